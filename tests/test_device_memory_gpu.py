"""Device memory that runs out, on the host alone: a child process is started with
tests/native/alloc_limit.c before the CUDA runtime, which refuses allocations.

A call that cannot have its memory reports it, leaves the handle as it was and
works once there is room; what a call allocates together it has whole or not at
all.  The step's slot maps are optional: they are given back to whatever else needs
the room, and the results are the same without them.
"""
import ctypes as C
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from cupf_b200 import abi, cases
from cupf_b200.dense import DenseSolver
from cupf_b200.server import Server
from cupf_b200.solver import APTSolver
from tests.test_slot_maps_gpu import SHAPES, crowded

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
OOM = 3  # CUPF_ERR_OOM


@pytest.fixture(scope="module")
def child(built, tmp_path_factory):
    """Run a function of this module in a process whose allocations can be refused."""
    so = str(tmp_path_factory.mktemp("alloc") / "alloc_limit.so")
    subprocess.run(["gcc", "-O2", "-shared", "-fPIC", "-o", so,
                    os.path.join(ROOT, "tests", "native", "alloc_limit.c"), "-ldl", "-lpthread"],
                   check=True)

    def run(name):
        r = subprocess.run([sys.executable, "-c",
                            "import tests.test_device_memory_gpu as t; t.%s(); print('done')" % name],
                           cwd=ROOT, env=dict(os.environ, LD_PRELOAD=so), capture_output=True,
                           text=True, timeout=300)
        assert r.returncode == 0 and r.stdout.endswith("done\n"), r.stdout + r.stderr
    return run


def shim():
    s = C.CDLL(None)
    s.alloc_refuse_from.argtypes = [C.c_long]
    s.alloc_limit.argtypes = [C.c_size_t]
    s.alloc_live.restype = C.c_size_t
    s.alloc_refused.restype = C.c_long
    return s


def refused(a, n, call, *args):
    """The call with all but its first n allocations refused."""
    a.alloc_refuse_from(n)
    with pytest.raises(abi.CupfError) as e:
        call(*args)
    a.alloc_refuse_from(-1)
    assert e.value.status == OOM


def same(a, b):
    assert np.array_equal(a[1], b[1])
    assert np.array_equal(a[0].view(np.uint32), b[0].view(np.uint32))


def line(seed=5):
    return cases.line_case(64, 40, 96, num_pf=5, num_grains=30, seed=seed, bc="110")


def scratch_refused():
    """The second buffer of the read-back scratch refused: set_slots and get_slots fail,
    the state goes on as if they had not been called, and both work afterwards."""
    a, c = shim(), line()
    with APTSolver(c) as s:
        s.init_from_argmax(c.phi, c.alpha)
        s.step(30)
        ph, ids = s.get_slots()
        s.step(21)
        want = s.get_slots()
    # a state of few occupied planes: another item shape than the running one's
    low = np.where(np.arange(ph.size) % (c.params.fnx * c.params.fny * c.params.fnz) <
                   3 * c.params.fnx * c.params.fny, ids, -1).astype(np.int32)
    with APTSolver(c) as s:
        s.init_from_argmax(c.phi, c.alpha)
        s.step(30)
        for n in (0, 1):
            refused(a, n, s.set_slots, ph, low, 0)
            s.step(7)
            refused(a, n, s.get_slots)
        s.step(7)
        same(s.get_slots(), want)
        s.set_slots(ph, ids, 30)
        s.step(21)
        same(s.get_slots(), want)


def moves(solver, c, a):
    """Steps and frame moves, the second past the archive's first capacity; with `a`
    every allocation on the way is refused at first."""
    solver.step(20)
    for n in (0, 1) if a else ():
        refused(a, n, solver.move_domain, 1, 10 ** 6, 0)
    tip, _, _ = solver.move_domain(1, 10 ** 6, 0)
    out = [solver.move_domain(tip, tip - 2, 0)]
    solver.step(9)
    mc = 4 * c.params.fnz + 5  # two layers fit, four more are moved
    if a:
        refused(a, 0, solver.move_domain, tip, tip - 3, mc)
    out.append(solver.move_domain(tip, tip - 3, mc))
    assert out[0][2] >= 3 and out[1][2] >= 4
    solver.step(9)
    return out, solver.get_archive(8 * c.params.fnz), solver.get_slots()


def archive_refused():
    c = line()
    got = []
    for a in (None, shim()):
        with APTSolver(c) as s:
            s.init_from_argmax(c.phi, c.alpha)
            got.append(moves(s, c, a))
    assert got[0][0] == got[1][0]
    for u, v in zip(got[0][1], got[1][1]):
        assert np.array_equal(u, v)
    same(got[0][2], got[1][2])


def volumes_and_nuclei_refused():
    a, c = shim(), line()
    p = c.params
    p.nuc_rad, p.pts_cell, p.nuc_Nmax0, p.nuc_Nmax = 0.16, 2, 5.0, 5.0
    with APTSolver(c) as s:
        s.init_from_argmax(c.phi, c.alpha)
        s.step(5)
        _, alpha = s.collect(clear=True)
        for n in (0, 1):
            refused(a, n, s.grain_volumes, p.num_theta)
        v = s.grain_volumes(p.num_theta)
        inner = alpha.reshape(p.fnz, p.fny, p.fnx)[1:-1, 1:-1, 1:-1]
        assert np.array_equal(v[1:], np.bincount(inner.ravel(), minlength=p.num_theta + 1)[1:])
        for n in (0, 1, 2):
            refused(a, n, s.nucl_init)
        s.nucl_init()
        s.nucleate()
        s.step(2)
        s.sync()


@pytest.mark.parametrize("name", ["scratch_refused", "archive_refused", "volumes_and_nuclei_refused"])
def test_refused_allocations_leave_the_handle_whole(child, name):
    child(name)


def map_bytes(p, precision="fp32"):
    align = 2 if precision == "fp32" else 4
    return -(-p.fnx // align) * align * p.fny * p.fnz * (4 * p.num_pf + 2)


def whole_run(s, c, state):
    """Every call that allocates on the way."""
    s.set_slots(*state, 0)
    s.step(20)
    tip, mc, _ = s.move_domain(1, 10 ** 6, 0)
    moved = s.move_domain(tip, tip - 1, mc)
    s.step(11)
    phi, alpha = s.collect(clear=True)
    return (moved, alpha, phi, s.grain_volumes(c.params.num_theta), s.qoi_sums(),
            *s.get_slots())


def equal(a, b):
    for u, v in zip(a, b):
        assert np.array_equal(np.asarray(u), np.asarray(v))


def maps_give_way():
    """A device that holds the simulation and all it allocates later, but not its maps
    too: every call succeeds, for this handle, a second one and the full-PF solver."""
    a, c = shim(), line()
    with APTSolver(c) as s:
        s.init_from_argmax(c.phi, c.alpha)
        state = s.get_slots()
    for prec in ("fp32", "fp16"):
        with APTSolver(c, precision=prec) as s:
            want = whole_run(s, c, state)
            need = a.alloc_live() - map_bytes(c.params, prec)
        a.alloc_limit(need + 4096)
        with APTSolver(c, precision=prec) as s:
            held = a.alloc_live()
            got = whole_run(s, c, state)
            assert a.alloc_refused() > 0
            assert a.alloc_live() == need
        equal(got, want)
        # the maps were there before the scratch was
        with APTSolver(c, precision=prec) as s:
            s.init_from_argmax(c.phi, c.alpha)
            assert a.alloc_live() == held
        # refused from the start: the same states
        a.alloc_limit(held - 1)
        with APTSolver(c, precision=prec) as s:
            assert a.alloc_live() == held - map_bytes(c.params, prec)
            a.alloc_limit(0)
            equal(whole_run(s, c, state), want)
    a.alloc_limit(2 * need + 4096)
    with APTSolver(c, precision="fp16") as s, APTSolver(c, precision="fp16") as t:
        equal(whole_run(s, c, state), want)
        equal(whole_run(t, c, state), want)
    a.alloc_limit(0)
    d = cases.line_case(24, 24, 32, num_pf=1, num_grains=6, seed=1)
    with DenseSolver(d):
        full = a.alloc_live()
    with APTSolver(c) as s:
        s.init_from_argmax(c.phi, c.alpha)
        a.alloc_limit(a.alloc_live() + full - 1)
        with DenseSolver(d):
            s.step(5)
            s.sync()


def maps_give_way_across_threads():
    """A second simulation created while the first is stepping in another thread."""
    a, c = shim(), line()
    with APTSolver(c) as s:
        s.init_from_argmax(c.phi, c.alpha)
        s.step(1000)
        want = s.collect(clear=True)
        need = a.alloc_live() - map_bytes(c.params)
    a.alloc_limit(2 * need + 4096)
    with APTSolver(c) as s:
        s.init_from_argmax(c.phi, c.alpha)
        go = threading.Thread(target=lambda: [s.step(10) for _ in range(100)])
        go.start()
        with APTSolver(c) as t:
            t.init_from_argmax(c.phi, c.alpha)
            t.step(1000)
            equal(t.collect(clear=True), want)
        go.join()
        equal(s.collect(clear=True), want)


def captured_steps_keep_their_maps():
    """Steps captured in a graph on the handle's stream: the maps they point to are not
    given back afterwards, and the graph's steps are the steps."""
    a, c = shim(), line()
    with APTSolver(c) as s:
        s.init_from_argmax(c.phi, c.alpha)
        s.step(12)
        want = s.get_slots()
    rt = C.CDLL("libcudart.so.12")
    graph, run = C.c_void_p(), C.c_void_p()
    with APTSolver(c) as s:
        s.init_from_argmax(c.phi, c.alpha)
        s.step(10)
        s.sync()
        stream = C.c_void_p(s.stream)
        assert rt.cudaStreamBeginCapture(stream, 2) == 0  # relaxed
        with APTSolver(c) as other:  # created while the stream is being captured
            refused(a, 0, other.set_slots, *want)
            s.step(2)
        assert rt.cudaStreamEndCapture(stream, C.byref(graph)) == 0
        assert rt.cudaGraphInstantiate(C.byref(run), graph, C.c_ulonglong(0)) == 0
        live = a.alloc_live()
        refused(a, 0, s.get_slots)
        assert a.alloc_live() == live
        assert rt.cudaGraphLaunch(run, stream) == 0
        s.sync()
        same(s.get_slots(), want)
        assert rt.cudaGraphExecDestroy(run) == 0 and rt.cudaGraphDestroy(graph) == 0


def forms_of_the_merge():
    """Crowded lists (holes, repeated ids, more grains than slots) with and without maps:
    rows merged by the warp's passes, by their own lanes, and both."""
    a = shim()
    for interior, npf, bc in SHAPES:
        c = cases.line_case(*interior, num_pf=npf, num_grains=12, seed=3, bc=bc)
        ph, ids = crowded(c, npf, 12)
        for prec in ("fp32", "fp16", "bf16"):
            for tile in (8, 4):
                got = []
                for maps in (True, False):
                    with APTSolver(c, precision=prec) as s:
                        live = a.alloc_live()
                    a.alloc_limit(0 if maps else live - 1)
                    with APTSolver(c, precision=prec) as s:
                        assert (a.alloc_live() == live) == maps
                        a.alloc_limit(0)
                        s.set_tile(tile)
                        s.set_slots(ph, ids, 0)
                        s.merge_overflows()
                        s.step(11)
                        got.append((s.merge_overflows(), *s.get_slots()))
                    if not maps:
                        equal(got[0], got[1])


@pytest.mark.parametrize("name", ["maps_give_way", "maps_give_way_across_threads",
                                  "captured_steps_keep_their_maps", "forms_of_the_merge"])
def test_slot_maps_give_way(child, name):
    child(name)


RUNNING = 1
REQUESTS = [((48, 44, 40), 1), ((40, 56, 48), 2), ((56, 40, 64), 3)]


def request(shape, seed):
    return cases.line_case(*shape, num_pf=8, num_grains=20, seed=seed)


def required(c, precision):
    """Bytes a request is admitted by (its maps are not among them)."""
    p = c.params
    pair, align = (8, 2) if precision == "fp32" else (4, 4)
    xp = -(-p.fnx // align) * align
    return (2 * xp * p.fny * p.fnz * p.num_pf * pair + p.fnx * p.fny * p.fnz * 8 +
            2 * -(-(p.fnx - 2) // 32) * -(-(p.fny - 2) // 4) * (p.fnz - 2) + 4096)


def server(precision, **kw):
    return Server(precision=precision, steps_per_round=16, autotune=False, **kw)


def alone(cs, precision):
    out = []
    for c in cs:
        with server(precision) as srv:
            r = srv.submit(c, 70)
            srv.run_until_done([r])
            out.append(srv.result(r))
    return out


def check_results(srv, rids, want):
    srv.run_until_done(rids)
    for r, w in zip(rids, want):
        got = srv.result(r)
        assert np.array_equal(got["alpha"], w["alpha"]) and got["qoi"] == w["qoi"]


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
def test_maps_never_hold_up_a_later_request(built, precision):
    """Requests that fit the budget together, submitted one after the other while the
    earlier ones hold slot maps, are all resident at once."""
    cs = [request(*r) for r in REQUESTS]
    want = alone(cs, precision)
    need = [required(c, precision) for c in cs]
    assert need[0] + map_bytes(cs[0].params, precision) <= sum(need[:2])
    for several in (2, 3):
        with server(precision, hbm_budget_bytes=sum(need[:several])) as srv:
            rids = []
            for c in cs[:several]:
                rids.append(srv.submit(c, 70))
                srv.pump()
                assert srv.status(rids[-1]) == RUNNING
            check_results(srv, rids, want)


def served_without_map_memory():
    """The device refuses the maps' memory to a request, or needs a resident one's back
    for the next: both requests run, with the same results."""
    a = shim()
    cs = [request(*r) for r in REQUESTS[:2]]
    for precision in ("fp32", "fp16"):
        want = alone(cs, precision)
        maps = [map_bytes(c.params, precision) for c in cs]
        with server(precision) as srv:
            empty = a.alloc_live()
            rids = []
            held = []
            for c in cs:
                rids.append(srv.submit(c, 70))
                srv.pump()
                held.append(a.alloc_live())
            check_results(srv, rids, want)
        for limit in (held[0] - 1, held[0] - maps[0] // 2, held[1] - sum(maps) + 65536):
            before = a.alloc_refused()
            with server(precision) as srv:
                assert a.alloc_live() <= empty
                rids = [srv.submit(cs[0], 70)]
                a.alloc_limit(limit)
                srv.pump()
                a.alloc_limit(held[1] - sum(maps) + 65536)
                rids.append(srv.submit(cs[1], 70))
                srv.pump()
                assert [srv.status(r) for r in rids] == [RUNNING, RUNNING]
                assert a.alloc_refused() > before
                a.alloc_limit(0)
                check_results(srv, rids, want)


@pytest.mark.parametrize("name", ["served_without_map_memory"])
def test_server_without_map_memory(child, name):
    child(name)
