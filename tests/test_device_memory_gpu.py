"""Device memory that runs out, on the host alone: a child process is started with
tests/native/alloc_limit.c before the CUDA runtime, which refuses allocations.

A call that cannot have its memory reports it, leaves the handle as it was and
works once there is room; what a call allocates together it has whole or not at
all.
"""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

from cupf_b200 import abi, cases
from cupf_b200.solver import APTSolver

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
    s.alloc_fail_next.argtypes = [C.c_long]
    s.alloc_limit.argtypes = [C.c_size_t]
    s.alloc_live.restype = C.c_size_t
    s.alloc_refused.restype = C.c_long
    return s


def refused(call, *args):
    with pytest.raises(abi.CupfError) as e:
        call(*args)
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
            a.alloc_fail_next(n)
            refused(s.set_slots, ph, low, 0)
            s.step(7)
            a.alloc_fail_next(n)
            refused(s.get_slots)
        s.step(7)
        same(s.get_slots(), want)
        s.set_slots(ph, ids, 30)
        s.step(21)
        same(s.get_slots(), want)


def moves(solver, c, a):
    """Steps and frame moves, the second past the archive's first capacity; with `a`
    every allocation on the way is refused once."""
    solver.step(20)
    for n in (0, 1) if a else ():
        a.alloc_fail_next(n)
        refused(solver.move_domain, 1, 10 ** 6, 0)
    tip, _, _ = solver.move_domain(1, 10 ** 6, 0)
    out = [solver.move_domain(tip, tip - 2, 0)]
    solver.step(9)
    mc = 4 * c.params.fnz + 5  # two layers fit, four more are moved
    if a:
        a.alloc_fail_next(0)
        refused(solver.move_domain, tip, tip - 3, mc)
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
            a.alloc_fail_next(n)
            refused(s.grain_volumes, p.num_theta)
        v = s.grain_volumes(p.num_theta)
        inner = alpha.reshape(p.fnz, p.fny, p.fnx)[1:-1, 1:-1, 1:-1]
        assert np.array_equal(v[1:], np.bincount(inner.ravel(), minlength=p.num_theta + 1)[1:])
        for n in (0, 1, 2):
            a.alloc_fail_next(n)
            refused(s.nucl_init)
        s.nucl_init()
        s.nucleate()
        s.step(2)
        s.sync()


@pytest.mark.parametrize("name", ["scratch_refused", "archive_refused", "volumes_and_nuclei_refused"])
def test_refused_allocations_leave_the_handle_whole(child, name):
    child(name)
