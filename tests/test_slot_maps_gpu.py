"""The step's slot maps (apt_step.cuh): a cell's merge is kept from step to step and
redone only where a list its stencil reads changed.  Whatever changes a list has to
be seen: the states and overflow counts equal the CPU oracle's, which merges every
cell every step, bit for bit.

* crowded random lists with holes and repeated ids (set_slots accepts them), more
  grains than slots, every slot count, boundary code and tile edge;
* undercooling that leaves cells unwritten (types 3 and 4), whose lists are those of
  two steps before;
* tile shape, z chunk and quiet items switched between steps, state replaced;
* a server request whose budget has no room for maps.
"""
import numpy as np
import pytest

from cupf_b200 import cases
from cupf_b200.server import Server
from cupf_b200.solver import APTSolver
from tests.helpers import compare_states

pytestmark = pytest.mark.gpu


def crowded(c, seed, grains, empty=0.35):
    """Random slots: each cell's slots hold random grains (repeats and holes among
    them) with random phi, in clumps of a few cells."""
    p = c.params
    rng = np.random.default_rng(seed)
    shp = (p.num_pf, p.fnz, p.fny, p.fnx)
    coarse = [max(1, (n + 2) // 3) for n in shp[1:]]
    ids = rng.integers(1, grains + 1, (p.num_pf, *coarse)).astype(np.int32)
    ids[rng.random(ids.shape) < empty] = -1
    for ax, n in enumerate(shp[1:]):
        ids = np.repeat(ids, 3, axis=ax + 1).take(range(n), axis=ax + 1)
    flip = rng.random(shp) < 0.05
    ids[flip] = rng.integers(1, grains + 1, int(flip.sum()))
    ids[:, shp[1] // 2:] = np.where(rng.random(ids[:, shp[1] // 2:].shape) < 0.7, -1,
                                    ids[:, shp[1] // 2:])
    ph = np.where(ids >= 0, rng.uniform(-0.99995, 1.0, shp), -1.0).astype(np.float32)
    ph, ids = ph.reshape(-1).copy(), ids.reshape(-1).copy()
    cases.fill_bc(p, ph, ids)
    return ph, ids


SHAPES = [((33, 9, 18), 1, "111"), ((31, 17, 13), 2, "000"), ((34, 16, 20), 3, "101"),
          ((32, 8, 21), 4, "110"), ((65, 7, 17), 5, "011"), ((3, 25, 19), 6, "010"),
          ((40, 12, 16), 7, "100"), ((38, 23, 24), 8, "110"), ((36, 18, 20), 8, "001")]


@pytest.mark.parametrize("spec", SHAPES, ids=lambda s: "%dx%dx%d_np%d_%s" % (*s[0], s[1], s[2]))
def test_crowded_lists_match_oracle(built, spec):
    from oracle import CpuOracle
    interior, npf, bc = spec
    c = cases.line_case(*interior, num_pf=npf, num_grains=12, seed=3, bc=bc)
    ph0, id0 = crowded(c, npf, 12)
    stats = np.zeros(2, np.int64)
    o_ph, o_id, _, _ = CpuOracle().run_f32(c, ph0, id0, 9, stats=stats)
    with APTSolver(c) as s:
        s.set_slots(ph0, id0, 0)
        s.merge_overflows()
        for _ in range(9):
            s.step(1)
        ovf = s.merge_overflows()
        ph, ids = s.get_slots()
    assert compare_states(c.params, ph, ids, o_ph, o_id)[:2] == (0, 0)
    assert ovf == (int(stats[0]), int(stats[1]))


@pytest.mark.parametrize("kind", ["cone", "paraboloid"])
def test_unwritten_cells_match_oracle(built, kind):
    from oracle import CpuOracle
    # a cone angle at which the device's tanf and cosf equal the C library's (the
    # undercooling then agrees bit for bit, as the comparison needs)
    extra = {"angle": 0.8} if kind == "cone" else {}
    make = cases.cone_case if kind == "cone" else cases.paraboloid_case
    c = make(44, 19, 28, num_pf=4, num_grains=25, seed=5, bc="110", **extra)
    ph0, id0 = crowded(c, 7, 25, empty=0.6)
    o_ph, o_id, _, _ = CpuOracle().run_f32(c, ph0, id0, 14)
    with APTSolver(c) as s:
        s.set_slots(ph0, id0, 0)
        s.step(14)
        ph, ids = s.get_slots()
    assert compare_states(c.params, ph, ids, o_ph, o_id)[:2] == (0, 0)


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
def test_switches_and_replaced_state_between_steps(built, precision):
    c = cases.line_case(50, 38, 44, num_pf=6, num_grains=40, seed=9, bc="110")
    other = cases.line_case(50, 38, 44, num_pf=6, num_grains=40, seed=10, bc="110")
    with APTSolver(c, precision=precision) as s:
        s.init_from_argmax(c.phi, c.alpha)
        s.step(60)
        want = s.get_slots()
    with APTSolver(c, precision=precision) as s:
        s.init_from_argmax(other.phi, other.alpha)  # another run's maps first
        s.step(25)
        s.init_from_argmax(c.phi, c.alpha)
        for n, change in ((7, lambda: s.set_skip_quiet(False)), (8, lambda: s.set_tile(4)),
                          (9, lambda: s.set_tuning(3)), (11, lambda: s.set_skip_quiet(True)),
                          (12, lambda: s.set_tile(8)), (13, lambda: None)):
            s.step(n)
            change()
        got = s.get_slots()
    assert np.array_equal(got[1], want[1])
    assert np.array_equal(got[0].view(np.uint32), want[0].view(np.uint32))


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
def test_server_without_room_for_maps(built, precision):
    c = cases.line_case(48, 44, 40, num_pf=8, num_grains=20, seed=1)
    p = c.params
    pair, align = (8, 2) if precision == "fp32" else (4, 4)
    xp = -(-p.fnx // align) * align
    need = (2 * xp * p.fny * p.fnz * p.num_pf * pair + p.fnx * p.fny * p.fnz * 8 +
            2 * -(-(p.fnx - 2) // 32) * -(-(p.fny - 2) // 4) * (p.fnz - 2) + 4096)
    out = []
    for budget in (need, 0):
        with Server(precision=precision, steps_per_round=16, autotune=False,
                    hbm_budget_bytes=budget) as srv:
            r = srv.submit(c, 70)
            srv.run_until_done([r])
            out.append(srv.result(r))
    assert np.array_equal(out[0]["alpha"], out[1]["alpha"]) and out[0]["qoi"] == out[1]["qoi"]
