"""The tile height the library picks when a state is loaded: on small line cases on both
sides of its rule the step is not slower than with the other height (each with the z chunk
that the library picks for it)."""
import pytest

from cupf_b200 import cases
from cupf_b200.solver import APTSolver

pytestmark = pytest.mark.gpu


def step_time(c, tile):
    with APTSolver(c) as s:
        if tile:
            s.set_tile(tile)
        s.init_from_argmax(c.phi, c.alpha)
        s.step(50)
        return min(s.time_steps(50) for _ in range(5))


@pytest.mark.parametrize("grid,num_pf,grains", [((24, 24, 32), 5, 10), ((40, 40, 40), 8, 15),
                                                ((48, 48, 48), 8, 20), ((64, 64, 128), 8, 40),
                                                ((64, 64, 64), 6, 35), ((64, 64, 128), 5, 40)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else str(v))
def test_chosen_height_is_the_faster_one(built, grid, num_pf, grains):
    c = cases.line_case(*grid, num_pf=num_pf, num_grains=grains, seed=0, bc="110")
    # runs of one height differ by a percent or two, the heights by 5 to 30
    assert step_time(c, 0) <= 1.08 * min(step_time(c, 8), step_time(c, 4))
