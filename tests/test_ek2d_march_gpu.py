"""The 2D march at the edges of its strips (30 columns a warp) and row chunks (2 to 32
rows), with a rotated crystal and noise: a few steps of every interior cell against the
FP64 oracle."""
import numpy as np
import pytest

from cupf_b200 import ek2d
from cupf_b200.ek2d import EK2DSolver
from oracle import Ek2dOracle

pytestmark = pytest.mark.gpu

STEPS = 6
SIZES = [(8, 10), (29, 33), (30, 31), (31, 64), (59, 20), (60, 97), (61, 40), (90, 130)]


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "%dx%d" % s)
def test_march_edges_match_oracle(built, size, prec):
    nx, ny = size
    c = ek2d.directional_case(nx, ny, 40, front_frac=0.5, sites=2, amp=0.4, eta=0.02, alpha0=20.0,
                              seed=11, asp_ratio=(ny + 0.5) / nx)
    o = Ek2dOracle()
    s = o.new_state(c, np.float64)
    o.run(c, s, STEPS, prestep=True)
    with EK2DSolver(c, precision=prec) as sv:
        sv.set_state(c.psi, c.U)
        sv.prestep()
        sv.step(STEPS)
        d = sv.get_state_f64()
    inner = np.s_[1:-1, 1:-1]
    # Per step, psi and U round once at their own size and take dt times a rate built
    # from a few dozen rounded operations on fluxes of size hi^2 |dpsi| (the hardware
    # approximations add an ulp or two each): 64 roundings of that size a step.  The
    # rates' roundings are FP32 ones in FP64 runs too: the oracle forms some of its
    # constants from the float parameters in float (the device's FP64 run is within
    # 1e-14 of a restatement that forms them in double, the oracle 1e-9 from both).
    eps, eps32 = 2.0 ** (-24 if prec == "fp32" else -52), 2.0 ** -24
    p = c.params
    flux = max(1.0, float(np.abs(np.diff(c.psi, axis=0)).max())) * float(p.hi) ** 2
    for name in ("psi", "U"):
        size_of = float(np.abs(s[name][inner]).max())
        tol = (STEPS + 1) * (4 * eps * size_of + 64 * eps32 * float(p.dt) * flux)
        err = float(np.abs(d[name][inner] - s[name][inner]).max())
        assert err <= tol, (name, err, tol)
