"""The 2D march at the edges of its strips (30 columns a warp) and row chunks (2 to 32
rows), with a rotated crystal: a few steps of every interior cell, in every storage with
noise against the FP64 oracle, and in FP64 without noise against a restatement whose
constants are formed in double like the library's."""
import numpy as np
import pytest

from cupf_b200 import ek2d
from cupf_b200.ek2d import EK2DSolver
from oracle import Ek2dOracle

pytestmark = pytest.mark.gpu

STEPS = 6
SIZES = [(8, 10), (29, 33), (30, 31), (31, 64), (59, 20), (60, 97), (61, 40), (90, 130)]


def case(size, eta):
    nx, ny = size
    return ek2d.directional_case(nx, ny, 40, front_frac=0.5, sites=2, amp=0.4, eta=eta, alpha0=20.0,
                                 seed=11, asp_ratio=(ny + 0.5) / nx)


def run(c, prec):
    with EK2DSolver(c, precision=prec) as sv:
        sv.set_state(c.psi, c.U)
        sv.prestep()
        sv.step(STEPS)
        return sv.get_state_f64()


def flux_size(c):
    """Size of the terms whose sum is a cell's rate: hi^2 times the largest difference."""
    psi = np.asarray(c.psi).reshape(c.fny, c.fnx)[1:-1, 1:-1]
    step = max(float(np.abs(np.diff(psi, axis=axis)).max()) for axis in (0, 1))
    return max(1.0, step) * float(c.params.hi) ** 2


@pytest.mark.parametrize("prec", ["fp32", "fp64", "fp16", "bf16"])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "%dx%d" % s)
def test_march_edges_match_oracle(built, size, prec):
    c = case(size, 0.02)
    o = Ek2dOracle()
    s = o.new_state(c, np.float64)
    o.run(c, s, STEPS, prestep=True)
    d = run(c, prec)
    inner = np.s_[1:-1, 1:-1]
    # Per step, psi and U round once at their own size and take dt times a rate built
    # from a few dozen rounded operations on fluxes of size hi^2 |dpsi| (the hardware
    # approximations add an ulp or two each): 64 roundings of that size a step.  The
    # rates' roundings are FP32 ones in FP64 runs too: the oracle forms some of its
    # constants from the float parameters in float (1e-9 from the library's FP64 run).
    eps, eps32 = 2.0 ** (-52 if prec == "fp64" else -24), 2.0 ** -24
    p = c.params
    rates = 64 * eps32 * float(p.dt) * flux_size(c)
    names = ("psi", "U") if prec in ("fp32", "fp64") else ("phi", "U")
    for name in names:
        size_of = float(np.abs(s[name][inner]).max())
        per_step = 4 * eps * size_of + rates
        if prec in ("fp16", "bf16"):
            # 16-bit storage rounds stochastically, by less than a unit in the last place
            # (2^-10 or 2^-7 of the value).  phi: FP16 stores psi, and 2^-10 |psi| moves
            # phi = tanh(psi / sqrt2) by at most 0.45 of 2^-10; BF16 stores 1 - |phi| <= 1.
            # U is stored less U0, at most 1 + the largest change.  A step carries the
            # error of the one before on, at most doubled by the neighbours' (cfl 0.2), and
            # a cell at the edge of the noise band may get its noise in one run only.
            ulp = 2.0 ** (-10 if prec == "fp16" else -7)
            stored = (0.45 if prec == "fp16" else 1.0) if name == "phi" else \
                float(np.abs(s["U"][inner] - float(p.U0)).max())
            noise = 0.5 * float(p.dt_sqrt) * float(p.hi) * 0.02 * (1.0 - 0.995 ** 2)
            per_step = 2.0 * (ulp * stored + noise) + rates
        err = float(np.abs(d[name][inner] - s[name][inner]).max())
        assert err <= (STEPS + 1) * per_step, (name, err, (STEPS + 1) * per_step)


def restated(c):
    """The model's step in numpy doubles: edge fluxes of psi (anisotropic) and of U (with
    the anti-trapping current), U first, then psi with the new U (PF.cu:440-598)."""
    p = c.params
    f = lambda n: float(getattr(p, n))
    k, hi, sq2, dt, eps = f("k"), f("hi"), f("sqrt2"), f("dt"), f("eps")
    ps, U = (np.asarray(a, np.float32).astype(np.float64).reshape(c.fny, c.fnx) for a in (c.psi, c.U))
    D = np.zeros_like(ps)

    def halo(a):
        a[:, 0], a[:, -1] = a[:, -2], a[:, 1]
        a[0], a[-1] = a[2], a[-3]
        return a

    def anisotropy(x, z):
        ux, uz = f("cosa") * x + f("sina") * z, f("cosa") * z - f("sina") * x
        m = ux * ux + uz * uz
        i = np.where(m > eps, 1.0 / np.where(m > eps, m * m, 1.0), 0.0)
        return (np.where(m > eps, f("a_s") * (1 + f("epsilon") * (ux ** 4 + uz ** 4) * i), 1.0),
                -f("a_12") * ux * uz * (ux * ux - uz * uz) * i)

    def normal(n, x, z):
        m = x * x + z * z
        return np.where(m > eps, n / np.sqrt(np.where(m > eps, m, 1.0)), 0.0)

    def edges(axis):
        """psi and U fluxes of the edges along x (axis 1) or y (axis 0)."""
        cut = (slice(1, -1), slice(None)) if axis == 1 else (slice(None), slice(1, -1))
        lo, up = (slice(None, -1), slice(1, None))
        at = lambda a, s: a[cut][(slice(None), s) if axis == 1 else (s, slice(None))]
        diff = lambda a: at(a, up) - at(a, lo)
        q = lambda a: np.diff(0.25 * (a[:-1, :-1] + a[:-1, 1:] + a[1:, :-1] + a[1:, 1:]), axis=1 - axis)
        n_ps, t_ps, n_ph, t_ph = diff(ps), q(ps), diff(ph), q(ph)
        x, z = (n_ph, t_ph) if axis == 1 else (t_ph, n_ph)
        A, Ap = anisotropy(x, z)
        J = A * (A * n_ps + (Ap if axis == 0 else -Ap) * t_ps)
        F = (0.5 * hi * f("Dl_tilde") * (2 - at(ph, lo) - at(ph, up)) * diff(U) +
             0.5 * (at(jat, lo) + at(jat, up)) * normal(n_ph, x, z))
        return np.diff(J, axis=axis), np.diff(F, axis=axis)

    halo(ps), halo(U)
    t0, t1 = (float(t) for t in c.t_mac[:2])
    pulled = 0.0
    rows = np.arange(c.fny, dtype=np.float64)[1:-1, None]
    for n in range(STEPS + 1):  # n = 0: the step before the loop, psi alone
        R, G = 0.0, float(c.Gt[0])
        if n:
            w = (n * dt * f("tau0") - t0) / (t1 - t0)
            R, G = ((1 - w) * float(a[0]) + w * float(a[1]) for a in (c.Rt, c.Gt))
        pulled += R * f("tau0") / f("W0") * dt
        ph = np.tanh(ps / sq2)
        jat = 0.5 * (1 + (1 - k) * U) * (1 - ph * ph) * D
        (xJ, xF), (yJ, yF) = edges(1), edges(0)
        i = np.s_[1:-1, 1:-1]
        Un = U[i]
        if n:
            Un = Un + dt * ((xF + yF) * hi + sq2 * jat[i]) / (1 + k - (1 - k) * ph[i])
        grad = lambda a: (0.5 * (a[1:-1, 2:] - a[1:-1, :-2]), 0.5 * (a[2:, 1:-1] - a[:-2, 1:-1]))
        A2 = anisotropy(*grad(ph))[0] ** 2
        gx, gz = grad(ps)
        lT = f("c_infm") * (1 / k - 1) / G / f("W0")
        Up = ((p.y0 + (rows - 1) * (f("dx") * f("W0"))) / f("W0") - pulled) / lT
        rhs = ((xJ + yJ - sq2 * A2 * ph[i] * (gx * gx + gz * gz)) * hi * hi + sq2 * ph[i] -
               f("lamd") * (1 - ph[i] ** 2) * sq2 * (Un + Up))
        d = rhs / (np.maximum(1 - (1 - k) * Up, k) * A2)
        ps[i], U[i], D[i] = ps[i] + dt * d, Un, d
        halo(ps), halo(U), halo(D)
    return {"psi": ps, "U": U}


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "%dx%d" % s)
def test_march_edges_match_double_restatement(built, size):
    c = case(size, 0.0)
    want, got = restated(c), run(c, "fp64")
    # roundings as above, all of them FP64 ones
    eps = 2.0 ** -52
    for name in ("psi", "U"):
        tol = (STEPS + 1) * (4 * eps * float(np.abs(want[name]).max()) +
                             64 * eps * float(c.params.dt) * flux_size(c))
        err = float(np.abs(got[name] - want[name])[1:-1, 1:-1].max())
        assert err <= tol, (name, err, tol)
