"""Performance cases of the framework's solvers, through their public entry points.

Each case is one pass of a user's program: a solver that is already set up
(`prepare`) advances by some steps and its result is read back (`run`), the way
the drivers' loops and the benchmark call it.  A pass leaves the solver in the
advanced state, so the next pass carries the same simulation on.

Families:
  line    3D APT directional solidification (cupf_b200.solver.APTSolver): steps,
          then the argmax fields, the grain volumes and the interface sums;
  pool    3D APT melt pool: the driver's loop of step, nucleation pass, frame
          check every 20 steps, step;
  dense   one phase field per grain (cupf_b200.dense.DenseSolver);
  ek2d    the 2D Echebarria-Karma line model (cupf_b200.ek2d.EK2DSolver);
  serve   a burst of requests through the batching server (cupf_b200.server).

`exact` restates each family's step in plain torch, in 64 bits.
"""
import math

import numpy as np
import torch

from cupf_b200 import cases, ek2d
from cupf_b200.dense import DenseSolver
from cupf_b200.ek2d import EK2DSolver
from cupf_b200.server import DONE, Server
from cupf_b200.solver import APTSolver

LS = -0.995          # a cell is solid above this phi
ID_DROP = -0.9999    # a slot loses its grain id below this phi
GRAINS_PER_AREA = 600.0 / (256 * 256)  # grain density of the 600-grain line workload
FRAME_CHECK = 20     # steps between the melt-pool loop's frame checks


def _line(name, nx, ny, nz, grains, num_pf, prec, steps, bc="110"):
    c = dict(kind="line", nx=nx, ny=ny, nz=nz, grains=grains, num_pf=num_pf, prec=prec,
             steps=steps, bc=bc)
    return dict(name=name, **c) if name else c


def _pool(name, nx, ny, nz, grains, prec, steps):
    c = dict(kind="pool", nx=nx, ny=ny, nz=nz, grains=grains, num_pf=8, prec=prec, steps=steps)
    return dict(name=name, **c) if name else c


def _dense(name, nx, ny, nz, grains, steps):
    c = dict(kind="dense", nx=nx, ny=ny, nz=nz, grains=grains, steps=steps)
    return dict(name=name, **c) if name else c


def _ek2d(name, nx, ny, prec, steps):
    c = dict(kind="ek2d", nx=nx, ny=ny, prec=prec, steps=steps)
    return dict(name=name, **c) if name else c


def _serve(name, requests, prec, steps):
    c = dict(kind="serve", requests=requests, prec=prec, steps=steps)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a few steps on a very small grid with read-back: launches and host calls count
        _line("line_24x24x32_fp32", 24, 24, 32, 12, 5, "fp32", 10),
        # the small line workload: 20 grains, 5 slots per cell, 200 steps
        _line("line_64_fp32", 64, 64, 64, 20, 5, "fp32", 200),
        # a grid that no tile divides, mirrored in x, six slots per cell
        _line("line_117x75x139_fp32", 117, 75, 139, 80, 6, "fp32", 50, bc="010"),
        # the throughput workload: 600 grains, 8 slots per cell
        _line("line_256x256x512_fp32", 256, 256, 512, 600, 8, "fp32", 50),
        # split-precision storage at the size of a large served request
        _line("line_128x128x256_fp16", 128, 128, 256, 150, 8, "fp16", 100),
        # moving window with nucleation under the analytic melt pool
        _pool("pool_128x128x384_fp32", 128, 128, 384, 100, "fp32", 40),
        # one field per grain, the benchmark's size
        _dense("dense_128_80grains", 128, 128, 128, 80, 40),
        # one field per grain on a small odd grid
        _dense("dense_45x38x52_12grains", 45, 38, 52, 12, 50),
        # 2D directional solidification at full size, with its frame check
        _ek2d("ek2d_2048x8192_fp32", 2048, 8192, "fp32", 100),
        # the same in 16-bit storage on an odd grid
        _ek2d("ek2d_1000x2050_fp16", 1000, 2050, "fp16", 100),
        # the short runs and 64-bit precision that convergence checks use
        _ek2d("ek2d_128x512_fp64", 128, 512, "fp64", 100),
        # a burst of the served stream: eight requests of its four grid shapes
        _serve("serve_8_fp16", 8, "fp16", 100),
    ]


def draw(rng):
    """One more case of the ranges above (3D grids of 24 to 256 cells a side and up
    to 256x256x512, 2D grids of 100x200 to 2048x8192)."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["line", "line", "line", "pool", "dense", "ek2d", "ek2d"])
    if kind == "line":
        nx, ny, nz = size(24, 256), size(24, 256), size(32, 512)
        grains = max(10, int(GRAINS_PER_AREA * nx * ny * rng.uniform(0.3, 1.2)))
        return _line(None, nx, ny, nz, grains, rng.choice([4, 5, 6, 8, 8]),
                     rng.choice(["fp32", "fp32", "fp16", "bf16"]), rng.randrange(10, 50),
                     rng.choice(["110", "110", "010", "000"]))
    if kind == "pool":
        nx, ny, nz = size(48, 160), size(48, 160), size(96, 384)
        return _pool(None, nx, ny, nz, max(10, int(GRAINS_PER_AREA * nx * ny * 0.6)),
                     rng.choice(["fp32", "fp16"]), 20 * rng.randrange(1, 3))
    if kind == "dense":
        nx, ny, nz = size(32, 128), size(32, 128), size(32, 128)
        return _dense(None, nx, ny, nz, max(6, min(80, int(0.005 * nx * ny))),
                      rng.randrange(10, 40))
    return _ek2d(None, size(100, 2048), size(200, 8192), rng.choice(["fp32", "fp32", "fp16", "bf16"]),
                 rng.randrange(20, 100))


# ---------------------------------------------------------------- inputs

def _numbers(seed):
    """Seed of the substrate and orientations, and the gradient and pulling speed
    around the workloads' G = 1 K/um and R = 0.05 m/s."""
    rng = np.random.default_rng(seed)
    return int(rng.integers(0, 1 << 30)), float(rng.uniform(0.9, 1.1)), float(rng.uniform(0.045, 0.055))


def _line_case(case, seed):
    sub, G, R = _numbers(seed)
    return cases.line_case(case["nx"], case["ny"], case["nz"], num_pf=case.get("num_pf", 8),
                           num_grains=case["grains"], seed=sub, G=G, R=R,
                           bc=case.get("bc", "110"))


def _pool_case(case, seed):
    sub, G, _ = _numbers(seed)
    d = cases.derive_params({**cases.LINE_CONSTANTS, "R": 0.5})
    t_end = 20000 * float(d["dt"]) * float(d["tau0"])  # the workload's 20,000 steps
    # the pool's size goes with the window's (radius 60 um, length 120 um in 256 x 256 cells)
    r0 = 60.0 * min(case["nx"], case["ny"]) / 256.0
    return cases.meltpool_case(case["nx"], case["ny"], case["nz"], num_pf=case["num_pf"],
                               num_grains=case["grains"], seed=sub, r0=r0, mp_len=2 * r0, G=G,
                               t_end=t_end)


def _ek2d_case(case, seed):
    rng = np.random.default_rng(seed)
    nx, ny = case["nx"], case["ny"]
    return ek2d.directional_case(nx, ny, 2 * (case["steps"] // 2), sites=max(2, min(32, nx // 64)),
                                 amp=float(rng.uniform(0.008, 0.012)),
                                 seed=int(rng.integers(0, 1 << 30)),
                                 asp_ratio=(ny + 0.5) / nx)  # odd sizes: no rounding to ny - 1


def _serve_cases(case, seed):
    """Two requests of each of the stream's grid shapes, with its ranges of grain
    counts, gradients and pulling speeds."""
    rng = np.random.default_rng(seed)
    shapes = [(48, 48, 48), (96, 96, 96), (128, 128, 256), (192, 192, 192)]
    out = []
    for n in range(case["requests"]):
        out.append(cases.line_case(*shapes[n % len(shapes)], num_pf=8,
                                   num_grains=10 + 290 * n // max(1, case["requests"] - 1),
                                   seed=int(rng.integers(0, 10000)), G=float(rng.uniform(0.1, 10.0)),
                                   R=float(rng.uniform(0.01, 0.5)), bc="110"))
    return out


class _EK2D(EK2DSolver):
    def __del__(self):
        self.close()


class _Server(Server):
    def __del__(self):
        self.close()


def _pinned(n, dtype):
    return torch.empty(n, dtype=dtype, pin_memory=torch.cuda.is_available()).numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ek2d":
        c = _ek2d_case(case, seed)
        s = _EK2D(c, precision=case["prec"])
        s.set_state(c.psi, c.U)
        s.prestep()
        # FP64 results are read in FP64; the others into page-locked host arrays
        out = None if case["prec"] == "fp64" else [_pinned(c.fnx * c.fny, torch.float32)
                                                   for _ in range(4)]
        return {"case": case, "solver": s, "out": out}
    if kind == "serve":
        return {"case": case, "requests": _serve_cases(case, seed),
                "server": _Server(precision=case["prec"], num_pf=8, steps_per_round=50)}
    c = _pool_case(case, seed) if kind == "pool" else _line_case(case, seed)
    out = (_pinned(c.length, torch.float32), _pinned(c.length, torch.int32))
    if kind == "dense":
        s = DenseSolver(c)
        s.init_from_argmax(c.phi, c.alpha)
        s.prestep()
        return {"case": case, "solver": s, "out": out}
    s = APTSolver(c, precision=case["prec"])
    s.init_from_argmax(c.phi, c.alpha)
    if kind == "pool":
        s.nucl_init()
    return {"case": case, "solver": s, "out": out, "fnz": c.params.fnz, "tip": 1, "moves": 0,
            "done": 0}


def run(state):
    case = state["case"]
    kind, steps = case["kind"], case["steps"]
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(c, steps) for c in state["requests"]]
        srv.run_until_done(ids)
        got = []
        for i in ids:
            r = srv.result(i)
            got.append({"alpha": r["alpha"], "volumes": r["volumes"], "qoi": list(r["qoi"])})
            srv.release(i)
        return got
    s = state["solver"]
    if kind == "ek2d":
        s.step(steps)
        st = s.get_state_f64() if state["out"] is None else s.get_state(out=state["out"])
        got = {"phi": st["phi"], "U": st["U"], "y": s.get_y()}
        if case["prec"] in ("fp32", "fp64"):
            got["psi"] = st["psi"]  # 16-bit storage bounds the far field's psi
        if case["prec"] == "fp64":
            got["dpsi"] = st["dpsi"]  # a difference of large terms: rounding noise in 32 bits
        return got
    if kind == "dense":
        s.step(steps)
        phi, alpha = s.collect(clear=True, out=state["out"])
        return {"phi": phi, "alpha": alpha}
    if kind == "line":
        s.step(steps)
        phi, alpha = s.collect(clear=True, out=state["out"])
        return {"phi": phi, "alpha": alpha, "volumes": s.grain_volumes(case["grains"]),
                "qoi": list(s.qoi_sums())}
    # melt pool: step, nucleation pass, frame check, step
    thres = int(0.8 * state["fnz"])
    for _ in range(steps // 2):
        s.step(1)
        s.nucleate(False, count=False)
        state["done"] += 2
        if state["done"] % FRAME_CHECK == 0:
            state["tip"], state["moves"], _ = s.move_domain(state["tip"], thres, state["moves"])
        s.step(1)
    phi, alpha = s.collect(clear=True, out=state["out"])
    loss = s.get_archive(1)[1]
    return {"phi": phi, "alpha": alpha, "z": s.get_z(), "loss": loss, "tip": state["tip"],
            "moves": state["moves"]}


# ---------------------------------------------------------------- the work of a pass

def _line_work(nx, ny, nz, num_pf, pair, steps):
    """Steps of one line simulation: the cells that hold a grain (the solid quarter
    and the interface's tail of about ten cells above it) read and write their
    slots once a step; about three of a cell's slots are updated, at about 100
    operations each.  The rest of the window is empty and stays so."""
    cells = nx * ny * min(nz, 0.25 * nz + 10)
    return cells * num_pf * pair * 2 * steps, cells * 3 * 100 * steps


def work(case):
    kind, steps = case["kind"], case["steps"]
    if kind == "serve":
        b = f = 0.0
        for nx, ny, nz in [(48, 48, 48), (96, 96, 96), (128, 128, 256), (192, 192, 192)]:
            wb, wf = _line_work(nx, ny, nz, 8, 4, steps)
            b += case["requests"] / 4 * (wb + 4 * nx * ny * nz)
            f += case["requests"] / 4 * wf
        return {"bytes": b, "flops": f}
    if kind == "ek2d":
        v = {"fp32": 4, "fp16": 2, "bf16": 2, "fp64": 8}[case["prec"]]
        cells = case["nx"] * case["ny"]
        # psi, U and dpsi read and written a step; about 150 operations a cell
        return {"bytes": cells * (6 * v * steps + 3 * v + 4 * max(4, v)),
                "flops": 150.0 * cells * steps}
    cells = case["nx"] * case["ny"] * case["nz"]
    if kind == "dense":
        # per cell its list's length, and about 1.5 present grains: list entry
        # (value and grain) read and written, field value written and reset
        return {"bytes": cells * (8 + 1.5 * 20) * steps + 16.0 * cells,
                "flops": 1.5 * 100 * cells * steps}
    pair = 8 if case["prec"] == "fp32" else 4
    if kind == "pool":
        # the solid around the pool fills about 0.85 of the window
        b = 0.85 * cells * case["num_pf"] * pair * 2 * steps
        return {"bytes": b + 8.0 * cells, "flops": 0.85 * cells * 2 * 100 * steps}
    b, f = _line_work(case["nx"], case["ny"], case["nz"], case["num_pf"], pair, steps)
    # read-back: every slot once more for the argmax and the interface sums, 8 B a cell out
    return {"bytes": b + cells * (case["num_pf"] * pair + 8.0), "flops": f}


def tolerance(case):
    """About four times the difference from `exact` (measured on a B200): 3D FP32 phi
    4e-8 to 1.2e-6 (a cell or two on the other side of a threshold), the 2D fields
    in FP32 1e-8 to 1e-7; 16-bit phi 4e-3 (3D), 8e-5 (2D FP16), 9e-4 (2D BF16)."""
    kind, prec = case["kind"], case.get("prec", "fp32")
    if prec == "fp64":
        return {"rel": 1e-13, "max": 1e-11}
    if prec == "fp32":
        return {"rel": 1e-6, "max": 1e-3} if kind == "ek2d" else {"rel": 5e-6, "max": 0.05,
                                                                 "differ": 1e-4}
    if kind == "ek2d":
        return {"rel": 4e-4, "max": 0.05} if prec == "fp16" else {"rel": 4e-3, "max": 0.2}
    return {"rel": 1.5e-2, "max": 0.5, "differ": 2e-3}


# ---------------------------------------------------------------- 64-bit restatement

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _source(n, bc):
    """Source index of every coordinate: mirrored (0) or periodic (1) halo."""
    s = list(range(n))
    s[0] = 2 if bc == 0 else n - 2
    s[n - 1] = n - 3 if bc == 0 else 1
    return s


def _halo(a, p, mirror_all=False):
    """Fill the halo of the last three axes of `a`, each coordinate by itself."""
    bx, by, bz = (0, 0, 0) if mirror_all else (p.bcX, p.bcY, p.bcZ)
    for axis, n, bc in ((-3, p.fnz, bz), (-2, p.fny, by), (-1, p.fnx, bx)):
        s = _source(n, bc)
        for i in (0, n - 1):
            a.select(axis, i).copy_(a.select(axis, s[i]).clone())
    return a


def _points(a, k1):
    """The seven stencil points (below, y-, x-, centre, x+, y+, above) of the
    interior cells of planes 1 .. k1-1."""
    def v(dz, dy, dx):
        return a[..., 1 + dz:k1 + dz, 1 + dy:a.shape[-2] - 1 + dy, 1 + dx:a.shape[-1] - 1 + dx]
    return [v(-1, 0, 0), v(0, -1, 0), v(0, 0, -1), v(0, 0, 0), v(0, 0, 1), v(0, 1, 0), v(1, 0, 0)]


def _slot_update(p, v, sa, ca, sb, cb, repul, Up, full):
    """New phi of one grain from its values at the seven points."""
    D, Bm, Lx, C, Rx, T, U = v
    ux, uy, uz = (Rx - Lx) * 0.5, (T - Bm) * 0.5, (U - D) * 0.5
    if full:
        rx = ca * cb * ux + sa * uy + ca * sb * uz
        ry = -sa * cb * ux + ca * uy - sa * sb * uz
        rz = -sb * ux + cb * uz
    else:
        rx = ca * cb * ux + sa * cb * uy - sb * uz
        ry = -sa * ux + ca * uy
        rz = ca * sb * ux + sa * sb * uy + cb * uz
    mag = rx * rx + ry * ry + rz * rz
    kd = float(p.kin_delta)
    a_s = 1.0 + 3.0 * kd
    q = rx ** 4 + ry ** 4 + rz ** 4
    m = mag > float(p.eps)
    A = torch.where(m, a_s * (1.0 - 4.0 * kd / a_s * q / torch.where(m, mag * mag, 1.0)), 1.0)
    hi = float(p.hi)
    w = 1.0 - C * C
    E1 = (Rx + Lx + T + Bm + U + D - 6.0 * C) * hi * hi + w * C
    inner = w * w - 6.0 * (C + 1.0) * repul
    return C + float(p.dt) * (E1 - float(p.lamd) * Up * inner) / A


class _ExactAPT:
    """The APT step: ids of the seven points merged in first-seen order into at most
    num_pf slots, each slot updated; an entry past the last slot lands in slot 0 of
    the next point."""

    def __init__(self, c):
        self.c, self.p = c, c.params
        p, dev = self.p, _device()
        shape = (p.num_pf, p.fnz, p.fny, p.fnx)
        self.ph = torch.full(shape, -1.0, dtype=torch.float64, device=dev)
        self.id = torch.full(shape, -1, dtype=torch.int32, device=dev)
        phi = torch.from_numpy(c.phi).to(dev).double().reshape(shape[1:])
        alpha = torch.from_numpy(c.alpha).to(dev).reshape(shape[1:])
        m = phi > LS
        self.ph[0][m] = phi[m]
        self.id[0][m] = alpha[m]
        _halo(self.ph, p), _halo(self.id, p)
        ng = p.num_theta
        tab = [torch.from_numpy(np.asarray(t, np.float64)).to(dev) for t in
               (c.sint[:ng + 1], c.cost[:ng + 1], c.sint[ng:], c.cost[ng:])]
        self.tab = tab  # entry g: sine and cosine of grain g's two angles
        self.z = torch.from_numpy(c.z).to(dev).double()
        self.n = 0

    def step(self):
        p, NP = self.p, self.p.num_pf
        self.n += 1
        t = self.n * float(p.dt) * float(p.tau0)
        held = (self.id >= 0).flatten(2).any(2).any(0).nonzero()
        k1 = min(p.fnz - 1, int(held.max()) + 2)  # planes above hold nothing and get nothing
        P, I = _points(self.ph, k1), _points(self.id, k1)
        shape = P[0].shape[1:]
        L = [torch.full(shape, -1, dtype=torch.int32, device=self.ph.device) for _ in range(NP)]
        V = [[torch.full(shape, -1.0, dtype=torch.float64, device=self.ph.device)
              for _ in range(NP)] for _ in range(7)]
        n = torch.zeros(shape, dtype=torch.int32, device=self.ph.device)
        for s in range(7):
            for q in range(NP):
                idv, pv = I[s][q], P[s][q]
                m = idv != -1
                if not bool(m.any()):
                    continue
                pos = n.clone()
                found = torch.zeros_like(m)
                for j in range(NP - 1, -1, -1):
                    e = (L[j] == idv) & m
                    pos = torch.where(e, j, pos)
                    found |= e
                for j in range(NP):
                    e = m & (pos == j)
                    L[j] = torch.where(e, idv, L[j])
                    V[s][j] = torch.where(e, pv, V[s][j])
                over = m & ~found & (n >= NP)
                if s < 6 and bool(over.any()):
                    V[s + 1][0] = torch.where(over, pv, V[s + 1][0])
                n += (m & ~found & (n < NP)).int()
        Up = ((float(p.G) * (self.z[1:k1] - float(p.z0))
               - float(p.underCoolingRate) * 1e6 * t) / float(p.L_cp))[:, None, None]
        terms = [0.25 * (V[3][j] + 1.0) ** 2 for j in range(NP)]
        nph, nid = torch.full_like(self.ph, -1.0), torch.full_like(self.id, -1)
        for j in range(NP):
            used = j < n
            g = L[j].clamp(min=0)
            g = torch.where(g > p.num_theta, g % p.num_theta + 1, g).long()
            near = V[3][j] > LS
            sa, ca, sb, cb = (torch.where(near, tb[g], d) for tb, d in
                              zip(self.tab, (0.0, 1.0, 0.0, 1.0)))
            repul = sum((terms[q] for q in range(NP) if q != j), torch.zeros_like(terms[0]))
            v = _slot_update(p, [V[s][j] for s in range(7)], sa, ca, sb, cb, repul, Up, False)
            nph[j, 1:k1, 1:-1, 1:-1] = torch.where(used, v, -1.0)
            nid[j, 1:k1, 1:-1, 1:-1] = torch.where(used & ~(v < ID_DROP), L[j], -1)
        self.ph, self.id = _halo(nph, p), _halo(nid, p)

    def read(self):
        p = self.p
        best, at = self.ph[0].clone(), self.id[0].clone()
        for j in range(1, p.num_pf):
            m = self.ph[j] > best
            best, at = torch.where(m, self.ph[j], best), torch.where(m, self.id[j], at)
        m = best > LS
        alpha = torch.where(m, at, 0)
        inner = alpha[1:-1, 1:-1, 1:-1].reshape(-1)
        key = torch.where((inner >= 1) & (inner <= p.num_theta), inner, 0).long()
        d, bm, lx, c, rx, tp, u = _points(best, p.fnz - 1)
        vol = float((0.5 * (1.0 + c)).sum())
        area = float((0.5 * torch.sqrt((0.5 * (rx - lx)) ** 2 + (0.5 * (tp - bm)) ** 2
                                       + (0.5 * (u - d)) ** 2)).sum())
        return {"phi": torch.where(m, best, 0.0).reshape(-1), "alpha": alpha.reshape(-1),
                "volumes": torch.bincount(key, minlength=p.num_theta + 1),
                "qoi": [vol, area, vol / ((p.fnx - 2) * (p.fny - 2))]}


def _exact_apt(c, steps):
    a = _ExactAPT(c)
    for _ in range(steps):
        a.step()
    return a.read()


def _exact_dense(c, steps):
    """Every grain's field at every cell; the repulsion sums over all other grains."""
    p, dev = c.params, _device()
    ng = p.num_theta
    shape = (p.fnz, p.fny, p.fnx)
    phi = torch.from_numpy(c.phi).to(dev).double().reshape(shape)
    alpha = torch.from_numpy(c.alpha).to(dev).reshape(shape)
    ph = torch.full((ng,) + shape, -1.0, dtype=torch.float64, device=dev)
    for g in range(ng):
        m = (phi > LS) & (alpha == g + 1)
        ph[g][m] = phi[m]
    _halo(ph, p, True)
    z = torch.from_numpy(c.z).to(dev).double()
    R = float(np.float32(c.meta["R"]))
    for n in range(steps + 1):  # n = 0: the update at t = 0 before the loop
        t = n * float(p.dt) * float(p.tau0)
        Up = (float(p.G) * (z[1:-1] - R * 1e6 * t - 2.0) / float(p.L_cp))[:, None, None]
        total = (0.25 * (ph[:, 1:-1, 1:-1, 1:-1] + 1.0) ** 2).sum(0)
        out = torch.empty_like(ph)
        for g in range(ng):
            v = _points(ph[g], p.fnz - 1)
            near = v[3] > LS
            o = [float(c.sint[g + 1]), float(c.cost[g + 1]), float(c.sint[g + 1 + ng]),
                 float(c.cost[g + 1 + ng])]
            sa, ca, sb, cb = (torch.where(near, w, d) for w, d in zip(o, (0.0, 1.0, 0.0, 1.0)))
            repul = total - 0.25 * (v[3] + 1.0) ** 2
            out[g, 1:-1, 1:-1, 1:-1] = _slot_update(p, v, sa, ca, sb, cb, repul, Up, True)
        ph = _halo(out, p, True)
    best, at = ph.max(0)
    m = best > LS
    return {"phi": torch.where(m, best, -1.0).reshape(-1),
            "alpha": torch.where(m, at.int() + 1, 0).reshape(-1)}


def _exact_ek2d(c, steps):
    """The line model's step: edge fluxes of psi (anisotropic) and U (with the
    anti-trapping current), U first, then psi with the new U; frame check every
    tipp steps."""
    p, dev = c.params, _device()
    f = lambda n: float(getattr(p, n))
    fnx, fny = c.fnx, c.fny
    k, hi, sq2, dt, eps = f("k"), f("hi"), f("sqrt2"), f("dt"), f("eps")
    W0, dxd = f("W0"), f("dx") * f("W0")

    def halo(a):
        a[:, 0], a[:, -1] = a[:, -2].clone(), a[:, 1].clone()
        a[0], a[-1] = a[2].clone(), a[-3].clone()
        return a

    ps, U = (halo(torch.from_numpy(np.asarray(a, np.float32)).to(dev).double().reshape(fny, fnx))
             for a in (c.psi, c.U))
    Dp = torch.zeros_like(ps)
    rows = torch.arange(fny, dtype=torch.float64, device=dev)[1:-1, None]
    cur_tip, thres, shifts, intR = 1, int((1.0 - f("blank")) * fny), 0, 0.0

    def length(G):
        return (f("c_infm") * (1.0 / k - 1.0) / G) / W0

    def aniso(x, y):
        ux, uz = f("cosa") * x + f("sina") * y, f("cosa") * y - f("sina") * x
        m = ux * ux + uz * uz
        on = m > eps
        inv = 1.0 / torch.where(on, m * m, 1.0)
        A = torch.where(on, f("a_s") * (1.0 + f("epsilon") * (ux ** 4 + uz ** 4) * inv), 1.0)
        Ap = torch.where(on, -f("a_12") * ux * uz * (ux * ux - uz * uz) * inv, 0.0)
        return A, Ap

    def unit(n, a, b):
        n2 = a * a + b * b
        on = n2 > eps
        return torch.where(on, n / torch.sqrt(torch.where(on, n2, 1.0)), 0.0)

    def advance(merge, lT):
        nonlocal ps, U, Dp
        ph = torch.tanh(ps / sq2)
        jat = 0.5 * (1.0 + (1.0 - k) * U) * (1.0 - ph * ph) * Dp
        qs, qp = (0.25 * (a[:-1, :-1] + a[:-1, 1:] + a[1:, :-1] + a[1:, 1:]) for a in (ps, ph))
        # x edges of rows 1 .. fny-2, y edges of columns 1 .. fnx-2
        x_ps, x_ph = (a[1:-1, 1:] - a[1:-1, :-1] for a in (ps, ph))
        x_tps, x_tph = qs[1:] - qs[:-1], qp[1:] - qp[:-1]
        y_ps, y_ph = (a[1:, 1:-1] - a[:-1, 1:-1] for a in (ps, ph))
        y_tps, y_tph = qs[:, 1:] - qs[:, :-1], qp[:, 1:] - qp[:, :-1]
        A, Ap = aniso(x_ph, x_tph)
        xJ = A * (A * x_ps - Ap * x_tps)
        A, Ap = aniso(y_tph, y_ph)
        yJ = A * (A * y_ps + Ap * y_tps)
        phC, UC = ph[1:-1, 1:-1], U[1:-1, 1:-1]
        Un = UC
        if merge:
            c1 = hi * f("Dl_tilde") * 0.5
            xF = (c1 * (2.0 - ph[1:-1, :-1] - ph[1:-1, 1:]) * (U[1:-1, 1:] - U[1:-1, :-1])
                  + 0.5 * (jat[1:-1, :-1] + jat[1:-1, 1:]) * unit(x_ph, x_ph, x_tph))
            yF = (c1 * (2.0 - ph[:-1, 1:-1] - ph[1:, 1:-1]) * (U[1:, 1:-1] - U[:-1, 1:-1])
                  + 0.5 * (jat[:-1, 1:-1] + jat[1:, 1:-1]) * unit(y_ph, y_tph, y_ph))
            div = (xF[:, 1:] - xF[:, :-1] + yF[1:] - yF[:-1]) * hi + sq2 * jat[1:-1, 1:-1]
            Un = UC + dt * div / (1.0 + k - (1.0 - k) * phC)
        g = lambda a: ((a[1:-1, 2:] - a[1:-1, :-2]) * 0.5, (a[2:, 1:-1] - a[:-2, 1:-1]) * 0.5)
        A2 = aniso(*g(ph))[0] ** 2
        gx, gz = g(ps)
        Up = ((p.y0 + (shifts - 1.0 + rows) * dxd) / W0 - intR) / lT
        rhs = ((xJ[:, 1:] - xJ[:, :-1] + yJ[1:] - yJ[:-1]
                - sq2 * A2 * phC * (gx * gx + gz * gz)) * hi * hi
               + sq2 * phC - f("lamd") * (1.0 - phC * phC) * sq2 * (Un + Up))
        d = rhs / ((1.0 - (1.0 - k) * Up).clamp(min=k) * A2)
        nps, nU, nD = torch.empty_like(ps), torch.empty_like(ps), torch.empty_like(ps)
        nps[1:-1, 1:-1], nU[1:-1, 1:-1], nD[1:-1, 1:-1] = ps[1:-1, 1:-1] + dt * d, Un, d
        ps, U, Dp = halo(nps), halo(nU), halo(nD)

    advance(False, length(float(c.Gt[0])))
    t0, t1 = float(c.t_mac[0]), float(c.t_mac[1])
    for n in range(1, steps + 1):
        x = (n * dt * f("tau0") - t0) / (t1 - t0)
        kt = min(max(int(math.floor(x)), 0), len(c.t_mac) - 2)
        w = x - kt
        R, G = ((1.0 - w) * float(a[kt]) + w * float(a[kt + 1]) for a in (c.Rt, c.Gt))
        intR += R * f("tau0") / W0 * dt
        advance(True, length(G))
        if n % p.tipp == 0:
            mean = torch.tanh(ps / sq2).sum(1).cpu().numpy() / fnx
            while mean[cur_tip] > f("ls") and cur_tip < fny - 1:
                cur_tip += 1
            m = 0
            while cur_tip >= thres:
                m, cur_tip = m + 1, cur_tip - 1
            if m:
                old = ps.clone()
                ps[1:fny - 1 - m], U[1:fny - 1 - m] = old[1 + m:fny - 1], U[1 + m:fny - 1].clone()
                e2, e1 = old[fny - 3], old[fny - 2]
                for j in range(fny - 1 - m, fny - 1):
                    e2, e1 = e1, 2.0 * e1 - e2
                    ps[j], U[j] = e1, f("U0")
                halo(ps), halo(U)
                shifts += m
    y = p.y0 + (np.arange(fny) - 1.0 + shifts) * dxd
    return {"psi": ps, "phi": torch.tanh(ps / sq2), "U": U, "dpsi": Dp, "y": y}


def exact(case, seed):
    kind, steps = case["kind"], case["steps"]
    if kind == "line":
        return _exact_apt(_line_case(case, seed), steps)
    if kind == "serve":
        got = [_exact_apt(c, steps) for c in _serve_cases(case, seed)]
        return [{n: r[n] for n in ("alpha", "volumes", "qoi")} for r in got]
    if kind == "dense":
        return _exact_dense(_line_case(case, seed), steps)
    if kind == "ek2d":
        st = _exact_ek2d(_ek2d_case(case, seed), steps)
        names = {"fp64": ("phi", "U", "y", "psi", "dpsi"), "fp32": ("phi", "U", "y", "psi")}
        return {n: st[n] for n in names.get(case["prec"], ("phi", "U", "y"))}
    return None  # nucleation and the moving window: random decisions, no short restatement
