// ek2d.cuh — 2D Echebarria–Karma directional-solidification step (psi/U line
// model of cuPF 2DdendriteMPI/line_model/PF.cu) for sm_100a.
//
// One launch advances the whole grid by one step (ek2d_march_kernel, below):
// each warp marches up a strip of 30 columns, computing for every cell
//   - the phase field, U and dpsi of the next row (decoded: psi and
//     phi = tanh(psi/sqrt2)) and the anti-trapping flux density
//     jat = (1+(1-k)U)(1-phi^2) dpsi / 2;
//   - plaquette means of psi and phi at the cell corners (psipjp .. phimjm of
//     merge_PF, PF.cu:444-453);
//   - the fluxes through its right and upper edges: the anisotropic psi flux J
//     (atheta/aptheta, PF.cu:119-146, 475-538) and the solute flux of U with
//     its anti-trapping part (PF.cu:460-551).  Each edge is computed once and
//     shared by the two cells it separates (the reference computes it from
//     both sides);
//   - U' = U + dt*div(U flux)/tau_U (PF.cu:553-556), then the psi right-hand
//     side with the new U (PF.cu:563-590), dpsi = rhs/tau_psi,
//     psi' = psi + dt*dpsi (+ noise), and the stores.
// The reference's merge_PF (PF.cu:379-610) fuses the same U-then-psi update in
// one kernel over a 128-wide band of a linear index; the pre-loop rhs_psi
// (PF.cu:150-280) is the same psi update with U left unchanged (`prestep`).
//
// Boundary: x periodic, y mirrored about rows 1 and fny-2 (set_BC,
// PF.cu:35-73).  The reference refills the halo of the state it is about to
// read; here every writer of an interior cell that some halo cell copies also
// writes that copy, so each step's output already carries its halo.
//
// Storage S: FP32 (the reference's), FP16 / BF16 (split precision: the phase
// field (psi bounded to +-50 W0 in FP16; phi as its distance to the bulk value
// in BF16), U - U0 and dpsi in 16 bits, the phase field and U stored with
// stochastic rounding, arithmetic in FP32) or FP64 (double arithmetic
// throughout).  Up = (y/W0 - intR)/lT_tilde of each row
// is formed in FP64 from the host's FP64 time integration.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "philox.cuh"
#include "rounding.cuh"

namespace cupf {
namespace ek2d {


// ---- storage formats -------------------------------------------------------
//
// Every format stores three planes: the phase field, U and dpsi.  ld_pp()
// decodes the phase-field plane into (psi, phi), st_ps()/st_ps_sr() encode a
// new psi; U and dpsi use ld/ldU and st/stU/st_sr.

template <class T>
__device__ __forceinline__ T tanh_t(T x);

// The hardware approximations (1 or 2 ulp) as single instructions: subnormal inputs and
// results go to zero instead of through the scaling that the non-flushing forms add.
// That changes no result of the step: 2^x and the reciprocals of tanh and of the code add
// to or divide by a number of at least 1, U's and psi's denominators are at least k
// times the anisotropy squared, and m * m is taken where m > eps (1e-8 by default).
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float ex2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
constexpr float kLog2e = 1.44269504f;

// FP32 / FP64: psi itself, as the reference stores it; phi = tanh(psi/sqrt2).
template <class TT>
struct StPlain {
  using V = TT;
  using T = TT;
  static constexpr bool kSR = false;
  __device__ static T ld(V v) { return v; }
  __device__ static T ldU(V v, T) { return v; }
  __device__ static V st(T x) { return x; }
  __device__ static V stU(T x, T) { return x; }
  __device__ static V st_sr(T x, uint32_t) { return x; }
  __device__ static void ld_pp(V v, T inv_sqrt2, T& ps, T& ph) {
    ps = v;
    ph = tanh_t(ps * inv_sqrt2);
  }
  __device__ static V st_ps(T ps) { return ps; }
  __device__ static V st_ps_sr(T ps, uint32_t) { return ps; }
  __device__ static void st_ps_U_sr(T ps, T u, uint32_t, V& vps, V& vu) {
    vps = ps;
    vu = u;
  }
};
using StF32 = StPlain<float>;
using StF64 = StPlain<double>;

// 16-bit storage (split precision).  psi is a signed distance that reaches
// thousands of W0 across the domain; stored as it is in 16 bits its spacing
// there exceeds the grid's own psi increments, and rounding noise in
// |grad psi|^2 then drives the far field toward solid.  psi is therefore held
// to |psi| <= kPsiClamp = 50 W0 in the 16-bit modes: far enough that the bound
// does not reach back to the front (a bound of 12.5 W0, where phi is already
// +-1 to float precision, moved the front by about a cell in 3000 steps; 25 W0
// by 0.02 cells; 50 W0 by none measurable), and small enough that FP16 keeps a
// spacing of at most 0.03 W0 there.
//   FP16 stores psi itself (spacing 2^-11 |psi|: 5e-4 at the interface centre,
//   4e-3 at |psi| = 4-8).
//   BF16, with 8 significant bits, stores phi as its distance to the nearest
//   bulk value, with phi's sign,
//     u = copysign(1 - |phi|, phi),   phi = copysign(1 - |u|, u),
//     |psi| = sqrt2 atanh(1 - |u|) = (ln(2 - |u|) - ln|u|)/sqrt2,
//   which keeps psi to about 2.8e-3 everywhere (BF16 has FP32's exponent range,
//   so u of |psi| = 50, 4e-31, is representable).
// U is stored as its offset from the far-field value U0.
constexpr float kPsiClamp = 50.0f;

template <bool BF>
struct StH16 {
  using V = unsigned short;
  using T = float;
  static constexpr bool kSR = true;
  __device__ static T ld(V v) {
    return BF ? __bfloat162float(__ushort_as_bfloat16(v)) : __half2float(__ushort_as_half(v));
  }
  __device__ static T ldU(V v, T U0) { return __fadd_rn(ld(v), U0); }
  __device__ static V st(T x) {
    return BF ? __bfloat16_as_ushort(__float2bfloat16_rn(x)) : __half_as_ushort(__float2half_rn(x));
  }
  __device__ static V stU(T x, T U0) { return st(__fsub_rn(x, U0)); }
  // stochastic rounding by the hardware conversion (cvt.rs): x with r[31:16]
  __device__ static uint32_t sr2(T hi, T lo, uint32_t r) {
    return BF ? sr_pack_bf16x2(hi, lo, r) : sr_pack_fp16x2(hi, lo, r);
  }
  __device__ static V st_sr(T x, uint32_t r) { return (V)(sr2(x, 0.0f, r) >> 16); }
  __device__ static void ld_pp(V v, T inv_sqrt2, T& ps, T& ph) {
    if (!BF) {
      ps = ld(v);
      ph = tanh_t(ps * inv_sqrt2);
      return;
    }
    const float u = ld(v), a = fabsf(u);
    ph = copysignf(1.0f - a, u);
    const float m = (a > 0.0f) ? fminf(0.70710678f * (__logf(2.0f - a) - __logf(a)), kPsiClamp)
                               : kPsiClamp;
    ps = copysignf(m, u);
  }
  // the stored value of a psi: psi bounded to +-kPsiClamp (FP16), or its u:
  // 1 - tanh(|psi|/sqrt2) = 2/(1 + e^(sqrt2 |psi|)) with psi's sign (BF16)
  __device__ static float code(float ps) {
    const float x = fminf(fabsf(ps), kPsiClamp);
    if (!BF) return copysignf(x, ps);
    return copysignf(2.0f * rcp_approx(1.0f + ex2_approx((1.41421356f * kLog2e) * x)), ps);
  }
  __device__ static V st_ps(T ps) { return st(code(ps)); }
  __device__ static V st_ps_sr(T ps, uint32_t r) { return st_sr(code(ps), r); }
  // the phase field's code and U - U0 in one conversion: r[31:16] round the
  // first, r[15:0] the second
  __device__ static void st_ps_U_sr(T ps, T u, uint32_t r, V& vps, V& vu) {
    const uint32_t d = sr2(code(ps), u, r);
    vps = (V)(d >> 16);
    vu = (V)(d & 0xFFFFu);
  }
};
using StF16 = StH16<false>;
using StBF16 = StH16<true>;

// ---- launch arguments ------------------------------------------------------

// Constants of the FP32-arithmetic step (flux_consts), with the factors that multiply
// a whole flux or difference folded together.  Part of the arguments: the arithmetic
// reads them as constant operands instead of holding them in registers.
struct FluxConsts {
  float cosa, sina, a_s, ase, a12;
  float j0, j1;      // jat/2 = (j0 + j1 U) (1 - phi^2) dpsi
  float g0, g1;      // solute conductance g0 + g1 (phi_a + phi_b)
  float dthi, dts;   // dt hi, 2 sqrt2 dt
  float opk, nomk;   // tau_U = opk + nomk phi
  float hi2, sqrt2, inv_sqrt2, nex, nlam;
  float eps, eps4, k, dt, U0;
};

struct EkArgs {
  const void* in;     // three planes (psi, U, dpsi), each fny rows of `pitch` values
  void* out;
  long long plane;    // values per plane
  int pitch, fnx, fny;
  int prestep;        // 1: psi update only, U unchanged (rhs_psi)
  int rows;           // output rows each warp marches over
  float k, hi, Dl_tilde, eps, sqrt2, lamd, dt, cosa, sina, a_s, epsilon, a_12, U0;
  float noise_amp;    // dt_sqrt*hi*eta; 0 disables the noise term
  double up_a, up_b;  // Up of memory row j = up_a + j*up_b
  uint32_t seed, step;
  FluxConsts fc;
};

inline FluxConsts flux_consts(const EkArgs& a) {
  FluxConsts c;
  c.cosa = a.cosa;
  c.sina = a.sina;
  c.a_s = a.a_s;
  c.ase = a.a_s * a.epsilon;
  c.a12 = a.a_12;
  c.j0 = 0.25f;
  c.j1 = 0.25f * (1.0f - a.k);
  const float hd = a.hi * a.Dl_tilde * 0.5f;
  c.g0 = 2.0f * hd;
  c.g1 = -hd;
  c.dthi = a.dt * a.hi;
  c.dts = 2.0f * a.sqrt2 * a.dt;
  c.opk = 1.0f + a.k;
  c.nomk = a.k - 1.0f;
  c.hi2 = a.hi * a.hi;
  c.sqrt2 = a.sqrt2;
  c.inv_sqrt2 = 1.0f / a.sqrt2;
  c.nex = -0.25f * a.sqrt2;
  c.nlam = -a.lamd * a.sqrt2;
  c.eps = a.eps;
  c.eps4 = 4.0f * a.eps;
  c.k = a.k;
  c.dt = a.dt;
  c.U0 = a.U0;
  return c;
}

// Constants of the FP64 step.
struct Consts {
  double k, omk, opk, hi, hiDl_half, eps, sqrt2, inv_sqrt2, lamd, dt, cosa, sina, a_s, epsilon,
      a_12, U0, noise_amp;
};

__device__ __forceinline__ Consts consts(const EkArgs& a) {
  Consts c;
  c.k = a.k;
  c.omk = 1.0 - (double)a.k;
  c.opk = 1.0 + (double)a.k;
  c.hi = a.hi;
  c.hiDl_half = (double)a.hi * (double)a.Dl_tilde * 0.5;
  c.eps = a.eps;
  c.sqrt2 = a.sqrt2;
  c.inv_sqrt2 = 1.0 / (double)a.sqrt2;
  c.lamd = a.lamd;
  c.dt = a.dt;
  c.cosa = a.cosa;
  c.sina = a.sina;
  c.a_s = a.a_s;
  c.epsilon = a.epsilon;
  c.a_12 = a.a_12;
  c.U0 = a.U0;
  c.noise_amp = a.noise_amp;
  return c;
}

// Math of the step.  FP64 storage uses correctly rounded double operations
// throughout.  The FP32-arithmetic storages (FP32, FP16, BF16) use the
// hardware approximations (reciprocal, reciprocal square root, 2^x; 1 or 2 ulp
// each), far below the per-step differences the model's own rounding makes,
// and tanh from its exponential form tanh(x) = 1 - 2/(1 + e^(2x)) (exact limits
// +-1 at large |x|; absolute error of a few 1e-7 near 0).
template <>
__device__ __forceinline__ float tanh_t<float>(float x) {
  return fmaf(-2.0f, rcp_approx(1.0f + ex2_approx((2.0f * kLog2e) * x)), 1.0f);
}
template <>
__device__ __forceinline__ double tanh_t<double>(double x) {
  return tanh(x);
}

// |phi| strictly inside the interface band, as the reference's
// (double)phi > -0.995 && (double)phi < 0.995 (PF.cu:592): for a float, that
// is |phi| < 0.995f exactly (0.995f rounds above 0.995).
__device__ __forceinline__ bool in_band(float ph) { return fabsf(ph) < 0.995f; }
__device__ __forceinline__ bool in_band(double ph) { return fabs(ph) < 0.995; }

// Anisotropy of the interface normal (phx, phz) rotated by the misorientation:
// A = atheta (PF.cu:119-131), Ap = aptheta (PF.cu:135-146).
__device__ __forceinline__ void aniso(double phx, double phz, const Consts& c, double& A, double& Ap) {
  const double ux = c.cosa * phx + c.sina * phz;
  const double uz = c.cosa * phz - c.sina * phx;
  const double ux2 = ux * ux, uz2 = uz * uz;
  const double m = ux2 + uz2;
  if (m > c.eps) {
    const double inv = 1.0 / (m * m);
    A = c.a_s * (1.0 + c.epsilon * (ux2 * ux2 + uz2 * uz2) * inv);
    Ap = -c.a_12 * ux * uz * (ux2 - uz2) * inv;
  } else {
    A = 1.0;
    Ap = 0.0;
  }
}

__device__ __forceinline__ double aniso_a(double phx, double phz, const Consts& c) {
  const double ux = c.cosa * phx + c.sina * phz;
  const double uz = c.cosa * phz - c.sina * phx;
  const double ux2 = ux * ux, uz2 = uz * uz;
  const double m = ux2 + uz2;
  if (m > c.eps) return c.a_s * (1.0 + c.epsilon * ((ux2 * ux2 + uz2 * uz2) / (m * m)));
  return 1.0;
}

// Write one cell's three values at (j, i) and at every halo cell that copies it:
// column fnx-1 copies column 1 and column 0 copies column fnx-2 (periodic x),
// row 0 copies row 2 and row fny-1 copies row fny-3 (mirrored y), corners both.
template <class V>
__device__ __forceinline__ void put_with_halo(V* ps, V* U, V* D, int pitch, int fnx, int fny,
                                              int j, int i, V vps, V vU, V vD) {
  auto put = [&](int jj, int ii) {
    const long long o = (long long)jj * pitch + ii;
    ps[o] = vps;
    U[o] = vU;
    D[o] = vD;
  };
  put(j, i);
  const bool xl = (i == 1), xr = (i == fnx - 2);
  if (xl) put(j, fnx - 1);
  if (xr) put(j, 0);
  if (j == 2) {
    put(0, i);
    if (xl) put(0, fnx - 1);
    if (xr) put(0, 0);
  }
  if (j == fny - 3) {
    put(fny - 1, i);
    if (xl) put(fny - 1, fnx - 1);
    if (xr) put(fny - 1, 0);
  }
}

// Fluxes through one cell edge, from the differences across it (normal) and
// along it (tangential, from the plaquette means at its two ends), and the
// values of the two cells it separates (a below/left, b above/right):
// J = A (A dpsi_n -+ Ap dpsi_t), the anisotropic psi flux of merge_PF
// (PF.cu:475-538), and Uf, the solute flux with its anti-trapping part
// (PF.cu:460-551).  kY selects the y-edge form (normal = z).
template <bool kY>
__device__ __forceinline__ void edge_flux(const Consts& c, bool merge, double psx, double psz,
                                          double phx, double phz, double pha, double phb, double Ua,
                                          double Ub, double ja, double jb, double& J, double& Uf) {
  double A, Ap;
  aniso(phx, phz, c, A, Ap);
  J = kY ? A * (A * psz + Ap * psx) : A * (A * psx - Ap * psz);
  if (merge) {
    const double n2 = phx * phx + phz * phz;
    const double nn = (n2 > c.eps) ? (kY ? phz : phx) * (1.0 / sqrt(n2)) : 0.0;
    Uf = c.hiDl_half * (2.0 - pha - phb) * (Ub - Ua) + 0.5 * (ja + jb) * nn;
  }
}

__device__ __forceinline__ double jat_of(const Consts& c, double U, double ph, double D) {
  return 0.5 * (1.0 + c.omk * U) * (1.0 - ph * ph) * D;
}

// Stored values of one cell's new psi, U and dpsi.
template <class S, class T = typename S::T, class V = typename S::V>
__device__ __forceinline__ void encode_cell(const EkArgs& a, bool merge, uint32_t step_key, int gi,
                                            int gj, T psn, T Un, T dps, V& vps, V& vU, V& vD) {
  const T U0 = (T)a.U0;
  if (S::kSR) {
    // one 32-bit draw per cell and step: its two 16-bit halves round the
    // phase field and U independently; dpsi is rewritten from scratch every
    // step, not accumulated, so it rounds to nearest
    const uint32_t r = mix32((uint32_t)(gi + a.fnx * gj) ^ step_key);
    if (merge) {
      S::st_ps_U_sr(psn, Un - U0, r, vps, vU);
    } else {
      vps = S::st_ps_sr(psn, r);
      vU = S::stU(Un, U0);
    }
  } else {
    vps = S::st_ps(psn);
    vU = S::stU(Un, U0);
  }
  vD = S::st(dps);
}

// One cell's update and stores (PF.cu:553-598): U' from the divergence of the
// solute fluxes, then psi' with the new U, dpsi = rhs/tau_psi, the optional
// noise term, and the stores with their halo copies.
__device__ __forceinline__ void cell_update(const EkArgs& a, const Consts& c, bool merge, int gi,
                                            int gj, double psC, double phC, double UC, double jatC,
                                            double JR, double JL, double JT, double JB, double UR,
                                            double UL, double UT, double UB, double phR, double phL,
                                            double phT, double phB, double psR, double psL, double psT,
                                            double psB, double* o_ps, double* o_U, double* o_D) {
  double Un = UC;
  if (merge) {
    const double rhsU = ((UR - UL) + (UT - UB)) * c.hi + c.sqrt2 * jatC;
    const double tauU = c.opk - c.omk * phC;
    Un = UC + c.dt * (rhsU / tauU);
  }
  const double phxn = (phR - phL) * 0.5;
  const double phzn = (phT - phB) * 0.5;
  const double psxn = (psR - psL) * 0.5;
  const double pszn = (psT - psB) * 0.5;
  double A2 = aniso_a(phxn, phzn, c);
  A2 = A2 * A2;
  const double gradps2 = psxn * psxn + pszn * pszn;
  const double extra = -c.sqrt2 * A2 * phC * gradps2;
  const double Up = a.up_a + (double)gj * a.up_b;
  const double rhs = ((JR - JL) + (JT - JB) + extra) * c.hi * c.hi + c.sqrt2 * phC -
                     c.lamd * (1.0 - phC * phC) * c.sqrt2 * (Un + Up);
  const double tp = 1.0 - c.omk * Up;
  const double tau = ((tp >= c.k) ? tp : c.k) * A2;
  const double dps = rhs / tau;
  double noise = 0.0;
  if (c.noise_amp != 0.0 && in_band(phC)) {
    const Philox4 rn = philox4x32_10((uint32_t)gi, (uint32_t)gj, a.step, 0x4E4F4953u, a.seed, 0x5EEDu);
    noise = c.noise_amp * (uniform01(rn.v[0]) - 0.5);
  }
  const double psn = psC + c.dt * dps + noise;
  put_with_halo(o_ps, o_U, o_D, a.pitch, a.fnx, a.fny, gj, gi, psn, Un, dps);
}

// ---- register-marching step kernel ------------------------------------------
//
// A warp owns a strip of MW = 30 output columns: lane l holds column x0-1+l, so
// lanes 0 and 31 carry the strip's halo columns.  The warp marches up a.rows
// output rows, keeping three rows of its own column (r-1, r, r+1) and two of its right
// neighbour (r, r+1) in registers; the left neighbour's values, plaquette means
// and x-edge fluxes come by warp shuffle.  Each edge flux is computed once: a
// lane computes the x-edge on its right and the y-edge above it, the y-edge
// below it was computed in the previous row.  The next row's loads are issued a
// row ahead of their use.  No shared memory, no barriers.
constexpr int MW = 30;
constexpr int MWARPS = 4;
// The warps of the launch take (strip, row chunk) pairs in order, strips
// fastest, whatever the grid's width: no idle warps beside a narrow grid.
struct MarchPos {
  int group, chunk;
  bool on;
};
__device__ __forceinline__ MarchPos march_pos(int ngroups, int nchunks) {
  const int w = blockIdx.x * MWARPS + (int)(threadIdx.x >> 5);
  return MarchPos{w % ngroups, w / ngroups, w < ngroups * nchunks};
}

// FP64 storage: one strip a warp, scalar arithmetic.
__global__ void __launch_bounds__(MWARPS * 32) ek2d_march_kernel(EkArgs a) {
  const Consts c = consts(a);
  const bool merge = !a.prestep;
  const double* in_ps = static_cast<const double*>(a.in);
  const double* in_U = in_ps + a.plane;
  const double* in_D = in_U + a.plane;
  double* o_ps = static_cast<double*>(a.out);
  double* o_U = o_ps + a.plane;
  double* o_D = o_U + a.plane;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const MarchPos pos = march_pos((a.fnx - 2 + MW - 1) / MW, (a.fny - 2 + a.rows - 1) / a.rows);
  if (!pos.on) return;             // whole warp: uniform
  const int x0 = 1 + pos.group * MW;  // first output column of the strip
  const int gi = x0 - 1 + lane;
  const bool col_ok = gi < a.fnx;
  const bool out_col = lane >= 1 && lane <= MW && gi <= a.fnx - 2;
  const int y0 = 1 + pos.chunk * a.rows;

  // raw values of the next row to decode, loaded one row ahead of their use so
  // that the load latency overlaps the current row's arithmetic
  double raw_ps{}, raw_U{}, raw_D{};
  bool raw_ok = false;
  auto issue = [&](int r) {
    raw_ok = col_ok && r < a.fny;
    if (raw_ok) {
      const long long o = (long long)r * a.pitch + gi;
      raw_ps = in_ps[o];
      raw_U = in_U[o];
      raw_D = in_D[o];
    }
  };
  auto load = [&](double& ps, double& ph, double& U, double& jat) {
    ps = ph = U = jat = 0.0;
    if (raw_ok) {
      StF64::ld_pp(raw_ps, c.inv_sqrt2, ps, ph);
      U = StF64::ldU(raw_U, c.U0);
      jat = jat_of(c, U, ph, StF64::ld(raw_D));
    }
  };
  auto right = [&](double v) { return __shfl_down_sync(FULL, v, 1); };
  auto left = [&](double v) { return __shfl_up_sync(FULL, v, 1); };

  // row r+1 ("c") and its right neighbour; row r ("b"); row r-1 ("a")
  double ps_c, ph_c, U_c, j_c, Rps_c, Rph_c, RU_c, Rj_c;
  double ps_b, ph_b, U_b, j_b, Rps_b, Rph_b, RU_b, Rj_b;
  double ps_a, ph_a;
  auto fetch_c = [&]() {  // decode the issued row into "c"
    load(ps_c, ph_c, U_c, j_c);
    Rps_c = right(ps_c);
    Rph_c = right(ph_c);
    RU_c = right(U_c);
    Rj_c = right(j_c);
  };
  auto shift = [&]() {
    ps_a = ps_b;
    ph_a = ph_b;
    ps_b = ps_c; ph_b = ph_c; U_b = U_c; j_b = j_c;
    Rps_b = Rps_c; Rph_b = Rph_c; RU_b = RU_c; Rj_b = Rj_c;
  };
  // plaquette means at (x+1/2, r+1/2) from rows b and c
  auto plaq = [&](double& qs, double& qp) {
    qs = (((ps_b + Rps_b) + ps_c) + Rps_c) * 0.25;
    qp = (((ph_b + Rph_b) + ph_c) + Rph_c) * 0.25;
  };
  // y-edge (x, r+1/2) between rows b and c
  auto yedge = [&](double qs, double qp, double& J, double& Uf) {
    const double Lqs = left(qs), Lqp = left(qp);
    edge_flux<true>(c, merge, qs - Lqs, ps_c - ps_b, qp - Lqp, ph_c - ph_b, ph_b, ph_c, U_b, U_c,
                    j_b, j_c, J, Uf);
  };

  // launched before the previous step has ended: nothing above reads what that writes
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  issue(y0 - 1);
  fetch_c();
  shift();
  issue(y0);
  fetch_c();
  issue(y0 + 1);
  double qs_hi, qp_hi;
  plaq(qs_hi, qp_hi);
  double yJ_hi, yU_hi = 0.0;
  yedge(qs_hi, qp_hi, yJ_hi, yU_hi);

  for (int t = 0; t < a.rows; ++t) {
    const int r = y0 + t;
    if (r > a.fny - 2) break;  // uniform across the warp
    shift();
    fetch_c();      // row r+1, issued one row earlier
    issue(r + 2);   // in flight during this row's arithmetic
    const double qs_lo = qs_hi, qp_lo = qp_hi;
    plaq(qs_hi, qp_hi);
    // x-edge (x+1/2, r)
    double xJ, xU = 0.0;
    edge_flux<false>(c, merge, Rps_b - ps_b, qs_hi - qs_lo, Rph_b - ph_b, qp_hi - qp_lo, ph_b, Rph_b,
                     U_b, RU_b, j_b, Rj_b, xJ, xU);
    const double yJ_lo = yJ_hi, yU_lo = yU_hi;
    yedge(qs_hi, qp_hi, yJ_hi, yU_hi);
    const double xJ_L = left(xJ), xU_L = left(xU);
    const double Lps = left(ps_b), Lph = left(ph_b);
    if (out_col)
      cell_update(a, c, merge, gi, r, ps_b, ph_b, U_b, j_b, xJ, xJ_L, yJ_hi, yJ_lo, xU, xU_L, yU_hi,
                  yU_lo, Rph_b, Lph, ph_c, ph_a, Rps_b, Lps, ps_c, ps_a, o_ps, o_U, o_D);
  }
}


// ---- the FP32-arithmetic storages' march
//
// The same march with the constants folded (FluxConsts) and the shared parts of the
// two edges and the update formed once: 1 - phi^2 and jat/2 are carried with a row,
// one reciprocal root per edge serves the normal and the anisotropy's 1/m^2 (the
// squared gradient is the same before and after the rotation up to its rounding), and
// the row's Up is formed in FP64 once per row by one lane instead of by every lane.
// Bound by instruction issue: 2048x8192 FP32 181 us per step with the general form, 160
// with this one (its 24 bytes per cell would take 61), 2048x4096 FP16 102 and 86.
// 1/m^2 as the root's fourth power is good to about five ulp (a reciprocal of m * m to
// three).  Against FP64 runs that shows nowhere: relative error of U, phi after 60 steps
// of 300x620 8.7e-8, 1.5e-8 with either and 8.6e-8, 1.5e-8 in the general form; after 100
// of 1000x2050 5.9e-8, 9.2e-9 with either and 5.8e-8, 9.4e-9; the reciprocal costs 3 %.

// edge_flux from the sums of the two cells' phi and jat/2 and the difference of
// their U.
template <bool kY, bool kMerge>
__device__ __forceinline__ void edge_flux32(const FluxConsts& c, float psx, float psz, float phx,
                                            float phz, float sph, float dU, float sj, float& J,
                                            float& Uf) {
  const float m = fmaf(phx, phx, phz * phz);
  const bool on = m > c.eps;
  const float r = on ? rsqrt_approx(m) : 0.0f;
  const float ux = fmaf(c.cosa, phx, c.sina * phz), uz = fmaf(c.cosa, phz, -c.sina * phx);
  const float ux2 = ux * ux, uz2 = uz * uz;
  const float r2 = r * r, inv = r2 * r2;
  const float q = fmaf(ux2, ux2, uz2 * uz2);
  const float A = fmaf(q * inv, c.ase, on ? c.a_s : 1.0f);
  const float Ap = (ux * uz) * (ux2 - uz2) * (inv * c.a12);  // -aptheta
  J = A * (kY ? fmaf(A, psz, -Ap * psx) : fmaf(A, psx, Ap * psz));
  if (kMerge) Uf = fmaf(sj, (kY ? phz : phx) * r, fmaf(c.g1, sph, c.g0) * dU);
}

template <class S, bool kMerge>
__global__ void __launch_bounds__(MWARPS * 32) ek2d_march32_kernel(const __grid_constant__ EkArgs a) {
  using V = typename S::V;
  const FluxConsts& c = a.fc;
  const V* in = static_cast<const V*>(a.in);
  V* out = static_cast<V*>(a.out);
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const MarchPos pos = march_pos((a.fnx - 2 + MW - 1) / MW, (a.fny - 2 + a.rows - 1) / a.rows);
  if (!pos.on) return;  // whole warp: uniform
  // lanes past the grid load its last column and store none
  const int gi = pos.group * MW + lane, li = min(gi, a.fnx - 1);
  const bool out_col = lane >= 1 && lane <= MW && gi <= a.fnx - 2;
  const bool rim_col = gi == 1 || gi == a.fnx - 2;  // some halo cell copies it
  const int y0 = 1 + pos.chunk * a.rows, y1 = min(y0 + a.rows, a.fny - 1);
  const uint32_t step_key = mix32(a.step ^ (a.seed * 0x9E3779B9u));
  const float Up_lane = (float)(a.up_a + (double)(y0 + lane) * a.up_b);  // rows <= 32

  // raw values of the next row, loaded one row ahead of their use so that the load
  // latency overlaps the current row's arithmetic (rows past the grid: the last row)
  V raw_ps, raw_U, raw_D;
  auto issue = [&](int r) {
    const V* p = in + (long long)min(r, a.fny - 1) * a.pitch + li;
    raw_ps = p[0];
    raw_U = p[a.plane];
    raw_D = p[2 * a.plane];
  };
  auto right = [&](float v) { return __shfl_down_sync(FULL, v, 1); };
  auto left = [&](float v) { return __shfl_up_sync(FULL, v, 1); };
  // row r+1 ("c") and its right neighbour; row r ("b"); row r-1 ("a"); w = 1 - phi^2,
  // j = jat/2
  float ps_c, ph_c, U_c, w_c, j_c, Rps_c, Rph_c, RU_c, Rj_c;
  float ps_b, ph_b, U_b, w_b, j_b, Rps_b, Rph_b, RU_b, Rj_b;
  float ps_a, ph_a;
  auto fetch_c = [&]() {  // decode the issued row into "c"
    S::ld_pp(raw_ps, c.inv_sqrt2, ps_c, ph_c);
    U_c = S::ldU(raw_U, c.U0);
    w_c = fmaf(-ph_c, ph_c, 1.0f);
    j_c = fmaf(c.j1, U_c, c.j0) * w_c * S::ld(raw_D);
    Rps_c = right(ps_c);
    Rph_c = right(ph_c);
    if (kMerge) {
      RU_c = right(U_c);
      Rj_c = right(j_c);
    }
  };
  auto shift = [&]() {
    ps_a = ps_b;
    ph_a = ph_b;
    ps_b = ps_c; ph_b = ph_c; U_b = U_c; w_b = w_c; j_b = j_c;
    Rps_b = Rps_c; Rph_b = Rph_c; RU_b = RU_c; Rj_b = Rj_c;
  };
  // plaquette means at (x+1/2, r+1/2) from rows b and c
  auto plaq = [&](float& qs, float& qp) {
    qs = (((ps_b + Rps_b) + ps_c) + Rps_c) * 0.25f;
    qp = (((ph_b + Rph_b) + ph_c) + Rph_c) * 0.25f;
  };
  // y-edge (x, r+1/2) between rows b and c
  auto yedge = [&](float qs, float qp, float& J, float& Uf) {
    edge_flux32<true, kMerge>(c, qs - left(qs), ps_c - ps_b, qp - left(qp), ph_c - ph_b, ph_b + ph_c,
                              U_c - U_b, j_b + j_c, J, Uf);
  };

  // launched before the previous step has ended: nothing above reads what that writes
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  issue(y0 - 1);
  fetch_c();
  shift();
  issue(y0);
  fetch_c();
  issue(y0 + 1);
  float qs_hi, qp_hi;
  plaq(qs_hi, qp_hi);
  float yJ_hi, yU_hi = 0.0f;
  yedge(qs_hi, qp_hi, yJ_hi, yU_hi);

  V* o = out + (long long)y0 * a.pitch + gi;
#pragma unroll 2
  for (int r = y0; r < y1; ++r, o += a.pitch) {
    shift();
    fetch_c();     // row r+1, issued one row earlier
    issue(r + 2);  // in flight during this row's arithmetic
    const float qs_lo = qs_hi, qp_lo = qp_hi;
    plaq(qs_hi, qp_hi);
    // x-edge (x+1/2, r)
    float xJ, xU = 0.0f;
    edge_flux32<false, kMerge>(c, Rps_b - ps_b, qs_hi - qs_lo, Rph_b - ph_b, qp_hi - qp_lo,
                               ph_b + Rph_b, RU_b - U_b, j_b + Rj_b, xJ, xU);
    const float yJ_lo = yJ_hi, yU_lo = yU_hi;
    yedge(qs_hi, qp_hi, yJ_hi, yU_hi);
    const float dJ = (xJ - left(xJ)) + (yJ_hi - yJ_lo);
    const float psx = Rps_b - left(ps_b), phx = Rph_b - left(ph_b);  // twice the central
    const float psz = ps_c - ps_a, phz = ph_c - ph_a;                // differences
    const float Up = __shfl_sync(FULL, Up_lane, r - y0);
    float Un = U_b;
    if (kMerge) {
      const float dF = (xU - left(xU)) + (yU_hi - yU_lo);
      Un = fmaf(fmaf(c.dts, j_b, dF * c.dthi), rcp_approx(fmaf(c.nomk, ph_b, c.opk)), U_b);
    }
    // psi with the new U (PF.cu:563-590); the anisotropy is the same of twice the gradient
    const float ux = fmaf(c.cosa, phx, c.sina * phz), uz = fmaf(c.cosa, phz, -c.sina * phx);
    const float ux2 = ux * ux, uz2 = uz * uz, m = ux2 + uz2;
    const float A = m > c.eps4
                        ? fmaf(fmaf(ux2, ux2, uz2 * uz2) * rcp_approx(m * m), c.ase, c.a_s)
                        : 1.0f;
    const float A2 = A * A;
    const float g4 = fmaf(psx, psx, psz * psz);
    const float lap = fmaf(A2 * ph_b * c.nex, g4, dJ);
    const float rhs = fmaf(w_b * (Un + Up), c.nlam, fmaf(lap, c.hi2, ph_b * c.sqrt2));
    const float tp = fmaxf(fmaf(c.nomk, Up, 1.0f), c.k);
    const float dps = rhs * rcp_approx(tp * A2);
    float psn = fmaf(c.dt, dps, ps_b);
    if (!out_col) continue;
    if (a.noise_amp != 0.0f && in_band(ph_b)) {
      const Philox4 rn = philox4x32_10((uint32_t)gi, (uint32_t)r, a.step, 0x4E4F4953u, a.seed, 0x5EEDu);
      psn += a.noise_amp * ((float)uniform01(rn.v[0]) - 0.5f);
    }
    V vps, vU, vD;
    encode_cell<S>(a, kMerge, step_key, gi, r, psn, Un, dps, vps, vU, vD);
    o[0] = vps;
    o[a.plane] = vU;
    o[2 * a.plane] = vD;
    if (rim_col || r == 2 || r == a.fny - 3)
      put_with_halo(out, out + a.plane, out + 2 * a.plane, a.pitch, a.fnx, a.fny, r, gi, vps, vU, vD);
  }
}

// ---- auxiliary kernels -------------------------------------------------------

// Reference-layout floats (psi, U, dpsi) -> storage, interior cells with their
// halo copies.  dpsi may be null (zeros).
template <class S>
__global__ void ek2d_import_kernel(const float* ps, const float* U, const float* D, void* out,
                                   long long plane, int pitch, int fnx, int fny, float U0) {
  using V = typename S::V;
  using T = typename S::T;
  const long long n = (long long)(fnx - 2) * (fny - 2);
  V* o_ps = static_cast<V*>(out);
  V* o_U = o_ps + plane;
  V* o_D = o_U + plane;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = 1 + (int)(e % (fnx - 2)), j = 1 + (int)(e / (fnx - 2));
    const long long src = (long long)j * fnx + i;
    put_with_halo(o_ps, o_U, o_D, pitch, fnx, fny, j, i, S::st_ps((T)ps[src]), S::stU((T)U[src], (T)U0),
                  S::st(D ? (T)D[src] : (T)0));
  }
}

// Storage -> reference layout (halos included) in float or double;
// phi = tanh(psi/sqrt2).
template <class S, class O>
__global__ void ek2d_export_kernel(const void* in, long long plane, int pitch, int fnx, int fny,
                                   float U0, float sqrt2, O* ps, O* ph, O* U, O* D) {
  using V = typename S::V;
  using T = typename S::T;
  const long long n = (long long)fnx * fny;
  const V* i_ps = static_cast<const V*>(in);
  const V* i_U = i_ps + plane;
  const V* i_D = i_U + plane;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % fnx), j = (int)(e / fnx);
    const long long o = (long long)j * pitch + i;
    T p, q;
    S::ld_pp(i_ps[o], (T)1 / (T)sqrt2, p, q);
    if (ps) ps[e] = (O)p;
    if (ph) ph[e] = (O)q;
    if (U) U[e] = (O)S::ldU(i_U[o], (T)U0);
    if (D) D[e] = (O)S::ld(i_D[o]);
  }
}

// Sum of phi over each row, halo columns included (one CTA per row, FP64).
template <class S>
__global__ void ek2d_row_sums_kernel(const void* in, int pitch, int fnx, float sqrt2, double* out) {
  using V = typename S::V;
  using T = typename S::T;
  const V* row = static_cast<const V*>(in) + (long long)blockIdx.x * pitch;
  double s = 0.0;
  const T inv = (T)1 / (T)sqrt2;
  for (int i = threadIdx.x; i < fnx; i += blockDim.x) {
    T p, q;
    S::ld_pp(row[i], inv, p, q);
    s += (double)q;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  __shared__ double warp_sums[32];
  if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += warp_sums[w];
    out[blockIdx.x] = t;
  }
}

// Move the frame up by `k` rows (k single-row moves of move_frame/copy_frame,
// PF.cu:625-668): row j takes row j+k; the top k rows continue the linear
// extrapolation psi_new = 2 psi[fny-2] - psi[fny-3] one row at a time, and U
// there is U0.  dpsi is not moved (the reference moves psi, phi and U only).
template <class S>
__global__ void ek2d_shift_kernel(const void* in, void* out, long long plane, int pitch, int fnx,
                                  int fny, int k, float U0) {
  using V = typename S::V;
  using T = typename S::T;
  const long long n = (long long)(fnx - 2) * (fny - 2);
  const V* i_ps = static_cast<const V*>(in);
  const V* i_U = i_ps + plane;
  const V* i_D = i_U + plane;
  V* o_ps = static_cast<V*>(out);
  V* o_U = o_ps + plane;
  V* o_D = o_U + plane;
  const V vU0 = S::stU((T)U0, (T)U0);
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = 1 + (int)(e % (fnx - 2)), j = 1 + (int)(e / (fnx - 2));
    V vps, vU;
    if (j + k <= fny - 2) {
      const long long src = (long long)(j + k) * pitch + i;
      vps = i_ps[src];
      vU = i_U[src];
    } else {
      T em2, em1, q;
      S::ld_pp(i_ps[(long long)(fny - 3) * pitch + i], (T)0.70710678118654752, em2, q);
      S::ld_pp(i_ps[(long long)(fny - 2) * pitch + i], (T)0.70710678118654752, em1, q);
      const int m = j - (fny - 2 - k);
      for (int t = 0; t < m; ++t) {
        const T en = (T)2 * em1 - em2;
        em2 = em1;
        em1 = en;
      }
      vps = S::st_ps(em1);
      vU = vU0;
    }
    put_with_halo(o_ps, o_U, o_D, pitch, fnx, fny, j, i, vps, vU, i_D[(long long)j * pitch + i]);
  }
}

}  // namespace ek2d
}  // namespace cupf
