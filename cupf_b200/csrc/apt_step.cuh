// apt_step.cuh — the fused APT step kernel for sm_100a.
//
// One launch = one explicit step of the reference's APTsetBC3D + APTrhs_psi
// pair (3DgrainMPI/APTPhaseField.cu:93-174, 178-354): boundary fill, neighbour
// grain-id gather with the first-seen merge, per-slot anisotropic update.
//
// Work decomposition: a CTA owns a TX x TY column tile of interior (x, y) cells
// (TX = 32, one warp per tile row; TY = 8 or 4, a template parameter the host
// picks per simulation, the server by timing) and a z chunk of ZC planes; one
// thread per (x, y) column marches z.  Planes of
// the input pair buffer (all NUM_PF slots, tile plus one-cell halo) stream into
// shared memory through a ring of STAGES stages filled by TMA
// (cp.async.bulk.tensor.4d, one 4-D box {TX+2, TY+2, 1, NP} per plane) and
// completed on per-stage mbarriers.  Computing plane k needs planes k-1, k, k+1
// resident; plane k+2 is in flight.
//
// Boundary fill: plane indices 0 and fnz-1 are loaded from their mapped source
// planes (TMA coordinate remap), and the x/y halo cells are read from HBM,
// where they hold their mapped interior source: the step writes every cell it
// computes also into the halo cells that map to it, and every other writer of
// the pair buffers (initialisation, import, nucleation, domain shift) is
// followed by a fill of the halo.  Halo edges and corners, which no 7-point
// stencil reads, are not maintained by the step.
//
// Slot maps.  An output slot j of a cell holds one grain; the slot where each of
// the 7 stencil points holds that grain follows from the points' ordered id
// lists alone (the first-seen merge in the reference's order (D,B,L,C,R,T,U) x
// slot).  It is kept per cell as one word per output slot, the slot map: 4 bits
// per point, NUM_PF where the point lacks the grain.  The lists change seldom (a
// front or tail crossing the cell), so the map belongs to the simulation's state
// beside the pairs: a step merges again only the cells whose own or face
// neighbours' lists changed in the step before.  Whoever changes a cell's list
// marks the cells that read it (mark_readers) for the next step; whoever replaces
// the whole state invalidates every map.  A few marked cells are merged by the warp
// together, four a pass with a lane per stencil point, so that scattered cells do not
// hold up a warp's other lanes; a row with many by its own lanes (row_merge), as every
// row is where the device has no room for maps.
//
// What bounds it: instruction issue and latency, not bytes.  128x128x256 line case, NUM_PF
// = 8, on a B200, us per step over steps 1-20, 21-50 and 51-150 (all-empty items left
// alone): FP32 220, 181, 163, where no maps are kept 273, 286, 286, and with the merge of
// every cell that the maps replaced 213, 232, 230; FP16 202, 156, 144; 231, 236, 242; 182,
// 200, 198.  In the first steps, while every grain's tail grows a cell a step, a quarter
// of the cells and more are merged: there the maps cost more than they save.
//
// The reference's aliasing write on merge overflow (local_phs[s][NUM_PF] ==
// local_phs[s+1][0]) is restated: such cells are merged every step.
#pragma once

#include "apt_storage.cuh"
#include "apt_update.cuh"

namespace cupf {

constexpr int TX = 32;
// Three planes in use and one in flight; a stage also holds a row of empty pairs
// (slot NUM_PF, never written by the loads), which an absent grain's code reads.
constexpr int STAGES = 4;

// Column-tile heights the step is built for (the box height is TY + 2 cells; the
// box width is the storage format's kBW).
constexpr bool tile_height_built(int ty) { return ty == 8 || ty == 4; }
template <int TY>
constexpr int tile_threads() {
  return TX * TY;
}

template <int NP, class S, int TY>
struct StepSmem {
  static constexpr int BW = S::kBW;
  static constexpr int BH = TY + 2;
  static constexpr int BCELLS = BW * BH;
  static constexpr int kBoxBytes = NP * BCELLS * S::kBytes;  // bytes one TMA plane load delivers
  // stage stride (TMA dst: 128 B aligned), with the row of empty pairs
  static constexpr int kStageBytes = ((NP + 1) * BCELLS * S::kBytes + 127) & ~127;
  static constexpr int kStagePairs = kStageBytes / S::kBytes;
  // 16-bit pairs in 32x8 tiles: the centre plane's phi values decoded once per
  // plane into FP32 (slot-major like a stage, plus the row of -1), read by the
  // five stencil points in that plane.  Three CTAs per SM still fit; for 32x4
  // tiles the extra row would cost one.
  static constexpr bool kDecode = S::kBytes == 4 && TY == 8;
  static constexpr int kDecOff = STAGES * kStageBytes;
  static constexpr int kDecBytes = kDecode ? (NP + 1) * BCELLS * 4 : 0;
  // per warp: its cells' slot-map words, and the merged cells' results and alias words
  static constexpr int kWordOff = kDecOff + kDecBytes;
  static constexpr int kBarOff = kWordOff + TY * (NP + 2) * 32 * 4;
  // + abort word, issued count, item index
  static constexpr int kBytes = kBarOff + STAGES * 8 + 16;
};

// Slot-map words: 4-bit slot code of stencil point s in bits 4s..4s+3; the top 4
// bits of slot 0's word hold the cell's slot count, or one of these marks.
constexpr uint32_t kMapCodes = 0x0FFFFFFFu;
constexpr uint32_t kMapEveryStep = 0xEu;  // merge overflow: merge this cell every step
constexpr uint32_t kMapInvalid = 0xFu;    // nothing known (also what a byte-wise fill with 0xFF leaves)

__device__ __forceinline__ uint32_t map_code(uint32_t w, int s) { return (w >> (4 * s)) & 0xFu; }

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Wait for a stage with a bounded spin: by default about one second of SM
// clock (kWaitCycles), then give up and report (the caller records an error and
// carries on so that every thread still reaches every barrier).  A try_wait may
// itself suspend the thread for a hardware-chosen interval, so a bound shorter
// than kShortWait is kept with non-blocking probes only.
constexpr long long kWaitCycles = 1ll << 31;
constexpr long long kShortWait = 1ll << 20;
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity,
                                                  long long limit = kWaitCycles) {
  if (limit < kShortWait) {
    const long long t0 = clock64();
    do {
      if (mbar_test_wait(bar, parity)) return true;
    } while (clock64() - t0 <= limit);
    return false;
  }
  if (mbar_try_wait(bar, parity)) return true;
  long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (clock64() - t0 > limit) return false;
  }
  return true;
}

__device__ __forceinline__ void tma_load_plane(void* dst, const CUtensorMap* map, uint64_t* bar,
                                               int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(0), "r"(smem_u32(bar))
      : "memory");
}

// Copy one word from global to shared memory without a register (asynchronous; this
// thread's copies have landed after copy_wait).
__device__ __forceinline__ void copy_word(uint32_t* dst, const uint32_t* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Per-CTA shared-memory state, carved from the dynamic allocation.
template <int NP, class S, int TY>
struct CtaSmem {
  using P = typename S::T;
  using Smem = StepSmem<NP, S, TY>;
  P* stages;
  float* dec;     // decoded centre plane (Smem::kDecode)
  uint32_t* wbuf; // merged cells (Smem::kWordOff)
  uint64_t* bars;
  int* s_abort;   // global plane sequence number of the first failed wait, + 1
  int* s_issued;  // plane sequence numbers issued so far (written by thread 0)
  int* s_item;    // work item handed to the CTA
  __device__ explicit CtaSmem(unsigned char* smem) {
    stages = reinterpret_cast<P*>(smem);
    dec = reinterpret_cast<float*>(smem + Smem::kDecOff);
    wbuf = reinterpret_cast<uint32_t*>(smem + Smem::kWordOff);
    bars = reinterpret_cast<uint64_t*>(smem + Smem::kBarOff);
    s_abort = reinterpret_cast<int*>(smem + Smem::kBarOff + STAGES * 8);
    s_issued = s_abort + 1;
    s_item = s_abort + 2;
  }
  __device__ void init() {
    if (threadIdx.x == 0) {
      for (int s = 0; s < STAGES; ++s) mbar_init(&bars[s], 1);
      *s_abort = 0;
      *s_issued = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int c = threadIdx.x; c < Smem::BCELLS; c += blockDim.x) {
      for (int s = 0; s < STAGES; ++s)
        stages[(size_t)s * Smem::kStagePairs + NP * Smem::BCELLS + c] = S::empty();
      if (Smem::kDecode) dec[NP * Smem::BCELLS + c] = -1.0f;
    }
    __syncthreads();
  }
  // After a timed-out wait no further loads are issued; before the CTA exits
  // (and its shared memory is reused) wait, bounded by the default limit
  // whatever the launch's own, for those in flight.
  __device__ void drain() {
    __syncthreads();
    if (threadIdx.x == 0 && *s_abort) {
      for (int q = *s_abort - 1; q < *s_issued; ++q)
        mbar_wait_bounded(&bars[q % STAGES], (uint32_t)((q / STAGES) & 1));
    }
  }
};

// The merge of one cell by its own lane: the first-seen order over (D,B,L,C,R,T,U) x
// slot.  Writes the cell's slot-map words to wcol and returns what the warp's merge
// (step_item) does: the slot count in bits 28..31, merge overflows aliased (low byte)
// and dropped (second byte), a list of the centre's that loses a grain (bit 16), an
// overflow (bit 17), with its alias word second.  pD, pC, pU: the cell in its planes.
//
// The list starts as the point below's.  An entry of another point whose grain stands
// in that same slot needs no search (a cell's slots stand in the first-seen order of
// its own neighbourhood, which starts with the column); the few others are looked up
// one by one, in order.
template <int NP, class S, int BW, int BCELLS>
__device__ __forceinline__ uint2 merge_cell(const typename S::T* pD, const typename S::T* pC,
                                            const typename S::T* pU, uint32_t* wcol) {
  auto point = [&](int s) {
    return s == 0 ? pD : s == 6 ? pU : pC + (s == 1 ? -BW : s == 2 ? -1 : s == 4 ? 1 : s == 5 ? BW : 0);
  };
  int list[NP];  // the grains placed so far; below -1: none
  uint32_t occ = 0;
  bool odd = false;  // a hole or a repeated grain in the list of the point below
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    const int id = S::id(pD[p * BCELLS]);
    occ |= (uint32_t)(id != -1) << p;
    list[p] = id != -1 ? id : -2 - p;
#pragma unroll
    for (int q = 0; q < p; ++q) odd = odd || list[p] == list[q];
  }
  odd = odd || (occ & (occ + 1)) != 0;
  uint32_t todo[2] = {odd ? occ : 0u, 0u};  // entries to look up: 8 bits a point, 4 points a word
  int cnt = odd ? 0 : __popc(occ);
  uint32_t w[NP];
#pragma unroll
  for (int p = 0; p < NP; ++p) {
    if (odd) list[p] = -2;
    w[p] = (uint32_t)NP * 0x1111111u;
    if (list[p] >= 0) w[p] -= (uint32_t)(NP - p);
  }
#pragma unroll
  for (int s = 1; s < 7; ++s) {
    const typename S::T* pt = point(s);
#pragma unroll
    for (int p = 0; p < NP; ++p) {
      const int id = S::id(pt[p * BCELLS]);
      if (id == list[p]) w[p] -= (uint32_t)(NP - p) << (4 * s);
      if (id != list[p] && id != -1) todo[s >> 2] |= 1u << (8 * (s & 3) + p);
    }
  }
#pragma unroll
  for (int p = 0; p < NP; ++p) wcol[p * 32] = w[p];
  uint32_t info = 0, al = 0xFFFFFFFFu;
  while (todo[0] | todo[1]) {
    const bool hi = todo[0] == 0;
    const int b = __ffs(hi ? todo[1] : todo[0]) - 1;
    if (hi)
      todo[1] &= todo[1] - 1;
    else
      todo[0] &= todo[0] - 1;
    const int s = (b >> 3) + (hi ? 4 : 0), p = b & 7;
    const int id = S::id(point(s)[p * BCELLS]);
    int j = cnt;
#pragma unroll
    for (int q = NP - 1; q >= 0; --q)
      if (list[q] == id) j = q;
    if (j == NP) {  // overflow: the last entry's value is the one aliased
      info = (info | 1u << 17 | (uint32_t)(s == 3) << 16) + (s < 6 ? 1u : 0x100u);
      if (s < 6) al = (al & ~(0xFu << (4 * s + 4))) | ((uint32_t)p << (4 * s + 4));
      continue;
    }
    if (j == cnt) {
#pragma unroll
      for (int q = 0; q < NP; ++q)
        if (q == j) list[q] = id;
      ++cnt;
    }
    // the last slot holding the id, as the reference's later write wins; an id repeated
    // in the centre's list does not survive the step
    const uint32_t old = wcol[j * 32], at = map_code(old, s);
    if (at == (uint32_t)NP) {
      wcol[j * 32] = old - ((uint32_t)(NP - p) << (4 * s));
    } else {
      if ((uint32_t)p > at) wcol[j * 32] = old + (((uint32_t)p - at) << (4 * s));
      info |= (uint32_t)(s == 3) << 16;
    }
  }
  if (info & (1u << 17)) {
    // a point's own grain of slot 0 overwrites the value aliased there
#pragma unroll
    for (int s = 1; s < 7; ++s)
      if (map_code(wcol[0], s) != (uint32_t)NP) al |= 0xFu << (4 * s);
  }
  return make_uint2(info | ((uint32_t)cnt << 28), al);
}

// The same out of line.
template <int NP, class S, int BW, int BCELLS>
__device__ __noinline__ uint2 merge_cell_call(const typename S::T* pD, const typename S::T* pC,
                                              const typename S::T* pU, uint32_t* wcol) {
  return merge_cell<NP, S, BW, BCELLS>(pD, pC, pU, wcol);
}

// A row with more marked cells than this is merged by its own lanes; 0: by the warp's
// passes whatever their number, as long as maps are kept.  The line lies where a row by
// its own lanes costs what its passes do: the fewer the slots, the cheaper the former, and
// with up to three the passes are not built at all (most cells of an interface then
// overflow and are merged every step).  Measured on a B200, us per step over the first 20
// steps and over steps 51-150:
//   NUM_PF = 8 FP32, passes only -> 28: line 128x128x256 233, 164 -> 220, 163; pool
//     256x256x768 5380, 4673 -> 5200, 4620.  16-bit pairs there keep to the passes, since
//     the pool's FP64 model leaves little of the instruction cache: 28 marks 5241, 4597
//     against 5114, 4414 (line 198, 144 against 202, 144);
//   28 -> this, FP32: NUM_PF = 6 200x150x100 150.4, 112.7 -> 149.9, 112.6; 5 128^3 90.8, 73.5
//     -> 89.3, 73.4; 4 160x128x128 96.3, 82.0 -> 94.3, 81.1; 3 128^3 74.3, 67.1 -> 67.3, 61.8;
//     2 62.7, 56.9 -> 54.4, 50.2; 1 47.6, 45.1 -> 45.3, 42.8;
//   never -> this, FP16: 7 160x160x128 164.5, 120.8 -> 158.9, 121.1; 6 141.5, 100.5 -> 133.8,
//     100.7; 5 98.4, 76.0 -> 92.9, 76.0; 4 109.0, 87.8 -> 99.2, 87.3; 3 84.7, 72.7 -> 72.0,
//     66.2; 2 72.4, 62.1 -> 58.7, 54.6; 1 56.3, 48.9 -> 46.3, 43.8.
// Without maps (NUM_PF = 8, steps 51-150): FP32 line 317 with passes, 286 by lanes, pool
// 7611 and 5894; FP16 276 and 242, 7000 and 5667.
template <int NP, class S>
constexpr int row_merge() {
  return NP <= 3 ? 0
         : NP == 4 ? 12
         : NP == 5 ? 20
         : NP == 6 ? (S::kBytes == 8 ? 24 : 20)
         : NP == 7 ? (S::kBytes == 8 ? 28 : 24)
                   : (S::kBytes == 8 ? 28 : 0);
}

// One work item: the column tile (txi, tyi) over the z chunk zci of one
// simulation.  qbase is the CTA's running plane sequence number: plane q of
// this item is sequence number qbase + q, which fixes its stage (mod STAGES)
// and the mbarrier phase parity; every issued plane is waited exactly once, in
// order, so the phases stay consistent across items.
template <int NP, class S, int TY>
__device__ __forceinline__ void step_item(const CUtensorMap* tmap, const StepArgs& a, int txi,
                                          int tyi, int zci, CtaSmem<NP, S, TY>& sm, int& qbase) {
  static_assert(NP <= 8, "slot codes are 4-bit fields, merge entries 8 per stencil point");
  using Smem = StepSmem<NP, S, TY>;
  constexpr int NTHREADS = tile_threads<TY>();
  using P = typename S::T;
  constexpr int BW = Smem::BW;
  constexpr int BCELLS = Smem::BCELLS;
  constexpr bool kDec = Smem::kDecode;
  constexpr int kRowMerge = row_merge<NP, S>();
  constexpr unsigned FULL = 0xffffffffu;
  // offsets of the centre plane's stencil points B, L, C, R, T from the cell
  constexpr int ctr_off[7] = {0, -BW, -1, 0, 1, BW, 0};
  P* stages = sm.stages;
  uint64_t* bars = sm.bars;
  int* s_abort = sm.s_abort;
  int* s_issued = sm.s_issued;
  P* gout = static_cast<P*>(a.out);

  const int tid = threadIdx.x;
  const int tx = tid % TX, ty = tid / TX;
  const int lane = tx;  // TX == warp size: a warp is one tile row
  const int x0 = 1 + TX * txi;  // first interior x of the tile
  const int y0 = 1 + TY * tyi;
  const int k_begin = 1 + a.zc * zci;
  const int k_end = min(k_begin + a.zc, a.fnz - 1);
  const int nplanes = k_end - k_begin + 2;  // planes k_begin-1 .. k_end
  const long long ss = a.slot_stride;
  const long long plane_pairs = (long long)a.xp * a.fny;
  const int q0 = qbase;

  auto issue = [&](int q) {  // plane index q -> logical z = k_begin - 1 + q
    const int g = q0 + q;
    const int s = g % STAGES;
    const int zl = k_begin - 1 + q;
    const int zp = bc_map(zl, a.fnz, a.bcZ);
    mbar_arrive_expect_tx(&bars[s], Smem::kBoxBytes);
    tma_load_plane(stages + (size_t)s * Smem::kStagePairs, tmap, &bars[s], x0 - 1, y0 - 1, zp);
    *s_issued = g + 1;
  };

  // the previous item (if any) is done with every stage before they refill
  __syncthreads();
  if (tid == 0 && !*s_abort) {
    fence_proxy_async();
    const int npre = min(STAGES, nplanes);
    for (int q = 0; q < npre; ++q) issue(q);
  }

  // Wait for plane q.
  auto land = [&](int q) {
    const int g = q0 + q;
    const int s = g % STAGES;
    const uint32_t parity = (uint32_t)((g / STAGES) & 1);
    if (!*s_abort && !mbar_wait_bounded(&bars[s], parity, a.wait_limit)) {
      atomicCAS(s_abort, 0, g + 1);
      atomicExch(a.err, ERR_TMA_TIMEOUT);
    }
  };

  // bit 0: this thread wrote a slot other than the exact empty pair (an occupied
  // slot, or one whose id was just dropped: it keeps its last phi) or left one
  // unwritten; bits 1 and 2: the same in the item's bottom and top plane
  uint32_t live = 0;
  // merge overflows of this thread's cells (StepArgs::overflows), aliased ones
  // in the low 16 bits and dropped ones in the high 16 (at most 7 NP per cell
  // and plane), summed per warp at the end of the item
  uint32_t n_ovf = 0;

  const int gx = x0 + tx, gy = y0 + ty;
  const bool valid = gx <= a.fnx - 2 && gy <= a.fny - 2;
  const int c = (ty + 1) * BW + (tx + 1);
  // offsets (in pairs, 0 = none) from this cell to the x/y halo cells whose
  // boundary map sources it (APTsetBC3D, APTPhaseField.cu:93-174)
  const int hdx0 = bc_map(0, a.fnx, a.bcX) == gx ? -gx : 0;
  const int hdx1 = bc_map(a.fnx - 1, a.fnx, a.bcX) == gx ? a.fnx - 1 - gx : 0;
  const int hdy0 = bc_map(0, a.fny, a.bcY) == gy ? -gy * a.xp : 0;
  const int hdy1 = bc_map(a.fny - 1, a.fny, a.bcY) == gy ? (a.fny - 1 - gy) * a.xp : 0;
  // (false for a whole warp away from the faces)
  const bool halo_any = __any_sync(FULL, valid && (hdx0 | hdx1 | hdy0 | hdy1) != 0);
  // the line profile and the liquid-start undercooling depend on z only: one
  // evaluation per plane instead of one per cell (32 planes at a time, one a lane)
  const bool plane_T = a.use_iuc || a.thermalType == 0 || a.thermalType == 1;
  const float kLS = __uint_as_float(kLSFloatBits);
  const float kDrop = __uint_as_float(kDropFloatBits);
  const KineConst kc = kine_const(a.kin_delta);
  // this lane's part of a warp's merges: stencil point lane % 8 (7: none) of the
  // pass's cell lane / 8; offset in pairs from the point's plane to the first cell
  // of the warp's row
  const int m_grp = lane >> 3, m_pt = lane & 7;
  const int m_off = (ty + 1) * BW + 1 +
                    (m_pt == 1 ? -BW : m_pt == 2 ? -1 : m_pt == 4 ? 1 : m_pt == 5 ? BW : 0);
  uint32_t* wbuf = sm.wbuf + ty * ((NP + 2) * 32);
  uint32_t* wcol = wbuf + lane;  // this cell's words, 32 apart

  // the next plane's word 0 and change marks, loaded a plane ahead
  const long long cell0 = (long long)k_begin * plane_pairs + (long long)gy * a.xp + gx;
  uint32_t next_w0 = kMapInvalid << 28;
  uint8_t next_r0 = 0, next_r1 = 0;
  auto prefetch = [&](long long cell) {
    if (a.map) {
      next_w0 = a.map[cell];
      next_r0 = a.redo_in[cell];
      next_r1 = a.redo_out[cell];
    }
  };
  if (valid) prefetch(cell0);

  float Up_lane = 0.0f;
  land(0);
  land(1);
  for (int k = k_begin; k < k_end; ++k) {
    const int qk = k - k_begin + 1;
    const long long cell = cell0 + (long long)(k - k_begin) * plane_pairs;
    const uint32_t w0 = next_w0 & kMapCodes;
    int n = (int)(next_w0 >> 28);
    // a mark left in redo_out by an earlier step (the item was not computed since)
    // counts too; a neighbour setting it for the next step meanwhile costs only a
    // merge with the same result
    const bool need = valid && (n > NP || next_r0 || next_r1);
    const bool had_mark = next_r0 != 0;
    if (!valid || need) n = 0;
    // the cell's words into its column of the warp's buffer
    if (n > 0) wcol[0] = w0;
#pragma unroll
    for (int j = 1; j < NP; ++j)
      if (j < n) copy_word(wcol + j * 32, a.map + j * ss + cell);
    if (valid && k + 1 < k_end) prefetch(cell + plane_pairs);
    if (plane_T && (qk & 31) == 1) {  // lane l: plane k + l
      float T;
      tinterp(a, 0, 0, min(k + lane, a.fnz - 1), &T);
      Up_lane = __fdiv_rn(T, a.L_cp);
    }
    const float Up_plane = __shfl_sync(FULL, Up_lane, (qk - 1) & 31);
    land(qk + 1);
    const int sD = (q0 + qk - 1) % STAGES, sC = (q0 + qk) % STAGES, sU = (q0 + qk + 1) % STAGES;
    P* stC = stages + (size_t)sC * Smem::kStagePairs;
    // every thread has finished the previous plane at this barrier
    bool occ = true;
    if (kDec)
      occ = __syncthreads_or(n > 0 || need) != 0;
    else
      __syncthreads();
    if (tid == 0 && qk >= 2 && qk - 2 + STAGES < nplanes && !*s_abort) {
      fence_proxy_async();
      issue(qk - 2 + STAGES);
    }
    // decode the centre plane's phi once (unless no cell reads it)
    if constexpr (kDec) {
      if (occ) {
        // four pairs per thread and pass (a stage and the decoded plane start on
        // 16-byte boundaries; NP * BCELLS is a multiple of 4)
        static_assert((NP * BCELLS) % 4 == 0, "vector decode");
        const uint4* st = reinterpret_cast<const uint4*>(stC);
        float4* d4 = reinterpret_cast<float4*>(sm.dec);
        for (int e = tid; e < NP * BCELLS / 4; e += NTHREADS) {
          const uint4 v = st[e];
          d4[e] = make_float4(S::phi(v.x), S::phi(v.y), S::phi(v.z), S::phi(v.w));
        }
        __syncthreads();
      }
    }
    const P* plD = stages + (size_t)sD * Smem::kStagePairs;
    const P* plU = stages + (size_t)sU * Smem::kStagePairs;

    // ---- merge of the warp's marked cells: first-seen order over (D,B,L,C,R,T,U) x
    // slot.  In a pass eight lanes take a cell, lane s the list of point s; each turn
    // places the first grain not placed yet, and every lane finds the slot it has in its
    // own list.  The turns give a word per point; its transpose the words per slot.
    uint32_t alias = 0xFFFFFFFFu;  // slot at point s-1 whose value sits in slot 0 of point s
    bool force_mark = false;
    uint32_t todo = __ballot_sync(FULL, need);
    uint32_t info = 0;
    if (todo && (NP <= 3 || !a.map || (kRowMerge && __popc(todo) > kRowMerge))) {
      if (need) {  // most of the row, or every cell of every step: a lane per cell
        uint2 r;
        // inline where that is the faster (NUM_PF = 5 FP32, 64^3: 16.6 against 16.9; the
        // other way round 4 FP32, 96^3: 39.8 against 38.4, and the pool in 16-bit pairs)
        if constexpr ((S::kBytes == 8 && NP >= 5) || NP <= 3)
          r = merge_cell<NP, S, BW, BCELLS>(plD + c, stC + c, plU + c, wcol);
        else
          r = merge_cell_call<NP, S, BW, BCELLS>(plD + c, stC + c, plU + c, wcol);
        info = r.x;
        if (info & (1u << 17)) alias = r.y;
      }
    } else if (todo) {
      const P* mp = (m_pt == 0 ? plD : m_pt == 6 ? plU : stC) + m_off;
      do {
        int src = -1;  // the pass's cells: the lowest four marked lanes
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          if (m_grp == g) src = __ffs(todo) - 1;
          todo &= todo - 1;
        }
        const bool on = src >= 0 && m_pt < 7;
        const P* mc = mp + max(src, 0);
        int id[NP];
        uint32_t un = 0;  // slots of this point's list whose grain is not placed yet
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          id[p] = S::id(mc[p * BCELLS]);
          un |= (uint32_t)(id[p] != -1) << p;
        }
        if (!on) un = 0;
        uint32_t codes = m_pt < 7 ? (uint32_t)NP * 0x11111111u : 0u;
        uint32_t dup = 0;
        int cnt = 0;
#pragma unroll
        for (int j = 0; j < NP; ++j) {
          const uint32_t act = __ballot_sync(FULL, un != 0);
          if (!act) break;
          const uint32_t mine = (act >> (8 * m_grp)) & 0xFFu;
          const int cand = S::id(mc[(un ? __ffs(un) - 1 : 0) * BCELLS]);
          const int gid = __shfl_sync(FULL, cand, 8 * m_grp + (mine ? __ffs(mine) - 1 : 0));
          uint32_t m = 0;
#pragma unroll
          for (int p = 0; p < NP; ++p) m |= (uint32_t)(id[p] == gid) << p;
          if (!mine || !on) m = 0;
          un &= ~m;
          // the last slot holding the id, as the reference's later write wins
          if (m) codes -= ((uint32_t)NP - (31u - (uint32_t)__clz(m))) << (4 * j);
          dup |= m & (m - 1);
          cnt += mine != 0;
        }
        // an id repeated in the centre's list does not survive the step
        uint32_t res = (uint32_t)cnt << 28;
        if (__any_sync(FULL, un | (m_pt == 3 ? dup : 0u))) {
          // merge overflow: local_phs[s][NUM_PF] aliases local_phs[s+1][0], which
          // point s+1's own grain of slot 0 overwrites; past the array at s == 6
          const uint32_t below = __shfl_up_sync(FULL, un, 1);
          const bool spill = m_pt >= 1 && m_pt <= 6 && below && (codes & 0xFu) == (uint32_t)NP;
          uint32_t al = 0xFFFFFFFFu;
          if (spill) al = ~(0xFu << (4 * m_pt)) | ((31u - (uint32_t)__clz(below)) << (4 * m_pt));
          // entries aliased (low byte) and dropped (second byte); a list that loses
          // an overflowing or repeated grain of the centre (bit 16); overflow (bit 17)
          uint32_t q = m_pt < 6 ? (uint32_t)__popc(un) : (uint32_t)__popc(un) << 8;
          uint32_t f = (m_pt == 3 && (un | dup) ? 1u << 16 : 0u) | (un ? 1u << 17 : 0u);
#pragma unroll
          for (int d = 1; d < 8; d <<= 1) {
            al &= __shfl_xor_sync(FULL, al, d);
            q += __shfl_xor_sync(FULL, q, d);
            f |= __shfl_xor_sync(FULL, f, d);
          }
          res |= q | f;
          if (src >= 0 && m_pt == 7) wbuf[(NP + 1) * 32 + src] = al;
        }
        // transpose the eight lanes' 4-bit fields: lane j gets slot j's word
#pragma unroll
        for (int d = 4; d; d >>= 1) {
          const uint32_t keep = d == 4 ? 0x0000FFFFu : d == 2 ? 0x00FF00FFu : 0x0F0F0F0Fu;
          const uint32_t o = __shfl_xor_sync(FULL, codes, d);
          codes = (m_pt & d) ? (codes & ~keep) | ((o >> (4 * d)) & keep)
                             : (codes & keep) | ((o & keep) << (4 * d));
        }
        if (src >= 0) {
          if (m_pt < NP) wbuf[m_pt * 32 + src] = codes;
          if (m_pt == 7) wbuf[NP * 32 + src] = res;
        }
      } while (todo);
      __syncwarp();
      if (need) {
        info = wbuf[NP * 32 + lane];
        if (info & (1u << 17)) alias = wbuf[(NP + 1) * 32 + lane];
      }
      __syncwarp();  // the buffer is rewritten at the next plane
    }
    if (need) {
      n = (int)(info >> 28);
      if (info & 0x3FFFFu) {
        force_mark = (info >> 16) & 1u;
        n_ovf += (info & 0xFFu) + ((info & 0xFF00u) << 8);
      }
      if (a.map) {
        const uint32_t mark0 = info & (1u << 17) ? kMapEveryStep : (uint32_t)n;
        a.map[cell] = (n ? wcol[0] : 0u) | (mark0 << 28);
#pragma unroll
        for (int j = 1; j < NP; ++j)
          if (j < n) a.map[j * ss + cell] = wcol[j * 32];
        if (had_mark) a.redo_in[cell] = 0;
      }
    }
    copy_wait();
    if (!valid) continue;

    P* outp = gout + cell;
    // write pair v to output slot j of this cell and to the halo cells it sources
    auto put = [&](int j, P v) {
      P* o = outp + j * ss;
      *o = v;
      if (halo_any) {
        if (hdx0) o[hdx0] = v;
        if (hdx1) o[hdx1] = v;
        if (hdy0) o[hdy0] = v;
        if (hdy1) o[hdy1] = v;
      }
    };
#pragma unroll
    for (int j = 0; j < NP; ++j)
      if (j >= n) put(j, S::empty());
    if (n == 0) continue;

    const P* pC = stC + c;
    const P* pts[7] = {plD + c, pC - BW, pC - 1, pC, pC + 1, pC + BW, plU + c};
    // Value of a slot-map word's grain at stencil point s.  The five points of the
    // centre plane read the decoded plane where there is one.
    auto phi_at = [&](uint32_t wj, int s) -> float {
      const uint32_t cd = s == 6 ? wj >> 24 : map_code(wj, s);
      if (kDec && s >= 1 && s <= 5) return sm.dec[cd * BCELLS + c + ctr_off[s]];
      return S::phi(pts[s][cd * BCELLS]);
    };
    const bool aliased = alias != 0xFFFFFFFFu;
    auto alias_at = [&](int s) -> float {  // slot 0's value at point s, where it is an alias
      return S::phi(pts[s - 1][map_code(alias, s) * BCELLS]);
    };
    // phi + 1 at the centre for every slot (the repulsion sum's terms); the loops
    // over slots stop at n, so a warp runs only as many iterations as its
    // fullest cell
    float phc1[NP];
#pragma unroll
    for (int q = 0; q < NP; ++q) phc1[q] = 0.0f;
#pragma unroll
    for (int q = 0; q < NP; ++q) {
      if (q >= n) break;
      phc1[q] = __fadd_rn(phi_at(wcol[q * 32], 3), 1.0f);
    }
    if (aliased && map_code(alias, 3) != 0xFu) phc1[0] = __fadd_rn(alias_at(3), 1.0f);

    // rounding bits of this cell and step: keyed on the cell's reference-layout
    // index and the step number, so a simulation rounds the same alone or batched
    uint32_t cell_key = 0;
    if (S::kStochastic)
      cell_key = mix32((uint32_t)(gx + a.fnx * (gy + a.fny * k)) ^ mix32(a.sr_key));

    float Up = Up_plane;
    bool upd = true;
    if (!plane_T) {
      float T;
      upd = tinterp(a, gx, gy, k, &T);
      Up = __fdiv_rn(T, a.L_cp);
    }

    bool clive = false;
    bool changed = force_mark;  // the cell's id list differs from the one it came in with
    // New value of output slot j < n, slot-map word wj.
    auto update_slot = [&](int j, uint32_t wj) -> P {
      // the grain's id: at the centre if that holds it, else at another point (the
      // row of empty pairs gives -1)
      const uint32_t cC = map_code(wj, 3);
      int id = S::id(pC[cC * BCELLS]);
      // orientation of the grain (APTPhaseField.cu:259-273), used only where the
      // centre holds it: loads issued before the stencil values are gathered so
      // their latency overlaps; ids are >= 0 there (cupf_apt_set_slots rejects
      // other negative ids) and the clamp only keeps an absent or corrupted id
      // from reading outside the tables
      int tid2 = id;
      if (id > a.num_theta)  // id % num_theta + 1
        tid2 = id - (int)div_invariant((uint32_t)id, a.nt_magic, a.nt_sh1, a.nt_sh2) * a.num_theta + 1;
      const bool tab_ok = (unsigned)tid2 <= (unsigned)a.num_theta;
      const int ti = tab_ok ? tid2 : 0;
      float4 t_o = __ldg(a.orient + ti);  // {sint[ti], cost[ti], sint[ti+NG], cost[ti+NG]}
      float ph7[7];
#pragma unroll
      for (int s = 0; s < 7; ++s) ph7[s] = phi_at(wj, s);
      if (id == -1) {
#pragma unroll
        for (int s = 0; s < 7; ++s)
          if (s != 3) id = max(id, S::id(pts[s][(s == 6 ? wj >> 24 : map_code(wj, s)) * BCELLS]));
      }
      if (j == 0 && aliased) {
#pragma unroll
        for (int s = 1; s < 7; ++s)
          if (map_code(alias, s) != 0xFu) ph7[s] = alias_at(s);
      }
      float sina = 0.0f, cosa = 1.0f, sinb = 0.0f, cosb = 1.0f;
      if (ph7[3] > kLS) {  // (double)phC > LS
        // an aliased centre value belongs to another grain than slot 0's
        int to = ti;
        bool ok = tab_ok;
        if (j == 0 && aliased && cC == (uint32_t)NP) {
          to = id;
          if (id > a.num_theta)
            to = id - (int)div_invariant((uint32_t)id, a.nt_magic, a.nt_sh1, a.nt_sh2) * a.num_theta + 1;
          ok = (unsigned)to <= (unsigned)a.num_theta;
          t_o = __ldg(a.orient + (ok ? to : 0));
        }
        if (ok) {
          sina = t_o.x;
          cosa = t_o.y;
          sinb = t_o.z;
          cosb = t_o.w;
        }
      }
      // repulsion sum over the other slots (APTPhaseField.cu:328-335): the
      // reference accumulates r += 0.25 (phi+1)(phi+1) with the product fused,
      // r' = RN(0.25 q q + r).  Kept four times larger, R = 4 r, the same sum is
      // R' = RN(q q + R) = 4 RN(0.25 q q + r) exactly (scaling by a power of two
      // commutes with rounding; every term is far from the subnormal range), so
      // one fused multiply-add per term and one multiply at the end give the
      // reference's bits.
      static_assert(Contract::REP == 1, "the scaled sum restates the fused form only");
      float rsum = 0.0f;
#pragma unroll
      for (int q = 0; q < NP; ++q)  // past n the terms are +0
        if (q != j) rsum = __fmaf_rn(phc1[q], phc1[q], rsum);
      const float repul = __fmul_rn(0.25f, rsum);
      const float nv = slot_update(a, kc, ph7, sina, cosa, sinb, cosb, repul, Up);
      const bool drop = nv < kDrop;  // (double)nv < -0.9999
      const int oid = drop ? -1 : id;
      // The list stays as it was only if every kept grain sat in this same slot and
      // every dropped one was absent (a grain of any slot past n is one of the n).
      changed |= cC != (drop ? (uint32_t)NP : (uint32_t)j);
      // slot j's rounding bits: the cell's hashed key times a distinct odd
      // constant per slot (a bijection of a uniform 32-bit value, one multiply)
      if (S::kStochastic) return S::make_sr(nv, oid, cell_key * ((uint32_t)(2 * j + 1) * 0x9E3779B9u));
      return S::make(nv, oid);
    };
    // one loop body run to the cell's slot count (unrolled over NUM_PF it overruns the
    // instruction cache: 1.16 times the time per step, FP32, 128x128x256, NUM_PF = 8)
    if (upd) {
#pragma unroll 1
      for (int j = 0; j < n; ++j) {
        const P v = update_slot(j, wcol[j * 32]);
        clive |= !S::is_empty(v);
        put(j, v);
      }
    }
    if (!upd) clive = changed = true;  // the reference leaves the slots unwritten
    if (changed && a.map)
      mark_readers(a.redo_out, gx, gy, k, a.fnx, a.fny, a.fnz, a.xp, a.bcX, a.bcY, a.bcZ);
    if (clive) live |= 1u | (k == k_begin ? 2u : 0u) | (k == k_end - 1 ? 4u : 0u);
  }

  // record which of the item's output, its bottom plane and its top plane hold
  // only exact empty pairs (flag bits 0, 1, 2)
  const int busy = __syncthreads_or(live & 1u), busy_lo = __syncthreads_or(live & 2u),
            busy_hi = __syncthreads_or(live & 4u);
  if (tid == 0 && a.quiet_out)
    a.quiet_out[(zci * a.nty + tyi) * a.ntx + txi] =
        (uint8_t)((busy ? 0 : 1) | (busy_lo ? 0 : 2) | (busy_hi ? 0 : 4));
  if (a.overflows) {
    const uint32_t wa = __reduce_add_sync(0xffffffffu, n_ovf & 0xFFFFu);
    const uint32_t wd = __reduce_add_sync(0xffffffffu, n_ovf >> 16);
    if ((tid & 31) == 0 && (wa | wd)) {
      atomicAdd(a.overflows, (unsigned long long)wa);
      atomicAdd(a.overflows + 1, (unsigned long long)wd);
    }
  }
  if (tid == 0 && a.active_cells) {
    const int wx = min(TX, a.fnx - 1 - x0), wy = min(TY, a.fny - 1 - y0);
    atomicAdd(a.active_cells, (unsigned long long)(wx * wy * (k_end - k_begin)));
  }

  qbase = q0 + nplanes;
}

// True when the step may leave work item (txi, tyi, zci) alone: its cells in
// the output buffer already hold only exact empty pairs (id -1, phi -1), and its
// cells and the face-neighbour cells its 7-point stencil reads in the input
// buffer hold no id.  Those neighbours are the whole items across the x and y
// faces (or the items the boundary map sends a halo cell to), and across the z
// faces the top plane of the item below and the bottom plane of the item above
// (flag bits 2 and 1; a halo plane maps to an arbitrary plane, so there the
// whole item's bit 0).  Every cell of such an item would be written as the empty
// pair again.
template <int TY>
__device__ __forceinline__ bool item_quiet(const StepArgs& a, const uint8_t* quiet_in,
                                           const uint8_t* quiet_out, int txi, int tyi, int zci) {
  const int per = a.ntx * a.nty;
  const int it = zci * per + tyi * a.ntx + txi;
  if (!(quiet_out[it] & 1) || !(quiet_in[it] & 1)) return false;
  auto q = [&](int tx, int ty, int zc, int bit) {
    return (quiet_in[zc * per + ty * a.ntx + tx] & bit) != 0;
  };
  const int x0 = 1 + TX * txi, x1 = min(x0 + TX - 1, a.fnx - 2);
  const int y0 = 1 + TY * tyi, y1 = min(y0 + TY - 1, a.fny - 2);
  const int k0 = 1 + a.zc * zci, k1 = min(k0 + a.zc, a.fnz - 1);
  const int xl = bc_map(x0 - 1, a.fnx, a.bcX), xr = bc_map(x1 + 1, a.fnx, a.bcX);
  const int yl = bc_map(y0 - 1, a.fny, a.bcY), yr = bc_map(y1 + 1, a.fny, a.bcY);
  const bool below = k0 - 1 >= 1
                         ? q(txi, tyi, zci - 1, 4)
                         : q(txi, tyi, (bc_map(k0 - 1, a.fnz, a.bcZ) - 1) / a.zc, 1);
  const bool above = k1 <= a.fnz - 2 ? q(txi, tyi, zci + 1, 2)
                                     : q(txi, tyi, (bc_map(k1, a.fnz, a.bcZ) - 1) / a.zc, 1);
  return below && above && q((xl - 1) / TX, tyi, zci, 1) && q((xr - 1) / TX, tyi, zci, 1) &&
         q(txi, (yl - 1) / TY, zci, 1) && q(txi, (yr - 1) / TY, zci, 1);
}

// The work items of a persistent launch: CTA b starts with item b; further items
// come from the launch's atomic counter, which a launch with no more items than
// CTAs never touches.  Otherwise each CTA counts itself done once it has drawn past
// the end; the last one resets both words, so the next launch (or graph replay)
// starts from zero.
// Every item is taken only while the error word is clear: after a failed
// load the steps still queued compute nothing, in launches of either kind.
struct WorkItems {
  int* work;
  int nitems;
  int* s_item;
  const int* err;
  int ticket;  // the first item, then -1 (draw from the counter) or nitems
  __device__ WorkItems(int* work, int nitems, int* s_item, const int* err)
      : work(work), nitems(nitems), s_item(s_item), err(err), ticket(blockIdx.x) {}
  // The CTA's next item, -1 when none is left (every thread gets the same).
  __device__ __forceinline__ int next() {
    if (nitems <= (int)gridDim.x) {  // one item a CTA
      const int it = ticket < nitems ? ticket : -1;
      ticket = nitems;
      if (it < 0) return it;
      // one thread's reading decides for the CTA: the word may be set meanwhile
      return __syncthreads_or(threadIdx.x == 0 && *(volatile const int*)err != 0) ? -1 : it;
    }
    __syncthreads();  // every thread has read the previous index
    if (threadIdx.x == 0) {
      int it = ticket >= 0 ? ticket : (int)gridDim.x + atomicAdd(work, 1);
      ticket = -1;
      // a CTA that gave up on a load set the error word: take no further items
      // (read with the ticket, once per item, not per plane)
      if (*(volatile const int*)err != 0) it = nitems;
      if (it >= nitems) {
        it = -1;
        __threadfence();
        if (atomicAdd(work + 1, 1) == (int)gridDim.x - 1) {
          atomicExch(work, 0);
          atomicExch(work + 1, 0);
        }
      }
      *s_item = it;
    }
    __syncthreads();
    return *s_item;
  }
};

// One launch = one step of one simulation.  Persistent CTAs pull work items
// (column tile x z chunk) from an atomic counter, z-chunk-major so the chunks
// nearest the bottom (the solid, where cells carry the most grain ids in a
// directional-solidification run) start first and the light liquid chunks fill
// in behind them.
// Resident CTAs per SM the step is compiled for.  32x8 tiles: three where three
// CTAs' shared memory fits (16-bit pairs, or FP32 up to NUM_PF = 5), else two.
// 32x4 tiles: twice that (the same registers per thread), or as many as their
// shared memory fits on one SM (228 KB) when fewer.
template <int NP, class S, int TY>
constexpr int step_min_blocks() {
  constexpr int tall = StepSmem<NP, S, 8>::kBytes <= 74 * 1024 ? 3 : 2;
  constexpr int by_smem = (228 * 1024) / StepSmem<NP, S, TY>::kBytes;
  return TY == 8 ? tall : (2 * tall < by_smem ? 2 * tall : by_smem);
}

template <int NP, class S, int TY>
__global__ void __launch_bounds__(tile_threads<TY>(), step_min_blocks<NP, S, TY>())
    apt_step_kernel(const __grid_constant__ CUtensorMap tmap, const StepArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  CtaSmem<NP, S, TY> sm(smem);
  sm.init();
  const int per_chunk = a.ntx * a.nty;
  const int nitems = per_chunk * a.nzc;
  int qbase = 0;
  // launched before the previous step has ended (launch_dependent): nothing above reads
  // what that writes
  cudaGridDependencySynchronize();
  cudaTriggerProgrammaticLaunchCompletion();
  WorkItems items(a.work, nitems, sm.s_item, a.err);
  for (;;) {
    const int it = items.next();
    if (it < 0) break;
    const int zci = it / per_chunk;
    const int r = it - zci * per_chunk;
    if (a.quiet_out && item_quiet<TY>(a, a.quiet_in, a.quiet_out, r % a.ntx, r / a.ntx, zci)) continue;
    step_item<NP, S, TY>(&tmap, a, r % a.ntx, r / a.ntx, zci, sm, qbase);
  }
  sm.drain();
}

}  // namespace cupf
