// apt_aux.cuh — the non-step kernels of the B200 APT solver.
//
// All operate on the pair-plane buffers described in apt_common.cuh.  None of
// them is on the per-step hot path; they run at init, at QoI / moving-domain
// events and on read-back.
#pragma once

#include "apt_storage.cuh"

namespace cupf {

struct Grid {
  int fnx, fny, fnz, xp, np;
  long long ss;  // slot stride in pairs
  __host__ __device__ long long plane() const { return (long long)xp * fny; }
  __host__ __device__ long long at(int i, int j, int k) const {
    return (long long)k * plane() + (long long)j * xp + i;
  }
  __host__ __device__ long long length() const { return (long long)fnx * fny * fnz; }
};

// Materialise the halo: every cell with a coordinate on the boundary takes the
// record of its mapped interior source (each coordinate mapped independently,
// = sequential z, y, x face fills of APTsetBC3D, APTPhaseField.cu:93-174).
// Cells are enumerated face by face without repetition.
__host__ __device__ __forceinline__ long long halo_cells(const Grid& g) {
  return 2ll * g.fnx * g.fny + 2ll * g.fnx * (g.fnz - 2) + 2ll * (g.fny - 2) * (g.fnz - 2);
}

// Halo cell idx (0 .. halo_cells-1): the two z planes, then the two y faces of
// the interior planes, then the two x faces of the interior rows.
__device__ __forceinline__ void halo_cell(long long idx, const Grid& g, int& i, int& j, int& k) {
  const long long nz2 = 2ll * g.fnx * g.fny;
  const long long ny2 = 2ll * g.fnx * (g.fnz - 2);
  const long long nx2 = 2ll * (g.fny - 2) * (g.fnz - 2);
  long long r = idx;
  if (r < nz2) {
    k = (r < nz2 / 2) ? 0 : g.fnz - 1;
    r %= (long long)g.fnx * g.fny;
    j = (int)(r / g.fnx);
    i = (int)(r % g.fnx);
  } else if ((r -= nz2) < ny2) {
    j = (r < ny2 / 2) ? 0 : g.fny - 1;
    r %= (long long)g.fnx * (g.fnz - 2);
    k = 1 + (int)(r / g.fnx);
    i = (int)(r % g.fnx);
  } else {
    r -= ny2;
    i = (r < nx2 / 2) ? 0 : g.fnx - 1;
    r %= (long long)(g.fny - 2) * (g.fnz - 2);
    k = 1 + (int)(r / (g.fny - 2));
    j = 1 + (int)(r % (g.fny - 2));
  }
}

template <class S>
__global__ void fill_halo_kernel(typename S::T* buf, Grid g, int bcX, int bcY, int bcZ) {
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < halo_cells(g);
       idx += (long long)gridDim.x * blockDim.x) {
    int i, j, k;
    halo_cell(idx, g, i, j, k);
    const long long d = g.at(i, j, k);
    const long long s = g.at(bc_map(i, g.fnx, bcX), bc_map(j, g.fny, bcY), bc_map(k, g.fnz, bcZ));
    for (int p = 0; p < g.np; ++p) buf[p * g.ss + d] = buf[p * g.ss + s];
  }
}

// set_minus1 + APTini_PF on both buffers (PhaseField.cu:51-57, APTPhaseField.cu:78-89):
// every slot (-1, -1), then slot 0 = (phi, alpha) where phi > LS.  phi/alpha in
// reference layout (index i + j*fnx + k*fnx*fny).
template <class S>
__global__ void init_kernel(typename S::T* A, typename S::T* B, const float* __restrict__ phi,
                            const int* __restrict__ alpha, Grid g) {
  const long long L = g.length();
  for (long long C = blockIdx.x * (long long)blockDim.x + threadIdx.x; C < L;
       C += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(C % g.fnx);
    const int j = (int)((C / g.fnx) % g.fny);
    const int k = (int)(C / ((long long)g.fnx * g.fny));
    const long long d = g.at(i, j, k);
    const float v = phi[C];
    typename S::T s0 = S::empty();
    if ((double)v > LS) s0 = S::make(v, alpha[C]);
    A[d] = s0;
    B[d] = s0;
    for (int p = 1; p < g.np; ++p) {
      A[p * g.ss + d] = S::empty();
      B[p * g.ss + d] = S::empty();
    }
  }
}

// APTcollect_PF (APTPhaseField.cu:55-75): argmax over slots, first max wins; the
// outputs change only where the max is above LS.
template <class S>
__global__ void collect_kernel(const typename S::T* __restrict__ buf, float* phi, int* alpha,
                               Grid g) {
  const long long L = g.length();
  for (long long C = blockIdx.x * (long long)blockDim.x + threadIdx.x; C < L;
       C += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(C % g.fnx);
    const int j = (int)((C / g.fnx) % g.fny);
    const int k = (int)(C / ((long long)g.fnx * g.fny));
    const long long d = g.at(i, j, k);
    typename S::T best = buf[d];
    float bv = S::phi(best);
    for (int p = 1; p < g.np; ++p) {
      const typename S::T v = buf[p * g.ss + d];
      const float f = S::phi(v);
      if (f > bv) {
        best = v;
        bv = f;
      }
    }
    if ((double)bv > LS) {
      phi[C] = bv;
      alpha[C] = S::id(best);
    }
  }
}

// pair planes -> reference layout (ph[slot*length + C], ids[slot*length + C])
template <class S>
__global__ void export_kernel(const typename S::T* __restrict__ buf, float* ph, int* ids, Grid g) {
  const long long L = g.length();
  for (long long C = blockIdx.x * (long long)blockDim.x + threadIdx.x; C < L * g.np;
       C += (long long)gridDim.x * blockDim.x) {
    const int p = (int)(C / L);
    const long long c = C - p * L;
    const int i = (int)(c % g.fnx);
    const int j = (int)((c / g.fnx) % g.fny);
    const int k = (int)(c / ((long long)g.fnx * g.fny));
    const typename S::T v = buf[p * g.ss + g.at(i, j, k)];
    ph[C] = S::phi(v);
    ids[C] = S::id(v);
  }
}

template <class S>
__global__ void import_kernel(typename S::T* buf, const float* __restrict__ ph,
                              const int* __restrict__ ids, Grid g) {
  const long long L = g.length();
  for (long long C = blockIdx.x * (long long)blockDim.x + threadIdx.x; C < L * g.np;
       C += (long long)gridDim.x * blockDim.x) {
    const int p = (int)(C / L);
    const long long c = C - p * L;
    const int i = (int)(c % g.fnx);
    const int j = (int)((c / g.fnx) % g.fny);
    const int k = (int)(c / ((long long)g.fnx * g.fny));
    buf[p * g.ss + g.at(i, j, k)] = S::make(ph[C], ids[C]);
  }
}

// Per-layer sum of phi over every slot and cell (halo included), one block per
// layer, double accumulation in a fixed order (deterministic; the reference
// accumulates with float atomics, PhaseField.cu:366-378).  A warp takes rows, its
// lanes the cells of a row, with the slots' loads in flight together: 128x128x384,
// NUM_PF = 8 FP32 (403 MB) 81 us on a B200, 312 with 256 threads and one load each.
constexpr int kLayerThreads = 1024;
template <class S>
__global__ void __launch_bounds__(kLayerThreads)
    layer_sum_kernel(const typename S::T* __restrict__ buf, double* sums, Grid g) {
  const int k = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double acc = 0.0;
  for (int j = warp; j < g.fny; j += kLayerThreads / 32) {
    const typename S::T* row = buf + g.at(0, j, k);
    for (int i = lane; i < g.fnx; i += 32) {
      int p = 0;
      for (; p + 4 <= g.np; p += 4) {
        typename S::T v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = row[(p + u) * g.ss + i];
#pragma unroll
        for (int u = 0; u < 4; ++u) acc += (double)S::phi(v[u]);
      }
      for (; p < g.np; ++p) acc += (double)S::phi(row[p * g.ss + i]);
    }
  }
  __shared__ double red[kLayerThreads];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int s = kLayerThreads / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) sums[k] = red[0];
}

// One layer of a domain move in one pass over the slots: the argmax of every cell
// (collect_kernel), and the interior shifted down one plane into dst
// (APTmove_frame, APTPhaseField.cu:357-410: dst[k] = src[k+1] for k < fnz-2, the top
// interior layer (-1, -1)); with `halo` dst also takes src's halo cells unchanged.
// One thread a cell: a block takes 32 x 8 cells of one plane (move_layer_blocks).
// Bound by bytes: 128x128x384, NUM_PF = 8 FP32 142 us on a B200 (about 860 MB, 6 TB/s);
// as three kernels with 64-bit index divisions 380.
inline unsigned move_layer_blocks(const Grid& g) {
  return (unsigned)((g.fnx + 31) / 32) * (unsigned)((g.fny + 7) / 8) * (unsigned)g.fnz;
}
template <class S>
__global__ void move_layer_kernel(const typename S::T* __restrict__ src, typename S::T* dst,
                                  float* phi, int* alpha, Grid g, int halo) {
  const int nbx = (g.fnx + 31) / 32, nby = (g.fny + 7) / 8, t = (int)(blockIdx.x % (nbx * nby));
  const int i = t % nbx * 32 + (threadIdx.x & 31), j = t / nbx * 8 + (threadIdx.x >> 5);
  const int k = (int)(blockIdx.x / (nbx * nby));
  if (i >= g.fnx || j >= g.fny) return;
  const bool inner = i > 0 && i < g.fnx - 1 && j > 0 && j < g.fny - 1 && k > 0 && k < g.fnz - 1;
  const long long d = g.at(i, j, k);
  const long long to = inner ? (k > 1 ? d - g.plane() : -1) : (halo ? d : -1);
  const bool top = inner && k == g.fnz - 2;
  typename S::T best{};
  float bv = 0.0f;
  for (int p = 0; p < g.np; ++p) {
    const typename S::T v = src[p * g.ss + d];
    const float f = S::phi(v);
    if (p == 0 || f > bv) {
      best = v;
      bv = f;
    }
    if (to >= 0) dst[p * g.ss + to] = v;
    if (top) dst[p * g.ss + d] = S::empty();
  }
  if ((double)bv > LS) {
    const long long C = ((long long)k * g.fny + j) * g.fnx + i;
    phi[C] = bv;
    alpha[C] = S::id(best);
  }
}

// Quiet-item flags after the domain moved down by m planes (new plane k holds old
// plane k + m, planes past the top are empty): an item is quiet when every item
// that held its new planes was (bit 0; bits 1 and 2, its bottom and top plane,
// are set only with bit 0).  src: flags before the move, dst: after.
static __global__ void quiet_shift_kernel(const uint8_t* __restrict__ src, uint8_t* dst, int per_chunk,
                                          int nzc, int zc, int fnz, int m) {
  const long long n = (long long)per_chunk * nzc;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i / per_chunk), t = (int)(i - (long long)c * per_chunk);
    const int k0 = 1 + zc * c, k1 = min(k0 + zc, fnz - 1);  // planes [k0, k1)
    const int lo = k0 + m, hi = min(k1 - 1 + m, fnz - 2);   // old planes they hold
    uint8_t q = 1;
    for (int cc = (lo - 1) / zc; lo <= hi && cc <= (hi - 1) / zc; ++cc)
      q &= src[(long long)cc * per_chunk + t] & 1;
    dst[i] = q ? 7 : 0;  // plane bits only from a wholly empty item
  }
}

template <class S>
__global__ void copy_interior_kernel(const typename S::T* __restrict__ src, typename S::T* dst,
                                     Grid g) {
  const int ni = g.fnx - 2, nj = g.fny - 2, nk = g.fnz - 2;
  const long long total = (long long)ni * nj * nk * g.np;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    long long r = idx;
    const int i = 1 + (int)(r % ni);
    r /= ni;
    const int j = 1 + (int)(r % nj);
    r /= nj;
    const int k = 1 + (int)(r % nk);
    const int p = (int)(r / nk);
    const long long d = p * g.ss + g.at(i, j, k);
    dst[d] = src[d];
  }
}

// Archive the bottom interior layer of the argmax map and count it into the
// lost area (APTPhaseField.cu:383-388): alpha_full[move*plane + C] = alpha[C] for
// C in layer 1 (all i, j), loss_area[alpha-1] += 1 for alpha in 1..num_theta.
static __global__ void archive_kernel(const int* __restrict__ alpha, int* alpha_full, int* loss_area,
                               int fnx, int fny, int move_count, int num_theta) {
  const long long plane = (long long)fnx * fny;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < plane;
       c += (long long)gridDim.x * blockDim.x) {
    const int a = alpha[plane + c];
    alpha_full[move_count * plane + plane + c] = a;
    if (a >= 1 && a <= num_theta) atomicAdd(loss_area + a - 1, 1);
  }
}

// Voxel count per grain id over the interior of the argmax map, plus the first
// (k, j, i)-order index where each id occurs (for the reference's first-seen
// ordering, QOI.cpp:198-231).  counts[0] = interior cells with no grain.
// A warp takes rows.  Neighbouring cells mostly share a grain, so the lanes of a
// warp holding the same id add their count in one atomic from the lowest of them,
// which also holds their smallest index; the cells with no grain (most of a window
// that is still liquid) are counted in registers, one atomic a warp at its end:
// 256x256x512 146 us on a B200, about 620 with an atomic for them in every warp row.
static __global__ void volume_kernel(const int* __restrict__ alpha, int fnx, int fny, int fnz, int ng,
                              unsigned long long* counts, long long* first) {
  const int lane = threadIdx.x & 31, nj = fny - 2;
  const int nwarps = gridDim.x * (blockDim.x >> 5);
  const long long rows = (long long)nj * (fnz - 2);
  unsigned long long none = 0;
  for (long long r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < rows; r += nwarps) {
    const int k = 1 + (int)(r / nj), j = 1 + (int)(r - (long long)(k - 1) * nj);
    const long long row = ((long long)k * fny + j) * fnx;
    for (int i0 = 1; i0 < fnx - 1; i0 += 32) {
      const int i = i0 + lane;
      const bool on = i < fnx - 1;
      const int a = on ? alpha[row + i] : 0;
      const int key = (a >= 1 && a <= ng) ? a : 0;
      none += on && key == 0;
      const unsigned grains = __ballot_sync(0xffffffffu, key != 0);
      if (key) {
        const unsigned peers = __match_any_sync(grains, key);
        if (lane == __ffs(peers) - 1) {
          atomicAdd(counts + key, (unsigned long long)__popc(peers));
          atomicMin(first + key, row + i);
        }
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) none += __shfl_down_sync(0xffffffffu, none, o);
  if (lane == 0 && none) atomicAdd(counts, none);
}

// Candidate cells of the 3D junction search (QOI3D::searchJunctionsOnImage,
// QOI.cpp:233-311): a solid cell (alpha != 0) whose 19-point neighbourhood
// (offsets with di^2 + dj^2 + dk^2 <= 2, itself included) holds no liquid cell,
// exactly four distinct grain ids and no id more than ten times.  The indices
// (reference layout) are appended in arbitrary order; `count` receives how many
// cells qualify even past `cap`.  `distinct[idx]` (interior cells in (k, j, i)
// order) receives the number of distinct values, liquid included, that the
// reference's scan inserts into its hash map at that cell (0 where alpha == 0):
// the host needs their running maximum to reproduce the map's bucket count,
// which fixes the order of the grain ids in each record.
static __global__ void junction_candidates_kernel(const int* __restrict__ alpha, int fnx, int fny,
                                                  int fnz, long long* out, long long cap,
                                                  unsigned long long* count,
                                                  unsigned char* distinct) {
  const long long ni = fnx - 2, nj = fny - 2, nk = fnz - 2;
  const long long total = ni * nj * nk, plane = (long long)fnx * fny;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long i = 1 + idx % ni, j = 1 + (idx / ni) % nj, k = 1 + idx / (ni * nj);
    const long long C = k * plane + j * fnx + i;
    if (alpha[C] == 0) {
      distinct[idx] = 0;
      continue;
    }
    int vals[19], cnt[19];
    int nd = 0, maxc = 0;
    bool zero = false;
    for (int dk = -1; dk <= 1; ++dk)
      for (int dj = -1; dj <= 1; ++dj)
        for (int di = -1; di <= 1; ++di) {
          if (di * di + dj * dj + dk * dk > 2) continue;
          const int v = alpha[C + dk * plane + dj * fnx + di];
          zero |= (v == 0);
          int f = -1;
          for (int q = 0; q < nd; ++q)
            if (vals[q] == v) f = q;
          if (f < 0) {
            vals[nd] = v;
            cnt[nd] = 0;
            f = nd++;
          }
          maxc = max(maxc, ++cnt[f]);
        }
    distinct[idx] = (unsigned char)nd;
    if (zero || nd != 4 || maxc > 10) continue;
    const unsigned long long slot = atomicAdd(count, 1ull);
    if ((long long)slot < cap) out[slot] = C;
  }
}

// Candidate cells of the line-configuration junction search
// (QOILine::searchJunctionsOnImage, QOI.cpp:103-160) over `nl` stacked x-y
// layers of an argmax map (the layers at the sampled tip heights): interior
// cells whose 3x3 in-plane neighbourhood holds at least three distinct values,
// none more than five times.  out receives the cells' indices in the stacked
// layers (layer * fnx * fny + j * fnx + i) in no particular order, up to cap;
// count receives their number.
static __global__ void line_junction_kernel(const int* __restrict__ layers, int nl, int fnx,
                                            int fny, long long* out, long long cap,
                                            unsigned long long* count) {
  const long long ni = fnx - 2, nj = fny - 2;
  const long long total = ni * nj * nl, plane = (long long)fnx * fny;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long i = 1 + idx % ni, j = 1 + (idx / ni) % nj, l = idx / (ni * nj);
    const long long C = l * plane + j * fnx + i;
    int v[9];
#pragma unroll
    for (int dj = -1; dj <= 1; ++dj)
#pragma unroll
      for (int di = -1; di <= 1; ++di) v[(dj + 1) * 3 + di + 1] = __ldg(layers + C + dj * fnx + di);
    int nd = 0, maxc = 0;
#pragma unroll
    for (int a = 0; a < 9; ++a) {
      bool first = true;
      int c = 0;
#pragma unroll
      for (int b = 0; b < 9; ++b) {
        c += (v[b] == v[a]);
        if (b < a && v[b] == v[a]) first = false;
      }
      nd += first;
      maxc = max(maxc, c);
    }
    if (nd < 3 || maxc > 5) continue;
    const unsigned long long slot = atomicAdd(count, 1ull);
    if ((long long)slot < cap) out[slot] = C;
  }
}

// FP64 interface QoIs over the interior, from m = max-over-slots phi of each cell:
//   part[2*b]   = sum (1 + m) / 2              (solid volume, cell units)
//   part[2*b+1] = sum |grad m| / 2             (interface area, cell units; a
//                 diffuse interface integrates |grad phi| to 2 across its width)
// with central differences of m on the 6 neighbours (halo cells filled first).
// One partial pair per block; the host adds the partials in block order.
// A block takes 32 x 8 cell columns over chunks of planes and marches up: every
// plane's m, with a one-cell rim, is formed once in shared memory (a cell's slots
// are read 1.4 times in all instead of seven times), three planes at a time.  Chunks
// of 32 planes, halved down to 2 while the grid has fewer than the launch has blocks.
// Bound by the latency of a plane's loads between its two barriers: 256x256x512, NUM_PF =
// 8 FP32 934 us on a B200, 1657 with seven reads a cell.
template <class S>
__global__ void __launch_bounds__(256)
    qoi_sums_kernel(const typename S::T* __restrict__ buf, Grid g, double* part) {
  constexpr int W = 34, H = 10;
  __shared__ float m[3][W * H];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int ntx = (g.fnx - 2 + 31) / 32, nty = (g.fny - 2 + 7) / 8;
  int np = 32;
  while (np > 2 && (long long)ntx * nty * ((g.fnz - 2 + np - 1) / np) < gridDim.x) np /= 2;
  const int nzc = (g.fnz - 2 + np - 1) / np;
  double vol = 0.0, area = 0.0;
  for (int it = blockIdx.x; it < ntx * nty * nzc; it += gridDim.x) {
    const int x0 = 32 * (it % ntx), y0 = 8 * (it / ntx % nty);  // the rim's first cell
    const int k0 = 1 + np * (it / (ntx * nty)), k1 = min(k0 + np, g.fnz - 1);
    auto plane = [&](int k) {
      for (int c = threadIdx.x; c < W * H; c += 256) {
        const int i = x0 + c % W, j = y0 + c / W;
        if (i >= g.fnx || j >= g.fny) continue;
        const typename S::T* q = buf + g.at(i, j, k);
        float v = S::phi(q[0]);
        for (int p = 1; p < g.np; ++p) v = fmaxf(v, S::phi(q[p * g.ss]));
        m[k % 3][c] = v;
      }
    };
    __syncthreads();  // the previous item's planes have been read
    plane(k0 - 1);
    plane(k0);
    const int i = x0 + 1 + tx, j = y0 + 1 + ty, c = (ty + 1) * W + tx + 1;
    const bool on = i < g.fnx - 1 && j < g.fny - 1;
    for (int k = k0; k < k1; ++k) {
      plane(k + 1);
      __syncthreads();
      if (on) {
        const float* mc = m[k % 3] + c;
        vol += 0.5 * (1.0 + (double)mc[0]);
        const double gx = 0.5 * ((double)mc[1] - mc[-1]);
        const double gy = 0.5 * ((double)mc[W] - mc[-W]);
        const double gz = 0.5 * ((double)m[(k + 1) % 3][c] - m[(k + 2) % 3][c]);
        area += 0.5 * sqrt(gx * gx + gy * gy + gz * gz);
      }
      __syncthreads();  // plane k - 1 makes room for k + 2
    }
  }
  __shared__ double rv[256], ra[256];
  rv[threadIdx.x] = vol;
  ra[threadIdx.x] = area;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if ((int)threadIdx.x < s) {
      rv[threadIdx.x] += rv[threadIdx.x + s];
      ra[threadIdx.x] += ra[threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = rv[0];
    part[2 * blockIdx.x + 1] = ra[0];
  }
}

}  // namespace cupf
