// Gaussian-gridding spread (NUFFT type-1 spreading) of many channels.
//
// Pipeline (all on one stream):
//   1. bin_count   : knot mapping per point, home cell -> tile id, tile
//                    histogram; per-channel sum |v| (sets the fixed-point
//                    scale of the FP32 path).
//   2. tile_scan   : exclusive scans of the histogram and of the number of
//                    work items per tile (a tile is split into chunks of at
//                    most FLPR_TUNE_SPREAD_ITEM_POINTS points).
//   3. bin_scatter : one contiguous record per point, in tile order.
//   4. accumulate  : every work item is spread into a copy of its tile plus a
//                    halo of msp cells, in registers (2-D and 3-D) or in
//                    shared memory (1-D, wide stencils, tiny grids), which
//                    is then added to the global accumulator with one atomic
//                    per non-zero cell.
//   5. finalize    : accumulator -> real grid (float or double) times 1/n.
//
// FLPR_PREC_F32 accumulates 64-bit fixed point: integer addition is
// associative, so the result does not depend on the order of the atomics
// and the grid is deterministic.  FLPR_PREC_F64 accumulates float64.
#include "common.cuh"

namespace flpr {

// points per work item: tuning(FLPR_TUNE_SPREAD_ITEM_POINTS), carried in SpreadGeom
constexpr int kSpreadThreads = 256;
constexpr int kMaxTaps1 = 25;  // 2*msp+1 for msp <= 12 (msp = 0: binning with weight 1)

struct SpreadGeom {
  int d;
  int L[3];
  int T[3];        // tile extent per axis
  int ntile[3];    // tiles per axis
  int W[3];        // tile + halo extent per axis
  int msp;
  int ntaps1;      // 2*msp+1
  int64_t cells;   // prod(L)
  int tile_cells;  // prod(W)
  int ntiles;
  int item_points;  // points per work item (one CTA)
  double four_tau[3];
  KnotAxis ax[3];
};

struct ChanPtrs {
  const double* col[FLPR_MAX_CHANNELS];
};

// Home cell and tile of a point; also its unwrapped knot index m.  ax: the
// knot maps of the axes (the geometry's, or a device-computed copy).
__device__ __forceinline__ int point_tile(const SpreadGeom& g, const KnotAxis* ax,
                                          const double* __restrict__ x, int64_t i, int* m_out,
                                          double* k_out) {
  int tile = 0;
  for (int a = 0; a < g.d; ++a) {
    double k = knot_of(x[i * g.d + a], ax[a]);
    int m = (int)rint(ddiv(k, ax[a].hx));
    int home = m % g.L[a];
    if (home < 0) home += g.L[a];
    tile = tile * g.ntile[a] + home / g.T[a];
    if (m_out) m_out[a] = m;
    if (k_out) k_out[a] = k;
  }
  return tile;
}

// Knot maps of the axes into shared memory: from d_kmap (d x 9, the layout
// of the host geometry's rows) when given, else from the geometry.
__device__ __forceinline__ void load_axes(const SpreadGeom& g, const double* __restrict__ d_kmap,
                                          KnotAxis* s_ax) {
  if (threadIdx.x < g.d) {
    const int a = threadIdx.x;
    if (d_kmap) {
      const double* k = d_kmap + 9 * a;
      s_ax[a] = KnotAxis{k[0], k[1], k[2], k[3], k[4], k[5], k[6], k[7], k[8]};
    } else {
      s_ax[a] = g.ax[a];
    }
  }
}

// Knot maps (d x 9: mean, std, centre, centred minimum, scale, ks, r0, shift,
// hx) from the point statistics (4 x d: minimum, maximum, mean, M2), with
// the operations, in the order, of the host geometry: z-score with ddof 1
// (model.py:58-68), mid-range centring, the knot-range mapping
// (convolution.py:190-208) and the centring shift (nufftn_type1.py:164-166).
// One thread per axis.  nm1 = n - 1 (negative for one point: std NaN).
struct KnotConsts {
  double ks[3], r0[3], hx[3];
};

__global__ void knot_map_kernel(int d, double nm1, const double* __restrict__ st, KnotConsts kc,
                                double* __restrict__ kmap) {
  const int a = threadIdx.x;
  if (a >= d) return;
  const double xmin = st[a], xmax = st[d + a], mean = st[2 * d + a], m2 = st[3 * d + a];
  double sd = nm1 > 0.0 ? __dsqrt_rn(ddiv(m2, nm1)) : NAN;
  if (sd == 0.0) sd = 1.0;
  const double xs_min = ddiv(dsub(xmin, mean), sd);
  const double xs_max = ddiv(dsub(xmax, mean), sd);
  const double center = ddiv(dadd(xs_max, xs_min), 2.0);
  const double lo = dsub(xs_min, center);
  const double hi = dsub(xs_max, center);
  double scale = dsub(hi, lo);
  if (scale == 0.0) scale = 1.0;
  const double ks = kc.ks[a], r0 = kc.r0[a];
  double c[2];
  for (int e = 0; e < 2; ++e) {
    double xn = dadd(dmul(ddiv(dsub(e == 0 ? lo : hi, lo), scale), ks), r0);
    xn = dadd(xn, 0.5);
    xn = np_mod(xn, 1.0);
    c[e] = dsub(xn, 0.5);
  }
  const double kmin = dsub(dmul(dadd(c[0], c[1]), 0.5), 0.5);
  const double shift = dsub(-0.5, kmin);
  double* o = kmap + 9 * a;
  o[0] = mean;
  o[1] = sd;
  o[2] = center;
  o[3] = lo;
  o[4] = scale;
  o[5] = ks;
  o[6] = r0;
  o[7] = shift;
  o[8] = kc.hx[a];
}

// Points per tile and, in blocks of their own, each channel's sum of |v|:
// blocks [0, nbh) count, then nbc blocks per channel follow.  A grid of few
// tiles counts in shared memory first, since thousands of points would wait
// for the same few global counters; and a channel per block leaves a thread's
// loads free of one another (one pass over points and then channels in turn:
// 62 us for 1e6 points and 11 channels on 512^2, 29 us for 1e5 on a 1-D grid
// of 1024; now 40 and 4.4 us).
constexpr int kFewTiles = 512;

__global__ void __launch_bounds__(256)
bin_count_kernel(SpreadGeom g, int64_t n, const double* __restrict__ x,
                 const double* __restrict__ d_kmap, int* __restrict__ counts, int nchan,
                 int ones_channel, ChanPtrs cp, double* __restrict__ absum, int nbh, int nbc) {
  if (blockIdx.x >= nbh) {
    const int b = blockIdx.x - nbh, c = b / nbc, part = b - c * nbc;
    const double* __restrict__ col = cp.col[c];
    double v = 0.0;
#pragma unroll 4
    for (int64_t i = part * 256LL + threadIdx.x; i < n; i += nbc * 256LL) v += fabs(col[i]);
    __shared__ double sh[8];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int k = 1; k < 8; ++k) v += sh[k];
      atomicAdd(&absum[ones_channel + c], v);
    }
    return;
  }
  __shared__ KnotAxis s_ax[3];
  __shared__ int s_cnt[kFewTiles];
  const bool few = g.ntiles <= kFewTiles;
  load_axes(g, d_kmap, s_ax);
  if (few)
    for (int t = threadIdx.x; t < g.ntiles; t += 256) s_cnt[t] = 0;
  __syncthreads();
  int* cnt = few ? s_cnt : counts;
  for (int64_t i = blockIdx.x * 256LL + threadIdx.x; i < n; i += nbh * 256LL)
    atomicAdd(&cnt[point_tile(g, s_ax, x, i, nullptr, nullptr)], 1);
  if (few) {
    __syncthreads();
    for (int t = threadIdx.x; t < g.ntiles; t += 256)
      if (s_cnt[t]) atomicAdd(&counts[t], s_cnt[t]);
  }
  if (ones_channel && blockIdx.x == 0 && threadIdx.x == 0) absum[0] = (double)n;
}

// Exclusive scans over the tile histogram (points and work items per tile) in
// two launches: blocks of kScanTiles tiles scan their own counts (four tiles
// per thread, warp shuffles, the warp totals scanned by warp 0) and leave
// their totals, then every block adds the totals before it.  One block alone
// took 1.4 us per 1024 tiles, 22 us for a 2-D grid and 350 us for a 3-D grid
// of 256^3 in its one-cell slabs.  A histogram of one block needs one launch.
constexpr int kScanTiles = 4096;

__global__ void __launch_bounds__(1024)
tile_scan_kernel(int ntiles, int item_points, const int* __restrict__ counts,
                 int* __restrict__ offsets, int* __restrict__ items, int* __restrict__ cursor,
                 int2* __restrict__ totals) {
  __shared__ int wa[32], wb[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t0 = blockIdx.x * kScanTiles + 4 * threadIdx.x;
  int a[4], b[4], sa = 0, sb = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int c = t0 + k < ntiles ? counts[t0 + k] : 0;
    a[k] = sa;
    b[k] = sb;
    sa += c;
    sb += (c + item_points - 1) / item_points;
  }
  int ia = sa, ib = sb;  // inclusive warp scans
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int va = __shfl_up_sync(0xffffffffu, ia, o);
    const int vb = __shfl_up_sync(0xffffffffu, ib, o);
    if (lane >= o) {
      ia += va;
      ib += vb;
    }
  }
  if (lane == 31) {
    wa[warp] = ia;
    wb[warp] = ib;
  }
  __syncthreads();
  if (warp == 0) {
    int xa = wa[lane], xb = wb[lane];  // 32 warps
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int va = __shfl_up_sync(0xffffffffu, xa, o);
      const int vb = __shfl_up_sync(0xffffffffu, xb, o);
      if (lane >= o) {
        xa += va;
        xb += vb;
      }
    }
    wa[lane] = xa;  // inclusive warp totals
    wb[lane] = xb;
  }
  __syncthreads();
  const int pa = (warp ? wa[warp - 1] : 0) + ia - sa, pb = (warp ? wb[warp - 1] : 0) + ib - sb;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (t0 + k < ntiles) {
      offsets[t0 + k] = pa + a[k];
      items[t0 + k] = pb + b[k];
      cursor[t0 + k] = 0;
    }
  if (threadIdx.x == 0) {
    totals[blockIdx.x] = make_int2(wa[31], wb[31]);
    if (gridDim.x == 1) {
      offsets[ntiles] = wa[31];
      items[ntiles] = wb[31];
    }
  }
}

__global__ void __launch_bounds__(1024)
tile_scan_add_kernel(int ntiles, const int2* __restrict__ totals, int* __restrict__ offsets,
                     int* __restrict__ items) {
  __shared__ int s_a, s_b;
  if (threadIdx.x == 0) s_a = s_b = 0;
  __syncthreads();
  int sa = 0, sb = 0;
  for (int k = threadIdx.x; k < (int)blockIdx.x; k += blockDim.x) {
    sa += totals[k].x;
    sb += totals[k].y;
  }
  for (int o = 16; o > 0; o >>= 1) {
    sa += __shfl_xor_sync(0xffffffffu, sa, o);
    sb += __shfl_xor_sync(0xffffffffu, sb, o);
  }
  if ((threadIdx.x & 31) == 0 && (sa | sb)) {
    atomicAdd(&s_a, sa);
    atomicAdd(&s_b, sb);
  }
  __syncthreads();
  const int pa = s_a, pb = s_b;
  for (int k = threadIdx.x; k < kScanTiles; k += blockDim.x) {
    const int t = blockIdx.x * kScanTiles + k;
    if (t < ntiles) {
      offsets[t] += pa;
      items[t] += pb;
    }
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    offsets[ntiles] = pa + totals[blockIdx.x].x;
    items[ntiles] = pb + totals[blockIdx.x].y;
  }
}

// Sorted records, one per point in tile order:
//   rec_base[pos]  local base cell of the point inside its tile, packed 10
//                  bits per axis (T <= 1024); rec_idx[pos] its index;
//   rec[pos * stride + ..]  the knot offsets k_a - hx_a m_a of the d axes,
//                  then the values of all channels (1 for the constant one),
//                  padded to an even count of doubles.
// A record is contiguous because its readers want all of it: they take the
// points of one tile in an order of their own, and 16-byte pieces of one
// record cost a quarter of the sectors that one scattered double per array
// does, on the write side too (each warp turns its 32 records through shared
// memory so that neighbouring lanes write neighbouring pieces).
constexpr int kScatterSlots = 16;  // doubles of a record staged at a time

__host__ __device__ inline int rec_stride(int d, int nchan) { return (d + nchan + 1) & ~1; }

template <bool FEW>
__global__ void __launch_bounds__(256)
bin_scatter_kernel(SpreadGeom g, int64_t n, const double* __restrict__ x,
                   const double* __restrict__ d_kmap, const int* __restrict__ offsets,
                   int* __restrict__ cursor, int nchan, int ones_channel, ChanPtrs cp,
                   int* __restrict__ rec_base, int* __restrict__ rec_idx,
                   double* __restrict__ rec) {
  constexpr int SS = kScatterSlots + 2;  // staging stride: 16-byte rows on distinct banks
  __shared__ KnotAxis s_ax[3];
  __shared__ __align__(16) double s_rec[8][32 * SS];
  __shared__ int s_cnt[FEW ? kFewTiles : 1];
  load_axes(g, d_kmap, s_ax);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int d = g.d, stride = rec_stride(d, nchan);
  double* sr = s_rec[warp];
  // A grid of few tiles ranks a block's points in shared memory and moves each
  // tile's cursor once for all of them: one cursor atomic per point made the
  // points of 1-D grids queue (1e5 points, grid 1024: 32 us, now 9.6).
  // whole blocks go round together: the last one has idle lanes and warps
  for (int64_t ib = (int64_t)blockIdx.x * 256; ib < n; ib += (int64_t)gridDim.x * 256) {
    const int64_t i0 = ib + warp * 32, i = i0 + lane;
    const int cnt = (int)max((int64_t)0, min((int64_t)32, n - i0));
    int m[3];
    double k[3];
    int pos = 0, t = 0, rank = 0;
    if (lane < cnt) t = point_tile(g, s_ax, x, i, m, k);
    if constexpr (FEW) {
      for (int j = threadIdx.x; j < g.ntiles; j += 256) s_cnt[j] = 0;
      __syncthreads();
      if (lane < cnt) rank = atomicAdd(&s_cnt[t], 1);
      __syncthreads();
      for (int j = threadIdx.x; j < g.ntiles; j += 256)
        if (s_cnt[j]) s_cnt[j] = atomicAdd(&cursor[j], s_cnt[j]);
      __syncthreads();
    }
    if (lane < cnt) {
      pos = offsets[t] + (FEW ? s_cnt[t] + rank : atomicAdd(&cursor[t], 1));
      int packed = 0;
      for (int a = 0; a < d; ++a) {
        int home = m[a] % g.L[a];
        if (home < 0) home += g.L[a];
        packed |= (home % g.T[a]) << (10 * a);
      }
      rec_base[pos] = packed;
      rec_idx[pos] = (int)i;
    }
    for (int s0 = 0; s0 < stride; s0 += kScatterSlots) {
      const int ns = min(kScatterSlots, stride - s0);
      if (lane < cnt) {
        for (int j = 0; j < ns; ++j) {
          const int slot = s0 + j, c = slot - d;
          double v = 0.0;
          if (c < 0) {
            v = dsub(k[slot], dmul(g.ax[slot].hx, (double)m[slot]));
          } else if (c < nchan) {
            v = ones_channel && c == 0 ? 1.0 : cp.col[c - ones_channel][i];
          }
          sr[lane * SS + j] = v;
        }
      }
      __syncwarp();
      const int nch = ns / 2;
      for (int t0 = 0; t0 < cnt * nch; t0 += 32) {
        const int e = t0 + lane, r = e / nch, ch = e - r * nch;
        const int64_t p = __shfl_sync(0xffffffffu, pos, r & 31);
        if (e < cnt * nch)
          *reinterpret_cast<double2*>(rec + p * stride + s0 + 2 * ch) =
              *reinterpret_cast<const double2*>(sr + r * SS + 2 * ch);
      }
      __syncwarp();
    }
    if constexpr (FEW) __syncthreads();  // the next round clears the ranks
  }
}

template <typename Acc>
struct AccOps;

template <>
struct AccOps<long long> {
  template <typename Real>
  __device__ static void add_shared(long long* p, Real v, Real scale) {
    long long q = (sizeof(Real) == 4) ? __float2ll_rn((float)(v * scale))
                                      : __double2ll_rn((double)(v * scale));
    if (q != 0) atomicAdd(reinterpret_cast<unsigned long long*>(p), (unsigned long long)q);
  }
  __device__ static void add_global(long long* p, long long v) {
    atomicAdd(reinterpret_cast<unsigned long long*>(p), (unsigned long long)v);
  }
};

template <>
struct AccOps<double> {
  template <typename Real>
  __device__ static void add_shared(double* p, Real v, Real) { atomicAdd(p, (double)v); }
  __device__ static void add_global(double* p, double v) { atomicAdd(p, v); }
};

// Fixed-point scale 2^e per channel so that |sum| over any subset of
// contributions stays below 2^50 (each point adds at most |v| to a cell when
// the taps do not wrap onto the same cell): every rounded product and every
// partial sum is then an integer that a double holds exactly, so the 2-D
// path can round and add in FP64 registers and still be exact and
// independent of the order of the points.  The quantum, 2^-50 of the
// channel's absolute sum, is far below the FP32 rounding of the grid.
constexpr int kFixedBits = 50;

__device__ __forceinline__ double fixed_scale(double absum, int margin_bits) {
  if (!(absum > 0.0)) return 1.0;
  int e = 0;
  frexp(absum, &e);  // absum < 2^e
  return ldexp(1.0, kFixedBits - e - margin_bits);
}

__device__ __forceinline__ float fexp(float v) { return expf(v); }
__device__ __forceinline__ double fexp(double v) { return exp(v); }

// One CTA per work item (a tile, or a chunk of at most g.item_points points of
// a tile).  Threads take (point, tap row) pairs: a tap row fixes the tap
// offsets of all axes but the last, and the thread walks the NT1 taps of the
// last axis, adding every channel of the point into the shared-memory copy of
// the tile plus its halo of msp cells.  The tile is then added to the global
// accumulator with one atomic per non-zero cell.  (In 1-D the lanes' values
// lie a record apart: 378 us for 1e6 points and 12 channels, 361 from an array
// per channel, whose scatter took 290 us, the records' 71.)
template <typename Acc, typename Real, int NT1>
__global__ void __launch_bounds__(kSpreadThreads)
tile_accumulate_kernel(SpreadGeom g, int nchan, int cgroup,
                       const int* __restrict__ offsets, const int* __restrict__ items,
                       const int* __restrict__ rec_base, const double* __restrict__ rec,
                       int stride, const double* __restrict__ absum, int margin_bits,
                       Acc* __restrict__ gacc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Acc* acc = reinterpret_cast<Acc*>(smem_raw);
  const int c_begin = blockIdx.y * cgroup;
  const int nc = min(nchan, c_begin + cgroup) - c_begin;
  const int tc = g.tile_cells;

  const int item = blockIdx.x;
  if (item >= items[g.ntiles]) return;
  int lo = 0, hi = g.ntiles;  // tile owning this item: largest t with items[t] <= item
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (items[mid] <= item) lo = mid; else hi = mid;
  }
  const int tile = lo;
  const int p_begin = offsets[tile] + (item - items[tile]) * g.item_points;
  const int p_end = min(offsets[tile + 1], p_begin + g.item_points);
  int tcoord[3] = {0, 0, 0};
  {
    int r = tile;
    for (int a = g.d - 1; a >= 0; --a) {
      tcoord[a] = r % g.ntile[a];
      r /= g.ntile[a];
    }
  }
  __shared__ Real scale[32];
  for (int i = threadIdx.x; i < nc * tc; i += blockDim.x) acc[i] = Acc(0);
  if (threadIdx.x < 32)
    scale[threadIdx.x] = (threadIdx.x < nc)
                             ? (Real)fixed_scale(absum ? absum[c_begin + threadIdx.x] : 0.0, margin_bits)
                             : Real(1);
  __syncthreads();

  constexpr int MSP = (NT1 - 1) / 2;
  const int d = g.d;
  const int rows = d == 1 ? 1 : (d == 2 ? NT1 : NT1 * NT1);
  const int np = p_end - p_begin;
  const int Wl = g.W[d - 1];
  const Real hxl = (Real)g.ax[d - 1].hx;
  const Real ftl = (Real)g.four_tau[d - 1];
  for (int t = threadIdx.x; t < np * rows; t += blockDim.x) {
    const int pp = t / rows;
    const int p = p_begin + pp;
    const int row = t - pp * rows;
    const int packed = rec_base[p];
    int j[2] = {0, 0};
    if (d == 2) {
      j[0] = row;
    } else if (d == 3) {
      j[0] = row / NT1;
      j[1] = row - j[0] * NT1;
    }
    // weight and local cell of the tap row (all axes but the last)
    Real wrow = Real(1);
    int cell = 0;
    for (int a = 0; a < d - 1; ++a) {
      const Real fr = (Real)rec[(int64_t)p * stride + a];
      const Real diff = fr - (Real)g.ax[a].hx * (Real)(j[a] - MSP);
      wrow *= fexp(-(diff * diff) / (Real)g.four_tau[a]);
      cell = cell * g.W[a] + ((packed >> (10 * a)) & 1023) + j[a];
    }
    cell = cell * Wl + ((packed >> (10 * (d - 1))) & 1023);
    const Real frl = (Real)rec[(int64_t)p * stride + d - 1];
    Real w[NT1];
#pragma unroll
    for (int jl = 0; jl < NT1; ++jl) {
      const Real diff = frl - hxl * (Real)(jl - MSP);
      w[jl] = wrow * fexp(-(diff * diff) / ftl);
    }
    for (int c = 0; c < nc; ++c) {
      const Real v = (Real)rec[(int64_t)p * stride + d + c_begin + c];
      const Real sc = scale[c];
      Acc* dst = acc + c * tc + cell;
#pragma unroll
      for (int jl = 0; jl < NT1; ++jl) AccOps<Acc>::add_shared(dst + jl, v * w[jl], sc);
    }
  }
  __syncthreads();

  // flush: one global atomic per non-zero cell of the tile + halo
  for (int idx = threadIdx.x; idx < nc * tc; idx += blockDim.x) {
    Acc v = acc[idx];
    if (v == Acc(0)) continue;
    int c = idx / tc;
    int r = idx - c * tc;
    int64_t gi = 0;
    int loc[3] = {0, 0, 0};
    for (int a = g.d - 1; a >= 0; --a) {
      loc[a] = r % g.W[a];
      r /= g.W[a];
    }
    for (int a = 0; a < g.d; ++a) {
      int gc = tcoord[a] * g.T[a] + loc[a] - g.msp;
      gc %= g.L[a];
      if (gc < 0) gc += g.L[a];
      gi = gi * g.L[a] + gc;
    }
    AccOps<Acc>::add_global(&gacc[(int64_t)(c_begin + c) * g.cells + gi], v);
  }
}

// ---- 2-D and 3-D path: one or two warps per work item ------------------------
// Tiles of 8 x 8 cells of the last two axes.  The warps of a CTA (one, or two that split the
// channels) take the points of one work item: they sort them by cell
// (counting sort of their indices), then walk them row of cells by row of
// cells, 32 points at a time staged in shared memory (per-axis tap weights
// and the records, copied in the background).  Lane (jm, group) holds, in
// registers, the W = NT1 + 7 cells of one halo row for UC channels: halo row
// r belongs to the lanes with jm = r mod NT1, so at tile row l0 they take tap
// jy = (jm - l0) mod NT1, every lane of the NT1 footprint rows works, and a
// row leaves the registers once, when the walk has passed it.  It goes
// through a small shared buffer to one global atomic per non-zero cell: no
// atomics on shared memory, no accumulator tile.  In the fixed-point
// accumulator every product is rounded to an integer before it is added, so
// sums are exact and the grid does not depend on the order of the points.
//
// In 3-D a tile is one cell thick on the first axis, and the NT1 taps of that
// axis take the place of the channels: tap plane j of a point has the value
// e0[j] v, and a warp takes one channel (27 lanes, three planes each, for 9
// taps).  A point so costs 30 multiply-adds per lane where a thread for each
// halo column of an 8 x 8 x 8 tile, rounding every product by two additions,
// took 37 operations and left more than half of its lanes idle.
//
// Bound by the FP64 pipe (UC (NT1 + 1) multiply-adds per point and warp, about
// 2.2 cycles each), beside which the FP32 grids issue two integer adds per
// product, and by latency: the next point's values are read and scaled beside
// this point's sums, and UC stays at 3 or less, which leaves registers for 12
// to 16 warps.  1e6 points, 12 channels, FP32 grid 512^2: 340 us, where an
// atomic per tile row on a shared tile took 527; 2e6 points, 12 channels, FP64:
// 421 us (758); 1e7 points, one channel, FP32 grid 128^3: 2.80 ms, where a
// thread per halo column took 7.63.
constexpr int kT2 = 8;            // tile edge of the 2-D path
constexpr int kItem2 = 1024;      // most points of a work item

// Register accumulators of the tile kernels.  Fixed point with quantum q (a
// power of two): the product v w is rounded once, to the nearest multiple of
// q, by the fused multiply-add t = v w + 1.5 * 2^52 q (every double in
// [2^52 q, 2^53 q) is a multiple of q, and |v w| < 2^50 q keeps t there).  The
// bit pattern of t is that of the bias plus v w / q, so the register adds the
// bit patterns as integers: no carry is lost in the low 51 bits, where the
// bias has none, and the sum (below 2^50 in magnitude) is their value as a
// signed number.  The sum is exact and independent of the order of the points,
// and v enters with all its bits.  (Adding in the multiply-add itself, with the
// sum in place of the bias, rounds a product halfway between two multiples by
// the parity of the sum so far; keeping such products away by setting v's last
// bit costs that bit, and rounds every one of them up.)  Float64 accumulation
// adds the fused product.
template <typename Acc>
struct RegSum;
template <>
struct RegSum<long long> {
  using T = unsigned long long;
  __device__ static double bias(double q) { return 6755399441055744.0 * q; }  // 1.5 * 2^52 q
  __device__ static void add(T& a, double v, double w, double bias) {
    a += (T)__double_as_longlong(__fma_rn(v, w, bias));
  }
  __device__ static long long value(T a) { return (long long)(a << 13) >> 13; }
};
template <>
struct RegSum<double> {
  using T = double;
  __device__ static double bias(double) { return 0.0; }
  __device__ static void add(T& a, double v, double w, double) { a = __fma_rn(v, w, a); }
  __device__ static double value(T a) { return a; }
};

// Tap weights of one axis from the knot's offset f to its cell:
// val exp(-(f - hx j)^2 / ft), j = -MSP .. MSP, into w: an exponential per tap.
// (The products e0 r^j C_j, two exponentials and a reciprocal per axis, save
// 10% of a 2-D FP64 spread and 15% of a 3-D one and err 1.6 times as much in
// the root mean square of a 2-D stencil.)
template <int NT1>
__device__ __forceinline__ void tap_weights(double f, double val, double hx, double ft,
                                            double inv_ft, double* __restrict__ w) {
#pragma unroll 3
  for (int j = 0; j < NT1; ++j) {
    const double t = f - hx * (double)(j - (NT1 - 1) / 2);
    // the quotient (t^2) / ft, corrected by its residual (Markstein); a single
    // tap has ft infinite and weight 1
    const double p = t * t, q = p * inv_ft;
    w[j] = val * exp(-(NT1 == 1 ? q : __fma_rn(__fma_rn(-q, ft, p), inv_ft, q)));
  }
}

// Tile that owns work item `item`: the largest t with items[t] <= item.  One
// warp probes 32 places at a time (three dependent loads for 16,384 tiles
// instead of fourteen).
__device__ __forceinline__ int item_tile(const int* __restrict__ items, int ntiles, int item,
                                         int lane) {
  int lo = 0, hi = ntiles;  // items[lo] <= item < items[hi]
  while (hi - lo > 1) {
    const int step = (hi - lo + 31) / 32;
    const int t = lo + lane * step;
    const unsigned le = __ballot_sync(0xffffffffu, t < hi && items[t] <= item);
    lo += (31 - __clz(le)) * step;  // lane 0 always holds
    hi = min(hi, lo + step);
  }
  return lo;
}

template <int BYTES>
__device__ __forceinline__ void copy_async(double* dst, const double* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// Channel groups of a warp: as many footprints of NT1 lanes as fit.
__host__ __device__ constexpr int groups2(int nt1) { return nt1 < 4 ? 8 : 32 / nt1; }

// Warps of one SM (one per CTA) that UC channels per lane leave registers for.
__host__ __device__ constexpr int warps2(int nt1, int uc) {
  const int regs = 2 * uc * (nt1 + 7) + 46;  // accumulators and working registers
  return regs <= 128 ? 16 : (regs <= 176 ? 12 : (regs <= 200 ? 10 : 8));
}

// Shared memory of one CTA.  The rows that the lanes still hold at the end
// go through the space of the staged points.  A warp's NCW "channels" are its
// value channels in 2-D and the tap planes of its one channel in 3-D.
template <typename Acc, int D, int NT1, int UC, int NW>
struct Stage2 {
  static constexpr int W = kT2 + NT1 - 1;     // halo cells per axis
  static constexpr int GPL = groups2(NT1);    // channel groups of a warp
  static constexpr int NCW = UC * GPL;        // channels of a warp
  static constexpr int NCB = NCW * NW;        // channels of the CTA
  static constexpr int NVB = D == 2 ? NCB : NW;  // value channels of the CTA
  static constexpr int WXS = (NT1 + 1) & ~1;  // even row stride: two weights per load
  static constexpr int RS = D == 2 ? (2 + NVB + 1) & ~1 : 3 + NVB;  // staged record
  static constexpr int VS = D == 2 ? RS : NCB;  // stride of the values the lanes read
  static constexpr int WR = W | 1;            // row-buffer stride of one channel
  struct Points {
    double rec[2][33 * RS];  // records of this batch and of the next (and one read ahead)
    double wx[32 * WXS];     // weights of the last axis
    double wy[33 * NT1];     // weights of the axis before it
    double val[D == 3 ? 33 * VS : 1];  // 3-D: axis-0 weights times the channels' values
    Acc row[NCB * WR];
    unsigned short order[kItem2];
    unsigned char cell[kItem2];
  };
  union {
    Points st;
    Acc rows[NT1 * NCB * WR];
  };
  double bias[NVB];
  int off[kT2 * kT2 + 1];
  int cur[kT2 * kT2];
  int col[W];  // grid columns of the halo
  int64_t plane[D == 3 ? NT1 : 1];  // 3-D: start of the grid planes of the tap planes
};

// Adds `nrows` halo rows from grid row gr0 on, (rows, NCW, WR) sums of
// one warp's lanes for its first nc channels, to the global accumulator: one
// atomic per non-zero cell.  v_w: its first value channel in the CTA.
template <typename Acc, int D, typename S>
__device__ __forceinline__ void add_rows(const SpreadGeom& g, const S& sh, const Acc* buf,
                                         int nrows, int gr0, int c_begin, int v_w, int nc,
                                         int lane, Acc* __restrict__ gacc) {
  constexpr int W = S::W, N = S::NCW * W, U = (N + 31) / 32;
  const int Lr = g.L[D - 2], Lc = g.L[D - 1];
  for (int r = 0; r < nrows; ++r) {
    int gr = (gr0 + r) % Lr;
    if (gr < 0) gr += Lr;
    Acc* grow = gacc + (int64_t)(c_begin + v_w) * g.cells + (int64_t)gr * Lc;
    const Acc* rb = buf + r * S::NCW * S::WR;
    Acc v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int idx = u * 32 + lane, c = idx / W, j = idx - c * W;
      v[u] = c < nc ? rb[c * S::WR + j] : Acc(0);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int idx = u * 32 + lane, c = idx / W, j = idx - c * W;
      if (v[u] != Acc(0))
        AccOps<Acc>::add_global(grow + (D == 2 ? (int64_t)c * g.cells : sh.plane[c]) + sh.col[j], v[u]);
    }
  }
}

template <int NW>
__device__ __forceinline__ void sync2() {
  if constexpr (NW == 1)
    __syncwarp();
  else
    __syncthreads();
}

template <typename Acc, int D, int NT1, int UC, int NW>
__global__ void __launch_bounds__(32 * NW, warps2(NT1, UC) / NW)
tile_accumulate_reg_kernel(SpreadGeom g, int nchan, const int* __restrict__ offsets,
                           const int* __restrict__ items, const int* __restrict__ rec_base,
                           const double* __restrict__ rec, int stride,
                           const double* __restrict__ absum, int margin_bits,
                           Acc* __restrict__ gacc) {
  using S = Stage2<Acc, D, NT1, UC, NW>;
  using R = RegSum<Acc>;
  constexpr int MSP = (NT1 - 1) / 2;
  constexpr int NLC = kT2 * kT2;
  constexpr int NT = 32 * NW;
  constexpr int W = S::W, GPL = S::GPL, NCW = S::NCW, NVB = S::NVB, WXS = S::WXS, RS = S::RS,
                VS = S::VS, WR = S::WR;
  __shared__ __align__(16) unsigned char s_raw[sizeof(S)];
  S& sh = *reinterpret_cast<S*>(s_raw);
  int* const off = sh.off;
  int* const cur = sh.cur;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c_begin = blockIdx.y * NVB;
  const int nv = min(nchan - c_begin, NVB);  // value channels here
  const int v_w = D == 2 ? warp * NCW : warp;                        // this warp's first one
  const int nc_w = D == 2 ? min(max(nv - v_w, 0), NCW) : (warp < nv ? NT1 : 0);
  const int jm = lane % NT1, grp = lane / NT1;
  const bool active = grp < GPL && grp * UC < nc_w;
  const double hy = g.ax[D - 2].hx, hx = g.ax[D - 1].hx;
  const double ify = 1.0 / g.four_tau[D - 2], ifx = 1.0 / g.four_tau[D - 1];
  const double ifz = 1.0 / g.four_tau[0];
  for (int c = tid; c < NVB; c += NT) {
    const double sc = (c < nv && absum != nullptr) ? fixed_scale(absum[c_begin + c], margin_bits) : 1.0;
    sh.bias[c] = R::bias(1.0 / sc);
  }
  // items in a grid-stride loop: most CTAs of a launch sized by the tiles of
  // the whole (padded) grid would find none
  const int nitems = items[g.ntiles];
  for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
    const int tile = item_tile(items, g.ntiles, item, lane);
    const int p_begin = offsets[tile] + (item - items[tile]) * g.item_points;
    const int np = min(offsets[tile + 1] - p_begin, g.item_points);
    const int tcx = tile % g.ntile[D - 1], tcy = tile / g.ntile[D - 1] % g.ntile[D - 2];
    sync2<NW>();  // the last item's readers are done
    if (tid < W) {
      const int gc = (tcx * kT2 + tid - MSP) % g.L[D - 1];
      sh.col[tid] = gc < 0 ? gc + g.L[D - 1] : gc;
    }
    if (D == 3 && tid < NT1) {
      int gp = (tile / (g.ntile[D - 1] * g.ntile[D - 2]) + tid - MSP) % g.L[0];
      if (gp < 0) gp += g.L[0];
      sh.plane[tid] = (int64_t)gp * g.L[1] * g.L[D - 1];
    }
    // counting sort by cell
    for (int i = tid; i < NLC; i += NT) cur[i] = 0;
    sync2<NW>();
#pragma unroll 4
    for (int i = tid; i < np; i += NT) {
      const int packed = rec_base[p_begin + i];
      const int lc = ((packed >> (10 * (D - 2))) & 1023) * kT2 + ((packed >> (10 * (D - 1))) & 1023);
      sh.st.cell[i] = (unsigned char)lc;
      atomicAdd(&cur[lc], 1);
    }
    sync2<NW>();
    if (warp == 0) {
      const int a0 = cur[2 * lane], a1 = cur[2 * lane + 1];
      int incl = a0 + a1;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      const int excl = incl - a0 - a1;
      off[2 * lane] = excl;
      off[2 * lane + 1] = excl + a0;
      if (lane == 31) off[NLC] = incl;
      __syncwarp();
      cur[2 * lane] = excl;
      cur[2 * lane + 1] = excl + a0;
    }
    sync2<NW>();
    for (int i = tid; i < np; i += NT)
      sh.st.order[atomicAdd(&cur[sh.st.cell[i]], 1)] = (unsigned short)i;
    sync2<NW>();

    // records of the 32 points from b0 on, copied in the background: the knot
    // offsets, then this CTA's channels, in pieces of 16 bytes (3-D: three
    // offsets, so 8 bytes)
    constexpr int PC = D == 2 ? 2 : 1;
    const int npc = D == 2 ? 1 + (nv + 1) / 2 : 3 + nv;
    const int dpt = NT / npc, dpc = NT - dpt * npc;
    const int pt0 = tid / npc, pc0 = tid - pt0 * npc;
    const double* rec_t = rec + (int64_t)p_begin * stride;
    auto fetch = [&](int b0, int half) {
      const int cnt = min(32, np - b0);
      for (int pt = pt0, pc = pc0; pt < cnt;) {
        copy_async<8 * PC>(&sh.st.rec[half][pt * RS + PC * pc],
                           rec_t + (int64_t)sh.st.order[b0 + pt] * stride +
                               (PC * pc >= D ? c_begin : 0) + PC * pc);
        pc += dpc;
        pt += dpt;
        if (pc >= npc) {
          pc -= npc;
          ++pt;
        }
      }
    };
    fetch(0, 0);

    // idle lanes repeat group 0 and drop it
    const int c_w = warp * NCW, vofs = c_w + (active ? grp * UC : 0);
    double bias[UC];
#pragma unroll
    for (int k = 0; k < UC; ++k) bias[k] = sh.bias[D == 2 ? vofs + k : v_w];
    typename R::T a[UC][W];
#pragma unroll
    for (int k = 0; k < UC; ++k)
#pragma unroll
      for (int j = 0; j < W; ++j) a[k][j] = 0;
    int row = 0, half = 0;
    for (int b0 = 0; b0 < np; b0 += 32, half ^= 1) {
      const int b1 = min(b0 + 32, np);
      copies_wait();
      sync2<NW>();  // this batch's records are there, the last one's readers done
      if (b0 + lane < b1) {
        const double* r = &sh.st.rec[half][lane * RS];
        if (NW == 1 || warp == 0)
          tap_weights<NT1>(r[D - 2], 1.0, hy, g.four_tau[D - 2], ify, sh.st.wy + lane * NT1);
        if (NW == 1 || warp == 1)
          tap_weights<NT1>(r[D - 1], 1.0, hx, g.four_tau[D - 1], ifx, sh.st.wx + lane * WXS);
        if (D == 3 && warp < nv)
          tap_weights<NT1>(r[0], r[3 + warp], g.ax[0].hx, g.four_tau[0], ifz,
                           sh.st.val + lane * VS + c_w);
      }
      sync2<NW>();
      fetch(b1, half ^ 1);
      for (;;) {
        int jy = jm - row % NT1;
        if (jy < 0) jy += NT1;
        const int* ro = off + row * kT2;
        int pp = max(ro[0], b0) - b0;
        const double* yp = sh.st.wy + pp * NT1 + jy;
        const double* vp = (D == 2 ? sh.st.rec[half] + 2 : sh.st.val) + pp * VS + vofs;
        const double2* xp = reinterpret_cast<const double2*>(sh.st.wx + pp * WXS);
        double v[UC];  // the next point's values times its axis-0 weight
#pragma unroll
        for (int k = 0; k < UC; ++k) v[k] = *yp * vp[k];
#pragma unroll
        for (int cr = 0; cr < kT2; ++cr) {
          const int pe = min(ro[cr + 1], b1) - b0;
#pragma unroll 1
          for (; pp < pe; ++pp) {
            yp += NT1;
            vp += VS;
            const double wyn = *yp;
            double u[UC], w[WXS];
#pragma unroll
            for (int k = 0; k < UC; ++k) u[k] = vp[k];
#pragma unroll
            for (int jx = 0; jx < NT1; jx += 2) {
              const double2 q = xp[jx / 2];
              w[jx] = q.x;
              w[jx + 1] = q.y;
            }
            xp += WXS / 2;
#pragma unroll
            for (int jx = 0; jx < NT1; ++jx)
#pragma unroll
              for (int k = 0; k < UC; ++k) R::add(a[k][cr + jx], v[k], w[jx], bias[k]);
#pragma unroll
            for (int k = 0; k < UC; ++k) v[k] = wyn * u[k];
          }
        }
        if (ro[kT2] > b1) break;      // the row goes on in the next batch
        if (row >= W - NT1) break;    // every lane on its last row
        // halo row `row` is complete: its lanes hand it over and start row + NT1
        Acc* rb = sh.st.row + c_w * WR;
        if (active && jm == row % NT1) {
          Acc* rp = rb + grp * UC * WR;
#pragma unroll
          for (int k = 0; k < UC; ++k)
#pragma unroll
            for (int j = 0; j < W; ++j) {
              rp[k * WR + j] = R::value(a[k][j]);
              a[k][j] = 0;
            }
        }
        __syncwarp();
        add_rows<Acc, D, S>(g, sh, rb, 1, tcy * kT2 + row - MSP, c_begin, v_w, nc_w, lane, gacc);
        __syncwarp();
        ++row;
      }
    }
    // the last NT1 rows, each in its own lanes
    sync2<NW>();
    Acc* rb = sh.rows + (size_t)warp * NT1 * NCW * WR;
    if (active) {
      int r = (jm - (W - NT1)) % NT1;  // position of this lane's row among W - NT1 .. W - 1
      if (r < 0) r += NT1;
      Acc* rp = rb + (r * NCW + grp * UC) * WR;
#pragma unroll
      for (int k = 0; k < UC; ++k)
#pragma unroll
        for (int j = 0; j < W; ++j) rp[k * WR + j] = R::value(a[k][j]);
    }
    __syncwarp();
    add_rows<Acc, D, S>(g, sh, rb, NT1, tcy * kT2 + (W - NT1) - MSP, c_begin, v_w, nc_w, lane, gacc);
  }
}

// Grid value = accumulator / fixed-point scale (a power of two, so the
// product with its inverse is exact) / n.  Thread per cell, all channels.
template <typename Acc, typename Out, bool kFixed>
__global__ void finalize_kernel(int nchan, int64_t cells, const Acc* __restrict__ gacc,
                                const double* __restrict__ absum, int margin_bits, double inv_n,
                                Out* __restrict__ out) {
  __shared__ double inv_scale[FLPR_MAX_CHANNELS];
  for (int c = threadIdx.x; c < nchan; c += blockDim.x)
    inv_scale[c] = kFixed ? 1.0 / fixed_scale(absum[c], margin_bits) : 1.0;
  __syncthreads();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < cells;
       i += (int64_t)gridDim.x * blockDim.x) {
    for (int c = 0; c < nchan; ++c) {
      const int64_t k = (int64_t)c * cells + i;
      const double v = (double)gacc[k] * inv_scale[c];
      out[k] = (Out)(v * inv_n);
    }
  }
}

// 2-D and 3-D grids of at least 8 x 8 cells on their last two axes take the
// register path, with up to 13 taps per axis in 2-D and 9 in 3-D (what the
// lanes hold; the wider stencils of the oversampled accuracies go through
// shared-memory atomics).
static bool use_reg_path(int d, const int* L, int msp) {
  return d >= 2 && L[d - 2] >= kT2 && L[d - 1] >= kT2 && 2 * msp + 1 <= (d == 2 ? 13 : 9);
}

static void make_geom(SpreadGeom& g, int d, const int* L, int msp, const double* tau,
                      const double* kmap) {
  memset(&g, 0, sizeof(g));
  const bool reg = use_reg_path(d, L, msp);
  g.d = d;
  g.msp = msp;
  g.ntaps1 = 2 * msp + 1;
  g.item_points = tuning(FLPR_TUNE_SPREAD_ITEM_POINTS);
  static const int tile2[3] = {16, 16, 1};
  static const int tile3[3] = {8, 8, 8};
  g.cells = 1;
  g.tile_cells = 1;
  g.ntiles = 1;
  for (int a = 0; a < 3; ++a) {
    if (a < d) {
      g.L[a] = L[a];
      int T = d == 1 ? 256 : (reg ? (a < d - 2 ? 1 : kT2) : (d == 2 ? (L[0] < kT2 || L[1] < kT2 ? kT2 : tile2[a])
                                                                  : tile3[a]));
      if (d == 3 && !reg) {
        // wide stencils (oversampled accuracies): smaller tiles, so that one
        // channel's tile plus halo fits shared memory
        const size_t kMax3 = (size_t)200 * 1024;
        while (T > 1 && sizeof(long long) * (size_t)(T + 2 * msp) * (T + 2 * msp) *
                                (T + 2 * msp) > kMax3)
          T >>= 1;
      }
      if (T > L[a]) T = L[a];
      g.T[a] = T;
      g.ntile[a] = (L[a] + T - 1) / T;
      g.W[a] = T + 2 * msp;
      g.cells *= L[a];
      g.tile_cells *= g.W[a];
      g.ntiles *= g.ntile[a];
      g.four_tau[a] = 4.0 * tau[a];
      const double* k = kmap + 9 * a;
      g.ax[a] = KnotAxis{k[0], k[1], k[2], k[3], k[4], k[5], k[6], k[7], k[8]};
    } else {
      g.L[a] = 1;
      g.T[a] = 1;
      g.ntile[a] = 1;
      g.W[a] = 1;
    }
  }
}

// Points per work item, the same for the spread and for the deposits that
// read its records.  Grids with few tiles (small 1-D grids): about four items
// per SM.  Register path, one or two warps per item, which walk its points one
// after another: at least 24 warps' worth of items per SM (two rounds of the
// resident ones), 256 to 1024 points; where those would leave the device
// empty, 32 to 128, at 3 warps' worth, since every item adds its halo to the
// grid (spread and deposits, 6 channels: 5e3 points on 70^2 97 us with 256, 84
// with 32; 2e4 on 40^2 131 with 256, 91 with 64; 12 channels, 1e5 points on
// 200^2: 178 with 256, 190 with 128).
// All of it times the setting over its default, with a batch of the staged
// points at least.
static void size_items(SpreadGeom& g, int64_t n, bool reg) {
  if (reg) {
    const int64_t per = n / (24LL * sm_count());
    int64_t ip = 32;
    while (ip < 8 * per && ip < 256) ip <<= 1;
    while (ip < per && ip < kItem2) ip <<= 1;
    ip = ip * g.item_points / kTuneItemPoints;
    g.item_points = (int)(ip < 32 ? 32 : (ip > kItem2 ? kItem2 : ip));
    return;
  }
  const int64_t target = 4LL * sm_count();
  if (g.ntiles < target) {
    const int64_t per = (n + target - 1) / target;
    int ip = 256;
    while (ip < per && ip < g.item_points) ip <<= 1;
    if (ip < g.item_points) g.item_points = ip;
  }
}

static int margin_bits_for(const SpreadGeom& g) {
  int m = 1;
  for (int a = 0; a < g.d; ++a)
    if (g.L[a] < g.ntaps1) m += 4;  // taps wrap onto the same cell
  return m;
}

static int channel_group(const SpreadGeom& g, int nchan, size_t acc_bytes) {
  // 1-D/2-D: four CTAs per SM; 3-D tiles are larger: two CTAs per SM, or
  // one when a wide stencil's tile needs more
  size_t budget = (g.d == 3 ? 110 : 55) * 1024;
  if (g.d == 3 && acc_bytes * (size_t)g.tile_cells > budget) budget = (size_t)200 * 1024;
  int cg = (int)(budget / (acc_bytes * (size_t)g.tile_cells));
  if (cg > 32) cg = 32;  // fixed-point scales of one group live in 32 shared slots
  if (cg > nchan) cg = nchan;
  return cg;
}

struct SpreadWs {
  int* counts;
  int* offsets;
  int* items;
  int* cursor;
  int* rec_base;
  int* rec_idx;
  int2* totals;
  double* rec;
  double* absum;
  void* gacc;
};

template <typename A>
static void spread_layout(A& ar, int d, int64_t n, int ntiles, int nchan, int64_t cells,
                          SpreadWs* w) {
  auto p1 = ar.template take<int>(ntiles);
  auto p2 = ar.template take<int>(ntiles + 1);
  auto p3 = ar.template take<int>(ntiles + 1);
  auto p4 = ar.template take<int>(ntiles);
  auto p5 = ar.template take<int>(n);
  auto p6 = ar.template take<double>((size_t)rec_stride(d, nchan) * n);
  auto p8 = ar.template take<double>(FLPR_MAX_CHANNELS);
  auto p9 = ar.template take<double>((size_t)nchan * cells);
  auto p10 = ar.template take<int>(n);
  auto p11 = ar.template take<int2>((ntiles + kScanTiles - 1) / kScanTiles);
  if (w) {
    w->counts = (int*)p1;
    w->offsets = (int*)p2;
    w->items = (int*)p3;
    w->cursor = (int*)p4;
    w->rec_base = (int*)p5;
    w->rec = (double*)p6;
    w->absum = (double*)p8;
    w->gacc = (void*)p9;
    w->rec_idx = (int*)p10;
    w->totals = (int2*)p11;
  }
}

struct SizeArena {
  size_t used = 0;
  template <typename T>
  T* take(size_t count) {
    used = align_up(used) + align_up(count * sizeof(T));
    return nullptr;
  }
};

template <int NT1>
static int launch_accumulate(const SpreadGeom& g, int nchan, int cg,
                             const SpreadWs& w, bool fixed, int margin, size_t smem, dim3 grid,
                             cudaStream_t s) {
  if (fixed) {
    auto k = tile_accumulate_kernel<long long, double, NT1>;
    FLPR_CUDA(raise_dyn_smem(k, smem));
    FLPR_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout,
                                   cudaSharedmemCarveoutMaxShared));
    k<<<grid, kSpreadThreads, smem, s>>>(g, nchan, cg, w.offsets, w.items, w.rec_base, w.rec,
                                         rec_stride(g.d, nchan), w.absum, margin,
                                         (long long*)w.gacc);
  } else {
    auto k = tile_accumulate_kernel<double, double, NT1>;
    FLPR_CUDA(raise_dyn_smem(k, smem));
    FLPR_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout,
                                   cudaSharedmemCarveoutMaxShared));
    k<<<grid, kSpreadThreads, smem, s>>>(g, nchan, cg, w.offsets, w.items, w.rec_base, w.rec,
                                         rec_stride(g.d, nchan), nullptr, margin,
                                         (double*)w.gacc);
  }
  FLPR_LAUNCH_CHECK();
  return FLPR_OK;
}

template <typename Acc, int D, int NT1, int UC, int NW>
static int launch_reg_k(const SpreadGeom& g, int nchan, const SpreadWs& w, const double* absum,
                        int margin, int64_t max_items, cudaStream_t s) {
  auto k = tile_accumulate_reg_kernel<Acc, D, NT1, UC, NW>;
  FLPR_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 cudaSharedmemCarveoutMaxShared));
  constexpr int NVB = Stage2<Acc, D, NT1, UC, NW>::NVB;
  // a CTA per item in 2-D (dealing them out in turn cost 5% there); in 3-D
  // the slabs of the padded grid are 8 times the occupied ones and more: four
  // rounds of the resident CTAs, each taking items in turn
  const int64_t cap = D == 2 ? max_items : 4LL * sm_count() * (warps2(NT1, UC) / NW);
  const unsigned nb = (unsigned)(max_items < cap ? max_items : cap);
  k<<<dim3(nb, (unsigned)((nchan + NVB - 1) / NVB)), 32 * NW, 0, s>>>(
      g, nchan, w.offsets, w.items, w.rec_base, w.rec, rec_stride(D, nchan), absum, margin,
      (Acc*)w.gacc);
  FLPR_LAUNCH_CHECK();
  return FLPR_OK;
}

#define FLPR_REG(D, U, N)                                                                         \
  return fixed ? launch_reg_k<long long, D, NT1, U, N>(g, nchan, w, w.absum, margin, max_items, s) \
               : launch_reg_k<double, D, NT1, U, N>(g, nchan, w, nullptr, margin, max_items, s);

// Channels per lane and warps per item: the channels spread over the lane
// groups of one warp while that needs at most three per lane, else of two
// warps, which share the sort, the records and (one axis each) the weights.
template <int NT1>
static int launch_accumulate_2d(const SpreadGeom& g, int nchan, const SpreadWs& w, bool fixed,
                                int margin, int64_t max_items, cudaStream_t s) {
  constexpr int GPL = groups2(NT1);
  const int uc = (nchan + GPL - 1) / GPL;
  if (uc <= 1) FLPR_REG(2, 1, 1)
  if (uc == 2) FLPR_REG(2, 2, 1)
  if (uc == 3) FLPR_REG(2, 3, 1)
  if (uc == 4) FLPR_REG(2, 2, 2)
  FLPR_REG(2, 3, 2)
}

// 3-D: one channel per warp, two warps when there is more than one.
template <int NT1>
static int launch_accumulate_3d(const SpreadGeom& g, int nchan, const SpreadWs& w, bool fixed,
                                int margin, int64_t max_items, cudaStream_t s) {
  constexpr int UC = (NT1 + groups2(NT1) - 1) / groups2(NT1);
  if (nchan == 1) FLPR_REG(3, UC, 1)
  FLPR_REG(3, UC, 2)
}
#undef FLPR_REG

static int finalize(const SpreadGeom& g, int64_t n, int nchan, bool fixed, int margin,
                    const SpreadWs& w, void* d_grid_out, cudaStream_t s);

}  // namespace flpr

using namespace flpr;

extern "C" {

size_t flpr_spread_ws(int d, int64_t n, const int* h_L, int msp, int nchan, int prec) {
  if (d < 1 || d > 3 || n < 1 || nchan < 1) return 0;
  SpreadGeom g;
  double tau[3] = {1, 1, 1}, kmap[27] = {0};
  make_geom(g, d, h_L, msp, tau, kmap);
  SizeArena ar;
  spread_layout(ar, d, n, g.ntiles, nchan, g.cells, nullptr);
  return ar.used;
}

// d_kmap: when not null, the knot maps (d x 9) are read on the device from
// there (h_kmap then only supplies the knot spacings, column 8).
static int spread_impl(int d, int64_t n, const double* d_x, const double* h_kmap,
                       const double* d_kmap, const int* h_L, int msp, const double* h_tau,
                       int nchan, int ones_channel, const double* const* h_cols,
                       void* d_grid_out, int prec, void* d_ws, size_t ws_bytes, void* stream) {
  FLPR_CHECK_ARG(d >= 1 && d <= 3, "spread: d=%d not in [1,3]", d);
  FLPR_CHECK_ARG(n >= 1 && n < (int64_t)1 << 31, "spread: n=%lld out of range", (long long)n);
  FLPR_CHECK_ARG(msp >= 0 && 2 * msp + 1 <= kMaxTaps1, "spread: msp=%d not in [0,12]", msp);
  FLPR_CHECK_ARG(nchan >= 1 && nchan <= FLPR_MAX_CHANNELS, "spread: nchan=%d", nchan);
  FLPR_CHECK_ARG(ones_channel == 0 || ones_channel == 1, "spread: ones_channel must be 0/1");
  FLPR_CHECK_ARG(prec == FLPR_PREC_F32 || prec == FLPR_PREC_F64, "spread: bad precision");
  for (int a = 0; a < d; ++a) FLPR_CHECK_ARG(h_L[a] >= 1, "spread: L[%d]=%d", a, h_L[a]);
  if (ws_bytes < flpr_spread_ws(d, n, h_L, msp, nchan, prec)) {
    set_error("spread: workspace too small");
    return FLPR_ERR_WORKSPACE;
  }
  cudaStream_t s = as_stream(stream);
  SpreadGeom g;
  make_geom(g, d, h_L, msp, h_tau, h_kmap);
  size_items(g, n, use_reg_path(d, h_L, msp));
  ChanPtrs cp;
  memset(&cp, 0, sizeof(cp));
  for (int c = 0; c < nchan - ones_channel; ++c) cp.col[c] = h_cols[c];
  Arena ar(d_ws, ws_bytes);
  SpreadWs w;
  const bool fixed = (prec == FLPR_PREC_F32);
  spread_layout(ar, d, n, g.ntiles, nchan, g.cells, &w);
  const int margin = margin_bits_for(g);
  FLPR_CUDA(cudaMemsetAsync(w.counts, 0, sizeof(int) * g.ntiles, s));
  FLPR_CUDA(cudaMemsetAsync(w.absum, 0, sizeof(double) * FLPR_MAX_CHANNELS, s));
  FLPR_CUDA(cudaMemsetAsync(w.gacc, 0, sizeof(double) * (size_t)nchan * g.cells, s));

  int nb = (int)((n + 255) / 256);
  if (nb > 8 * sm_count()) nb = 8 * sm_count();
  // per-channel sums of |v|: the fixed-point scales of the FP32 grid and of
  // the sorted adjoint deposits (flpr_deposit_sorted) in either precision
  int nbc = (int)((n + 2047) / 2048);  // eight values per thread, then longer loops
  if (nbc > sm_count()) nbc = sm_count();
  bin_count_kernel<<<nb + nbc * (nchan - ones_channel), 256, 0, s>>>(
      g, n, d_x, d_kmap, w.counts, nchan, ones_channel, cp, w.absum, nb, nbc);
  FLPR_LAUNCH_CHECK();
  const int nsb = (g.ntiles + kScanTiles - 1) / kScanTiles;
  tile_scan_kernel<<<nsb, 1024, 0, s>>>(g.ntiles, g.item_points, w.counts, w.offsets, w.items,
                                        w.cursor, w.totals);
  FLPR_LAUNCH_CHECK();
  if (nsb > 1) {
    tile_scan_add_kernel<<<nsb, 1024, 0, s>>>(g.ntiles, w.totals, w.offsets, w.items);
    FLPR_LAUNCH_CHECK();
  }
  // records and tap weights are float64 in both precisions: FP32 weights
  // lose ~1e-6 on the far taps (exponents near 8), which ill-conditioned
  // local systems in sparse corners amplify; only the accumulator differs
  // one point per thread up to 32 CTAs per SM: every thread waits for the
  // slot its cursor atomic returns, so more of them in flight hide it
  int nbs = (int)((n + 255) / 256);
  if (nbs > 32 * sm_count()) nbs = 32 * sm_count();
  auto scatter = g.ntiles <= kFewTiles ? bin_scatter_kernel<true> : bin_scatter_kernel<false>;
  scatter<<<nbs, 256, 0, s>>>(g, n, d_x, d_kmap, w.offsets, w.cursor, nchan,
                                         ones_channel, cp, w.rec_base, w.rec_idx, w.rec);
  FLPR_LAUNCH_CHECK();

  int64_t max_items = (int64_t)g.ntiles + (n + g.item_points - 1) / g.item_points;
  if (d == 2 && use_reg_path(d, h_L, msp)) {
    int st = FLPR_OK;
    switch (g.ntaps1) {
      case 1: st = launch_accumulate_2d<1>(g, nchan, w, fixed, margin, max_items, s); break;
      case 3: st = launch_accumulate_2d<3>(g, nchan, w, fixed, margin, max_items, s); break;
      case 5: st = launch_accumulate_2d<5>(g, nchan, w, fixed, margin, max_items, s); break;
      case 7: st = launch_accumulate_2d<7>(g, nchan, w, fixed, margin, max_items, s); break;
      case 9: st = launch_accumulate_2d<9>(g, nchan, w, fixed, margin, max_items, s); break;
      case 11: st = launch_accumulate_2d<11>(g, nchan, w, fixed, margin, max_items, s); break;
      case 13: st = launch_accumulate_2d<13>(g, nchan, w, fixed, margin, max_items, s); break;
      default: set_error("spread: msp=%d not supported (0..12)", g.msp); return FLPR_ERR_ARG;
    }
    if (st != FLPR_OK) return st;
    return finalize(g, n, nchan, fixed, margin, w, d_grid_out, s);
  }
  if (d == 3 && use_reg_path(d, h_L, msp)) {
    int st = FLPR_OK;
    switch (g.ntaps1) {
      case 1: st = launch_accumulate_3d<1>(g, nchan, w, fixed, margin, max_items, s); break;
      case 3: st = launch_accumulate_3d<3>(g, nchan, w, fixed, margin, max_items, s); break;
      case 5: st = launch_accumulate_3d<5>(g, nchan, w, fixed, margin, max_items, s); break;
      case 7: st = launch_accumulate_3d<7>(g, nchan, w, fixed, margin, max_items, s); break;
      case 9: st = launch_accumulate_3d<9>(g, nchan, w, fixed, margin, max_items, s); break;
      default: set_error("spread: msp=%d not supported by the 3-D path", g.msp); return FLPR_ERR_ARG;
    }
    if (st != FLPR_OK) return st;
    return finalize(g, n, nchan, fixed, margin, w, d_grid_out, s);
  }
  const size_t acc_bytes = 8;
  int cg = channel_group(g, nchan, acc_bytes);
  FLPR_CHECK_ARG(cg >= 1, "spread: tile does not fit shared memory");
  int ngroups = (nchan + cg - 1) / cg;
  size_t smem = acc_bytes * (size_t)cg * g.tile_cells;
  dim3 grid((unsigned)max_items, (unsigned)ngroups);
  int status = FLPR_OK;
  switch (g.ntaps1) {
    case 1: status = launch_accumulate<1>(g, nchan, cg, w, fixed, margin, smem, grid, s); break;
    case 3: status = launch_accumulate<3>(g, nchan, cg, w, fixed, margin, smem, grid, s); break;
    case 5: status = launch_accumulate<5>(g, nchan, cg, w, fixed, margin, smem, grid, s); break;
    case 7: status = launch_accumulate<7>(g, nchan, cg, w, fixed, margin, smem, grid, s); break;
    case 9: status = launch_accumulate<9>(g, nchan, cg, w, fixed, margin, smem, grid, s); break;
    case 11: status = launch_accumulate<11>(g, nchan, cg, w, fixed, margin, smem, grid, s); break;
    case 13: status = launch_accumulate<13>(g, nchan, cg, w, fixed, margin, smem, grid, s); break;
    case 15: status = launch_accumulate<15>(g, nchan, cg, w, fixed, margin, smem, grid, s); break;
    case 17: status = launch_accumulate<17>(g, nchan, cg, w, fixed, margin, smem, grid, s); break;
    case 19: status = launch_accumulate<19>(g, nchan, cg, w, fixed, margin, smem, grid, s); break;
    case 21: status = launch_accumulate<21>(g, nchan, cg, w, fixed, margin, smem, grid, s); break;
    case 23: status = launch_accumulate<23>(g, nchan, cg, w, fixed, margin, smem, grid, s); break;
    case 25: status = launch_accumulate<25>(g, nchan, cg, w, fixed, margin, smem, grid, s); break;
    default: set_error("spread: msp=%d not supported (0..12)", g.msp); return FLPR_ERR_ARG;
  }
  if (status != FLPR_OK) return status;
  return finalize(g, n, nchan, fixed, margin, w, d_grid_out, s);
}

int flpr_spread(int d, int64_t n, const double* d_x, const double* h_kmap, const int* h_L,
                int msp, const double* h_tau, int nchan, int ones_channel,
                const double* const* h_cols, void* d_grid_out, int prec, void* d_ws,
                size_t ws_bytes, void* stream) {
  FLPR_CHECK_ARG(h_kmap != nullptr, "spread: null knot map");
  return spread_impl(d, n, d_x, h_kmap, nullptr, h_L, msp, h_tau, nchan, ones_channel, h_cols,
                     d_grid_out, prec, d_ws, ws_bytes, stream);
}

int flpr_spread_dkmap(int d, int64_t n, const double* d_x, const double* d_kmap,
                      const double* h_hx, const int* h_L, int msp, const double* h_tau,
                      int nchan, int ones_channel, const double* const* h_cols,
                      void* d_grid_out, int prec, void* d_ws, size_t ws_bytes, void* stream) {
  FLPR_CHECK_ARG(d >= 1 && d <= 3, "spread: d=%d not in [1,3]", d);
  FLPR_CHECK_ARG(d_kmap != nullptr && h_hx != nullptr, "spread: null knot map");
  double hk[27] = {0.0};
  for (int a = 0; a < d; ++a) hk[9 * a + 8] = h_hx[a];
  return spread_impl(d, n, d_x, hk, d_kmap, h_L, msp, h_tau, nchan, ones_channel, h_cols,
                     d_grid_out, prec, d_ws, ws_bytes, stream);
}

int flpr_spread_grid64(int d, int64_t n, const int* h_L, int msp, int nchan, const void* d_ws,
                       size_t ws_bytes, double* d_grid64, void* stream) {
  return flpr_spread_grid64_channels(d, n, h_L, msp, nchan, nchan, d_ws, ws_bytes, d_grid64,
                                     stream);
}

int flpr_spread_grid64_channels(int d, int64_t n, const int* h_L, int msp, int nchan, int nout,
                                const void* d_ws, size_t ws_bytes, double* d_grid64,
                                void* stream) {
  FLPR_CHECK_ARG(d >= 1 && d <= 3, "spread_grid64: d=%d not in [1,3]", d);
  FLPR_CHECK_ARG(n >= 1 && nchan >= 1 && nchan <= FLPR_MAX_CHANNELS, "spread_grid64: n/nchan");
  FLPR_CHECK_ARG(nout >= 1 && nout <= nchan, "spread_grid64: nout=%d not in [1, %d]", nout, nchan);
  FLPR_CHECK_ARG(d_ws != nullptr && d_grid64 != nullptr, "spread_grid64: null pointer");
  for (int a = 0; a < d; ++a) FLPR_CHECK_ARG(h_L[a] >= 1, "spread_grid64: L[%d]=%d", a, h_L[a]);
  if (ws_bytes < flpr_spread_ws(d, n, h_L, msp, nchan, FLPR_PREC_F32)) {
    set_error("spread_grid64: workspace too small");
    return FLPR_ERR_WORKSPACE;
  }
  SpreadGeom g;
  double tau[3] = {1, 1, 1}, kmap[27] = {0};
  make_geom(g, d, h_L, msp, tau, kmap);
  Arena ar(const_cast<void*>(d_ws), ws_bytes);
  SpreadWs w;
  spread_layout(ar, d, n, g.ntiles, nchan, g.cells, &w);
  int64_t fb64 = (g.cells + 255) / 256;
  if (fb64 > 16 * sm_count()) fb64 = 16 * sm_count();
  finalize_kernel<long long, double, true><<<(int)fb64, 256, 0, as_stream(stream)>>>(
      nout, g.cells, (const long long*)w.gacc, w.absum, margin_bits_for(g), 1.0 / (double)n,
      d_grid64);
  FLPR_LAUNCH_CHECK();
  return FLPR_OK;
}

int flpr_spread_order(int d, int64_t n, const int* h_L, int msp, int nchan, const void* d_ws,
                      size_t ws_bytes, const int** d_order) {
  FLPR_CHECK_ARG(d >= 1 && d <= 3, "spread_order: d=%d not in [1,3]", d);
  FLPR_CHECK_ARG(n >= 1 && nchan >= 1 && nchan <= FLPR_MAX_CHANNELS, "spread_order: n/nchan");
  FLPR_CHECK_ARG(d_ws != nullptr && d_order != nullptr, "spread_order: null pointer");
  for (int a = 0; a < d; ++a) FLPR_CHECK_ARG(h_L[a] >= 1, "spread_order: L[%d]=%d", a, h_L[a]);
  if (ws_bytes < flpr_spread_ws(d, n, h_L, msp, nchan, FLPR_PREC_F32)) {
    set_error("spread_order: workspace too small");
    return FLPR_ERR_WORKSPACE;
  }
  SpreadGeom g;
  double tau[3] = {1, 1, 1}, kmap[27] = {0};
  make_geom(g, d, h_L, msp, tau, kmap);
  Arena ar(const_cast<void*>(d_ws), ws_bytes);
  SpreadWs w;
  spread_layout(ar, d, n, g.ntiles, nchan, g.cells, &w);
  *d_order = w.rec_idx;
  return FLPR_OK;
}

int flpr_knot_map(int d, int64_t n, const double* d_stats, const double* h_ks,
                  const double* h_r0, const double* h_hx, double* d_kmap, void* stream) {
  FLPR_CHECK_ARG(d >= 1 && d <= 3, "knot_map: d=%d not in [1,3]", d);
  FLPR_CHECK_ARG(n >= 1, "knot_map: n=%lld", (long long)n);
  FLPR_CHECK_ARG(d_stats && h_ks && h_r0 && h_hx && d_kmap, "knot_map: null pointer");
  KnotConsts kc{};
  for (int a = 0; a < d; ++a) {
    kc.ks[a] = h_ks[a];
    kc.r0[a] = h_r0[a];
    kc.hx[a] = h_hx[a];
  }
  knot_map_kernel<<<1, 32, 0, as_stream(stream)>>>(d, (double)(n - 1), d_stats, kc, d_kmap);
  FLPR_LAUNCH_CHECK();
  return FLPR_OK;
}

}  // extern "C"

namespace flpr {

static int finalize(const SpreadGeom& g, int64_t n, int nchan, bool fixed, int margin,
                    const SpreadWs& w, void* d_grid_out, cudaStream_t s) {
  int64_t fb64 = (g.cells + 255) / 256;
  if (fb64 > 16 * sm_count()) fb64 = 16 * sm_count();
  const int fb = (int)fb64;
  double inv_n = 1.0 / (double)n;
  if (fixed) {
    finalize_kernel<long long, float, true><<<fb, 256, 0, s>>>(nchan, g.cells, (long long*)w.gacc,
                                                         w.absum, margin, inv_n,
                                                         (float*)d_grid_out);
  } else {
    finalize_kernel<double, double, false><<<fb, 256, 0, s>>>(nchan, g.cells, (double*)w.gacc, nullptr,
                                                       margin, inv_n, (double*)d_grid_out);
  }
  FLPR_LAUNCH_CHECK();
  return FLPR_OK;
}

}  // namespace flpr

// ---- adjoint deposits from the tile-sorted records --------------------------
// The dual form of the GCV / Hutchinson sums (see flpr_deposit) needs, per
// cell g of the raw grid, Q[g][c] = sum_i w_ig v_ic and the corner-pair
// weights B of the multilinear stencils.  Here one CTA takes the same work
// item as the spread (the points of one spreading tile, in tile order, with
// their point indices and channel values already in the records) and
// accumulates its deposits in a shared-memory window of the raw grid around
// the tile; the window goes to the global sums with one atomic per non-zero
// cell.  Every contribution is rounded to a 64-bit fixed-point integer
// (quantum 2^-62 of the channel's absolute sum; of n for the pair weights),
// so the sums are exact and do not depend on the order of the points: the
// deposits, and with them the FP32 fit, are bitwise reproducible.  The
// output arrays Q and B hold the integers until the finishing pass turns
// them into doubles in place.
namespace flpr {

constexpr int kDepThreads = 256;
constexpr int kDepHalo = 2;       // raw-grid cells of margin around a spreading tile
constexpr int kDepMaxChan = 32;

struct DepositGeom {
  int G[2];
  double x0[2], dx[2];
  int m0[2];     // spreading cell of raw-grid node 0, per axis (a window hint only)
  int win[2];    // window extent (raw-grid cells) per axis
  int C;         // value channels
  int ones;      // 1: spread channel 0 was the constant (not deposited)
  int64_t n;     // points
};

__host__ __device__ constexpr int dep_pairs(int D) { return (1 << D) * ((1 << D) + 1) / 2; }

__device__ __forceinline__ double dep_scale(double absum, int extra_bits) {
  if (!(absum > 0.0)) return 1.0;
  int e = 0;
  frexp(absum, &e);  // absum < 2^e
  return ldexp(1.0, 62 - extra_bits - e);
}

template <int D>
__global__ void __launch_bounds__(kDepThreads)
tile_deposit_kernel(SpreadGeom g, DepositGeom dg, int64_t n, const double* __restrict__ x,
                    const int* __restrict__ offsets, const int* __restrict__ items,
                    const int* __restrict__ rec_idx, const double* __restrict__ rec, int stride,
                    const double* __restrict__ absum, unsigned long long* __restrict__ qacc,
                    unsigned long long* __restrict__ bacc) {
  constexpr int NC = 1 << D;
  constexpr int NP = dep_pairs(D);
  extern __shared__ __align__(16) unsigned long long sacc[];  // window cells x (C + NP)
  __shared__ double s_scale[kDepMaxChan + 1];
  const int C = dg.C, wst = C + NP;
  const int W0 = dg.win[0], W1 = D == 2 ? dg.win[1] : 1;
  const int item = blockIdx.x;
  if (item >= items[g.ntiles]) return;
  int lo = 0, hi = g.ntiles;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (items[mid] <= item) lo = mid; else hi = mid;
  }
  const int tile = lo;
  const int p_begin = offsets[tile] + (item - items[tile]) * g.item_points;
  const int p_end = min(offsets[tile + 1], p_begin + g.item_points);
  // raw-grid window of the tile: node j sits at spreading cell (m0 + j) mod L
  // (the knots are centred on the periodic grid); points whose stencil
  // leaves the window go straight to the global sums
  int org[2] = {0, 0};
  {
    int tc[2] = {tile, 0};
    if (D == 2) {
      tc[0] = tile / g.ntile[1];
      tc[1] = tile - tc[0] * g.ntile[1];
    }
#pragma unroll
    for (int a = 0; a < D; ++a) {
      int j = (tc[a] * g.T[a] - dg.m0[a]) % g.L[a];
      if (j < 0) j += g.L[a];
      org[a] = j - kDepHalo;
    }
  }
  for (int i = threadIdx.x; i < W0 * W1 * wst; i += kDepThreads) sacc[i] = 0ull;
  if (threadIdx.x < C) s_scale[threadIdx.x] = dep_scale(absum[dg.ones + threadIdx.x], 0);
  if (threadIdx.x == 0) s_scale[C] = dep_scale((double)n, 1);  // pair weights: sum <= n
  __syncthreads();
  // batches of kDepThreads points: first one thread per point forms its
  // corner weights and cells (the window cell, or -1 - the global cell when
  // the stencil leaves the window), then the (point, channel) deposits and
  // the pair weights are spread over all threads, neighbours taking the
  // channels of one point, which lie side by side in its record and in the
  // window (1e6 points, 11 channels, a 1-D grid of 1024: 115 us; a channel's
  // points side by side, a record apart: 181)
  __shared__ double s_w[kDepThreads * (1 << D)];
  __shared__ int s_cell[kDepThreads * (1 << D)];
  for (int b0 = p_begin; b0 < p_end; b0 += kDepThreads) {
    const int nb = min(kDepThreads, p_end - b0);
    if (threadIdx.x < nb) {
      const int p = b0 + threadIdx.x;
      const int64_t i = rec_idx[p];
      int ix[2] = {0, 0};
      double fr[2] = {0.0, 0.0};
#pragma unroll
      for (int a = 0; a < D; ++a) {
        axis_cell(x[i * D + a], dg.x0[a], dg.dx[a], dg.G[a], &ix[a], &fr[a]);
        if (fr[a] != fr[a]) fr[a] = 0.0;  // no cell; integers hold no NaN
      }
      bool inside = true;
#pragma unroll
      for (int a = 0; a < D; ++a) {
        const int l = ix[a] - org[a];
        inside = inside && l >= 0 && l + 1 < dg.win[a];
      }
#pragma unroll
      for (int k = 0; k < NC; ++k) {
        double wk = 1.0;
        int gi = 0, li = 0;
#pragma unroll
        for (int a = 0; a < D; ++a) {
          const int bit = (k >> (D - 1 - a)) & 1;
          wk *= bit ? fr[a] : (1.0 - fr[a]);
          gi = gi * dg.G[a] + ix[a] + bit;
          li = li * dg.win[a] + ix[a] + bit - org[a];
        }
        s_w[threadIdx.x * NC + k] = wk;
        s_cell[threadIdx.x * NC + k] = inside ? li : -1 - gi;
      }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nb * (C + 1); e += kDepThreads) {
      const bool chan = e < nb * C;
      const int t = chan ? e / C : e - nb * C, c = chan ? e - t * C : C;
      const double* w = s_w + t * NC;
      const int* cell = s_cell + t * NC;
      if (chan) {
        const double vs = rec[(int64_t)(b0 + t) * stride + D + dg.ones + c] * s_scale[c];
#pragma unroll
        for (int k = 0; k < NC; ++k) {
          const long long q = __double2ll_rn(w[k] * vs);
          if (q == 0) continue;
          if (cell[k] >= 0)
            atomicAdd(&sacc[cell[k] * wst + c], (unsigned long long)q);
          else
            atomicAdd(&qacc[(int64_t)(-1 - cell[k]) * C + c], (unsigned long long)q);
        }
      } else {
        int pr = 0;
#pragma unroll
        for (int k = 0; k < NC; ++k) {
#pragma unroll
          for (int k2 = k; k2 < NC; ++k2, ++pr) {
            const long long q =
                __double2ll_rn((k == k2 ? 1.0 : 2.0) * w[k] * w[k2] * s_scale[C]);
            if (q == 0) continue;
            if (cell[0] >= 0)
              atomicAdd(&sacc[cell[0] * wst + C + pr], (unsigned long long)q);
            else
              atomicAdd(&bacc[(int64_t)(-1 - cell[0]) * NP + pr], (unsigned long long)q);
          }
        }
      }
    }
    __syncthreads();  // the next batch overwrites the point table
  }
  __syncthreads();
  // window -> global sums, one atomic per non-zero entry
  for (int e = threadIdx.x; e < W0 * W1 * wst; e += kDepThreads) {
    const unsigned long long v = sacc[e];
    if (v == 0ull) continue;
    const int cell = e / wst, j = e - cell * wst;
    const int l0 = D == 2 ? cell / W1 : cell, l1 = D == 2 ? cell - l0 * W1 : 0;
    const int g0 = org[0] + l0, g1 = org[1] + l1;
    if (g0 < 0 || g0 >= dg.G[0] || (D == 2 && (g1 < 0 || g1 >= dg.G[1]))) continue;  // stays 0
    const int64_t gc = D == 2 ? (int64_t)g0 * dg.G[1] + g1 : g0;
    if (j < C)
      atomicAdd(&qacc[gc * C + j], v);
    else
      atomicAdd(&bacc[gc * NP + (j - C)], v);
  }
}

// The 2-D deposits of windows up to kDepCells cells per axis (tiles of 8 cells
// and less).  A CTA takes one spread work item in batches of one point per
// thread, sorted by raw-grid cell in shared memory (corner weights and scaled
// channel values staged there).  A warp then takes one row of cells and up to
// 11 channels: lane (jy, c) sums, in 64-bit integer registers, corner row jy
// of channel c for the cells of the row, ten more lanes sum the corner-pair
// weights, and each sum goes to the global arrays with one atomic, the lanes
// of a cell's channels side by side.  1e6 points, 11 channels, a 512^2 grid:
// 188 us; an atomic per point, corner and channel on a shared window took
// 332 us, bound by the atomics.
constexpr int kDepCells = 11;                     // cells per axis of the window
constexpr int kDepKeys = kDepCells * kDepCells;   // the last key: outside the window
constexpr int kDepGroup = 11;                     // channels of a warp (22 lanes, 10 pairs)

inline size_t dep2_smem(int C) {
  return sizeof(double) * (size_t)kDepThreads * (4 + (C | 1));
}

__global__ void __launch_bounds__(kDepThreads, 3)
tile_deposit2_kernel(SpreadGeom g, DepositGeom dg, const double* __restrict__ x,
                     const int* __restrict__ offsets, const int* __restrict__ items,
                     const int* __restrict__ rec_idx, const double* __restrict__ rec, int stride,
                     const double* __restrict__ absum, unsigned long long* __restrict__ qacc,
                     unsigned long long* __restrict__ bacc) {
  constexpr int NP = dep_pairs(2);
  extern __shared__ __align__(16) double s_dyn[];
  __shared__ double s_scale[kDepMaxChan + 1];
  __shared__ int cnt[128], off[kDepKeys + 2];
  __shared__ unsigned char s_pos[kDepThreads];  // sorted place of each point of the batch
  __shared__ int s_gi[kDepThreads];             // raw cell (row major) of points outside
  const int C = dg.C, vstr = C | 1;
  double* s_w = s_dyn;                     // kDepThreads x 4 corner weights
  double* s_v = s_w + kDepThreads * 4;     // kDepThreads x vstr scaled values
  const int item = blockIdx.x;
  if (item >= items[g.ntiles]) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tile = item_tile(items, g.ntiles, item, lane);
  const int p_begin = offsets[tile] + (item - items[tile]) * g.item_points;
  const int p_end = min(offsets[tile + 1], p_begin + g.item_points);
  // raw-grid window of the tile: node j sits at spreading cell (m0 + j) mod L
  // (the knots are centred on the periodic grid); points whose stencil
  // leaves the window go straight to the global sums
  int org[2];
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    const int tc = a == 0 ? tile / g.ntile[1] : tile % g.ntile[1];
    int j = (tc * g.T[a] - dg.m0[a]) % g.L[a];
    if (j < 0) j += g.L[a];
    org[a] = j - kDepHalo;
  }
  if (tid < C) s_scale[tid] = dep_scale(absum[dg.ones + tid], 0);
  if (tid == kDepMaxChan) s_scale[kDepMaxChan] = dep_scale((double)dg.n, 1);
  const int ngrp = (C + kDepGroup - 1) / kDepGroup;
  for (int b0 = p_begin; b0 < p_end; b0 += kDepThreads) {
    const int nb = min(kDepThreads, p_end - b0);
    __syncthreads();  // the last batch's readers are done
    if (tid < 128) cnt[tid] = 0;
    __syncthreads();
    int key = 0, rank = 0, ix[2] = {0, 0};
    double fr[2] = {0.0, 0.0};
    if (tid < nb) {
      const int64_t i = rec_idx[b0 + tid];
      bool inside = true;
#pragma unroll
      for (int a = 0; a < 2; ++a) {
        axis_cell(x[i * 2 + a], dg.x0[a], dg.dx[a], dg.G[a], &ix[a], &fr[a]);
        if (fr[a] != fr[a]) fr[a] = 0.0;  // no cell; integers hold no NaN
        const int l = ix[a] - org[a];
        inside = inside && l >= 0 && l < kDepCells;
      }
      key = inside ? (ix[0] - org[0]) * kDepCells + ix[1] - org[1] : kDepKeys;
      rank = atomicAdd(&cnt[key], 1);
    }
    __syncthreads();
    if (warp == 0) {  // exclusive scan of the 122 counts
      int c4[4], sum = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        c4[k] = sum;
        sum += cnt[4 * lane + k];
      }
      int incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (4 * lane + k < kDepKeys + 2) off[4 * lane + k] = incl - sum + c4[k];
    }
    __syncthreads();
    if (tid < nb) {
      const int pos = off[key] + rank;
      s_pos[tid] = (unsigned char)pos;
      if (key == kDepKeys) s_gi[pos] = ix[0] * dg.G[1] + ix[1];
      double* w = s_w + 4 * pos;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        w[k] = (k & 2 ? fr[0] : 1.0 - fr[0]) * (k & 1 ? fr[1] : 1.0 - fr[1]);
    }
    __syncthreads();
    for (int e = tid; e < nb * C; e += kDepThreads) {
      const int t = e / C, c = e - t * C;
      s_v[s_pos[t] * vstr + c] = rec[(int64_t)(b0 + t) * stride + 2 + dg.ones + c] * s_scale[c];
    }
    __syncthreads();
    // warp items: (row of cells, group of channels)
    for (int wi = warp; wi < kDepCells * ngrp; wi += kDepThreads / 32) {
      const int l0 = wi / ngrp, gb = wi - l0 * ngrp;
      const int* ro = off + l0 * kDepCells;
      if (ro[0] == ro[kDepCells]) continue;
      const int c0 = gb * kDepGroup, nc = min(kDepGroup, C - c0);
      // channel lane: weights of corner row jy, value of channel c; pair lane:
      // weight k of the pair (k, k2) times weight k2, first sum only
      const bool chan = lane < 2 * nc, pair = !chan && gb == 0 && lane - 2 * nc < NP;
      const int jy = chan && lane >= nc, c = chan ? lane - jy * nc : 0;
      int k = 0, k2 = 0;
      {
        int p = pair ? lane - 2 * nc : 0;
        while (p >= 4 - k) {
          p -= 4 - k;
          ++k;
        }
        k2 = k + p;
      }
      const double pf = (k == k2 ? 1.0 : 2.0) * s_scale[kDepMaxChan];
      unsigned long long a[kDepCells + 1];
#pragma unroll
      for (int j = 0; j <= kDepCells; ++j) a[j] = 0ull;
      int pp = ro[0];
#pragma unroll
      for (int cr = 0; cr < kDepCells; ++cr) {
        const int pe = ro[cr + 1];
#pragma unroll 1
        for (; pp < pe; ++pp) {
          const double* w = s_w + 4 * pp;
          double w0, w1, v;
          if (chan) {
            const double2 u = *reinterpret_cast<const double2*>(w + 2 * jy);
            w0 = u.x;
            w1 = u.y;
            v = s_v[pp * vstr + c0 + c];
          } else {
            w0 = w[k] * w[k2];
            w1 = 0.0;
            v = pf;
          }
          a[cr] += (unsigned long long)__double2ll_rn(w0 * v);
          a[cr + 1] += (unsigned long long)__double2ll_rn(w1 * v);
        }
      }
      if (chan || pair) {
        unsigned long long* base = chan ? qacc + c0 + c : bacc + lane - 2 * nc;
        const int64_t cell0 = (int64_t)(org[0] + l0 + jy) * dg.G[1] + org[1];
        const int step = chan ? C : NP;
#pragma unroll
        for (int j = 0; j <= kDepCells; ++j)
          if (a[j] != 0ull) atomicAdd(base + (cell0 + j) * step, a[j]);
      }
    }
    // points whose stencil leaves the window
    const int po = off[kDepKeys], nout = nb - po;
    for (int e = tid; e < nout * (C + 1); e += kDepThreads) {
      const int c = e / nout, t = po + e - c * nout;
      const double* w = s_w + 4 * t;
      const int64_t gi = s_gi[t];
      if (c < C) {
        const double vs = s_v[t * vstr + c];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const long long q = __double2ll_rn(w[k] * vs);
          if (q != 0)
            atomicAdd(&qacc[(gi + (k >> 1) * dg.G[1] + (k & 1)) * C + c], (unsigned long long)q);
        }
      } else {
        int pr = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int k2 = k; k2 < 4; ++k2, ++pr) {
            const long long q = __double2ll_rn((k == k2 ? 1.0 : 2.0) * w[k] * w[k2] * s_scale[kDepMaxChan]);
            if (q != 0) atomicAdd(&bacc[gi * NP + pr], (unsigned long long)q);
          }
      }
    }
  }
}

// per-block sums of squares of every channel over a fixed range of point
// indices (the columns in their own order: the result does not depend on
// the order of the sorted records); part[b * C + c]
__global__ void __launch_bounds__(kDepThreads)
sumsq_kernel(int64_t n, int C, ChanPtrs cp, double* __restrict__ part) {
  __shared__ double red[kDepThreads / 32];
  const int c = blockIdx.y;
  const int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
  const int64_t i0 = blockIdx.x * chunk, i1 = min(n, i0 + chunk);
  const double* __restrict__ col = cp.col[c];
  double sq = 0.0;
#pragma unroll 4
  for (int64_t i = i0 + threadIdx.x; i < i1; i += kDepThreads) {
    const double v = col[i];
    sq += v * v;
  }
  for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sq;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int k = 0; k < kDepThreads / 32; ++k) t += red[k];
    part[(int64_t)blockIdx.x * C + c] = t;
  }
}

// integers -> doubles in place (Q (M, C), B (M, NP))
__global__ void deposit_finish_kernel(int64_t M, int C, int NP, const double* __restrict__ absum,
                                      int ones, int64_t n, double* __restrict__ Q,
                                      double* __restrict__ B) {
  __shared__ double inv[kDepMaxChan + 1];
  if (threadIdx.x < C) inv[threadIdx.x] = 1.0 / dep_scale(absum[ones + threadIdx.x], 0);
  if (threadIdx.x == 0) inv[C] = 1.0 / dep_scale((double)n, 1);
  __syncthreads();
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < M * C;
       i += (int64_t)gridDim.x * blockDim.x) {
    const long long v = reinterpret_cast<const long long*>(Q)[i];
    Q[i] = (double)v * inv[i % C];
  }
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < M * NP;
       i += (int64_t)gridDim.x * blockDim.x) {
    const long long v = reinterpret_cast<const long long*>(B)[i];
    B[i] = (double)v * inv[C];
  }
}

// sq[c] = sum over the items' partials, in item order (one block per channel)
__global__ void deposit_sq_kernel(int nitems, int C, const double* __restrict__ part,
                                  double* __restrict__ sq) {
  __shared__ double sh[256];
  const int c = blockIdx.x;
  double s = 0.0;
  for (int it = threadIdx.x; it < nitems; it += blockDim.x) s += part[(int64_t)it * C + c];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int k = blockDim.x / 2; k > 0; k >>= 1) {
    if (threadIdx.x < k) sh[threadIdx.x] += sh[threadIdx.x + k];
    __syncthreads();
  }
  if (threadIdx.x == 0) sq[c] = sh[0];
}

constexpr int kSumsqBlocks = 512;

static int64_t max_items_of(const SpreadGeom& g, int64_t n) {
  return (int64_t)g.ntiles + (n + g.item_points - 1) / g.item_points;
}

}  // namespace flpr

extern "C" {

size_t flpr_deposit_sorted_ws(int d, int64_t n, const int* h_L, int msp, int nchan) {
  if (d < 1 || d > 2 || n < 1 || nchan < 1) return 0;
  SpreadGeom g;
  double tau[3] = {1, 1, 1}, kmap[27] = {0};
  make_geom(g, d, h_L, msp, tau, kmap);
  return align_up(sizeof(double) * (size_t)kSumsqBlocks * (size_t)nchan);
}

int flpr_deposit_sorted(int d, int64_t n, const double* d_x, const int* h_L, int msp, int nchan,
                        int ones_channel, const double* const* h_cols,
                        const void* d_spread_ws, size_t spread_ws_bytes,
                        const double* h_ax, const int* h_G, const int* h_m0, double* d_Q,
                        double* d_B, double* d_sq, void* d_ws, size_t ws_bytes, void* stream) {
  FLPR_CHECK_ARG(d == 1 || d == 2, "deposit_sorted: d=%d (1 or 2)", d);
  FLPR_CHECK_ARG(ones_channel == 0 || ones_channel == 1, "deposit_sorted: ones_channel");
  const int C = nchan - ones_channel;
  FLPR_CHECK_ARG(n >= 1 && C >= 1 && C <= kDepMaxChan, "deposit_sorted: n=%lld C=%d",
                 (long long)n, C);
  FLPR_CHECK_ARG(d_x && h_cols && d_spread_ws && h_ax && h_G && h_m0 && d_Q && d_B && d_sq && d_ws,
                 "deposit_sorted: null pointer");
  for (int a = 0; a < d; ++a)
    FLPR_CHECK_ARG(h_G[a] >= 2 && h_L[a] >= 1, "deposit_sorted: G[%d]=%d", a, h_G[a]);
  if (spread_ws_bytes < flpr_spread_ws(d, n, h_L, msp, nchan, FLPR_PREC_F32) ||
      ws_bytes < flpr_deposit_sorted_ws(d, n, h_L, msp, nchan)) {
    set_error("deposit_sorted: workspace too small");
    return FLPR_ERR_WORKSPACE;
  }
  cudaStream_t s = as_stream(stream);
  SpreadGeom g;
  double tau[3] = {1, 1, 1}, kmap[27] = {0};
  make_geom(g, d, h_L, msp, tau, kmap);
  size_items(g, n, use_reg_path(d, h_L, msp));  // the work items the spread used
  Arena ar(const_cast<void*>(d_spread_ws), spread_ws_bytes);
  SpreadWs w;
  spread_layout(ar, d, n, g.ntiles, nchan, g.cells, &w);
  DepositGeom dg;
  memset(&dg, 0, sizeof(dg));
  int64_t M = 1;
  for (int a = 0; a < d; ++a) {
    dg.G[a] = h_G[a];
    dg.x0[a] = h_ax[2 * a];
    dg.dx[a] = h_ax[2 * a + 1];
    dg.m0[a] = h_m0[a];
    dg.win[a] = g.T[a] + 2 * kDepHalo;
    M *= h_G[a];
  }
  dg.C = C;
  dg.ones = ones_channel;
  dg.n = n;
  const int NP = dep_pairs(d);
  const int wcells = dg.win[0] * (d == 2 ? dg.win[1] : 1);
  const size_t smem = sizeof(unsigned long long) * (size_t)wcells * (size_t)(C + NP);
  FLPR_CHECK_ARG(smem <= (size_t)200 * 1024, "deposit_sorted: window does not fit shared memory");
  FLPR_CUDA(cudaMemsetAsync(d_Q, 0, sizeof(double) * (size_t)M * C, s));
  FLPR_CUDA(cudaMemsetAsync(d_B, 0, sizeof(double) * (size_t)M * NP, s));
  const int64_t nitems = max_items_of(g, n);
  double* part = static_cast<double*>(d_ws);
  ChanPtrs cp;
  memset(&cp, 0, sizeof(cp));
  for (int c = 0; c < C; ++c) cp.col[c] = h_cols[c];
  if (d == 2 && dg.win[0] <= kDepCells + 1 && dg.win[1] <= kDepCells + 1) {
    const size_t sm2 = dep2_smem(C);
    FLPR_CUDA(fit_carveout(tile_deposit2_kernel, kDepThreads, sm2));
    tile_deposit2_kernel<<<(unsigned)nitems, kDepThreads, sm2, s>>>(
        g, dg, d_x, w.offsets, w.items, w.rec_idx, w.rec, rec_stride(d, nchan), w.absum,
        reinterpret_cast<unsigned long long*>(d_Q), reinterpret_cast<unsigned long long*>(d_B));
  } else if (d == 2) {
    // wider tiles (stencils of more than 13 taps; the package's fits keep
    // records of up to 13, so only direct callers get here)
    auto k = tile_deposit_kernel<2>;
    FLPR_CUDA(raise_dyn_smem(k, smem));
    k<<<(unsigned)nitems, kDepThreads, smem, s>>>(
        g, dg, n, d_x, w.offsets, w.items, w.rec_idx, w.rec, rec_stride(d, nchan), w.absum,
        reinterpret_cast<unsigned long long*>(d_Q), reinterpret_cast<unsigned long long*>(d_B));
  } else {
    auto k = tile_deposit_kernel<1>;
    FLPR_CUDA(raise_dyn_smem(k, smem));
    k<<<(unsigned)nitems, kDepThreads, smem, s>>>(
        g, dg, n, d_x, w.offsets, w.items, w.rec_idx, w.rec, rec_stride(d, nchan), w.absum,
        reinterpret_cast<unsigned long long*>(d_Q), reinterpret_cast<unsigned long long*>(d_B));
  }
  FLPR_LAUNCH_CHECK();
  int64_t fb = (M * (C > NP ? C : NP) + 255) / 256;
  if (fb > 8 * sm_count()) fb = 8 * sm_count();
  deposit_finish_kernel<<<(int)fb, 256, 0, s>>>(M, C, NP, w.absum, ones_channel, n, d_Q, d_B);
  FLPR_LAUNCH_CHECK();
  sumsq_kernel<<<dim3(kSumsqBlocks, C), kDepThreads, 0, s>>>(n, C, cp, part);
  FLPR_LAUNCH_CHECK();
  deposit_sq_kernel<<<C, 256, 0, s>>>(kSumsqBlocks, C, part, d_sq);
  FLPR_LAUNCH_CHECK();
  return FLPR_OK;
}

}  // extern "C"
