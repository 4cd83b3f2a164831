// gd_pipeline.cu -- the exact-DBSCAN kernels.
//
// Replaces, in the reference (CUDA-DClust+):
//   host bbox + bin widths        main.cu:166-207           -> k_bbox_chunk, k_params_inst
//   INDEXING_STRUCTURE/insertData indexing.cu:54-118        -> k_keys (cell keys)
//   thrust::sort_by_key           main.cu:332               -> gdprim::radix_sort_pairs
//   INDEXING_ADJUSTMENT           indexing.cu:23-51         -> k_runs, k_cells
//   DBSCAN kernel + searchPoints  dbscan.cu:254-474         -> k_core_cell (float32 band),
//                                                              k_core_point (float64), k_core_heavy
//   MarkAsCandidate + host merge  dbscan.cu:189-222, 25-187 -> k_links, k_flood, k_union_scan,
//                                                              k_union_heavy, k_asym_resolve
//                                                              (device union-find)
//   GetDbscanResult               dbscan.cu:225-251         -> k_roots, k_label, k_border_*,
//                                                              k_scatter_labels
//
// A run clusters K >= 1 independent instances at once: every cell key carries
// the instance id above the instance's local cell key, so one radix sort, one
// cell list and one launch per phase (per dimension present) serve them all.
//
// Grid: fine cells of side f = eps * m (m > 0.5, below 1/sqrt(dim)), in blocks of
// 64 (8x8 or 4x4x4), keyed by block and place in the block.  Two points of one cell
// are always neighbours (cell diagonal below eps), and every neighbour of a point lies within +-2 cells per axis.
// A cell holding >= minpts points is therefore all core ("dense") without a
// single distance evaluation, and all core points of a cell are in one cluster.
//
// Precision modes (template flag F32):
//   F32 = false: every pair decision is the float64 predicate (gd_internal.cuh).
//   F32 = true : the pair is first measured in float32 on bbox-centred
//                coordinates; only pairs whose float32 d2 falls inside a proven
//                rounding band around eps^2 are re-tested with the float64
//                predicate.  Outside the band the float32 decision provably
//                equals the float64 one, so labels stay bit-exact.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <type_traits>

#include "gd_internal.cuh"
#include "gd_launch.h"
#include "gd_lookback.cuh"

namespace gd {

// ------------------------------------------------------------------ bbox
// Doubles ordered as int64 (monotone for non-NaN values): min/max run on the
// integer pipe instead of the much slower float64 pipe of this GPU.
__device__ __forceinline__ double dbl_of(long long o) {
  return __longlong_as_double(o >= 0 ? o : o ^ 0x7fffffffffffffffLL);
}

__global__ void k_bbox_init(const gdl::Bufs B, int K) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < K; i += gridDim.x * blockDim.x)
    for (int k = 0; k < 6; ++k) B.bbox[i * 6 + k] = k < 3 ? LLONG_MAX : LLONG_MIN;
}

constexpr int kBboxThreads = 256;

// Calls f(l, x) for every point l in [l0, l1) of an instance whose coordinates
// start at pts (row-major, D doubles per point), x holding its coordinates;
// the block's threads share the range.  With pts 16-byte aligned the points
// come in 16-byte vector loads (2D: one per point, four points in flight per
// thread; 3D: three per pair of points, l0 even), otherwise in scalar loads.
template <int D, class F>
__device__ __forceinline__ void for_points(const double* __restrict__ pts, int64_t l0, int64_t l1,
                                           F&& f) {
  const int t = threadIdx.x, NT = blockDim.x;
  if ((reinterpret_cast<uintptr_t>(pts) & 15) == 0 && (D == 2 || (l0 & 1) == 0)) {
    const double2* __restrict__ p2 = reinterpret_cast<const double2*>(pts);
    if constexpr (D == 2) {
      for (int64_t base = l0; base < l1; base += 4 * NT) {
        double2 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int64_t l = base + u * NT + t;
          if (l < l1) v[u] = __ldg(p2 + l);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int64_t l = base + u * NT + t;
          if (l < l1) {
            const double x[3] = {v[u].x, v[u].y, 0.0};
            f(l, x);
          }
        }
      }
    } else {
      const int64_t q0 = l0 >> 1, q1 = l1 >> 1;  // whole pairs: points [2 q0, 2 q1)
      for (int64_t base = q0; base < q1; base += 2 * NT) {
        double2 v[2][3];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int64_t q = base + u * NT + t;
          if (q < q1) {
            v[u][0] = __ldg(p2 + 3 * q);
            v[u][1] = __ldg(p2 + 3 * q + 1);
            v[u][2] = __ldg(p2 + 3 * q + 2);
          }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int64_t q = base + u * NT + t;
          if (q < q1) {
            const double a[3] = {v[u][0].x, v[u][0].y, v[u][1].x};
            f(2 * q, a);
            const double b[3] = {v[u][1].y, v[u][2].x, v[u][2].y};
            f(2 * q + 1, b);
          }
        }
      }
      if ((l1 & 1) && t == 0 && l1 - 1 >= l0) {  // odd last point
        const int64_t l = l1 - 1;
        const double x[3] = {pts[3 * l], pts[3 * l + 1], pts[3 * l + 2]};
        f(l, x);
      }
    }
    return;
  }
  for (int64_t l = l0 + t; l < l1; l += NT) {
    double x[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int k = 0; k < D; ++k) x[k] = pts[l * D + k];
    f(l, x);
  }
}

// Order-preserving int64 image of a double's bits (monotone for non-NaN values).
__device__ __forceinline__ long long ord_of(double v) {
  const long long bv = __double_as_longlong(v);
  return bv >= 0 ? bv : bv ^ 0x7fffffffffffffffLL;
}

// one block per chunk of one instance; one atomic per block and bound
__global__ void __launch_bounds__(kBboxThreads) k_bbox_chunk(const gdl::Bufs B) {
  const Chunk c = B.chunks[blockIdx.x];
  const InstDesc I = B.inst[c.inst];
  const int dim = I.dim;
  long long lo[3] = {LLONG_MAX, LLONG_MAX, LLONG_MAX}, hi[3] = {LLONG_MIN, LLONG_MIN, LLONG_MIN};
  bool bad = false;
  const double* __restrict__ pts = B.coords + I.co_off;
  auto take = [&](int64_t, const double* x) {
    for (int k = 0; k < 3; ++k) {
      if (k >= dim) break;
      const long long bv = __double_as_longlong(x[k]);
      bad |= (bv & 0x7ff0000000000000LL) == 0x7ff0000000000000LL;
      const long long o = ord_of(x[k]);
      lo[k] = min(lo[k], o);
      hi[k] = max(hi[k], o);
    }
  };
  if (dim == 2) for_points<2>(pts, c.begin - I.pt_off, c.end - I.pt_off, take);
  else for_points<3>(pts, c.begin - I.pt_off, c.end - I.pt_off, take);
  __shared__ long long s[6][kBboxThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo[k] = min(lo[k], __shfl_xor_sync(kFull, lo[k], o));
      hi[k] = max(hi[k], __shfl_xor_sync(kFull, hi[k], o));
    }
    if (lane == 0) { s[k][w] = lo[k]; s[3 + k][w] = hi[k]; }
  }
  if (__any_sync(kFull, bad) && lane == 0) atomicOr(&B.Bi->flags, kFlagNonFinite);
  __syncthreads();
  if (threadIdx.x < 6) {
    const int k = threadIdx.x;
    if ((k % 3) < dim) {
      long long v = s[k][0];
      for (int j = 1; j < kBboxThreads / 32; ++j) v = k < 3 ? min(v, s[k][j]) : max(v, s[k][j]);
      if (k < 3) atomicMin(B.bbox + c.inst * 6 + k, v);
      else atomicMax(B.bbox + c.inst * 6 + k, v);
    }
  }
}

// An instance's grid and float32 band from its bounding box [lo, hi] (its points'
// least and greatest coordinates; not read when it has none).
__device__ void fill_params(DevParams& p, const InstDesc& I, int inst, const double* lo,
                            const double* hi, double mult, uint64_t dense_floor,
                            uint64_t dense_per_point, uint64_t rows_floor) {
  const int D = I.dim;
  const double eps = I.eps;
  int fl = 0;
  for (int k = 0; k < 3; ++k) {
    const bool on = k < D && I.n > 0;
    p.lo[k] = on ? lo[k] : 0.0;
    p.hi[k] = on ? hi[k] : 0.0;
    p.centre[k] = on ? 0.5 * lo[k] + 0.5 * hi[k] : 0.0;
    p.G[k] = 1;
  }
  p.dim = D;
  p.minpts = I.minpts;
  p.eps = eps;
  p.eps2 = __dmul_rn(eps, eps);
  p.f = __dmul_rn(eps, mult);
  p.inv_f = 1.0 / p.f;
  p.pt_off = I.pt_off;
  p.n = I.n;
  p.co_off = I.co_off;
  p.inst = inst;
  double cells = 1.0;
  uint64_t C = 1;
  uint64_t NB = 1;
  for (int k = 0; k < 3; ++k) p.Bk[k] = 1;
  for (int k = 0; k < D; ++k) {
    double t = floor(__dmul_rn(__dsub_rn(p.hi[k], p.lo[k]), p.inv_f)) + 1.0;
    if (!(t < 2147483648.0)) { fl |= kFlagGridTooLarge; t = 1.0; }
    p.G[k] = (int64_t)t;
    cells *= t;
    C *= (uint64_t)p.G[k];
    const int sh = D == 2 ? block_shift<2>() : block_shift<3>();
    p.Bk[k] = (int32_t)((p.G[k] + (1 << sh) - 1) >> sh);
    NB *= (uint64_t)p.Bk[k];
  }
  // cell counts must fit 62 bits; keys (whole blocks) then fit 64: rounding the
  // axes up to blocks costs at most a factor of 4 near the limit (3D, one axis
  // of a single cell), and 4 * 4e18 < 2^64
  if (!(cells < 4.0e18)) {
    fl |= kFlagGridTooLarge;
    NB = 1;
  }
  // Block lookup.  Direct (one 32-byte entry per block, cleared per run) up to
  // one block per point or the floor; else a table of the block rows (8 bytes
  // each) up to kRowsPerPoint per point or the floor: a row holds few blocks, so
  // its search is short and the table stays in cache; else the hash of the
  // occupied rows.
  uint64_t limit = (uint64_t)I.n * dense_per_point;
  if (limit < dense_floor) limit = dense_floor;
  p.NB = NB;
  p.rows = NB / (uint64_t)p.Bk[D - 1];
  if (NB <= limit) {
    p.sparse = 0;
  } else {
    uint64_t rlimit = dense_per_point ? (uint64_t)I.n * kRowsPerPoint : 0;
    if (rlimit < rows_floor) rlimit = rows_floor;
    p.sparse = (fl & kFlagGridTooLarge) || p.rows > rlimit ? 1 : 2;
  }
  udiv_magic((uint64_t)p.Bk[1], p.dm[0], p.ds[0]);
  udiv_magic((uint64_t)p.Bk[2], p.dm[1], p.ds[1]);
  p.small = NB <= 0xffffffffull ? 1 : 0;
  p.dm32[0] = udiv_magic32((uint32_t)p.Bk[1]);
  p.dm32[1] = udiv_magic32((uint32_t)p.Bk[2]);
  p.key_bits = 64 - __clzll((long long)((NB << kBlockBits) - 1));
  p.cell_bits = C > 1 ? 64 - __clzll((long long)(C - 1)) : 0;
  // box-test shortcut and float32 filter need every |x| <= eps * 2^30
  double maxabs = 0, R = 0;
  for (int k = 0; k < D; ++k) {
    maxabs = fmax(maxabs, fmax(fabs(p.lo[k]), fabs(p.hi[k])));
    R = fmax(R, fmax(p.hi[k] - p.centre[k], p.centre[k] - p.lo[k]));
  }
  if (maxabs <= eps * 1073741824.0) {
    p.eps2_in = __dmul_rn(p.eps2, 1.0 - 1.0 / 524288.0);    // 1 - 2^-19
  } else {
    p.eps2_in = -1.0;
    fl |= kFlagNoShortcut;
  }
  {
    // float32 band.  a_k = fl32(x_k - c_k) is off from x_k - c_k by at most
    // ea = R 2^-24 (R bounds |x_k - c_k|).  For a pair with true squared distance
    // S, the float32 value s = fl(fl(u0^2) + ...), u_k = fl32(a_pk - a_qk), obeys
    //   |s - S| <= (S + 4 ea sqrt(D S) + 4 D ea^2)(D + 3) 2^-24
    //              + 4 ea sqrt(D S) + 4 D ea^2  =: B(S)
    // (coordinate error, one rounding per subtraction, D roundings in the FMA
    // chain).  Evaluated at S = 2 eps^2 and padded by 1.5 this is bmax.  Then
    //   s < L = eps^2 (1 - 2^-17) - bmax  =>  S < eps^2 (1 - 2^-17)
    //        =>  float64 d2 <= eps2_in  =>  neighbour both ways (box test passes);
    //   s > H = eps^2 (1 + 2^-17) + bmax  =>  float64 d2 > eps2  =>  not a neighbour.
    // L is rounded down and H up to float32.  Pairs with L <= s <= H take the
    // float64 predicate.  When the bound is not small every pair takes it.
    const double u32 = 1.0 / 16777216.0;               // 2^-24
    R = R * (1.0 + 1e-12) + 1e-300;
    // |fl32(x - c) - (x - c)| and the error of a float32 cell origin (either
    // way of computing it, see cell_origin32), with a small margin
    const double ea = R * u32 * (1.0 + 1.0 / 65536.0);
    const double e2 = p.eps2;
    const double rs = sqrt(2.0 * e2) * sqrt((double)D);
    double bmax = (2.0 * e2 + 4.0 * ea * rs + 4.0 * D * ea * ea) * (D + 3) * u32
                  + 4.0 * ea * rs + 4.0 * D * ea * ea;
    bmax *= 1.5;
    const double L = e2 * (1.0 - 1.0 / 131072.0) - bmax;   // 2^-17
    const double H = e2 * (1.0 + 1.0 / 131072.0) + bmax;
    const bool ok = !(fl & kFlagNoShortcut) && e2 > 1e-30 && R < 1e30 && L > 0.25 * e2 &&
                    H < 4.0 * e2;
    p.eps2_lo32 = ok ? __double2float_rd(L) : -1.0f;
    p.eps2_hi32 = ok ? __double2float_ru(H) : INFINITY;
    // Cell-level classification.  A point's position inside its cell,
    // u_k = (fl32(x_k - c_k) - o_k) / f with o_k the cell origin in the same
    // centred float32 frame, is within uerr of the truth (coordinate and origin
    // errors 2 ea, three float32 roundings, and the 2^-20-cell slack of the
    // float64 cell assignment of candidate points).  A stencil cell whose
    // farthest corner is within eps (1 - 2^-7) holds only neighbours (float64
    // d2 <= eps2_in, so the box test passes too); one whose nearest face is
    // beyond eps (1 + 2^-7) holds none.  Thresholds are in squared cell units.
    const double inv_m2 = (eps / p.f) * (eps / p.f);
    const double uerr = 4.0 * ea / p.f + 1.0 / 262144.0;               // + 2^-18
    const double mi = 1.0 - 1.0 / 128.0, mo = 1.0 + 1.0 / 128.0;
    p.inv_f32 = __double2float_rn(1.0 / p.f);
    p.uerr = __double2float_ru(uerr);
    p.thr_in = __double2float_rd(inv_m2 * mi * mi * (1.0 - 1.0 / 65536.0));
    p.thr_out = __double2float_ru(inv_m2 * mo * mo * (1.0 + 1.0 / 65536.0));
    p.prune = (!(fl & kFlagNoShortcut) && uerr <= 1.0 / 256.0 && R < 1e30 && e2 > 1e-30) ? 1 : 0;
  }
  {
    // float pairs for cell_origin32's float32 path: every cell index below 2^24
    // (exact in float) and magnitudes far from float under- and overflow
    bool fast = p.f >= 0x1p-60 && p.f <= 0x1p60;
    p.f_hi = __double2float_rn(p.f);
    p.f_lo = __double2float_rn(p.f - (double)p.f_hi);
    for (int k = 0; k < 3; ++k) {
      const double b = k < D ? p.lo[k] - p.centre[k] : 0.0;
      fast = fast && p.G[k] < (1 << 24) && fabs(b) <= 0x1p60;
      p.b_hi[k] = __double2float_rn(b);
      p.b_lo[k] = __double2float_rn(b - (double)p.b_hi[k]);
    }
    p.fast_origin = fast ? 1 : 0;
  }
  {
    // Float32 cell keys.  k_keys computes t64 = fl64(fl64(x - lo) * inv_f) and
    // floor(t64).  Its float32 path takes x32 = x rounded toward zero (from the
    // bits, |x32 - x| <= |x| 2^-23), lo32 = fl32(lo), i32 = fl32(inv_f) and
    // t32 = fl32(fl32(x32 - lo32) * i32).  With T = (x - lo) inv_f exact,
    //   |t32 - T| <= (|x| 2^-23 + |lo| 2^-24) inv_f (1 + 2^-22) + T (3 2^-24 + 2^-47)
    //   |t64 - T| <= T 2^-52,
    // and 0 <= T <= (hi - lo) inv_f < G + 1.  key_band is 1.25 times the sum
    // (rounded up to float): a t32 farther than that from every integer has
    // floor(t32) = floor(t64).
    double maxabs_k = 0.0, loabs = 0.0;
    for (int k = 0; k < D; ++k) {
      maxabs_k = fmax(maxabs_k, fmax(fabs(p.lo[k]), fabs(p.hi[k])));
      loabs = fmax(loabs, fabs(p.lo[k]));
    }
    double gmax = 1.0;
    for (int k = 0; k < D; ++k) gmax = fmax(gmax, (double)p.G[k]);
    const double band = 1.25 * ((maxabs_k * 0x1p-23 + loabs * 0x1p-24) * p.inv_f * (1.0 + 0x1p-22) +
                                (gmax + 1.0) * (3.0 * 0x1p-24 + 0x1p-47));
    bool kf = I.n > 0 && band < 0.125 && gmax < 0x1p21 && maxabs_k < 0x1p100 && p.inv_f < 0x1p100 &&
              maxabs_k * p.inv_f < 0x1p100;
    for (int k = 0; k < 3; ++k) p.key_lo32[k] = k < D ? __double2float_rn(p.lo[k]) : 0.0f;
    p.key_inv32 = __double2float_rn(p.inv_f);
    p.key_band = __double2float_ru(band);
    p.key_fast = kf ? 1 : 0;
  }
  p.flags = fl;
  p.ent_off = 0;
  p.row_off = 0;
  p.kmask = 0;
  p.LB = 0;
}

// One thread per instance.
__global__ void k_params_inst(const gdl::Bufs B, int K, double mult2, double mult3,
                              uint64_t dense_floor, uint64_t dense_per_point,
                              uint64_t rows_floor) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= K) return;
  const InstDesc I = B.inst[i];
  double lo[3], hi[3];
  for (int k = 0; k < 3; ++k) {
    lo[k] = dbl_of(B.bbox[i * 6 + k]);
    hi[k] = dbl_of(B.bbox[i * 6 + 3 + k]);
  }
  DevParams p;
  fill_params(p, I, i, lo, hi, I.dim == 2 ? mult2 : mult3, dense_floor, dense_per_point, rows_floor);
  B.Pv[i] = p;
}

// One block: the run layout -- key widths, cell-table offsets (exclusive scan
// over every instance's table length), flags.
__global__ void __launch_bounds__(1024) k_layout(const gdl::Bufs B, int K) {
  __shared__ unsigned long long s_part[32], s_part2[32];
  __shared__ int s_red[5][32];
  __shared__ unsigned long long s_carry, s_carry2;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int lb = 0, cb = 0, fl = 0, sp = 0, xf = 0, md = 2, k2 = 0;
  for (int i = threadIdx.x; i < K; i += blockDim.x) {
    const DevParams& p = B.Pv[i];
    if (p.n > 0) lb = max(lb, p.key_bits);
    if (p.n > 0) cb = max(cb, p.cell_bits);
    fl |= p.flags;
    sp |= p.sparse == 1;
    xf |= p.prune;
    if (p.n > 0 && !(p.eps2_lo32 > 0.0f)) xf |= 2;
    md = max(md, p.dim);
    k2 += p.dim == 2;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    lb = max(lb, __shfl_xor_sync(kFull, lb, o));
    cb = max(cb, __shfl_xor_sync(kFull, cb, o));
    fl |= __shfl_xor_sync(kFull, fl, o);
    sp |= __shfl_xor_sync(kFull, sp, o);
    xf |= __shfl_xor_sync(kFull, xf, o);
    md = max(md, __shfl_xor_sync(kFull, md, o));
    k2 += __shfl_xor_sync(kFull, k2, o);
  }
  if (lane == 0) {
    s_red[0][w] = lb;
    s_red[1][w] = fl | (sp << 16) | (xf << 17);
    s_red[2][w] = md;
    s_red[3][w] = k2;
    s_red[4][w] = cb;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int LB = 0, F = 0, MD = 2, K2 = 0, CB = 0;
    for (int j = 0; j < 32; ++j) {
      LB = max(LB, s_red[0][j]);
      F |= s_red[1][j];
      MD = max(MD, s_red[2][j]);
      K2 += s_red[3][j];
      CB = max(CB, s_red[4][j]);
    }
    int IB = 0;
    while (IB < 31 && ((K - 1) >> IB)) ++IB;
    BatchInfo bi;
    bi.K = K;
    bi.LB = LB;
    bi.IB = IB;
    bi.key64 = LB + IB > 32 ? 1 : 0;
    bi.any_sparse = (F >> 16) & 1;
    bi.any_xf = (F >> 17) & 1;
    bi.flags = (F & 0xffff) | B.Bi->flags |
               (CB + IB > 62 || LB + IB > 64 ? kFlagGridTooLarge : 0);
    bi.max_dim = MD;
    bi.K2 = K2;
    bi.band_off = (F >> 18) & 1;
    bi.ent_total = 0;
    bi.row_total = 0;
    bi.grid_cells = 0;
    *B.Bi = bi;
    s_carry = 0;
    s_carry2 = 0;
  }
  __syncthreads();
  const int LB = B.Bi->LB;
  const uint64_t kmask = LB >= 64 ? ~0ull : ((1ull << LB) - 1ull);
  // exclusive scans of the table sizes, 1024 instances at a time: block entries
  // of direct tables, rows of row tables (none for the hash).  Their totals give the grid's
  // cells too (20,000 instances: 114 us; with a shared 64-bit atomic per instance for those
  // cells 805).
  for (int base = 0; base < K; base += 1024) {
    const int i = base + threadIdx.x;
    unsigned long long vo = 0, vs = 0;
    if (i < K) {
      const DevParams& p = B.Pv[i];
      vo = p.sparse == 0 ? p.NB : 0;
      vs = p.sparse == 2 ? p.rows : 0;
    }
    unsigned long long io = vo, is = vs;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long t = __shfl_up_sync(kFull, io, o), u = __shfl_up_sync(kFull, is, o);
      if (lane >= o) {
        io += t;
        is += u;
      }
    }
    if (lane == 31) {
      s_part[w] = io;
      s_part2[w] = is;
    }
    __syncthreads();
    if (w == 0) {
      const unsigned long long t = s_part[lane], u = s_part2[lane];
      unsigned long long ti = t, ui = u;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long a = __shfl_up_sync(kFull, ti, o), c = __shfl_up_sync(kFull, ui, o);
        if (lane >= o) {
          ti += a;
          ui += c;
        }
      }
      s_part[lane] = ti - t;
      s_part2[lane] = ui - u;
    }
    __syncthreads();
    const unsigned long long eo = s_carry + s_part[w] + io - vo;
    const unsigned long long es = s_carry2 + s_part2[w] + is - vs;
    if (i < K) {
      B.Pv[i].ent_off = (uint32_t)eo;
      B.Pv[i].row_off = es;
      B.Pv[i].kmask = kmask;
      B.Pv[i].LB = LB;
    }
    __syncthreads();
    if (threadIdx.x == 1023) {
      s_carry = eo + vo;
      s_carry2 = es + vs;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    B.Bi->ent_total = s_carry;
    B.Bi->row_total = s_carry2;
    B.Bi->grid_cells = (s_carry << kBlockBits) + s_carry2;
  }
}

// ------------------------------------------------------------------ keys
// Instance id above the LB local key bits (LB = 64 only for a single instance).
__device__ __forceinline__ uint64_t inst_key(int inst, int LB) {
  return LB >= 64 ? 0 : (uint64_t)inst << LB;
}

template <class Key>
__device__ __forceinline__ int inst_of(Key key, int LB) {
  return LB >= 64 ? 0 : (int)((uint64_t)key >> LB);
}

// floor(fl64(fl64(x - lo) * inv_f)) as an int: t is finite; out-of-range
// values saturate, and the caller's clamp takes them to the grid's edge.
__device__ __forceinline__ int cell_index_f64(double x, double lo, double inv_f) {
  return __double2int_rd(__dmul_rn(__dsub_rn(x, lo), inv_f));
}

// Cell along one axis: kfast, lo32, inv32 and band as in DevParams::key_*; G1: the
// axis' last cell.
__device__ __forceinline__ int cell_of_coord(double x, bool kfast, double lo, double inv_f,
                                             float lo32, float inv32, float band, int G1) {
  // 32-bit cell index: conversions to 64-bit integers run on this GPU's
  // narrow float64 pipe; every cell index is below 2^31 (grids are checked)
  int q;
  bool fast = false;
  if (kfast) {
    // float32 cell position (no float64 instruction), used when it is
    // farther than key_band from a cell boundary.  key_fast means |x| < 2^100 and
    // positions in [-1, 2^21 + 1].
    const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
    const unsigned hw = (unsigned)(bits >> 32);
    // sign, the exponent's low 8 bits with the bias moved by 896 (a flip of the
    // highest), 23 mantissa bits; below 2^-126: 0, off by less than 2^-26 cells
    const unsigned m = (__funnelshift_l((unsigned)bits, hw, 3) ^ 0x40000000u) & 0x7fffffffu;
    const float x32 = __uint_as_float((hw & 0x80000000u) | ((hw & 0x7fffffffu) < 0x38100000u ? 0u : m));
    const float t = __fmul_rn(__fsub_rn(x32, lo32), inv32);
    // floor without a conversion instruction: for |t| < 2^22,
    // t + 1.5 * 2^23 rounded down lies in [2^23, 2^24), where floats are
    // the integers, so it is floor(t) + 1.5 * 2^23 exactly and its
    // mantissa bits hold floor(t) + 2^22
    const float s = __fadd_rd(t, 12582912.0f);
    const float fr = __fsub_rn(t, __fsub_rn(s, 12582912.0f));
    q = (int)(__float_as_uint(s) - 0x4b400000u);
    fast = fr > band && fr < 1.0f - band;
  }
  // the float64 formula for the few coordinates near a cell boundary
  if (!fast) q = cell_index_f64(x, lo, inv_f);
  return min(max(q, 0), G1);
}

// Local key from the cells along each axis.
__device__ __forceinline__ uint64_t key_of_cell(int D, const int* c, int B1, int B2) {
  return D == 2 ? ((uint64_t)(unsigned)(c[0] >> 3) * (unsigned)B1 + (unsigned)(c[1] >> 3)) << kBlockBits |
                      (unsigned)((c[0] & 7) << 3 | (c[1] & 7))
                : (((uint64_t)(unsigned)(c[0] >> 2) * (unsigned)B1 + (unsigned)(c[1] >> 2)) * (unsigned)B2 +
                   (unsigned)(c[2] >> 2)) << kBlockBits |
                      (unsigned)((c[0] & 3) << 4 | (c[1] & 3) << 2 | (c[2] & 3));
}

// One block per chunk: cell key of every point, instance id above the local key.
// Memory bound if the instructions per coordinate stay few (10M 2D / 20M 3D points: 42
// and 91 us, floors 30 and 83; with the range checks and the select over a run-time
// dimension that the host's key_fast conditions make needless, 71 and 140 us).
template <class Key>
__global__ void __launch_bounds__(256) k_keys(const gdl::Bufs B, Key* __restrict__ keys) {
  const Chunk c = B.chunks[blockIdx.x];
  const DevParams& P = B.Pv[c.inst];
  const double inv_f = P.inv_f;
  double lo[3];
  int G1[3];
  float lo32[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    lo[k] = P.lo[k];
    G1[k] = (int)(P.G[k] - 1);
    lo32[k] = P.key_lo32[k];
  }
  const uint64_t hi = inst_key(P.inst, P.LB);
  const int B1 = P.Bk[1], B2 = P.Bk[2];
  const bool kfast = P.key_fast != 0;
  const float band = P.key_band, inv32 = P.key_inv32;
  const double* __restrict__ pts = B.coords + P.co_off;
  Key* __restrict__ out = keys + P.pt_off;
  auto points = [&](auto dim) {
    constexpr int D = decltype(dim)::value;
    for_points<D>(pts, c.begin - P.pt_off, c.end - P.pt_off, [&](int64_t l, const double* xs) {
      int q[3] = {0, 0, 0};
#pragma unroll
      for (int k = 0; k < D; ++k)
        q[k] = cell_of_coord(xs[k], kfast, lo[k], inv_f, lo32[k], inv32, band, G1[k]);
      out[l] = (Key)(hi + key_of_cell(D, q, B1, B2));
    });
  };
  if (P.dim == 2) points(std::integral_constant<int, 2>{});
  else points(std::integral_constant<int, 3>{});
}

// Coordinates of one point in 16-byte loads where the address allows (a 2D
// point at a 16-byte boundary is one load; a 3D point is a 16-byte and an
// 8-byte load, in the order its alignment allows).
template <int D>
__device__ __forceinline__ void load_coords(const double* __restrict__ src, double* v) {
  const bool a16 = (reinterpret_cast<uintptr_t>(src) & 15) == 0;
  if (D == 2) {
    if (a16) {
      const double2 t = __ldg(reinterpret_cast<const double2*>(src));
      v[0] = t.x;
      v[1] = t.y;
    } else {
      v[0] = __ldg(src);
      v[1] = __ldg(src + 1);
    }
  } else {
    if (a16) {
      const double2 t = __ldg(reinterpret_cast<const double2*>(src));
      v[0] = t.x;
      v[1] = t.y;
      v[2] = __ldg(src + 2);
    } else {
      v[0] = __ldg(src);
      const double2 t = __ldg(reinterpret_cast<const double2*>(src + 1));
      v[1] = t.x;
      v[2] = t.y;
    }
  }
}

// Sorted copies: float64 points (16 or 24 bytes each) and centred float32 ones (8 or 16
// bytes).  The float64 ones are written in every mode: the points are the caller's, who may
// change or free them once the first expand has returned, and later expands of the index
// re-test the float32 band's pairs (20M 3D points in that mode: 110 us of 4.9 ms).  2D positions come first in a mixed run,
// so each point lies at its position times its own size.  ONE: a single
// instance (its parameters are Pv[0], no key is read).  kGatherU points per
// thread and pass, so that as many random loads are in flight.
#ifndef GD_GATHER_U
#define GD_GATHER_U 4
#endif
constexpr int kGatherU = GD_GATHER_U;
template <class Key, bool XF, bool ONE>
__global__ void k_gather(const gdl::Bufs B, int64_t n) {
  const int LB = B.Bi->LB;
  const Key* __restrict__ keys = static_cast<const Key*>(B.keys);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i0 < n; i0 += kGatherU * stride) {
    double v[kGatherU][3];
    const DevParams* Pp[kGatherU];
#pragma unroll
    for (int u = 0; u < kGatherU; ++u) {
      const int64_t i = i0 + u * stride;
      Pp[u] = nullptr;
      if (i < n) {
        const int64_t g = B.ids[i];
        const DevParams& P = B.Pv[ONE ? 0 : inst_of(keys[i], LB)];
        Pp[u] = &P;
        const double* src = B.coords + P.co_off + (g - P.pt_off) * P.dim;
        if (P.dim == 2) load_coords<2>(src, v[u]);
        else load_coords<3>(src, v[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < kGatherU; ++u) {
      const int64_t i = i0 + u * stride;
      if (i >= n) continue;
      const DevParams& P = *Pp[u];
      const int D = P.dim;
      if (D == 2) {
        reinterpret_cast<double2*>(B.X)[i] = make_double2(v[u][0], v[u][1]);
      } else {
#pragma unroll
        for (int k = 0; k < 3; ++k) B.X[3 * i + k] = v[u][k];
      }
      if (XF) {
        const float f0 = __double2float_rn(__dsub_rn(v[u][0], P.centre[0]));
        const float f1 = __double2float_rn(__dsub_rn(v[u][1], P.centre[1]));
        if (D == 2) {
          reinterpret_cast<float2*>(B.Xf)[i] = make_float2(f0, f1);
        } else {
          const float f2 = __double2float_rn(__dsub_rn(v[u][2], P.centre[2]));
          reinterpret_cast<float4*>(B.Xf)[i] = make_float4(f0, f1, f2, 0.0f);
        }
      }
    }
  }
}

// ---------------------------------------------------------------- bit masks
// Number of set bits of a mask below position i (0 <= i <= its length): the
// word prefix count plus the set bits of i's word below it.
__device__ __forceinline__ uint32_t bit_rank(const uint32_t* __restrict__ bits,
                                             const uint32_t* __restrict__ pre, int64_t i) {
  const int64_t w = i >> 5;
  return pre[w] + (uint32_t)__popc(bits[w] & ((1u << (i & 31)) - 1u));
}

// Cell index m of sorted position i: the cell starts at or before i, less one.
__device__ __forceinline__ int cell_of(const gdl::Bufs& B, int64_t i) {
  const int64_t w = i >> 5;
  return (int)(B.runpre[w] + (uint32_t)__popc(B.runbits[w] & (0xffffffffu >> (31 - (i & 31))))) -
         1;
}

// Cells, in one pass over the sorted keys: a bit per position that starts a cell
// (its key differs from the one before) with per-word prefix counts, and every
// cell's first position (reps) and key (ckeys).  A tile is 8192 positions (16 warps
// of 16 words): counts are scanned in the block, the tile's prefix comes by look-back
// while the keys wait in registers.  The last tile closes reps and counts the cells;
// in runs of 2D and 3D instances the first cell of a 3D instance marks the border.
// (Bits, scan, list and closing had been four launches reading the keys twice: C2
// 22 + 6 + 36 + 4 us.)
constexpr int kRunThreads = 512, kRunWords = 16, kRunTile = kRunThreads * kRunWords;
template <class Key>
__global__ void __launch_bounds__(kRunThreads)
k_runs(const gdl::Bufs B, int64_t n, Key* __restrict__ ckeys, unsigned tiles,
       gdprim::LookbackCtl* ctl, unsigned long long* status) {
  __shared__ uint32_t s_warp[32];
  __shared__ unsigned s_tile, s_epoch;
  __shared__ uint32_t s_agg, s_excl;
  const Key* __restrict__ keys = static_cast<const Key*>(B.keys);
  unsigned long long* timeouts = B.ctr + kCtrWaitTimeouts;
  gdprim::lb_begin(ctl, &s_tile, &s_epoch);
  const unsigned tile = s_tile, epoch = s_epoch;
  if (tile >= tiles) {
    // a counter left inconsistent (never expected): no tile, report it
    if (threadIdx.x == 0) atomicAdd(timeouts, 1ull);
    gdprim::lb_end(ctl, tiles, epoch);
    return;
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t seg = (int64_t)tile * kRunTile + (int64_t)w * 32 * kRunWords;
  Key k[kRunWords];
#pragma unroll
  for (int u = 0; u < kRunWords; ++u) {
    const int64_t i = seg + u * 32 + lane;
    k[u] = i < n ? keys[i] : (Key)0;
  }
  // the key before the segment, then each word's last key
  Key last = seg > 0 && seg < n ? keys[seg - 1] : (Key)0;
  unsigned bits[kRunWords], cnt = 0;
#pragma unroll
  for (int u = 0; u < kRunWords; ++u) {
    const int64_t i = seg + u * 32 + lane;
    Key prev = __shfl_up_sync(kFull, k[u], 1);
    if (lane == 0) prev = last;
    last = __shfl_sync(kFull, k[u], 31);
    bits[u] = __ballot_sync(kFull, i < n && (i == 0 || k[u] != prev));
    cnt += (unsigned)__popc(bits[u]);
  }
  // warp totals scanned in the block (one thread per warp carries the total)
  const uint32_t ex = gdprim::block_excl_scan<kRunThreads>(lane == 0 ? cnt : 0u, s_warp, &s_agg);
  const uint32_t excl =
      gdprim::lb_tile_prefix(status, tile, gdprim::lb_tag(epoch), &s_agg, &s_excl, timeouts);
  uint32_t m = excl + __shfl_sync(kFull, ex, 0);
  const int K2 = B.Bi->K2, LB = B.Bi->LB;
  const bool mixed = K2 > 0 && K2 < B.Bi->K;
#pragma unroll
  for (int u = 0; u < kRunWords; ++u) {
    const int64_t i0 = seg + u * 32, i = i0 + lane;
    if (i0 >= n) break;  // warp-uniform
    if (lane == 0) {
      B.runbits[i0 >> 5] = bits[u];
      B.runpre[i0 >> 5] = m;
    }
    if ((bits[u] >> lane) & 1u) {
      const uint32_t c = m + (uint32_t)__popc(bits[u] & ((1u << lane) - 1u));
      B.reps[c] = (int)i;
      ckeys[c] = k[u];
      if (mixed && inst_of(k[u], LB) >= K2 && (i == 0 || inst_of(keys[i - 1], LB) < K2))
        B.ctr[kCtrCells2D] = c;
    }
    m += (uint32_t)__popc(bits[u]);
  }
  if (tile == tiles - 1u && threadIdx.x == 0) {
    const uint32_t M = excl + s_agg;
    *B.M = M;
    B.reps[M] = (int)n;
    B.ctr[kCtrCells] = M;
    if (K2 == 0) B.ctr[kCtrCells2D] = 0;
    else if (!mixed || inst_of(keys[n - 1], LB) < K2) B.ctr[kCtrCells2D] = M;
  }
  gdprim::lb_end(ctl, tiles, epoch);
}

// Block entries and row lookups, a lane per cell.  A block's cells are
// consecutive in key order, mostly within one warp: the run of lanes of one block
// forms its occupancy word together; where the block of the last lane goes past the
// warp's end the warp reads on (at most 63 cells), and the lane of the block's first
// cell writes the entry (core word and roots empty).  Every cell notes
// where its block's entry is.  The first and last cell of a block row write the
// row's cell range (row table or hash slot).  (Entries lie at first cells where some
// instance has no direct table; a warp that starts inside a block finds that cell by two
// reads together.  Each lane stepping back key by key: 4096 instances 2.25 ms, now 1.88.)
template <class Key>
__global__ void __launch_bounds__(256) k_cells(const gdl::Bufs B) {
  const Key* __restrict__ ckeys = static_cast<const Key*>(B.ckeys);
  const int LB = B.Bi->LB;
  const int64_t M = *B.M;
  const int lane = threadIdx.x & 31;
  for (int64_t m0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); m0 < M;
       m0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = m0 + lane;
    const uint64_t key = (uint64_t)ckeys[m < M ? m : M - 1];
    const uint64_t blk = key >> kBlockBits;  // with the instance id
    uint64_t pb = __shfl_up_sync(kFull, blk, 1);
    if (lane == 0) pb = m > 0 ? (uint64_t)ckeys[m - 1] >> kBlockBits : ~0ull;
    const bool first = m < M && (m == 0 || pb != blk);
    const unsigned firsts = __ballot_sync(kFull, first);
    // this lane's run: lanes [rs, re) hold cells of its block
    const unsigned heads = firsts | 1u;
    const unsigned upto = (unsigned)((2ull << lane) - 1ull);
    const int rs = 31 - __clz(heads & upto);
    const unsigned after = heads & ~upto;
    const int nv = M - m0 < 32 ? (int)(M - m0) : 32;
    const int re = after ? __ffs(after) - 1 : nv;
    // the run's occupancy word, its cells of two points and more, of three and more,
    // gathered at its first lane: a segmented OR over the lanes that follow
    const int len = B.pop && m < M ? B.reps[m + 1] - B.reps[m] : 1;
    const uint32_t b = 1u << (key & 31);
    const bool up = (key & 32) != 0;
    uint32_t lo = up ? 0u : b, hi = up ? b : 0u;
    BlockPop pop;
    pop.two[0] = len > 1 ? lo : 0u;
    pop.two[1] = len > 1 ? hi : 0u;
    pop.three[0] = len > 2 ? lo : 0u;
    pop.three[1] = len > 2 ? hi : 0u;
    auto gather = [&](uint32_t& x) {
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_down_sync(kFull, x, o);
        if (lane + o < re) x |= y;
      }
    };
    gather(lo);
    gather(hi);
    if (B.pop) {
      gather(pop.two[0]);
      gather(pop.two[1]);
      gather(pop.three[0]);
      gather(pop.three[1]);
    }
    // the block of the warp's last lane goes on past it: the warp reads on together
    const int rl = 31 - __clz(heads);
    if (m0 + 32 < M && ((firsts >> rl) & 1u)) {
      const uint64_t bl = __shfl_sync(kFull, blk, 31);
      for (int64_t c0 = m0 + 32;; c0 += 32) {
        const int64_t c = c0 + lane;
        const uint64_t k = c < M ? (uint64_t)ckeys[c] : 0;
        const bool same = c < M && k >> kBlockBits == bl;
        if (!__any_sync(kFull, same)) break;
        const uint32_t cb = same ? 1u << (k & 31) : 0u;
        const bool cu = (k & 32) != 0;
        const int cl = B.pop && same ? B.reps[c + 1] - B.reps[c] : 1;
        const uint32_t l0 = cu ? 0u : cb, h0 = cu ? cb : 0u;
        const uint32_t a0 = __reduce_or_sync(kFull, l0), a1 = __reduce_or_sync(kFull, h0);
        if (lane == rl) {
          lo |= a0;
          hi |= a1;
        }
        if (B.pop) {
          const uint32_t t0 = __reduce_or_sync(kFull, cl > 1 ? l0 : 0u);
          const uint32_t t1 = __reduce_or_sync(kFull, cl > 1 ? h0 : 0u);
          const uint32_t u0 = __reduce_or_sync(kFull, cl > 2 ? l0 : 0u);
          const uint32_t u1 = __reduce_or_sync(kFull, cl > 2 ? h0 : 0u);
          if (lane == rl) {
            pop.two[0] |= t0;
            pop.two[1] |= t1;
            pop.three[0] |= u0;
            pop.three[1] |= u1;
          }
        }
        if (!__all_sync(kFull, same)) break;
      }
    }
    // the first cell of the block of the warp's first lane, where it lies before the
    // warp (at most 63 cells back); only entries at first cells ask for it
    int64_t f0 = m0;
    if (B.nbr && !(firsts & 1u)) {
      const uint64_t b0 = __shfl_sync(kFull, blk, 0);
      for (int r = 0; r < 2; ++r) {
        const int64_t c = f0 - 1 - lane;
        const bool same = c >= 0 && (uint64_t)ckeys[c] >> kBlockBits == b0;
        const unsigned other = ~__ballot_sync(kFull, same);
        f0 -= other ? __ffs(other) - 1 : 32;
        if (other) break;
      }
    }
    if (m >= M) continue;
    const DevParams& P = B.Pv[inst_of(key, LB)];
    const uint64_t lblk = (key & P.kmask) >> kBlockBits;
    const int mode = P.sparse;
    uint32_t e = P.ent_off + (uint32_t)lblk;
    // (the block's first cell: the run's first lane, or before the warp)
    if (mode != 0) e = B.ent_base + (uint32_t)(rs == 0 ? f0 : m0 + rs);
    B.cellent[m] = e;
    if (first) {
      BlockEnt E;
      E.occ = (unsigned long long)hi << 32 | lo;
      E.base = (uint32_t)m;
      E.lo = kNoEnt;
      E.core = 0;
      E.hi = kNoEnt;
      E.uni = kNoEnt;
      B.ent[e] = E;
      if (B.pop) B.pop[e] = pop;
    }
    if (mode == 0) continue;
    // the row's first key and the first key past it (no key of the run lies
    // between a row's last one and the latter)
    const int a = P.dim - 2;
    const uint64_t Bz = (uint64_t)P.Bk[P.dim - 1];
    const uint64_t row = udiv_by(lblk, P.dm[a], P.ds[a]);
    const uint64_t k0 = inst_key(P.inst, LB) + ((row * Bz) << kBlockBits);
    const uint64_t k1 = k0 + (Bz << kBlockBits) - 1;  // the row's last possible key
    const bool rfirst = m == 0 || (uint64_t)ckeys[m - 1] < k0;
    const bool rlast = m == M - 1 || (uint64_t)ckeys[m + 1] > k1;
    if (!rfirst && !rlast) continue;
    uint2* slot = nullptr;
    if (mode == 2) {
      slot = B.rowtab + P.row_off + row;
    } else {
      const uint32_t mask = B.hmask;
      uint32_t h = hash_key(k0) & mask;
      for (uint32_t probe = 0; probe <= mask; ++probe) {
        const unsigned long long prev = atomicCAS(B.hkeys + h, kHashEmpty, (unsigned long long)k0);
        if (prev == kHashEmpty || prev == k0) {
          slot = B.hvals + h;
          break;
        }
        h = (h + 1) & mask;
      }
    }
    if (slot) {
      if (rfirst) slot->x = (uint32_t)m;
      if (rlast) slot->y = (uint32_t)(m + 1);
    }
  }
}

// ------------------------------------------------------------- cell helpers
template <int D>
struct CellXYZ {
  int c[3];  // per-axis cell indices (each below 2^31)
};

template <int D>
__device__ __forceinline__ CellXYZ<D> decompose(uint64_t key, const DevParams& P) {
  constexpr int S = block_shift<D>(), SM = (1 << S) - 1;
  CellXYZ<D> r;
  const unsigned in = (unsigned)key & 63u;
  uint64_t k = key >> kBlockBits;
  if (P.small) {
    // fewer than 2^32 blocks: the same division on 32 bits
    unsigned q = (unsigned)k;
    if (D == 3) {
      const unsigned k2 = udiv_by32(q, P.dm32[1], P.ds[1]);
      r.c[2] = (int)((q - k2 * (unsigned)P.Bk[2]) << S | (in & SM));
      q = k2;
    } else {
      r.c[2] = 0;
    }
    const unsigned k1 = udiv_by32(q, P.dm32[0], P.ds[0]);
    r.c[1] = (int)((q - k1 * (unsigned)P.Bk[1]) << S | (D == 3 ? (in >> S) & SM : in & SM));
    r.c[0] = (int)(k1 << S | in >> (D == 3 ? 2 * S : S));
    return r;
  }
  if (D == 3) {
    const uint64_t k2 = udiv_by(k, P.dm[1], P.ds[1]);
    r.c[2] = (int)((unsigned)(k - k2 * (uint64_t)(unsigned)P.Bk[2]) << S | (in & SM));
    k = k2;
  } else {
    r.c[2] = 0;
  }
  const uint64_t k1 = udiv_by(k, P.dm[0], P.ds[0]);
  r.c[1] = (int)((unsigned)(k - k1 * (uint64_t)(unsigned)P.Bk[1]) << S |
                 (D == 3 ? (in >> S) & SM : in & SM));
  r.c[0] = (int)((unsigned)k1 << S | in >> (D == 3 ? 2 * S : S));
  return r;
}

// Coordinates of sorted position i: float64 copy, centred float32 copy.
template <int D>
__device__ __forceinline__ void ld_x(const gdl::Bufs& B, int64_t i, double* v) {
  if (D == 2) {
    const double2 t = reinterpret_cast<const double2*>(B.X)[i];
    v[0] = t.x;
    v[1] = t.y;
  } else {
#pragma unroll
    for (int k = 0; k < D; ++k) v[k] = B.X[3 * i + k];
  }
}
template <int D>
__device__ __forceinline__ void ld_f(const gdl::Bufs& B, int64_t i, float* v) {
  if (D == 2) {
    const float2 t = reinterpret_cast<const float2*>(B.Xf)[i];
    v[0] = t.x;
    v[1] = t.y;
  } else {
    const float4 t = reinterpret_cast<const float4*>(B.Xf)[i];
    v[0] = t.x;
    v[1] = t.y;
    v[D - 1] = t.z;
  }
}
// One candidate (sorted position q) in the layout the mode tests with.
template <int D, bool F32>
struct Cand {
  double x[D];
  float f[D];
};

template <int D, bool F32>
__device__ __forceinline__ void load_cand(Cand<D, F32>& c, const gdl::Bufs& B, int64_t q) {
  if (F32) ld_f<D>(B, q, c.f);
  else ld_x<D>(B, q, c.x);
}

// Per-warp staging of up to 32 "A" points (the points of the cell in work).
template <int D>
struct WarpStage {
  double x[32][D];
  float f[32][D];
};

struct Tally {
  uint32_t t64 = 0, t32 = 0, band = 0, asym = 0;
};

// float32 distance (centred copies); FMA-rounded as the band derivation assumes
template <int D>
__device__ __forceinline__ float dist2_f32(const float* a, const float* b) {
  float u = __fsub_rn(a[0], b[0]);
  float s = __fmul_rn(u, u);
  float v = __fsub_rn(a[1], b[1]);
  s = __fmaf_rn(v, v, s);
  if (D == 3) {
    float w = __fsub_rn(a[2], b[2]);
    s = __fmaf_rn(w, w, s);
  }
  return s;
}

// Directed test "cand is a neighbour of centre".  One side is a staged point
// (sorted position si; float64 coordinates sx in float64 mode), the other a
// candidate (sorted position q; coordinates in registers).  stage_is_centre
// selects which is the centre of the query box.  In float32-band mode the
// float64 coordinates of both are loaded only for a band re-test.
template <int D, bool F32, class PP>
__device__ __forceinline__ bool pair_test(const double* sx, const float* sf, const Cand<D, F32>& c,
                                          const gdl::Bufs& B, int64_t q, int64_t si,
                                          bool stage_is_centre, const PP& P, Tally& t) {
  if (F32) {
    ++t.t32;
    float s = dist2_f32<D>(sf, c.f);
    if (s < P.eps2_lo32) return true;
    if (s > P.eps2_hi32) return false;
    ++t.band;
    double qx[D], px[D];
    ld_x<D>(B, q, qx);
    ld_x<D>(B, si, px);
    ++t.t64;
    double d2 = dist2_f64<D>(px, qx);
    return stage_is_centre ? pred_from_d2<D>(d2, px, qx, P) : pred_from_d2<D>(d2, qx, px, P);
  } else {
    ++t.t64;
    double d2 = dist2_f64<D>(sx, c.x);
    return stage_is_centre ? pred_from_d2<D>(d2, sx, c.x, P) : pred_from_d2<D>(d2, c.x, sx, P);
  }
}

// Symmetric test for core-core links: true when the pair is a neighbour in both
// directions; counts pairs that are neighbours in exactly one direction.
template <int D, bool F32, class PP>
__device__ __forceinline__ bool link_test(const double* sx, const float* sf, const Cand<D, F32>& c,
                                          const gdl::Bufs& B, int a, int q, const PP& P,
                                          Tally& t) {
  double qx[D], ax[D];
  if (F32) {
    ++t.t32;
    float s = dist2_f32<D>(sf, c.f);
    if (s < P.eps2_lo32) return true;
    if (s > P.eps2_hi32) return false;
    ++t.band;
    // float64 coordinates of both, for the band re-test only
    ld_x<D>(B, q, qx);
    ld_x<D>(B, a, ax);
  } else {
#pragma unroll
    for (int k = 0; k < D; ++k) {
      qx[k] = c.x[k];
      ax[k] = sx[k];
    }
  }
  sx = ax;
  ++t.t64;
  double d2 = dist2_f64<D>(sx, qx);
  if (d2_le(d2, P.eps2_in)) return true;
  if (!d2_le(d2, P.eps2)) return false;
  bool f = box_f64<D>(sx, qx, P.eps), b = box_f64<D>(qx, sx, P.eps);
  if (f != b) {
    // q is a neighbour of a but not a of q (f), or the reverse: a directed
    // link that the merge replay (k_asym_resolve) needs.
    ++t.asym;
    unsigned long long slot = atomicAdd(B.ctr + kCtrAsymEdges, 1ull);
    if (slot < (unsigned long long)kAsymCap) {
      B.asym[2 * slot] = f ? a : q;
      B.asym[2 * slot + 1] = f ? q : a;
    }
  }
  return f && b;
}

__device__ __forceinline__ void flush_tally(const Tally& t, unsigned long long* ctr) {
  // one atomic per warp per counter
  unsigned long long a = t.t64, b = t.t32, c = t.band, d = t.asym;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(kFull, a, o);
    b += __shfl_xor_sync(kFull, b, o);
    c += __shfl_xor_sync(kFull, c, o);
    d += __shfl_xor_sync(kFull, d, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (a) atomicAdd(ctr + kCtrTests64, a);
    if (b) atomicAdd(ctr + kCtrTests32, b);
    if (c) atomicAdd(ctr + kCtrBand, c);
    if (d) atomicAdd(ctr + kCtrAsym, d);
  }
}

// The lanes sharing this lane's value v, for values that sit in runs of
// consecutive lanes (lanes holding sorted points: a cell's points are
// neighbours).  act: the lanes taking part; the result is the run of
// consecutive active lanes with v that holds this lane (0 for an inactive
// lane).  Equal values split by an inactive lane give two runs.  All 32 lanes
// call it.  (__match_any_sync gives the same sets for such values, at a
// higher cost.)
__device__ __forceinline__ unsigned run_peers(unsigned act, int v) {
  const int lane = threadIdx.x & 31;
  const int prev = __shfl_up_sync(kFull, v, 1);
  const bool on = (act >> lane) & 1u;
  const bool prev_on = ((act << 1) >> lane) & 1u;             // lane - 1 active (0 for lane 0)
  const bool head = on && (!prev_on || prev != v);
  const unsigned heads = __ballot_sync(kFull, head);
  if (!on) return 0u;
  const unsigned upto = (unsigned)((2ull << lane) - 1ull);   // lanes 0..lane
  const int s = 31 - __clz(heads & upto);                     // this run's head
  const unsigned stop = (heads | ~act) & ~upto;               // next head or gap
  const int e = stop ? __ffs(stop) - 1 : 32;
  return (unsigned)(((1ull << e) - 1ull) & ~((1ull << s) - 1ull));
}

template <bool KEY64>
__device__ __forceinline__ uint64_t key_at(const gdl::Bufs& B, int64_t i) {
  if (KEY64) return static_cast<const unsigned long long*>(B.keys)[i];
  return static_cast<const uint32_t*>(B.keys)[i];
}

// key of cell m (instance id and local key)
template <bool KEY64>
__device__ __forceinline__ uint64_t ckey_at(const gdl::Bufs& B, int64_t m) {
  if (KEY64) return static_cast<const unsigned long long*>(B.ckeys)[m];
  return static_cast<const uint32_t*>(B.ckeys)[m];
}

// The cell a kernel thread/warp works on: instance parameters and local key.
struct CellCtx {
  const DevParams* P;
  uint64_t local;
};

template <bool KEY64>
__device__ __forceinline__ CellCtx cell_ctx(const gdl::Bufs& B, int64_t m, int LB) {
  const uint64_t key = ckey_at<KEY64>(B, m);
  CellCtx c;
  c.P = B.Pv + (KEY64 ? inst_of(key, LB) : (int)(key >> LB));
  c.local = key & c.P->kmask;
  return c;
}

// ------------------------------------------------------------ block lookups
// Entries of blocks z0 and z0 + 1 (last axis; z0 >= -1) of block row `row`,
// kNoEnt when unwanted, outside the grid or (row table, hash) not occupied.
// Direct tables: one address computation, no load.  Row tables and the hash:
// the row's cell range, then a binary search over its cells' keys for the
// first cell of the first wanted block; the next block follows its cells.
template <int D, bool KEY64>
__device__ __forceinline__ void find_pair(const gdl::Bufs& B, const DevParams& P, uint64_t row,
                                           int z0, bool want0, bool want1, uint32_t& e0,
                                           uint32_t& e1) {
  e0 = kNoEnt;
  e1 = kNoEnt;
  const int Bz = P.Bk[D - 1];
  want0 = want0 && z0 >= 0;
  want1 = want1 && z0 + 1 < Bz;
  if (P.sparse == 0) {
    const uint32_t e = P.ent_off + (uint32_t)row * (uint32_t)Bz + (uint32_t)z0;
    if (want0) e0 = e;
    if (want1) e1 = e + 1;
    return;
  }
  if (!want0 && !want1) return;
  const uint64_t k0 = inst_key(P.inst, P.LB) + ((row * (uint64_t)Bz) << kBlockBits);
  uint2 rc = make_uint2(0, 0);
  if (P.sparse == 2) {
    rc = B.rowtab[P.row_off + row];
  } else {
    const uint32_t hmask = B.hmask;
    uint32_t h = hash_key(k0) & hmask;
    for (uint32_t probe = 0; probe <= hmask; ++probe) {
      const unsigned long long kk = B.hkeys[h];
      if (kk == k0) {
        rc = B.hvals[h];
        break;
      }
      if (kk == kHashEmpty) break;
      h = (h + 1) & hmask;
    }
  }
  const uint64_t kf = k0 + ((uint64_t)(want0 ? z0 : z0 + 1) << kBlockBits);
  uint32_t a = rc.x, b = rc.y;
  while (a < b) {
    const uint32_t mid = (a + b) >> 1;
    if (ckey_at<KEY64>(B, mid) < kf) a = mid + 1;
    else b = mid;
  }
  if (a >= rc.y) return;
  const uint64_t zb = (ckey_at<KEY64>(B, a) - k0) >> kBlockBits;
  if (want0 && zb == (uint64_t)z0) {
    e0 = B.ent_base + a;
    if (!want1) return;
    a += (uint32_t)__popcll(B.ent[e0].occ);
    if (a < rc.y && (ckey_at<KEY64>(B, a) - k0) >> kBlockBits == (uint64_t)(z0 + 1))
      e1 = B.ent_base + a;
  } else if (want1 && zb == (uint64_t)(z0 + 1)) {
    e1 = B.ent_base + a;
  }
}

// The same for row r of the stencil of cell m (its block row is `row`).  Direct
// tables: computed; otherwise read from the cell's neighbour entries (k_neighbors).
template <int D>
__device__ __forceinline__ void block_pair(const gdl::Bufs& B, const DevParams& P, int64_t m, int r,
                                           uint64_t row, int z0, bool want0, bool want1,
                                           uint32_t& e0, uint32_t& e1) {
  e0 = kNoEnt;
  e1 = kNoEnt;
  if (P.sparse == 0) {
    const int Bz = P.Bk[D - 1];
    const uint32_t e = P.ent_off + (uint32_t)row * (uint32_t)Bz + (uint32_t)z0;
    if (want0 && z0 >= 0) e0 = e;
    if (want1 && z0 + 1 < Bz) e1 = e + 1;
    return;
  }
  const uint2 v = B.nbr[4 * m + r];
  if (want0) e0 = v.x;
  if (want1) e1 = v.y;
}

// The first 16 bytes of an entry (occupied cells, first cell, lo); an empty
// one for kNoEnt.
struct EntHead {
  unsigned long long occ;
  uint32_t base, lo;
};
__device__ __forceinline__ EntHead ent_head(const gdl::Bufs& B, uint32_t e) {
  EntHead h{0, 0, 0};
  if (e != kNoEnt) {
    const uint4 v = *reinterpret_cast<const uint4*>(B.ent + e);
    h.occ = (unsigned long long)v.y << 32 | v.x;
    h.base = v.z;
    h.lo = v.w;
  }
  return h;
}
// its other half: core cells, hi
struct EntTail {
  unsigned long long core;
  uint32_t hi, uni;
};
__device__ __forceinline__ EntTail ent_tail(const gdl::Bufs& B, uint32_t e) {
  EntTail h{0, 0, 0};
  if (e != kNoEnt) {
    const uint4 v = *(reinterpret_cast<const uint4*>(B.ent + e) + 1);
    h.core = (unsigned long long)v.y << 32 | v.x;
    h.hi = v.z;
    h.uni = v.w;
  }
  return h;
}

// index of the occupied cell at `bit` of a block
__device__ __forceinline__ int ent_cell(unsigned long long occ, uint32_t base, int bit) {
  return (int)(base + (uint32_t)__popcll(occ & ((1ull << bit) - 1ull)));
}

// Cell (x, y, z): its index, or -1 when outside the grid or empty (the warp
// kernels' lookup, one cell per lane).
template <int D, bool KEY64>
__device__ __forceinline__ int find_cell(const gdl::Bufs& B, const DevParams& P, int64_t x,
                                         int64_t y, int64_t z) {
  constexpr int S = block_shift<D>(), SM = (1 << S) - 1;
  if (x < 0 || x >= P.G[0] || y < 0 || y >= P.G[1]) return -1;
  if (D == 3 && (z < 0 || z >= P.G[2])) return -1;
  const int64_t last = D == 3 ? z : y;
  const uint64_t row = D == 3 ? (uint64_t)(x >> S) * (unsigned)P.Bk[1] + (uint64_t)(y >> S)
                              : (uint64_t)(x >> S);
  uint32_t e0, e1;
  find_pair<D, KEY64>(B, P, row, (int)(last >> S), true, false, e0, e1);
  const EntHead h = ent_head(B, e0);
  const int bit = D == 3 ? (int)((x & SM) << (2 * S) | (y & SM) << S | (z & SM))
                         : (int)((x & SM) << S | (y & SM));
  if (!((h.occ >> bit) & 1ull)) return -1;
  return ent_cell(h.occ, h.base, bit);
}

// cell range of dimension D: 2D instances' cells come first
template <int D>
__device__ __forceinline__ void dim_range(const gdl::Bufs& B, int64_t& mlo, int64_t& mhi) {
  const int64_t M = *B.M, M2 = (int64_t)B.ctr[kCtrCells2D];
  mlo = D == 2 ? 0 : M2;
  mhi = D == 2 ? M2 : M;
}

// ------------------------------------------------------------ stencil tables
// Offsets within +-2 cells, built at compile time.  kHalf[d][pass]: the half
// stencil (o > 0 lexicographically) split into the union passes (union_pass).
// kFullSt[d]: all offsets, nearest first (the warp kernels).
struct OffTab {
  signed char o[128][3];
  int n;
};

// by the smallest possible distance between the cells, then by how many axes
// are off
constexpr int off_rank(int x, int y, int z) {
  const int ax = x < 0 ? -x : x, ay = y < 0 ? -y : y, az = z < 0 ? -z : z;
  const int gx = ax > 1 ? ax - 1 : 0, gy = ay > 1 ? ay - 1 : 0, gz = az > 1 ? az - 1 : 0;
  return (gx * gx + gy * gy + gz * gz) * 8 + ax + ay + az;
}

// Union passes over the half stencil, run in order with a compression between
// them, so that by the later, larger passes most neighbour cells are in A's
// set already and settle from one parent load instead of a root chase and a
// link search.  3D: 0 the face neighbours (one axis off by one), 1 the rest of
// the 3^3 shell, 2 the cells two away along some axis (on C3 the face pass cut
// the union phase from 2.79 to 2.08 ms).  2D: 0 the 3^2 shell, 1 the rest (a
// separate face pass there cost more than it saved).
constexpr int kUnionPasses = 3;

__host__ __device__ constexpr int union_passes(int D) { return D == 3 ? 3 : 2; }

constexpr int union_pass(int D, int x, int y, int z) {
  const int ax = x < 0 ? -x : x, ay = y < 0 ? -y : y, az = z < 0 ? -z : z;
  if (ax > 1 || ay > 1 || az > 1) return union_passes(D) - 1;
  return D == 3 && ax + ay + az != 1 ? 1 : 0;
}

constexpr bool half_pos(int x, int y, int z) {
  return x > 0 || (x == 0 && (y > 0 || (y == 0 && z > 0)));
}

constexpr OffTab make_half(int D, int pass) {
  OffTab t{};
  const int zr = D == 3 ? 2 : 0;
  for (int x = -2; x <= 2; ++x)
    for (int y = -2; y <= 2; ++y)
      for (int z = -zr; z <= zr; ++z) {
        if (!half_pos(x, y, z) || union_pass(D, x, y, z) != pass) continue;
        t.o[t.n][0] = (signed char)x;
        t.o[t.n][1] = (signed char)y;
        t.o[t.n][2] = (signed char)z;
        ++t.n;
      }
  return t;
}

constexpr OffTab make_full(int D) {
  OffTab t{};
  const int zr = D == 3 ? 2 : 0;
  for (int rank = 0; rank < 40; ++rank)
    for (int x = -2; x <= 2; ++x)
      for (int y = -2; y <= 2; ++y)
        for (int z = -zr; z <= zr; ++z) {
          if (off_rank(x, y, z) != rank) continue;
          t.o[t.n][0] = (signed char)x;
          t.o[t.n][1] = (signed char)y;
          t.o[t.n][2] = (signed char)z;
          ++t.n;
        }
  return t;
}
static_assert(make_full(2).n == 25 && make_full(3).n == 125, "whole stencils");

__constant__ OffTab kHalf[2][kUnionPasses] = {{make_half(2, 0), make_half(2, 1), make_half(2, 2)},
                                              {make_half(3, 0), make_half(3, 1), make_half(3, 2)}};

// Union pass masks by a cell's place in its block and the stencil block (row
// r = first-axis half [x 2 + second-axis half], last-axis half k: 2 r + k;
// half 0 is the block of c - 2): the block's cells that are in the pass's half
// stencil of that cell.
struct PassMasks {
  unsigned long long m[kUnionPasses][64][8];
};

constexpr PassMasks make_pass_masks(int D) {
  PassMasks t{};
  const int S = D == 2 ? 3 : 2, SIDE = 1 << S, zr = D == 3 ? 2 : 0;
  for (int lb = 0; lb < 64; ++lb) {
    const int cx = D == 3 ? lb >> 4 : lb >> 3, cy = D == 3 ? (lb >> 2) & 3 : lb & 7;
    const int cz = D == 3 ? lb & 3 : 0;
    for (int x = -2; x <= 2; ++x)
      for (int y = -2; y <= 2; ++y)
        for (int z = -zr; z <= zr; ++z) {
          if (!half_pos(x, y, z)) continue;
          // cell and stencil block start per axis, shifted by one block to stay >= 0
          const int X = cx + x + SIDE, Y = cy + y + SIDE, Z = cz + z + SIDE;
          const int hx = (X >> S) - ((cx - 2 + SIDE) >> S), hy = (Y >> S) - ((cy - 2 + SIDE) >> S);
          const int hz = D == 3 ? (Z >> S) - ((cz - 2 + SIDE) >> S) : 0;
          const int in = D == 3 ? (X & 3) << 4 | (Y & 3) << 2 | (Z & 3) : (X & 7) << 3 | (Y & 7);
          const int blk = D == 3 ? hx * 4 + hy * 2 + hz : hx * 2 + hy;
          t.m[union_pass(D, x, y, z)][lb][blk] |= 1ull << in;
        }
  }
  return t;
}

// (global memory: the lanes of a warp read different entries)
__device__ const PassMasks kPassMasks[2] = {make_pass_masks(2), make_pass_masks(3)};
__constant__ OffTab kFullSt[2] = {make_full(2), make_full(3)};

// Per-warp list of the stencil's non-empty cells, nearest first: cell r holds
// the points lo[r] .. lo[r] + len, and pre[r] is the exclusive prefix of the
// lengths (the cells concatenated).
struct CellList {
  int lo[128];
  int pre[128];
};

// fills the list (each lane looks up every 32nd stencil cell); returns the
// points, and the cells in ncells
template <int D, bool KEY64>
__device__ __forceinline__ int build_cells(const gdl::Bufs& B, CellList& CL, const CellXYZ<D>& cc,
                                           const DevParams& P, int lane, int& ncells) {
  const OffTab& T = kFullSt[D - 2];
  int total = 0, cells = 0;
  for (int t0 = 0; t0 < T.n; t0 += 32) {
    const int t = t0 + lane;
    int lo = 0, len = 0;
    if (t < T.n) {
      const int c = find_cell<D, KEY64>(B, P, (int64_t)cc.c[0] + T.o[t][0],
                                        (int64_t)cc.c[1] + T.o[t][1], (int64_t)cc.c[2] + T.o[t][2]);
      if (c >= 0) {
        lo = B.reps[c];
        len = B.reps[c + 1] - lo;
      }
    }
    int inc = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(kFull, inc, o);
      if (lane >= o) inc += v;
    }
    const unsigned has = __ballot_sync(kFull, len > 0);
    if (len > 0) {
      const int at = cells + __popc(has & ((1u << lane) - 1u));
      CL.lo[at] = lo;
      CL.pre[at] = total + inc - len;
    }
    cells += __popc(has);
    total += __shfl_sync(kFull, inc, 31);
  }
  __syncwarp();
  ncells = cells;
  return total;
}

// sorted position of concatenated candidate c (0 <= c < total)
__device__ __forceinline__ int cell_list_pos(const CellList& CL, int ncells, int c) {
  int r = 0;
#pragma unroll
  for (int step = 64; step; step >>= 1)
    if (r + step < ncells && CL.pre[r + step] <= c) r += step;
  return CL.lo[r] + (c - CL.pre[r]);
}

constexpr int kWarpsPerBlock = 8;
constexpr int kCellThreads = kWarpsPerBlock * 32;

// ----------------------------------------------- cell-level classification
// Origin (low corner) of cell cc in the centred float32 frame.
template <int D>
__device__ __forceinline__ void cell_origin32(const CellXYZ<D>& cc, const DevParams& P, float* o) {
  if (P.fast_origin) {
    // o = fl32((lo - centre) + c f) from float pairs: c f_hi by an exact
    // two-product (fma), added to b_hi by an exact two-sum, the small terms
    // (product error, c f_lo, b_lo) summed in float; one final rounding.  The
    // result is within |o| 2^-24 (1 + 2^-20) of the exact value (c < 2^24 is
    // exact in float; the pairs carry 48 bits), which the position error
    // bound (uerr, via ea) covers.
#pragma unroll
    for (int k = 0; k < D; ++k) {
      const float c = (float)(int)cc.c[k];
      const float p = __fmul_rn(c, P.f_hi);
      const float e = __fmaf_rn(c, P.f_hi, -p);
      const float q = __fmul_rn(c, P.f_lo);
      const float a = P.b_hi[k];
      const float s = __fadd_rn(a, p);
      const float v = __fsub_rn(s, a);
      const float t = __fadd_rn(__fsub_rn(a, __fsub_rn(s, v)), __fsub_rn(p, v));
      const float low = __fadd_rn(__fadd_rn(t, e), __fadd_rn(q, P.b_lo[k]));
      o[k] = __fadd_rn(s, low);
    }
    return;
  }
#pragma unroll
  for (int k = 0; k < D; ++k)
    o[k] = __double2float_rn(
        __dsub_rn(__dadd_rn(P.lo[k], __dmul_rn((double)cc.c[k], P.f)), P.centre[k]));
}

// A point's position inside its own cell, in cell units (error <= P.uerr).
template <int D, class PP>
__device__ __forceinline__ void frac_pos(const float* xf, const float* o, const PP& P, float* u) {
#pragma unroll
  for (int k = 0; k < D; ++k) u[k] = __fmul_rn(__fsub_rn(xf[k], o[k]), P.inv_f32);
}

// Cell at offset (ox, oy, oz) from the point's cell: 1 every point in it is a
// neighbour (both ways), -1 none is, 0 must be tested.
template <int D, class PP>
__device__ __forceinline__ int classify(const float* u, int ox, int oy, int oz, const PP& P) {
  const int off[3] = {ox, oy, oz};
  float smax = 0.0f, smin = 0.0f;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    const float a = u[k] - (float)off[k];  // position relative to the box [off, off + 1]
    const float b = a - 1.0f;
    const float mx = fmaxf(fabsf(a), fabsf(b)) + P.uerr;
    const float mn = fmaxf(fmaxf(-a, b) - P.uerr, 0.0f);
    smax = fmaf(mx, mx, smax);
    smin = fmaf(mn, mn, smin);
  }
  if (smax <= P.thr_in) return 1;
  if (smin >= P.thr_out) return -1;
  return 0;
}

// ------------------------------------------------------- thread front ends
// Most work items need little: isolated noise points whose stencil holds fewer
// than minpts points, cells whose neighbour links are found by the first test,
// border points with a handful of candidate cores.  The front-end kernels give
// one thread to each point, chunk of points (core count, border search) or core
// cell (union scan) and finish those cases inline (bounded work per thread); a
// cell that needs more is appended to the heavy list and handled by the
// warp-cooperative *_heavy kernel that follows.  The stencil's 25 or 125 cells come
// as the occupancy words of 4 or 8 blocks, so empty cells cost nothing.  (Rows of 5
// cells, each looked up by itself, had cost 5 or 25 lookups per walk, by binary
// search outside the densest grids.)
constexpr int kScanThreadsPerBlock = 256;
// The walk kernels (core count, union scan, border search) take their list
// entries from a global cursor in batches of 32 (a union scan over a long list: 64,
// as its entries are short: C3 union 1.32 ms at 32, 1.30 at 64; a 1M-point 2D
// expand, whose lists are a few passes long: 0.24 ms core at 64, 0.21 at 32), 32 per
// pass of a warp: work is handed out as it is done, so no warp is left with a tail of
// costly entries after the others finish (a static grid-stride split left
// whole SMs idle behind a few slow warps).
constexpr int kUnionSmall = 1 << 20;
struct WalkCursor {
  unsigned long long* c;  // kCtrWalkCursor2/3, zero at launch
  int span;               // list entries of this dimension (< 2^31)
  int batch;              // entries handed out at a time
  int next, end;          // the warp's batch, relative to its first entry (warp-uniform)
  // the warp's next 32 entries are [next, min(next + 32, end)); false when the
  // list is used up (all lanes call it)
  __device__ __forceinline__ bool advance(int lane) {
    if (next < end) return true;
    unsigned long long got = 0;
    if (lane == 0) got = atomicAdd(c, (unsigned long long)batch);
    got = __shfl_sync(kFull, got, 0);
    if (got >= (unsigned long long)span) return false;
    next = (int)got;
    end = span - next > batch ? next + batch : span;
    return true;
  }
};
template <int D>
__device__ __forceinline__ WalkCursor walk_cursor(const gdl::Bufs& B, int64_t jlo, int64_t jhi,
                                               int batch) {
  return WalkCursor{B.ctr + (D == 2 ? kCtrWalkCursor2 : kCtrWalkCursor3), (int)(jhi - jlo), batch,
                    0, 0};
}
// Resident 256-thread blocks per SM the front-end kernels are compiled for
// (register budget 65536 / (256 * blocks) per thread).  These kernels are
// bound by memory latency, so occupancy beats registers (a few spilled bytes
// cost less than a lost block).
#ifndef GD_CORE_MIN_BLOCKS
#define GD_CORE_MIN_BLOCKS 8
#endif
#ifndef GD_CORE_CELL_MIN_BLOCKS
#define GD_CORE_CELL_MIN_BLOCKS 7
#endif
#ifndef GD_UNION_MIN_BLOCKS
#define GD_UNION_MIN_BLOCKS 6
#endif
#ifndef GD_BORDER_MIN_BLOCKS
#define GD_BORDER_MIN_BLOCKS 8
#endif
constexpr int kCoreMinBlocks = GD_CORE_MIN_BLOCKS;
constexpr int kCoreCellMinBlocks = GD_CORE_CELL_MIN_BLOCKS;
constexpr int kUnionMinBlocks = GD_UNION_MIN_BLOCKS;
constexpr int kBorderMinBlocks = GD_BORDER_MIN_BLOCKS;
constexpr int kBorderThreads = 128;
// The pair-test budgets of one thread (core count per point, link search per
// cell pair, border search per point) come with the buffers (Bufs::tn_*): the
// context sets them, the autotuner varies them.

// warp-aggregated append to the heavy list (all 32 lanes must call it)
__device__ __forceinline__ void heavy_push(const gdl::Bufs& B, int slot, bool push, int64_t m,
                                           unsigned long long mask) {
  const unsigned bal = __ballot_sync(kFull, push);
  if (!bal) return;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(bal) - 1;
  unsigned long long base = 0;
  if (lane == leader) base = atomicAdd(B.ctr + slot, (unsigned long long)__popc(bal));
  base = __shfl_sync(kFull, base, leader);
  if (push) {
    const unsigned long long at = base + (unsigned long long)__popc(bal & ((1u << lane) - 1u));
    B.hv_cell[at] = (int)m;
    B.hv_mask[at] = mask;
  }
}

template <int D, bool F32>
__device__ __forceinline__ void load_point(double* x, float* f, const gdl::Bufs& B, int64_t i,
                                           bool prune) {
  // float32-band mode tests from the float32 copy; the float64 coordinates
  // are loaded by the band re-test itself
  if (!F32) ld_x<D>(B, i, x);
  if (F32 || prune) ld_f<D>(B, i, f);
}

// The +-2 stencil of a cell over its blocks: per axis the first block, and the
// cells of the axis as bits counted from that block's first cell (w5: within
// two, w3: within one); the axis' cells fall into two blocks at most.
template <int D>
struct Stencil {
  static constexpr int S = block_shift<D>(), SIDE = 1 << S, ROWS = D == 3 ? 4 : 2;
  int b0[D];
  uint32_t w5[D];
  __device__ __forceinline__ void init(const CellXYZ<D>& cc) {
#pragma unroll
    for (int k = 0; k < D; ++k) {
      b0[k] = (cc.c[k] - 2) >> S;
      w5[k] = 31u << ((cc.c[k] - 2) & (SIDE - 1));
    }
  }
  // offset of the first cell of axis k's first block from the cell
  __device__ __forceinline__ int off0(const CellXYZ<D>& cc, int k) const {
    return (int)((unsigned)b0[k] << S) - cc.c[k];
  }
  static __device__ __forceinline__ uint32_t part(uint32_t w, int i) {
    return i ? w >> SIDE : w & ((1u << SIDE) - 1u);
  }
  // block row r: its index among the grid's block rows, or -1 outside the grid
  __device__ __forceinline__ int64_t row(int r, const DevParams& P) const {
    const int bx = b0[0] + (D == 3 ? r >> 1 : r);
    if (bx < 0 || bx >= P.Bk[0]) return -1;
    if (D == 2) return bx;
    const int by = b0[1] + (r & 1);
    if (by < 0 || by >= P.Bk[1]) return -1;
    return (int64_t)bx * P.Bk[1] + by;
  }
  // place along axis k of the cell at `bit` of a block
  static __device__ __forceinline__ int bit_off(int bit, int k) {
    return k == 0 ? bit >> (D == 3 ? 2 * S : S) : (D == 3 && k == 1 ? (bit >> S) & (SIDE - 1)
                                                                    : bit & (SIDE - 1));
  }
};

// Masks of the stencil's blocks from per-axis cell sets (Stencil::w5 or a part of
// it): an axis' cells as words of a block mask, for each half of the axis.  The
// middle (3D) and the last axis repeat in both words.
template <int D>
struct StencilWords {
  using St = Stencil<D>;
  uint32_t xl[2], xh[2], y[2], z[2];
  static __device__ __forceinline__ uint32_t first(uint32_t m) {  // half of the axis: one word
    return D == 3 ? (m & 1u) * 0xffffu | ((m >> 1) & 1u) * 0xffff0000u
                  : ((m | m << 7 | m << 14 | m << 21) & 0x01010101u) * 255u;
  }
  __device__ __forceinline__ void init(const uint32_t* w) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t px = St::part(w[0], i), pz = St::part(w[D - 1], i);
      xl[i] = first(px & ((1u << (St::SIDE / 2)) - 1u));
      xh[i] = first(px >> (St::SIDE / 2));
      const uint32_t py = D == 3 ? St::part(w[1], i) : 0u;
      y[i] = D == 3 ? ((py | py << 3 | py << 6 | py << 9) & 0x1111u) * 15u * 0x10001u : ~0u;
      z[i] = pz * (D == 3 ? 0x11111111u : 0x01010101u);
    }
  }
  // masks of row r's two blocks
  __device__ __forceinline__ void row(int r, uint2& m0, uint2& m1) const {
    const int ri = D == 3 ? r >> 1 : r;
    const uint32_t a = ri ? xl[1] : xl[0], b = ri ? xh[1] : xh[0];
    const uint32_t c = D == 3 ? ((r & 1) ? y[1] : y[0]) : ~0u;
    m0 = make_uint2(a & c & z[0], b & c & z[0]);
    m1 = make_uint2(a & c & z[1], b & c & z[1]);
  }
};
__device__ __forceinline__ unsigned long long u64_of(uint2 v) {
  return (unsigned long long)v.y << 32 | v.x;
}

// Neighbour entries of every cell whose instance has no direct table: per row of its
// stencil the entries of the row's two blocks.  The filter, the core walks, the union
// passes and the border search all look up the same blocks, by a binary search in a
// row that takes four to seven dependent loads; here each is searched once and then
// read in one load beside its cell's (sparse batches: 60.5 -> 55.2 ms, 4,096 instances).
template <bool KEY64>
__global__ void __launch_bounds__(256) k_neighbors(const gdl::Bufs B) {
  const int LB = B.Bi->LB;
  const int64_t M = *B.M;
  for (int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; m < M;
       m += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t key = ckey_at<KEY64>(B, m);
    const DevParams& P = B.Pv[inst_of(key, LB)];
    if (P.sparse == 0) continue;
    auto rows = [&](auto dim) {
      constexpr int D = decltype(dim)::value;
      const CellXYZ<D> cc = decompose<D>(key & P.kmask, P);
      Stencil<D> st;
      st.init(cc);
      // the second block of an axis is met unless the five cells fit one block
      const bool two = ((cc.c[D - 1] - 2) & (Stencil<D>::SIDE - 1)) + 4 >= Stencil<D>::SIDE;
      for (int r = 0; r < Stencil<D>::ROWS; ++r) {
        uint32_t e0 = kNoEnt, e1 = kNoEnt;
        const int64_t row = st.row(r, P);
        if (row >= 0)
          find_pair<D, KEY64>(B, P, (uint64_t)row, st.b0[D - 1], true, two, e0, e1);
        B.nbr[4 * m + r] = make_uint2(e0, e1);
      }
    };
    if (P.dim == 2) rows(std::integral_constant<int, 2>{});
    else rows(std::integral_constant<int, 3>{});
  }
}

// Squared largest / smallest distance (plus / minus the position error) along
// one axis from a point at in-cell position a (cell units) to the cell slab at
// offset o.
template <class PP>
__device__ __forceinline__ void axis_terms(float a, int o, const PP& P, float& mx2, float& mn2) {
  const float x = a - (float)o, y = x - 1.0f;
  const float mx = fmaxf(fabsf(x), fabsf(y)) + P.uerr;
  const float mn = fmaxf(fmaxf(-x, y) - P.uerr, 0.0f);
  mx2 = mx * mx;
  mn2 = mn * mn;
}

// Axes whose slab distance terms a float64 core walk keeps in shared memory (the
// 3D walk forms the others again).
__host__ __device__ constexpr int core_axes(int d) { return d == 3 ? 1 : d; }
constexpr int kCoreThreads = 128;
constexpr int kCoreWarps = kCoreThreads / 32;

// Points in the stencil of a cell, counted up to `enough`: occupied cells, cells of
// two and more, and the rest of the cells of three and more one by one.
template <int D>
__device__ __forceinline__ int stencil_points(const gdl::Bufs& B, const DevParams& P, int64_t cell,
                                              uint64_t local, int enough) {
  using St = Stencil<D>;
  const CellXYZ<D> cc = decompose<D>(local, P);
  St st;
  st.init(cc);
  StencilWords<D> W5;
  W5.init(st.w5);
  int pts = 0;
  for (int r = 0; r < St::ROWS && pts < enough; ++r) {
    const int64_t row = st.row(r, P);
    if (row < 0) continue;
    uint2 m[2];
    W5.row(r, m[0], m[1]);
    uint32_t e[2];
    block_pair<D>(B, P, cell, r, (uint64_t)row, st.b0[D - 1], (m[0].x | m[0].y) != 0,
                         (m[1].x | m[1].y) != 0, e[0], e[1]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (e[h] == kNoEnt) continue;
      const EntHead a = ent_head(B, e[h]);
      const unsigned long long M = u64_of(m[h]), o = a.occ & M;
      if (!o) continue;
      const BlockPop p = B.pop[e[h]];
      pts += __popcll(o) + __popcll((p.two[0] | (unsigned long long)p.two[1] << 32) & M);
      for (unsigned long long w = (p.three[0] | (unsigned long long)p.three[1] << 32) & M;
           w && pts < enough; w &= w - 1) {
        const int c = ent_cell(a.occ, a.base, __ffsll((long long)w) - 1);
        pts += B.reps[c + 1] - B.reps[c] - 2;
      }
    }
  }
  return pts;
}

// Cells whose stencil holds fewer than minpts points: no point of theirs is a core
// point, and none needs a walk (a bit per cell in fbits).  A thread per cell.
// Float32-band mode only: there it saves the batch workload, three of whose points in
// four are noise, a quarter of the core phase (32.5 -> 25.1 ms) and costs a
// single-instance run nothing (C3: core 1.85 -> 1.73 ms, index 1.58 -> 1.70).  The
// float64 walk drops such points before it tests them; there the extra pass cost more
// than it saved (2D tracks 1.03 -> 1.09 ms).
template <bool KEY64>
__global__ void __launch_bounds__(256) k_core_filter(const gdl::Bufs B) {
  const int LB = B.Bi->LB;
  const int64_t M = *B.M;
  const int lane = threadIdx.x & 31;
  for (int64_t m0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); m0 < M;
       m0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = m0 + lane;
    bool skip = false;
    if (m < M) {
      const uint64_t key = ckey_at<KEY64>(B, m);
      const DevParams& P = B.Pv[inst_of(key, LB)];
      const int minpts = P.minpts;
      if (B.reps[m + 1] - B.reps[m] < minpts)
        skip = (P.dim == 2 ? stencil_points<2>(B, P, m, key & P.kmask, minpts)
                           : stencil_points<3>(B, P, m, key & P.kmask, minpts)) < minpts;
    }
    const unsigned b = __ballot_sync(kFull, skip);
    if (lane == 0) B.fbits[m0 >> 5] = b;
  }
}

// Core flags of points in dense cells (at least minpts points: all core, no
// test), with their cells' core counts.  Every other
// point gets its bit in the walk list's mask (listed in sorted order
// afterwards), so that k_core_point's warps hold only neighbouring points that
// walk.  ONE: a single instance (its parameters are Pv[0]).
// chunk: points per walk list entry (1, or k_core_cell's chunk).
template <bool KEY64, bool ONE>
__global__ void k_core_split(const gdl::Bufs B, int64_t n, int chunk, int clear) {
  const int LB = B.Bi->LB;
  const int lane = threadIdx.x & 31;
  unsigned long long dense = 0;
  // a later expand of the index: the blocks' words start empty again
  const int64_t Mc = clear ? (int64_t)*B.M : 0;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < Mc;
       c += (int64_t)gridDim.x * blockDim.x) {
    BlockEnt& E = B.ent[B.cellent[c]];
    if (E.base != (uint32_t)c) continue;
    E.lo = kNoEnt;
    E.core = 0;
    E.hi = kNoEnt;
  }
  // two groups of 32 points per warp and pass, their loads issued together
  constexpr int U = 2;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t g0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); g0 < n;
       g0 += U * stride) {
    int m[U], b[U], e[U], mp[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = g0 + u * stride + lane;
      const int64_t ic = i < n ? i : n - 1;
      m[u] = cell_of(B, ic);
      mp[u] = B.Pv[ONE ? 0 : (int)(key_at<KEY64>(B, ic) >> LB)].minpts;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      b[u] = B.reps[m[u]];
      e[u] = B.reps[m[u] + 1];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i0 = g0 + u * stride;
      if (i0 >= n) break;  // warp-uniform
      const int64_t i = i0 + lane;
      const bool dn = i < n && e[u] - b[u] >= mp[u];
      if (dn) {
        B.core[i] = 1;
        if (i == b[u]) {
          B.cellcore[m[u]] = e[u] - b[u];
          ++dense;
        }
      }
      // the walk list: the chunk starts among the points outside dense cells, but for
      // the cells that k_core_filter settled
      const bool out = B.pop && i < n && !dn && ((B.fbits[m[u] >> 5] >> (m[u] & 31)) & 1u);
      if (out) B.core[i] = 0;
      const unsigned wl = __ballot_sync(kFull, i < n && !dn && !out && (((int)i - b[u]) & (chunk - 1)) == 0);
      if (lane == 0) B.lbits[i0 >> 5] = wl;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dense += __shfl_xor_sync(kFull, dense, o);
  if (lane == 0 && dense) atomicAdd(B.ctr + kCtrDenseCells, dense);
}

// Core flags of the points outside dense cells, float32-band mode: a thread per
// chunk of up to kCoreChunk consecutive points of one cell, taken from the walk
// list (chunk starts, in sorted order) through the walk cursor.  The chunk shares
// one stencil walk: the stencil comes as a few 64-cell occupancy words (4 block
// lookups in 2D, 8 in 3D, two at a time; home row first), masked to the cells
// within one (pass 0) and then two (pass 1) of the own cell, whose points count at
// once; slabs out of reach of the chunk's bounding box leave the masks.
// Every candidate of an occupied cell is loaded once and tested against all the
// chunk's points in registers -- a float32 test is about nine instructions, less
// than the steps that reach a candidate, so sharing those pays more than any
// finer rule on what to test.  Only cells of more than kCoreBigCell points are
// classified first, as a whole and per point (wholly inside eps: count, wholly
// outside: skip; from 1, 2, 5 points on the batch's core phase took 20.7, 20.1 and 18.7
// ms, from 8 on 18.4, and no less beyond).
// A chunk whose tests pass its budget sends its cell to the warp kernel, which
// recomputes the whole cell.  The budget counts every candidate (most cells are not classified
// first), so it is kCellBudget times the context's per point: a whole 3D stencil of 8 points per
// cell.  (2M 3D points, uniform, 4 per cell, minPts 87, the mean neighbour count: core phase
// 3.91 ms at one times the budget, 2.55 at two, four, eight and sixteen; 9 per cell: 6.03, 6.02,
// 3.98, 3.97, 3.97.)  A cell of more than half the budget that is not settled whole goes to the
// warp kernel at once: its points are a long serial chain (200 clumps of 5,000 2D points, spread
// 0.05 to 5 at eps 0.5, minPts 5 and 50: 381 and 1129 us without the rule, 147 and 282 from 128
// points on, 134 and 270 from 64, 157 and 354 from 256; five minPts on 1M even 2D points take 0.6 %
// longer with the line at 128 than without the rule, 2 % at 64).  Per-cell core counts are atomics
// (cleared before the launch).
//
// Passes [p0, p1).  3D runs pass 0 for every listed chunk first: a chunk with an
// undecided point keeps its points' counts in lab[] (kDecided for decided ones)
// and its bit in fbits, and a second launch runs pass 1 for that compacted list
// only, so that its warps hold only chunks that need the long walk.
#ifndef GD_CORE_CHUNK
#define GD_CORE_CHUNK 2
#endif
constexpr int kCoreChunk = GD_CORE_CHUNK;
constexpr int kCoreBigCell = 8;
constexpr int kCellBudget = 4;
constexpr int kDecided = 0x3fffffff;
template <int D, bool KEY64>
__global__ void __launch_bounds__(kCoreThreads, kCoreCellMinBlocks)
k_core_cell(const gdl::Bufs B, int64_t n, int p0, int p1) {
  using St = Stencil<D>;
  constexpr int C = kCoreChunk;
  const int lane = threadIdx.x & 31;
  const int LB = B.Bi->LB;
  const bool second = p0 > 0;    // the list and counts of a first launch
  const bool split = p1 < 2;     // a second launch follows
  // this dimension's part of the walk list: 2D instances' points come first
  const int64_t p3 = B.reps[(int64_t)B.ctr[kCtrCells2D]];
  const int64_t L = (int64_t)*B.lcount;
  const int64_t L2 =
      p3 < n ? (int64_t)(second ? bit_rank(B.fbits, B.fpre, p3) : bit_rank(B.lbits, B.lpre, p3))
             : L;
  const int64_t jlo = D == 2 ? 0 : L2, jhi = D == 2 ? L2 : L;
  WalkCursor wc = walk_cursor<D>(B, jlo, jhi, 32);
  Tally t;
  while (wc.advance(lane)) {
    const int64_t j = jlo + wc.next + lane;
    const bool valid = wc.next + lane < wc.end;
    wc.next += 32;
    const int64_t i = valid ? (int64_t)B.blist[j] : 0;
    int m = -1, na = 0, minpts = 0;
    bool over = false;
    int cnt[C];
    uint32_t was = 0;  // points decided by the first launch
    if (valid) {
      m = cell_of(B, i);
      const int b = B.reps[m], e = B.reps[m + 1];
      na = min(C, e - (int)i);
      const CellCtx cx = cell_ctx<KEY64>(B, m, LB);
      const DevParams& P = *cx.P;
      const PredParams Q = pred_params(P);
      minpts = Q.minpts;
      const bool prune = Q.prune != 0;
      const CellXYZ<D> cc = decompose<D>(cx.local, P);
      St st;
      st.init(cc);
      // the chunk's points; absent ones repeat the first and count as decided
      float pf[C][D];
      int present = 0;
#pragma unroll
      for (int a = 0; a < C; ++a) {
        const int64_t ia = a < na ? i + a : i;
        ld_f<D>(B, ia, pf[a]);
        cnt[a] = a < na ? (second ? B.lab[ia] : e - b) : kDecided;
        if (a < na && second && cnt[a] == kDecided) was |= 1u << a;
        present += cnt[a] < minpts;
      }
      float o[D], ulo[D], uhi[D];  // cell origin, the undecided points' bounds in the cell
      if (prune) {
        cell_origin32<D>(cc, P, o);
#pragma unroll
        for (int k = 0; k < D; ++k) {
          float lo = INFINITY, hi = -INFINITY;
#pragma unroll
          for (int a = 0; a < C; ++a)
            if (cnt[a] < minpts) {
              lo = fminf(lo, pf[a][k]);
              hi = fmaxf(hi, pf[a][k]);
            }
          ulo[k] = __fmul_rn(__fsub_rn(lo, o[k]), Q.inv_f32) - Q.uerr;
          uhi[k] = __fmul_rn(__fsub_rn(hi, o[k]), Q.inv_f32) + Q.uerr;
          uint32_t near = 14u;
          const float l2 = ulo[k] + 1.0f, h2 = 2.0f - uhi[k];  // to the slabs at -2 and +2
          if (!(l2 > 0.0f && l2 * l2 >= Q.thr_out)) near |= 1u;
          if (!(h2 > 0.0f && h2 * h2 >= Q.thr_out)) near |= 16u;
          st.w5[k] = near << ((cc.c[k] - 2) & (St::SIDE - 1));
        }
      }
      int budget = kCellBudget * B.tn_core * present;
      bool done = present == 0;
      // one occupied cell: place `bit` of block (row r, half h) of the stencil
      auto visit = [&](int q0, int qe, int bit, int r, int h) {
        if (prune && qe - q0 > kCoreBigCell) {
          // out of reach of all the points, or settled for each of them?
          int off[3] = {0, 0, 0};
          float smin = 0.0f;
#pragma unroll
          for (int k = 0; k < D; ++k) {
            const int half = k == D - 1 ? h : (D == 3 ? (k == 0 ? r >> 1 : r & 1) : r);
            off[k] = st.off0(cc, k) + (half << St::S) + St::bit_off(bit, k);
            const float d = (float)off[k];
            const float mn = fmaxf(fmaxf(d - uhi[k], ulo[k] - 1.0f - d), 0.0f);
            smin = fmaf(mn, mn, smin);
          }
          if (smin >= Q.thr_out) return;
          int cl[C];
          bool open = false;
#pragma unroll
          for (int a = 0; a < C; ++a) {
            cl[a] = -1;
            if (cnt[a] < minpts) {
              float u[D];
              frac_pos<D>(pf[a], o, Q, u);
              cl[a] = classify<D>(u, off[0], off[1], off[2], Q);
              open |= cl[a] == 0;
            }
          }
          if (!open) {
#pragma unroll
            for (int a = 0; a < C; ++a)
              if (cl[a] > 0) cnt[a] += qe - q0;
            done = true;
#pragma unroll
            for (int a = 0; a < C; ++a) done = done && cnt[a] >= minpts;
            return;
          }
        }
        if (qe - q0 > B.tn_core / 2) budget = 0;  // a crowded cell is a warp's work
        for (int q = q0; q < qe; ++q) {
          budget -= present;
          if (budget < 0) {
            over = true;
            done = true;
            return;
          }
          float f[D];
          ld_f<D>(B, q, f);
          bool band = false;
#pragma unroll
          for (int a = 0; a < C; ++a) {
            const float s2 = dist2_f32<D>(pf[a], f);
            const bool in = s2 < Q.eps2_lo32;
            cnt[a] += in ? 1 : 0;
            band |= !in && !(s2 > Q.eps2_hi32);
          }
          if (band) {
            // the float64 predicate for the points whose float32 test cannot say
            double qx[D];
            ld_x<D>(B, q, qx);
#pragma unroll
            for (int a = 0; a < C; ++a) {
              if (a >= na) continue;
              const float s2 = dist2_f32<D>(pf[a], f);
              if (s2 < Q.eps2_lo32 || s2 > Q.eps2_hi32) continue;
              double px[D];
              ld_x<D>(B, i + a, px);
              ++t.band;
              ++t.t64;
              cnt[a] += pred_from_d2<D>(dist2_f64<D>(px, qx), px, qx, Q) ? 1 : 0;
            }
          }
        }
        t.t32 += present * (qe - q0);
        done = true;
#pragma unroll
        for (int a = 0; a < C; ++a) done = done && cnt[a] >= minpts;
      };
      // the own block's row and half first
      const int hz = (cc.c[D - 1] >> St::S) - st.b0[D - 1];
      const int home = D == 3 ? ((cc.c[0] >> St::S) - st.b0[0]) * 2 + (cc.c[1] >> St::S) - st.b0[1]
                              : (cc.c[0] >> St::S) - st.b0[0];
      for (int ps = p0; ps < p1 && !done; ++ps) {
        StencilWords<D> W5, W3;
        {
          uint32_t w3[D];
#pragma unroll
          for (int k = 0; k < D; ++k) w3[k] = st.w5[k] & (14u << ((cc.c[k] - 2) & (St::SIDE - 1)));
          W3.init(w3);
          if (ps > 0) W5.init(st.w5);
        }
        for (int tt = 0; tt < St::ROWS && !done; ++tt) {
          const int r = tt ^ home;
          const int64_t row = st.row(r, P);
          if (row < 0) continue;
          uint2 m0, m1;
          W3.row(r, m0, m1);
          if (ps > 0) {
            uint2 f0, f1;
            W5.row(r, f0, f1);
            m0 = make_uint2(f0.x & ~m0.x, f0.y & ~m0.y);
            m1 = make_uint2(f1.x & ~m1.x, f1.y & ~m1.y);
          }
          unsigned long long M0 = u64_of(m0), M1 = u64_of(m1);
          if (ps == 0 && tt == 0) {
            // the own cell is counted already
            const unsigned long long own = ~(1ull << (cx.local & 63));
            if (hz == 0) M0 &= own;
            else M1 &= own;
          }
          uint32_t e0, e1;
          block_pair<D>(B, P, m, r, (uint64_t)row, st.b0[D - 1], M0 != 0, M1 != 0, e0, e1);
          EntHead a = ent_head(B, e0);
          const EntHead a1 = ent_head(B, e1);
          unsigned long long w = a.occ & M0, wn = a1.occ & M1;
          int h = 0;
          while (!done) {
            if (!w) {
              if (!wn) break;
              w = wn;
              wn = 0;
              a = a1;
              h = 1;
            }
            const int bit = __ffsll((long long)w) - 1;
            w &= w - 1;
            const int c = ent_cell(a.occ, a.base, bit);
            visit(B.reps[c], B.reps[c + 1], bit, r, h);
          }
        }
      }
    }
    // results: core flags; in a first launch the undecided chunks go on
    int ncore = 0;
    if (valid && !over) {
      bool go_on = false;
#pragma unroll
      for (int a = 0; a < C; ++a) {
        if (a >= na || ((was >> a) & 1u)) continue;
        const bool isc = cnt[a] >= minpts;
        if (split) {
          B.lab[i + a] = isc ? kDecided : cnt[a];
          go_on |= !isc;
        }
        if (isc || !split) B.core[i + a] = isc ? 1 : 0;
        ncore += isc;
      }
      if (go_on) atomicOr(B.fbits + (i >> 5), 1u << (i & 31));
    }
    // per-cell core count
    if (ncore > 0) atomicAdd(B.cellcore + m, ncore);
    // cells with an undecided chunk, once per warp
    const unsigned om = __ballot_sync(kFull, over);
    bool lead = false;
    if (over) lead = lane == __ffs(__match_any_sync(om, m)) - 1;
    heavy_push(B, kCtrHeavyCore, lead, m, 0);
  }
  flush_tally(t, B.ctr);
}

// Core flags of the points outside dense cells, float64 mode: a thread per listed
// point, warps taking the list from the walk cursor.  A float64 test occupies
// this GPU's narrow float64 pipe for a whole warp slot however few lanes take
// part, so tests are made only on full warps, and only for points they can
// decide.  First every point classifies its stencil's occupied cells (same block
// words as k_core_cell, no float64): wholly inside eps they count, wholly outside
// they are dropped, the rest stay as bits of their block's word.  A point whose
// undecided cells cannot lift its count to minpts is no core point, untested.
// Then the warp pools: each lane hands out its open candidates one at a time into
// the warp's pair buffer until its count reaches minpts, and whenever the buffer
// holds 32 pairs the warp tests them, a lane per pair.  A point whose own open candidates pass
// the budget sends its cell to the warp kernel, and so does a warp whose candidates pass 32 of
// them.  (200 clumps of 5,000 2D points, spread 0.05 to 5 at eps 0.5, minPts 5 and 50: core phase
// 851 and 1126 us with the warp's rule alone, a few lanes handing out thousands; 194 and 443 so,
// 223 and 491 at twice the budget.)
// Passes as in k_core_cell (2D: both in one walk).
// a lane's open candidates are counted up to this many (32 lanes' sum fits an int)
constexpr int kPoolCap = 0x03ffffff;
template <int D>
struct PairStage {
  double x[32][D];
  double e2in[32], e2[32];
  int inst[32];
  int cnt[32];     // hits among the tested pairs
  int q[64];       // pair buffer: candidate, owner lane
  int own[64];
};
template <int D, bool KEY64>
__global__ void __launch_bounds__(kCoreThreads, kCoreMinBlocks)
k_core_point(const gdl::Bufs B, int64_t n, int p0, int p1) {
  using St = Stencil<D>;
  constexpr int AX = core_axes(D);
  // per thread and axis (the last AX): squared largest / smallest distance terms
  // to the five cell slabs at offsets -2..2
  __shared__ float2 slt[AX][5][kCoreThreads];
  // the blocks with undecided cells (their bits, the entry)
  __shared__ unsigned long long siw[2 * St::ROWS][kCoreThreads];
  __shared__ uint32_t sie[2 * St::ROWS][kCoreThreads];
  __shared__ PairStage<D> stage[kCoreWarps];
  const int lane = threadIdx.x & 31;
  PairStage<D>& S = stage[threadIdx.x >> 5];
  const int LB = B.Bi->LB;
  const bool second = p0 > 0;    // the list and counts of a first launch
  const bool split = p1 < 2;     // a second launch follows
  // this dimension's part of the walk list: 2D instances' points come first
  const int64_t p3 = B.reps[(int64_t)B.ctr[kCtrCells2D]];
  const int64_t L = (int64_t)*B.lcount;
  const int64_t L2 =
      p3 < n ? (int64_t)(second ? bit_rank(B.fbits, B.fpre, p3) : bit_rank(B.lbits, B.lpre, p3))
             : L;
  const int64_t jlo = D == 2 ? 0 : L2, jhi = D == 2 ? L2 : L;
  WalkCursor wc = walk_cursor<D>(B, jlo, jhi, 32);
  Tally t;
  while (wc.advance(lane)) {
    const int64_t j = jlo + wc.next + lane;
    const bool valid = wc.next + lane < wc.end;
    wc.next += 32;
    const int64_t i = valid ? (int64_t)B.blist[j] : 0;
    int m = -1;
    int cnt = 0, ptot = 0, ni = 0, minpts = 0;
    if (valid) {
      m = cell_of(B, i);
      const CellCtx cx = cell_ctx<KEY64>(B, m, LB);
      const DevParams& P = *cx.P;
      const PredParams Q = pred_params(P);
      minpts = Q.minpts;
      cnt = second ? B.lab[i] : B.reps[m + 1] - B.reps[m];
      const bool prune = Q.prune != 0;
      const CellXYZ<D> cc = decompose<D>(cx.local, P);
      St st;
      st.init(cc);
      double px[D];
      float pf[D], u[D];
      load_point<D, false>(px, pf, B, i, prune);
#pragma unroll
      for (int k = 0; k < D; ++k) S.x[lane][k] = px[k];
      S.e2in[lane] = Q.eps2_in;
      S.e2[lane] = Q.eps2;
      S.inst[lane] = P.inst;
      if (prune) {
        float o[D];
        cell_origin32<D>(cc, P, o);
        frac_pos<D>(pf, o, Q, u);
#pragma unroll
        for (int k = 0; k < D; ++k) {
          uint32_t near = 0;
#pragma unroll
          for (int j = 0; j < 5; ++j) {
            float a2, b2;
            axis_terms(u[k], j - 2, Q, a2, b2);
            if (k >= D - AX) slt[k - (D - AX)][j][threadIdx.x] = make_float2(a2, b2);
            if (b2 < Q.thr_out) near |= 1u << j;  // the slab is not beyond eps by itself
          }
          st.w5[k] = near << ((cc.c[k] - 2) & (St::SIDE - 1));
        }
      }
      // cells of this launch: within one (split), the others (second), or all
      StencilWords<D> W5, W3;
      {
        uint32_t w3[D];
#pragma unroll
        for (int k = 0; k < D; ++k) w3[k] = st.w5[k] & (14u << ((cc.c[k] - 2) & (St::SIDE - 1)));
        W3.init(w3);
        W5.init(st.w5);
      }
      const unsigned long long own = 1ull << (cx.local & 63);
      const int home = D == 3 ? ((cc.c[0] >> St::S) - st.b0[0]) * 2 + (cc.c[1] >> St::S) - st.b0[1]
                              : (cc.c[0] >> St::S) - st.b0[0];
      const int hz = (cc.c[D - 1] >> St::S) - st.b0[D - 1];
      for (int tt = 0; tt < St::ROWS && cnt < minpts; ++tt) {
        const int r = tt ^ home;
        const int64_t row = st.row(r, P);
        if (row < 0) continue;
        uint2 a[2], f[2];
        W3.row(r, a[0], a[1]);
        W5.row(r, f[0], f[1]);
        unsigned long long M[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          M[h] = split ? u64_of(a[h]) : (second ? u64_of(f[h]) & ~u64_of(a[h]) : u64_of(f[h]));
          if (tt == 0 && h == hz) M[h] &= ~own;  // the own cell is counted already
        }
        uint32_t e[2];
        block_pair<D>(B, P, m, r, (uint64_t)row, st.b0[D - 1], M[0] != 0, M[1] != 0, e[0], e[1]);
        EntHead hd[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) hd[h] = ent_head(B, e[h]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          unsigned long long w = hd[h].occ & M[h], open = 0;
          while (w && cnt < minpts) {
            const int bit = __ffsll((long long)w) - 1;
            w &= w - 1;
            int cls = 0;
            if (prune) {
              float smax = 0.0f, smin = 0.0f;
#pragma unroll
              for (int k = 0; k < D; ++k) {
                const int half = k == D - 1 ? h : (D == 3 ? (k == 0 ? r >> 1 : r & 1) : r);
                const int j = st.off0(cc, k) + 2 + (half << St::S) + St::bit_off(bit, k);
                float2 lt;
                if (k >= D - AX) lt = slt[k - (D - AX)][j][threadIdx.x];
                else axis_terms(u[k], j - 2, Q, lt.x, lt.y);
                smax += lt.x;
                smin += lt.y;
              }
              cls = smax <= Q.thr_in ? 1 : (smin >= Q.thr_out ? -1 : 0);
            }
            if (cls < 0) continue;
            const int c = ent_cell(hd[h].occ, hd[h].base, bit);
            const int len = B.reps[c + 1] - B.reps[c];
            if (cls > 0) {
              cnt += len;
            } else {
              open |= 1ull << bit;
              ptot = min(ptot + min(len, kPoolCap), kPoolCap);
            }
          }
          if (open) {
            siw[ni][threadIdx.x] = open;
            sie[ni][threadIdx.x] = e[h];
            ++ni;
          }
        }
      }
      // before a second launch the tests are always made (it walks other cells)
      if (cnt >= minpts || (!split && ptot < kPoolCap && cnt + ptot < minpts)) ni = 0;
      if (ni == 0) ptot = 0;
    }
    // ---- pooled tests; a lane hands out one candidate per step, so that one of more than a
    // budget of its own would keep the warp (its cell goes to the warp kernel)
    bool over = ptot > B.tn_core;
    if (over) ni = ptot = 0;
    int pool = ptot;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) pool += __shfl_xor_sync(kFull, pool, o);
    if (pool > 32 * B.tn_core) {  // too much for the warp: the warp kernel takes the cells
      over = over || ni > 0;
      ni = 0;
      pool = 0;
    }
    S.cnt[lane] = 0;
    __syncwarp();
    if (pool > 0) {
      unsigned long long w = 0, occ = 0;
      uint32_t base = 0;
      int k = 0, q = 0, qe = 0, nbuf = 0;
      bool alive = ni > 0;
      while (true) {
        if (alive) {
          if (q == qe) {
            if (!w) {
              if (k == ni) {
                alive = false;
              } else {
                w = siw[k][threadIdx.x];
                const EntHead a = ent_head(B, sie[k][threadIdx.x]);
                occ = a.occ;
                base = a.base;
                ++k;
              }
            }
            if (alive) {
              const int c = ent_cell(occ, base, __ffsll((long long)w) - 1);
              w &= w - 1;
              q = B.reps[c];
              qe = B.reps[c + 1];
            }
          }
          alive = alive && cnt + S.cnt[lane] < minpts;
        }
        const unsigned bal = __ballot_sync(kFull, alive);
        if (alive) {
          const int at = nbuf + __popc(bal & ((1u << lane) - 1u));
          S.q[at] = q++;
          S.own[at] = lane;
        }
        nbuf += __popc(bal);
        __syncwarp();
        if (nbuf >= 32 || (bal == 0 && nbuf > 0)) {
          const int take = min(nbuf, 32);
          nbuf -= take;
          if (lane < take) {
            const int qq = S.q[nbuf + lane], ow = S.own[nbuf + lane];
            double qx[D];
            ld_x<D>(B, qq, qx);
            ++t.t64;
            const double d2 = dist2_f64<D>(S.x[ow], qx);
            bool hit = d2_le(d2, S.e2in[ow]);
            if (!hit && d2_le(d2, S.e2[ow])) hit = box_f64<D>(S.x[ow], qx, B.Pv[S.inst[ow]].eps);
            if (hit) atomicAdd(&S.cnt[ow], 1);
          }
          __syncwarp();
        }
        if (bal == 0 && nbuf == 0) break;
      }
      cnt += S.cnt[lane];
    }
    __syncwarp();
    const bool isc = valid && !over && cnt >= minpts;
    // undecided after pass 0: on to the second launch
    const bool go_on = split && valid && !over && !isc;
    if (go_on) {
      B.lab[i] = cnt;
      atomicOr(B.fbits + (i >> 5), 1u << (i & 31));
    }
    if (valid && !over && !go_on) B.core[i] = isc ? 1 : 0;
    // per-cell core count, one atomic per cell and warp
    const unsigned grp = run_peers(__ballot_sync(kFull, isc), m);
    if (isc && lane == __ffs(grp) - 1) atomicAdd(B.cellcore + m, __popc(grp));
    // cells with an undecided point, once per warp
    const unsigned om = __ballot_sync(kFull, over);
    bool lead = false;
    if (over) lead = lane == __ffs(__match_any_sync(om, m)) - 1;
    heavy_push(B, kCtrHeavyCore, lead, m, 0);
  }
  flush_tally(t, B.ctr);
}

// Bounded link search between the core points of cells A and B by one thread:
// 1 found (neighbours both ways), 0 none exists, -1 budget spent.  With cell
// classification, a core point of A that has all of B within reach links at
// once (B holds a core point), and one that has none of B in reach is skipped.
template <int D, bool F32>
__device__ __forceinline__ int inline_link(const gdl::Bufs& B, int64_t n, int bA, int eA, int bB,
                                           int eB, const float* oA, int ox, int oy, int oz,
                                           const DevParams& P, const PredParams& Q, Tally& t) {
  const bool prune = Q.prune != 0;
  int budget = B.tn_link;
  for (int a = bA; a < eA; ++a) {
    if (!B.core[a]) continue;
    double ax[D];
    float af[D];
    load_point<D, F32>(ax, af, B, a, prune);
    if (prune) {
      float u[D];
      frac_pos<D>(af, oA, Q, u);
      const int cls = classify<D>(u, ox, oy, oz, Q);
      if (cls > 0) return 1;
      if (cls < 0) continue;
    }
    for (int q = bB; q < eB; ++q) {
      if (!B.core[q]) continue;
      if (budget-- == 0) return -1;
      Cand<D, F32> cd;
      load_cand<D, F32>(cd, B, q);
      if (link_test<D, F32>(ax, af, cd, B, a, q, Q, t)) return 1;
    }
  }
  return 0;
}

// Pairs of cells that a thread does not search: it classifies the first cell's points one by
// one, and skips the second one's that are not core points, without counting either.  (2M 3D
// points at 40,000 Zipf-popular positions, the most popular one with 190,000 points, float32
// mode: union phase 49.9 ms, 15.5 so; 400,000 2D points likewise 5.5 and 1.2; the line at 64 or
// 1024 points within 5 %.)
constexpr int kLinkPoints = 256;
constexpr long long kLinkPairs = 1ll << 16;
__device__ __forceinline__ bool crowded_pair(int na, int nb) {
  return na > kLinkPoints || (long long)na * nb > kLinkPairs;
}

// Link between core cells m and c (at offset (ox, oy, oz) from m), m's
// representative in ca: the representatives first -- on the workloads nine face
// neighbours in ten are linked by that one test -- then the search.
template <int D, bool F32>
__device__ __forceinline__ int cell_link(const gdl::Bufs& B, int64_t n, const DevParams& P,
                                         const CellXYZ<D>& cc, int m, int c,
                                         const Cand<D, F32>& ca, int ox, int oy, int oz, Tally& t) {
  Cand<D, F32> cd;
  load_cand<D, F32>(cd, B, B.cellrep[c]);
  bool apart;
  if (F32) {
    ++t.t32;
    const float s2 = dist2_f32<D>(ca.f, cd.f);
    if (s2 < P.eps2_lo32) return 1;
    apart = s2 > P.eps2_hi32;
  } else {
    ++t.t64;
    const double d2 = dist2_f64<D>(ca.x, cd.x);
    if (d2_le(d2, P.eps2_in)) return 1;
    apart = !d2_le(d2, P.eps2);
  }
  if (apart && B.cellcore[m] == 1 && B.cellcore[c] == 1) return 0;  // the only pair
  const int bA = B.reps[m], eA = B.reps[m + 1], bB = B.reps[c], eB = B.reps[c + 1];
  if (crowded_pair(eA - bA, eB - bB)) return -1;
  const PredParams Q = pred_params(P);
  float oA[D];
  if (Q.prune) cell_origin32<D>(cc, P, oA);
  return inline_link<D, F32>(B, n, bA, eA, bB, eB, oA, ox, oy, oz, P, Q, t);
}

// ---- link searches by a warp.
// Core point a of one cell against the core points [b0, b1) of another: whether one is its
// neighbour both ways.  A warp, a lane per candidate.
template <int D, bool F32>
__device__ __forceinline__ bool warp_link_row(const gdl::Bufs& B, int a, int b0, int b1,
                                               const PredParams& Q, Tally& t) {
  const int lane = threadIdx.x & 31;
  double ax[D];
  float af[D];
  if (F32) ld_f<D>(B, a, af);
  else ld_x<D>(B, a, ax);
  for (int qb = b0; qb < b1; qb += 32) {
    const int q = qb + lane;
    bool hit = false;
    if (q < b1 && B.core[q]) {
      Cand<D, F32> c;
      load_cand<D, F32>(c, B, q);
      hit = link_test<D, F32>(ax, af, c, B, a, q, Q, t);
    }
    if (__any_sync(kFull, hit)) return true;
  }
  return false;
}

// The core points [a0, a0 + na), na <= 32, of the cell with origin oA against those of [b0, b1),
// at offset o: whether a pair are neighbours both ways.  A lane per point of the first cell
// finds out which of them have the other cell wholly inside or outside their reach; the others
// are tested all at once with a lane each and the other cell's points one by one, or one by one
// with a lane per point of that cell, whichever takes fewer steps.
template <int D, bool F32>
__device__ __forceinline__ bool warp_link_rows(const gdl::Bufs& B, int a0, int na, int b0, int b1,
                                               const float* oA, const int* o, const PredParams& Q,
                                               Tally& t) {
  const int lane = threadIdx.x & 31;
  int cls = -1;
  double ax[D];
  float af[D];
  if (lane < na && B.core[a0 + lane]) {
    cls = 0;
    load_point<D, F32>(ax, af, B, a0 + lane, Q.prune != 0);
    if (Q.prune) {
      float u[D];
      frac_pos<D>(af, oA, Q, u);
      cls = classify<D>(u, o[0], o[1], o[2], Q);
    }
  }
  if (__any_sync(kFull, cls > 0)) return true;  // (the other cell holds a core point)
  unsigned open = __ballot_sync(kFull, cls == 0);
  if (!open) return false;
  // (the steps of the first way are the cheaper)
  if (5ll * __popc(open) * ((b1 - b0 + 31) / 32) >= 4ll * (b1 - b0)) {
    for (int q = b0; q < b1; ++q) {
      if (!B.core[q]) continue;
      bool hit = false;
      if (cls == 0) {
        Cand<D, F32> c;
        load_cand<D, F32>(c, B, q);
        hit = link_test<D, F32>(ax, af, c, B, a0 + lane, q, Q, t);
      }
      if (__any_sync(kFull, hit)) return true;
    }
    return false;
  }
  for (; open; open &= open - 1)
    if (warp_link_row<D, F32>(B, a0 + __ffs(open) - 1, b0, b1, Q, t)) return true;
  return false;
}

// bit of offset (ox, oy, oz) in the kHalf[D][pass] table, or -1 if it is not there
struct HalfBits {
  signed char b[2][kUnionPasses][5][5][5];
};

constexpr HalfBits make_half_bits() {
  HalfBits h{};
  for (int d = 0; d < 2; ++d)
    for (int p = 0; p < kUnionPasses; ++p) {
      for (int x = 0; x < 5; ++x)
        for (int y = 0; y < 5; ++y)
          for (int z = 0; z < 5; ++z) h.b[d][p][x][y][z] = -1;
      const OffTab t = make_half(d + 2, p);
      for (int i = 0; i < t.n; ++i)
        h.b[d][p][t.o[i][0] + 2][t.o[i][1] + 2][t.o[i][2] + 2] = (signed char)i;
    }
  return h;
}

__constant__ HalfBits kHalfBits = make_half_bits();

template <int D>
__device__ __forceinline__ int half_bit(int pass, int ox, int oy, int oz) {
  return kHalfBits.b[D - 2][pass][ox + 2][oy + 2][oz + 2];
}

// Union scan of one pass, one thread per listed core cell A: the pass's half
// stencil as masks over at most 4 (2D) or 8 (3D) block entries, whose core words
// leave only the cells holding a core point.  The parents of a block's cells are
// read in groups of four, through the cache: a parent equal to A's current root,
// or to A's root when the pass began, settles the cell from one load even if it
// is stale, since sets only merge.  The others are looked at again from fresh
// loads and searched for a link.  The entries also hold the
// root of the block's core cells at the pass's start, where they share one: if it
// is A's, the whole block is settled by its entry.
template <int D, bool F32, bool KEY64>
__global__ void __launch_bounds__(kScanThreadsPerBlock, kUnionMinBlocks)
k_union_scan(const gdl::Bufs B, int64_t n, int pass) {
  using St = Stencil<D>;
  __shared__ unsigned long long siw[2 * St::ROWS][kScanThreadsPerBlock];
  __shared__ uint32_t sie[2 * St::ROWS][kScanThreadsPerBlock];
  const int lane = threadIdx.x & 31;
  const int LB = B.Bi->LB;
  // this dimension's part of the core-cell list: 2D instances' cells come first
  const int64_t M2 = (int64_t)B.ctr[kCtrCells2D];
  const int64_t L = (int64_t)*B.lcount;
  const int64_t L2 = M2 < n ? (int64_t)bit_rank(B.lbits, B.lpre, M2) : L;
  const int64_t jlo = D == 2 ? 0 : L2, jhi = D == 2 ? L2 : L;
  WalkCursor wc = walk_cursor<D>(B, jlo, jhi, jhi - jlo < kUnionSmall ? 32 : 64);
  Tally t;
  while (wc.advance(lane)) {
    const int64_t j = jlo + wc.next + lane;
    const bool valid = wc.next + lane < wc.end;
    wc.next += 32;
    const int64_t m = valid ? (int64_t)B.blist[j] : 0;
    unsigned long long open = 0;
    if (valid) {
      const CellCtx cx = cell_ctx<KEY64>(B, m, LB);
      const DevParams& P = *cx.P;
      const CellXYZ<D> cc = decompose<D>(cx.local, P);
      St st;
      st.init(cc);
      const unsigned long long* __restrict__ masks = kPassMasks[D - 2].m[pass][cx.local & 63];
      // A's parent as the compression before this pass left it: A's root at
      // the start of the pass.  Neighbours' parents were compressed at the
      // same time, so one equal to it puts the cell in A's set however the
      // pass's unions have moved the root since (ra, the current root, is
      // checked too).
      const int ra0 = reinterpret_cast<volatile int*>(B.parent)[m];
      int ra = uf_find(B.parent, (int)m);
      // A's representative: its first core point
      const int qa = B.cellrep[m];
      Cand<D, F32> ca;
      load_cand<D, F32>(ca, B, qa);
      // one cell holding a core point (index c) at offset (ox, oy, oz).  Its
      // points are looked up only when a link search is needed.
      auto visit_core = [&](int c, int ox, int oy, int oz) {
        // ra: a root of A's set, refreshed only when c's root differs.  A
        // parent equal to ra puts c in A's set from one load (ra stays in
        // A's set whatever is hooked later; the pass before compressed the
        // parents to roots).
        const int pc = reinterpret_cast<volatile int*>(B.parent)[c];
        if (pc == ra || pc == ra0) return;
        const int rc = pc == c ? c : uf_find(B.parent, pc);
        if (rc == ra) return;
        ra = uf_find(B.parent, ra);
        if (rc == ra) return;
        const int res = cell_link<D, F32>(B, n, P, cc, (int)m, c, ca, ox, oy, oz, t);
        if (res > 0) {
          uf_union(B.parent, (int)m, c);
          ra = uf_find(B.parent, ra);
        } else if (res < 0) {
          // the pass masks keep every visited offset in this pass's half stencil
          const int bit = half_bit<D>(pass, ox, oy, oz);
          if (bit >= 0) open |= 1ull << bit;
        }
      };
      // the blocks with cells to look at; those are visited afterwards, so that
      // the warp's lanes visit theirs together whatever blocks they lie in
      int ni = 0;
      uint32_t codes = 0;
      for (int r = 0; r < St::ROWS; ++r) {
        const unsigned long long M0 = masks[2 * r], M1 = masks[2 * r + 1];
        if (!(M0 | M1)) continue;
        const int64_t row = st.row(r, P);
        if (row < 0) continue;
        uint32_t e[2];
        block_pair<D>(B, P, m, r, (uint64_t)row, st.b0[D - 1], M0 != 0, M1 != 0, e[0], e[1]);
        EntHead hd[2];
        EntTail tl[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          hd[h] = ent_head(B, e[h]);
          tl[h] = ent_tail(B, e[h]);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          unsigned long long w = tl[h].core & (h ? M1 : M0), slow;
          if ((int)(pass == 0 ? tl[h].uni : pass == 1 ? hd[h].lo : tl[h].hi) == ra0) w = 0;
          slow = 0;
          while (w) {
            int bit[4], pr[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              bit[q] = w ? __ffsll((long long)w) - 1 : -1;
              w &= w - 1;
              pr[q] = bit[q] >= 0 ? B.parent[ent_cell(hd[h].occ, hd[h].base, bit[q])] : ra;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (pr[q] != ra && pr[q] != ra0) slow |= 1ull << bit[q];
          }
          if (slow) {
            siw[ni][threadIdx.x] = slow;
            sie[ni][threadIdx.x] = e[h];
            codes |= (uint32_t)(2 * r + h) << (4 * ni);
            ++ni;
          }
        }
      }
      unsigned long long w = 0, occ = 0;
      uint32_t base = 0;
      int d[3] = {0, 0, 0}, k = 0;
      while (true) {
        if (!w) {
          if (k == ni) break;
          w = siw[k][threadIdx.x];
          const EntHead a = ent_head(B, sie[k][threadIdx.x]);
          occ = a.occ;
          base = a.base;
          const int code = (int)(codes >> (4 * k)) & 7;
          d[0] = st.off0(cc, 0) + ((D == 3 ? code >> 2 : code >> 1) << St::S);
          if (D == 3) d[1] = st.off0(cc, 1) + (((code >> 1) & 1) << St::S);
          d[D - 1] = st.off0(cc, D - 1) + ((code & 1) << St::S);
          ++k;
        }
        const int bit = __ffsll((long long)w) - 1;
        w &= w - 1;
        visit_core(ent_cell(occ, base, bit), d[0] + St::bit_off(bit, 0), d[1] + St::bit_off(bit, 1),
                   D == 3 ? d[2] + St::bit_off(bit, 2) : 0);
      }
    }
    heavy_push(B, kCtrHeavyUnion, open != 0, m, open);
  }
  flush_tally(t, B.ctr);
}

// Border labels, one thread per listed non-core point (k_label lists them,
// consecutive lanes holding consecutive sorted points).  Each point walks its
// stencil and takes the smallest cluster id among the cells whose core points
// have it in their neighbourhood (centre = the core point, as the reference's
// expansion queries from the core point).  Cells whose id cannot improve on
// the best so far are skipped; with classification, a cell wholly inside eps
// gives its id without tests and one wholly outside is skipped.  A point whose
// tests pass the budget sends its cell to the warp kernel.  The own block comes first: in it
// lie most of the near cells, whose first hit settles all cells of the same cluster (2M 3D
// points, 4 per cell, half of them border points: label phase 646 us in block order, 389 so,
// float64 mode 1841 and 874; cells within one of the own first in every block 344 and 514, but
// 48.4 -> 50.8 ms on 4,096 instances, most of whose points are noise).
template <int D, bool F32, bool KEY64>
__global__ void __launch_bounds__(kBorderThreads, kBorderMinBlocks) k_border_point(const gdl::Bufs B, int64_t n) {
  using St = Stencil<D>;
  // per thread and axis: squared largest / smallest distance terms to the five
  // cell slabs at offsets -2..2
  __shared__ float2 slt[D][5][kBorderThreads];
  __shared__ unsigned long long siw[2 * St::ROWS][kBorderThreads];
  __shared__ uint32_t sie[2 * St::ROWS][kBorderThreads];
  const int lane = threadIdx.x & 31;
  const int LB = B.Bi->LB;
  // this dimension's part of the list: 2D instances' points come first
  const int64_t p3 = B.reps[(int64_t)B.ctr[kCtrCells2D]];
  const int64_t L = (int64_t)*B.lcount;
  const int64_t L2 = p3 < n ? (int64_t)bit_rank(B.lbits, B.lpre, p3) : L;
  const int64_t jlo = D == 2 ? 0 : L2, jhi = D == 2 ? L2 : L;
  WalkCursor wc = walk_cursor<D>(B, jlo, jhi, 32);
  Tally t;
  while (wc.advance(lane)) {
    const int64_t j = jlo + wc.next + lane;
    const bool valid = wc.next + lane < wc.end;
    wc.next += 32;
    int m = -1;
    bool over = false;
    if (valid) {
      const int64_t i = (int64_t)B.blist[j];
      m = cell_of(B, i);
      const CellCtx cx = cell_ctx<KEY64>(B, m, LB);
      const DevParams& P = *cx.P;
      const PredParams Q = pred_params(P);
      const bool prune = Q.prune != 0;
      const CellXYZ<D> cc = decompose<D>(cx.local, P);
      St st;
      st.init(cc);
      double px[D];
      float pf[D];
      load_point<D, F32>(px, pf, B, i, prune);
      if (prune) {
        float u[D], o[D];
        cell_origin32<D>(cc, P, o);
        frac_pos<D>(pf, o, Q, u);
#pragma unroll
        for (int k = 0; k < D; ++k) {
          uint32_t near = 0;
#pragma unroll
          for (int j = 0; j < 5; ++j) {
            float a2, b2;
            axis_terms(u[k], j - 2, Q, a2, b2);
            slt[k][j][threadIdx.x] = make_float2(a2, b2);
            if (b2 < Q.thr_out) near |= 1u << j;  // the slab is not beyond eps by itself
          }
          st.w5[k] = near << ((cc.c[k] - 2) & (St::SIDE - 1));
        }
      }
      int best = INT_MAX, budget = B.tn_border;
      // the blocks with core cells in the stencil, the own block's row and half first, then
      // their cells
      StencilWords<D> W5;
      W5.init(st.w5);
      int ni = 0;
      uint32_t codes = 0;
      const int home = D == 3 ? ((cc.c[0] >> St::S) - st.b0[0]) * 2 + (cc.c[1] >> St::S) - st.b0[1]
                              : (cc.c[0] >> St::S) - st.b0[0];
      const int hz = (cc.c[D - 1] >> St::S) - st.b0[D - 1];
      for (int tt = 0; tt < St::ROWS; ++tt) {
        const int r = tt ^ home;
        const int64_t row = st.row(r, P);
        if (row < 0) continue;
        uint2 mk[2];
        W5.row(r, mk[0], mk[1]);
        uint32_t e[2];
        block_pair<D>(B, P, m, r, (uint64_t)row, st.b0[D - 1], (mk[0].x | mk[0].y) != 0,
                             (mk[1].x | mk[1].y) != 0, e[0], e[1]);
        unsigned long long w[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) w[h] = e[h] != kNoEnt ? B.ent[e[h]].core & u64_of(mk[h]) : 0ull;
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          const int h = g ^ hz;
          const unsigned long long wh = h ? w[1] : w[0];
          if (wh) {
            siw[ni][threadIdx.x] = wh;
            sie[ni][threadIdx.x] = h ? e[1] : e[0];
            codes |= (uint32_t)(2 * r + h) << (4 * ni);
            ++ni;
          }
        }
      }
      unsigned long long w = 0, occ = 0;
      uint32_t base = 0;
      int d[D], kk = 0;
#pragma unroll
      for (int k = 0; k < D; ++k) d[k] = 0;
      while (!over) {
        if (!w) {
          if (kk == ni) break;
          const EntHead a = ent_head(B, sie[kk][threadIdx.x]);
          const int code = (int)(codes >> (4 * kk)) & 7;
          w = siw[kk][threadIdx.x];
          ++kk;
          if ((int)a.lo >= best) {  // none of its clusters can improve on the best so far
            w = 0;
            continue;
          }
          occ = a.occ;
          base = a.base;
          d[0] = st.off0(cc, 0) + 2 + ((D == 3 ? code >> 2 : code >> 1) << St::S);
          if (D == 3) d[1] = st.off0(cc, 1) + 2 + (((code >> 1) & 1) << St::S);
          d[D - 1] = st.off0(cc, D - 1) + 2 + ((code & 1) << St::S);
        }
        const int bit = __ffsll((long long)w) - 1;
        w &= w - 1;
        const int c = ent_cell(occ, base, bit);
        const int cB = B.cellcid[c];
        if (cB >= best) continue;
        int cls = 0;
        if (prune) {
          float smax = 0.0f, smin = 0.0f;
#pragma unroll
          for (int k = 0; k < D; ++k) {
            const float2 lt = slt[k][d[k] + St::bit_off(bit, k)][threadIdx.x];
            smax += lt.x;
            smin += lt.y;
          }
          cls = smax <= Q.thr_in ? 1 : (smin >= Q.thr_out ? -1 : 0);
        }
        if (cls > 0) {
          best = cB;  // every point of that cell, a core among them, is in reach
        } else if (cls == 0) {
          const int q = B.reps[c], qe = B.reps[c + 1];
          for (int qq = q; qq < qe; ++qq) {
            if (!B.core[qq]) continue;
            if (budget-- == 0) {
              over = true;
              break;
            }
            Cand<D, F32> cd;
            load_cand<D, F32>(cd, B, qq);
            if (pair_test<D, F32>(px, pf, cd, B, qq, i, false, Q, t)) {
              best = cB;
              break;
            }
          }
        }
      }
      if (!over) B.lab[i] = best == INT_MAX ? kNoise : best;
    }
    // cells with an undecided point, once per warp
    const unsigned om = __ballot_sync(kFull, over);
    bool lead = false;
    if (over) lead = lane == __ffs(__match_any_sync(om, m)) - 1;
    heavy_push(B, kCtrHeavyBorder, lead, m, 0);
  }
  flush_tally(t, B.ctr);
}

// ------------------------------------------------------------- core flags
// Heavy cells, one warp each: dense cells (>= minpts points) are all core;
// other queued cells stream the points of their stencil's cells (looked up one
// per lane and concatenated, nearest first) 32 at
// a time, one candidate per lane, and every staged point of the cell gets
// __ballot_sync + __popc of the lanes holding a neighbour.  The warp stops as
// soon as every staged point has reached minpts.
template <int D, bool F32, bool KEY64>
__global__ void __launch_bounds__(kCellThreads) k_core_heavy(const gdl::Bufs B, int64_t n) {
  __shared__ WarpStage<D> stage[kWarpsPerBlock];
  __shared__ CellList lists[kWarpsPerBlock];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  WarpStage<D>& S = stage[w];
  CellList& CL = lists[w];
  const int LB = B.Bi->LB;
  int64_t mlo, mhi;
  dim_range<D>(B, mlo, mhi);
  const int64_t W = (int64_t)gridDim.x * kWarpsPerBlock;
  Tally t;
  unsigned long long dense = 0;
  const int64_t H = (int64_t)B.ctr[kCtrHeavyCore];
  for (int64_t h = (int64_t)blockIdx.x * kWarpsPerBlock + w; h < H; h += W) {
    const int64_t m = B.hv_cell[h];
    if (m < mlo || m >= mhi) continue;
    const int b = B.reps[m], e = B.reps[m + 1], sz = e - b;
    const CellCtx cx = cell_ctx<KEY64>(B, m, LB);
    const DevParams& P = *cx.P;
    const PredParams Q = pred_params(P);
    if (sz >= Q.minpts) {
      for (int i = b + lane; i < e; i += 32) B.core[i] = 1;
      if (lane == 0) { B.cellcore[m] = sz; ++dense; }
      continue;
    }
    const CellXYZ<D> cc = decompose<D>(cx.local, P);
    int ncells = 0;
    const int total = build_cells<D, KEY64>(B, CL, cc, P, lane, ncells);
    int ncore = 0;
    for (int c0 = 0; c0 < sz; c0 += 32) {
      const int na = min(32, sz - c0);
      if (lane < na) {
        if (F32) ld_f<D>(B, b + c0 + lane, S.f[lane]);
        else ld_x<D>(B, b + c0 + lane, S.x[lane]);
      }
      __syncwarp();
      int mycnt = 0;
      bool done = false;
      for (int base = 0; base < total && !done; base += 32) {
        const int c = base + lane;
        const bool valid = c < total;
        int q = 0;
        Cand<D, F32> cd;
        if (valid) {
          q = cell_list_pos(CL, ncells, c);
          load_cand<D, F32>(cd, B, q);
        }
        for (int j = 0; j < na; ++j) {
          bool hit = valid && pair_test<D, F32>(S.x[j], S.f[j], cd, B, q, b + c0 + j, true, Q, t);
          unsigned bal = __ballot_sync(kFull, hit);
          if (lane == j) mycnt += __popc(bal);
        }
        done = __all_sync(kFull, lane >= na || mycnt >= Q.minpts);
      }
      const bool isc = lane < na && mycnt >= Q.minpts;
      if (lane < na) B.core[b + c0 + lane] = isc ? 1 : 0;
      ncore += __popc(__ballot_sync(kFull, isc));
      __syncwarp();
    }
    if (lane == 0) B.cellcore[m] = ncore;
  }
  flush_tally(t, B.ctr);
  if (lane == 0 && dense) atomicAdd(B.ctr + kCtrDenseCells, dense);
}

// ------------------------------------------------------------- union-find
// Each core cell's representative (its first core point) and its bit in its
// block's core word, and the mask of the core-cell list (listed in order for the
// union; a word per warp over [0, n)).  The cell whose bit is the block's first
// lists the block (blklist, in no particular order) and clears its link words.
// A round of a thread block takes kCoreCellsU x 256 cells and one atomic for its list
// entries (an atomic per warp, all at one address, bounds such a kernel: about 0.7 ns
// each).
constexpr int kCoreCellsU = 4;
template <bool KEY64>
__global__ void __launch_bounds__(256) k_core_cells(const gdl::Bufs B, int64_t n) {
  const int64_t M = *B.M;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __shared__ uint32_t s_cnt[32];
  __shared__ unsigned long long s_at;
  const int64_t per = 256 * kCoreCellsU;
  // words of the mask beyond the cells are cleared before the launch
  for (int64_t r0 = blockIdx.x * per; r0 < M; r0 += gridDim.x * per) {
    unsigned news[kCoreCellsU];
#pragma unroll
    for (int u = 0; u < kCoreCellsU; ++u) {
      const int64_t m0 = r0 + (w * kCoreCellsU + u) * 32, m = m0 + lane;
      const bool f = m < M && B.cellcore[m] > 0;
      bool fresh = false;
      if (f) {
        int q = B.reps[m];
        while (!B.core[q]) ++q;
        B.cellrep[m] = q;
        B.compmin[m] = (int)B.ids[q];  // the sort is stable: its smallest core index
        const uint32_t e = B.cellent[m];
        fresh = atomicOr(&B.ent[e].core, 1ull << ((unsigned)ckey_at<KEY64>(B, m) & 63u)) == 0;
        if (fresh) B.links[e] = BlockLinks{};
      }
      const unsigned bl = __ballot_sync(kFull, f);
      if (lane == 0 && m0 < M) B.lbits[m0 >> 5] = bl;
      news[u] = __ballot_sync(kFull, fresh);
      if (lane == 0) s_cnt[w * kCoreCellsU + u] = (uint32_t)__popc(news[u]);
    }
    __syncthreads();
    if (w == 0) {
      const uint32_t c = s_cnt[lane];
      uint32_t inc = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kFull, inc, o);
        if (lane >= o) inc += v;
      }
      s_cnt[lane] = inc - c;
      if (lane == 31 && inc) s_at = atomicAdd(B.ctr + kCtrBlocks, (unsigned long long)inc);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < kCoreCellsU; ++u)
      if ((news[u] >> lane) & 1u)
        B.blklist[s_at + s_cnt[w * kCoreCellsU + u] + __popc(news[u] & ((1u << lane) - 1u))] =
            (uint32_t)(r0 + (w * kCoreCellsU + u) * 32 + lane);
    __syncthreads();
  }
}

// Union inside blocks, in two steps without a chain to follow: which of a block's
// core cells that share a face are linked through their representatives (in float64
// mode: or because all of the neighbour is in the representative's reach), as one
// word per direction (k_links, a thread per listed core cell), then the connected
// parts of those words by bit floods (k_flood, a thread per block), whose cells get
// the part's first cell as parent.  The union passes then start from blocks mostly
// in one part each, and look for the links that the representatives do not show.
// (A first pass over single cells had spent its time in the finds and hooks of
// these links: C3 0.95 ms.)
template <int D>
struct LinkDirs {
  static constexpr int N = D;
  // the neighbour along axis d: its bit distance, and the places that have it in the block
  static __device__ constexpr int sh(int d) {
    return D == 3 ? (d == 0 ? 16 : d == 1 ? 4 : 1) : (d == 0 ? 8 : 1);
  }
  static __device__ constexpr unsigned long long in(int d) {
    return D == 3 ? (d == 0 ? 0x0000ffffffffffffull
                            : d == 1 ? 0x0fff0fff0fff0fffull : 0x7777777777777777ull)
                  : (d == 0 ? 0x00ffffffffffffffull : 0x7f7f7f7f7f7f7f7full);
  }
};

template <int D, bool F32, bool KEY64>
__global__ void __launch_bounds__(256) k_links(const gdl::Bufs B, int64_t n) {
  using Dir = LinkDirs<D>;
  const int LB = B.Bi->LB;
  const int64_t M2 = (int64_t)B.ctr[kCtrCells2D];
  const int64_t L = (int64_t)*B.lcount;
  const int64_t L2 = M2 < n ? (int64_t)bit_rank(B.lbits, B.lpre, M2) : L;
  const int64_t jlo = D == 2 ? 0 : L2, jhi = D == 2 ? L2 : L;
  Tally t;
  for (int64_t j = jlo + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < jhi;
       j += (int64_t)gridDim.x * blockDim.x) {
    const int a = (int)B.blist[j];
    const uint64_t key = ckey_at<KEY64>(B, a);
    const int bit = (int)key & 63;
    const uint32_t e = B.cellent[a];
    const int qa = B.cellrep[a];
    const EntHead hd = ent_head(B, e);
    const unsigned long long core = ent_tail(B, e).core;
    const DevParams& P = B.Pv[inst_of(key, LB)];
    unsigned has = 0;
    int rq[Dir::N];
#pragma unroll
    for (int d = 0; d < Dir::N; ++d)
      if ((((core >> Dir::sh(d)) & Dir::in(d)) >> bit) & 1ull) {
        has |= 1u << d;
        rq[d] = B.cellrep[ent_cell(hd.occ, hd.base, bit + Dir::sh(d))];
      }
    if (!has) continue;
    unsigned hit = 0;
    if constexpr (F32) {
      float f[D];
      ld_f<D>(B, qa, f);
#pragma unroll
      for (int d = 0; d < Dir::N; ++d)
        if ((has >> d) & 1u) {
          float g[D];
          ld_f<D>(B, rq[d], g);
          ++t.t32;
          if (dist2_f32<D>(f, g) < P.eps2_lo32) hit |= 1u << d;
        }
    } else {
      if (P.prune) {
        const PredParams Q = pred_params(P);
        float o[D], f[D], u[D];
        cell_origin32<D>(decompose<D>(key & P.kmask, P), P, o);
        ld_f<D>(B, qa, f);
        frac_pos<D>(f, o, Q, u);
#pragma unroll
        for (int d = 0; d < Dir::N; ++d)
          if (classify<D>(u, d == 0, d == 1, d == 2, Q) > 0) hit |= 1u << d;
        hit &= has;
      }
      if (hit != has) {
        double x[D];
        ld_x<D>(B, qa, x);
#pragma unroll
        for (int d = 0; d < Dir::N; ++d)
          if (((has & ~hit) >> d) & 1u) {
            double y[D];
            ld_x<D>(B, rq[d], y);
            ++t.t64;
            if (d2_le(dist2_f64<D>(x, y), P.eps2_in)) hit |= 1u << d;
          }
      }
    }
#pragma unroll
    for (int d = 0; d < Dir::N; ++d)
      if ((hit >> d) & 1u) atomicOr(&B.links[e].w[d][bit >> 5], 1u << (bit & 31));
  }
  flush_tally(t, B.ctr);
}

__global__ void k_flood(const gdl::Bufs B) {
  const int64_t M2 = (int64_t)B.ctr[kCtrCells2D];
  const int64_t NBk = (int64_t)B.ctr[kCtrBlocks];
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < NBk;
       j += (int64_t)gridDim.x * blockDim.x) {
    const int mc = (int)B.blklist[j];  // a cell of the block
    const uint32_t e = B.cellent[mc];
    const EntHead hd = ent_head(B, e);
    unsigned long long left = B.ent[e].core;
    const unsigned long long occ = hd.occ;
    const int m0 = (int)hd.base;
    const BlockLinks lk = B.links[e];
    uint32_t uni = kNoEnt;
    unsigned long long l[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) l[d] = (unsigned long long)lk.w[d][1] << 32 | lk.w[d][0];
    const bool two = m0 < M2;
    const int s0 = two ? LinkDirs<2>::sh(0) : LinkDirs<3>::sh(0);
    const int s1 = two ? LinkDirs<2>::sh(1) : LinkDirs<3>::sh(1);
    while (left) {
      unsigned long long part = left & (0ull - left), before;
      const int root = ent_cell(occ, (uint32_t)m0, __ffsll((long long)part) - 1);
      do {
        before = part;
        part |= (part & l[0]) << s0 | ((part >> s0) & l[0]);
        part |= (part & l[1]) << s1 | ((part >> s1) & l[1]);
        part |= (part & l[2]) << 1 | ((part >> 1) & l[2]);  // (3D; no bits in 2D)
      } while (part != before);
      left &= ~part;
      uni = uni == kNoEnt ? (uint32_t)root : kMixedRoot;
      for (unsigned long long w = part; w; w &= w - 1)
        B.parent[ent_cell(occ, (uint32_t)m0, __ffsll((long long)w) - 1)] = root;
    }
    B.ent[e].uni = uni;
  }
}

// Heavy link searches, one warp per queued cell A: for each still-open
// half-stencil neighbour B (pass 0: offsets within +-1, pass 1: the rest) whose
// core points are in another component, look for one core-core pair that are
// neighbours both ways (warp_link_rows) and unite the two cells.  (Two blocks per SM leave room
// for the search without spills: two crowds of 8,000 points, float32 mode, 350 -> 327 ms.)
template <int D, bool F32, bool KEY64>
__global__ void __launch_bounds__(kCellThreads, 2)
k_union_heavy(const gdl::Bufs B, int64_t n, int pass) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int LB = B.Bi->LB;
  int64_t mlo, mhi;
  dim_range<D>(B, mlo, mhi);
  const int64_t W = (int64_t)gridDim.x * kWarpsPerBlock;
  const OffTab& T = kHalf[D - 2][pass];
  Tally t;
  const int64_t H = (int64_t)B.ctr[kCtrHeavyUnion];
  for (int64_t h = (int64_t)blockIdx.x * kWarpsPerBlock + w; h < H; h += W) {
    const int64_t m = B.hv_cell[h];
    if (m < mlo || m >= mhi) continue;
    const unsigned long long open = B.hv_mask[h];
    const int b = B.reps[m];
    const int e = B.reps[m + 1];
    const CellCtx cx = cell_ctx<KEY64>(B, m, LB);
    const DevParams& P = *cx.P;
    const PredParams Q = pred_params(P);
    const CellXYZ<D> cc = decompose<D>(cx.local, P);
    float oA[D];
    if (Q.prune) cell_origin32<D>(cc, P, oA);
    for (int t0 = 0; t0 < T.n; t0 += 32) {
      const int tt = t0 + lane;
      bool cand = false;
      int bB = 0, eB = 0, cB = 0;
      if (tt < T.n && ((open >> tt) & 1ull)) {
        const int c = find_cell<D, KEY64>(B, P, (int64_t)cc.c[0] + T.o[tt][0],
                                          (int64_t)cc.c[1] + T.o[tt][1],
                                          (int64_t)cc.c[2] + T.o[tt][2]);
        if (c >= 0) {
          cB = c;
          bB = B.reps[c];
          eB = B.reps[c + 1];
          cand = B.cellcore[cB] > 0 && uf_find(B.parent, cB) != uf_find(B.parent, (int)m);
        }
      }
      unsigned mask = __ballot_sync(kFull, cand);
      while (mask) {
        const int src = __ffs(mask) - 1;
        mask &= mask - 1;
        const int cbB = __shfl_sync(kFull, bB, src);
        const int ceB = __shfl_sync(kFull, eB, src);
        const int ccB = __shfl_sync(kFull, cB, src);
        if (uf_find(B.parent, (int)m) == uf_find(B.parent, ccB)) continue;
        const signed char* ob = T.o[t0 + src];
        const int o[3] = {ob[0], ob[1], ob[2]};
        bool found = false;
        for (int a = b; a < e && !found; a += 32)
          found = warp_link_rows<D, F32>(B, a, min(32, e - a), cbB, ceB, oA, o, Q, t);
        if (found && lane == 0) uf_union(B.parent, (int)m, ccB);
        __syncwarp();
      }
    }
  }
  flush_tally(t, B.ctr);
}

// Merge replay for one-directional core links.  Components of the symmetric
// core graph are what the reference's sequential expansion produces when every
// core-core neighbour relation is mutual.  When core a has core b in its
// neighbourhood but not the reverse (the query box and the distance test can
// disagree in the last bit), the reference's scan (dbscan_rtree_exp.cpp:363-404)
// lets the cluster that expands a swallow b's component if that component is
// still unvisited -- which depends on the order clusters open.  This kernel
// replays exactly that order over the few components touched by such links:
// components in order of their smallest core index; each unassigned one opens
// a cluster that absorbs every unassigned component reachable along directed
// links.  Absorbed roots are re-parented under the opening root.  One thread;
// the list holds at most kAsymCap links (more is reported as an error).
// cell(q): the cell of sorted position q.
template <class F>
__device__ void asym_resolve(const gdl::Bufs& B, AsymWork& W, F&& cell) {
  const int* __restrict__ cellmin = B.compmin;  // per root: the component's smallest core index
  int* parent = B.parent;
  const int* __restrict__ asym_list = B.asym;
  unsigned long long E = B.ctr[kCtrAsymEdges];
  if (E == 0) return;
  if (E > (unsigned long long)kAsymCap) return;  // reported by the host
  int *from = W.from, *to = W.to, *node = W.node, *assigned = W.assigned;
  int ne = 0, nv = 0;
  for (unsigned long long i = 0; i < E; ++i) {
    int a = asym_list[2 * i], b = asym_list[2 * i + 1];
    int ra = uf_find(parent, cell(a));
    int rb = uf_find(parent, cell(b));
    if (ra == rb) continue;
    from[ne] = ra;
    to[ne] = rb;
    ++ne;
    int r2[2] = {ra, rb};
    for (int k = 0; k < 2; ++k) {
      bool seen = false;
      for (int v = 0; v < nv && !seen; ++v) seen = node[v] == r2[k];
      if (!seen) node[nv++] = r2[k];
    }
  }
  // order the components by smallest core index (insertion sort, small)
  for (int i = 1; i < nv; ++i) {
    int x = node[i], j = i - 1;
    while (j >= 0 && cellmin[node[j]] > cellmin[x]) { node[j + 1] = node[j]; --j; }
    node[j + 1] = x;
  }
  // links as indices into the ordered node list
  for (int e = 0; e < ne; ++e) {
    int fi = 0, ti = 0;
    for (int u = 0; u < nv; ++u) {
      if (node[u] == from[e]) fi = u;
      if (node[u] == to[e]) ti = u;
    }
    from[e] = fi;
    to[e] = ti;
  }
  for (int v = 0; v < nv; ++v) assigned[v] = -1;
  for (int v = 0; v < nv; ++v) {
    if (assigned[v] >= 0) continue;
    assigned[v] = node[v];
    // grow the opened cluster along directed links until nothing changes
    bool grew = true;
    while (grew) {
      grew = false;
      for (int e = 0; e < ne; ++e) {
        if (assigned[from[e]] == node[v] && assigned[to[e]] < 0) {
          assigned[to[e]] = node[v];
          grew = true;
        }
      }
    }
  }
  for (int v = 0; v < nv; ++v)
    if (assigned[v] != node[v]) parent[node[v]] = assigned[v];
}

__global__ void k_asym_resolve(const gdl::Bufs B) {
  __shared__ AsymWork W;
  if (threadIdx.x == 0 && blockIdx.x == 0)
    asym_resolve(B, W, [&](int q) { return cell_of(B, q); });
}

// parent[m] <- root (full path compression).  slot[D] (for the cells of that
// dimension, -1: none): the word of each block's entry (0: lo, 1: hi) that gets
// the block's root when all its core cells have the same one, kMixedRoot when not,
// for the next union pass (one atomic per run of lanes of one block).
__global__ void k_compress(const gdl::Bufs B, int slot2, int slot3) {
  const int64_t M = *B.M, M2 = (int64_t)B.ctr[kCtrCells2D];
  const int lane = threadIdx.x & 31;
  for (int64_t m0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); m0 < M;
       m0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = m0 + lane;
    const bool on = m < M && B.cellcore[m] > 0;
    int r = 0;
    uint32_t e = 0;
    if (on) {
      r = uf_find(B.parent, (int)m);
      B.parent[m] = r;
      e = B.cellent[m];
    }
    const int slot = m < M2 ? slot2 : slot3;
    const bool mk = on && slot >= 0;
    const unsigned grp = run_peers(__ballot_sync(kFull, mk), (int)e);
    if (mk) {
      const unsigned lo = __reduce_min_sync(grp, (unsigned)r), hi = __reduce_max_sync(grp, (unsigned)r);
      if (lane == __ffs(grp) - 1) {
        uint32_t* u = slot == 0 ? &B.ent[e].lo : &B.ent[e].hi;
        uint32_t old = lo == hi ? atomicCAS(u, kNoEnt, lo) : kMixedRoot;
        if (old != kNoEnt && old != lo) atomicExch(u, kMixedRoot);
      }
    }
  }
}

// The smallest core index of every component, kept at its root (compmin starts as
// every core cell's own).  Roots are the cells of smallest index; most cells find a
// smaller value already in place, so few atomics are left.
__global__ void k_comp_min(const gdl::Bufs B) {
  const int64_t M = *B.M;
  const int lane = threadIdx.x & 31;
  for (int64_t m0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); m0 < M;
       m0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = m0 + lane;
    const bool on = m < M && B.cellcore[m] > 0;
    int r = 0;
    if (on) {
      r = uf_find(B.parent, (int)m);
      B.parent[m] = r;
    }
    const bool sub = on && r != (int)m;
    const unsigned grp = run_peers(__ballot_sync(kFull, sub), r);
    if (sub) {
      const int mn = (int)__reduce_min_sync(grp, (unsigned)B.compmin[m]);
      if (lane == __ffs(grp) - 1 && mn < *reinterpret_cast<volatile int*>(B.compmin + r))
        atomicMin(B.compmin + r, mn);
    }
  }
}

// every root marks its component's smallest core index (a bit over global
// point indices; cluster numbers are the ranks of these bits)
__global__ void k_roots(const gdl::Bufs B) {
  const int64_t M = *B.M;
  for (int64_t m = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; m < M;
       m += (int64_t)gridDim.x * blockDim.x) {
    BlockEnt& E = B.ent[B.cellent[m]];
    if (E.base == (uint32_t)m) E.lo = INT_MAX;  // smallest cluster id, set by k_cell_ids
    if (B.cellcore[m] == 0) continue;
    if (uf_find(B.parent, (int)m) == (int)m) {
      const uint32_t cm = (uint32_t)B.compmin[m];
      atomicOr(B.fbits + (cm >> 5), 1u << (cm & 31));
    }
  }
}

// Per cell: the cluster id of its core points (the rank of its root's mark,
// less the marks of the instances before it: cluster numbers restart at 0 in
// every instance), INT_MAX without core points.
// Each block's smallest id goes to its entry (one atomic per run of lanes of
// one block).
template <bool KEY64>
__global__ void k_cell_ids(const gdl::Bufs B) {
  const int LB = B.Bi->LB;
  const int64_t M = *B.M;
  const int lane = threadIdx.x & 31;
  for (int64_t m0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); m0 < M;
       m0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t m = m0 + lane;
    int cid = INT_MAX;
    uint32_t e = 0;
    const bool on = m < M && B.cellcore[m] > 0;
    if (on) {
      const DevParams& P = B.Pv[inst_of(ckey_at<KEY64>(B, m), LB)];
      const int64_t root_min = B.compmin[uf_find(B.parent, (int)m)];
      cid = (int)(bit_rank(B.fbits, B.fpre, root_min) - bit_rank(B.fbits, B.fpre, P.pt_off));
      e = B.cellent[m];
    }
    if (m < M) B.cellcid[m] = cid;
    const unsigned grp = run_peers(__ballot_sync(kFull, on), (int)e);
    if (on) {
      const unsigned mn = __reduce_min_sync(grp, (unsigned)cid);
      if (lane == __ffs(grp) - 1) atomicMin(&B.ent[e].lo, mn);
    }
  }
}

// The mask of the border-search list: every non-core point (listed in sorted
// order afterwards, so neighbouring list entries are neighbouring points, 2D
// instances' first), a word per warp.
__global__ void k_label(const gdl::Bufs B, int64_t n) {
  const int lane = threadIdx.x & 31;
  // four groups of 32 points per warp and pass, their loads issued together
  constexpr int U = 4;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t g0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); g0 < n;
       g0 += U * stride) {
    uint8_t c[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = g0 + u * stride + lane;
      c[u] = i < n ? B.core[i] : (uint8_t)1;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i0 = g0 + u * stride;
      if (i0 >= n) break;  // warp-uniform
      const unsigned nc = __ballot_sync(kFull, !c[u]);
      if (lane == 0) B.lbits[i0 >> 5] = nc;
    }
  }
}

// Border points: one warp per cell with non-core points (only non-dense cells
// have any).  Each staged non-core point takes the smallest cluster id among
// the cells whose core points have it in their neighbourhood (centre = the core
// point, as the reference's expansion queries from the core point).  Lanes look
// the stencil cells up in parallel; cells whose cluster id cannot improve any
// staged point are skipped.
template <int D, bool F32, bool KEY64>
__global__ void __launch_bounds__(kCellThreads) k_border_heavy(const gdl::Bufs B, int64_t n) {
  __shared__ WarpStage<D> stage[kWarpsPerBlock];
  __shared__ int sIdx[kWarpsPerBlock][32];
  const int LB = B.Bi->LB;
  int64_t mlo, mhi;
  dim_range<D>(B, mlo, mhi);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  WarpStage<D>& S = stage[w];
    const int64_t W = (int64_t)gridDim.x * kWarpsPerBlock;
  const OffTab& T = kFullSt[D - 2];
  Tally t;
  const int64_t H = (int64_t)B.ctr[kCtrHeavyBorder];
  for (int64_t h = (int64_t)blockIdx.x * kWarpsPerBlock + w; h < H; h += W) {
    const int64_t m = B.hv_cell[h];
    if (m < mlo || m >= mhi) continue;
    const int b = B.reps[m], e = B.reps[m + 1];
    const CellCtx cx = cell_ctx<KEY64>(B, m, LB);
    const DevParams& P = *cx.P;
    const PredParams Q = pred_params(P);
    const CellXYZ<D> cc = decompose<D>(cx.local, P);
    for (int c0 = b; c0 < e; c0 += 32) {
      // stage this chunk's non-core points
      const int i = c0 + lane;
      const bool nc = i < e && !B.core[i];
      const unsigned ncm = __ballot_sync(kFull, nc);
      const int na = __popc(ncm);
      if (na == 0) continue;
      if (nc) {
        const int slot = __popc(ncm & ((1u << lane) - 1u));
        sIdx[w][slot] = i;
        if (F32) ld_f<D>(B, i, S.f[slot]);
        else ld_x<D>(B, i, S.x[slot]);
      }
      __syncwarp();
      int best = INT_MAX;  // lane j < na: best cluster of staged point j
      for (int t0 = 0; t0 < T.n; t0 += 32) {
        const int tt = t0 + lane;
        bool has = false;
        int bB = 0, eB = 0, cid = INT_MAX;
        if (tt < T.n) {
          const int c = find_cell<D, KEY64>(B, P, (int64_t)cc.c[0] + T.o[tt][0],
                                            (int64_t)cc.c[1] + T.o[tt][1],
                                            (int64_t)cc.c[2] + T.o[tt][2]);
          if (c >= 0) {
            bB = B.reps[c];
            eB = B.reps[c + 1];
            cid = B.cellcid[c];  // INT_MAX without core points
            has = cid != INT_MAX;
          }
        }
        unsigned mask = __ballot_sync(kFull, has);
        while (mask) {
          const int src = __ffs(mask) - 1;
          mask &= mask - 1;
          const int cB = __shfl_sync(kFull, cid, src);
          const int cbB = __shfl_sync(kFull, bB, src);
          const int ceB = __shfl_sync(kFull, eB, src);
          unsigned wantm = __ballot_sync(kFull, lane < na && cB < best);
          for (int qb = cbB; qb < ceB && wantm; qb += 32) {
            const int q = qb + lane;
            const bool valid = q < ceB && B.core[q];
            Cand<D, F32> c;
            if (valid) load_cand<D, F32>(c, B, q);
            unsigned pending = wantm;
            while (pending) {
              const int j = __ffs(pending) - 1;
              pending &= pending - 1;
              bool hit = valid && pair_test<D, F32>(S.x[j], S.f[j], c, B, q, sIdx[w][j], false, Q, t);
              if (__any_sync(kFull, hit)) {
                if (lane == j) best = cB;
                wantm &= ~(1u << j);
              }
            }
          }
        }
      }
      if (lane < na) B.lab[sIdx[w][lane]] = best == INT_MAX ? kNoise : best;
      __syncwarp();
    }
  }
  flush_tally(t, B.ctr);
}

// labels back to the caller's point order (core points: their cell's cluster;
// the others: the border search's label or NOISE); counts
__global__ void k_scatter_labels(const gdl::Bufs B, int64_t n, int* __restrict__ out,
                                 uint8_t* __restrict__ core_out) {
  unsigned long long nn = 0, nc = 0;
  // four points per thread and pass, in straight-line phases so that each
  // phase's loads are in flight together: ids, core flags, run words; then
  // both candidate labels (the border search's, and the cell's cluster for a
  // core point); then the stores
  constexpr int U = 4;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i0 < n; i0 += U * stride) {
    uint32_t j[U], rb[U], rp[U];
    uint8_t c[U];
    int l[U], lc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = i0 + u * stride < n ? i0 + u * stride : n - 1;
      j[u] = B.ids[i];
      c[u] = B.core[i];
      rb[u] = B.runbits[i >> 5];
      rp[u] = B.runpre[i >> 5];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = i0 + u * stride < n ? i0 + u * stride : n - 1;
      const int m = (int)(rp[u] + (uint32_t)__popc(rb[u] & (0xffffffffu >> (31 - (i & 31))))) - 1;
      l[u] = B.lab[i];
      lc[u] = B.cellcid[m];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (i0 + u * stride >= n) continue;
      const int lab = c[u] ? lc[u] : l[u];
      out[j[u]] = lab;
      if (core_out) core_out[j[u]] = c[u];
      nn += lab == kNoise;
      nc += c[u];
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    nn += __shfl_xor_sync(kFull, nn, o);
    nc += __shfl_xor_sync(kFull, nc, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (nn) atomicAdd(B.ctr + kCtrNoise, nn);
    if (nc) atomicAdd(B.ctr + kCtrCore, nc);
  }
}

// clusters of every instance: the root marks in its range of global indices
__global__ void k_cluster_counts(const gdl::Bufs B, int K, int64_t* out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < K; i += gridDim.x * blockDim.x) {
    const InstDesc I = B.inst[i];
    out[i] = (int64_t)bit_rank(B.fbits, B.fpre, I.pt_off + I.n) -
             (int64_t)bit_rank(B.fbits, B.fpre, I.pt_off);
  }
}

#include "gd_small.cuh"

}  // namespace gd
// ------------------------------------------------------------------ launchers
namespace gdl {

using namespace gd;

static int grid_for(int64_t work, int threads, int sms, int per_sm) {
  int64_t g = (work + threads - 1) / threads;
  int64_t cap = (int64_t)sms * per_sm;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

int grids(const Bufs& B, int K, int nchunks, double mult2, double mult3, uint64_t dense_floor,
          uint64_t dense_per_point, uint64_t rows_floor, cudaStream_t s) {
  k_bbox_init<<<(K + 255) / 256, 256, 0, s>>>(B, K);
  if (nchunks > 0) k_bbox_chunk<<<nchunks, kBboxThreads, 0, s>>>(B);
  k_params_inst<<<(K + 127) / 128, 128, 0, s>>>(B, K, mult2, mult3, dense_floor, dense_per_point,
                                                rows_floor);
  k_layout<<<1, 1024, 0, s>>>(B, K);
  return 3 + (nchunks > 0 ? 1 : 0);
}

int keys(const Bufs& B, bool key64, int nchunks, void* keys_out, cudaStream_t s) {
  if (nchunks <= 0) return 0;
  if (key64)
    k_keys<unsigned long long><<<nchunks, 256, 0, s>>>(B, static_cast<unsigned long long*>(keys_out));
  else
    k_keys<uint32_t><<<nchunks, 256, 0, s>>>(B, static_cast<uint32_t*>(keys_out));
  return 1;
}

int gather(const Bufs& B, bool key64, int64_t n, bool xf, bool one, int sms, cudaStream_t s) {
  const int g = grid_for(n, 256, sms, 8);
  using U64 = unsigned long long;
#define GD_GATHER(KEY, XF)                                                  \
  do {                                                                      \
    if (one) k_gather<KEY, XF, true><<<g, 256, 0, s>>>(B, n);               \
    else k_gather<KEY, XF, false><<<g, 256, 0, s>>>(B, n);                  \
  } while (0)
  if (key64) {
    if (xf) GD_GATHER(U64, true);
    else GD_GATHER(U64, false);
  } else {
    if (xf) GD_GATHER(uint32_t, true);
    else GD_GATHER(uint32_t, false);
  }
#undef GD_GATHER
  return 1;
}

// kernels of one exclusive scan over nw words
static int scan_launches(int64_t nw) { return gdprim::scan_launches(nw); }

// the set bits of B.lbits over [0, n) listed in order into B.blist, their
// count in *B.lcount
static int list_bits(const Bufs& B, int64_t n, void* scan_temp, cudaStream_t s) {
  const int64_t nw = (n + 31) / 32;
  gdprim::list_bits(B.lbits, B.lpre, nw, B.blist, scan_temp, B.lcount, s, B.ctr + kCtrWaitTimeouts);
  return nw > 0 ? 1 : 0;
}

int runs(const Bufs& B, bool key64, int64_t n, void* scan_temp, cudaStream_t s) {
  const int64_t T = (n + kRunTile - 1) / kRunTile;
  using U64 = unsigned long long;
  void* ck = const_cast<void*>(B.ckeys);
  gdprim::LookbackCtl* ctl = gdprim::lb_ctl(scan_temp);
  unsigned long long* st = gdprim::lb_status(scan_temp);
  if (key64)
    k_runs<U64><<<(unsigned)T, kRunThreads, 0, s>>>(B, n, static_cast<U64*>(ck), (unsigned)T, ctl, st);
  else
    k_runs<uint32_t><<<(unsigned)T, kRunThreads, 0, s>>>(B, n, static_cast<uint32_t*>(ck),
                                                         (unsigned)T, ctl, st);
  return 1;
}

int cells(const Bufs& B, bool key64, int64_t n, int sms, cudaStream_t s) {
  const int g = grid_for(n, 256, sms, 8);
  if (key64) k_cells<unsigned long long><<<g, 256, 0, s>>>(B);
  else k_cells<uint32_t><<<g, 256, 0, s>>>(B);
  if (!B.nbr) return 1;
  if (key64) k_neighbors<true><<<g, 256, 0, s>>>(B);
  else k_neighbors<false><<<g, 256, 0, s>>>(B);
  return 2;
}

#define GD_L1(D, f32, key64, KERNEL, GRID, THREADS, ...)                          \
  do {                                                                            \
    if (f32) {                                                                    \
      if (key64) KERNEL<D, true, true><<<GRID, THREADS, 0, s>>>(__VA_ARGS__);     \
      else KERNEL<D, true, false><<<GRID, THREADS, 0, s>>>(__VA_ARGS__);          \
    } else {                                                                      \
      if (key64) KERNEL<D, false, true><<<GRID, THREADS, 0, s>>>(__VA_ARGS__);    \
      else KERNEL<D, false, false><<<GRID, THREADS, 0, s>>>(__VA_ARGS__);         \
    }                                                                             \
  } while (0)

// one launch per dimension present (bit 0: 2D instances, bit 1: 3D instances)
#define GD_LAUNCH_DIMS(dims, f32, key64, KERNEL, GRID, THREADS, ...)              \
  do {                                                                            \
    if ((dims) & 1) GD_L1(2, f32, key64, KERNEL, GRID, THREADS, __VA_ARGS__);     \
    if ((dims) & 2) GD_L1(3, f32, key64, KERNEL, GRID, THREADS, __VA_ARGS__);     \
  } while (0)

static int per_dim(int dims) { return ((dims & 1) ? 1 : 0) + ((dims & 2) ? 1 : 0); }

int core(const Bufs& B, int64_t n, int dims, bool f32, bool key64, bool one, bool fresh, int sms,
         void* scan_temp, cudaStream_t s) {
  cudaMemsetAsync(B.ctr + kCtrHeavyCore, 0, 8, s);
  cudaMemsetAsync(B.cellcore, 0, (size_t)B.cells * 4, s);  // per-cell core counts
  // dense cells at once; the other points listed in sorted order for the walk
  const int g = grid_for(n, 256, sms, 8);
  const int chunk = f32 ? kCoreChunk : 1;
  if (B.pop) {
    if (key64) k_core_filter<true><<<g, 256, 0, s>>>(B);
    else k_core_filter<false><<<g, 256, 0, s>>>(B);
  }
  if (key64) {
    if (one) k_core_split<true, true><<<g, 256, 0, s>>>(B, n, chunk, fresh ? 0 : 1);
    else k_core_split<true, false><<<g, 256, 0, s>>>(B, n, chunk, fresh ? 0 : 1);
  } else {
    if (one) k_core_split<false, true><<<g, 256, 0, s>>>(B, n, chunk, fresh ? 0 : 1);
    else k_core_split<false, false><<<g, 256, 0, s>>>(B, n, chunk, fresh ? 0 : 1);
  }
  int L = (B.pop ? 2 : 1) + list_bits(B, n, scan_temp, s);
  cudaMemsetAsync(B.ctr + kCtrWalkCursor2, 0, 16, s);
  // 3D walks split after pass 0 (the 3^3 shell)
  if (dims & 2) cudaMemsetAsync(B.fbits, 0, (size_t)B.nw * 4, s);
  auto walk = [&](auto dim, int q0, int q1) {
    constexpr int D = decltype(dim)::value;
    if (f32) {
      const int grid = sms * kCoreCellMinBlocks;
      if (key64) k_core_cell<D, true><<<grid, kCoreThreads, 0, s>>>(B, n, q0, q1);
      else k_core_cell<D, false><<<grid, kCoreThreads, 0, s>>>(B, n, q0, q1);
    } else {
      const int grid = sms * kCoreMinBlocks;
      if (key64) k_core_point<D, true><<<grid, kCoreThreads, 0, s>>>(B, n, q0, q1);
      else k_core_point<D, false><<<grid, kCoreThreads, 0, s>>>(B, n, q0, q1);
    }
  };
  if (dims & 1) walk(std::integral_constant<int, 2>{}, 0, 2);
  if (dims & 2) {
    walk(std::integral_constant<int, 3>{}, 0, 1);
    // the undecided 3D points, listed in sorted order
    gdprim::list_bits(B.fbits, B.fpre, B.nw, B.blist, scan_temp, B.lcount, s,
                      B.ctr + kCtrWaitTimeouts);
    cudaMemsetAsync(B.ctr + kCtrWalkCursor3, 0, 8, s);
    walk(std::integral_constant<int, 3>{}, 1, 2);
    L += 2;
  }
  GD_LAUNCH_DIMS(dims, f32, key64, k_core_heavy, sms * 8, kCellThreads, B, n);
  return L + 2 * per_dim(dims);
}

int unite(const Bufs& B, int64_t n, int dims, bool f32, bool key64, int sms, void* scan_temp,
          cudaStream_t s) {
  cudaMemsetAsync(B.lbits, 0, (size_t)B.nw * 4, s);
  cudaMemsetAsync(B.ctr + kCtrBlocks, 0, 8, s);
  if (key64) k_core_cells<true><<<grid_for(n, 256 * kCoreCellsU, sms, 8), 256, 0, s>>>(B, n);
  else k_core_cells<false><<<grid_for(n, 256 * kCoreCellsU, sms, 8), 256, 0, s>>>(B, n);
  int L = 1 + list_bits(B, n, scan_temp, s);
  const int lgrid = grid_for(n, 256, sms, 8);
  GD_LAUNCH_DIMS(dims, f32, key64, k_links, lgrid, 256, B, n);
  k_flood<<<grid_for(n, 128, sms, 16), 128, 0, s>>>(B);
  L += per_dim(dims) + 1;
  int launched = 0;
  for (int pass = 0; pass < kUnionPasses; ++pass) {
    // the dimensions that have this pass
    const int pd = dims & ((pass < union_passes(2) ? 1 : 0) | (pass < union_passes(3) ? 2 : 0));
    if (!pd) continue;
    cudaMemsetAsync(B.ctr + kCtrHeavyUnion, 0, 8, s);
    cudaMemsetAsync(B.ctr + kCtrWalkCursor2, 0, 16, s);
    GD_LAUNCH_DIMS(pd, f32, key64, k_union_scan, sms * 8, kScanThreadsPerBlock, B, n, pass);
    GD_LAUNCH_DIMS(pd, f32, key64, k_union_heavy, sms * 8, kCellThreads, B, n, pass);
    // every parent to its root: the next pass then finds most neighbours in
    // A's set from one load (parent[q] == A's root).  After the last pass the
    // root marks and cluster ids find their roots themselves.
    const bool last = pass == kUnionPasses - 1 ||
                      !(dims & ((pass + 1 < union_passes(2) ? 1 : 0) |
                                (pass + 1 < union_passes(3) ? 2 : 0)));
    // (the entries' word for pass 1 is lo, for pass 2 hi)
    if (!last)
      k_compress<<<grid_for(n, 256, sms, 8), 256, 0, s>>>(B, pass + 1 < union_passes(2) ? pass : -1,
                                                          pass + 1 < union_passes(3) ? pass : -1);
    launched += 2 * per_dim(pd) + (last ? 0 : 1);
  }
  k_comp_min<<<grid_for(n, 256, sms, 8), 256, 0, s>>>(B);
  k_asym_resolve<<<1, 32, 0, s>>>(B);
  return L + launched + 2;
}

int roots(const Bufs& B, bool key64, int64_t n, int sms, void* scan_temp, cudaStream_t s) {
  cudaMemsetAsync(B.fbits, 0, (size_t)(B.nwf + 1) * 4, s);
  k_roots<<<grid_for(n, 256, sms, 8), 256, 0, s>>>(B);
  // total clusters into the small block (read with the counters)
  gdprim::exclusive_scan_popc(B.fbits, B.fpre, B.nwf, scan_temp, B.K, s, B.ctr + kCtrWaitTimeouts);
  if (key64) k_cell_ids<true><<<grid_for(n, 256, sms, 8), 256, 0, s>>>(B);
  else k_cell_ids<false><<<grid_for(n, 256, sms, 8), 256, 0, s>>>(B);
  return 2 + scan_launches(B.nwf);
}

int label(const Bufs& B, int64_t n, int sms, void* scan_temp, cudaStream_t s) {
  k_label<<<grid_for(n, 256, sms, 8), 256, 0, s>>>(B, n);
  return 1 + list_bits(B, n, scan_temp, s);
}

int border(const Bufs& B, int64_t n, int dims, bool f32, bool key64, int sms, cudaStream_t s) {
  cudaMemsetAsync(B.ctr + kCtrHeavyBorder, 0, 8, s);
  cudaMemsetAsync(B.ctr + kCtrWalkCursor2, 0, 16, s);
  GD_LAUNCH_DIMS(dims, f32, key64, k_border_point, sms * kBorderMinBlocks, kBorderThreads, B, n);
  GD_LAUNCH_DIMS(dims, f32, key64, k_border_heavy, sms * 8, kCellThreads, B, n);
  return 2 * per_dim(dims);
}

int scatter_labels(const Bufs& B, int64_t n, int* out, uint8_t* core_out, int sms,
                   cudaStream_t s) {
  k_scatter_labels<<<grid_for(n, 256, sms, 8), 256, 0, s>>>(B, n, out, core_out);
  return 1;
}

// blocks of a small run's kernels: one resident block per SM at most
static int small_grid(int64_t lanes, int sms) {
  const int64_t g = (lanes + kSmallThreads - 1) / kSmallThreads;
  return (int)(g < 1 ? 1 : (g > sms ? sms : g));
}

cudaError_t small_index(const Bufs& B, const SmallArgs& A, int sms, cudaStream_t s) {
  void* args[] = {const_cast<Bufs*>(&B), const_cast<SmallArgs*>(&A)};
  const void* f = A.dim == 2 ? (const void*)k_small_index<2> : (const void*)k_small_index<3>;
  return cudaLaunchCooperativeKernel(f, dim3(small_grid(A.n, sms)), dim3(kSmallThreads), args, 0, s);
}

cudaError_t small_expand(const Bufs& B, const SmallArgs& A, bool f32, int minpts, int* out, int sms,
                         cudaStream_t s) {
  void* args[] = {const_cast<Bufs*>(&B), const_cast<SmallArgs*>(&A), &minpts, &out};
  const void* f = A.dim == 2
                      ? (f32 ? (const void*)k_small_expand<2, true> : (const void*)k_small_expand<2, false>)
                      : (f32 ? (const void*)k_small_expand<3, true> : (const void*)k_small_expand<3, false>);
  const int G = A.dim == 2 ? SmallWalk<2>::G : SmallWalk<3>::G;
  return cudaLaunchCooperativeKernel(f, dim3(small_grid((int64_t)A.n * G, sms)), dim3(kSmallThreads),
                                     args, (size_t)B.nwf * 4, s);
}

int small_points(const Bufs& B, int n, int dim, double* out, int sms, cudaStream_t s) {
  k_small_points<<<grid_for(n, 256, sms, 8), 256, 0, s>>>(B, n, dim, out);
  return 1;
}

int small_scatter(const Bufs& B, int n, int* out, uint8_t* core_out, int sms, cudaStream_t s) {
  k_small_scatter<<<grid_for(n, 256, sms, 8), 256, 0, s>>>(B, n, out, core_out);
  return 1;
}

int cluster_counts(const Bufs& B, int K, int64_t* out, cudaStream_t s) {
  k_cluster_counts<<<(K + 255) / 256, 256, 0, s>>>(B, K, out);
  return 1;
}

}  // namespace gdl
