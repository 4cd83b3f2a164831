// gd_small.cuh -- one small instance in two cooperative kernels (included by
// gd_pipeline.cu, namespace gd).
//
// A small instance spends its time in launches and in dependent loads, not in work:
// the general pipeline's 40 launches took 0.33 of the 0.39 ms of a 1,000-point run.
// Here the index build is one kernel and the expand another, their phases separated
// by grid-wide barriers (about 1 us each), and every stencil walk takes a group of
// lanes -- one lane per block of the stencil, 4 in 2D and 8 in 3D -- so that a walk's
// chain of loads is a quarter or an eighth as long.
//
// The index needs no sort: points set their cell's bit in their block's occupancy
// word, each occupied block then takes a run of cell numbers from a counter, points
// take their place in their cell from the cell's counter, and each cell takes a run
// of positions from another.  Cells of a block are consecutive and in bit order, as
// the walks need; the order of blocks, and of points in a cell, is whatever the
// counters gave, which no label depends on.  Blocks are found directly (one entry per
// block) where there are few, else by a hash of block keys.
//
// Both kernels are launched cooperatively (every block resident), so the barrier's
// waits end; they are still bounded, and one that gives up makes its block leave and
// is reported (kCtrWaitTimeouts): the host then takes the general path.


constexpr unsigned kBarrierPolls = 1u << 25;  // 2 s of sleep, about 15 s with the loads

// All blocks of the launch; false when the wait gave up (the block must leave).
__device__ __forceinline__ bool grid_barrier(const SmallArgs& A, unsigned long long* timeouts) {
  if (gridDim.x == 1) {
    __syncthreads();
    return true;
  }
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    unsigned gen;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(gen) : "l"(A.bar + 1) : "memory");
    __threadfence();
    if (atomicAdd(A.bar, 1u) == gridDim.x - 1u) {
      A.bar[0] = 0;
      __threadfence();
      asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(A.bar + 1), "r"(gen + 1u) : "memory");
    } else {
      ok = 0;
      for (unsigned it = 0; it < kBarrierPolls; ++it) {
        unsigned g;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(g) : "l"(A.bar + 1) : "memory");
        if (g != gen) {
          ok = 1;
          break;
        }
        if (it > 64) __nanosleep(64);
      }
      if (!ok) atomicAdd(timeouts, 1ull);
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// One lane's share of a counter that the warp's lanes draw on together.
__device__ __forceinline__ uint32_t warp_draw(unsigned long long* c, uint32_t want) {
  const int lane = threadIdx.x & 31;
  uint32_t inc = want;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(kFull, inc, o);
    if (lane >= o) inc += v;
  }
  const uint32_t total = __shfl_sync(kFull, inc, 31);
  unsigned long long at = 0;
  if (lane == 0 && total) at = atomicAdd(c, (unsigned long long)total);
  return (uint32_t)__shfl_sync(kFull, at, 0) + inc - want;
}

// Entry of a block, kNoEnt when outside the grid or (hash) not occupied.
template <int D>
__device__ __forceinline__ uint32_t small_ent(const gdl::Bufs& B, const DevParams& P, int x, int y,
                                              int z) {
  if (x < 0 || x >= P.Bk[0] || y < 0 || y >= P.Bk[1]) return kNoEnt;
  if (D == 3 && (z < 0 || z >= P.Bk[2])) return kNoEnt;
  uint64_t blk = (uint64_t)(unsigned)x * (unsigned)P.Bk[1] + (unsigned)y;
  if (D == 3) blk = blk * (unsigned)P.Bk[2] + (unsigned)z;
  if (P.sparse == 0) return (uint32_t)blk;
  const uint32_t mask = B.hmask;
  uint32_t h = hash_key(blk) & mask;
  for (uint32_t probe = 0; probe <= mask; ++probe) {
    const unsigned long long k = B.hkeys[h];
    if (k == blk) return h;
    if (k == kHashEmpty) break;
    h = (h + 1) & mask;
  }
  return kNoEnt;
}

// ---------------------------------------------------------------- index build
template <int D>
__global__ void __launch_bounds__(kSmallThreads) k_small_index(const gdl::Bufs B, const SmallArgs A) {
  __shared__ DevParams P;
  __shared__ long long s_b[7][kSmallThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int n = A.n, T = gridDim.x * kSmallThreads, t0 = blockIdx.x * kSmallThreads + threadIdx.x;
  unsigned long long* timeouts = B.ctr + kCtrWaitTimeouts;
  {
    // bounds of the block's points
    long long lo[D], hi[D], bad = 0;
#pragma unroll
    for (int k = 0; k < D; ++k) {
      lo[k] = LLONG_MAX;
      hi[k] = LLONG_MIN;
    }
    for (int l = t0; l < n; l += T)
#pragma unroll
      for (int k = 0; k < D; ++k) {
        const double x = A.coords[(int64_t)l * D + k];
        bad |= (__double_as_longlong(x) & 0x7ff0000000000000LL) == 0x7ff0000000000000LL;
        const long long o = ord_of(x);
        lo[k] = min(lo[k], o);
        hi[k] = max(hi[k], o);
      }
    bad = __any_sync(kFull, bad != 0);
#pragma unroll
    for (int k = 0; k < D; ++k) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        lo[k] = min(lo[k], __shfl_xor_sync(kFull, lo[k], o));
        hi[k] = max(hi[k], __shfl_xor_sync(kFull, hi[k], o));
      }
      if (lane == 0) {
        s_b[k][w] = lo[k];
        s_b[3 + k][w] = hi[k];
      }
    }
    if (lane == 0) s_b[6][w] = bad;
    __syncthreads();
    if (threadIdx.x < 7 && (threadIdx.x == 6 || threadIdx.x % 3 < D)) {
      const int k = threadIdx.x;
      long long v = s_b[k][0];
      for (int j = 1; j < kSmallThreads / 32; ++j)
        v = k < 3 ? min(v, s_b[k][j]) : max(v, s_b[k][j]);
      A.part[blockIdx.x * 8 + k] = v;
    }
  }
  if (!grid_barrier(A, timeouts)) return;
  // every block: the same bounds, the same grid
  if (w < 7 && (w == 6 || w % 3 < D)) {
    long long v = w < 3 ? LLONG_MAX : LLONG_MIN;
    for (int j = lane; j < (int)gridDim.x; j += 32) {
      const long long x = A.part[j * 8 + w];
      v = w < 3 ? min(v, x) : max(v, x);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const long long x = __shfl_xor_sync(kFull, v, o);
      v = w < 3 ? min(v, x) : max(v, x);
    }
    if (lane == 0) s_b[w][0] = v;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
    for (int k = 0; k < D; ++k) {
      lo[k] = dbl_of(s_b[k][0]);
      hi[k] = dbl_of(s_b[3 + k][0]);
    }
    const InstDesc I{0, n, 0, A.eps, D, 1};
    fill_params(P, I, 0, lo, hi, A.mult, A.direct_max, 0, 0);
    int fl = P.flags | (s_b[6][0] > 0 ? kFlagNonFinite : 0) |
             (P.cell_bits > 62 ? kFlagGridTooLarge : 0);
    if (P.sparse != 0) {
      P.sparse = 1;
      if (A.hash_slots == 0) fl |= kFlagNotSmall;
    }
    P.flags = fl;
    P.LB = P.key_bits;
    P.kmask = P.LB >= 64 ? ~0ull : (1ull << P.LB) - 1ull;
    if (blockIdx.x == 0) {
      B.Pv[0] = P;
      BatchInfo bi{};
      bi.K = 1;
      bi.LB = P.LB;
      bi.flags = fl;
      bi.max_dim = D;
      bi.K2 = D == 2 ? 1 : 0;
      bi.any_xf = 1;
      bi.band_off = !(P.eps2_lo32 > 0.0f);
      bi.grid_cells = P.sparse == 0 ? P.NB << kBlockBits : 0;
      bi.any_sparse = P.sparse == 1;
      *B.Bi = bi;
    }
  }
  __syncthreads();
  if (P.flags & (kFlagNonFinite | kFlagGridTooLarge | kFlagNotSmall)) return;  // (every block)
  const uint32_t ents = P.sparse == 0 ? (uint32_t)P.NB : A.hash_slots;
  for (uint32_t e = t0; e < ents; e += T) {
    B.ent[e] = BlockEnt{};
    if (P.sparse) B.hkeys[e] = kHashEmpty;
  }
  if (!grid_barrier(A, timeouts)) return;
  // cells: occupancy bits
  for (int l = t0; l < n; l += T) {
    int c[3] = {0, 0, 0};
#pragma unroll
    for (int k = 0; k < D; ++k)
      c[k] = cell_of_coord(A.coords[(int64_t)l * D + k], P.key_fast != 0, P.lo[k], P.inv_f,
                           P.key_lo32[k], P.key_inv32, P.key_band, (int)(P.G[k] - 1));
    const uint64_t key = key_of_cell(D, c, P.Bk[1], P.Bk[2]);
    const uint64_t blk = key >> kBlockBits;
    uint32_t e = (uint32_t)blk;
    if (P.sparse) {
      const uint32_t mask = B.hmask;
      uint32_t h = hash_key(blk) & mask;
      e = 0;
      for (uint32_t probe = 0; probe <= mask; ++probe) {  // more slots than points: one is free
        const unsigned long long prev = atomicCAS(B.hkeys + h, kHashEmpty, (unsigned long long)blk);
        if (prev == kHashEmpty || prev == blk) {
          e = h;
          break;
        }
        h = (h + 1) & mask;
      }
    }
    const unsigned long long bit = 1ull << (key & 63);
    if (!(*reinterpret_cast<volatile unsigned long long*>(&B.ent[e].occ) & bit))
      atomicOr(&B.ent[e].occ, bit);
    A.ptkey[l] = (uint64_t)e << kBlockBits | (key & 63);
  }
  if (!grid_barrier(A, timeouts)) return;
  // cell numbers: a run per block
  for (uint32_t e0 = t0 - lane; e0 < ents; e0 += T) {
    const uint32_t e = e0 + lane;
    unsigned long long occ = e < ents ? B.ent[e].occ : 0ull;
    uint32_t m = warp_draw(B.ctr + kCtrCells, (uint32_t)__popcll(occ));
    if (!occ) continue;
    BlockEnt E{};
    E.occ = occ;
    E.base = m;
    B.ent[e] = E;
    for (; occ; occ &= occ - 1, ++m) {
      A.cellkey[m] = (uint64_t)e << kBlockBits | (unsigned)(__ffsll((long long)occ) - 1);
      B.cellcore[m] = 0;
    }
  }
  if (!grid_barrier(A, timeouts)) return;
  // places in the cells
  for (int l = t0; l < n; l += T) {
    const uint64_t k = A.ptkey[l];
    const EntHead h = ent_head(B, (uint32_t)(k >> kBlockBits));
    const int m = ent_cell(h.occ, h.base, (int)(k & 63));
    A.ptcell[l] = (uint32_t)m;
    A.ptpos[l] = (uint32_t)atomicAdd(B.cellcore + m, 1);
  }
  if (!grid_barrier(A, timeouts)) return;
  // positions: a run per cell
  const int M = (int)*reinterpret_cast<volatile unsigned long long*>(B.ctr + kCtrCells);
  for (int m0 = t0 - lane; m0 < M; m0 += T) {
    const int m = m0 + lane;
    const uint32_t len = m < M ? (uint32_t)B.cellcore[m] : 0u;
    const uint32_t at = warp_draw(B.ctr + kCtrBlocks, len);
    if (m < M) A.crange[m] = make_uint2(at, at + len);
  }
  if (!grid_barrier(A, timeouts)) return;
  // sorted points
  for (int l = t0; l < n; l += T) {
    const uint32_t m = A.ptcell[l];
    const int64_t i = A.crange[m].x + A.ptpos[l];
    B.ids[i] = (uint32_t)l;
    A.pcell[i] = m;
    double x[3];
    float f[3];
#pragma unroll
    for (int k = 0; k < D; ++k) {
      x[k] = A.coords[(int64_t)l * D + k];
      B.X[i * D + k] = x[k];
      f[k] = __double2float_rn(__dsub_rn(x[k], P.centre[k]));
    }
    if (D == 2) reinterpret_cast<float2*>(B.Xf)[i] = make_float2(f[0], f[1]);
    else reinterpret_cast<float4*>(B.Xf)[i] = make_float4(f[0], f[1], f[2], 0.0f);
  }
}

// --------------------------------------------------------------------- expand
// A lane's part of a cell's stencil: one block (first-axis half, [middle-axis half,]
// last-axis half by lane).
template <int D>
struct SmallWalk {
  using St = Stencil<D>;
  static constexpr int G = D == 3 ? 8 : 4;  // lanes per group
  CellXYZ<D> cc;
  int half[D];
  St st;
  uint32_t e;
  // cell given by its key (entry << 6 | place) and its entry's block coordinates
  __device__ __forceinline__ void init(const gdl::Bufs& B, const DevParams& P, uint64_t ck, int g) {
    const uint32_t own = (uint32_t)(ck >> kBlockBits);
    const uint64_t blk = P.sparse == 0 ? own : B.hkeys[own];
    cc = decompose<D>(blk << kBlockBits | (ck & 63), P);
    st.init(cc);
    half[0] = D == 3 ? g >> 2 : g >> 1;
    if (D == 3) half[1] = (g >> 1) & 1;
    half[D - 1] = g & 1;
    e = small_ent<D>(B, P, st.b0[0] + half[0], st.b0[1] + half[1], D == 3 ? st.b0[D - 1] + half[D - 1] : 0);
  }
  // this block's cells of the stencil w[] (per-axis sets as Stencil::w5)
  __device__ __forceinline__ unsigned long long mask(const uint32_t* w) const {
    StencilWords<D> W;
    W.init(w);
    const uint32_t yz = (D == 3 ? (half[1] ? W.y[1] : W.y[0]) : ~0u) & (half[D - 1] ? W.z[1] : W.z[0]);
    return (unsigned long long)((half[0] ? W.xh[1] : W.xh[0]) & yz) << 32 |
           ((half[0] ? W.xl[1] : W.xl[0]) & yz);
  }
  // offset along axis k of the block's cell at `bit` from the cell
  __device__ __forceinline__ int off(int bit, int k) const {
    return st.off0(cc, k) + (half[k] << St::S) + St::bit_off(bit, k);
  }
  // mask of this group's lanes
  static __device__ __forceinline__ unsigned group() {
    return (G == 8 ? 0xffu : 0xfu) << ((threadIdx.x & 31) & ~(G - 1));
  }
};

// ---- link searches that a lane does not finish.  A lane of the union spends at most
// kSmallLinkTests tests on a cell pair, and none on a crowded one (crowded_pair): two crowded
// cells that are apart by a little more than eps would otherwise keep one lane busy for |A| |B|
// tests while every other block waits at the barrier.  The cells with open pairs are listed with
// those pairs as a mask (offsets of the step's half stencil) and searched after the barrier, a
// warp per cell; pairs of more than kSmallWarpPairs point pairs
// then by a block each, and those of more than kSmallBlockPairs by the whole grid, one after the
// other.  (Two crowds of 5,000 points each, 1.1 eps apart, float64, whole call: 0.70 ms in 2D
// and 0.79 in 3D; 20,000 each: 6.4 and 8.6.  The general path's warp per pair: 0.25 and 0.32 s;
// 4.8 and 6.1 s.)
// The lists lie in buffers of the index build that are free by now: each cell's mask in ptkey,
// the listed cells in ptcell (each once per step), large pairs in ptpos, n / 2 of them: the
// blocks' in its first 3 n / 8, the grid's behind them; a warp searches a pair itself where there
// is no room.  The grid's cells have more than 1,024 points on one side; there are at most
// n / 1025 of those, each in at most 124 pairs (62 in each half of the 3D stencil): below n / 8.
constexpr long long kSmallWarpPairs = 1ll << 14, kSmallBlockPairs = 1ll << 20;
__host__ __device__ constexpr int small_block_cap(int n) { return n / 2 - n / 8; }
__host__ __device__ constexpr int small_grid_cap(int n) { return n / 8; }

constexpr int kShell3 = make_half(3, 1).n;
static_assert(kShell3 + make_half(3, 2).n <= 64 && make_half(2, 1).n <= 64, "a mask per step");

// Index of an offset among the step's half stencil (step 0: pass 0; step 1: the others).
template <int D>
__device__ __forceinline__ int small_open_bit(int step, int ox, int oy, int oz) {
  const int ax = max(abs(ox), max(abs(oy), abs(oz)));
  if (step == 0) return half_bit<D>(0, ox, oy, oz);
  return D == 3 && ax > 1 ? kShell3 + half_bit<D>(2, ox, oy, oz) : half_bit<D>(1, ox, oy, oz);
}

// two cells' roots equal (one answer for the warp)
__device__ __forceinline__ bool small_same(const gdl::Bufs& B, int a, int b) {
  int same = 0;
  if ((threadIdx.x & 31) == 0) same = uf_find(B.parent, a) == uf_find(B.parent, b);
  return __shfl_sync(kFull, same, 0) != 0;
}

// The listed cells' open pairs, a warp per cell.
template <int D, bool F32>
__device__ __noinline__ void small_link_cells(const gdl::Bufs& B, const SmallArgs& A,
                                              const DevParams& P, int step, int listed,
                                              unsigned long long* nbig) {
  constexpr int S = block_shift<D>(), SM = (1 << S) - 1;
  const int lane = threadIdx.x & 31;
  const int W = gridDim.x * (kSmallThreads / 32);
  const PredParams Q = pred_params(P);
  uint2* big = reinterpret_cast<uint2*>(A.ptpos);
  const int n0 = kHalf[D - 2][step].n, n1 = step == 0 ? 0 : kHalf[D - 2][2].n;
  Tally t;
  for (int h = blockIdx.x * (kSmallThreads / 32) + (threadIdx.x >> 5); h < listed; h += W) {
    const int m = (int)A.ptcell[h];
    const unsigned long long open = A.ptkey[m];
    __syncwarp();
    if (lane == 0) A.ptkey[m] = 0;  // for the next step
    const uint64_t ck = A.cellkey[m];
    const uint32_t own = (uint32_t)(ck >> kBlockBits);
    const uint64_t blk = P.sparse == 0 ? own : B.hkeys[own];
    const CellXYZ<D> cc = decompose<D>(blk << kBlockBits | (ck & 63), P);
    const uint2 ra = A.crange[m];
    float oA[D];
    if (Q.prune) cell_origin32<D>(cc, P, oA);
    for (int t0 = 0; t0 < n0 + n1; t0 += 32) {
      const int tt = t0 + lane;
      int c = -1;
      uint2 rb = make_uint2(0, 0);
      if (tt < n0 + n1 && ((open >> tt) & 1ull)) {
        const signed char* o = tt < n0 ? kHalf[D - 2][step].o[tt] : kHalf[D - 2][2].o[tt - n0];
        const int x = cc.c[0] + o[0], y = cc.c[1] + o[1], z = cc.c[2] + o[2];
        const EntHead e = ent_head(B, small_ent<D>(B, P, x >> S, y >> S, D == 3 ? z >> S : 0));
        const int bit = D == 3 ? (x & SM) << (2 * S) | (y & SM) << S | (z & SM)
                               : (x & SM) << S | (y & SM);
        if ((e.occ >> bit) & 1ull) {
          c = ent_cell(e.occ, e.base, bit);
          rb = A.crange[c];
        }
      }
      for (unsigned mask = __ballot_sync(kFull, c >= 0); mask; mask &= mask - 1) {
        const int src = __ffs(mask) - 1, k = t0 + src;
        const int cb = __shfl_sync(kFull, c, src);
        const int b0 = (int)__shfl_sync(kFull, rb.x, src), b1 = (int)__shfl_sync(kFull, rb.y, src);
        if (small_same(B, m, cb)) continue;
        const long long tests = (long long)(ra.y - ra.x) * (b1 - b0);
        if (tests > kSmallWarpPairs) {
          const bool grid = tests > kSmallBlockPairs;
          int room = 0;
          if (lane == 0) {
            const unsigned long long at = atomicAdd(nbig + (grid ? 1 : 0), 1ull);
            room = at < (unsigned long long)(grid ? small_grid_cap(A.n) : small_block_cap(A.n));
            if (room)
              big[(grid ? small_block_cap(A.n) : 0) + at] = make_uint2((uint32_t)m, (uint32_t)cb);
          }
          if (__shfl_sync(kFull, room, 0)) continue;
        }
        const signed char* ob = k < n0 ? kHalf[D - 2][step].o[k] : kHalf[D - 2][2].o[k - n0];
        const int o[3] = {ob[0], ob[1], ob[2]};
        bool found = false;
        for (int a = (int)ra.x; a < (int)ra.y && !found; a += 32)
          found = warp_link_rows<D, F32>(B, a, min(32, (int)ra.y - a), b0, b1, oA, o, Q, t);
        if (found && lane == 0) uf_union(B.parent, m, cb);
        __syncwarp();
      }
    }
  }
  flush_tally(t, B.ctr);
}

// A large pair: a warp (w of W) per point of the first cell.
template <int D, bool F32>
__device__ __forceinline__ void small_link_pair(const gdl::Bufs& B, const SmallArgs& A, uint2 pair,
                                                int w, int W, const PredParams& Q, Tally& t) {
  const int m = (int)pair.x, c = (int)pair.y;
  const uint2 ra = A.crange[m], rb = A.crange[c];
  for (int a = (int)ra.x + w; a < (int)ra.y; a += W) {
    if (!B.core[a]) continue;
    if (small_same(B, m, c)) break;
    if (warp_link_row<D, F32>(B, a, (int)rb.x, (int)rb.y, Q, t)) {
      if ((threadIdx.x & 31) == 0) uf_union(B.parent, m, c);
      __syncwarp();
      break;
    }
  }
}

// The large pairs: a block each, then the whole grid.
template <int D, bool F32>
__device__ __noinline__ void small_link_big(const gdl::Bufs& B, const SmallArgs& A,
                                            const DevParams& P, const unsigned long long* nbig) {
  constexpr int NW = kSmallThreads / 32;
  const int w = threadIdx.x >> 5;
  const PredParams Q = pred_params(P);
  const uint2* big = reinterpret_cast<const uint2*>(A.ptpos);
  const int nb = (int)min(nbig[0], (unsigned long long)small_block_cap(A.n));
  const int ng = (int)min(nbig[1], (unsigned long long)small_grid_cap(A.n));
  Tally t;
  for (int p = blockIdx.x; p < nb; p += gridDim.x)
    small_link_pair<D, F32>(B, A, big[p], w, NW, Q, t);
  for (int p = 0; p < ng; ++p)
    small_link_pair<D, F32>(B, A, big[small_block_cap(A.n) + p], blockIdx.x * NW + w,
                            gridDim.x * NW, Q, t);
  flush_tally(t, B.ctr);
}

// ---- points with many open candidates, a warp each.  A group of 4 or 8 lanes tests them a
// lane per block, one per step: a point beside a crowded cell would keep one lane busy for
// thousands of steps, and the warp with it.  (260,000 2D points in clumps with spreads from
// 0.01 to 20 at eps 0.5, float64, minPts 4, whole call: 3.43 ms, so 0.75.)
// Neighbours of point i (sorted position), counted up to minpts.
template <int D, bool F32>
__device__ __noinline__ int small_count_point(const gdl::Bufs& B, const SmallArgs& A,
                                              const DevParams& P, int i, int minpts) {
  using W = SmallWalk<D>;
  const int lane = threadIdx.x & 31;
  const PredParams Q = pred_params(P);
  const bool prune = Q.prune != 0;
  const int m = (int)A.pcell[i];
  const uint2 own = A.crange[m];
  int cnt = (int)(own.y - own.x);
  double px[D];
  float pf[D], u[D];
  load_point<D, F32>(px, pf, B, i, prune);
  Tally t;
  for (int g = 0; g < W::G && cnt < minpts; ++g) {
    W wk;
    wk.init(B, P, A.cellkey[m], g);
    if (prune) {
      float o[D];
      cell_origin32<D>(wk.cc, P, o);
      frac_pos<D>(pf, o, Q, u);
    }
    const EntHead h = ent_head(B, wk.e);
    for (unsigned long long v = h.occ & wk.mask(wk.st.w5); v && cnt < minpts; v &= v - 1) {
      const int bit = __ffsll((long long)v) - 1;
      const int c = ent_cell(h.occ, h.base, bit);
      if (c == m) continue;
      const int cls = prune ? classify<D>(u, wk.off(bit, 0), wk.off(bit, 1),
                                          D == 3 ? wk.off(bit, D - 1) : 0, Q) : 0;
      if (cls < 0) continue;
      const uint2 r = A.crange[c];
      if (cls > 0) {
        cnt += (int)(r.y - r.x);
        continue;
      }
      for (uint32_t q0 = r.x; q0 < r.y && cnt < minpts; q0 += 32) {
        const uint32_t q = q0 + lane;
        bool hit = false;
        if (q < r.y) {
          Cand<D, F32> cd;
          load_cand<D, F32>(cd, B, q);
          hit = pair_test<D, F32>(px, pf, cd, B, q, i, true, Q, t);
        }
        cnt += __popc(__ballot_sync(kFull, hit));
      }
    }
  }
  flush_tally(t, B.ctr);
  return cnt;
}

// Smallest cluster id below `best` among the cells whose core points have point i in their
// neighbourhood, else `best`.
template <int D, bool F32>
__device__ __noinline__ int small_border_point(const gdl::Bufs& B, const SmallArgs& A,
                                               const DevParams& P, int i, int best) {
  using W = SmallWalk<D>;
  const int lane = threadIdx.x & 31;
  const PredParams Q = pred_params(P);
  const bool prune = Q.prune != 0;
  const int m = (int)A.pcell[i];
  double px[D];
  float pf[D], u[D];
  load_point<D, F32>(px, pf, B, i, prune);
  Tally t;
  for (int g = 0; g < W::G; ++g) {
    W wk;
    wk.init(B, P, A.cellkey[m], g);
    if (wk.e == kNoEnt) continue;
    if (prune) {
      float o[D];
      cell_origin32<D>(wk.cc, P, o);
      frac_pos<D>(pf, o, Q, u);
    }
    const EntHead h = ent_head(B, wk.e);
    for (unsigned long long v = ent_tail(B, wk.e).core & wk.mask(wk.st.w5); v; v &= v - 1) {
      const int bit = __ffsll((long long)v) - 1;
      const int c = ent_cell(h.occ, h.base, bit);
      const int cB = B.cellcid[c];
      if (cB >= best) continue;
      const int cls = prune ? classify<D>(u, wk.off(bit, 0), wk.off(bit, 1),
                                          D == 3 ? wk.off(bit, D - 1) : 0, Q) : 0;
      if (cls < 0) continue;
      bool in = cls > 0;
      const uint2 r = A.crange[c];
      for (uint32_t q0 = r.x; q0 < r.y && !in; q0 += 32) {
        const uint32_t q = q0 + lane;
        bool hit = false;
        if (q < r.y && B.core[q]) {
          Cand<D, F32> cd;
          load_cand<D, F32>(cd, B, q);
          hit = pair_test<D, F32>(px, pf, cd, B, q, i, false, Q, t);
        }
        in = __any_sync(kFull, hit);
      }
      if (in) best = cB;
    }
  }
  flush_tally(t, B.ctr);
  return best;
}

// Two blocks' registers fit an SM, so that runs on different streams do not wait for each
// other's end (100,000 2D points, 4 threads with a context each: 7,600 runs a second, with one
// block per SM, which needs no spills, 5,300; one thread: 4,030 and 4,140).
template <int D, bool F32>
__global__ void __launch_bounds__(kSmallThreads, 2)
k_small_expand(const __grid_constant__ gdl::Bufs B, const __grid_constant__ SmallArgs A, int minpts,
               int* __restrict__ out) {
  using W = SmallWalk<D>;
  __shared__ DevParams P;
  extern __shared__ uint32_t s_pre[];  // prefix counts of the cluster marks
  __shared__ uint32_t s_warp[32];
  const int lane = threadIdx.x & 31, g = lane & (W::G - 1);
  const unsigned grp = W::group();
  const int n = A.n, T = gridDim.x * kSmallThreads, t0 = blockIdx.x * kSmallThreads + threadIdx.x;
  const int gT = T / W::G, g0 = t0 / W::G;
  unsigned long long* timeouts = B.ctr + kCtrWaitTimeouts;
  for (int k = threadIdx.x; k < (int)(sizeof(DevParams) / 4); k += kSmallThreads)
    reinterpret_cast<uint32_t*>(&P)[k] = reinterpret_cast<const uint32_t*>(B.Pv)[k];
  __syncthreads();
  if (P.flags & (kFlagNonFinite | kFlagGridTooLarge | kFlagNotSmall)) return;  // (every block)
  // a wait of the index build gave up: cells, ids and places may be an earlier call's
  __shared__ int s_off;
  if (threadIdx.x == 0) {
    s_off = *reinterpret_cast<volatile unsigned long long*>(timeouts) != 0;
    P.minpts = minpts;
  }
  __syncthreads();
  if (s_off) return;
  const PredParams Q = pred_params(P);
  const bool prune = Q.prune != 0;
  const int M = (int)B.ctr[kCtrCells];
  const int nwf = (int)B.nwf;
  Tally t;
  // ---- cells and marks cleared; the points outside dense cells listed
  for (int m = t0; m < M; m += T) {
    const uint2 r = A.crange[m];
    B.cellcore[m] = (int)(r.y - r.x) >= minpts ? (int)(r.y - r.x) : 0;
    B.cellmin[m] = INT_MAX;
    B.parent[m] = m;
    A.ptkey[m] = 0;  // no link search open
    B.ent[A.cellkey[m] >> kBlockBits].core = 0;
  }
  for (int k = t0; k < nwf; k += T) B.fbits[k] = 0;
  if (t0 < 4) B.ctr[kCtrSmallPairs + t0] = 0;
  for (int i0 = t0 - lane; i0 < n; i0 += T) {
    const int i = i0 + lane;
    bool walk = false;
    if (i < n) {
      const uint2 r = A.crange[A.pcell[i]];
      walk = (int)(r.y - r.x) < minpts;
    }
    const uint32_t at = warp_draw(B.ctr + kCtrWalkCursor2, walk ? 1u : 0u);
    if (walk) A.list[at] = (uint32_t)i;
  }
  if (!grid_barrier(A, timeouts)) return;
  const int L = (int)*reinterpret_cast<volatile unsigned long long*>(B.ctr + kCtrWalkCursor2);
  // ---- core flags: dense cells' points at once, then a group per listed point.
  // Each lane classifies its block's cells; where the group's sure neighbours and
  // open candidates leave the decision open, the lanes test their candidates one
  // per step, the warp's groups in step together, until the group's count or its
  // candidates decide.
  for (int i = t0; i < n; i += T) {
    const int m = (int)A.pcell[i];
    const uint2 r = A.crange[m];
    if ((int)(r.y - r.x) < minpts) continue;
    B.core[i] = 1;
    if (i == (int)r.x) atomicAdd(B.ctr + kCtrDenseCells, 1ull);
    const int id = (int)B.ids[i];
    if (id < *reinterpret_cast<volatile int*>(B.cellmin + m)) atomicMin(B.cellmin + m, id);
  }
  for (int j0 = (t0 - lane) / W::G; j0 < L; j0 += gT) {
    const int j = j0 + lane / W::G;
    const bool valid = j < L;
    const int i = valid ? (int)A.list[j] : 0;
    int m = 0, add = 0, open = 0;
    double px[D];
    float pf[D];
    unsigned long long w = 0;  // open cells
    EntHead h{0, 0, 0};
    int own = 0;
    if (valid) {
      m = (int)A.pcell[i];
      const uint2 r = A.crange[m];
      own = (int)(r.y - r.x);
      W wk;
      wk.init(B, P, A.cellkey[m], g);
      float u[D];
      load_point<D, F32>(px, pf, B, i, prune);
      if (prune) {
        float o[D];
        cell_origin32<D>(wk.cc, P, o);
        frac_pos<D>(pf, o, Q, u);
      }
      h = ent_head(B, wk.e);
      for (unsigned long long v = h.occ & wk.mask(wk.st.w5); v; v &= v - 1) {
        const int bit = __ffsll((long long)v) - 1;
        const int c = ent_cell(h.occ, h.base, bit);
        if (c == m) continue;
        const int cls = prune ? classify<D>(u, wk.off(bit, 0), wk.off(bit, 1),
                                            D == 3 ? wk.off(bit, D - 1) : 0, Q) : 0;
        if (cls < 0) continue;
        const uint2 q = A.crange[c];
        if (cls > 0) {
          add += (int)(q.y - q.x);
        } else {
          w |= 1ull << bit;
          open += (int)(q.y - q.x);
        }
      }
    }
#pragma unroll
    for (int o = W::G / 2; o > 0; o >>= 1) {
      add += __shfl_xor_sync(kFull, add, o);
      open += __shfl_xor_sync(kFull, open, o);
    }
    int cnt = own + add;
    const bool undecided = valid && cnt < minpts && cnt + open >= minpts;
    // (the whole group)
    const bool heavy = undecided && open > (F32 ? kSmallPointTests32 : kSmallPointTests);
    bool more = undecided && !heavy && w != 0;
    uint32_t q = 0, qe = 0;
    while (true) {
      bool hit = false;
      if (more) {
        if (q == qe) {
          const uint2 r = A.crange[ent_cell(h.occ, h.base, __ffsll((long long)w) - 1)];
          w &= w - 1;
          q = r.x;
          qe = r.y;
        }
        Cand<D, F32> cd;
        load_cand<D, F32>(cd, B, q);
        hit = pair_test<D, F32>(px, pf, cd, B, q, i, true, Q, t);
        ++q;
      }
      cnt += __popc(__ballot_sync(kFull, hit) & grp);
      more = more && cnt < minpts && (q < qe || w != 0);
      if (!__any_sync(kFull, more)) break;
    }
    for (unsigned hv = __ballot_sync(kFull, heavy && g == 0); hv; hv &= hv - 1) {
      const int src = __ffs(hv) - 1;
      const int c = small_count_point<D, F32>(B, A, P, __shfl_sync(kFull, i, src), minpts);
      if (src == (lane & ~(W::G - 1))) cnt = c;
    }
    if (valid && g == 0) {
      const bool isc = cnt >= minpts;
      B.core[i] = isc ? 1 : 0;
      if (isc) {
        atomicAdd(B.cellcore + m, 1);
        const int id = (int)B.ids[i];
        if (id < *reinterpret_cast<volatile int*>(B.cellmin + m)) atomicMin(B.cellmin + m, id);
      }
    }
  }
  if (!grid_barrier(A, timeouts)) return;
  // ---- core words, each core cell's representative (its first core point)
  for (int m = t0; m < M; m += T) {
    if (B.cellcore[m] == 0) continue;
    B.compmin[m] = B.cellmin[m];
    uint32_t q = A.crange[m].x;
    while (!B.core[q]) ++q;
    A.cellrep[m] = q;
    const uint64_t k = A.cellkey[m];
    atomicOr(&B.ent[k >> kBlockBits].core, 1ull << (k & 63));
  }
  if (!grid_barrier(A, timeouts)) return;
  // ---- union, a group per core cell: first the near neighbours (pass 0 of the
  // half stencil), then, from compressed parents, the others, most of which settle
  // from one parent load.  Pairs that pass a lane's budget follow after the barrier.
  for (int step = 0; step < 2; ++step) {
    unsigned long long* nopen = B.ctr + (step == 0 ? kCtrHeavyCore : kCtrHeavyUnion);
    unsigned long long* nbig = B.ctr + kCtrSmallPairs + 2 * step;
    for (int m = g0; m < M; m += gT) {
      if (B.cellcore[m] == 0) continue;  // (the whole group)
      const uint64_t ck = A.cellkey[m];
      unsigned long long w = kPassMasks[D - 2].m[0][ck & 63][g];
      if (step > 0) {
        w = 0;
        for (int ps = 1; ps < union_passes(D); ++ps) w |= kPassMasks[D - 2].m[ps][ck & 63][g];
      }
      if (!w) continue;
      W wk;
      wk.init(B, P, ck, g);
      if (wk.e == kNoEnt) continue;
      w &= ent_tail(B, wk.e).core;
      if (!w) continue;
      const EntHead h = ent_head(B, wk.e);
      const int ra0 = *reinterpret_cast<volatile int*>(B.parent + m);
      if (step > 0) {
        // parents four at a time; one equal to A's settles the cell
        unsigned long long slow = 0;
        while (w) {
          int bit[4], pr[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            bit[k] = w ? __ffsll((long long)w) - 1 : -1;
            w &= w - 1;
            pr[k] = bit[k] >= 0
                        ? *reinterpret_cast<volatile int*>(B.parent + ent_cell(h.occ, h.base, bit[k]))
                        : ra0;
          }
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (pr[k] != ra0) slow |= 1ull << bit[k];
        }
        w = slow;
        if (!w) continue;
      }
      const uint2 r = A.crange[m];
      Cand<D, F32> ca;
      load_cand<D, F32>(ca, B, A.cellrep[m]);
      const bool single = B.cellcore[m] == 1;
      float oA[D];
      if (prune) cell_origin32<D>(wk.cc, P, oA);
      while (w) {
        const int bit = __ffsll((long long)w) - 1;
        w &= w - 1;
        const int c = ent_cell(h.occ, h.base, bit);
        if (step > 0 && uf_find(B.parent, m) == uf_find(B.parent, c)) continue;
        // the representatives first, then the search
        Cand<D, F32> cd;
        load_cand<D, F32>(cd, B, A.cellrep[c]);
        bool linked, apart;
        if (F32) {
          ++t.t32;
          const float s2 = dist2_f32<D>(ca.f, cd.f);
          linked = s2 < Q.eps2_lo32;
          apart = s2 > Q.eps2_hi32;
        } else {
          ++t.t64;
          const double d2 = dist2_f64<D>(ca.x, cd.x);
          linked = d2_le(d2, Q.eps2_in);
          apart = !d2_le(d2, Q.eps2);
        }
        if (!linked && !(apart && single && B.cellcore[c] == 1)) {
          const uint2 q = A.crange[c];
          const int ox = wk.off(bit, 0), oy = wk.off(bit, 1), oz = D == 3 ? wk.off(bit, D - 1) : 0;
          const int res = crowded_pair((int)(r.y - r.x), (int)(q.y - q.x))
                              ? -1
                              : inline_link<D, F32>(B, n, (int)r.x, (int)r.y, (int)q.x, (int)q.y,
                                                    oA, ox, oy, oz, P, Q, t);
          linked = res > 0;
          if (res < 0 && atomicOr(A.ptkey + m, 1ull << small_open_bit<D>(step, ox, oy, oz)) == 0)
            A.ptcell[atomicAdd(nopen, 1ull)] = (uint32_t)m;
        }
        if (linked) uf_union(B.parent, m, c);
      }
    }
    if (!grid_barrier(A, timeouts)) return;
    const int listed = (int)*reinterpret_cast<volatile unsigned long long*>(nopen);
    if (listed) {
      small_link_cells<D, F32>(B, A, P, step, listed, nbig);
      if (!grid_barrier(A, timeouts)) return;
      const volatile unsigned long long* nb = nbig;
      if (nb[0] + nb[1]) {
        small_link_big<D, F32>(B, A, P, nbig);
        if (!grid_barrier(A, timeouts)) return;
      }
    }
    if (step == 0) {
      for (int m = t0; m < M; m += T)
        if (B.cellcore[m] > 0) B.parent[m] = uf_find(B.parent, m);
      if (!grid_barrier(A, timeouts)) return;
    }
  }
  // ---- components: smallest core index at the root
  for (int m = t0; m < M; m += T) {
    if (B.cellcore[m] == 0) continue;
    const int r = uf_find(B.parent, m), mn = B.cellmin[m];
    if (r != m && mn < *reinterpret_cast<volatile int*>(B.compmin + r)) atomicMin(B.compmin + r, mn);
  }
  if (!grid_barrier(A, timeouts)) return;
  if (*reinterpret_cast<volatile unsigned long long*>(B.ctr + kCtrAsymEdges) != 0) {
    if (t0 == 0) asym_resolve(B, *A.asym, [&](int q) { return (int)A.pcell[q]; });
    if (!grid_barrier(A, timeouts)) return;
  }
  // ---- cluster marks
  for (int m = t0; m < M; m += T) {
    if (B.cellcore[m] == 0) continue;
    if (uf_find(B.parent, m) == m) {
      const uint32_t cm = (uint32_t)B.compmin[m];
      atomicOr(B.fbits + (cm >> 5), 1u << (cm & 31));
    }
  }
  if (!grid_barrier(A, timeouts)) return;
  // ---- cluster numbers: every block ranks the marks for itself
  {
    const int per = (nwf + kSmallThreads - 1) / kSmallThreads;
    const int k0 = threadIdx.x * per, k1 = min(k0 + per, nwf);
    uint32_t sum = 0;
    for (int k = k0; k < k1; ++k) sum += (uint32_t)__popc(B.fbits[k]);
    __shared__ uint32_t s_total;
    uint32_t ex = gdprim::block_excl_scan<kSmallThreads>(sum, s_warp, &s_total);
    for (int k = k0; k < k1; ++k) {
      s_pre[k] = ex;
      ex += (uint32_t)__popc(B.fbits[k]);
    }
    __syncthreads();
    if (t0 == 0) *B.K = s_total;
  }
  for (int m = t0; m < M; m += T) {
    int cid = INT_MAX;
    if (B.cellcore[m] > 0) {
      const uint32_t rm = (uint32_t)B.compmin[uf_find(B.parent, m)];
      cid = (int)(s_pre[rm >> 5] + (uint32_t)__popc(B.fbits[rm >> 5] & ((1u << (rm & 31)) - 1u)));
    }
    B.cellcid[m] = cid;
  }
  if (!grid_barrier(A, timeouts)) return;
  // ---- labels: core points their cell's, the others a border search
  uint32_t noise = 0, ncore = 0;
  for (int i = t0; i < n; i += T) {
    if (!B.core[i]) continue;
    const int best = B.cellcid[A.pcell[i]];
    ++ncore;
    if (out) out[B.ids[i]] = best;
    else B.lab[i] = best;
  }
  for (int j0 = (t0 - lane) / W::G; j0 < L; j0 += gT) {
    const int j = j0 + lane / W::G;
    const int i = j < L ? (int)A.list[j] : 0;
    const bool search = j < L && !B.core[i];  // (the whole group)
    int best = INT_MAX, budget = kSmallPointTests;
    bool heavy = false;
    if (search) {
      const int m = (int)A.pcell[i];
      W wk;
      wk.init(B, P, A.cellkey[m], g);
      unsigned long long w = 0;
      EntHead h{0, 0, 0};
      if (wk.e != kNoEnt) w = ent_tail(B, wk.e).core & wk.mask(wk.st.w5);
      if (w) {
        h = ent_head(B, wk.e);
        double px[D];
        float pf[D], u[D];
        load_point<D, F32>(px, pf, B, i, prune);
        if (prune) {
          float o[D];
          cell_origin32<D>(wk.cc, P, o);
          frac_pos<D>(pf, o, Q, u);
        }
        while (w && !heavy) {
          const int bit = __ffsll((long long)w) - 1;
          w &= w - 1;
          const int c = ent_cell(h.occ, h.base, bit);
          const int cB = B.cellcid[c];
          if (cB >= best) continue;
          const int cls = prune ? classify<D>(u, wk.off(bit, 0), wk.off(bit, 1),
                                              D == 3 ? wk.off(bit, D - 1) : 0, Q) : 0;
          if (cls < 0) continue;
          if (cls > 0) {
            best = cB;
            continue;
          }
          const uint2 q = A.crange[c];
          for (uint32_t qq = q.x; qq < q.y; ++qq) {
            if (budget-- == 0) {
              heavy = true;
              break;
            }
            if (!B.core[qq]) continue;
            Cand<D, F32> cd;
            load_cand<D, F32>(cd, B, qq);
            if (pair_test<D, F32>(px, pf, cd, B, qq, i, false, Q, t)) {
              best = cB;
              break;
            }
          }
        }
      }
    }
#pragma unroll
    for (int o = W::G / 2; o > 0; o >>= 1) best = min(best, __shfl_xor_sync(kFull, best, o));
    // (a group's lowest lane stands for it)
    const unsigned hb = __ballot_sync(kFull, heavy);
    for (unsigned hv = __ballot_sync(kFull, g == 0 && (hb & grp)); hv; hv &= hv - 1) {
      const int src = __ffs(hv) - 1;
      const int b = small_border_point<D, F32>(B, A, P, __shfl_sync(kFull, i, src),
                                               __shfl_sync(kFull, best, src));
      if (src == (lane & ~(W::G - 1))) best = b;
    }
    if (search && g == 0) {
      if (best == INT_MAX) best = kNoise;
      noise += best == kNoise;
      if (out) out[B.ids[i]] = best;
      else B.lab[i] = best;
    }
  }
  flush_tally(t, B.ctr);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    noise += __shfl_xor_sync(kFull, noise, o);
    ncore += __shfl_xor_sync(kFull, ncore, o);
  }
  if (lane == 0) {
    if (noise) atomicAdd(B.ctr + kCtrNoise, (unsigned long long)noise);
    if (ncore) atomicAdd(B.ctr + kCtrCore, (unsigned long long)ncore);
  }
}

// labels (and core flags) back to the caller's order, where the expand did not
// write them itself
__global__ void k_small_scatter(const gdl::Bufs B, int n, int* __restrict__ out,
                                uint8_t* __restrict__ core_out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t j = B.ids[i];
    out[j] = B.lab[i];
    if (core_out) core_out[j] = B.core[i];
  }
}

// the points back in the caller's order
__global__ void k_small_points(const gdl::Bufs B, int n, int dim, double* __restrict__ out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int64_t j = B.ids[i];
    for (int k = 0; k < dim; ++k) out[j * dim + k] = B.X[(int64_t)i * dim + k];
  }
}
