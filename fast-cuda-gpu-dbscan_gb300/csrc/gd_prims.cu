// gd_prims.cu -- device primitives: exclusive scan and a stable LSD radix sort.
//
// Scans are single-pass, with decoupled look-back (gd_lookback.cuh).
//
// Scan (u32): tiles of 8192 elements (512 threads x 16 contiguous items), one
// launch (k_scan_onepass): reads 4 B, writes 4 B/elem.  Against the earlier
// reduce / partials / down-sweep kernels it saves two launches per scan (C2:
// union and label phases about 10 us faster each).
// Radix sort (u32 or u64 key, u32 value), 8- or 9-bit digits, tiles of 4096 pairs
// (256 threads x 16 items; each warp owns a contiguous 512-element segment so
// warp-local ranking in item order is stable):
//   k_rs_upsweep     per-tile digit histograms       reads 4 B/pair
//   exclusive scan over the [digit][tile] histogram (k_scan_onepass)
//   k_rs_downsweep   rank in tile, regroup in shared memory, scatter
//                                                    reads 8 B, writes 8 B/pair
// A onesweep variant (one histogram kernel for all passes, per-digit look-back
// in the scatter kernel) was measured slower on C2 (index phase 0.78 -> 0.94
// ms): with about 760 tiles in flight the serial per-digit look-back chains
// cost more than the upsweep and the histogram scan they replace.
// This replaces thrust::sort_by_key (main.cu:332).
#include <algorithm>

#include "gd_internal.cuh"
#include "gd_lookback.cuh"

namespace gdprim {

namespace {

constexpr int kScanThreads = 512;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;

// value of one scanned element: the element itself, or (POPC) the number of
// set bits of a 32-bit word
template <bool POPC>
__device__ __forceinline__ uint32_t scan_val(uint32_t x) {
  return POPC ? (uint32_t)__popc(x) : x;
}

// Single-pass exclusive scan (decoupled look-back).
template <bool POPC>
__global__ void __launch_bounds__(kScanThreads)
k_scan_onepass(const uint32_t* in, uint32_t* out, int64_t n, unsigned tiles, LookbackCtl* ctl,
               unsigned long long* status, uint32_t* total_dev, unsigned long long* timeouts) {
  __shared__ uint32_t s_warp[32];
  __shared__ unsigned s_tile, s_epoch;
  __shared__ uint32_t s_agg, s_excl;
  lb_begin(ctl, &s_tile, &s_epoch);
  const unsigned tile = s_tile, epoch = s_epoch;
  const uint32_t tag = lb_tag(epoch);
  if (tile >= tiles) {
    // a counter left inconsistent (never expected): no tile, report it
    if (threadIdx.x == 0 && timeouts) atomicAdd(timeouts, 1ull);
    lb_end(ctl, tiles, epoch);
    return;
  }
  const int64_t base = (int64_t)tile * kScanTile + (int64_t)threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  const bool full = base + kScanItems <= n;
  if (full) {
    const uint4* p = reinterpret_cast<const uint4*>(in + base);
#pragma unroll
    for (int q = 0; q < kScanItems / 4; ++q) {
      const uint4 a = p[q];
      v[4 * q] = a.x; v[4 * q + 1] = a.y; v[4 * q + 2] = a.z; v[4 * q + 3] = a.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) v[i] = base + i < n ? in[base + i] : 0u;
  }
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) v[i] = scan_val<POPC>(v[i]);
  uint32_t sum = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) sum += v[i];
  uint32_t ex = block_excl_scan<kScanThreads>(sum, s_warp, &s_agg);
  const uint32_t excl = lb_tile_prefix(status, tile, tag, &s_agg, &s_excl, timeouts);
  if (threadIdx.x == 0 && tile == tiles - 1u && total_dev) *total_dev = excl + s_agg;
  ex += excl;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    uint32_t t = v[i];
    v[i] = ex;
    ex += t;
  }
  if (full) {
    uint4* p = reinterpret_cast<uint4*>(out + base);
#pragma unroll
    for (int q = 0; q < kScanItems / 4; ++q)
      p[q] = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
  } else {
#pragma unroll
    for (int i = 0; i < kScanItems; ++i)
      if (base + i < n) out[base + i] = v[i];
  }
  lb_end(ctl, tiles, epoch);
}

// ---------------------------------------------------------------- radix sort
constexpr int kRsThreads = 256;
constexpr int kRsWarps = kRsThreads / 32;
// tiles from which an upsweep block takes four (a chip's worth of blocks stays: 256)
constexpr int64_t kRsFour = 1024;
constexpr int kRsMaxBins = 512;  // digits of 8 or 9 bits
// items per thread: 16 for 32-bit keys (4096-pair tiles), 8 for 64-bit keys
template <class K>
constexpr int rs_items() { return sizeof(K) == 4 ? 16 : 8; }
// Blocks per SM that the downsweep's registers leave room for, and when it loads its
// values.  32-bit keys: three blocks, the values loaded after the ranking so that they
// arrive during the tile scan (10M pairs, three passes: 193 us; loaded with the keys 202;
// four blocks 198).  64-bit keys, half as many items per thread: five blocks, values
// loaded with the keys (131M pairs, whole index: 16.57 ms; four blocks 16.66, three
// 17.0, late loads 17.2).
template <class K>
constexpr int rs_min_blocks() { return sizeof(K) == 4 ? 3 : 5; }
constexpr int kRsMinTile = kRsThreads * 8;

// A tile's place.  Plain: tile t of T, counts at [digit][tile].  By instance: a chunk of
// one instance holds kChunkPoints / TILE tiles (the last chunk's perhaps empty), and the
// counts lie [instance][digit][tile of the instance], so that their one scan gives every
// instance's pairs their place among its own.
struct RsPlace {
  int64_t base, end;      // pairs [base, end) (the tile's, or more)
  int64_t hist, stride;   // counts of digit d at hist + d * stride
};
template <int TILE, int BINS, bool SEG>
__device__ __forceinline__ RsPlace rs_place(const SortChunks& sc, int64_t tile, int64_t n, int64_t T,
                                            bool first) {
  RsPlace p;
  if constexpr (!SEG) {
    p.base = tile * TILE;
    p.end = n;
    p.hist = tile;
    p.stride = T;
  } else {
    constexpr int TPC = (int)(gd::kChunkPoints / TILE);
    const int64_t ci = tile / TPC;
    const gd::Chunk c = sc.chunks[ci];
    const int64_t sub = tile % TPC, off = c.begin - sc.Pv[c.inst].pt_off;
    const int64_t c0 = ci - off / gd::kChunkPoints;  // the instance's first chunk
    const int64_t b = first ? c.begin : (int64_t)c.sorted;
    p.base = b + sub * TILE;
    p.end = b + (c.end - c.begin);
    p.stride = (sc.Pv[c.inst].n + gd::kChunkPoints - 1) / gd::kChunkPoints * TPC;
    p.hist = c0 * TPC * BINS + (ci - c0) * TPC + sub;
  }
  return p;
}

// A block counts the digits of G consecutive tiles (G | T), so that a digit's counts,
// T apart from the next digit's, leave in one store of G (20M keys, three passes: a
// tile per block 90 us, four 75; 2M keys: 17, but four tiles leave too few blocks, 50).
template <class K, int ITEMS, int RB, int G, bool SEG>
__global__ void __launch_bounds__(kRsThreads)
k_rs_upsweep(const K* __restrict__ keys, int64_t n, int shift, uint32_t* __restrict__ hist,
             int64_t T, const SortChunks sc, bool first) {
  constexpr int WSEG = 32 * ITEMS, TILE = kRsThreads * ITEMS, BINS = 1 << RB;
  constexpr int BPT = BINS / kRsThreads;
  constexpr uint32_t MASK = BINS - 1;
  // warp-private digit counts (shared-memory atomics), summed at the end
  __shared__ uint32_t h[kRsWarps][BINS];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int ww = 0; ww < kRsWarps; ++ww)
    for (int d = threadIdx.x; d < BINS; d += kRsThreads) h[ww][d] = 0;
  __syncthreads();
  uint32_t tot[BPT][G];
  const RsPlace at = rs_place<TILE, BINS, SEG>(sc, (int64_t)blockIdx.x * G, n, T, first);
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const int64_t seg = at.base + g * TILE + w * WSEG;
    // every item's key in flight at once, then the counts
    uint32_t d[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
      const int64_t e = seg + i * 32 + lane;
      d[i] = e < at.end ? (uint32_t)(__ldg(keys + e) >> shift) & MASK : 0xffffffffu;
    }
#pragma unroll
    for (int i = 0; i < ITEMS; ++i)
      if (d[i] != 0xffffffffu) atomicAdd(&h[w][d[i]], 1u);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < BPT; ++q) {
      tot[q][g] = 0;
#pragma unroll
      for (int ww = 0; ww < kRsWarps; ++ww) {
        uint32_t& c = h[ww][q * kRsThreads + threadIdx.x];
        tot[q][g] += c;
        if (g + 1 < G) c = 0;
      }
    }
    if (g + 1 < G) __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < BPT; ++q) {
    uint32_t* out = hist + at.hist + (int64_t)(q * kRsThreads + threadIdx.x) * at.stride;
    if constexpr (G == 4)
      *reinterpret_cast<uint4*>(out) = make_uint4(tot[q][0], tot[q][1], tot[q][2], tot[q][3]);
    else if constexpr (G == 2)
      *reinterpret_cast<uint2*>(out) = make_uint2(tot[q][0], tot[q][1]);
    else
#pragma unroll
      for (int g = 0; g < G; ++g) out[g] = tot[q][g];
  }
}

template <class K, int ITEMS, int RB, bool SEG>
__global__ void __launch_bounds__(kRsThreads, rs_min_blocks<K>())
k_rs_downsweep(const K* __restrict__ kin, const uint32_t* __restrict__ vin,
               K* __restrict__ kout, uint32_t* __restrict__ vout, int64_t n,
               int shift, const uint32_t* __restrict__ goff, int64_t T, const SortChunks sc,
               bool first) {
  constexpr int WSEG = 32 * ITEMS, TILE = kRsThreads * ITEMS, BINS = 1 << RB;
  constexpr int BPT = BINS / kRsThreads;  // digits per thread in the tile scan
  constexpr uint32_t MASK = BINS - 1;
  constexpr bool LATE = sizeof(K) == 4;
  static_assert(TILE <= 65535, "per-warp digit offsets are 16-bit");
  __shared__ K s_keys[TILE];
  __shared__ uint32_t s_vals[TILE];
  __shared__ uint16_t s_cnt[kRsWarps][BINS];  // per-warp digit counts, then offsets
  __shared__ uint32_t s_dstart[BINS];
  __shared__ int32_t s_gbase[BINS];
  __shared__ uint32_t s_warp[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const RsPlace at = rs_place<TILE, BINS, SEG>(sc, blockIdx.x, n, T, first);
  const int64_t base = at.base, end = at.end;
  if (base >= end) return;  // an empty tile of a last chunk
  const int valid_count = (int)min((int64_t)TILE, end - base);
  for (int i = lane; i < BINS; i += 32) s_cnt[w][i] = 0;
  __syncwarp();
  const unsigned lt_mask = (1u << lane) - 1u;
  K k[ITEMS];
  uint32_t v[ITEMS], r[ITEMS];
  const int64_t seg = base + w * WSEG;
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    int64_t e = seg + i * 32 + lane;
    k[i] = e < end ? __ldg(kin + e) : ~(K)0;
    if (!LATE) v[i] = vin && e < end ? __ldg(vin + e) : (uint32_t)e;
  }
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    uint32_t d = (uint32_t)(k[i] >> shift) & MASK;
    // lanes holding the same digit: one ballot per digit bit (measured faster
    // than __match_any_sync here)
    unsigned peers = gd::kFull;
#pragma unroll
    for (int bit = 0; bit < RB; ++bit) {
      const unsigned bb = __ballot_sync(gd::kFull, (d >> bit) & 1u);
      peers &= ((d >> bit) & 1u) ? bb : ~bb;
    }
    uint32_t b = s_cnt[w][d];
    __syncwarp();
    if (lane == __ffs(peers) - 1) s_cnt[w][d] = (uint16_t)(b + (uint32_t)__popc(peers));
    __syncwarp();
    r[i] = b + (uint32_t)__popc(peers & lt_mask);
  }
  if constexpr (LATE)  // the values, on their way during the tile scan
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const int64_t e = seg + i * 32 + lane;
    v[i] = vin && e < end ? __ldg(vin + e) : (uint32_t)e;
  }
  __syncthreads();
  {
    // digits threadIdx.x * BPT .. + BPT - 1: offsets across warps, then the
    // tile's digit starts
    uint32_t tots[BPT], sum = 0;
#pragma unroll
    for (int q = 0; q < BPT; ++q) {
      const int d = threadIdx.x * BPT + q;
      uint32_t tot = 0;
#pragma unroll
      for (int ww = 0; ww < kRsWarps; ++ww) {
        const uint32_t c = s_cnt[ww][d];
        s_cnt[ww][d] = (uint16_t)tot;
        tot += c;
      }
      tots[q] = tot;
      sum += tot;
    }
    uint32_t ex = block_excl_scan<kRsThreads>(sum, s_warp, nullptr);
#pragma unroll
    for (int q = 0; q < BPT; ++q) {
      const int d = threadIdx.x * BPT + q;
      s_dstart[d] = ex;
      s_gbase[d] = (int32_t)goff[at.hist + (int64_t)d * at.stride] - (int32_t)ex;
      ex += tots[q];
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    uint32_t d = (uint32_t)(k[i] >> shift) & MASK;
    uint32_t pos = s_dstart[d] + s_cnt[w][d] + r[i];
    s_keys[pos] = k[i];
    s_vals[pos] = v[i];
  }
  __syncthreads();
  for (int j = threadIdx.x; j < valid_count; j += kRsThreads) {
    K key = s_keys[j];
    uint32_t d = (uint32_t)(key >> shift) & MASK;
    int64_t g = (int64_t)s_gbase[d] + j;
    kout[g] = key;
    vout[g] = s_vals[j];
  }
}

// Set bits of a mask listed in one pass: per-word prefix counts (pre) and the
// positions of the set bits in order (out[pre[w] + r] = 32 w + (bit r of word w)).
// A tile is 512 words, one per thread: word counts are scanned in the block, the
// tile's prefix comes by look-back, and each warp then writes its 32 words one at
// a time with a lane per bit, so each word's entries go out in one store.  One
// launch where a scan and a compaction took two.
constexpr int kListThreads = 512, kListWords = 1, kListTile = kListThreads * kListWords;
__global__ void __launch_bounds__(kListThreads)
k_list_bits(const uint32_t* __restrict__ words, uint32_t* __restrict__ pre, int64_t nw,
            uint32_t* __restrict__ out, unsigned tiles, LookbackCtl* ctl,
            unsigned long long* status, uint32_t* total_dev, unsigned long long* timeouts) {
  __shared__ uint32_t s_warp[32];
  __shared__ unsigned s_tile, s_epoch;
  __shared__ uint32_t s_agg, s_excl;
  __shared__ uint32_t s_w[kListTile], s_p[kListTile];
  lb_begin(ctl, &s_tile, &s_epoch);
  const unsigned tile = s_tile, epoch = s_epoch;
  if (tile >= tiles) {
    // a counter left inconsistent (never expected): no tile, report it
    if (threadIdx.x == 0 && timeouts) atomicAdd(timeouts, 1ull);
    lb_end(ctl, tiles, epoch);
    return;
  }
  const int64_t base = (int64_t)tile * kListTile;
  uint32_t v[kListWords], sum = 0;
#pragma unroll
  for (int i = 0; i < kListWords; ++i) {
    const int64_t w = base + threadIdx.x * kListWords + i;
    v[i] = w < nw ? words[w] : 0u;
    sum += (uint32_t)__popc(v[i]);
  }
  uint32_t ex = block_excl_scan<kListThreads>(sum, s_warp, &s_agg);
  const uint32_t excl = lb_tile_prefix(status, tile, lb_tag(epoch), &s_agg, &s_excl, timeouts);
  if (threadIdx.x == 0 && tile == tiles - 1u && total_dev) *total_dev = excl + s_agg;
  ex += excl;
#pragma unroll
  for (int i = 0; i < kListWords; ++i) {
    const int k = threadIdx.x * kListWords + i;
    if (base + k < nw) pre[base + k] = ex;
    s_w[k] = v[i];
    s_p[k] = ex;
    ex += (uint32_t)__popc(v[i]);
  }
  __syncwarp();  // a warp's words were written by its own lanes
  const int lane = threadIdx.x & 31, k0 = (threadIdx.x >> 5) * 32 * kListWords;
  const unsigned below = (1u << lane) - 1u;
#pragma unroll 4
  for (int k = k0; k < k0 + 32 * kListWords; ++k) {
    const uint32_t x = s_w[k];
    if ((x >> lane) & 1u)
      out[s_p[k] + (uint32_t)__popc(x & below)] = (uint32_t)((base + k) << 5) + (uint32_t)lane;
  }
  lb_end(ctl, tiles, epoch);
}

__global__ void k_iota(uint32_t* v, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    v[i] = (uint32_t)i;
}

inline size_t align_up(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace

// scan temp: control block (64 B), then the status words
size_t scan_temp_bytes(int64_t n) {
  const int64_t T = (n + kScanTile - 1) / kScanTile;
  return align_up(sizeof(LookbackCtl) + (size_t)(T > 0 ? T : 1) * 8);
}

int scan_launches(int64_t n) { return n > 0 ? 1 : 0; }

template <bool POPC>
void scan_impl(const uint32_t* in, uint32_t* out, int64_t n, void* temp, uint32_t* total_dev,
               cudaStream_t s, unsigned long long* timeouts) {
  if (n <= 0) {
    if (total_dev) cudaMemsetAsync(total_dev, 0, sizeof(uint32_t), s);
    return;
  }
  const int64_t T = (n + kScanTile - 1) / kScanTile;
  k_scan_onepass<POPC><<<(unsigned)T, kScanThreads, 0, s>>>(in, out, n, (unsigned)T, lb_ctl(temp),
                                                            lb_status(temp), total_dev, timeouts);
}

void exclusive_scan_u32(const uint32_t* in, uint32_t* out, int64_t n, void* temp,
                        uint32_t* total_dev, cudaStream_t s, unsigned long long* timeouts) {
  scan_impl<false>(in, out, n, temp, total_dev, s, timeouts);
}

void exclusive_scan_popc(const uint32_t* words, uint32_t* pre, int64_t nw, void* temp,
                         uint32_t* total_dev, cudaStream_t s, unsigned long long* timeouts) {
  scan_impl<true>(words, pre, nw, temp, total_dev, s, timeouts);
}

void list_bits(const uint32_t* words, uint32_t* pre, int64_t nw, uint32_t* out, void* temp,
               uint32_t* total_dev, cudaStream_t s, unsigned long long* timeouts) {
  if (nw <= 0) {
    cudaMemsetAsync(total_dev, 0, sizeof(uint32_t), s);
    return;
  }
  const int64_t T = (nw + kListTile - 1) / kListTile;
  k_list_bits<<<(unsigned)T, kListThreads, 0, s>>>(words, pre, nw, out, (unsigned)T, lb_ctl(temp),
                                                   lb_status(temp), total_dev, timeouts);
}

// sort temp: the [digit][tile] histogram.  Its scan keeps its state in the
// caller's scan temp, which holds nothing but scan state: were the two in one
// buffer, a larger sort's status words would lie where a smaller sort left its
// histogram, and a count that looks like a tagged word would pass for a prefix.
int64_t sort_scan_elems(int64_t n, int chunks) {
  const int64_t plain = ((n + kRsMinTile - 1) / kRsMinTile + 3) / 4 * 4;
  return std::max(plain, chunks * (gd::kChunkPoints / kRsMinTile)) * kRsMaxBins;
}

size_t sort_temp_bytes(int64_t n, int chunks) {
  return align_up((size_t)sort_scan_elems(n, chunks) * sizeof(uint32_t));
}

// The points lie instance by instance already, so the id's bits need no pass (120M points
// in 4096 instances, 48-bit keys of 36 local bits: six passes and 49.8 ms a run, by
// instance four and 48.5); chunks that are half empty or more would cost more in empty
// tiles' counts.
bool sort_by_instance(int64_t n, int chunks, int local, int bits) {
  auto passes = [](int b) { return (b + sort_digit_bits(b) - 1) / sort_digit_bits(b); };
  return local > 0 && passes(local) < passes(bits) && chunks * gd::kChunkPoints <= 2 * n;
}

template <class K, int RB, bool SEG>
int sort_passes(K* keys[2], uint32_t* vals[2], int64_t n, int passes, bool vals_in_is_iota,
                void* temp, void* scan_temp, cudaStream_t s, unsigned long long* timeouts,
                const SortChunks& sc) {
  constexpr int ITEMS = rs_items<K>();
  constexpr int TILE = kRsThreads * ITEMS;
  // four tiles per upsweep block where that leaves enough blocks; the histogram is then
  // for a multiple of four tiles, the last ones perhaps empty
  constexpr int TPC = (int)(gd::kChunkPoints / TILE);  // (by instance: a chunk's)
  int64_t T = SEG ? (int64_t)sc.count * TPC : (n + TILE - 1) / TILE;
  const bool four = !SEG && T >= kRsFour;
  const int64_t tiles = T;
  if (four) T = (T + 3) & ~(int64_t)3;
  const int64_t h = T << RB;
  uint32_t* hist = static_cast<uint32_t*>(temp);
  int cur = 0;
  for (int p = 0; p < passes; ++p) {
    int shift = RB * p;
    const bool first = p == 0;
    if constexpr (SEG)
      k_rs_upsweep<K, ITEMS, RB, TPC, true><<<(unsigned)sc.count, kRsThreads, 0, s>>>(
          keys[cur], n, shift, hist, T, sc, first);
    else if (four)
      k_rs_upsweep<K, ITEMS, RB, 4, false><<<(unsigned)(T / 4), kRsThreads, 0, s>>>(keys[cur], n, shift, hist,
                                                                           T, sc, first);
    else
      k_rs_upsweep<K, ITEMS, RB, 1, false><<<(unsigned)T, kRsThreads, 0, s>>>(keys[cur], n, shift, hist, T, sc,
                                                                       first);
    exclusive_scan_u32(hist, hist, h, scan_temp, nullptr, s, timeouts);
    const uint32_t* vin = (p == 0 && vals_in_is_iota) ? nullptr : vals[cur];
    k_rs_downsweep<K, ITEMS, RB, SEG><<<(unsigned)tiles, kRsThreads, 0, s>>>(
        keys[cur], vin, keys[cur ^ 1], vals[cur ^ 1], n, shift, hist, T, sc, first);
    cur ^= 1;
  }
  return cur;
}

int sort_digit_bits(int bits) { return (bits + 8) / 9 < (bits + 7) / 8 ? 9 : 8; }

int sort_launches(int64_t n, int bits) {
  if (n <= 0) return 0;
  const int rb = sort_digit_bits(bits);
  const int passes = (bits + rb - 1) / rb;
  return passes ? passes * 3 : 1;  // upsweep, scan, downsweep per pass
}

// Digits of 9 bits where they save a pass (a 26-bit key: 3 passes, not 4),
// else of 8 bits.
template <class K>
int radix_sort_pairs(K* keys[2], uint32_t* vals[2], int64_t n, int bits, bool vals_in_is_iota,
                     void* temp, void* scan_temp, cudaStream_t s, unsigned long long* timeouts,
                     const SortChunks& sc) {
  if (n <= 0) return 0;
  const int rb = sort_digit_bits(bits);
  const int passes = (bits + rb - 1) / rb;
  if (passes == 0) {
    if (vals_in_is_iota) k_iota<<<1024, 256, 0, s>>>(vals[0], n);
    return 0;
  }
  auto* f = sc.chunks ? (rb == 9 ? sort_passes<K, 9, true> : sort_passes<K, 8, true>)
                      : (rb == 9 ? sort_passes<K, 9, false> : sort_passes<K, 8, false>);
  return f(keys, vals, n, passes, vals_in_is_iota, temp, scan_temp, s, timeouts, sc);
}

template int radix_sort_pairs<uint32_t>(uint32_t* [2], uint32_t* [2], int64_t, int, bool, void*,
                                        void*, cudaStream_t, unsigned long long*, const SortChunks&);
template int radix_sort_pairs<unsigned long long>(unsigned long long* [2], uint32_t* [2], int64_t,
                                                  int, bool, void*, void*, cudaStream_t,
                                                  unsigned long long*, const SortChunks&);

}  // namespace gdprim
