// gd_lookback.cuh -- block scans and the decoupled look-back that the single-pass
// kernels share (gd_prims.cu: scans and list compaction, gd_pipeline.cu: cell list).
//
// Each tile publishes its aggregate, reads its predecessors' published values back
// to the nearest inclusive prefix, and publishes its own inclusive prefix.  Tiles
// take their index from an atomic counter when their block starts, so a tile only
// waits on tiles that running blocks hold and every wait ends; each wait is still
// bounded (kWaitPolls polls), and a wait that gives up counts the predecessor as 0
// -- every offset then stays at or below its true value, so no write leaves its
// array -- and is reported through the caller's counter.
//
// The state between launches lives in the caller's scan temp, which must be zero
// when first used and hold nothing else: a control block (tile counter,
// finished-block counter, launch epoch) that the last block of each launch resets,
// and the status words, tagged with the launch's epoch so that words left by
// earlier launches read as not ready.
#pragma once

#include "gd_internal.cuh"

namespace gdprim {

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t t = __shfl_up_sync(gd::kFull, v, o);
    if (lane >= o) v += t;
  }
  return v;
}

// exclusive scan of one value per thread across a block of NT threads
template <int NT>
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* s_warp,
                                                    uint32_t* block_total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  constexpr int NW = NT / 32;
  uint32_t inc = warp_incl_scan(v, lane);
  if (lane == 31) s_warp[w] = inc;
  __syncthreads();
  if (w == 0) {
    uint32_t t = lane < NW ? s_warp[lane] : 0u;
    uint32_t ti = warp_incl_scan(t, lane);
    if (lane < NW) s_warp[lane] = ti - t;
    if (lane == NW - 1 && block_total) *block_total = ti;
  }
  __syncthreads();
  uint32_t r = s_warp[w] + inc - v;
  __syncthreads();
  return r;
}

// ------------------------------------------------------------ look-back state
struct LookbackCtl {
  unsigned int tile;   // next tile index of the running launch
  unsigned int done;   // blocks of the running launch that finished
  unsigned int epoch;  // launches completed on this control block
  unsigned int pad[13];
};
static_assert(sizeof(LookbackCtl) == 64, "control block is 64 bytes");

// A predecessor tile's block is already running when its tile is waited on, so
// its aggregate follows within microseconds; 2^14 polls (about 16 ms) only end
// waits that could never succeed.
constexpr unsigned kWaitPolls = 1u << 14;

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// status word: tag (bits 63..34), kind (33..32: 1 aggregate, 2 inclusive
// prefix), value (31..0)
__device__ __forceinline__ unsigned long long lb_word(uint32_t tag, uint32_t kind, uint32_t v) {
  return ((unsigned long long)tag << 34) | ((unsigned long long)kind << 32) | v;
}

// A tile's status word once it carries this launch's tag: its kind (1 or 2)
// and value; kind 0 (value 0) when kWaitPolls polls saw nothing.
__device__ __forceinline__ uint32_t lb_wait(const unsigned long long* p, uint32_t tag,
                                            uint32_t& v) {
  for (unsigned it = 0; it < kWaitPolls; ++it) {
    const unsigned long long w = ld_relaxed_u64(p);
    const uint32_t kind = (uint32_t)(w >> 32) & 3u;
    if ((uint32_t)(w >> 34) == tag && kind != 0u) {
      v = (uint32_t)w;
      return kind;
    }
    if (it >= 4) __nanosleep(64);
  }
  v = 0;
  return 0;
}

// Block start: the tile index (from the counter) and the launch's tag.
__device__ __forceinline__ void lb_begin(LookbackCtl* ctl, unsigned* s_tile, unsigned* s_epoch) {
  if (threadIdx.x == 0) {
    *s_tile = atomicAdd(&ctl->tile, 1u);
    *s_epoch = *reinterpret_cast<volatile unsigned*>(&ctl->epoch);
  }
  __syncthreads();
}

__device__ __forceinline__ uint32_t lb_tag(unsigned epoch) { return (epoch & 0x3fffffffu) + 1u; }

// Block end, after every thread is done with the status words: the last block
// of the launch resets the counters and advances the epoch for the next one.
__device__ __forceinline__ void lb_end(LookbackCtl* ctl, unsigned tiles, unsigned epoch) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&ctl->done, 1u) == tiles - 1u) {
      ctl->tile = 0u;
      ctl->done = 0u;
      ctl->epoch = epoch + 1u;
    }
  }
}

// Exclusive prefix of tile `tile` from its predecessors' status words, by one
// warp (32 predecessors per round, nearest first).  *gave_up: a wait ran out.
__device__ __forceinline__ uint32_t lb_warp_prefix(const unsigned long long* status, int64_t tile,
                                                   uint32_t tag, bool* gave_up) {
  const int lane = threadIdx.x & 31;
  uint32_t excl = 0;
  bool lost = false;
  for (int64_t top = tile - 1; top >= 0; top -= 32) {
    const int64_t k = top - lane;
    uint32_t v = 0, kind = 2;  // before tile 0: an inclusive prefix of 0
    if (k >= 0) kind = lb_wait(status + k, tag, v);
    lost |= __any_sync(gd::kFull, kind == 0u);
    // nearest lane holding a prefix (or a wait that gave up): sum up to it
    const unsigned stop = __ballot_sync(gd::kFull, kind != 1u);
    const int last = stop ? __ffs(stop) - 1 : 31;
    uint32_t add = lane <= last ? v : 0u;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) add += __shfl_xor_sync(gd::kFull, add, o);
    excl += add;
    if (stop) break;
  }
  *gave_up = lost;
  return excl;
}

// Block-wide: the tile's exclusive prefix from its aggregate (held by thread 0's
// warp in *s_agg), published on the way; every thread gets it.  tiles - 1's inclusive
// prefix is the total (*s_excl + aggregate there).
__device__ __forceinline__ uint32_t lb_tile_prefix(unsigned long long* status, unsigned tile,
                                                   uint32_t tag, const uint32_t* s_agg,
                                                   uint32_t* s_excl, unsigned long long* timeouts) {
  if (threadIdx.x < 32) {
    const uint32_t agg = *s_agg;
    unsigned long long* my = status + tile;
    if (threadIdx.x == 0) st_relaxed_u64(my, lb_word(tag, tile == 0 ? 2u : 1u, agg));
    bool lost = false;
    const uint32_t excl = tile == 0 ? 0u : lb_warp_prefix(status, (int64_t)tile, tag, &lost);
    if (threadIdx.x == 0) {
      if (tile != 0) st_relaxed_u64(my, lb_word(tag, 2u, excl + agg));
      *s_excl = excl;
      if (lost && timeouts) atomicAdd(timeouts, 1ull);
    }
  }
  __syncthreads();
  return *s_excl;
}

// control block and status words in scan temp memory
__host__ __device__ inline LookbackCtl* lb_ctl(void* temp) { return static_cast<LookbackCtl*>(temp); }
__host__ __device__ inline unsigned long long* lb_status(void* temp) {
  return reinterpret_cast<unsigned long long*>(static_cast<char*>(temp) + sizeof(LookbackCtl));
}

}  // namespace gdprim
