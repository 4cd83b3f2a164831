// gd_internal.cuh -- device-side declarations shared by the gbdbscan kernels.
//
// Data layout in HBM for one clustering instance of n points in d dimensions
// (d = 2 or 3), after the index build:
//   keys[n]   u32   fine-cell key of each point, sorted ascending (u64 for
//                   sparse grids)
//   ids[n]    u32   original point index of each sorted position
//   X[n][d]   f64   coordinates of each sorted position
//   ent[]     32 B  block entries: 64 cells each (8x8 in 2D, 4x4x4 in 3D), found
//                   directly by block key, through a table of block rows, or
//                   through a hash of the occupied block rows (k_cells)
//   ckeys[M]        key of every non-empty cell
//   reps[M+1] i32   sorted position of the first point of every non-empty cell
// Per non-empty cell, indexed by its cell index m (0..M-1, key order; the
// walks reach it from a block entry's occupancy word without loading reps):
//   cellcore[m]  number of core points in the cell
//   compmin[m]   smallest original index among the cell's core points (general path: that of
//                its first core position, ids ascend within a cell; small path: cellmin[m])
//   parent[m]    union-find parent (a cell index)
//   cellcid[m]   cluster id of the cell's core points (INT_MAX: none)
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace gd {

constexpr int kNoise = -2;            // common.h:8 NOISE
constexpr int kWarp = 32;
constexpr unsigned kFull = 0xffffffffu;

// One clustering instance as the caller describes it (uploaded per run).
struct InstDesc {
  int64_t pt_off;      // first point of the instance in the concatenated point list
  int64_t n;           // its points
  int64_t co_off;      // its first coordinate (in doubles) in the concatenated buffer
  double eps;
  int32_t dim;         // 2 or 3
  int32_t minpts;
};

// A run of points of one instance (bbox and key kernels take one block each).
struct Chunk {
  int32_t inst;
  int32_t sorted;      // its first position with the instances in their own order
  int64_t begin;       // global point indices [begin, end)
  int64_t end;
};
constexpr int64_t kChunkPoints = 8192;

// Whole-run layout, computed on the device after the per-instance grids.
struct BatchInfo {
  int32_t K;           // instances
  int32_t LB;          // local key bits (widest instance grid)
  int32_t IB;          // instance-id bits
  int32_t key64;       // 1: keys are 64-bit
  uint64_t ent_total;  // block entries of all directly addressed instances
  uint64_t row_total;  // row-table entries of all instances that use one
  uint64_t grid_cells; // cells of direct tables + rows of row tables
  int32_t any_sparse;  // some instance uses the hash of occupied block rows
  int32_t flags;       // OR of the instances' kFlag* bits
  int32_t any_xf;      // some instance wants the centred float32 copy
  int32_t max_dim;
  int32_t K2;          // instances [0, K2) are 2D, [K2, K) 3D
  int32_t band_off;    // some instance has no valid float32 band (all its pairs
                       // take the float64 predicate)
};

// Grid and predicate parameters of one instance, computed on the device from
// its bounding box.
struct DevParams {
  double lo[3];        // per-dimension minimum (grid origin)
  double hi[3];        // per-dimension maximum
  double centre[3];    // bounding-box centre (origin of the float32 copy)
  double f;            // fine cell side
  double inv_f;        // 1 / f
  double eps;          // epsilon
  double eps2;         // fl(eps * eps), the reference's threshold
  double eps2_in;      // float64 d2 <= eps2_in implies the box test passes
  float eps2_lo32;     // float32 d2 below this: certainly a neighbour
  float eps2_hi32;     // float32 d2 above this: certainly not a neighbour
  int64_t G[3];        // cells per dimension
  int32_t Bk[3];       // blocks per dimension (8 cells a side in 2D, 4 in 3D)
  uint64_t NB;         // total blocks
  uint64_t rows;       // block rows: NB / Bk[dim-1]
  int32_t dim;
  int32_t minpts;
  int32_t key_bits;    // bits of a local key (block key, then 6 bits in the block)
  int32_t cell_bits;   // bits of the plain cell count (the refusal limit is on these)
  int32_t flags;       // kFlag*
  int32_t sparse;      // block lookup: 0 directly by block key; 2 table of block rows
                       // (blocks inside a row by binary search); 1 hash of occupied rows
  int32_t prune;       // 1: cell-level inside/outside classification enabled
  float inv_f32;       // fl32(1 / f)
  float uerr;          // bound on the error of a point's in-cell position (cell units)
  float thr_in;        // sum of squared max distances (cell units) below: all neighbours
  float thr_out;       // sum of squared min distances (cell units) above: none
  int64_t pt_off;      // first point (global index)
  int64_t n;           // points
  int64_t co_off;      // first coordinate in the concatenated buffer
  uint32_t ent_off;    // direct table: the instance's first block entry
  uint64_t row_off;    // row table: the instance's first row
  uint64_t kmask;      // mask of the local key bits
  int32_t LB;          // local key bits of the run (copied from BatchInfo)
  int32_t inst;        // instance index
  // exact division of block keys by Bk[1] and Bk[2] (multiply-high method, see
  // udiv_magic): multiplier and shift per divisor
  uint64_t dm[2];
  int32_t ds[2];
  uint32_t dm32[2];    // the same on 32 bits, for fewer than 2^32 blocks (small)
  int32_t small;
  // float32 cell origins without float64 arithmetic (cell_origin32): the cell
  // side and lo - centre per axis as float pairs (hi + lo), valid when fast_origin
  float f_hi, f_lo;
  float b_hi[3], b_lo[3];
  int32_t fast_origin;
  // float32 cell keys (k_keys): lo and 1/f in float, and the bound on
  // |t32 - t64| in cell units; a coordinate whose float32 cell position is
  // farther than key_band from a cell boundary takes its cell from it, the
  // others from the float64 formula.  Valid when key_fast.
  float key_lo32[3], key_inv32, key_band;
  int32_t key_fast;
};

// Division by an invariant integer d >= 1 through a multiply-high (Granlund &
// Montgomery, "Division by invariant integers using multiplication", 1994,
// Fig. 4.1, N = 64): with l = ceil(log2 d) and m = floor(2^64 (2^l - d) / d) + 1,
// q = (t + ((k - t) >> 1)) >> (l - 1), t = mulhi(m, k), for every 64-bit k
// (l = 0, i.e. d = 1: q = k).  d < 2^32.
__host__ __device__ inline void udiv_magic(uint64_t d, uint64_t& m, int32_t& l) {
  l = 0;
  while (l < 64 && (1ull << l) < d) ++l;
  if (l == 0) { m = 0; return; }
  // floor((2^l - d) * 2^64 / d) in two 32-bit digits (d < 2^32: both partial
  // remainders shifted by 32 fit 64 bits; 2^l - d < d)
  const uint64_t r0 = ((1ull << l) - d) << 32;
  const uint64_t q1 = r0 / d, r1 = (r0 - q1 * d) << 32;
  const uint64_t q = (q1 << 32) | (r1 / d);
  m = q + 1;
}

__device__ __forceinline__ uint64_t udiv_by(uint64_t k, uint64_t m, int32_t l) {
  if (l == 0) return k;
  const uint64_t t = __umul64hi(m, k);
  return (t + ((k - t) >> 1)) >> (l - 1);
}

// The 32-bit form (N = 32): same shift, m = floor(2^32 (2^l - d) / d) + 1.
__host__ __device__ inline uint32_t udiv_magic32(uint32_t d) {
  int l = 0;
  while (l < 32 && (1ull << l) < d) ++l;
  if (l == 0) return 0;
  return (uint32_t)((((1ull << l) - d) << 32) / d) + 1u;
}

__device__ __forceinline__ uint32_t udiv_by32(uint32_t k, uint32_t m, int32_t l) {
  if (l == 0) return k;
  const uint32_t t = __umulhi(m, k);
  return (t + ((k - t) >> 1)) >> (l - 1);
}

// The predicate constants a cell kernel keeps in registers.
struct PredParams {
  double eps, eps2, eps2_in;
  float eps2_lo32, eps2_hi32, uerr, thr_in, thr_out, inv_f32;
  int32_t minpts, prune;
};

__device__ __forceinline__ PredParams pred_params(const DevParams& P) {
  PredParams q;
  q.eps = P.eps;
  q.eps2 = P.eps2;
  q.eps2_in = P.eps2_in;
  q.eps2_lo32 = P.eps2_lo32;
  q.eps2_hi32 = P.eps2_hi32;
  q.uerr = P.uerr;
  q.thr_in = P.thr_in;
  q.thr_out = P.thr_out;
  q.inv_f32 = P.inv_f32;
  q.minpts = P.minpts;
  q.prune = P.prune;
  return q;
}

// Blocks of 64 cells: the low 6 bits of a key are the cell's place in its
// block, x-major, the bits above the block's key, x-major over the blocks.  A
// block's occupied cells are one 64-bit word, its cells are consecutive in key
// order, and the +-2 stencil of a cell meets at most two blocks per axis: 4
// lookups in 2D and 8 in 3D answer for all 25 or 125 cells.
constexpr int kBlockBits = 6;
template <int D>
__host__ __device__ constexpr int block_shift() { return D == 2 ? 3 : 2; }

// One block.  Direct tables: indexed by block key; otherwise by the block's
// first cell.
struct alignas(32) BlockEnt {
  unsigned long long occ;   // occupied cells
  uint32_t base;            // index of the block's first cell
  uint32_t lo;              // the root its core cells share before union pass 1 (kNoEnt:
                            // unset, kMixedRoot: several); border search: their smallest
                            // cluster id
  unsigned long long core;  // cells holding a core point
  uint32_t hi;              // the root its core cells share before union pass 2
  uint32_t uni;             // the root its core cells share before union pass 0
};
static_assert(sizeof(BlockEnt) == 32, "one sector per block entry");
constexpr uint32_t kNoEnt = 0xffffffffu, kMixedRoot = 0xfffffffeu;

// Links between core cells of one block that share a face: per axis the cells
// linked to the next one along it.
struct alignas(8) BlockLinks {
  uint32_t w[3][2];
};

// Cells of a block holding two points and more, three and more.
struct alignas(16) BlockPop {
  uint32_t two[2], three[2];
};

// A grid with too many blocks for a direct table takes a table of its block
// rows when it has at most this many rows per point (or the table floor).
constexpr uint64_t kRowsPerPoint = 8;

constexpr int kFlagNonFinite = 1;     // NaN or Inf coordinate
constexpr int kFlagGridTooLarge = 2;  // cell counts and instance ids beyond 62 bits
constexpr int kFlagNotSmall = 8;      // the grid is not for the small kernels
constexpr int kFlagNoShortcut = 4;    // |x| too large relative to eps for the
                                      // box-test shortcut / float32 filter

// Device counters (u64), zeroed per run.
enum Counter {
  kCtrCells = 0,        // M, number of non-empty cells
  kCtrTests64,          // float64 distance evaluations
  kCtrTests32,          // float32 distance evaluations
  kCtrBand,             // float32 evaluations that fell in the re-test band
  kCtrAsym,             // core pairs that are neighbours in one direction only
  kCtrClusters,         // K
  kCtrCore,             // core points
  kCtrNoise,            // noise points
  kCtrDenseCells,       // cells with >= minpts points
  kCtrAsymEdges,        // one-directional core pairs recorded for the merge replay
  kCtrHeavyCore,        // cells queued for warp-cooperative core counting
  kCtrHeavyUnion,       // cells queued for warp-cooperative link searches
  kCtrHeavyBorder,      // cells queued for warp-cooperative border search
  kCtrCells2D,          // cells of 2D instances (they sort first)
  kCtrWalkCursor2,      // walk-list entries handed out (2D, 3D); cleared before each walk launch
  kCtrWalkCursor3,
  kCtrWaitTimeouts,     // look-back waits (scans, sort) and small runs' barrier waits that gave up
  kCtrBlocks,           // blocks holding a core point (small runs: positions handed out)
  kCtrSmallPairs,       // small runs: large cell pairs for blocks and for the grid, in each of
                        // the union's two steps (4 words, cleared by the expand)
  kCtrCount = 22
};

// Capacity of the list of one-directional core-core pairs (see k_asym_resolve).
constexpr int kAsymCap = 2048;

// Work space of the merge replay (k_asym_resolve).
struct AsymWork {
  int from[kAsymCap], to[kAsymCap];
  int node[2 * kAsymCap], assigned[2 * kAsymCap];
};

// A small run's arguments beside its buffers (gd_small.cuh).
struct SmallArgs {
  const double* coords;
  int n, dim;
  double eps, mult;
  uint64_t direct_max;       // blocks a direct table may have
  uint32_t hash_slots;       // slots of the block hash (power of two); 0: direct grids only
  unsigned* bar;             // barrier: arrivals, generation (zero when first used)
  long long* part;           // 8 words per block: bounds of its points, non-finite flag
  // (index; in the expand these three hold the lists of open link searches)
  unsigned long long* ptkey; // per point: entry << 6 | place in the block
  uint32_t* ptcell;          // per point: its cell
  uint32_t* ptpos;           // per point: its place in the cell
  uint32_t* pcell;           // per position: its cell
  uint64_t* cellkey;         // per cell: entry << 6 | place in the block
  uint2* crange;             // per cell: its positions [x, y)
  uint32_t* list;            // positions outside dense cells (per expand)
  uint32_t* cellrep;         // per core cell: its first core point (position)
  AsymWork* asym;
};

constexpr int kSmallThreads = 512;
// pair tests one lane of a small run spends on a cell pair before the pair goes to a warp
constexpr int kSmallLinkTests = 64;
// open candidates from which a point goes to a warp (core count), and candidates that a lane
// looks at for a point's border search before it does.  (Both lines at half and twice the value
// on sets with crowded cells, 300 to 260,000 points, and on the blobs: 64 instead of 256 costs
// 30,000 3D blob points 16 % and 128 2 %, 512 costs 260,000 points in clumps of different spread
// 20 %; link tests at 256 cost 1,000 to 30,000 points at Zipf-popular positions 10 to 20 %.
// Float32 tests cost a lane less beside the classification that a warp does again: at 256 and
// 512, 130,000 3D points of a few per position take 1.35 and 1.23 times as long as at 1024; at
// 2048 260,000 points in clumps 1.25 times.)
constexpr int kSmallPointTests = 256, kSmallPointTests32 = 1024;
// Single runs of at most this many points take the small kernels when their grid has
// a direct block table.  The lines lie where the general pipeline's launches stop
// dominating: 2D 482 -> 341 us at 128k points, 510 -> 398 at 256k (blobs, float64); 3D
// 756 -> 648 at 128k, but 789 -> 960 at 256k.  With a block hash at most
// kSmallHashPoints: larger sparse sets are the general path's row tables'.
constexpr int64_t small_points(int dim) { return dim == 2 ? 262144 : 131072; }
constexpr int64_t kSmallHashPoints = 16384;
__host__ __device__ constexpr uint64_t small_direct_max(int64_t n) {
  return n < 4096 ? 8192 : 2 * (uint64_t)n;
}
__host__ __device__ constexpr uint32_t small_hash_slots(int64_t n) {
  if (n > kSmallHashPoints) return 0;
  uint32_t h = 1024;
  while (h < 2 * (uint64_t)n) h <<= 1;
  return h;
}

// Hash of occupied block rows (sparse grids): open addressing, linear probing.
constexpr unsigned long long kHashEmpty = ~0ull;
__host__ __device__ __forceinline__ uint32_t hash_key(unsigned long long k) {
  return (uint32_t)((k * 0x9E3779B97F4A7C15ull) >> 32);
}

// ---- float64 predicate, bit-exact with the reference's CPU DBSCAN ----------
// Neighbour test with centre p and candidate q: the query box
// [fl(p-eps), fl(p+eps)] with inclusive bounds (cpu-dbscan/Rtree.h:1573-1588)
// and fl(fl(dx*dx) + fl(dy*dy) [+ fl(dz*dz)]) <= fl(eps*eps), dx = fl(p - q)
// (cpu-dbscan/dbscan_rtree_exp.cpp:351-358, 431-432).  The _rn intrinsics keep
// the compiler from fusing multiply-adds, which would change the bits.
template <int D>
__device__ __forceinline__ double dist2_f64(const double* p, const double* q) {
  double a = __dsub_rn(p[0], q[0]);
  double s = __dmul_rn(a, a);
  double b = __dsub_rn(p[1], q[1]);
  s = __dadd_rn(s, __dmul_rn(b, b));
  if (D == 3) {
    double c = __dsub_rn(p[2], q[2]);
    s = __dadd_rn(s, __dmul_rn(c, c));
  }
  return s;
}

template <int D>
__device__ __forceinline__ bool box_f64(const double* p, const double* q, double eps) {
#pragma unroll
  for (int k = 0; k < D; ++k) {
    double lo = __dsub_rn(p[k], eps);
    double hi = __dadd_rn(p[k], eps);
    if (lo > q[k] || q[k] > hi) return false;
  }
  return true;
}

// d2 <= t for a squared distance d2 (a sum of squares of finite values: +0 or
// positive, never -0 or NaN) and any t other than NaN, from the bit patterns:
// non-negative doubles order as their bits do as signed integers, and a
// negative t has a negative pattern, below every d2.  An integer compare keeps
// the test off this GPU's narrow float64 pipe.
__device__ __forceinline__ bool d2_le(double d2, double t) {
  return __double_as_longlong(d2) <= __double_as_longlong(t);
}

// Full predicate given d2 = dist2_f64(p, q).
template <int D, class PP>
__device__ __forceinline__ bool pred_from_d2(double d2, const double* p, const double* q,
                                             const PP& P) {
  if (d2_le(d2, P.eps2_in)) return true;
  if (!d2_le(d2, P.eps2)) return false;
  return box_f64<D>(p, q, P.eps);
}

// ---- union-find over cells (lock-free; the larger index hooks under the smaller)
__device__ __forceinline__ int uf_find(int* parent, int x) {
  volatile int* par = parent;
  int p = par[x];
  while (p != x) {
    int gp = par[p];
    if (gp != p) par[x] = gp;
    x = p;
    p = gp;
  }
  return x;
}

__device__ __forceinline__ void uf_union(int* parent, int a, int b) {
  while (true) {
    a = uf_find(parent, a);
    b = uf_find(parent, b);
    if (a == b) return;
    if (b < a) { int t = a; a = b; b = t; }
    // hook b under a
    int old = atomicCAS(parent + b, b, a);
    if (old == b) return;
    b = old;
  }
}

}  // namespace gd

// ---- host-side primitive launchers (gd_prims.cu) ---------------------------
namespace gdprim {
// temp bytes needed by exclusive_scan_u32 / exclusive_scan_popc for n
// elements.  Temp memory must be zero when first used and is then kept
// consistent by the primitives themselves (one stream at a time).
size_t scan_temp_bytes(int64_t n);
// kernels one scan of n elements launches
int scan_launches(int64_t n);
// out[i] = sum_{j<i} in[i]; in == out allowed.  Returns the total in *total_dev
// (device pointer, may be null).  timeouts (may be null): incremented when a
// look-back wait gave up (the result is then wrong but every write in bounds).
void exclusive_scan_u32(const uint32_t* in, uint32_t* out, int64_t n, void* temp,
                        uint32_t* total_dev, cudaStream_t s,
                        unsigned long long* timeouts = nullptr);
// pre[w] = number of set bits in words[0, w) (exclusive scan of popcounts),
// total in *total_dev (may be null); words and pre 16-byte aligned, distinct.
void exclusive_scan_popc(const uint32_t* words, uint32_t* pre, int64_t nw, void* temp,
                         uint32_t* total_dev, cudaStream_t s,
                         unsigned long long* timeouts = nullptr);
// the set bits of words[0, nw): pre as above, and their positions in ascending
// order, out[pre[w] + r] = 32 w + (position of the r-th set bit of word w); temp and
// timeouts as for the scan
void list_bits(const uint32_t* words, uint32_t* pre, int64_t nw, uint32_t* out, void* temp,
               uint32_t* total_dev, cudaStream_t s, unsigned long long* timeouts = nullptr);
// temp bytes needed by radix_sort_pairs for n elements (either key width), and
// the elements its scan temp must allow for (scan_temp_bytes of that many)
// (chunks: as for radix_sort_pairs, 0 without)
size_t sort_temp_bytes(int64_t n, int chunks = 0);
int64_t sort_scan_elems(int64_t n, int chunks = 0);
// The chunks of a run of several instances, for a sort instance by instance.
struct SortChunks {
  const gd::Chunk* chunks = nullptr;
  const gd::DevParams* Pv = nullptr;
  int count = 0;
};
// Whether a run of n points in `chunks` chunks, with keys of `local` bits below the
// instance id's, is sorted instance by instance on the local bits alone.
bool sort_by_instance(int64_t n, int chunks, int local, int bits);
// Stable LSD radix sort of (key, value) pairs on the low `bits` key bits,
// K = uint32_t or unsigned long long.  keys/vals: ping-pong buffers [0] and
// [1]; input in [0].  If vals_in_is_iota, vals[0] is not read and the values
// are taken as 0..n-1.  With chunks: the pairs of each instance by themselves, on the
// low `bits` bits, the instances in their own order (input: in that of the points).
// Returns the index (0 or 1) of the buffer that holds the
// result.  timeouts as for the scan.
template <class K>
int radix_sort_pairs(K* keys[2], uint32_t* vals[2], int64_t n, int bits, bool vals_in_is_iota,
                     void* temp, void* scan_temp, cudaStream_t s,
                     unsigned long long* timeouts = nullptr, const SortChunks& sc = {});
// kernels one radix_sort_pairs call launches
int sort_launches(int64_t n, int bits);
// digit width radix_sort_pairs uses for a `bits`-bit key (8 or 9)
int sort_digit_bits(int bits);
}  // namespace gdprim
