// Checks of the context's code around failures that cannot be caused from outside: this
// program holds gd_api.cu itself, so that it can set a counter or refuse an allocation
// between two calls.  Kernels come from libgbdbscan.so.  Usage: ctx_checks NAME; prints
// what differs and exits 1 when a check does not hold.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include "gd_launch.h"

// a small index build after which the wait counter is set, where asked for
namespace gdl {
int index_gives_up = 0;
cudaError_t small_index_checked(const Bufs& B, const gd::SmallArgs& A, int sms, cudaStream_t s) {
  const cudaError_t e = small_index(B, A, sms, s);
  if (index_gives_up) cudaMemsetAsync(B.ctr + gd::kCtrWaitTimeouts, 1, 1, s);
  return e;
}
}  // namespace gdl
#define small_index small_index_checked

// device allocations of more than malloc_limit bytes are refused
size_t malloc_limit = ~(size_t)0, malloc_calls = 0;
cudaError_t limited_malloc(void** p, size_t bytes) {
  ++malloc_calls;
  return bytes > malloc_limit ? cudaErrorMemoryAllocation : cudaMalloc(p, bytes);
}
#define cudaMalloc limited_malloc
#include "gd_api.cu"
#undef cudaMalloc
#include "gd_server.cpp"

namespace {

int bad = 0;
#define CHECK(x)                                              \
  do {                                                        \
    if (!(x)) {                                               \
      std::printf("line %d: %s (%s)\n", __LINE__, #x, gd_last_error()); \
      bad = 1;                                                \
    }                                                         \
  } while (0)

// n points in dim dimensions: clumps and noise over a square or cube of the given side
std::vector<double> points(int64_t n, int dim, double side, unsigned seed) {
  std::mt19937_64 g(seed);
  std::uniform_real_distribution<double> u(0, side);
  std::normal_distribution<double> z(0, 0.4);
  std::vector<double> c(60 * dim), p(n * dim);
  for (double& v : c) v = u(g);
  for (int64_t i = 0; i < n; ++i)
    for (int k = 0; k < dim; ++k) p[i * dim + k] = i % 5 ? c[(i % 60) * dim + k] + z(g) : u(g);
  return p;
}

void* on_device(const void* p, size_t bytes) {
  void* d = nullptr;
  if (cudaMalloc(&d, bytes) != cudaSuccess) std::abort();
  cudaMemcpy(d, p, bytes, cudaMemcpyHostToDevice);
  return d;
}

// labels of the general path, from a context of its own
std::vector<int32_t> general(const std::vector<double>& p, int dim, double eps, int minpts) {
  gd_ctx* c = nullptr;
  std::vector<int32_t> lab(p.size() / dim);
  gd_instance I{(int64_t)lab.size(), dim, minpts, eps};
  CHECK(gd_ctx_create(0, &c) == GD_OK);
  CHECK(gd_batch_dbscan(c, 1, &I, p.data(), 0, lab.data(), nullptr, nullptr) == GD_OK);
  gd_ctx_destroy(c);
  return lab;
}

void set_counter(gd_ctx* c, int which, unsigned long long v) {
  cudaStreamSynchronize(c->stream);
  cudaMemcpy(c->dCtr() + which, &v, 8, cudaMemcpyHostToDevice);
}

// An expand whose index build gave up (a barrier wait ran out) must not touch anything.
void expand_after_a_failed_index() {
  const std::vector<double> p = points(3000, 2, 40, 1);
  gd_ctx* c = nullptr;
  CHECK(gd_ctx_create(0, &c) == GD_OK);
  gd_points g{p.data(), 3000, 2, 0};
  CHECK(gd_index_build(c, &g, 0.3) == GD_OK && c->is_small);
  std::vector<int32_t> out(3000, 77);
  int* d = static_cast<int*>(on_device(out.data(), 3000 * 4));
  set_counter(c, gd::kCtrWaitTimeouts, 1);
  CHECK(gdl::small_expand(c->small_bufs(), c->sa, false, 5, d, c->sms, c->stream) == cudaSuccess);
  CHECK(cudaStreamSynchronize(c->stream) == cudaSuccess);
  cudaMemcpy(out.data(), d, 3000 * 4, cudaMemcpyDeviceToHost);
  CHECK(std::count(out.begin(), out.end(), 77) == 3000);
  cudaFree(d);
  gd_ctx_destroy(c);
}

std::vector<int32_t> result(gd_ctx* c, int64_t n) {
  std::vector<int32_t> lab(n);
  CHECK(gd_get_result(c, lab.data(), nullptr, 0, nullptr, nullptr) == GD_OK);
  return lab;
}

// A small run that gives up in its index build or in an expand gets its labels from the
// general path, and the context goes on working: further expands, then another small run.
void a_small_run_gives_up() {
  for (int dim = 2; dim <= 3; ++dim)
    for (int prec = 0; prec < 2; ++prec) {
      const int64_t n = 5000;
      const std::vector<double> p = points(n, dim, dim == 2 ? 40 : 12, 7 + dim);
      const std::vector<int32_t> w5 = general(p, dim, 0.3, 5), w9 = general(p, dim, 0.3, 9);
      double* d = static_cast<double*>(on_device(p.data(), p.size() * 8));
      const gd_points host{p.data(), n, dim, 0}, dev{d, n, dim, 1};
      gd_ctx* c = nullptr;
      CHECK(gd_ctx_create(0, &c) == GD_OK);
      CHECK(gd_ctx_set_precision(c, prec) == GD_OK);
      gdl::index_gives_up = 1;
      CHECK(gd_index_build(c, &host, 0.3) == GD_OK && !c->is_small);
      gdl::index_gives_up = 0;
      CHECK(gd_expand(c, 5) == GD_OK && result(c, n) == w5);
      for (const gd_points* g : {&host, &dev}) {
        CHECK(gd_index_build(c, g, 0.3) == GD_OK && c->is_small);
        CHECK(gd_expand(c, 9) == GD_OK && result(c, n) == w9 && c->is_small);
        CHECK(gd_expand(c, 5) == GD_OK);
        set_counter(c, gd::kCtrWaitTimeouts, 1);
        if (g->on_device) CHECK(cudaMemset(d, 0, p.size() * 8) == cudaSuccess);
        CHECK(result(c, n) == w5 && !c->is_small);
        CHECK(gd_expand(c, 9) == GD_OK && result(c, n) == w9);
        CHECK(gd_expand(c, 5) == GD_OK && result(c, n) == w5);
      }
      std::vector<int32_t> lab(n);
      CHECK(gd_dbscan(c, &host, 0.3, 9, lab.data(), nullptr) == GD_OK && lab == w9 && c->is_small);
      cudaFree(d);
      gd_ctx_destroy(c);
    }
}

gd_status batch(gd_ctx* c, const std::vector<double>& p, int dim, double eps, int minpts,
                std::vector<int32_t>& lab) {
  lab.assign(p.size() / dim, 0);
  const gd_instance I{(int64_t)lab.size(), dim, minpts, eps};
  return gd_batch_dbscan(c, 1, &I, p.data(), 0, lab.data(), nullptr, nullptr);
}

// A small run leaves a large run's buffers where they are.
void a_small_run_after_a_large_one() {
  const std::vector<double> large = points(300000, 3, 60, 3), small = points(1000, 2, 20, 4);
  gd_ctx* c = nullptr;
  CHECK(gd_ctx_create(0, &c) == GD_OK);
  std::vector<int32_t> lab;
  CHECK(batch(c, large, 3, 0.3, 8, lab) == GD_OK);
  const void* slab = c->run_slab;
  const size_t bytes = c->X.bytes;
  std::vector<int32_t> got(1000);
  const gd_points g{small.data(), 1000, 2, 0};
  malloc_calls = 0;
  malloc_limit = 4 << 20;  // the buffers of 1,000 points
  CHECK(gd_dbscan(c, &g, 0.3, 5, got.data(), nullptr) == GD_OK && c->is_small);
  malloc_limit = ~(size_t)0;
  CHECK(got == general(small, 2, 0.3, 5));
  CHECK(c->run_slab == slab && c->X.bytes == bytes);
  malloc_calls = 0;
  CHECK(batch(c, large, 3, 0.3, 8, lab) == GD_OK && malloc_calls == 0);
  CHECK(gd_dbscan(c, &g, 0.3, 5, got.data(), nullptr) == GD_OK && malloc_calls == 0);
  gd_ctx_destroy(c);
}

// A run that fits the device is not refused for the sizes that earlier runs left.
void kept_sizes_do_not_refuse_a_run() {
  gd_ctx* c = nullptr;
  CHECK(gd_ctx_create(0, &c) == GD_OK);
  std::vector<int32_t> lab;
  // a hashed 3D grid, then a larger set on a direct 2D grid
  const std::vector<double> wide = points(200000, 3, 1e5, 5), dense = points(260000, 2, 40, 6);
  const std::vector<int32_t> want = general(dense, 2, 0.3, 8);
  gd_ctx* own = nullptr;  // what the second run takes by itself
  CHECK(gd_ctx_create(0, &own) == GD_OK && batch(own, dense, 2, 0.3, 8, lab) == GD_OK);
  size_t alone = 0, both = 0;
  for (DevBuf* b : own->run_set) alone += b->bytes;
  gd_ctx_destroy(own);
  CHECK(batch(c, wide, 3, 0.3, 8, lab) == GD_OK);
  for (DevBuf* b : c->run_set) both += b->bytes;
  CHECK(both > alone);
  malloc_limit = alone;
  CHECK(batch(c, dense, 2, 0.3, 8, lab) == GD_OK && lab == want);
  malloc_limit = ~(size_t)0;
  gd_ctx_destroy(c);
}

// A run whose buffers do not fit at a cell per point gets them by the counted cells: same
// labels over direct, row-table and hashed grids and a mixed batch, for repeated expands, and
// with every walk handed to the warp kernels (the heavy lists' size).
void buffers_by_the_counted_cells() {
  struct Case { int64_t n; int dim; double side; };
  for (int prec = 0; prec < 2; ++prec)
    for (const Case& k : {Case{300000, 2, 100}, Case{300000, 2, 3e6}, Case{150000, 3, 40},
                          Case{150000, 3, 3e3}, Case{150000, 3, 1e5}})
      for (int warps = 0; warps < 2; ++warps) {
        const std::vector<double> p = points(k.n, k.dim, k.side, 11);
        const gd_points g{p.data(), k.n, k.dim, 0};
        gd_ctx* c = nullptr;
        CHECK(gd_ctx_create(0, &c) == GD_OK && gd_ctx_set_precision(c, prec) == GD_OK);
        if (warps) {
          const gd_tuning t{0, 0, 0, 0, 0, 0};
          CHECK(gd_ctx_set_tuning(c, &t) == GD_OK);
        }
        std::vector<int32_t> want[3];
        const int mp[3] = {8, 4, 20};
        CHECK(gd_index_build(c, &g, 0.3) == GD_OK && !c->is_small && !c->lean);
        for (int e = 0; e < 3; ++e) {
          CHECK(gd_expand(c, mp[e]) == GD_OK);
          want[e] = result(c, k.n);
        }
        size_t all = 0;
        for (DevBuf* b : c->run_set) all += b->bytes;
        CHECK(gd_ctx_trim(c) == GD_OK);
        malloc_limit = all - 1;
        CHECK(gd_index_build(c, &g, 0.3) == GD_OK && c->lean && c->cells_cap < k.n);
        for (int e = 0; e < 3; ++e) {
          CHECK(gd_expand(c, mp[e]) == GD_OK);
          CHECK(result(c, k.n) == want[e]);
        }
        // the room is there again
        malloc_limit = ~(size_t)0;
        CHECK(gd_index_build(c, &g, 0.3) == GD_OK && (!c->lean || prec == 0));
        CHECK(gd_expand(c, 8) == GD_OK && result(c, k.n) == want[0]);
        gd_ctx_destroy(c);
      }
  // a batch of both dimensions and all three lookups
  std::vector<double> p;
  std::vector<gd_instance> inst;
  for (int i = 0; i < 24; ++i) {
    const int dim = 2 + i % 2;
    const double side[2][3] = {{30, 2e4, 3e6}, {30, 150, 2e4}};
    const std::vector<double> q = points(3000 + 997 * i, dim, side[dim - 2][i / 2 % 3], i);
    inst.push_back({(int64_t)q.size() / dim, dim, 5 + i % 3, 0.3});
    p.insert(p.end(), q.begin(), q.end());
  }
  int64_t n = 0;
  for (const gd_instance& i : inst) n += i.n;
  for (int prec = 0; prec < 2; ++prec) {
    gd_ctx* c = nullptr;
    CHECK(gd_ctx_create(0, &c) == GD_OK && gd_ctx_set_precision(c, prec) == GD_OK);
    std::vector<int32_t> want(n), lab(n);
    auto run = [&](std::vector<int32_t>& out) {
      return gd_batch_dbscan(c, (int)inst.size(), inst.data(), p.data(), 0, out.data(), nullptr,
                             nullptr);
    };
    CHECK(run(want) == GD_OK && !c->lean);
    size_t all = 0;
    for (DevBuf* b : c->run_set) all += b->bytes;
    CHECK(gd_ctx_trim(c) == GD_OK);
    malloc_limit = all - 1;
    CHECK(run(lab) == GD_OK && c->lean && lab == want);
    malloc_limit = ~(size_t)0;
    gd_ctx_destroy(c);
  }
}

// The server admits requests by an estimate of their device memory, which a batch's buffers
// must not pass: every lookup alone, and mixed so that most instances have a direct table and
// the batch still holds slots and a row hash.
void server_estimate() {
  for (int prec = 0; prec < 2; ++prec)
    for (int mix = 0; mix < 5; ++mix) {
      std::vector<double> p;
      std::vector<gd_instance> inst;
      for (int i = 0; i < 40; ++i) {
        const int dim = 3, n = 13200;  // (the row hash has almost four slots per point)
        // blocks of just below one per point: direct; rows below 8 per point: table; else hash
        const double block = 4 * 0.3 / std::sqrt(3.0), direct = 22.9 * block, rows = 323 * block;
        const double side = mix == 0   ? direct
                            : mix == 1 ? rows
                            : mix == 2 ? 2e4
                            : mix == 3 ? (i ? direct : 2e4)
                                       : (i ? rows : 2e4);
        std::mt19937_64 g(i);
        std::uniform_real_distribution<double> u(0, side);
        for (int k = 0; k < n * dim; ++k) p.push_back(u(g));
        inst.push_back({n, dim, 5, 0.3});
      }
      const int64_t n = (int64_t)p.size() / 3;
      std::vector<int32_t> lab(n);
      gd_ctx* c = nullptr;
      CHECK(gd_ctx_create(0, &c) == GD_OK && gd_ctx_set_precision(c, prec) == GD_OK);
      CHECK(gd_batch_dbscan(c, (int)inst.size(), inst.data(), p.data(), 0, lab.data(), nullptr,
                            nullptr) == GD_OK);
      size_t bytes = c->coords.bytes + c->out.bytes;
      for (DevBuf* b : c->run_set) bytes += b->bytes;
      for (DevBuf* b : c->table_set) bytes += b->bytes;
      std::printf("precision %d mix %d: %.1f bytes per point\n", prec, mix, (double)bytes / n);
      CHECK((int64_t)bytes <= n * kBytesPerPoint + (int64_t)inst.size() * kBytesPerRequest);
      CHECK((mix == 0) == (c->bi.row_total == 0 && !c->bi.any_sparse));
      gd_ctx_destroy(c);
    }
}

}  // namespace

int main(int argc, char** argv) {
  const std::string name = argc > 1 ? argv[1] : "";
  if (name == "expand_after_a_failed_index") expand_after_a_failed_index();
  else if (name == "a_small_run_gives_up") a_small_run_gives_up();
  else if (name == "a_small_run_after_a_large_one") a_small_run_after_a_large_one();
  else if (name == "kept_sizes_do_not_refuse_a_run") kept_sizes_do_not_refuse_a_run();
  else if (name == "buffers_by_the_counted_cells") buffers_by_the_counted_cells();
  else if (name == "server_estimate") server_estimate();
  else return 2;
  return bad;
}
