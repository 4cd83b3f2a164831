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

#include "gd_api.cu"

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

}  // namespace

int main(int argc, char** argv) {
  const std::string name = argc > 1 ? argv[1] : "";
  if (name == "expand_after_a_failed_index") expand_after_a_failed_index();
  else return 2;
  return bad;
}
