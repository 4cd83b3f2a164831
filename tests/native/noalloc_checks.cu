// gd_dbscan_noalloc around a barrier wait that gives up: this program holds gd_noalloc.cu
// itself and sets the wait counter behind the index build or the expand.  Kernels come from
// libgbdbscan.so.  Prints what differs and exits 1 when a check does not hold.
#include <cstdio>
#include <random>
#include <vector>

#include "gd_launch.h"

namespace gdl {
int gives_up = 0;  // 1: index build, 2: expand
cudaError_t small_index_checked(const Bufs& B, const gd::SmallArgs& A, int sms, cudaStream_t s) {
  const cudaError_t e = small_index(B, A, sms, s);
  if (gives_up == 1) cudaMemsetAsync(B.ctr + gd::kCtrWaitTimeouts, 1, 1, s);
  return e;
}
cudaError_t small_expand_checked(const Bufs& B, const gd::SmallArgs& A, bool f32, int minpts,
                                 int* out, int sms, cudaStream_t s) {
  const cudaError_t e = small_expand(B, A, f32, minpts, out, sms, s);
  if (gives_up == 2) cudaMemsetAsync(B.ctr + gd::kCtrWaitTimeouts, 1, 1, s);
  return e;
}
}  // namespace gdl
#define small_index small_index_checked
#define small_expand small_expand_checked
#include "gd_noalloc.cu"

int main() {
  int bad = 0;
  for (int dim = 2; dim <= 3; ++dim)
    for (int prec = 0; prec < 2; ++prec) {
      const int64_t n = 4000;
      std::mt19937_64 g(dim);
      std::normal_distribution<double> z(0, 1.0);
      std::vector<double> p(n * dim);
      for (int64_t i = 0; i < n; ++i)
        for (int k = 0; k < dim; ++k) p[i * dim + k] = z(g) + 6.0 * (i % 9) * (k == 0);
      double* d = nullptr;
      int32_t* out = nullptr;
      if (cudaMalloc(&d, p.size() * 8) != cudaSuccess || cudaMalloc(&out, n * 4) != cudaSuccess)
        return 3;
      cudaMemcpy(d, p.data(), p.size() * 8, cudaMemcpyHostToDevice);
      std::vector<int32_t> want(n), lab(n);
      int64_t clusters[4] = {};
      for (int how = 0; how < 4; ++how) {  // sound, index gives up, expand gives up, sound
        gdl::gives_up = how % 3;
        const gd_status st =
            gd_dbscan_noalloc(d, n, dim, 0.25, 6, prec, out, &clusters[how], nullptr);
        cudaMemcpy((how ? lab : want).data(), out, n * 4, cudaMemcpyDeviceToHost);
        if (st != GD_OK || (how && (lab != want || clusters[how] != clusters[0]))) {
          std::printf("dim %d precision %d case %d: status %d\n", dim, prec, how, (int)st);
          bad = 1;
        }
      }
      cudaFree(d);
      cudaFree(out);
    }
  return bad;
}
