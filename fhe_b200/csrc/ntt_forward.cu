// to_ntt: Montgomery enter and the exact forward transform.
// One of the files that instantiate the transforms (ntt.cuh), each a few kinds so that
// they compile side by side.
#include "kernels.cuh"
#include "ntt.cuh"

namespace fhe_b200 {

cudaError_t launch_to_ntt(const PrimeTables &t, int log_n, int polys, int limbs, int prime_base,
                          const int64_t *x, long long x_stride, int64_t *y, long long y_stride,
                          cudaStream_t s) {
  EnterLoad ld{x, x_stride, t.r_squared, t.r_mod, t.q, t.k};
  PlainStore st{y, y_stride};
  return forward_ntt(log_n, polys, limbs, prime_base, t, ld, st, y, y_stride, s);
}

}  // namespace fhe_b200
