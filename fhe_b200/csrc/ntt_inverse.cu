// to_intt: the exact inverse transform, N^-1 and Montgomery exit.
// One of the files that instantiate the transforms (ntt.cuh), each a few kinds so that
// they compile side by side.
#include "kernels.cuh"
#include "ntt.cuh"

namespace fhe_b200 {

cudaError_t launch_to_intt(const PrimeTables &t, int log_n, int polys, int limbs, int prime_base,
                           const int64_t *x, long long x_stride, int64_t *y, long long y_stride,
                           cudaStream_t s) {
  PlainLoad ld{x, x_stride};
  EnterExitStore<false> st{y, y_stride, t.n_inverse, t.q, t.k, t.exit_shoup};
  return inverse_ntt(log_n, polys, limbs, prime_base, t, ld, st, y, y_stride, s);
}

}  // namespace fhe_b200
