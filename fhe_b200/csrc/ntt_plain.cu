// The plain per-limb transforms, and the forward one that attaches the special primes.
// One of the files that instantiate the transforms (ntt.cuh), each a few kinds so that
// they compile side by side.
#include "kernels.cuh"
#include "ntt.cuh"

namespace fhe_b200 {

cudaError_t launch_attach_special_ntt(const PrimeTables &t, const KeySwitchTables &ks, int log_n,
                                      int polys, int limbs, int moduli_id, const int64_t *x,
                                      long long x_stride, int64_t *y, long long y_stride,
                                      cudaStream_t s) {
  const long long n = 1LL << log_n;
  const size_t special_bytes = static_cast<size_t>(ks.special_count) * n * sizeof(int64_t);
  for (int p = 0; p < polys; p++) {
    const cudaError_t e = cudaMemsetAsync(y + p * y_stride + limbs * n, 0, special_bytes, s);
    if (e != cudaSuccess) return e;
  }
  ProductEnterLoad ld{x, x_stride, ks.p_product_mult_r, t.r_squared, t.q, t.k};
  PlainStore st{y, y_stride};
  return forward_ntt(log_n, polys, limbs, moduli_id, t, ld, st, y, y_stride, s);
}

cudaError_t launch_ntt_plain(const PrimeTables &t, int log_n, int polys, int limbs, int prime_base,
                             int64_t *x, long long stride, bool inverse, cudaStream_t s) {
  PlainLoad ld{x, stride};
  PlainStore st{x, stride};
  if (inverse) return inverse_ntt(log_n, polys, limbs, prime_base, t, ld, st, x, stride, s);
  return forward_ntt(log_n, polys, limbs, prime_base, t, ld, st, x, stride, s);
}

}  // namespace fhe_b200
