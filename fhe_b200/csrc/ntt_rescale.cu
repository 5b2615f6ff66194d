// The lazy rescale fused into the forward transform.
// One of the files that instantiate the transforms (ntt.cuh), each a few kinds so that
// they compile side by side.
#include "kernels.cuh"
#include "ntt.cuh"

namespace fhe_b200 {

cudaError_t launch_rescale_to_ntt(const PrimeTables &t, const KeySwitchTables &ks, int log_n,
                                  int polys, int limbs, int src_moduli_id, const int64_t *x,
                                  long long x_stride, int64_t *y, long long y_stride,
                                  cudaStream_t s, const ExactLimbs &exact, int first_polys,
                                  const int64_t *second) {
  const long long row = static_cast<long long>(src_moduli_id) * ks.prime_count;
  PlainStore st{y, y_stride};
  if (exact.poly == ExactLimbs::kAllExact) {
    RescaleEnterLoad<false> ld{x, x_stride, first_polys, second, src_moduli_id, ks.rescale_scale + row,
                               ks.rescale_shoup + 2 * row, t.r_squared, t.q, t.k, t.r_mod,
                               ks.rescale_enter_shoup + 2 * row, exact};
    // A 60-bit dropped prime's words are too wide for the exact form in doubles.
    return forward_ntt(log_n, polys, limbs, src_moduli_id + 1, t, ld, st, y, y_stride, s, nullptr, nullptr,
                       ExactLimbs{}, !t.fp_primes.has(src_moduli_id));
  }
  RescaleEnterLoad<true> ld{x, x_stride, first_polys, second, src_moduli_id, ks.rescale_scale + row,
                            ks.rescale_shoup + 2 * row, t.r_squared, t.q, t.k, t.r_mod,
                            ks.rescale_enter_shoup + 2 * row, exact};
  return forward_ntt<RescaleEnterLoad<true>, PlainStore, kNttMixed>(
      log_n, polys, limbs, src_moduli_id + 1, t, ld, st, y, y_stride, s, nullptr, nullptr, exact);
}

}  // namespace fhe_b200
