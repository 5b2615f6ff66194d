// ModUp's forward and ModDown's inverse transform, whose words only matter modulo q.
// One of the files that instantiate the transforms (ntt.cuh), each a few kinds so that
// they compile side by side.
#include "kernels.cuh"
#include "ntt.cuh"

namespace fhe_b200 {

cudaError_t launch_extended_ntt(const PrimeTables &t, const DevicePartitions &dp, int log_n,
                                int moduli_id, int64_t *ext, cudaStream_t s, bool skip_own) {
  const long long stride = static_cast<long long>(dp.extended) << log_n;
  PlainLoad ld{ext, stride};
  PlainStore st{ext, stride};
  // Value-only: the extended polynomial reaches the output only through the key
  // inner product's reduction to [0, q) and ModDown's reduced inverse transform.
  return forward_ntt<PlainLoad, PlainStore, kNttValueOnly>(log_n, dp.count, dp.extended, moduli_id, t,
                                                           ld, st, ext, stride, s,
                                                           skip_own ? dp.start : nullptr,
                                                           skip_own ? dp.size : nullptr);
}

cudaError_t launch_mod_down_intt(const PrimeTables &t, int log_n, int moduli_id, int extended,
                                 int64_t *acc, cudaStream_t s, int polys) {
  if (polys < 1 || polys > 2) return cudaErrorInvalidValue;
  const long long stride = static_cast<long long>(extended) << log_n;
  PlainLoad ld{acc, stride};
  EnterExitStore<true> st{acc, stride, t.n_inverse, t.q, t.k, t.exit_shoup};
  // Value-only: the store reduces every word to [0, q).
  return inverse_ntt<PlainLoad, EnterExitStore<true>, kNttValueOnly>(log_n, polys, extended,
                                                                     moduli_id, t, ld, st, acc,
                                                                     stride, s);
}

}  // namespace fhe_b200
