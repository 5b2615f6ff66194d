// The tensor product fused into the inverse transform.
// One of the files that instantiate the transforms (ntt.cuh), each a few kinds so that
// they compile side by side.
#include "kernels.cuh"
#include "ntt.cuh"

namespace fhe_b200 {

namespace {

constexpr int kThreads = 256;

inline unsigned blocks_for(long long work) {
  long long b = (work + kThreads - 1) / kThreads;
  return static_cast<unsigned>(b < 1 ? 1 : b);
}

struct TensorLoad {
  static constexpr bool kFp = false;
  const int64_t *a;
  const int64_t *b;
  long long poly_stride;  // limbs * n
  const uint64_t *q;
  const uint64_t *k;
  // Optional sink of the third polynomial's NTT-form words into each partition's own
  // limbs of ModUp's extended buffer [count][extended][N].
  int64_t *own_ext = nullptr;
  const int *part_start = nullptr;
  const int *part_size = nullptr;
  int part_count = 0;
  int extended = 0;
  bool third_only = false;  // a one-polynomial launch of the third polynomial
  struct Raw {
    int64_t a0, a1, b0, b1;
    int gi, n;
  };
  __device__ __forceinline__ Raw raw(int poly, int limb, int gi, int n) const {
    const long long i = static_cast<long long>(limb) * n + gi;
    if (third_only) poly = 2;
    return {poly != 2 ? a[i] : 0, poly != 0 ? a[poly_stride + i] : 0, poly != 2 ? b[i] : 0,
            poly != 0 ? b[poly_stride + i] : 0, gi, n};
  }
  __device__ __forceinline__ int64_t word(const Raw &x, int poly, int limb, int prime) const {
    const uint64_t qq = q[prime], kk = k[prime];
    if (third_only) poly = 2;
    if (poly == 0) return mont_mult_lazy(x.a0, x.b0, qq, kk);
    if (poly == 2) {
      const int64_t v = mont_mult_lazy(x.a1, x.b1, qq, kk);
      if (own_ext != nullptr) {
        int p = 0;
        while (p + 1 < part_count && limb >= part_start[p] + part_size[p]) p++;
        own_ext[(static_cast<long long>(p) * extended + limb) * x.n + x.gi] = v;
      }
      return v;
    }
    const int64_t qs = static_cast<int64_t>(qq);
    return guard(guard(mont_mult_lazy(x.a0, x.b1, qq, kk) + mont_mult_lazy(x.a1, x.b0, qq, kk), qs << 1), qs);
  }
};

// The tensor's third polynomial d2 = a1 b1 as a streaming pass before a plain mixed
// inverse transform (TensorLoad's words, with 16-byte accesses by a full grid: the
// loader pass of d2 alone waits on its loads and fills under one wave), and its
// NTT-form words into each partition's own limbs of ModUp's extended buffer when one
// is given.  Same words either way.
__global__ void __launch_bounds__(256)
    tensor_third_kernel(PrimeTables t, TensorLoad ld, int log_n, int limbs, int prime_base,
                        int64_t *y) {
  chained_kernel_begin();
  const long long pairs = static_cast<long long>(limbs) << (log_n - 1);
  const long long n = 1LL << log_n;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < pairs;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long w = 2 * i;
    const int limb = static_cast<int>(w >> log_n);
    const int prime = prime_base + limb;
    const uint64_t q = t.q[prime], k = t.k[prime];
    const longlong2 a = *reinterpret_cast<const longlong2 *>(ld.a + ld.poly_stride + w);
    const longlong2 b = *reinterpret_cast<const longlong2 *>(ld.b + ld.poly_stride + w);
    longlong2 v;
    v.x = mont_mult_lazy(a.x, b.x, q, k);
    v.y = mont_mult_lazy(a.y, b.y, q, k);
    *reinterpret_cast<longlong2 *>(y + w) = v;
    if (ld.own_ext != nullptr) {
      int p = 0;
      while (p + 1 < ld.part_count && limb >= ld.part_start[p] + ld.part_size[p]) p++;
      *reinterpret_cast<longlong2 *>(ld.own_ext + (static_cast<long long>(p) * ld.extended) * n + w) = v;
    }
  }
}

}  // namespace

cudaError_t launch_tensor_to_intt(const PrimeTables &t, int log_n, int limbs, int prime_base,
                                  const int64_t *a, const int64_t *b, int64_t *y, cudaStream_t s,
                                  int64_t *own_ext, const DevicePartitions *dp,
                                  const ExactLimbs &exact, bool third_only) {
  const long long stride = static_cast<long long>(limbs) << log_n;
  const int polys = third_only ? 1 : 3;
  TensorLoad ld{a, b, stride, t.q, t.k};
  ld.third_only = third_only;
  if (own_ext != nullptr) {
    if (dp == nullptr) return cudaErrorInvalidValue;
    ld.own_ext = own_ext;
    ld.part_start = dp->start;
    ld.part_size = dp->size;
    ld.part_count = dp->count;
    ld.extended = dp->extended;
  }
  if (exact.poly == ExactLimbs::kAllExact) {
    EnterExitStore<false> st{y, stride, t.n_inverse, t.q, t.k, t.exit_shoup};
    return inverse_ntt(log_n, polys, limbs, prime_base, t, ld, st, y, stride, s);
  }
  MixedExitStore st{y, stride, t.n_inverse, t.q, t.k, t.exit_shoup, exact};
  const bool aligned = (reinterpret_cast<uintptr_t>(a) & 15) == 0 &&
                       (reinterpret_cast<uintptr_t>(b) & 15) == 0 &&
                       (reinterpret_cast<uintptr_t>(y) & 15) == 0 &&
                       (own_ext == nullptr || (reinterpret_cast<uintptr_t>(own_ext) & 15) == 0);
  if (third_only && log_n >= 9 && aligned) {
    // d2 first, then a plain mixed inverse transform in place.
    note_launch();
    launch_chained(tensor_third_kernel, blocks_for(static_cast<long long>(limbs) << (log_n - 1)), kThreads, 0, s,
        t, ld, log_n, limbs, prime_base, y);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    PlainLoad pl{y, stride};
    return inverse_ntt<PlainLoad, MixedExitStore, kNttMixed>(log_n, 1, limbs, prime_base, t, pl, st, y,
                                                             stride, s, exact);
  }
  return inverse_ntt<TensorLoad, MixedExitStore, kNttMixed>(log_n, polys, limbs, prime_base, t, ld,
                                                            st, y, stride, s, exact);
}

}  // namespace fhe_b200
