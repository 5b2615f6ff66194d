// Tensor-core ModDown epilogue (tcgen05.mma kind::i8 on sm_100a).
//
// The reference divides every normal limb by the special primes one after another
// (core_key_switch.cpp:123-160).  Unrolled, limb j of a coefficient becomes
//   v_j = x_j * prod_s pinv_s - sum_s d_s * prod_{t>=s} pinv_t   (mod q_j),
// where d_s is the divisor of step s (special limb K-1-s after s divisions) and
// pinv_s the step's inverse special prime modulo q_j; its final make_unsigned
// leaves v_j canonical in [0, q_j), so any exact evaluation gives the same word.
// Here the sum over s runs on the INT8 tensor pipe:
//   * A (128 coefficients x kb bytes): the 8 little-endian bytes of every d_s as an
//     unsigned word, then one byte [d_s < 0] per divisor (a negative d_s read as
//     unsigned is d_s + 2^64, which the sign byte takes back);
//   * B (per moduli id, built on the host): for target j, the 8 bytes of
//     e_saj = w'_sj 2^(8a) R mod q_j against byte a of d_s, where
//     w'_sj = -prod_{t>=s} pinv_t mod q_j, and of z_sj = -2^64 w'_sj R mod q_j
//     against the sign byte of d_s;
//   * D (tensor memory, S32): 8 columns per target, column b = the exact partial sum
//     of byte b of the constants (each below 2^24), so X_j = sum_b D_b 2^(8b) is
//     congruent to R sum_s d_s w'_sj and below 2^81; one MMA round covers 16
//     targets, so a CTA holds 128 tensor-memory columns and the B of one round, and
//     four CTAs fit on an SM.
// The epilogue folds the 8 partial sums into a 128-bit word, takes one REDC of it
// (a word below q_j + 2^19), adds x_j prod pinv (one Shoup product) and reduces the
// total (below 4 q_j) to [0, q_j).  A target whose prime fp_prime accepts has plain
// constants (no factor R) and is folded, added and rescaled in doubles: about 30
// instructions in place of 90.  Each thread finishes its targets in registers (the rescale's
// dropped limb, target 0, goes to the other half through shared memory first), and the
// next round's B is copied while this one is folded, the first under the triangle.
// The divisor triangle (K(K-1)/2 divisions per coefficient) stays on the CUDA
// cores, as in the CUDA-core form.
#include <cstring>
#include <vector>

#include "kernels.cuh"
#include "modarith.cuh"
#include "umma.cuh"

namespace fhe_b200 {

namespace {

using namespace umma;

constexpr int row_bytes(int K) { return (9 * K + 31) / 32 * 32; }  // d_s bytes + sign bytes

// Four CTAs per SM (64 registers) where that costs no spills, fewer otherwise.
template <int K, bool DOUBLES>
__global__ void __launch_bounds__(kTcThreads, K <= 10 ? 4 : (K <= 13 ? 3 : 1))
    mod_down_tc_kernel(PrimeTables t, KeySwitchTables ks, ModDownTcTables tc, int n,
                       int moduli_id, int L, const int64_t *acc, EpilogueOps ops, int64_t *out,
                       TcStatus status) {
  chained_kernel_begin();
  constexpr int KB = row_bytes(K);
  constexpr int kBBytes = kTcColumns * KB;
  extern __shared__ __align__(128) uint8_t smem[];
  uint8_t *sA = smem;                   // [128 rows][KB], core matrices
  uint8_t *sB = smem + kTcCoeffs * KB;  // two rounds: [128 columns][KB] each
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tmem_base;
  __shared__ int64_t first_limb[kTcCoeffs];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int poly = blockIdx.y;
  const int coeff0 = blockIdx.x * kTcCoeffs;
  const int P = ks.prime_count;
  const int64_t *x = acc + static_cast<long long>(poly) * (L + K) * n + coeff0;

  load_b_round<KB>(sB, tc.b, 0);
  // The triangle's constants in shared memory from eight special primes on, read at fixed
  // offsets (entries past a step's limbs are zero): from the tables each product takes three
  // loads and their addresses (K = 10: 16 products at N = 2^16 893 us, 864 with the copy).
  // Below, the copy and its barrier cost more than they give (K = 4: eight rotations 277 us,
  // 286 with it).
  constexpr bool kCopy = K >= 8;
  __shared__ uint64_t special_q[kCopy ? K : 1], special_k[kCopy ? K : 1];
  __shared__ int64_t special_inverse[kCopy ? K * K : 1];
  if (kCopy) {
    for (int i = tid; i < K * K; i += kTcThreads) {
      const int s = i / K, limb = i % K;
      special_inverse[i] = limb < K - 1 - s ? ks.p_inverse_mult_r[s * P + moduli_id + L + limb] : 0;
      if (i < K) {
        special_q[i] = t.q[moduli_id + L + i];
        special_k[i] = t.k[moduli_id + L + i];
      }
    }
    __syncthreads();
  }

  // 1. Divisor triangle.  From eight special primes on, two adjacent lanes share a
  // coefficient: lane `side` holds the special limbs i = 2 j + side, and each step's divisor
  // comes from its owner by a shuffle; one thread a coefficient left half the warps waiting
  // at the barrier below and ran a chain twice as long (K = 10: serving batch 10946 -> 10585
  // us).  Below, it gains nothing: at K = 6 246.7 us with one lane and 246.2 with two (one
  // product at N = 2^17), at K = 4 two lanes were slower (eight rotations 1307 -> 1326 us).
  // The lanes then write alternate 16-byte chunks of the A row.
  constexpr int kLanes = K >= 8 ? 2 : 1;
  if (tid < kTcCoeffs * kLanes) {
    const int c = tid / kLanes, side = tid % kLanes;
    constexpr int kOwn = (K + kLanes - 1) / kLanes;
    int64_t sp[kOwn];
#pragma unroll
    for (int j = 0; j < kOwn; j++) {
      const int i = kLanes * j + side;
      sp[j] = i < K ? x[static_cast<long long>(L + i) * n + c] : 0;
    }
    uint64_t w[KB / 8];
#pragma unroll
    for (int i = 0; i < KB / 8; i++) w[i] = 0;
#pragma unroll
    for (int s = 0; s < K; s++) {
      const int own = (K - 1 - s) / kLanes;
      const int64_t d = kLanes == 1 ? sp[own]
                                    : __shfl_sync(0xffffffffu, sp[own], (lane & ~1) | ((K - 1 - s) & 1));
      w[s] = static_cast<uint64_t>(d);
      if (d < 0) w[K + (s >> 3)] |= 1ull << (8 * (s & 7));
#pragma unroll
      for (int j = 0; j < kOwn; j++) {
        if (kLanes * j >= K - 1 - s) continue;
        const int i = kLanes * j + side;  // the odd lane may have none left: its product is dropped
        const int limb = i < K ? i : K - 1, prime = moduli_id + L + limb;
        const uint64_t q = kCopy ? special_q[limb] : t.q[prime];
        const int64_t q2 = static_cast<int64_t>(q << 1);
        const int64_t v = mont_mult_const(kCopy ? special_inverse[s * K + limb] : ks.p_inverse_mult_r[s * P + prime],
                                          guard(sp[j] + q2 - d, q2), q, kCopy ? special_k[limb] : t.k[prime]);
        sp[j] = i < K - 1 - s ? v : sp[j];
      }
    }
#pragma unroll
    for (int ch = 0; ch < KB / 16; ch++) {
      if (ch % kLanes != side) continue;
      const uint4 v = make_uint4(static_cast<uint32_t>(w[2 * ch]), static_cast<uint32_t>(w[2 * ch] >> 32),
                                 static_cast<uint32_t>(w[2 * ch + 1]),
                                 static_cast<uint32_t>(w[2 * ch + 1] >> 32));
      *reinterpret_cast<uint4 *>(sA + core_offset(c, ch * 16, kTcCoeffs)) = v;
    }
  }
  if (warp == 0) tmem_alloc(&tmem_base);
  if (tid == 0) mbar_init(&mbar);
  async_copies_wait();
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base;
  const uint32_t bar = smem_addr(&mbar);

  // 2. One MMA round per 16 targets; each thread finishes 8 targets of its coefficient, two at
  // a time.  The loop over the pairs is not unrolled and a launch without targets in doubles is
  // compiled without them: unrolled, the eight copies of both forms' arithmetic and stores
  // waited on the instruction cache (71 launches of the bootstrap, 54-bit primes: 2282 us
  // unrolled, 1974 as a loop, 1757 without the doubles; 16 products at N = 2^16: 1008 and
  // 860 us; eight rotations at K = 4: 309 and 285 us).
  const int lane_base = (warp & 3) * 32;
  const int row = lane_base + lane;
  const int half = warp >> 2;
  const uint32_t tmem_row = tmem + (static_cast<uint32_t>(lane_base) << 16);
  const int64_t *base = poly < ops.base_polys  // uniform per CTA
                            ? ops.base + static_cast<long long>(poly) * L * n + coeff0 + row
                            : nullptr;
  // Target j: x_j divided by the special primes, canonical, and the caller's addend.
  auto divided = [&](int j, const uint32_t *d, int64_t xj) -> int64_t {
    const int prime = moduli_id + j;
    const uint64_t q = t.q[prime];
    int64_t v;
    if (DOUBLES && fp_prime(q) && (static_cast<uint64_t>(xj) >> kFpWordBits) == 0) {
      const FpPrime f{fp_from_word(q), t.inv_q[prime]};
      const double sum = fold_fp(d, f) + fp_mul(fp_from_word(static_cast<uint64_t>(xj)),
                                                fp_from_word(static_cast<uint64_t>(tc.c_shoup[2 * j])), f);
      v = fp_to_word(fp_canonical(fp_reduce(sum, f), f));
    } else {
      uint64_t lo, hi;
      fold8(d, lo, hi);
      // REDC(X) < q + 2^19, and x_j prod pinv by Shoup's product is below 2q.  (A plain sum of
      // an fp_prime target whose word is out of range takes one more factor R.)
      if (DOUBLES && fp_prime(q)) {
        const uint64_t r = static_cast<uint64_t>(redc_wide(lo, hi, q, t.k[prime]));
        lo = static_cast<uint64_t>(mont_mult(static_cast<int64_t>(r), t.r_squared[prime], q, t.k[prime]));
      } else {
        lo = static_cast<uint64_t>(redc_wide(lo, hi, q, t.k[prime]));
      }
      const uint64_t u = lo + shoup_mult(static_cast<uint64_t>(tc.c_shoup[2 * j]),
                                         static_cast<uint64_t>(tc.c_shoup[2 * j + 1]),
                                         static_cast<uint64_t>(xj), q);
      uint64_t r = u >= (q << 1) ? u - (q << 1) : u;
      v = static_cast<int64_t>(r >= q ? r - q : r);
    }
    if (base == nullptr) return v;
    const int64_t qs = static_cast<int64_t>(q);
    return guard(guard(base[static_cast<long long>(j) * n] + v, qs << 1), qs);
  };
  const int32_t place = ops.signed_perm == nullptr ? 0 : ops.signed_perm[coeff0 + row];
  const uint64_t q_half = t.q[moduli_id] >> 1;  // of the dropped prime (unsigned, as get_rounder)
  const long long rescale_row = static_cast<long long>(moduli_id) * P;
  int64_t y0 = 0;
  // Target j's word on its way out: rescaled by the first limb (core_rescale.cpp:5-25), moved
  // by the caller's permutation (rotate_ after key_switch_mod_down, core.cpp:939-952), or as
  // it is.
  auto put = [&](int j, int64_t v) {
    const int prime = moduli_id + j;
    const uint64_t q = t.q[prime];
    const int64_t qs = static_cast<int64_t>(q), q2 = qs << 1;
    if (ops.rescale) {
      const bool up = static_cast<uint64_t>(y0) > q_half;
      const int64_t *shoup = ks.rescale_shoup + 2 * (rescale_row + prime);
      if (DOUBLES && fp_prime(q) && static_cast<uint64_t>(v) < static_cast<uint64_t>(q2) &&
          static_cast<uint64_t>(y0) <= static_cast<uint64_t>(q2)) {
        // Both words in the lazy range: the difference's product is canonical.
        const FpPrime f{fp_from_word(q), t.inv_q[prime]};
        double r = fp_canonical(fp_mul(fp_from_word(static_cast<uint64_t>(v)) - fp_from_word(static_cast<uint64_t>(y0)),
                                       fp_from_word(static_cast<uint64_t>(shoup[0])), f), f);
        r = up ? r + 1.0 : r;
        v = fp_to_word(r >= f.q ? r - f.q : r);
      } else {
        v = rescale_word_shoup(v, y0, up ? 1 : 0, q, t.k[prime], ks.rescale_scale[rescale_row + prime], shoup);
      }
      out[static_cast<long long>(poly) * (L - 1) * n + static_cast<long long>(j - 1) * n + coeff0 + row] = v;
      return;
    }
    int at = coeff0 + row;
    if (ops.signed_perm != nullptr) {
      if (place < 0) v = -v;
      v = v < 0 ? v + qs : guard(v, qs);
      at = place < 0 ? ~place : place;
    }
    out[static_cast<long long>(poly) * L * n + static_cast<long long>(j) * n + at] = v;
  };

  bool ok = true;
  int round = 0;
  for (; round < tc.rounds; round++) {
    if (round > 0) {
      async_copies_wait();
      fence_async_smem();
      __syncthreads();
    }
    if (tid == 0) {
      mma_round(tmem, sA, sB + (round & 1) * kBBytes, KB);
      mma_commit(bar);
    }
    // The other buffer's MMAs have completed: every thread passed their wait.
    if (round + 1 < tc.rounds) load_b_round<KB>(sB + ((round + 1) & 1) * kBBytes, tc.b, round + 1);
    // The halves of the CTA take the round's pairs of targets in turn, so that a round of few
    // targets keeps both busy.  A pair's words x_j are loaded while the MMAs or the pair
    // before it run.
    auto target = [&](int pair) { return round * kTcTargets + 4 * pair + 2 * half; };
    auto word = [&](int j) -> int64_t { return j < L ? x[static_cast<long long>(j) * n + row] : 0; };
    int64_t xa = word(target(0)), xb = word(target(0) + 1);
    ok = __syncthreads_and(mbar_wait(bar, round & 1, status.wait_limit)) != 0;
    if (!ok) break;
    tc_fence_after();
    if (round == 0 && ops.rescale) {
      if (half == 0) {
        uint32_t d[16];
        tmem_load16(tmem_row, d);
        first_limb[row] = divided(0, d, xa);
      }
      __syncthreads();
      y0 = first_limb[row];
    }
#pragma unroll 1
    for (int pair = 0; pair < kTcTargets / 4; pair++) {
      const int j0 = target(pair);
      if (j0 >= L) break;  // uniform across the warp
      uint32_t d[16];
      tmem_load16(tmem_row + (j0 - round * kTcTargets) * 8, d);
      const int64_t xw[2] = {xa, xb};
      if (pair + 1 < kTcTargets / 4) {
        xa = word(target(pair + 1));
        xb = word(target(pair + 1) + 1);
      }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int j = j0 + h;
        if (j < L && !(ops.rescale && j == 0)) put(j, divided(j, d + 8 * h, xw[h]));
      }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
  }
  if (!ok) {
    // The round's MMAs may still be running: wait for them (bounded) before the
    // tensor memory is given back.
    async_copies_wait();
    if (tid == 0) *static_cast<volatile int *>(status.error) = 1;
    if (warp == 0) mbar_wait(bar, round & 1);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem);
}

template <int K, bool DOUBLES>
cudaError_t launch_tc(dim3 grid, size_t smem, const PrimeTables &t, const KeySwitchTables &ks,
                      const ModDownTcTables &tc, int n, int moduli_id, int limbs, const int64_t *acc,
                      const EpilogueOps &ops, int64_t *out, const TcStatus &status, cudaStream_t s) {
  // To the most any supported shape needs, so no attribute call falls inside a graph capture.
  static DeviceOnce raised;
  const cudaError_t e = raise_smem_limit(mod_down_tc_kernel<K, DOUBLES>, 200 * 1024, raised);
  if (e != cudaSuccess) return e;
  note_launch();
  return launch_chained(mod_down_tc_kernel<K, DOUBLES>, grid, kTcThreads, smem, s, t, ks, tc, n, moduli_id,
                        limbs, acc, ops, out, status);
}

size_t tc_smem_bytes(int K) {
  return static_cast<size_t>(kTcCoeffs + 2 * kTcColumns) * row_bytes(K);
}

using u128 = unsigned __int128;

uint64_t mul_mod(uint64_t a, uint64_t b, uint64_t m) {
  return static_cast<uint64_t>(static_cast<u128>(a) * b % m);
}

uint64_t pow_mod(uint64_t b, uint64_t e, uint64_t m) {
  uint64_t r = 1 % m;
  b %= m;
  for (; e; e >>= 1, b = mul_mod(b, b, m))
    if (e & 1) r = mul_mod(r, b, m);
  return r;
}

}  // namespace

bool mod_down_tc_supported(int special_count, int limbs, int n) {
  return special_count >= 1 && special_count <= 16 && limbs >= 1 && n >= kTcCoeffs &&
         n % kTcCoeffs == 0;
}

ModDownTcHost make_mod_down_tc_tables(const std::vector<uint64_t> &q,
                                      const std::vector<std::vector<int64_t>> &p_inverse_mult_r,
                                      int moduli_id, int limbs, int special_count) {
  const int K = special_count, L = limbs;
  ModDownTcHost h;
  h.kb = row_bytes(K);
  h.rounds = (L + kTcTargets - 1) / kTcTargets;
  h.b.assign(static_cast<size_t>(h.rounds) * kTcColumns * h.kb, 0);
  h.c_r.resize(L);
  h.c_shoup.resize(2 * static_cast<size_t>(L));
  for (int j = 0; j < L; j++) {
    const int prime = moduli_id + j;
    const uint64_t m = q[prime];
    const uint64_t r = pow_mod(2, 62, m);
    const uint64_t r_inv = pow_mod(r, m - 2, m);  // m is prime
    std::vector<uint64_t> w(K);
    uint64_t prod = 1 % m;
    for (int s = K - 1; s >= 0; s--) {
      const uint64_t pr = static_cast<uint64_t>(p_inverse_mult_r[s][prime]) % m;
      prod = mul_mod(prod, mul_mod(pr, r_inv, m), m);  // times p_s^-1 mod q_j
      w[s] = prod;
    }
    h.c_r[j] = static_cast<int64_t>(mul_mod(prod, r, m));
    h.c_shoup[2 * j] = static_cast<int64_t>(prod);
    h.c_shoup[2 * j + 1] = static_cast<int64_t>((static_cast<u128>(prod) << 64) / m);
    const uint64_t two64 = static_cast<uint64_t>((static_cast<u128>(1) << 64) % m);
    const int round = j / kTcTargets, jl = j % kTcTargets;
    uint8_t *b = h.b.data() + static_cast<size_t>(round) * kTcColumns * h.kb;
    for (int s = 0; s < K; s++) {
      // w'_sj R, or plain where the target is folded in doubles
      const uint64_t wn = fp_prime(m) ? (m - w[s]) % m : mul_mod((m - w[s]) % m, r, m);
      const uint64_t z = (m - mul_mod(two64, wn, m)) % m;  // -2^64 w'_sj R
      uint64_t e = wn;  // w'_sj 2^(8a) R for a = 0, 1, ...
      for (int a = 0; a < 8; a++) {
        for (int bb = 0; bb < 8; bb++)
          b[core_offset(jl * 8 + bb, s * 8 + a, kTcColumns)] = static_cast<uint8_t>(e >> (8 * bb));
        e = static_cast<uint64_t>((static_cast<u128>(e) << 8) % m);
      }
      for (int bb = 0; bb < 8; bb++)
        b[core_offset(jl * 8 + bb, 8 * K + s, kTcColumns)] = static_cast<uint8_t>(z >> (8 * bb));
    }
  }
  return h;
}

cudaError_t launch_mod_down_epilogue_tc(const PrimeTables &t, const KeySwitchTables &ks,
                                        const ModDownTcTables &tc, int n, int moduli_id,
                                        int limbs, const int64_t *acc, const EpilogueOps &ops,
                                        int64_t *out, const TcStatus &status, cudaStream_t s) {
  const int K = ks.special_count;
  if (!mod_down_tc_supported(K, limbs, n) || tc.b == nullptr || status.error == nullptr ||
      tc.kb != row_bytes(K) || tc.rounds != (limbs + kTcTargets - 1) / kTcTargets ||
      (ops.base_polys > 0 && ops.base == nullptr) || (ops.rescale && ops.signed_perm != nullptr) ||
      ops.polys < 1 || ops.polys > 2 || ops.base_polys > ops.polys)
    return cudaErrorInvalidValue;
  const size_t smem = tc_smem_bytes(K);
  const dim3 grid(n / kTcCoeffs, ops.polys);
  bool doubles = false;
  for (int j = 0; j < limbs; j++) doubles = doubles || t.fp_primes.has(moduli_id + j);
  switch (K) {
#define FHE_TC_CASE(KK)                                                                                   \
  case KK:                                                                                                \
    return doubles                                                                                        \
               ? launch_tc<KK, true>(grid, smem, t, ks, tc, n, moduli_id, limbs, acc, ops, out, status, s) \
               : launch_tc<KK, false>(grid, smem, t, ks, tc, n, moduli_id, limbs, acc, ops, out, status, s);
    FHE_TC_CASE(1) FHE_TC_CASE(2) FHE_TC_CASE(3) FHE_TC_CASE(4) FHE_TC_CASE(5) FHE_TC_CASE(6)
    FHE_TC_CASE(7) FHE_TC_CASE(8) FHE_TC_CASE(9) FHE_TC_CASE(10) FHE_TC_CASE(11) FHE_TC_CASE(12)
    FHE_TC_CASE(13) FHE_TC_CASE(14) FHE_TC_CASE(15) FHE_TC_CASE(16)
#undef FHE_TC_CASE
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fhe_b200
