// Batched negacyclic NTT / inverse NTT for the B200 CKKS engine.
//
// The transform of one limb (N = 2^log_n words) is split into passes.  A pass
// performs S consecutive radix-2 stages on independent sub-transforms of 2^S words
// each: "strided" passes take one word out of every T = 2^(log_n - S) (the early
// forward stages / late inverse stages), "contiguous" passes take 2^S adjacent
// words.  A CTA stages a tile of sub-transforms in shared memory; inside a tile the
// stages are done three or four at a time in registers, so shared memory is touched
// once per three or four stages.  The first round of a pass reads global memory
// through a Loader and the last round writes through a Storer, which is where the
// element-wise work before and after a transform (Montgomery enter, N^-1 scaling,
// key products ...) is fused.
//
// Each butterfly is exactly the reference's (operation/ntt.cpp:46-134 forward,
// Cooley-Tukey with the bit-reversed psi table; 177-272 inverse, Gentleman-Sande
// with the "backward paint" table), so the output words are bit-identical whatever
// the pass split.
//
// The limbs of the 40- and 41-bit scaling primes are computed in doubles (ntt_pass_fp),
// the others in integers (ntt_pass_int).
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "kernels.cuh"
#include "modarith.cuh"

namespace fhe_b200 {

void note_launch(unsigned count);

// Which words a transform must reproduce (template parameter VALUE_ONLY):
//   kNttExact      every butterfly is the reference's, every word identical;
//   kNttValueOnly  only each result's value modulo q matters (Harvey's butterflies
//                  on Shoup twiddles where the words are in range);
//   kNttMixed      value-only except the limbs that NttPass::exact names, which take
//                  the exact butterflies (a CTA transforms one limb, so the choice is
//                  uniform per CTA).
constexpr int kNttExact = 0;
constexpr int kNttValueOnly = 1;
constexpr int kNttMixed = 2;

struct NttPass {
  int log_n;
  int stages;       // S, the stages of this pass
  int stride_log;   // log2(T); 0 for contiguous passes
  int columns_log;  // log2(sub-transforms per CTA tile) of the integer limbs
  int first;        // stages done before this pass
  int polys;
  int limbs;
  int prime_base;  // prime index of limb 0
  // Optional: polynomial p's limbs [skip_start[p], skip_start[p] + skip_size[p]) are
  // left untouched (ModUp's partitions' own limbs, already in NTT form).
  const int *skip_start = nullptr;
  const int *skip_size = nullptr;
  // A kNttMixed transform keeps the exact butterflies on these limbs only.
  ExactLimbs exact;
};

// A Loader reads word gi of (poly, limb) as it lies (raw), so that a thread has all its
// loads in flight before it works on any, and makes the transform's word of it:
//   word   as an integer;
//   fp     on a limb in doubles (kFp: it has them; the generic form converts `word`).
//          EXACT: the exact word, an integer in [0, 2q), or `bad` is set and the CTA takes
//          the integer pass.  Otherwise any value congruent modulo q and below 2^42, for
//          raw words that are not `odd` (negative, or 2^42 and more);
//   fp_any the same for odd ones.
// A Storer takes the result as an integer word, or as a double: EXACT the exact word,
// otherwise a value below 2^50 whose word may be any of [0, 2q); `before` reads what lies
// there where the store adds to it, again ahead of all stores.
// Constants per prime are read once a thread (Const).

__device__ __forceinline__ bool fp_odd(int64_t w) { return (static_cast<uint64_t>(w) >> kFpWordBits) != 0; }
__device__ __forceinline__ double fp_small(int64_t w) { return fp_from_word(static_cast<uint64_t>(w)); }
// An exact word of [0, 2q).
__device__ __forceinline__ double fp_exact_word(int64_t w, const FpPrime &f, bool &bad) {
  const double x = fp_from_word(static_cast<uint64_t>(w) & 0x000FFFFFFFFFFFFFull);
  bad = bad || fp_odd(w) || x >= 2.0 * f.q;
  return x;
}
// A double as a word of [0, 2q): an exact one as it is, a value reduced to about q / 2
// around zero and shifted by q.
template <bool EXACT>
__device__ __forceinline__ int64_t fp_store_word(double x, const FpPrime &f) {
  return fp_to_word(EXACT ? x : fp_reduce(x, f) + f.q);
}

struct NoConst {};

// Reads word gi of (poly, limb) from a [poly][limb][N] buffer.
struct PlainLoad {
  static constexpr bool kFp = true;
  using Raw = int64_t;
  using Const = NoConst;
  const int64_t *src;
  long long poly_stride;
  __device__ __forceinline__ Raw raw(int poly, int limb, int gi, int n) const {
    return src[poly * poly_stride + (long long)limb * n + gi];
  }
  __device__ __forceinline__ int64_t word(Raw w, int, int, int) const { return w; }
  __device__ __forceinline__ Const constants(int, const FpPrime &) const { return {}; }
  template <bool EXACT>
  __device__ __forceinline__ bool odd(Raw w) const { return fp_odd(w); }
  template <bool EXACT>
  __device__ __forceinline__ double fp(Raw w, const Const &, const FpPrime &f, bool &bad) const {
    return EXACT ? fp_exact_word(w, f, bad) : fp_small(w);
  }
  __device__ __forceinline__ double fp_any(Raw w, const Const &, const FpPrime &f) const {
    return fp_from_any_word(w, f);
  }
};

struct PlainStore {
  using Const = NoConst;
  int64_t *dst;
  long long poly_stride;
  __device__ __forceinline__ void word(int poly, int limb, int, int gi, int n, int64_t v) const {
    dst[poly * poly_stride + (long long)limb * n + gi] = v;
  }
  __device__ __forceinline__ Const constants(int, const FpPrime &) const { return {}; }
  __device__ __forceinline__ int64_t before(int, int, int) const { return 0; }
  template <bool EXACT>
  __device__ __forceinline__ void fp(int poly, int limb, int prime, int gi, int n, const Const &,
                                     const FpPrime &f, int64_t, double x) const {
    word(poly, limb, prime, gi, n, fp_store_word<EXACT>(x, f));
  }
};

// The words between the two passes of a transform: as PlainLoad and PlainStore, but the
// values of an FP64 limb that only matter modulo q stay the doubles they are.
struct MidLoad : PlainLoad {
  template <bool EXACT>
  __device__ __forceinline__ bool odd(Raw w) const { return EXACT && fp_odd(w); }
  template <bool EXACT>
  __device__ __forceinline__ double fp(Raw w, const Const &, const FpPrime &f, bool &bad) const {
    return EXACT ? fp_exact_word(w, f, bad) : fp_bits(static_cast<uint64_t>(w));
  }
};
struct MidStore : PlainStore {
  template <bool EXACT>
  __device__ __forceinline__ void fp(int poly, int limb, int prime, int gi, int n, const Const &,
                                     const FpPrime &f, int64_t, double x) const {
    word(poly, limb, prime, gi, n, EXACT ? fp_to_word(x) : static_cast<int64_t>(fp_raw(x)));
  }
};

// A constant multiplier: the plain residue, its quotient by q, the Montgomery word 2^-62.
struct FpFactor {
  double w, w_over_q, w_mont;
};
__device__ __forceinline__ FpFactor fp_factor(int64_t plain, int64_t mont, const FpPrime &f) {
  const double w = fp_small(plain);
  return {w, w * f.inv_q, fp_small(mont) * kFpMontScale};
}

// mont_enter by a per-prime constant on the way in: to_ntt_ (core_ntt.cpp:91-100).
struct EnterLoad {
  static constexpr bool kFp = true;
  using Raw = int64_t;
  using Const = FpFactor;
  const int64_t *src;
  long long poly_stride;
  const int64_t *constant;  // indexed by prime
  const int64_t *plain;     // constant R^-1, indexed by prime
  const uint64_t *q;
  const uint64_t *k;
  __device__ __forceinline__ Raw raw(int poly, int limb, int gi, int n) const {
    return src[poly * poly_stride + (long long)limb * n + gi];
  }
  __device__ __forceinline__ int64_t word(Raw x, int, int, int prime) const {
    return mont_mult_lazy(x, constant[prime], q[prime], k[prime]);
  }
  __device__ __forceinline__ Const constants(int prime, const FpPrime &f) const {
    return fp_factor(plain[prime], constant[prime], f);
  }
  template <bool EXACT>
  __device__ __forceinline__ bool odd(Raw x) const { return fp_odd(x); }
  template <bool EXACT>
  __device__ __forceinline__ double fp(Raw x, const Const &c, const FpPrime &f, bool &bad) const {
    if (!EXACT) return fp_mul(fp_small(x), c.w, c.w_over_q, f.q);
    bad = bad || fp_odd(x);
    return fp_mont_mult(fp_small(x & ((int64_t(1) << kFpWordBits) - 1)), c.w, c.w_over_q, c.w_mont, f);
  }
  __device__ __forceinline__ double fp_any(Raw x, const Const &c, const FpPrime &f) const {
    return fp_mul(fp_from_any_word(x, f), c.w, c.w_over_q, f.q);
  }
};

// rescale_once_ (core_rescale.cpp:5-25) and to_ntt_'s enter on the way in: limb
// `limb` of the rescaled text is made from limbs limb + 1 and 0 of the source, whose
// first prime is prime - limb - 1 (the rounder compares unsigned, as get_rounder).
//
// MIXED: the limbs outside `exact` only matter modulo q.  Their word is
// ((x_j - x_0) q_0^-1 + rounder) R mod q, the value of the two steps, formed as one
// Shoup product of the difference by q_0^-1 R plus the rounder's R, in [0, 2q); a
// difference still negative after adding 2q (words far out of range) takes the
// exact steps, whose value is the same.
template <bool MIXED = false>
struct RescaleEnterLoad {
  static constexpr bool kFp = true;
  struct Raw {
    int64_t x0, xj;
  };
  struct Const {
    FpFactor enter;        // R: r_mod, r_squared
    double rescale;        // q_0^-1 (exact)
    double rescale_enter;  // q_0^-1 R (a value)
    uint64_t half;         // of the dropped prime
  };
  const int64_t *src;             // [poly][limbs + 1][N]
  long long poly_stride;
  int first_polys;                // polynomials from this one on come from `second`
  const int64_t *second;
  int dropped;                    // the dropped prime
  const int64_t *rescale_scale;   // its row, indexed by prime
  const int64_t *rescale_shoup;   // the same row's (C, C') pairs
  const int64_t *r_squared;
  const uint64_t *q;
  const uint64_t *k;
  const int64_t *r_mod;        // R mod q, indexed by prime
  const int64_t *enter_shoup;  // the row's rescale_enter_shoup pairs
  ExactLimbs exact;            // MIXED
  __device__ __forceinline__ Raw raw(int poly, int limb, int gi, int n) const {
    const int64_t *s = poly < first_polys ? src + poly * poly_stride : second + (poly - first_polys) * poly_stride;
    return {s[gi], s[static_cast<long long>(limb + 1) * n + gi]};
  }
  __device__ __forceinline__ int64_t word(Raw x, int poly, int limb, int prime) const {
    const int64_t rounder = static_cast<uint64_t>(x.x0) > (q[dropped] >> 1) ? 1 : 0;
    const uint64_t qq = q[prime], kk = k[prime];
    if (MIXED && !exact.exact(poly, limb)) {
      const int64_t q2 = static_cast<int64_t>(qq << 1);
      int64_t d = x.xj - x.x0;
      d = d >= 0 ? d : d + q2;
      if (d >= 0) {
        const uint64_t y = shoup_mult(static_cast<uint64_t>(enter_shoup[2 * prime]),
                                      static_cast<uint64_t>(enter_shoup[2 * prime + 1]),
                                      static_cast<uint64_t>(d), qq) +
                           (rounder ? static_cast<uint64_t>(r_mod[prime]) : 0);  // [0, 3q)
        return static_cast<int64_t>(y) >= q2 ? static_cast<int64_t>(y) - q2 : static_cast<int64_t>(y);
      }
    }
    const int64_t v = rescale_word_shoup(x.xj, x.x0, rounder, qq, kk, rescale_scale[prime],
                                         rescale_shoup + 2 * prime);
    return mont_mult_lazy(v, r_squared[prime], qq, kk);
  }
  __device__ __forceinline__ Const constants(int prime, const FpPrime &f) const {
    return {fp_factor(r_mod[prime], r_squared[prime], f), fp_small(rescale_shoup[2 * prime]),
            fp_small(enter_shoup[2 * prime]), q[dropped] >> 1};
  }
  template <bool EXACT>
  __device__ __forceinline__ bool odd(Raw x) const { return fp_odd(x.x0 | x.xj); }
  // The difference, its product by q_0^-1 (a value: by q_0^-1 R) and the rounder as above.
  // The exact word's steps need the difference non-negative after one 2q (their result is
  // then canonical before the enter).
  template <bool EXACT>
  __device__ __forceinline__ double fp(Raw x, const Const &c, const FpPrime &f, bool &bad) const {
    const bool up = static_cast<uint64_t>(x.x0) > c.half;
    if (!EXACT) {
      const double y = fp_mul(fp_small(x.xj) - fp_small(x.x0), c.rescale_enter, f);
      return up ? y + c.enter.w : y;
    }
    constexpr int64_t kMask = (int64_t(1) << kFpWordBits) - 1;
    double d = fp_small(x.xj & kMask) - fp_small(x.x0 & kMask);
    d = fp_negative(d) ? d + 2.0 * f.q : d;
    bad = bad || odd<true>(x) || fp_negative(d);
    double r = fp_canonical(fp_mul(d, c.rescale, f), f);
    r = up ? r + 1.0 : r;
    r = r >= f.q ? r - f.q : r;
    return fp_mont_mult(r, c.enter.w, c.enter.w_over_q, c.enter.w_mont, f);
  }
  __device__ __forceinline__ double fp_any(Raw x, const Const &c, const FpPrime &f) const {
    const double y = fp_mul(fp_from_any_word(x.xj, f) - fp_from_any_word(x.x0, f), c.rescale_enter, f);
    return static_cast<uint64_t>(x.x0) > c.half ? y + c.enter.w : y;
  }
};

// attach_special_prime_chains_ (core.cpp:1127-1155) on the way in: x * P R^-1
// (mont_enter_scalar_ by P * R mod q) then to_ntt_'s enter.
struct ProductEnterLoad {
  static constexpr bool kFp = false;
  using Raw = int64_t;
  const int64_t *src;
  long long poly_stride;
  const int64_t *p_product;  // P * R mod q, indexed by prime
  const int64_t *r_squared;
  const uint64_t *q;
  const uint64_t *k;
  __device__ __forceinline__ Raw raw(int poly, int limb, int gi, int n) const {
    return src[poly * poly_stride + (long long)limb * n + gi];
  }
  __device__ __forceinline__ int64_t word(Raw x, int, int, int prime) const {
    const uint64_t qq = q[prime], kk = k[prime];
    return mont_mult_lazy(mont_mult_lazy(x, p_product[prime], qq, kk), r_squared[prime], qq, kk);
  }
};

// mont_enter_exit by N^-1*R on the way out: to_intt_ (core_ntt.cpp:131-148),
// optionally followed by reduce_2q_to_q (mod_down, core_key_switch.cpp:121).  With
// the reduction the word is the canonical residue of v N^-1 R^-1, so for v in
// [0, 2^62) one Shoup product by that constant and one subtraction give it.
template <bool REDUCE>
struct EnterExitStore {
  using Const = FpFactor;
  int64_t *dst;
  long long poly_stride;
  const int64_t *n_inverse;
  const uint64_t *q;
  const uint64_t *k;
  const int64_t *exit_shoup;  // PrimeTables::exit_shoup
  __device__ __forceinline__ void word(int poly, int limb, int prime, int gi, int n, int64_t v) const {
    const uint64_t qq = q[prime], kk = k[prime];
    if (REDUCE && (static_cast<uint64_t>(v) >> kMontBits) == 0) {
      const uint64_t r = shoup_mult(static_cast<uint64_t>(exit_shoup[2 * prime]),
                                    static_cast<uint64_t>(exit_shoup[2 * prime + 1]),
                                    static_cast<uint64_t>(v), qq);
      dst[poly * poly_stride + (long long)limb * n + gi] = static_cast<int64_t>(r >= qq ? r - qq : r);
      return;
    }
    int64_t y = mont_exit(mont_mult_lazy(v, n_inverse[prime], qq, kk), qq, kk);
    if (REDUCE) y = guard(y, static_cast<int64_t>(qq));
    dst[poly * poly_stride + (long long)limb * n + gi] = y;
  }
  __device__ __forceinline__ Const constants(int prime, const FpPrime &f) const {
    return fp_factor(exit_shoup[2 * prime], 0, f);
  }
  __device__ __forceinline__ int64_t before(int, int, int) const { return 0; }
  template <bool EXACT>
  __device__ __forceinline__ void fp(int poly, int limb, int, int gi, int n, const Const &c,
                                     const FpPrime &f, int64_t, double x) const {
    const double r = fp_canonical(fp_mul(x, c.w, c.w_over_q, f.q), f);
    dst[poly * poly_stride + (long long)limb * n + gi] =
        fp_to_word(EXACT && !REDUCE ? fp_exit_word(x, r, f) : r);
  }
};

// to_intt_'s exit (EnterExitStore<false>) after a mixed inverse transform: the exact
// limbs keep mont_exit(mont_mult(v, N^-1 R)); the others, whose words only matter
// modulo q, take one Shoup product by N^-1 R^-1, a word in [0, 2q) of the same value.
struct MixedExitStore {
  using Const = FpFactor;
  int64_t *dst;
  long long poly_stride;
  const int64_t *n_inverse;
  const uint64_t *q;
  const uint64_t *k;
  const int64_t *exit_shoup;  // PrimeTables::exit_shoup
  ExactLimbs exact;
  __device__ __forceinline__ void word(int poly, int limb, int prime, int gi, int n, int64_t v) const {
    const uint64_t qq = q[prime], kk = k[prime];
    int64_t *d = dst + poly * poly_stride + (long long)limb * n + gi;
    if (!exact.exact(poly, limb) && (static_cast<uint64_t>(v) >> kMontBits) == 0) {
      *d = static_cast<int64_t>(shoup_mult(static_cast<uint64_t>(exit_shoup[2 * prime]),
                                           static_cast<uint64_t>(exit_shoup[2 * prime + 1]),
                                           static_cast<uint64_t>(v), qq));
      return;
    }
    *d = mont_exit(mont_mult_lazy(v, n_inverse[prime], qq, kk), qq, kk);
  }
  __device__ __forceinline__ Const constants(int prime, const FpPrime &f) const {
    return fp_factor(exit_shoup[2 * prime], 0, f);
  }
  __device__ __forceinline__ int64_t before(int, int, int) const { return 0; }
  template <bool EXACT>
  __device__ __forceinline__ void fp(int poly, int limb, int, int gi, int n, const Const &c,
                                     const FpPrime &f, int64_t, double x) const {
    const double r = fp_canonical(fp_mul(x, c.w, c.w_over_q, f.q), f);
    dst[poly * poly_stride + (long long)limb * n + gi] = fp_to_word(EXACT ? fp_exit_word(x, r, f) : r);
  }
};

// ------------------------------------------------------------------- tiles --
//
// A tile's words are numbered in the order of their global indices: a contiguous tile's
// word c 2^S + i, a strided one's i 2^columns_log + c for element i of column c.  The
// stages act on tile bits [low, low + S), low = columns_log in strided tiles and 0 in
// contiguous ones, from the top down forward and from the bottom up inverse.  A round
// takes the next W of them (3 in integers, 4 in doubles): a thread holds the 2^W words
// that differ in W adjacent tile bits [d, d + W), and where fewer stages are left than
// that, the window's other bits are just carried.
struct NttRound {
  int d;       // lowest bit of the window
  int b0, b1;  // the stages' bits
};
template <bool INVERSE, int W>
__device__ __forceinline__ NttRound ntt_round(int done, int low, int S, int top) {
  const int count = S - done < W ? S - done : W;
  NttRound r;
  r.b0 = INVERSE ? low + done : low + S - done - count;
  r.b1 = r.b0 + count;
  r.d = r.b0 < top - W ? r.b0 : top - W;
  return r;
}
template <int W>
__device__ __forceinline__ int ntt_group_word(int group, int d) {  // its window bits are 0
  return ((group >> d) << (d + W)) | (group & ((1 << d) - 1));
}

// Shared-memory place of a tile word.  A 128-byte bank row holds 16 words and a half-warp's
// 8-byte accesses are served together: with these XORs every access of the FP64 rounds and
// of the coalesced copies is free of bank conflicts in every default shape, and the integer
// rounds' stay within two wavefronts (simulated).  Linear over XOR, so that a thread's words
// are its first one's place XOR constants of the round.
__device__ __forceinline__ int tile_place(int at) {
  return at ^ ((at >> 4) & 15) ^ (((at >> 6) & 1) << 3);
}

// The default split of N = 2^log_n, 13 <= log_n <= 17: the stages of the strided pass.
__host__ __device__ constexpr int ntt_strided_stages(int log_n) {
  return log_n >= 16 ? 8 : (log_n >= 14 ? 7 : 6);
}
// A shape known at compile time (LOG_N > 0), or the one that a launch brings (LOG_N = 0).
template <int LOG_N, bool STRIDED, bool INVERSE>
__device__ __forceinline__ void ntt_fold_shape(NttPass &a, int tile_log) {
  if (LOG_N > 0) {
    constexpr int kStrided = ntt_strided_stages(LOG_N > 0 ? LOG_N : 13);
    a.log_n = LOG_N;
    a.stages = STRIDED ? kStrided : LOG_N - kStrided;
    a.stride_log = STRIDED ? LOG_N - kStrided : 0;
    a.first = STRIDED == INVERSE ? LOG_N - a.stages : 0;
    a.columns_log = tile_log - a.stages;
  }
}

// Words of the tiles of a shape known at compile time: 16 a thread in doubles and 8 in
// integers with 128 threads; 8 with 256 threads where a launch is all integers.
constexpr int kNttThreads = 128, kNttIntThreads = 256;
constexpr int kNttFpTileLog = 11, kNttIntTileLog = 10, kNttAllIntTileLog = 11;

// One CTA's tile of a pass, in integers.  `value_limb`: the limb only matters modulo q
// (uniform per CTA) and its prime has Shoup's twiddle pairs.
template <int LOG_N, bool STRIDED, bool INVERSE, int VALUE_ONLY, int THREADS, class Loader, class Storer>
__device__ __forceinline__ void ntt_pass_int(const NttPass &a, const PrimeTables &t, const Loader &load,
                                             const Storer &store, int poly, int limb, int block,
                                             bool value_limb, int64_t *tile) {
  constexpr int W = 3, kWords = 1 << W;
  constexpr int kUnroll = LOG_N > 0 ? 8 : 1;  // of the rounds
  const int columns_log = a.columns_log;
  const int prime = a.prime_base + limb;
  const uint64_t q = t.q[prime];
  const uint64_t k = t.k[prime];
  const int64_t q2 = static_cast<int64_t>(q << 1);
  const int n = 1 << a.log_n;
  const int S = a.stages;
  // Twiddles of the general product: a mixed pass has exact limbs, which need the
  // reference's words; the same values serve its value-only limbs out of range.
  const int64_t *tw = (VALUE_ONLY == kNttValueOnly ? (INVERSE ? t.root_inverse_reduced : t.root_reduced)
                                                   : (INVERSE ? t.root_inverse : t.root)) +
                     static_cast<size_t>(prime) * (n - 1);
  // Value-only limbs' in-range words multiply by Shoup's (W, W') pairs instead.
  const longlong2 *tws =
      VALUE_ONLY ? reinterpret_cast<const longlong2 *>(INVERSE ? t.root_inverse_shoup : t.root_shoup) +
                       static_cast<size_t>(prime) * n
                 : nullptr;
  // A forward value-only pass after the first reads words in [0, 4q).
  const uint64_t in_bound = (value_limb && !INVERSE && a.first > 0) ? (q << 2) : (q << 1);
  const bool last_pass = !INVERSE && a.first + S == a.log_n;
  const int tile_log = columns_log + S;
  const int low = STRIDED ? columns_log : 0;
  // Global index of tile word `at`, and of tile bit b as an exponent.
  const int origin = STRIDED ? block << columns_log : block << tile_log;
  auto global_word = [&](int at) {
    return STRIDED ? origin + (at & ((1 << columns_log) - 1)) + ((at >> columns_log) << a.stride_log)
                   : origin + at;
  };
  auto global_bit = [&](int b) { return STRIDED && b >= columns_log ? b - columns_log + a.stride_log : b; };
  // Round 0 checks the words it loads; if every group of the CTA was in range, the
  // tile stays in range through the later rounds, which then skip the check.
  bool slow = false;
  bool tile_lazy = false;

#pragma unroll kUnroll
  for (int done = 0; done < S; done += W) {
    const NttRound rd = ntt_round<INVERSE, W>(done, low, S, tile_log);
    const bool first_round = done == 0, last_round = done + W >= S;
    int place[W];
    int step[W];
#pragma unroll
    for (int b = 0; b < W; b++) {
      place[b] = tile_place(1 << (rd.d + b));
      step[b] = 1 << global_bit(rd.d + b);
    }
    const int top_bit = global_bit(rd.d + W - 1);
#pragma unroll 1
    for (int gid = threadIdx.x; gid < 1 << (tile_log - W); gid += THREADS) {
      const int at = ntt_group_word<W>(gid, rd.d);
      const int tb = tile_place(at);
      const int gi0 = global_word(at);  // global index of the group's first word
      auto word_place = [&](int e) {
        return tb ^ (e & 1 ? place[0] : 0) ^ (e & 2 ? place[1] : 0) ^ (e & 4 ? place[2] : 0);
      };
      auto word_index = [&](int e) {
        return gi0 + (e & 1 ? step[0] : 0) + (e & 2 ? step[1] : 0) + (e & 4 ? step[2] : 0);
      };
      int64_t x[kWords];
      if (first_round) {
        typename Loader::Raw raw[kWords];
#pragma unroll
        for (int e = 0; e < kWords; e++) raw[e] = load.raw(poly, limb, word_index(e), n);
#pragma unroll
        for (int e = 0; e < kWords; e++) x[e] = load.word(raw[e], poly, limb, prime);
      } else {
#pragma unroll
        for (int e = 0; e < kWords; e++) x[e] = tile[word_place(e)];
      }
      // For q < 2^60, words in [0, 2q) stay there through every butterfly (the
      // reference's lazy range; twiddles are below 2q), and for them the
      // butterfly's signed compares and sign-extended product reduce to the short
      // forms below (same words); any other word takes the reference's forms.
      bool in_range = tile_lazy;
      if (first_round) {
        in_range = q < (uint64_t(1) << 60);
#pragma unroll
        for (int e = 0; e < kWords; e++) in_range = in_range && static_cast<uint64_t>(x[e]) < in_bound;
        slow = slow || !in_range;
      }
      auto stages = [&](auto lazy, auto shoup) {
        constexpr bool kLazy = decltype(lazy)::value;
        // guard(a + b, q2) and guard(a + q2 - b, q2) (unit.h:13)
        auto add_guard = [&](int64_t a1, int64_t b1) -> int64_t {
          if (kLazy) {
            const int64_t y = a1 + b1 - q2;
            return y < 0 ? y + q2 : y;
          }
          return guard(a1 + b1, q2);
        };
        auto sub_guard = [&](int64_t a1, int64_t b1) -> int64_t {
          if (kLazy) {
            const int64_t y = a1 - b1;
            return y < 0 ? y + q2 : y;
          }
          return guard(a1 + q2 - b1, q2);
        };
        auto product = [&](int64_t w, int64_t v) -> int64_t {
          if (kLazy) return mont_mult_small(static_cast<uint64_t>(w), static_cast<uint64_t>(v), q, k);
          return mont_mult_const(w, v, q, k);
        };
        // The twiddle of table entry i: the Montgomery word, or for Harvey's form
        // on in-range words the Shoup pair (its product is the same value mod q).
        constexpr bool kShoup = kLazy && decltype(shoup)::value;
        struct Twiddle {
          int64_t w, wp;
        };
        auto twiddle = [&](int i) -> Twiddle {
          if (kShoup) {
            const longlong2 v = __ldg(tws + i);
            return {v.x, v.y};
          }
          return {__ldg(tw + i), 0};
        };
        auto value_product = [&](const Twiddle &w, int64_t v) -> int64_t {
          return static_cast<int64_t>(shoup_mult(static_cast<uint64_t>(w.w), static_cast<uint64_t>(w.wp),
                                                 static_cast<uint64_t>(v), q));
        };
        // The butterflies of one stage that share a twiddle are blocks of consecutive
        // words of the group, and the blocks' twiddles consecutive table entries.
#pragma unroll
        for (int j = 0; j < W; j++) {
          const int bit = INVERSE ? j : W - 1 - j;  // of the window
          const int half = 1 << bit;
          if (rd.d + bit < rd.b0 || rd.d + bit >= rd.b1) continue;
          // The window's bits are adjacent in the global index too, or carried.
          const int gb = top_bit - (W - 1 - bit);
          // forward, stage s = log_n - 1 - gb: twiddle root[2^s - 1 + (gi >> (log_n - s))]
          // (ntt.cpp:46-134); inverse, distance 2^gb: root_inverse[N - N / 2^gb +
          // (gi >> (gb + 1))] (ntt.cpp:177-272)
          const int wi = (INVERSE ? n - (n >> gb) : (n >> (gb + 1)) - 1) + (gi0 >> (gb + 1));
#pragma unroll
          for (int h = 0; h < kWords / 2; h++) {
            if (h >= kWords / 2 / half) continue;
            const Twiddle w = twiddle(wi + h);
#pragma unroll
            for (int e2 = 0; e2 < kWords / 2; e2++) {
              if (e2 >= half) continue;
              const int e = h * 2 * half + e2;
              if (!INVERSE) {
                if (kShoup) {
                  // Harvey's form: words in [0, 4q), one guard per butterfly;
                  // Shoup's product is below 2q.
                  int64_t uu = x[e] - q2;
                  uu = uu < 0 ? uu + q2 : uu;
                  const int64_t p = value_product(w, x[e + half]);
                  x[e] = uu + p;
                  x[e + half] = uu - p + q2;
                } else {
                  const int64_t uu = x[e];
                  const int64_t p = product(w.w, x[e + half]);
                  x[e] = add_guard(uu, p);
                  x[e + half] = sub_guard(uu, p);
                }
              } else {
                const int64_t uu = x[e];
                const int64_t vv = x[e + half];
                x[e] = add_guard(uu, vv);
                // Harvey's form: the product's operand in (0, 4q) needs no guard.
                x[e + half] = kShoup ? value_product(w, uu - vv + q2) : product(w.w, sub_guard(uu, vv));
              }
            }
          }
        }
      };
      if (in_range) {
        if constexpr (VALUE_ONLY != kNttExact) {
          if (value_limb) {
            stages(std::true_type{}, std::true_type{});
          } else {
            stages(std::true_type{}, std::false_type{});
          }
        } else {
          stages(std::true_type{}, std::false_type{});
        }
      } else {
        stages(std::false_type{}, std::false_type{});
      }
      if (last_round) {
#pragma unroll
        for (int e = 0; e < kWords; e++) {
          if (VALUE_ONLY && value_limb && !INVERSE && last_pass && in_range) {
            const int64_t y = x[e] - q2;  // [0, 4q) -> [0, 2q)
            x[e] = y < 0 ? x[e] : y;
          }
          store.word(poly, limb, prime, word_index(e), n, x[e]);
        }
      } else {
#pragma unroll
        for (int e = 0; e < kWords; e++) tile[word_place(e)] = x[e];
      }
    }
    if (first_round && !last_round) {
      tile_lazy = __syncthreads_or(slow) == 0;
    } else if (!last_round) {
      __syncthreads();
    }
  }
}

// One CTA's tile of 2^11 words of a pass over a limb whose prime fp_prime accepts, in
// doubles (modarith.cuh, "FP64 products"): a butterfly is 8 FP64 instructions where only
// values modulo q matter and about 14 where the word is the reference's, against 35 and 45
// on the integer pipes, and needs no guard in the first case: forward words grow by at most
// (1/2 + 2^-6) q a stage (below 2^45 after 17), inverse sums double, and are reduced after
// every pass and, in passes of more than 8 stages, after the second round (below 2^50
// throughout).  EXACT words stay integers in [0, 2q) as the reference's lazy butterflies
// leave them; a CTA that loads any other word returns false before it stores anything, and
// takes the integer pass.  Radix-16 rounds: against radix-8 at 256 threads that is one
// exchange and one barrier instead of two at 8 stages, and twice the loads in flight
// (hoisted rotations at N = 2^16, when it was chosen: 1585 us with radix-8, 1501 with
// radix-16).  A loop over one round's body, to spare the instruction cache, measured slower
// then (the index arithmetic no longer folds): 558 against 429 us for the transforms below.
// Bound by latency and the FP64 pipe (40 % active).  Exact forward and inverse transform of
// four ciphertexts of 24 limbs at N = 2^16: 696 us with every limb in integers, 403 us now
// (2 x 201 MB in and out).
//
// In a contiguous pass (of at most 9 stages) a warp owns 512 adjacent words, whole
// sub-transforms, from load to store: its rounds exchange words inside the warp, and the
// words that a thread holds side by side (first round of the inverse, last of the forward)
// go through shared memory too, so that every global access is coalesced.
template <int LOG_N, bool STRIDED, bool INVERSE, bool EXACT, class Loader, class Storer>
__device__ __forceinline__ bool ntt_pass_fp(const NttPass &a, const PrimeTables &t, const Loader &load,
                                            const Storer &store, int poly, int limb, int block, double *tile) {
  constexpr int W = 4, kWords = 1 << W;
  const int prime = a.prime_base + limb;
  const int n = 1 << a.log_n;
  const int S = a.stages;
  const FpPrime f{static_cast<double>(t.q[prime]), t.inv_q[prime]};
  const double q2 = 2.0 * f.q;
  const double *tw = reinterpret_cast<const double *>(INVERSE ? t.root_inverse_shoup : t.root_shoup) +
                     static_cast<size_t>(prime) * 2 * n;
  const int columns_log = kNttFpTileLog - S;
  const int low = STRIDED ? columns_log : 0;
  const int top = STRIDED ? kNttFpTileLog : 9;  // contiguous: the bits of a warp's words
  const int origin = STRIDED ? block << columns_log : block << kNttFpTileLog;
  auto global_word = [&](int at) {
    return STRIDED ? origin + (at & ((1 << columns_log) - 1)) + ((at >> columns_log) << a.stride_log)
                   : origin + at;
  };
  // Table entry of the first twiddle of the stage on global bit gb for the group at gi0.
  auto twiddle_index = [&](int gb, int gi0) {
    return (INVERSE ? n - (n >> gb) : n >> (gb + 1)) + (gi0 >> (gb + 1));
  };
  const int copy_word = (threadIdx.x >> 5) * 512 + (threadIdx.x & 31);  // contiguous copies: 16 rows of 32
  bool bad = false;

  typename Storer::Const sc = store.constants(prime, f);
  auto store_words = [&](auto index, auto value) {
    int64_t before[kWords];
#pragma unroll
    for (int e = 0; e < kWords; e++) before[e] = store.before(limb, index(e), n);
#pragma unroll
    for (int e = 0; e < kWords; e++)
      store.template fp<EXACT>(poly, limb, prime, index(e), n, sc, f, before[e], value(e));
  };
  // Loads 16 words, index(e) and their places slot(e), converts them and hands them to put;
  // two-word raws eight at a time, for the registers they take.
  constexpr int kChunk = sizeof(typename Loader::Raw) > sizeof(int64_t) ? kWords / 2 : kWords;
  auto load_words = [&](auto index, auto slot, auto put) {
#pragma unroll
    for (int e0 = 0; e0 < kWords; e0 += kChunk) {
      typename Loader::Raw raw[kChunk];
#pragma unroll
      for (int e = 0; e < kChunk; e++) raw[e] = load.raw(poly, limb, index(e0 + e), n);
      if constexpr (Loader::kFp) {
        const typename Loader::Const lc = load.constants(prime, f);
        bool odd = false;
#pragma unroll
        for (int e = 0; e < kChunk; e++) odd = odd || (!EXACT && load.template odd<EXACT>(raw[e]));
        if (!odd) {
#pragma unroll
          for (int e = 0; e < kChunk; e++) put(e0 + e, load.template fp<EXACT>(raw[e], lc, f, bad));
          continue;
        }
        // Rare (words of a 60-bit dropped prime, or out of range): one at a time, by way of
        // the thread's own places in the tile.
#pragma unroll 1
        for (int e = e0; e < e0 + kChunk; e++)
          tile[slot(e)] = load.fp_any(load.raw(poly, limb, index(e), n), lc, f);
#pragma unroll
        for (int e = 0; e < kChunk; e++) put(e0 + e, tile[slot(e0 + e)]);
      } else {
#pragma unroll
        for (int e = 0; e < kChunk; e++) {
          const int64_t w = load.word(raw[e], poly, limb, prime);
          put(e0 + e, EXACT ? fp_exact_word(w, f, bad) : (fp_odd(w) ? fp_from_any_word(w, f) : fp_small(w)));
        }
      }
    }
  };

  if (!STRIDED && INVERSE) {
    const auto place = [&](int i) { return tile_place(copy_word + i * 32); };
    load_words([&](int i) { return origin + copy_word + i * 32; }, place,
               [&](int i, double v) { tile[place(i)] = v; });
  }
#pragma unroll
  for (int done = 0; done < S; done += W) {
    const NttRound rd = ntt_round<INVERSE, W>(done, low, S, top);
    const bool first_round = done == 0, last_round = done + W >= S;
    const int at = ntt_group_word<W>(threadIdx.x, rd.d);
    const int tb = tile_place(at);
    const int gi0 = global_word(at);
    const int low_bit = STRIDED ? rd.d - columns_log + a.stride_log : rd.d;  // of the global index
    const int p0 = tile_place(1 << rd.d), p1 = tile_place(2 << rd.d), p2 = tile_place(4 << rd.d),
              p3 = tile_place(8 << rd.d);
    auto word_place = [&](int e) {
      return tb ^ (e & 1 ? p0 : 0) ^ (e & 2 ? p1 : 0) ^ (e & 4 ? p2 : 0) ^ (e & 8 ? p3 : 0);
    };
    auto word_index = [&](int e) { return gi0 + (e << low_bit); };
    // The round's twiddles, before the barrier: they do not wait for the words.  A stage's
    // are consecutive entries from a multiple of their number (the forward rows start at
    // entry 1): slot 2^j + h for block h of the stage with 2^j blocks.
    double w[kWords];
#pragma unroll
    for (int j = 0; j < W; j++) {
      const int bit = W - 1 - j, gb = low_bit + bit;
      if (rd.d + bit < rd.b0 || rd.d + bit >= rd.b1) continue;
      const double *p = tw + twiddle_index(gb, gi0);
      if (j == 0) {
        w[1] = __ldg(p);
      } else {
#pragma unroll
        for (int h = 0; h < kWords / 2; h += 2) {
          if (h >= 1 << j) continue;
          const double2 v = __ldg(reinterpret_cast<const double2 *>(p + h));
          w[(1 << j) + h] = v.x;
          w[(1 << j) + h + 1] = v.y;
        }
      }
    }
    double x[kWords];
    if (first_round && (STRIDED || !INVERSE)) {
      load_words(word_index, word_place, [&](int e, double v) { x[e] = v; });
    } else {
      if (EXACT && !STRIDED && first_round) {
        if (__syncthreads_or(bad)) return false;
      } else if (!STRIDED) {
        __syncwarp();
      }
#pragma unroll
      for (int e = 0; e < kWords; e++) x[e] = tile[word_place(e)];
    }
#pragma unroll
    for (int j = 0; j < W; j++) {
      const int bit = INVERSE ? j : W - 1 - j;
      const int half = 1 << bit, blocks = 1 << (W - 1 - bit);
      if (rd.d + bit < rd.b0 || rd.d + bit >= rd.b1) continue;
      const double *mont = tw + n + twiddle_index(low_bit + bit, gi0);  // EXACT
#pragma unroll
      for (int h = 0; h < kWords / 2; h++) {
        if (h >= blocks) continue;
        const double wp = w[blocks + h], wq = wp * f.inv_q, wm = EXACT ? __ldg(mont + h) : 0.0;
#pragma unroll
        for (int e2 = 0; e2 < kWords / 2; e2++) {
          if (e2 >= half) continue;
          const int e = h * 2 * half + e2;
          const double uu = x[e], vv = x[e + half];
          const double p = INVERSE ? vv
                                   : (EXACT ? fp_mont_mult(vv, wp, wq, wm, f)
                                            : fp_mul(vv, wp, wq, f.q));
          // guard(u + p, 2q) and guard(u - p + 2q, 2q) on words of [0, 2q)
          double sum = uu + p, d = uu - p;
          if (EXACT) {
            sum -= q2;
            sum = fp_negative(sum) ? sum + q2 : sum;
            d = fp_negative(d) ? d + q2 : d;
          }
          x[e] = sum;
          x[e + half] = !INVERSE ? d
                                 : (EXACT ? fp_mont_mult(d, wp, wq, wm, f)
                                          : fp_mul(d, wp, wq, f.q));
        }
      }
    }
    if (INVERSE && !EXACT && ((last_round && a.first + S < a.log_n) || (S > 8 && done == W))) {
#pragma unroll
      for (int e = 0; e < kWords; e++) x[e] = fp_reduce(x[e], f);
    }
    if (last_round && (STRIDED || INVERSE)) {
      store_words(word_index, [&](int e) { return x[e]; });
      break;
    }
    // (to the places that this thread read, so nobody else waits for them)
#pragma unroll
    for (int e = 0; e < kWords; e++) tile[word_place(e)] = x[e];
    if (STRIDED || (EXACT && first_round && !INVERSE)) {
      if (EXACT && first_round) {
        if (__syncthreads_or(bad)) return false;
      } else {
        __syncthreads();
      }
    }
  }
  if (!STRIDED && !INVERSE) {
    __syncwarp();
    store_words([&](int i) { return origin + copy_word + i * 32; },
                [&](int i) { return tile[tile_place(copy_word + i * 32)]; });
  }
  return true;
}

// Limbs in the order a pass's CTAs take them: those in integers first, since they take
// longest and have twice as many CTAs each.
constexpr int kNttMaxLimbs = PrimeSet::kPrimes;
static_assert(kNttMaxLimbs <= 256, "limbs are listed as bytes");
struct NttLimbOrder {
  int integer_limbs = 0;
  uint8_t limb[kNttMaxLimbs] = {};
};

// Both kinds of limbs, a shape known at compile time.  80 registers and six CTAs an SM where
// values count (at five ModUp's transforms of a product at N = 2^17 take 1005 us, 977 at six);
// the exact ones, which hold more constants, 96 and five (both transforms of a text at
// N = 2^14 10.9 us a call, 11.9 at six; four inverse ones at N = 2^16 208 and 217).
// The mixed passes, which hold the value, the exact and the integer form, spill at 80 (the lazy
// rescale's by about 100 bytes a thread, the tensor loader's, on the path without the fold, by
// 260 and more).  Fewer loads in flight spill less and are slower: the tensor's transform of
// a product at N = 2^17 648 us, 652 with four elements' loads at a time and 688 with two.
template <int LOG_N, bool STRIDED, bool INVERSE, class Loader, class Storer, int VALUE_ONLY>
__global__ void __launch_bounds__(kNttThreads, VALUE_ONLY == kNttExact ? 5 : 6)
    ntt_pass_kernel(NttPass a, NttLimbOrder order, PrimeTables t, Loader load, Storer store) {
  chained_kernel_begin();
  __shared__ double tile[1 << kNttFpTileLog];
  constexpr int kIntTiles = LOG_N - kNttIntTileLog, kFpTiles = LOG_N - kNttFpTileLog;
  const int integer_blocks = (order.integer_limbs * a.polys) << kIntTiles;
  const bool integer = static_cast<int>(blockIdx.x) < integer_blocks;
  const int b = integer ? blockIdx.x : blockIdx.x - integer_blocks;
  const int tiles_log = integer ? kIntTiles : kFpTiles;
  const int row = b >> tiles_log;
  int block = b & ((1 << tiles_log) - 1), count = 1;
  const int poly = row % a.polys;
  const int limb = order.limb[row / a.polys + (integer ? 0 : order.integer_limbs)];
  if (a.skip_start != nullptr && limb >= a.skip_start[poly] &&
      limb < a.skip_start[poly] + a.skip_size[poly])
    return;  // uniform per CTA, before any barrier
  const bool value_limb =
      VALUE_ONLY == kNttValueOnly || (VALUE_ONLY == kNttMixed && !a.exact.exact(poly, limb));
  if (!integer) {
    ntt_fold_shape<LOG_N, STRIDED, INVERSE>(a, kNttFpTileLog);
    if constexpr (VALUE_ONLY != kNttExact) {
      if (value_limb) {
        ntt_pass_fp<LOG_N, STRIDED, INVERSE, false>(a, t, load, store, poly, limb, block, tile);
        return;
      }
    }
    if constexpr (VALUE_ONLY != kNttValueOnly) {
      if (ntt_pass_fp<LOG_N, STRIDED, INVERSE, true>(a, t, load, store, poly, limb, block, tile)) return;
    }
    // The tile's two halves in integers, with exact butterflies (no Shoup pairs).
    block *= 2;
    count = 2;
  }
  ntt_fold_shape<LOG_N, STRIDED, INVERSE>(a, kNttIntTileLog);
#pragma unroll 1
  for (int i = 0; i < count; i++) {
    if (i > 0) __syncthreads();
    ntt_pass_int<LOG_N, STRIDED, INVERSE, VALUE_ONLY, kNttThreads>(
        a, t, load, store, poly, limb, block + i, VALUE_ONLY == kNttValueOnly || (value_limb && integer),
        reinterpret_cast<int64_t *>(tile));
  }
}

// Every limb in integers: the default shape of N = 2^16 (the bootstrap preset's 54-bit
// primes) at compile time, or a shape that the launch brings.
template <int LOG_N, bool STRIDED, bool INVERSE, class Loader, class Storer, int VALUE_ONLY>
__global__ void __launch_bounds__(kNttIntThreads, 4)
    ntt_int_kernel(NttPass a, PrimeTables t, Loader load, Storer store) {
  chained_kernel_begin();
  extern __shared__ __align__(16) int64_t tile_smem[];
  const int poly = blockIdx.y % a.polys;
  const int limb = blockIdx.y / a.polys;
  if (a.skip_start != nullptr && limb >= a.skip_start[poly] &&
      limb < a.skip_start[poly] + a.skip_size[poly])
    return;  // uniform per CTA, before any barrier
  ntt_fold_shape<LOG_N, STRIDED, INVERSE>(a, kNttAllIntTileLog);
  // A prime with rows of doubles has no Shoup pairs here: it takes the exact butterflies,
  // whose words are as good.
  const bool value_limb =
      (VALUE_ONLY == kNttValueOnly || (VALUE_ONLY == kNttMixed && !a.exact.exact(poly, limb))) &&
      !t.fp_primes.has(a.prime_base + limb);
  ntt_pass_int<LOG_N, STRIDED, INVERSE, VALUE_ONLY, kNttIntThreads>(a, t, load, store, poly, limb,
                                                                    blockIdx.x, value_limb, tile_smem);
}

// Pass plan of a transform of 2^log_n words: for two passes, the tuned or default
// split and tile shapes (ntt_tuning, kernels.cuh).  Every plan performs the same
// butterflies, so every plan gives the same words.
struct NttPlan {
  int passes;   // 1 or 2
  int s_first;  // S of the strided (outer) pass, or log_n for a single pass
  int s_second; // S of the contiguous (inner) pass
  int first_columns_log;   // sub-transforms per CTA of the strided pass
  int second_columns_log;  // sub-transforms per CTA of the contiguous pass
  bool standard;           // the default shape of N = 2^13 .. 2^17
};

inline NttPlan ntt_plan(int log_n) {
  if (log_n <= 11) return {1, log_n, 0, 0, 0, false};
  const NttTuning tu = ntt_tuning(log_n), def = ntt_default_tuning(log_n);
  const int s_first = log_n - tu.s_second;
  // A group of eight words has to fit a tile.
  auto at_least = [](int columns_log, int s) { return columns_log + s < 3 ? 3 - s : columns_log; };
  return {2, s_first, tu.s_second, at_least(tu.first_columns_log, s_first),
          at_least(tu.second_tile_log - tu.s_second, tu.s_second),
          log_n >= 13 && tu.s_second == def.s_second && tu.first_columns_log == def.first_columns_log &&
              tu.second_tile_log == def.second_tile_log};
}

template <int LOG_N, bool STRIDED, bool INVERSE, int VALUE_ONLY, class Loader, class Storer>
cudaError_t launch_ntt_int(const NttPass &a, const PrimeTables &t, const Loader &ld, const Storer &st,
                           cudaStream_t stream) {
  const dim3 grid((1 << a.log_n) >> (a.columns_log + a.stages), a.polys * a.limbs);
  const size_t smem = sizeof(int64_t) << (a.columns_log + a.stages);
  auto kernel = ntt_int_kernel<LOG_N, STRIDED, INVERSE, Loader, Storer, VALUE_ONLY>;
  // To the most any valid plan uses, so no attribute call lands inside a graph capture.
  static DeviceOnce raised;
  const cudaError_t e = raise_smem_limit(kernel, kNttMaxSmem, raised);
  if (e != cudaSuccess) return e;
  if (smem > static_cast<size_t>(kNttMaxSmem)) return cudaErrorInvalidValue;
  note_launch(1);
  launch_chained(kernel, grid, kNttIntThreads, smem, stream, a, t, ld, st);
  return cudaGetLastError();
}

template <bool STRIDED, bool INVERSE, int VALUE_ONLY, class Loader, class Storer>
cudaError_t launch_ntt_pass(const NttPass &a, bool standard, bool integer, const PrimeTables &t,
                            const Loader &ld, const Storer &st, cudaStream_t stream) {
  NttLimbOrder order;
  int in_doubles = 0;
  if (standard && !integer && a.limbs <= kNttMaxLimbs) {
    for (int pass = 0, at = 0; pass < 2; pass++)
      for (int j = a.limbs - 1; j >= 0; j--)
        if (t.fp_primes.has(a.prime_base + j) == (pass == 1)) {
          order.limb[at++] = static_cast<uint8_t>(j);
          in_doubles += pass;
        }
    order.integer_limbs = a.limbs - in_doubles;
  }
  if (in_doubles == 0) {
    if (standard && a.log_n == 16)
      return launch_ntt_int<16, STRIDED, INVERSE, VALUE_ONLY>(a, t, ld, st, stream);
    return launch_ntt_int<0, STRIDED, INVERSE, VALUE_ONLY>(a, t, ld, st, stream);
  }
  const unsigned blocks = static_cast<unsigned>(a.polys) *
                          ((static_cast<unsigned>(order.integer_limbs) << (a.log_n - kNttIntTileLog)) +
                           (static_cast<unsigned>(in_doubles) << (a.log_n - kNttFpTileLog)));
  note_launch(1);
  switch (a.log_n) {
#define FHE_NTT_CASE(L)                                                               \
  case L:                                                                             \
    launch_chained(ntt_pass_kernel<L, STRIDED, INVERSE, Loader, Storer, VALUE_ONLY>,  \
                   blocks, kNttThreads, 0, stream, a, order, t, ld, st);              \
    break;
    FHE_NTT_CASE(13) FHE_NTT_CASE(14) FHE_NTT_CASE(15) FHE_NTT_CASE(16) FHE_NTT_CASE(17)
#undef FHE_NTT_CASE
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

// A transform in one pass (N = 2^3 .. 2^11) or two: strided then contiguous forward, the
// other way round inverse.  The first pass reads through `ld`, the last one writes through
// `st`; intermediate data lives in `work` ([poly][limb][N], stride work_stride), which may
// alias the final destination.
template <bool INVERSE, int VALUE_ONLY, class Loader, class Storer>
cudaError_t run_ntt(NttPass a, const PrimeTables &tables, const Loader &ld, const Storer &st, int64_t *work,
                    long long work_stride, cudaStream_t stream, bool integer = false) {
  const NttPlan plan = ntt_plan(a.log_n);
  PrimeTables t = tables;
  if (VALUE_ONLY != kNttExact && plan.passes == 2 && !plan.standard && t.shoup_tables != nullptr &&
      t.shoup_tables->ready(stream)) {
    // Pairs in place of the rows of doubles, which only the default shapes read.  A caller's
    // shape with exact butterflies on these limbs: one rotation at N = 2^17 and 40 limbs
    // 1969 us, 1699 with the pairs (the default shape, in doubles: 1061).
    t.root_shoup = t.shoup_tables->root;
    t.root_inverse_shoup = t.shoup_tables->root_inverse;
    t.fp_primes = PrimeSet{};
  }
  a.first = 0;
  if (plan.passes == 1) {
    a.stages = a.log_n;
    a.stride_log = 0;
    a.columns_log = 0;
    return launch_ntt_int<0, false, INVERSE, VALUE_ONLY>(a, t, ld, st, stream);
  }
  auto shape = [&](bool strided) {
    a.stages = strided ? plan.s_first : plan.s_second;
    a.stride_log = strided ? plan.s_second : 0;
    a.columns_log = strided ? plan.first_columns_log : plan.second_columns_log;
  };
  MidStore mid_store{{work, work_stride}};
  MidLoad mid_load{{work, work_stride}};
  shape(!INVERSE);
  const cudaError_t e = launch_ntt_pass<!INVERSE, INVERSE, VALUE_ONLY>(a, plan.standard, integer, t, ld,
                                                                       mid_store, stream);
  if (e != cudaSuccess) return e;
  a.first = a.stages;
  shape(INVERSE);
  return launch_ntt_pass<INVERSE, INVERSE, VALUE_ONLY>(a, plan.standard, integer, t, mid_load, st, stream);
}

// Batched forward NTT of `polys` x `limbs` limbs.  `integer`: every limb in integers.
template <class Loader, class Storer, int VALUE_ONLY = kNttExact>
cudaError_t forward_ntt(int log_n, int polys, int limbs, int prime_base, const PrimeTables &t,
                        const Loader &ld, const Storer &st, int64_t *work, long long work_stride,
                        cudaStream_t stream, const int *skip_start = nullptr,
                        const int *skip_size = nullptr, const ExactLimbs &exact = ExactLimbs{},
                        bool integer = false) {
  const NttPass a{log_n, 0, 0, 0, 0, polys, limbs, prime_base, skip_start, skip_size, exact};
  return run_ntt<false, VALUE_ONLY>(a, t, ld, st, work, work_stride, stream, integer);
}

template <class Loader, class Storer, int VALUE_ONLY = kNttExact>
cudaError_t inverse_ntt(int log_n, int polys, int limbs, int prime_base, const PrimeTables &t,
                        const Loader &ld, const Storer &st, int64_t *work, long long work_stride,
                        cudaStream_t stream, const ExactLimbs &exact = ExactLimbs{}) {
  const NttPass a{log_n, 0, 0, 0, 0, polys, limbs, prime_base, nullptr, nullptr, exact};
  return run_ntt<true, VALUE_ONLY>(a, t, ld, st, work, work_stride, stream);
}

}  // namespace fhe_b200
