// Host check of the FP64 products (fhe_b200/csrc/modarith.cuh compiles as plain C++):
// for primes of 40 and 41 bits, random operands and the edges of their ranges,
//   fp_mul       is congruent to v w and within 3/4 q of zero, for |v| <= 2^50;
//   fp_mont_mult is the word of the reference's Montgomery product, for v in [0, 2^42)
//                and lazy Montgomery words in [0, 2q);
//   fp_exit_word is the word of mont_exit(mont_mult(v, N^-1 R));
//   fp_from_any_word and the word conversions keep the value.
// Usage: fp_check <iterations> <seed> <prime> ...; prints the mismatch count.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "modarith.cuh"

using namespace fhe_b200;
using i128 = __int128;

static uint64_t negated_inverse(uint64_t q) {
  uint64_t x = 1;
  for (int i = 0; i < 7; i++) x *= 2 - q * x;
  return (0 - x) & kMontMask;
}

int main(int argc, char **argv) {
  const long iterations = std::atol(argv[1]);
  std::mt19937_64 rng(std::atoll(argv[2]));
  long bad = 0;
  for (int a = 3; a < argc; a++) {
    const uint64_t q = std::strtoull(argv[a], nullptr, 10), k = negated_inverse(q);
    if (!fp_prime(q)) bad++;
    const FpPrime f{static_cast<double>(q), 1.0 / static_cast<double>(q)};
    auto mod = [&](i128 x) { return static_cast<uint64_t>(((x % static_cast<i128>(q)) + q) % q); };
    auto power = [&](uint64_t b, uint64_t e) {
      uint64_t r = 1;
      for (; e; e >>= 1, b = mod(static_cast<i128>(b) * b))
        if (e & 1) r = mod(static_cast<i128>(r) * b);
      return r;
    };
    const uint64_t r_inverse = power((uint64_t(1) << 62) % q, q - 2);
    const uint64_t n_inverse_r = mod(static_cast<i128>(power(65536, q - 2)) * ((uint64_t(1) << 62) % q));
    const uint64_t exit_c = mod(static_cast<i128>(mod(static_cast<i128>(n_inverse_r) * r_inverse)) * r_inverse);
    const uint64_t edges[] = {0, 1, 2, q - 1, q, q + 1, 2 * q - 1};
    for (long it = 0; it < iterations; it++) {
      uint64_t word = rng() % (2 * q), v = rng() % (2 * q);
      if (it % 3 == 0) v = edges[rng() % 7];
      if (it % 5 == 0) word = edges[rng() % 7];
      if (it % 7 == 0) v = rng() & ((uint64_t(1) << 42) - 1);
      if (it % 11 == 0) v = (uint64_t(1) << 42) - 1 - (rng() & 15);
      const uint64_t w = mod(static_cast<i128>(word) * r_inverse);  // the plain residue
      const double wd = static_cast<double>(w);
      // A residue near zero is where the Montgomery word differs from it: v = x / w.
      if (it % 2 == 0 && w != 0) v = mod(static_cast<i128>(power(w, q - 2)) * (rng() & 0x7FFFFF)) + (it % 4 ? q : 0);
      const int64_t got = fp_to_word(
          fp_mont_mult(fp_from_word(v), wd, wd * f.inv_q, static_cast<double>(word) * kFpMontScale, f));
      if (got != mont_mult_small(word, v, q, k)) bad++;
      const double r = fp_canonical(fp_mul(fp_from_word(v), static_cast<double>(exit_c), f), f);
      if (fp_to_word(fp_exit_word(fp_from_word(v), r, f)) !=
          mont_exit(mont_mult(static_cast<int64_t>(v), static_cast<int64_t>(n_inverse_r), q, k), q, k))
        bad++;
      int64_t s = static_cast<int64_t>(rng() & ((uint64_t(1) << 51) - 1)) - (int64_t(1) << 50);
      if (it % 9 == 0) s = it % 2 ? (int64_t(1) << 50) : -(int64_t(1) << 50);
      const double p = fp_mul(static_cast<double>(s), wd, f);
      if (!(p >= -0.75 * f.q && p <= 0.75 * f.q) || p != static_cast<double>(static_cast<int64_t>(p)) ||
          mod(static_cast<int64_t>(p)) != mod(static_cast<i128>(s) * static_cast<i128>(w)))
        bad++;
      const double reduced = fp_reduce(static_cast<double>(s), f);
      if (!(reduced >= -0.51 * f.q && reduced <= 0.51 * f.q) || mod(static_cast<int64_t>(reduced)) != mod(s)) bad++;
      const int64_t any = static_cast<int64_t>(rng());
      const double small = fp_from_any_word(any, f);
      if (!(small > -4398046511104.0 && small < 4398046511104.0) || mod(static_cast<int64_t>(small)) != mod(any))
        bad++;
    }
  }
  std::printf("%ld\n", bad);
  return 0;
}
