"""Key switching at every number of special primes against the CPU oracle: the divisor
triangle on one lane and on two (an odd count leaves the second lane without a limb in
places), Garner's digits in doubles for partitions of up to 16 limbs, and the ends of the
tensor-core rounds (their targets go to the CTA's halves in pairs)."""
import numpy as np
import pytest

from inputs import uniform_limbs
from oracle import oracle

pytestmark = pytest.mark.gpu

NTT, SPECIAL = 2, 16
RELIN, ROTATION = 3, 6


def check(e, ctx, L, seed):
    mid = e.chain_count - L
    rng = np.random.default_rng(seed)
    n, q = e.coeff_count, e.moduli[mid:e.chain_count]
    t3, ct = uniform_limbs(rng, q, 3, n), uniform_limbs(rng, q, 2, n)
    key = uniform_limbs(rng, e.moduli[mid:], 2 * e.partition_count(mid), n)
    rk = e.upload(key, mid, NTT | SPECIAL, RELIN)
    fk = e.upload_fixed_rotation_key(key, mid, 5)
    assert np.array_equal(e.relinearize(e.upload(t3, mid, NTT), rk).download(),
                          ctx.relinearize(mid, t3, mid, key)), L
    assert np.array_equal(e.rotate(e.upload(ct, mid), fk).download(),
                          ctx.rotate(mid, ct, mid, key, 5)), L
    if L >= 3:  # the rescaled store
        a = uniform_limbs(rng, e.moduli[mid - 1:e.chain_count], 2, n)
        b = uniform_limbs(rng, e.moduli[mid - 1:e.chain_count], 2, n)
        got = e.multiply_relinearize_rescale(e.upload(a, mid - 1), e.upload(b, mid - 1), rk).download()
        assert np.array_equal(got, ctx.mult_relin_rescale(mid - 1, a, b, mid, key)), L


@pytest.mark.parametrize("preset,K", [(1, K) for K in range(1, 17)] + [(2, 4), (2, 5), (2, 9), (2, 16)])
def test_every_special_count_matches_the_oracle(preset, K):
    from fhe_b200 import Engine

    e = Engine(log_coeff_count=16, special_prime_count=K, scheme_preset=preset)
    e.set_tensor_cores(True)
    try:
        ctx = oracle.Context(16, e.moduli, K)
        for L in sorted({2, min(K + 2, e.chain_count - 2)}):  # the larger: a partition of K limbs and one of 2
            check(e, ctx, L, 100 * K + L)
    finally:
        e.close()


@pytest.mark.parametrize("preset", [1, 2])
def test_the_ends_of_a_round_match_the_oracle(engines, preset):
    e = engines(16, 4, preset)
    ctx = oracle.Context(16, e.moduli, 4)
    for L in (1, 3, 4, 5, 7, 15, 16, 17, 18):
        check(e, ctx, L, 7000 + L)
