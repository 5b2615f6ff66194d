"""Decode's CRT at every limb count: the same integers modulo more primes give the same
doubles, whatever number of 64-bit words the kernel holds them in."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PLAINTEXT = 5


def residues(values, moduli):
    return np.array([[int(v) % int(q) for v in values] for q in moduli], dtype=np.int64)[None]


@pytest.mark.parametrize("log_n,special,limb_counts", [
    (13, 1, (2, 3, 4)), (16, 10, (2, 5, 11, 29)),
    (17, 6, (2, 3, 4, 5, 6, 7, 8, 11, 13, 15, 16, 19, 20, 25, 31, 40, 47)),
])
def test_the_limb_count_does_not_change_the_slots(engines, log_n, special, limb_counts):
    e = engines(log_n, special, 1)
    rng = np.random.default_rng(log_n)
    values = np.zeros(e.coeff_count, dtype=object)
    values[:64] = rng.integers(-2 ** 50, 2 ** 50, 64)
    values[64:67] = [-1, 1, 0]
    sparse = np.flatnonzero(values)
    slots = []
    for limbs in limb_counts:
        q = e.moduli[e.chain_count - limbs:e.chain_count]
        x = np.zeros((1, limbs, e.coeff_count), dtype=np.int64)
        x[:, :, sparse] = residues(values[sparse], q)
        slots.append(e.decode(e.upload(x, e.chain_count - limbs, kind=PLAINTEXT), complex_output=True))
    for s in slots[1:]:
        assert np.array_equal(s, slots[0])
    # Integers near Q / 2 and Q / 3 as constant polynomials: every slot has their value, the
    # sign past Q / 2 negative.  The words are summed in doubles: one rounding a word.  Where
    # those exceed a double's range (more than 25 limbs), powers of two within it.
    for limbs in limb_counts:
        q = [int(v) for v in e.moduli[e.chain_count - limbs:e.chain_count]]
        big = 1
        for v in q:
            big *= v
        values = (big // 2 - 1, big // 2 + 1, big // 3, big - big // 3)
        if big.bit_length() > 1023:  # 2^(64 w) overflows past w = 15, as in the reference
            values = (1, big - 1, 2 ** 1000, big - 2 ** 1000)
        for m in values:
            x = np.zeros((1, limbs, e.coeff_count), dtype=np.int64)
            x[:, :, :1] = residues([m], q)
            got = e.decode(e.upload(x, e.chain_count - limbs, kind=PLAINTEXT))
            want = float(m if 2 * m < big else m - big)
            assert np.allclose(got, want, rtol=2.0 ** -52 * (limbs + 2 * log_n), atol=0)
