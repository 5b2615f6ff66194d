"""The transforms of the 40- and 41-bit primes in doubles: their products against the
integer forms (on the CPU), and on the GPU every default shape against a tuned shape, whose
passes run in integers, word for word, words outside the lazy range included."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from fhe_b200 import _lib
from inputs import uniform_limbs

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "fhe_b200", "csrc")
NTT, SPECIAL, RELIN, ROTATION = 2, 16, 3, 6


def moduli_of(log_n, special):
    cfg, info, q = _lib.FheConfig(log_n, -1, special, -1, 1), _lib.FheEngineInfo(), (ctypes.c_uint64 * 200)()
    assert _lib.load().fhe_parameters_query(ctypes.byref(cfg), ctypes.byref(info), q, 200) == 0
    return [int(x) for x in q[:info.prime_count]]


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_products_in_doubles_match_the_integer_forms(tmp_path):
    exe = str(tmp_path / "fp_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, "-o", exe,
                    os.path.join(HERE, "fp_check.cpp")], check=True)
    primes = sorted({q for log_n, k in ((13, 1), (16, 10), (17, 6)) for q in moduli_of(log_n, k) if q < 1 << 41})
    primes = primes[:2] + primes[-2:]
    out = subprocess.run([exe, "200000", "1", *map(str, primes)], check=True, capture_output=True, text=True)
    assert out.stdout.strip() == "0"


def both_shapes(log_n, fn):
    """fn() under the default shape and under one whose passes run in integers."""
    lib = _lib.load()
    saved = [ctypes.c_int() for _ in range(3)]
    assert lib.fhe_ntt_tuning_get(log_n, *map(ctypes.byref, saved)) == 0
    default = fn()
    assert lib.fhe_ntt_tuning_set(log_n, 6, 2, 11) == 0
    try:
        return default, fn()
    finally:
        lib.fhe_ntt_tuning_set(log_n, *[v.value for v in saved])


@pytest.mark.gpu
@pytest.mark.parametrize("log_n,special", [(13, 1), (14, 1), (15, 2), (16, 10), (17, 6)])
@pytest.mark.parametrize("words", ["canonical", "lazy", "wild"])
def test_doubles_give_the_words_of_the_integer_passes(engines, log_n, special, words):
    e = engines(log_n, special, 1)
    mid = max(1, e.chain_count - 6)
    rng = np.random.default_rng(100 * log_n + special)
    q = e.moduli[mid:e.chain_count]

    def text(polys):
        x = uniform_limbs(rng, q, polys, e.coeff_count)
        x[0, :, :4] = 0
        if words != "canonical":  # half the words in [q, 2q), the edges among them
            pick = rng.random(x.shape) < 0.5
            x += np.where(pick, np.asarray(q, dtype=np.int64)[None, :, None], 0)
            x[-1, :, 5] = 2 * np.asarray(q, dtype=np.int64) - 1
        if words == "wild":  # words no operation makes: negative, 2q and more, 2^45
            at = rng.integers(0, e.coeff_count, 3)
            x[0, 0, at[0]], x[0, 1, at[1]], x[0, -1, at[2]] = -5, 2 * int(q[1]), 1 << 45
        return x

    a, b = text(2), text(2)
    key = uniform_limbs(rng, e.moduli[mid:], 2 * e.partition_count(mid), e.coeff_count)
    rk = e.upload(key, mid, NTT | SPECIAL, RELIN)
    fk = e.upload(key, mid, NTT | SPECIAL, ROTATION)
    fk.set_delta(1)

    def run():
        x = e.upload(a, mid)
        out = [e.ntt(x).download(), e.intt(e.upload(a, mid, NTT)).download(),
               e.multiply_plaintext(x, e.upload(b[:1], mid, kind=5)).download(),
               e.rotate(x, fk).download()]
        for inverse in (False, True):
            y = e.upload(a, mid)
            e.ntt_limbs(y.device_pointer(), mid, len(q), 2, len(q) * e.coeff_count, inverse=inverse)
            out.append(y.download())
        if words != "wild":
            out.append(e.multiply(x, e.upload(b, mid), rk).download())
        return out

    for i, (got, want) in enumerate(zip(*both_shapes(log_n, run))):
        assert np.array_equal(got, want), i
