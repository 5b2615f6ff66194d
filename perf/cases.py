"""The calls whose speed this framework is measured by.

Each case is one pass through the engine's public entry points on seeded messages:
the client's encryption and decryption, the server's products, rotations, plaintext
dot products, transforms and serving batches, and a bootstrap, from the smallest ring
(N = 2^13) to the largest (N = 2^17).  Engines and keys are what a program keeps for
its lifetime: they are made once per parameter set from a fixed seed; the messages,
and the ciphertexts they are encrypted to, come from the case's seed.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from fhe_b200 import Engine

DEFAULT, BOOTSTRAP = 1, 2  # scheme presets: 40-bit scale, 54-bit scale with a 60-bit base

# (log2 N, special primes, preset): the reference's tiers and the key-switching set
# with ten special primes; the highest level at which a key switches.
SETS = {
    (13, 1, DEFAULT): 1,
    (14, 1, DEFAULT): 6,
    (15, 2, DEFAULT): 16,
    (16, 4, DEFAULT): 35,
    (16, 10, DEFAULT): 26,
    (17, 6, DEFAULT): 76,
    (16, 4, BOOTSTRAP): 25,
}

# What a serving program's rotation keys reach (powers of two), and their number.
ROTATION_KEYS = 8


def _case(op, log_n, special, preset=DEFAULT, name=None, **more):
    c = dict(op=op, log_n=log_n, special=special, preset=preset, **more)
    return dict(c, name=name) if name else c


def listed():
    return [
        # A client's message on the reference's default engine: encode, encrypt with a
        # public key at the top level; the message is shorter than the slots.
        _case("encrypt", 14, 1, name="encrypt_n14", level=7, count=5000, complex=False),
        # A client reading a complex result at N = 2^16: decrypt, decode all slots.
        _case("decrypt", 16, 4, name="decrypt_n16", level=9, complex=True),
        # The smallest server call: a plaintext-weighted sum of two ciphertexts on the
        # smallest ring, where launches and latency are all there is.
        _case("dot", 13, 1, name="dot_n13", level=2, terms=2),
        # One product on the default engine (N = 2^14, one special prime).
        _case("hmult", 14, 1, name="hmult_n14", level=6, batch=1),
        # One product deep in a circuit: few limbs left at N = 2^16.
        _case("hmult", 16, 10, name="hmult_n16_low", level=5, batch=1),
        # The headline: a batch of products at the top key-switching level.
        _case("hmult", 16, 10, name="hmult_n16_batch", level=26, batch=16),
        # One product at the largest ring's top level: 13 partitions, a 2 GB key.
        _case("hmult", 17, 6, name="hmult_n17", level=76, batch=1),
        # One rotation with a fixed key on a middle ring, a ragged last partition.
        _case("rotate", 15, 2, name="rotate_n15", level=11, count=1),
        # Hoisted rotations of one ciphertext (the inner loop of a linear transform).
        _case("rotate", 16, 4, name="rotate_n16_hoisted", level=20, count=8),
        # A serving step: pairs at uneven levels, multiplied, rescaled and rotated.
        _case("serve", 16, 10, name="serve_n16", low=2, high=24, batch=24),
        # Both transforms on their own, over four ciphertexts of 24 limbs.
        _case("transform", 16, 10, name="transform_n16", level=22, count=4),
        # A bootstrap with the medium three-stage key.
        _case("bootstrap", 16, 4, BOOTSTRAP, name="bootstrap_n16", level=3),
    ]


def _spread(rng: random.Random, low: int, high: int) -> int:
    """A whole number of [low, high], spread over the logarithm where that spans a decade."""
    if high < 10 * low:
        return rng.randint(low, high)
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 0.49))))))


def draw(rng):
    op = rng.choice(["encrypt", "decrypt", "dot", "hmult", "hmult", "hmult", "rotate", "rotate",
                     "serve", "transform", "bootstrap"])
    if op == "bootstrap":
        return _case(op, 16, 4, BOOTSTRAP, level=rng.randint(1, 14))
    if op == "serve":
        low = rng.randint(2, 8)
        return _case(op, 16, 10, low=low, high=rng.randint(low + 4, 24), batch=rng.randint(3, 23))
    sets = [s for s in SETS if s[0] > 13 or op in ("encrypt", "decrypt", "dot", "transform")]
    log_n, special, preset = rng.choice(sets)
    top = SETS[(log_n, special, preset)]
    if op == "encrypt":
        return _case(op, log_n, special, preset, level=_spread(rng, 1, top),
                     count=_spread(rng, 1, 1 << (log_n - 1)), complex=rng.random() < 0.5)
    if op == "decrypt":
        return _case(op, log_n, special, preset, level=_spread(rng, 1, min(top, 35)),
                     complex=rng.random() < 0.5)
    if op == "dot":
        return _case(op, log_n, special, preset, level=2 if log_n == 13 else _spread(rng, 2, top),
                     terms=_spread(rng, 1, 12 if log_n < 17 else 3))
    if op == "transform":
        return _case(op, log_n, special, preset, level=_spread(rng, 1, top),
                     count=_spread(rng, 1, 12 if log_n < 17 else 2))
    if op == "rotate":
        return _case(op, log_n, special, preset, level=_spread(rng, 1, top),
                     count=rng.randint(1, ROTATION_KEYS if log_n < 17 else 2))
    return _case("hmult", log_n, special, preset, level=_spread(rng, 2, top),
                 batch=_spread(rng, 1, 15) if log_n < 17 else 1)


# ------------------------------------------------------- engines, keys, messages --


class _Program:
    """An engine and the keys a program holds, made on first use."""

    def __init__(self, log_n: int, special: int, preset: int):
        self.engine = Engine(log_coeff_count=log_n, special_prime_count=special,
                             scheme_preset=preset)
        self.keys = {}
        self.engine.seed([11, 22, 33, 44, 55, 66, 77, 88], [1, 2])
        self.secret = self.engine.create_secret_key()

    def key(self, kind, *args):
        """A key of the given kind; its random words depend on the kind alone."""
        at = (kind, *args)
        if at not in self.keys:
            e, sk = self.engine, self.secret
            e.seed([len(kind), *args, 0, 0, 0, 0, 0, 0, 0][:8], [3, 4])
            self.keys[at] = {
                "public": lambda: e.create_public_key(sk),
                "relinearization": lambda: e.create_relinearization_key(sk),
                "conjugation": lambda: e.create_conjugation_key(sk),
                "rotation": lambda: e.create_fixed_rotation_key(sk, *args),
                "bootstrap": lambda: e.create_bootstrap_key(sk, 3, "medium"),
            }[kind]()
        return self.keys[at]


_programs: dict = {}


def _program(case) -> _Program:
    at = (case["log_n"], case["special"], case["preset"])
    if at not in _programs:
        _programs[at] = _Program(*at)
    return _programs[at]


def _message(rng, count: int, complex_values: bool):
    re = rng.uniform(-1.0, 1.0, count)
    return re + 1j * rng.uniform(-1.0, 1.0, count) if complex_values else re


class _Words:
    """An engine object's limbs where they lie, as a CUDA array that keeps it alive."""

    def __init__(self, data):
        i = data.info()
        self.data = data
        self.__cuda_array_interface__ = {
            "shape": (i["polys"], i["chains"], data.engine.coeff_count),
            "typestr": "<i8", "data": (data.device_pointer(), False), "version": 2}


def _words(data) -> torch.Tensor:
    return torch.as_tensor(_Words(data), device="cuda")


def _rng_seed(seed: int) -> list:
    return [seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF, 5, 6, 7, 8, 9, 10]


def prepare(case, seed):
    p = _program(case)
    e, op = p.engine, case["op"]
    rng = np.random.default_rng(seed)
    s = {"case": case, "engine": e, "seed": _rng_seed(seed)}
    if op == "encrypt":
        s["message"] = _message(rng, case["count"], case["complex"])
        s["public"] = p.key("public")
        return s
    if op == "dot":
        s["weights"] = [e.encode(_message(rng, e.slot_count, False), case["level"])
                        for _ in range(case["terms"])]
    if op in ("hmult", "serve", "bootstrap"):
        s["relinearization"] = p.key("relinearization")
    if op == "rotate":
        s["rotations"] = [p.key("rotation", 1 << i) for i in range(case["count"])]
    if op == "serve":
        s["rotations"] = [p.key("rotation", 1 << (3 * i % ROTATION_KEYS))
                          for i in range(case["batch"])]
    if op == "bootstrap":
        s["conjugation"] = p.key("conjugation")
        s["bootstrap"] = p.key("bootstrap")
    e.seed(s["seed"], [0, 1])

    def ciphertext(level):
        values = _message(rng, e.slot_count, case.get("complex", True))
        s.setdefault("message", values)
        return e.encrypt(e.encode(values, level), p.secret)

    if op == "serve":
        span = case["high"] - case["low"] + 1
        levels = [case["low"] + 7 * i % span for i in range(case["batch"])]
    else:
        levels = [case["level"]] * {"dot": case.get("terms"), "hmult": case.get("batch"),
                                    "transform": case.get("count")}.get(op, 1)
    s["a"] = [ciphertext(level) for level in levels]
    if op in ("hmult", "serve"):
        s["b"] = [ciphertext(level) for level in levels]
    if op == "decrypt":
        s["secret"] = p.secret
    return s


def run(state):
    e, case = state["engine"], state["case"]
    op = case["op"]
    if op == "encrypt":
        e.seed(state["seed"], [0, 1])
        plain = e.encode(state["message"], case["level"])
        return [_words(plain), _words(e.encrypt(plain, state["public"]))]
    if op == "decrypt":
        return e.decode(e.decrypt(state["a"][0], state["secret"]), complex_output=case["complex"])
    if op == "dot":
        total = e.multiply_plaintext(state["a"][0], state["weights"][0])
        for x, w in zip(state["a"][1:], state["weights"][1:]):
            total = e.add(total, e.multiply_plaintext(x, w))
        return _words(total if case["level"] < 3 else e.rescale(total))
    if op == "hmult":
        a, b, rk = state["a"], state["b"], state["relinearization"]
        if len(a) == 1:
            return _words(e.multiply_relinearize_rescale(a[0], b[0], rk))
        return [_words(y) for y in e.multiply_relinearize_rescale_batch(a, b, rk)]
    if op == "rotate":
        if case["count"] == 1:
            return _words(e.rotate(state["a"][0], state["rotations"][0]))
        return [_words(y) for y in e.rotate_batch(state["a"][0], state["rotations"])]
    if op == "serve":
        return [_words(y) for y in e.multiply_rotate_batch(
            state["a"], state["b"], state["relinearization"], state["rotations"])]
    if op == "transform":
        out = []
        for x in state["a"]:
            y = e.ntt(x)
            out += [_words(y), _words(e.intt(y))]
        return out
    return _words(e.bootstrap(state["a"][0], state["relinearization"], state["conjugation"],
                              state["bootstrap"]))


def exact(case, seed):
    """The slots a decrypted message has; ciphertext words have no value of their own."""
    if case["op"] != "decrypt":
        return None
    return _message(np.random.default_rng(seed), 1 << (case["log_n"] - 1), case["complex"])


# ----------------------------------------------------------------------- work --


def work(case):
    """Limbs in and out once (8 N bytes each), keys once; three operations (a modular
    product, a sum and a difference) per butterfly of the transforms that cannot be
    left out and two per term of the limb-wise sums."""
    log_n, special, op = case["log_n"], case["special"], case["op"]
    n = 1 << log_n
    butterflies = 3 * n // 2 * log_n  # operations of one limb's transform

    def key_switch(limbs):
        """(key limbs read, operations) of one key switch of a text of `limbs` limbs."""
        parts = -(-limbs // special)
        extended = limbs + special
        transforms = limbs + (parts * extended - limbs) + 2 * extended
        products = limbs * (min(limbs, special) - 1) // 2 + limbs * extended  # digits, ModUp
        products += 2 * parts * extended + 2 * special * (limbs + special // 2)
        return 2 * parts * extended, transforms * butterflies + 2 * n * products

    def product(level):
        """(limbs in and out, key limbs, operations): lazy rescale, tensor, key switch, rescale."""
        limbs = level + 1
        key, ops = key_switch(limbs)
        ops += 4 * limbs * butterflies + 2 * n * (4 * limbs + 4 * limbs + 2 * limbs)
        return 2 * 2 * (limbs + 1) + 2 * (limbs - 1), key, ops

    limbs, ops = 0, 0
    if op == "encrypt":
        text = case["level"] + 2
        ops = 3 * text * butterflies + 2 * n * 4 * text + 10 * n * log_n
        limbs = 2 * text + text + 2 * text + case["count"] * (2 if case["complex"] else 1) / n
    elif op == "decrypt":
        text = case["level"] + 2
        ops = 2 * text * butterflies + 2 * n * 3 * text + 10 * n * log_n
        limbs = 2 * text + text + (1 if case["complex"] else 0.5)
    elif op == "dot":
        text = case["level"] + 2
        ops = case["terms"] * (3 * (text - 1) * butterflies + 2 * n * 5 * text)
        limbs = case["terms"] * 3 * text + 2 * (text - 2)
    elif op == "hmult":
        io, key, one = product(case["level"])
        limbs, ops = case["batch"] * io + key, case["batch"] * one
    elif op == "rotate":
        text = case["level"] + 2
        key, one = key_switch(text)
        limbs = 2 * text + case["count"] * (2 * text + key)
        ops = case["count"] * one
    elif op == "serve":
        span = case["high"] - case["low"] + 1
        most = 0
        for i in range(case["batch"]):
            level = case["low"] + 7 * i % span
            io, key, one = product(level)
            rotation_key, rotation = key_switch(level)
            most = max(most, key)
            limbs += io + rotation_key
            ops += one + rotation
        limbs += most
    elif op == "transform":
        text = case["level"] + 2
        limbs = case["count"] * 3 * 2 * text
        ops = case["count"] * 2 * 2 * text * butterflies
    else:
        # The medium three-stage key (13 GB) and about 80 key switches of its rotations and
        # products, half the chain high on average.
        limbs = 25000 + 2 * 5 + 2 * 12
        ops = 80 * key_switch(14)[1]
    return {"bytes": 8.0 * n * limbs, "flops": float(ops)}
