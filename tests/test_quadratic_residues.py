"""CPU checks, in exact arithmetic and with the kernels' own FP32 and FP64
operations, of the quadratic residue numbers the tensor-core forms' exact
recompute uses (ozaki.cu): images of an element from its 16-bit limbs, the
residue byte of a product sum, and the reconstruction of both parts."""
import math
import random
import re
import os
from fractions import Fraction

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                   "ascend-open-source-contributions_b200", "csrc", "ozaki.cu")
BETA, MAX_N = 47, 4096
F = np.float32
MAGIC = F(12582912.0)


def _table(name):
    body = re.search(name + r"\[kOzMods\] = \{([^}]*)\}", open(SRC).read()).group(1)
    return [int(x) for x in body.split(",")]


MODULI, ROOTS = _table("kOzModuli"), _table("kOzRoots")


def _balanced(v, p):
    r = v % p
    return r if r <= p // 2 else r - p


def _limbs(t):
    """limbs16: the word arithmetic of the kernel."""
    w = (0x4338000000000000 + t) & (2 ** 64 - 1)
    lo, hi = w & 0xFFFFFFFF, (w >> 32) - 0x43380000
    l0 = (lo & 0xFFFF) - (0x10000 if lo & 0x8000 else 0)
    m1 = (lo >> 16) + (1 if l0 < 0 else 0)
    return l0, (m1 - 65536 if m1 >= 32768 else m1), hi + (1 if m1 >= 32768 else 0)


def _mod_byte(s, p):
    """mod_bits2 on one FP32 value (each FMA's result is exact or rounded once)."""
    inv = F(1.0) / F(p)
    q = F(F(float(s) * float(inv) + float(MAGIC)) - MAGIC)  # the FP64 sum rounds once to FP32 (24 + 24 bits < 53)
    r = float(s) - float(q) * p
    assert r == int(r) and abs(r) <= 125
    b = (0x4B400000 + int(r)) & 0xFF
    return b - 256 if b >= 128 else b


def test_moduli_and_roots():
    M = math.prod(MODULI)
    for i, (p, r) in enumerate(zip(MODULI, ROOTS)):
        assert (r * r + 1) % p == 0
        assert all(math.gcd(p, q) == 1 for q in MODULI[:i])
    assert 2 * MAX_N * 2 ** (2 * BETA) <= M // 8


@pytest.mark.parametrize("p,r", list(zip(MODULI, ROOTS)))
def test_images_and_products_mod_p(p, r):
    rng = random.Random(p)
    edge = [0, 1, -1, 2 ** BETA, -2 ** BETA, 2 ** 31, 2 ** 31 - 1, -2 ** 31, 32767, 32768, -32768, -32769,
            2 ** 47 - 2 ** 16, 2 ** 32 - 1, 2 ** 32 - 32768, 65535 * 65536]
    c1, c2 = _balanced(2 ** 16, p), _balanced(2 ** 32, p)
    d = [_balanced(r * 2 ** e, p) for e in (0, 16, 32)]

    def images(x, y):
        a, b = _limbs(x), _limbs(y)
        for v, l in ((x, a), (y, b)):
            assert l[2] * 2 ** 32 + l[1] * 2 ** 16 + l[0] == v and all(abs(t) <= 2 ** 15 for t in l)
        sa = a[2] * c2 + a[1] * c1 + a[0]
        sb = b[2] * d[2] + b[1] * d[1] + b[0] * d[0]
        assert max(abs(sa), abs(sb), abs(sa + sb), abs(sa - sb)) < 2 ** 24
        return _mod_byte(sa + sb, p), _mod_byte(sa - sb, p)

    draws = [(rng.choice(edge), rng.choice(edge)) for _ in range(200)]
    draws += [(rng.randint(-2 ** BETA, 2 ** BETA), rng.randint(-2 ** BETA, 2 ** BETA)) for _ in range(200)]
    inv, bias = 2 ** 32 // p, -(-2 ** 26 // p) * p
    sums, re, im = [0, 0], 0, 0
    for (x, y), (u, v) in zip(draws, reversed(draws)):
        a, b = images(x, y), images(u, v)
        assert (a[0] - (x + r * y)) % p == 0 and (a[1] - (x - r * y)) % p == 0
        sums = [s + g * h for s, g, h in zip(sums, a, b)]
        re, im = re + x * u - y * v, im + x * v + y * u
    out = []
    for s in sums:
        X = s + bias
        byte = X - ((X * inv) >> 32) * p
        assert 0 <= byte < 256 and (byte - s) % p == 0
        out.append(byte)
    half, root = pow(2, -1, p), pow(2 * r, -1, p)
    assert (sum(out) * half - re) % p == 0 and ((out[0] - out[1]) * root - im) % p == 0
    # the residue byte over the whole range of a sum of MAX_N products
    for s in [125 * 125 * MAX_N, -125 * 125 * MAX_N, 0, 1, -1] + [rng.randint(-2 ** 26, 2 ** 26) for _ in range(2000)]:
        X = s + bias
        byte = X - ((X * inv) >> 32) * p
        assert 0 <= byte < 256 and (byte - s) % p == 0


def test_reconstruction_of_both_parts():
    M = math.prod(MODULI)
    mask = 2 ** 40 - 1
    split = lambda v: [float((v >> (40 * l)) & mask) for l in range(3)]  # noqa: E731
    w = []
    for p, r in zip(MODULI, ROOTS):
        W = M // p
        w.append([split(W * pow(2 * W % p, -1, p)), split(W * pow(2 * W * r % p, -1, p))])
    m, k2, k1 = split(M), float(Fraction(2 ** 80, M)), float(Fraction(2 ** 40, M))
    rng = random.Random(11)
    bound = 2 * MAX_N * 2 ** (2 * BETA)
    for _ in range(3000):
        x = [rng.choice([0, 1, -1, bound, -bound, rng.randint(-bound, bound), rng.randint(-2 ** 30, 2 ** 30)])
             for _ in range(2)]
        s = [[0.0] * 3, [0.0] * 3]
        for i, (p, r) in enumerate(zip(MODULI, ROOTS)):
            # any byte congruent to the product may be stored, up to p + p / 32
            y = [(x[0] + r * x[1]) % p, (x[0] - r * x[1]) % p]
            y = [v + p if v + p <= p + p // 32 and rng.random() < 0.5 else v for v in y]
            for part, v in enumerate((y[0] + y[1], y[0] - y[1])):
                for l in range(3):
                    s[part][l] += v * w[i][part][l]
                    assert abs(s[part][l]) < 2.0 ** 53
        for part in range(2):
            S = sum(int(s[part][l]) << (40 * l) for l in range(3))
            est = s[part][2] * k2 + s[part][1] * k1
            assert abs(est - float(Fraction(S, M))) < 2.0 ** -30
            k = round(est)
            assert S - k * M == x[part]
            d = [int(s[part][l]) - k * int(m[l]) for l in range(3)]
            assert all(abs(v) <= 2 ** 53 for v in d)
            got = (float(d[2]) * 2.0 ** 40 + float(d[1])) * 2.0 ** 40 + float(d[0])
            assert abs(got - x[part]) <= abs(x[part]) * 2.0 ** -52
