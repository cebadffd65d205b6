"""The tracers' branch-free FP64 reciprocal, quotient and square root against IEEE
division and square root (the host's, and CUDA's `/` and sqrt): equal to the bit.

Operands: random ones over the stated range of magnitudes, its ends, 0, divisors
of all ones and near it (whose reciprocals lie next to a midpoint between doubles),
and the operands whose quotients and roots lie nearest to such a midpoint. Those
follow from modular arithmetic: A / B is j / (B 2^54) from the midpoint M 2^-54 for
M = j / B mod 2^54 and A = (B M - j) / 2^54, and sqrt(A 2^s) next to M for M^2 = j
mod 2^s and A = (M^2 - j) / 2^s."""
import ctypes as C
import os
import random
import subprocess

import numpy as np
import pytest

from bellhopcuda_b200 import build as recipe

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("math") / "device_math_check.so")
    subprocess.check_call([recipe.nvcc(), *recipe.ARCH, "-O3", "-std=c++17", "-fmad=false", "-I" + recipe.CSRC, "-shared",
                           "-Xcompiler", "-fPIC", os.path.join(HERE, "device_math_check.cu"), "-o", so])
    lib = C.CDLL(so)

    def call(op, a, b):
        a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)
        out = np.empty_like(a)
        p = lambda v: v.ctypes.data_as(C.POINTER(C.c_double))
        assert lib.device_math(op, p(a), p(b), p(out), len(a)) == 0
        return out
    return call


def mantissas(rng, n):
    """odd integers of 53 bits: random, all ones and down from it, one and up from it"""
    out = []
    while len(out) < n:
        k = rng.randrange(4)
        if k == 0:
            out.append(rng.getrandbits(52) | (1 << 52) | 1)
        elif k == 1:
            out.append((1 << 53) - 1 - 2 * rng.randrange(1 << rng.randrange(1, 40)))
        elif k == 2:
            out.append((1 << 52) + 1 + 2 * rng.randrange(1 << rng.randrange(1, 40)))
        else:
            out.append((1 << 53) - 1 - 2 * (len(out) % 512))
    return out


def hard_quotients(rng, n):
    a, b = [], []
    for B in mantissas(rng, n):
        j = rng.choice([1, -1, 3, -3, 5, -5, 7, -7])
        M = j * pow(B, -1, 1 << 54) % (1 << 54)
        A = (B * M - j) >> 54
        if M >= 1 << 53 and 0 < A < 1 << 53:
            a.append(float(A))
            b.append(float(B))
    return np.array(a), np.array(b)


def hard_roots():
    out = []
    for s in (54, 55):
        for j in list(range(1, 4000, 8)) + list(range(-7, -4000, -8)):
            x = 1
            for k in range(3, s):
                if (x * x - j) % (1 << (k + 1)):
                    x += 1 << (k - 1)
            m = 1 << s
            for M in {x % m, -x % m, (x + m // 2) % m, (-x + m // 2) % m}:
                if 1 << 53 <= M < 1 << 54 and (M * M - j) >> s < 1 << 53:
                    out.append(float((M * M - j) >> s) * 2.0 ** (s % 2))
    return np.array(out)


def scaled(rng, m, span):
    return m * 2.0 ** rng.integers(-span, span, len(m))


def same(x, y):
    return np.array_equal(x.view(np.int64), y.view(np.int64))


def test_divisors(device):
    rng = random.Random(5)
    g = np.random.default_rng(5)
    b = np.concatenate([np.array(mantissas(rng, 100000), np.float64) * 2.0 ** -52, g.uniform(1.0, 2.0, 400000)])
    wide = np.concatenate([scaled(g, b, 890) * g.choice([-1.0, 1.0], len(b)), [2.0 ** 900, 2.0 ** -900, 1.0, 3.0]])
    assert same(device(0, wide, wide), 1.0 / wide)
    assert same(device(7, wide, np.abs(wide)), 1.0 / np.abs(wide))
    not_ones = wide[(wide > 0.0) | (wide.view(np.int64) & ((1 << 52) - 1) != (1 << 52) - 1)]
    assert same(device(7, not_ones, not_ones), 1.0 / not_ones)
    # the six b whose squares' reciprocals lie so near a midpoint that one Newton step misses it
    six = np.array([0x17e23ea0c37857, 0x18da7d634a84b0, 0x1f0cba276f78fb, 0x108360cd3ed557, 0x175a6a5d5f9e1e,
                    0x1aac5548dbdf1c], np.float64) * 2.0 ** -52
    half = np.concatenate([scaled(g, b, 440), [2.0 ** 449, 2.0 ** -449, 1500.0], six, 1024.0 * six])
    assert same(device(2, half, half), 1.0 / (half * half))
    assert same(device(5, np.ones_like(wide), wide), 1.0 / wide)


def test_quotients(device):
    g = np.random.default_rng(6)
    a, b = hard_quotients(random.Random(6), 40000)
    assert len(a) > 10000
    k = np.concatenate([[0.0], g.uniform(-2.0, 2.0, 1000000)])
    no = b != 2.0 ** 53 - 1.0   # all ones: positive divisors only
    x = np.concatenate([a, -a * 2.0 ** -300, a[no], scaled(g, k, 400)])
    y = np.concatenate([b, b * 2.0 ** 200, -b[no], scaled(g, g.uniform(1.0, 2.0, len(k)) * g.choice([-1.0, 1.0], len(k)), 400)])
    x[-len(k)], y[-len(k)] = 0.0, 3.0
    ref = x / y
    assert same(device(1, x, y), ref) and same(device(5, x, y), ref)
    z = np.concatenate([np.array(mantissas(random.Random(7), 200000), np.float64) * 2.0 ** -52,
                        scaled(g, g.uniform(1.0, 2.0, 400000), 200)])
    w = scaled(g, g.uniform(1.0, 2.0, len(z)), 400)
    assert same(device(3, w, z), w / (z * z))


def test_roots(device):
    g = np.random.default_rng(8)
    a = hard_roots()
    assert len(a) > 1000
    ones = np.array(mantissas(random.Random(8), 100000), np.float64)
    x = np.concatenate([a, scaled(g, np.concatenate([ones, g.uniform(1.0, 4.0, 1000000)]), 420), [2.0 ** -900, 2.0 ** 900]])
    assert same(device(4, x, x), np.sqrt(x)) and same(device(6, x, x), np.sqrt(x))
    ends = np.array([0.0, 5e-324, 1e-310, 1e-300, 1e-280, 1e-270, 1e270, 1e280, 1.7e308, np.inf])
    assert same(device(8, ends, ends), np.sqrt(ends)) and same(device(8, x, x), np.sqrt(x))
