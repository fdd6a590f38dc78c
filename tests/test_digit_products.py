"""The digit products of the FP64 K3 contractions (fdga_digits.cuh; fdga_k3_oz.cu on tcgen05, fdga_k3_mma.cu on
warp-level products), emulated in integers with the number of digits read from the sources.

A value below its bound 2^F is rounded to Y = v 2^(8S-2-F) and cut into S balanced base-256 digits; the products
of digits s, t with s + t = g < S add up in one FP32 accumulator (16 products at a time); the others are dropped.
With S = 8 a product term loses at most 7·2^-62 (the seven pairs of g = 8) + 2^-62 (the rounding of both) + the
pairs beyond, below 2^-58.9 of its two bounds.  Sums of up to K = 128 terms are exact in the accumulators; for
K ≤ 256 the diagonals g ≥ 5 can pass 2^24 and then round by a unit per addition, below 2^-44 of the bounds.
The form with eight 7-bit digits that the tcgen05 kernel had before dropped up to 2^-53.2 of its bounds."""
import os
import re
from fractions import Fraction

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fddgasolver.jl_gb300", "csrc")
KERNELS = ["fdga_k3_oz.cu", "fdga_k3_mma.cu"]
TERM = 2.0 ** -58.9


def digits_of(kernel):
    src = open(os.path.join(CSRC, kernel), encoding="utf-8").read()
    return int(re.search(r"constexpr int S = (\d+);", src).group(1))


def bound_exponent(v):
    """F with every |v| < 2^F (the largest exponent field; 0 for zeros)."""
    return max((int(np.frexp(x)[1]) for x in v if x), default=0)


def fixed(x, F, S):
    y = Fraction(x) * Fraction(2) ** (8 * S - 2 - F)
    return int(y + Fraction(1, 2)) if y >= 0 else -int(-y + Fraction(1, 2))


def cut(Y, S):
    """Digits from the most significant: adding 0x80 to every byte leaves byte - 128 as the digit."""
    u = (Y + int("80" * 8, 16)) % 2 ** 64
    return [((u >> (8 * (S - 1 - s))) & 255) - 128 for s in range(S)]


def digit_dot(a, b, S):
    """(the emulated Σ a b, the sum's two bounds as a Fraction)."""
    FA, FB = bound_exponent(a), bound_exponent(b)
    da, db = (np.array([cut(fixed(x, F, S), S) for x in v]) for v, F in ((a, FA), (b, FB)))
    acc = np.zeros(S, dtype=np.float32)
    for k in range(0, len(a), 16):
        for s in range(S):
            for t in range(S - s):
                acc[s + t] += np.float32(int(da[k:k + 16, s] @ db[k:k + 16, t]))
    E = FA + FB - 2 * (8 * S - 2)
    c = sum(int(acc[g]) * 256 ** (2 * (S - 1) - g) for g in range(S))
    return Fraction(c) * Fraction(2) ** E, Fraction(2) ** (FA + FB)


def exact_dot(a, b):
    return sum((Fraction(x) * Fraction(y) for x, y in zip(a, b)), Fraction(0))


@pytest.mark.parametrize("kernel", KERNELS)
def test_digits_restore_the_value(kernel):
    S = digits_of(kernel)
    rng = np.random.default_rng(1)
    for x in np.concatenate([rng.standard_normal(50), 2.0 ** -np.arange(9), -1 + 2.0 ** -np.arange(1, 53)]):
        F = bound_exponent([x])
        d = cut(fixed(x, F, S), S)
        assert all(-128 <= v <= 127 for v in d) and abs(d[0]) <= 64
        assert Fraction(sum(v * 256 ** (S - 1 - s) for s, v in enumerate(d))) * Fraction(2) ** (F - 8 * S + 2) == Fraction(x)


@pytest.mark.parametrize("kernel", KERNELS)
def test_one_product_of_the_worst_digits(kernel):
    """Digits 32, -128, ..., -128 on both sides (the dropped products all positive)."""
    S = digits_of(kernel)
    Y = 32 * 256 ** (S - 1) - sum(128 * 256 ** s for s in range(S - 1))
    d = cut(Y, S)
    assert d == [32] + [-128] * (S - 1)
    kept = sum(d[s] * d[t] * 256 ** (2 * (S - 1) - s - t) for s in range(S) for t in range(S - s))
    lost = Fraction(abs(Y * Y - kept), 2 ** (2 * (8 * S - 2)))
    assert lost + Fraction(1, 2 ** (8 * S - 2)) <= TERM
    assert lost < 2.0 ** -53.2  # the former eight 7-bit digits


@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("kind", ["flat", "decaying", "opposed", "apart", "constant"])
@pytest.mark.parametrize("K", [16, 48, 128, 256])
def test_dot_products(kernel, kind, K):
    S = digits_of(kernel)
    rng = np.random.default_rng(K)
    w = np.arange(1, K + 1) / 4.0
    for _ in range(4):
        a, b = rng.standard_normal(K), rng.standard_normal(K)
        if kind == "decaying":
            a, b = a / (1 + w * w), b / (1 + w * w)
        elif kind == "opposed":
            a, b = a / w ** 4, b * w ** 4
        elif kind == "apart":  # the largest entries of the two at different ω
            a[0], b[-1] = 2.0 ** 30, -2.0 ** 30
        elif kind == "constant":  # every digit -128: the accumulators' largest sums
            a = b = np.full(K, -128.0 / 255.0)
        c, B = digit_dot(a, b, S)
        tol = K * TERM * B + (0 if K <= 128 else Fraction(2) ** -44 * B)
        assert abs(c - exact_dot(a, b)) <= tol
        if kind in ("flat", "decaying") and K <= 128:  # terms near their bounds: no worse than an FP64 sum's own bound
            assert abs(c - exact_dot(a, b)) <= K * 2.0 ** -53 * sum(abs(Fraction(x) * Fraction(y)) for x, y in zip(a, b))
