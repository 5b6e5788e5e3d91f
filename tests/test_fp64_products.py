"""Products of the FP64 form (dqmc_gb300/csrc/k_ozaki.cu, exact form): 9 slices
of 7 bits with a check per element, FP64 dot products where the slices hold too
little of an element.

CPU: digits and magnitudes restated on Python integers.  GPU: single elements
against the exact product within the bounds of both ways, for operands graded
along rows, columns and, in opposite directions, along the inner index; the
error of whole matrices against that of FP64 multiply-adds (mode 0)."""
import math
from fractions import Fraction

import numpy as np
import pytest

from test_split_gemm import digits

S, BITS = 9, 7


def test_nine_digits_reconstruct_the_value():
    rng = np.random.default_rng(1)
    top = (1 << 62) - (1 << 9)
    for X in [0, 1, -1, top, -top, 1 << 61, -(1 << 61), 32, -32, 31] + [int(v) for v in rng.integers(-top, top, 1000)]:
        d = digits(X, S, BITS)
        assert abs(d[0]) <= 1 << BITS
        assert all(abs(v) <= 1 << (BITS - 1) for v in d[1:])
        assert X == sum(Fraction(v) * Fraction(2) ** (62 - (p + 1) * BITS) for p, v in enumerate(d))


def oz_mag(x, E):
    b = int(np.float64(abs(x)).view(np.uint64))
    if b == 0:
        return 0
    f = (b >> 52) - 1023 - E + 127
    return 67 << 7 if f < 67 else f << 7 | (b >> 45 & 0x7F)


def test_magnitudes():
    rng = np.random.default_rng(2)
    bf16 = lambda v: float(np.uint32(v << 16).view(np.float32))
    for x in list(rng.standard_normal(200) * 10.0 ** rng.uniform(-17, 0, 200)) + [0.5, 2.0 ** -60, -(2.0 ** -59)]:
        for E in (1, 3):
            y = abs(math.ldexp(x, -E))
            assert y < 1
            m = bf16(oz_mag(x, E))
            assert y * (1 - 2.0 ** -7) < m <= y or (y < 2.0 ** -60 and m == 2.0 ** -60)
    assert bf16(oz_mag(0.0, 0)) == 0.0 and bf16(oz_mag(5e-324, 0)) == 2.0 ** -60


def operands(kind, n, seed=0):
    rng = np.random.default_rng(seed)
    c = lambda: rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    A, B, k = c(), c(), np.linspace(0.0, 1.0, n)
    if kind == "rows and columns":
        return A * 10.0 ** (12 * k - 6)[:, None], B * 10.0 ** (5 - 10 * k)[None, :]
    if kind == "opposite":      # along the inner index
        return A * 10.0 ** (-8 * k)[None, :], B * 10.0 ** (8 * k)[:, None]
    if kind == "crossed":       # rows and columns of either direction: no scaling of the inner index helps
        s = np.where(np.arange(n) % 2, 1.0, -1.0)
        return A * 10.0 ** (8 * np.outer(s, k - 0.5)), B * 10.0 ** (8 * np.outer(k - 0.5, s))
    if kind == "decaying":
        d = np.exp(-0.3 * np.abs(np.subtract.outer(np.arange(n), np.arange(n))))
        return A * d, B * d
    if kind == "triangular":
        return np.triu(A), np.tril(B)
    if kind == "unitary":
        return np.linalg.qr(A)[0], np.linalg.qr(B)[0]
    if kind == "identity":
        return np.eye(n) + 0j, B * 10.0 ** (-9 * rng.uniform(size=(n, n)))
    return A, B


KINDS = ["plain", "rows and columns", "opposite", "crossed", "decaying", "triangular", "unitary", "identity"]


def exact_element(a, b):
    """sum a b of complex vectors (rationals), and sum |a| |b|."""
    def ints(v):   # v 2^600
        m, e = np.frexp(v)
        return [int(x * 2.0 ** 53) << (int(y) + 547) for x, y in zip(m, e)]

    ar, ai, br, bi = ints(a.real), ints(a.imag), ints(b.real), ints(b.imag)
    re = sum(x * y - u * v for x, y, u, v in zip(ar, br, ai, bi))
    im = sum(x * v + u * y for x, y, u, v in zip(ar, br, ai, bi))
    return Fraction(re, 1 << 1200), Fraction(im, 1 << 1200), float(np.abs(a) @ np.abs(b))


def chain_of(L, inflight=0, **kw):
    from dqmc_gb300 import api
    return api.DQMC(api.ModelParams(L=L, slices=10, safe_mult=10, inflight=inflight, **kw))


@pytest.mark.gpu
@pytest.mark.parametrize("inflight", [0, 8])
@pytest.mark.parametrize("L", [2, 4, 6, 8, 10, 12, 14, 16])
def test_elements_against_the_exact_product(L, inflight):
    """n = 16 .. 1024: tiles of 8, 16 and 24 columns, split K and not, one to seven chunks."""
    chain = chain_of(L, inflight)
    n = 4 * L * L
    rows = sorted({r for r in (0, 1, 63, n // 2, 127, 128, n - 2, n - 1) if r < n})
    cols = sorted({c for c in (0, 7, 8, 15, 23, 24, n // 2 + 1, n - 1) if c < n})
    # slices: 2 n real terms of at most (2 + S / 4 + 1 / 2) 2^-62 of the scales, which are below 2^8 / sqrt(2 n)
    # sqrt(2) sum |a| |b|; dot product: n / 16 + 7 roundings of partial sums; and the last rounding
    slices = math.sqrt(2 * n) * (2.5 + S / 4) * 2.0 ** (-62 + 8 + 0.5)
    dot = (n / 16 + 8) * 2.0 ** -52.5
    for kind in KINDS:
        A, B = operands(kind, n, seed=L)
        C = chain.gemm_check(A, B, 1)
        for r in rows:
            for c in cols:
                re, im, mag = exact_element(A[r], B[:, c])
                err = math.hypot(float(Fraction(C[r, c].real) - re), float(Fraction(C[r, c].imag) - im))
                assert err <= (slices + dot) * mag + 2.0 ** -52.5 * abs(C[r, c]), (kind, r, c, err / max(mag, 1e-300))
    chain.close()


@pytest.mark.gpu
@pytest.mark.parametrize("L", [4, 8, 14])
@pytest.mark.parametrize("kind", KINDS)
def test_no_further_off_than_multiply_adds(L, kind):
    """rms over elements of the error relative to sum |a| |b|, 40 x 40 elements."""
    chain = chain_of(L)
    n = 4 * L * L
    A, B = operands(kind, n, seed=100 + L)
    C = [chain.gemm_check(A, B, m) for m in (0, 1)]
    rng = np.random.default_rng(L)
    R, Q = rng.choice(n, 24, replace=False), rng.choice(n, 24, replace=False)
    e2 = [0.0, 0.0]
    for r in R:
        for c in Q:
            re, im, mag = exact_element(A[r], B[:, c])
            if mag == 0.0:
                assert C[0][r, c] == C[1][r, c] == 0
                continue
            for m in (0, 1):
                v = C[m][r, c]
                e2[m] += (float(Fraction(v.real) - re) / mag) ** 2 + (float(Fraction(v.imag) - im) / mag) ** 2
    assert e2[1] <= e2[0], [math.sqrt(e / 576) for e in e2]
    chain.close()


@pytest.mark.gpu
@pytest.mark.parametrize("L", [4, 8, 16])   # split K from n = 256 on, n = 1024 without
def test_special_values_as_in_multiply_adds(L):
    chain = chain_of(L)
    n = 4 * L * L
    A, B = operands("plain", n, seed=7)
    A[3, 5] = np.inf
    A[n - 1, 2] = np.nan
    B[4, n - 2] = -np.inf
    A[1] = 0.0            # zero row: zeros, NaN where it meets the infinite column
    B[:, 2] = 0.0
    A[6] *= 5e-310        # a denormal row
    C = [chain.gemm_check(A, B, m) for m in (0, 1)]
    for part in (np.real, np.imag):
        x, y = part(C[0]), part(C[1])
        assert np.array_equal(np.isnan(x), np.isnan(y))
        assert np.array_equal(np.isposinf(x), np.isposinf(y)) and np.array_equal(np.isneginf(x), np.isneginf(y))
    assert np.all(C[1][1, 2:n - 2] == 0) and np.all(np.delete(C[1][:, 2], [3, n - 1]) == 0)
    ok = np.isfinite(C[0][6])
    assert np.abs(C[1][6, ok] - C[0][6, ok]).max() <= 2 * n * 5e-324 * 4
    chain.close()


@pytest.mark.gpu
def test_products_are_reproducible():
    """Split K adds integers in any order, the magnitudes among them."""
    chain = chain_of(8)
    A, B = operands("decaying", 256, seed=3)
    want = chain.gemm_check(A, B, 1)
    for _ in range(10):
        assert np.array_equal(chain.gemm_check(A, B, 1), want)
    chain.close()


@pytest.mark.gpu
def test_greens_of_oppositely_graded_factors():
    """G = (1 + Tl Tr^dag)^-1 for Tl falling and Tr rising by 10^8 along the inner
    index: 64-bit rounding of Tl Tr^dag, whose entries are of order n."""
    n = 64
    chain = chain_of(4)
    rng = np.random.default_rng(11)
    g = 10.0 ** (8 * np.linspace(0, 1, n))
    c = lambda: rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    Tl, Tr = c() / g[None, :], c() * g[None, :]
    one, d = np.eye(n) + 0j, np.ones(n)
    G, _ = chain.calculate_greens_udt(one, d, Tl, one, d, Tr)
    chain.close()
    X = np.eye(n) + ((Tl * g[None, :]) @ (Tr / g[None, :]).conj().T)   # rounding of g: n 2^-53 per entry
    want = np.linalg.inv(X)
    # |dG| <= |G| |dX| |G| with |dX| <= n 2^-52 |Tl| |Tr|^T, and the inverse's own n 2^-53 cond
    mag = (np.abs(Tl) * g[None, :]) @ (np.abs(Tr) / g[None, :]).T
    nG = np.linalg.norm(want, 2)
    bound = nG * nG * np.linalg.norm(n * 2.0 ** -51 * mag + n * 2.0 ** -52 * np.abs(X), 2)
    assert np.abs(G - want).max() <= bound, (np.abs(G - want).max(), bound)
