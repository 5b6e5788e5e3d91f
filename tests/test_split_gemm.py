"""The split-BF16 GEMM (dqmc_gb300/csrc/k_ozaki.cu, oz_slice.cuh).

CPU: the digit cutting and the rounding of the two-word sums, restated step
for step on Python integers.  GPU: products at the edges of tiles, K chunks and
slices within the bound that the slicing gives, and at 56 bits no further from
the exact product than the FP64 FMA kernel."""
import math
from fractions import Fraction

import numpy as np
import pytest

M64 = (1 << 64) - 1


def digits(X, S, bits):
    """oz_next_digit on a 62-bit fixed-point integer, S times."""
    out = []
    for p in range(1, S + 1):
        s = 62 - p * bits
        if s <= 0:
            out.append(X << -s)
            X = 0
            continue
        q = (X + (1 << (s - 1)) - 1 + ((X >> s) & 1)) >> s
        X -= q << s
        out.append(q)
    return out


@pytest.mark.parametrize("S,bits", [(2, 7), (6, 7), (8, 7), (8, 8)])
def test_digits_reconstruct_the_value(S, bits):
    rng = np.random.default_rng(S * 10 + bits)
    top = (1 << 62) - (1 << 9)
    for X in [0, 1, -1, top, -top, 1 << 61, -(1 << 61)] + [int(v) for v in rng.integers(-top, top, 400)]:
        if S * bits > 62:
            X &= ~0xFF   # a double's 53 bits: the low bits of the fixed point are zero
        d = digits(X, S, bits)
        assert abs(d[0]) <= 1 << bits
        assert all(abs(v) <= 1 << (bits - 1) for v in d[1:])
        rest = X - sum(Fraction(v) * Fraction(2) ** (62 - (p + 1) * bits) for p, v in enumerate(d))
        assert abs(rest) <= Fraction(2) ** (61 - S * bits)


def wide_ldexp(hi, lo, sh, e):
    h0 = hi & M64
    l = (h0 << sh) & M64
    h = (hi >> (64 - sh)) & M64
    l = (l + (lo & M64)) & M64
    h = (h + ((lo >> 63) & M64) + (1 if l < (lo & M64) else 0)) & M64
    neg = h >> 63 == 1
    if neg:
        l = -l & M64
        h = ((h ^ M64) + (1 if l == 0 else 0)) & M64
    ex = e + 64
    if h == 0:
        h, l, ex = l, 0, e
    if h == 0:
        return 0.0
    lz = 64 - h.bit_length()
    m = ((h << lz) | (l >> (64 - lz))) & M64 if lz else h
    sticky = (l << lz) & M64 != 0
    q = m >> 11
    rem = m & 0x7FF
    q += 1 if rem + ((q & 1) | (1 if sticky else 0)) > 0x400 else 0
    bits = ((63 - lz + ex + 1023 - 1) << 52) + q
    v = np.uint64(bits & M64).view(np.float64)
    return -float(v) if neg else float(v)


def test_wide_sum_rounds_once():
    rng = np.random.default_rng(5)
    cases = [(0, 0), (0, 1), (0, -1), (1, -1), (-1, 1), (1 << 47, -(1 << 47)), (-(1 << 47), (1 << 47) - 1)]
    for _ in range(4000):
        s = int(rng.integers(1, 48))
        cases.append((int(rng.integers(-(1 << s), 1 << s)), int(rng.integers(-(1 << 47), 1 << 47))))
    for k in range(20, 40):   # ties and their neighbours
        cases += [((1 << 53) + 1 << 20 >> k, d) for d in (-1, 0, 1)]
    for hi, lo in cases:
        for sh, e in ((28, -63), (32, -72)):
            v = (hi << sh) + lo
            assert wide_ldexp(hi, lo, sh, e) == math.ldexp(float(v), e)   # float(int) rounds to nearest even


def _matrix(kind, n, rng):
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    if kind == "unitary":
        return np.linalg.qr(a)[0]
    if kind == "rows":
        return a * np.logspace(-6, 6, n)[:, None]
    if kind == "cols":
        return a * np.logspace(6, -6, n)[None, :]
    return a


def _expo(x):
    """2^E, E the frexp exponent of the largest component."""
    return 2.0 ** np.frexp(x)[1]


@pytest.mark.gpu
@pytest.mark.parametrize("L,bits", [(2, 0), (2, 60), (4, 0), (4, 14), (4, 56), (6, 0), (6, 48), (10, 0), (16, 0)])
@pytest.mark.parametrize("kind", ["plain", "rows", "cols"])
def test_split_product_within_its_bound(L, bits, kind):
    from dqmc_gb300 import api
    chain = api.DQMC(api.ModelParams(L=L, slices=10, safe_mult=10, precision="mixed", ozaki_bits=bits))
    n = 4 * L * L
    rng = np.random.default_rng(100 * L + bits)
    A, B = _matrix(kind, n, rng), _matrix("plain", n, rng)
    C = chain.gemm_check(A, B, 1)
    want = (A.astype(np.clongdouble) @ B.astype(np.clongdouble)) if n <= 144 else A @ B
    kp = 2 * ((n + 15) // 16 * 16)
    S, w = next((S, S * b) for S in range(2, 9) for b in [min(8, math.floor((24 - math.log2(kp * S)) / 2))]
                if S * b >= (bits or 40))
    big = lambda X, ax: np.maximum(np.abs(X.real).max(ax), np.abs(X.imag).max(ax))
    # per term: both operands truncated by 2^-(w+1), pairs p + q > S + 1 dropped (< (S / 4 + 1/2) 2^-w); 2n terms per part
    term = (1.0 + S / 4.0 + 0.5) * 2.0 ** -w
    bound = 2 * n * term * np.outer(_expo(big(A, 1)), _expo(big(B, 0)))
    bound = np.sqrt(2.0) * bound + 2.0 ** -50 * np.abs(want) + (n * 2.0 ** -52 * (np.abs(A) @ np.abs(B)) if n > 144 else 0)
    err = np.abs(C - want)
    assert np.all(err <= bound), float((err / bound).max())
    chain.close()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["plain", "unitary", "rows", "cols"])
def test_56_bits_no_further_off_than_fma(kind):
    from dqmc_gb300 import api
    chain = api.DQMC(api.ModelParams(L=4, slices=10, safe_mult=10, precision="mixed", ozaki_bits=56))
    rng = np.random.default_rng(9)
    A, B = _matrix(kind, 64, rng), _matrix("unitary" if kind == "unitary" else "plain", 64, rng)
    want = A.astype(np.clongdouble) @ B.astype(np.clongdouble)
    err = [float(np.linalg.norm((chain.gemm_check(A, B, m) - want).astype(complex) / np.linalg.norm(A, axis=1)[:, None]))
           for m in (0, 1)]
    assert err[1] <= err[0], err
    chain.close()


@pytest.mark.gpu
def test_nan_and_inf_reach_the_product():
    from dqmc_gb300 import api
    chain = api.DQMC(api.ModelParams(L=6, slices=10, safe_mult=10, precision="mixed"))
    rng = np.random.default_rng(3)
    n = 144
    for bad in (np.nan, np.inf):
        A, B = _matrix("plain", n, rng), _matrix("plain", n, rng)
        A[5, 7] = bad
        B[3, 140] = -bad
        ok = np.isfinite(chain.gemm_check(A, B, 1))
        want = np.ones((n, n), bool)
        want[5] = False
        want[:, 140] = False
        assert np.array_equal(ok, want)
    chain.close()


@pytest.mark.gpu
@pytest.mark.parametrize("L,bits", [(2, 0), (2, 56), (4, 0), (4, 56), (6, 0), (6, 48), (8, 0), (10, 0), (12, 0)])
def test_tile_width_keeps_the_bits(L, bits):
    # tiles of 8 (n <= 144), 16 (n = 256, with split K) and 32 columns: sums are
    # exact, so the product is that of the 32 columns which chains in flight take
    from dqmc_gb300 import api
    n = 4 * L * L
    rng = np.random.default_rng(L)
    A, B = _matrix("rows", n, rng), _matrix("plain", n, rng)
    got = []
    for inflight in (0, 8):
        chain = api.DQMC(api.ModelParams(L=L, slices=10, safe_mult=10, precision="mixed", ozaki_bits=bits,
                                         inflight=inflight))
        got.append(chain.gemm_check(A, B, 1))
        chain.close()
    assert np.array_equal(got[0], got[1])
