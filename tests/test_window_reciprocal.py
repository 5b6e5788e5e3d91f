"""1 / det M in k_local_window: Newton's iteration from a single-precision seed
(recip_newton, restated with exactly rounded FMAs), and ratios whose squared
modulus leaves the range of double."""
import ctypes
from fractions import Fraction

import numpy as np
import pytest

from oracle.dqmc_ref import synthetic_field


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def recip_newton(x):
    y = float(np.float32(1.0) / np.float32(x))
    y = fma(fma(-x, y, 1.0), y, y)
    return fma(fma(-x, y, 1.0), y, y)


def test_newton_against_the_division():
    """Seed within 2^-23, squared twice, and the roundings of the last step: 1 ulp."""
    rng = np.random.default_rng(3)
    xs = [1.0, 2.0 - 2.0 ** -52, 1.0 + 2.0 ** -52, 1.5, 4.0 / 3.0] + list(rng.uniform(1.0, 2.0, 2000))
    for e in (-100, -99, -37, -1, 0, 1, 52, 99, 100):
        for x in xs if e in (-100, 0, 100) else xs[:300]:
            v = float(np.ldexp(x, e))
            want = Fraction(1) / Fraction(v)
            got = recip_newton(v)
            assert abs(Fraction(got) - want) <= Fraction(np.spacing(float(want))), v


@pytest.mark.gpu
@pytest.mark.parametrize("g", [1.0, 1e30, 1e42])
def test_ratios_of_any_size(g):
    """The block of G of one site scaled to g: its ratio is about 1e-8 g^4 (1e160 at
    the last), and the update takes the block back to order one, up to the
    cancellation of 64-bit rounding on g.  Against k_local_updates."""
    torch = pytest.importorskip("torch")
    from dqmc_gb300 import api
    L, M, site = 4, 10, 5
    mp = api.ModelParams(L=L, slices=M, safe_mult=10)
    N, n = mp.N, mp.n
    chain = api.DQMC(mp, synthetic_field(N, M, 12))
    chain.init()
    G0 = np.array(chain.greens)
    own = site + N * np.arange(4)
    if g != 1.0:
        G0[own, own] = g
    chain.greens = G0
    delta = np.asfortranarray(np.random.default_rng(4).uniform(-0.2, 0.2, (3, N)))
    unif = np.full(N, 2.0)          # accepted where p > 1
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    G = dev(np.asfortranarray(G0).ravel(order="F").view(np.float64))
    f, d, u = dev(chain.get_field().ravel(order="F")), dev(delta.ravel(order="F")), dev(unif)
    act, acc = dev(np.array([chain.boson_action])), torch.zeros(N, dtype=torch.uint8).cuda()
    slice1 = chain.current_slice
    _, got, det, _ = chain.local_updates(delta, unif, return_details=True)
    torch.cuda.synchronize()
    cp = mp.to_c()
    assert chain.lib.dqmc_local_updates_noalloc(ctypes.byref(cp), ptr(G), ptr(f), slice1, ptr(d), ptr(u), ptr(acc),
                                                ptr(act), None) == 0
    want = G.cpu().numpy().view(np.complex128).reshape((n, n), order="F")
    assert np.array_equal(got, acc.cpu().numpy().astype(bool))
    if g > 1.0:
        assert got[site] and abs(det[site]) > 1e-10 * g ** 4
    # 64 roundings of entries up to g in the block's rows and columns, as in test_rank4_updates
    assert np.abs(chain.greens - want).max() <= 64 * 16 * 2.0 ** -53 * max(1.0, g)
    chain.close()
