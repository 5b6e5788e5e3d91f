"""Slice matrices on both kernels of dqmc_gb300/csrc/k_slice.cu (a thread per
output component up to n = 144, a thread per block above and for B^dag M) against
the oracle, over every mode of multiply_B_*."""
import numpy as np
import pytest

from oracle import dqmc_ref as R


@pytest.mark.gpu
@pytest.mark.parametrize("L", [2, 4, 6, 8])
def test_slice_modes(L):
    from dqmc_gb300 import api
    p = R.Params(L=L, slices=10, delta_tau=0.1, safe_mult=5, lambda_=1.0, r=1.0, c=1.0, u=1.0, mu1=-0.5, mu2=-0.5,
                 box=0.2)
    phi = R.synthetic_field(p.N, p.slices, 90 + L)
    ref = R.DQMCRef(p, phi)
    chain = api.DQMC(api.ModelParams(L=L, slices=10, safe_mult=5), phi)
    rng = np.random.default_rng(L)
    A = rng.standard_normal((p.n, p.n)) + 1j * rng.standard_normal((p.n, p.n))
    # four sparse factors of at most 4 terms per entry: 20 roundings, amplified by
    # the factors' norms (below 3 each side)
    for sl in (1, 7, 10):
        for name in ("multiply_B_left", "multiply_B_right", "multiply_B_inv_left", "multiply_B_inv_right",
                     "multiply_daggered_B_left"):
            want = getattr(ref, name)(sl, A.copy())
            assert np.max(np.abs(getattr(chain, name)(sl, A) - want)) < 60 * 2.3e-16 * np.max(np.abs(want)), (sl, name)
    # a round trip through B and its inverse, left and right
    for fwd, back in (("multiply_B_left", "multiply_B_inv_left"), ("multiply_B_right", "multiply_B_inv_right")):
        got = getattr(chain, back)(3, getattr(chain, fwd)(3, A))
        assert np.max(np.abs(got - A)) < 400 * 2.3e-16 * np.max(np.abs(A))
    chain.close()
