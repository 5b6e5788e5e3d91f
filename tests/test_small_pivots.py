"""Pivots whose squared modulus leaves the range of double: the blocked LU
(n > 576) reports them as singular, the unblocked one divides by them."""
import numpy as np
import pytest


def greens(L, scale):
    """G of D = scale on the left, 1 / scale on the right: the separated matrix is
    (1 + Tl Tr^dag) / scale with 1 + Tl Tr^dag = 1 + 4."""
    from dqmc_gb300 import api
    n = 4 * L * L
    chain = api.DQMC(api.ModelParams(L=L, slices=10, safe_mult=10))
    one = np.eye(n) + 0j
    try:
        return chain.calculate_greens_udt(one, np.full(n, scale), 2 * one, one, np.full(n, 1.0 / scale), 2 * one)[0]
    finally:
        chain.close()


@pytest.mark.gpu
@pytest.mark.parametrize("L", [4, 14])
def test_moderate_scales(L):
    G = greens(L, 2.0 ** 300)
    assert np.allclose(G, np.eye(len(G)) / 5, rtol=1e-13, atol=1e-300)


@pytest.mark.gpu
def test_blocked_lu_reports_a_pivot_without_reciprocal():
    from dqmc_gb300 import api
    with pytest.raises(api.DQMCError, match="[Ss]ingular"):
        greens(14, 2.0 ** 600)


@pytest.mark.gpu
def test_unblocked_lu_divides_by_it():
    G = greens(4, 2.0 ** 600)
    assert np.allclose(G, np.eye(64) / 5, rtol=1e-13, atol=1e-300)
