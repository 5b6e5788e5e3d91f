"""The cluster LU panels and the trailing update (dqmc_gb300/csrc/k_lu.cu)
through calculate_greens of given UDTs, at the edges of their ranges: one panel
narrower than LU_PB, one full panel, ragged last panels, the largest lattice of
the unblocked form and the smallest of the blocked one, on clusters of 16 and 8
CTAs, against numpy in 64 bits."""
import numpy as np
import pytest


def _udt(n, rng, top):
    q = lambda: np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))[0]
    t = np.triu(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)), 1) / np.sqrt(n) + np.eye(n)
    return q(), np.logspace(top, -top, n), t[:, rng.permutation(n)]


def _greens(Ul, Dl, Tl, Ur, Dr, Tr):
    lp, lm, rp, rm = np.maximum(Dl, 1), np.minimum(Dl, 1), np.maximum(Dr, 1), np.minimum(Dr, 1)
    X = (Ul.conj().T @ Ur) / lp[:, None] / rp[None, :] + lm[:, None] * (Tl @ Tr.conj().T) * rm[None, :]
    G = (Ur / rp[None, :]) @ np.linalg.solve(X, Ul.conj().T / lp[:, None])
    return G, -(np.linalg.slogdet(X)[1] + np.log(lp).sum() + np.log(rp).sum()), np.linalg.cond(X)


@pytest.mark.gpu
@pytest.mark.parametrize("L", [2, 4, 6, 8, 12, 14])
@pytest.mark.parametrize("cluster", [0, 8])
def test_greens_of_udts(L, cluster, monkeypatch):
    from dqmc_gb300 import api
    monkeypatch.setenv("DQMC_TUNE", f"lu_cluster={cluster}")
    chain = api.DQMC(api.ModelParams(L=L, slices=10, safe_mult=10))
    n = 4 * L * L
    rng = np.random.default_rng(L)
    udts = _udt(n, rng, 3.0) + _udt(n, rng, 2.0)
    G, ld = chain.calculate_greens_udt(*udts)
    want, ldw, cond = _greens(*udts)
    # backward-stable solves on both sides: a few n eps times the condition number
    tol = 8 * n * 2.3e-16 * cond
    assert np.max(np.abs(G - want)) < tol * max(1.0, np.max(np.abs(want)))
    assert abs(ld - ldw) < tol * n
    chain.close()


@pytest.mark.gpu
@pytest.mark.parametrize("L", [4, 6, 14])
def test_nan_leaves_the_chain_usable(L):
    # a NaN is no pivot: it travels to the result, and the next call is as ever
    from dqmc_gb300 import api
    chain = api.DQMC(api.ModelParams(L=L, slices=10, safe_mult=10))
    n = 4 * L * L
    rng = np.random.default_rng(L)
    udts = _udt(n, rng, 3.0) + _udt(n, rng, 2.0)
    good, _ = chain.calculate_greens_udt(*udts)
    for fill in (np.nan, -np.nan):
        bad = [x.copy() for x in udts]
        bad[0][:, n // 2] = fill
        try:
            G, _ = chain.calculate_greens_udt(*bad)
            assert np.isnan(G).any()
        except api.DQMCError:
            pass
        again, _ = chain.calculate_greens_udt(*udts)
        assert np.array_equal(again, good)
        A = np.array(udts[0])
        u, d, t = chain.decompose_udt(A)
        A[:, n // 3] = fill
        try:
            u1, d1, t1 = chain.decompose_udt(A)
            assert np.isnan(u1).any() or np.isnan(d1).any() or np.isnan(t1).any()
        except api.DQMCError:
            pass
        for x, y in zip(chain.decompose_udt(np.array(udts[0])), (u, d, t)):
            assert np.array_equal(x, y)
    chain.close()
