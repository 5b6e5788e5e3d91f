"""The column-pivoted QR (k_qr_cols and its hand-over from k_qrp,
dqmc_gb300/csrc/k_linalg.cu) through decompose_udt: the smallest lattice, part
filled last groups of rows, the largest that is held entirely, and the two that
start in k_qrp; graded columns force norm recomputations, equal columns force ties,
a rank-one matrix forces zero norms.  Chains in flight take k_qrp for all steps
where the held columns are too few, with the same bits."""
import numpy as np
import pytest


def _matrix(kind, n, rng):
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    if kind == "graded":
        a = a * np.logspace(5, -5, n)[rng.permutation(n)][None, :]
    elif kind == "dependent":   # columns that lose all but 1e-9 of their norm to others
        h = n // 2
        a[:, h:2 * h] = a[:, :h] @ (rng.standard_normal((h, h)) / np.sqrt(h)) + 1e-9 * a[:, h:2 * h]
    elif kind == "equal norms":
        a = np.linalg.qr(a)[0]
    return a


@pytest.mark.gpu
@pytest.mark.parametrize("L", [2, 4, 6, 8, 10, 12, 14, 16])
@pytest.mark.parametrize("kind", ["graded", "dependent", "equal norms"])
def test_decomposition(L, kind):
    from dqmc_gb300 import api
    n = 4 * L * L
    A = _matrix(kind, n, np.random.default_rng(L))
    got = []
    for inflight in (0, 16):
        chain = api.DQMC(api.ModelParams(L=L, slices=10, safe_mult=10, inflight=inflight))
        got.append(chain.decompose_udt(A))
        chain.close()
    U, D, T = got[0]
    for x, y in zip(*got):
        assert np.array_equal(x, y)
    # Householder QR: columns backward stable to a few n eps, Q orthogonal to the same
    tol = 16 * n * 2.3e-16
    assert np.max(np.abs(U.conj().T @ U - np.eye(n))) < tol
    assert np.all(np.linalg.norm((U * D[None, :]) @ T - A, axis=0) < tol * np.linalg.norm(A, axis=0))
    # pivoting: no later column is longer than the pivot at its step
    R = D[:, None] * T
    order = np.argsort(np.count_nonzero(np.abs(T) > 0, axis=0), kind="stable")
    R = R[:, order]
    tails = np.sqrt(np.cumsum((np.abs(R) ** 2)[::-1], axis=0)[::-1])
    assert np.all(np.triu(tails, 1).max(axis=1) <= D * (1 + 1e-6))
