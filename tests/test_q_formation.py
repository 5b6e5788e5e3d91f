"""U of the pivoted UDT decomposition in the FP64 form: formed in blocks of
reflectors by the split products, it may be no further from orthonormal than
reflectors applied one by one in FP64, whose error is about n^(1/2) u per column
(u = 2^-53, complex: twice that), and U D T has to give A back."""
import numpy as np
import pytest

from dqmc_gb300 import api

U53 = 2.0 ** -53


@pytest.mark.gpu
@pytest.mark.parametrize("L", [4, 6, 8, 10])   # one block of 32 and a remainder rule each side of n = 144
@pytest.mark.parametrize("zero_columns", [0, 3])   # reflectors with tau = 0
def test_u_orthonormal(L, zero_columns):
    n = 4 * L * L
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) * np.logspace(5, -5, n)[rng.permutation(n)]
    if zero_columns:
        # unit columns are pivoted first and leave reflectors without a tail
        A[:zero_columns, :] = 0.0
        A[:, :zero_columns] = 0.0
        A[np.arange(zero_columns), np.arange(zero_columns)] = 1e9
    p = api.ModelParams(L=L, slices=10, precision="fp64")
    mc = api.DQMC(p, rng.uniform(-1, 1, (3, p.N, 10)))
    U, D, T = mc.decompose_udt(A)
    eye = U.conj().T @ U - np.eye(n)
    assert np.linalg.norm(eye) / np.sqrt(n) <= 4.0 * np.sqrt(n) * U53
    back = (U * D[None, :]) @ T
    # per column: the error of A's column is bounded by n u times its norm
    err = np.linalg.norm(back - A, axis=0)
    assert np.all(err <= 8.0 * n * U53 * np.linalg.norm(A, axis=0))
