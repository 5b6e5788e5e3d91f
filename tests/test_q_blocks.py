"""U of the UDT decomposition in the FP64 form against the block size of its
formation (DQMC_TUNE wy=): the setting counts for every n, and since the 63-bit
products leave no error in U, its results agree within the rounding of U's own
columns."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("L", [4, 6, 10, 14])
def test_block_sizes_agree(L, monkeypatch):
    from dqmc_gb300 import api
    n = 4 * L * L
    rng = np.random.default_rng(n)
    A = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) * 10.0 ** -np.linspace(0, 8, n)
    U, launches = {}, {}
    for b in (16, 64, 128):
        monkeypatch.setenv("DQMC_TUNE", f"wy={b}")
        chain = api.DQMC(api.ModelParams(L=L, slices=10, safe_mult=10))
        chain.reset_timing(True)
        U[b] = chain.decompose_udt(A)[0]
        launches[b] = chain.timing()["kinds"]["apply_q"]["launches"]
        chain.close()
        assert np.linalg.norm(U[b].conj().T @ U[b] - np.eye(n)) <= 4.0 * n * 2.0 ** -53
    assert launches[16] > launches[64] and (n <= 64 or launches[64] > launches[128])
    # the same reflectors: n / 16 block steps of one rounding per entry (2^-53 times the column), both sides
    for b in (16, 64):
        assert np.linalg.norm(U[b] - U[128], axis=0).max() <= 2.0 * np.sqrt(n / 16 + 4) * 2.0 ** -53 * 4
