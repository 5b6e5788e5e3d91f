"""G of chains in flight against G from scratch, right after stabilisations: the
LU panels' clusters share SMs with the other chains' kernels, so their warps run
far apart, which a chain alone on the GPU does not show."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("cluster", [0, 8])
def test_chains_in_flight_agree_with_scratch(cluster, monkeypatch):
    import torch
    from dqmc_gb300 import api
    monkeypatch.setenv("DQMC_TUNE", f"lu_cluster={cluster}")
    Ls = [6, 8, 10, 12] * 4
    M, s = 20, 10
    rng = np.random.default_rng(7)
    b = api.Batch([api.ModelParams(L=L, slices=M, safe_mult=s, precision="mixed", delay=16) for L in Ls],
                  [rng.uniform(-1, 1, (3, L * L, M)) for L in Ls])
    b.init()
    for calls in (9, 1) * 8:
        d = [torch.from_numpy(rng.uniform(-0.2, 0.2, (calls, L * L, 3))).cuda() for L in Ls]
        u = [torch.from_numpy(rng.uniform(size=(calls, L * L))).cuda() for L in Ls]
        b.sweep_device(calls, [x.data_ptr() for x in d], [x.data_ptr() for x in u])
        for c in b.chains:
            G = np.array(c.greens)
            scratch, _ = c.calc_greens_and_logdet(c.state[0])
            # the mixed form's stabilisation and s wraps: 1e-9 at the largest of these lattices
            assert np.max(np.abs(G - scratch)) < 1e-7
