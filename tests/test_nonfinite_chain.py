"""A chain whose G is not finite: the calls report it wherever their arrays lie."""
import ctypes

import numpy as np
import pytest


def nonfinite_chain(api):
    p = api.ModelParams(L=4, slices=20, safe_mult=10)
    chain = api.DQMC(p, np.random.default_rng(1).uniform(-1, 1, (3, 16, 20)))
    chain.init()
    chain.greens = np.full((64, 64), np.nan + 0j)
    with pytest.raises(api.DQMCError) as e:
        for _ in range(40):   # until a stabilisation compares G with the fresh one
            chain.propagate()
    return chain, e.value.code


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["host", "device"])
def test_equal_time_correlators_report_it(where):
    torch = pytest.importorskip("torch")
    from dqmc_gb300 import api
    chain, code = nonfinite_chain(api)
    N = 16
    if where == "host":
        out = [np.zeros(N), np.zeros(N), np.zeros(2 * N), np.zeros(2 * N)]
        ptr = [x.ctypes.data for x in out]
    else:
        out = [torch.zeros(k * N, dtype=torch.float64).cuda() for k in (1, 1, 2, 2)]
        ptr = [x.data_ptr() for x in out]
        torch.cuda.synchronize()
    rc = chain.lib.dqmc_measure_equal_time(chain.h, None, *[ctypes.cast(p, api._D) for p in ptr],
                                           1 if where == "device" else 0)
    assert rc == code
    chain.close()
