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


@pytest.mark.gpu
@pytest.mark.parametrize("call", ["dqmc_local_updates", "dqmc_update"])
def test_local_updates_return_the_ratios_beside_the_error(call):
    """A ratio that is not finite is an error; the per-site outputs say where it is."""
    from dqmc_gb300 import api
    chain = api.DQMC(api.ModelParams(L=4, slices=20, safe_mult=20), np.random.default_rng(1).uniform(-1, 1, (3, 16, 20)))
    chain.init()
    G = np.array(chain.greens)
    G[9, 9] = np.nan
    chain.greens = G
    delta, unif = np.zeros((3, 16), order="F"), np.full(16, 2.0)   # no acceptance: the NaN stays at its site
    acc, det, pac = np.full(16, 7, np.uint8), np.full(16, 7.0 + 0j), np.full(16, 7.0)
    D = lambda a: a.ctypes.data_as(api._D)
    rate = ctypes.c_double(-1.0)
    rc = getattr(chain.lib, call)(chain.h, D(delta), D(unif), acc.ctypes.data_as(ctypes.c_void_p), D(det), D(pac),
                                  ctypes.byref(rate))
    assert rc != 0
    assert not (acc == 7).any() and not (det == 7.0).any() and not (pac == 7.0).any()
    assert np.isnan(det[9]) and (call == "dqmc_update" or np.isfinite(np.delete(det, 9)).all())
    chain.close()
