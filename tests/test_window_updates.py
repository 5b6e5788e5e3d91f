"""Windowed local updates (k_local_window, k_local_factors) at the edges of
their ranges against the oracle: windows shorter than a cluster, ragged last
windows, several sites per CTA, depths above the largest window, chains capped
to 8-CTA clusters, and all-accepted or all-rejected windows."""
import dataclasses

import numpy as np
import pytest

from oracle import dqmc_ref as R

P = R.Params(L=6, slices=10, delta_tau=0.1, safe_mult=5, lambda_=1.0, r=1.0, c=1.0, u=1.0, mu1=-0.5, mu2=-0.5,
             box=0.2)


def _run(p, delay, inflight, unif=None, precision="fp64"):
    from dqmc_gb300 import api
    calls = 3
    phi = R.synthetic_field(p.N, p.slices, 50 + p.L)
    delta, u = R.synthetic_streams(p.N, calls, p.box, 60 + delay)
    if unif is not None:
        u = np.full_like(u, unif)
    ref = R.DQMCRef(p, phi)
    ref.init()
    rec = []
    ref.sweep(calls, delta, u, record=rec)
    gpu = api.DQMC(api.ModelParams(L=p.L, slices=p.slices, safe_mult=p.safe_mult, delay=delay, inflight=inflight,
                                   precision=precision), phi)
    gpu.init()
    res = gpu.sweep(calls, delta, u, return_accepted=True)
    acc = np.array([r[2] for r in rec]).reshape(calls, p.N)
    tol = 1e-10 if precision == "fp64" else 1e-8
    assert np.array_equal(res["accepted_mask"], acc)
    assert np.array_equal(gpu.get_field(), ref.phi)
    assert np.max(np.abs(gpu.greens - ref.greens)) < tol * max(1.0, np.max(np.abs(ref.greens)))
    assert abs(gpu.boson_action - ref.boson_action_value) < 1e-10 * abs(ref.boson_action_value)
    gpu.close()
    return acc.mean()


@pytest.mark.gpu
@pytest.mark.parametrize("delay", [0, 2, 3, 8, 17, 31, 32, 64])
@pytest.mark.parametrize("inflight", [0, 16])
def test_depths_and_cluster_sizes(delay, inflight):
    _run(P, delay, inflight)


@pytest.mark.gpu
@pytest.mark.parametrize("L", [2, 4, 8])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_lattices(L, precision):
    _run(dataclasses.replace(P, L=L), 16, 0, precision=precision)


@pytest.mark.gpu
@pytest.mark.parametrize("unif,rate", [(-1.0, 1.0), (1e6, None)])
def test_full_and_nearly_empty_windows(unif, rate):
    """A uniform below every probability accepts all sites; one above all
    accepts only those with p > 1."""
    got = _run(P, 16, 0, unif=unif)
    assert rate is None or got == rate


@pytest.mark.gpu
@pytest.mark.parametrize("L,delay", [(8, 16), (10, 3), (12, 16), (14, 40), (16, 16)])
def test_factors_beside_the_window(L, delay):
    """Follower clusters of 8 and 16 vectors per CTA, ragged last CTAs among
    them, against the factors as a launch of their own (chains in flight): the
    sums are the same up to the split over lanes, 4 p terms of FP64 rounding per
    window and at most 2 N / 16 windows."""
    from dqmc_gb300 import api
    calls = 2
    phi = R.synthetic_field(L * L, 10, 70 + L)
    delta, u = R.synthetic_streams(L * L, calls, 0.2, 80 + L)
    got = []
    for inflight in (0, 8):
        c = api.DQMC(api.ModelParams(L=L, slices=10, safe_mult=10, delay=delay, inflight=inflight), phi)
        c.init()
        res = c.sweep(calls, delta, u, return_accepted=True)
        got.append((res["accepted_mask"], np.array(c.greens), c.get_field()))
        c.close()
    assert np.array_equal(got[0][0], got[1][0])
    assert np.array_equal(got[0][2], got[1][2])
    windows = 2 * calls * (L * L // 16 + 1)
    tol = windows * 4 * 32 * 2.3e-16
    assert np.max(np.abs(got[0][1] - got[1][1])) < tol * max(1.0, np.max(np.abs(got[1][1])))
