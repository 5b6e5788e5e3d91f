"""Local updates at depths 0 and 1: rank-4 updates in 64 bits, whatever the form
of the stabilisation.  The windows of both forms against k_local_updates (one
rank-4 update of all of G per acceptance, in FP64 multiply-adds) through the
allocation-free entry point, which shares no code with them."""
import ctypes

import numpy as np
import pytest

from oracle.dqmc_ref import synthetic_field, synthetic_streams


@pytest.mark.gpu
@pytest.mark.parametrize("precision,bits", [("fp64", 0), ("mixed", 14), ("mixed", 0)])
@pytest.mark.parametrize("delay", [0, 1])
@pytest.mark.parametrize("L", [2, 6, 10, 16])
def test_depths_0_and_1_are_fp64_updates(L, delay, precision, bits):
    torch = pytest.importorskip("torch")
    from dqmc_gb300 import api
    lib = api.load_library()
    M = 10
    mp = api.ModelParams(L=L, slices=M, safe_mult=10, delay=delay, precision=precision, ozaki_bits=bits)
    N, n = mp.N, mp.n
    phi = synthetic_field(N, M, 900 + L)
    start = api.DQMC(api.ModelParams(L=L, slices=M, safe_mult=10), phi)   # an FP64 G to start from
    start.init()
    G0 = np.array(start.greens)
    start.close()
    chain = api.DQMC(mp, phi)
    chain.init()
    chain.greens = G0
    slice1 = chain.current_slice
    delta, unif = synthetic_streams(N, 1, 0.2, 910 + L)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    G = dev(np.asfortranarray(G0).ravel(order="F").view(np.float64))
    f, d, u = dev(chain.get_field().ravel(order="F")), dev(delta[0].ravel(order="F")), dev(unif[0])
    act, acc = dev(np.array([chain.boson_action])), torch.zeros(N, dtype=torch.uint8).cuda()
    _, got, _, _ = chain.local_updates(delta[0], unif[0], return_details=True)
    torch.cuda.synchronize()
    cp = api.ModelParams(L=L, slices=M, safe_mult=10).to_c()
    assert lib.dqmc_local_updates_noalloc(ctypes.byref(cp), ptr(G), ptr(f), slice1, ptr(d), ptr(u), ptr(acc), ptr(act),
                                          None) == 0
    want = G.cpu().numpy().view(np.complex128).reshape((n, n), order="F")
    assert np.array_equal(got, acc.cpu().numpy().astype(bool)) and got.any()
    # per acceptance a rank-4 term of rounding 8 2^-53 on entries of order one, and its effect on the later ones
    tol = 64 * max(16, int(got.sum())) * 2.0 ** -53 * max(1.0, np.abs(want).max())
    assert np.abs(chain.greens - want).max() <= tol, (np.abs(chain.greens - want).max(), tol)
    chain.close()


@pytest.mark.gpu
@pytest.mark.parametrize("delay", [0, 16])
def test_flush_where_the_target_has_no_slices(delay):
    """L = 2: 57 .. 60 bits can be had at K = n = 16, not at the flush's K = 64."""
    from dqmc_gb300 import api
    from oracle import dqmc_ref as R
    p = R.Params(L=2, slices=10, delta_tau=0.1, safe_mult=5, lambda_=1.0, r=1.0, c=1.0, u=1.0, mu1=-0.5, mu2=-0.5,
                 box=0.2)
    phi = R.synthetic_field(4, 10, 5)
    delta, u = R.synthetic_streams(4, 10, 0.2, 6)
    ref = R.DQMCRef(p, phi)
    ref.init()
    rec = []
    ref.sweep(10, delta, u, record=rec)
    for bits in (57, 60):
        c = api.DQMC(api.ModelParams(L=2, slices=10, safe_mult=5, precision="mixed", ozaki_bits=bits, delay=delay), phi)
        c.init()
        res = c.sweep(10, delta, u, return_accepted=True)
        assert np.array_equal(res["accepted_mask"], np.array([r[2] for r in rec]).reshape(10, 4))
        assert np.abs(c.greens - ref.greens).max() < 1e-10 * max(1.0, np.abs(ref.greens).max())
        c.close()
