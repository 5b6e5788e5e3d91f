"""Depths below 8: windows of 2 k sites that end after k acceptances
(k_local_window), from all accepted to hardly any, with follower clusters and
without, against the oracle."""
import pytest

from test_window_updates import P, _run


@pytest.mark.gpu
@pytest.mark.parametrize("delay", [2, 3, 5, 7])
@pytest.mark.parametrize("inflight", [0, 16])
@pytest.mark.parametrize("unif", [-1.0, None, 1e6])
def test_rounds_end_after_k_acceptances(delay, inflight, unif):
    got = _run(P, delay, inflight, unif=unif)
    assert unif != -1.0 or got == 1.0


def test_flush_model():
    """The bench's count of flushes with work: k = 2 takes windows of 4 sites up to 2 acceptances."""
    from bench import real_flush_count
    a = [1, 1, 0, 0, 0, 1, 0, 1, 0, 0, 0, 0]
    # sites 0-1 | 2-5 (one acceptance) | 6-9 (one) | 10-11 (none)
    assert real_flush_count(a, 1, 12, 2) == 3
    assert real_flush_count(a * 2, 2, 12, 16) == 2 and real_flush_count([0] * 12, 1, 12, 2) == 0
