"""The arrival counters of a window launch with follower clusters
(k_local_window, k_local_prepare), restated: clusters draw a ticket, ticket 0
decides the window, the others arrive once they have read the state, and the
window advances the state when all have.  Where a follower comes too late for
the bounded wait, the counters must not let a later launch decide a window
before its followers have read the state, or decide one twice."""
import itertools

import pytest

FOLLOWERS = 3


class Device:
    def __init__(self):
        self.arrive = [0, 0]   # followers that have read the state, clusters started
        self.state = 0         # next site; a window is 16 sites
        self.err = False
        self.decided = []      # windows decided, by their first site

    def prepare(self):
        self.arrive = [0, 0]
        self.state = 0

    def launch(self, order, late):
        """order: the clusters as they start; late: those that start after the window has given up waiting."""
        first = self.state     # what a cluster reads when it starts
        window = None
        read = []

        def start():
            nonlocal window
            ticket = self.arrive[1]
            self.arrive[1] += 1
            if self.err:
                return
            if ticket == 0:
                window = self.state
            else:
                read.append(self.state)
                self.arrive[0] += 1

        for c in order:
            if c not in late:
                start()
        if window is not None:
            self.decided.append(window)
            if self.err or self.arrive[0] != FOLLOWERS:
                self.err = True        # counters and state stay
            else:
                self.arrive = [0, 0]
                self.state = window + 16
        elif not self.err:
            self.err = True            # followers without a window give up
        for c in order:
            if c in late:
                start()
        assert all(r == first for r in read), "a follower read the state of another window"


def slice_of(dev, late_in_first=()):
    dev.prepare()
    for rnd in range(4):
        dev.launch(range(FOLLOWERS + 1), late_in_first if rnd == 0 else ())


def test_all_in_time():
    dev = Device()
    slice_of(dev)
    assert dev.decided == [0, 16, 32, 48] and not dev.err


@pytest.mark.parametrize("late", [c for k in (1, 2, 3) for c in itertools.combinations(range(FOLLOWERS + 1), k)])
def test_late_followers(late):
    dev = Device()
    slice_of(dev, late)
    # the window that timed out is the only one of its slice, and reported
    assert dev.err and dev.decided in ([], [0])
    # the next call (the host has taken the error) starts clean
    dev.err, dev.decided = False, []
    slice_of(dev)
    assert dev.decided == [0, 16, 32, 48] and not dev.err
