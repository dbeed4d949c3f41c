"""The served stream's client (starlab_b200/stream.py) on fake servers: a
latency counts from the call's arrival, whatever held its submission back, and
only a server with a request ring holds calls back (no GPU)."""
import threading
import time

import numpy as np

from starlab_b200.stream import run_served

SERVE = 0.02


class Fake:
    """Serves one call at a time; every call takes SERVE seconds."""

    def __init__(self):
        self.mu, self.busy = threading.Lock(), threading.Lock()
        self.flying = self.most = 0
        self.sent = []

    def open_cluster(self, n, eps2):
        return 0

    def set_j(self, *a):
        pass

    def submit(self, *a):
        with self.mu:
            self.flying += 1
            self.most = max(self.most, self.flying)
            self.sent.append(time.perf_counter())
            return len(self.sent) - 1

    def wait(self, rid):
        with self.busy:
            time.sleep(SERVE)
        with self.mu:
            self.flying -= 1
        return None, None, None, None, time.perf_counter() - self.sent[rid]


class Ringed(Fake):
    ring_calls = 2


def stream(n):
    z = np.zeros((3, 3))
    return [(np.ones(3), z, z, z, z)], [(0.0, 0, 1, 0, 1e-6)] * n


def test_latency_counts_from_arrival_when_the_ring_holds_calls_back():
    srv = Ringed()
    lat, wall, inter = run_served(srv, *stream(10))
    assert srv.most <= Ringed.ring_calls
    assert inter == 30 and len(lat) == 10
    # all ten arrive at once and are served in turn: the last one has waited
    # for all (from its submission it would be three calls at the most)
    assert max(lat) >= 9.5 * SERVE and max(lat) <= wall + 1e-3
    assert np.all(np.sort(lat) >= (np.arange(10) + 0.9) * SERVE)


def test_a_server_without_a_ring_gets_every_call_when_it_is_due():
    srv = Fake()
    lat, _, _ = run_served(srv, *stream(10))
    assert srv.most >= 8 and srv.sent[-1] - srv.sent[0] < 5 * SERVE
    assert max(lat) >= 9.5 * SERVE
