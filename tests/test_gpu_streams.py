"""Hubs, CTA tables and sorted vertices of one scope on streams of their own: every combination of
the three groups, whole graphs and out-of-core batches, repeated and concurrent runs, against the
oracle and against the same kernels on one stream (profiling on)."""
import threading

import numpy as np
import pytest

import galp_gb300
import oracle
from galp_gb300 import tools

pytestmark = pytest.mark.gpu


def _graph(small, groups, ctas, hubs, seed):
    rng = np.random.default_rng(seed)
    degs = rng.permutation(np.concatenate([rng.integers(0, 33, small), rng.integers(33, 1025, groups),
                                           rng.integers(1025, 12289, ctas), rng.integers(12289, 20000, hubs)]))
    n = len(degs)
    off = np.zeros(n + 1, np.int64)
    off[1:] = np.cumsum(degs)
    nbr = rng.integers(0, n, off[-1], dtype=np.int64) % max(n // 3, 1)  # ties and repeats
    return galp_gb300.Graph(off, nbr.astype(np.int32))


MIXES = [(4000, 300, 20, 3), (4000, 0, 0, 2), (0, 200, 0, 3), (0, 0, 9, 4), (0, 0, 0, 5), (4000, 300, 20, 1)]


@pytest.mark.parametrize("mix", MIXES)
def test_groups(mix):
    g = _graph(*mix, seed=sum(mix))
    it, want, counts = oracle.run_par(g.offsets, g.neighbors, 5, early_exit=False)
    with galp_gb300.Propagator(g, early_exit=0) as p:
        for prof in (0, 1, 0, 0):
            tools.profile(p, prof)
            p.run(5)
            assert np.array_equal(p.get_labels(), want) and list(p.updates) == list(counts)


@pytest.mark.parametrize("policy", [1, 2])
def test_batches(policy):
    g = _graph(4000, 300, 20, 3, seed=9)
    res = []
    for prof in (1, 0, 0):
        with galp_gb300.Propagator(g, policy=policy, buffer_pow=16, early_exit=0) as p:
            tools.profile(p, prof)
            p.run(4)
            res.append((p.get_labels().copy(), list(p.updates)))
    for lab, upd in res[1:]:
        assert np.array_equal(lab, res[0][0]) and upd == res[0][1]


def test_threads():
    g = _graph(4000, 300, 20, 3, seed=11)
    _, want, _ = oracle.run_par(g.offsets, g.neighbors, 6, early_exit=False)
    got = [None] * 4

    def work(i):
        with galp_gb300.Propagator(g, early_exit=0) as p:
            for _ in range(5):
                p.run(6)
            got[i] = p.get_labels().copy()

    th = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert all(x is not None and np.array_equal(x, want) for x in got)
