"""Small vertices of up to four neighbours, whose lanes gather their own labels in the separate
kernel: every mix of degrees around four within a tile, ties of two and more, tiles at the list's
end, whole graphs, a frontier and out-of-core batches, against the oracle."""
import numpy as np
import pytest

import galp_gb300
import oracle
from galp_gb300 import tools

pytestmark = pytest.mark.gpu


def _graph(degs, pool, seed):
    rng = np.random.default_rng(seed)
    off = np.concatenate([[0], np.cumsum(degs)]).astype(np.int64)
    return galp_gb300.Graph(off, rng.integers(0, min(pool, len(degs)), off[-1]).astype(np.int32))


@pytest.mark.parametrize("top", [0, 1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 1000, 40_000])
def test_degrees(n, top):
    rng = np.random.default_rng(n + top)
    for pool in (3, n):  # few labels, or mostly different ones
        g = _graph(rng.integers(0, top + 1, n), pool, top)
        with galp_gb300.Propagator(g, early_exit=0) as p:
            tools.profile(p, 1)  # the separate kernels
            for k in (1, 4):
                p.run(k)
                _, want, counts = oracle.run_par(g.offsets, g.neighbors, k, early_exit=False)
                assert np.array_equal(p.get_labels(), want) and p.updates == list(counts)


@pytest.mark.parametrize("policy", [1, 2])
def test_out_of_core(policy):
    g = _graph(np.random.default_rng(7).integers(0, 5, 50_000), 50_000, 8)
    with galp_gb300.Propagator(g, policy=policy, buffer_pow=12, early_exit=0) as p:
        p.run(4)
        _, want, counts = oracle.run_par(g.offsets, g.neighbors, 4, policy=policy, buffer_pow=12, early_exit=False)
        assert np.array_equal(p.get_labels(), want) and p.updates == list(counts)


def test_frontier():
    rng = np.random.default_rng(3)
    n = 30_000
    a, b = rng.integers(0, n, 40_000), rng.integers(0, n, 40_000)
    key = np.unique(np.concatenate([a * n + b, b * n + a])[np.tile(a != b, 2)])
    off = np.zeros(n + 1, np.int64)
    np.add.at(off, key // n + 1, 1)
    g = galp_gb300.Graph(np.cumsum(off), (key % n).astype(np.int32))
    with galp_gb300.Propagator(g, frontier=1, early_exit=0) as p:
        assert tools.schedule_info(p).flags & tools.SchedInfo.FRONTIER
        tools.set_variant(p, frontier_frac=1.0)
        for k in (2, 9):
            p.run(k)
            _, want, counts = oracle.run_par(g.offsets, g.neighbors, k, early_exit=False)
            assert np.array_equal(p.get_labels(), want) and p.updates == list(counts)
