"""Small-vertex counting (at most 32 neighbours, sorted in registers) at the edges of its
tiles: lists that end inside a warp or a degree window, every degree from 0 to 32, the
largest degree of each sorting network, and labels that tie two, several or all ways."""
import numpy as np
import pytest

import galp_gb300
import oracle
from galp_gb300 import tools

pytestmark = pytest.mark.gpu


def _graph(degs, pool, seed):
    """Unsorted adjacency: vertex v draws degs[v] neighbours (repeats allowed) from `pool`
    vertices spread over the graph."""
    rng = np.random.default_rng(seed)
    n = len(degs)
    off = np.zeros(n + 1, np.int64)
    off[1:] = np.cumsum(degs)
    ids = rng.choice(n, size=min(pool, n), replace=False)
    return galp_gb300.Graph(off, rng.choice(ids, size=int(off[-1])).astype(np.int32))


def _check(g, niter=4, **opts):
    with galp_gb300.Propagator(g, early_exit=0, **opts) as p:
        tools.profile(p, 1)  # the separate kernels, whatever the size
        for k in range(1, niter + 1):
            p.run(k)
            got = p.get_labels()
            _, want, counts = oracle.run(g.offsets, g.neighbors, k, early_exit=False)
            assert np.array_equal(got, want), f"run({k}): {np.count_nonzero(got != want)} labels differ"
            assert list(p.updates) == list(counts)


@pytest.mark.parametrize("n", [1, 31, 33, 127, 128, 129, 1000, 20011])
def test_every_degree_at_list_ends(n):
    rng = np.random.default_rng(n)
    _check(_graph(rng.integers(0, 33, n), 5 + n // 3, n))


@pytest.mark.parametrize("deg", [1, 4, 5, 8, 9, 12, 16, 17, 20, 24, 25, 28, 29, 31, 32])
@pytest.mark.parametrize("pool", [2, 40, 3000])
def test_uniform_degree(deg, pool):
    # pool 2: long runs (up to the whole list); 40: ties of several labels; 3000: all distinct
    _check(_graph(np.full(3001, deg), pool, deg * 7 + pool))


def test_one_label_everywhere():
    # every list one run: a full row of 32 equal labels
    n = 300
    off = np.arange(n + 1, dtype=np.int64) * 32
    _check(galp_gb300.Graph(off, np.full(32 * n, 7, np.int32)))
