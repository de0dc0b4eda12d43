"""Counting of 33 to 1024 neighbours by groups of lanes (sorted in registers): the edges of
the groups and of the labels per lane, runs that span lanes, ties of every kind, lists that
leave a warp's last tile partly filled, and spills carried over between variant rows."""
import numpy as np
import pytest

import galp_gb300
import oracle
from galp_gb300 import tools

pytestmark = pytest.mark.gpu


def _graph(degs, pool, seed):
    """Vertex v draws degs[v] neighbours (repeats allowed, unsorted) from `pool` vertices
    spread over the graph."""
    rng = np.random.default_rng(seed)
    n = len(degs)
    off = np.zeros(n + 1, np.int64)
    off[1:] = np.cumsum(degs)
    ids = rng.choice(n, size=min(pool, n), replace=False)
    nbr = rng.choice(ids, size=int(off[-1])).astype(np.int32)
    return galp_gb300.Graph(off, nbr)


def _check(g, niter=3, **opts):
    with galp_gb300.Propagator(g, early_exit=0, **opts) as p:
        tools.profile(p, 1)  # the separate kernels, whatever the size
        for k in range(1, niter + 1):
            p.run(k)
            got = p.get_labels()
            _, want, counts = oracle.run_par(g.offsets, g.neighbors, k, early_exit=False)
            assert np.array_equal(got, want), f"run({k}): {np.count_nonzero(got != want)} labels differ"
            assert list(p.updates) == list(counts)


EDGES = sorted({d for G in (2, 4, 8, 16, 32) for N in (20, 24, 32) for d in (G * N, G * N + 1)} |
               {33, 48, 1023})


@pytest.mark.parametrize("deg", EDGES)
@pytest.mark.parametrize("pool", [3, 300, 5000])
def test_uniform_degree(deg, pool):
    # pool 3: runs over many lanes; 300: ties of several labels; 5000: mostly distinct
    n = max(40, 60000 // deg)
    _check(_graph(np.full(n, deg), pool, deg * 7 + pool))


@pytest.mark.parametrize("n", [1, 2, 17, 33, 500, 3000])
def test_mixed_degrees(n):
    rng = np.random.default_rng(n)
    degs = np.exp(rng.uniform(np.log(20), np.log(2500), n)).astype(np.int64)
    _check(_graph(degs, 4 + n, n + 1))


def test_one_label_everywhere():
    # a group whose labels are one run from its first lane to its last
    for deg in (33, 100, 1024):
        off = np.arange(201, dtype=np.int64) * deg
        _check(galp_gb300.Graph(off, np.full(200 * deg, 7, np.int32)))


def test_frontier_keeps_sorted_spills():
    # the frontier keeps the spilled runs (in label order) of vertices none of whose neighbours
    # changed, and resolves them again at other run bases
    g = galp_gb300.generate_rmat(15, 16, seed=11)
    assert ((g.degrees() > 1024) & (g.degrees() <= 2048)).any()
    for rows in ((3, 1), (1, 3)):
        with galp_gb300.Propagator(g, frontier=1, early_exit=0) as p:
            for row in rows:
                tools.dispatch_set(p, 2, row)
                p.run(8)
                _, want, counts = oracle.run(g.offsets, g.neighbors, 8, early_exit=False)
                assert np.array_equal(p.get_labels(), want) and list(p.updates) == list(counts)
