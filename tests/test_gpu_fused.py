"""Runs of small graphs and batches in one kernel: vertices in every counting phase, chunks of
vertices that the blocks resolve at their edges, graphs that span chunks or share one, early
exits, repeated runs, and sizes beyond which the separate kernels run."""
import numpy as np
import pytest

import galp_gb300
import oracle
from galp_gb300 import tools

pytestmark = pytest.mark.gpu


def _graph(degs, pool, seed, ordered=False):
    """Vertex v draws degs[v] neighbours from `pool` vertices spread over the graph; ordered =
    distinct and ascending (the first iteration's closed form)."""
    rng = np.random.default_rng(seed)
    n = len(degs)
    ids = np.sort(rng.choice(n, size=min(pool, n), replace=False))
    if ordered:
        degs = np.minimum(degs, len(ids))
        nbr = [np.sort(rng.choice(ids, size=d, replace=False)) for d in degs]
    else:
        nbr = [rng.choice(ids, size=d) for d in degs]
    off = np.zeros(n + 1, np.int64)
    off[1:] = np.cumsum(degs)
    return galp_gb300.Graph(off, np.concatenate(nbr + [np.zeros(0, np.int64)]).astype(np.int32))


def _launches(p):
    return tools.schedule_info(p).launches


def _check(g, niters=(1, 2, 5), fused=True, **opts):
    with galp_gb300.Propagator(g, **opts) as p:
        for k in niters:
            before = _launches(p)
            p.run(k)
            assert (_launches(p) - before == 1) == fused
            it, want, counts = oracle.run_par(g.offsets, g.neighbors, k, early_exit=opts.get("early_exit", 1) != 0)
            assert p.iters_run == it and list(p.updates) == list(counts)
            assert np.array_equal(p.get_labels(), want)


@pytest.mark.parametrize("ordered", [False, True])
@pytest.mark.parametrize("n", [1, 2, 33, 511, 513, 4864, 30000])
def test_chunk_edges(n, ordered):
    rng = np.random.default_rng(n)
    _check(_graph(rng.integers(0, 40, n), 3 + n // 4, n, ordered), early_exit=0)


@pytest.mark.parametrize("top", [1025, 3000, 6145, 12288])
def test_large_vertices(top):
    # one block each, beside lane groups and small vertices; both block shapes (1 M entries)
    rng = np.random.default_rng(top)
    degs = np.concatenate([rng.integers(0, 33, 4000), rng.integers(33, 1025, 300), rng.integers(1025, top + 1, 30),
                           [top]])
    degs = rng.permutation(degs)
    _check(_graph(degs, 3000, top), early_exit=0)
    _check(_graph(np.tile(degs, 3), 9000, top + 1), niters=(3,), early_exit=0)


def test_early_exit_and_repeats():
    g = galp_gb300.generate_sbm([100] * 30, 14.0, 1.0, seed=4)
    _check(g, niters=(40, 3, 40))


def test_limits():
    g = galp_gb300.generate_sbm([400] * 100, 5.0, 1.0, seed=4)
    _check(g, niters=(2,))
    with galp_gb300.Propagator(g, frontier=1) as p:  # a frontier run keeps the separate kernels
        before = _launches(p)
        p.run(3)
        assert _launches(p) - before > 3
    n = (1 << 21) + 5  # too many vertices
    off = np.arange(n + 1, dtype=np.int64)
    _check(galp_gb300.Graph(off, np.roll(np.arange(n, dtype=np.int32), 1)), niters=(2,), fused=False)


@pytest.mark.parametrize("early_exit", [0, 1])
def test_batches(early_exit):
    rng = np.random.default_rng(7)
    gs = []
    # sizes from empty graphs and single vertices to one that spans many chunks
    for i, n in enumerate([0, 1, 2, 5, 0, 40, 300, 1500, 17, 20000, 3, 129, 0, 900, 2500]):
        kind = i % 3
        if n < 3:
            gs.append(galp_gb300.Graph(np.arange(n + 1, dtype=np.int64) * (n > 1), np.zeros(n * (n > 1), np.int32)))
        elif kind == 0:
            gs.append(_graph(rng.integers(0, 60, n), 2 + n // 3, i))
        else:
            sizes = [max(1, n // 5)] * 5
            gs.append(galp_gb300.generate_sbm(sizes, 10.0, 1.0 + kind, seed=i))
    with galp_gb300.Batch(gs, early_exit=early_exit) as b:
        for k in (1, 4, 30):
            before = _launches(b)
            b.run(k)
            assert _launches(b) - before == 1
            for i, g in enumerate(gs):
                it, want, counts = oracle.run_par(g.offsets, g.neighbors, k, early_exit=bool(early_exit))
                got_it, got = b.graph_stats(i)
                assert np.array_equal(b.labels(i), want), f"graph {i} of {k}"
                if g.n:
                    assert got_it == it and got == list(counts)
