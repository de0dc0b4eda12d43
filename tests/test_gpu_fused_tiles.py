"""One-kernel runs: tiles fixed to a warp (counted by a plan kept in shared memory) and tiles
claimed from the list, lane-group and small tiles of every row length, on both block shapes."""
import numpy as np
import pytest

import galp_gb300
import oracle
from galp_gb300 import tools

pytestmark = pytest.mark.gpu

SMS, NARROW = 152, 16  # resident blocks, warps of the narrow shape
FIXED = SMS * NARROW   # tiles fixed to a warp when no block has a larger vertex


def _check(degs, seed, niter=4, one=True):
    rng = np.random.default_rng(seed)
    n = len(degs)
    off = np.zeros(n + 1, np.int64)
    off[1:] = np.cumsum(degs)
    pool = rng.integers(0, n, max(n // 4, 3), dtype=np.int64)  # ties, repeated labels
    nbr = pool[rng.integers(0, len(pool), off[-1])].astype(np.int32)
    g = galp_gb300.Graph(off, nbr)
    _, want, counts = oracle.run_par(g.offsets, g.neighbors, niter, early_exit=False)
    with galp_gb300.Propagator(g, early_exit=0) as p:
        for _ in range(2):
            before = tools.schedule_info(p).launches
            p.run(niter)
            assert (tools.schedule_info(p).launches - before == 1) == one
            assert np.array_equal(p.get_labels(), want) and list(p.updates) == list(counts)


@pytest.mark.parametrize("extra", [-33, -1, 0, 1, 32, 1000])
def test_fixed_and_claimed(extra):
    # 32 small vertices a tile: just below and above one tile for every warp
    n = FIXED * 32 + extra
    _check(np.random.default_rng(extra + 99).integers(0, 12, n), 105 + extra)


@pytest.mark.parametrize("deg", [1, 4, 5, 16, 17, 31, 32, 33, 40, 41, 48, 49, 64, 160, 161, 192, 193, 256, 640, 641,
                                 768, 769, 1023, 1024])
def test_row_lengths(deg):
    n = 70 if deg > 32 else 131
    _check(np.full(n, deg), deg)
    rng = np.random.default_rng(deg)
    _check(rng.permutation(np.concatenate([np.full(n, deg), rng.integers(0, deg + 1, n)])), deg + 1)


@pytest.mark.parametrize("large", [1, 100, SMS - 1, SMS, 2 * SMS + 5])
def test_few_free_blocks(large):
    rng = np.random.default_rng(large)
    _check(rng.permutation(np.concatenate([rng.integers(1025, 1400, large), rng.integers(33, 200, 500),
                                           rng.integers(0, 33, 9000)])), large)


def test_wide():
    # above 2 M entries: no plans
    rng = np.random.default_rng(3)
    _check(rng.permutation(np.concatenate([rng.integers(1025, 3000, 60), rng.integers(33, 1025, 3000),
                                           rng.integers(0, 33, 60000)])), 3)


@pytest.mark.parametrize("n, deg, one", [(1 << 20, 2, True), ((1 << 20) + 7, 8, True), ((1 << 20) + 7, 7, False),
                                         ((1 << 21) + 1, 9, False)])
def test_size_rule(n, deg, one):
    _check(np.full(n, deg), deg, niter=2, one=one)


@pytest.mark.parametrize("n", [1, 32, 33, 300, 511, 2047, 2048, 2049])  # one cluster up to 64 tiles
def test_cluster(n):
    rng = np.random.default_rng(n)
    _check(rng.integers(0, 20, n), n, niter=9)
    _check(np.concatenate([rng.integers(0, 20, n), rng.integers(33, 1025, 9)]), n + 1, niter=9)


@pytest.mark.parametrize("sizes", [[511] * 152, [513] * 152, [700, 30, 1] * 151 + [5000], [1024] * 152, [1030] * 152,
                                   [1, 60, 4000] * 58, [1700] * 152])
def test_batch_rows(sizes):
    # one, two and three vertices per thread and round, several rounds; graphs that end early
    rng = np.random.default_rng(len(sizes) + sizes[0])
    gs = []
    for i, n in enumerate(sizes):
        deg = rng.integers(0, 9, n) if i % 3 else np.full(n, min(n, 4))
        off = np.zeros(n + 1, np.int64)
        off[1:] = np.cumsum(deg)
        gs.append(galp_gb300.Graph(off, rng.integers(0, max(n // (1 + i % 4), 1), off[-1]).astype(np.int32)))
    with galp_gb300.Batch(gs) as b:
        for k in (1, 6):
            before = tools.schedule_info(b).launches
            b.run(k)
            assert tools.schedule_info(b).launches - before == 1
            for i, g in enumerate(gs):
                it, want, counts = oracle.run_par(g.offsets, g.neighbors, k)
                got_it, got = b.graph_stats(i)
                assert np.array_equal(b.labels(i), want), f"graph {i} of {k}"
                assert got_it == it and got == list(counts)


@pytest.mark.parametrize("n, deg, one", [((1 << 18) // 64, 16, True), ((1 << 18) // 64, 17, False),
                                         ((1 << 18) // 64 + 1, 3, False)])
def test_batch_size_rule(n, deg, one):
    rng = np.random.default_rng(n + deg)
    gs = [galp_gb300.Graph(np.arange(n + 1, dtype=np.int64) * deg, rng.integers(0, n // 2, n * deg).astype(np.int32))
          for _ in range(64)]
    with galp_gb300.Batch(gs, early_exit=0) as b:
        before = tools.schedule_info(b).launches
        b.run(3)
        assert (tools.schedule_info(b).launches - before == 1) == one
        for i, g in enumerate(gs):
            _, want, counts = oracle.run_par(g.offsets, g.neighbors, 3, early_exit=False)
            assert np.array_equal(b.labels(i), want) and b.graph_stats(i)[1] == list(counts)
