"""Batches above the one-kernel limits: the captured graph of a run follows what was set since."""
import numpy as np
import pytest

import galp_gb300
import oracle
from galp_gb300 import tools

pytestmark = pytest.mark.gpu


def _batch(count=4100):
    """More graphs than one kernel takes, with vertices in every counting range."""
    rng = np.random.default_rng(count)
    gs = [galp_gb300.generate_sbm([8] * 4, 5.0, 1.0, seed=i) for i in range(40)]
    big = rng.permutation(np.concatenate([rng.integers(1025, 3000, 12), rng.integers(33, 1025, 60),
                                          rng.integers(1, 33, 4000)]))
    off = np.zeros(len(big) + 1, np.int64)
    off[1:] = np.cumsum(big)
    gs.append(galp_gb300.Graph(off, rng.integers(0, len(big), off[-1]).astype(np.int32)))
    return [gs[i % 40] for i in range(count - 1)] + gs[40:]


def _rows(b):
    return [int(x) for x in tools.dispatch_log(b)[1] if x >= 0]


def test_a_new_dispatch_mode_is_captured_again():
    with galp_gb300.Batch(_batch(), early_exit=0) as b:
        b.run(4)
        want = b.all_labels()
        assert set(_rows(b)) == {0}
        for row in (2, 8, 10, 0):
            tools.dispatch_set(b, 2, row)
            b.run(4)
            assert set(_rows(b)) == {row} and np.array_equal(b.all_labels(), want)
        tools.dispatch_set(b, 2, 8)
        b.run(4)
        tools.dispatch_set(b, 0)
        b.run(4)
        assert set(_rows(b)) == {0} and np.array_equal(b.all_labels(), want)


def test_a_small_batch_follows_its_dispatch_mode():
    gs = [galp_gb300.generate_sbm([50] * k, 9.0, 2.0, seed=k) for k in (4, 9, 30)]
    with galp_gb300.Batch(gs, early_exit=0) as b:
        b.run(4)
        want = b.all_labels()
        for mode, row in ((2, 8), (0, 0), (2, 2), (2, 10), (0, 0)):
            tools.dispatch_set(b, mode, row)
            b.run(4)
            assert set(_rows(b)) == {row} and np.array_equal(b.all_labels(), want)


def _csr(lists):
    off = np.zeros(len(lists) + 1, np.int64)
    off[1:] = np.cumsum([len(x) for x in lists])
    return galp_gb300.Graph(off, np.concatenate([np.zeros(0, np.int64), *lists]).astype(np.int32))


def _kinds(ordered):
    """Graphs from empty to a few thousand vertices, in every counting range, some of which end early;
    ordered: all lists strictly increasing (the closed first iteration)."""
    rng = np.random.default_rng(ordered)

    def lists(degs, n):
        return [np.sort(rng.choice(n, d, replace=False)) if ordered else rng.integers(0, n, d)
                for d in np.minimum(degs, n)]

    gs = [_csr([]), _csr([np.zeros(0, np.int64)]), _csr([np.array([1]), np.array([0])])]
    for n in (5, 17, 40, 129, 300):
        gs.append(_csr(lists(rng.integers(0, 40, n), n)))
    gs.append(_csr(lists(rng.integers(33, 1025, 1500), 1500)))
    gs.append(_csr(lists(np.concatenate([rng.integers(1025, 2600, 15), rng.integers(0, 33, 2600)]), 2615)))
    gs.append(_csr([np.array([v ^ 1]) for v in range(64)]))  # pairs: they swap labels for ever
    gs.append(galp_gb300.generate_sbm([40] * 30, 14.0, 1.0, seed=4))
    gs.append(galp_gb300.generate_sbm([300] * 4, 60.0, 2.0, seed=5))
    gs.append(_csr([np.zeros(0, np.int64)] * 70))
    return gs


@pytest.mark.parametrize("early_exit", [1, 0])
@pytest.mark.parametrize("ordered", [True, False])
@pytest.mark.parametrize("fill", ["graphs", "vertices"])
def test_captured_batch_equals_the_oracle(fill, ordered, early_exit):
    kinds = _kinds(ordered)
    if fill == "graphs":  # more than 4,096 graphs
        small = [i for i, g in enumerate(kinds) if g.n < 70]
        which = list(range(len(kinds))) + [small[i % len(small)] for i in range(4100)]
    else:                 # more than 2^18 vertices
        which = list(range(len(kinds))) * ((1 << 18) // sum(g.n for g in kinds) + 1)
    with galp_gb300.Batch([kinds[i] for i in which], early_exit=early_exit) as b:
        assert b.count > 4096 or b.n > 1 << 18
        assert bool(tools.schedule_info(b).flags & tools.SchedInfo.SORTED) == ordered
        for niter in (1, 4, 25, 4):
            before = tools.schedule_info(b).launches
            b.run(niter)
            after = tools.schedule_info(b).launches
            assert after - before > 3 * niter  # captured anew for each iteration count
            b.run(niter)
            assert tools.schedule_info(b).launches == after  # and replayed
            want = [oracle.run_par(g.offsets, g.neighbors, niter, early_exit=bool(early_exit)) for g in kinds]
            got = np.split(b.all_labels(), b.graph_v0[1:-1])
            ended = set()
            for j, i in enumerate(which):
                it, lab, counts = want[i]
                assert np.array_equal(got[j], lab), f"graph {j} (kind {i}) of {niter}"
                if kinds[i].n and j < 3 * len(kinds):
                    assert b.graph_stats(j) == (it, list(counts))
                    ended.add(it)
            assert len(ended) > 2 or niter < 25 or not early_exit
