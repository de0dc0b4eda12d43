"""Batches above the one-kernel limits: the captured graph of a run follows what was set since."""
import numpy as np
import pytest

import galp_gb300
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
