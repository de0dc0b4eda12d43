"""The batch autotuner times the run that the batch takes and leaves it in force."""
import numpy as np
import pytest

import galp_gb300
from galp_gb300 import tools

pytestmark = pytest.mark.gpu


def _run_launches(b, niter):
    before = tools.schedule_info(b).launches
    b.run(niter)
    return tools.schedule_info(b).launches - before


def _steady_ms(b, niter):
    ms = []
    for _ in range(20):
        b.run(niter)
        ms.append(b.stats.device_ms)
    return min(ms)


def test_small_vertices_have_nothing_to_choose():
    # planted partitions whose vertices all have at most 32 neighbours: one kernel, and as separate
    # kernels no launch shape with an effect
    gs = [galp_gb300.generate_sbm([40] * k, 7.0, 2.0, seed=k) for k in range(4, 60)]
    assert max(g.degrees().max() for g in gs) <= 32
    with galp_gb300.Batch(gs) as b:
        b.run(10)
        want = b.all_labels()
        before = _steady_ms(b, 10)
        res = b.tune(10)
        assert res["trials"] == 3 and res["dispatch_row"] == -1  # one kernel, separate kernels twice
        assert _run_launches(b, 10) == 1 and np.array_equal(b.all_labels(), want)
        # several times what the one kernel takes is the separate kernels' time
        assert res["best_ms"] < 1.5 * before


def test_a_row_is_kept_only_above_the_one_kernel():
    rng = np.random.default_rng(3)
    gs = []
    for i in range(12):
        deg = rng.permutation(np.concatenate([rng.integers(1025, 1500 + 400 * (i % 2), 2), rng.integers(33, 900, 20),
                                              rng.integers(1, 33, 1500)]))
        off = np.zeros(len(deg) + 1, np.int64)
        off[1:] = np.cumsum(deg)
        gs.append(galp_gb300.Graph(off, rng.integers(0, len(deg), off[-1]).astype(np.int32)))
    with galp_gb300.Batch(gs, early_exit=0) as b:
        b.run(6)
        want = b.all_labels()
        before = _steady_ms(b, 6)
        res = b.tune(6)
        assert res["trials"] == 1 + 2 + 3 + 3 + 4 and res["dispatch_row"] in (-1, 0, 2, 8, 10)
        assert res["best_ms"] < 1.5 * before
        assert (_run_launches(b, 6) == 1) == (res["dispatch_row"] == -1)
        assert np.array_equal(b.all_labels(), want)


def test_profiled_batches_are_tuned_as_they_run():
    gs = [galp_gb300.generate_sbm([60] * k, 20.0, 9.0, seed=k) for k in range(4, 30)]
    with galp_gb300.Batch(gs) as b:
        tools.profile(b, 1)  # its runs take the separate kernels
        res = b.tune(4)
        assert res["trials"] == 2 + 3 + 3 and res["dispatch_row"] == -1
        tools.profile(b, 0)
        assert _run_launches(b, 4) == 1
