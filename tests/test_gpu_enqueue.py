"""Results read after an enqueued run are that run's, whether or not galp_sync came before and
whatever run came before it."""
import numpy as np
import pytest

import galp_gb300
import oracle
from galp_gb300 import tools

pytestmark = pytest.mark.gpu

# one kernel; separate kernels (a vertex above 12,288 neighbours)
GRAPHS = {"one_kernel": lambda: galp_gb300.generate_sbm([100] * 30, 9.0, 4.0, seed=2),
          "separate": lambda: galp_gb300.generate_rmat(17, 16, seed=11)}


@pytest.mark.parametrize("kind", list(GRAPHS))
@pytest.mark.parametrize("sync", [True, False])
def test_labels_of_an_enqueued_run(kind, sync):
    g = GRAPHS[kind]()
    with galp_gb300.Propagator(g, early_exit=0) as p:
        for before, k in ((6, 3), (3, 4), (0, 5)):
            if before:
                p.run(before)
            p.enqueue(k)
            if sync:
                p.sync()
            _, want, counts = oracle.run_par(g.offsets, g.neighbors, k, early_exit=False)
            assert np.array_equal(p.get_labels(), want)
            assert len(tools.dispatch_log(p)[1]) == k
            if not sync:
                p.sync()  # still gives the run's statistics
                assert p.stats.device_ms > 0
            assert p.iters_run == k and p.updates == list(counts)
            assert np.array_equal(p.get_labels(), want)


@pytest.mark.parametrize("sync", [True, False])
def test_labels_of_an_enqueued_batch(sync):
    gs = [galp_gb300.generate_sbm([40] * k, 7.0, 3.0, seed=k) for k in (3, 20, 9)]
    with galp_gb300.Batch(gs, early_exit=0) as b:
        for before, k in ((6, 3), (3, 4), (0, 5)):
            if before:
                b.run(before)
            b.enqueue(k)
            if sync:
                b.sync()
            want = [oracle.run_par(g.offsets, g.neighbors, k, early_exit=False)[1] for g in gs]
            assert np.array_equal(b.all_labels(), np.concatenate(want))
            for i in range(len(gs)):
                assert np.array_equal(b.labels(i), want[i])
            b.sync()
