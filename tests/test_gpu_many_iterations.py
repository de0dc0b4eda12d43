"""Runs of more iterations than the statistics record (GALP_MAX_ITERS): the dispatcher goes by the
iteration before, not by the record."""
import numpy as np
import pytest

import galp_gb300
import oracle
from galp_gb300 import tools

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("opts", [{}, {"dispatch": 1}, {"frontier": 1}, {"frontier": 1, "dispatch": 1}])
@pytest.mark.parametrize("niter", [65, 150])
def test_exact_beyond_the_record(opts, niter):
    # pairs swap their labels for ever beside communities that converge
    g = galp_gb300.generate_sbm([100] * 30, 14.0, 1.0, seed=4)
    pairs = g.n + (np.arange(400) ^ 1)
    both = galp_gb300.Graph(np.concatenate([g.offsets, g.offsets[-1] + 1 + np.arange(400)]),
                            np.concatenate([g.neighbors, pairs]).astype(np.int32))
    it, want, counts = oracle.run_par(both.offsets, both.neighbors, niter, early_exit=False)
    with galp_gb300.Propagator(both, early_exit=0, **opts) as p:
        p.run(niter)
        assert p.iters_run == it == niter
        assert list(p.stats.updates) == list(counts[:64])
        assert np.array_equal(p.get_labels(), want)
        assert len(tools.dispatch_log(p)[1]) == 64
