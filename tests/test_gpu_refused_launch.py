"""One-kernel runs whose launch is refused: a cluster falls back to a cooperative launch, that to the
separate kernels (a batch to its captured graph), with the same labels and counts."""
import ctypes

import numpy as np
import pytest

import galp_gb300
import oracle
from galp_gb300 import tools

pytestmark = pytest.mark.gpu


def _refuse(p, bits):
    L = galp_gb300.load_library()
    L.galp_debug_launch.argtypes = [ctypes.c_void_p, ctypes.c_int32]
    L.galp_debug_launch.restype = ctypes.c_int
    assert L.galp_debug_launch(p._h, bits) == 0


def _one_kernel(p, gs, niter=5):
    """Run, check against the oracle, and say whether the run was one launch."""
    before = tools.schedule_info(p).launches
    p.run(niter)
    one = tools.schedule_info(p).launches - before == 1
    want = [oracle.run_par(g.offsets, g.neighbors, niter, early_exit=False) for g in gs]
    got = p.get_labels() if hasattr(p, "get_labels") else p.all_labels()
    assert np.array_equal(got, np.concatenate([w[1] for w in want]))
    if len(gs) > 1:
        assert [p.graph_stats(i)[1] for i in range(len(gs))] == [list(w[2]) for w in want]
    else:
        assert p.updates == list(want[0][2])
    assert p.stats.err == 0 and p.stats.iters_run == niter
    return one


SMALL = [galp_gb300.generate_sbm([64] * 16, 8.0, 2.0, seed=7)]   # one cluster
LARGE = [galp_gb300.generate_sbm([256] * 64, 16.0, 2.0, seed=1)]  # a cooperative launch
MANY = [galp_gb300.generate_sbm([50] * k, 9.0, 2.0, seed=k) for k in (3, 5, 60)]


def test_cluster_refused():
    with galp_gb300.Propagator(SMALL[0], early_exit=0) as p:
        assert _one_kernel(p, SMALL)
        _refuse(p, 1)
        assert _one_kernel(p, SMALL) and _one_kernel(p, SMALL, 1)
        _refuse(p, 0)
        assert _one_kernel(p, SMALL)


@pytest.mark.parametrize("gs,bits", [(SMALL, 3), (LARGE, 2), (MANY, 2)])
@pytest.mark.parametrize("first", [False, True])
def test_cooperative_launch_refused(gs, bits, first):
    make = (lambda: galp_gb300.Batch(gs, early_exit=0)) if len(gs) > 1 else \
        (lambda: galp_gb300.Propagator(gs[0], early_exit=0))
    with make() as p:
        if not first:
            assert _one_kernel(p, gs)
        _refuse(p, bits)
        assert not _one_kernel(p, gs)
        _refuse(p, 0)
        # from here on separate kernels, a batch's captured (and counted) once per iteration count
        for niter in (5, 2, 5, 5):
            _one_kernel(p, gs, niter)
        if len(gs) == 1:
            assert not _one_kernel(p, gs)


def test_refused_while_a_run_is_queued():
    g = LARGE[0]
    with galp_gb300.Propagator(g, early_exit=0) as p:
        p.enqueue(4)
        _refuse(p, 2)
        p.enqueue(3)  # gives the one-kernel run's memory back
        p.sync()
        assert p.iters_run == 3
        assert np.array_equal(p.get_labels(), oracle.run_par(g.offsets, g.neighbors, 3, early_exit=False)[1])
