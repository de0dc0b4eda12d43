"""A barrier wait of a one-kernel run that runs out: the call reports GALP_ETIMEOUT with the
statistics of a run that never got anywhere, runs enqueued behind it report it too instead of
racing through half-counted barriers, and the run after galp_sync is exact again.  The test hook
makes the waits expect an arrival that never comes, with a short limit."""
import ctypes

import numpy as np
import pytest

import galp_gb300
import oracle
from galp_gb300 import tools

pytestmark = pytest.mark.gpu

ETIMEOUT = -4


def _break(p, on):
    L = galp_gb300.load_library()
    L.galp_debug_barrier.argtypes = [ctypes.c_void_p, ctypes.c_int64, ctypes.c_int32]
    L.galp_debug_barrier.restype = ctypes.c_int
    assert L.galp_debug_barrier(p._h, 2000 if on else 0, int(on)) == 0


def _times_out(p, call):
    with pytest.raises(galp_gb300.GalpError) as e:
        call()
    assert e.value.code == ETIMEOUT
    assert p.stats.err & 1 and p.stats.iters_run == 0 and p.stats.runs_last == 0
    assert not any(p.stats.updates)


def _exact(p, gs, niter):
    p.run(niter)
    want = [oracle.run_par(g.offsets, g.neighbors, niter, early_exit=False) for g in gs]
    got = p.get_labels() if hasattr(p, "get_labels") else p.all_labels()
    assert np.array_equal(got, np.concatenate([w[1] for w in want]))
    assert p.stats.err == 0 and p.stats.iters_run == niter


def _contexts():
    # 512-thread shape (fixed tiles), 768-thread shape, a batch
    narrow = galp_gb300.generate_sbm([256] * 64, 16.0, 2.0, seed=1)
    wide = galp_gb300.generate_sbm([500] * 300, 16.0, 2.0, seed=2)
    parts = [galp_gb300.generate_sbm([90] * k, 9.0, 2.0, seed=k) for k in range(5, 45)]
    yield lambda: galp_gb300.Propagator(narrow, early_exit=0), [narrow]
    yield lambda: galp_gb300.Propagator(wide, early_exit=0), [wide]
    yield lambda: galp_gb300.Batch(parts, early_exit=0), parts


@pytest.mark.parametrize("case", range(3))
def test_timeout_is_reported_and_recovers(case):
    make, gs = list(_contexts())[case]
    with make() as p:
        _break(p, True)
        _times_out(p, lambda: p.run(4))  # the context's first run
        assert len(tools.dispatch_log(p)[1]) == 0
        _break(p, False)
        _exact(p, gs, 4)
        _break(p, True)
        _times_out(p, lambda: p.run(4))  # after a run that ended
        _break(p, False)
        before = tools.schedule_info(p).launches
        _exact(p, gs, 3)
        assert tools.schedule_info(p).launches - before == 1


@pytest.mark.parametrize("case", range(3))
@pytest.mark.parametrize("first", [False, True])
def test_runs_enqueued_behind_a_timeout(case, first):
    make, gs = list(_contexts())[case]
    with make() as p:
        if not first:
            _exact(p, gs, 2)
        _break(p, True)
        p.enqueue(5)
        _break(p, False)
        p.enqueue(5)
        p.enqueue(3)
        _times_out(p, p.sync)
        for k in (3, 5, 5):
            _exact(p, gs, k)


def test_separate_kernels_behind_a_timeout():
    make, gs = list(_contexts())[0]
    with make() as p:
        _break(p, True)
        p.enqueue(5)
        _break(p, False)
        tools.profile(p, 1)  # this run takes the separate kernels and is not disturbed
        p.enqueue(3)
        tools.profile(p, 0)
        with pytest.raises(galp_gb300.GalpError) as e:
            p.sync()
        assert e.value.code == ETIMEOUT
        _, want, _ = oracle.run_par(gs[0].offsets, gs[0].neighbors, 3, early_exit=False)
        assert p.stats.iters_run == 3 and np.array_equal(p.get_labels(), want)
        _exact(p, gs, 4)
