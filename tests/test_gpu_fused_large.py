"""One-kernel runs of graphs with vertices above 1024 neighbours against the separate kernels: as
fast within what the two differ by, and not taken at all with very many of them."""
import ctypes

import numpy as np
import pytest

import galp_gb300
from galp_gb300 import tools

pytestmark = pytest.mark.gpu


def _graph(degs, seed):
    rng = np.random.default_rng(seed)
    degs = rng.permutation(degs)
    off = np.concatenate([[0], np.cumsum(degs)]).astype(np.int64)
    return galp_gb300.Graph(off, rng.integers(0, len(degs), off[-1]).astype(np.int32))


def _run_ms(p):
    ms = []
    for _ in range(6):
        p.run(10)
        ms.append(p.stats.device_ms)
    return min(ms)


def test_large_tied_vertices_do_not_wait_for_each_other():
    # 660 vertices of 12,000 neighbours over 600 K vertices: a block meets its few of them in several
    # rounds of the resolve phase (one after the other they took 1.8 times the separate kernels)
    g = _graph(np.concatenate([np.full(660, 12000), np.full(600_000, 20)]), 1)
    with galp_gb300.Propagator(g, early_exit=0) as p:
        p.run(10)
        want = p.get_labels()
        assert tools.schedule_info(p).launches == 1
        one = _run_ms(p)
        L = galp_gb300.load_library()
        L.galp_debug_launch.argtypes = [ctypes.c_void_p, ctypes.c_int32]
        assert L.galp_debug_launch(p._h, 3) == 0
        separate = _run_ms(p)
        assert np.array_equal(p.get_labels(), want)
    assert one < 1.35 * separate, (one, separate)
