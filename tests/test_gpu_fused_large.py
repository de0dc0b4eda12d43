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


@pytest.mark.parametrize("per_block, one", [(1, True), (8, True), (9, False)])
def test_how_many_large_vertices(per_block, one):
    import torch

    blocks = min(torch.cuda.get_device_properties(0).multi_processor_count, 256)
    large = 8 * blocks + 1 if per_block > 8 else per_block * blocks
    g = _graph(np.concatenate([np.full(large, 1025), np.full(3000, 5)]), 2)
    with galp_gb300.Propagator(g, early_exit=0) as p:
        p.run(3)
        assert (tools.schedule_info(p).launches == 1) == one
    gs = [_graph(np.concatenate([np.full(k, 1025), np.full(400, 5)]), 3) for k in (large // 2, large - large // 2)]
    with galp_gb300.Batch(gs, early_exit=0) as b:
        b.run(3)
        assert (tools.schedule_info(b).launches == 1) == one


def test_very_many_large_vertices_take_their_own_kernels():
    # 20,000 vertices of 1,100 neighbours: one block each in one kernel took twice the separate
    # kernels' time; a run is now no slower than the same kernels one after the other
    g = _graph(np.full(20000, 1100), 4)
    with galp_gb300.Propagator(g, early_exit=0) as p:
        p.run(10)
        got = _run_ms(p)
        tools.profile(p, 1)
        assert got < 1.1 * _run_ms(p)
