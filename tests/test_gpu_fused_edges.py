"""The edges of one-kernel runs at this device's own number of multiprocessors: tiles fixed to a
warp and claimed ones, blocks without a fixed tile, chunks of one, two and three rows."""
import numpy as np
import pytest

from test_gpu_fused_tiles import NARROW, _check, test_batch_rows as check_batch_rows

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def blocks():
    import torch

    return min(torch.cuda.get_device_properties(0).multi_processor_count, 256)


@pytest.mark.parametrize("extra", [-1, 0, 1])
def test_fixed_and_claimed(blocks, extra):
    n = blocks * NARROW * 32 + extra
    _check(np.random.default_rng(extra + 7).integers(0, 12, n), 300 + extra)


@pytest.mark.parametrize("times, extra", [(1, -1), (1, 0), (2, 5)])
def test_few_free_blocks(blocks, times, extra):
    rng = np.random.default_rng(times)
    large = times * blocks + extra
    _check(rng.permutation(np.concatenate([rng.integers(1025, 1400, large), rng.integers(33, 200, 500),
                                           rng.integers(0, 33, 9000)])), large)


@pytest.mark.parametrize("size", [511, 513, 1024, 1030])
def test_batch_rows(blocks, size):
    check_batch_rows([size] * blocks)


@pytest.mark.parametrize("n, mid, deg", [(1 << 20, 60000, 33), (1 << 20, 15000, 130), (1 << 21, 530000, 35),
                                         (1 << 21, 31000, 600)])
def test_queue_of_tied_vertices(n, mid, deg):
    # all vertices above 32 neighbours in the first blocks' chunks: more of them than the queue holds,
    # and fewer over many rounds; both block shapes
    degs = np.concatenate([np.full(mid, deg), np.zeros(n - mid, np.int64)])
    _check(degs, mid, niter=3)
