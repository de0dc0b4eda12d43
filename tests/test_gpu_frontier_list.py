"""The frontier's list of changed vertices: kept without holding the counting up where most vertices
change, exact whatever part of a warp's vertices changes."""
import numpy as np
import pytest

import galp_gb300
import oracle
from galp_gb300 import tools

pytestmark = pytest.mark.gpu


def _grid(w):
    v = np.arange(w * w)
    x, y = v % w, v // w
    nbr = np.stack([((y - 1) % w) * w + x, y * w + (x - 1) % w, y * w + (x + 1) % w, ((y + 1) % w) * w + x], 1)
    return galp_gb300.Graph(np.arange(w * w + 1, dtype=np.int64) * 4, np.sort(nbr, 1).reshape(-1).astype(np.int32))


@pytest.mark.parametrize("n, p", [(33, 1.0), (3000, 0.5), (100_000, 0.02), (100_000, 0.9)])
def test_parts_of_warps_change(n, p):
    # a share p of the vertices swaps labels in pairs for ever, the others stand still
    rng = np.random.default_rng(n)
    pairs = rng.permutation(n)[: int(n * p) // 2 * 2].reshape(-1, 2)
    to = np.arange(n)
    to[pairs[:, 0]], to[pairs[:, 1]] = pairs[:, 1], pairs[:, 0]
    deg = np.where(to == np.arange(n), 0, 1)
    off = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
    g = galp_gb300.Graph(off, to[deg > 0].astype(np.int32))
    for frac in (1.0, 0.05):
        with galp_gb300.Propagator(g, frontier=1, early_exit=0) as q:
            assert tools.schedule_info(q).flags & tools.SchedInfo.FRONTIER
            tools.set_variant(q, frontier_frac=frac)
            for k in (2, 5):
                q.run(k)
                _, want, counts = oracle.run_par(g.offsets, g.neighbors, k, early_exit=False)
                assert np.array_equal(q.get_labels(), want) and q.updates == list(counts)


def test_changes_do_not_hold_the_counting_up():
    # a torus of 3 M vertices, most of which change in every iteration
    g = _grid(1732)

    def ms(**opts):
        with galp_gb300.Propagator(g, early_exit=0, **opts) as p:
            t = []
            for _ in range(6):
                p.run(10)
                t.append(p.stats.device_ms)
            return min(t)

    plain, frontier = ms(), ms(frontier=1)
    assert frontier < 1.27 * plain, (frontier, plain)
