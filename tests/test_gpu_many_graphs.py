"""Batches of very many small graphs: the scan of the run sums, the graphs' run bases and the end of
an iteration are spread over the device; exact at every number of sums around the rounds of the
scan, with empty graphs and graphs without edges anywhere, also at the end."""
import numpy as np
import pytest

import galp_gb300
import oracle
from galp_gb300 import tools

pytestmark = pytest.mark.gpu


def _kinds():
    """Small graphs by kind: offsets and neighbours."""
    rng = np.random.default_rng(5)
    kinds = [(np.zeros(1, np.int64), np.zeros(0, np.int32)), (np.zeros(4, np.int64), np.zeros(0, np.int32)),
             (np.zeros(2, np.int64), np.zeros(0, np.int32))]
    for n in (2, 3, 9, 20):
        deg = rng.integers(0, 6, n)
        off = np.concatenate([[0], np.cumsum(deg)]).astype(np.int64)
        kinds.append((off, rng.integers(0, n, off[-1]).astype(np.int32)))
    kinds.append((np.arange(5, dtype=np.int64), np.array([1, 0, 3, 2], np.int32)))  # swaps labels for ever
    return kinds


def _batch(kinds, which):
    n = np.array([len(k[0]) - 1 for k in kinds], np.int64)[which]
    m = np.array([len(k[1]) for k in kinds], np.int64)[which]
    v0 = np.concatenate([[0], np.cumsum(n)])
    e0 = np.concatenate([[0], np.cumsum(m)])
    off = np.concatenate([kinds[k][0][:-1] + e0[i] for i, k in enumerate(which)] + [e0[-1:]])
    nbr = np.concatenate([kinds[k][1] + v0[i] for i, k in enumerate(which)]).astype(np.int32)
    return dict(offsets=off, neighbors=nbr, graph_v0=v0)


@pytest.mark.parametrize("early_exit", [1, 0])
@pytest.mark.parametrize("sums", [8191, 8192, 8193, 32767, 32768, 32769, 40960, 40961, 70000])
def test_rounds_of_the_scan(sums, early_exit):
    # as many sums as given: one per 1,024 vertices and one per graph
    kinds = _kinds()
    which = np.random.default_rng(sums).integers(0, len(kinds), sums)
    which[-3:] = 0
    n = np.array([len(k[0]) - 1 for k in kinds])[which]
    from_end = np.cumsum(n[::-1])[::-1]
    size = np.arange(sums, 0, -1) + (from_end + 1023) // 1024  # sums of the batch that begins at graph i
    which = which[np.argmin(np.abs(size - sums)):]
    for niter in (1, 3, 7):
        want = [oracle.run(*k, niter, early_exit=bool(early_exit)) for k in kinds]
        with galp_gb300.Batch(early_exit=early_exit, **_batch(kinds, which)) as b:
            b.run(niter)
            b.run(niter)
            assert np.array_equal(b.all_labels(), np.concatenate([want[k][1] for k in which]))
            for i in list(range(0, len(which), 997)) + list(range(len(which) - 9, len(which))):
                if len(kinds[which[i]][0]) > 1:
                    assert b.graph_stats(i) == (want[which[i]][0], list(want[which[i]][2]))
            assert b.stats.runs_last == _runs(kinds, which, niter, early_exit)


def _runs(kinds, which, niter, early_exit):
    """Distinct neighbour labels over all vertices in the last iteration that the batch ran (graphs
    that ended keep their labels)."""
    iters = max(oracle.run(*k, niter, early_exit=bool(early_exit))[0] for k in kinds)
    per = []
    for off, nbr in kinds:
        lab = oracle.run(off, nbr, iters - 1, early_exit=bool(early_exit))[1] if iters > 1 else np.arange(len(off) - 1)
        per.append(sum(len(set(lab[nbr[off[v]:off[v + 1]]])) for v in range(len(off) - 1)))
    return int(np.array(per)[which].sum())


def test_graphs_do_not_cost_more_than_their_vertices():
    # 300,000 graphs of 20 vertices: the scan, the bases and the iteration's end stay below the counting
    rng = np.random.default_rng(1)
    G, n, deg = 300_000, 20, 4
    v = np.arange(G * n, dtype=np.int64)
    nbr = (v - v % n)[:, None] + rng.integers(0, n, (G * n, deg))
    with galp_gb300.Batch(offsets=np.arange(G * n + 1, dtype=np.int64) * deg, neighbors=nbr.reshape(-1).astype(np.int32),
                          graph_v0=np.arange(G + 1, dtype=np.int64) * n, early_exit=0) as b:
        b.run(5)
        tools.profile(b, 2)
        b.run(5)
        tools.profile_kernels(b)
        b.run(5)
        ms = {k: t for k, (t, _) in tools.profile_kernels(b).items()}
    books = sum(ms.get(k, 0.0) for k in ("scan_sums_kernel", "scan_kernel", "batch_bases_kernel", "batch_finalize_kernel"))
    assert books < ms["count_small_sort_kernel"], ms
