"""Workloads that users of galp_gb300 run, for timing and for comparing builds.

Every case goes through the public Python entry points (galp_gb300.Propagator,
galp_gb300.Batch, the seeded generators): a graph in host memory (or a batch in device
memory) is clustered for ten iterations, and the labels, the number of iterations and the
change counts come back.  `mode` says what a pass is:

  run     a program that keeps its context and clusters the graph again: run + get_labels
  whole   the command line's use, once per graph: create the context from the host CSR
          (upload, schedule, checks), run, read the labels, destroy it
  batch   many independent graphs clustered together by one Batch

Labels are whole numbers and exact by construction, so there is no 64-bit reference
to state here: outputs are compared for equality.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import galp_gb300

NITER = 10


def listed():
    return [
        # the smallest call: a planted partition of 1,024 vertices (the smoke check's graph),
        # where launches and latency are all there is
        dict(name="sbm_1k", mode="run", graph="sbm", n=1024, blocks=16, deg_in=8.0, deg_out=2.0),
        # 64 communities of 256: the small benchmark configuration
        dict(name="sbm_16k", mode="run", graph="sbm", n=16384, blocks=64, deg_in=16.0, deg_out=2.0),
        # a million-vertex LFR-style graph with the method a user of the lock-free hash picks
        dict(name="lfr_1m", mode="run", graph="lfr", n=1_000_000, kmean=20.0, mu=0.3, method=1),
        # skewed degrees at a size where every launch is short: scale 16
        dict(name="rmat_16", mode="run", graph="rmat", scale=16, edge_factor=16),
        # the active-vertex frontier under the learned dispatcher
        dict(name="rmat_20_frontier", mode="run", graph="rmat", scale=20, edge_factor=16, frontier=1, dispatch=1),
        # ordinary size: scale 22, in-core defaults
        dict(name="rmat_22", mode="run", graph="rmat", scale=22, edge_factor=16),
        # the largest: half a billion entries in-core (the scale-24 benchmark configuration)
        dict(name="rmat_24", mode="run", graph="rmat", scale=24, edge_factor=16),
        # as many entries over four times the vertices: sparse, mostly tiny degrees, labels
        # that do not stay in L2
        dict(name="rmat_26_sparse", mode="run", graph="rmat", scale=26, edge_factor=4),
        # out-of-core with overlapped copies: neighbours streamed in batches of 2^22 entries
        dict(name="rmat_22_ooc", mode="run", graph="rmat", scale=22, edge_factor=16, policy=2, buffer_pow=22),
        # the command line's use: one graph, one context, from host CSR to host labels
        dict(name="rmat_20_whole", mode="whole", graph="rmat", scale=20, edge_factor=16),
        # a small batch: graphs of a few hundred to a few thousand vertices
        dict(name="batch_96", mode="batch", count=96, nmin=200, nmax=5000, deg_in=12.0, deg_out=3.0),
        # a quarter of the 4,096-graph batched configuration
        dict(name="batch_1024", mode="batch", count=1024, nmin=1000, nmax=200_000, deg_in=12.0, deg_out=3.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sbm", "lfr", "rmat", "rmat", "rmat_opts", "ooc", "whole", "batch"])
    if kind == "sbm":
        n = _log_int(rng, 500, 300_000)
        return dict(mode="run", graph="sbm", n=n, blocks=max(2, _log_int(rng, 4, max(5, n // 20))),
                    deg_in=round(rng.uniform(6.0, 24.0), 2), deg_out=round(rng.uniform(1.0, 5.0), 2),
                    method=rng.randrange(2))
    if kind == "lfr":
        return dict(mode="run", graph="lfr", n=_log_int(rng, 5_000, 1_000_000), kmean=round(rng.uniform(10.0, 30.0), 2),
                    mu=round(rng.uniform(0.15, 0.5), 3), method=rng.randrange(2))
    if kind == "batch":
        count = _log_int(rng, 16, 1024)
        nmax = _log_int(rng, 2_000, 200_000)
        return dict(mode="batch", count=count, nmin=min(1000, max(100, nmax // 20)), nmax=nmax,
                    deg_in=round(rng.uniform(8.0, 16.0), 2), deg_out=round(rng.uniform(1.0, 5.0), 2))
    edge_factor = _log_int(rng, 4, 28)
    top = 27 - max(2, math.ceil(math.log2(edge_factor)))  # at most 2^27 sampled edges
    if kind == "rmat":
        scale = rng.randint(11, top)
        return dict(mode="run", graph="rmat", scale=scale, edge_factor=edge_factor, method=rng.randrange(2))
    if kind == "rmat_opts":
        return dict(mode="run", graph="rmat", scale=rng.randint(12, min(top, 22)), edge_factor=edge_factor,
                    frontier=rng.randrange(2), dispatch=1)
    if kind == "ooc":
        return dict(mode="run", graph="rmat", scale=rng.randint(16, min(top, 22)), edge_factor=edge_factor,
                    policy=rng.choice([1, 2, 2]), buffer_pow=rng.randint(20, 24))
    return dict(mode="whole", graph="rmat", scale=rng.randint(12, min(top, 22)), edge_factor=edge_factor)


def _rmat_vertices(scale, edge_factor):
    """Vertices kept of an R-MAT graph: five standard deviations below the expected number
    that have an edge (a vertex whose ID has j one-bits ends an edge with probability
    0.76^(scale-j) 0.24^j), so that the number does not depend on the seed."""
    ne = edge_factor << scale
    e = sum(math.comb(scale, j) * -math.expm1(-2 * ne * 0.76 ** (scale - j) * 0.24 ** j) for j in range(scale + 1))
    return int(e - 5 * math.sqrt(e))


def _rmat(scale, edge_factor, seed):
    """R-MAT (0.57, 0.19, 0.19, 0.05) on the device: symmetrised, no self-loops or
    duplicates, isolated vertices deleted, IDs compacted and cut at _rmat_vertices (the few
    vertices above, of the lowest degrees, go with their edges).  Host arrays (offsets
    int64, neighbours int32)."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    ne = edge_factor << scale
    u = torch.zeros(ne, dtype=torch.int32, device="cuda")
    v = torch.zeros(ne, dtype=torch.int32, device="cuda")
    for _ in range(scale):
        r = torch.rand(ne, device="cuda", generator=gen)
        ub = r >= 0.76
        vb = ((r >= 0.57) & ~ub) | (r >= 0.95)
        u.mul_(2).add_(ub)
        v.mul_(2).add_(vb)
        del r, ub, vb
    keep = u != v
    u, v = u[keep].long(), v[keep].long()
    del keep
    key = torch.cat([(u << scale) | v, (v << scale) | u])
    del u, v
    key = torch.sort(key).values
    first = torch.ones(key.numel(), dtype=torch.bool, device="cuda")
    torch.ne(key[1:], key[:-1], out=first[1:])
    key = key[first]
    del first
    nz = torch.zeros(1 << scale, dtype=torch.bool, device="cuda")
    nz[key >> scale] = True
    newid = (torch.cumsum(nz, 0) - 1).to(torch.int32)
    src, nbr = newid[key >> scale], newid[key & ((1 << scale) - 1)]
    del key, nz, newid
    n = _rmat_vertices(scale, edge_factor)
    keep = (src < n) & (nbr < n)
    src, nbr = src[keep], nbr[keep]
    del keep
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(src, minlength=n), 0, out=off[1:])
    g = galp_gb300.Graph(off.cpu().numpy(), nbr.cpu().numpy())
    del off, src, nbr
    torch.cuda.empty_cache()
    return g


def _batch(case, seed):
    """Planted-partition graphs concatenated on the device: n log-uniform in [nmin, nmax],
    4 to 256 equal communities each.  Device (offsets, neighbours), host graph_v0."""
    count = case["count"]
    rng = np.random.default_rng(count)  # the sizes belong to the case, the edges to the seed
    ns = np.exp(rng.uniform(np.log(case["nmin"]), np.log(case["nmax"]), count)).astype(np.int64)
    ks = rng.integers(4, 257, count)
    v0 = np.zeros(count + 1, np.int64)
    v0[1:] = np.cumsum(ns)
    N = int(v0[-1])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    dn, dv0 = torch.from_numpy(ns).cuda(), torch.from_numpy(v0[:-1]).cuda()
    csize = torch.from_numpy((ns + ks - 1) // ks).cuda()

    def pairs(deg, inside):
        per = (dn.double() * deg / 2).long()
        g = torch.repeat_interleave(torch.arange(count, device="cuda"), per)
        a = (torch.rand(g.numel(), device="cuda", dtype=torch.float64, generator=gen) * dn[g]).long()
        lo, span = torch.zeros_like(a), dn[g]
        if inside:
            lo = (a // csize[g]) * csize[g]
            span = torch.minimum(span - lo, csize[g])
        b = lo + (torch.rand(g.numel(), device="cuda", dtype=torch.float64, generator=gen) * span).long()
        return a + dv0[g], b + dv0[g]

    a0, b0 = pairs(case["deg_in"], True)
    a1, b1 = pairs(case["deg_out"], False)
    a, b = torch.cat([a0, a1]), torch.cat([b0, b1])
    del a0, a1, b0, b1
    keep = a != b
    a, b = a[keep], b[keep]
    key = torch.cat([a * N + b, b * N + a])
    del a, b, keep
    key = torch.unique(key)
    nbr = (key % N).to(torch.int32)
    off = torch.zeros(N + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(key // N, minlength=N), 0, out=off[1:])
    del key
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    return off, nbr, v0


def _graph(case, seed):
    if case["graph"] == "sbm":
        n, k = case["n"], case["blocks"]
        sizes = np.full(k, n // k, np.int64)
        sizes[: n % k] += 1
        return galp_gb300.generate_sbm(sizes, case["deg_in"], case["deg_out"], seed)
    if case["graph"] == "lfr":
        return galp_gb300.generate_lfr(case["n"], kmean=case["kmean"], mu=case["mu"], seed=seed)
    return _rmat(case["scale"], case["edge_factor"], seed)


def _options(case):
    return {k: case[k] for k in ("method", "policy", "buffer_pow", "frontier", "dispatch") if k in case}


def prepare(case, seed):
    seed = int(seed) % (1 << 31)
    if case["mode"] == "batch":
        off, nbr, v0 = _batch(case, seed)
        b = galp_gb300.Batch(offsets=off.data_ptr(), neighbors=nbr.data_ptr(), graph_v0=v0, n=off.numel() - 1,
                             m=nbr.numel())
        return dict(mode="batch", ctx=b)
    g = _graph(case, seed)
    if case["mode"] == "whole":
        return dict(mode="whole", graph=g, opts=_options(case))
    return dict(mode="run", ctx=galp_gb300.Propagator(g, **_options(case)))


def _updates(p):
    """Labels changed per iteration, zero after the last one run."""
    return np.array(p.stats.updates[:NITER], np.int64)


def run(state):
    if state["mode"] == "batch":
        b = state["ctx"]
        b.run(NITER)
        return dict(labels=b.all_labels(), iters=int(b.stats.iters_run))
    if state["mode"] == "whole":
        with galp_gb300.Propagator(state["graph"], **state["opts"]) as p:
            p.run(NITER)
            return dict(labels=p.get_labels(), iters=p.iters_run, updates=_updates(p))
    p = state["ctx"]
    p.run(NITER)
    return dict(labels=p.get_labels(), iters=p.iters_run, updates=_updates(p))


def _size(case):
    """Vertices and CSR entries, about (the exact ones come with the seed)."""
    if case["mode"] == "batch":
        lo, hi = case["nmin"], case["nmax"]
        n = case["count"] * (hi - lo) / math.log(hi / lo)
        return n, n * (case["deg_in"] + case["deg_out"])
    if case["graph"] == "sbm":
        return case["n"], case["n"] * (case["deg_in"] + case["deg_out"])
    if case["graph"] == "lfr":
        return case["n"], 0.92 * case["n"] * case["kmean"]
    s, ef = case["scale"], case["edge_factor"]
    # the share of edges left without duplicates grows slowly with the scale
    return _rmat_vertices(s, ef), 2 * (ef << s) * max(0.6, 1 - 0.4 * 2 ** (-(s - 10) / 3.5) * (ef / 16) ** 0.3)


def work(case):
    """Per iteration: every neighbour ID (4 bytes), every offset (8), every old label (4)
    and every new label (4), once; ten iterations.  Labels gathered more than once are not
    counted again.  No floating-point operations."""
    n, m = _size(case)
    return dict(bytes=float(NITER * (4 * m + 16 * n)), flops=0.0)
