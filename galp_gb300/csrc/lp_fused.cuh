// lp_fused.cuh -- a whole in-core run of a small graph in one kernel.
//
// A run of a graph whose iteration takes a few microseconds of work is bound by its launches:
// a dozen kernels per iteration at 2 to 6 us each.  fused_run_kernel does every iteration in
// one cooperative launch (one block per SM at most, all of them resident), with two grid-wide
// barriers per iteration:
//
//   count    vertices of more than 1024 neighbours by the block (hash table in shared
//            memory), lane-group and small tiles by warps (the code of the separate
//            kernels), one list of tiles for all warps of the grid; each warp adds its
//            vertices' distinct counts to the sums of the chunks of vertices they belong to
//   barrier
//   resolve  each block scans the distinct counts of its own chunk from the chunk sums and
//            resolves the chunk's tied vertices where it meets them
//   barrier  every block reads the change counts and decides the early exit alike
//
// Batches of graphs run the same way, with run positions, change counts and early exits per
// graph: the sums are then those of the pieces in which graphs and chunks cut the vertices.
//
// Bound by the latency of a tile (two round trips to L2 per eight rows of gathers) and of the
// barriers (1.7 us each) on the smallest graphs; a warp's first tile is therefore the same in every
// iteration, with its neighbours in shared memory, and its gathers are 16 in flight.  On skewed
// graphs bound by the balance between the blocks: the other tiles are claimed from the list.
// Passes of ten iterations, tiles dealt out in fixed order, each kind by itself and gathered by the
// separate kernels' code -> this (us): planted partitions of 10 K entries 158 -> 124 (115 as a cluster), 294 K 230 ->
// 160; R-MAT 16 423 -> 342; LFR of 560 K entries 309 -> 200; batch of 96 graphs 432 -> 400 (372 with three rows per round).
//
// Shares of a run's time, count / wait at the barrier after it / resolve / wait: R-MAT 16 60 / 20 /
// 13 / 8 %, the batch of 96 graphs 51 / 12 / 27 / 11, LFR of a million vertices 80 / 2 / 15 / 2,
// planted partitions of 294 K entries 38 / 20 / 24 / 17, of 10 K 36 / 15 / 34 / 15.
//
// Labels, change counts, run counts and the dispatch log are those of the separate kernels.
#pragma once

#include "lp_index.h"
#include "lp_pipeline.cuh"

namespace galp {

// Block shapes: 512 threads where latency is all there is (up to kFusedNarrowEntries), with plans of
// the fixed tiles; 768 above, for more of the gathers in flight, without (their 96 KB would come out
// of the L1 cache: LFR of 5.5 M entries 663 -> 886 us).  768 threads have 80 registers: they store a
// gathered row before the next is loaded (tile_gather), all eight loaded first would spill (planted
// partitions of 3.8 M entries 454 -> 519).  512 against 768 threads (us): R-MAT 16 (1.8 M) 342 and
// 380, LFR of 1.9 M 357 and 362, R-MAT 18 with edge factor 4 (2.0 M) 437 and 436, planted partitions
// of 3.8 M 466 and 454, LFR of 5.5 M 691 and 663.
constexpr int kFusedNarrow = 512, kFusedWide = 768;  // batches: always narrow
constexpr int64_t kFusedNarrowEntries = 1 << 21;
constexpr int kFusedMaxBlocks = 256;
// Up to these sizes a run is one kernel (above kFusedAnyVertices only with kFusedDense entries per
// vertex: of a sparse graph's run the resolve phase is the larger part, and its separate kernel has
// more threads).  Passes of ten iterations, separate kernels against one (us): planted partitions of
// 10 K entries 336 and 115, 294 K 496 and 160, 3.8 M 713 and 454; R-MAT 16 (1.8 M) 699 and 342; LFR
// of 5.5 M entries 916 and 663, 18 M 1964 and 1768, 24 M (700 K vertices) 2131 and 1865; planted
// partitions of a million vertices with 5 M entries 1078 and 1071, 15 M 1516 and 1458, 25 M 1825 and
// 1846; 1.5 M vertices with 7.5 M entries 1367 and 1446, with 21 M (LFR) 2386 and 2165.  Batches,
// whose separate kernels are one CUDA-graph launch and whose resolve phase does more per vertex (the
// context's first pass, with the capture, and a later one): 16 graphs with 312 K entries 440 / 286
// and 234 / 197, 96 with 1.8 M (156 K vertices) 600 / 383 and 444 / 372, 100 with 3.7 M (202 K)
// 939 / 612 and 606 / 523, 60 with 3.4 M (254 K) 818 / 581 and 633 / 562; above the vertex limit
// 220 with 3.2 M (278 K) 678 / 478 and 657 / 567, 300 with 1.7 M (362 K) 1113 / 480 and 761 / 572.
constexpr int64_t kFusedMaxEntries = 1 << 25, kFusedMaxVertices = 1 << 21;
constexpr int64_t kFusedAnyVertices = 1 << 20, kFusedDense = 8;
constexpr int64_t kFusedMaxBatchEntries = 1 << 22, kFusedMaxBatchVertices = 1 << 18;
// Vertices above kGroupMax neighbours, per multiprocessor: each takes a whole block here, four of
// those up to 2048 share a multiprocessor in a kernel of their own.  Random graphs, ten iterations,
// one kernel against the separate ones (ms): 4 M entries with 390 of 2,048 neighbours 1.08 and 1.27,
// with 1,454 of 1,100 1.16 and 1.15, with 3,636 0.90 and 0.71; 20 M with 18,181 of 1,100 4.5 and 2.2,
// with 333 of 12,000 8.0 and 7.4; LFR of 7 M with 782 0.75 and 0.94, of 24 M with 1,967 2.26 and
// 2.17; batches of 2 M entries with 976 of 2,048 1.1 times as fast, with 1,816 of 1,100 0.88.
constexpr int64_t kFusedLarge = 8;
// Runs of up to kFusedClusterTiles tiles, all small or lane-group ones, are one thread-block cluster:
// its hardware barrier replaces the counter in global memory (0.6 us less each), and the launch is
// not cooperative.  One block per tile and the counter against the cluster (us): 512 vertices with
// 5 K entries 133 and 117, 1,024 with 10 K 133 and 115, 2,048 with 20 K (64 tiles) 139 and 122,
// 1,349 with 24 K (R-MAT 11) 141 and 140, four graphs of together 1,070 vertices 162 and 151; with
// more tiles 16 SMs are too few for the work: 2,700 vertices with 51 K (R-MAT 12) 156 and 165,
// 4,096 with 113 K 143 and 148.
constexpr int kFusedClusterBlocks = 16, kFusedClusterTiles = 64;
constexpr int kFusedMaxGraphs = 4096;
constexpr long long kFusedSpinLimit = 1ll << 21;  // polls of a barrier wait (about a second)

// Device memory of the run's barriers and sums, zero before the first run.  Every run leaves it so,
// except one whose wait ran out (Ctl::gave_up): runs enqueued behind it return at once, and
// galp_sync clears both.
struct FusedState {
    unsigned arrived;                        // blocks that have reached a barrier of this run
    unsigned left;                           // blocks that have ended it
    unsigned long long changes[3];           // of iteration i in entry i % 3
    unsigned long long runs[3];              // distinct labels, likewise
    int claimed[3];                          // tiles handed out beyond the fixed ones, likewise
};

struct FusedArgs {
    PipeArgs p;               // lab_in, lab_out, disp and the tied lists are not used
    int32_t *lab0, *lab1;
    FusedState *state;
    long long *sums;          // [3][pieces]: distinct labels per piece, of iteration i in row i % 3; zero
    int pieces;               // blocks + graphs
    DispatchArgs d;           // for the log (its rule is the fixed one)
    int64_t n, m;
    long long thr;            // early-exit threshold
    int niter;
    int shortcut;             // adjacency strictly increasing: the first iteration in closed form
    int chunk;                // vertices per block in the resolve phase
    int slots;                // table slots for vertices above kGroupMax
    int agg_mode;
    int cluster;              // the grid is one cluster
    long long spin_limit;     // polls before a barrier wait gives up
    unsigned more;            // arrivals awaited beyond the blocks' own (0; tests only)
    // batches
    unsigned long long *g_changes;  // [3][graphs]: labels changed, likewise
    int32_t *g_active, *g_iters;
    long long *g_counts;            // [graphs][max_iter]
    int g_max_iter, early_exit;
};

// The run's k-th barrier (k = 1, 2, ...) of all blocks; false when the wait ran out (Ctl::gave_up
// is set, and the block must return: the others give up in the same way).  In a run
// that is one cluster no wait can run out: all its blocks are resident, and none returns early.  The
// arrivals only count up, so a block waits for one number and nobody resets anything until the
// last block leaves the run.
__device__ __forceinline__ bool grid_barrier(const FusedArgs &a, Ctl *ctl, int *failed, unsigned k)
{
    FusedState *st = a.state;
    if (a.cluster) {
        asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
        return true;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&st->arrived) : "memory");
        unsigned now = 0;
        bool waits;
        long long i = 0;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(&st->arrived) : "memory");
            waits = barrier_waits(now - a.more, k, gridDim.x);
        } while (waits && ++i < a.spin_limit);
        if (waits) {
            atomicExch(&ctl->gave_up, 1);
            *failed = 1;
        }
    }
    __syncthreads();
    return !*failed;
}

// Dynamic shared memory: the warps' tile buffers, or the block's hash table, or the resolve
// phase's buffers.
// The queue of tied vertices above 32 neighbours takes several rounds' worth of them: a vertex above
// 1024 keeps its warp for up to 0.3 ms, which a block that empties the queue in every round waits
// for in every round (600 K random vertices of 20 neighbours and 666 of 12,000, ten iterations
// 14.2 -> 8.4 ms, separate kernels 7.6; without such vertices no change).
template <bool BATCH, int THREADS, int ROWS>
struct FusedResolve {
    static constexpr int kWarps = THREADS / 32;
    static constexpr int kPer = ROWS;  // vertices per thread and round
    static constexpr int kRound = kPer * THREADS;
    static constexpr int kQueue = BATCH ? 6 * THREADS : 8 * THREADS;
    int hist[kWarps][256];
    long long qa[kQueue];               // run base,
    long long qN[BATCH ? kQueue : 1];   // (batches) its graph's runs,
    int qv[kQueue];                     // vertex
    uint8_t qf[BATCH ? kQueue : 1];     // (batches) 1 = last of its graph, 2 = its graph still runs
    uint8_t grun[THREADS];  // (batches) whether the chunk's graphs still run
};
union FusedTile {
    TileBuf small;
    GroupBuf group;
};
template <int THREADS>
constexpr size_t kFusedTiles = sizeof(FusedTile) * (THREADS / 32);  // the plans lie behind
template <int THREADS>
constexpr int kFusedPlan = THREADS > kFusedNarrow ? 0 : 16;
template <int THREADS>
constexpr size_t kFusedSmem =
    kFusedTiles<THREADS> + (kFusedPlan<THREADS> ? sizeof(int32_t) * kPlanWords * (THREADS / 32) : 0);
static_assert(sizeof(FusedResolve<true, kFusedNarrow, 3>) <= kFusedTiles<kFusedNarrow> &&
                  sizeof(FusedResolve<false, kFusedNarrow, 1>) <= kFusedTiles<kFusedNarrow> &&
                  sizeof(FusedResolve<false, kFusedWide, 2>) <= kFusedTiles<kFusedWide>,
              "the resolve buffers fit the tile buffers");

// State of a vertex in the resolve phase, loaded in one round trip whether it is tied or not.
struct FusedVertex {
    int d, kw, r, g, gprev;    // g: its graph, gprev: the graph of the vertex before
    int32_t c0, c1, old, now;  // its label before, and after the count where it is not tied
    int64_t o0;
};

// ROWS: vertices per thread and round of the resolve phase.  A round is a chain of loads, scans and
// block barriers (about 5,000 cycles in batches), and rows beyond the block's vertices are paid for
// too: batches in the narrow shape take the rows that their chunk of vertices fills, up to three.
// One, two and three rows (us, on the device): 96 graphs with 165 K vertices (1,086 a block) 348, 344
// and 320, 150 with 180 K (1,186) 357, 352 and 328; 96 with 146 K (960) 285, 270 and 281, 200 with
// 132 K (871) 287, 271 and 284; 96 with 22 K (145) 137, 145 and 160.
template <bool BATCH, int kFusedThreads, int ROWS>
__global__ void __launch_bounds__(kFusedThreads, 1) fused_run_kernel(FusedArgs a)
{
    using Resolve = FusedResolve<BATCH, kFusedThreads, ROWS>;
    constexpr int kFusedWarps = Resolve::kWarps, kPer = Resolve::kPer, kRound = Resolve::kRound;
    extern __shared__ __align__(16) unsigned char fused_smem[];
    __shared__ GroupTiles T;
    __shared__ int red[5 * kFusedWarps], red2[2 * kFusedWarps];
    __shared__ long long wsum[kFusedWarps], wall[kFusedWarps], wlast[kFusedWarps];
    __shared__ unsigned long long sruns;
    __shared__ int sctr, qn, failed;
    PipeArgs p = a.p;
    p.lab_in = a.lab0;
    p.lab_out = a.lab1;
    FusedState *st = a.state;
    Ctl *ctl = p.ctl;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int nb = gridDim.x, b = blockIdx.x;
    const int nmid = p.nmid_s + p.nmid_l + p.nmid_x, ncta = nmid - p.gcut[5];
    FusedTile *tiles = reinterpret_cast<FusedTile *>(fused_smem);
    const BlockRed5<kFusedThreads> br{red, red2};
    if (tid == 0) {
        failed = *(volatile int *)&ctl->gave_up;
        T.set(p, p.gcut[5]);
    }
    if (b == 0) {  // the run's bookkeeping: nobody else touches it before the first barrier
        if (tid == 0) {
            ctl->active = 0;
            ctl->iter = 0;
            ctl->err = 0;
            ctl->N = 0;
            ctl->thr = a.thr;
            ctl->max_iter = a.niter;
            ctl->ticket = 0;
            ctl->changes = 0;
            ctl->changed_n = 0;
            ctl->frontier_off = 0;
            ctl->tied_mid = 0;
            st->changes[0] = 0;
        }
        if (tid < 64) ctl->counts[tid] = 0;
    }
    if (b == nb - 1) {  // the dispatch log, which the last block writes
        if (tid < kMaxLogIters) a.d.var_log[tid] = -1;
        for (int i = tid; i < kMaxLogIters * kFeat; i += kFusedThreads) a.d.feat_log[i] = 0.f;
    }
    for (int64_t v = (int64_t)b * kFusedThreads + tid; v < a.n; v += (int64_t)nb * kFusedThreads)
        a.lab0[v] = (int32_t)(BATCH ? v - __ldg(&p.g_v0[__ldg(&p.gid[v])]) : v);
    if (BATCH)
        for (int g = b * kFusedThreads + tid; g < p.ngraphs; g += nb * kFusedThreads) {
            a.g_active[g] = 1;
            a.g_iters[g] = 0;
            a.g_changes[g] = 0;
        }
    // the block's vertices in the resolve phase, their first and last graph, and the chunks
    // these two lie in
    const int64_t v0 = (int64_t)b * a.chunk, v1 = min(v0 + a.chunk, a.n);
    int gf = 0, gl = v0 < v1 ? 0 : -1, f0 = 0, f1 = nb, l0 = 0, l1 = 0;  // no vertices: no pieces
    if (BATCH && v0 < v1) {
        gf = __ldg(&p.gid[v0]);
        gl = __ldg(&p.gid[v1 - 1]);
        f0 = (int)(__ldg(&p.g_v0[gf]) / a.chunk);
        f1 = (int)((__ldg(&p.g_v0[gf + 1]) - 1) / a.chunk) + 1;
        l0 = (int)(__ldg(&p.g_v0[gl]) / a.chunk);
        l1 = (int)((__ldg(&p.g_v0[gl + 1]) - 1) / a.chunk) + 1;
    }
    auto piece_of = [&](int v) { return v < 0 ? 0 : v / a.chunk + (BATCH ? __ldg(&p.gid[v]) : 0); };
    // whether graph g still runs in iteration i: its last change count decides, whether or not
    // the thread that keeps g_active has seen it yet
    auto running = [&](int g, int i) {
        if (i == 0) return true;
        if (!*((volatile int32_t *)&a.g_active[g])) return false;
        const unsigned long long c = *((volatile unsigned long long *)&a.g_changes[(size_t)((i - 1) % 3) * p.ngraphs + g]);
        const double ng = (double)(__ldg(&p.g_v0[g + 1]) - __ldg(&p.g_v0[g]));
        return !((a.early_exit && (double)c <= ng * 1e-5) || i >= a.g_max_iter);
    };
    // count the changes of a warp's vertices for their graphs (row s of g_changes)
    auto graph_changes = [&](bool chg, int g, int s) {
        const int g0 = __reduce_max_sync(kFull, chg ? g : 0);
        if (__all_sync(kFull, !chg || g == g0)) {
            const int c = __popc(__ballot_sync(kFull, chg));
            if (lane == 0 && c) atomicAdd(&a.g_changes[(size_t)s * p.ngraphs + g0], (unsigned long long)c);
        } else if (chg) {
            atomicAdd(&a.g_changes[(size_t)s * p.ngraphs + g], 1ull);
        }
    };
    unsigned barriers = 0;
    __syncthreads();
    if (failed) return;  // a run before this one left the barriers and sums half-way
    // tiles: the lane groups' (largest degrees first), then the small vertices'.  Every warp of a
    // block without vertices above kGroupMax has its first tile fixed, consecutive ones on different
    // blocks, with its vertices and offsets in registers for all iterations; the other tiles are
    // claimed one by one.
    const int ngroup = T.count(), ntiles = ngroup + ((p.nsmall + 31) >> 5);
    const int nfree = max(nb - ncta, 0), nfixed = nfree * kFusedWarps;
    auto head_of = [&](int t) {
        if (t < ngroup) return group_head<true>(p, T, t, false);
        TileHead h{-1, 0, 0, 0, 0, 1};
        const int i = (t - ngroup) * 32 + lane;
        if (t < ntiles && i < p.nsmall) tile_head<true>(p, h, p.small_v[i], false);
        return h;
    };
    const int tile0 = b >= ncta ? w * nfree + b - ncta : -1;
    const TileHead head0 = head_of(tile0 >= 0 ? tile0 : ntiles);
    // its plan: the block's table is never used, so it stays
    constexpr int kPlanPer = kFusedPlan<kFusedThreads>;
    int32_t *plan = reinterpret_cast<int32_t *>(fused_smem + kFusedTiles<kFusedThreads>) + w * kPlanWords;
    if (!kPlanPer || tile0 < 0 || tile0 >= ntiles) {
        plan = nullptr;
    } else {
        int first = 0, n = 32;  // the lane's part of its vertex's neighbours
        if (tile0 < ngroup) {
            n = group_shape_of<true>(head0.deg, head0.g).N;  // as group_tile with a plan
            first = (lane & ((1 << head0.g) - 1)) * n;
        }
        const int cnt = head0.v >= 0 ? head0.deg - first : 0;
#pragma unroll 8
        for (int j = 0; j < 32; ++j)
            plan[j * 32 + lane] = j < n && j < cnt ? __ldg(&p.nbr[head0.o0 - p.nbr_shift + first + j]) : -1;
        __syncwarp();
    }
    if (!a.shortcut && !grid_barrier(a, ctl, &failed, ++barriers)) return;  // labels gathered by other blocks
    int it = 0;
    long long runs = 0, last_changes = 0;
    for (;;) {
        p.lab_in = it & 1 ? a.lab1 : a.lab0;
        p.lab_out = it & 1 ? a.lab0 : a.lab1;
        long long *sums = a.sums + (size_t)(it % 3) * a.pieces;
        unsigned long long counted = 0;  // distinct labels of the warp's vertices (batches)
        if (tid == 0) sruns = 0;
        unsigned long long changes = 0;
        const bool first = it == 0 && a.shortcut;
        if (b == nb - 1 && w == kFusedWarps - 1 && !first && it < kMaxLogIters) {
            // this iteration's entry of the dispatch log
            if (lane < kFeat)
                a.d.feat_log[it * kFeat + lane] = dispatch_feature(a.d, lane, it, last_changes, runs);
            if (lane == 0) a.d.var_log[it] = a.d.fixed_variant_dense;
        }
        if (first) {
            for (int64_t v = (int64_t)b * kFusedThreads + tid; v < a.n; v += (int64_t)nb * kFusedThreads) {
                const int64_t o0 = __ldg(&p.off[v]);
                const int64_t deg = __ldg(&p.off[v + 1]) - o0;
                AllCandidates q{deg};
                if (BATCH) {  // run positions and labels of the vertex's graph
                    const int g = __ldg(&p.gid[v]);
                    const int64_t vg = __ldg(&p.g_v0[g]);
                    int32_t nl = (int32_t)(v - vg);
                    if (deg > 0) {
                        const int64_t e0 = __ldg(&p.off[vg]), e1 = __ldg(&p.off[__ldg(&p.g_v0[g + 1])]);
                        const int r = resolve_rank(o0 - e0, deg, e1 - e0, v == __ldg(&p.g_last[g]), q);
                        nl = (int32_t)(__ldg(&p.nbr[o0 + r]) - vg);
                    }
                    p.lab_out[v] = nl;
                    count_change(changes, nl, (int32_t)(v - vg));
                } else {
                    int32_t nl = (int32_t)v;
                    if (deg > 0) nl = __ldg(&p.nbr[o0 + resolve_rank(o0, deg, a.m, v == p.last_v, q)]);
                    p.lab_out[v] = nl;
                    count_change(changes, nl, (int32_t)v);
                }
                p.dcnt[v] = (int32_t)deg;
            }
        } else {
            // vertices above kGroupMax neighbours, the largest first, one block each
            if (b < ncta) {
                unsigned long long *tab = reinterpret_cast<unsigned long long *>(fused_smem);
                for (int s = tid; s < a.slots; s += kFusedThreads) tab[s] = 0ull;
                uint32_t gen = 0;
                for (int i = b; i < ncta; i += nb) {
                    __syncthreads();
                    ++gen;  // far below kT64GenMax: at most ncta vertices per pass
                    const int v = p.mid_v[nmid - 1 - i];
                    const int64_t o0 = __ldg(&p.off[v]);
                    const int deg = (int)(__ldg(&p.off[v + 1]) - o0);
                    const int32_t old = get_label<true>(&p.lab_in[v]);
                    const uint32_t cap = (uint32_t)min(a.slots, 4 * pad32(deg));
                    const bool agg = a.agg_mode == 1 || (a.agg_mode == 0 && 2 * p.dcnt[v] <= deg);
                    constexpr int PER = 8;
                    Sum5 obs = sum5_empty();
                    for (int base = 0; base < deg; base += kFusedThreads * PER) {
                        int nbr[PER];
#pragma unroll
                        for (int u = 0; u < PER; ++u) {
                            const int e = base + tid + u * kFusedThreads;
                            nbr[u] = e < deg ? ld_nbr(&p.nbr[o0 + e]) : -1;
                        }
                        uint32_t lb[PER];
#pragma unroll
                        for (int u = 0; u < PER; ++u)
                            lb[u] = nbr[u] >= 0 ? (uint32_t)gather_label<true>(&p.lab_in[nbr[u]]) : kEmpty;
#pragma unroll
                        for (int u = 0; u < PER; ++u) {
                            if (base + u * kFusedThreads >= deg) break;  // block-uniform
                            t64_insert_row(tab, cap, gen, lb[u], agg, obs);
                        }
                    }
                    const Sum5 s = br.reduce(obs);
                    int rmin = 0, rmax = s.d - 1;
                    if (s.k > 1) {
                        if (s.k < s.d) {
                            t64_ranks(tab, (int)cap, tid, kFusedThreads, gen, s.mn, s.mx, rmin, rmax);
                            br.reduce2(rmin, rmax);
                        }
                        if (s.k > 2) {
                            if (tid == 0) sctr = 0;
                            __syncthreads();
                            t64_spill(tab, (int)cap, tid, kFusedThreads, gen, p.run_lab + o0, p.run_cnt + o0, &sctr);
                        }
                    }
                    if (tid == 0) {
                        finish_counted(p, v, s, rmin, rmax, changes, old);
                        atomicAdd((unsigned long long *)&sums[piece_of(v)], (unsigned long long)s.d);
                        counted += (unsigned long long)s.d;
                    }
                }
                __syncthreads();
            }
            auto claim = [&] {
                if (ntiles <= nfixed) return ntiles;
                int c = 0;
                if (lane == 0) c = atomicAdd(&st->claimed[it % 3], 1);
                return nfixed + __shfl_sync(kFull, c, 0);
            };
            for (int t = tile0 >= 0 ? tile0 : claim(); t < ntiles; t = claim()) {
                TileHead hd = head0;
                if (t != tile0) hd = head_of(t);
                else if (hd.v >= 0) hd.old = get_label<true>(&p.lab_in[hd.v]);
                int d;
                if (t < ngroup) {
                    d = group_tile<true, kPlanPer>(p, tiles[w].group, hd, changes, t == tile0 ? plan : nullptr);
                    if ((lane & ((1 << hd.g) - 1)) || hd.v < 0) d = 0;  // the group's first lane counts
                } else {
                    bool chg;
                    d = small_tile<true, kPlanPer>(p, tiles[w].small, hd, changes, chg, t == tile0 ? plan : nullptr);
                }
                add_runs(sums, piece_of(hd.v), d);
                counted += (unsigned)d;
            }
            if (BATCH) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) counted += __shfl_xor_sync(kFull, counted, o);
                __syncthreads();  // sruns is zero
                if (lane == 0 && counted) atomicAdd(&sruns, counted);
                __syncthreads();
                if (tid == 0 && sruns) atomicAdd(&st->runs[it % 3], sruns);
            }
        }
        if (!grid_barrier(a, ctl, &failed, ++barriers)) return;
        // entries of the iterations to come: their last readers passed the barrier before this one
        {
            long long *later = a.sums + (size_t)((it + 2) % 3) * a.pieces;
            for (int i = b + gf + tid; i <= b + gl; i += kFusedThreads) later[i] = 0;
            if (b == 0 && tid == 0) {
                st->changes[(it + 1) % 3] = 0;
                st->runs[(it + 2) % 3] = 0;
                st->claimed[(it + 1) % 3] = 0;
            }
            if (BATCH)
                for (int g = b * kFusedThreads + tid; g < p.ngraphs; g += nb * kFusedThreads)
                    a.g_changes[(size_t)((it + 1) % 3) * p.ngraphs + g] = 0;
        }
        if (!first) {
            Resolve &R = *reinterpret_cast<Resolve *>(fused_smem);
            // a round: kRound vertices, kPer per lane (a warp's are consecutive, row after row)
            auto load = [&](FusedVertex(&x)[kPer], int64_t vb) {
#pragma unroll
                for (int u = 0; u < kPer; ++u) {
                    const int64_t v = vb + (w * kPer + u) * 32 + lane;
                    x[u] = FusedVertex{};
                    if (v < v1) {
                        x[u].d = p.dcnt[v];
                        x[u].kw = p.sm_kw[v];
                        x[u].c0 = p.sm_c0[v];
                        x[u].c1 = p.sm_c1[v];
                        x[u].r = p.sm_r[v];
                        x[u].old = get_label<true>(&p.lab_in[v]);
                        x[u].o0 = __ldg(&p.off[v]);
                        if (BATCH) {
                            x[u].now = get_label<true>(&p.lab_out[v]);
                            x[u].g = __ldg(&p.gid[v]);
                            x[u].gprev = v > v0 ? __ldg(&p.gid[v - 1]) : -1;
                        }
                    }
                }
            };
            FusedVertex x[kPer];
            load(x, v0);
            // batches: the chunk's graphs, whether each still runs
            if (BATCH)
                for (int j = tid; j <= gl - gf && j < kFusedThreads; j += kFusedThreads) R.grun[j] = running(gf + j, it);
            // the run base of the chunk in its (first) graph and that graph's runs; in batches
            // also the runs of the chunk's last graph
            {
                long long below = 0, all = 0, last = 0;
                if (tid < nb) {
                    if (tid >= f0 && tid < f1) {
                        all = *((volatile long long *)&sums[tid + gf]);
                        if (tid < b) below = all;
                    }
                    if (BATCH && tid >= l0 && tid < l1) last = *((volatile long long *)&sums[tid + gl]);
                }
                below = warp_sum_ll(below);
                all = warp_sum_ll(all);
                if (BATCH) last = warp_sum_ll(last);
                if (lane == 0) {
                    wsum[w] = below;
                    wall[w] = all;
                    if (BATCH) wlast[w] = last;
                }
                __syncthreads();
            }
            long long base = 0, runs_first = 0, runs_last = 0;
#pragma unroll
            for (int i = 0; i < kFusedMaxBlocks / 32; ++i) {
                base += wsum[i];
                runs_first += wall[i];
                if (BATCH) runs_last += wlast[i];
            }
            runs = BATCH ? (long long)*((volatile unsigned long long *)&st->runs[it % 3]) : runs_first;
            // batches: `base` counts from the chunk's first vertex, `start` is its value at the
            // start of the current graph (the first graph's lies `base` runs before the chunk)
            long long start = BATCH ? -base : 0;
            if (BATCH) base = 0;
            bool emptied = true;  // the queue, in the round before
            for (int64_t vb = v0; vb < v1; vb += kRound) {
                if (vb > v0) load(x, vb);
                int incl[kPer];  // distinct labels of the warp's vertices up to and with this one
                int wtotal = 0;
#pragma unroll
                for (int u = 0; u < kPer; ++u) {
                    incl[u] = x[u].d;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int y = __shfl_up_sync(kFull, incl[u], o);
                        if (lane >= o) incl[u] += y;
                    }
                    incl[u] += wtotal;
                    wtotal = __shfl_sync(kFull, incl[u], 31);
                }
                __syncthreads();  // the sums of the round before are read
                if (lane == 31) wsum[w] = wtotal;
                if (tid == 0 && emptied) qn = 0;
                __syncthreads();
                long long before = base;
                for (int i = 0; i < kFusedWarps; ++i) {
                    if (i < w) before += wsum[i];
                    base += wsum[i];
                }
                // batches: the run base at the start of each vertex's graph.  The bases ascend, so it
                // is the largest of those of the graph starts up to the vertex.
                long long s0[kPer];
                if (BATCH) {
                    long long carry = LLONG_MIN;
#pragma unroll
                    for (int u = 0; u < kPer; ++u) {
                        const int64_t v = vb + (w * kPer + u) * 32 + lane;
                        const bool starts = v < v1 && v > v0 && x[u].g != x[u].gprev;
                        s0[u] = starts ? before + incl[u] - x[u].d : LLONG_MIN;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const long long y = __shfl_up_sync(kFull, s0[u], o);
                            if (lane >= o) s0[u] = max(s0[u], y);
                        }
                        s0[u] = max(s0[u], carry);
                        carry = __shfl_sync(kFull, s0[u], 31);
                    }
                    if (lane == 31) wall[w] = carry;
                    __syncthreads();
                    long long from = start;
                    for (int i = 0; i < kFusedWarps; ++i) {
                        if (i < w) from = max(from, wall[i]);
                        start = max(start, wall[i]);
                    }
#pragma unroll
                    for (int u = 0; u < kPer; ++u) s0[u] = max(s0[u], from);
                }
#pragma unroll
                for (int u = 0; u < kPer; ++u) {
                    const int64_t v = vb + (w * kPer + u) * 32 + lane;
                    const bool tied = x[u].d > 0 && (x[u].kw & 0xFFFF) > 1;
                    long long at = before + incl[u] - x[u].d, N = runs_first;
                    bool is_last = v == p.last_v, run = true;
                    if (BATCH && v < v1) {
                        const int j = x[u].g - gf;
                        run = j < kFusedThreads ? R.grun[j] != 0 : running(x[u].g, it);
                        if (tied) {
                            at -= s0[u];
                            N = x[u].g == gf ? runs_first
                                : x[u].g == gl ? runs_last
                                               : *((volatile long long *)&sums[b + x[u].g]);
                            is_last = v == __ldg(&p.g_last[x[u].g]);
                        }
                    }
                    int32_t nl = x[u].now;
                    bool queued = false;
                    if (tied) {
                        if (x[u].kw >= 0) {
                            const int q = atomicAdd(&qn, 1);
                            R.qv[q] = (int)v;
                            R.qa[q] = at;
                            if (BATCH) {
                                R.qN[q] = N;
                                R.qf[q] = (is_last ? 1 : 0) | (run ? 2 : 0);
                            }
                            queued = true;
                        } else {
                            int64_t from = -1;
                            nl = resolve_small(p, RunScope{at, N, is_last}, x[u].kw, x[u].d, x[u].c0, x[u].c1, x[u].r,
                                               x[u].o0, from);
                            if (from >= 0) nl = p.run_lab[from];
                            if (run) p.lab_out[v] = nl;
                            count_change(changes, nl, x[u].old);
                        }
                    }
                    if (BATCH) {
                        // a graph that has ended keeps its labels; the others count their changes
                        if (v < v1 && !queued && !run) p.lab_out[v] = x[u].old;
                        graph_changes(v < v1 && !queued && run && nl != x[u].old, x[u].g, it % 3);
                    }
                }
                __syncthreads();
                emptied = vb + kRound >= v1 || qn > Resolve::kQueue - kRound;  // block-uniform
                for (int q = w; emptied && q < qn; q += kFusedWarps) {
                    const int u = R.qv[q];
                    const RunScope rs{R.qa[q], BATCH ? R.qN[q] : runs_first, BATCH ? (R.qf[q] & 1) != 0 : u == p.last_v};
                    const bool run_u = !BATCH || (R.qf[q] & 2);
                    const int32_t ul = resolve_mid(p, u, rs, R.hist[w]);
                    if (lane == 0) {
                        const int32_t old = get_label<true>(&p.lab_in[u]);
                        p.lab_out[u] = run_u ? ul : old;
                        count_change(changes, ul, old);
                        if (BATCH && run_u && ul != old)
                            atomicAdd(&a.g_changes[(size_t)(it % 3) * p.ngraphs + __ldg(&p.gid[u])], 1ull);
                    }
                }
            }
        } else {
            runs = a.m;
            if (BATCH)  // the change counts per graph, zero since the barrier
                for (int64_t vb = (int64_t)b * kFusedThreads + w * 32; vb < a.n; vb += (int64_t)nb * kFusedThreads) {
                    const int64_t v = vb + lane;
                    const bool chg = v < a.n && get_label<true>(&p.lab_out[v]) != get_label<true>(&p.lab_in[v]);
                    graph_changes(chg, chg ? __ldg(&p.gid[v]) : 0, 0);
                }
        }
        {
            unsigned long long c = changes;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(kFull, c, o);
            if (lane == 0 && c) atomicAdd(&st->changes[it % 3], c);
        }
        if (!grid_barrier(a, ctl, &failed, ++barriers)) return;
        last_changes = (long long)*((volatile unsigned long long *)&st->changes[it % 3]);
        if (b == 0 && tid == 0 && it < 64) ctl->counts[it] = (unsigned long long)last_changes;
        ++it;
        if (BATCH) {
            int any = 0;
            for (int g = tid; g < p.ngraphs; g += kFusedThreads) any |= running(g, it);
            // the graph's keeper records its count; after that g_active may say what the count
            // already says
            any = __syncthreads_or(any);
            for (int g = b * kFusedThreads + tid; g < p.ngraphs; g += nb * kFusedThreads) {
                if (!a.g_active[g]) continue;
                a.g_counts[(size_t)g * a.g_max_iter + it - 1] =
                    (long long)a.g_changes[(size_t)((it - 1) % 3) * p.ngraphs + g];
                a.g_iters[g] = it;
                if (!running(g, it)) a.g_active[g] = 0;
            }
            if (!any || it >= a.niter) break;
        } else if (last_changes <= a.thr || it >= a.niter) {
            break;
        }
    }
    for (int i = 0; i < 3; ++i)
        for (int j = b + gf + tid; j <= b + gl; j += kFusedThreads) a.sums[(size_t)i * a.pieces + j] = 0;
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&st->left, 1u) == (unsigned)nb - 1) {  // the last block of the run
            st->left = 0;
            st->arrived = 0;
        }
        if (b == 0) {
            ctl->iter = it;
            ctl->N = runs;
            // (st->runs of other blocks' last read lies before the last barrier)
            for (int i = 0; i < 3; ++i) {
                st->runs[i] = 0;
                st->claimed[i] = 0;
            }
        }
    }
}

}  // namespace galp
