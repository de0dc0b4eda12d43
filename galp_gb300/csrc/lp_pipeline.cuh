// lp_pipeline.cuh -- count -> scan -> resolve: the exact label-propagation update
// without inter-block waiting.
//
// One iteration over a scope (whole graph, one out-of-core batch):
//
//   count   vertices are degree-bucketed and counted with no dependence between blocks:
//             small (degree <= 32, and degree 0): one lane per vertex, labels sorted in
//               registers (or one warp per pack of <= 32 label slots);
//             33..1024: a group of lanes per vertex, labels sorted in registers;
//             1025..12288: one CTA per vertex, shared-memory hash table;
//             big (> 12288): hash partitions (big_insert, hub_count, lp_kernels.cuh).
//           Each vertex gets its distinct-label count d; a vertex with a unique
//           most-frequent label is final and written at once.  A tied vertex leaves a
//           summary (smallest/largest candidate, their ranks, #candidates, max count)
//           and its (label, count) runs in a spill area at its own CSR positions.
//           Its d joins the sum of its block of vertices.
//   scan    exclusive scan of those sums (the run base of a vertex is the position of its
//           first run in the reference's run array,
//           label_propagation/src/dpp/kernel.cuh:66-82 scatter_indexes).
//   resolve goes over the vertices in order with their run bases: each tied vertex picks
//           its winner by the reference's positional tie rule (resolve_rank, lp_resolve.h)
//           from its summary, or from its spilled runs; those above 32 neighbours in a
//           kernel of their own, one warp each.
//
// Spill layout (indexed by CSR position relative to the scope's first entry):
//   run_lab[e0 + r] label, run_cnt[e0 + r] count of the vertex's r-th run; small vertices
//   write their sorted labels (or, counted in packs, their runs in label order), vertices
//   sorted by lane groups their runs in label order (kSpillSorted), CTA-table vertices
//   their table's occupied entries unsorted (queried by order statistics).
#pragma once

#include <utility>

#include "rmat_rng.h"
#include "lp_index.h"
#include "lp_kernels.cuh"
#include "lp_dispatch.cuh"

namespace galp {

constexpr int kMidSMax = 256;        // mid bucket: 33..256 neighbours
constexpr int kMidWarps = 8;         // warps (vertices) per CTA of count_mid_sort_kernel
constexpr int kRunBlock = 1024;      // vertices per sum of distinct counts, and per resolve block
constexpr int kLargeMax = 2048;      // large bucket: 257..2048; above 1024 one 256-thread CTA each
constexpr int kXlMax = 12288;        // xl bucket: 2049..12288, one CTA each (512 or 1024 threads)
constexpr int kXlSlots = 2 * kXlMax; // 192 KB of shared-memory table (64-bit slots)
constexpr int kXlThreads = 1024;
constexpr int kXlAMax = 6144;        // xl vertices up to here: 512-thread CTAs, 96 KB tables

struct PipeArgs {
    const int32_t *nbr;     // neighbour buffer holding CSR entries [nbr_shift, ...)
    int64_t nbr_shift;
    const int64_t *off;
    const int32_t *lab_in;
    int32_t *lab_out;
    Ctl *ctl;
    // static buckets of the scope
    const int32_t *pack_v0;
    const uint8_t *pack_nv;
    int32_t npacks;
    const int32_t *small_v; // the same vertices one by one, in order of degree within windows
    int32_t nsmall;
    const int32_t *mid_v;   // mid (33..256), then large (257..2048), then xl (2049..12288) vertices
    int32_t nmid_s, nmid_l, nmid_x;
    // per-vertex state (global vertex index)
    int32_t *dcnt;          // distinct labels
    int64_t *runbase;       // run base (in its scope or graph) of hubs and of listed tied vertices
    int32_t *sm_c0, *sm_c1; // smallest / largest candidate label
    int32_t *sm_kw;         // candidates | max count << 16 (| kSmallVertex or kSpillSorted)
    int32_t *sm_r;          // rank of smallest | rank of largest << 16
    // spill, indexed by CSR position - nbr_shift
    int32_t *run_lab;
    uint16_t *run_cnt;
    int32_t *tied_mid;      // tied vertices above 32 neighbours (listed by resolve_kernel)
    // scan
    int64_t v0, v1;         // scope vertices
    // distinct counts summed per block of kRunBlock vertices (batches: per piece of a block that
    // lies in one graph, see run_piece), zero between iterations; and their exclusive scan
    long long *sums;
    long long *run_at;
    long long *round_sum;   // sums of kScanRound sums each, where several blocks scan
    int32_t last_v;
    // frontier mode (null = every vertex is recounted and no changes are recorded)
    const uint8_t *dirty;   // 1 = a neighbour's label changed in the previous iteration
    int32_t *changed;       // vertices whose label changes in this iteration
    const DispatchState *disp;  // this iteration's variant (mid-list split, inserts, frontier)
    // batched mode (null g_v0 = one graph): graph g owns vertices [g_v0[g], g_v0[g+1]), its
    // own run positions (g_base[g] = run base of its first vertex), labels and last vertex
    const int64_t *g_v0;
    int64_t *g_base;
    const int32_t *g_active;          // 0: the graph has ended and keeps its labels
    unsigned long long *g_changes;    // labels changed per graph in this iteration
    const int32_t *g_last;
    const int32_t *gid;     // graph of every vertex
    int32_t ngraphs;
    int32_t lab27;          // every label below 2^27 - 1 (32-bit sort keys in packs)
    int32_t small_sort;     // small vertices: 0 match-based packs, 1 sort-based packs (needs lab27),
                            // 2 one thread per vertex, sorted in registers
    int32_t gcut[6];        // mid-list positions of the first vertex above 32 << i neighbours
    int32_t gstart;         // first mid-list position counted by lane groups (mid_sort: above 256)
};

constexpr int kSmallVertex = (int)0x80000000u;  // in sm_kw: at most 32 neighbours

// Run position scope of a vertex: its run base a, the scope's run count N, and whether it
// is the scope's last run-owning vertex (the whole graph, or its graph in batched mode).
struct RunScope {
    long long a, N;
    bool is_last;
};

// of vertex v, whose run base is a in the scope
__device__ __forceinline__ RunScope run_scope(const PipeArgs &p, int v, long long a)
{
    if (!p.g_v0) return RunScope{a, p.ctl->N, v == p.last_v};
    const int g = __ldg(&p.gid[v]);
    const long long base = p.g_base[g];
    return RunScope{a - base, p.g_base[g + 1] - base, v == p.g_last[g]};
}

__device__ __forceinline__ void count_change(unsigned long long &changes, int32_t nl, int32_t old)
{
    changes += (nl != old);
}

// Frontier mode and this iteration not switched to a full recount.
__device__ __forceinline__ bool frontier_on(const PipeArgs &p)
{
    return p.dirty && !*((volatile int *)&p.ctl->frontier_off);
}

// Loads of the current labels.  LIVE: the running kernel itself wrote them in an earlier phase
// (a grid-wide barrier lies between), so the non-coherent path must not be used.
template <bool LIVE>
__device__ __forceinline__ int32_t get_label(const int32_t *p)
{
    if constexpr (LIVE) {
        int32_t v;
        asm volatile("ld.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
        return v;
    } else {
        return __ldg(p);
    }
}
template <bool LIVE>
__device__ __forceinline__ int32_t gather_label(const int32_t *p)
{
    if constexpr (LIVE) {
        int32_t v;
        asm volatile("{\n\t.reg .b64 pol;\n\tcreatepolicy.fractional.L2::evict_last.b64 pol, 1.0;\n\t"
            "ld.global.L2::cache_hint.b32 %0, [%1], pol;\n\t}" : "=r"(v) : "l"(p));
        return v;
    } else {
        return ld_label(p);
    }
}

// The label of vertex id, INT_MAX where id < 0.  LIVE loads are volatile, so a condition around one
// would be a branch that the compiler moves no other load across: the condition is in the load.
template <bool LIVE>
__device__ __forceinline__ int32_t gather_label_if(const int32_t *lab, int id)
{
    if constexpr (LIVE) {
        int32_t v;
        asm volatile("{\n\t.reg .b64 pol;\n\t.reg .pred some;\n\tsetp.ge.s32 some, %2, 0;\n\tmov.b32 %0, 0x7fffffff;\n\t"
            "createpolicy.fractional.L2::evict_last.b64 pol, 1.0;\n\t"
            "@some ld.global.L2::cache_hint.b32 %0, [%1], pol;\n\t}" : "=&r"(v) : "l"(lab + id), "r"(id));
        return v;
    } else {
        return id >= 0 ? gather_label<false>(&lab[id]) : INT_MAX;
    }
}

// Record a changed vertex for the next iteration's frontier (single thread).
__device__ __forceinline__ void note_change(const PipeArgs &p, int32_t v, int32_t nl, int32_t old)
{
    if (p.changed && nl != old) p.changed[atomicAdd(&p.ctl->changed_n, 1)] = v;
}

__device__ __forceinline__ void flush_changes(unsigned long long changes, Ctl *ctl)
{
    unsigned long long c = changes;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) c += __shfl_xor_sync(kFull, c, off);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(&ctl->changes, c);
}

// Sum that vertex v's distinct count belongs to.  Blocks and graphs cut the vertices into
// pieces; block + graph numbers them in vertex order (with gaps, whose sums stay 0).
__device__ __forceinline__ int run_piece(const PipeArgs &p, int v)
{
    return (int)((v - p.v0) / kRunBlock) + (p.g_v0 ? __ldg(&p.gid[v]) : 0);
}

// Add a warp's distinct counts d (0 in lanes without one) to their sums.
__device__ __forceinline__ void add_runs(long long *sums, int piece, int d)
{
    const int c0 = __reduce_max_sync(kFull, d ? piece : 0);
    if (__all_sync(kFull, !d || piece == c0)) {
        const int all = __reduce_add_sync(kFull, d);
        if ((threadIdx.x & 31) == 0 && all) atomicAdd((unsigned long long *)&sums[c0], (unsigned long long)all);
    } else if (d) {
        atomicAdd((unsigned long long *)&sums[piece], (unsigned long long)d);
    }
}
__device__ __forceinline__ void add_runs(const PipeArgs &p, int v, int d)  // one thread
{
    atomicAdd((unsigned long long *)&p.sums[run_piece(p, v)], (unsigned long long)d);
}

// warp-aggregated append of the lanes with `pred` to list[ctr++]
__device__ __forceinline__ void warp_append(bool pred, int32_t value, int32_t *list, int *ctr)
{
    const unsigned m = __ballot_sync(kFull, pred);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    int base = 0;
    if (lane == __ffs(m) - 1) base = atomicAdd(ctr, __popc(m));
    base = __shfl_sync(kFull, base, __ffs(m) - 1);
    if (pred) list[base + __popc(m & ((1u << lane) - 1))] = value;
}

// Warp-private shared-memory buffer in front of a shared append-only list (the tied
// vertices above 32 neighbours): a warp appends with one ballot, and the buffer reaches the
// list with one global atomic per kWarpBuf entries instead of one per append.
constexpr int kWarpBuf = 64;
struct WarpBuf {
    int32_t *buf;  // kWarpBuf entries of this warp's shared memory
    int n = 0;     // warp-uniform fill
    __device__ void flush(int32_t *list, int *ctr)
    {
        if (!n) return;
        const int lane = threadIdx.x & 31;
        int base = 0;
        if (lane == 0) base = atomicAdd(ctr, n);
        base = __shfl_sync(kFull, base, 0);
        for (int i = lane; i < n; i += 32) list[base + i] = buf[i];
        __syncwarp();
        n = 0;
    }
    __device__ void append(bool pred, int32_t value, int32_t *list, int *ctr)
    {
        const unsigned m = __ballot_sync(kFull, pred);
        if (!m) return;
        if (n + __popc(m) > kWarpBuf) flush(list, ctr);
        const int lane = threadIdx.x & 31;
        if (pred) buf[n + __popc(m & ((1u << lane) - 1))] = value;
        n += __popc(m);
        __syncwarp();
    }
};

// warp-level version of note_change (all lanes call it)
__device__ __forceinline__ void warp_note_changes(const PipeArgs &p, bool changed, int32_t v)
{
    if (p.changed) warp_append(changed, v, p.changed, &p.ctl->changed_n);
}

// Per-vertex results of a counted pack: the values live at each vertex's first slot lane
// and move to the vertex lanes, which write the vertex state (all lanes call this).
__device__ __forceinline__ void finish_small_pack(const PipeArgs &p, bool vl, int v, int deg, int pos, int d, int k,
                                                  int W, int cmin, int cmax, int rmin, int rmax,
                                                  unsigned long long &changes)
{
    const int lane = threadIdx.x & 31;
    // results live at each vertex's first slot lane; bring them to the vertex lanes
    const int src = (vl && deg > 0) ? pos : lane;
    // d, k, W <= 32 and ranks < 32: one word
    const uint32_t packed = (uint32_t)d | ((uint32_t)k << 6) | ((uint32_t)W << 12) | ((uint32_t)rmin << 18) |
                            ((uint32_t)rmax << 23);
    const uint32_t pk_v = __shfl_sync(kFull, packed, src);
    const int d_v = (int)(pk_v & 63), k_v = (int)((pk_v >> 6) & 63), W_v = (int)((pk_v >> 12) & 63);
    const int r0_v = (int)((pk_v >> 18) & 31), r1_v = (int)((pk_v >> 23) & 31);
    const int c0_v = __shfl_sync(kFull, cmin, src);
    const int c1_v = __shfl_sync(kFull, cmax, src);
    const bool tied = vl && deg > 0 && k_v > 1;
    bool chg = false;
    if (vl) {
        p.dcnt[v] = deg > 0 ? d_v : 0;
        const int32_t old = __ldg(&p.lab_in[v]);
        if (deg > 0) p.sm_kw[v] = k_v | (W_v << 16) | kSmallVertex;
        if (!tied) {
            const int32_t nl = deg > 0 ? c0_v : old;
            p.lab_out[v] = nl;
            count_change(changes, nl, old);
            chg = nl != old;
        } else {
            p.sm_c0[v] = c0_v;
            p.sm_c1[v] = c1_v;
            p.sm_r[v] = r0_v | (r1_v << 16);
        }
    }
    add_runs(p.sums, vl && deg > 0 ? run_piece(p, v) : 0, vl && deg > 0 ? d_v : 0);
    warp_note_changes(p, chg, v);
}

// ---------------------------------------------------------------------------
// small vertices: one warp per pack
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256, 6) count_small_kernel(PipeArgs p)
{
    if (!ctl_active(p.ctl)) return;
    const bool fr = frontier_on(p);
    const int lane = threadIdx.x & 31;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    unsigned long long changes = 0;
    for (int pk = gw; pk < p.npacks; pk += nw) {
        const int v0 = p.pack_v0[pk], nv = p.pack_nv[pk];
        // vertex lanes: offsets, degrees, slot positions
        const bool vl = lane < nv;
        const int v = v0 + lane;
        if (fr && !__any_sync(kFull, vl && p.dirty[v])) {
            // no label around this pack changed: counts and summaries carry over; labels
            // of untied vertices stay, tied vertices are resolved again (run bases move)
            bool tied = false;
            if (vl && (__ldg(&p.off[v + 1]) > __ldg(&p.off[v]))) tied = (p.sm_kw[v] & 0xFFFF) > 1;
            if (vl && !tied) p.lab_out[v] = __ldg(&p.lab_in[v]);
            add_runs(p.sums, vl ? run_piece(p, v) : 0, vl ? p.dcnt[v] : 0);
            continue;
        }
        // The pack's CSR entries are contiguous: slot lane i holds entry obase + i.  Vertex
        // lanes read their offsets (an offset minus obase is the vertex's first slot lane);
        // the slot lanes of one vertex form a segment [first, last] found from the mask of
        // segment starts.
        const int64_t ol = __ldg(&p.off[v0 + min(lane, nv)]);
        const int64_t obase = __shfl_sync(kFull, ol, 0);
        const int64_t oend = nv < 32 ? __shfl_sync(kFull, ol, nv) : __ldg(&p.off[v0 + 32]);
        const int64_t onext = __shfl_down_sync(kFull, ol, 1);
        const int deg = vl ? (int)((lane == 31 ? oend : onext) - ol) : 0;
        const int pos = (int)(ol - obase);
        const int total = (int)(oend - obase);
        const bool valid = lane < total;
        const unsigned starts = __reduce_or_sync(kFull, (vl && deg > 0) ? (1u << pos) : 0u);
        const unsigned upto = (2u << lane) - 1u;  // lanes 0..lane
        const int j = valid ? 31 - __clz(starts & upto) : lane;  // segment id = its first lane
        const unsigned later_start = starts & ~upto;
        const int seg_last = valid ? (later_start ? __ffs(later_start) - 2 : total - 1) : lane;
        const int64_t oj = obase + j;  // the owner's first CSR entry
        int lab = 0;
        if (valid) lab = ld_label(&p.lab_in[ld_nbr(&p.nbr[obase + lane - p.nbr_shift])]);
        const unsigned vm = valid ? (((seg_last == 31) ? kFull : ((2u << seg_last) - 1u)) & ~((1u << j) - 1u))
                                  : (1u << lane);
        if (p.small_sort && p.lab27) {
            // Sort-based counting: sort the pack by (vertex lane << 27 | label) in one 32-bit
            // key (padding lanes last; a vertex keeps its slot lanes), then every run of equal
            // keys is one distinct label: heads give d, run lengths give counts, and
            // candidates come out in label order (cmin/cmax and their ranks by bit scans).
            uint32_t sk = valid ? (((uint32_t)j << 27) | (uint32_t)lab) : 0xFFFFFFFFu;
#pragma unroll
            for (int kk = 2; kk <= 32; kk <<= 1) {
#pragma unroll
                for (int jj = kk >> 1; jj > 0; jj >>= 1) {
                    const uint32_t ok = __shfl_xor_sync(kFull, sk, jj);
                    const bool up = (lane & kk) == 0, lower = (lane & jj) == 0;
                    sk = ((lower == up) ? (ok < sk) : (ok > sk)) ? ok : sk;
                }
            }
            const int first = __ffs(vm) - 1, last = 31 - __clz(vm);
            const int slab = (int)(sk & ((1u << 27) - 1));
            const uint32_t prevk = __shfl_up_sync(kFull, sk, 1);
            const bool head = valid && (lane == first || prevk != sk);
            const unsigned hm = __ballot_sync(kFull, head) & vm;
            const unsigned later = hm & ~((2u << lane) - 1u);
            const int cnt = head ? (later ? __ffs(later) - 1 : last + 1) - lane : 0;
            const int W = seg_max(cnt, lane, first, last);
            const unsigned cm = __ballot_sync(kFull, head && cnt == W) & vm;
            const int k = __popc(cm), d = __popc(hm);
            const int lo = cm ? __ffs(cm) - 1 : lane, hi = cm ? 31 - __clz(cm) : lane;
            const int cmin = __shfl_sync(kFull, slab, lo), cmax = __shfl_sync(kFull, slab, hi);
            const int rmin = __popc(hm & ((1u << lo) - 1)), rmax = __popc(hm & ((1u << hi) - 1));
            if (head && k > 2) {
                const int64_t e = oj - p.nbr_shift + __popc(hm & ((1u << lane) - 1));
                p.run_lab[e] = slab;
                p.run_cnt[e] = (uint16_t)cnt;
            }
            finish_small_pack(p, vl, v, deg, pos, d, k, W, cmin, cmax, rmin, rmax, changes);
            continue;
        }
        const unsigned eq = __match_any_sync(kFull, valid ? (uint32_t)lab : (0x80000000u | (uint32_t)lane)) & vm;
        const int cnt = __popc(eq);
        const bool leader = valid && ((__ffs(eq) - 1) == lane);
        const unsigned lm = __ballot_sync(kFull, leader);
        const int first = __ffs(vm) - 1, last = 31 - __clz(vm);
        const int W = seg_max(valid ? cnt : 0, lane, first, last);
        const bool cand = leader && cnt == W;
        const unsigned cm = __ballot_sync(kFull, cand);
        const int k = __popc(cm & vm);
        const int d = __popc(lm & vm);
        int cmin, cmax, rmin = 0, rmax = 0;
        if (__all_sync(kFull, !valid || k == 1)) {
            const unsigned m = cm & vm;
            cmin = cmax = __shfl_sync(kFull, lab, m ? (__ffs(m) - 1) : lane);
        } else {
            cmin = seg_min(cand ? lab : INT_MAX, lane, first, last);
            cmax = seg_max(cand ? lab : -1, lane, first, last);
            rmin = __popc(__ballot_sync(kFull, leader && lab < cmin) & vm);
            rmax = __popc(__ballot_sync(kFull, leader && lab < cmax) & vm);
            if (p.lab27 && __any_sync(kFull, valid && k > 2)) {
                // resolving a vertex with more than two candidates may need its runs in
                // label order: sort the pack by (vertex lane << 27 | label) in one 32-bit
                // key (labels below 2^27 - 1; padding lanes sort last), then spill the
                // runs of those vertices; run lengths come from the run heads
                uint32_t sk = valid ? (((uint32_t)j << 27) | (uint32_t)lab) : 0xFFFFFFFFu;
#pragma unroll
                for (int kk = 2; kk <= 32; kk <<= 1) {
#pragma unroll
                    for (int jj = kk >> 1; jj > 0; jj >>= 1) {
                        const uint32_t ok = __shfl_xor_sync(kFull, sk, jj);
                        const bool up = (lane & kk) == 0, lower = (lane & jj) == 0;
                        sk = ((lower == up) ? (ok < sk) : (ok > sk)) ? ok : sk;
                    }
                }
                const int slab = (int)(sk & ((1u << 27) - 1));
                const uint32_t prevk = __shfl_up_sync(kFull, sk, 1);
                const bool head = valid && (lane == first || prevk != sk);
                const unsigned hm = __ballot_sync(kFull, head) & vm;
                const int rank = __popc(hm & ((1u << lane) - 1));
                const unsigned later = hm & ~((2u << lane) - 1u);
                const int sc = (later ? __ffs(later) - 1 : last + 1) - lane;
                if (head && k > 2) {
                    const int64_t e = oj - p.nbr_shift + rank;
                    p.run_lab[e] = slab;
                    p.run_cnt[e] = (uint16_t)sc;
                }
            } else if (__any_sync(kFull, valid && k > 2)) {
                // labels of 27 bits or more: 64-bit (vertex, label) keys
                unsigned long long sk =
                    valid ? (((unsigned long long)(unsigned)j << 32) | (unsigned)lab) : (0xFFFFFFFF00000000ull | lane);
                int sc = valid ? cnt : 0;
#pragma unroll
                for (int kk = 2; kk <= 32; kk <<= 1) {
#pragma unroll
                    for (int jj = kk >> 1; jj > 0; jj >>= 1) {
                        const unsigned long long ok = __shfl_xor_sync(kFull, sk, jj);
                        const int oc = __shfl_xor_sync(kFull, sc, jj);
                        const bool up = (lane & kk) == 0, lower = (lane & jj) == 0;
                        if ((lower == up) ? (ok < sk) : (ok > sk)) {
                            sk = ok;
                            sc = oc;
                        }
                    }
                }
                const int slab = (int)(unsigned)sk;
                const int prev = __shfl_up_sync(kFull, slab, 1);
                const bool head = valid && (lane == first || prev != slab);
                const unsigned hm = __ballot_sync(kFull, head) & vm;
                const int rank = __popc(hm & ((1u << lane) - 1));
                if (head && k > 2) {
                    const int64_t e = oj - p.nbr_shift + rank;
                    p.run_lab[e] = slab;
                    p.run_cnt[e] = (uint16_t)sc;
                }
            }
        }
        finish_small_pack(p, vl, v, deg, pos, d, k, W, cmin, cmax, rmin, rmax, changes);
    }
    flush_changes(changes, p.ctl);
}

// ---------------------------------------------------------------------------
// mid, large and xl vertices: generation-tagged hash tables in shared memory
// ---------------------------------------------------------------------------
//
// A slot is one 64-bit word: generation (19 bits) | label (31 bits) | count (14 bits).
// Every vertex a table serves gets a new generation, so slots left by earlier vertices
// read as free and the table is never cleared between vertices; an insert either adds
// to the slot holding its label or claims a stale slot with one compare-and-swap.
// Degrees stay below 2^14 on these paths and labels below 2^31.
constexpr int kT64GenShift = 45;
constexpr uint32_t kT64GenMax = (1u << 19) - 1;
constexpr unsigned long long kT64CntMask = (1ull << 14) - 1;

__device__ __forceinline__ unsigned long long t64_tag(uint32_t gen, uint32_t label)
{
    return ((unsigned long long)gen << kT64GenShift) | ((unsigned long long)label << 14);
}

// Adds c occurrences of label.  Returns the label's count right after this insert and
// sets `claimed` when the insert took a new slot (the label's first insert).
__device__ __forceinline__ uint32_t t64_insert(unsigned long long *tab, uint32_t cap, uint32_t gen, uint32_t label,
                                               uint32_t c, bool &claimed)
{
    const unsigned long long tag = t64_tag(gen, label);
    uint32_t h = hslot(label, cap);
    // Plain loads: a slot that holds this vertex's generation never changes its label, and
    // a stale view of a free slot is caught by the compare-and-swap.
    unsigned long long cur = tab[h];
    for (;;) {
        if ((cur & ~kT64CntMask) == tag) {
            // the count is the low 14 bits of the low word (little-endian), and the total
            // stays below 2^14: a 32-bit add never carries into the label
            claimed = false;
            return (atomicAdd((unsigned int *)&tab[h], c) & (uint32_t)kT64CntMask) + c;
        }
        if ((uint32_t)(cur >> kT64GenShift) != gen) {  // stale: claim it
            const unsigned long long prev = atomicCAS(&tab[h], cur, tag | c);
            if (prev == cur) {
                claimed = true;
                return c;
            }
            cur = prev;  // taken meanwhile: look at it again
            continue;
        }
        h = (h + 1 == cap) ? 0 : h + 1;
        cur = tab[h];
    }
}

// Per-vertex summary: distinct labels d, maximum count W, number k of labels with count
// W and the smallest / largest of them.
struct Sum5 {
    int d, W, k, mn, mx;
};

__device__ __forceinline__ Sum5 sum5_empty() { return Sum5{0, 0, 0, INT_MAX, -1}; }

// Fold the count a label has right after one of its inserts (d is left to the caller).
// The counts a label passes through rise strictly and its last insert sees its final
// count, so folding every insert of a vertex gives its maximum count W, the number k
// of labels that reach W (each sees W exactly once) and their smallest and largest
// label, with no pass over the table; d is the number of slot claims.
__device__ __forceinline__ void sum5_observe(Sum5 &s, int lab, int c)
{
    if (c > s.W) {
        s.W = c;
        s.k = 1;
        s.mn = s.mx = lab;
    } else if (c == s.W) {
        s.k++;
        s.mn = min(s.mn, lab);
        s.mx = max(s.mx, lab);
    }
}

__device__ __forceinline__ Sum5 sum5_warp(const Sum5 &s)
{
    Sum5 r;
    r.W = __reduce_max_sync(kFull, s.W);
    const bool top = s.W == r.W;
    r.d = __reduce_add_sync(kFull, s.d);
    r.k = __reduce_add_sync(kFull, top ? s.k : 0);
    r.mn = __reduce_min_sync(kFull, top ? s.mn : INT_MAX);
    r.mx = __reduce_max_sync(kFull, top ? s.mx : -1);
    return r;
}

// Ranks of cmin and cmax among the vertex's distinct labels (partial counts).
__device__ __forceinline__ void t64_ranks(const unsigned long long *tab, int cap, int t0, int stride, uint32_t gen,
                                          int cmin, int cmax, int &a0, int &a1)
{
    a0 = a1 = 0;
    for (int i = t0; i < cap; i += stride) {
        const unsigned long long x = tab[i];
        if ((uint32_t)(x >> kT64GenShift) == gen) {
            const int lab = (int)((x >> 14) & 0x7FFFFFFF);
            a0 += lab < cmin;
            a1 += lab < cmax;
        }
    }
}

// Write the vertex's (label, count) entries, unsorted, to its spill positions; `ctr` is
// a shared counter the group has zeroed.
__device__ __forceinline__ void t64_spill(const unsigned long long *tab, int cap, int t0, int stride, uint32_t gen,
                                          int32_t *rl, uint16_t *rc, int *ctr)
{
    const int lane = threadIdx.x & 31;
    for (int i0 = t0 - lane; i0 < cap; i0 += stride) {  // warp-uniform trip count
        const int i = i0 + lane;
        const unsigned long long x = i < cap ? tab[i] : 0ull;
        const bool occ = i < cap && (uint32_t)(x >> kT64GenShift) == gen;
        const unsigned m = __ballot_sync(kFull, occ);
        if (!m) continue;
        int base = 0;
        if (lane == __ffs(m) - 1) base = atomicAdd(ctr, __popc(m));
        base = __shfl_sync(kFull, base, __ffs(m) - 1);
        if (occ) {
            const int at = base + __popc(m & ((1u << lane) - 1));
            rl[at] = (int32_t)((x >> 14) & 0x7FFFFFFF);
            rc[at] = (uint16_t)(x & kT64CntMask);
        }
    }
}

// Insert one row of gathered labels: lanes holding the same label add once when
// `aggregate` (heavy labels would otherwise serialise on one slot).  Each insert's
// observed count folds into `obs`; obs.d counts the claims.
__device__ __forceinline__ void t64_insert_row(unsigned long long *tab, uint32_t cap, uint32_t gen, uint32_t lb,
                                               bool aggregate, Sum5 &obs)
{
    uint32_t c = 1;
    bool mine = lb != kEmpty;
    if (aggregate) {
        const unsigned same = __match_any_sync(kFull, lb);
        mine = mine && (int)(threadIdx.x & 31) == __ffs(same) - 1;
        c = (uint32_t)__popc(same);
    }
    if (mine) {
        bool claimed;
        const uint32_t now = t64_insert(tab, cap, gen, lb, c, claimed);
        obs.d += claimed;
        sum5_observe(obs, (int)lb, (int)now);
    }
}

// Finish a counted vertex: per-vertex state, and its label unless it is tied.  One thread.
constexpr int kSpillSorted = 1 << 30;  // in sm_kw: the vertex's spilled runs are in label order
__device__ __forceinline__ void finish_counted(const PipeArgs &p, int v, const Sum5 &s, int rmin, int rmax,
                                               unsigned long long &changes, int32_t old, int flags = 0)
{
    p.dcnt[v] = s.d;
    p.sm_kw[v] = s.k | (s.W << 16) | flags;
    if (s.k == 1) {
        p.lab_out[v] = s.mn;
        count_change(changes, s.mn, old);
        note_change(p, v, s.mn, old);
        return;
    }
    p.sm_c0[v] = s.mn;
    p.sm_c1[v] = s.mx;
    p.sm_r[v] = rmin | (rmax << 16);
}

// Frontier: a clean vertex keeps its counts; it is re-resolved if tied, else keeps its
// label.  One thread.
__device__ __forceinline__ void carry_clean(const PipeArgs &p, int v)
{
    if ((p.sm_kw[v] & 0xFFFF) <= 1) p.lab_out[v] = __ldg(&p.lab_in[v]);
}

// ----- sorting networks in registers -----
// Batcher's odd-even merge sort (K. E. Batcher, "Sorting networks and their applications",
// 1968) for the next power of two, cut to the first N wires: the wires above would hold the
// largest keys and never exchange.  The comparators are compile-time constants, so a network
// is straight-line code of one min and one max per comparator.
struct NetPair {
    int a, b;
};
template <int N>
struct SortNet {
    static __host__ __device__ constexpr int pow2()
    {
        int p = 1;
        while (p < N) p *= 2;
        return p;
    }
    // the c-th comparator, or with c < 0 the number of comparators in .a
    static __host__ __device__ constexpr NetPair get(int c)
    {
        const int P = pow2();
        int at = 0;
        for (int p = 1; p < P; p *= 2)
            for (int k = p; k >= 1; k /= 2)
                for (int j = k % p; j + k < P; j += 2 * k)
                    for (int i = 0; i < k && i + j + k < P; ++i)
                        if ((i + j) / (2 * p) == (i + j + k) / (2 * p) && i + j + k < N) {
                            if (at == c) return NetPair{i + j, i + j + k};
                            ++at;
                        }
        return NetPair{at, 0};
    }
    static constexpr int size = get(-1).a;
    template <int C>
    static __device__ __forceinline__ void step(int32_t (&x)[N])
    {
        constexpr NetPair q = get(C);
        const int32_t lo = min(x[q.a], x[q.b]), hi = max(x[q.a], x[q.b]);
        x[q.a] = lo;
        x[q.b] = hi;
    }
    template <int... C>
    static __device__ __forceinline__ void steps(int32_t (&x)[N], std::integer_sequence<int, C...>)
    {
        (step<C>(x), ...);
    }
    static __device__ __forceinline__ void sort(int32_t (&x)[N])
    {
        steps(x, std::make_integer_sequence<int, size>{});
    }
};

// Sort the first N words of a lane's row in registers, write them back and return the mask
// of positions that differ from the one before (position 0 always set).
template <int N>
__device__ __forceinline__ uint32_t small_sort_row(int32_t *row)
{
    int32_t x[N];
#pragma unroll
    for (int j = 0; j < N; j += 4) {
        const int4 q = *reinterpret_cast<const int4 *>(row + j);
        x[j] = q.x;
        x[j + 1] = q.y;
        x[j + 2] = q.z;
        x[j + 3] = q.w;
    }
    SortNet<N>::sort(x);
    uint32_t h = 1u;
#pragma unroll
    for (int j = 1; j < N; ++j)
        if (x[j] != x[j - 1]) h |= 1u << j;
#pragma unroll
    for (int j = 0; j < N; j += 4) *reinterpret_cast<int4 *>(row + j) = make_int4(x[j], x[j + 1], x[j + 2], x[j + 3]);
    return h;
}

// Order every window of kSmallWindow entries of a scope's small-vertex list by degree
// (stable), once per graph: a warp's 32 vertices then have about equal degrees, while their
// neighbour lists and per-vertex outputs stay within the window's few cache lines.
constexpr int kSmallWindow = 128;
__global__ void __launch_bounds__(kSmallWindow) small_window_kernel(int32_t *small_v, int nsmall, const int64_t *off)
{
    __shared__ uint8_t sdeg[kSmallWindow];
    const int tid = threadIdx.x;
    for (int64_t w0 = (int64_t)blockIdx.x * kSmallWindow; w0 < nsmall; w0 += (int64_t)gridDim.x * kSmallWindow) {
        const int cnt = (int)min((int64_t)kSmallWindow, nsmall - w0);
        int v = 0, deg = 0;
        if (tid < cnt) {
            v = small_v[w0 + tid];
            deg = (int)(off[v + 1] - off[v]);
            sdeg[tid] = (uint8_t)deg;
        }
        __syncthreads();
        if (tid < cnt) {
            int r = 0;
            for (int i = 0; i < cnt; ++i) r += sdeg[i] < deg || (sdeg[i] == deg && i < tid);
            small_v[w0 + r] = v;
        }
        __syncthreads();
    }
}

// Row of a small vertex in its warp's shared memory: 36 words, so that the 16-byte accesses
// of 8 lanes to their own rows fall in distinct banks.
constexpr int kSmallRow = 36;

// ----- a warp's tile of sorted rows -----
//
// One tile: the labels of up to 32 vertices (1024 CSR entries), gathered together into the
// warp's shared memory.  The entries of the tile's vertices follow one another in slots; a
// warp copies 32 slots at a time, whatever vertices they belong to, and the owner of a slot
// follows from the mask of vertex starts in its row of slots.
struct TileBuf {
    int32_t rows[32 * kSmallRow];  // per lane: its labels, padded with INT_MAX
    int64_t dlt[32];        // i-th vertex to count: CSR position minus slot
    int32_t at[32];         // its row's first word minus its first slot
    uint2 info[32];         // row of slots: mask of vertex starts, starts in earlier rows
    // index of the vertex that owns the lane's slot in a row (lanes past the tile's total: any)
    __device__ __forceinline__ int owner(int row) const
    {
        const uint2 q = info[row];
        return (int)q.y + __popc(q.x & ((2u << (threadIdx.x & 31)) - 1u)) - 1;
    }
};

// Gather a tile of one vertex per lane: the lane's `deg` labels, whose first entry is at e0
// of the neighbour buffer, go to its row, padded to n words (a multiple of 4).
// SLIM (where registers are short): a row's labels are stored before the next row's are loaded.
template <bool LIVE, bool SLIM>
__device__ __forceinline__ void tile_gather(const PipeArgs &p, TileBuf &B, int deg, int64_t e0, int n)
{
    const int lane = threadIdx.x & 31;
    int pos = deg;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, pos, o);
        if (lane >= o) pos += y;
    }
    const int total = __shfl_sync(kFull, pos, 31);
    pos -= deg;
    B.info[lane] = make_uint2(0u, 0u);
    const unsigned nz = __ballot_sync(kFull, deg > 0);
    const int rank = __popc(nz & ((1u << lane) - 1u));
    __syncwarp();
    if (deg > 0) {
        B.dlt[rank] = e0 - pos;
        B.at[rank] = lane * kSmallRow - pos;
        atomicOr(&B.info[pos >> 5].x, 1u << (pos & 31));
    }
    for (int j = 0; j < n; j += 4)
        *reinterpret_cast<int4 *>(B.rows + lane * kSmallRow + j) = make_int4(INT_MAX, INT_MAX, INT_MAX, INT_MAX);
    __syncwarp();
    const int starts = __popc(B.info[lane].x);
    int before = starts;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, before, o);
        if (lane >= o) before += y;
    }
    B.info[lane].y = (uint32_t)(before - starts);
    __syncwarp();
    constexpr int PER = 8;  // rows in flight
    for (int r0 = 0; r0 * 32 < total; r0 += PER) {
        int id[PER], at[PER];
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            id[u] = -1;
            if ((r0 + u) * 32 >= total) continue;  // warp-uniform
            const int s = (r0 + u) * 32 + lane;
            const int own = B.owner(r0 + u);
            if (s < total) {
                id[u] = ld_nbr(&p.nbr[B.dlt[own] + s]);
                at[u] = B.at[own] + s;
            }
        }
        if constexpr (SLIM) {
#pragma unroll
            for (int u = 0; u < PER; ++u)
                if (id[u] >= 0) B.rows[at[u]] = gather_label<LIVE>(&p.lab_in[id[u]]);
        } else {  // all loads before the first store: the warp waits once for the eight rows
            int32_t lb[PER];
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                if (LIVE && (r0 + u) * 32 >= total) continue;  // warp-uniform
                lb[u] = gather_label_if<LIVE>(p.lab_in, id[u]);
            }
#pragma unroll
            for (int u = 0; u < PER; ++u)
                if (id[u] >= 0) B.rows[at[u]] = lb[u];
        }
    }
    __syncwarp();
}

// What a lane needs of its vertex before counting it: loaded one tile ahead.
struct TileHead {
    int v, deg, g;  // vertex (-1 = none), its neighbours, log2 of its lanes
    int64_t o0;     // first CSR entry
    int32_t old;    // current label
    int dirty;      // 0: frontier mode and no neighbour label changed
};

template <bool LIVE>
__device__ __forceinline__ void tile_head(const PipeArgs &p, TileHead &h, int v, bool fr)
{
    h.v = v;
    h.o0 = __ldg(&p.off[v]);
    h.deg = (int)(__ldg(&p.off[v + 1]) - h.o0);
    h.old = get_label<LIVE>(&p.lab_in[v]);
    h.dirty = fr ? (int)p.dirty[v] : 1;
}

// Plan of a tile that a warp counts again and again: word j * 32 + lane is the neighbour whose
// label is the j-th of the lane's row, -1 = none.
constexpr int kPlanWords = 32 * 32;

// Fill the rows (`stride` words apart) by a plan, the first n labels of each (a multiple of 4),
// PER of them in flight.
template <int PER>
__device__ __forceinline__ void plan_gather(const PipeArgs &p, const int32_t *plan, int32_t *rows, int stride, int n)
{
    const int lane = threadIdx.x & 31;
    for (int j0 = 0; j0 < n; j0 += PER) {
        int32_t x[PER];
#pragma unroll
        for (int u = 0; u < PER; ++u) x[u] = j0 + u < n ? plan[(j0 + u) * 32 + lane] : -1;
#pragma unroll
        for (int u = 0; u < PER; ++u) x[u] = gather_label_if<true>(p.lab_in, x[u]);
#pragma unroll
        for (int u = 0; u < PER; u += 4)
            if (j0 + u < n)
                *reinterpret_cast<int4 *>(rows + lane * stride + j0 + u) = make_int4(x[u], x[u + 1], x[u + 2], x[u + 3]);
    }
    __syncwarp();
}

// A lane's at most 4 labels, gathered by itself and sorted into its row; the mask of run heads as
// small_sort_row.  Lanes of a tile lie close together in the neighbour list, and setting up the
// common gather costs more than the gather: ten iterations over 20 M vertices in pairs 3.6 -> 2.8 ms
// in this kernel, in a ring 4.0 -> 3.2, in a torus 5.1 -> 3.7, with two random neighbours 6.1 -> 6.3.
__device__ __forceinline__ uint32_t small_direct_row(const PipeArgs &p, int32_t *row, int deg, int64_t e0)
{
    int id[4];
    int32_t x[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) id[j] = j < deg ? ld_nbr(&p.nbr[e0 + j]) : -1;
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = gather_label_if<false>(p.lab_in, id[j]);
    SortNet<4>::sort(x);
    *reinterpret_cast<int4 *>(row) = make_int4(x[0], x[1], x[2], x[3]);
    return 1u | (x[1] != x[0] ? 2u : 0u) | (x[2] != x[1] ? 4u : 0u) | (x[3] != x[2] ? 8u : 0u);
}

// Count the warp's 32 small vertices (one per lane), with the tile buffer B (PLAN: rows in flight
// by the tile's plan, 0 = it has none).  Writes their state and the labels of untied ones (chg: it
// changed); returns the lane's distinct count.
//
// Kernels that keep plans have few tiles per warp, and the straight-line code of the networks is
// mostly fetched for one tile: they use fewer of them (rows of 8, 16, 24, 32; group rows of 32).
// Passes with all networks and with these (us): R-MAT 14 188 and 176, R-MAT 17 with edge factor 4
// 297 and 277, LFR of 1.9 M entries 357 and 331.  R-MAT 24, whose warps run the same code over and
// over, would lose: 49.9 and 50.6 ms.
template <bool LIVE, int PLAN = 0>
__device__ __forceinline__ int small_tile(const PipeArgs &p, TileBuf &B, const TileHead &hd,
                                          unsigned long long &changes, bool &chg, const int32_t *plan = nullptr)
{
    const int lane = threadIdx.x & 31;
    const int v = hd.v;
    const int deg = (v >= 0 && hd.dirty) ? hd.deg : 0;  // neighbours to count
    constexpr bool FEW = PLAN > 0;
    int n4 = (__reduce_max_sync(kFull, deg) + 3) >> 2;
    if (FEW) n4 = (n4 + 1) & ~1;
    const bool direct = !LIVE && n4 <= 1;  // every lane gathers its own
    if (PLAN && plan) plan_gather<PLAN ? PLAN : 4>(p, plan, B.rows, kSmallRow, 4 * n4);
    else if (!direct) tile_gather<LIVE, LIVE && PLAN == 0>(p, B, deg, hd.o0 - p.nbr_shift, 4 * n4);
    int32_t *row = B.rows + lane * kSmallRow;
    uint32_t h = 0u;
    if (!LIVE && direct) h = small_direct_row(p, row, deg, hd.o0 - p.nbr_shift);
    else switch (n4) {  // warp-uniform
    case 0: break;
    case 1: if (!FEW) h = small_sort_row<4>(row); break;
    case 2: h = small_sort_row<8>(row); break;
    case 3: if (!FEW) h = small_sort_row<12>(row); break;
    case 4: h = small_sort_row<16>(row); break;
    case 5: if (!FEW) h = small_sort_row<20>(row); break;
    case 6: h = small_sort_row<24>(row); break;
    case 7: if (!FEW) h = small_sort_row<28>(row); break;
    default: h = small_sort_row<32>(row); break;
    }
    const uint32_t valid = deg >= 32 ? kFull : (1u << deg) - 1u;
    h &= valid;
    const uint32_t cont = ~h & valid;
    // heads of runs of at least W labels: such a run has W - 1 continuations behind its head
    uint32_t m = h;
    int W = 1;
    for (;;) {
        const uint32_t t = m & __funnelshift_rc(cont, 0u, W);  // a shift of 32 gives 0
        if (!t) break;
        m = t;
        ++W;
    }
    const int k = __popc(m);
    chg = false;
    if (v >= 0) {
        if (!hd.dirty) {
            // no label around the vertex changed: its counts carry over
            if (hd.deg == 0 || (p.sm_kw[v] & 0xFFFF) <= 1) p.lab_out[v] = hd.old;
        } else if (deg == 0) {
            p.dcnt[v] = 0;
            p.lab_out[v] = hd.old;
        } else {
            p.dcnt[v] = __popc(h);
            p.sm_kw[v] = k | (W << 16) | kSmallVertex;
            if (k == 1) {
                const int32_t nl = row[__ffs(m) - 1];
                p.lab_out[v] = nl;
                count_change(changes, nl, hd.old);
                chg = nl != hd.old;
            } else {
                const int lo = __ffs(m) - 1, hi = 31 - __clz(m);
                p.sm_c0[v] = k == 2 ? row[lo] : (int32_t)h;
                p.sm_c1[v] = k == 2 ? row[hi] : (int32_t)m;
                p.sm_r[v] = __popc(h & ((1u << lo) - 1u)) | (__popc(h & ((1u << hi) - 1u)) << 16);
            }
        }
    }
    unsigned spill = __ballot_sync(kFull, k > 2);
    if (PLAN && plan) {
        // one vertex after the other (the owners of slots are not at hand)
        __syncwarp();  // every lane's row is sorted (the vote does not order shared memory)
#pragma unroll 1
        while (spill) {
            const int src = __ffs(spill) - 1;
            spill &= spill - 1;
            const int64_t e = __shfl_sync(kFull, hd.o0 - p.nbr_shift, src);
            const int dg = __shfl_sync(kFull, deg, src);
            if (lane < dg) p.run_lab[e + lane] = B.rows[src * kSmallRow + lane];
        }
    } else if (direct) {
        if (k > 2)
            for (int j = 0; j < deg; ++j) p.run_lab[hd.o0 - p.nbr_shift + j] = row[j];
    } else if (spill) {
        const int total = __reduce_add_sync(kFull, deg);
        const unsigned nz = __ballot_sync(kFull, deg > 0);
        if (deg > 0 && k <= 2) B.dlt[__popc(nz & ((1u << lane) - 1u))] = LLONG_MIN;
        __syncwarp();
        for (int r = 0; r * 32 < total; ++r) {
            const int s = r * 32 + lane;
            const int own = B.owner(r);
            if (s < total) {
                const int64_t e = B.dlt[own];
                if (e != LLONG_MIN) p.run_lab[e + s] = B.rows[B.at[own] + s];
            }
        }
    }
    __syncwarp();  // the tile buffer may be written again
    return __popc(h);
}

// Small vertices (at most 32 neighbours; `small_sort` 2): a warp takes 32 vertices of about
// equal degree (small_window_kernel), gathers their labels together and sorts each vertex's
// labels in one lane's registers.
//
//   gather  32 CSR entries per row whatever vertices they belong to, eight rows in flight;
//           the owner of an entry follows from the mask of vertex starts in its row; labels
//           go to the owner's row of shared memory (padded with INT_MAX, no label).  Tiles of
//           at most four neighbours each: small_direct_row.
//   sort    a network sized to the warp's largest degree in steps of 4; the mask h of run
//           heads gives everything else: d = popc(h), and the heads m of runs of maximum
//           length W by W steps of m & (continuations >> W).
//   spill   vertices with more than two candidates keep their sorted labels at their CSR
//           positions and h, m in place of the candidate labels (SmallMaskQuery).
//
// Bound by the load/store pipe (70 % of its wavefronts on planted partitions of degree 15:
// the label gathers alone are 32 per row), then by the latency of the two dependent loads.
// A warp has the order of its vertices to itself, so there is no barrier between warps: a
// version that ordered 128 vertices inside the block, with three barriers and per-lane
// result selects, took 42 ms where this one takes 25.  Ten iterations, this kernel's share
// (an insertion sort per thread in shared memory before): 1,024 planted partitions of
// together 526 M entries 55.5 -> 24.9 ms, R-MAT 24 9.8 -> 4.4 ms, R-MAT 26 with edge
// factor 4 20.2 -> 11.5 ms, LFR of a million vertices 2.0 -> 0.73 ms.
constexpr int kSmallThreads = 128;
constexpr int kSmallBlocks = 8;  // resident blocks per SM
__global__ void __launch_bounds__(kSmallThreads, kSmallBlocks) count_small_sort_kernel(PipeArgs p)
{
    constexpr int NW = kSmallThreads / 32;
    __shared__ __align__(16) TileBuf stile[NW];
    __shared__ int32_t cbuf[NW][kWarpBuf];
    if (!ctl_active(p.ctl)) return;
    const bool fr = frontier_on(p);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned long long changes = 0;
    WarpBuf cb{cbuf[w]};  // changed vertices (frontier mode)
    // a block takes NW * 32 list entries per round; its warps take the quarters of a degree
    // window in turn, so that none has only the window's highest degrees
    ListWalk walk(blockIdx.x, gridDim.x, kSmallThreads, p.nsmall);
    int turn = w;
    auto head = [&](int rounds) {
        TileHead h{-1, 0, 0, 0, 0, 1};
        const int i = walk.entry(rounds, turn * 32 + lane);
        if (i >= 0) tile_head<false>(p, h, p.small_v[i], fr);
        turn = (turn + 1) & (NW - 1);
        return h;
    };
    TileHead nxt = head(0);
    for (; walk.more(); walk.next()) {
        const TileHead hd = nxt;
        nxt = head(1);
        bool chg;
        int d = small_tile<false>(p, stile[w], hd, changes, chg);
        if (!hd.dirty) d = p.dcnt[hd.v];
        add_runs(p.sums, d ? run_piece(p, hd.v) : 0, d);
        if (p.changed) cb.append(chg, hd.v, p.changed, &p.ctl->changed_n);
    }
    if (p.changed) cb.flush(p.changed, &p.ctl->changed_n);
    flush_changes(changes, p.ctl);
}

// What a warp or CTA needs of a mid-list vertex before counting it: loaded one vertex ahead, so
// these dependent loads (list entry, then offsets and state) are in flight while the
// previous vertex is counted.
struct CtaHead {
    int v;         // vertex, -1 past the end of the range
    int deg;
    int64_t o0;    // first CSR entry
    int dcnt;      // distinct labels in the previous iteration (aggregation rule)
    int32_t old;   // current label
    int dirty;     // 0: frontier mode and no neighbour label changed
};

__device__ __forceinline__ CtaHead cta_head(const PipeArgs &p, int first, int i, int count, bool fr)
{
    CtaHead h{-1, 0, 0, 0, 0, 1};
    if (i < count) {
        h.v = p.mid_v[first + i];
        h.o0 = __ldg(&p.off[h.v]);
        h.deg = (int)(__ldg(&p.off[h.v + 1]) - h.o0);
        h.dcnt = p.dcnt[h.v];
        h.old = __ldg(&p.lab_in[h.v]);
        h.dirty = fr ? (int)p.dirty[h.v] : 1;
    }
    return h;
}

// ----- vertices of 33..1024 neighbours sorted by groups of lanes -----

// Sort x[OFF .. OFF + CNT), a bitonic sequence, within a lane: half-cleaners while the length
// is even (they hold for any even length), a sorting network for an odd rest.
template <int OFF, int CNT, int N, int... C>
__device__ __forceinline__ void bitonic_rest(int32_t (&x)[N], std::integer_sequence<int, C...>)
{
    ((void)[&] {
        constexpr NetPair q = SortNet<CNT>::get(C);
        const int32_t lo = min(x[OFF + q.a], x[OFF + q.b]), hi = max(x[OFF + q.a], x[OFF + q.b]);
        x[OFF + q.a] = lo;
        x[OFF + q.b] = hi;
    }(), ...);
}

template <int OFF, int CNT, int N>
__device__ __forceinline__ void bitonic_lane(int32_t (&x)[N])
{
    if constexpr (CNT > 1 && CNT % 2 == 0) {
#pragma unroll
        for (int j = 0; j < CNT / 2; ++j) {
            const int32_t lo = min(x[OFF + j], x[OFF + j + CNT / 2]), hi = max(x[OFF + j], x[OFF + j + CNT / 2]);
            x[OFF + j] = lo;
            x[OFF + j + CNT / 2] = hi;
        }
        bitonic_lane<OFF, CNT / 2>(x);
        bitonic_lane<OFF + CNT / 2, CNT / 2>(x);
    } else if constexpr (CNT > 1) {
        bitonic_rest<OFF, CNT>(x, std::make_integer_sequence<int, SortNet<CNT>::size>{});
    }
}

// A lane's number of labels N, the words from its row to the next lane's (16-byte accesses of
// 8 lanes to their own rows fall in distinct banks) and j / N as j * rcp >> 16 (j < 32 N).
struct GroupShape {
    int N, stride, rcp;
};
__host__ __device__ constexpr GroupShape group_shape(int N)
{
    return N == 20   ? GroupShape{20, 20, 3277}
           : N == 24 ? GroupShape{24, 28, 2731}
                     : GroupShape{32, 36, 2048};
}

// Sort the N words of every lane's row over groups of 2^g consecutive lanes (lane-major
// order), write the rows back and return the lane's mask of positions that differ from
// the one before (the group's first position always set).  Each lane sorts its row, then
// level L merges pairs of sorted runs of 2^(L-1) lanes: a flip against the mirrored lane,
// half-cleaners between lanes, and the bitonic rest within the lane.
template <int N>
__device__ __forceinline__ uint32_t group_sort_rows(int32_t *rows, int g)
{
    const int lane = threadIdx.x & 31;
    int32_t *row = rows + lane * group_shape(N).stride;
    int32_t x[N];
#pragma unroll
    for (int j = 0; j < N; j += 4) {
        const int4 q = *reinterpret_cast<const int4 *>(row + j);
        x[j] = q.x;
        x[j + 1] = q.y;
        x[j + 2] = q.z;
        x[j + 3] = q.w;
    }
    SortNet<N>::sort(x);
#pragma unroll 1
    for (int L = 1; L <= g; ++L) {
        const int flip = (1 << L) - 1;
        bool low = !(lane & (1 << (L - 1)));
#pragma unroll
        for (int j = 0; j < N / 2; ++j) {
            const int32_t a = __shfl_xor_sync(kFull, x[N - 1 - j], flip), b = __shfl_xor_sync(kFull, x[j], flip);
            x[j] = low ? min(x[j], a) : max(x[j], a);
            x[N - 1 - j] = low ? min(x[N - 1 - j], b) : max(x[N - 1 - j], b);
        }
#pragma unroll 1
        for (int D = 1 << (L - 1) >> 1; D >= 1; D >>= 1) {
            low = !(lane & D);
#pragma unroll
            for (int j = 0; j < N; ++j) {
                const int32_t a = __shfl_xor_sync(kFull, x[j], D);
                x[j] = low ? min(x[j], a) : max(x[j], a);
            }
        }
        bitonic_lane<0, N>(x);
    }
    const int32_t before = __shfl_up_sync(kFull, x[N - 1], 1);
    uint32_t h = (lane & ((1 << g) - 1)) == 0 || x[0] != before ? 1u : 0u;
#pragma unroll
    for (int j = 1; j < N; ++j)
        if (x[j] != x[j - 1]) h |= 1u << j;
#pragma unroll
    for (int j = 0; j < N; j += 4) *reinterpret_cast<int4 *>(row + j) = make_int4(x[j], x[j + 1], x[j + 2], x[j + 3]);
    return h;
}

// Move the run heads (mask h) of every lane's row to the front of its group's rows, in order
// (the lane's first head has rank `at` in the group), candidates (mask m) with the sign bit set.
template <int N>
__device__ __forceinline__ void group_compact(int32_t *rows, int g, uint32_t h, uint32_t m, int at)
{
    constexpr int stride = group_shape(N).stride;
    const int lane = threadIdx.x & 31;
    int32_t x[N];
#pragma unroll
    for (int j = 0; j < N; j += 4) {
        const int4 q = *reinterpret_cast<const int4 *>(rows + lane * stride + j);
        x[j] = q.x;
        x[j + 1] = q.y;
        x[j + 2] = q.z;
        x[j + 3] = q.w;
    }
    __syncwarp();
    int32_t *out = rows + (lane >> g << g) * stride + at;
#pragma unroll
    for (int j = 0; j < N; ++j)
        if ((h >> j) & 1u) *out++ = x[j] | (int32_t)(((m >> j) & 1u) << 31);
    __syncwarp();
}

// One warp per tile of 32 / G vertices of the degree-sorted mid list, G = 2^g lanes each,
// where 16 G < degree <= 32 G: g = 1 (33..64 neighbours) to 5 (513..1024).  The labels are
// gathered in rows of 32, spread over the group's lanes, N = 20, 24 or 32 labels each (the
// smallest that holds the tile's largest degree), and sorted across the group; run lengths
// come from the lanes' head masks, with the part of a run that goes on into later lanes
// added to its head's lane.  Vertices with more than two candidates spill their runs in
// label order, with the maximum count for candidates and 0 for others.
//
// About 4.5 warp instructions per entry in tie-heavy iterations, none of them divergent or
// behind a barrier, where tables in shared memory (one warp, 64 or 128 threads per vertex)
// took 8 to 10 at 13 to 22 active lanes; half of them are the networks' minima and maxima,
// which run at half rate.  Ten iterations of R-MAT 24: 20.0 -> 16.6 ms here (15.6 since all
// eight rows of a gather are loaded before the first is stored) and, the spilled runs being in
// order, 2.6 -> 0.85 ms in resolve_mid; R-MAT 26 with edge factor 4: 28.9 -> 23.2 and 6.0 -> 1.8.
// Longer lists stay with the tables: a warp sorting 2048 labels, 64 to
// a lane, gained 16 % where there are tens of thousands of such vertices and lost 80 % where
// there are a few (one warp then takes 27 us for one).  Labels brought in by asynchronous
// copies, the next tile's during the sort, were slower (4-byte copies run at half the rate
// of loads: 17.1 ms here, and 33 instead of 25 for the small vertices above).
constexpr int kGroupMax = 1024;
struct GroupBuf {
    int32_t rows[32 * 36];
    int64_t ent[16];  // the tile's vertices: first entry in the neighbour buffer,
    int32_t deg[16];  // labels to gather
};

// The classes' list ranges and tiles, largest degrees first: tile t of a class g is the one with
// upto[g + 1] <= t < upto[g], list entries first[g] + (t - upto[g + 1]) * (32 >> g) ...
struct GroupTiles {
    int first[6], last[6], upto[7];
    __device__ void set(const PipeArgs &p, int pos1)  // one thread
    {
        int tiles = 0;
        for (int g = 5; g >= 1; --g) {
            const int f = max(p.gcut[g - 1], p.gstart), l = min(p.gcut[g], pos1), per = 32 >> g;
            tiles += (max(l - f, 0) + per - 1) / per;
            first[g] = f;
            last[g] = l;
            upto[g] = tiles;
        }
        upto[6] = 0;
    }
    __device__ __forceinline__ int count() const { return upto[1]; }
};

template <bool LIVE>
__device__ __forceinline__ TileHead group_head(const PipeArgs &p, const GroupTiles &T, int t, bool fr)
{
    TileHead h{-1, 0, 1, 0, 0, 1};
    if (t < T.count()) {
        h.g = 5;
        while (t >= T.upto[h.g]) --h.g;
        const int i = T.first[h.g] + (t - T.upto[h.g + 1]) * (32 >> h.g) + ((int)(threadIdx.x & 31) >> h.g);
        if (i < T.last[h.g]) tile_head<LIVE>(p, h, p.mid_v[i], fr);
    }
    return h;
}

// The shape for a tile whose lanes belong to vertices of `deg` labels to count.  FEW: one length
// for all, 32 labels per lane.
template <bool FEW>
__device__ __forceinline__ GroupShape group_shape_of(int deg, int g)
{
    if (FEW) return group_shape(32);
    const int n = (__reduce_max_sync(kFull, deg) + (1 << g) - 1) >> g;
    return n <= 20 ? group_shape(20) : n <= 24 ? group_shape(24) : group_shape(32);
}

// Count the warp's tile of vertices (one per group of lanes; PLAN and plan as for small tiles).
// Writes their state and the labels of untied ones; returns the group's distinct count.
template <bool LIVE, int PLAN = 0>
__device__ __forceinline__ int group_tile(const PipeArgs &p, GroupBuf &B, const TileHead &hd,
                                          unsigned long long &changes, const int32_t *plan = nullptr)
{
    const int lane = threadIdx.x & 31;
    int32_t *rows = B.rows;
    const int v = hd.v, g = hd.g, G = 1 << g, sub = lane & (G - 1);
    const bool leader = sub == 0;
    const int deg = (v >= 0 && hd.dirty) ? hd.deg : 0;  // neighbours to count
    constexpr bool FEW = PLAN > 0;
    const GroupShape sh = group_shape_of<FEW>(deg, g);
    const int N = sh.N, stride = sh.stride;
    if (PLAN && plan) {
        plan_gather<PLAN ? PLAN : 4>(p, plan, rows, stride, N);
    } else {
        if (leader) {
            B.ent[lane >> g] = hd.o0 - p.nbr_shift;
            B.deg[lane >> g] = deg;
        }
        for (int j = 0; j < N; j += 4)
            *reinterpret_cast<int4 *>(rows + lane * stride + j) = make_int4(INT_MAX, INT_MAX, INT_MAX, INT_MAX);
        __syncwarp();
        // gather: row r holds entries 32 (r mod G) ... of the tile's vertex r / G
        constexpr int PER = 8;  // rows in flight
        for (int r0 = 0; r0 < 32; r0 += PER) {
            int id[PER];
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                const int q = (r0 + u) >> g, j = ((r0 + u) & (G - 1)) * 32 + lane;
                id[u] = j < B.deg[q] ? ld_nbr(&p.nbr[B.ent[q] + j]) : -1;
            }
            if constexpr (LIVE && PLAN == 0) {  // as for small tiles
#pragma unroll
                for (int u = 0; u < PER; ++u) {
                    const int q = (r0 + u) >> g, j = ((r0 + u) & (G - 1)) * 32 + lane;
                    if (id[u] >= 0)
                        rows[(q << g) * stride + j + (j * sh.rcp >> 16) * (stride - N)] =
                            gather_label<LIVE>(&p.lab_in[id[u]]);
                }
            } else {
                int32_t lb[PER];
#pragma unroll
                for (int u = 0; u < PER; ++u) lb[u] = gather_label_if<LIVE>(p.lab_in, id[u]);
#pragma unroll
                for (int u = 0; u < PER; ++u) {
                    const int q = (r0 + u) >> g, j = ((r0 + u) & (G - 1)) * 32 + lane;
                    if (id[u] >= 0) rows[(q << g) * stride + j + (j * sh.rcp >> 16) * (stride - N)] = lb[u];
                }
            }
        }
        __syncwarp();
    }
    uint32_t h;
    if (!FEW && N == 20) h = group_sort_rows<20>(rows, g);  // warp-uniform
    else if (!FEW && N == 24) h = group_sort_rows<24>(rows, g);
    else h = group_sort_rows<32>(rows, g);
    const int cnt = min(max(deg - sub * N, 0), N);  // labels in this lane
    const uint32_t valid = cnt >= 32 ? kFull : (1u << cnt) - 1u;
    h &= valid;
    const uint32_t cont = ~h & valid;
    // labels of the following lanes that continue this lane's last run: sums of the lanes'
    // leading continuations up to and with the first lane that has a head
    int ext = h ? __ffs(h) - 1 : cnt;
    bool stop = h != 0u;
    for (int o = 1; o < G; o <<= 1) {
        const int e2 = __shfl_down_sync(kFull, ext, o);
        const bool s2 = __shfl_down_sync(kFull, (int)stop, o);
        if (sub + o < G && !stop) {
            ext += e2;
            stop = s2;
        }
    }
    ext = __shfl_down_sync(kFull, ext, 1);
    if (sub == G - 1) ext = 0;
    const int lp = h ? 31 - __clz(h) : 0;     // the last head of the lane ...
    const int tail = h ? cnt - lp + ext : 0;  // ... and the length of its run
    uint32_t m = h & ~(1u << lp);             // the other heads, as for small vertices
    int W = m ? 1 : 0;
    while (m) {
        const uint32_t more = m & __funnelshift_rc(cont, 0u, W);  // a shift of 32 gives 0
        if (!more) break;
        m = more;
        ++W;
    }
    int top = max(W, tail);
    for (int o = G >> 1; o; o >>= 1) top = max(top, __shfl_xor_sync(kFull, top, o));
    m = (W == top ? m : 0u) | (tail == top && h ? 1u << lp : 0u);
    // distinct labels and candidates of the group, and the rank of the lane's first head
    int k = __popc(m), d = __popc(h);
    for (int o = 1; o < G; o <<= 1) {
        const int y = __shfl_up_sync(kFull, d, o);
        if (sub >= o) d += y;
    }
    const int rank0 = d - __popc(h);
    for (int o = G >> 1; o; o >>= 1) k += __shfl_xor_sync(kFull, k, o);
    d = __shfl_sync(kFull, d, lane | (G - 1));
    // the smallest and largest candidate and their ranks, from the lanes that hold them
    const unsigned gm = (G == 32 ? kFull : ((1u << G) - 1u)) << (lane - sub);
    const unsigned holders = __ballot_sync(kFull, m != 0u) & gm;
    const int lo = m ? __ffs(m) - 1 : 0, hi = m ? 31 - __clz(m) : 0;
    const int l0 = holders ? __ffs(holders) - 1 : lane, l1 = holders ? 31 - __clz(holders) : lane;
    Sum5 sm;
    sm.d = d;
    sm.W = top;
    sm.k = k;
    sm.mn = __shfl_sync(kFull, rows[lane * stride + lo], l0);
    sm.mx = __shfl_sync(kFull, rows[lane * stride + hi], l1);
    const int rmin = __shfl_sync(kFull, rank0 + __popc(h & ((1u << lo) - 1u)), l0);
    const int rmax = __shfl_sync(kFull, rank0 + __popc(h & ((1u << hi) - 1u)), l1);
    if (leader && v >= 0) {
        if (!hd.dirty) carry_clean(p, v);
        else finish_counted(p, v, sm, rmin, rmax, changes, hd.old, kSpillSorted);
    }
    unsigned spill = __ballot_sync(kFull, leader && deg > 0 && k > 2);
    if (spill) {
        if (!FEW && N == 20) group_compact<20>(rows, g, h, m, rank0);
        else if (!FEW && N == 24) group_compact<24>(rows, g, h, m, rank0);
        else group_compact<32>(rows, g, h, m, rank0);
        const int64_t e0 = hd.o0 - p.nbr_shift;
        while (spill) {  // one vertex after the other, coalesced
            const int src = __ffs(spill) - 1;
            spill &= spill - 1;
            const int64_t e = __shfl_sync(kFull, e0, src);
            const int dd = __shfl_sync(kFull, d, src), ww = __shfl_sync(kFull, top, src);
            for (int r = lane; r < dd; r += 32) {
                const int32_t x = rows[src * stride + r];
                p.run_lab[e + r] = x & INT_MAX;
                p.run_cnt[e + r] = x < 0 ? (uint16_t)ww : (uint16_t)0;
            }
        }
    }
    __syncwarp();  // the tile buffer may be written again
    return d;
}

constexpr int kGroupThreads = 128;
constexpr int kGroupBlocks = 5;  // resident blocks per SM: 6, 4 and 8 were 1 to 9 % slower
__global__ void __launch_bounds__(kGroupThreads, kGroupBlocks) count_group_kernel(PipeArgs p)
{
    constexpr int NW = kGroupThreads / 32;
    __shared__ __align__(16) GroupBuf stile[NW];
    __shared__ GroupTiles T;
    if (!ctl_active(p.ctl)) return;
    const bool fr = frontier_on(p);
    const int w = threadIdx.x >> 5;
    unsigned long long changes = 0;
    if (threadIdx.x == 0) T.set(p, p.disp->pos1);
    __syncthreads();
    const int nw = gridDim.x * NW;
    int t = blockIdx.x * NW + w;
    TileHead nxt = group_head<false>(p, T, t, fr);
    for (; t < T.count(); t += nw) {
        const TileHead hd = nxt;
        nxt = group_head<false>(p, T, t + nw, fr);
        int d = group_tile<false>(p, stile[w], hd, changes);
        if (!hd.dirty) d = p.dcnt[hd.v];
        if ((threadIdx.x & ((1 << hd.g) - 1)) == 0 && hd.v >= 0) add_runs(p, hd.v, d);
    }
    flush_changes(changes, p.ctl);
}

// One warp per mid vertex (33..256 neighbours), counted the segmented sort + reduce way
// (the reference's method 0, dpp/segmented_sort.cuh and the boundary/scan/reduce steps of
// dpp/kernel.cuh, within one warp): the vertex's labels are sorted by a 256-key bitonic
// network (8 keys per lane; sorted position i lives in lane i / 8, register i % 8; unused
// keys are 0xFFFFFFFF and sort last), run heads are the positions whose label differs from
// the previous one, and a run's count is the distance to the next head.  The summary and
// the spill (runs in label order, which the unsorted-spill queries accept) are the ones
// the hash kernels produce.  Variant `mid_sort` 1; no table, no shared memory but the tied
// buffer.
__device__ __forceinline__ void warp_bitonic256(uint32_t (&a)[8], int lane)
{
#pragma unroll
    for (int k = 2; k <= 256; k <<= 1) {
#pragma unroll
        for (int jj = k >> 1; jj > 0; jj >>= 1) {
            if (jj >= 8) {  // partner in lane ^ (jj / 8), same register
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int i = lane * 8 + j;
                    const uint32_t o = __shfl_xor_sync(kFull, a[j], jj >> 3);
                    const bool up = (i & k) == 0, lower = (i & jj) == 0;
                    a[j] = (lower == up) ? min(a[j], o) : max(a[j], o);
                }
            } else {  // partner in this lane's registers
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int pj = j ^ jj;
                    if (pj > j) {
                        const bool up = ((lane * 8 + j) & k) == 0;
                        const uint32_t x = a[j], y = a[pj];
                        a[j] = up ? min(x, y) : max(x, y);
                        a[pj] = up ? max(x, y) : min(x, y);
                    }
                }
            }
        }
    }
}

__global__ void __launch_bounds__(32 * kMidWarps) count_mid_sort_kernel(PipeArgs p)
{
    if (!ctl_active(p.ctl)) return;
    const bool fr = frontier_on(p);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int gw = blockIdx.x * kMidWarps + w;
    const int nw = gridDim.x * kMidWarps;
    unsigned long long changes = 0;
    const int nwarp_v = p.gstart;  // the degree-sorted mid list's prefix of up to 256 neighbours
    for (int i = gw; i < nwarp_v; i += nw) {
        const int v = p.mid_v[i];
        if (fr && !p.dirty[v]) {
            if (lane == 0) {
                carry_clean(p, v);
                add_runs(p, v, p.dcnt[v]);
            }
            continue;
        }
        const int64_t o0 = __ldg(&p.off[v]);
        const int deg = (int)(__ldg(&p.off[v + 1]) - o0);  // 33..256
        uint32_t a[8];
        {
            int nb[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int e = j * 32 + lane;  // coalesced loads; placement does not matter to the sort
                nb[j] = e < deg ? ld_nbr(&p.nbr[o0 + e - p.nbr_shift]) : -1;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) a[j] = nb[j] >= 0 ? (uint32_t)ld_label(&p.lab_in[nb[j]]) : 0xFFFFFFFFu;
        }
        warp_bitonic256(a, lane);
        // run heads: position i is valid when i < deg and a head when its label differs
        // from position i - 1's (the previous lane's last key for register 0)
        const uint32_t prev_last = __shfl_up_sync(kFull, a[7], 1);
        unsigned hm = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int pos = lane * 8 + j;
            const uint32_t prev = j ? a[j - 1] : prev_last;
            if (pos < deg && (pos == 0 || a[j] != prev)) hm |= 1u << j;
        }
        // the first head at or after the next lane (suffix minimum over lanes), else deg
        int first = hm ? lane * 8 + __ffs(hm) - 1 : deg;
        int after = deg;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int o = __shfl_down_sync(kFull, first, off);
            if (lane + off < 32) first = min(first, o);
        }
        after = __shfl_down_sync(kFull, first, 1);  // minimum over lanes > this one
        if (lane == 31) after = deg;
        // heads before this lane, for the runs' ranks
        const int nh = __popc(hm);
        int before = nh;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int o = __shfl_up_sync(kFull, before, off);
            if (lane >= off) before += o;
        }
        before -= nh;
        // this lane's runs: count = next head position - head position
        Sum5 part = sum5_empty();
        int cnt[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            cnt[j] = 0;
            if (hm & (1u << j)) {
                const unsigned later = hm & ~((2u << j) - 1u);
                const int next = later ? lane * 8 + __ffs(later) - 1 : after;
                cnt[j] = next - (lane * 8 + j);
                part.d += 1;
                sum5_observe(part, (int)a[j], cnt[j]);
            }
        }
        const Sum5 sm = sum5_warp(part);
        // ranks of the smallest and largest candidate: heads before them (labels ascend)
        int rmin = 0, rmax = sm.d - 1;
        if (sm.k > 1) {
            int lo = 0, hi = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (hm & (1u << j)) {
                    lo += (int)a[j] < sm.mn;
                    hi += (int)a[j] < sm.mx;
                }
            rmin = __reduce_add_sync(kFull, lo);
            rmax = __reduce_add_sync(kFull, hi);
            if (sm.k > 2) {  // spill the runs in label order
                int32_t *rl = p.run_lab + (o0 - p.nbr_shift);
                uint16_t *rc = p.run_cnt + (o0 - p.nbr_shift);
                int r = before;
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (hm & (1u << j)) {
                        rl[r] = (int32_t)a[j];
                        rc[r] = (uint16_t)cnt[j];
                        ++r;
                    }
            }
        }
        if (lane == 0) {
            finish_counted(p, v, sm, rmin, rmax, changes, __ldg(&p.lab_in[v]));
            add_runs(p, v, sm.d);
        }
        __syncwarp();
    }
    flush_changes(changes, p.ctl);
}

// Block-wide Sum5 / pair reductions with one barrier each: warps publish partials, then
// every warp folds all of them.  Buffers hold one entry per warp (W = THREADS / 32): buf
// is [5][W], buf2 [2][W].  The kernel's end-of-vertex barrier orders a buffer's reads
// before its next writes.
template <int THREADS>
struct BlockRed5 {
    static constexpr int W = THREADS / 32;
    int *buf;   // [5][W]
    int *buf2;  // [2][W]
    __device__ Sum5 reduce(Sum5 s) const
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        s = sum5_warp(s);
        if (lane == 0) {
            buf[0 * W + warp] = s.d;
            buf[1 * W + warp] = s.W;
            buf[2 * W + warp] = s.k;
            buf[3 * W + warp] = s.mn;
            buf[4 * W + warp] = s.mx;
        }
        __syncthreads();
        Sum5 t = sum5_empty();
        if (lane < W) t = Sum5{buf[lane], buf[W + lane], buf[2 * W + lane], buf[3 * W + lane], buf[4 * W + lane]};
        return sum5_warp(t);
    }
    __device__ void reduce2(int &a, int &b) const
    {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        a = __reduce_add_sync(kFull, a);
        b = __reduce_add_sync(kFull, b);
        if (lane == 0) {
            buf2[warp] = a;
            buf2[W + warp] = b;
        }
        __syncthreads();
        const int x = lane < W ? buf2[lane] : 0, y = lane < W ? buf2[W + lane] : 0;
        a = __reduce_add_sync(kFull, x);
        b = __reduce_add_sync(kFull, y);
    }
};

// ----- bulk copies into shared memory (cp.async.bulk) with mbarrier completion -----
__device__ __forceinline__ uint32_t smem_u32(const void *ptr)
{
    return (uint32_t)__cvta_generic_to_shared(ptr);
}

__device__ __forceinline__ void mbar_init(unsigned long long *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// One thread: expect `bytes` on the barrier, then copy them global -> shared (both
// addresses 16-byte aligned, bytes a multiple of 16).
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, unsigned long long *bar)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait for the barrier's phase `parity`; false after kStageSpinLimit polls.
constexpr long long kStageSpinLimit = 1ll << 22;
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, uint32_t parity)
{
    for (long long i = 0; i < kStageSpinLimit; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// One CTA of THREADS threads per vertex of degree <= SLOTS/2 (table of SLOTS 64-bit
// slots in dynamic shared memory), for a range of the degree-sorted mid list.
//
// Software pipelining across the CTA's vertices: the next vertex's head (CtaHead) and, in
// CTAs of up to 256 threads that do not stage, its first PER * THREADS neighbour IDs are
// loaded into registers while the current vertex's labels are gathered and counted, so a
// vertex starts with its label gathers instead of three dependent global round trips.
//
// STAGE: the next vertex's neighbour IDs are copied into a shared-memory stage by one
// bulk copy (cp.async.bulk, completion on an mbarrier) while the current vertex is
// counted, so the IDs are read from shared memory and no thread waits on their global
// loads.  The copy starts at the 16-byte boundary below the vertex's first entry and
// ends at the one above its last (the neighbour buffers carry 16 bytes of padding).  A
// wait that runs out (it cannot for a valid address) sets kErrStage, waits for that copy
// once more before the CTA exits and counts the remaining vertices from global loads.
// Not in frontier mode (clean vertices need no IDs).
template <int THREADS, int SLOTS, bool STAGE = false>
__global__ void __launch_bounds__(THREADS, THREADS >= 1024 ? 1 : THREADS >= 512 ? 2 : THREADS >= 256 ? 4
                                           : THREADS >= 128 ? 8 : 16)
    count_cta_kernel(PipeArgs p, int which)
{
    extern __shared__ __align__(16) unsigned long long cta_tab[];
    __shared__ int red[5 * (THREADS / 32)], red2[2 * (THREADS / 32)];
    __shared__ int sctr;
    __shared__ __align__(8) unsigned long long stage_bar;
    __shared__ int stage_ok;
    if (!ctl_active(p.ctl)) return;
    // ranges of the degree-sorted mid list: 1 [pos_a, pos2), 2 [pos2, pos_b), 3 [pos_b, end)
    const DispatchState &ds = *p.disp;
    const int first = which == 1 ? ds.pos_a : which == 2 ? ds.pos2 : ds.pos_b;
    const int end = which == 1 ? ds.pos2 : which == 2 ? ds.pos_b : p.nmid_s + p.nmid_l + p.nmid_x;
    const int count = end - first;
    const bool fr = frontier_on(p);
    const int tid = threadIdx.x;
    const BlockRed5<THREADS> br{red, red2};
    unsigned long long changes = 0;
    for (int s = tid; s < SLOTS; s += THREADS) cta_tab[s] = 0ull;
    uint32_t gen = 0;
    // staging: thread 0 copies the neighbour IDs of list entry i into the stage
    const bool staged = STAGE && !fr;
    int32_t *stage = reinterpret_cast<int32_t *>(cta_tab + SLOTS);
    uint32_t parity = 0, lost_parity = 2;
    auto stage_issue = [&](int i) {
        if (i >= count) return;
        const int vn = p.mid_v[first + i];
        const int64_t a = __ldg(&p.off[vn]) - p.nbr_shift;
        const int64_t b = __ldg(&p.off[vn + 1]) - p.nbr_shift;
        const int64_t a4 = a & ~(int64_t)3, b4 = (b + 3) & ~(int64_t)3;
        // the proxy fence orders the threads' reads of the stage before the copy's writes
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        bulk_load(stage, p.nbr + a4, (uint32_t)(4 * (b4 - a4)), &stage_bar);
    };
    if (staged && tid == 0) {
        mbar_init(&stage_bar, 1);
        stage_ok = 1;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        stage_issue(blockIdx.x);
    }
    __syncthreads();
    constexpr int PER = 8;  // a thread's loads in flight together per round
    // The first round of a vertex's neighbour IDs, loaded one vertex ahead (not staged; CTAs
    // of up to 256 threads: in the 512- and 1024-thread CTAs the extra registers cost the
    // gathers more than the early IDs save).
    constexpr bool kAhead = THREADS <= 256;
    const bool ahead = kAhead && !staged;
    auto ids_ahead = [&](int (&nb)[PER], const CtaHead &h) {
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int e = tid + u * THREADS;
            nb[u] = (ahead && h.v >= 0 && h.dirty && e < h.deg) ? ld_nbr(&p.nbr[h.o0 + e - p.nbr_shift]) : -1;
        }
    };
    CtaHead nxt = cta_head(p, first, blockIdx.x, count, fr);
    int nbn[PER];
    ids_ahead(nbn, nxt);
    for (int i = blockIdx.x; i < count; i += gridDim.x) {
        const CtaHead h = nxt;
        const int v = h.v;
        int nb0[PER];
#pragma unroll
        for (int u = 0; u < PER; ++u) nb0[u] = nbn[u];
        nxt = cta_head(p, first, i + gridDim.x, count, fr);
        if (!h.dirty) {
            if (tid == 0) {
                carry_clean(p, v);
                add_runs(p, v, h.dcnt);
            }
            ids_ahead(nbn, nxt);
            continue;
        }
        if (++gen > kT64GenMax) {
            for (int s = tid; s < SLOTS; s += THREADS) cta_tab[s] = 0ull;
            __syncthreads();
            gen = 1;
        }
        const int64_t o0 = h.o0;
        const int deg = h.deg;
        // this vertex's IDs in the stage (the copy was issued one vertex earlier)
        bool from_stage = false;
        if (staged && stage_ok) {
            const bool got = mbar_wait(&stage_bar, parity);
            if (!got) stage_ok = 0;  // any thread that gave up turns staging off for the CTA
            __syncthreads();
            from_stage = stage_ok != 0;
            if (!from_stage) {
                lost_parity = parity;  // the copy still in flight completes this phase
                if (tid == 0) atomicOr(&p.ctl->err, kErrStage);
            }
            parity ^= 1u;
        }
        const int skip = (int)((o0 - p.nbr_shift) & 3);
        // probe range: the whole table up to 4 slots per neighbour (load <= 1/4 where the
        // table allows, at most 1/2): the longest probe of a warp's inserts sets its pace
        const uint32_t cap = (uint32_t)min(SLOTS, 4 * pad32(deg));
        // warp-aggregated inserts when the vertex had at most half as many distinct labels
        // as neighbours in the previous iteration (agg_mode 0); always (1); never (2)
        const int mode = p.disp->agg_mode;
        const bool agg = mode == 1 || (mode == 0 && 2 * h.dcnt <= deg);
        Sum5 obs = sum5_empty();
        // gather in rounds of PER loads per thread in flight together; the first round's IDs
        // are in registers already (or in the stage)
        for (int base = 0; base < deg; base += THREADS * PER) {
            int nb[PER];
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                const int e = base + tid + u * THREADS;
                if (base == 0 && ahead) nb[u] = nb0[u];
                else nb[u] = (e < deg) ? (from_stage ? stage[skip + e] : ld_nbr(&p.nbr[o0 + e - p.nbr_shift])) : -1;
            }
            uint32_t lb[PER];
#pragma unroll
            for (int u = 0; u < PER; ++u) lb[u] = (nb[u] >= 0) ? (uint32_t)ld_label(&p.lab_in[nb[u]]) : kEmpty;
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                if (base + u * THREADS >= deg) break;  // block-uniform
                t64_insert_row(cta_tab, cap, gen, lb[u], agg, obs);
            }
        }
        // the next vertex's first IDs (its head has arrived during the gathers and inserts)
        // load while this vertex is reduced, ranked, spilled and finished
        ids_ahead(nbn, nxt);
        // the reduction's barrier also completes the table for the rank and spill passes,
        // and every thread's reads of the stage: the next vertex's copy may start
        const Sum5 s = br.reduce(obs);
        if (from_stage && tid == 0) stage_issue(i + gridDim.x);
        int rmin = 0, rmax = s.d - 1;  // when every distinct label is a candidate
        if (s.k > 1) {
            if (s.k < s.d) {
                t64_ranks(cta_tab, (int)cap, tid, THREADS, gen, s.mn, s.mx, rmin, rmax);
                br.reduce2(rmin, rmax);
            }
            if (s.k > 2) {
                if (tid == 0) sctr = 0;
                __syncthreads();
                t64_spill(cta_tab, (int)cap, tid, THREADS, gen, p.run_lab + (o0 - p.nbr_shift),
                          p.run_cnt + (o0 - p.nbr_shift), &sctr);
            }
        }
        if (tid == 0) {
            finish_counted(p, v, s, rmin, rmax, changes, h.old);
            add_runs(p, v, s.d);
        }
        __syncthreads();
    }
    // a copy that a wait gave up on still lands in this CTA's shared memory: wait for it
    // (bounded) before the CTA exits
    if (staged && lost_parity < 2) (void)mbar_wait(&stage_bar, lost_parity);
    flush_changes(changes, p.ctl);
}

// One CTA per hub partition (grid-stride over the scope's partitions): count the
// partition's (label, count) pairs in a shared-memory table sized to them (all pairs of a
// label fall in one partition, so its count is complete here), fold the counts each
// insert observes into the partition's summary, append its distinct labels to the hub's
// distinct list and reset the partition's fill for the next scope.
//
// Three shapes: 1024 threads with 16384-slot tables (one CTA per SM), 512 threads with
// 8192-slot tables (three per SM) for partitions of half the size (hub_part_shift 1), and
// 256 threads with 4096-slot tables (six per SM) for a quarter (hub_part_shift >= 2).
template <int kT, int TAB>
__global__ void __launch_bounds__(kT, kT >= 1024 ? 1 : kT >= 512 ? 3 : 6) hub_count_kernel(IterArgs p)
{
    extern __shared__ __align__(16) uint32_t hub_tab[];  // TAB keys, then TAB counts
    __shared__ int red[5 * (kT / 32)], red2[2 * (kT / 32)];
    __shared__ int sfill, sbase, sctr;
    if (!ctl_active(p.ctl)) return;
    uint32_t *key = hub_tab;
    uint32_t *cnt = hub_tab + TAB;
    const BlockRed5<kT> br{red, red2};
    const int tid = threadIdx.x, lane = tid & 31;
    for (int x = blockIdx.x; x < p.nparts; x += gridDim.x) {
        const int gp = p.q0 + x;
        const int bi = p.part_big[gp];
        const int pcap = p.hub_pcap[bi];
        if (tid == 0) sfill = min(p.pfill[gp], pcap);
        __syncthreads();
        const int fill = sfill;
        uint32_t tcap = 64;  // load <= 1/2 when every pair is a distinct label
        while (tcap < 2u * (uint32_t)fill && tcap < (uint32_t)TAB) tcap <<= 1;
        for (int s2 = tid; s2 < (int)tcap; s2 += kT) {
            key[s2] = kEmpty;
            cnt[s2] = 0;
        }
        __syncthreads();
        const unsigned long long *src = p.pairs + p.hub_pbase[bi] + (int64_t)(gp - p.hub_p0[bi]) * pcap;
        Sum5 obs = sum5_empty();
        constexpr int PER = 8;  // a thread's pair loads in flight together
        for (int j0 = 0; j0 < fill; j0 += kT * PER) {
            unsigned long long xs[PER];
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                const int j = j0 + tid + u * kT;
                xs[u] = j < fill ? src[j] : ~0ull;  // a pair is never all ones (labels < 2^31)
            }
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                if (xs[u] == ~0ull) continue;
                const uint32_t L = (uint32_t)(xs[u] >> 32), c = (uint32_t)xs[u];
                uint32_t h = hslot(L, tcap);
                // a full table (more distinct labels than slots: pairs repeating few labels
                // made it small) ends the probe after one round and flags the run
                for (uint32_t probe = 0;; ++probe) {
                    if (probe == tcap) {
                        atomicOr(&p.ctl->err, kErrHubOverflow);
                        break;
                    }
                    const uint32_t prev = atomicCAS(&key[h], kEmpty, L);
                    if (prev == kEmpty || prev == L) {
                        obs.d += prev == kEmpty;
                        sum5_observe(obs, (int)L, (int)(atomicAdd(&cnt[h], c) + c));
                        break;
                    }
                    h = (h + 1 == tcap) ? 0 : h + 1;
                }
            }
        }
        const Sum5 sm = br.reduce(obs);  // its barrier also completes the table
        if (tid == 0) {
            sbase = sm.d ? atomicAdd(&p.bstat[bi].d, sm.d) : 0;
            sctr = 0;
            p.psum[gp] = make_int4(sm.W, sm.k, sm.mn, sm.mx);
            p.pfill[gp] = 0;
        }
        __syncthreads();
        unsigned long long *list = p.big_list + p.big_ooff[bi] + sbase;
        for (int s0 = 0; s0 < (int)tcap; s0 += kT) {
            const int s2 = s0 + tid;
            const bool used = s2 < (int)tcap && key[s2] != kEmpty;
            const unsigned m = __ballot_sync(kFull, used);
            if (!m) continue;
            int at = 0;
            if (lane == __ffs(m) - 1) at = atomicAdd(&sctr, __popc(m));
            at = __shfl_sync(kFull, at, __ffs(m) - 1) + __popc(m & ((1u << lane) - 1));
            if (used) list[at] = ((unsigned long long)key[s2] << 32) | cnt[s2];
        }
        __syncthreads();
    }
}

// Measurement probe: one pass over the CSR that streams every neighbour ID and gathers its
// label with the loads the counting kernels use (streaming IDs, evict-last label gathers),
// 8 entries per thread in flight, and nothing else; the block XORs the labels into one
// word.  Its time is the floor of any update that gathers every neighbour's label.
__global__ void __launch_bounds__(kTB) gather_probe_kernel(const int32_t *nbr, int64_t m, const int32_t *lab,
                                                           unsigned long long *acc)
{
    constexpr int PER = 8;
    uint32_t x = 0;
    const int64_t stride = (int64_t)gridDim.x * kTB * PER;
    for (int64_t base = (int64_t)blockIdx.x * kTB * PER + threadIdx.x; base < m; base += stride) {
        int nb[PER];
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int64_t e = base + (int64_t)u * kTB;
            nb[u] = e < m ? ld_nbr(&nbr[e]) : -1;
        }
#pragma unroll
        for (int u = 0; u < PER; ++u) x ^= nb[u] >= 0 ? (uint32_t)ld_label(&lab[nb[u]]) : 0u;
    }
    x = __reduce_xor_sync(kFull, x);
    if ((threadIdx.x & 31) == 0 && x) atomicXor(acc, (unsigned long long)x);
}

// One warp per big vertex: fold its partitions' summaries; when every distinct label is
// a candidate the ranks are 0 and d - 1.  Its distinct count joins the others.
__global__ void big_combine_kernel(IterArgs p, PipeArgs q)
{
    if (!ctl_active(p.ctl)) return;
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < p.nbig; i += nw) {
        const int bi = p.b0 + i;
        int W = 0, k = 0, mn = INT_MAX, mx = -1;
        for (int c = p.hub_p0[bi] + lane; c < p.hub_p0[bi + 1]; c += 32) {
            const int4 o = p.psum[c];
            if (o.x > W) {
                W = o.x;
                k = o.y;
                mn = o.z;
                mx = o.w;
            } else if (o.x == W) {
                k += o.y;
                mn = min(mn, o.z);
                mx = max(mx, o.w);
            }
        }
        const int Ww = __reduce_max_sync(kFull, W);
        const bool top = W == Ww;
        k = __reduce_add_sync(kFull, top ? k : 0);
        mn = __reduce_min_sync(kFull, top ? mn : INT_MAX);
        mx = __reduce_max_sync(kFull, top ? mx : -1);
        if (lane == 0) {
            BigStat &st = p.bstat[bi];
            st.W = Ww;
            st.k = k;
            st.cmin = mn;
            st.cmax = mx;
            if (k == st.d) {
                st.rmin = 0;
                st.rmax = st.d - 1;
            }
            const int v = p.big_v[bi];
            q.dcnt[v] = st.d;
            add_runs(q, v, st.d);
        }
    }
}

// ---------------------------------------------------------------------------
// scan of the distinct counts' sums
// ---------------------------------------------------------------------------

// Exclusive scan of the sums (which are zero again afterwards), the scope's number of runs, the
// graphs' run bases, an empty tied list.  Up to kScanOneBlock sums one block does it all, round
// after round; more (whose rounds and graphs would follow one another) are scanned by a block per
// round, from the rounds' sums (scan_sums_kernel), and the graphs' bases have a kernel of their own.
// One block or several, us per iteration: 20 K graphs 29 and 23, 100 K 130 and 23, a million 1950
// and 30; with fewer graphs two launches more are worth about two rounds.
constexpr int kScanThreads = 1024;
constexpr int kScanRound = kScanThreads * 8;
constexpr int kScanOneBlock = 4 * kScanRound;

// Run base of graph g, an empty one too: its first sum (empty graphs have one that nothing adds to)
__device__ __forceinline__ int64_t graph_base(const PipeArgs &p, int g)
{
    return p.run_at[(int64_t)(p.g_v0[g] - p.v0) / kRunBlock + g];
}

__global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(PipeArgs p, int npieces)
{
    __shared__ long long ws[kScanThreads / 32];
    if (!ctl_active(p.ctl)) return;
    const int tid = threadIdx.x;
    const int64_t i0 = (int64_t)blockIdx.x * kScanRound;
    long long s = 0;
#pragma unroll
    for (int u = 0; u < kScanRound / kScanThreads; ++u) {
        const int64_t i = i0 + u * kScanThreads + tid;
        if (i < npieces) s += p.sums[i];
    }
    s = warp_sum_ll(s);
    if ((tid & 31) == 0) ws[tid >> 5] = s;
    __syncthreads();
    if (tid < 32) {
        s = warp_sum_ll(ws[tid]);
        if (tid == 0) p.round_sum[blockIdx.x] = s;
    }
}

__global__ void __launch_bounds__(kScanThreads) scan_kernel(PipeArgs p, int npieces)
{
    constexpr int NW = kScanThreads / 32, PER = kScanRound / kScanThreads;
    __shared__ long long ws[NW];
    if (!ctl_active(p.ctl)) return;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const bool several = gridDim.x > 1;
    long long base = 0;
    if (several) {  // the sums of the rounds before
        for (int i = tid; i < (int)blockIdx.x; i += kScanThreads) base += p.round_sum[i];
        base = warp_sum_ll(base);
        if (lane == 0) ws[w] = base;
        __syncthreads();
        base = warp_sum_ll(ws[lane]);
        __syncthreads();
    }
    const int64_t end = several ? min((int64_t)npieces, ((int64_t)blockIdx.x + 1) * kScanRound) : npieces;
    // rounds of kScanRound sums; a warp takes 32 * PER consecutive ones, row after row
    for (int64_t i0 = (int64_t)blockIdx.x * kScanRound; i0 < end; i0 += kScanRound) {
        long long x[PER], s = 0;
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int64_t i = i0 + (w * PER + u) * 32 + lane;
            x[u] = i < end ? p.sums[i] : 0;
        }
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const long long own = x[u];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const long long y = __shfl_up_sync(kFull, x[u], o);
                if (lane >= o) x[u] += y;
            }
            const long long row = __shfl_sync(kFull, x[u], 31);
            x[u] += s - own;
            s += row;
        }
        if (lane == 0) ws[w] = s;
        __syncthreads();
        long long before = base, all = ws[lane];
        for (int i = 0; i < w; ++i) before += ws[i];
        all = warp_sum_ll(all);
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int64_t i = i0 + (w * PER + u) * 32 + lane;
            if (i < end) {
                p.run_at[i] = before + x[u];
                p.sums[i] = 0;
            }
        }
        base += all;
        __syncthreads();
    }
    if (blockIdx.x == gridDim.x - 1 && tid == 0) {
        p.ctl->N = base;
        p.ctl->tied_mid = 0;
    }
    if (p.g_v0 && !several)
        for (int g = tid; g <= p.ngraphs; g += kScanThreads) p.g_base[g] = g < p.ngraphs ? graph_base(p, g) : base;
}

__global__ void __launch_bounds__(kTB) batch_bases_kernel(PipeArgs p)
{
    if (!ctl_active(p.ctl)) return;
    for (int64_t g = (int64_t)blockIdx.x * kTB + threadIdx.x; g <= p.ngraphs; g += (int64_t)gridDim.x * kTB)
        p.g_base[g] = g < p.ngraphs ? graph_base(p, (int)g) : p.ctl->N;
}

// ---------------------------------------------------------------------------
// resolution of tied vertices
// ---------------------------------------------------------------------------

// Sorted spilled runs of a small vertex, scanned by one thread.
struct SpillRunQuery {
    const int32_t *lab;
    const uint16_t *cnt;
    int d, W;
    __device__ int first_ge(int64_t x) const
    {
        for (int r = (int)(x < 0 ? 0 : x); r < d; ++r)
            if ((int)cnt[r] == W) return r;
        return -1;
    }
    __device__ int last_lt(int64_t y) const
    {
        for (int r = (int)(y < d ? y : d) - 1; r >= 0; --r)
            if ((int)cnt[r] == W) return r;
        return -1;
    }
    __device__ int tile_pick(int64_t) const { return -1; }  // d <= 32 never spans a tile
};

// A small vertex with more than two candidates as count_small_sort_kernel leaves it: h has
// the run heads among its sorted labels (at its CSR positions), m the heads of candidates.
struct SmallMaskQuery {
    uint32_t h, m;
    int pos = 0;  // head of the candidate that the last query found
    // position of the head of rank x (0 <= x < popc(h))
    __device__ int at(int x) const
    {
        uint32_t b = h;
        int r = 0;
#pragma unroll
        for (int step = 16; step; step >>= 1) {
            const int c = __popc(b & ((1u << step) - 1u));
            if (x >= c) {
                x -= c;
                r += step;
                b >>= step;
            }
        }
        return r;
    }
    __device__ int rank(int head)
    {
        pos = head;
        return __popc(h & ((1u << head) - 1u));
    }
    __device__ int first_ge(int64_t x)
    {
        if (x >= __popc(h)) return -1;
        const uint32_t c = x <= 0 ? m : m & ~((1u << at((int)x)) - 1u);
        return c ? rank(__ffs(c) - 1) : -1;
    }
    __device__ int last_lt(int64_t y)
    {
        if (y <= 0) return -1;
        const uint32_t c = y >= __popc(h) ? m : m & ((1u << at((int)y)) - 1u);
        return c ? rank(31 - __clz(c)) : -1;
    }
    __device__ int tile_pick(int64_t) const { return -1; }  // d <= 32 never spans a tile
};

// New label of a tied small vertex with run scope rs, from its state (one thread); e: its first
// entry in the spill area.  Where that holds the label, its entry is left in `from`.
__device__ __forceinline__ int32_t resolve_small(const PipeArgs &p, const RunScope &rs, int kw, int d, int32_t c0,
                                                 int32_t c1, int rr, int64_t e, int64_t &from)
{
    const int k = kw & 0xFFFF, W = (kw >> 16) & 0x3FFF;
    if (k > 2 && p.small_sort == 2) {
        SmallMaskQuery mq{(uint32_t)c0, (uint32_t)c1};
        (void)resolve_rank(rs.a, d, rs.N, rs.is_last, mq);  // its result is the last query's
        from = e + mq.pos;
        return 0;
    }
    const int rmin = rr & 0xFFFF, rmax = rr >> 16;
    SummaryQuery q(k, d, rmin, rmax);
    int r = resolve_rank(rs.a, d, rs.N, rs.is_last, q);
    if (!q.fail && r == rmin) return c0;
    if (!q.fail && r == rmax) return c1;
    SpillRunQuery sq{p.run_lab + e, p.run_cnt + e, d, W};
    if (q.fail) r = resolve_rank(rs.a, d, rs.N, rs.is_last, sq);
    from = e + r;
    return 0;
}

// Unsorted spilled (label, count) entries of a mid/large vertex, one warp.
struct SpillTableQuery {
    const int32_t *lab;
    const uint16_t *cnt;
    int d, W, rmin, rmax;
    int *hist;
    int lane;
    __device__ uint32_t select(int x)
    {
        uint32_t prefix = 0;
        int remaining = x;
        for (int shift = 24; shift >= 0; shift -= 8) {
            for (int b = lane; b < 256; b += 32) hist[b] = 0;
            __syncwarp();
            const uint32_t hi_mask = (shift == 24) ? 0u : (0xFFFFFFFFu << (shift + 8));
            for (int i = lane; i < d; i += 32) {
                const uint32_t k = (uint32_t)lab[i];
                if ((k & hi_mask) == (prefix & hi_mask)) atomicAdd(&hist[(k >> shift) & 255], 1);
            }
            __syncwarp();
            int c[8];
            int local = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                c[i] = hist[lane * 8 + i];
                local += c[i];
            }
            int incl = local;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int o = __shfl_up_sync(kFull, incl, off);
                if (lane >= off) incl += o;
            }
            const int excl = incl - local;
            const unsigned who = __ballot_sync(kFull, remaining >= excl && remaining < incl);
            const int src = who ? (__ffs(who) - 1) : 31;
            int digit = 0, before = 0;
            if (lane == src) {
                int acc = excl, i = 0;
                for (; i < 7; ++i) {
                    if (remaining < acc + c[i]) break;
                    acc += c[i];
                }
                digit = lane * 8 + i;
                before = acc;
            }
            digit = __shfl_sync(kFull, digit, src);
            before = __shfl_sync(kFull, before, src);
            prefix |= (uint32_t)digit << shift;
            remaining -= before;
            __syncwarp();
        }
        return prefix;
    }
    __device__ int rank_of(uint32_t c) const
    {
        int n = 0;
        for (int i = lane; i < d; i += 32) n += (uint32_t)lab[i] < c;
        return __reduce_add_sync(kFull, n);
    }
    __device__ int first_ge(int64_t x)
    {
        if (x >= d) return -1;
        if (x <= rmin) return rmin;
        const uint32_t L = select((int)x);
        uint32_t best = kEmpty;
        for (int i = lane; i < d; i += 32) {
            const uint32_t k = (uint32_t)lab[i];
            if ((int)cnt[i] == W && k >= L && k < best) best = k;
        }
        best = __reduce_min_sync(kFull, best);
        return best == kEmpty ? -1 : rank_of(best);
    }
    __device__ int last_lt(int64_t y)
    {
        if (y > rmax) return rmax;
        if (y <= rmin) return -1;
        const uint32_t L = select((int)y);
        int best = -1;
        for (int i = lane; i < d; i += 32) {
            const uint32_t k = (uint32_t)lab[i];
            if ((int)cnt[i] == W && k < L && (int)k > best) best = (int)k;
        }
        best = __reduce_max_sync(kFull, best);
        return best < 0 ? -1 : rank_of((uint32_t)best);
    }
    // Among candidates of rank in [lo, lo + kTile) (a whole tile), the one of highest
    // tile_priority; ranks by full passes (only vertices of > 4352 distinct labels
    // whose last tile holds no candidate get here).
    __device__ int tile_pick(int64_t lo)
    {
        int best = -1, bestr = -1;
        for (int i0 = 0; i0 < d; i0 += 32) {
            const int i = i0 + lane;
            const bool c = i < d && (int)cnt[i] == W;
            unsigned m = __ballot_sync(kFull, c);
            while (m) {
                const int src = __ffs(m) - 1;
                m &= m - 1;
                const uint32_t lab_c = (uint32_t)__shfl_sync(kFull, i < d ? lab[i] : 0, src);
                const int r = rank_of(lab_c);
                if (r >= lo && r < lo + kTile && tile_priority(r - lo) > best) {
                    best = tile_priority(r - lo);
                    bestr = r;
                }
            }
        }
        return bestr;
    }
};

// Spilled runs in label order (vertices counted by lane groups), one warp: the run of
// rank r is entry r.
struct SpillSortedQuery {
    const uint16_t *cnt;
    int d, W, rmin, rmax;
    int lane;
    __device__ int first_ge(int64_t x) const
    {
        if (x <= rmin) return rmin;
        if (x > rmax) return -1;
        for (int r0 = (int)x;; r0 += 32) {  // rank rmax is a candidate
            const int r = r0 + lane;
            const unsigned m = __ballot_sync(kFull, r <= rmax && (int)cnt[r] == W);
            if (m) return r0 + __ffs(m) - 1;
        }
    }
    __device__ int last_lt(int64_t y) const
    {
        if (y > rmax) return rmax;
        if (y <= rmin) return -1;
        for (int r0 = (int)y - 32;; r0 -= 32) {  // rank rmin is a candidate
            const int r = r0 + lane;
            const unsigned m = __ballot_sync(kFull, r >= rmin && (int)cnt[r] == W);
            if (m) return r0 + 31 - __clz(m);
        }
    }
    __device__ int tile_pick(int64_t) const { return -1; }  // d <= kGroupMax never spans a tile
};

// New label of a tied mid-list vertex with run scope rs (one warp; hist: 256 ints of its shared
// memory).
__device__ __forceinline__ int32_t resolve_mid(const PipeArgs &p, int v, const RunScope &rs, int *hist)
{
    const int lane = threadIdx.x & 31;
    const int kw = p.sm_kw[v], rr = p.sm_r[v];
    const int k = kw & 0xFFFF, W = (kw >> 16) & 0x3FFF, rmin = rr & 0xFFFF, rmax = rr >> 16;
    const int d = p.dcnt[v];
    SummaryQuery q(k, d, rmin, rmax);
    int r = resolve_rank(rs.a, d, rs.N, rs.is_last, q);
    if (!q.fail && r == rmin) return p.sm_c0[v];
    if (!q.fail && r == rmax) return p.sm_c1[v];
    const int64_t e = __ldg(&p.off[v]) - p.nbr_shift;
    if (kw & kSpillSorted) {
        SpillSortedQuery sq{p.run_cnt + e, d, W, rmin, rmax, lane};
        if (q.fail) r = resolve_rank(rs.a, d, rs.N, rs.is_last, sq);
        return (r == rmin) ? p.sm_c0[v] : (r == rmax) ? p.sm_c1[v] : p.run_lab[e + r];
    }
    SpillTableQuery tq{p.run_lab + e, p.run_cnt + e, d, W, rmin, rmax, hist, lane};
    if (q.fail) r = resolve_rank(rs.a, d, rs.N, rs.is_last, tq);
    return (r == rmin) ? p.sm_c0[v] : (r == rmax) ? p.sm_c1[v] : (int32_t)tq.select(r);
}

// Count a row of changed vertices (one per lane) for their graphs (batches): a warp's rows mostly
// lie in one graph, whose changes it keeps until the graph is another one.
struct GraphChanges {
    int g = -1, n = 0;  // warp-uniform
    __device__ __forceinline__ void flush(const PipeArgs &p)
    {
        if (n && (threadIdx.x & 31) == 0) atomicAdd(&p.g_changes[g], (unsigned long long)n);
        n = 0;
    }
    __device__ __forceinline__ void add(const PipeArgs &p, bool chg, int gv)
    {
        const unsigned m = __ballot_sync(kFull, chg);
        if (!m) return;
        const int g0 = __shfl_sync(kFull, gv, __ffs(m) - 1);
        if (__all_sync(kFull, !chg || gv == g0)) {
            if (g0 != g) flush(p);
            g = g0;
            n += __popc(m);
        } else if (chg) {
            atomicAdd(&p.g_changes[gv], 1ull);
        }
    }
};

// The scope's vertices in order, with their run bases: ties of at most 32 neighbours are resolved
// here, larger ones listed with their run base for resolve_mid_kernel, hubs (which have no
// summary: sm_kw is 0) get their run base.  Batches: a graph that has ended keeps its labels,
// the others count their changes.
//
// One pass where a reduction and a scan over all vertices, tied lists filled by the counting
// kernels and, for batches, a pass of comparing and committing labels stood before: ten
// iterations of 1,024 planted partitions (36 M vertices) 12.4 -> 6.5 ms with scan_kernel, and
// five launches per iteration fewer.  Bound by the latency of its dependent loads (d and kw,
// then the summary and offset, then the spilled label), which is why the rows' loads of one kind
// go out together; 2 or 4 blocks per SM were 3 to 20 % slower.
constexpr int kResolveBlocks = 3;  // resident blocks per SM
template <bool BATCH>
__global__ void __launch_bounds__(kTB, kResolveBlocks) resolve_kernel(PipeArgs p)
{
    constexpr int PER = kRunBlock / kTB;
    __shared__ long long ws[kNW];
    __shared__ int32_t tbuf[kNW][kWarpBuf];
    if (!ctl_active(p.ctl)) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t b0 = p.v0 + (int64_t)blockIdx.x * kRunBlock;
    const int64_t v0 = b0 + w * (PER * 32) + lane;
    // the rows' loads of one kind together, so that the chain of dependent loads is paid once
    int d[PER], kw[PER], g[PER];
    int32_t old[PER], nl[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        const int64_t v = v0 + u * 32;
        const bool in = v < p.v1;
        d[u] = in ? p.dcnt[v] : 0;
        kw[u] = in ? p.sm_kw[v] : 1;
        old[u] = BATCH && in ? __ldg(&p.lab_in[v]) : 0;
        nl[u] = BATCH && in ? p.lab_out[v] : 0;
        g[u] = BATCH && in ? __ldg(&p.gid[v]) : 0;
    }
    long long at[PER];  // runs of the warp's vertices before the vertex
    {
        bool hub = false;  // a row without one has less than 2^31 runs
#pragma unroll
        for (int u = 0; u < PER; ++u) hub |= d[u] > kXlMax;
        const bool wide = !BATCH && __any_sync(kFull, hub);
        long long s = 0;
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            long long row, incl;
            if (!wide) {
                int x = d[u];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(kFull, x, o);
                    if (lane >= o) x += y;
                }
                incl = x;
                row = __shfl_sync(kFull, x, 31);
            } else {
                incl = d[u];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const long long y = __shfl_up_sync(kFull, incl, o);
                    if (lane >= o) incl += y;
                }
                row = __shfl_sync(kFull, incl, 31);
            }
            at[u] = s + incl - d[u];
            s += row;
        }
        if (lane == 0) ws[w] = s;
    }
    // small tied vertices (small), larger ones and hubs (rest; k = 0 in hubs)
    int64_t o0[PER];
    int32_t c0[PER], c1[PER], rr[PER];
    bool small[PER], rest[PER], runs[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        const int64_t v = v0 + u * 32;
        const int k = kw[u] & 0xFFFF;
        const bool pick = d[u] > 0 && k != 1;
        small[u] = pick && kw[u] < 0;
        rest[u] = pick && kw[u] >= 0;
        o0[u] = small[u] ? __ldg(&p.off[v]) : 0;
        c0[u] = small[u] ? p.sm_c0[v] : 0;
        c1[u] = small[u] ? p.sm_c1[v] : 0;
        rr[u] = small[u] && (k == 2 || p.small_sort != 2) ? p.sm_r[v] : 0;
        if (!BATCH) old[u] = small[u] ? __ldg(&p.lab_in[v]) : 0;
        runs[u] = !BATCH || __ldg(&p.g_active[g[u]]) != 0;
    }
    __syncthreads();
    long long base = p.run_at[run_piece(p, (int)b0)];
    for (int i = 0; i < w; ++i) base += ws[i];
    int64_t from[PER];  // spill entry that holds the new label, or -1
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        from[u] = -1;
        if (small[u]) {
            const int64_t v = v0 + u * 32;
            nl[u] = resolve_small(p, run_scope(p, (int)v, base + at[u]), kw[u], d[u], c0[u], c1[u], rr[u],
                                  o0[u] - p.nbr_shift, from[u]);
        }
    }
#pragma unroll
    for (int u = 0; u < PER; ++u)
        if (from[u] >= 0) nl[u] = p.run_lab[from[u]];
    WarpBuf tb{tbuf[w]};
    GraphChanges gc;
    unsigned long long changes = 0;
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        const int64_t v = v0 + u * 32;
        const bool listed = rest[u] && (kw[u] & 0xFFFF) != 0;
        if (rest[u]) p.runbase[v] = base + at[u];
        if (small[u]) {
            if (runs[u]) p.lab_out[v] = nl[u];
            count_change(changes, nl[u], old[u]);
        }
        tb.append(listed, (int32_t)v, p.tied_mid, &p.ctl->tied_mid);
        if (BATCH) {
            if (v < p.v1 && !listed && !runs[u]) p.lab_out[v] = old[u];
            gc.add(p, v < p.v1 && !listed && runs[u] && nl[u] != old[u], g[u]);
        }
    }
    tb.flush(p.tied_mid, &p.ctl->tied_mid);
    if (!BATCH && p.changed) {  // the warp's changed vertices, with one addition to the list's length
        unsigned m[PER];
        int n = 0;
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            m[u] = __ballot_sync(kFull, small[u] && nl[u] != old[u]);
            n += __popc(m[u]);
        }
        int to = 0;
        if (lane == 0 && n) to = atomicAdd(&p.ctl->changed_n, n);
        to = __shfl_sync(kFull, to, 0);
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            if ((m[u] >> lane) & 1u) p.changed[to + __popc(m[u] & ((1u << lane) - 1u))] = (int32_t)(v0 + u * 32);
            to += __popc(m[u]);
        }
    }
    if (BATCH) gc.flush(p);
    flush_changes(changes, p.ctl);
}

template <bool BATCH>
__global__ void __launch_bounds__(kTB) resolve_mid_kernel(PipeArgs p)
{
    __shared__ int hist[kNW][256];
    if (!ctl_active(p.ctl)) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int nt = *((volatile int *)&p.ctl->tied_mid);
    unsigned long long changes = 0;
    for (int i = blockIdx.x * kNW + w; i < nt; i += gridDim.x * kNW) {
        const int v = p.tied_mid[i];
        const int32_t nl = resolve_mid(p, v, run_scope(p, v, p.runbase[v]), hist[w]);
        if (lane == 0) {
            const int32_t old = __ldg(&p.lab_in[v]);
            count_change(changes, nl, old);
            note_change(p, v, nl, old);
            if (BATCH) {
                const int g = __ldg(&p.gid[v]);
                const bool runs = __ldg(&p.g_active[g]) != 0;
                p.lab_out[v] = runs ? nl : old;
                if (runs && nl != old) atomicAdd(&p.g_changes[g], 1ull);
            } else {
                p.lab_out[v] = nl;
            }
        }
    }
    flush_changes(changes, p.ctl);
}

// Frontier: mark the neighbours of every vertex that changed in the previous iteration
// (the graph is symmetric, so they are exactly the vertices whose neighbour labels
// changed).  One warp per changed vertex.  When the dispatcher chose a full recount for
// this iteration (e.g. most labels changed, so marking would touch most of the graph)
// nothing is marked and ctl->frontier_off tells the count kernels.
__global__ void __launch_bounds__(kTB) mark_dirty_kernel(const int64_t *off, const int32_t *nbr,
                                                         const int32_t *changed, const DispatchState *disp, Ctl *ctl,
                                                         uint8_t *dirty)
{
    const int lane = threadIdx.x & 31;
    const int nc = *((volatile int *)&ctl->changed_n);
    const bool dense = !disp->frontier;
    if (blockIdx.x == 0 && threadIdx.x == 0) ctl->frontier_off = dense ? 1 : 0;
    if (dense) return;
    for (int64_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nc; i += (gridDim.x * blockDim.x) >> 5) {
        const int u = changed[i];
        const int64_t e0 = off[u], e1 = off[u + 1];
        for (int64_t e = e0 + lane; e < e1; e += 32) dirty[nbr[e]] = 1;
    }
}

// ---------------------------------------------------------------------------
// first iteration on strictly increasing adjacency lists
// ---------------------------------------------------------------------------
//
// With labels = vertex IDs (the reference's initialize_labels, dpp/kernel.cuh:15-22) and
// every adjacency list strictly increasing, each vertex's neighbour labels are distinct
// and already sorted: d = degree, every run has count 1 (all are candidates), the run
// base of v is offsets[v] and the scope holds N = m runs.  The winning run r follows
// from the closed form alone and its label is the neighbour ID at offsets[v] + r.

// Every distinct label is a candidate (k == d).
struct AllCandidates {
    int64_t d;
    __device__ int first_ge(int64_t x) const { return x < d ? (int)(x < 0 ? 0 : x) : -1; }
    __device__ int last_lt(int64_t y) const { return y > 0 ? (int)((y < d ? y : d) - 1) : -1; }
    __device__ int tile_pick(int64_t lo) const { return (int)(lo + kTile - 1); }
};

__global__ void __launch_bounds__(kTB) first_iteration_kernel(PipeArgs p, int64_t n, int64_t m)
{
    if (!ctl_active(p.ctl)) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) p.ctl->N = m;  // one run per CSR entry
    unsigned long long changes = 0;
    GraphChanges gc;
    const int lane = threadIdx.x & 31;
    for (int64_t vb = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; vb < n;
         vb += (int64_t)gridDim.x * blockDim.x) {  // warp-uniform
        const int64_t v = vb + lane;
        int g = 0;
        bool chg = false;
        if (v < n) {
            const int64_t o0 = __ldg(&p.off[v]);
            const int64_t deg = __ldg(&p.off[v + 1]) - o0;
            const int32_t old = __ldg(&p.lab_in[v]);
            int32_t nl = old;
            if (deg > 0) {
                AllCandidates q{deg};
                if (!p.g_v0) {
                    const int r = resolve_rank(o0, deg, m, v == p.last_v, q);
                    nl = __ldg(&p.nbr[o0 + r]);
                } else {  // graph-local run positions and labels
                    g = __ldg(&p.gid[v]);
                    const int64_t vg = p.g_v0[g], e0 = __ldg(&p.off[vg]), e1 = __ldg(&p.off[p.g_v0[g + 1]]);
                    const int r = resolve_rank(o0 - e0, deg, e1 - e0, v == p.g_last[g], q);
                    nl = (int32_t)(__ldg(&p.nbr[o0 + r]) - vg);
                }
            }
            p.lab_out[v] = nl;
            p.dcnt[v] = (int32_t)deg;  // every neighbour label distinct (insert-aggregation hint)
            count_change(changes, nl, old);
            note_change(p, (int32_t)v, nl, old);
            if (p.g_v0) {
                g = __ldg(&p.gid[v]);
                chg = nl != old;
            }
        }
        if (p.g_v0) gc.add(p, chg, g);
    }
    if (p.g_v0) gc.flush(p);
    flush_changes(changes, p.ctl);
}

// Setup checks without the symmetry checksum, as two streaming passes:
//   csr_scan_kernel:     out[3] += neighbour IDs outside [0, n); out[0] += entries e >= 1
//                        with nbr[e] <= nbr[e-1] (all descents, row boundaries included);
//   row_start_kernel:    out[4] += those descents that sit at a row start (e = offsets[v]
//                        of a vertex with neighbours), which do not count.
// Adjacency lists are strictly increasing when out[0] == out[4].
__global__ void __launch_bounds__(kTB) csr_scan_kernel(const int32_t *nbr, int64_t m, int64_t n,
                                                       unsigned long long *out)
{
    unsigned long long desc = 0, outside = 0;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < m; e += (int64_t)gridDim.x * blockDim.x) {
        const int32_t u = __ldg(&nbr[e]);
        outside += (u < 0 || u >= n);
        if (e > 0) desc += (u <= __ldg(&nbr[e - 1]));
    }
    desc = __reduce_add_sync(kFull, (unsigned)desc);
    outside = __reduce_add_sync(kFull, (unsigned)outside);
    if ((threadIdx.x & 31) == 0) {
        if (desc) atomicAdd(&out[0], desc);
        if (outside) atomicAdd(&out[3], outside);
    }
}

__global__ void __launch_bounds__(kTB) row_start_kernel(const int64_t *off, const int32_t *nbr, int64_t n,
                                                        unsigned long long *out)
{
    unsigned long long b = 0;
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const int64_t e = off[v];
        if (e > 0 && off[v + 1] > e) b += (__ldg(&nbr[e]) <= __ldg(&nbr[e - 1]));
    }
    b = __reduce_add_sync(kFull, (unsigned)b);
    if ((threadIdx.x & 31) == 0 && b) atomicAdd(&out[4], b);
}

// One pass over the resident CSR at setup (warp per 32 consecutive vertices, lanes over
// the warp's edge range, row of each edge by a shuffle binary search over the 33 offsets):
//   out[3] += neighbour IDs outside [0, n) (the graph is rejected);
//   out[0] += adjacent entries of one row that are not strictly increasing
//             (0 enables the first-iteration shortcut);
//   out[1], out[2] += sum over entries (v, u) of g(v)k(u) - g(u)k(v) (mod 2^64) for two
//             hash pairs g, k.  The form is antisymmetric, so every graph whose edge
//             multiset is symmetric sums to 0 in both; an asymmetric one does so only by a
//             hash collision (about 2^-64 per sum).  Both 0 enables the frontier, whose
//             dirty marking pushes along out-edges.  Computed only when want_sym.
__device__ __forceinline__ uint64_t adj_hash(uint64_t x, uint64_t salt)
{
    return splitmix64_mix(x * 0x9E3779B97F4A7C15ull + salt);
}

__global__ void __launch_bounds__(kTB) adjacency_check_kernel(const int64_t *off, const int32_t *nbr, int64_t n,
                                                              int want_sym, unsigned long long *out)
{
    const int lane = threadIdx.x & 31;
    const int64_t nwb = (n + 31) >> 5;
    unsigned long long desc = 0, s1 = 0, s2 = 0, outside = 0;
    for (int64_t wb = (int64_t)(blockIdx.x * blockDim.x + threadIdx.x) >> 5; wb < nwb;
         wb += (int64_t)(gridDim.x * blockDim.x) >> 5) {
        const int64_t vb = wb << 5;
        const int64_t o = off[min(vb + lane, n)];  // lanes past n hold off[n]
        const int64_t oend = off[min(vb + 32, n)];
        const int64_t e_begin = __shfl_sync(kFull, o, 0);
        int32_t carry = 0;  // last entry of the previous chunk
        for (int64_t c = e_begin; c < oend; c += 32) {
            const int64_t e = c + lane;
            int r = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) {
                const int64_t oc = __shfl_sync(kFull, o, r + step);
                if (oc <= e) r += step;
            }
            const bool valid = e < oend;
            const int32_t u = valid ? __ldg(&nbr[e]) : 0;
            int32_t prev = __shfl_up_sync(kFull, u, 1);
            if (lane == 0) prev = carry;
            carry = __shfl_sync(kFull, u, 31);
            const int64_t row_start = __shfl_sync(kFull, o, r);
            if (valid) {
                if (e != row_start && u <= prev) ++desc;
                outside += (u < 0 || u >= n);
            }
            if (valid && want_sym) {
                const uint64_t v = (uint64_t)(vb + r);
                s1 += adj_hash(v, 0x1234567ull) * adj_hash((uint64_t)u, 0xABCDEF1ull) -
                      adj_hash((uint64_t)u, 0x1234567ull) * adj_hash(v, 0xABCDEF1ull);
                s2 += adj_hash(v, 0x7777777ull) * adj_hash((uint64_t)u, 0x3141592ull) -
                      adj_hash((uint64_t)u, 0x7777777ull) * adj_hash(v, 0x3141592ull);
            }
        }
    }
#pragma unroll
    for (int sh = 16; sh > 0; sh >>= 1) {
        desc += __shfl_xor_sync(kFull, desc, sh);
        s1 += __shfl_xor_sync(kFull, s1, sh);
        s2 += __shfl_xor_sync(kFull, s2, sh);
        outside += __shfl_xor_sync(kFull, outside, sh);
    }
    if (lane == 0) {
        if (desc) atomicAdd(&out[0], desc);
        if (want_sym) {
            atomicAdd(&out[1], s1);
            atomicAdd(&out[2], s2);
        }
        if (outside) atomicAdd(&out[3], outside);
    }
}

// ---------------------------------------------------------------------------
// batched mode: many independent graphs in one concatenated CSR
// ---------------------------------------------------------------------------

// Graph of every vertex (set up once).  One block per graph (grid-stride).
__global__ void __launch_bounds__(kTB) batch_gid_kernel(const int64_t *g_v0, int ngraphs, int32_t *gid)
{
    for (int g = blockIdx.x; g < ngraphs; g += gridDim.x)
        for (int64_t v = g_v0[g] + threadIdx.x; v < g_v0[g + 1]; v += blockDim.x) gid[v] = g;
}

// Initial labels: graph-local vertex IDs.  One block per graph (grid-stride).
// Sets *bad when an edge leaves its graph.  One block per graph (grid-stride).
__global__ void __launch_bounds__(kTB) batch_validate_kernel(const int64_t *off, const int32_t *nbr,
                                                             const int64_t *g_v0, int ngraphs, int *bad)
{
    for (int g = blockIdx.x; g < ngraphs; g += gridDim.x) {
        const int64_t v0 = g_v0[g], v1 = g_v0[g + 1];
        int b = 0;
        for (int64_t e = off[v0] + threadIdx.x; e < off[v1]; e += blockDim.x) {
            const int64_t u = nbr[e];
            b |= (u < v0 || u >= v1);
        }
        if (__any_sync(kFull, b) && (threadIdx.x & 31) == 0) atomicOr(bad, 1);
    }
}

__global__ void __launch_bounds__(kTB) batch_init_labels_kernel(const int64_t *g_v0, int ngraphs, int32_t *lab)
{
    for (int g = blockIdx.x; g < ngraphs; g += gridDim.x) {
        const int64_t v0 = g_v0[g], v1 = g_v0[g + 1];
        for (int64_t v = v0 + threadIdx.x; v < v1; v += blockDim.x) lab[v] = (int32_t)(v - v0);
    }
}

// After an iteration of a batch: per graph, the labels that changed and the reference's early
// exit (count <= n_g * 1e-5, dpp.cuh:88); the run goes on while some graph is active.  One thread
// per graph; the block that ends last keeps the run's books.
// Also the next iteration's dispatch state, where there is one (a.out).
constexpr int kFinalThreads = 1024;
__global__ void __launch_bounds__(kFinalThreads) batch_finalize_kernel(Ctl *ctl, const int64_t *g_v0, int32_t *g_active,
                                                                       int32_t *g_iters, long long *g_counts,
                                                                       unsigned long long *g_changes, int ngraphs,
                                                                       int max_iter, int it, int early_exit,
                                                                       DispatchArgs a)
{
    __shared__ int any, last;
    const bool several = gridDim.x > 1;
    if (threadIdx.x == 0) any = 0;
    __syncthreads();
    const bool on = ctl_active(ctl);  // else every graph ended earlier: all is settled
    for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; on && g < ngraphs;
         g += (int64_t)gridDim.x * blockDim.x) {
        if (!g_active[g]) continue;
        const unsigned long long t = g_changes[g];
        g_changes[g] = 0;
        if (it < max_iter) g_counts[g * max_iter + it] = (long long)t;
        g_iters[g] = it + 1;
        if ((early_exit && (double)t <= (double)(g_v0[g + 1] - g_v0[g]) * 1e-5) || it + 1 >= max_iter) g_active[g] = 0;
        else any = 1;
    }
    __syncthreads();
    if (several) {
        if (threadIdx.x == 0) {
            if (any) atomicExch(&ctl->more, 1);
            __threadfence();
            last = atomicAdd(&ctl->ticket, 1ull) == gridDim.x - 1;
        }
        __syncthreads();
        if (!last) return;
    }
    if (threadIdx.x == 0) {
        if (on) {
            const bool more = several ? atomicExch(&ctl->more, 0) != 0 : any != 0;
            const unsigned long long c = ctl->changes;
            ctl->last = c;
            if (ctl->iter < 64) ctl->counts[ctl->iter] = c;
            ctl->iter += 1;
            if (!more || ctl->iter >= ctl->max_iter) ctl->active = 0;
        }
        ctl->changes = 0;
        ctl->ticket = 0;
    }
    if (a.out) {
        __syncthreads();
        dispatch_step(a);
    }
}

__global__ void batch_init_kernel(int32_t *g_active, int32_t *g_iters, unsigned long long *g_changes, int ngraphs,
                                  int active)
{
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < ngraphs; g += gridDim.x * blockDim.x) {
        g_active[g] = active;
        g_iters[g] = 0;
        g_changes[g] = 0;
    }
}

}  // namespace galp
