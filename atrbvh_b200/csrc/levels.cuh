// The bottom-up order of a treelet pass, shared by the ATRBVH and TRBVH
// optimisers: node records, the level of every treelet root, the roots listed
// level by level, and the cluster that takes small ATRBVH trees' narrow levels.
#pragma once

#include "common.cuh"
#include "internal.h"
#include "treelet.cuh"

namespace atr {
namespace {

// The optimiser's per-node record, node-indexed in the batch layout (one
// 16-byte load gives a treelet leaf everything but its box):
//   x  subtree triangle count;
//   y  nodesSah of even iterations, z  nodesSah of odd iterations -- this
//      iteration's in component 1 + par (par = iteration & 1), the next
//      iteration's in the other;
//   w  big-node level: this iteration's until the node is finished, the next
//      iteration's after (only the level lists, built before any node is
//      finished, read this iteration's).
// The reference recomputes nodesSah bottom-up every iteration as
// (ci*A + left) + right, while a rewritten node stores the merge cost
// (left + right) + ci*A; the two can differ in the last bit, so the next
// iteration's values are kept in the recomputation's order.
__device__ __forceinline__ int rec_ns_cur(int par) { return 1 + par; }
__device__ __forceinline__ int rec_ns_next(int par) { return 2 - par; }
__device__ __forceinline__ float* rec_f(int4* r, int x, int c) { return reinterpret_cast<float*>(r + x) + c; }
__device__ __forceinline__ int* rec_i(int4* r, int x, int c) { return reinterpret_cast<int*>(r + x) + c; }
// A record from its fields, the nodesSah values placed by parity.
__device__ __forceinline__ int4 make_rec(int cnt, float ns_cur, float ns_next, int lvl, int par) {
    return par ? make_int4(cnt, __float_as_int(ns_next), __float_as_int(ns_cur), lvl)
               : make_int4(cnt, __float_as_int(ns_cur), __float_as_int(ns_next), lvl);
}

// formTreelet's argmax tree (Treelet.cuh:23-39) over m lanes -- lane i takes
// lane i + floor(c/2) when that value is strictly larger, c halving upward --
// returns the largest value and, among equal largest values, the lane that
// comes first in a fixed order that depends only on m.  tree_winner replays
// the tree on a tie pattern; argmax_priority ranks the lanes by removing
// winners one at a time.  The full-warp path then needs two warp reductions:
// the maximum value, then the lowest rank among the lanes holding it.
// The kernels copy the table to shared memory four bytes at a time.
struct alignas(16) ArgmaxPriority {
    uint8_t rank[kMaxTreelet + 1][32];
};
static_assert(alignof(ArgmaxPriority) >= sizeof(uint32_t) && sizeof(ArgmaxPriority) % sizeof(uint32_t) == 0,
              "whole aligned words");

constexpr int tree_winner(int m, uint32_t tied) {
    int val[32] = {};
    int idx[32] = {};
    for (int i = 0; i < 32; ++i) {
        val[i] = (i < m && ((tied >> i) & 1u)) ? 1 : 0;
        idx[i] = i;
    }
    int c = m, sh = m / 2;
    while (c > 1) {
        for (int i = 0; i < c - sh; ++i)  // ascending: lane i + sh is read before it is updated
            if (val[i + sh] > val[i]) {
                val[i] = val[i + sh];
                idx[i] = idx[i + sh];
            }
        c = (c + 1) / 2;
        sh = c / 2;
    }
    return idx[0];
}

constexpr ArgmaxPriority argmax_priority() {
    ArgmaxPriority t{};
    for (int m = 0; m <= kMaxTreelet; ++m)
        for (int i = 0; i < 32; ++i) t.rank[m][i] = 255;
    for (int m = 1; m <= kMaxTreelet; ++m) {
        uint32_t rem = m == 32 ? 0xffffffffu : ((1u << m) - 1u);
        int k = 0;
        while (rem) {
            const int w = tree_winner(m, rem);
            t.rank[m][w] = (uint8_t)k++;
            rem &= ~(1u << w);
        }
    }
    return t;
}

__device__ const ArgmaxPriority g_argmax_priority = argmax_priority();

// ---- level passes ---------------------------------------------------------------
// A node whose subtree holds at least gamma triangles ("big") is a treelet
// root; its results depend only on its subtree, so any order that finishes a
// node's big descendants first gives the reference's result.  The level of a
// big node is 1 + the largest level of its big children (0 for the others).
// Phase A finishes every node that is not big (subtree count, nodesSah, child
// record) and levels the big ones: k_levels climbs once from every leaf;
// k_levels_pp and k_levels_pp_hist take counts, nodesSah (and levels) from
// the LBVH build.  Phase B files big nodes of levels 1..L into per-level
// lists (in the same pass as the level counts: k_levels_pp_hist for the first
// iteration, k_level_hist for the others); phase C restructures each level's
// treelets in one launch, several per warp in lane groups; the dataflow kernel
// then climbs from the frontier below the levels above L.

constexpr int kMaxLevels = 64;  // largest L (ATR_TUNE_ATR_LEVELS)
constexpr int kListPer = 8;                  // nodes per thread of the level-list kernels
constexpr int kListBlock = 256 * kListPer;  // nodes per block of those kernels
// Nodes whose reads a thread of those kernels requests at once.  The passes are
// bound by latency and by their warps in flight: one node after another, each
// with its warp scan for the frontier, ATRBVH took 1,826 us at 4,194,304
// triangles and 5,252 at 16.8M; two at once (48 registers) and the scan only in
// warps that hold a node above the level passes 1,807 and 5,176, four (58) 1,814
// and 5,181, eight (74) 1,828 and 5,223.
constexpr int kListAhead = 2;
static_assert(kListPer % kListAhead == 0, "whole batches of nodes");

struct LevelRefs {
    int4* rec;             // per node (node-indexed): count, nodesSah x 2, level (see NextRefs)
    int par;               // iteration & 1
    float ct;              // the leaf cost constant (triangle leaves' records)
    uint32_t* counters;
    int4* kids;
    uint32_t* cursor;      // [L + 2]: entries filed per level (the level's count)
    uint2* order;          // (mesh, local node) of big nodes: level l's list at (l - 1) * cap
    uint32_t cap;          // entries per level list (at most n / gamma nodes share a level)
    uint2* frontier;       // climb starts of the dataflow pass
    uint32_t* n_frontier;
    uint2* top;            // (mesh, local node) of the big nodes above level L, the first kTopCap
    uint32_t* n_top;       // how many there are
    uint32_t* err;
};

// Lists a block's big nodes above level L (one atomic per warp).
constexpr uint32_t kTopCap = 2048;
__device__ __forceinline__ void list_top(const LevelRefs& lv, bool is_top, uint2 ent) {
    const uint32_t b = __ballot_sync(kFull, is_top);
    if (!b) return;
    uint32_t at = 0;
    if ((threadIdx.x & 31) == (uint32_t)(__ffs(b) - 1)) at = atomicAdd(lv.n_top, (uint32_t)__popc(b));
    at = __shfl_sync(kFull, at, __ffs(b) - 1) + __popc(b & lanemask_lt());
    if (is_top && at < kTopCap) lv.top[at] = ent;
}

constexpr int kLvBlock = 512;  // threads (leaves) per block of the phase-A climb

// Phase A of the first iteration: one climb from every leaf (sorted order)
// that finishes the nodes that are not treelet roots and levels the roots.
// With the radix tree's leaf ranges (a tree straight from the LBVH build), a
// node whose range lies inside the block's leaves is reached only by threads
// of the block, so its arrival counter and the first child's summary live in
// shared memory under block-scope ordering; only nodes whose range crosses a
// block boundary use a device-scope acquire-release atomic in global memory.
// Without ranges every node takes the global path.
__global__ void __launch_bounds__(kLvBlock) k_levels(TreeRefs g, Segs segs, LevelRefs lv, int tsize_all,
                                                     const uint8_t* __restrict__ seg_tsize,
                                                     const uint8_t* __restrict__ seg_iters, int iteration, float ci,
                                                     float ct, int L, const int2* __restrict__ ranges) {
    __shared__ uint32_t s_ctr[kLvBlock];
    __shared__ int4 s_rec[kLvBlock][2];  // per local node and side: (count, level, nodesSah, area)
    for (int k = threadIdx.x; k < kLvBlock; k += blockDim.x) s_ctr[k] = 0;
    __syncthreads();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= segs.n) return;
    const uint32_t m = segs.seg_of_tri(i);
    if (seg_iters && iteration >= (int)seg_iters[m]) return;
    const uint32_t s0 = segs.tri_begin(m);
    const uint32_t n = segs.tri_end(m) - s0;
    const int base = segs.node_base(m), cb = segs.inner_base(m);
    const int gamma = (seg_tsize ? (int)seg_tsize[m] : tsize_all) << iteration;
    const int64_t blo = (int64_t)blockIdx.x * blockDim.x, bhi = blo + blockDim.x - 1;
    const int li = (int)(i - s0);
    const int leaf = base + li + (int)n - 1;
    // Summary of the subtree this thread has just finished (the leaf first).
    const float la = g.area[leaf];
    int my_cnt = 1, my_lvl = 0, my_first = li, child = li + (int)n - 1;
    float my_nsah = __fmul_rn(ct, la), my_area = la;
    lv.rec[leaf] = make_int4(1, __float_as_int(my_nsah), __float_as_int(my_nsah), 0);
    const int cur_c = rec_ns_cur(lv.par);
    int cur = g.parent[leaf];
    while (cur >= 0) {
        const int x = base + cur;
        int sib_cnt, sib_lvl;
        float sib_nsah, sib_area;
        bool local = false;
        if (ranges) {
            const int2 rg = ranges[cb + cur];
            local = (int64_t)s0 + rg.x >= blo && (int64_t)s0 + rg.y <= bhi;
            if (local) {
                // Internal node cur covers [rg.x, rg.y] and is numbered by one
                // of its ends, so its slot lies inside the block.
                const int slot = (int)((int64_t)s0 + cur - blo);
                const int side = my_first == rg.x ? 0 : 1;
                s_rec[slot][side] = make_int4(my_cnt, my_lvl, __float_as_int(my_nsah), __float_as_int(my_area));
                __threadfence_block();
                if (atomicAdd(&s_ctr[slot], 1u) == 0u) return;
                __threadfence_block();
                const int4 r = s_rec[slot][side ^ 1];
                sib_cnt = r.x;
                sib_lvl = r.y;
                sib_nsah = __int_as_float(r.z);
                sib_area = __int_as_float(r.w);
                my_first = rg.x;
            }
        }
        const int lc = ld_cg(g.left + x), rc = ld_cg(g.right + x);
        const int sib = lc == child ? rc : lc;
        if (!local) {
            if (atomic_add_acq_rel_gpu(&lv.counters[cb + cur], 1u) == 0u) return;
            const int4 sr = __ldcg(lv.rec + base + sib);
            sib_cnt = sr.x;
            sib_lvl = is_internal(sib, n) ? sr.w : 0;
            sib_nsah = __int_as_float(cur_c == 1 ? sr.y : sr.z);
            sib_area = ld_cg(g.area + base + sib);
            if (ranges) my_first = min(my_first, ranges[cb + cur].x);
        }
        const bool mine_left = lc == child;
        const int cnt = my_cnt + sib_cnt;
        const float a = ld_cg(g.area + x);
        lv.kids[cb + cur] = make_int4(lc, rc, __float_as_int(mine_left ? my_area : sib_area),
                                      __float_as_int(mine_left ? sib_area : my_area));
        int lvl = 0;
        float ns = 0.0f;
        if (cnt < gamma) {
            ns = __fadd_rn(__fadd_rn(__fmul_rn(ci, a), mine_left ? my_nsah : sib_nsah), mine_left ? sib_nsah : my_nsah);
            lv.rec[x] = make_int4(cnt, __float_as_int(ns), __float_as_int(ns), 0);
        } else {
            lvl = 1 + max(my_lvl, sib_lvl);
            *rec_i(lv.rec, x, 0) = cnt;
            *rec_i(lv.rec, x, 3) = lvl;
        }
        my_cnt = cnt;
        my_lvl = lvl;
        my_nsah = ns;  // only read while the climb stays below the treelet roots (cnt < gamma)
        my_area = a;
        child = cur;
        cur = g.parent[x];
    }
}

// Files a block's nodes of levels 1..L into the level lists: thread-held
// levels me[q] (0: none) and entries ent[q].  Ranks within the block come from
// one shared atomic per level present in a warp (__match_any_sync), then one
// global reservation per level per block on lv.cursor (which ends as the
// level's count).  Nodes of one level have disjoint subtrees of at least gamma
// triangles each, so a list holds at most lv.cap of them; a reservation past
// that sets kErrLevelList and writes nothing.  Every thread of the block calls
// it; s_cnt holds L + 2 zeroed counters.
__device__ __forceinline__ void file_levels(const LevelRefs& lv, int L, const int (&me)[kListPer],
                                            const uint2 (&ent)[kListPer], uint32_t* s_cnt, uint32_t* s_base) {
    const int lane = threadIdx.x & 31;
    uint32_t key[kListPer];
#pragma unroll
    for (int q = 0; q < kListPer; ++q) {
        const uint32_t peers = __match_any_sync(kFull, me[q]);
        const int leader = __ffs(peers) - 1;
        uint32_t b = 0;
        if (lane == leader && me[q] > 0) b = atomicAdd(&s_cnt[me[q]], (uint32_t)__popc(peers));
        b = __shfl_sync(kFull, b, leader) + (uint32_t)__popc(peers & ((1u << lane) - 1u));
        key[q] = me[q] > 0 ? ((uint32_t)me[q] << 16) | b : 0u;  // rank < kListBlock
    }
    __syncthreads();
    for (int k = threadIdx.x; k < L + 2; k += blockDim.x)
        s_base[k] = s_cnt[k] ? atomicAdd(&lv.cursor[k], s_cnt[k]) : 0u;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kListPer; ++q)
        if (key[q]) {
            const uint32_t l = key[q] >> 16;
            const uint32_t at = s_base[l] + (key[q] & 0xffffu);
            if (at < lv.cap) lv.order[(size_t)(l - 1) * lv.cap + at] = ent[q];
            else set_error_bits(lv.err, kErrLevelList);
        }
}

// A block's big nodes above level L (one per thread, m and x) go to the top
// list, and their children at levels up to L to the dataflow pass's frontier.
__device__ __forceinline__ void list_above(const Segs& segs, const LevelRefs& lv, bool above, uint32_t m, uint32_t x,
                                           int lc, int rc, int L) {
    if (!__any_sync(kFull, above)) return;  // nearly every warp: a few hundred nodes are above
    list_top(lv, above, make_uint2(m, x));
    bool pl = false, pr = false;
    if (above) {
        const uint32_t n = segs.tri_end(m) - segs.tri_begin(m);
        const int nb = segs.node_base(m);
        pl = (is_internal(lc, n) ? *rec_i(lv.rec, nb + lc, 3) : 0) <= L;
        pr = (is_internal(rc, n) ? *rec_i(lv.rec, nb + rc, 3) : 0) <= L;
    }
    // Frontier entries: one atomic per warp.
    const uint32_t push = pl + pr;
    uint32_t incl = push;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, incl, o);
        if ((threadIdx.x & 31) >= o) incl += y;
    }
    const uint32_t total = __shfl_sync(kFull, incl, 31);
    uint32_t at = 0;
    if ((threadIdx.x & 31) == 31 && total) at = atomicAdd(lv.n_frontier, total);
    at = __shfl_sync(kFull, at, 31) + incl - push;
    if (pl) lv.frontier[at++] = make_uint2(m, (uint32_t)lc);
    if (pr) lv.frontier[at] = make_uint2(m, (uint32_t)rc);
}

// Phase A of iterations after the first: the previous iteration left every
// internal node's level for this one (next levels of the nodes it finished,
// kept current by treelet rewrites), and subtree counts, nodesSah and child
// records that are already final for nodes that are not treelet roots now.
// Count the levels, mark this iteration's non-roots as non-roots for the next
// one too, and list the frontier below the levels above L.
__global__ void __launch_bounds__(256) k_level_hist(Segs segs, LevelRefs lv, const uint8_t* __restrict__ seg_iters,
                                                    int iteration, int L) {
    __shared__ uint32_t s_cnt[kMaxLevels + 2];
    __shared__ uint32_t s_base[kMaxLevels + 2];
    for (int k = threadIdx.x; k < L + 2; k += blockDim.x) s_cnt[k] = 0;
    __syncthreads();
    int lvl[kListPer];
    uint2 lent[kListPer];
#pragma unroll
    for (int q0 = 0; q0 < kListPer; q0 += kListAhead) {
        int4 rec[kListAhead];
#pragma unroll
        for (int u = 0; u < kListAhead; ++u) {
            const uint32_t i = blockIdx.x * kListBlock + (q0 + u) * 256 + threadIdx.x;
            rec[u] = make_int4(0, 0, 0, -1);  // nothing to do
            lent[q0 + u] = make_uint2(0u, 0u);
            if (i < segs.n) {
                const uint32_t m = segs.seg_of_tri(i);
                const uint32_t s0 = segs.tri_begin(m);
                if ((!seg_iters || iteration < (int)seg_iters[m]) && i - s0 < segs.tri_end(m) - s0 - 1) {
                    lent[q0 + u] = make_uint2(m, i - s0);
                    rec[u] = lv.rec[segs.node_base(m) + (int)(i - s0)];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kListAhead; ++u) {
            const int q = q0 + u, me = rec[u].w;
            const uint32_t m = lent[q].x, x = lent[q].y;
            // Not a treelet root: its next nodesSah is this one (the level stays 0).
            if (me == 0)
                *rec_i(lv.rec, segs.node_base(m) + (int)x, rec_ns_next(lv.par)) = lv.par ? rec[u].z : rec[u].y;
            lvl[q] = me > 0 && me <= L ? me : 0;
            const bool above = me > L;
            int4 kd = make_int4(0, 0, 0, 0);
            if (above) kd = lv.kids[segs.inner_base(m) + (int)x];
            list_above(segs, lv, above, m, x, kd.x, kd.y, L);
        }
    }
    file_levels(lv, L, lvl, lent, s_cnt, s_base);
}

// ---- the top of the tree ------------------------------------------------------
// Above the levels that the level passes take, a level holds a few hundred
// roots down to one, so a level costs one treelet's latency plus whatever
// starts it.  One cluster of CTAs takes all of these levels in one launch: the
// roots are sorted by level once, a warp takes a root, and a hardware cluster
// barrier (release/acquire) stands between levels, in place of a launch per
// level or of the dataflow pass's fence, arrival atomic and sibling load per
// node.  A tree whose top does not fit (more than kTopCap roots or kTopLevels
// levels) is left to the dataflow pass, whose arrival counters are then cleared
// here; otherwise that pass's frontier is emptied.
// Bound by a treelet's latency, about 11,500 cycles on an idle SM (formation
// 3,800, leaves' data 900, merge 4,500, rewrite 900), and 2,000 for the barrier.
constexpr int kTopWarps = 16;  // warps per CTA
constexpr int kTopLevels = 512;

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

struct TopRefs {
    uint2* sorted;       // [kTopCap] roots by level
    uint32_t* offset;    // [kTopLevels + 1] start of each level above L
    uint32_t* levels;    // how many there are, or ~0: the top does not fit
    size_t counters;     // arrival counters to clear then
};

// f(root) by one warp for every listed root, level by level.  Every thread of the
// cluster calls it; s_off (kTopLevels + 1 words) and s_max are shared scratch.
template <class F>
__device__ __forceinline__ void top_levels(const Segs& segs, const LevelRefs& lv, const TopRefs& tr, int L,
                                           uint32_t* s_off, uint32_t* s_max, F f) {
    constexpr int T = kTopWarps * 32;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const uint32_t rank = blockIdx.x, ctas = gridDim.x;
    const uint32_t k_top = *lv.n_top;
    if (k_top == 0) return;  // no node above L (the frontier is empty too); the same in every CTA
    if (rank == 0) {
        // Counting sort by level.
        constexpr int kPer = kTopCap / T;
        uint2 ent[kPer];
        uint32_t lev[kPer];
        for (int k = tid; k <= kTopLevels; k += T) s_off[k] = 0;
        if (tid == 0) *s_max = 0;
        __syncthreads();
        const bool fits = k_top <= kTopCap;
#pragma unroll
        for (int q = 0; q < kPer; ++q) {
            const uint32_t k = q * T + tid;
            lev[q] = 0xffffffffu;
            if (fits && k < k_top) {
                ent[q] = lv.top[k];
                lev[q] = (uint32_t)(*rec_i(lv.rec, segs.node_base(ent[q].x) + (int)ent[q].y, 3) - L - 1);
                atomicMax(s_max, lev[q]);
                if (lev[q] < (uint32_t)kTopLevels) atomicAdd(&s_off[lev[q] + 1], 1u);
            }
        }
        __syncthreads();
        const bool ok = fits && *s_max < (uint32_t)kTopLevels;
        if (ok) {
            if (w == 0) {  // inclusive scan of s_off[1..kTopLevels]
                constexpr int kRun = kTopLevels / 32;
                uint32_t sum = 0;
#pragma unroll
                for (int j = 0; j < kRun; ++j) sum += s_off[1 + lane * kRun + j];
                uint32_t inc = sum;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(kFull, inc, o);
                    if (lane >= o) inc += y;
                }
                uint32_t run = inc - sum;
#pragma unroll
                for (int j = 0; j < kRun; ++j) {
                    run += s_off[1 + lane * kRun + j];
                    s_off[1 + lane * kRun + j] = run;
                }
            }
            __syncthreads();
            for (int k = tid; k <= kTopLevels; k += T) tr.offset[k] = s_off[k];
            __syncthreads();
#pragma unroll
            for (int q = 0; q < kPer; ++q)
                if (lev[q] != 0xffffffffu) tr.sorted[atomicAdd(&s_off[lev[q]], 1u)] = ent[q];
        }
        if (tid == 0) *tr.levels = ok ? *s_max + 1 : 0xffffffffu;
    }
    cluster_barrier();
    const uint32_t levels = __ldcg(tr.levels);
    if (levels == 0xffffffffu) {
        for (size_t k = (size_t)rank * T + tid; k < tr.counters; k += (size_t)ctas * T) lv.counters[k] = 0;
        return;
    }
    if (rank == 0 && tid == 0) *lv.n_frontier = 0;
    for (uint32_t k = tid; k <= levels; k += T) s_off[k] = __ldcg(tr.offset + k);
    __syncthreads();
    for (uint32_t l = 0; l < levels; ++l) {
        const uint32_t end = s_off[l + 1];
        // Consecutive roots go to different CTAs.
        for (uint32_t e = s_off[l] + (uint32_t)w * ctas + rank; e < end; e += (uint32_t)kTopWarps * ctas)
            f(__ldcg(tr.sorted + e));
        __syncwarp();
        cluster_barrier();
    }
}

// Launch shape of a top kernel: one cluster.
inline cudaLaunchConfig_t top_config(int ctas, cudaLaunchAttribute* at, cudaStream_t s) {
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = (unsigned)ctas;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(kTopWarps * 32);
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

// The largest cluster `kernel` may be launched with: 16 CTAs (above 8 is
// non-portable) where the device runs such a cluster, else 8.
template <class K>
int top_cluster(K kernel, int* ctas) {
    ATR_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchAttribute at{};
    const cudaLaunchConfig_t cfg = top_config(16, &at, nullptr);
    int clusters = 0;
    const cudaError_t e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg);
    if (e != cudaSuccess) cudaGetLastError();
    *ctas = e == cudaSuccess && clusters > 0 ? 16 : 8;
    return ATR_OK;
}

// Level passes of an iteration with this gamma: every level expected to hold
// more than kTopWidth roots (a level pass over fewer takes one treelet's
// latency, which the cluster of the top kernel does without a launch).  Roots
// per level fall by about 0.62 per level from n / (1.5 gamma) at level 1.
constexpr double kTopWidth = 200.0;
inline double level_roots(uint32_t n, int gamma) { return (double)n / (1.5 * (double)gamma); }
inline int auto_levels(uint32_t n, int gamma) {
    int L = 1;
    for (double r = level_roots(n, gamma) * 0.62; L < kMaxLevels && r > kTopWidth; r *= 0.62) ++L;
    return L;
}

// Scratch of the level lists.  Big nodes of one level root disjoint subtrees of
// at least gamma0 triangles (the smallest gamma), so each level's list holds at
// most n / gamma0; frontier nodes root disjoint subtrees too, so they number at
// most the triangles.
struct LevelScratch {
    int L;
    uint32_t n, cap;
    size_t b_ord, b_front, b_small, b_top;
    LevelScratch(uint32_t n_, uint32_t gamma0, int L_) : L(L_), n(n_) {
        cap = (n + gamma0 - 1) / gamma0;
        b_ord = align256((size_t)L * cap * 8);
        b_front = align256((size_t)n * 8);
        b_small = align256((size_t)((L + 2) + 2) * 4);
        b_top = align256(2 * kTopCap * sizeof(uint2) + (kTopLevels + 2) * 4);
    }
    size_t bytes() const { return L ? b_ord + b_front + b_small + b_top : 0; }
    void bind(char* p, size_t inner, uint32_t* d_error, LevelRefs& lv, TopRefs& tr) const {
        lv.order = reinterpret_cast<uint2*>(p); p += b_ord;
        lv.cap = cap;
        lv.err = d_error;
        lv.frontier = reinterpret_cast<uint2*>(p); p += b_front;
        lv.cursor = reinterpret_cast<uint32_t*>(p); p += b_small;
        lv.n_frontier = lv.cursor + (L + 2);
        lv.n_top = lv.n_frontier + 1;
        lv.top = reinterpret_cast<uint2*>(p);
        tr.sorted = lv.top + kTopCap;
        tr.offset = reinterpret_cast<uint32_t*>(tr.sorted + kTopCap);
        tr.levels = tr.offset + kTopLevels + 1;
        tr.counters = inner;
    }
};

}  // namespace
}  // namespace atr
