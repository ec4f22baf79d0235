// TRBVH: treelet restructuring by dynamic programming over leaf subsets
// (Karras & Aila 2013), treelet size 7, on sm_100a.
//
// Semantics follow BVHRT-Core/src/TRBVH.cu:329-479 and TRBVHOptimizer.cpp:91-106:
// the same bottom-up pass as ATRBVH; per treelet the 128 subset boxes and
// areas, leaf costs = nodesSah, and for every subset S of 2..7 leaves
//   C(S) = min(ci*A(S) + min_P [C(P) + C(S\P)], ct*A(S)*T)
// with T the treelet's triangle count (:126-128).  Partitions are enumerated
// and reduced exactly as the reference does (sizes 2..5 one lane per subset,
// (p - delta) & S order; size 6 four lanes per subset; size 7 all 32 lanes; the
// lower lane keeps ties), so the chosen partitions match.  The rebuild
// (:222-327) proceeds round by round; in each round left children take
// internal nodes before right children, each in lane order, and a right
// child's nodesSah is written from the left partition's cost as in :309.
// Subset boxes, costs and masks live in shared memory (the reference keeps
// the boxes in a per-warp global scratch buffer).
//
// An iteration runs level by level as ATRBVH's does (levels.cuh): one climb
// from every leaf finishes the nodes that are not treelet roots and levels the
// roots, one pass lists them, then each level's treelets are restructured in one
// launch, a warp each; the dataflow kernel k_trbvh takes the narrow levels above.
// Bound by the subset programme's issue on the wide levels and by one treelet's
// latency on the narrow ones.  300,007 uniform triangles, 3 iterations:
// 1.59 -> 0.90 ms against one climb that restructured treelets as its warps
// reached them (a warp's up to eight one after another, 17 % of the warps
// resident).  ATRBVH's cluster for the narrow levels is no gain here, cluster |
// dataflow: 1,003 triangles 304 | 288 us, 65,536 568 | 562, 262,144 850 | 843,
// 1,000,003 1,791 | 1,783, 16.8M 22.09 | 22.11 ms.

#include "common.cuh"
#include "internal.h"
#include "levels.cuh"
#include "treelet.cuh"

namespace atr {
namespace {

constexpr int kTrWarps = 8;
constexpr int kTr = 7;
constexpr int kSubsets = 1 << kTr;

struct TrShared {
    float mnx[kSubsets], mny[kSubsets], mnz[kSubsets];
    float mxx[kSubsets], mxy[kSubsets], mxz[kSubsets];
    float cost[kSubsets];
    int8_t mask[kSubsets];
    int4 kid[8];  // child records of the treelet's leaves while it grows
    int stack_node[8];
    int stack_set[8];
};

// Subsets of 7 leaves grouped by size (2..5), each group in ascending order.
struct SubsetTable {
    uint8_t by_size[112];
};
constexpr int kSizeStart[5] = {0, 21, 56, 91, 112};  // starts of sizes 2, 3, 4, 5 and the end
constexpr SubsetTable subset_table() {
    SubsetTable t{};
    int k = 0;
    for (int size = 2; size <= 5; ++size)
        for (int s = 1; s < kSubsets; ++s) {
            int c = 0;
            for (int b = 0; b < kTr; ++b) c += (s >> b) & 1;
            if (c == size) t.by_size[k++] = (uint8_t)s;
        }
    return t;
}
__device__ const SubsetTable g_subsets = subset_table();

// Costs of this lane's subset s of kSize leaves: its partitions in the
// reference's order, the first of equal minima kept.
template <int kSize>
__device__ __forceinline__ void best_partition(const TrShared& sm, int s, float& opt, int& optp) {
    const int delta = (s - 1) & s;
    int p = (-delta) & s;
    opt = FLT_MAX;
    optp = 0;
#pragma unroll
    for (int j = 0; j < (1 << (kSize - 1)) - 1; ++j) {
        const float c = __fadd_rn(sm.cost[p], sm.cost[p ^ s]);
        if (c < opt) { opt = c; optp = p; }
        p = (p - delta) & s;
    }
}

// The subsets of kSize leaves (processSchedule :100-134), one lane per subset.
template <int kSize>
__device__ __forceinline__ void size_round(TrShared& sm, const uint8_t* __restrict__ by_size, float ci, float ct,
                                           float T) {
    constexpr int b = kSizeStart[kSize - 2], e = kSizeStart[kSize - 1];
#pragma unroll
    for (int k0 = b; k0 < e; k0 += 32) {
        const int k = k0 + (int)(threadIdx.x & 31);
        if (k < e) {
            const int s = by_size[k];
            float opt;
            int optp;
            best_partition<kSize>(sm, s, opt, optp);
            const float area = sm.cost[s];
            sm.cost[s] = fminf(__fadd_rn(__fmul_rn(ci, area), opt), __fmul_rn(__fmul_rn(ct, area), T));
            sm.mask[s] = (int8_t)optp;
        }
    }
    __syncwarp();
}

// A child record from the tree itself.  Called by all lanes or one.
__device__ __forceinline__ int4 tree_kids(const TreeRefs& g, int nb, int x) {
    const int l = ld_cg(g.left + nb + x), r = ld_cg(g.right + nb + x);
    return make_int4(l, r, __float_as_int(ld_cg(g.area + nb + l)), __float_as_int(ld_cg(g.area + nb + r)));
}

// One treelet by the whole warp: root and its child record rk, nodesSah and
// triangle count.  KD and rec start at the mesh's first inner node and node.
// kTight: there are neither, child records come from the tree and nodesSah is in
// `ns`, which starts at the mesh's first node.
template <bool kTight>
__device__ bool process_trbvh(const TreeRefs& g, int nb, uint32_t n, int root, int4 rk, int4* KD, int4* rec, float* ns,
                              float root_sah, int tri_count, float ci, float ct, TrShared& sm,
                              const uint8_t* __restrict__ s_prio, const uint8_t* __restrict__ s_by_size) {
    const int lane = threadIdx.x & 31;
    int32_t* const P_ = g.parent + nb;
    int32_t* const Lf = g.left + nb;
    int32_t* const Rt = g.right + nb;
    float4* const BMN = g.bmin + nb;
    float4* const BMX = g.bmax + nb;
    float* const AR = g.area + nb;

    // formTreelet (Treelet.cuh:57-114), as the ATRBVH passes form it: lane k
    // holds treelet leaf k, an internal leaf's child record is on its way to
    // shared memory from the moment it joins.
    int internal_node = lane == 0 ? root : -1;
    int s_node = -1;
    float s_area = 0.0f;
    auto join = [&](int node, float area) {
        s_node = node;
        s_area = area;
        if constexpr (!kTight)
            if (is_internal(node, n)) cp_async16_cg(sm.kid + lane, KD + node);
    };
    if (lane < 2) join(lane == 0 ? rk.x : rk.y, __int_as_float(lane == 0 ? rk.z : rk.w));
#pragma unroll
    for (int it = 0; it < kTr - 2; ++it) {
        const int m = 2 + it;
        const uint32_t ev = (lane < m && is_internal(s_node, n)) ? __float_as_uint(s_area) + 1u : 0u;
        const uint32_t vmax = __reduce_max_sync(kFull, ev);
        const uint32_t tied = __ballot_sync(kFull, lane < m && ev == vmax);
        int largest = __ffs(tied) - 1;
        if (vmax > 0x7f800001u) {
            // A NaN area has no place in that order: the reference's own
            // shuffle tree, in which it neither replaces nor is replaced.
            float v = (lane < m && is_internal(s_node, n)) ? s_area : -FLT_MAX;
            int ix = lane;
            for (int c = m, sh = m / 2; c > 1; c = (c + 1) / 2, sh = c / 2) {
                const float ov = __shfl_down_sync(kFull, v, sh);
                const int oi = __shfl_down_sync(kFull, ix, sh);
                if (lane < c - sh && ov > v) { v = ov; ix = oi; }
            }
            largest = __shfl_sync(kFull, ix, 0);
        } else if (__popc(tied) != 1) {
            const uint32_t pk = ((tied >> lane) & 1u) ? (uint32_t)s_prio[m * 32 + lane] : 255u;
            const uint32_t pmin = __reduce_min_sync(kFull, pk);
            largest = __ffs(__ballot_sync(kFull, pk == pmin)) - 1;
        }
        const int rep = __shfl_sync(kFull, s_node, largest);
        if (!is_internal(rep, n)) {
            cp_async_wait_all();
            return false;
        }
        int4 k;
        if constexpr (kTight) {
            k = tree_kids(g, nb, rep);
        } else {
            if (lane == largest) cp_async_wait_all();
            __syncwarp();
            k = sm.kid[largest];
            __syncwarp();
        }
        if (lane == it + 1) internal_node = rep;
        if (lane == largest) join(k.x, __int_as_float(k.z));
        else if (lane == it + 2) join(k.y, __int_as_float(k.w));
    }
    float4 s_mn = make_float4(0.f, 0.f, 0.f, 0.f), s_mx = s_mn;
    float s_sah = 0.0f;
    if (lane < kTr) {
        s_mn = ld_cg(BMN + s_node);
        s_mx = ld_cg(BMX + s_node);
        s_sah = is_internal(s_node, n) ? ld_cg(kTight ? ns + s_node : rec_f(rec, s_node, 1)) : __fmul_rn(ct, s_area);
    }
    cp_async_wait_all();

    // Subset boxes and areas (calculateSubsetSurfaceAreas :37-98).
    // Lane l takes subsets 4l .. 4l + 3: leaves 2..6 by the bits of l, then
    // leaves 0 and 1 in the four ways.
    {
        float a0 = FLT_MAX, a1 = FLT_MAX, a2 = FLT_MAX, b0 = -FLT_MAX, b1 = -FLT_MAX, b2 = -FLT_MAX;
        float x0[2], x1[2], x2[2], y0[2], y1[2], y2[2];
#pragma unroll
        for (int i = 0; i < kTr; ++i) {
            const float m0 = __shfl_sync(kFull, s_mn.x, i), m1 = __shfl_sync(kFull, s_mn.y, i),
                        m2 = __shfl_sync(kFull, s_mn.z, i);
            const float n0 = __shfl_sync(kFull, s_mx.x, i), n1 = __shfl_sync(kFull, s_mx.y, i),
                        n2 = __shfl_sync(kFull, s_mx.z, i);
            if (i < 2) {
                x0[i] = m0; x1[i] = m1; x2[i] = m2;
                y0[i] = n0; y1[i] = n1; y2[i] = n2;
            } else if (lane & (1 << (i - 2))) {
                a0 = fminf(m0, a0); a1 = fminf(m1, a1); a2 = fminf(m2, a2);
                b0 = fmaxf(n0, b0); b1 = fmaxf(n1, b1); b2 = fmaxf(n2, b2);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int s = lane * 4 + j;
            float c0 = a0, c1 = a1, c2 = a2, d0 = b0, d1 = b1, d2 = b2;
#pragma unroll
            for (int i = 0; i < 2; ++i)
                if (j & (1 << i)) {
                    c0 = fminf(x0[i], c0); c1 = fminf(x1[i], c1); c2 = fminf(x2[i], c2);
                    d0 = fmaxf(y0[i], d0); d1 = fmaxf(y1[i], d1); d2 = fmaxf(y2[i], d2);
                }
            sm.mnx[s] = c0; sm.mny[s] = c1; sm.mnz[s] = c2;
            sm.mxx[s] = d0; sm.mxy[s] = d1; sm.mxz[s] = d2;
            sm.cost[s] = box_area(c0, c1, c2, d0, d1, d2);
        }
        sm.mask[lane * 4] = sm.mask[lane * 4 + 1] = sm.mask[lane * 4 + 2] = sm.mask[lane * 4 + 3] = 0;
    }
    __syncwarp();
    if (lane < kTr) sm.cost[1 << lane] = s_sah;
    __syncwarp();
    const float T = (float)tri_count;

    // Sizes 2..5: a size's costs follow from the smaller sizes'.
    size_round<2>(sm, s_by_size, ci, ct, T);
    size_round<3>(sm, s_by_size, ci, ct, T);
    size_round<4>(sm, s_by_size, ci, ct, T);
    size_round<5>(sm, s_by_size, ci, ct, T);

    // Size 6: four lanes per subset, reduced within the group (processSubsets :136-189).
    {
        float opt = FLT_MAX;
        int optp = 0;
        const int k = lane >> 2;
        const int s = (kSubsets - 1) & ~(1 << k);
        if (lane < 4 * kTr) {
            const int left_mask = -(1 << max(k - 1, 0));
            int base = (lane & 3) + 1;
            const int np = (1 << (kTr - 2)) - 1;
            int p = (((base & left_mask) << 1) | (base & ~left_mask)) << 1;
            for (int j = lane & 3; j < np; j += 4) {
                const float c = __fadd_rn(sm.cost[p], sm.cost[p ^ s]);
                if (c < opt) { opt = c; optp = p; }
                base += 4;
                p = (((base & left_mask) << 1) | (base & ~left_mask)) << 1;
            }
        }
#pragma unroll
        for (int sh = 2; sh > 0; sh >>= 1) {
            const float ov = __shfl_down_sync(kFull, opt, sh);
            const int op = __shfl_down_sync(kFull, optp, sh);
            if (ov < opt) { opt = ov; optp = op; }
        }
        __syncwarp();
        if (lane < 4 * kTr && (lane & 3) == 0) {
            const float area = sm.cost[s];
            sm.cost[s] = fminf(__fadd_rn(__fmul_rn(ci, area), opt), __fmul_rn(__fmul_rn(ct, area), T));
            sm.mask[s] = (int8_t)optp;
        }
        __syncwarp();
    }
    // Size 7: all lanes, 32-lane reduction (:193-219).
    {
        const int s = kSubsets - 1;
        float opt = FLT_MAX;
        int optp = 0;
        int p = (lane + 1) * 2;
        for (int j = lane; j < (1 << (kTr - 1)) - 1; j += 32) {
            const float c = __fadd_rn(sm.cost[p], sm.cost[p ^ s]);
            if (c < opt) { opt = c; optp = p; }
            p += 64;
        }
#pragma unroll
        for (int sh = 16; sh > 0; sh >>= 1) {
            const float ov = __shfl_down_sync(kFull, opt, sh);
            const int op = __shfl_down_sync(kFull, optp, sh);
            if (ov < opt) { opt = ov; optp = op; }
        }
        __syncwarp();
        if (lane == 0) {
            const float area = sm.cost[s];
            sm.cost[s] = fminf(__fadd_rn(__fmul_rn(ci, area), opt), __fmul_rn(__fmul_rn(ct, area), T));
            sm.mask[s] = (int8_t)optp;
        }
        __syncwarp();
    }

    // Rebuild (updateTreelet :222-327).
    if (!(sm.cost[kSubsets - 1] < root_sah)) return true;
    int e_node = lane == 0 ? root : 0;
    int e_set = lane == 0 ? kSubsets - 1 : 0;
    int size = 1;
    int cur = 1;
    const uint32_t lt = lanemask_lt();
    while (size > 0) {
        const bool act = lane < size;
        const int P = act ? (int)sm.mask[e_set] : 0;
        const int Q = act ? (int)(int8_t)(P ^ e_set) : 0;
        // Left children.
        const bool li = act && __popc((unsigned)P) > 1;
        const unsigned lb = __ballot_sync(kFull, li);
        const int lslot = cur + __popc(lb & lt);
        const int lint = __shfl_sync(kFull, internal_node, li ? lslot : 0);
        const int lsrc = act && !li ? __ffs(P) - 1 : 0;
        const int lleaf = __shfl_sync(kFull, s_node, lsrc);
        const float lleaf_area = __shfl_sync(kFull, s_area, lsrc);
        cur += __popc(lb);
        // Right children.
        const bool ri = act && __popc((unsigned)Q) > 1;
        const unsigned rb = __ballot_sync(kFull, ri);
        const int rslot = cur + __popc(rb & lt);
        const int rint = __shfl_sync(kFull, internal_node, ri ? rslot : 0);
        const int rsrc = act && !ri ? __ffs(Q) - 1 : 0;
        const int rleaf = __shfl_sync(kFull, s_node, rsrc);
        const float rleaf_area = __shfl_sync(kFull, s_area, rsrc);
        cur += __popc(rb);
        __syncwarp();
        if (act) {
            const int lc = li ? lint : lleaf;
            const int rc = ri ? rint : rleaf;
            float la = lleaf_area, ra = rleaf_area;
            Lf[e_node] = lc;
            P_[lc] = e_node;
            Rt[e_node] = rc;
            P_[rc] = e_node;
            if (li) {
                const float4 mn = make_float4(sm.mnx[P], sm.mny[P], sm.mnz[P], 0.0f);
                const float4 mx = make_float4(sm.mxx[P], sm.mxy[P], sm.mxz[P], 0.0f);
                BMN[lc] = mn;
                BMX[lc] = mx;
                AR[lc] = la = box_area(mn, mx);
                *(kTight ? ns + lc : rec_f(rec, lc, 1)) = sm.cost[P];
                const int pos = __popc(lb & lt);
                sm.stack_node[pos] = lc;
                sm.stack_set[pos] = P;
            }
            if (ri) {
                const float4 mn = make_float4(sm.mnx[Q], sm.mny[Q], sm.mnz[Q], 0.0f);
                const float4 mx = make_float4(sm.mxx[Q], sm.mxy[Q], sm.mxz[Q], 0.0f);
                BMN[rc] = mn;
                BMX[rc] = mx;
                AR[rc] = ra = box_area(mn, mx);
                *(kTight ? ns + rc : rec_f(rec, rc, 1)) = sm.cost[P];
                const int pos = __popc(lb) + __popc(rb & lt);
                sm.stack_node[pos] = rc;
                sm.stack_set[pos] = Q;
            }
            if constexpr (!kTight) KD[e_node] = make_int4(lc, rc, __float_as_int(la), __float_as_int(ra));
        }
        __syncwarp();
        size = __popc(lb) + __popc(rb);
        if (lane < size) {
            e_node = sm.stack_node[lane];
            e_set = sm.stack_set[lane];
        }
        __syncwarp();
    }
    return true;
}

// What the kernels keep in shared memory besides the warps' TrShared.
struct TrTables {
    __align__(4) uint8_t prio[(kMaxTreelet + 1) * 32];
    __align__(4) uint8_t by_size[112];
};
__device__ __forceinline__ void load_tables(TrTables& t) {
    for (int k = threadIdx.x; k < (kMaxTreelet + 1) * 8; k += blockDim.x)
        reinterpret_cast<uint32_t*>(t.prio)[k] = reinterpret_cast<const uint32_t*>(&g_argmax_priority.rank[0][0])[k];
    for (int k = threadIdx.x; k < 112; k += blockDim.x) t.by_size[k] = g_subsets.by_size[k];
    __syncthreads();
}

// The treelet rooted at q, by the calling warp; everything below q is final.
__device__ __forceinline__ void restructure_root(const TreeRefs& g, const Segs& segs, const LevelRefs& lv, uint2 q,
                                                 float ci, TrShared& sm, const TrTables& t) {
    const uint32_t s0 = segs.tri_begin(q.x);
    const uint32_t n = segs.tri_end(q.x) - s0;
    const int nb = segs.node_base(q.x), x = (int)q.y;
    int4* const kd = lv.kids + segs.inner_base(q.x);
    int4* const rec = lv.rec + nb;
    const int4 rk = __ldcg(kd + x);
    const int cnt = ld_cg(rec_i(rec, x, 0));
    const float sah = __fadd_rn(__fadd_rn(__fmul_rn(ci, ld_cg(g.area + nb + x)), ld_cg(rec_f(rec, rk.x, 1))),
                                ld_cg(rec_f(rec, rk.y, 1)));
    if ((threadIdx.x & 31) == 0) *rec_f(rec, x, 1) = sah;
    if (!process_trbvh<false>(g, nb, n, x, rk, kd, rec, nullptr, sah, cnt, ci, lv.ct, sm, t.prio, t.by_size) &&
        (threadIdx.x & 31) == 0)
        set_error_bits(lv.err, kErrTreeletClimb);
    __syncwarp();
}

// Every treelet root of level lev, a warp each.
__global__ void __launch_bounds__(kTrWarps * 32, 3) k_tr_level(TreeRefs g, Segs segs, LevelRefs lv, int lev, float ci) {
    __shared__ TrShared s_tr[kTrWarps];
    __shared__ TrTables s_t;
    const uint32_t beg = (uint32_t)(lev - 1) * lv.cap;
    const uint32_t end = beg + min(lv.cursor[lev], lv.cap);
    const uint32_t first = beg + blockIdx.x * kTrWarps;
    if (first >= end) return;  // no root for this block
    load_tables(s_t);
    const uint32_t w = threadIdx.x >> 5;
    for (uint32_t e = first + w; e < end; e += gridDim.x * kTrWarps)
        restructure_root(g, segs, lv, lv.order[e], ci, s_tr[w], s_t);
}

// The dataflow pass: climbs from the frontier below the levels above L (all
// that lies under a start is final); the second thread to reach a node finishes
// it, and a warp restructures the treelets its lanes reach one after another.
// Starts go to lane 0 of every warp first, then lane 1, ...
__global__ void __launch_bounds__(kTrWarps * 32) k_trbvh(TreeRefs g, Segs segs, LevelRefs lv, float ci) {
    __shared__ TrShared s_tr[kTrWarps];
    __shared__ TrTables s_t;
    const uint32_t n_start = *lv.n_frontier;
    if (blockIdx.x * kTrWarps >= n_start) return;
    load_tables(s_t);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t nwarps = gridDim.x * kTrWarps;
    uint32_t next = (uint32_t)lane * nwarps + blockIdx.x * kTrWarps + (uint32_t)w;
    int cur = -1, base = 0, cbase = 0;
    uint32_t mesh = 0;
    bool rewrote = false;
    while (__any_sync(kFull, cur >= 0 || next < n_start)) {
        if (cur < 0 && next < n_start) {
            const uint2 e = lv.frontier[next];
            next += 32u * nwarps;
            mesh = e.x;
            base = segs.node_base(mesh);
            cbase = segs.inner_base(mesh);
            cur = g.parent[base + (int)e.y];
        }
        bool second = false;
        int up = -1;
        if (cur >= 0) {
            up = ld_cg(g.parent + base + cur);
            if (rewrote) fence_acq_rel_gpu();
            if (atomic_add_acq_rel_gpu(&lv.counters[cbase + cur], 1u) == 0u) cur = -1;
            else second = true;
        }
        // Everything above the frontier is a root; its count and child record
        // are k_levels', kept current by the rewrites since.
        unsigned vote = __ballot_sync(kFull, second);
        rewrote = vote != 0;
        __syncwarp();
        while (vote) {
            const int rl = __ffs(vote) - 1;
            const uint2 q = make_uint2(__shfl_sync(kFull, mesh, rl), (uint32_t)__shfl_sync(kFull, cur, rl));
            restructure_root(g, segs, lv, q, ci, s_tr[w], s_t);
            vote &= vote - 1;
        }
        if (cur >= 0) cur = up;
    }
}

// One climb that restructures treelets as its warps reach them, for trees whose
// level passes find no memory: 20 bytes of scratch a triangle (counts and nodesSah
// per node, arrivals) in place of 75 to 82; and for trees of a few treelets, where
// it is one launch an iteration in place of the passes'.  Level passes | this, 3
// iterations, us: 2 triangles 76 | 28, 10 103 | 63, 50 148 | 118, 100 191 | 173, 150
// 180 | 200, 300 214 | 226, 20,011 456 | 499, 100,003 615 | 623, 1,000,003 1,783 |
// 2,716, 16.8M 22,100 | 39,700.
__global__ void __launch_bounds__(kTrWarps * 32) k_tr_tight(TreeRefs g, Segs segs, int32_t* __restrict__ counts,
                                                            float* __restrict__ nsah, uint32_t* __restrict__ counters,
                                                            const uint8_t* __restrict__ seg_iters, int iteration,
                                                            float ci, float ct, uint32_t* __restrict__ err) {
    __shared__ TrShared s_tr[kTrWarps];
    __shared__ TrTables s_t;
    load_tables(s_t);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    int cur = -1, base = 0, cbase = 0;
    uint32_t n = 2;
    if (i < segs.n) {
        const uint32_t m = segs.seg_of_tri(i), s0 = segs.tri_begin(m);
        n = segs.tri_end(m) - s0;
        base = segs.node_base(m);
        cbase = segs.inner_base(m);
        if (!seg_iters || iteration < (int)seg_iters[m]) {
            const int leaf = base + (int)(i - s0) + (int)n - 1;
            counts[leaf] = 1;
            nsah[leaf] = __fmul_rn(ct, g.area[leaf]);
            cur = g.parent[leaf];
        }
    }
    const int gamma = kTr << iteration;
    while (__any_sync(kFull, cur >= 0)) {
        int cnt = 0;
        float sah = 0.0f;
        if (cur >= 0) {
            // The other lanes' parts of the treelets below are ordered before this
            // by the warp barrier that follows them.
            fence_acq_rel_gpu();
            if (atomic_add_acq_rel_gpu(&counters[cbase + cur], 1u) == 0u) {
                cur = -1;
            } else {
                const int x = base + cur;
                const int l = base + ld_cg(g.left + x), r = base + ld_cg(g.right + x);
                cnt = ld_cg(counts + l) + ld_cg(counts + r);
                sah = __fadd_rn(__fadd_rn(__fmul_rn(ci, ld_cg(g.area + x)), ld_cg(nsah + l)), ld_cg(nsah + r));
                counts[x] = cnt;
                nsah[x] = sah;
            }
        }
        unsigned vote = __ballot_sync(kFull, cnt >= gamma);
        __syncwarp();
        while (vote) {
            const int rl = __ffs(vote) - 1;
            const int root = __shfl_sync(kFull, cur, rl), nb = __shfl_sync(kFull, base, rl);
            const int rcnt = __shfl_sync(kFull, cnt, rl);
            const float rsah = __shfl_sync(kFull, sah, rl);
            const uint32_t rn = __shfl_sync(kFull, n, rl);
            if (!process_trbvh<true>(g, nb, rn, root, tree_kids(g, nb, root), nullptr, nullptr, nsah + nb, rsah, rcnt,
                                     ci, ct, s_tr[w], s_t.prio, s_t.by_size) &&
                lane == 0)
                set_error_bits(err, kErrTreeletClimb);
            __syncwarp();
            vote &= vote - 1;
        }
        if (cur >= 0) cur = ld_cg(g.parent + base + cur);
    }
}

constexpr uint32_t kTightTriangles = 128;  // up to these the climb is the faster

int trbvh_tight(atr_ctx* ctx, const TreeRefs& g, const Segs& segs, size_t total_nodes, int iterations,
                const uint8_t* seg_iters, float ci, float ct) {
    const size_t inner = segs.n - segs.count, b4 = align256(total_nodes * 4);
    void* scratch = nullptr;
    ATR_TRY(ctx->alloc(&scratch, 2 * b4 + align256(inner * 4)));
    char* const p = static_cast<char*>(scratch);
    uint32_t* const counters = reinterpret_cast<uint32_t*>(p + 2 * b4);
    constexpr int kThreads = kTrWarps * 32;
    int st = ATR_OK;
    ctx->phase_begin("trbvh");
    for (int it = 0; it < iterations && st == ATR_OK; ++it) {
        st = zero_words_async(ctx, counters, inner);
        if (st != ATR_OK) break;
        k_tr_tight<<<(segs.n + kThreads - 1) / kThreads, kThreads, 0, ctx->stream>>>(
            g, segs, reinterpret_cast<int32_t*>(p), reinterpret_cast<float*>(p + b4), counters, seg_iters, it, ci, ct,
            ctx->d_error);
        ctx->launches += 1;
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) st = cuda_fail(e, "k_tr_tight launch", __FILE__, __LINE__);
    }
    ctx->phase_end();
    ctx->release(scratch);
    return st;
}

// Whether `bytes` of scratch can be had: eagerly the allocation itself tells; a
// captured one is only made when the graph is instantiated or launched, so the
// device's free memory decides for it.
int level_scratch(atr_ctx* ctx, void** p, size_t bytes, bool* fits) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    ATR_CUDA(cudaStreamIsCapturing(ctx->stream, &cap));
    *fits = true;
    if (cap != cudaStreamCaptureStatusNone) {
        size_t avail = 0, all = 0;
        ATR_CUDA(cudaMemGetInfo(&avail, &all));
        *fits = bytes <= avail;
        return *fits ? ctx->alloc(p, bytes) : ATR_OK;
    }
    const cudaError_t e = cudaMallocFromPoolAsync(p, bytes, ctx->pool, ctx->stream);
    if (e == cudaSuccess) return ATR_OK;
    *p = nullptr;
    if (e != cudaErrorMemoryAllocation) return cuda_fail(e, "cudaMallocAsync", __FILE__, __LINE__);
    cudaGetLastError();
    *fits = false;
    return ATR_OK;
}

}  // namespace

// TRBVH (treelet 7) over every mesh of `segs`; seg_iters optionally gives
// each mesh its own iteration count (`iterations` is then their maximum).
int trbvh_run(atr_ctx* ctx, const TreeRefs& g, const Segs& segs, size_t total_nodes, int iterations,
              const uint8_t* seg_iters, float ci, float ct, const int2* karras_ranges) {
    if (iterations <= 0) return ATR_OK;
    if (segs.n <= kTightTriangles) return trbvh_tight(ctx, g, segs, total_nodes, iterations, seg_iters, ci, ct);
    const size_t inner = segs.n - segs.count;
    const LevelScratch ls(segs.n, kTr, auto_levels(segs.n, kTr));
    const size_t b_rec = align256(total_nodes * 16), b_kid = align256(inner * 16), b_ctr = align256(inner * 4);
    void* scratch = nullptr;
    bool fits = false;
    ATR_TRY(level_scratch(ctx, &scratch, b_rec + b_kid + b_ctr + ls.bytes(), &fits));
    if (!fits) return trbvh_tight(ctx, g, segs, total_nodes, iterations, seg_iters, ci, ct);
    char* p = static_cast<char*>(scratch);
    LevelRefs lv{};
    TopRefs tr{};  // no cluster here
    lv.rec = reinterpret_cast<int4*>(p); p += b_rec;
    lv.kids = reinterpret_cast<int4*>(p); p += b_kid;
    lv.counters = reinterpret_cast<uint32_t*>(p); p += b_ctr;
    lv.ct = ct;
    ls.bind(p, inner, ctx->d_error, lv, tr);
    cudaStream_t s = ctx->stream;
    const unsigned climb = (segs.n + kLvBlock - 1) / kLvBlock, list = (segs.n + kListBlock - 1) / kListBlock;
    const unsigned grid = (unsigned)ctx->num_sms * 3;  // grid-stride over a level's roots
    cudaError_t e = cudaSuccess;
    ctx->phase_begin("trbvh");
    for (int it = 0; it < iterations && e == cudaSuccess; ++it) {
        const int L = auto_levels(segs.n, kTr << it);
        e = cudaMemsetAsync(lv.counters, 0, inner * 4, s);
        if (e == cudaSuccess && zero_words_async(ctx, lv.cursor, ls.b_small / 4) != ATR_OK) e = cudaErrorLaunchFailure;
        if (e != cudaSuccess) break;
        k_levels<<<climb, kLvBlock, 0, s>>>(g, segs, lv, kTr, nullptr, seg_iters, it, ci, ct, L,
                                            it == 0 ? karras_ranges : nullptr);
        k_level_hist<<<list, 256, 0, s>>>(segs, lv, seg_iters, it, L);
        for (int lev = 1; lev <= L; ++lev) k_tr_level<<<grid, kTrWarps * 32, 0, s>>>(g, segs, lv, lev, ci);
        // The climb's arrivals; the dataflow pass counts its own.
        if (zero_words_async(ctx, lv.counters, inner) != ATR_OK) e = cudaErrorLaunchFailure;
        if (e != cudaSuccess) break;
        k_trbvh<<<grid, kTrWarps * 32, 0, s>>>(g, segs, lv, ci);
        ctx->launches += 3 + (uint64_t)L;
    }
    ctx->phase_end();
    if (e == cudaSuccess) e = cudaGetLastError();
    ctx->release(scratch);
    if (e != cudaSuccess) return cuda_fail(e, "TRBVH launch", __FILE__, __LINE__);
    return ATR_OK;
}

}  // namespace atr

using namespace atr;

extern "C" int atr_optimize_trbvh(atr_ctx* ctx, atr_tree* tree, int tsize, int iterations, float ci, float ct) {
    ATR_REQUIRE(ctx && tree, ATR_ERR_INVALID_ARG, "atr_optimize_trbvh: NULL argument");
    ATR_REQUIRE(tsize == kTr, ATR_ERR_UNSUPPORTED,
                "atr_optimize_trbvh: treelet size %d unsupported (the reference's subset kernel covers 7)", tsize);
    ATR_REQUIRE(iterations >= 0 && iterations <= 24, ATR_ERR_INVALID_ARG, "atr_optimize_trbvh: iterations %d",
                iterations);
    const uint32_t n = tree->n;
    TreeRefs g{n, tree->parent, tree->left, tree->right, tree->bmin, tree->bmax, tree->area};
    Segs segs{nullptr, nullptr, 1u, n};
    const int2* ranges = tree->karras ? tree->range : nullptr;
    tree->karras = false;
    tree_topology_changed(tree);
    ctx->release(tree->prepass_block);
    tree->prepass_block = nullptr;
    tree->prepass = BuildPrepass{};
    return trbvh_run(ctx, g, segs, 2 * (size_t)n - 1, iterations, nullptr, ci, ct, ranges);
}
