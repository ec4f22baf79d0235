// Compact2 traversal layout with Woop triangles, built on the device.
//
// Byte-identical to the reference's host conversion
// gpu-ray-traversal/src/rt/cuda/CudaBVH.cpp:469-574 (createCompact for a
// collapsed tree) and :579-600 (woopifyTri), which walks the tree with a LIFO
// stack: popping node X allots node records to X's inner children (left, then
// right) and appends the Woop triangles of X's leaf children (left, then
// right, each followed by a 0x80000000 terminator).  Nodes are therefore
// popped in right-first preorder, and everything popped before a node X is its
// ancestors and, for every node of its path that is an inner left child, the
// right sibling's whole subtree.  A subtree of I inner nodes allots I - 1
// records below its root's, so the two running totals at X -- records allotted
// (S) and Woop entries written (W) before X is popped -- are sums over X's path
// of per-node steps that need subtree totals only:
//   S(c) = S(P) + inner children of P + [c left, sibling r inner] (I(r) - 1)
//   W(c) = W(P) + entries of P's leaf children + [c left, r inner] TW(r)
// and X's own record is 1 + S(P), plus one for a right child beside an inner
// left one.  Hence three passes and no scan, rank order or jump rounds:
//   1. bottom-up: subtree totals (I, TW); the thread that finishes a node
//      writes its inner children's steps;
//   2. the nodes with at least kTopInner inner nodes below sum their whole path;
//   3. every other node walks up to the nearest of those (a few links), and the
//      thread of each reachable inner node writes its 64-byte record and its
//      leaf children's Woop triangles.
// Bound by the latency of the climb's exchanges and of the write pass's gathers
// (boxes, vertices): 0.85 -> 0.54 ms for 4,194,304 clustered triangles and 3.6 ->
// 2.4 ms for a batch of 24.9M against a rank by pointer jumping (up to 25
// rounds), a scatter by rank, two scans and a slot pass.
// The Woop transform restates FW::MatrixBase::inverted
// (gpu-ray-traversal/src/framework/base/Math.hpp:961-983, 3x3 determinant
// :934-939) with round-to-nearest operations in the reference's order.

#include "common.cuh"
#include "internal.h"

namespace atr {

namespace {

// Nodes whose subtree holds at least this many inner nodes sum their path to
// the root once (pass 2); the walks of pass 3 stop at the nearest of them.
constexpr uint32_t kTopInner = 128;

struct FlatRefs {
    const int32_t* parent;
    const int32_t* left;
    const int32_t* right;
    const int32_t* data;
    const int32_t* count;
    const float4* bmin;
    const float4* bmax;
    const int32_t* tri;
};

// Segment view of thread gi: the mesh, its first node (nb), its first inner
// node (cb), its first triangle (s0), its triangle count (n) and the local
// index li of the leaf (and of the inner node) this thread owns.
struct SegPos {
    uint32_t m, s0, n, li;
    int nb, cb;
};
__device__ __forceinline__ SegPos seg_pos(const Segs& segs, uint32_t gi) {
    SegPos p;
    p.m = segs.seg_of_tri(gi);
    p.s0 = segs.tri_begin(p.m);
    p.n = segs.tri_end(p.m) - p.s0;
    p.li = gi - p.s0;
    p.nb = segs.node_base(p.m);
    p.cb = segs.inner_base(p.m);
    return p;
}

__device__ __forceinline__ bool c_leaf(const FlatRefs& t, int nb, int x) { return t.data[nb + x] >= 0; }

// A node's step from its parent: x the parent (local; -1 at the root), y the
// S step (-1: the parent is a leaf of the collapsed tree, so nothing below it
// is part of the layout), z the W step, w the inner nodes of the node's
// subtree, with kRightOfInner set for a right child beside an inner left one.
// Written for inner nodes only, so a walk must not start at a collapsed leaf.
constexpr uint32_t kRightOfInner = 0x80000000u;
__device__ __forceinline__ uint32_t step_inner(const int4& s) { return (uint32_t)s.w & ~kRightOfInner; }

// Pass 1.  A child's totals reach its parent through the parent's 64-bit slot
// (bit 63 marks them present, then I, then TW): the first arrival exchanges
// its totals in and stops, the second takes the sibling's out of the exchange.
// A leaf's I is 0 and an inner node's at least 1, so the totals also tell the
// two apart and a child's own arrays are not read.  Nothing else read here is
// written by this pass, so the exchanges need no ordering, and the next node's
// links load while the exchange is in flight.
__device__ __forceinline__ unsigned long long pack_totals(uint32_t inner, uint32_t tw) {
    return (1ull << 63) | ((unsigned long long)inner << 32) | tw;
}

__global__ void __launch_bounds__(256) k_flat_counts(FlatRefs t, Segs segs, int4* __restrict__ step,
                                                      unsigned long long* __restrict__ slots,
                                                      int64_t* __restrict__ nodes_out, int64_t* __restrict__ woop_out,
                                                      int64_t* __restrict__ depth_out) {
    const uint32_t gi = blockIdx.x * blockDim.x + threadIdx.x;
    if (gi == 0) *depth_out = 0;
    if (gi >= segs.n) return;
    const SegPos q = seg_pos(segs, gi);
    int ch = (int)q.li + (int)q.n - 1;
    int cur = t.parent[q.nb + ch];
    if (cur < 0) return;
    uint32_t mi = 0u, mw = 4u;  // inner nodes and Woop entries below ch: one triangle and its terminator
    int l = t.left[q.nb + cur], r = t.right[q.nb + cur], up = t.parent[q.nb + cur], dat = t.data[q.nb + cur];
    while (true) {
        int nl = 0, nr = 0, nup = -1, ndat = -1;
        if (up >= 0) {
            nl = t.left[q.nb + up];
            nr = t.right[q.nb + up];
            nup = t.parent[q.nb + up];
            ndat = t.data[q.nb + up];
        }
        const unsigned long long other = atomicExch(slots + q.cb + cur, pack_totals(mi, mw));
        if (other == 0ull) return;
        const uint32_t si = (uint32_t)(other >> 32) & 0x7fffffffu, sw = (uint32_t)other;
        const bool from_left = ch == l;
        const uint32_t il = from_left ? mi : si, ir = from_left ? si : mi;
        const uint32_t wl = from_left ? mw : sw, wr = from_left ? sw : mw;
        const bool cleaf = dat >= 0 && up >= 0;
        const int ds = (il ? 1 : 0) + (ir ? 1 : 0);
        const uint32_t dw = (il ? 0u : wl) + (ir ? 0u : wr);
        if (il)
            step[q.cb + l] = make_int4(cur, cleaf ? -1 : ds + (ir ? (int)ir - 1 : 0), (int)(dw + (ir ? wr : 0u)), (int)il);
        if (ir) step[q.cb + r] = make_int4(cur, cleaf ? -1 : ds, (int)dw, (int)(ir | (il ? kRightOfInner : 0u)));
        if (cleaf) {
            const int c = t.count[q.nb + cur];
            mi = 0u;
            mw = 3u * (uint32_t)(c > 1 ? c : 1) + 1u;
        } else {
            mi = 1u + il + ir;
            mw = wl + wr;
        }
        if (up < 0) {
            step[q.cb + cur] = make_int4(-1, 0, 0, (int)mi);
            nodes_out[q.m] = (int64_t)mi;
            woop_out[q.m] = (int64_t)mw;
            return;
        }
        ch = cur;
        cur = up;
        l = nl;
        r = nr;
        up = nup;
        dat = ndat;
    }
}

// Where a node stands: S, W, its depth (root 1), and whether it is part of
// the layout (w = 0) or below a leaf of the collapsed tree (w = 1).
// Pass 2: the nodes with large subtrees, over their whole path.
__global__ void __launch_bounds__(256) k_flat_top(Segs segs, const int4* __restrict__ step, int4* __restrict__ place,
                                                   const int32_t* __restrict__ data) {
    const uint32_t gi = blockIdx.x * blockDim.x + threadIdx.x;
    if (gi >= segs.n) return;
    const SegPos q = seg_pos(segs, gi);
    if (q.li >= q.n - 1) return;
    const int x = (int)q.li;
    // A collapsed leaf has no step; the root (node 0) has one whatever its data says.
    if (data[q.nb + x] >= 0 && x != 0) return;
    int4 s = __ldg(step + q.cb + x);
    if (step_inner(s) < kTopInner) return;
    int4 at = make_int4(0, 0, 1, 0);
    while (s.x >= 0) {
        if (s.y < 0) {
            at.w = 1;
            break;
        }
        at.x += s.y;
        at.y += s.z;
        at.z += 1;
        s = __ldg(step + q.cb + s.x);
    }
    place[q.cb + x] = at;
}

// The place of inner node x (local), whose step is s.
__device__ __forceinline__ int4 walk_up(const int4* __restrict__ step, const int4* __restrict__ place, int x, int4 s) {
    int4 at = make_int4(0, 0, 0, 0);
    while (true) {
        if (step_inner(s) >= kTopInner) {
            const int4 p = __ldg(place + x);
            return make_int4(at.x + p.x, at.y + p.y, at.z + p.z, p.w);
        }
        at.z += 1;
        if (s.x < 0) return at;
        if (s.y < 0) {
            at.w = 1;
            return at;
        }
        at.x += s.y;
        at.y += s.z;
        x = s.x;
        s = __ldg(step + x);
    }
}

__device__ __forceinline__ float det3(const float s[3][3]) {
    // v00*v11*v22 - v00*v12*v21 + v10*v21*v02 - v10*v22*v01 + v20*v01*v12 - v20*v02*v11
    float r = __fmul_rn(__fmul_rn(s[0][0], s[1][1]), s[2][2]);
    r = __fsub_rn(r, __fmul_rn(__fmul_rn(s[0][0], s[1][2]), s[2][1]));
    r = __fadd_rn(r, __fmul_rn(__fmul_rn(s[1][0], s[2][1]), s[0][2]));
    r = __fsub_rn(r, __fmul_rn(__fmul_rn(s[1][0], s[2][2]), s[0][1]));
    r = __fadd_rn(r, __fmul_rn(__fmul_rn(s[2][0], s[0][1]), s[1][2]));
    r = __fsub_rn(r, __fmul_rn(__fmul_rn(s[2][0], s[0][2]), s[1][1]));
    return r;
}

__device__ void woopify(const float4* __restrict__ v, int tri, float4* __restrict__ out) {
    const float4 a = v[3 * (size_t)tri], b = v[3 * (size_t)tri + 1], c = v[3 * (size_t)tri + 2];
    const float c0[3] = {__fsub_rn(a.x, c.x), __fsub_rn(a.y, c.y), __fsub_rn(a.z, c.z)};
    const float c1[3] = {__fsub_rn(b.x, c.x), __fsub_rn(b.y, c.y), __fsub_rn(b.z, c.z)};
    const float c2[3] = {__fsub_rn(__fmul_rn(c0[1], c1[2]), __fmul_rn(c0[2], c1[1])),
                         __fsub_rn(__fmul_rn(c0[2], c1[0]), __fmul_rn(c0[0], c1[2])),
                         __fsub_rn(__fmul_rn(c0[0], c1[1]), __fmul_rn(c0[1], c1[0]))};
    float M[4][4];
    for (int r = 0; r < 3; ++r) { M[r][0] = c0[r]; M[r][1] = c1[r]; M[r][2] = c2[r]; }
    M[0][3] = c.x; M[1][3] = c.y; M[2][3] = c.z;
    M[3][0] = 0.0f; M[3][1] = 0.0f; M[3][2] = 0.0f; M[3][3] = 1.0f;
    float R[3][4];  // rows 0..2 of the inverse are all the layout needs
    float d = 0.0f, si = 1.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float sj = si;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float s[3][3];
#pragma unroll
            for (int k = 0; k < 3; ++k)
#pragma unroll
                for (int l = 0; l < 3; ++l) s[k][l] = M[k < j ? k : k + 1][l < i ? l : l + 1];
            const float dd = __fmul_rn(det3(s), sj);
            if (i < 3) R[i][j] = dd;
            d = __fadd_rn(d, __fmul_rn(dd, M[j][i]));
            sj = -sj;
        }
        si = -si;
    }
    const float rd = d != 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) R[i][j] = __fmul_rn(__fmul_rn(R[i][j], rd), 4.0f);
    out[0] = make_float4(R[2][0], R[2][1], R[2][2], -R[2][3]);
    out[1] = make_float4(R[0][0], R[0][1], R[0][2], R[0][3]);
    out[2] = make_float4(R[1][0], R[1][1], R[1][2], R[1][3]);
}

// Pass 3.  One thread per reachable inner node: its 64-byte record in the mesh's node
// slice (first node 4 * cb in float4 units), the terminators of its leaf
// children's Woop lists in the mesh's Woop slice (first entry 4 * s0).  The
// Woop triangles of a warp's leaf children are then spread over the warp's
// lanes (an exclusive scan of the nodes' triangle counts in shared memory,
// item u to the node whose range holds it), so a node with long leaf lists
// does not hold the warp while the others idle.
constexpr int kWriteThreads = 128;

__global__ void __launch_bounds__(kWriteThreads) k_flat_write(FlatRefs t, Segs segs, const float4* __restrict__ verts,
                                                     const int4* __restrict__ step, const int4* __restrict__ place,
                                                     int4* __restrict__ nodes, float4* __restrict__ woop,
                                                     int32_t* __restrict__ tri_index,
                                                     unsigned long long* __restrict__ depth_out) {
    constexpr int W = kWriteThreads / 32;
    __shared__ uint32_t s_pre[W][32], s_n0[W][32], s_w[W][2][32], s_s0[W][32];
    __shared__ int32_t s_d[W][2][32];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const uint32_t gi = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t items[2] = {0u, 0u}, wk[2] = {0u, 0u};
    int32_t dk[2] = {0, 0};
    uint32_t s0 = 0;
    bool multi[2] = {false, false};
    uint32_t depth = 0;
    if (gi < segs.n) {
        const SegPos q = seg_pos(segs, gi);
        s0 = q.s0;
        const int x = (int)q.li;
        int4 st = make_int4(-1, 0, 0, 0), at = make_int4(0, 0, 0, 1);
        // The root is part of the layout whatever its data says.
        if (q.li < q.n - 1 && (t.data[q.nb + x] < 0 || t.parent[q.nb + x] < 0)) {
            st = __ldg(step + q.cb + x);
            at = walk_up(step + q.cb, place + q.cb, x, st);
        }
        if (at.w == 0) {
            depth = (uint32_t)at.z;
            float4* mw = woop + 4 * (size_t)q.s0;
            int32_t* mt = tri_index + 4 * (size_t)q.s0;
            const int ch[2] = {t.left[q.nb + x], t.right[q.nb + x]};
            int cref[2];
            uint32_t w = (uint32_t)at.y;
            int slot = 1 + at.x;  // of the next inner child
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int c = ch[k];
                if (!c_leaf(t, q.nb, c)) {
                    cref[k] = 4 * slot++;
                    continue;
                }
                cref[k] = ~(int)w;
                const int cnt = t.count[q.nb + c];
                multi[k] = cnt > 1;
                items[k] = (uint32_t)(cnt > 1 ? cnt : 1);
                wk[k] = w;
                dk[k] = t.data[q.nb + c];
                w += 3u * items[k];
                const float term = __int_as_float((int)0x80000000u);
                mw[w] = make_float4(term, term, term, term);
                mt[w] = 0;
                w += 1;
            }
            const float4 lm = t.bmin[q.nb + ch[0]], lx = t.bmax[q.nb + ch[0]];
            const float4 rm = t.bmin[q.nb + ch[1]], rx = t.bmax[q.nb + ch[1]];
            const int own = st.x < 0 ? 0 : 1 + at.x - st.y + (st.w < 0 ? 1 : 0);
            int4* dst = nodes + 4 * ((size_t)q.cb + (size_t)own);
            dst[0] = make_int4(__float_as_int(lm.x), __float_as_int(lx.x), __float_as_int(lm.y), __float_as_int(lx.y));
            dst[1] = make_int4(__float_as_int(rm.x), __float_as_int(rx.x), __float_as_int(rm.y), __float_as_int(rx.y));
            dst[2] = make_int4(__float_as_int(lm.z), __float_as_int(lx.z), __float_as_int(rm.z), __float_as_int(rx.z));
            dst[3] = make_int4(cref[0], cref[1], 0, 0);
        }
    }
    // One atomic per warp on the shared maximum.
    depth = __reduce_max_sync(kFull, depth);
    if (lane == 0 && depth > 0) atomicMax(depth_out, (unsigned long long)depth);
    // Items of this lane: items[0] triangles of the left leaf child, then
    // items[1] of the right.
    const uint32_t mine = items[0] + items[1];
    uint32_t incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += y;
    }
    const uint32_t total = __shfl_sync(kFull, incl, 31);
    s_pre[wp][lane] = incl - mine;
    s_n0[wp][lane] = items[0];
    s_w[wp][0][lane] = wk[0];
    s_w[wp][1][lane] = wk[1];
    // A single-triangle leaf's data is the triangle (sign bit set here);
    // a list leaf's data is its list offset.
    s_d[wp][0][lane] = dk[0] | (multi[0] ? 0 : (int32_t)0x80000000);
    s_d[wp][1][lane] = dk[1] | (multi[1] ? 0 : (int32_t)0x80000000);
    s_s0[wp][lane] = s0;
    __syncwarp();
    for (uint32_t u = lane; u < total; u += 32) {
        // The node holding item u: the last lane whose range starts at or
        // before u (lanes without items share the next lane's start).
        int o = 0;
#pragma unroll
        for (int step = 16; step > 0; step >>= 1)
            if (s_pre[wp][o + step] <= u) o += step;
        const uint32_t loc = u - s_pre[wp][o];
        const int k = loc < s_n0[wp][o] ? 0 : 1;
        const uint32_t j = loc - (k ? s_n0[wp][o] : 0u);
        const int32_t dd = s_d[wp][k][o];
        const uint32_t ms0 = s_s0[wp][o];
        const int d = dd & 0x7fffffff;
        const int tri = dd >= 0 ? t.tri[ms0 + (uint32_t)d + j] : d;
        const uint32_t w = s_w[wp][k][o] + 3u * j;
        woopify(verts + 3 * (size_t)ms0, tri, woop + 4 * (size_t)ms0 + w);
        int32_t* mt = tri_index + 4 * (size_t)ms0;
        mt[w] = tri;
        mt[w + 1] = 0;
        mt[w + 2] = 0;
    }
}

}  // namespace

// Compact2 layout of every mesh of segs into per-mesh slices of nodes (mesh m
// from node inner_base(m)), woop and tri_index (mesh m from entry 4 *
// tri_begin(m)).  d_sizes receives 2 * count + 1 int64: nodes per mesh, Woop
// entries per mesh, then the deepest inner level over all meshes.  Stream
// ordered: nothing here waits for the device.
int flatten_segs(atr_ctx* ctx, const Segs& segs, const CollapsedOut& c, const float4* verts, int4* nodes,
                 float4* woop, int32_t* tri_index, int64_t* d_sizes) {
    const uint32_t n = segs.n;
    const uint32_t m = n - segs.count;  // inner nodes over all meshes
    cudaStream_t s = ctx->stream;
    void* scratch = nullptr;
    const size_t b4 = align256((size_t)m * 16);
    ATR_TRY(ctx->alloc(&scratch, 2 * b4 + align256((size_t)m * 8)));
    char* p = static_cast<char*>(scratch);
    int4* step = reinterpret_cast<int4*>(p); p += b4;
    int4* place = reinterpret_cast<int4*>(p); p += b4;
    unsigned long long* slots = reinterpret_cast<unsigned long long*>(p);
    const FlatRefs t{c.parent, c.left, c.right, c.data, c.count, c.bmin, c.bmax, c.tri_indices};
    const unsigned gb = (n + 255) / 256;
    int64_t* const depth_out = d_sizes + 2 * segs.count;
    // The count climb reads a zero slot as "no sibling yet": a failed clear must stop here.
    int st = zero_words_async(ctx, reinterpret_cast<uint32_t*>(slots), (size_t)m * 2);
    if (st == ATR_OK) {
        k_flat_counts<<<gb, 256, 0, s>>>(t, segs, step, slots, d_sizes, d_sizes + segs.count, depth_out);
        k_flat_top<<<gb, 256, 0, s>>>(segs, step, place, c.data);
        k_flat_write<<<(n + kWriteThreads - 1) / kWriteThreads, kWriteThreads, 0, s>>>(
            t, segs, verts, step, place, nodes, woop, tri_index, reinterpret_cast<unsigned long long*>(depth_out));
        ctx->launches += 3;
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) st = cuda_fail(e, "flatten kernels", __FILE__, __LINE__);
    }
    ctx->release(scratch);
    return st;
}

}  // namespace atr

using namespace atr;

extern "C" {

int atr_flatten_compact2(atr_ctx* ctx, const atr_collapsed* c, const atr_scene* scene, atr_compact** out) {
    ATR_REQUIRE(ctx && c && scene && out, ATR_ERR_INVALID_ARG, "atr_flatten_compact2: NULL argument");
    ATR_REQUIRE(c->n == scene->n || c->split, ATR_ERR_INVALID_ARG,
                "atr_flatten_compact2: tree/scene size mismatch");
    *out = nullptr;
    const uint32_t n = c->n;
    atr_compact* cp = new atr_compact();
    cp->ctx = ctx;
    // Upper bounds: every inner node, and 3 entries per triangle + 1 terminator per triangle.
    int st = ctx->alloc(reinterpret_cast<void**>(&cp->nodes), (size_t)(n - 1) * 64);
    if (st == ATR_OK) st = ctx->alloc(reinterpret_cast<void**>(&cp->woop), (size_t)n * 4 * 16);
    if (st == ATR_OK) st = ctx->alloc(reinterpret_cast<void**>(&cp->tri_index), (size_t)n * 4 * 4);
    int64_t* sizes = nullptr;
    if (st == ATR_OK) st = ctx->alloc(reinterpret_cast<void**>(&sizes), 24);
    if (st != ATR_OK) {
        ctx->release(sizes);
        atr_compact_destroy(cp);
        return st;
    }
    const Segs segs{nullptr, nullptr, 1u, n};
    const CollapsedOut co{c->parent, c->left, c->right, c->data, c->count, c->bmin, c->bmax, c->tri_indices};
    ctx->phase_begin("flatten");
    st = flatten_segs(ctx, segs, co, scene->verts, cp->nodes, cp->woop, cp->tri_index, sizes);
    ctx->phase_end();
    if (st == ATR_OK) {
        int64_t h[3] = {0, 0, 0};
        st = read_back(ctx, h, sizes, sizeof(h), false);
        cp->num_nodes = h[0];
        cp->num_woop = h[1];
        cp->max_depth = (int32_t)h[2];
    }
    ctx->release(sizes);
    if (st != ATR_OK) { atr_compact_destroy(cp); return st; }
    *out = cp;
    return ATR_OK;
}

int atr_compact_destroy(atr_compact* cp) {
    if (!cp) return ATR_OK;
    cp->ctx->release(cp->nodes);
    cp->ctx->release(cp->woop);
    cp->ctx->release(cp->tri_index);
    delete cp;
    return ATR_OK;
}

int atr_compact_download(atr_ctx* ctx, const atr_compact* cp, int32_t* nodes, float* woop, int32_t* tri) {
    ATR_REQUIRE(ctx && cp, ATR_ERR_INVALID_ARG, "atr_compact_download: NULL argument");
    cudaStream_t s = ctx->stream;
    if (nodes) ATR_CUDA(cudaMemcpyAsync(nodes, cp->nodes, (size_t)cp->num_nodes * 64, cudaMemcpyDeviceToHost, s));
    if (woop) ATR_CUDA(cudaMemcpyAsync(woop, cp->woop, (size_t)cp->num_woop * 16, cudaMemcpyDeviceToHost, s));
    if (tri) ATR_CUDA(cudaMemcpyAsync(tri, cp->tri_index, (size_t)cp->num_woop * 4, cudaMemcpyDeviceToHost, s));
    return atr_ctx_synchronize(ctx);
}

int atr_compact_view_get(const atr_compact* cp, atr_compact_view* v) {
    ATR_REQUIRE(cp && v, ATR_ERR_INVALID_ARG, "atr_compact_view_get: NULL argument");
    v->num_nodes = cp->num_nodes;
    v->num_woop = cp->num_woop;
    v->nodes = reinterpret_cast<int32_t*>(cp->nodes);
    v->woop = reinterpret_cast<float*>(cp->woop);
    v->tri_index = cp->tri_index;
    v->max_depth = cp->max_depth;
    return ATR_OK;
}

}  // extern "C"
