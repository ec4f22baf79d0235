// Closest-hit / any-hit traversal of the Compact2 layout on sm_100a.
//
// Per ray this is gpu-ray-traversal/src/rt/kernels/kepler_dynamic_fetch.cu:95-317
// as one lane executes it: slab tests of both children, nearer child first,
// the farther one pushed; a leaf reached during the descent is processed
// before the descent continues (the reference may postpone it while other
// lanes still descend, which only changes the culling bound used for nodes
// whose leaves cannot hold a closer hit); Woop ray/triangle tests with
// t > tmin, t < hitT, u >= 0, v >= 0, u + v <= 1 keep the first hit on ties.
// The span helpers keep the reference's integer min/max on float bits
// (CudaTracerKernels.hpp:182-189).  Arithmetic: slab = fma(bound, 1/d, -o/d),
// Woop dot products as fma chains, IEEE reciprocal; the CPU oracle uses the
// same operations.
//
// Warps are persistent: lanes whose ray is done wait until fewer than 20 lanes
// of the warp have work (the reference's dynamic fetch; 16 in the largest
// layouts, 8 for a camera's rays in small ones), then take new rays from a global
// counter.  Between two fetches the warp steps as one, every step
// either a descent or a leaf test, chosen by vote: left to diverge, the lanes
// of a warp met again only by chance and an instruction served 6.6 of 32 lanes
// (1M sorted incoherent rays; 8.8 for pinhole rays); voting serves 11 and 13.
// What a ray does, and in which order, does not depend on the schedule.  Bound
// by issue (0.65 per cycle and scheduler) and by L1/L2 latency: 1M sorted
// incoherent rays 1.07 -> 0.84 ms, 2.07M pinhole rays 0.57 -> 0.46 ms, a bounce of
// each 0.66 -> 0.48 ms (4.2M triangles).  Measured and not kept: 12 or 16 blocks a
// SM (spills), prefetching the pushed child, fetching at 12 or 28 lanes.
//
#include <type_traits>

#include "common.cuh"
#include "internal.h"

namespace atr {

// Which layout each ray traverses: with groups == 0 every ray uses the arrays
// as given; otherwise rays [ray_off[g], ray_off[g+1]) trace mesh
// group_mesh[g] of a batch whose mesh m starts at node 4 * (tri_off[m] - m)
// (float4 units) and Woop entry 4 * tri_off[m].
struct RayMeshMap {
    const uint32_t* ray_off;
    const uint32_t* group_mesh;
    const uint32_t* tri_off;
    uint32_t groups;
};

namespace {

constexpr int kSentinel = 0x76543210;

// How a warp steps: lanes with work below which it fetches rays; how many times as
// many lanes must wait to descend as at leaves for a descent; and the kernel's
// variant.  kNear's figures are compiled in (read from arguments they cost up to
// 0.6 %).  kFar: a leaf step runs each lane's leaf to its end.  kClose: as kNear, but
// while a warp's rays have one origin (a camera's) it fetches below 8 lanes: their
// paths are short and end together, and a fetch takes as long as several steps.
enum Variant { kNear = 0, kFar = 1, kClose = 2 };
struct Stepping {
    Variant variant;
    int fetch, weight;
};
constexpr Stepping kNearSteps = {kNear, 20, 2};
constexpr int kCameraFetch = 8;
// By the bytes of the layout's nodes and Woop entries (126 MB of L2).  Far beyond
// L2 the fetches' misses bound the trace, and more lanes at work lose more than they
// hide: a leaf's remaining sectors leave the L1 between two of its lane's steps, and
// rays in flight push each other's nodes out.  8.4M random rays, closest | any hit,
// ms, by each lane at its own step (as before the vote) / kNear / kFar, 20, 2 / kFar,
// 16, 1:
//   uniform    62 MB    8.0 / 5.59 / 5.64 / 5.71   | 6.8 / 4.75 / 4.78 / 4.85
//   uniform   459 MB   13.8 / 10.0 / 9.98 / 9.99   | 7.5 / 5.91 / 5.88 / 5.80
//   clustered 447 MB    5.6 / 3.46 / 3.44 / 3.75   | 4.7 / 2.80 / 2.82 / 3.04
//   uniform   679 MB   17.3 / 14.9 / 14.2 / 13.8   | 8.3 / 7.66 / 7.30 / 7.07
//   clustered 665 MB    6.1 / 4.14 / 4.08 / 4.30   | 4.8 / 3.05 / 3.03 / 3.20
//   uniform   898 MB   20.9 / 20.0 / 19.2 / 18.2   | 9.2 / 9.38 / 8.93 / 8.51
//   clustered 875 MB    6.3 / 4.53 / 4.40 / 4.53   | 4.9 / 3.34 / 3.28 / 3.35
//   uniform  1.33 GB   27.6 / 28.4 / 27.5 / 25.3   | 10.8 / 11.6 / 11.2 / 10.5
//   clustered 1.28 GB   6.8 / 5.78 / 5.53 / 5.39   | 5.0 / 4.18 / 4.11 / 3.92
//   uniform  1.77 GB   33.7 / 35.3 / 34.5 / 31.4   | 12.0 / 13.1 / 12.8 / 11.9
//   uniform  2.63 GB   44.7 / 47.4 / 46.3 / 42.0   | 13.6 / 15.3 / 14.9 / 13.9
// With at most twice the rays that the GPU holds at once (189,440) rays do not push
// each other out yet: 16.8M uniform triangles, closest hit of 100,003, 300,007 and
// 400,009 rays by kNear / kFar, 16, 1: 0.80 / 0.79, 1.50 / 1.55, 2.04 / 1.90.
// In layouts of up to 4 MB a camera's rays end early: 8.3M pinhole rays, us, kNear /
// kClose: 1,000 uniform triangles (0.1 MB) 246 / 231, clustered 10,007 (1.2 MB) 282 /
// 262, 30,011 (3.6 MB) 356 / 332; beyond, clustered 65,536 (7.7 MB) 452 / 414 but
// uniform 811 / 843.
Stepping stepping(size_t layout_bytes, int64_t rays, int64_t held) {
    if (layout_bytes <= 4000000 && rays > held) return {kClose, 20, 2};  // else every warp fetches once
    if (rays <= 2 * held) return kNearSteps;
    if (layout_bytes >= 1100000000) return {kFar, 16, 1};
    if (layout_bytes >= 600000000) return {kFar, 20, 2};
    return kNearSteps;
}

__device__ __forceinline__ int imin(int a, int b) { return a < b ? a : b; }
__device__ __forceinline__ int imax(int a, int b) { return a > b ? a : b; }

__device__ __forceinline__ float span_begin(float a0, float a1, float b0, float b1, float c0, float c1, float d) {
    const int t = imax(imin(__float_as_int(c0), __float_as_int(c1)), __float_as_int(d));
    return __int_as_float(imax(imax(__float_as_int(fminf(a0, a1)), __float_as_int(fminf(b0, b1))), t));
}
__device__ __forceinline__ float span_end(float a0, float a1, float b0, float b1, float c0, float c1, float d) {
    const int t = imin(imax(__float_as_int(c0), __float_as_int(c1)), __float_as_int(d));
    return __int_as_float(imin(imin(__float_as_int(fmaxf(a0, a1)), __float_as_int(fmaxf(b0, b1))), t));
}

// A node's 64 bytes in two 32-byte loads: the lanes of a warp visit different
// nodes, so each load instruction costs the L1 one lookup per lane (1M sorted
// incoherent rays: 1.12 -> 1.07 ms against four 16-byte loads).
__device__ __forceinline__ void ld32(const float4* p, float4& a, float4& b) {
    asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(p));
}

constexpr int kTraceThreads = 128;
constexpr int kSharedStack = 16;

template <int kStack, bool kMapped, Variant kVariant>
__global__ void __launch_bounds__(kTraceThreads) k_trace(const float4* __restrict__ nodes_all,
                                               const float4* __restrict__ woop_all,
                                               const int* __restrict__ tri_all, RayMeshMap map,
                                               const float4* __restrict__ rays, int64_t nrays, int any_hit,
                                               int4* __restrict__ results, unsigned long long* __restrict__ counter,
                                               unsigned long long* __restrict__ other,
                                               int lanes, Stepping far, uint32_t* __restrict__ err) {
    // The stack's top entry is held in a register (top), so a pop does not
    // wait for a load; of the sp entries below it the first kSharedStack are
    // in shared memory (one bank per lane whatever the lanes' depths), the
    // rest in local memory (16 entries take 5 % off incoherent rays; 4 or 8 less).
    __shared__ int s_stack[kSharedStack][kTraceThreads];
    int stack[kStack > kSharedStack ? kStack - kSharedStack : 1];
    // The launch before this one, which used the other counter, is done; the next
    // one starts from it.
    if (other && blockIdx.x == 0 && threadIdx.x == 0) *other = 0ull;
    const int lane = threadIdx.x & 31;
    if (lane >= lanes) return;
    const unsigned team = lanes == 32 ? kFull : (1u << lanes) - 1u;
    const Stepping how = kVariant == kFar ? far : kNearSteps;
    const int fetch = (how.fetch * lanes + 31) / 32;
    int top = kSentinel;
    float ox = 0, oy = 0, oz = 0, tmin = 0, dx = 0, dy = 0, dz = 0, hitT = 0;
    float idx = 0, idy = 0, idz = 0, oodx = 0, oody = 0, oodz = 0;
    int nodeAddr = kSentinel, leafAddr = 0, hitIndex = -1, sp = 0;
    long long rayidx = 0;
    bool has = false, overflow = false;
    bool more = true;  // the same in every lane: rays are left to fetch
    const float4* nodes = nodes_all;
    const float4* woop = woop_all;
    const int* tri_index = tri_all;

    auto pop = [&]() {
        nodeAddr = top;
        if (--sp >= 0) top = sp < kSharedStack ? s_stack[sp][threadIdx.x] : stack[max(sp - kSharedStack, 0)];
    };
    // Both children of the inner node nodeAddr against the ray: on to the
    // nearer one, the farther one pushed; the first leaf met is set aside.
    auto node_step = [&]() {
        float4 n0, n1, nz, cn;
        ld32(nodes + nodeAddr, n0, n1);
        ld32(nodes + nodeAddr + 2, nz, cn);
        int c0 = __float_as_int(cn.x), c1 = __float_as_int(cn.y);
        const float c0lox = __fmaf_rn(n0.x, idx, -oodx), c0hix = __fmaf_rn(n0.y, idx, -oodx);
        const float c0loy = __fmaf_rn(n0.z, idy, -oody), c0hiy = __fmaf_rn(n0.w, idy, -oody);
        const float c0loz = __fmaf_rn(nz.x, idz, -oodz), c0hiz = __fmaf_rn(nz.y, idz, -oodz);
        const float c1loz = __fmaf_rn(nz.z, idz, -oodz), c1hiz = __fmaf_rn(nz.w, idz, -oodz);
        const float c0min = span_begin(c0lox, c0hix, c0loy, c0hiy, c0loz, c0hiz, tmin);
        const float c0max = span_end(c0lox, c0hix, c0loy, c0hiy, c0loz, c0hiz, hitT);
        const float c1lox = __fmaf_rn(n1.x, idx, -oodx), c1hix = __fmaf_rn(n1.y, idx, -oodx);
        const float c1loy = __fmaf_rn(n1.z, idy, -oody), c1hiy = __fmaf_rn(n1.w, idy, -oody);
        const float c1min = span_begin(c1lox, c1hix, c1loy, c1hiy, c1loz, c1hiz, tmin);
        const float c1max = span_end(c1lox, c1hix, c1loy, c1hiy, c1loz, c1hiz, hitT);
        const bool swp = c1min < c0min;
        const bool t0 = c0max >= c0min, t1 = c1max >= c1min;
        if (!t0 && !t1) {
            pop();
        } else {
            nodeAddr = t0 ? c0 : c1;
            if (t0 && t1) {
                if (swp) { const int tmp = nodeAddr; nodeAddr = c1; c1 = tmp; }
                if (sp + 1 >= kStack) {  // deeper than the stack: give the ray up
                    overflow = true;
                    nodeAddr = kSentinel;
                    leafAddr = 0;
                    return;
                }
                if (sp < kSharedStack) s_stack[sp][threadIdx.x] = top;
                else stack[max(sp - kSharedStack, 0)] = top;
                ++sp;
                top = c1;
            }
        }
        if (nodeAddr < 0 && leafAddr >= 0) {
            leafAddr = nodeAddr;
            pop();
        }
    };
    // The next triangle of the leaf set aside, and whether it was the last: a
    // triangle is always followed by another or by the terminator, so all of
    // these loads lie in the list and can be in flight together.
    auto leaf_step = [&]() {
        const int tri = ~leafAddr;
        const float4 v00 = __ldg(woop + tri);
        const int next = __ldg(reinterpret_cast<const int*>(woop + tri + 3));
        bool last = true;
        if (__float_as_int(v00.x) != (int)0x80000000u) {
            last = next == (int)0x80000000u;
            const float Oz = __fmaf_rn(-oz, v00.z, __fmaf_rn(-oy, v00.y, __fmaf_rn(-ox, v00.x, v00.w)));
            const float invDz = __frcp_rn(__fmaf_rn(dz, v00.z, __fmaf_rn(dy, v00.y, __fmul_rn(dx, v00.x))));
            const float t = __fmul_rn(Oz, invDz);
            if (t > tmin && t < hitT) {
                const float4 v11 = __ldg(woop + tri + 1), v22 = __ldg(woop + tri + 2);
                const float Ox = __fmaf_rn(oz, v11.z, __fmaf_rn(oy, v11.y, __fmaf_rn(ox, v11.x, v11.w)));
                const float Dx = __fmaf_rn(dz, v11.z, __fmaf_rn(dy, v11.y, __fmul_rn(dx, v11.x)));
                const float u = __fmaf_rn(t, Dx, Ox);
                const float Oy = __fmaf_rn(oz, v22.z, __fmaf_rn(oy, v22.y, __fmaf_rn(ox, v22.x, v22.w)));
                const float Dy = __fmaf_rn(dz, v22.z, __fmaf_rn(dy, v22.y, __fmul_rn(dx, v22.x)));
                const float v = __fmaf_rn(t, Dy, Oy);
                if (u >= 0.0f && v >= 0.0f && __fadd_rn(u, v) <= 1.0f) {
                    hitT = t;
                    hitIndex = tri;
                    if (any_hit) {
                        nodeAddr = kSentinel;
                        last = true;
                    }
                }
            }
        }
        if (!last) {
            leafAddr -= 3;  // ~(tri + 3)
        } else {
            leafAddr = nodeAddr;
            if (nodeAddr < 0) pop();
        }
    };

    while (true) {
        if (more) {
            // Lanes without a ray take the next ones.
            const unsigned idle = __ballot_sync(team, !has);
            const int leader = __ffs(idle) - 1;
            unsigned long long base = 0;
            if (lane == leader) base = atomicAdd(counter, (unsigned long long)__popc(idle));
            base = __shfl_sync(team, base, leader);
            more = (long long)base + __popc(idle) < nrays;
            if (!has) {
                rayidx = (long long)base + __popc(idle & lanemask_lt());
                has = rayidx < nrays;
                if (has) {
                    if constexpr (kMapped) {
                        uint32_t lo = 0, hi = map.groups;
                        while (hi - lo > 1) {
                            const uint32_t mid = (lo + hi) >> 1;
                            if ((long long)__ldg(map.ray_off + mid) <= rayidx) lo = mid; else hi = mid;
                        }
                        const uint32_t mesh = __ldg(map.group_mesh + lo);
                        const uint32_t s0 = __ldg(map.tri_off + mesh);
                        nodes = nodes_all + 4 * ((size_t)s0 - mesh);
                        woop = woop_all + 4 * (size_t)s0;
                        tri_index = tri_all + 4 * (size_t)s0;
                    }
                    const float4 o = __ldg(rays + 2 * rayidx), d = __ldg(rays + 2 * rayidx + 1);
                    ox = o.x; oy = o.y; oz = o.z; tmin = o.w;
                    dx = d.x; dy = d.y; dz = d.z; hitT = d.w;
                    const float ooeps = 8.271806125530277e-25f;  // 2^-80
                    idx = __frcp_rn(fabsf(dx) > ooeps ? dx : copysignf(ooeps, dx));
                    idy = __frcp_rn(fabsf(dy) > ooeps ? dy : copysignf(ooeps, dy));
                    idz = __frcp_rn(fabsf(dz) > ooeps ? dz : copysignf(ooeps, dz));
                    oodx = __fmul_rn(ox, idx);
                    oody = __fmul_rn(oy, idy);
                    oodz = __fmul_rn(oz, idz);
                    top = kSentinel;
                    sp = 0;
                    leafAddr = 0;
                    nodeAddr = 0;
                    hitIndex = -1;
                    overflow = false;
                }
            }
        }
        // Steps until fewer than `fetch` lanes have work (or none, once there
        // are no rays to fetch).  A lane either descends or tests its leaf; each
        // warp step is one of the two: descent unless the lanes at leaves are
        // more than half as many (a leaf step is short and frees its lane), or,
        // in the largest layouts, more.
        int enough = more ? fetch : 1;
        if constexpr (kVariant == kClose) {
            // One origin, but for chance: only the schedule depends on it.
            const unsigned from = __float_as_uint(ox) ^ 31u * __float_as_uint(oy) ^ 961u * __float_as_uint(oz);
            const unsigned first = __shfl_sync(team, from, 0);
            if (__all_sync(team, !has || from == first) && more) enough = (kCameraFetch * lanes + 31) / 32;
        }
        while (true) {
            const bool leaf = has && leafAddr < 0;
            const bool inner = has && !leaf && nodeAddr != kSentinel;
            const unsigned bi = __ballot_sync(team, inner), bl = __ballot_sync(team, leaf);
            if (__popc(bi | bl) < enough) break;
            if (__popc(bi) >= how.weight * __popc(bl)) {
                // Two steps a vote: most lanes that descend do so again.
                if (inner) {
                    node_step();
                    if ((unsigned)nodeAddr < (unsigned)kSentinel && leafAddr >= 0) node_step();
                }
            } else {
                if (leaf) {
                    do leaf_step();
                    while (kVariant == kFar && leafAddr < 0);
                }
                if constexpr (kVariant == kFar) __syncwarp(team);
            }
        }
        if (has && nodeAddr == kSentinel && leafAddr >= 0) {
            if (overflow) set_error_bits(err, kErrTraceStack);
            const int id = hitIndex == -1 ? -1 : __ldg(tri_index + hitIndex);
            results[rayidx] = make_int4(id, __float_as_int(hitT), 0, 0);
            has = false;
        }
        if (!more && !__any_sync(team, has)) break;
    }
}

template <int kStack, bool kMapped, Variant kVariant>
void launch_trace(atr_ctx* ctx, const int4* nodes, const float4* woop, const int32_t* tri, const RayMeshMap& map,
                  const float4* rays, int64_t n, int any_hit, int4* res, unsigned long long* counter,
                  unsigned long long* other, const Stepping& how, size_t layout_bytes) {
    const int blocks_per_sm = ctx->trace_blocks[kStack > 64][kMapped][kVariant];
    // Rays per warp: the paths of a warp's rays add up as far as they differ, so
    // few rays are spread over as many warps as run at once (1,000 rays through
    // 20,011 triangles: 57 us at one ray a warp, 93 at 32; 50,000 rays: 103 us at
    // 32 or 16, 117 at 8).  Not over a handful of triangles, whose paths are a few
    // steps and end together (3,072 and 76,800 rays over 12: 12.3 and 14.8 us
    // spread, 10.4 and 12.6 at 32; random rays over 100 already gain from it).
    constexpr size_t kFewSteps = 4096;  // bytes of nodes and Woop entries
    constexpr int W = kTraceThreads / 32;
    const int64_t warps = (int64_t)ctx->num_sms * blocks_per_sm * W;
    int lanes = 32;
    while (layout_bytes > kFewSteps && lanes > 1 && n <= warps * (lanes / 2)) lanes /= 2;
    const int64_t need = (n + W * lanes - 1) / (W * lanes);
    int64_t grid = (int64_t)ctx->num_sms * blocks_per_sm;
    if (need < grid) grid = need;
    k_trace<kStack, kMapped, kVariant><<<(unsigned)grid, kTraceThreads, 0, ctx->stream>>>(
        reinterpret_cast<const float4*>(nodes), woop, tri, map, rays, n, any_hit, res, counter, other, lanes, how,
        ctx->d_error);
    ctx->launches += 1;
}

template <int kStack>
void launch_trace(atr_ctx* ctx, const int4* nodes, const float4* woop, const int32_t* tri, const RayMeshMap& map,
                  const float4* rays, int64_t n, int any_hit, int4* res, unsigned long long* counter,
                  unsigned long long* other, const Stepping& how, size_t layout_bytes) {
    auto run = [&](auto mapped, auto variant) {
        launch_trace<kStack, mapped.value, variant.value>(ctx, nodes, woop, tri, map, rays, n, any_hit, res, counter,
                                                          other, how, layout_bytes);
    };
    auto by_variant = [&](auto mapped) {
        switch (how.variant) {
            case kNear: run(mapped, std::integral_constant<Variant, kNear>{}); break;
            case kFar: run(mapped, std::integral_constant<Variant, kFar>{}); break;
            case kClose: run(mapped, std::integral_constant<Variant, kClose>{}); break;
        }
    };
    if (map.groups) by_variant(std::true_type{});
    else by_variant(std::false_type{});
}

// Cosine-weighted diffuse bounce per primary hit (the workload of
// gpu-ray-traversal/src/rt/ray/RayGenKernels.cu:114-223 with one sample):
// origin backed off the hit by 1e-4 along the ray, geometric normal facing
// the ray, direction from a counter-based hash of (seed, ray); misses get
// tmax = -1 and never hit.
__global__ void __launch_bounds__(256) k_bounce(const float4* __restrict__ verts, const float4* __restrict__ rays,
                                                const int4* __restrict__ res, int64_t n, uint64_t seed,
                                                float4* __restrict__ out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 o = rays[2 * i], d = rays[2 * i + 1];
    const int4 r = res[i];
    if (r.x < 0) {
        out[2 * i] = o;
        out[2 * i + 1] = make_float4(d.x, d.y, d.z, -1.0f);
        return;
    }
    const float t = fmaxf(__int_as_float(r.y) - 1e-4f, 0.0f);
    const float4 p = make_float4(o.x + d.x * t, o.y + d.y * t, o.z + d.z * t, 0.0f);
    const float4 a = verts[3 * (size_t)r.x], b = verts[3 * (size_t)r.x + 1], c = verts[3 * (size_t)r.x + 2];
    const float e1x = b.x - a.x, e1y = b.y - a.y, e1z = b.z - a.z;
    const float e2x = c.x - a.x, e2y = c.y - a.y, e2z = c.z - a.z;
    float nx = e1y * e2z - e1z * e2y, ny = e1z * e2x - e1x * e2z, nz = e1x * e2y - e1y * e2x;
    float len = sqrtf(nx * nx + ny * ny + nz * nz);
    if (len == 0.0f) { nx = 1.0f; ny = 0.0f; nz = 0.0f; len = 1.0f; }
    nx /= len; ny /= len; nz /= len;
    if (nx * d.x + ny * d.y + nz * d.z > 0.0f) { nx = -nx; ny = -ny; nz = -nz; }
    // Orthonormal basis around n.
    float tx, ty, tz;
    if (fabsf(nx) > fabsf(nz)) { tx = -ny; ty = nx; tz = 0.0f; } else { tx = 0.0f; ty = -nz; tz = ny; }
    const float tl = rsqrtf(tx * tx + ty * ty + tz * tz);
    tx *= tl; ty *= tl; tz *= tl;
    const float bx = ny * tz - nz * ty, by = nz * tx - nx * tz, bz = nx * ty - ny * tx;
    // Two uniforms from a 64-bit mix of (seed, i).
    unsigned long long h = seed ^ (0x9E3779B97F4A7C15ull * (unsigned long long)(i + 1));
    h ^= h >> 30; h *= 0xBF58476D1CE4E5B9ull; h ^= h >> 27; h *= 0x94D049BB133111EBull; h ^= h >> 31;
    const float u1 = (float)(h >> 40) * (1.0f / 16777216.0f);
    const float u2 = (float)((h >> 16) & 0xFFFFFF) * (1.0f / 16777216.0f);
    const float rr = sqrtf(u1), phi = 6.2831853f * u2;
    const float x = rr * cosf(phi), y = rr * sinf(phi), z = sqrtf(fmaxf(0.0f, 1.0f - u1));
    float wx = x * tx + y * bx + z * nx, wy = x * ty + y * by + z * ny, wz = x * tz + y * bz + z * nz;
    const float wl = rsqrtf(wx * wx + wy * wy + wz * wz);
    out[2 * i] = p;
    out[2 * i + 1] = make_float4(wx * wl, wy * wl, wz * wl, 1e30f);
}

}  // namespace

// Blocks of each instance that an SM holds (once per context: contexts launch from
// threads of their own).
int trace_prepare(atr_ctx* ctx) {
    auto set = [&](int* b, auto kernel) {
        const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(b, kernel, kTraceThreads, 0);
        if (e != cudaSuccess || *b < 1) *b = 1;
        return e;
    };
    auto& b = ctx->trace_blocks;
    ATR_CUDA(set(&b[0][0][kNear], k_trace<64, false, kNear>));
    ATR_CUDA(set(&b[0][0][kFar], k_trace<64, false, kFar>));
    ATR_CUDA(set(&b[0][0][kClose], k_trace<64, false, kClose>));
    ATR_CUDA(set(&b[0][1][kNear], k_trace<64, true, kNear>));
    ATR_CUDA(set(&b[0][1][kFar], k_trace<64, true, kFar>));
    ATR_CUDA(set(&b[0][1][kClose], k_trace<64, true, kClose>));
    ATR_CUDA(set(&b[1][0][kNear], k_trace<256, false, kNear>));
    ATR_CUDA(set(&b[1][0][kFar], k_trace<256, false, kFar>));
    ATR_CUDA(set(&b[1][0][kClose], k_trace<256, false, kClose>));
    ATR_CUDA(set(&b[1][1][kNear], k_trace<256, true, kNear>));
    ATR_CUDA(set(&b[1][1][kFar], k_trace<256, true, kFar>));
    ATR_CUDA(set(&b[1][1][kClose], k_trace<256, true, kClose>));
    return ATR_OK;
}

int trace_run(atr_ctx* ctx, const int4* nodes, const float4* woop, const int32_t* tri, const RayMeshMap& map,
              int max_depth, size_t layout_bytes, const float4* rays, int64_t n, int any_hit, int4* res) {
    if (n == 0) return ATR_OK;
    // The ray counter: one of the context's two, used in turn; the launch that uses
    // one clears the other for the next (a count of finished warps that let the last
    // one clear a single counter cost 4 us a launch).  A captured trace gets one of
    // its own, since its graph may run on any stream beside others.
    unsigned long long* counter = ctx->d_trace + ctx->trace_turn;
    unsigned long long* other = ctx->d_trace + (ctx->trace_turn ^ 1);
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    ATR_CUDA(cudaStreamIsCapturing(ctx->stream, &cap));
    unsigned long long* own = nullptr;
    if (cap != cudaStreamCaptureStatusNone) {
        ATR_TRY(ctx->alloc(reinterpret_cast<void**>(&own), 8));
        cudaMemsetAsync(own, 0, 8, ctx->stream);
        counter = own;
        other = nullptr;
    }
    int st = ATR_OK;
    const Stepping how =
        stepping(layout_bytes, n, (int64_t)ctx->num_sms * ctx->trace_blocks[0][0][kNear] * kTraceThreads);
    ctx->phase_begin("trace");
    if (max_depth + 1 < 64)
        launch_trace<64>(ctx, nodes, woop, tri, map, rays, n, any_hit, res, counter, other, how, layout_bytes);
    else if (max_depth + 1 < 256)
        launch_trace<256>(ctx, nodes, woop, tri, map, rays, n, any_hit, res, counter, other, how, layout_bytes);
    else st = ATR_ERR_UNSUPPORTED;
    ctx->phase_end();
    ctx->release(own);
    if (st == ATR_ERR_UNSUPPORTED) {
        set_error("trace: layout depth %d exceeds the traversal stack", max_depth);
        return st;
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        // Whether this launch ran or not, both counters are zero behind it.
        if (!own) cudaMemsetAsync(ctx->d_trace, 0, 16, ctx->stream);
        return cuda_fail(e, "k_trace launch", __FILE__, __LINE__);
    }
    if (!own) ctx->trace_turn ^= 1;  // the launch uses up its counter and clears the other
    return ATR_OK;
}

int trace_batch(atr_ctx* ctx, const int4* nodes, const float4* woop, const int32_t* tri, const uint32_t* ray_off,
                const uint32_t* group_mesh, const uint32_t* tri_off, uint32_t groups, int max_depth, size_t layout_bytes,
                const float4* rays, int64_t n, int any_hit, int4* res) {
    const RayMeshMap map{ray_off, group_mesh, tri_off, groups};
    return trace_run(ctx, nodes, woop, tri, map, max_depth, layout_bytes, rays, n, any_hit, res);
}

}  // namespace atr

using namespace atr;

extern "C" {

int atr_trace(atr_ctx* ctx, const atr_compact* cp, const float* rays, int64_t n, int any_hit, int32_t* results) {
    ATR_REQUIRE(ctx && cp && rays && results, ATR_ERR_INVALID_ARG, "atr_trace: NULL argument");
    ATR_REQUIRE(n >= 0, ATR_ERR_INVALID_ARG, "atr_trace: negative ray count");
    const RayMeshMap map{nullptr, nullptr, nullptr, 0u};
    return trace_run(ctx, cp->nodes, cp->woop, cp->tri_index, map, cp->max_depth,
                     (size_t)cp->num_nodes * 64 + (size_t)cp->num_woop * 16, reinterpret_cast<const float4*>(rays), n, any_hit, reinterpret_cast<int4*>(results));
}

int atr_gen_bounce_rays(atr_ctx* ctx, const atr_scene* scene, const float* rays, const int32_t* results, int64_t n,
                        uint64_t seed, float* out) {
    ATR_REQUIRE(ctx && scene && rays && results && out, ATR_ERR_INVALID_ARG, "atr_gen_bounce_rays: NULL argument");
    if (n <= 0) return ATR_OK;
    k_bounce<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(
        scene->verts, reinterpret_cast<const float4*>(rays), reinterpret_cast<const int4*>(results), n, seed,
        reinterpret_cast<float4*>(out));
    ctx->launches += 1;
    ATR_CUDA(cudaGetLastError());
    return ATR_OK;
}

}  // extern "C"
