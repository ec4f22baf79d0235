// What the ATRBVH and TRBVH kernels share of a treelet and its tree.
#pragma once

#include "common.cuh"

namespace atr {

constexpr int kMaxTreelet = 20;
constexpr int kMaxDist = kMaxTreelet * (kMaxTreelet - 1) / 2;  // 190

__device__ __forceinline__ bool is_internal(int idx, uint32_t n) { return (uint32_t)idx < n - 1u; }

// Row/column of flat index k of the strictly lower triangular matrix stored
// row by row (r(r-1)/2 + c): BVHRT-Core/src/TriangularMatrix.cuh:150-168.
__device__ __forceinline__ void trm_rc(int k, int& r, int& c) {
    r = (int)__fmul_rn(__fadd_rn(1.0f, __fsqrt_rn((float)(8 * k + 1))), 0.5f);
    if (r * (r - 1) / 2 > k) --r;
    if ((r + 1) * r / 2 <= k) ++r;
    c = k - r * (r - 1) / 2;
}
__device__ __forceinline__ int trm_idx(int r, int c) { return r * (r - 1) / 2 + c; }

struct Box {
    float mnx, mny, mnz, mxx, mxy, mxz;
};

__device__ __forceinline__ Box shfl_box(const Box& b, int src) {
    Box o;
    o.mnx = __shfl_sync(kFull, b.mnx, src);
    o.mny = __shfl_sync(kFull, b.mny, src);
    o.mnz = __shfl_sync(kFull, b.mnz, src);
    o.mxx = __shfl_sync(kFull, b.mxx, src);
    o.mxy = __shfl_sync(kFull, b.mxy, src);
    o.mxz = __shfl_sync(kFull, b.mxz, src);
    return o;
}

// Surface area of the union of two boxes (Commons.cuh:156-164).
__device__ __forceinline__ float union_area(const Box& a, const Box& b) {
    return sa3(__fsub_rn(fmaxf(a.mxx, b.mxx), fminf(a.mnx, b.mnx)),
               __fsub_rn(fmaxf(a.mxy, b.mxy), fminf(a.mny, b.mny)),
               __fsub_rn(fmaxf(a.mxz, b.mxz), fminf(a.mnz, b.mnz)));
}

struct TreeRefs {
    uint32_t n;
    int32_t* parent;
    int32_t* left;
    int32_t* right;
    float4* bmin;
    float4* bmax;
    float* area;
};

}  // namespace atr
