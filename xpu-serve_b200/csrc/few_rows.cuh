// Products of a handful of rows with 32 weight rows a CTA of eight warps, on mma.sync m16n8k16 (weight rows on the M side, eight rows
// of x a product on the N side): what the experts' products for few tokens and the per-head products of latent attention share.
#pragma once

#include "common.cuh"

namespace {

constexpr int kFewWarps = 8;
constexpr int kFewRows = 32;          // weight rows a CTA
constexpr int kFewAhead = 4;          // k blocks of 32 a warp has in flight

__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 load_weights(const __nv_bfloat16* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ uint4 load_rows(const __nv_bfloat16* p) {     // (volatile, as the weights': asked for where it stands)
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// Adds w . x^T to acc[m][t]: w[q] points at the lane's 8 elements (from `piece` = (lane & 3) * 8 on) of weight row lane / 4 + 8 q,
// x[t] at those of row 8 t + lane / 4. The warps take the 32-wide k blocks in turn; a lane's 16 bytes of a row are 8 consecutive k,
// and the same assignment of k to fragment slots serves both operands. K is a multiple of 8.
template <int NT>
__device__ __forceinline__ void few_rows_multiply(const __nv_bfloat16* const (&w)[4], const __nv_bfloat16* const (&x)[NT], int K, int piece,
                                                  int warp, float (&acc)[2][NT][4]) {
    auto multiply = [&](const uint4 (&a)[4], const uint4 (&b)[NT]) {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const uint4 lo = a[2 * m], hi = a[2 * m + 1];
                mma_bf16(acc[m][t], lo.x, hi.x, lo.y, hi.y, b[t].x, b[t].y);
                mma_bf16(acc[m][t], lo.z, hi.z, lo.w, hi.w, b[t].z, b[t].w);
            }
    };
    int k0 = warp * 32;
    for (; k0 + (kFewAhead - 1) * kFewWarps * 32 + 32 <= K; k0 += kFewAhead * kFewWarps * 32) {
        uint4 a[kFewAhead][4], b[kFewAhead][NT];
#pragma unroll
        for (int s = 0; s < kFewAhead; ++s) {
#pragma unroll
            for (int q = 0; q < 4; ++q) a[s][q] = load_weights(w[q] + k0 + s * kFewWarps * 32);
#pragma unroll
            for (int t = 0; t < NT; ++t) b[s][t] = load_rows(x[t] + k0 + s * kFewWarps * 32);
        }
#pragma unroll
        for (int s = 0; s < kFewAhead; ++s) multiply(a[s], b[s]);
    }
    for (; k0 < K; k0 += kFewWarps * 32) {             // a lane's piece is whole or past the end
        uint4 a[4], b[NT];
        const bool there = k0 + piece < K;
#pragma unroll
        for (int q = 0; q < 4; ++q) a[q] = there ? load_weights(w[q] + k0) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int t = 0; t < NT; ++t) b[t] = there ? *reinterpret_cast<const uint4*>(x[t] + k0) : make_uint4(0u, 0u, 0u, 0u);
        multiply(a, b);
    }
}

}  // namespace
