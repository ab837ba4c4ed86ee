// Routed experts for few tokens (a decode step): one product kernel that finds each expert's rows by itself.
//
// A step of T tokens chooses T * top rows (token, choice) over E experts; with a handful of tokens an expert has one or two of
// them and what the product costs is its weights' bytes. The tile products of the long steps (gemm_tc.cu) want the rows sorted,
// padded to tiles of 128 and gathered, and give each CTA 256 weight rows, too few CTAs to keep memory busy. Here:
//   - no plan and no gather: rows keep their own index (token * top + choice) from the router to the combine, and a CTA finds
//     the rows of its expert by one look over the T * top ids;
//   - a CTA takes 32 weight rows of one expert, its eight warps take k blocks of 32 in turn; a lane loads 16 bytes of four weight
//     rows and of its token's row straight into mma.sync fragments (the contraction's order within a block is free, so the
//     operands' registers are filled as they lie in memory), eight columns a product; the warps' sums meet in shared memory in
//     the order of the warps. A row's result does not depend on the other rows of the step.
// Bound by the weights' bytes of the experts that are met. Measured on B200 (8 tokens, top 4 of 16 experts of 1,024 at width 2,048:
// 177 MB of weights, kernels alone): gate/up and down 35 + 20 us (3.2 TB/s, cold), where gather, two tcgen05 products over padded
// tiles of 128 rows and the plan took 120; a decode step of four such layers 0.69 -> 0.63 ms. A product's time follows the
// groups of eight columns that it carries, whatever an expert's count is: the tcgen05 products take over at 17 tokens, or at 33 for
// small experts (ops/lib.py moe_few_tokens has both sides; 32 rows an expert are the most that an instance here holds).
#include "common.cuh"
#include "few_rows.cuh"

namespace {

enum FewEpilogue : int { FEW_STORE = 0, FEW_GATED = 1, FEW_RELU_SQ = 2 };

struct FewParams {
    const __nv_bfloat16* x;        // [rows / share, K]: row i reads x[i / share]
    const __nv_bfloat16* w;        // [E, N, K]
    __nv_bfloat16* out;            // [rows, N] (N / 2 gated)
    const int32_t* ids;            // [rows] the row's expert, -1: none
    int rows, share, N, K, epilogue;
    int64_t ldx, ldo;
    float limit, alpha, shift;     // the gated epilogue: limit 0 silu(g) * u, else the clamped unit
};

// NT groups of eight rows of an expert.
template <int NT>
__global__ void __launch_bounds__(kFewWarps * 32)
moe_few_rows_kernel(const FewParams p) {
    __shared__ int list[NT * 8];
    __shared__ int count;
    __shared__ float sums[kFewWarps][2 * NT * 4][32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int e = blockIdx.y, n0 = blockIdx.x * kFewRows;
    pdl_launch_dependents();
    pdl_wait();
    if (warp == 0) {                                   // the expert's rows, in order
        int have = 0;
        for (int i0 = 0; i0 < p.rows; i0 += 32) {
            const bool mine = i0 + lane < p.rows && p.ids[i0 + lane] == e;
            const unsigned who = __ballot_sync(0xffffffffu, mine);
            const int at = have + __popc(who & ((1u << lane) - 1u));
            if (mine && at < NT * 8) list[at] = i0 + lane;
            have += __popc(who);
        }
        if (lane == 0) count = min(have, NT * 8);      // (a token names an expert once, so an expert has at most T rows)
    }
    __syncthreads();
    const int rows = count;
    if (rows == 0) return;
    const int piece = (lane & 3) * 8, r = lane >> 2;
    const __nv_bfloat16* w[4];                         // weight rows n0 + r, + 8, + 16, + 24 (past N: the last row, not stored)
#pragma unroll
    for (int q = 0; q < 4; ++q)
        w[q] = p.w + ((int64_t)e * p.N + min(n0 + r + 8 * q, p.N - 1)) * p.K + piece;
    const __nv_bfloat16* x[NT];                        // (columns past the expert's rows read its first row and are not stored)
#pragma unroll
    for (int t = 0; t < NT; ++t) x[t] = p.x + (int64_t)(list[t * 8 + r < rows ? t * 8 + r : 0] / p.share) * p.ldx + piece;
    float acc[2][NT][4];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[m][t][j] = 0.0f;
    few_rows_multiply<NT>(w, x, p.K, piece, warp, acc);
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int j = 0; j < 4; ++j) sums[warp][(m * NT + t) * 4 + j][lane] = acc[m][t][j];
    __syncthreads();
    // a thread finishes the two weight rows r and r + 8 of one 16-row block for one row of the step
    for (int item = threadIdx.x; item < 2 * NT * 2 * 32; item += kFewWarps * 32) {
        const int l = item & 31, j = (item >> 5) & 1, mt = item >> 6, t = mt % NT, m = mt / NT;
        const int col = t * 8 + (l & 3) * 2 + j;
        if (col >= rows) continue;
        float lo = 0.0f, hi = 0.0f;
#pragma unroll
        for (int v = 0; v < kFewWarps; ++v) {
            lo += sums[v][mt * 4 + j][l];
            hi += sums[v][mt * 4 + j + 2][l];
        }
        __nv_bfloat16* out = p.out + (int64_t)list[col] * p.ldo;
        const int row = n0 + m * 16 + (l >> 2);
        if (p.epilogue == FEW_GATED) {                 // blocks of 8 gate rows and the 8 up rows of the same outputs; N is a multiple of 16
            if (row + 8 >= p.N) continue;
            float g = lo, u = hi, y;
            if (p.limit > 0.0f) {
                g = fminf(g, p.limit);
                u = fminf(fmaxf(u, -p.limit), p.limit);
                y = g / (1.0f + __expf(-p.alpha * g)) * (u + p.shift);
            } else {
                y = g / (1.0f + __expf(-g)) * u;
            }
            out[((n0 + m * 16) >> 1) + (l >> 2)] = __float2bfloat16_rn(y);
            continue;
        }
        if (p.epilogue == FEW_RELU_SQ) {
            lo = fmaxf(lo, 0.0f);
            hi = fmaxf(hi, 0.0f);
            lo *= lo;
            hi *= hi;
        }
        if (row < p.N) out[row] = __float2bfloat16_rn(lo);
        if (row + 8 < p.N) out[row + 8] = __float2bfloat16_rn(hi);
    }
}

}  // namespace

// out[i] = epilogue(w[ids[i]] . x[i / share]) for i < rows, bfloat16; rows whose id is negative are not written. At most 32 rows
// an expert. epilogue 0: store; 1: gated (w's rows in blocks of 8 gate and 8 up rows; out has N / 2 columns); 2: max(v, 0)^2.
XS_API int xs_moe_few_rows(const void* x, int64_t ldx, int share, const void* w, void* out, int64_t ldo, const int32_t* ids, int rows,
                           int most_an_expert, int E, int N, int K, int epilogue, float limit, float alpha, float shift,
                           cudaStream_t stream) {
    if (rows == 0) return 0;
    XS_REQUIRE(rows > 0 && share > 0 && E > 0 && E <= 65535 && N > 0 && K > 0 && K % 8 == 0, "moe_few_rows: %d rows, %d experts, N %d, K %d", rows, E, N, K);
    XS_REQUIRE(most_an_expert > 0 && most_an_expert <= 32, "moe_few_rows: up to %d rows an expert (at most 32)", most_an_expert);
    XS_REQUIRE(ldx % 8 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)w % 16 == 0, "moe_few_rows: operands are not in 16-byte pieces");
    XS_REQUIRE(epilogue >= 0 && epilogue <= 2 && (epilogue != FEW_GATED || N % 16 == 0), "moe_few_rows: epilogue %d, N %d", epilogue, N);
    FewParams p;
    p.x = (const __nv_bfloat16*)x;
    p.w = (const __nv_bfloat16*)w;
    p.out = (__nv_bfloat16*)out;
    p.ids = ids;
    p.rows = rows; p.share = share; p.N = N; p.K = K; p.epilogue = epilogue;
    p.ldx = ldx; p.ldo = ldo;
    p.limit = limit; p.alpha = alpha; p.shift = shift;
    const dim3 grid(ceil_div_i(N, kFewRows), E);
    if (most_an_expert <= 8) xs_launch(moe_few_rows_kernel<1>, grid, dim3(kFewWarps * 32), 0, stream, p);
    else if (most_an_expert <= 16) xs_launch(moe_few_rows_kernel<2>, grid, dim3(kFewWarps * 32), 0, stream, p);
    else xs_launch(moe_few_rows_kernel<4>, grid, dim3(kFewWarps * 32), 0, stream, p);
    XS_LAUNCH_CHECK("moe_few_rows");
    return 0;
}
