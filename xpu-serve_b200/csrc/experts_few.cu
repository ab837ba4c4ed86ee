// Routed experts for few tokens (a decode step): one product kernel that finds each expert's rows by itself.
//
// A step of T tokens chooses T * top rows (token, choice) over E experts; with a handful of tokens an expert has one or two of
// them and what the product costs is its weights' bytes. The tile products of the long steps (gemm_tc.cu) want the rows sorted,
// padded to tiles of 128 and gathered, and give each CTA 256 weight rows, too few CTAs to keep memory busy. Here there is no plan and
// no gather: rows keep their own index (token * top + choice) from the router to the combine, and a CTA finds the rows of its expert
// by one look over the T * top ids. A row's result does not depend on the other rows of the step while one kernel takes it. Two kernels:
//   - up to 16 tokens (`moe_stream_kernel`): a warp streams 16 weight rows over the whole of K through a ring of its own in shared
//     memory, the expert's rows of x lie beside the rings. All CTAs of a step are resident at once and hold 64 to 80 KB of weights in
//     flight each, most of it asked for before the router's choice is known;
//   - otherwise, and where x's rows leave no room for two CTAs an SM (`moe_few_rows_kernel`): a CTA takes 32 weight rows of one expert,
//     its eight warps take k blocks of 32 in turn straight into mma.sync fragments; the warps' sums meet in shared memory.
// Bound by the weights' bytes of the experts that are met. Measured on B200, gate/up and down back to back in a graph, weights from
// memory, us, second kernel -> first (the bytes' time): 16 experts of 1,024 at width 2,048, top 4: 1 token 21.5 -> 17.7 (8), 4 tokens
// 38.9 -> 26.6 (19), 8 tokens 54.0 -> 33.8 (29), 16 tokens 54.5 -> 40 (31); 64 of 512, top 8: 8 tokens 70 -> 56 (43), 16 tokens 96 -> 67
// (54); 16 of 2,816 at width 4,096: 8 tokens 203 -> 174 (149), 16 tokens 230 (x's rows leave one CTA an SM: 246 on the first). Why the
// second is slower: a warp's two rounds of loads with nothing in flight between them, three CTAs an SM that start and end together.
// A product's time follows the groups of eight columns that it carries, whatever an expert's count is: the tcgen05 products take over
// at 17 tokens, or at 33 for small experts (ops/lib.py moe_few_tokens has both sides; 32 rows an expert are the most here).
#include <atomic>

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

// The sums of weight rows n + r and n + r + 8 (n a multiple of 16) of one row of the step go out through the epilogue.
__device__ __forceinline__ void few_finish(const FewParams& p, __nv_bfloat16* out, int n, int r, float lo, float hi) {
    const int row = n + r;
    if (p.epilogue == FEW_GATED) {                     // blocks of 8 gate rows and the 8 up rows of the same outputs; N is a multiple of 16
        if (row + 8 >= p.N) return;
        float g = lo, u = hi, y;
        if (p.limit > 0.0f) {
            g = fminf(g, p.limit);
            u = fminf(fmaxf(u, -p.limit), p.limit);
            y = g / (1.0f + __expf(-p.alpha * g)) * (u + p.shift);
        } else {
            y = g / (1.0f + __expf(-g)) * u;
        }
        out[(n >> 1) + r] = __float2bfloat16_rn(y);
        return;
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
        few_finish(p, p.out + (int64_t)list[col] * p.ldo, n0 + m * 16, l >> 2, lo, hi);
    }
}

// The same product with a warp per 16 weight rows over the whole of K: nothing is shared between warps but the expert's rows of x.
// A CTA owns 16 WARPS weight rows of one expert: eight warps, or, where all experts that can be met are at most one such CTA an SM,
// four with rings of eight stages (1 token: 22.0 -> 17.7 us). Each warp streams its 16 rows through a ring of its own (STAGES x 16 rows x 64 k, cp.async,
// 16-byte pieces swizzled by row so that ldmatrix has no bank conflicts): no barrier of the CTA, no sums to meet. `eager`: the ring
// is asked for before the wait for the kernel that chose the experts (worth it where most experts are met).
constexpr int kStageK = 64, kStageBytes = 16 * kStageK * 2;

__device__ __forceinline__ uint32_t shared_at(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, int bytes) {      // the first `bytes` (0 or 16), else zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at));
}

template <int NT, int STAGES, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 2)
moe_stream_kernel(const FewParams p, int eager) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ int list[NT * 8];
    __shared__ int count;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int e = blockIdx.y, n0 = (blockIdx.x * WARPS + warp) * 16;
    const uint32_t ring = shared_at(smem) + warp * STAGES * kStageBytes;
    const uint32_t xs = shared_at(smem) + WARPS * STAGES * kStageBytes;
    const int stages = (p.K + kStageK - 1) / kStageK;
    const int pitch = stages * kStageK * 2 + 16;         // bytes of a row of x: eight rows' pieces lie in different banks
    pdl_launch_dependents();
    // a lane copies piece (lane & 7) of rows lane / 8 + 4 j (past N: the last row, not stored)
    const int piece = lane & 7, r0 = lane >> 3;
    const __nv_bfloat16* w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = p.w + ((int64_t)e * p.N + min(n0 + r0 + 4 * j, p.N - 1)) * p.K + piece * 8;
    auto ask = [&](int s) {
        if (s < stages) {
            const uint32_t to = ring + (s % STAGES) * kStageBytes;
            const int k = s * kStageK;
            const int bytes = k + piece * 8 < p.K ? 16 : 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int r = r0 + 4 * j;
                copy16(to + r * 128 + ((piece ^ (r & 7)) << 4), bytes > 0 ? w[j] + k : p.w, bytes);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (eager) {
#pragma unroll
        for (int s = 0; s < STAGES - 1; ++s) ask(s);
    }
    pdl_wait();
    if (warp == 0) {                                     // the expert's rows, in order
        int have = 0;
        for (int i0 = 0; i0 < p.rows; i0 += 32) {
            const bool mine = i0 + lane < p.rows && p.ids[i0 + lane] == e;
            const unsigned who = __ballot_sync(0xffffffffu, mine);
            const int at = have + __popc(who & ((1u << lane) - 1u));
            if (mine && at < NT * 8) list[at] = i0 + lane;
            have += __popc(who);
        }
        if (lane == 0) count = min(have, NT * 8);        // (a token names an expert once, so an expert has at most T rows)
    }
    __syncthreads();
    const int rows = count;
    if (rows == 0) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        return;
    }
    if (!eager) {
#pragma unroll
        for (int s = 0; s < STAGES - 1; ++s) ask(s);
    }
    // the expert's rows of x, a warp a row at a time; zeros past them and past K
    const int pieces = stages * 8;
    for (int r = warp; r < NT * 8; r += WARPS) {
        const bool live = r < rows;
        const __nv_bfloat16* from = live ? p.x + (int64_t)(list[r] / p.share) * p.ldx : p.x;
        for (int c = lane; c < pieces; c += 32)
            copy16(xs + r * pitch + c * 16, c * 8 < p.K ? from + c * 8 : from, live && c * 8 < p.K ? 16 : 0);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    float acc[2][NT][4];                                 // even and odd pairs of k steps: two chains
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[c][t][j] = 0.0f;
    const int ar = lane & 15, ac = lane >> 4;            // ldmatrix: this lane's row and half of a weight tile
    for (int s = 0; s < stages; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncwarp();                                    // every lane's pieces of stage s are here, stage s - 1 has been read
        ask(s + STAGES - 1);
        const uint32_t at = ring + (s % STAGES) * kStageBytes + ar * 128;
#pragma unroll
        for (int h = 0; h < 2; ++h) {                    // 32 k
            uint32_t a[2][4];
#pragma unroll
            for (int q = 0; q < 2; ++q) ldmatrix4(a[q], at + (((h * 4 + q * 2 + ac) ^ (ar & 7)) << 4));
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                uint32_t b[4];
                ldmatrix4(b, xs + (t * 8 + (lane & 7)) * pitch + (s * 8 + h * 4 + (lane >> 3)) * 16);
                mma_bf16(acc[h][t], a[0][0], a[0][1], a[0][2], a[0][3], b[0], b[1]);
                mma_bf16(acc[h][t], a[1][0], a[1][1], a[1][2], a[1][3], b[2], b[3]);
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    // lane: weight rows n0 + lane / 4 and + 8, columns 2 (lane & 3) and the next
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int col = t * 8 + (lane & 3) * 2 + j;
            if (col >= rows) continue;
            float lo = acc[0][t][j] + acc[1][t][j], hi = acc[0][t][j + 2] + acc[1][t][j + 2];
            few_finish(p, p.out + (int64_t)list[col] * p.ldo, n0, lane >> 2, lo, hi);
        }
}

constexpr size_t kMostSmem = 226 * 1024, kHalfSmem = 113 * 1024;      // of a CTA, and of each of two on an SM
size_t stream_smem(int nt, int stages, int warps, int K) { return (size_t)warps * stages * kStageBytes + (size_t)nt * 8 * ((size_t)ceil_div_i(K, kStageK) * kStageK * 2 + 16); }

template <int NT, int STAGES, int WARPS>
int launch_stream(const FewParams& p, int E, int eager, cudaStream_t stream) {
    const size_t smem = stream_smem(NT, STAGES, WARPS, p.K);
    static std::atomic<bool> done{false};
    if (!done.load(std::memory_order_acquire)) {
        if (cudaFuncSetAttribute(moe_stream_kernel<NT, STAGES, WARPS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMostSmem) != cudaSuccess) return -1;
        done.store(true, std::memory_order_release);
    }
    return xs_launch(moe_stream_kernel<NT, STAGES, WARPS>, dim3(ceil_div_i(p.N, 16 * WARPS), E), dim3(WARPS * 32), smem, stream, p,
                     eager) == cudaSuccess ? 0 : -1;
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
    const int eager = rows >= E;
    const int groups = most_an_expert <= 8 ? 1 : 2;
    // few CTAs for the experts that can be met: smaller ones, each with a deeper ring
    const bool narrow = groups == 1 && (int64_t)(rows < E ? rows : E) * ceil_div_i(N, 128) <= 148;
    int rc = 1;                                          // 1: not taken
    if (most_an_expert <= 16) {
        if (narrow && stream_smem(1, 8, 4, K) <= kMostSmem) rc = launch_stream<1, 8, 4>(p, E, eager, stream);
        else if (groups == 1 && stream_smem(1, 5, 8, K) <= kHalfSmem) rc = launch_stream<1, 5, 8>(p, E, eager, stream);
        else if (groups == 1 && stream_smem(1, 4, 8, K) <= kHalfSmem) rc = launch_stream<1, 4, 8>(p, E, eager, stream);
        else if (groups == 1 && stream_smem(1, 5, 8, K) <= kMostSmem) rc = launch_stream<1, 5, 8>(p, E, eager, stream);
        else if (groups == 2 && stream_smem(2, 3, 8, K) <= kHalfSmem) rc = launch_stream<2, 3, 8>(p, E, eager, stream);
    }
    XS_REQUIRE(rc >= 0, "moe_few_rows: launch failed: %s", cudaGetErrorString(cudaGetLastError()));
    if (rc == 0) return 0;
    const dim3 grid(ceil_div_i(N, kFewRows), E);
    if (most_an_expert <= 8) xs_launch(moe_few_rows_kernel<1>, grid, dim3(kFewWarps * 32), 0, stream, p);
    else if (most_an_expert <= 16) xs_launch(moe_few_rows_kernel<2>, grid, dim3(kFewWarps * 32), 0, stream, p);
    else xs_launch(moe_few_rows_kernel<4>, grid, dim3(kFewWarps * 32), 0, stream, p);
    XS_LAUNCH_CHECK("moe_few_rows");
    return 0;
}
