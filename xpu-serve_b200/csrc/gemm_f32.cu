// out[M, N] = x[M, K] . w[N, K]^T (+ bias[N]) in float32 on CUDA-core FMAs: the float32 path's product where rows start on
// 16-byte boundaries (gemm_generic.cu keeps the other cases and the element types).
//
// Order of the sums: 32 consecutive k into a partial by fused multiply-adds in ascending k, partials added in ascending k, for
// every output and in every kernel here. It is the order of gemm_generic.cu, so a row's result is the same bit for bit whatever
// the other rows of the call are, and whichever kernel takes them.
//
// Two kernels:
//   few rows (up to 64, 4, 8 or 16 at a time): bound by the weights' bytes. A CTA takes 8 weight rows at a time and streams them
//     past x in stages of 1,024 k (cp.async, two stages, a 16-byte piece of every row a thread), a thread multiplying one 32-k chunk
//     of one weight row. The chunks' partials meet in shared memory, where one thread an output adds them in order while the next
//     stage is multiplied. Weight rows' 16-byte pieces are swizzled by row, x's by chunk, so that neither load has bank conflicts.
//     (With 128 threads, stages of 512 k and one or two weight rows a thread the SM had one warp a scheduler: 2.0 TB/s.)
//   more rows: bound by the FMA units. 64 x 128 outputs a CTA of 128 threads, 8 x 8 a thread, both operands in stages of 32 k as
//     they lie in memory (rows of k, 36 floats apart: the eight rows of a 16-byte load's phase fall into different banks), so
//     nothing is transposed; a stage is exactly one partial. Where such tiles are few for the device's SMs, 64 x 64 a CTA and 4 x 8 a
//     thread: a warp alone multiplies no more often than every second cycle, so an SM of one tile wants its outputs on more warps
//     (one of 64 x 64 with 8 x 8 a thread took as long as one of 64 x 128: 424 us at K 6656, on four warps 270). With the device
//     full 8 x 8 is the better one, since it reads less from shared memory a product.
//
// Measured on B200 (products of the 350M shape, weights from memory, us; before: the 64 x 64 tile of gemm_generic.cu, whose time
// does not depend on the rows):
//     N 13312 K 1024    4 rows 210 -> 13.5 (4.0 TB/s)   16 rows 212 -> 32   64 rows 221 -> 76    1,294 rows 1,569 -> 832 (42 TFLOP/s)
//     N  1024 K 6656    4 rows 1,218 -> 14.7            16 rows 1,232 -> 20   64 rows 1,264 -> 72   1,294 rows 1,144 -> 615
//     N 65536 K 1024    4 rows 462 -> 52 (5.2 TB/s)     16 rows 464 -> 140
// Tiles of both kinds (us, L2 flushed; 64 x 128 of 8 x 8 / 64 x 64 of 4 x 8):
//     rows                65          128          300          700          1,294
//     N 13312 K 1024   117 / 102   119 / 104   225 / 254    444 / 492    832 / 907
//     N  3072 K 1024    74 / 49     74 / 49     75 / 80     119 / 135    225 / 223
//     N  2048 K 1024    74 / 47     74 / 47     74 / 74     117 / 102    182 / 168
//     N  1024 K 1024    72 / 47     72 / 47     74 / 47      74 / 78     117 / 102
//     N  1024 K 6656   424 / 270   424 / 270   436 / 272    438 / 471    709 / 615
// n tiles on the SM that has the most take 56 n + 18 us (64 x 128) or 31 n + 16 (64 x 64) at K 1024: hence the line between them.
// Passes of 16 rows against the 64 x 64 tiles (us): N 1024 K 1024 35 / 47 at 160 rows, 41 / 47 at 192, 51 / 47 at 256; K 6656 166 /
// 271 at 160, 256 / 272 at 256; N 2048 K 1024 39 / 47 at 96 rows, 47 / 47 at 128, 53 / 47 at 144; N 3072 K 1024 43 / 47 at 80, 51 / 48
// at 96: passes up to 14 x 1,024 passes times outputs a row.
#include <atomic>

#include "common.cuh"

namespace {

constexpr int kChunk = 32;            // k of one partial sum
constexpr int kStages = 3;            // of the tile kernel
constexpr int kFewThreads = 256, kFewRows = 8;      // few rows: threads and weight rows a CTA
constexpr int kStageK = 4 * kFewThreads;            // few rows: k of a stage, a 16-byte piece of every row a thread
constexpr int kFewRowsMost = 64;
constexpr int kFewOutputs = 14 * 1024;               // passes of 16 rows times outputs a row
constexpr int kSmemOfSm = 228 * 1024; // shared memory of an SM, of which each CTA takes 1 KB for itself
constexpr int kDevices = 64;          // devices that remember their shared-memory limit (further ones set it each time)

__device__ __forceinline__ uint32_t smem_at(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// 16 bytes, of which the first `bytes` (0 to 16) are read and the rest are zeros.
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Up to MR rows of x.
template <int MR>
__global__ void __launch_bounds__(kFewThreads, MR <= 4 ? 2 : 1)
gemm_f32_few_rows_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                         float* __restrict__ out, int M, int N, int K, int64_t ldx, int64_t ldw, int64_t ldo) {
    constexpr int kChunks = kStageK / kChunk;                     // 32
    constexpr int kStageFloats = (kFewRows + MR) * kStageK;
    constexpr int kOuts = kFewRows * MR;                          // 32, 64 or 128: at most one a thread
    extern __shared__ __align__(16) float sm[];
    float* parts = sm + 2 * kStageFloats;                         // [2][kChunks][MR][kFewRows]
    const int m0 = blockIdx.y * MR;
    const int r = threadIdx.x & 7, c = threadIdx.x >> 3;          // a thread multiplies chunk c of weight row r
    // and copies the 16-byte piece r of chunk c of every row: its place in a row of the stage, for weight rows turned by the row
    const int piece = threadIdx.x * 4;
    pdl_launch_dependents();
    const int stages = (K + kStageK - 1) / kStageK;
    const int tiles = (N + kFewRows - 1) / kFewRows;
    // the CTA's tiles are walked as one run of stages: the next tile's weights are on their way while this one's are multiplied
    const int total = ((tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x) * stages;
    auto load_w = [&](float* stage, int n0, int k0) {
        const int bytes = min(16, max(0, (K - k0 - piece) * 4));
        const float* from = w + (int64_t)n0 * ldw + k0 + piece;
        const uint32_t to = smem_at(stage + c * kChunk);
#pragma unroll
        for (int q = 0; q < kFewRows; ++q) {
            const int there = n0 + q < N ? bytes : 0;
            copy16(to + (uint32_t)(q * kStageK + ((r ^ q) << 2)) * 4u, there > 0 ? from + (int64_t)q * ldw : w, there);
        }
    };
    auto load_x = [&](float* stage, int k0) {
        const int bytes = min(16, max(0, (K - k0 - piece) * 4));
        const float* from = x + (int64_t)m0 * ldx + k0 + piece;
        const uint32_t to = smem_at(stage + kFewRows * kStageK + c * kChunk + ((r ^ (c & 7)) << 2));
#pragma unroll
        for (int q = 0; q < MR; ++q) {
            const int there = m0 + q < M ? bytes : 0;
            copy16(to + (uint32_t)(q * kStageK) * 4u, there > 0 ? from + (int64_t)q * ldx : x, there);
        }
    };
    int load_n = blockIdx.x * kFewRows, load_s = 0;               // the stage to be asked for next
    auto next_load = [&] {
        if (++load_s == stages) {
            load_s = 0;
            load_n += gridDim.x * kFewRows;
        }
    };
    if (total > 0) load_w(sm, load_n, 0);
    pdl_wait();                                                   // x is written by the kernel before this one
    if (total > 0) load_x(sm, 0);
    copies_commit();
    next_load();
    float acc = 0.0f;
    int n0 = blockIdx.x * kFewRows, s_at = 0;                     // the stage whose partials are added next
    // adds a stage's partials; behind a tile's last stage, stores its outputs
    auto add_parts = [&](const float* from) {
        const int o = threadIdx.x;
        if (o < kOuts) {
#pragma unroll
            for (int j = 0; j < kChunks; ++j) acc += from[j * kOuts + o];
            if (s_at == stages - 1) {
                const int m = m0 + o / kFewRows, n = n0 + o % kFewRows;
                if (m < M && n < N) out[(int64_t)m * ldo + n] = bias != nullptr ? acc + bias[n] : acc;
                acc = 0.0f;
            }
        }
        if (++s_at == stages) {
            s_at = 0;
            n0 += gridDim.x * kFewRows;
        }
    };
    for (int g = 0; g < total; ++g) {
        copies_wait<0>();
        __syncthreads();                      // stage g is here, stage g - 1 has been read, its partials are written
        if (g + 1 < total) {
            float* to = sm + ((g + 1) & 1) * kStageFloats;
            load_w(to, load_n, load_s * kStageK);
            load_x(to, load_s * kStageK);
            next_load();
        }
        copies_commit();
        const float* ws = sm + (g & 1) * kStageFloats + r * kStageK + c * kChunk;
        const float* xs = sm + (g & 1) * kStageFloats + kFewRows * kStageK + c * kChunk;
        float part[MR];
#pragma unroll
        for (int m = 0; m < MR; ++m) part[m] = 0.0f;
#pragma unroll
        for (int i = 0; i < kChunk / 4; ++i) {
            const float4 b = *reinterpret_cast<const float4*>(ws + ((i ^ r) << 2));
            float4 a[MR];
#pragma unroll
            for (int m = 0; m < MR; ++m) a[m] = *reinterpret_cast<const float4*>(xs + m * kStageK + ((i ^ (c & 7)) << 2));
#pragma unroll
            for (int m = 0; m < MR; ++m) part[m] = fmaf(a[m].x, b.x, part[m]);
#pragma unroll
            for (int m = 0; m < MR; ++m) part[m] = fmaf(a[m].y, b.y, part[m]);
#pragma unroll
            for (int m = 0; m < MR; ++m) part[m] = fmaf(a[m].z, b.z, part[m]);
#pragma unroll
            for (int m = 0; m < MR; ++m) part[m] = fmaf(a[m].w, b.w, part[m]);
        }
        if (g > 0) add_parts(parts + ((g - 1) & 1) * kChunks * kOuts);
        float* to = parts + ((g & 1) * kChunks + c) * kOuts + r;
#pragma unroll
        for (int m = 0; m < MR; ++m) to[m * kFewRows] = part[m];
    }
    __syncthreads();
    if (total > 0) add_parts(parts + ((total - 1) & 1) * kChunks * kOuts);
}

constexpr int BM = 64, kRow = kChunk + 4;

// RT x 8 outputs a thread, CTAS CTAs an SM.
template <int BN, int RT, int CTAS>
__global__ void __launch_bounds__(BN / 8 * (BM / RT), CTAS)
gemm_f32_tile_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                     float* __restrict__ out, int M, int N, int K, int64_t ldx, int64_t ldw, int64_t ldo) {
    extern __shared__ __align__(16) float sm[];
    constexpr int kTileFloats = (BM + BN) * kRow, TX = BN / 8, TY = BM / RT, kStep = TX * TY / 8;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
    const int stages = (K + kChunk - 1) / kChunk;
    // a thread copies the piece tid & 7 of the rows tid / 8, + kStep, + 2 kStep, ... of each operand
    const int piece = threadIdx.x & 7, row = threadIdx.x >> 3;
    auto load = [&](int s, bool weights, bool inputs) {
        float* to = sm + (s % kStages) * kTileFloats;
        const int k = s * kChunk + piece * 4;
        const int left = min(16, max(0, (K - k) * 4));
        if (inputs) {
#pragma unroll
            for (int q = 0; q < BM / kStep; ++q) {
                const int m = m0 + row + kStep * q;
                const int n_bytes = m < M ? left : 0;
                copy16(smem_at(to + (row + kStep * q) * kRow + piece * 4), n_bytes > 0 ? x + (int64_t)m * ldx + k : x, n_bytes);
            }
        }
        if (weights) {
#pragma unroll
            for (int q = 0; q < BN / kStep; ++q) {
                const int n = n0 + row + kStep * q;
                const int n_bytes = n < N ? left : 0;
                copy16(smem_at(to + (BM + row + kStep * q) * kRow + piece * 4), n_bytes > 0 ? w + (int64_t)n * ldw + k : w, n_bytes);
            }
        }
    };
    pdl_launch_dependents();
#pragma unroll
    for (int s = 0; s < kStages - 1; ++s)
        if (s < stages) load(s, true, false);
    pdl_wait();
#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) {
        if (s < stages) load(s, false, true);
        copies_commit();
    }
    float acc[RT][8];
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
    for (int s = 0; s < stages; ++s) {
        copies_wait<kStages - 2>();
        __syncthreads();
        if (s + kStages - 1 < stages) load(s + kStages - 1, true, true);
        copies_commit();
        const float* xs = sm + (s % kStages) * kTileFloats + ty * kRow;
        const float* ws = sm + (s % kStages) * kTileFloats + (BM + tx) * kRow;
        float part[RT][8];
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) part[i][j] = 0.0f;
#pragma unroll 2
        for (int k = 0; k < kChunk; k += 4) {
            float4 a[RT];
#pragma unroll
            for (int i = 0; i < RT; ++i) a[i] = *reinterpret_cast<const float4*>(xs + TY * i * kRow + k);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float4 b = *reinterpret_cast<const float4*>(ws + TX * j * kRow + k);
#pragma unroll
                for (int i = 0; i < RT; ++i) part[i][j] = fmaf(a[i].x, b.x, part[i][j]);
#pragma unroll
                for (int i = 0; i < RT; ++i) part[i][j] = fmaf(a[i].y, b.y, part[i][j]);
#pragma unroll
                for (int i = 0; i < RT; ++i) part[i][j] = fmaf(a[i].z, b.z, part[i][j]);
#pragma unroll
                for (int i = 0; i < RT; ++i) part[i][j] = fmaf(a[i].w, b.w, part[i][j]);
            }
        }
#pragma unroll
        for (int i = 0; i < RT; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] += part[i][j];
    }
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        const int m = m0 + ty + TY * i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int n = n0 + tx + TX * j;
            if (n < N) out[(int64_t)m * ldo + n] = bias != nullptr ? acc[i][j] + bias[n] : acc[i][j];
        }
    }
}

// Lets a kernel of more than 48 KB of shared memory run on the current device: once a device, as the attribute is a device's.
template <typename K>
cudaError_t opt_in(K* kernel, size_t smem, std::atomic<bool> (&done)[kDevices]) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess || (device < kDevices && done[device].load(std::memory_order_acquire))) return e;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess && device < kDevices) done[device].store(true, std::memory_order_release);
    return e;
}

template <int MR>
cudaError_t launch_few(const float* x, const float* w, const float* bias, float* out, int M, int N, int K, int64_t ldx, int64_t ldw,
                       int64_t ldo, cudaStream_t stream) {
    const size_t smem = (2 * (size_t)(kFewRows + MR) * kStageK + 2 * (kStageK / kChunk) * kFewRows * MR) * sizeof(float);
    static std::atomic<bool> done[kDevices];
    const cudaError_t e = opt_in(gemm_f32_few_rows_kernel<MR>, smem, done);
    if (e != cudaSuccess) return e;
    const int tiles = ceil_div_i(N, kFewRows), chunks = ceil_div_i(M, MR);
    const int fit = 148 * (smem <= 110 * 1024 ? 2 : 1);           // CTAs that are resident at one time
    return xs_launch(gemm_f32_few_rows_kernel<MR>, dim3(tiles < fit ? tiles : fit, chunks), dim3(kFewThreads), smem, stream, x, w, bias,
                     out, M, N, K, ldx, ldw, ldo);
}

template <int BN, int RT, int CTAS>
cudaError_t launch_tile(const float* x, const float* w, const float* bias, float* out, int M, int N, int K, int64_t ldx, int64_t ldw,
                        int64_t ldo, cudaStream_t stream) {
    const size_t needs = (size_t)kStages * (BM + BN) * kRow * sizeof(float);
    // No more CTAs an SM than an even share: the CTAs of this launch that start while the kernel before it still runs take the places
    // that it left, which gave some SMs four tiles where three would do (N 1024, K 6656, 1,294 rows in a run of launches: 800 us
    // instead of 616; with the limit 607).
    const int64_t share = ((int64_t)ceil_div_i(N, BN) * ceil_div_i(M, BM) + 147) / 148;
    const size_t fills = share < CTAS ? (size_t)(kSmemOfSm / (int)share - 1024) & ~(size_t)15 : 0, smem = fills > needs ? fills : needs;
    static std::atomic<bool> done[kDevices];
    const cudaError_t e = opt_in(gemm_f32_tile_kernel<BN, RT, CTAS>, kSmemOfSm - 1024, done);
    if (e != cudaSuccess) return e;
    return xs_launch(gemm_f32_tile_kernel<BN, RT, CTAS>, dim3(ceil_div_i(N, BN), ceil_div_i(M, BM)), dim3(BN / 8 * (BM / RT)), smem, stream,
                     x, w, bias, out, M, N, K, ldx, ldw, ldo);
}

}  // namespace

// Whether the kernels here take a product: rows that start on 16-byte boundaries.
bool xs_gemm_f32_takes(const void* x, const void* w, int64_t ldx, int64_t ldw) {
    return (uintptr_t)x % 16 == 0 && (uintptr_t)w % 16 == 0 && ldx % 4 == 0 && ldw % 4 == 0;
}

int xs_gemm_f32(const float* x, const float* w, const float* bias, float* out, int M, int N, int K, int64_t ldx, int64_t ldw,
                int64_t ldo, cudaStream_t stream) {
    cudaError_t e;
    // (between 17 and 64 rows: the tiles where they are enough to fill half of the device's SMs; above, passes of 16 rows of narrow
    // products)
    if (M <= 16 || (M <= kFewRowsMost && ceil_div_i(N, 64) < 74) || (int64_t)ceil_div_i(M, 16) * N <= kFewOutputs) {
        e = M <= 4 ? launch_few<4>(x, w, bias, out, M, N, K, ldx, ldw, ldo, stream)
            : M <= 8 ? launch_few<8>(x, w, bias, out, M, N, K, ldx, ldw, ldo, stream)
                     : launch_few<16>(x, w, bias, out, M, N, K, ldx, ldw, ldo, stream);
    } else {
        XS_REQUIRE(ceil_div_i(M, BM) <= 65535, "gemm: %d rows exceed the grid limit", M);
        // (tiles on the SM that has the most; the figures are above)
        const int64_t rows = ceil_div_i(M, BM), narrow = (rows * ceil_div_i(N, 64) + 147) / 148, wide = (rows * ceil_div_i(N, 128) + 147) / 148;
        e = 5 * narrow < 9 * wide ? launch_tile<64, 4, 4>(x, w, bias, out, M, N, K, ldx, ldw, ldo, stream)
                                  : launch_tile<128, 8, 2>(x, w, bias, out, M, N, K, ldx, ldw, ldo, stream);
    }
    XS_REQUIRE(e == cudaSuccess, "gemm (float32): launch failed: %s", cudaGetErrorString(e));
    return 0;
}
