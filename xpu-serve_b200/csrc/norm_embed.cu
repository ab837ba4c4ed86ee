// Embedding gather, fused residual-add + RMSNorm, SwiGLU activation, error state.
//
// RMSNorm(x, w, eps) = x * (mean(x^2) + eps)^(-1/2) * w over the last dimension, no +1
// offset, all in float32 (reference: src/graph/graph.h:57, kernel
// src/backend/sycl/sycl_kernels.cpp:1543-1559). The residual stream is float32 in every
// precision mode; a branch's output joins it here.
#include <stdarg.h>
#include <stdio.h>

#include "common.cuh"

static thread_local char g_error[512] = "";

void xs_set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_error, sizeof(g_error), fmt, ap);
    va_end(ap);
}

XS_API const char* xs_last_error() { return g_error; }

XS_API int xs_abi_version() { return 5; }

int g_xs_pdl = 1;
// 1: kernels of a step may overlap their start with the previous kernel's end (programmatic
// dependent launch); 0: plain stream order. Returns the previous setting.
XS_API int xs_set_pdl(int on) {
    const int old = g_xs_pdl;
    g_xs_pdl = on ? 1 : 0;
    return old;
}

// ------------------------------------------------------------------ embedding
// h[t, :] = table[ids[t], :] * scale as float32 (LFM3: scale 1, src/models/lfm3/lfm3_decoder.cpp:50).
template <typename TW>
__global__ void embed_kernel(const TW* __restrict__ table, const int32_t* __restrict__ ids,
                             float* __restrict__ h, int T, int H, float scale) {
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x;
    const TW* row = table + (int64_t)ids[t] * H;
    float* out = h + (int64_t)t * H;
    for (int c = threadIdx.x; c < H; c += blockDim.x) out[c] = to_f32(row[c]) * scale;
}

// The same for bfloat16 rows on 16-byte boundaries whose width is a multiple of 8: eight elements a thread, one load.
__global__ void embed_bf16x8_kernel(const __nv_bfloat16* __restrict__ table, const int32_t* __restrict__ ids, float* __restrict__ h, int T,
                                    int H, float scale) {
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x;
    const uint4* row = reinterpret_cast<const uint4*>(table + (int64_t)ids[t] * H);
    float4* out = reinterpret_cast<float4*>(h + (int64_t)t * H);
    for (int c = threadIdx.x; c < (H >> 3); c += blockDim.x) {
        const uint4 raw = row[c];
        const __nv_bfloat162* two = reinterpret_cast<const __nv_bfloat162*>(&raw);
        const float2 a = __bfloat1622float2(two[0]), b = __bfloat1622float2(two[1]), e = __bfloat1622float2(two[2]), f = __bfloat1622float2(two[3]);
        out[2 * c] = make_float4(a.x * scale, a.y * scale, b.x * scale, b.y * scale);
        out[2 * c + 1] = make_float4(e.x * scale, e.y * scale, f.x * scale, f.y * scale);
    }
}

// A token's row plus a row of a second table chosen by a hash of the previous and the current token, plus a sine/cosine
// vector of the position, then an RMS norm (w == nullptr: none):
//     x = table[tok] * scale + pair[pos == 0 ? buckets : (prev * mul_prev + tok * mul_cur) mod buckets]
//     x[2 i] += sin(pos f_i),  x[2 i + 1] += cos(pos f_i)          (inv_freq holds the f_i in float32; the angle is float32)
//     h = x / sqrt(mean(x^2) + eps) * w
// The previous token of a step's first token of a sequence is what `last_token[slot]` holds; the block of that token then
// writes the sequence's last token of this step there, so the word is read before it is written whatever the order of blocks.
template <typename TW>
__global__ void embed_pair_kernel(const TW* __restrict__ table, const TW* __restrict__ pair, const int32_t* __restrict__ ids,
                                  const int32_t* __restrict__ positions, const int32_t* __restrict__ seq_of_token,
                                  const int32_t* __restrict__ cu_seqlens, const int32_t* __restrict__ slots,
                                  int32_t* __restrict__ last_token, const float* __restrict__ inv_freq,
                                  const float* __restrict__ w, float* __restrict__ h, int H, float scale, int buckets,
                                  long long mul_prev, long long mul_cur, float eps) {
    extern __shared__ float row[];
    __shared__ float scratch[32];
    __shared__ int prev_s;
    pdl_launch_dependents();
    const int t = blockIdx.x;
    const int seq = seq_of_token[t], pos = positions[t], tok = ids[t];
    const int first = cu_seqlens[seq], end = cu_seqlens[seq + 1];
    pdl_wait();
    if (threadIdx.x == 0) {
        int prev = 0;
        if (t == first) {
            const int slot = slots[seq];
            prev = last_token[slot];
            last_token[slot] = ids[end - 1];
        } else {
            prev = ids[t - 1];
        }
        prev_s = prev;
    }
    __syncthreads();
    const long long bucket = pos == 0 ? (long long)buckets : ((long long)prev_s * mul_prev + (long long)tok * mul_cur) % buckets;
    const TW* er = table + (int64_t)tok * H;
    const TW* pr = pair + bucket * H;
    float ss = 0.0f;
    for (int i = threadIdx.x; 2 * i < H; i += blockDim.x) {          // a thread takes the sine and the cosine of one angle
        float sn, cs;
        sincosf((float)pos * inv_freq[i], &sn, &cs);
        const int c = 2 * i;
        const float v0 = to_f32(er[c]) * scale + to_f32(pr[c]) + sn;
        row[c] = v0;
        ss += v0 * v0;
        if (c + 1 < H) {
            const float v1 = to_f32(er[c + 1]) * scale + to_f32(pr[c + 1]) + cs;
            row[c + 1] = v1;
            ss += v1 * v1;
        }
    }
    float* out = h + (int64_t)t * H;
    if (w == nullptr) {
        __syncthreads();
        for (int c = threadIdx.x; c < H; c += blockDim.x) out[c] = row[c];
        return;
    }
    ss = block_sum(ss, scratch);          // (its barriers also order the row's writes before the reads below)
    const float inv = 1.0f / sqrtf(ss / (float)H + eps);
    for (int c = threadIdx.x; c < H; c += blockDim.x) out[c] = row[c] * inv * w[c];
}

// logits = cap * tanh(logits / cap), in place: a soft limit that some architectures put on their logits.
__global__ void logit_cap_kernel(float* __restrict__ logits, int64_t n, float cap, float inv_cap) {
    pdl_launch_dependents();
    pdl_wait();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        logits[i] = cap * tanhf(logits[i] * inv_cap);
}

__global__ void logit_scale_kernel(float* __restrict__ logits, int64_t n, float scale) {
    pdl_launch_dependents();
    pdl_wait();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) logits[i] *= scale;
}

XS_API int xs_embed(const void* table, int table_dtype, const int32_t* ids, float* h, int T, int H, float scale,
                    cudaStream_t stream) {
    if (T == 0) return 0;
    XS_REQUIRE(T > 0 && H > 0, "embed: %d tokens of width %d", T, H);
    if (table_dtype == XS_BF16 && H % 8 == 0 && ((uintptr_t)table | (uintptr_t)h) % 16 == 0) {
        xs_launch(embed_bf16x8_kernel, dim3(T), dim3(H >= 1024 ? 256 : 128), 0, stream, (const __nv_bfloat16*)table, ids, h, T, H, scale);
        XS_LAUNCH_CHECK("embed");
        return 0;
    }
    XS_DISPATCH_DTYPE(table_dtype, TW,
                      xs_launch(embed_kernel<TW>, dim3(T), dim3(256), 0, stream, (const TW*)table, ids, h, T, H, scale));
    XS_LAUNCH_CHECK("embed");
    return 0;
}

XS_API int xs_embed_pair(const void* table, const void* pair, int table_dtype, const int32_t* ids, const int32_t* positions,
                         const int32_t* seq_of_token, const int32_t* cu_seqlens, const int32_t* slots, int32_t* last_token,
                         const float* inv_freq, const float* w, float* h, int T, int H, float scale, int buckets,
                         long long mul_prev, long long mul_cur, float eps, cudaStream_t stream) {
    if (T == 0) return 0;
    XS_REQUIRE(T > 0 && H > 0 && buckets > 0 && mul_prev >= 0 && mul_cur >= 0, "embed_pair: %d tokens of width %d, %d buckets", T, H, buckets);
    XS_REQUIRE((size_t)H * 4 <= 200 * 1024, "embed_pair: width %d does not fit shared memory (limit 51200)", H);
    const size_t smem = (size_t)H * sizeof(float);
#define XS_GO(TW)                                                                                                          \
    do {                                                                                                                   \
        if (smem > 48 * 1024)                                                                                              \
            cudaFuncSetAttribute(embed_pair_kernel<TW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);           \
        xs_launch(embed_pair_kernel<TW>, dim3(T), dim3(H >= 2048 ? 512 : 256), smem, stream, (const TW*)table,             \
                  (const TW*)pair, ids, positions, seq_of_token, cu_seqlens, slots, last_token, inv_freq, w, h, H, scale,  \
                  buckets, mul_prev, mul_cur, eps);                                                                        \
    } while (0)
    XS_DISPATCH_DTYPE(table_dtype, TW, XS_GO(TW));
#undef XS_GO
    XS_LAUNCH_CHECK("embed_pair");
    return 0;
}

// logits *= scale, in place: a constant that some architectures put between the head and the softmax.
XS_API int xs_logit_scale(float* logits, int64_t n, float scale, cudaStream_t stream) {
    if (n == 0) return 0;
    XS_REQUIRE(n > 0, "logit scale: %lld values", (long long)n);
    const int blocks = (int)(n / 1024 < 1 ? 1 : (n / 1024 > 1184 ? 1184 : n / 1024));
    xs_launch(logit_scale_kernel, dim3(blocks), dim3(256), 0, stream, logits, n, scale);
    XS_LAUNCH_CHECK("logit_scale");
    return 0;
}

XS_API int xs_logit_cap(float* logits, int64_t n, float cap, cudaStream_t stream) {
    if (n == 0) return 0;
    XS_REQUIRE(n > 0 && cap > 0.0f, "logit cap: %lld values, cap %g", (long long)n, (double)cap);
    const int blocks = (int)(n / 1024 < 1 ? 1 : (n / 1024 > 1184 ? 1184 : n / 1024));
    xs_launch(logit_cap_kernel, dim3(blocks), dim3(256), 0, stream, logits, n, cap, 1.0f / cap);
    XS_LAUNCH_CHECK("logit_cap");
    return 0;
}

// ------------------------------------------------------- add + RMSNorm (fused)
// For each output row i (source row r = rows ? rows[i] : i):
//   v = h[r]                                   float32
//   if m:      b = m[r];  if post_w: b = RMSNorm(b, post_w, eps_post)
//              v = v + b;  h[r] = v            the residual sum stays float32
//   if w:      y[i] = RMSNorm(v, w, eps)       written in y's element type
//   else if y: y[i] = v                        (a layer whose sublayers read the stream itself)
// One block per row; the row lives in shared memory between the passes.
template <typename TM, typename TY>
__global__ void add_rmsnorm_kernel(float* __restrict__ h, const TM* __restrict__ m,
                                   const float* __restrict__ post_w, const float* __restrict__ w,
                                   TY* __restrict__ y, const int32_t* __restrict__ rows, int H, float eps_post, float eps) {
    extern __shared__ float row[];
    __shared__ float scratch[32];
    pdl_launch_dependents();
    pdl_wait();
    const int i = blockIdx.x;
    const int64_t r = rows ? rows[i] : i;
    float* hr = h + r * H;
    float ss = 0.0f;
    if (m != nullptr) {
        const TM* mr = m + r * H;
        if (post_w != nullptr) {
            float bs = 0.0f;
            for (int c = threadIdx.x; c < H; c += blockDim.x) {
                const float b = to_f32(mr[c]);
                row[c] = b;
                bs += b * b;
            }
            bs = block_sum(bs, scratch);
            const float inv = 1.0f / sqrtf(bs / (float)H + eps_post);
            for (int c = threadIdx.x; c < H; c += blockDim.x) {
                const float v = hr[c] + row[c] * inv * post_w[c];
                row[c] = v;
                hr[c] = v;
                ss += v * v;
            }
        } else {
            for (int c = threadIdx.x; c < H; c += blockDim.x) {
                const float v = hr[c] + to_f32(mr[c]);
                row[c] = v;
                hr[c] = v;
                ss += v * v;
            }
        }
    } else {
        for (int c = threadIdx.x; c < H; c += blockDim.x) {
            const float v = hr[c];
            row[c] = v;
            ss += v * v;
        }
    }
    if (w == nullptr) {
        // no norm reads the stream: y (when given) is the sum itself in y's element type
        if (y != nullptr) {
            __syncthreads();
            TY* yc = y + (int64_t)i * H;
            for (int c = threadIdx.x; c < H; c += blockDim.x) yc[c] = from_f32<TY>(row[c]);
        }
        return;
    }
    ss = block_sum(ss, scratch);
    const float inv = 1.0f / sqrtf(ss / (float)H + eps);
    TY* yr = y + (int64_t)i * H;
    for (int c = threadIdx.x; c < H; c += blockDim.x) yr[c] = from_f32<TY>(row[c] * inv * w[c]);
}


// The same operation for widths that are a multiple of 4 and at most 16 * 1024: each thread keeps
// up to four float4 of the row in registers, so the row is read once and every pass after the
// first runs on registers.
template <typename TM>
__device__ __forceinline__ float4 load4(const TM* p);
template <>
__device__ __forceinline__ float4 load4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <>
__device__ __forceinline__ float4 load4<__nv_bfloat16>(const __nv_bfloat16* p) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(__nv_bfloat16* p, float4 v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    uint2 raw;
    raw.x = *reinterpret_cast<const unsigned*>(&a);
    raw.y = *reinterpret_cast<const unsigned*>(&b);
    *reinterpret_cast<uint2*>(p) = raw;
}

// (Few rows: all it does is wait. The norms' weights are asked for before the wait for the previous kernel, and each sum has a place of its
// own: 5 rows of 1,024 in a chain of decode kernels, branch norm and norm, 3.0 -> 2.4 us.)
template <typename TM, typename TY, int NV>
__global__ void add_rmsnorm_vec_kernel(float* __restrict__ h, const TM* __restrict__ m,
                                       const float* __restrict__ post_w, const float* __restrict__ w,
                                       TY* __restrict__ y, const int32_t* __restrict__ rows, int H, float eps_post,
                                       float eps) {
    __shared__ float scratch[2][32];
    pdl_launch_dependents();
    const int i = blockIdx.x;
    float4 pw[NV], ww[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int c = threadIdx.x + k * blockDim.x;
        const bool there = c < (H >> 2);
        pw[k] = there && post_w != nullptr ? load4<float>(post_w + 4 * c) : make_float4(1.f, 1.f, 1.f, 1.f);
        ww[k] = there && w != nullptr ? load4<float>(w + 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    pdl_wait();
    const int64_t r = rows ? rows[i] : i;
    float* hr = h + r * H;
    const int chunks = H >> 2;
    float4 v[NV];
    float ss = 0.0f;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int c = threadIdx.x + k * blockDim.x;
        v[k] = c < chunks ? ld_written4(hr + 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (m != nullptr) {
        const TM* mr = m + r * H;
        float4 b[NV];
        float bs = 0.0f;
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const int c = threadIdx.x + k * blockDim.x;
            b[k] = c < chunks ? ld_written4(mr + 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
            bs += b[k].x * b[k].x + b[k].y * b[k].y + b[k].z * b[k].z + b[k].w * b[k].w;
        }
        float inv = 1.0f;
        if (post_w != nullptr) {
            bs = block_sum_first(bs, scratch[0]);
            inv = 1.0f / sqrtf(bs / (float)H + eps_post);
        }
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            const int c = threadIdx.x + k * blockDim.x;
            if (c >= chunks) continue;
            if (post_w != nullptr) {
                v[k].x += b[k].x * inv * pw[k].x;
                v[k].y += b[k].y * inv * pw[k].y;
                v[k].z += b[k].z * inv * pw[k].z;
                v[k].w += b[k].w * inv * pw[k].w;
            } else {
                v[k].x += b[k].x;
                v[k].y += b[k].y;
                v[k].z += b[k].z;
                v[k].w += b[k].w;
            }
            store4(hr + 4 * c, v[k]);
        }
    }
    if (w == nullptr) {
        if (y != nullptr) {
            TY* yc = y + (int64_t)i * H;
#pragma unroll
            for (int k = 0; k < NV; ++k) {
                const int c = threadIdx.x + k * blockDim.x;
                if (c < chunks) store4(yc + 4 * c, v[k]);
            }
        }
        return;
    }
#pragma unroll
    for (int k = 0; k < NV; ++k) ss += v[k].x * v[k].x + v[k].y * v[k].y + v[k].z * v[k].z + v[k].w * v[k].w;
    ss = block_sum_first(ss, scratch[1]);
    const float inv = 1.0f / sqrtf(ss / (float)H + eps);
    TY* yr = y + (int64_t)i * H;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int c = threadIdx.x + k * blockDim.x;
        if (c >= chunks) continue;
        store4(yr + 4 * c, make_float4(v[k].x * inv * ww[k].x, v[k].y * inv * ww[k].y, v[k].z * inv * ww[k].z, v[k].w * inv * ww[k].w));
    }
}

XS_API int xs_add_rmsnorm(float* h, const void* m, int m_dtype, const float* post_w, const float* w, void* y,
                          int y_dtype, const int32_t* rows, int n_rows, int H, float eps_post, float eps,
                          cudaStream_t stream) {
    if (n_rows == 0) return 0;
    XS_REQUIRE(n_rows > 0 && H > 0, "add_rmsnorm: %d rows of width %d", n_rows, H);
    XS_REQUIRE((size_t)H * 4 <= 200 * 1024, "add_rmsnorm: width %d does not fit shared memory (limit 51200)", H);
    XS_REQUIRE(w == nullptr || y != nullptr, "add_rmsnorm: a norm weight without an output");
    const bool aligned = H % 4 == 0 && ((uintptr_t)h % 16 == 0) && ((uintptr_t)m % 16 == 0) && ((uintptr_t)y % 16 == 0) &&
                         ((uintptr_t)w % 16 == 0) && ((uintptr_t)post_w % 16 == 0);
    if (aligned && H <= 16 * 1024) {
        const int chunks = H / 4;
        const int threads = chunks <= 128 ? 128 : chunks <= 1024 ? 256 : chunks <= 2048 ? 512 : 1024;
        const int nv = (chunks + threads - 1) / threads;
#define XS_VEC(TM, TY, NV)                                                                                          \
    xs_launch(add_rmsnorm_vec_kernel<TM, TY, NV>, dim3(n_rows), dim3(threads), 0, stream, h, (const TM*)m, post_w, \
              w, (TY*)y, rows, H, eps_post, eps)
#define XS_VEC_NV(TM, TY)                       \
    do {                                        \
        if (nv <= 1) XS_VEC(TM, TY, 1);         \
        else if (nv == 2) XS_VEC(TM, TY, 2);    \
        else XS_VEC(TM, TY, 4);                 \
    } while (0)
        XS_DISPATCH_DTYPE(m_dtype, TM, XS_DISPATCH_DTYPE(y_dtype, TY, XS_VEC_NV(TM, TY)));
#undef XS_VEC_NV
#undef XS_VEC
        XS_LAUNCH_CHECK("add_rmsnorm");
        return 0;
    }
    const size_t smem = (size_t)H * sizeof(float);
    const int threads = H >= 2048 ? 512 : 256;
#define XS_GO(TM, TY)                                                                                    \
    do {                                                                                                 \
        if (smem > 48 * 1024)                                                                            \
            cudaFuncSetAttribute(add_rmsnorm_kernel<TM, TY>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                 (int)smem);                                                             \
        xs_launch(add_rmsnorm_kernel<TM, TY>, dim3(n_rows), dim3(threads), smem, stream, h, (const TM*)m, \
                  post_w, w, (TY*)y, rows, H, eps_post, eps);                                            \
    } while (0)
    XS_DISPATCH_DTYPE(m_dtype, TM, XS_DISPATCH_DTYPE(y_dtype, TY, XS_GO(TM, TY)));
#undef XS_GO
    XS_LAUNCH_CHECK("add_rmsnorm");
    return 0;
}

// ----------------------------------------------------------------- SwiGLU act
// out[t, f] = silu(gate[t, f]) * up[t, f], silu(z) = z / (1 + exp(-z))
// (src/models/common/blocks.cpp:23-27; src/backend/cpu_ref/ops.cpp:242-247).
// Layout of a gate/up row: interleave 0: [F gate | F up]; interleave 8: blocks of 16 columns,
// 8 gate then the 8 up of the same f (how the stacked weight is ordered for the fused epilogue
// of the few-row product).
// ACT 1: the gate's activation is the tanh form of gelu instead, 0.5 g (1 + tanh(sqrt(2 / pi) (g + 0.044715 g^3))).
__device__ __forceinline__ float silu_f(float g) { return g / (1.0f + expf(-g)); }
// (0.5 (1 + tanh(a)) = 1 / (1 + exp(-2 a)): one exponential, as silu)
__device__ __forceinline__ float gelu_tanh_f(float g) { return g / (1.0f + expf(-1.5957691216057308f * (g + 0.044715f * g * g * g))); }
template <int ACT>
__device__ __forceinline__ float gate_act_f(float g) { return ACT == 1 ? gelu_tanh_f(g) : silu_f(g); }

template <typename T, int ACT>
__global__ void silu_mul_kernel(const T* __restrict__ gu, T* __restrict__ out, int64_t total, int F, int64_t ld,
                                int interleave) {
    pdl_launch_dependents();
    pdl_wait();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t t = i / F;
        const int f = (int)(i - t * F);
        const int64_t gi = interleave ? (int64_t)(f / interleave) * 2 * interleave + f % interleave : f;
        const int64_t ui = interleave ? gi + interleave : (int64_t)F + f;
        out[i] = from_f32<T>(gate_act_f<ACT>(to_f32(gu[t * ld + gi])) * to_f32(gu[t * ld + ui]));
    }
}

// 8 outputs a thread, 16-byte loads and stores; F a multiple of 8, rows 16-byte aligned.
template <int ACT>
__global__ void silu_mul_bf16x8_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out,
                                       int64_t total8, int F8, int64_t ld, int interleave) {
    pdl_launch_dependents();
    pdl_wait();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total8; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t t = i / F8;
        const int j = (int)(i - t * F8);
        const __nv_bfloat16* row = gu + t * ld;
        const uint4 g = *reinterpret_cast<const uint4*>(row + (interleave ? 16 * j : 8 * j));
        const uint4 u = *reinterpret_cast<const uint4*>(row + (interleave ? 16 * j + 8 : 8 * (int64_t)F8 + 8 * j));
        const __nv_bfloat162* gp = reinterpret_cast<const __nv_bfloat162*>(&g);
        const __nv_bfloat162* up = reinterpret_cast<const __nv_bfloat162*>(&u);
        uint4 o;
        __nv_bfloat162* op = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float2 gf = __bfloat1622float2(gp[k]), uf = __bfloat1622float2(up[k]);
            op[k] = __floats2bfloat162_rn(gate_act_f<ACT>(gf.x) * uf.x, gate_act_f<ACT>(gf.y) * uf.y);
        }
        *reinterpret_cast<uint4*>(out + t * 8 * (int64_t)F8 + 8 * j) = o;
    }
}

// act 0: silu(gate) * up; 1: gelu_tanh(gate) * up.
XS_API int xs_gated_act(const void* gu, void* out, int dtype, int T, int F, int64_t ld, int interleave, int act,
                        cudaStream_t stream) {
    if (T == 0) return 0;
    XS_REQUIRE(T > 0 && F > 0 && ld >= 2 * (int64_t)F, "gated_act: %d rows, %d columns, stride %lld", T, F, (long long)ld);
    XS_REQUIRE(interleave == 0 || (interleave == 8 && F % 8 == 0), "gated_act: interleave %d with %d columns", interleave, F);
    XS_REQUIRE(act == 0 || act == 1, "gated_act: activation code %d (0 silu, 1 gelu_tanh)", act);
    if (dtype == XS_BF16 && F % 8 == 0 && ld % 8 == 0 && (uintptr_t)gu % 16 == 0 && (uintptr_t)out % 16 == 0) {
        const int64_t total8 = (int64_t)T * (F / 8);
        const int blocks = (int)((total8 + 255) / 256 < 148 * 32 ? (total8 + 255) / 256 : 148 * 32);
        if (act == 1)
            xs_launch(silu_mul_bf16x8_kernel<1>, dim3(blocks), dim3(256), 0, stream, (const __nv_bfloat16*)gu, (__nv_bfloat16*)out,
                      total8, F / 8, ld, interleave);
        else
            xs_launch(silu_mul_bf16x8_kernel<0>, dim3(blocks), dim3(256), 0, stream, (const __nv_bfloat16*)gu, (__nv_bfloat16*)out,
                      total8, F / 8, ld, interleave);
        XS_LAUNCH_CHECK("gated_act");
        return 0;
    }
    const int64_t total = (int64_t)T * F;
    const int blocks = (int)((total + 255) / 256 < 148 * 16 ? (total + 255) / 256 : 148 * 16);
    XS_DISPATCH_DTYPE(dtype, TT, do {
        if (act == 1) xs_launch(silu_mul_kernel<TT, 1>, dim3(blocks), dim3(256), 0, stream, (const TT*)gu, (TT*)out, total, F, ld, interleave);
        else xs_launch(silu_mul_kernel<TT, 0>, dim3(blocks), dim3(256), 0, stream, (const TT*)gu, (TT*)out, total, F, ld, interleave);
    } while (0));
    XS_LAUNCH_CHECK("gated_act");
    return 0;
}

XS_API int xs_silu_mul(const void* gu, void* out, int dtype, int T, int F, int64_t ld, int interleave,
                       cudaStream_t stream) {
    return xs_gated_act(gu, out, dtype, T, F, ld, interleave, 0, stream);
}

// ------------------------------------------------------------ zero state rows
// state[slots[i], :] = 0 for a freshly opened sequence.
__global__ void zero_rows_kernel(uint8_t* __restrict__ base, const int32_t* __restrict__ slots, int64_t row_bytes) {
    uint8_t* row = base + (int64_t)slots[blockIdx.x] * row_bytes;
    for (int64_t i = threadIdx.x; i < row_bytes; i += blockDim.x) row[i] = 0;
}

XS_API int xs_zero_rows(void* base, const int32_t* slots, int n, int64_t row_bytes, cudaStream_t stream) {
    if (n == 0 || row_bytes == 0) return 0;
    zero_rows_kernel<<<n, 256, 0, stream>>>((uint8_t*)base, slots, row_bytes);
    XS_LAUNCH_CHECK("zero_rows");
    return 0;
}
