// Norms that sit on a branch's output, and the clamped gated activation.
//
// llm_norm_add:     residual[t] (+)= branch[t] * rsqrt(mean(branch[t]^2) + eps) * weight   (float32 statistics and sum),
//                   and optionally a copy of the new residual row in the engine's type, which the next sub-layer reads.
//                   One block per row, the row held in registers between the two passes, sums in a fixed order.
//                   With a second gain the new residual row is normed as well, into rows of the engine's type: the norm
//                   in front of the next sub-layer of a design that has norms on both sides of its sub-layers.
//                   A branch may arrive as the k-split parts of a product (few rows only): they are added in split order as they are read
//                   and the sum is rounded to the type the product has, so a row does not depend on who adds its parts.
// llm_rmsnorm_rows: out[t] = in[t] * rsqrt(mean(in[t]^2) + eps) * weight for rows of the engine's type with strides of their
//                   own (some columns of a wider product), float32 statistics.
// llm_glu_clamped:  act = g * sigmoid(slope * g) * (u + 1) with g = min(gate, limit), u = clamp(up, -limit, limit),
//                   from one [T, 2 * inner] row of gate columns followed by up columns.
// llm_glu_act:      act = f(gate) * up from such a row, f = silu (0) or the tanh form of gelu (1).
#include "common.cuh"

namespace {

constexpr int kNormThreads = 256;
constexpr int kNormPer = 8;          // elements a thread holds: rows up to 2048 * ... are walked in rounds of 2048

template <typename TB, typename TW, typename TC>
__global__ void __launch_bounds__(kNormThreads)
norm_add_kernel(float* __restrict__ residual, const TB* __restrict__ branch, const TW* __restrict__ weight,
                TC* __restrict__ cast, int width, float eps, int accumulate, const TW* __restrict__ next_weight,
                TC* __restrict__ next_out) {
    pdl_trigger();
    pdl_wait();
    __shared__ float red[32];
    const size_t row = blockIdx.x;
    const TB* b = branch + row * width;
    float* res = residual + row * width;
    float ss = 0.f;
    float held[kNormPer];
    // first pass: sum of squares (the first kNormPer rounds of the row stay in registers)
#pragma unroll
    for (int j = 0; j < kNormPer; ++j) {
        const int i = threadIdx.x + j * kNormThreads;
        held[j] = i < width ? to_f32(b[i]) : 0.f;
        ss += held[j] * held[j];
    }
    for (int i = threadIdx.x + kNormPer * kNormThreads; i < width; i += kNormThreads) {
        const float v = to_f32(b[i]);
        ss += v * v;
    }
    const float total = block_sum(ss, red);
    const float inv = 1.0f / sqrtf(total / (float)width + eps);
#pragma unroll
    for (int j = 0; j < kNormPer; ++j) {
        const int i = threadIdx.x + j * kNormThreads;
        if (i < width) {
            float y = held[j] * inv * to_f32(weight[i]);
            if (accumulate) y += res[i];
            res[i] = y;
            held[j] = y;
            if (cast) cast[row * width + i] = from_f32<TC>(y);
        }
    }
    float ss2 = 0.f;
    for (int i = threadIdx.x + kNormPer * kNormThreads; i < width; i += kNormThreads) {
        float y = to_f32(b[i]) * inv * to_f32(weight[i]);
        if (accumulate) y += res[i];
        res[i] = y;
        ss2 += y * y;
        if (cast) cast[row * width + i] = from_f32<TC>(y);
    }
    if (!next_out) return;                 // the same for the whole block
    // the norm of the new row (what was held is zero beyond the row's end)
#pragma unroll
    for (int j = 0; j < kNormPer; ++j) ss2 += held[j] * held[j];
    const float inv2 = 1.0f / sqrtf(block_sum(ss2, red) / (float)width + eps);
#pragma unroll
    for (int j = 0; j < kNormPer; ++j) {
        const int i = threadIdx.x + j * kNormThreads;
        if (i < width) next_out[row * width + i] = from_f32<TC>(held[j] * inv2 * to_f32(next_weight[i]));
    }
    for (int i = threadIdx.x + kNormPer * kNormThreads; i < width; i += kNormThreads)
        next_out[row * width + i] = from_f32<TC>(res[i] * inv2 * to_f32(next_weight[i]));
}

// The same for few rows, when a row's time is what counts and not the rows in flight: 1024 threads a row, and everything a thread
// will need is asked for at once (the gains even before the kernel ahead has finished) instead of in three dependent rounds of twelve loads.
// The sums are those of the kernel above: 256 threads add the same numbers in the same order, out of shared memory.  One row of 3072 numbers took
// 8.3 us there.  With the other kernels of few rows (token shift 21 us, head norms 11.7, wkv decays 13) and the product's parts read here instead of
// added by a kernel ahead, a prompt of 1111 tokens and eight decode steps at the Rodapel 3B sizes went from 7.41 to 6.77 ms.
constexpr int kFewThreads = 1024, kFewPer = 4, kFewWidth = kFewThreads * kFewPer;
constexpr int kFewRows = 148;        // a block of 1024 threads to an SM

// From which width on the wide block is the faster one, in us a call of the other kernel and of this one: bfloat16 branch without a second norm 2.3 and
// 2.1 (768 numbers, 8 rows), 5.5 and 2.6 (3072, 148 rows), but 1.8 and 2.0 (512, one row); float32 2.4 and 2.3 (1536), 3.6 and 2.5 (3072, 148 rows), but
// 1.8 and 2.2 (512); with a second norm 4.4 and 3.5 (3072, 148 rows), 3.0 and 3.0 (1536), but 2.4 and 2.8 (512, 37 rows).
int few_width(int branch_dtype, bool second) { return second ? 2048 : branch_dtype == LLM_BF16 ? 768 : 1536; }

template <typename TB, typename TW, typename TC>
__global__ void __launch_bounds__(kFewThreads)
norm_add_few_kernel(float* __restrict__ residual, const TB* __restrict__ branch, const TW* __restrict__ weight, TC* __restrict__ cast,
                    int width, float eps, int accumulate, const TW* __restrict__ next_weight, TC* __restrict__ next_out, int splits,
                    size_t split_stride) {
    pdl_trigger();
    extern __shared__ float row_buf[];       // width floats
    __shared__ float red[kNormThreads / 32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const size_t row = blockIdx.x;
    float b[kFewPer], w[kFewPer], nw[kFewPer], r[kFewPer];
#pragma unroll
    for (int j = 0; j < kFewPer; ++j) {
        const int i = tid + j * kFewThreads;
        w[j] = i < width ? to_f32(weight[i]) : 0.f;
        nw[j] = next_out && i < width ? to_f32(next_weight[i]) : 0.f;
    }
    pdl_wait();
#pragma unroll
    for (int j = 0; j < kFewPer; ++j) {
        const int i = tid + j * kFewThreads;
        r[j] = accumulate && i < width ? residual[row * width + i] : 0.f;
        if (splits == 0) b[j] = i < width ? to_f32(branch[row * width + i]) : 0.f;
    }
    if (splits > 0) {
        const float* parts = reinterpret_cast<const float*>(branch) + row * width;
        float e[kFewPer][kMaxParts];
#pragma unroll
        for (int j = 0; j < kFewPer; ++j)
#pragma unroll
            for (int k = 0; k < kMaxParts; ++k)
                if (k < splits && tid + j * kFewThreads < width) e[j][k] = parts[k * split_stride + tid + j * kFewThreads];
#pragma unroll
        for (int j = 0; j < kFewPer; ++j) {
            b[j] = tid + j * kFewThreads < width ? e[j][0] : 0.f;
#pragma unroll
            for (int k = 1; k < kMaxParts; ++k)
                if (k < splits && tid + j * kFewThreads < width) b[j] += e[j][k];
            b[j] = to_f32(from_f32<TB>(b[j]));             // as a kernel that adds the parts into rows of this type leaves them
        }
    }
    // sums of squares as kNormThreads threads take them: element tid + kNormThreads * j, from round `from` to the row's end, then from 0
    auto square_sum = [&](int from) {
        float ss = 0.f;
        if (warp < kNormThreads / 32) {
            for (int i = tid + from * kNormThreads; i < width; i += kNormThreads) ss += row_buf[i] * row_buf[i];
            for (int i = tid; i < width && i < from * kNormThreads; i += kNormThreads) ss += row_buf[i] * row_buf[i];
            ss = warp_sum(ss);
            if (lane == 0) red[warp] = ss;
        }
        __syncthreads();
        return warp_sum(lane < kNormThreads / 32 ? red[lane] : 0.f);
    };
#pragma unroll
    for (int j = 0; j < kFewPer; ++j)
        if (tid + j * kFewThreads < width) row_buf[tid + j * kFewThreads] = b[j];
    __syncthreads();
    const float inv = 1.0f / sqrtf(square_sum(0) / (float)width + eps);
#pragma unroll
    for (int j = 0; j < kFewPer; ++j) {
        const int i = tid + j * kFewThreads;
        if (i < width) {
            const float scaled = b[j] * inv;
            const float y = accumulate ? fmaf(scaled, w[j], r[j]) : scaled * w[j];
            b[j] = y;
            residual[row * width + i] = y;
            if (cast) cast[row * width + i] = from_f32<TC>(y);
            if (next_out) row_buf[i] = y;
        }
    }
    if (!next_out) return;                 // the same for the whole block
    __syncthreads();
    const float inv2 = 1.0f / sqrtf(square_sum(kNormPer) / (float)width + eps);
#pragma unroll
    for (int j = 0; j < kFewPer; ++j) {
        const int i = tid + j * kFewThreads;
        if (i < width) next_out[row * width + i] = from_f32<TC>(b[j] * inv2 * nw[j]);
    }
}

template <typename T>
__global__ void __launch_bounds__(128)
rmsnorm_rows_kernel(const T* __restrict__ in, long long ld_in, T* __restrict__ out, long long ld_out, const float* __restrict__ weight,
                    int width, float eps) {
    pdl_trigger();
    pdl_wait();
    __shared__ float red[32];
    const T* x = in + (size_t)blockIdx.x * ld_in;
    T* y = out + (size_t)blockIdx.x * ld_out;
    float ss = 0.f;
    for (int i = threadIdx.x; i < width; i += blockDim.x) { const float v = to_f32(x[i]); ss += v * v; }
    const float inv = 1.0f / sqrtf(block_sum(ss, red) / (float)width + eps);
    for (int i = threadIdx.x; i < width; i += blockDim.x) y[i] = from_f32<T>(to_f32(x[i]) * inv * weight[i]);
}

__device__ __forceinline__ float gelu_tanh_f(float z) {
    return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}

template <typename T>
__global__ void glu_act_kernel(const T* __restrict__ gu, T* __restrict__ act, int tokens, int inner, int kind) {
    pdl_trigger();
    pdl_wait();
    const size_t n = (size_t)tokens * inner;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const size_t t = i / inner, c = i % inner;
        const float g = to_f32(gu[t * 2 * inner + c]), u = to_f32(gu[t * 2 * inner + inner + c]);
        act[i] = from_f32<T>((kind == 1 ? gelu_tanh_f(g) : g / (1.0f + expf(-g))) * u);
    }
}

__device__ __forceinline__ float glu_clamped(float g, float u, float limit, float slope) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit);
    return g / (1.0f + expf(-slope * g)) * (u + 1.0f);
}

template <typename T>
__global__ void glu_clamped_kernel(const T* __restrict__ gu, T* __restrict__ act, int tokens, int inner, float limit, float slope) {
    pdl_trigger();
    pdl_wait();
    const size_t n = (size_t)tokens * inner;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const size_t t = i / inner, c = i % inner;
        act[i] = from_f32<T>(glu_clamped(to_f32(gu[t * 2 * inner + c]), to_f32(gu[t * 2 * inner + inner + c]), limit, slope));
    }
}

// Eight neighbouring numbers a thread, for rows and halves of rows that start on 16 bytes, and a row of blocks a token (the kernel above divides in
// 64 bits for every number and loads one at a time).  us in bfloat16, above and here: 1111 rows of 8192 26.4 and 11.7, 37 of 8192 2.2 and 1.8, 148
// of 2048 2.2 and 2.0, but 16 of 8192 1.7 and 1.8, 8 of 2048 1.3 and 1.8.
constexpr size_t kGluVec = 200000;         // numbers from which on there are threads enough for all SMs

template <typename T>
__global__ void __launch_bounds__(256)
glu_clamped_vec_kernel(const T* __restrict__ gu, T* __restrict__ act, int tokens, int inner, float limit, float slope) {
    pdl_trigger();
    pdl_wait();
    constexpr int kPieces = sizeof(T) / 2;           // 16-byte loads of eight numbers
    for (int t = blockIdx.y; t < tokens; t += gridDim.y) {
        const T* gr = gu + (size_t)t * 2 * inner;
        T* ar = act + (size_t)t * inner;
        for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < inner / 8; c += gridDim.x * blockDim.x) {
            uint4 g[kPieces], u[kPieces], a[kPieces];
#pragma unroll
            for (int e = 0; e < kPieces; ++e) {
                g[e] = reinterpret_cast<const uint4*>(gr + 8 * c)[e];
                u[e] = reinterpret_cast<const uint4*>(gr + inner + 8 * c)[e];
            }
            const T *gp = reinterpret_cast<const T*>(g), *up = reinterpret_cast<const T*>(u);
            T* ap = reinterpret_cast<T*>(a);
#pragma unroll
            for (int e = 0; e < 8; ++e) ap[e] = from_f32<T>(glu_clamped(to_f32(gp[e]), to_f32(up[e]), limit, slope));
#pragma unroll
            for (int e = 0; e < kPieces; ++e) reinterpret_cast<uint4*>(ar + 8 * c)[e] = a[e];
        }
    }
}

}  // namespace

// Rows up to which llm_norm_add takes the parts of a product (width up to 4096).
LLM_API int llm_norm_add_few_rows(int width) { return width <= kFewWidth ? kFewRows : 0; }

// branch [tokens, width] of `branch_dtype`; weight float32 or bfloat16 (`weight_dtype`); cast: null or [tokens, width] of
// `cast_dtype`.  accumulate == 0 writes the normed row instead of adding it (an embedding's norm).  splits > 0: `branch` is float32 parts
// [splits][tokens][width], `split_stride` numbers apart, of rows of `branch_dtype` (at most llm_norm_add_few_rows() rows, of at most 4096 numbers).
LLM_API int llm_norm_add(float* residual, const void* branch, int branch_dtype, const void* weight, int weight_dtype,
                         void* cast, int cast_dtype, int tokens, int width, float eps, int accumulate, const void* next_weight,
                         void* next_out, int splits, long long split_stride, cudaStream_t stream) {
    if (tokens == 0) return 0;
    if (width <= 0) LLM_FAIL(-1, "norm_add: width %d", width);
    const bool few = tokens <= kFewRows && width <= kFewWidth;
    if (splits < 0 || splits > kMaxParts || (splits > 0 && !few))
        LLM_FAIL(-1, "norm_add: %d parts of %d rows of %d numbers are not taken", splits, tokens, width);
    if ((next_weight == nullptr) != (next_out == nullptr)) LLM_FAIL(-1, "norm_add: the second norm needs a gain and a place for its rows");
    return llm_dispatch_dtype(branch_dtype, [&](auto tb) {
        using TB = decltype(tb);
        return llm_dispatch_dtype(weight_dtype, [&](auto tw) {
            using TW = decltype(tw);
            return llm_dispatch_dtype(cast || next_out ? cast_dtype : LLM_BF16, [&](auto tc) {
                using TC = decltype(tc);
                if (splits > 0 || (few && width >= few_width(branch_dtype, next_out != nullptr)))
                    llm_launch(norm_add_few_kernel<TB, TW, TC>, (unsigned)tokens, kFewThreads, sizeof(float) * width, stream, residual,
                               (const TB*)branch, (const TW*)weight, (TC*)cast, width, eps, accumulate, (const TW*)next_weight, (TC*)next_out,
                               splits, (size_t)split_stride);
                else
                    llm_launch(norm_add_kernel<TB, TW, TC>, (unsigned)tokens, kNormThreads, 0, stream, residual, (const TB*)branch,
                               (const TW*)weight, (TC*)cast, width, eps, accumulate, (const TW*)next_weight, (TC*)next_out);
                LLM_CHECK_LAUNCH("norm_add");
                return 0;
            });
        });
    });
}

// in / out: rows of `dtype` with strides ld_in / ld_out (in elements); weight float32 [width].
LLM_API int llm_rmsnorm_rows(const void* in, long long ld_in, void* out, long long ld_out, const float* weight, int dtype, int tokens,
                             int width, float eps, cudaStream_t stream) {
    if (tokens == 0) return 0;
    if (width <= 0) LLM_FAIL(-1, "rmsnorm_rows: width %d", width);
    return llm_dispatch_dtype(dtype, [&](auto tag) {
        using T = decltype(tag);
        llm_launch(rmsnorm_rows_kernel<T>, (unsigned)tokens, 128, 0, stream, (const T*)in, ld_in, (T*)out, ld_out, weight, width, eps);
        LLM_CHECK_LAUNCH("rmsnorm_rows");
        return 0;
    });
}

// kind: 0 silu, 1 the tanh form of gelu.
LLM_API int llm_glu_act(const void* gu, void* act, int dtype, int tokens, int inner, int kind, cudaStream_t stream) {
    if (tokens == 0 || inner == 0) return 0;
    if (kind != 0 && kind != 1) LLM_FAIL(-1, "glu_act: activation code %d is not known", kind);
    const size_t n = (size_t)tokens * inner;
    const unsigned blocks = (unsigned)((n + 255) / 256 < 148 * 16 ? (n + 255) / 256 : 148 * 16);
    return llm_dispatch_dtype(dtype, [&](auto tag) {
        using T = decltype(tag);
        llm_launch(glu_act_kernel<T>, blocks, 256, 0, stream, (const T*)gu, (T*)act, tokens, inner, kind);
        LLM_CHECK_LAUNCH("glu_act");
        return 0;
    });
}

LLM_API int llm_glu_clamped(const void* gu, void* act, int dtype, int tokens, int inner, float limit, float slope,
                            cudaStream_t stream) {
    if (tokens == 0 || inner == 0) return 0;
    const size_t n = (size_t)tokens * inner;
    const bool vec = inner % 8 == 0 && !(((uintptr_t)gu | (uintptr_t)act) & 15) && n >= kGluVec;
    const int work = inner / 8, threads = vec && work < 256 ? (work + 31) / 32 * 32 : 256;
    const dim3 grid = vec ? dim3((work + threads - 1) / threads, tokens < 65535 ? tokens : 65535)
                          : dim3((unsigned)((n + 255) / 256 < 148 * 16 ? (n + 255) / 256 : 148 * 16));
    return llm_dispatch_dtype(dtype, [&](auto tag) {
        using T = decltype(tag);
        llm_launch(vec ? glu_clamped_vec_kernel<T> : glu_clamped_kernel<T>, grid, threads, 0, stream, (const T*)gu, (T*)act, tokens, inner, limit, slope);
        LLM_CHECK_LAUNCH("glu_clamped");
        return 0;
    });
}

LLM_TRACE_EXPORT(branch_norm)
