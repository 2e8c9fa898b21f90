// Paged causal attention in float32 for head sizes 64 and 128: the same sums in the same order as attention_generic.cu (which
// keeps the other head sizes), laid out for prompts and for single decoded tokens.
//
// A query at position p walks its keys in tiles of 32 that start at multiples of 32 of the key position; per tile the running maximum
// moves, the sums so far are scaled by exp(old - new), and the tile's terms are added: scores over the head's numbers in order, the
// denominator's 32 terms by a butterfly (16, 8, 4, 2, 1), the output's 32 terms in order.  Every kernel keeps that order, so a token's
// result is bit for bit the same as a prompt's last token, in a portion of a prompt, or decoded by itself.
//
// attn_f32_tile_kernel    64 queries of one request and one head a block, 128 threads with 4 queries x 4 keys (scores) and 4 queries x 8 or
//                         16 numbers (output) each, keys and values through two shared-memory buffers by cp.async.  Bound by the FMA
//                         pipes and the shared memory that feeds them (6 loads of 16 bytes for 32 FMAs).
// attn_f32_single_kernel  one token and head a block: all scores of up to 1024 keys at a time by 256 threads, then the output's chain over
//                         the keys, a number a thread, from value tiles that cp.async keeps ahead.  Bound by the chain's latency.
// Measured in whole steps of the 1B shape (32 heads on 8 of 64 numbers, 16 layers), against one warp per token and head: a prompt of 777
// tokens 33.7 -> 15.5 ms a step (attention 1290 -> about 150 us a layer), five requests of 300 to 900 tokens decoding 7.1 -> 2.3 ms.
#include "common.cuh"

namespace {

constexpr int kTileQ = 64, kTileK = 32;

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool live) {
    const int n = live ? 16 : 0;                       // nothing to read: the 16 bytes become zero
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ bool finite4(float4 v) {
    const float big = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
    return big <= 3.402823466e38f && v.x == v.x && v.y == v.y && v.z == v.z && v.w == v.w;
}

// The butterfly of warp_sum over 32 terms of which a thread holds c, c + 8, c + 16, c + 24 (c = its place among eight lanes).
__device__ __forceinline__ float sum32(const float (&p)[4]) {
    float v = (p[0] + p[2]) + (p[1] + p[3]);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <int D>
__global__ void __launch_bounds__(128)
attn_f32_tile_kernel(const float* __restrict__ q, int q_stride, const float* __restrict__ cache, const int* __restrict__ block_table,
                     int table_width, const int* __restrict__ tiles, int n_tiles, float* __restrict__ out, int out_stride, int heads,
                     int kv_heads, int page_size, int window, float scale) {
    pdl_trigger();
    pdl_wait();
    constexpr int LDK = D + 4, LDP = kTileK + 4, ND = D / 32;        // ND float4 of the output per thread and query
    extern __shared__ __align__(16) float smem_f[];
    float* Qs = smem_f;                                // [64][LDK]
    float* Ks = Qs + kTileQ * LDK;                     // [2][32][LDK]
    float* Vs = Ks + 2 * kTileK * LDK;                 // [2][32][D]
    float* Ps = Vs + 2 * kTileK * D;                   // [64][LDP]
    // the lists run from the shortest context to the longest: the longest start first
    const int* tile = tiles + 4 * (n_tiles - 1 - (int)blockIdx.y);
    const int row0 = tile[0], rows = tile[1], pos0 = tile[2], request = tile[3];
    const int h = blockIdx.x, hk = h / (heads / kv_heads);
    const int* table = block_table + (size_t)request * table_width;
    const int tid = threadIdx.x, cg = tid & 7, rg = tid >> 3;
    const size_t plane = (size_t)kv_heads * page_size * D, head_off = (size_t)hk * page_size * D;
    const int last = pos0 + rows - 1, first = window > 0 ? max(0, pos0 - window + 1) : 0;

    for (int i = tid; i < kTileQ * (D / 4); i += 128) {
        const int r = i / (D / 4), c = (i % (D / 4)) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < rows) v = *reinterpret_cast<const float4*>(q + (size_t)(row0 + r) * q_stride + (size_t)h * D + c);
        *reinterpret_cast<float4*>(Qs + r * LDK + c) = v;
    }
    auto fetch = [&](int k0, int buf) {                // four threads a key: its row of the key plane and of the value plane
        const int j = tid >> 2, key = k0 + j;
        const bool live = key >= first && key <= last;
        const size_t off = live ? (size_t)table[key / page_size] * 2 * plane + head_off + (size_t)(key % page_size) * D : 0;
#pragma unroll
        for (int i = 0; i < D / 16; ++i) {
            const int c = ((tid & 3) + 4 * i) * 4;
            cp_async16(Ks + ((size_t)buf * kTileK + j) * LDK + c, cache + off + c, live);
            cp_async16(Vs + ((size_t)buf * kTileK + j) * D + c, cache + off + plane + c, live);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float o[4][ND][4], m[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY; l[i] = 0.f;
#pragma unroll
        for (int n = 0; n < ND; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) o[i][n][e] = 0.f;
    }
    const int k_begin = first & ~(kTileK - 1);
    fetch(k_begin, 0);
    int buf = 0;
    for (int k0 = k_begin; k0 <= last; k0 += kTileK, buf ^= 1) {
        if (k0 + kTileK <= last) {
            fetch(k0 + kTileK, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        // values that are not finite must not reach a query that does not see them (0 * inf): looked for by the thread that fetched them
        bool odd = false;
#pragma unroll
        for (int i = 0; i < D / 16; ++i)
            odd |= !finite4(*reinterpret_cast<const float4*>(Vs + ((size_t)buf * kTileK + (tid >> 2)) * D + ((tid & 3) + 4 * i) * 4));
        odd = __syncthreads_or(odd);

        // scores: queries rg + 16 i, keys cg + 8 j
        const float* Kb = Ks + (size_t)buf * kTileK * LDK;
        float s[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 4
        for (int d = 0; d < D; d += 4) {
            float4 a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(Qs + (rg + 16 * i) * LDK + d);
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(Kb + (cg + 8 * j) * LDK + d);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    s[i][j] = fmaf(b[j].x, a[i].x, s[i][j]);
                    s[i][j] = fmaf(b[j].y, a[i].y, s[i][j]);
                    s[i][j] = fmaf(b[j].z, a[i].z, s[i][j]);
                    s[i][j] = fmaf(b[j].w, a[i].w, s[i][j]);
                }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int pos = pos0 + rg + 16 * i, lo = window > 0 ? max(0, pos - window + 1) : 0;
            float p[4], mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = k0 + cg + 8 * j;
                p[j] = key >= lo && key <= pos ? scale * s[i][j] : -INFINITY;
                mx = fmaxf(mx, p[j]);
            }
#pragma unroll
            for (int w = 4; w > 0; w >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
            const bool sees = k0 <= pos && k0 + kTileK > lo;              // the query sees a key of this tile
            const float m_new = fmaxf(m[i], mx), corr = sees ? expf(m[i] - m_new) : 1.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = k0 + cg + 8 * j;
                p[j] = key >= lo && key <= pos ? expf(p[j] - m_new) : 0.f;
                Ps[(rg + 16 * i) * LDP + cg + 8 * j] = p[j];
            }
            const float sum = sum32(p);
            if (sees) {
                l[i] = l[i] * corr + sum;
                m[i] = m_new;
            }
#pragma unroll
            for (int n = 0; n < ND; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) o[i][n][e] *= corr;
        }
        __syncwarp();                                  // a query's eight threads are in one warp, and only they read its row of Ps
        const float* Vb = Vs + (size_t)buf * kTileK * D + cg * 4;
        if (!odd) {
#pragma unroll 2
            for (int j = 0; j < kTileK; j += 4) {
                float4 p[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) p[i] = *reinterpret_cast<const float4*>(Ps + (rg + 16 * i) * LDP + j);
#pragma unroll
                for (int jj = 0; jj < 4; ++jj)
#pragma unroll
                    for (int n = 0; n < ND; ++n) {
                        const float4 v = *reinterpret_cast<const float4*>(Vb + (j + jj) * D + n * 32);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float pj = jj == 0 ? p[i].x : jj == 1 ? p[i].y : jj == 2 ? p[i].z : p[i].w;
                            o[i][n][0] = fmaf(pj, v.x, o[i][n][0]);
                            o[i][n][1] = fmaf(pj, v.y, o[i][n][1]);
                            o[i][n][2] = fmaf(pj, v.z, o[i][n][2]);
                            o[i][n][3] = fmaf(pj, v.w, o[i][n][3]);
                        }
                    }
            }
        } else {
            for (int j = 0; j < kTileK; ++j)
#pragma unroll
                for (int n = 0; n < ND; ++n) {
                    const float4 v = *reinterpret_cast<const float4*>(Vb + j * D + n * 32);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float pj = Ps[(rg + 16 * i) * LDP + j];
                        if (pj == 0.f) continue;
                        o[i][n][0] = fmaf(pj, v.x, o[i][n][0]);
                        o[i][n][1] = fmaf(pj, v.y, o[i][n][1]);
                        o[i][n][2] = fmaf(pj, v.z, o[i][n][2]);
                        o[i][n][3] = fmaf(pj, v.w, o[i][n][3]);
                    }
                }
        }
        __syncthreads();                               // the buffer is free for the tile after next
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = rg + 16 * i;
        if (r >= rows) continue;
        const float inv = 1.0f / l[i];
#pragma unroll
        for (int n = 0; n < ND; ++n)
            *reinterpret_cast<float4*>(out + (size_t)(row0 + r) * out_stride + (size_t)h * D + n * 32 + cg * 4) =
                make_float4(o[i][n][0] * inv, o[i][n][1] * inv, o[i][n][2] * inv, o[i][n][3] * inv);
    }
}

constexpr int kSingleThreads = 256, kSpan = 1024;      // keys whose scores lie in shared memory at a time

template <int D>
__global__ void __launch_bounds__(kSingleThreads)
attn_f32_single_kernel(const float* __restrict__ q, int q_stride, const float* __restrict__ cache, const int* __restrict__ block_table,
                       int table_width, const int* __restrict__ items, const int* __restrict__ token_request,
                       const int* __restrict__ positions, float* __restrict__ out, int out_stride, int heads, int kv_heads, int page_size,
                       int window, float scale) {
    pdl_trigger();
    pdl_wait();
    constexpr int kStages = 512 / D;                   // value tiles of 32 keys on their way or being used: 64 KiB
    extern __shared__ __align__(16) float smem_f[];
    float* Vs = smem_f;                                // [kStages][32][D]
    __shared__ __align__(16) float qs[D], p[kSpan];
    __shared__ float tile_max[kSpan / 32], tile_sum[kSpan / 32], tile_corr[kSpan / 32];
    const int t = items[blockIdx.y], h = blockIdx.x, hk = h / (heads / kv_heads);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int pos = positions[t], lo = window > 0 ? max(0, pos - window + 1) : 0;
    const int* table = block_table + (size_t)token_request[t] * table_width;
    const size_t plane = (size_t)kv_heads * page_size * D, head_off = (size_t)hk * page_size * D;
    auto row_of = [&](int key) { return (size_t)table[key / page_size] * 2 * plane + head_off + (size_t)(key % page_size) * D; };
    const int k_begin = lo & ~31, n_tiles = (pos - k_begin) / 32 + 1;
    auto fetch = [&](int i) {                          // value tile i of the walk; eight threads a key
        if (i < n_tiles) {
            const int j = tid >> 3, key = k_begin + 32 * i + j;
            const bool live = key >= lo && key <= pos;
            const size_t off = live ? row_of(key) + plane : 0;
#pragma unroll
            for (int c = 0; c < D / 32; ++c) {
                const int e = ((tid & 7) + 8 * c) * 4;
                cp_async16(Vs + ((size_t)(i % kStages) * 32 + j) * D + e, cache + off + e, live);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < kStages - 1; ++i) fetch(i);
    for (int i = tid; i < D; i += kSingleThreads) qs[i] = q[(size_t)t * q_stride + (size_t)h * D + i];
    __syncthreads();

    float m = -INFINITY, l = 0.f, acc = 0.f;           // m and l alike in all threads; acc: output number tid
    for (int span0 = 0; span0 < n_tiles; span0 += kSpan / 32) {
        const int span_tiles = min(kSpan / 32, n_tiles - span0), k0 = k_begin + span0 * 32;
        for (int i = warp; i < span_tiles; i += kSingleThreads / 32) {
            const int key = k0 + i * 32 + lane;
            float s = -INFINITY;
            if (key >= lo && key <= pos) {
                const float* k = cache + row_of(key);
                float4 kv[16];
                float dot = 0.f;
#pragma unroll
                for (int c0 = 0; c0 < D; c0 += 64) {
#pragma unroll
                    for (int c = 0; c < 16; ++c) kv[c] = *reinterpret_cast<const float4*>(k + c0 + 4 * c);
#pragma unroll
                    for (int c = 0; c < 16; ++c) {
                        const float4 qv = *reinterpret_cast<const float4*>(qs + c0 + 4 * c);
                        dot = fmaf(kv[c].x, qv.x, dot);
                        dot = fmaf(kv[c].y, qv.y, dot);
                        dot = fmaf(kv[c].z, qv.z, dot);
                        dot = fmaf(kv[c].w, qv.w, dot);
                    }
                }
                s = scale * dot;
            }
            p[i * 32 + lane] = s;
            const float mx = warp_max(s);
            if (lane == 0) tile_max[i] = mx;
        }
        __syncthreads();
        for (int i = warp; i < span_tiles; i += kSingleThreads / 32) {
            float before = lane < i ? tile_max[lane] : -INFINITY;         // (a span has 32 tiles)
            before = fmaxf(m, warp_max(before));
            const float m_new = fmaxf(before, tile_max[i]);
            const int key = k0 + i * 32 + lane;
            const float e = key >= lo && key <= pos ? expf(p[i * 32 + lane] - m_new) : 0.f;
            p[i * 32 + lane] = e;
            const float sum = warp_sum(e);
            if (lane == 0) {
                tile_sum[i] = sum;
                tile_corr[i] = expf(before - m_new);
            }
        }
        for (int i = 0; i < span_tiles; ++i) m = fmaxf(m, tile_max[i]);
        for (int i = 0; i < span_tiles; ++i) {
            fetch(span0 + i + kStages - 1);
            asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
            __syncthreads();                           // tile span0 + i has landed for all; (first round: the span's p are written)
            const float corr = tile_corr[i];
            l = l * corr + tile_sum[i];
            if (tid < D) {
                acc *= corr;
                const float* v = Vs + (size_t)((span0 + i) % kStages) * 32 * D + tid;
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    const float4 pj = *reinterpret_cast<const float4*>(p + i * 32 + j);
                    if (pj.x != 0.f) acc = fmaf(pj.x, v[j * D], acc);
                    if (pj.y != 0.f) acc = fmaf(pj.y, v[(j + 1) * D], acc);
                    if (pj.z != 0.f) acc = fmaf(pj.z, v[(j + 2) * D], acc);
                    if (pj.w != 0.f) acc = fmaf(pj.w, v[(j + 3) * D], acc);
                }
            }
            __syncthreads();                           // the stage may be refilled (and, after the last tile, p)
        }
    }
    if (tid < D) out[(size_t)t * out_stride + (size_t)h * D + tid] = acc * (1.0f / l);
}

template <int D> size_t tile_smem() { return sizeof(float) * (kTileQ * (D + 4) + 2 * kTileK * (D + 4) + 2 * kTileK * D + kTileQ * (kTileK + 4)); }

template <typename Kern>
int set_smem(Kern kern, size_t bytes, const char* name) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) LLM_FAIL(-2, "%s: cudaFuncSetAttribute: %s", name, cudaGetErrorString(e));
    return 0;
}

int check(int heads, int kv_heads, int head_dim, const char* name) {
    if (head_dim != 64 && head_dim != 128) LLM_FAIL(-1, "%s: head_dim %d is not 64 or 128", name, head_dim);
    if (kv_heads <= 0 || heads <= 0 || heads % kv_heads) LLM_FAIL(-1, "%s: heads %d is not a multiple of kv_heads %d", name, heads, kv_heads);
    return 0;
}

}  // namespace

LLM_API int llm_attention_f32_supported(int heads, int kv_heads, int head_dim) {
    return (head_dim == 64 || head_dim == 128) && kv_heads > 0 && heads % kv_heads == 0;
}

// tiles: [n_tiles][4] = first token row, rows (at most 64), position of the first row, request; consecutive positions of one request.
LLM_API int llm_attention_f32_tiles(const float* q, int q_stride, const float* cache, const int* block_table, int table_width,
                                    const int* tiles, int n_tiles, float* out, int out_stride, int heads, int kv_heads, int head_dim,
                                    int page_size, int window, float scale, cudaStream_t stream) {
    if (n_tiles == 0) return 0;
    if (int rc = check(heads, kv_heads, head_dim, "attention_f32_tiles")) return rc;
    if (n_tiles > 65535) LLM_FAIL(-1, "attention_f32_tiles: %d tiles are too many for one launch", n_tiles);
    const dim3 grid(heads, n_tiles);
    auto go = [&](auto kern, size_t smem) {
        if (int rc = set_smem(kern, smem, "attention_f32_tiles")) return rc;
        llm_launch(kern, grid, 128, smem, stream, q, q_stride, cache, block_table, table_width, tiles, n_tiles, out, out_stride, heads,
                   kv_heads, page_size, window, scale);
        LLM_CHECK_LAUNCH("attention_f32_tiles");
        return 0;
    };
    return head_dim == 64 ? go(attn_f32_tile_kernel<64>, tile_smem<64>()) : go(attn_f32_tile_kernel<128>, tile_smem<128>());
}

// items: the token rows of single decoded tokens.
LLM_API int llm_attention_f32_single(const float* q, int q_stride, const float* cache, const int* block_table, int table_width,
                                     const int* items, int n_items, const int* token_request, const int* positions, float* out,
                                     int out_stride, int heads, int kv_heads, int head_dim, int page_size, int window, float scale,
                                     cudaStream_t stream) {
    if (n_items == 0) return 0;
    if (int rc = check(heads, kv_heads, head_dim, "attention_f32_single")) return rc;
    if (n_items > 65535) LLM_FAIL(-1, "attention_f32_single: %d tokens are too many for one launch", n_items);
    const dim3 grid(heads, n_items);
    auto go = [&](auto kern) {
        if (int rc = set_smem(kern, 64 * 1024, "attention_f32_single")) return rc;
        llm_launch(kern, grid, kSingleThreads, 64 * 1024, stream, q, q_stride, cache, block_table, table_width, items, token_request,
                   positions, out, out_stride, heads, kv_heads, page_size, window, scale);
        LLM_CHECK_LAUNCH("attention_f32_single");
        return 0;
    };
    return head_dim == 64 ? go(attn_f32_single_kernel<64>) : go(attn_f32_single_kernel<128>);
}

LLM_TRACE_EXPORT(attention_f32)
