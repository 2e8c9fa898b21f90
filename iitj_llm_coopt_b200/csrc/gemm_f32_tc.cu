// float32 matrix products on the fifth-generation tensor cores: y = x . W^T with x [T, K] and W [N, K] row-major, float32
// in and out, at float32 precision.  Every factor is taken apart into three bfloat16 pieces that add up to it exactly,
//
//     v = hi + mid + lo,   hi = v cut to 8 significant bits,  mid = the rest rounded to 8 bits,  lo = what then remains,
//
// and the product is the sum of the six piece products that reach 2^-24 of it (hi.hi; hi.mid, mid.hi; mid.mid, hi.lo, lo.hi),
// accumulated in float32.  The tensor cores cut a sum off where they add to it instead of rounding it, which would cost
// precision along a long k range; therefore the large piece product (hi.hi) stays in tensor memory for 128 k at a time (eight
// instructions), and these chunks are added in registers, rounded to nearest.  The five small products (2^-8 of the sum; lo.mid
// rides along) have accumulators of their own for a whole segment of the k range.  Relative error (2-norm, against 64 bits, normal factors) at
// K = 128 / 512 / 2048 / 8192: 1.2e-7 / 1.3e-7 / 1.5e-7 / 1.9e-7; a chain of fused multiply-adds has 2.0e-7 / 4.0e-7 / 8.0e-7 / 1.6e-6.
// Factors of one sign, whose sums shrink with every cut: K = 64 / 256 / 2048 0.9e-7 / 1.8e-7 / 1.8e-7 against 1.2e-7 / 2.5e-7 / 6.9e-7;
// a first chunk of 128 k was as far off as the chain up to K = 132 (1.81e-7 against 1.75e-7 at 128), so K up to 192 has chunks of 64.
// Numbers below 2^-110 lose bits: the last of their pieces lie below the smallest bfloat16 number, 2^-133.
//
// Order of a sum: chunks of 128 k (64 up to K = 192) in order, the small products of a segment with the last chunk of the segment.  Segments
// depend on K alone (an eighth of it, at least 256), so an output element is the same whatever else is in the call and
// however the call is cut into tiles and blocks.
//
// One block owns 128 rows of W (SwiGLU: 64 gate rows and the 64 up rows of the same features) and a tile of 16 to 80 tokens:
//   loader      W in boxes of 32 k (128 bytes a row, 128-byte swizzle) by TMA, requested before the kernel ahead has finished
//   converters  two groups of four warps, a row a thread: 32 floats a step and group from shared memory, three pieces, into tensor memory as the A operand
//               (the weights' pieces then cost the product no shared-memory bandwidth)
//   x           split_planes_kernel lays the pieces out once and TMA loads them.  (Taking x apart in every block costs a proxy fence
//               a step on top of the work: products of few tokens took 2300 clocks a step that way.)
//   issuers     two warps, one for the large and one for the small products: sixteen tcgen05.mma a step of 64 k
//   epilogue    four or eight warps, a row a thread: chunks out of tensor memory, sums in registers
// A step's barriers (a wait takes 200 clocks even when there is nothing to wait for, a commit 100) cost the issuer and the converters
// about 1000 clocks whatever the tile, as much as the products of 80 tokens take: hence steps of 64 k and not fewer, and two issuers.
// Products with few tiles share the k range out over a cluster of blocks (segments whole): every block keeps the sums of its
// chunks in shared memory, and the blocks then add all chunks of their part of the tile in order, over distributed shared memory.
//
// What bounds it: a decode step the HBM bytes of W, a prompt the tensor cores at seven bfloat16 products per float32 product (six of
// them of use: 278 TFLOP/s of the measured bf16 rate) and the barriers above.  Measured with the planes, cold weights, against the
// product on the CUDA cores (gemm_f32.cu): 5 tokens, 2048 x 2048 195 -> 10 us, 2048 x 8192 770 -> 28 us; one token, 128256 x 2048
// 1006 -> 172 us (6.1 TB/s); 777 tokens, 2048 x 2048 256 -> 69 us, 2048 x 8192 993 -> 214 us (122 TFLOP/s), SwiGLU 8192 x 2048 1483 ->
// 356 us (146 TFLOP/s; 331 us before boxes were handed back after the vote and the small products had one shape).
//
// Listed form (llm_gemm_f32_tc_listed): the rows were sorted by weight matrix on the device (the experts of a routed feed-forward);
// a block takes its tile from the list, blocks beyond the list's count leave at once.
//
// Infinities and NaNs arrive through hi.hi as they would in a plain product (a NaN gets its quiet bit in hi first); the small products,
// which then hold inf - inf, are left out when they are not finite.  Waits are bounded: a wait that runs out records a code in the status word of the bfloat16 product
// (11 producer, 12 issuer, 13 epilogue, 14 converter), and the block falls through to its teardown.
#include "tcgen05_common.cuh"

LLM_API int llm_gemm_grouped_tile_rows();      // gemm_grouped.cu

namespace {

typedef __nv_bfloat16 bf16;

constexpr int kRows = 128;               // rows of W per block (UMMA M)
constexpr int kStepK = 64;               // k of a step: two boxes of W of 32 float32 a row
constexpr int kBoxBytes = kRows * 32 * 4;
constexpr int kChunkSteps = 2;           // steps whose hi.hi products stay in one accumulator ...
constexpr int kShortSteps = 3;           // ... but one where the k range has at most so many
// Ring stages; of W: boxes, an even number, so that a stage is always read by the same group of converters.  (Boxes land in any
// order: a group that shared a stage could come to wait for the stage's second box before the first, the other group's, had landed,
// and a wait by parity that is two phases early passes at once.)
constexpr int kMaxW = 12, kMaxX = 4;
constexpr int kACols = 96;               // tensor-memory columns of the A pieces of one step
constexpr int kMaxA = 4;                 // steps whose A pieces lie in tensor memory at a time
constexpr int kSmallTokens = 16;         // up to here the smaller kernel
constexpr int kListedRows = 64;          // rows of a listed tile, at most (gemm_grouped.cu)
constexpr int kMaxTile = 80;             // tokens of a tile: 4 x 80 accumulator columns and two slots of A fill tensor memory

struct Args {
    float* out;
    int* status;
    int n, ldc, tokens, swiglu;          // swiglu: W holds gate rows, then up rows
    // listed form (tiles != null): rows sorted by group beforehand, a weight matrix each (llm_moe_plan writes the list)
    const int* tiles;                    // tiles[0] = count, entry i at tiles[4 + 4 * i] = (group, first row, rows, -)
    int clamped;                         // the gate's form: 0 silu(w g) * (w u), 1 clamped
    float limit, slope;
    const float* row_scale;              // w of form 0, one per row (null: 1)
    int steps, seg_steps, segs;          // steps of 64 k; steps of a segment (a multiple of 2); segments
    int cluster;                         // blocks that share a tile's k range (a divisor of segs)
    int tt, t_tiles;                     // tokens of a tile (a multiple of 16); token tiles
    int w_stages, x_stages, a_slots;
    int tmem_cols;
    int ring_bytes, x_bytes;             // shared memory: W ring | x pieces | chunk sums (cluster > 1)
    int sum_cols;                        // the smaller kernel: tokens whose chunk sums are kept (cluster > 1)
};

__device__ __forceinline__ void give_up_f32(const Args& a, int code) { atomicCAS(a.status, 0, (code << 16) | (int)(blockIdx.x & 0xffff)); }

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}

// Two neighbouring numbers taken apart; each result word holds both numbers' pieces (the first in the low half).
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    const uint32_t ua = __float_as_uint(a), ub = __float_as_uint(b);
    hi = __byte_perm(ua, ub, 0x7632);
    const float ra = a - __uint_as_float(ua & 0xffff0000u), rb = b - __uint_as_float(ub & 0xffff0000u);      // exact
    const __nv_bfloat162 m = __floats2bfloat162_rn(ra, rb);
    mid = *reinterpret_cast<const uint32_t*>(&m);
    const float la = ra - __uint_as_float(mid << 16), lb = rb - __uint_as_float(mid & 0xffff0000u);          // exact, 8 bits
    lo = __byte_perm(__float_as_uint(la), __float_as_uint(lb), 0x7632);
}

// False only if no number behind the pieces `lo` (several pairs' words, or-ed) is infinite or a NaN: those have a NaN there.
__device__ __forceinline__ bool maybe_not_finite(uint32_t lo) { return (lo & 0x7f80u) == 0x7f80u || (lo & 0x7f800000u) == 0x7f800000u; }
// The quiet bits of those of two numbers that are NaNs, where hi has them: a NaN whose payload lies in the 16 bits that are cut off
// would become an infinity.
__device__ __forceinline__ uint32_t quiet_nan2(uint32_t a, uint32_t b) {
    return ((a & 0x7fffffffu) > 0x7f800000u ? 0x40u : 0u) | ((b & 0x7fffffffu) > 0x7f800000u ? 0x400000u : 0u);
}

__device__ __forceinline__ float finite_or_zero(float v) { return fabsf(v) <= 3.402823466e38f ? v : 0.f; }

__device__ __forceinline__ float cluster_read(const float* local, uint32_t rank) {
    uint32_t addr;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"((uint32_t)__cvta_generic_to_shared(local)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
// The sum of `count` chunks that lie `per_block` to a block of the cluster, in order: chunk c of block r at p + c * stride of that
// block's shared memory.  Four lanes (l = 0 .. 3, eight lanes apart) share a sum: each has sixteen remote reads in flight (one takes
// about half a microsecond), then they add their terms one lane after the other.  The result is in the lane with l = 3.
__device__ __forceinline__ float cluster_sum(const float* p, int stride, int count, int per_block, int l) {
    float t = 0.f;
    for (int j0 = 0; j0 < count; j0 += 64) {
        const int mine = j0 + 16 * l;
        int r = mine / per_block, c = mine % per_block;
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j)
            if (mine + j < count) {
                v[j] = cluster_read(p + (size_t)c * stride, r);
                if (++c == per_block) { c = 0; ++r; }
            }
#pragma unroll
        for (int turn = 0; turn < 4; ++turn) {
            const float before = __shfl_sync(0xffffffffu, t, (threadIdx.x & 7) + 8 * ((turn + 3) & 3));
            if (l == turn) {
                t = before;
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (mine + j < count) t += v[j];
            }
        }
    }
    return t;
}

// What becomes of a gate and an up number of result row `r` (gemm_grouped.cu's two forms; a plain SwiGLU is form 0 with w = 1).
__device__ __forceinline__ float glu(const Args& a, float g, float u, int r) {
    if (a.clamped) {
        g = fminf(g, a.limit);
        u = fminf(fmaxf(u, -a.limit), a.limit);
        return g / (1.0f + expf(-a.slope * g)) * (u + 1.0f);
    }
    const float w = a.row_scale ? a.row_scale[r] : 1.0f;
    g *= w;
    return g / (1.0f + expf(-g)) * (u * w);
}

// SMALL: one tile of at most 16 tokens; fewer threads of fewer registers, so that two blocks share an SM and the next product's
// blocks can start on their weights while this one's finish.  CHUNK: steps of a chunk.
template <bool SMALL, int CHUNK>
__global__ void __launch_bounds__(SMALL ? 512 : 640, SMALL ? 2 : 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const Args a) {
    constexpr int kEpiWarps = SMALL ? 4 : 8;
    constexpr int kFirstEpi = 12;
    constexpr int kCols = SMALL ? 16 : 40;           // columns (tokens) of an epilogue thread
    extern __shared__ unsigned char smem_raw[];
    unsigned char* ring = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* xp = ring + a.ring_bytes;
    float* sums = reinterpret_cast<float*>(xp + a.x_bytes);
    __shared__ __align__(8) uint64_t w_full[kMaxW], w_empty[kMaxW], x_full[kMaxX], x_empty[kMaxX];
    __shared__ __align__(8) uint64_t a_full[kMaxA], a_empty[kMaxA], chunk_full[2], hi_free[2], corr_full, corr_free;
    __shared__ uint32_t tmem_base_slot;
    __shared__ volatile int failed;

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int rank = a.cluster > 1 ? (int)llm_cluster_rank() : 0;
    // the token tiles of a block of W's rows are neighbours in the grid, so that W comes from HBM once
    const int tile = blockIdx.x / a.cluster;
    const int feat0 = (tile / a.t_tiles) * (a.swiglu ? kRows / 2 : kRows);
    int tok0 = (tile % a.t_tiles) * a.tt, tok_end = min(a.tokens, tok0 + a.tt), w_row0 = feat0;
    if (a.tiles) {
        pdl_wait();                                    // the list is an earlier kernel's
        const int i = tile % a.t_tiles;
        if (i >= a.tiles[0]) return;                   // the whole cluster
        const int* e = a.tiles + 4 + 4 * i;
        tok0 = e[1];
        tok_end = tok0 + min(e[2], a.tt);
        w_row0 = e[0] * a.n * (a.swiglu ? 2 : 1) + feat0;
    }
    const int block_steps = a.segs / a.cluster * a.seg_steps;
    const int step0 = rank * block_steps, n_steps = min(a.steps - step0, block_steps);
    const int n_chunks = (n_steps + CHUNK - 1) / CHUNK;
    const int x_stage = 3 * a.tt * 128;                // a stage of x: 64 k of the three pieces

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.w_stages; ++s) { mbar_init(&w_full[s], 1); mbar_init(&w_empty[s], 4); }
        for (int s = 0; s < a.x_stages; ++s) { mbar_init(&x_full[s], 1); mbar_init(&x_empty[s], 2); }
        for (int s = 0; s < a.a_slots; ++s) { mbar_init(&a_full[s], 8); mbar_init(&a_empty[s], 2); }
        for (int s = 0; s < 2; ++s) { mbar_init(&chunk_full[s], 1); mbar_init(&hi_free[s], kEpiWarps); }
        mbar_init(&corr_full, 1);
        mbar_init(&corr_free, kEpiWarps);
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(a.tmem_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base_slot, 0);
    const uint32_t t_hi = tmem, t_corr = tmem + 2 * a.tt, t_a = tmem + 4 * a.tt;

    pdl_trigger();
    if (warp == 0) {
        // ---- loader of W: the weights depend on no earlier kernel ----------------------------------------------
        const int boxes = 2 * n_steps, k_first = step0 * kStepK;
        uint32_t phase = 1;
        bool free_now = true;                          // what a poll after the box before has found
        for (int b = 0, s = 0; b < boxes; ++b) {
            if (b >= a.w_stages && !free_now && !mbar_wait_all(&w_empty[s], phase)) { if (lane == 0) give_up_f32(a, 11); failed = 1; break; }
            if (elect_one()) {
                unsigned char* st = ring + (size_t)s * kBoxBytes;
                mbar_expect_tx(&w_full[s], kBoxBytes);
                tma_load_2d(st, &map_w, &w_full[s], k_first + 32 * b, w_row0);
                if (a.swiglu) tma_load_2d(st + kBoxBytes / 2, &map_w, &w_full[s], k_first + 32 * b, a.n + w_row0);
            }
            __syncwarp();
            if (++s == a.w_stages) { s = 0; phase ^= 1; }
            if (b + 1 >= a.w_stages) {
                const bool now = mbar_poll(&w_empty[s], phase);
                free_now = __all_sync(0xffffffffu, now);
            }
        }
    } else if (warp == 2) {
        // ---- loader of x's pieces: three boxes of 64 k ----------------------------------------------------------
        pdl_wait();
        uint32_t phase = 1;
        for (int j = 0, s = 0; j < n_steps; ++j) {
            if (j >= a.x_stages && !mbar_wait_all(&x_empty[s], phase)) { if (lane == 0) give_up_f32(a, 11); failed = 1; break; }
            if (elect_one()) {
                mbar_expect_tx(&x_full[s], x_stage);
#pragma unroll
                for (int p = 0; p < 3; ++p)
                    tma_load_2d(xp + (size_t)s * x_stage + p * a.tt * 128, &map_x, &x_full[s], (step0 + j) * kStepK, p * a.tokens + tok0);
            }
            __syncwarp();
            if (++s == a.x_stages) { s = 0; phase ^= 1; }
        }
    } else if (warp == 1 || warp == 3) {
        // ---- issuers: warp 1 of the large products, warp 3 of the small ones (counters run along: a division costs them 100 clocks) --
        const bool large = warp == 1;
        const uint32_t idesc1 = umma_idesc(kRows, a.tt), idesc2 = umma_idesc(kRows, 2 * a.tt);
        const uint64_t plane = (uint64_t)(a.tt * 128) >> 4, desc0 = umma_desc(xp), desc_stage = (uint64_t)x_stage >> 4;
        uint64_t desc = desc0;
        uint32_t x_phase = 0, a_phase = 0;
        int xs = 0, as = 0, seg_left = a.seg_steps, seg = 0;
        bool x_ok = false, a_ok = false, hi_ok = false;       // what a poll during the step before has found
        for (int i = 0; i < n_steps; ++i) {
            const int c = i / CHUNK;
            const bool seg_start = seg_left == a.seg_steps, chunk_start = i % CHUNK == 0;
            bool ok = x_ok || mbar_wait_all(&x_full[xs], x_phase);
            if (large && chunk_start && c >= 2) ok = ok && (hi_ok || mbar_wait_all(&hi_free[c & 1], ((c / 2) - 1) & 1));
            if (!large && seg_start && i > 0) ok = ok && mbar_wait_all(&corr_free, (seg++) & 1);
            ok = ok && (a_ok || mbar_wait_all(&a_full[as], a_phase));
            if (!ok) { if (lane == 0) give_up_f32(a, 12); failed = 1; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a0 = t_a + as * kACols, d_hi = t_hi + (c & 1) * a.tt;
            const bool last = i == n_steps - 1;
            if (elect_one()) {
                if (large) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_ts(d_hi, a0 + 8 * k, desc + 2 * k, idesc1, !(chunk_start && k == 0));
                    umma_commit(&a_empty[as]);
                    umma_commit(&x_empty[xs]);
                    if (i % CHUNK == CHUNK - 1 || last) umma_commit(&chunk_full[c & 1]);
                } else {
                    // The pieces of x lie one after the other, so that one instruction multiplies a piece of W with two of them and adds to
                    // both halves of t_corr.  All three have one shape and one accumulator: only such instructions are promised to run in
                    // the order of their issue (lo.hi by itself, half as wide, was not).  Five instructions of one product each cost a
                    // step of five tokens 2.23 ms against 2.22; lo.mid comes with the width and is below what the sum can hold.
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t ah = a0 + 8 * k, am = ah + 32, al = ah + 64;
                        const uint64_t bh = desc + 2 * k, bm = bh + plane;
                        umma_ts(t_corr, ah, bm, idesc2, !(seg_start && k == 0));          // hi.mid | hi.lo
                        umma_ts(t_corr, am, bh, idesc2, 1u);                              // mid.hi | mid.mid
                        umma_ts(t_corr, al, bh, idesc2, 1u);                              // lo.hi  | lo.mid
                    }
                    umma_commit(&a_empty[as]);
                    umma_commit(&x_empty[xs]);
                    if (seg_left == 1 || last) umma_commit(&corr_full);
                }
            }
            __syncwarp();
            desc += desc_stage;
            if (++xs == a.x_stages) { xs = 0; x_phase ^= 1; desc = desc0; }
            if (++as == a.a_slots) { as = 0; a_phase ^= 1; }
            if (--seg_left == 0) seg_left = a.seg_steps;
            const int cn = (i + 1) / CHUNK;
            const bool x_now = mbar_poll(&x_full[xs], x_phase), a_now = mbar_poll(&a_full[as], a_phase);
            const bool hi_now = large && cn >= 2 && mbar_poll(&hi_free[cn & 1], ((cn / 2) - 1) & 1);
            x_ok = __all_sync(0xffffffffu, x_now); a_ok = __all_sync(0xffffffffu, a_now); hi_ok = __all_sync(0xffffffffu, hi_now);
        }
    } else if (warp >= 4 && warp < kFirstEpi) {
        // ---- converters: W's pieces into tensor memory; each group of four warps has one of the two boxes of every step ------------
        const int q = warp & 3, group = (warp - 4) >> 2, row = q * 32 + lane, sw = row & 7;
        uint32_t phase = 0, a_phase = 1;
        bool w_ok = false;                                     // what a poll during the step before has found
        for (int i = 0, s = group, as = 0; i < n_steps; ++i) {
            if (!w_ok && !mbar_wait_all(&w_full[s], phase)) { if (lane == 0) give_up_f32(a, 14); failed = 1; break; }
            const unsigned char* st = ring + (size_t)s * kBoxBytes + row * 128;
            // the whole box is taken apart before the wait for the slot, so that only the stores lie between a slot's last product and
            // its next one
            const bool a_now = i < a.a_slots || mbar_poll(&a_empty[as], a_phase);
            uint32_t hi[16], mid[16], lo[16], all = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float4 v = *reinterpret_cast<const float4*>(st + ((j ^ sw) << 4));
                split2(v.x, v.y, hi[2 * j], mid[2 * j], lo[2 * j]);
                split2(v.z, v.w, hi[2 * j + 1], mid[2 * j + 1], lo[2 * j + 1]);
                all |= lo[2 * j] | lo[2 * j + 1];
            }
            // The box may be handed back only when its numbers lie in registers: an arrival does not wait for loads that were issued
            // before it, and beside a kernel that keeps the SM's load path busy they can take longer than the box's successor needs to
            // land (measured beside attention: rows of a later box in 96 of 96 products of 5 x 2 * 8192 x 2048).  The vote takes a piece
            // of every number that was read, and the arrival cannot pass what depends on it.
            if (__any_sync(0xffffffffu, maybe_not_finite(all))) {
#pragma unroll 1
                for (int j = 0; j < 8; ++j) {
                    const uint4 v = *reinterpret_cast<const uint4*>(st + ((j ^ sw) << 4));
                    const uint32_t first = quiet_nan2(v.x, v.y), second = quiet_nan2(v.z, v.w);
#pragma unroll
                    for (int i = 0; i < 16; ++i) hi[i] |= i == 2 * j ? first : i == 2 * j + 1 ? second : 0u;
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // (these loads, too, come before the box's successor)
            }
            const bool a_ok = __all_sync(0xffffffffu, a_now);
            __syncwarp();
            if (lane == 0) mbar_arrive(&w_empty[s]);            // the box has been read
            __syncwarp();
            if ((s += 2) >= a.w_stages) { s -= a.w_stages; phase ^= 1; }
            const bool w_now = mbar_poll(&w_full[s], phase);
            if (!a_ok && !mbar_wait_all(&a_empty[as], a_phase)) { if (lane == 0) give_up_f32(a, 14); failed = 1; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t ta = t_a + as * kACols + 16 * group + ((uint32_t)(q * 32) << 16);
            __syncwarp();
            tmem_st16(ta, hi);
            tmem_st16(ta + 32, mid);
            tmem_st16(ta + 64, lo);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            w_ok = __all_sync(0xffffffffu, w_now);
            __syncwarp();
            if (lane == 0) mbar_arrive(&a_full[as]);
            __syncwarp();
            if (++as == a.a_slots) { as = 0; a_phase ^= 1; }
        }
    } else if (warp >= kFirstEpi) {
        // ---- epilogue: chunks out of tensor memory ----------------------------------------------------------------
        const int q = warp & 3, col0 = ((warp - kFirstEpi) >> 2) * kCols, row = q * 32 + lane;
        const uint32_t lane_off = (uint32_t)(q * 32) << 16;
        float total[kCols];
#pragma unroll
        for (int j = 0; j < kCols; ++j) total[j] = 0.f;
        bool ok = true;
        int seg_left = a.seg_steps / CHUNK, seg = 0;
        for (int c = 0; c < n_chunks; ++c) {
            const bool seg_end = --seg_left == 0 || c == n_chunks - 1;
            if (seg_left == 0) seg_left = a.seg_steps / CHUNK;
            if (!mbar_wait_all(&chunk_full[c & 1], (c / 2) & 1) || (seg_end && !mbar_wait_all(&corr_full, (seg++) & 1))) { if (lane == 0) give_up_f32(a, 13); failed = 1; ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int g = 0; g < kCols; g += 8) {
                if (col0 + g < a.tt) {
                    uint32_t v[8], w[8];
                    if (seg_end) {
                        tmem_ld8(t_corr + col0 + g + lane_off, v);
                        tmem_ld8(t_corr + a.tt + col0 + g + lane_off, w);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                        for (int j = 0; j < 8; ++j) w[j] = __float_as_uint(finite_or_zero(__uint_as_float(v[j]) + __uint_as_float(w[j])));
                    }
                    tmem_ld8(t_hi + (c & 1) * a.tt + col0 + g + lane_off, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        float t = __uint_as_float(v[j]);
                        if (seg_end) t += __uint_as_float(w[j]);
                        if (a.cluster > 1) {
                            if (!SMALL || col0 + g + j < a.sum_cols) sums[((size_t)c * (SMALL ? a.sum_cols : a.tt) + col0 + g + j) * kRows + row] = t;
                        } else {
                            total[g + j] += t;
                        }
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&hi_free[c & 1]);
                if (seg_end) mbar_arrive(&corr_free);
            }
            __syncwarp();
        }
        if (a.cluster == 1) {
            pdl_wait();                                    // nothing is stored before the previous kernel has finished
            if (a.swiglu) {
                // rows 0 .. 63 are gate rows, 64 .. 127 the up rows of the same features: through the ring, which has been read, to
                // all threads of the block (below)
                float* rows = reinterpret_cast<float*>(ring);
#pragma unroll
                for (int j = 0; j < kCols; ++j)
                    if (ok && col0 + j < a.tt) rows[(size_t)(col0 + j) * kRows + row] = total[j];
            } else if (ok && feat0 + row < a.n) {
#pragma unroll
                for (int j = 0; j < kCols; ++j) {
                    const int tok = tok0 + col0 + j;
                    if (tok < tok_end) a.out[(size_t)tok * a.ldc + feat0 + row] = total[j];
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (a.cluster == 1 && a.swiglu && !failed) {
        pdl_wait();
        const float* rows = reinterpret_cast<const float*>(ring);
        const int live = tok_end - tok0;
#pragma unroll 4
        for (int e = threadIdx.x; e < live * 64; e += blockDim.x) {
            const int col = e >> 6, row = e & 63;
            if (feat0 + row < a.n)
                a.out[(size_t)(tok0 + col) * a.ldc + feat0 + row] = glu(a, rows[col * kRows + row], rows[col * kRows + 64 + row], tok0 + col);
        }
    }
    if (a.cluster > 1) {
        __syncwarp();
        llm_cluster_sync();                                // every block's chunk sums lie in its shared memory
        pdl_wait();
        const int rows = a.swiglu ? kRows / 2 : kRows, live = tok_end - tok0;
        const int all_chunks = (a.steps + CHUNK - 1) / CHUNK;
        const int per_block = a.segs / a.cluster * (a.seg_steps / CHUNK);         // (the last block may have fewer)
        const int l = (threadIdx.x >> 3) & 3, per_pass = blockDim.x / 4, stride = (SMALL ? a.sum_cols : a.tt) * kRows;
        for (int e0 = rank * per_pass; e0 < live * rows; e0 += a.cluster * per_pass) {
            const int e = e0 + (threadIdx.x >> 5) * 8 + (threadIdx.x & 7);
            const int col = min(e / rows, live - 1), row = e % rows;             // (all lanes take part in the sums)
            const float* p = sums + (size_t)col * kRows + row;
            const float g = cluster_sum(p, stride, all_chunks, per_block, l);
            const float u = a.swiglu ? cluster_sum(p + kRows / 2, stride, all_chunks, per_block, l) : 0.f;
            if (l == 3 && e < live * rows && feat0 + row < a.n)
                a.out[(size_t)(tok0 + col) * a.ldc + feat0 + row] = a.swiglu ? glu(a, g, u, tok0 + col) : g;
        }
        __syncwarp();
        llm_cluster_sync();                                // nobody leaves while its shared memory is being read
    }
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(a.tmem_cols));
    }
}

// planes[p][t][k], p = hi, mid, lo: the bfloat16 pieces of x, four numbers a thread; columns K .. kp - 1 are zero.  Listed form: of
// the first live_rows[0] rows alone, row t being row source[t] of x (null: t).
__global__ void __launch_bounds__(256)
split_planes_kernel(const float* __restrict__ x, bf16* __restrict__ planes, int tokens, int K, int kp, const int* __restrict__ source,
                    const int* __restrict__ live_rows) {
    pdl_trigger();
    pdl_wait();
    const int quads = kp / 4, live = live_rows ? min(tokens, live_rows[0]) : tokens;
    const size_t plane = (size_t)tokens * kp;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < (size_t)live * quads; i += (size_t)gridDim.x * blockDim.x) {
        const int t = (int)(i / quads), k = (int)(i % quads) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k < K) v = *reinterpret_cast<const float4*>(x + (size_t)(source ? source[t] : t) * K + k);
        uint2 h, m, l;
        split2(v.x, v.y, h.x, m.x, l.x);
        split2(v.z, v.w, h.y, m.y, l.y);
        h.x |= quiet_nan2(__float_as_uint(v.x), __float_as_uint(v.y));
        h.y |= quiet_nan2(__float_as_uint(v.z), __float_as_uint(v.w));
        bf16* d = planes + (size_t)t * kp + k;
        *reinterpret_cast<uint2*>(d) = h;
        *reinterpret_cast<uint2*>(d + plane) = m;
        *reinterpret_cast<uint2*>(d + 2 * plane) = l;
    }
}

constexpr int kSmemLimit = 226 * 1024;      // of 227 KiB a block; the static arrays take the rest

struct Plan { int tt, cluster, w_stages, x_stages, a_slots, tmem_cols, smem; };

// Clusters of 1 to 8 blocks that run at a time: one block to an SM as cudaOccupancyMaxActiveClusters gives it (the SMs of a GPC are no multiple of
// eight), two to an SM as the times below fit it.
constexpr int kClusters[2][9] = {{0, 148, 74, 45, 33, 26, 22, 15, 15}, {0, 296, 148, 90, 74, 52, 44, 30, 35}};

// us of a product of at most 16 tokens: `tiles` tiles of 128 features in clusters of `cl` blocks of `cta_steps` steps each, `per_sm` blocks to an SM.
// A wave is a chain of barriers (1.1 us a step where two blocks share an SM) and, in a cluster, a pass over the sums for every `cl` tokens; the waves
// and the stream of the weights hide in each other for the most part.  Fitted to 939 cuts of 30 products (n 512 to 50000, k 512 to 18944) at 1, 4, 8, 12
// and 16 tokens; the cut it takes is 0.3 % off the fastest on average, 9 % at most.  (An estimate without the passes and with one block to an SM only
// where two don't fit was 7.6 % off, 16 x 14000 x 1500 2.2 times: 48.7 us for 21.7.  16 x 12000 x 5000 77 -> 57 us, one token by 9000 x 3000 32 -> 26,
// by 2048 x 8192 24, by 18944 x 3584 65 -> 45.)
double few_us(long long tiles, int cl, int cta_steps, int per_sm, int tokens, int steps) {
    const long long waves = (tiles + kClusters[per_sm - 1][cl] - 1) / kClusters[per_sm - 1][cl];
    const double sums = cl > 1 ? 1.2 + 1.9 * ((tokens + cl - 1) / cl - 1) : 0.0;
    const double chain = waves * (cta_steps * (per_sm == 2 ? 1.08 : 0.59) + 6.6 + sums), stream = tiles * kRows * steps * kStepK * 4.0 / 5.8e6 + 1.5;
    return chain > stream ? chain + 0.34 * stream : stream + 0.34 * chain;
}

// The cut of a product into tiles of `tt` tokens and clusters over the k range: the one with the least estimated clocks.  A step of
// 64 k costs a block the larger of its tensor-core time (12 clocks a token) and its shared-memory time (64 KiB of W written and
// read, 1152 bytes a token, at 128 bytes a clock), and about 1000 clocks of barriers whatever its size.  Few tokens (at most 16): few_us.
// Listed form: `listed` tiles are expected, of `tokens` rows at most.
Plan make_plan(int tokens, int n, int swiglu, int steps, int seg_steps, int sms, int listed) {
    const int segs = (steps + seg_steps - 1) / seg_steps;
    const bool small = tokens <= kSmallTokens;
    const long long f_tiles = swiglu ? (n + 63) / 64 : (n + kRows - 1) / kRows;
    Plan best{};
    double best_cost = 1e30;
    const int most = tokens >= kMaxTile ? kMaxTile : (tokens + 15) / 16 * 16;
    for (int tt = small || listed ? most : 16; tt <= most; tt += 16)
        for (int cl = 1; cl <= segs; ++cl)
            for (int per_sm = 1; per_sm <= (small ? 2 : 1); ++per_sm) {
                if (segs % cl) continue;
                const long long ctas = f_tiles * (listed ? listed : (tokens + tt - 1) / tt) * cl;
                const int cta_steps = segs / cl * seg_steps < steps ? segs / cl * seg_steps : steps;
                const int chunks = (cta_steps + kChunkSteps - 1) / kChunkSteps;
                const int sums = cl > 1 ? chunks * (small ? tokens : tt) * kRows * 4 : 0, x_stage = 3 * tt * 128;
                auto w_stages = [&](int xs) {
                    const int room = ((per_sm == 2 ? 112 * 1024 : kSmemLimit) - 1024 - sums - xs * x_stage) / kBoxBytes / 2 * 2;
                    return room < kMaxW ? room : kMaxW;
                };
                const int ws = w_stages(2);
                if (ws < 4) continue;
                int xs = 2;
                while (xs < kMaxX && w_stages(xs + 1) == ws) ++xs;
                const double mma = 12.0 * tt, smem_clk = (65536.0 + 1152.0 * tt) / 128.0, barriers = 1000.0;
                const double step_clk = mma > smem_clk ? mma : smem_clk;
                const double cost = small ? few_us(ctas / cl, cl, cta_steps, per_sm, tokens, steps)
                                          : (double)((ctas + sms - 1) / sms) * (cta_steps * (step_clk > barriers ? step_clk : barriers) + 3000.0) +
                                                (cl > 1 ? 2000.0 + 40.0 * chunks * cl * tt / 16 : 0.0);
                if (cost < best_cost) {
                    best_cost = cost;
                    const int cols = per_sm == 2 || 4 * tt + 2 * kACols <= 256 ? 256 : 512, slots = (cols - 4 * tt) / kACols;
                    best = Plan{tt, cl, ws, xs, slots < kMaxA ? slots : kMaxA, cols, ws * kBoxBytes + xs * x_stage + sums + 1024};
                }
            }
    return best;
}

template <bool SMALL, int CHUNK>
int launch(const CUtensorMap& mw, const CUtensorMap& mx, const Args& a, dim3 grid, int smem, cudaStream_t stream) {
    auto kern = gemm_f32_tc_kernel<SMALL, CHUNK>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
    if (e != cudaSuccess) LLM_FAIL(-2, "gemm_f32_tc: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    if (a.cluster > 1)
        llm_launch_cluster(kern, grid, SMALL ? 512 : 640, smem, stream, (unsigned)a.cluster, mw, mx, a);
    else
        llm_launch(kern, grid, SMALL ? 512 : 640, smem, stream, mw, mx, a);
    LLM_CHECK_LAUNCH("gemm_f32_tc");
    return 0;
}

}  // namespace

// 1 if llm_gemm_f32_tc takes a product with rows of K floats (TMA: rows that start on 16-byte boundaries).
LLM_API int llm_gemm_f32_tc_supported(int K, const void* x, const void* w) {
    return K >= 4 && K % 4 == 0 && !((uintptr_t)x & 15) && !((uintptr_t)w & 15);
}

// bfloat16 elements of scratch that a call with `tokens` rows needs.
LLM_API long long llm_gemm_f32_tc_scratch(int tokens, int K) { return 3LL * tokens * ((K + 7) / 8 * 8); }

namespace {

// `tokens`: rows of x's pieces (and of the result); `groups` weight matrices; listed form: max_tiles > 0.
int run(const float* x, const int* source, const float* w, int tokens, int groups, int max_tiles, int K, void* planes, Args a, cudaStream_t stream) {
    if (!llm_gemm_f32_tc_supported(K, x, w)) LLM_FAIL(-1, "gemm_f32_tc: rows of %d floats do not start on 16-byte boundaries", K);
    if (!planes || ((uintptr_t)planes & 15)) LLM_FAIL(-1, "gemm_f32_tc: scratch for the pieces of x, on a 16-byte boundary, is needed");
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        LLM_FAIL(-2, "gemm_f32_tc: no device");
    a.tokens = tokens;
    a.status = const_cast<int*>(llm_gemm_bf16_status_word());
    if (!a.status) LLM_FAIL(-2, "gemm_f32_tc: no status word");
    a.steps = (K + kStepK - 1) / kStepK;
    a.seg_steps = ((a.steps + 7) / 8 + 1) / 2 * 2;
    if (a.seg_steps < 4) a.seg_steps = 4;
    a.segs = (a.steps + a.seg_steps - 1) / a.seg_steps;
    const int tile_tokens = max_tiles && tokens > kListedRows ? kListedRows : tokens;
    const Plan p = make_plan(tile_tokens, a.n, a.swiglu, a.steps, a.seg_steps, sms, max_tiles < tokens ? max_tiles : tokens);
    if (!p.tt) LLM_FAIL(-1, "gemm_f32_tc: no cut of %d x %d x %d fits", tokens, a.n, K);
    a.cluster = p.cluster; a.tt = p.tt; a.w_stages = p.w_stages; a.x_stages = p.x_stages; a.a_slots = p.a_slots;
    a.ring_bytes = p.w_stages * kBoxBytes;
    a.x_bytes = p.x_stages * 3 * p.tt * 128;
    a.tmem_cols = p.tmem_cols;
    a.sum_cols = tile_tokens;
    a.t_tiles = max_tiles ? max_tiles : (tokens + p.tt - 1) / p.tt;
    const long long blocks_x = (long long)(a.swiglu ? (a.n + 63) / 64 : (a.n + kRows - 1) / kRows) * a.t_tiles * p.cluster;
    if (blocks_x > 0x7fffffffLL) LLM_FAIL(-1, "gemm_f32_tc: %d tokens by %d are too many for one launch", tokens, a.n);
    const dim3 grid((unsigned)blocks_x);
    const int kp = (K + 7) / 8 * 8;
    CUtensorMap mw, mx;
    if (int rc = llm_tensor_map_2d_f32(w, (uint64_t)groups * a.n * (a.swiglu ? 2 : 1), K, a.swiglu ? kRows / 2 : kRows, 32, &mw)) return rc;
    if (int rc = llm_tensor_map_2d(planes, 3ull * tokens, kp, p.tt, 64, &mx)) return rc;
    const size_t quads = (size_t)tokens * (kp / 4);
    const int blocks = (int)((quads + 255) / 256 < 148 * 8 ? (quads + 255) / 256 : 148 * 8);
    llm_launch(split_planes_kernel, blocks, 256, 0, stream, x, (bf16*)planes, tokens, K, kp, source, a.tiles ? a.tiles + 1 : nullptr);
    LLM_CHECK_LAUNCH("gemm_f32_tc_planes");
    const auto go = a.steps <= kShortSteps ? (tile_tokens <= kSmallTokens ? launch<true, 1> : launch<false, 1>)
                                           : (tile_tokens <= kSmallTokens ? launch<true, kChunkSteps> : launch<false, kChunkSteps>);
    return go(mw, mx, a, grid, p.smem, stream);
}

}  // namespace

// out [tokens, ldc] = x [tokens, K] . w [n, K]^T, or with swiglu silu(x . w[0:n]^T) * (x . w[n:2n]^T); rows of x and w contiguous.
LLM_API int llm_gemm_f32_tc(const float* x, const float* w, float* out, int tokens, int n, int K, int ldc, int swiglu,
                            void* planes, cudaStream_t stream) {
    if (tokens == 0 || n == 0) return 0;
    Args a{};
    a.out = out; a.n = n; a.ldc = ldc; a.swiglu = swiglu ? 1 : 0;
    return run(x, nullptr, w, tokens, 1, 0, K, planes, a, stream);
}

// The listed form of llm_gemm_grouped: out [rows, ldc] = row r of x (row source[r], null: r) . w[group of r]^T for the rows that the
// device's list of tiles names (of llm_gemm_grouped_tile_rows rows at most; tiles[1]: how many rows are live), with that entry's glu
// forms (0 none, 1 clamped, 2 silu with a factor per row).  w [groups, n (2n with glu), K].
LLM_API int llm_gemm_f32_tc_listed(const float* x, const int* source, const float* w, float* out, int rows, int n, int K, int groups,
                                   const int* tiles, int max_tiles, int form, float limit, float slope, const float* row_scale,
                                   void* planes, cudaStream_t stream) {
    if (rows <= 0 || n <= 0 || groups <= 0 || max_tiles <= 0) return 0;
    if (form < 0 || form > 2) LLM_FAIL(-1, "gemm_f32_tc: glu form %d is not known", form);
    if (form == 1 && limit < 0.f) LLM_FAIL(-1, "gemm_f32_tc: the clamp's limit %g is negative", (double)limit);
    if (llm_gemm_grouped_tile_rows() != kListedRows) LLM_FAIL(-1, "gemm_f32_tc: tiles of %d rows", llm_gemm_grouped_tile_rows());
    if ((long long)groups * n * 2 > 0x7fffffffLL) LLM_FAIL(-1, "gemm_f32_tc: %d matrices of %d rows are too many", groups, n);
    Args a{};
    a.out = out; a.n = n; a.ldc = n; a.swiglu = form ? 1 : 0;
    a.tiles = tiles; a.clamped = form == 1; a.limit = limit; a.slope = slope; a.row_scale = form == 2 ? row_scale : nullptr;
    return run(x, source, w, rows, groups, max_tiles, K, planes, a, stream);
}

LLM_TRACE_EXPORT(gemm_f32_tc)
