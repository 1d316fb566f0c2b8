// Y[M][N] = X[M][K] * W[N][K]^T (+ addend) in 32 bits on the tensor cores, sm_100a.
//
// A float is the exact sum of three bfloat16 values (8 bits of the significand each; the second at most 2^-8, the third
// 2^-17 of the float's power of two), so a product of floats is nine products of bfloat16 values, each of them exact in 32
// bits.  The three smallest are left out: together less than 2^-24 of the product, a rounding of it, and 2^-28 on average.
// The other six are summed by tcgen05.mma.  The tensor cores cut off what they add instead of rounding it, so an accumulator
// lives for one block of 32 k only: it is read back, added to a sum in registers (rounded to nearest) and begun again.
//
//   * TMA brings blocks of both operands into a ring in shared memory and eight or twelve warps, four to a block, cut
//     them in three: the weights, operand A, into tensor memory (a lane a feature), the tokens, operand B, back into
//     shared memory (K-major, 64-byte swizzle).  With the weights' parts in shared memory too its bandwidth bound (a block of
//     128 x 128 took 1,650 clocks of it, 768 of the tensor cores); as it is the cutting warps' latency does (9216 x 1024,
//     201 tokens: issue slots 51 % busy, shared memory 31 %, tensor memory 35 %, DRAM 12 %).
//   * One lane issues the MMAs, 128 features by up to 208 tokens; four to sixteen warps add finished accumulators up.
//     Each role runs as far ahead as the rings and the accumulators let it.
//   * K is cut over a cluster where a matrix has too few feature tiles; the parts are added in rank order through
//     distributed shared memory.
//   * How K is cut depends on N and K alone and a value on its row of X and of W alone: the same bits in every batch.
//   * Values without three bfloat16 parts (infinities, NaN, beyond the largest bfloat16, parts below the smallest
//     normal one) are found by what the element came to and the largest magnitudes of its two rows (see ``sure``); such
//     an element is summed again as multiply-adds.  The warps that cut look at every value (sums of squares, packed).
#include <float.h>

#include "gemm_f32.cuh"
#include "tcgen05.cuh"

using namespace fwb;
using namespace fwb::tc5;

namespace {

constexpr int KB = 32;                                  // k per block: a 64-byte row of bfloat16
constexpr int ROW_BYTES = KB * 2;
constexpr int A_PART = KB / 2, A_COLS = 3 * A_PART;     // columns of tensor memory: a part of the weights, all three

template <int NT>
struct SplitTile {
    static constexpr int RAW_W = BM * KB * 4, RAW = RAW_W + NT * KB * 4, RAW_STAGES = NT > 112 ? 3 : NT > 64 ? 5 : 6;
    static constexpr int STAGE = 3 * NT * ROW_BYTES, STAGES = NT > 112 ? 2 : NT > 64 ? 3 : 4;
    static constexpr int PIECES = NT / 16;              // 16-byte pieces of the tokens a thread has of a block
    static constexpr int TEAMS = NT > 112 ? 2 : 3, CUTTERS = 4 * TEAMS;     // warps that cut, four to a block
    static constexpr int ADDERS = NT > 112 ? 16 : NT > 16 ? 8 : 4, THREADS = 32 * (CUTTERS + ADDERS + 2);
    static constexpr int COLUMNS = NT * 4 / ADDERS;     // of an accumulator, a warp's
    static constexpr int BUFFERS = NT > 112 ? 2 : NT > 64 ? 3 : 4, TMEM_COLS = 512;
    static constexpr int SMEM = STAGES * STAGE + RAW_STAGES * RAW + 1024 + 256 + (BM + NT + 1) * 4;
    static_assert(BUFFERS * NT + STAGES * A_COLS <= TMEM_COLS, "tensor memory");
    static_assert(NT * BM * 4 <= STAGES * STAGE + RAW_STAGES * RAW, "the parts of a cluster go where the rings were");
    static_assert(RAW_STAGES >= STAGES && STAGES >= TEAMS, "a cutting warp's waits tell a slot's phases apart");
    static_assert(RAW % 1024 == 0 && STAGE * STAGES % 1024 == 0, "swizzled rows");
};

struct SplitParams {
    const float *x, *w, *addend;
    float* y;
    int M, N, K, ldx, ldy;
    int splits, tile_tokens;
    bool vectors;                // rows of Y and the addend start on 16-byte borders
    float lost;                  // see ``sure``
    int* status;
};

// K-major, 64-byte swizzle: rows of 64 bytes, 8-row groups 512 bytes apart.
__device__ __forceinline__ uint64_t make_smem_desc_64(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;                             // SWIZZLE_64B
    return d;
}
// D[tmem] (+)= A[tmem] * B[shared memory].
__device__ __forceinline__ void umma_bf16_tmem(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                               uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Stores 8 columns of the thread's lane (tcgen05.wait::st is the caller's).
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\ttcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float* v) {
    uint32_t r[4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n\ttcgen05.wait::ld.sync.aligned;"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr)
                 : "memory");
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ bool elect_one() {
    uint32_t chosen;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(chosen));
    return chosen != 0;
}
// Two values in one register, as packed arithmetic takes them (half the instructions of the warps that cut).
__device__ __forceinline__ float low(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float high(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }
// The leading bfloat16 parts of two values, which keep the rest.
__device__ __forceinline__ uint32_t take_bf16(uint64_t& v) {
    uint32_t parts;
    asm("{\n\t.reg .f32 a, b;\n\t.reg .b32 fa, fb;\n\t.reg .b64 both;\n\t"
        "mov.b64 {a, b}, %1;\n\t"
        "cvt.rn.bf16x2.f32 %0, b, a;\n\t"
        "shl.b32 fa, %0, 16;\n\t"
        "and.b32 fb, %0, 0xffff0000;\n\t"
        "mov.b64 both, {fa, fb};\n\t"
        "sub.rn.f32x2 %1, %1, both;\n\t}"
        : "=&r"(parts), "+l"(v));
    return parts;
}
__device__ __forceinline__ uint2 take_bf16(ulonglong2& v) {
    uint64_t a = v.x, b = v.y;
    const uint2 parts = make_uint2(take_bf16(a), take_bf16(b));
    v.x = a;
    v.y = b;
    return parts;
}

// What is asked of an element before its sum counts.  Of a value that has no three bfloat16 parts less than 2^-126 is
// missing (or all of it: infinities, NaN and what rounds past the largest bfloat16 show in the sum, which is not finite),
// and as much of a partial product that has no place among the normal floats.  With x and w the largest magnitudes in the
// row of X and the row of W that is less than K 2^-126 (x + w + 6), so an element 2^24 times as large is right to a
// rounding: K 2^-100 max(x, w), or 2^-40 while both are below TALL (K up to 2^24).  A sum over a row of zeros is zero.
// What is asked is the two rows' own affair: bits do not depend on the batch.
constexpr float TALL = 0x1p36f, TALL_SQUARE = 0x1p72f, SMALL = 0x1p-40f;
__device__ __forceinline__ bool sure(float v) { return fabsf(v) <= FLT_MAX && fabsf(v) >= SMALL; }
// x, w: 0 for a row of zeros, its largest magnitude from TALL on, else another positive number.
__device__ __forceinline__ bool sure(float v, float x, float w, float lost) {
    const float top = fmaxf(x, w), least = top >= TALL ? fmaxf(SMALL, lost * top) : SMALL;
    return fabsf(v) <= FLT_MAX && (fabsf(v) >= least || x == 0.0f || w == 0.0f);
}
// An element whose parts did not say what the values are (rows of whole 16-byte pieces, on their borders).
__device__ __noinline__ float plain_sum(const float* x, const float* w, int K) {
    float sum[4] = {};
    for (int k = 0; k < K; k += 4) {
        const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(w + k);
        sum[0] = fmaf(a.x, b.x, sum[0]);
        sum[1] = fmaf(a.y, b.y, sum[1]);
        sum[2] = fmaf(a.z, b.z, sum[2]);
        sum[3] = fmaf(a.w, b.w, sum[3]);
    }
    return (sum[0] + sum[1]) + (sum[2] + sum[3]);
}
// A token's sums that are not all sure, four features a lane: against the largest magnitudes that the cluster's CTAs found.
__device__ __noinline__ float4 look_closer(const SplitParams& prm, float4 sum, uint32_t w_top, uint32_t x_top, int t, int f) {
    const int splits = prm.splits, lane = threadIdx.x & 31;
    float x = lane < splits ? ld_dsmem_f32(x_top, lane) : 0.0f;
    x = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(x)));
    float4 of[8], w = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int r = 0; r < 8; ++r) of[r] = r < splits ? ld_dsmem_f32x4(w_top, r) : w;
#pragma unroll
    for (int r = 0; r < 8; ++r) w = make_float4(fmaxf(w.x, of[r].x), fmaxf(w.y, of[r].y), fmaxf(w.z, of[r].z), fmaxf(w.w, of[r].w));
    float v[4] = {sum.x, sum.y, sum.z, sum.w};
    const float tops[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (f + j < prm.N && !sure(v[j], x, tops[j], prm.lost))
            v[j] = plain_sum(prm.x + (size_t)t * prm.ldx, prm.w + (size_t)(f + j) * prm.K, prm.K);
    return make_float4(v[0], v[1], v[2], v[3]);
}
// Four neighbouring features of a token.
__device__ __forceinline__ void finish(const SplitParams& prm, int t, int f, float4 sum) {
    const float v[4] = {sum.x, sum.y, sum.z, sum.w};
    float* y = prm.y + (size_t)t * prm.ldy + f;
    const float* addend = prm.addend ? prm.addend + (size_t)t * prm.ldy + f : nullptr;
    if (f + 3 < prm.N && prm.vectors) {
        if (addend) {
            const float4 a = *reinterpret_cast<const float4*>(addend);
            sum = make_float4(sum.x + a.x, sum.y + a.y, sum.z + a.z, sum.w + a.w);
        }
        *reinterpret_cast<float4*>(y) = sum;
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (f + j < prm.N) y[j] = addend ? v[j] + addend[j] : v[j];
    }
}
// A maximum of floats that are not negative is one of their bits as integers.
__device__ __forceinline__ void raise(float* at, float v) { atomicMax(reinterpret_cast<int*>(at), __float_as_int(v)); }
__device__ __forceinline__ float top_of(float top, const float4& v) {
    return fmaxf(fmaxf(fmaxf(top, fabsf(v.x)), fmaxf(fabsf(v.y), fabsf(v.z))), fabsf(v.w));
}
__device__ __forceinline__ bool not_zero(const float4& v) {
    return ((__float_as_uint(v.x) | __float_as_uint(v.y) | __float_as_uint(v.z) | __float_as_uint(v.w)) << 1) != 0;
}
__device__ __forceinline__ void add_squares(uint64_t& s, const ulonglong2& v) {
    asm("fma.rn.f32x2 %0, %1, %1, %0;\n\tfma.rn.f32x2 %0, %2, %2, %0;" : "+l"(s) : "l"(v.x), "l"(v.y));
}
__device__ __forceinline__ bool may_be_tall(uint64_t s) { return !(low(s) + high(s) < TALL_SQUARE); }      // (or not finite)

template <int NT>
__global__ void __launch_bounds__(SplitTile<NT>::THREADS, 1)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                      const __grid_constant__ SplitParams prm) {
    using T = SplitTile<NT>;
    constexpr int STAGES = T::STAGES, RAW_STAGES = T::RAW_STAGES, PIECES = T::PIECES, BUFFERS = T::BUFFERS;
    constexpr int CUTTERS = T::CUTTERS, MMA_WARP = CUTTERS + T::ADDERS, LOAD_WARP = MMA_WARP + 1;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* raw = ring + STAGES * T::STAGE;             // rows of 32 floats: 128 of W (128-byte swizzle), then of X
    uint64_t* raw_full = reinterpret_cast<uint64_t*>(raw + RAW_STAGES * T::RAW);
    uint64_t* raw_empty = raw_full + RAW_STAGES;
    uint64_t* full_bar = raw_empty + RAW_STAGES;
    uint64_t* empty_bar = full_bar + STAGES;
    uint64_t* acc_full = empty_bar + STAGES;
    uint64_t* acc_empty = acc_full + BUFFERS;
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + BUFFERS);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);
    // of this CTA's k: what ``sure`` asks of its features and of its tokens, and whether any value is TALL
    float* w_top = reinterpret_cast<float*>(raw + RAW_STAGES * T::RAW + 256);
    float* x_top = w_top + BM;
    float* any_tall = x_top + NT;

    pdl_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int splits = prm.splits, rank = blockIdx.x % splits;      // = the rank in the cluster
    const int t0 = (blockIdx.x / splits) * prm.tile_tokens, f0 = blockIdx.y * BM;
    const int tokens = min(prm.M - t0, prm.tile_tokens), columns = (tokens + 15) & ~15;
    const int blocks = (prm.K + KB - 1) / KB;
    const int first = (int)((long)blocks * rank / splits), n_blocks = (int)((long)blocks * (rank + 1) / splits) - first;

    if (tid == 0) {
        for (int r = 0; r < RAW_STAGES; ++r) {
            mbar_init(&raw_full[r], 1);
            mbar_init(&raw_empty[r], 4);
        }
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 4);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < BUFFERS; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], T::ADDERS);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < BM + NT + 1; i += T::THREADS) w_top[i] = 0.0f;
    if (warp == MMA_WARP) tmem_alloc(tmem_holder, T::TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    pdl_wait();

    const uint32_t a_base = tmem_base + BUFFERS * NT;
    const int quarter = warp & 3, column0 = ((warp - CUTTERS) >> 2) * T::COLUMNS;       // of an adding warp
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const uint32_t plane = columns * ROW_BYTES;          // a part of the tokens
    float* parts = reinterpret_cast<float*>(ring);       // a CTA's sums: [token][128 features]

    if (warp < CUTTERS) {
        // of the tokens: piece p is 16 bytes at k = 4 (id & 7) of row row0 + 16 p
        const int id = tid & 127, row0 = id >> 3;
        const uint32_t swizzled = row0 * ROW_BYTES + ((((id & 7) >> 1) ^ ((row0 >> 1) & 3)) << 4) + (id & 1) * 8;
        bool w_any = false;                              // this thread's feature has a value other than zero
        uint32_t x_any = 0;                              // bit p: row row0 + 16 p of the tokens has one
        const uint32_t x_all = tokens > row0 ? (1u << ((tokens - row0 + 15) >> 4)) - 1 : 0;
        float w_most = 1.0f;
        for (int i = warp >> 2; i < n_blocks; i += T::TEAMS) {
            const int r = i % RAW_STAGES, s = i % STAGES;
            // The stage first: a wait goes by its phase's parity, and a team never waited for the blocks of the other
            // teams.  Block i - STAGES multiplied means that every block up to it, the slot's last tenant too, has
            // landed; the stage's own phases cannot run ahead, as this team's block before waited for i - TEAMS - STAGES.
            bool ok = i < STAGES || mbar_wait(&empty_bar[s], (i / STAGES - 1) & 1, abort_flag, 34, prm.status);
            if (ok) ok = mbar_wait(&raw_full[r], (i / RAW_STAGES) & 1, abort_flag, 35, prm.status);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint8_t* from = raw + (size_t)r * T::RAW;
            const ulonglong2* x = reinterpret_cast<const ulonglong2*>(from + T::RAW_W) + id;
            uint8_t* x_to = ring + (size_t)s * T::STAGE + swizzled;
            const uint32_t w_to = a_base + lane_base + s * A_COLS;
            ulonglong2 w[8];                             // thread = feature: its 32 k
#pragma unroll
            for (int c = 0; c < 8; ++c) w[c] = *reinterpret_cast<const ulonglong2*>(from + id * 128 + ((c ^ (id & 7)) << 4));
            uint64_t w_squares = 0, x_squares = 0;
#pragma unroll
            for (int c = 0; c < 8; ++c) add_squares(w_squares, w[c]);
#pragma unroll
            for (int part = 0; part < 3; ++part)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t pairs[8];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint2 four = take_bf16(w[4 * h + c]);
                        pairs[2 * c] = four.x;
                        pairs[2 * c + 1] = four.y;
                    }
                    tmem_st8(w_to + part * A_PART + 8 * h, pairs);
                }
#pragma unroll
            for (int p0 = 0; p0 < PIECES; p0 += 4) {
                if (p0 * 16 >= columns) break;
                ulonglong2 v[4];                         // all asked for before the first one is cut
#pragma unroll
                for (int p = 0; p < 4; ++p)
                    if (p0 + p < PIECES && (p0 + p) * 16 < columns) v[p] = x[(p0 + p) * 128];
#pragma unroll
                for (int p = 0; p < 4; ++p)
                    if (p0 + p < PIECES && (p0 + p) * 16 < columns) add_squares(x_squares, v[p]);
#pragma unroll
                for (int part = 0; part < 3; ++part)
#pragma unroll
                    for (int p = 0; p < 4; ++p)
                        if (p0 + p < PIECES && (p0 + p) * 16 < columns)
                            *reinterpret_cast<uint2*>(x_to + part * plane + (p0 + p) * 16 * ROW_BYTES) = take_bf16(v[p]);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full_bar[s]);
            // what ``sure`` asks, where a block may add to it: read once more while the copies lie there
            const float4* w_raw = reinterpret_cast<const float4*>(from + id * 128);          // (in another order)
            const float4* x_raw = reinterpret_cast<const float4*>(x);
            if (!w_any) {
                w_any = low(w_squares) + high(w_squares) != 0.0f;
                if (!w_any) {
#pragma unroll
                    for (int c = 0; c < 8; ++c) w_any |= not_zero(w_raw[c ^ (id & 7)]);
                }
            }
            if (x_any != x_all) {
#pragma unroll
                for (int p = 0; p < PIECES; ++p)
                    if (p * 16 < columns && not_zero(x_raw[p * 128])) x_any |= 1u << p;
            }
            if (may_be_tall(w_squares)) {
#pragma unroll 1
                for (int c = 0; c < 8; ++c) w_most = top_of(w_most, w_raw[c]);
            }
            if (may_be_tall(x_squares)) {
#pragma unroll 1
                for (int p = 0; p * 16 < columns; ++p) {
                    const float most = top_of(0.0f, x_raw[p * 128]);
                    if (most >= TALL) {
                        raise(x_top + row0 + p * 16, most);
                        *any_tall = 1.0f;
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&raw_empty[r]);
        }
        if (w_any) raise(w_top + id, w_most >= TALL ? w_most : 1.0f);
        if (w_most >= TALL) *any_tall = 1.0f;
#pragma unroll 1
        for (int p = 0; p < PIECES; ++p)
            if (x_any >> p & 1) raise(x_top + row0 + p * 16, 1.0f);
    } else if (warp == LOAD_WARP) {
        if (lane == 0) {
            const uint32_t bytes = (BM + prm.tile_tokens) * KB * 4;
            int i = 0;
            for (; i < n_blocks; ++i) {
                const int r = i % RAW_STAGES, k = (first + i) * KB;
                if (i >= RAW_STAGES && !mbar_wait(&raw_empty[r], (i / RAW_STAGES - 1) & 1, abort_flag, 36, prm.status)) break;
                uint8_t* to = raw + (size_t)r * T::RAW;
                mbar_expect_tx(&raw_full[r], bytes);
                tma_load_2d(to, &map_w, &raw_full[r], k, f0);
                tma_load_2d(to + T::RAW_W, &map_x, &raw_full[r], k, t0);
            }
            // after a wait that gave up: the copies on their way land before shared memory goes to another CTA
            for (int j = i > RAW_STAGES ? i - RAW_STAGES : 0; j < i; ++j)
                for (unsigned spin = 0; spin < WAIT_LIMIT && !mbar_test(&raw_full[j % RAW_STAGES], (j / RAW_STAGES) & 1); ++spin) {}
        }
    } else if (warp == MMA_WARP) {
        // the whole warp walks along, one lane issues: descriptors stay in uniform registers (88 -> 50 clocks an MMA)
        const uint32_t idesc = make_idesc_mn(BM, columns);
        const bool issuer = elect_one();
        for (int i = 0; i < n_blocks; ++i) {
            const int s = i % STAGES, b = i % BUFFERS;
            bool ok = mbar_wait(&full_bar[s], (i / STAGES) & 1, abort_flag, 31, prm.status);
            if (ok && i >= BUFFERS) ok = mbar_wait(&acc_empty[b], (i / BUFFERS - 1) & 1, abort_flag, 32, prm.status);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const uint32_t a = a_base + s * A_COLS, d = tmem_base + b * NT;
            const uint64_t x0 = make_smem_desc_64(smem_u32(ring) + s * T::STAGE);
            if (issuer) {
                const uint64_t x1 = x0 + (plane >> 4), x2 = x1 + (plane >> 4);
                uint32_t more = 0;
                auto product = [&](int part, uint64_t x) {
#pragma unroll
                    for (int k = 0; k < KB / UMMA_K; ++k) {
                        umma_bf16_tmem(d, a + part * A_PART + 8 * k, x + 2 * k, idesc, more);
                        more = 1;
                    }
                };
                product(2, x0);                          // the smallest first
                product(0, x2);
                product(1, x1);
                product(1, x0);
                product(0, x1);
                product(0, x0);
                umma_commit(&empty_bar[s]);
                umma_commit(&acc_full[b]);
            }
            __syncwarp();
        }
    } else {
        float acc[T::COLUMNS];
#pragma unroll
        for (int j = 0; j < T::COLUMNS; ++j) acc[j] = 0.0f;
        bool ok = true;
        for (int i = 0; i < n_blocks; ++i) {
            const int b = i % BUFFERS;
            ok = __all_sync(0xffffffffu, mbar_wait(&acc_full[b], (i / BUFFERS) & 1, abort_flag, 33, prm.status));
            if (!ok) break;
            tc_fence_after();
            const uint32_t from = tmem_base + lane_base + b * NT + column0;
#pragma unroll
            for (int c = 0; c < T::COLUMNS; c += 8) {
                if (column0 + c >= columns) break;
                float part[8];
                if (c + 8 <= T::COLUMNS) tmem_ld8(from + c, part);
                else tmem_ld4(from + c, part);
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (c + j < T::COLUMNS) acc[c + j] += part[j];
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[b]);
        }
        // the last accumulator is complete: nothing reads the rings any more
        if (ok) {
#pragma unroll
            for (int j = 0; j < T::COLUMNS; ++j) parts[(column0 + j) * BM + quarter * 32 + lane] = acc[j];
        }
    }
    tc_fence_before();
    if (splits == 1) __syncthreads();
    else cluster_sync_all();
    if (*abort_flag == 0) {
        const float tall = splits == 1 ? *any_tall : lane < splits ? ld_dsmem_f32(smem_u32(any_tall), lane) : 0.0f;
        const int f = f0 + lane * 4, features = prm.N - f;
#pragma unroll 1
        for (int t = rank + warp * splits; t < tokens; t += (T::THREADS / 32) * splits) {
            const float* at = parts + t * BM + lane * 4;
            float4 sum;
            if (splits == 1) {
                sum = *reinterpret_cast<const float4*>(at);
            } else {
                sum = ld_dsmem_f32x4(smem_u32(at), 0);
                for (int r = 1; r < splits; ++r) {
                    const float4 part = ld_dsmem_f32x4(smem_u32(at), r);
                    sum.x += part.x;
                    sum.y += part.y;
                    sum.z += part.z;
                    sum.w += part.w;
                }
            }
            const bool good = (sure(sum.x) || features < 1) && (sure(sum.y) || features < 2) &&
                              (sure(sum.z) || features < 3) && (sure(sum.w) || features < 4);
            if (!__all_sync(0xffffffffu, good && tall == 0.0f))
                sum = look_closer(prm, sum, smem_u32(w_top + lane * 4), smem_u32(x_top + t), t0 + t, f);
            finish(prm, t0 + t, f, sum);
        }
    }
    if (splits > 1) cluster_sync_all();                  // nobody leaves while a peer reads
    __syncwarp();
    if (warp == MMA_WARP) tmem_dealloc(tmem_base, T::TMEM_COLS);
}

// Boxes of 32 k by box_rows of a float matrix, rows row_stride values apart.
bool make_map_f32(CUtensorMap* map, const float* base, long rows, int K, long row_stride, int box_rows,
                  CUtensorMapSwizzle swizzle) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)row_stride * 4};
    cuuint32_t box[2] = {(cuuint32_t)KB, (cuuint32_t)box_rows};
    cuuint32_t elem[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int NT>
int launch(const CUtensorMap& map_w, const CUtensorMap& map_x, const SplitParams& prm, int token_tiles, cudaStream_t stream) {
    auto kernel = gemm_f32_split_kernel<NT>;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SplitTile<NT>::SMEM);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((unsigned)(prm.splits * token_tiles), (unsigned)((prm.N + BM - 1) / BM), 1);
    config.blockDim = dim3(SplitTile<NT>::THREADS);
    config.dynamicSmemBytes = SplitTile<NT>::SMEM;
    config.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = prm.splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attr;
    config.numAttrs = pdl_enabled() ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&config, kernel, map_w, map_x, prm);
    return e == cudaSuccess ? fwb_launch_status() : (int)e;
}

}  // namespace

// By the matrix alone, so that a row's bits do not depend on the batch.  Smaller matrices leave most SMs without a tile, and
// what a CTA needs to start (tensor memory, rings) shows: single launches, us, multiply-adds then this, 1 | 64 | 201 tokens:
// 128 x 128 8.3 8.5 | 8.9 8.3 | 8.5 12.5; 256 x 512 8.6 8.3 | 8.8 8.4 | 8.6 14.1.  In a chain of launches over 300 MB of
// weights: 1024 x 1024 10.2 5.9 | 14.8 8.6 | 18.5 16.5; 3072 x 1024 11.0 8.1 | 21.9 11.1 | 47.1 21.5; 9216 x 1024 20.9 13.0 |
// 38.7 17.3 | 121 34.8; 1024 x 4608 34.3 12.3 | 59.8 17.2 | 75.7 38.1; 65536 x 1024 132 72 | 262 98 | 834 229; 128 x 8192
// 48.8 17.0 | 103 23.1 | 104 56.1; 8192 x 128 4.7 4.7 | 8.2 6.9 | 23.4 13.6; with half of W's or of X's rows zero at most
// 1.2 times as long (3072 x 1024, 201 tokens).  Relative error at K = 1,024 2.1e-7, then 0.9e-7 (one slice of 1,024:
// 1.2e-7), at 4,608 4.3e-7 and 1.1e-7, at 128 0.9e-7 and 0.7e-7.
bool fwb::gemm_f32_split_takes(int N, int K) {
    return N >= 128 && K >= 128 && (long)N * K >= 1L << 20 && N <= 128 * 65535;
}

int fwb::gemm_f32_split(const float* X, const float* W, float* Y, const float* addend, int M, int N, int K, int ldx, int ldy,
                        cudaStream_t stream) {
    SplitParams prm{X, W, addend, Y, M, N, K, ldx, ldy, 1, 0, false, K * 0x1p-100f, status_word()};
    prm.vectors = !(ldy & 3) && !((uintptr_t)Y & 15) && !((uintptr_t)addend & 15);
    const int feature_tiles = (N + BM - 1) / BM, blocks = (K + KB - 1) / KB;
    // a CTA an SM; 15 clusters of eight find room at once, 33 of four.  So 1024 x 1024, eight feature tiles, takes two rounds
    // from 209 to some 300 tokens: 209 | 225 | 300 tokens 18.6 | 21.1 | 24.1 us by multiply-adds, 23.4 | 23.3 | 26.5 so (the
    // slices may not follow the tokens)
    for (int s = 8; s > 1 && prm.splits == 1; s >>= 1)
        if (feature_tiles * s <= (s == 8 ? 128 : s == 4 ? 136 : 148) && blocks >= 4 * s) prm.splits = s;
    // (how the tokens are cut changes no value)
    const int most = M <= 16 ? 16 : M <= 64 ? 64 : M <= 112 ? 112 : 208;
    const long token_tiles = ((long)M + most - 1) / most;
    if (token_tiles > (1 << 24)) return FWB_TOO_LARGE;
    prm.tile_tokens = (int)((((M + token_tiles - 1) / token_tiles) + 15) & ~15L);
    const int count = (M + prm.tile_tokens - 1) / prm.tile_tokens;
    CUtensorMap map_w, map_x;
    if (!make_map_f32(&map_w, W, N, K, K, BM, CU_TENSOR_MAP_SWIZZLE_128B) ||
        !make_map_f32(&map_x, X, M, K, ldx, prm.tile_tokens, CU_TENSOR_MAP_SWIZZLE_NONE))
        return FWB_UNSUPPORTED;
    switch (most) {
        case 16: return launch<16>(map_w, map_x, prm, count, stream);
        case 64: return launch<64>(map_w, map_x, prm, count, stream);
        case 112: return launch<112>(map_w, map_x, prm, count, stream);
        default: return launch<208>(map_w, map_x, prm, count, stream);
    }
}
