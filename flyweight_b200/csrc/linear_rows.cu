// Y[t][f] = sum_k X[t][k] * W[f][k] for a handful of tokens (decode steps): a weight reader.
//
// With so few tokens the product is bound by the weights' bytes when it runs alone, and inside a decode
// step -- some eighty dependent launches of a few microseconds each -- by what happens between the moment
// the activations are there and the moment the result is.  So nothing but the activations' own way stays
// behind griddepcontrol.wait: no tiles, no tensor memory, no cluster.
//
//   * A CTA owns `units` groups of eight features (for a gated product eight of the gate and the eight of
//     the up projection that go with them) over all of K; its eight warps cut K between them: per step of
//     the walk ("chunk") a warp takes KBLK adjacent 32-wide blocks.  No split of K over CTAs, so a sum, an
//     activation or a residual is finished where it is made.
//   * A ninth warp streams the weights through a ring in shared memory, row by row with bulk copies (a row's
//     piece is contiguous), from the kernel's first moment on: nothing in the stream writes weights.  Two
//     CTAs an SM: one ring an SM keeps 12 MB on the way, too little for HBM's latency under load (16384 x
//     2048, 8 tokens: 16.5 us with one, 11.1 with two; the bytes take 10.3), and the next kernel's CTAs
//     find room as soon as the first ones end.  Asking weights into L2 ahead of the ring was slower.
//   * mma.sync of 16 tokens x 8 features x 16 k; a lane's 16-byte read is eight k of one feature, and the k
//     of a block are dealt to the fragments' slots in that order for both operands.  Rows in shared memory
//     are 64 bytes apart modulo 128, which a quarter-warp's two rows need.
//   * Activations are read as A fragments from global memory, one chunk ahead; the NORMED form reads rows
//     of the fp32 residual, makes bf16(x * w) of them and keeps the rows' sums of squares for
//     the epilogue: (W (x w)) r = W (x w r).
//   * The warps' partial sums meet in shared memory and are added in warp order: the result does not depend on
//     how the features are cut over CTAs, nor on the number of tokens up to 16 (17 to 32 deal K to the warps in
//     shorter steps, which is another order of the same sums).
// Every wait on an mbarrier is bounded as in the tcgen05 products.
//
// Measured on B200 in a chain of launches over 300 MB of weights (us; tcgen05 kernel, this one; HBM time):
//   8 tokens   1024 x 1024  4.4 2.2 (0.3)   3072 x 1024  4.7 2.5 (1.0)   6144 x 2048  7.9 5.2 (3.8)
//              2048 x 8192 10.1 8.4 (5.1)  16384 x 2048 15.8 11.1 (10.3) 65536 x 2048 41.3 42.3 (41.0)
//  16 tokens   1024 x 1024  4.4 2.7         3072 x 1024  4.7 3.2         2048 x 8192 10.0 14.5
//  24 tokens   1024 x 1024  4.9 3.9         9216 x 1024 11.4 8.1         6144 x 2048  8.6 10.7
// (with more tokens every CTA reads more activations, so the tcgen05 kernel takes over as K and M grow)
#include "tcgen05.cuh"

using namespace fwb;
using namespace fwb::tc5;

namespace {

constexpr int WARPS = 8, THREADS = 32 * (WARPS + 1);
constexpr int SMEM_TARGET = 112 * 1024;        // two CTAs an SM
constexpr int MAX_SLOTS = 8;
constexpr long TWO_CTAS_FROM = 2 << 20;
// EPI_CONV: the rows are B | C | x of a gated short convolution, a token per request: three accumulators, and the
// epilogue is the convolution's step (csrc/shortconv.cu) on the bfloat16-rounded projections, state and all.
enum Epilogue : int { EPI_F32 = 0, EPI_BF16 = 1, EPI_ADD_F32 = 2, EPI_SWIGLU_BF16 = 3, EPI_CONV = 4 };
constexpr int accumulators_of(int epi) { return epi == EPI_CONV ? 3 : (epi == EPI_SWIGLU_BF16 ? 2 : 1); }

struct RowsParams {
    const __nv_bfloat16* x;      // [M][K], or
    const float* norm_x;         // NORMED: fp32 rows [.][K] (row t, or norm_rows[t])
    const float* norm_w;
    const int* norm_rows;
    float norm_eps;
    const __nv_bfloat16* w;      // [rows][K]
    void* y;                     // [M][ldy]
    const float* addend;         // [M][ldy] (may be y)
    int M, N, K, ldy;
    int up_row_offset, act;
    float limit;
    int units;                   // groups of eight features of one accumulator per CTA
    int slots;                   // depth of the ring
    int* status;
    // EPI_CONV: [N][conv_taps], [N] or null, a request's last conv_taps - 1 products at conv_slot[token] * conv_stride
    const float* conv_w;
    const float* conv_bias;
    float* conv_state;
    const int* conv_slot;
    long long conv_stride;
    int conv_taps;
};

__device__ __forceinline__ uint4 load_rows(const void* p) {     // written by the kernel before: not .nc
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void mma_16x8x16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                            uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// bytes between rows in shared memory: quarter-warps read two rows of 64 bytes each
__host__ __device__ constexpr int row_stride(int K) { return ((2 * K + 127) & ~127) + 64; }

// R8: groups of eight token rows.
template <int R8, int KBLK, int EPI, bool NORMED>
__global__ void __launch_bounds__(THREADS, 2) linear_rows_kernel(const RowsParams prm) {
    constexpr int NACC = accumulators_of(EPI);
    constexpr int MT = (R8 + 1) / 2;                   // 16-row tiles of the product
    constexpr int CHUNK = WARPS * KBLK * 32, W_STRIDE = row_stride(CHUNK), SLOT = 8 * W_STRIDE;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t full_bar[MAX_SLOTS], empty_bar[MAX_SLOTS];
    __shared__ int abort_word;
    __shared__ float squares[WARPS][8 * R8];           // NORMED: the warps' shares of the rows' sums of squares
    volatile int* abort_flag = &abort_word;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int all_units = (prm.N + 7) >> 3, slots = prm.slots;
    const int unit0 = blockIdx.x * prm.units;
    const int units = all_units - unit0 < prm.units ? all_units - unit0 : prm.units;
    const int groups = units * NACC, K = prm.K;
    const int chunks = (K + CHUNK - 1) / CHUNK, steps = chunks * groups;
    uint8_t* ring = smem;
    float* partial = reinterpret_cast<float*>(ring + slots * SLOT);                       // [warp][group][R8][32 lanes][2]
    float* norm_w = partial + WARPS * prm.units * NACC * R8 * 64;                         // [K], NORMED

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < slots; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], WARPS);
        }
        abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    int asked = 0;                                     // the weight warp's copies into the ring so far, eight rows each
    if (warp == WARPS) {
        // ---- weights
        int slot = 0, group = 0, k = 0;
        uint32_t parity = 1;                           // of the empty barrier: the ring's first round waits for nothing
        for (; asked < steps; ++asked) {
            // (the lanes poll each for itself and go on together: a vote, or one that gave up would leave the others behind)
            if (asked >= slots && !__all_sync(0xffffffffu, mbar_wait(&empty_bar[slot], parity, abort_flag, 21, prm.status)))
                break;
            const uint32_t bytes = (uint32_t)(K - k < CHUNK ? K - k : CHUNK) * 2;
            if (lane == 0) mbar_expect_tx(&full_bar[slot], 8 * bytes);
            __syncwarp();
            if (lane < 8) {
                const int feature = (unit0 + group / NACC) * 8 + lane;
                const size_t row = (feature < prm.N ? feature : prm.N - 1) + (size_t)(group % NACC) * prm.up_row_offset;
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(smem_u32(ring + slot * SLOT + lane * W_STRIDE)), "l"(prm.w + row * K + k), "r"(bytes),
                               "r"(smem_u32(&full_bar[slot])) : "memory");
            }
            if (++group == groups) group = 0, k += CHUNK;
            if (++slot == slots) slot = 0, parity ^= 1;
        }
    }
    if (NORMED && warp < WARPS) {
        // the norm's weight, a warp's own k only, while the kernel before this one still runs
#pragma unroll 4
        for (int k = warp * KBLK * 32 + lane * 4; k < K; k += CHUNK)
            *reinterpret_cast<float4*>(norm_w + k) = *reinterpret_cast<const float4*>(prm.norm_w + k);
        __syncwarp();
    }
    pdl_wait();

    if (warp < WARPS) {
        // ---- activations
        // as they lie in memory: 16 bytes of bf16, or (NORMED) 32 bytes of fp32
        constexpr int PIECES = NORMED ? 2 : 1;
        uint4 x_next[KBLK][R8][PIECES];
        const char* x_at[R8];
#pragma unroll
        for (int r = 0; r < R8; ++r) {
            const int row = g + 8 * r;
            if (row >= prm.M) x_at[r] = nullptr;
            else if (NORMED) x_at[r] = reinterpret_cast<const char*>(prm.norm_x + (size_t)(prm.norm_rows ? prm.norm_rows[row] : row) * K);
            else x_at[r] = reinterpret_cast<const char*>(prm.x + (size_t)row * K);
        }
        auto fetch_rows = [&](int k) {
#pragma unroll
            for (int b = 0; b < KBLK; ++b)
#pragma unroll
                for (int r = 0; r < R8; ++r)
#pragma unroll
                    for (int i = 0; i < PIECES; ++i)
                        x_next[b][r][i] = x_at[r] && k + b * 32 < K
                                              ? load_rows(x_at[r] + (size_t)(k + b * 32) * 2 * PIECES + 16 * i) : make_uint4(0, 0, 0, 0);
        };
        int x_k = warp * KBLK * 32 + t * 8;
        float square[R8];
#pragma unroll
        for (int r = 0; r < R8; ++r) square[r] = 0.0f;
        fetch_rows(x_k);

        // ---- the walk: chunk by chunk of K, in every chunk group by group of features
        int slot = 0, w_k = 0;
        uint32_t parity = 0;
        for (int chunk = 0; chunk < chunks; ++chunk) {
            uint4 xv[KBLK][R8];
#pragma unroll
            for (int b = 0; b < KBLK; ++b) {
                if constexpr (NORMED) {
                    float w[8] = {};
                    if (x_k + b * 32 < K) {
                        *reinterpret_cast<float4*>(w) = *reinterpret_cast<const float4*>(norm_w + x_k + b * 32);
                        *reinterpret_cast<float4*>(w + 4) = *reinterpret_cast<const float4*>(norm_w + x_k + b * 32 + 4);
                    }
#pragma unroll
                    for (int r = 0; r < R8; ++r) {
                        uint32_t packed[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint4 piece = x_next[b][r][PIECES == 2 ? i >> 1 : 0];
                            const float one = __uint_as_float(i & 1 ? piece.z : piece.x), two = __uint_as_float(i & 1 ? piece.w : piece.y);
                            square[r] = fmaf(one, one, square[r]);
                            square[r] = fmaf(two, two, square[r]);
                            __nv_bfloat162 h = __floats2bfloat162_rn(one * w[2 * i], two * w[2 * i + 1]);
                            packed[i] = *reinterpret_cast<uint32_t*>(&h);
                        }
                        xv[b][r] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
                    }
                } else {
#pragma unroll
                    for (int r = 0; r < R8; ++r) xv[b][r] = x_next[b][r][0];
                }
            }
            x_k += CHUNK;
            if (chunk + 1 < chunks) fetch_rows(x_k);
            const int live = K - w_k - warp * KBLK * 32 - t * 8;      // this lane's k below K, from its first one on
            for (int group = 0; group < groups; ++group) {
                // (nothing goes by the answer: after a wait that gave up every later one ends at its first poll, the sums
                // are worth nothing and nobody stores them.  A vote here costs 4 % of a decode step)
                mbar_wait(&full_bar[slot], parity, abort_flag, 22, prm.status);
                const uint8_t* from = ring + slot * SLOT + g * W_STRIDE + (warp * KBLK * 32 + t * 8) * 2;
                uint4 wv[KBLK];
#pragma unroll
                for (int b = 0; b < KBLK; ++b)
                    wv[b] = b * 32 < live ? *reinterpret_cast<const uint4*>(from + b * 64) : make_uint4(0, 0, 0, 0);
                __syncwarp();
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&empty_bar[slot])) : "memory");
                float acc[MT][2][4];
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[m][0][i] = acc[m][1][i] = 0.0f;
#pragma unroll
                for (int b = 0; b < KBLK; ++b)
#pragma unroll
                    for (int m = 0; m < MT; ++m) {
                        const uint4 one = xv[b][2 * m];
                        const uint4 two = 2 * m + 1 < R8 ? xv[b][2 * m + 1 < R8 ? 2 * m + 1 : 0] : make_uint4(0, 0, 0, 0);
                        mma_16x8x16(acc[m][0], one.x, two.x, one.y, two.y, wv[b].x, wv[b].y);
                        mma_16x8x16(acc[m][1], one.z, two.z, one.w, two.w, wv[b].z, wv[b].w);
                    }
                float2* mine = reinterpret_cast<float2*>(partial) + (size_t)((warp * prm.units * NACC + group) * R8) * 32 + lane;
#pragma unroll
                for (int r = 0; r < R8; ++r) {
                    float2 v = make_float2(acc[r / 2][0][(r & 1) * 2] + acc[r / 2][1][(r & 1) * 2],
                                           acc[r / 2][0][(r & 1) * 2 + 1] + acc[r / 2][1][(r & 1) * 2 + 1]);
                    if (chunk > 0) {
                        const float2 before = mine[r * 32];
                        v.x += before.x, v.y += before.y;
                    }
                    mine[r * 32] = v;
                }
                if (++slot == slots) slot = 0, parity ^= 1;
            }
            w_k += CHUNK;
        }
        if constexpr (NORMED) {
#pragma unroll
            for (int r = 0; r < R8; ++r) {
                float v = square[r];
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                if (t == 0) squares[warp][g + 8 * r] = v;
            }
        }
    }
    __syncthreads();
    if (*abort_flag) {
        // somebody gave up: the copies still in flight land before the block's shared memory is another's.  The slot's
        // last phase, for each slot, with a limit of its own (the abort flag would end mbar_wait at once)
        if (warp == WARPS && lane < slots && asked > lane) {
            const uint32_t last = (uint32_t)((asked - 1 - lane) / slots) & 1;
            for (unsigned spin = 0; spin < WAIT_LIMIT && !mbar_test(&full_bar[lane], last); ++spin) __nanosleep(64);
        }
        return;
    }

    // ---- the warps' sums together, and what the caller wants done with them
    const int width = units * 8;
    for (int i = threadIdx.x; i < width * prm.M; i += THREADS) {
        const int row = i / width, n = i - row * width, f = unit0 * 8 + n;
        if (f >= prm.N) continue;
        const size_t at = (size_t)row * prm.ldy + f;
        float add = 0.0f;
        if (EPI == EPI_ADD_F32) add = prm.addend[at];
        float sum[NACC], inv_rms = 1.0f;
        if constexpr (NORMED) {
            float sq = 0.0f;
#pragma unroll
            for (int wp = 0; wp < WARPS; ++wp) sq += squares[wp][row];
            inv_rms = rsqrtf(sq / (float)K + prm.norm_eps);
        }
#pragma unroll
        for (int a = 0; a < NACC; ++a) {
            const float* p = partial + (size_t)(((n >> 3) * NACC + a) * R8 + (row >> 3)) * 64 + ((row & 7) * 4 + ((n & 7) >> 1)) * 2 + (n & 1);
            float v = 0.0f;
#pragma unroll
            for (int wp = 0; wp < WARPS; ++wp) v += p[(size_t)wp * prm.units * NACC * R8 * 64];
            sum[a] = v * inv_rms;
        }
        if constexpr (EPI == EPI_CONV) {
            const int keep = prm.conv_taps - 1;
            const float b = __bfloat162float(__float2bfloat16_rn(sum[0])), c = __bfloat162float(__float2bfloat16_rn(sum[1]));
            const float u = b * __bfloat162float(__float2bfloat16_rn(sum[2]));
            const float* taps = prm.conv_w + (size_t)f * prm.conv_taps;
            float* kept = prm.conv_state + (size_t)prm.conv_slot[row] * prm.conv_stride + (size_t)f * keep;
            float v = prm.conv_bias ? prm.conv_bias[f] : 0.0f;
            for (int k = 0; k < keep; ++k) {
                const float old = kept[k];
                v = fmaf(taps[k], old, v);
                if (k > 0) kept[k - 1] = old;
            }
            kept[keep - 1] = u;
            v = fmaf(taps[keep], u, v);
            reinterpret_cast<__nv_bfloat16*>(prm.y)[at] = __float2bfloat16_rn(c * v);
        } else if (EPI == EPI_F32) reinterpret_cast<float*>(prm.y)[at] = sum[0];
        else if (EPI == EPI_ADD_F32) reinterpret_cast<float*>(prm.y)[at] = sum[0] + add;
        else if (EPI == EPI_BF16) reinterpret_cast<__nv_bfloat16*>(prm.y)[at] = __float2bfloat16_rn(output_act_f32(prm.act, sum[0]));
        else reinterpret_cast<__nv_bfloat16*>(prm.y)[at] = __float2bfloat16_rn(gated_fast(prm.act, prm.limit, sum[0], sum[NACC - 1]));
    }
}

template <int R8, int KBLK, int EPI, bool NORMED>
int launch(RowsParams prm, cudaStream_t stream) {
    constexpr int NACC = accumulators_of(EPI), SLOT = 8 * row_stride(WARPS * KBLK * 32);
    constexpr int MOST = 16 / (NACC * R8);             // units a CTA keeps partial sums of: 32 KiB
    const int all_units = (prm.N + 7) / 8;
    // two CTAs an SM, or as few more as the partial sums allow, evenly filled; one for a matrix that a single
    // ring an SM nearly holds
    int rounds = (long)prm.N * NACC * prm.K * 2 > TWO_CTAS_FROM ? 2 : 1;
    while ((all_units + 148 * rounds - 1) / (148 * rounds) > MOST) ++rounds;
    prm.units = (all_units + 148 * rounds - 1) / (148 * rounds);
    const int ctas = (all_units + prm.units - 1) / prm.units;
    const int fixed = WARPS * prm.units * NACC * R8 * 256 + (NORMED ? prm.K * 4 : 0);
    const int steps = prm.units * NACC * ((prm.K + WARPS * KBLK * 32 - 1) / (WARPS * KBLK * 32));
    int slots = (SMEM_TARGET - 2048 - fixed) / SLOT;
    slots = slots > MAX_SLOTS ? MAX_SLOTS : slots;
    slots = slots > steps ? steps : slots;
    prm.slots = slots < 3 ? 3 : slots;
    auto kernel = linear_rows_kernel<R8, KBLK, EPI, NORMED>;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    fwb::pdl(kernel, ctas, THREADS, fixed + prm.slots * SLOT, stream)(prm);
    return fwb_launch_status();
}

constexpr int MAX_ROWS = 32, MAX_NORMED_ROWS = 8, MAX_NORMED_K = 1024;    // normed: K in one chunk
constexpr int MAX_CONV_TAPS = 16;

template <int EPI, bool NORMED>
int launch_rows(const RowsParams& prm, cudaStream_t stream) {
    if constexpr (NORMED) return launch<1, 4, EPI, true>(prm, stream);
    else {
        if (prm.M > 16) return launch<4, 2, EPI, false>(prm, stream);
        if (prm.M > 8) return launch<2, 4, EPI, false>(prm, stream);
        return launch<1, 4, EPI, false>(prm, stream);
    }
}

bool shape_ok(const void* w, int M, int K, int most) { return M <= most && (K & 7) == 0 && ((uintptr_t)w & 15) == 0; }

}  // namespace

// X: [M][K] bf16, M <= 32; W: [rows][K] bf16; Y: [M][ldy].  Epilogues 0 fp32, 1 bf16 (with an output activation in
// the bits above the code), 2 fp32 + addend (which may be Y), 3 gated, as fwb_gemm_tcgen05.
FWB_API int fwb_linear_rows(const void* X, const void* W, void* Y, const float* addend, int M, int N, int K, int w_rows,
                            int ldy, int epilogue, int up_row_offset, float gate_limit, cudaStream_t stream) {
    const int act = epilogue >> 8;
    epilogue &= 0xff;
    if (M <= 0 || N <= 0) return FWB_OK;
    if (!X || !W || !Y || K <= 0 || ldy < N) return FWB_BAD_ARGUMENT;
    if (!shape_ok(W, M, K, MAX_ROWS) || ((uintptr_t)X & 15)) return FWB_UNSUPPORTED;
    if (epilogue == EPI_ADD_F32 && !addend) return FWB_BAD_ARGUMENT;
    if (epilogue == EPI_SWIGLU_BF16 && (up_row_offset < N || w_rows < up_row_offset + N)) return FWB_BAD_ARGUMENT;
    if (epilogue != EPI_SWIGLU_BF16 && w_rows < N) return FWB_BAD_ARGUMENT;
    const RowsParams prm{(const __nv_bfloat16*)X, nullptr, nullptr, nullptr, 0.0f, (const __nv_bfloat16*)W, Y, addend,
                         M, N, K, ldy, up_row_offset, act, gate_limit, 0, 0, status_word(),
                         nullptr, nullptr, nullptr, nullptr, 0, 0};
    switch (epilogue) {
        case EPI_F32: return launch_rows<EPI_F32, false>(prm, stream);
        case EPI_BF16: return launch_rows<EPI_BF16, false>(prm, stream);
        case EPI_ADD_F32: return launch_rows<EPI_ADD_F32, false>(prm, stream);
        case EPI_SWIGLU_BF16: return launch_rows<EPI_SWIGLU_BF16, false>(prm, stream);
        default: return FWB_UNSUPPORTED;
    }
}

// The same on RMS-normed rows of the fp32 residual (row t, or rows[t]), M <= 8: epilogues 0, 1, 3.
FWB_API int fwb_linear_rows_normed(const float* x_res, const float* norm_w, const int* rows, float eps, const void* W,
                                   void* Y, int M, int N, int K, int w_rows, int ldy, int epilogue, int up_row_offset,
                                   float gate_limit, cudaStream_t stream) {
    const int act = epilogue >> 8;
    epilogue &= 0xff;
    if (M <= 0 || N <= 0) return FWB_OK;
    if (!x_res || !norm_w || !W || !Y || K <= 0 || ldy < N) return FWB_BAD_ARGUMENT;
    if (!shape_ok(W, M, K, MAX_NORMED_ROWS) || ((uintptr_t)x_res & 15) || ((uintptr_t)norm_w & 15) || K > MAX_NORMED_K)
        return FWB_UNSUPPORTED;
    if (epilogue == EPI_SWIGLU_BF16 && (up_row_offset < N || w_rows < up_row_offset + N)) return FWB_BAD_ARGUMENT;
    if (epilogue != EPI_SWIGLU_BF16 && w_rows < N) return FWB_BAD_ARGUMENT;
    const RowsParams prm{nullptr, x_res, norm_w, rows, eps, (const __nv_bfloat16*)W, Y, nullptr,
                         M, N, K, ldy, up_row_offset, act, gate_limit, 0, 0, status_word(),
                         nullptr, nullptr, nullptr, nullptr, 0, 0};
    switch (epilogue) {
        case EPI_F32: return launch_rows<EPI_F32, true>(prm, stream);
        case EPI_BF16: return launch_rows<EPI_BF16, true>(prm, stream);
        case EPI_SWIGLU_BF16: return launch_rows<EPI_SWIGLU_BF16, true>(prm, stream);
        default: return FWB_UNSUPPORTED;
    }
}

// One step of a gated short convolution for requests of one token each (M <= 16, or 8 with the norm): in_proj rows B | C | x ([3H][K], H below one
// another) on X [M][K] bf16, or (norm_w given) on RMS-normed rows of the fp32 residual X, then
// z[t][c] = C (bias + sum_k taps[c][k] u) with u = B x behind the `conv_taps` - 1 products in slots[t], which move on.
// The projections are rounded to bfloat16 in between: the bits of fwb_linear_rows and fwb_shortconv.
FWB_API int fwb_linear_rows_conv(const void* X, const float* norm_w, float eps, const void* W, const float* conv_w,
                                 const float* conv_bias, float* state, long long state_stride, const int* slots, void* z,
                                 int M, int H, int K, int conv_taps, cudaStream_t stream) {
    if (M <= 0 || H <= 0) return FWB_OK;
    if (!X || !W || !conv_w || !state || !slots || !z || K <= 0) return FWB_BAD_ARGUMENT;
    if (conv_taps < 2 || conv_taps > MAX_CONV_TAPS) return FWB_UNSUPPORTED;       // as fwb_shortconv
    if (state_stride < (long long)H * (conv_taps - 1)) return FWB_BAD_ARGUMENT;
    if (!shape_ok(W, M, K, norm_w ? MAX_NORMED_ROWS : 16) || ((uintptr_t)X & 15)) return FWB_UNSUPPORTED;
    if (norm_w && (((uintptr_t)norm_w & 15) || K > MAX_NORMED_K)) return FWB_UNSUPPORTED;
    const RowsParams prm{(const __nv_bfloat16*)X, (const float*)X, norm_w, nullptr, eps, (const __nv_bfloat16*)W, z, nullptr,
                         M, H, K, H, H, 0, 0.0f, 0, 0, status_word(),
                         conv_w, conv_bias, state, slots, state_stride, conv_taps};
    if (norm_w) return launch<1, 4, EPI_CONV, true>(prm, stream);
    return M > 8 ? launch<2, 4, EPI_CONV, false>(prm, stream) : launch<1, 4, EPI_CONV, false>(prm, stream);
}
