// Y[M][N] = X[M][K] * W[N][K]^T (+ addend): the entry point of the true 32-bit matrix product, and the fallback of the
// bfloat16 path for shapes the tensor-core kernel refuses.  Any M, N, K >= 1.  The order in which an output element's
// products are added depends on the kernel alone, and which kernel runs on the types, N, K, ldx and the operands' alignment
// alone: the value at [m][n] does not depend on M or on which other rows share the launch.
//
//   gemm_f32_tcgen05.cu   fp32 throughout, 16-byte copies, N and K from 128 and N K from 2^20 on:
//                     exact thirds of the values on the tensor cores, closer to the exact sum than the
//                     others, which are plain multiply-adds.
//   gemm_f32_kernel   fp32 throughout, rows that 16-byte copies can read (K, ldx multiples of 4):
//                     eight partial sums an element (four quarters of every 64 k, even and odd k
//                     apart), added in a fixed order.
//   gemm_simt_kernel  everything else: one accumulator that walks k = 0..K-1.
#include "common.cuh"
#include "gemm_f32.cuh"

using namespace fwb;

namespace {

constexpr int TM = 64, TN = 64, TK = 16;

template <typename TX, typename TW, typename TY>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TX* __restrict__ X, const TW* __restrict__ W, TY* __restrict__ Y,
                 const float* __restrict__ addend, int M, int N, int K, int ldx, int ldy) {
    fwb::pdl_entry();
    __shared__ float xs[TK][TM + 4];
    __shared__ float ws[TK][TN + 4];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    const int tm = (tid / 16) * 4, tn = (tid % 16) * 4;
    const int lrow = tid / 4, lk = (tid % 4) * 4;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;

    for (int k0 = 0; k0 < K; k0 += TK) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = k0 + lk + j;
            const int m = m0 + lrow, n = n0 + lrow;
            xs[lk + j][lrow] = (m < M && k < K) ? to_f32<TX>(X[(size_t)m * ldx + k]) : 0.0f;
            ws[lk + j][lrow] = (n < N && k < K) ? to_f32<TW>(W[(size_t)n * K + k]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < TK; ++k) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = xs[k][tm + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = ws[k][tn + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + tm + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tn + j;
            if (n >= N) continue;
            float v = acc[i][j];
            if (addend) v += addend[(size_t)m * ldy + n];
            Y[(size_t)m * ldy + n] = from_f32<TY>(v);
        }
    }
}

// ---- fp32 operands in 16-byte pieces --------------------------------------------------------
// Bound by the fp32 pipes from a few dozen rows on and by the weights' bytes below.  Both operands are
// K-major, so they go to shared memory as they lie, by asynchronous 16-byte copies, three stages of
// 64 k deep, and a thread reads four consecutive k of a row at once.  Rows are 68 floats apart, which
// puts the eight rows that neighbouring lanes read on different banks.  An accumulator is a pair: even k and
// odd k, plain multiply-adds (packed ones, fma.rn.f32x2, gave the same bits and took 1.6 times as long for
// 201 x 1024 x 4608).  Four groups of 64 threads take 16 of the 64 k of every stage each: an output tile of
// 64 x 32 keeps eight warps busy, and a 201 x 1024 product fills 128 SMs.
// Measured on B200 in a chain of launches over 300 MB of weights (us; gemm_simt_kernel, then this one):
// 201 x 9216 x 1024 288 -> 121, 201 x 1024 x 4608 378 -> 76, 64 x 9216 x 1024 100 -> 39 (31 TFLOP/s),
// 8 x 1024 x 4608 403 -> 35, 1 x 9216 x 1024 94 -> 21 (matrices of that
// size have gone to the tensor cores since); relative error against 64 bits 5.7e-7 -> 2.1e-7 at K = 1024.
constexpr int FK = 64, FSTRIDE = FK + 4, FSTAGES = 3;

__device__ __forceinline__ void fma_four(float2& acc, const float4& a, const float4& b) {
    acc.x = fmaf(a.x, b.x, acc.x);
    acc.y = fmaf(a.y, b.y, acc.y);
    acc.x = fmaf(a.z, b.z, acc.x);
    acc.y = fmaf(a.w, b.w, acc.y);
}

template <int RM, int RN>
constexpr int f32_smem_bytes() {
    constexpr int ring = FSTAGES * 8 * (RM + RN) * FSTRIDE, partial = 3 * 8 * RM * (8 * RN + 4);
    return (ring > partial ? ring : partial) * 4;
}

// A tile of 8 RM rows x 8 RN columns; a thread of a group owns rows (lane & 7) + 8 i and columns (id / 8) + 8 j.
template <int RM, int RN, int PER_SM>
__global__ void __launch_bounds__(256, PER_SM)
gemm_f32_kernel(const float* __restrict__ X, const float* __restrict__ W, float* Y, const float* addend,
                int M, int N, int K, int ldx, int ldy) {
    constexpr int BM = 8 * RM, BN = 8 * RN, STAGE = (BM + BN) * FSTRIDE;
    constexpr int PROW = BN + 4;               // rows of a partial tile: a warp's 8 rows x 4 columns on 32 banks
    extern __shared__ __align__(16) float smem[];
    fwb::pdl_entry();
    const int tid = threadIdx.x, group = tid >> 6, id = tid & 63, tm = id & 7, tn = id >> 3;
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int chunks = (K + FK - 1) / FK;

    auto fetch = [&](int chunk) {
        if (chunk < chunks) {
            float* stage = smem + (chunk % FSTAGES) * STAGE;
            const int k0 = chunk * FK;
#pragma unroll
            for (int i = 0; i < (BM + BN) * (FK / 4); i += 256) {
                const int piece = i + tid, row = piece >> 4, k = k0 + (piece & 15) * 4;
                if ((BM + BN) * (FK / 4) % 256 != 0 && row >= BM + BN) break;
                const bool is_x = row < BM;
                const int at = is_x ? m0 + row : n0 + row - BM;
                const bool in = k < K && at < (is_x ? M : N);       // K is a multiple of 4: a piece is whole or absent
                const float* src = is_x ? X + (in ? (size_t)at * ldx + k : 0) : W + (in ? (size_t)at * K + k : 0);
                const uint32_t dst = (uint32_t)__cvta_generic_to_shared(stage + row * FSTRIDE + (piece & 15) * 4);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0)
                             : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float2 acc[RM][RN];
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN; ++j) acc[i][j] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int s = 0; s < FSTAGES - 1; ++s) fetch(s);
    for (int c = 0; c < chunks; ++c) {
        asm volatile("cp.async.wait_group %0;" ::"n"(FSTAGES - 2) : "memory");
        __syncthreads();                       // chunk c has landed for everybody; chunk c - 1 is read by nobody
        fetch(c + FSTAGES - 1);
        const float* xs = smem + (c % FSTAGES) * STAGE + tm * FSTRIDE + group * 16;
        const float* ws = smem + (c % FSTAGES) * STAGE + (BM + tn) * FSTRIDE + group * 16;
#pragma unroll
        for (int k = 0; k < 16; k += 4) {
            float4 a[RM], b[RN];
#pragma unroll
            for (int i = 0; i < RM; ++i) a[i] = *reinterpret_cast<const float4*>(xs + i * 8 * FSTRIDE + k);
#pragma unroll
            for (int j = 0; j < RN; ++j) b[j] = *reinterpret_cast<const float4*>(ws + j * 8 * FSTRIDE + k);
#pragma unroll
            for (int i = 0; i < RM; ++i)
#pragma unroll
                for (int j = 0; j < RN; ++j) fma_four(acc[i][j], a[i], b[j]);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                           // the ring is free: the groups' partial tiles go there
    if (group > 0) {
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < RN; ++j) smem[(group - 1) * BM * PROW + (tm + 8 * i) * PROW + tn + 8 * j] = acc[i][j].x + acc[i][j].y;
    }
    __syncthreads();
    if (group == 0) {
#pragma unroll
        for (int i = 0; i < RM; ++i)
#pragma unroll
            for (int j = 0; j < RN; ++j) {
                const int at = (tm + 8 * i) * PROW + tn + 8 * j;
                smem[at] = (((acc[i][j].x + acc[i][j].y) + smem[at]) + smem[BM * PROW + at]) + smem[2 * BM * PROW + at];
            }
    }
    __syncthreads();
    for (int at = tid; at < BM * BN; at += 256) {
        const int m = m0 + at / BN, n = n0 + at % BN;
        if (m >= M || n >= N) continue;
        float v = smem[at / BN * PROW + at % BN];
        if (addend) v += addend[(size_t)m * ldy + n];
        Y[(size_t)m * ldy + n] = v;
    }
}

template <int RM, int RN, int PER_SM>
int launch_f32(const float* X, const float* W, float* Y, const float* addend, int M, int N, int K, int ldx, int ldy,
               cudaStream_t stream) {
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_kernel<RM, RN, PER_SM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             f32_smem_bytes<RM, RN>());
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const dim3 grid((M + 8 * RM - 1) / (8 * RM), (N + 8 * RN - 1) / (8 * RN));
    if (grid.y > 65535) return FWB_TOO_LARGE;
    fwb::pdl(gemm_f32_kernel<RM, RN, PER_SM>, grid, 256, f32_smem_bytes<RM, RN>(), stream)(X, W, Y, addend, M, N, K, ldx, ldy);
    return fwb_launch_status();
}

// The tile: 16 or 32 rows for as few tokens; else 40 to 64 rows by 64 or 32 columns, whichever takes the least time by
// rounds over the SMs: 201 rows are four tiles of 56 or of 64.  A tile's time goes with its products and a constant
// (64 x 64: 143 us for four rounds at K = 1,024; 64 x 32: 25 us for one, 60 us for three).
int dispatch_f32(const float* X, const float* W, float* Y, const float* addend, int M, int N, int K, int ldx, int ldy,
                 cudaStream_t stream) {
    if (M <= 16) return launch_f32<2, 2, 2>(X, W, Y, addend, M, N, K, ldx, ldy, stream);
    if (M <= 32) return launch_f32<4, 4, 2>(X, W, Y, addend, M, N, K, ldx, ldy, stream);
    int rm = 8, rn = 8;
    bool alone = true;                         // a tile has an SM to itself: all the registers a thread can use
    long best = -1;
    for (int r = 8; r >= 5; --r)
        for (int c = 8; c >= 4; c -= 4) {
            const long tiles = (long)((M + 8 * r - 1) / (8 * r)) * ((N + 8 * c - 1) / (8 * c));
            const long cost = ((tiles + 147) / 148) * (r * c + 12);
            if (best < 0 || cost < best) best = cost, rm = r, rn = c, alone = c == 8 || tiles <= 148;
        }
#define FWB_F32(RM)                                                                                        \
    if (rm == RM)                                                                                          \
        return rn == 8 ? launch_f32<RM, 8, 1>(X, W, Y, addend, M, N, K, ldx, ldy, stream)                  \
               : alone ? launch_f32<RM, 4, 1>(X, W, Y, addend, M, N, K, ldx, ldy, stream)                  \
                       : launch_f32<RM, 4, 2>(X, W, Y, addend, M, N, K, ldx, ldy, stream)
    FWB_F32(8);
    FWB_F32(7);
    FWB_F32(6);
    FWB_F32(5);
#undef FWB_F32
    return FWB_UNSUPPORTED;
}

template <typename TX, typename TW, typename TY>
int launch(const void* X, const void* W, void* Y, const float* addend, int M, int N, int K, int ldx,
           int ldy, cudaStream_t stream) {
    dim3 grid((N + TN - 1) / TN, (M + TM - 1) / TM);
    if (grid.y > 65535) return FWB_TOO_LARGE;
    fwb::pdl(gemm_simt_kernel<TX, TW, TY>, grid, 256, 0, stream)((const TX*)X, (const TW*)W, (TY*)Y,
                                                           addend, M, N, K, ldx, ldy);
    return fwb_launch_status();
}

}  // namespace

// Dtype flags: 0 = float32, 1 = bfloat16.  `addend` (fp32, same layout as a fp32 Y,
// may alias Y) is added before the store; it needs y_bf16 == 0.
FWB_API int fwb_gemm_simt(const void* X, int x_bf16, const void* W, int w_bf16, void* Y, int y_bf16,
                          const float* addend, int M, int N, int K, int ldx, int ldy,
                          cudaStream_t stream) {
    if (M <= 0 || N <= 0) return FWB_OK;
    if (!X || !W || !Y || K <= 0 || ldx < K || ldy < N) return FWB_BAD_ARGUMENT;
    if (addend && y_bf16) return FWB_UNSUPPORTED;
    using bf = __nv_bfloat16;
    const int key = (x_bf16 ? 4 : 0) | (w_bf16 ? 2 : 0) | (y_bf16 ? 1 : 0);
    switch (key) {
        case 0:
            if (!(K & 3) && !(ldx & 3) && !((uintptr_t)X & 15) && !((uintptr_t)W & 15) && gemm_f32_split_takes(N, K))
                return gemm_f32_split((const float*)X, (const float*)W, (float*)Y, addend, M, N, K, ldx, ldy, stream);
            if (!(K & 3) && !(ldx & 3) && !((uintptr_t)X & 15) && !((uintptr_t)W & 15) && N <= 16 * 65535)
                return dispatch_f32((const float*)X, (const float*)W, (float*)Y, addend, M, N, K, ldx, ldy, stream);
            return launch<float, float, float>(X, W, Y, addend, M, N, K, ldx, ldy, stream);
        case 2: return launch<float, bf, float>(X, W, Y, addend, M, N, K, ldx, ldy, stream);
        case 4: return launch<bf, float, float>(X, W, Y, addend, M, N, K, ldx, ldy, stream);
        case 6: return launch<bf, bf, float>(X, W, Y, addend, M, N, K, ldx, ldy, stream);
        case 7: return launch<bf, bf, bf>(X, W, Y, addend, M, N, K, ldx, ldy, stream);
        case 5: return launch<bf, float, bf>(X, W, Y, addend, M, N, K, ldx, ldy, stream);
        default: return FWB_UNSUPPORTED;
    }
}
