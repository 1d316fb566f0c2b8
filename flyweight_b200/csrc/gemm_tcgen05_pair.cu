// bfloat16 matrix product for prompt-sized steps on CTA PAIRS (tcgen05 cta_group::2), sm_100a.
//
//   Y[t][f] = sum_k X[t][k] * W[f][k]
//
// Two CTAs of a cluster work on one tile of 256 features x 256 tokens per accumulator: each CTA
// holds 128 of the features (its half of operand A) and 128 of the tokens (its half of operand
// B) in shared memory, the leader CTA issues one tcgen05.mma.cta_group::2 (M = 256, N = 256,
// K = 16) that reads both halves of both operands, and each CTA's tensor memory receives the
// accumulator rows of its own 128 features for all 256 tokens.  Against the single-CTA kernel a
// CTA loads and reads half of the activations per MMA: that kernel's tensor pipe waits on shared-
// memory bandwidth (TMA fill plus operand reads exceed 128 B/clk), this one's does not.
//
// Per stage: both CTAs' producers fill their own shared memory by TMA (plain tile loads of this
// GPU's memory, one destination each) whose completion bytes are all counted on the LEADER's
// "full" barrier (the cta_group::2 form of the load allows the barrier to live in the pair's other
// CTA); the leader's MMA thread waits for that one barrier, issues the MMAs and commits with a
// cluster-wide arrive that frees the stage in both CTAs.
//
// The grid is one pair per two SMs and walks the tiles (tile p, p + pairs, ...): tensor memory holds
// two accumulators, so the epilogue warps of both CTAs store tile i while the tensor cores work on
// tile i + 1 and the ring never runs dry between tiles.  (A launch of one tile a pair left the tensor
// cores idle for the epilogue and the next CTA's start.)
//
// SwiGLU: a CTA's 128 rows of A are 64 gate rows f and the 64 up rows F + f that go with them (two
// boxes), so one accumulator holds both halves of 64 features, gate in lanes 0-63, up in lanes 64-127
// of the same column.  The warps of lane quarters q and q + 2 trade halves of every 16 columns through
// shared memory: the gate's warp finishes the first eight, the up's the other eight.
//
// Launched with programmatic stream serialisation like every kernel of the library; every mbarrier
// wait is bounded.
#include "tcgen05.cuh"

using namespace fwb;
using namespace fwb::tc5;

namespace {

constexpr int EPI_WARPS = 16;          // four per quarter of the TMEM lanes
constexpr int THREADS = 64 + 32 * EPI_WARPS;   // warp 0 producer, warp 1 MMA, then the epilogue warps
constexpr int SM_PAIRS = 148 / 2;
constexpr int A_BYTES = BM * BK * 2;                    // 16 KiB: this CTA's 128 rows of A
constexpr int TRADE_FLOATS = 8 * 32;                    // what a warp hands over of 16 columns
enum PairEpilogue : int { PAIR_F32 = 0, PAIR_BF16 = 1, PAIR_ADD_F32 = 2, PAIR_SWIGLU_BF16 = 3 };
// BN: tokens per tile, half of them in each CTA's shared memory
template <int BN>
struct PairTile {
    static constexpr int HALF_N = BN / 2;
    static constexpr int STAGE_BYTES = A_BYTES + HALF_N * BK * 2;
    static constexpr int STAGES = 192 * 1024 / STAGE_BYTES;
    static constexpr int TRADE_BYTES = 2 * EPI_WARPS * TRADE_FLOATS * 4;
    static constexpr int smem_bytes(bool gated) { return STAGES * STAGE_BYTES + (gated ? TRADE_BYTES : 0) + 1024 + 512; }
};

struct PairParams {
    void* y;
    int M, N, K, ldy;
    int up_row_offset;
    int gate_act;          // SwiGLU: the gate's activation (GATE_*); bf16 outputs: OUTPUT_*
    float gate_limit;
    int token_tiles, feature_tiles;
    int* status;
    // Grouped form: the rows of X are sorted by group (see fwb_gemm_tcgen05_grouped); group_tiles[0] token tiles,
    // then their (group, first row) pairs; a group's rows end at group_offsets[group + 1], its matrix begins
    // group * group_w_rows rows down W.
    const int* group_tiles;
    const int* group_offsets;
    int group_w_rows;
};

__device__ __forceinline__ void umma_bf16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                               uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrive (once all MMAs issued so far have completed) on the barrier at this offset in both CTAs.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
    const uint16_t mask = 3;
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
        ::"r"(smem_u32(bar)), "h"(mask)
        : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* holder, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(holder)),
                 "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t addr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
// Cluster-window address of `ptr`'s offset in CTA `rank`.
__device__ __forceinline__ uint32_t cluster_addr(const void* ptr, uint32_t rank) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(ptr)), "r"(rank));
    return remote;
}
// TMA tile load into this CTA's shared memory whose bytes are counted on a barrier that may live
// in the other CTA of the pair (given by its cluster-window address).
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, uint32_t bar_cluster_addr,
                                                 int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(bar_cluster_addr), "r"(x), "r"(y)
        : "memory");
}

// One arrival on the barrier at this cluster-window address.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}

template <int EPI, int BN, bool GROUPED>
__global__ void __launch_bounds__(THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                 const PairParams prm) {
    constexpr bool GATED = EPI == PAIR_SWIGLU_BF16;
    constexpr int CTA_FEATURES = GATED ? BM / 2 : BM;    // features a CTA has of a tile
    using T = PairTile<BN>;
    constexpr int STAGES = T::STAGES, STAGE_BYTES = T::STAGE_BYTES, HALF_N = T::HALF_N;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    float* trade = reinterpret_cast<float*>(tiles + STAGES * STAGE_BYTES);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(tiles + STAGES * STAGE_BYTES + (GATED ? T::TRADE_BYTES : 0));
    uint64_t* empty_bar = full_bar + STAGES;
    uint64_t* acc_full = empty_bar + STAGES;             // [2]: in both CTAs
    uint64_t* acc_empty = acc_full + 2;                  // [2]: the leader's, arrived on by both CTAs' epilogue warps
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 1);

    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();                // 0 = leader
    const int first_tile = blockIdx.x >> 1, tile_step = gridDim.x >> 1;
    const int n_kb = (prm.K + BK - 1) / BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 2 * EPI_WARPS);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc_pair(tmem_holder, 512);    // the same warp in both CTAs
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();          // both CTAs' barriers exist before anybody signals across
    tc_fence_after();
    const uint32_t tmem_base = *tmem_holder;

    // the list of token tiles is the work of an earlier kernel of this step: nothing is read before it is done
    if (GROUPED) pdl_wait();
    const int token_tiles = GROUPED ? prm.group_tiles[0] : prm.token_tiles;
    const int tiles_all = token_tiles * prm.feature_tiles;
    // token tiles are the fast index: pairs that run together share weight tiles in L2
    struct Place {
        int tok0, m_end, f, w_row;                       // first token, the rows' end, this CTA's first feature and row of W
    };
    auto place_of = [&](int tile) {
        Place at;
        const int token_tile = tile % token_tiles;
        at.f = (tile / token_tiles) * 2 * CTA_FEATURES + (int)rank * CTA_FEATURES;
        if (GROUPED) {
            const int group = prm.group_tiles[1 + 2 * token_tile];
            at.tok0 = prm.group_tiles[2 + 2 * token_tile];
            at.m_end = prm.group_offsets[group + 1];
            at.w_row = at.f + group * prm.group_w_rows;
        } else {
            at.tok0 = token_tile * BN;
            at.m_end = prm.M;
            at.w_row = at.f;
        }
        return at;
    };

    if (warp == 0) {
        if (lane == 0) {
            // every load of the pair reports to the leader's barrier of its stage; the leader arms it
            // with the bytes of both CTAs
            auto load_w = [&](int s, const Place& at, int kb) {
                uint8_t* stage = tiles + (size_t)s * STAGE_BYTES;
                const uint32_t bar = cluster_addr(&full_bar[s], 0);
                if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * STAGE_BYTES);
                tma_load_2d_pair(stage, &map_w, bar, kb * BK, at.w_row);
                if (GATED) tma_load_2d_pair(stage + A_BYTES / 2, &map_w, bar, kb * BK, prm.up_row_offset + at.w_row);
            };
            auto load_x = [&](int s, const Place& at, int kb) {
                tma_load_2d_pair(tiles + (size_t)s * STAGE_BYTES + A_BYTES, &map_x, cluster_addr(&full_bar[s], 0), kb * BK,
                                 at.tok0 + (int)rank * HALF_N);
            };
            const int ahead = first_tile >= tiles_all ? 0 : n_kb < STAGES ? n_kb : STAGES;
            if (ahead) {
                const Place at = place_of(first_tile);
                for (int i = 0; i < ahead; ++i) load_w(i, at, i);      // weights first: nothing in the stream writes them
                if (!GROUPED) pdl_wait();
                for (int i = 0; i < ahead; ++i) load_x(i, at, i);
            }
            int s = ahead % STAGES;
            uint32_t parity = ahead == STAGES ? 0 : 1;   // of the empty barrier; the ring's first round waits for nothing
            bool ok = true;
            for (int tile = first_tile; tile < tiles_all && ok; tile += tile_step) {
                const Place at = place_of(tile);
                for (int kb = tile == first_tile ? ahead : 0; kb < n_kb; ++kb) {
                    ok = mbar_wait(&empty_bar[s], parity, abort_flag, 11, prm.status);
                    if (!ok) break;
                    load_w(s, at, kb);
                    load_x(s, at, kb);
                    if (++s == STAGES) {
                        s = 0;
                        parity ^= 1;
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            constexpr uint32_t idesc = make_idesc_mn(2 * BM, BN);
            bool ok = true;
            int s = 0, turn = 0;
            uint32_t parity = 0;
            for (int tile = first_tile; tile < tiles_all && ok; tile += tile_step, ++turn) {
                const int b = turn & 1;
                // both CTAs' epilogues have read what this accumulator held two tiles ago
                if (turn >= 2) ok = mbar_wait_cluster(&acc_empty[b], ((turn >> 1) - 1) & 1, abort_flag, 17, prm.status);
                if (!ok) break;
                tc_fence_after();
                for (int kb = 0; kb < n_kb; ++kb) {
                    ok = mbar_wait_cluster(&full_bar[s], parity, abort_flag, 13, prm.status);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t stage = smem_u32(tiles + (size_t)s * STAGE_BYTES);
                    const uint64_t a_desc = make_smem_desc(stage), b_desc = make_smem_desc(stage + A_BYTES);
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k)
                        umma_bf16_pair(tmem_base + b * BN, a_desc + 2 * k, b_desc + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    umma_commit_pair(&empty_bar[s]);     // frees the stage in both CTAs
                    if (++s == STAGES) {
                        s = 0;
                        parity ^= 1;
                    }
                }
                umma_commit_pair(&acc_full[b]);          // accumulator complete, in both CTAs
            }
        }
    }
    __syncwarp();

    // ---------------------------------------------------------------- epilogue (both CTAs)
    if (warp >= 2) {
        if (!GROUPED) pdl_wait();
        const int quarter = warp & 3, group = (warp - 2) >> 2;
        const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
        constexpr int PER_GROUP = BN / (EPI_WARPS / 4);  // the warps of a quarter of the TMEM lanes share the token columns
        int turn = 0;
        for (int tile = first_tile; tile < tiles_all; tile += tile_step, ++turn) {
            const int b = turn & 1;
            bool ready = mbar_wait(&acc_full[b], (turn >> 1) & 1, abort_flag, 15, prm.status);
            // (after a wait that gave up nobody reads or stores, but everybody keeps meeting his partner's barriers)
            ready = __all_sync(0xffffffffu, ready && !*abort_flag);
            tc_fence_after();
            const Place at_tile = place_of(tile);
            const int tok0 = at_tile.tok0 + group * PER_GROUP, m_end = at_tile.m_end;
            const uint32_t from = lane_base + b * BN + group * PER_GROUP;
            if constexpr (GATED) {
                const bool up = quarter >= 2;
                const int f = at_tile.f + (quarter & 1) * 32 + lane;
                float* mine = trade + (size_t)(warp - 2) * TRADE_FLOATS + lane;
                const float* theirs = trade + (size_t)((warp - 2) ^ 2) * TRADE_FLOATS + lane;
                const int barrier = 1 + group * 2 + (quarter & 1);
#pragma unroll 1
                for (int c0 = 0; c0 < PER_GROUP; c0 += 16) {
                    float v[16] = {};
                    if (ready) tmem_ld16(from + c0, v);
                    const int buffer = (c0 >> 4 & 1) * EPI_WARPS * TRADE_FLOATS;
#pragma unroll
                    for (int j = 0; j < 8; ++j) mine[buffer + j * 32] = up ? v[j] : v[8 + j];
                    asm volatile("bar.sync %0, 64;" ::"r"(barrier) : "memory");
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float other = theirs[buffer + j * 32];
                        const float g = up ? other : v[j], u = up ? v[8 + j] : other;
                        const int t = tok0 + c0 + (up ? 8 : 0) + j;
                        if (ready && t < m_end && f < prm.N)
                            reinterpret_cast<__nv_bfloat16*>(prm.y)[(size_t)t * prm.ldy + f] =
                                __float2bfloat16_rn(gated_fast(prm.gate_act, prm.gate_limit, g, u));
                    }
                }
            } else {
                const int f = at_tile.f + quarter * 32 + lane;
#pragma unroll 1
                for (int c0 = 0; c0 < PER_GROUP && ready; c0 += 16) {
                    float v[16];
                    float sum[EPI == PAIR_ADD_F32 ? 16 : 1];
                    if constexpr (EPI == PAIR_ADD_F32) {          // Y += the product: asked for in front of the accumulator
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const int t = tok0 + c0 + j;
                            sum[j] = t < m_end && f < prm.N ? reinterpret_cast<const float*>(prm.y)[(size_t)t * prm.ldy + f] : 0.0f;
                        }
                    }
                    tmem_ld16(from + c0, v);
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const int t = tok0 + c0 + j;
                        if (t >= m_end || f >= prm.N) continue;
                        const size_t at = (size_t)t * prm.ldy + f;
                        if (EPI == PAIR_ADD_F32) reinterpret_cast<float*>(prm.y)[at] = v[j] + sum[EPI == PAIR_ADD_F32 ? j : 0];
                        else if (EPI == PAIR_F32) reinterpret_cast<float*>(prm.y)[at] = v[j];
                        else reinterpret_cast<__nv_bfloat16*>(prm.y)[at] = __float2bfloat16_rn(output_act_f32(prm.gate_act, v[j]));
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(cluster_addr(&acc_empty[b], 0));
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();          // neither CTA frees tensor memory or leaves while the other still works
    if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

template <int EPI, int BN, bool GROUPED>
int launch(const CUtensorMap& map_w, const CUtensorMap& map_x, const PairParams& prm, long most_tiles, cudaStream_t stream) {
    auto kernel = gemm_pair_kernel<EPI, BN, GROUPED>;
    constexpr int SMEM = PairTile<BN>::smem_bytes(EPI == PAIR_SWIGLU_BF16);
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(2 * (unsigned)(most_tiles < SM_PAIRS ? most_tiles : SM_PAIRS), 1, 1);
    config.blockDim = dim3(THREADS);
    config.dynamicSmemBytes = SMEM;
    config.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
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

// X: [M][K] bf16, W: [w_rows][K] bf16, Y: [M][ldy] fp32 (epilogues 0, 2) or bf16 (1, 3).
// epilogue: 0 = fp32, 1 = bf16 (an output activation in the bits above), 2 = fp32, Y += the product, 3 = SwiGLU (N = F, up rows at
// up_row_offset; the gate's activation in the bits above, its parameter in gate_limit).
// K % 8 == 0, bases 16-byte aligned.
FWB_API int fwb_gemm_tcgen05_pair(const void* X, const void* W, void* Y, int M, int N, int K, int w_rows,
                                  int ldy, int epilogue, int up_row_offset, float gate_limit, cudaStream_t stream) {
    const int gate_act = epilogue >> 8;     // bits above the epilogue code: the gate's, or a bf16 output's, activation
    epilogue &= 0xff;
    if (M <= 0 || N <= 0) return FWB_OK;
    if (!X || !W || !Y || K <= 0 || ldy < N) return FWB_BAD_ARGUMENT;
    if ((K & 7) || ((uintptr_t)X & 15) || ((uintptr_t)W & 15)) return FWB_UNSUPPORTED;
    const bool gated = epilogue == PAIR_SWIGLU_BF16;
    if (gated && (up_row_offset < N || w_rows < up_row_offset + N)) return FWB_BAD_ARGUMENT;
    if (!gated && w_rows < N) return FWB_BAD_ARGUMENT;
    PairParams prm;
    prm.y = Y;
    prm.M = M;
    prm.N = N;
    prm.K = K;
    prm.ldy = ldy;
    prm.up_row_offset = up_row_offset;
    prm.gate_act = gate_act;
    prm.gate_limit = gate_limit;
    prm.status = status_word();
    prm.group_tiles = prm.group_offsets = nullptr;
    prm.group_w_rows = 0;
    const int features = gated ? BM : 2 * BM;            // of a tile
    prm.feature_tiles = (N + features - 1) / features;
    // 128-token tiles where 256 would leave half of the pairs without one (1,024 features at 2,048 tokens)
    const bool narrow = (long)prm.feature_tiles * ((M + 255) / 256) * 2 <= SM_PAIRS;
    const int bn = narrow ? 128 : 256;
    prm.token_tiles = (M + bn - 1) / bn;
    const long tiles = (long)prm.token_tiles * prm.feature_tiles;
    if (tiles > 1073741823L) return FWB_TOO_LARGE;
    CUtensorMap map_w, map_x;
    if (!make_map(&map_w, W, w_rows, K, gated ? BM / 2 : BM)) return FWB_UNSUPPORTED;
    if (!make_map(&map_x, X, M, K, bn / 2)) return FWB_UNSUPPORTED;
    switch (epilogue) {
        case PAIR_F32:
            return narrow ? launch<PAIR_F32, 128, false>(map_w, map_x, prm, tiles, stream)
                          : launch<PAIR_F32, 256, false>(map_w, map_x, prm, tiles, stream);
        case PAIR_BF16:
            return narrow ? launch<PAIR_BF16, 128, false>(map_w, map_x, prm, tiles, stream)
                          : launch<PAIR_BF16, 256, false>(map_w, map_x, prm, tiles, stream);
        case PAIR_ADD_F32:
            return narrow ? launch<PAIR_ADD_F32, 128, false>(map_w, map_x, prm, tiles, stream)
                          : launch<PAIR_ADD_F32, 256, false>(map_w, map_x, prm, tiles, stream);
        case PAIR_SWIGLU_BF16:
            return narrow ? launch<PAIR_SWIGLU_BF16, 128, false>(map_w, map_x, prm, tiles, stream)
                          : launch<PAIR_SWIGLU_BF16, 256, false>(map_w, map_x, prm, tiles, stream);
        default: return FWB_UNSUPPORTED;
    }
}

// The grouped form of fwb_gemm_tcgen05_grouped (its arguments, checked there) for token tiles of 128 rows.
int fwb::tc5::gemm_pair_grouped(const void* X, const void* W, void* Y, const int* offsets, const int* tiles, int max_tiles,
                                int A, int N, int K, int n_groups, int group_w_rows, int ldy, int epilogue, int gate_act,
                                int up_row_offset, float gate_limit, cudaStream_t stream) {
    const bool gated = epilogue == PAIR_SWIGLU_BF16;
    PairParams prm;
    prm.y = Y;
    prm.M = A;
    prm.N = N;
    prm.K = K;
    prm.ldy = ldy;
    prm.up_row_offset = up_row_offset;
    prm.gate_act = gate_act;
    prm.gate_limit = gate_limit;
    prm.status = status_word();
    prm.group_tiles = tiles;
    prm.group_offsets = offsets;
    prm.group_w_rows = group_w_rows;
    const int features = gated ? BM : 2 * BM;
    prm.feature_tiles = (N + features - 1) / features;
    prm.token_tiles = max_tiles;
    const long most = (long)max_tiles * prm.feature_tiles;
    if (most > 1073741823L) return FWB_TOO_LARGE;
    CUtensorMap map_w, map_x;
    if (!make_map(&map_w, W, (long)n_groups * group_w_rows, K, gated ? BM / 2 : BM)) return FWB_UNSUPPORTED;
    if (!make_map(&map_x, X, A, K, 64)) return FWB_UNSUPPORTED;
    switch (epilogue) {
        case PAIR_F32: return launch<PAIR_F32, 128, true>(map_w, map_x, prm, most, stream);
        case PAIR_BF16: return launch<PAIR_BF16, 128, true>(map_w, map_x, prm, most, stream);
        default: return launch<PAIR_SWIGLU_BF16, 128, true>(map_w, map_x, prm, most, stream);
    }
}
