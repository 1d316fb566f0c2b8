// Causal grouped-query attention over the paged cache, plain SIMT, fp32 arithmetic.
//
// A block walks the keys that its tokens may see, lo..pos (lo = max(0, pos-window+1) with a window, else 0;
// with `keep` also the positions below it) in tiles of 32 positions that start at multiples of 32, stages each
// K and V tile in shared memory once, and lets its warps run an online softmax for the query heads of one KV
// head.  A tile never straddles a page (the page size is a multiple of 32).  The walk and the reduction order
// depend only on the token's own position, never on how the batch was cut, so the result for a token is the
// same in a whole prompt, in a portion, or as a single decoded token.
//
//   attention_f32_kernel   32 bits throughout, head sizes of whole 16-byte pieces: the tokens of a segment in
//                          runs of up to eight, a warp a token and up to four heads.
//   attention_simt_kernel  a block a token: the fallback of the bfloat16 path for head sizes or group sizes
//                          that the tensor-core kernels refuse, and odd head sizes.
#include "common.cuh"

using namespace fwb;

namespace {

constexpr int WARPS = 4;
constexpr int TILE = 32;
constexpr int MAX_HPW = 4;   // query heads per warp  -> 16 heads of a group per block (larger groups: more blocks)
constexpr int MAX_DPL = 8;   // head channels per lane -> head size <= 256

template <typename TQ, typename TC, typename TO>
__global__ void __launch_bounds__(WARPS * 32)
attention_simt_kernel(const TQ* __restrict__ q, const TC* __restrict__ k_pool,
                      const TC* __restrict__ v_pool, const int* __restrict__ positions,
                      const int* __restrict__ tok_seg, const int* __restrict__ block_table,
                      int max_pages, int page_size, TO* __restrict__ out, int nh, int nkv, int hd,
                      int window, float scale, const float* __restrict__ sink, float softcap, int keep) {
    fwb::pdl_entry();
    extern __shared__ float smem[];
    const int group = nh / nkv;
    // a block takes up to WARPS * MAX_HPW query heads of its KV head; a larger group is cut over blockIdx.z
    const int g0 = blockIdx.z * (WARPS * MAX_HPW);
    const int mine = group - g0 < WARPS * MAX_HPW ? group - g0 : WARPS * MAX_HPW;
    float* qs = smem;                         // [mine][hd]
    float* ks = qs + mine * hd;               // [TILE][hd+1]
    float* vs = ks + TILE * (hd + 1);         // [TILE][hd]
    const int t = blockIdx.x, kvh = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pos = positions[t];
    const int* table = block_table + (size_t)tok_seg[t] * max_pages;
    const int lo = fwb::first_visible_key(pos, window);

    for (int i = threadIdx.x; i < mine * hd; i += blockDim.x)
        qs[i] = to_f32<TQ>(q[((size_t)t * nh + (size_t)kvh * group + g0) * hd + i]);

    float m[MAX_HPW], l[MAX_HPW], acc[MAX_HPW][MAX_DPL];
#pragma unroll
    for (int a = 0; a < MAX_HPW; ++a) {
        // a sink: a key of score sink[head] (not scaled, not capped) whose value is zero starts the row
        const int g = warp + a * WARPS;
        const bool sunk = sink != nullptr && g < mine;
        m[a] = sunk ? sink[kvh * group + g0 + g] : -INFINITY;
        l[a] = sunk ? 1.0f : 0.0f;
#pragma unroll
        for (int d = 0; d < MAX_DPL; ++d) acc[a][d] = 0.0f;
    }
    const float inv_cap = softcap > 0.0f ? 1.0f / softcap : 0.0f;

    const KeyTiles walk = fwb::key_tiles(lo, pos, keep, TILE);
    for (int tile = 0; tile < walk.count; ++tile) {
        const int base = walk.at(tile) * TILE;
        __syncthreads();
        const int page = table[base / page_size];
        const size_t src = (((size_t)page * nkv + kvh) * page_size + (base % page_size)) * hd;
        const int valid = pos - base + 1 < TILE ? pos - base + 1 : TILE;   // rows of the tile in use
        for (int i = threadIdx.x; i < TILE * hd; i += blockDim.x) {
            const int r = i / hd, c = i - r * hd;
            const bool live = r < valid;
            ks[r * (hd + 1) + c] = live ? to_f32<TC>(k_pool[src + i]) : 0.0f;
            vs[i] = live ? to_f32<TC>(v_pool[src + i]) : 0.0f;
        }
        __syncthreads();
        const int kpos = base + lane;
        const bool seen = (kpos >= lo || kpos < keep) && kpos <= pos;
#pragma unroll
        for (int a = 0; a < MAX_HPW; ++a) {
            const int g = warp + a * WARPS;
            if (g >= mine) break;
            const float* qh = qs + g * hd;
            const float* kr = ks + lane * (hd + 1);
            float s = 0.0f;
            for (int d = 0; d < hd; ++d) s = fmaf(qh[d], kr[d], s);
            s *= scale;
            if (softcap > 0.0f) s = softcap * tanhf(s * inv_cap);
            s = seen ? s : -INFINITY;
            const float tile_max = warp_max(s);
            if (tile_max == -INFINITY) continue;   // nothing visible in this tile (warp-uniform)
            const float m_new = fmaxf(m[a], tile_max);
            const float p = seen ? expf(s - m_new) : 0.0f;
            const float corr = expf(m[a] - m_new);  // m[a] == -inf gives 0
            l[a] = l[a] * corr + warp_sum(p);
            m[a] = m_new;
#pragma unroll
            for (int d = 0; d < MAX_DPL; ++d) acc[a][d] *= corr;
            for (int j = 0; j < valid; ++j) {
                const float pj = __shfl_sync(0xffffffffu, p, j);
#pragma unroll
                for (int d = 0; d < MAX_DPL; ++d) {
                    const int c = lane + 32 * d;
                    if (c < hd) acc[a][d] = fmaf(pj, vs[j * hd + c], acc[a][d]);
                }
            }
        }
    }
#pragma unroll
    for (int a = 0; a < MAX_HPW; ++a) {
        const int g = warp + a * WARPS;
        if (g >= mine) break;
        const float inv = 1.0f / l[a];
        TO* dst = out + ((size_t)t * nh + (size_t)kvh * group + g0 + g) * hd;
#pragma unroll
        for (int d = 0; d < MAX_DPL; ++d) {
            const int c = lane + 32 * d;
            if (c < hd) dst[c] = from_f32<TO>(acc[a][d] * inv);
        }
    }
}

// ---- fp32, 16-byte pieces ---------------------------------------------------------------------
// Same sums in the same order as attention_simt_kernel.  The work is small (201 tokens of 16 heads: 42 million
// multiply-adds) and that kernel spends its time on staging every tile once a token, a value at a time, and on two
// reads of shared memory a multiply-add; here a tile serves a run of tokens, comes by 16-byte copies one tile ahead,
// and a key is read once for all heads of a warp.
// Tokens are cut into runs where their index is a multiple of the run's length and where a token does not stand next to
// the one before it in its sequence; a block whose token begins no run ends at once, so single decoded tokens keep a block
// each.  That block gives up to four heads to one warp and leaves the others to copy, and is the faster one for it: a decoded
// token, us, block a token then this, head size 64 and groups of 2 | 4: 1 x 1,000 keys 402 90 | 404 152, 1 x 8,000 2,999 660 |
// 3,004 1,129, 8 x 8,000 2,915 664 | 2,922 1,135; head size 128, 8 x 8,000 5,495 754 | 5,500 989.
constexpr int F32_WARPS = 8;

template <int HPW, int DPL>              // heads a warp, head channels a lane
__global__ void __launch_bounds__(F32_WARPS * 32)
attention_f32_kernel(const float* __restrict__ q, const float* __restrict__ k_pool, const float* __restrict__ v_pool,
                     const int* __restrict__ positions, const int* __restrict__ tok_seg,
                     const int* __restrict__ block_table, int max_pages, int page_size, float* __restrict__ out, int T,
                     int nh, int nkv, int hd, int window, float scale, const float* __restrict__ sink, float softcap, int keep) {
    fwb::pdl_entry();
    extern __shared__ __align__(16) float smem[];
    const int group = nh / nkv, g0 = blockIdx.z * (WARPS * MAX_HPW);
    const int mine = group - g0 < WARPS * MAX_HPW ? group - g0 : WARPS * MAX_HPW;
    const int warps_a_token = (mine + HPW - 1) / HPW, run = F32_WARPS / warps_a_token;
    const int t0 = blockIdx.x, kvh = blockIdx.y, seg = tok_seg[t0];
    auto goes_on = [&](int t) { return tok_seg[t] == tok_seg[t - 1] && positions[t] == positions[t - 1] + 1; };
    if (t0 % run != 0 && goes_on(t0)) return;
    int n = 1;
    while ((t0 + n) % run != 0 && t0 + n < T && goes_on(t0 + n)) ++n;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int hd4 = hd >> 2, k_row = hd + 4, buffer = TILE * (k_row + hd);
    float* qs = smem + 2 * buffer;                       // [n][mine][hd]
    float* ps = qs + run * mine * hd + warp * HPW * TILE;           // [HPW][TILE]
    const int ti = warp / warps_a_token, h0 = warp % warps_a_token * HPW;
    const bool active = ti < n;
    const int pos = active ? positions[t0 + ti] : -1, last = positions[t0 + n - 1];
    const int lo = fwb::first_visible_key(pos < 0 ? 0 : pos, window);
    const int* table = block_table + (size_t)seg * max_pages;
    const KeyTiles walk = fwb::key_tiles(fwb::first_visible_key(positions[t0], window), last, keep, TILE);

    auto fetch = [&](int tile) {
        if (tile < walk.count) {
            const int base = walk.at(tile) * TILE;
            const size_t src = (((size_t)table[base / page_size] * nkv + kvh) * page_size + (base % page_size)) * hd;
            float* ks = smem + (tile & 1) * buffer;
            for (int r = warp; r < TILE; r += F32_WARPS)
                for (int c = lane; c < 2 * hd4; c += 32) {
                    const bool is_v = c >= hd4;
                    const int at = is_v ? c - hd4 : c;
                    float* dst = ks + (is_v ? TILE * k_row + r * hd : r * k_row) + at * 4;
                    const float* from = (is_v ? v_pool : k_pool) + src + (size_t)r * hd + at * 4;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                                 ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(from), "r"(base + r <= last ? 16 : 0)
                                 : "memory");
                }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0);
    for (int i = threadIdx.x; i < n * mine * hd4; i += F32_WARPS * 32) {
        const int row = i / hd4;
        reinterpret_cast<float4*>(qs)[i] = reinterpret_cast<const float4*>(
            q + ((size_t)(t0 + row / mine) * nh + (size_t)kvh * group + g0 + row % mine) * hd)[i - row * hd4];
    }

    float m[HPW], l[HPW], acc[HPW][DPL];
#pragma unroll
    for (int a = 0; a < HPW; ++a) {
        // a sink: a key of score sink[head] (not scaled, not capped) whose value is zero starts the row
        const bool sunk = sink != nullptr && h0 + a < mine;
        m[a] = sunk ? sink[kvh * group + g0 + h0 + a] : -INFINITY;
        l[a] = sunk ? 1.0f : 0.0f;
#pragma unroll
        for (int d = 0; d < DPL; ++d) acc[a][d] = 0.0f;
    }
    const float inv_cap = softcap > 0.0f ? 1.0f / softcap : 0.0f;
    const float4* my_q[HPW];
#pragma unroll
    for (int a = 0; a < HPW; ++a)                        // (heads past the last one repeat it and are not stored)
        my_q[a] = reinterpret_cast<const float4*>(qs) + (size_t)((active ? ti : 0) * mine + (h0 + a < mine ? h0 + a : mine - 1)) * hd4;

    for (int tile = 0; tile < walk.count; ++tile) {
        fetch(tile + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const int base = walk.at(tile) * TILE, kpos = base + lane;
        const int valid = pos - base + 1 < TILE ? pos - base + 1 : TILE;       // rows of the tile that this token may see
        const bool seen = (kpos >= lo || kpos < keep) && kpos <= pos;
        if (__any_sync(0xffffffffu, seen)) {
            const float* ks = smem + (tile & 1) * buffer;
            const float* vs = ks + TILE * k_row;
            const float4* kr = reinterpret_cast<const float4*>(ks + lane * k_row);
            float s[HPW];
#pragma unroll
            for (int a = 0; a < HPW; ++a) s[a] = 0.0f;
#pragma unroll 4
            for (int d = 0; d < hd4; ++d) {
                const float4 k = kr[d];
#pragma unroll
                for (int a = 0; a < HPW; ++a) {
                    const float4 x = my_q[a][d];
                    s[a] = fmaf(x.x, k.x, s[a]);
                    s[a] = fmaf(x.y, k.y, s[a]);
                    s[a] = fmaf(x.z, k.z, s[a]);
                    s[a] = fmaf(x.w, k.w, s[a]);
                }
            }
            bool live[HPW];
            __syncwarp();                                // the probabilities of the tile before are read
#pragma unroll
            for (int a = 0; a < HPW; ++a) {
                s[a] *= scale;
                if (softcap > 0.0f) s[a] = softcap * tanhf(s[a] * inv_cap);
                s[a] = seen ? s[a] : -INFINITY;
                const float tile_max = warp_max(s[a]);
                live[a] = tile_max != -INFINITY;
                if (!live[a]) continue;
                const float m_new = fmaxf(m[a], tile_max);
                const float p = seen ? expf(s[a] - m_new) : 0.0f;
                const float corr = expf(m[a] - m_new);   // m[a] == -inf gives 0
                l[a] = l[a] * corr + warp_sum(p);
                m[a] = m_new;
#pragma unroll
                for (int d = 0; d < DPL; ++d) acc[a][d] *= corr;
                ps[a * TILE + lane] = p;
            }
            __syncwarp();
            int j = 0;
            for (; j + 4 <= valid; j += 4) {
                float4 p[HPW];
#pragma unroll
                for (int a = 0; a < HPW; ++a) p[a] = *reinterpret_cast<const float4*>(ps + a * TILE + j);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int d = 0; d < DPL; ++d) {
                        const int c = lane + 32 * d;
                        const float v = c < hd ? vs[(j + i) * hd + c] : 0.0f;
#pragma unroll
                        for (int a = 0; a < HPW; ++a)
                            if (live[a]) acc[a][d] = fmaf(i == 0 ? p[a].x : i == 1 ? p[a].y : i == 2 ? p[a].z : p[a].w, v, acc[a][d]);
                    }
            }
            for (; j < valid; ++j)
#pragma unroll
                for (int d = 0; d < DPL; ++d) {
                    const int c = lane + 32 * d;
                    const float v = c < hd ? vs[j * hd + c] : 0.0f;
#pragma unroll
                    for (int a = 0; a < HPW; ++a)
                        if (live[a]) acc[a][d] = fmaf(ps[a * TILE + j], v, acc[a][d]);
                }
        }
        __syncthreads();                                 // the buffer is read
    }
    if (!active) return;
#pragma unroll
    for (int a = 0; a < HPW; ++a) {
        if (h0 + a >= mine) break;
        const float inv = 1.0f / l[a];
        float* dst = out + ((size_t)(t0 + ti) * nh + (size_t)kvh * group + g0 + h0 + a) * hd;
#pragma unroll
        for (int d = 0; d < DPL; ++d) {
            const int c = lane + 32 * d;
            if (c < hd) dst[c] = acc[a][d] * inv;
        }
    }
}

template <int HPW, int DPL>
int launch_f32(const float* q, const float* k_pool, const float* v_pool, const int* positions, const int* tok_seg,
               const int* block_table, int max_pages, int page_size, float* out, int T, int nh, int nkv, int hd, int window,
               float scale, const float* sink, float softcap, int keep, int cuts, cudaStream_t stream) {
    // queries: at most eight warps of HPW heads
    const size_t smem = ((size_t)2 * TILE * (2 * hd + 4) + (size_t)F32_WARPS * HPW * (hd + TILE)) * sizeof(float);
    auto kernel = attention_f32_kernel<HPW, DPL>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    fwb::pdl(kernel, dim3(T, nkv, cuts), F32_WARPS * 32, smem, stream)(q, k_pool, v_pool, positions, tok_seg, block_table,
                                                                       max_pages, page_size, out, T, nh, nkv, hd, window,
                                                                       scale, sink, softcap, keep);
    return fwb_launch_status();
}

}  // namespace

// q, out: [T][nh*hd].  k_pool, v_pool: [pages][nkv][page_size][hd].  positions, tok_seg: [T].
// block_table: [S][max_pages].  The keys of every position <= a token's own must
// already be in the cache (this step's included).  Dtype flags: 0 fp32, 1 bf16.
FWB_API int fwb_attention_simt(const void* q, int q_bf16, const void* k_pool, const void* v_pool,
                               int cache_bf16, const int* positions, const int* tok_seg,
                               const int* block_table, int max_pages, int page_size, void* out,
                               int out_bf16, int T, int nh, int nkv, int hd, int window, float scale,
                               cudaStream_t stream);

// The general form.  sink: fp32 [nh] or null -- a score per head (not scaled, not capped) that joins the
// row's softmax denominator and has no value.  softcap > 0: score <- softcap * tanh(score / softcap)
// behind the scale.  keep > 0 (with a sliding window): the sequence's first `keep` positions stay visible
// however far the window has moved on.
FWB_API int fwb_attention_simt_sink(const void* q, int q_bf16, const void* k_pool, const void* v_pool,
                                    int cache_bf16, const int* positions, const int* tok_seg,
                                    const int* block_table, int max_pages, int page_size, void* out,
                                    int out_bf16, int T, int nh, int nkv, int hd, int window, float scale,
                                    const float* sink, float softcap, int keep, cudaStream_t stream) {
    if (T <= 0) return FWB_OK;
    if (keep < 0 || (keep > 0 && window <= 0)) return FWB_BAD_ARGUMENT;
    if (!q || !k_pool || !v_pool || !positions || !tok_seg || !block_table || !out)
        return FWB_BAD_ARGUMENT;
    if (nh <= 0 || nkv <= 0 || nh % nkv != 0 || hd <= 0 || max_pages <= 0) return FWB_BAD_ARGUMENT;
    if (page_size <= 0 || page_size % TILE != 0) return FWB_UNSUPPORTED;
    const int group = nh / nkv;
    const int cuts = (group + WARPS * MAX_HPW - 1) / (WARPS * MAX_HPW);
    if (hd > 32 * MAX_DPL || nkv > 65535 || cuts > 65535) return FWB_UNSUPPORTED;
    const size_t smem = ((size_t)(cuts > 1 ? WARPS * MAX_HPW : group) * hd + (size_t)TILE * (2 * hd + 1)) * sizeof(float);
    using bf = __nv_bfloat16;
    if (!q_bf16 && !cache_bf16 && !out_bf16 && hd % 4 == 0 &&
        !(((uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool) & 15)) {
#define FWB_F32(HPW, DPL)                                                                                            \
    return launch_f32<HPW, DPL>((const float*)q, (const float*)k_pool, (const float*)v_pool, positions, tok_seg,     \
                                block_table, max_pages, page_size, (float*)out, T, nh, nkv, hd, window, scale, sink, \
                                softcap, keep, cuts, stream)
        if (group <= 2) {
            if (hd <= 64) FWB_F32(2, 2);
            if (hd <= 128) FWB_F32(2, 4);
            FWB_F32(2, 8);
        }
        if (hd <= 64) FWB_F32(4, 2);
        if (hd <= 128) FWB_F32(4, 4);
        FWB_F32(4, 8);
#undef FWB_F32
    }
    dim3 grid(T, nkv, cuts);
#define FWB_ATTN(TQ, TC, TO)                                                                      \
    do {                                                                                          \
        auto kernel = attention_simt_kernel<TQ, TC, TO>;                                          \
        if (smem > 48 * 1024) {                                                                   \
            cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                                 (int)smem);                                      \
            if (e != cudaSuccess) return (int)e;                                                  \
        }                                                                                         \
        fwb::pdl(kernel, grid, WARPS * 32, smem, stream)((const TQ*)q, (const TC*)k_pool,               \
                                                   (const TC*)v_pool, positions, tok_seg,         \
                                                   block_table, max_pages, page_size, (TO*)out,   \
                                                   nh, nkv, hd, window, scale, sink, softcap, keep); \
    } while (0)
    if (!q_bf16 && !cache_bf16 && !out_bf16) FWB_ATTN(float, float, float);
    else if (q_bf16 && cache_bf16 && out_bf16) FWB_ATTN(bf, bf, bf);
    else return FWB_UNSUPPORTED;
#undef FWB_ATTN
    return fwb_launch_status();
}

FWB_API int fwb_attention_simt(const void* q, int q_bf16, const void* k_pool, const void* v_pool,
                               int cache_bf16, const int* positions, const int* tok_seg,
                               const int* block_table, int max_pages, int page_size, void* out,
                               int out_bf16, int T, int nh, int nkv, int hd, int window, float scale,
                               cudaStream_t stream) {
    return fwb_attention_simt_sink(q, q_bf16, k_pool, v_pool, cache_bf16, positions, tok_seg, block_table,
                                   max_pages, page_size, out, out_bf16, T, nh, nkv, hd, window, scale, nullptr,
                                   0.0f, 0, stream);
}
