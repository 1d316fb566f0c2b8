// The gated delta rule: a recurrent mixer whose per-request state is one [d][e] matrix per head.
//
// Per token and head, with unit vectors q (times d^-1/2) and k of size d, a value v of size e, a
// write strength beta in (0, 1) and a decay g in (0, 1):
//     S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
// so the read-out sees the token's own write.  q, k and v come from one fused projection
//     p[t] = [ q: G d | k: G d | v: H e | gate: H e | b: H | a: H ]        (fp32)
// through a short causal convolution over time per channel (taps [C][L], the last tap on the token
// itself) and silu; q and k are then made unit vectors per head (x / sqrt(sum x^2 + 1e-6)); query
// head h uses q/k head h / (H / G).  beta = sigmoid(b), g = exp(-exp(A_log) softplus(a + dt_bias)).
//
// Kernels (everything fp32; segments of many tokens also take delta_chunk and delta_runs, further down, which sum over
// their chunks in 64 bits):
//   delta_prepare   one block per token (or per four): convolution + silu, unit vectors, beta and g
//                   -> r[t] = [ q^: G d | k^: G d | v: H e | beta: H | g: H | q^.k^: G ]
//   delta_scan      one block per (16 or 32 columns of S, head, segment): the recurrence over the
//                   segment's tokens in order.  A column of S evolves independently of the others;
//                   four or eight adjacent lanes hold one column in registers, so a token costs two
//                   reductions over those lanes.  State in and out of the request's slot.  The first
//                   block of a segment also moves the convolution's last L-1 inputs on, for the next
//                   step (behind delta_prepare, which reads the old ones).
//   gated_head_norm out[t][h] = weight * o / sqrt(mean(o^2) + eps) * silu(gate)
// A request's slot is [ S: H d e | conv inputs: C (L-1) ] fp32, zero when the request starts.  A
// token's result depends on its request's earlier tokens only through that slot, and on nothing of the segments beside
// its own in the step: a segment's own length decides between scan and chunks.  In the scan every sum runs in an order
// fixed by the sizes, so it does not depend on how the sequence was cut into steps; the chunks of a long segment start
// where the segment does, so another cut is another order of the same sums.
#include "common.cuh"

using namespace fwb;

namespace {

constexpr int MAX_TAPS = 16;

struct DeltaShape {
    int H, G, d, e, L;      // heads, q/k heads, q/k size, value size, taps
    __host__ __device__ int cq() const { return G * d; }
    __host__ __device__ int cv() const { return H * e; }
    __host__ __device__ int channels() const { return 2 * G * d + H * e; }      // through the convolution
    __host__ __device__ int p_width() const { return channels() + H * e + 2 * H; }
    // (rows of r are padded to 16 bytes, so that 16-byte copies may start at a head's first channel)
    __host__ __device__ int r_width() const { return (channels() + 2 * H + G + 3) & ~3; }
};

__global__ void __launch_bounds__(512)
delta_prepare_kernel(const float* __restrict__ p, const float* __restrict__ taps, const float* __restrict__ a_log,
                     const float* __restrict__ dt_bias, const float* __restrict__ state, long long slot_stride,
                     const int* __restrict__ seg_start, const int* __restrict__ seg_slot,
                     const int* __restrict__ tok_seg, float* __restrict__ r, DeltaShape sh) {
    fwb::pdl_entry();
    extern __shared__ float c[];                  // the token's channels behind convolution and silu
    const int t = blockIdx.x;
    const int seg = tok_seg[t];
    const int local = t - seg_start[seg];         // tokens of this request in front of t in this step
    const int C = sh.channels(), P = sh.p_width(), R = sh.r_width(), L = sh.L;
    const float* hist = state + (size_t)seg_slot[seg] * slot_stride + (size_t)sh.H * sh.d * sh.e;
    for (int ch = threadIdx.x; ch < C; ch += blockDim.x) {
        float acc = 0.0f;
        for (int j = 0; j < L; ++j) {
            const int back = L - 1 - j;           // tap j multiplies the input `back` tokens ago
            const float x = back <= local ? p[(size_t)(t - back) * P + ch]
                                          : hist[(size_t)ch * (L - 1) + (L - 1) - (back - local)];
            acc = fmaf(taps[(size_t)ch * L + j], x, acc);
        }
        c[ch] = silu_f32(acc);
    }
    __syncthreads();
    float* out = r + (size_t)t * R;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const float q_scale = rsqrtf((float)sh.d);
    for (int head = warp; head < sh.G; head += warps) {            // query head and key head `head` together
        const float* q = c + (size_t)head * sh.d;
        const float* k = c + (size_t)(sh.G + head) * sh.d;
        float qq = 0.0f, kk = 0.0f, qk = 0.0f;
        for (int i = lane; i < sh.d; i += 32) {
            qq = fmaf(q[i], q[i], qq);
            kk = fmaf(k[i], k[i], kk);
            qk = fmaf(q[i], k[i], qk);
        }
        qq = warp_sum(qq), kk = warp_sum(kk), qk = warp_sum(qk);
        const float inv_q = (1.0f / sqrtf(qq + 1e-6f)) * q_scale, inv_k = 1.0f / sqrtf(kk + 1e-6f);
        for (int i = lane; i < sh.d; i += 32) {
            out[(size_t)head * sh.d + i] = q[i] * inv_q;
            out[(size_t)(sh.G + head) * sh.d + i] = k[i] * inv_k;
        }
        if (lane == 0) out[C + 2 * sh.H + head] = (qk * inv_q) * inv_k;      // q^ . k^, for the read-out
    }
    for (int i = threadIdx.x; i < sh.cv(); i += blockDim.x) out[2 * sh.cq() + i] = c[2 * sh.cq() + i];
    for (int h = threadIdx.x; h < sh.H; h += blockDim.x) {
        const float b = p[(size_t)t * P + C + sh.cv() + h];
        const float a = p[(size_t)t * P + C + sh.cv() + sh.H + h] + dt_bias[h];
        const float softplus = a > 20.0f ? a : log1pf(expf(a));
        out[C + h] = 1.0f / (1.0f + expf(-b));
        out[C + sh.H + h] = expf(-expf(a_log[h]) * softplus);
    }
}

// The same for four taps and channel counts in fours, PREP tokens a block: their rows of p are read once, 16 bytes a
// load, as a window that slides along (the kernel above reads every row once per tap), and only the channels of q and
// k stop in shared memory on their way.  Blocks (.., 0) have q and k, blocks (.., 1) the values: three small blocks an SM
// wait for their loads, norms and scalars in turn.
constexpr int PREP = 4;
__global__ void __launch_bounds__(256, 3)
delta_prepare_window_kernel(const float* __restrict__ p, const float* __restrict__ taps, const float* __restrict__ a_log,
                            const float* __restrict__ dt_bias, const float* __restrict__ state, long long slot_stride,
                            const int* __restrict__ seg_start, const int* __restrict__ seg_slot,
                            const int* __restrict__ tok_seg, float* __restrict__ r, int T, DeltaShape sh) {
    fwb::pdl_entry();
    extern __shared__ __align__(16) float c[];    // [PREP][2 G d]: q and k behind convolution and silu
    constexpr int L = 4;
    const int t0 = blockIdx.x * PREP, tokens = T - t0 < PREP ? T - t0 : PREP;
    const int C = sh.channels(), P = sh.p_width(), R = sh.r_width(), QK = 2 * sh.cq();
    int local[PREP];                              // tokens of its request in front of a token in this step
    const float* hist[PREP];
#pragma unroll
    for (int i = 0; i < PREP; ++i) {
        const int t = i < tokens ? t0 + i : t0, seg = tok_seg[t];
        local[i] = t - seg_start[seg];
        hist[i] = state + (size_t)seg_slot[seg] * slot_stride + (size_t)sh.H * sh.d * sh.e;
    }
    const int stop = blockIdx.y ? C : QK;
    for (int ch = (blockIdx.y ? QK : 0) + threadIdx.x * 4; ch < stop; ch += blockDim.x * 4) {
        float4 window[PREP + L - 1];
#pragma unroll
        for (int i = 0; i < PREP + L - 1; ++i) {
            const int t = t0 + i - (L - 1);
            window[i] = t >= 0 && t < T ? *reinterpret_cast<const float4*>(p + (size_t)t * P + ch) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        float4 w[4];                              // the taps of four channels
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = *reinterpret_cast<const float4*>(taps + (size_t)(ch + j) * L);
#pragma unroll
        for (int i = 0; i < PREP; ++i) {
            if (i >= tokens) break;
            float4 x[L];
#pragma unroll
            for (int j = 0; j < L; ++j) {
                const int back = L - 1 - j;       // tap j multiplies the input `back` tokens ago
                x[j] = window[i + j];
                if (back > local[i]) {
                    const float* from = hist[i] + (size_t)ch * (L - 1) + (L - 1) - (back - local[i]);
                    x[j] = make_float4(from[0], from[L - 1], from[2 * (L - 1)], from[3 * (L - 1)]);
                }
            }
            float4 v;
            v.x = silu_f32(fmaf(w[0].w, x[3].x, fmaf(w[0].z, x[2].x, fmaf(w[0].y, x[1].x, w[0].x * x[0].x))));
            v.y = silu_f32(fmaf(w[1].w, x[3].y, fmaf(w[1].z, x[2].y, fmaf(w[1].y, x[1].y, w[1].x * x[0].y))));
            v.z = silu_f32(fmaf(w[2].w, x[3].z, fmaf(w[2].z, x[2].z, fmaf(w[2].y, x[1].z, w[2].x * x[0].z))));
            v.w = silu_f32(fmaf(w[3].w, x[3].w, fmaf(w[3].z, x[2].w, fmaf(w[3].y, x[1].w, w[3].x * x[0].w))));
            if (ch < QK) *reinterpret_cast<float4*>(c + i * QK + ch) = v;
            else *reinterpret_cast<float4*>(r + (size_t)(t0 + i) * R + ch) = v;
        }
    }
    if (blockIdx.y) return;
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const float q_scale = rsqrtf((float)sh.d);
    for (int job = warp; job < tokens * sh.G; job += warps) {         // query head and key head `head` together
        const int i = job / sh.G, head = job - i * sh.G;
        const float* q = c + (size_t)i * QK + (size_t)head * sh.d;
        const float* k = q + sh.cq();
        float* out = r + (size_t)(t0 + i) * R;
        float qq = 0.0f, kk = 0.0f, qk = 0.0f;
        for (int n = lane; n < sh.d; n += 32) {
            qq = fmaf(q[n], q[n], qq);
            kk = fmaf(k[n], k[n], kk);
            qk = fmaf(q[n], k[n], qk);
        }
        qq = warp_sum(qq), kk = warp_sum(kk), qk = warp_sum(qk);
        const float inv_q = (1.0f / sqrtf(qq + 1e-6f)) * q_scale, inv_k = 1.0f / sqrtf(kk + 1e-6f);
        for (int n = lane; n < sh.d; n += 32) {
            out[(size_t)head * sh.d + n] = q[n] * inv_q;
            out[(size_t)(sh.G + head) * sh.d + n] = k[n] * inv_k;
        }
        if (lane == 0) out[C + 2 * sh.H + head] = (qk * inv_q) * inv_k;      // q^ . k^, for the read-out
    }
    for (int job = threadIdx.x; job < tokens * sh.H; job += blockDim.x) {
        const int i = job / sh.H, h = job - i * sh.H;
        const float* row = p + (size_t)(t0 + i) * P + C + sh.cv();
        const float a = row[sh.H + h] + dt_bias[h];
        const float softplus = a > 20.0f ? a : log1pf(expf(a));
        r[(size_t)(t0 + i) * R + C + h] = 1.0f / (1.0f + expf(-row[h]));
        r[(size_t)(t0 + i) * R + C + sh.H + h] = expf(-expf(a_log[h]) * softplus);
    }
}

// The request's last L-1 inputs of every channel, for the next step.  Runs in the kernel behind
// delta_prepare (which reads the old ones): the first block of every segment's scan does it.
__device__ __forceinline__ void delta_conv_advance(const float* __restrict__ p, float* __restrict__ slot, int t0,
                                                   int n, const DeltaShape& sh) {
    const int keep = sh.L - 1, P = sh.p_width();
    for (int ch = threadIdx.x; ch < sh.channels(); ch += blockDim.x) {
        float* hist = slot + (size_t)sh.H * sh.d * sh.e + (size_t)ch * keep;
        float next[MAX_TAPS];
        for (int j = 0; j < keep; ++j) {
            const int local = n - keep + j;       // the input that becomes entry j (oldest first)
            next[j] = local >= 0 ? p[(size_t)(t0 + local) * P + ch] : hist[j + n];
        }
        for (int j = 0; j < keep; ++j) hist[j] = next[j];
    }
}

__device__ __forceinline__ void copy_async_f32(float* dst_shared, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_shared)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy_async_16(float* dst_shared, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_shared)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// LPC adjacent lanes hold one column of S, DPL consecutive entries each (LPC * DPL >= d).  The tokens'
// q, k, v, beta, g and q.k arrive through a ring of asynchronous copies that runs three tokens ahead of the
// arithmetic.  Per token both sums over the *old* column, a = S.k and b = S.q, are taken in one pass and
// reduced over the LPC lanes together; then
//     u = beta (v - g a),   o = g b + u (q.k),   S <- g S + k u
// which is the recurrence in the order the header states (the read-out sees the token's write), with
// one reduction on the way to the next token instead of two.  In a slot, S lies column by column:
// S[h][column][d].  VEC: d and e are multiples of 4 and slots start on 16-byte borders: copies and
// state accesses of 16 bytes.
template <int DPL, int LPC, bool VEC>
__global__ void __launch_bounds__(128)
delta_scan_kernel(const float* __restrict__ r, const float* __restrict__ p, float* __restrict__ state,
                  long long slot_stride, const int* __restrict__ seg_start, const int* __restrict__ seg_slot,
                  float* __restrict__ o, int below, DeltaShape sh) {
    // The next kernel is released only behind the token loop: its blocks would otherwise sit on the SMs for
    // the whole scan, whose one warp a scheduler is slowed by every other resident warp.
    fwb::pdl_wait();
    constexpr int COLS = 128 / LPC, STRIDE = DPL + 4, STAGES = 4;     // (+4: lanes' float4 reads hit apart banks)
    constexpr int KQ = 2 * LPC * STRIDE;                              // floats of one stage's k and q
    __shared__ __align__(16) float kq[STAGES][KQ];
    __shared__ __align__(16) float vs[STAGES][COLS];
    __shared__ float scalars[STAGES][4];                              // beta, g, q.k
    const int seg = blockIdx.z, h = blockIdx.y;
    const int t0 = seg_start[seg], t1 = seg_start[seg + 1];
    if (t1 <= t0 || t1 - t0 >= below) return;                         // (a segment of that many tokens goes by chunks)
    const int d = sh.d, e = sh.e, R = sh.r_width();
    const int kv_head = h / (sh.H / sh.G);
    const int col_local = threadIdx.x / LPC, sub = threadIdx.x % LPC;
    const int col = blockIdx.x * COLS + col_local;
    const bool valid = col < e;
    float* slot = state + (size_t)seg_slot[seg] * slot_stride;
    if (blockIdx.x == 0 && h == 0 && sh.L > 1) delta_conv_advance(p, slot, t0, t1 - t0, sh);
    float* S_col = slot + ((size_t)h * e + (valid ? col : 0)) * d;
    float S[DPL];
    if (VEC) {
#pragma unroll
        for (int i = 0; i < DPL; i += 4) {
            const int dd = sub * DPL + i;
            const float4 v = (valid && dd < d) ? *reinterpret_cast<const float4*>(S_col + dd) : make_float4(0.f, 0.f, 0.f, 0.f);
            S[i] = v.x, S[i + 1] = v.y, S[i + 2] = v.z, S[i + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < DPL; ++i) {
            const int dd = sub * DPL + i;
            S[i] = (valid && dd < d) ? S_col[dd] : 0.0f;
        }
    }
    if (d < DPL * LPC || (int)(blockIdx.x + 1) * COLS > e) {
        // entries behind the head's last channel and columns behind the last are never copied: zeros
        for (int i = threadIdx.x; i < STAGES * KQ; i += blockDim.x) (&kq[0][0])[i] = 0.0f;
        for (int i = threadIdx.x; i < STAGES * COLS; i += blockDim.x) (&vs[0][0])[i] = 0.0f;
        __syncthreads();
    }
    const int q_at = kv_head * d, k_at = sh.cq() + kv_head * d, v_at = 2 * sh.cq() + h * e;
    // what this thread copies for every token (VEC): one 16-byte piece of k|q, the fourth warp's first
    // lanes the values, three lanes the token's scalars
    const int piece = threadIdx.x * 4;
    const bool has_piece = piece < 2 * d;
    const int piece_which = piece >= d ? 1 : 0, piece_dd = piece - piece_which * d;
    const int piece_src = (piece_which ? q_at : k_at) + piece_dd;
    const int piece_dst = piece_which * LPC * STRIDE + (piece_dd / DPL) * STRIDE + piece_dd % DPL;
    const int c4 = (threadIdx.x - 96) * 4;
    const bool has_v = threadIdx.x >= 96 && c4 < COLS && (int)blockIdx.x * COLS + c4 < e;
    const int v_src = v_at + blockIdx.x * COLS + c4;
    const int which_scalar = threadIdx.x - 120;                       // 0 beta, 1 g, 2 q.k
    const int scalar_src = which_scalar == 0 ? sh.channels() + h
                                             : (which_scalar == 1 ? sh.channels() + sh.H + h
                                                                  : sh.channels() + 2 * sh.H + kv_head);
    auto fetch = [&](int t, int stage) {
        if (t < t1) {
            const float* row = r + (size_t)t * R;
            if (VEC) {
                if (has_piece) copy_async_16(&kq[stage][piece_dst], row + piece_src);
                if (has_v) copy_async_16(&vs[stage][c4], row + v_src);
            } else {
                for (int i = threadIdx.x; i < 2 * d; i += blockDim.x) {
                    const int which = i >= d ? 1 : 0, dd = i - which * d;
                    copy_async_f32(&kq[stage][which * LPC * STRIDE + (dd / DPL) * STRIDE + dd % DPL],
                                   row + (which ? q_at : k_at) + dd);
                }
                if (threadIdx.x < COLS && blockIdx.x * COLS + threadIdx.x < e)
                    copy_async_f32(&vs[stage][threadIdx.x], row + v_at + blockIdx.x * COLS + threadIdx.x);
            }
            if (which_scalar >= 0 && which_scalar < 3) copy_async_f32(&scalars[stage][which_scalar], row + scalar_src);
        }
        copy_async_commit();
    };
    for (int j = 0; j < STAGES - 1; ++j) fetch(t0 + j, j);
    float* out_at = o + ((size_t)t0 * sh.H + h) * e + col;
    const size_t out_step = (size_t)sh.H * e;
    for (int t = t0; t < t1; ++t, out_at += out_step) {
        const int stage = (t - t0) % STAGES;
        copy_async_wait<STAGES - 2>();          // this token's copies have landed (mine; the barrier: everybody's)
        __syncthreads();                        // ... and everybody is done with the token before
        fetch(t + STAGES - 1, (t - t0 + STAGES - 1) % STAGES);
        const float beta = scalars[stage][0], g = scalars[stage][1], qk = scalars[stage][2];
        const float4* k4 = reinterpret_cast<const float4*>(&kq[stage][sub * STRIDE]);
        const float4* q4 = reinterpret_cast<const float4*>(&kq[stage][LPC * STRIDE + sub * STRIDE]);
        float a[4] = {0.0f, 0.0f, 0.0f, 0.0f}, b[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int i = 0; i < DPL / 4; ++i) {
            const float4 k = k4[i], q = q4[i];
            a[0] = fmaf(S[4 * i], k.x, a[0]), b[0] = fmaf(S[4 * i], q.x, b[0]);
            a[1] = fmaf(S[4 * i + 1], k.y, a[1]), b[1] = fmaf(S[4 * i + 1], q.y, b[1]);
            a[2] = fmaf(S[4 * i + 2], k.z, a[2]), b[2] = fmaf(S[4 * i + 2], q.z, b[2]);
            a[3] = fmaf(S[4 * i + 3], k.w, a[3]), b[3] = fmaf(S[4 * i + 3], q.w, b[3]);
        }
        float sk = (a[0] + a[1]) + (a[2] + a[3]), sq = (b[0] + b[1]) + (b[2] + b[3]);
#pragma unroll
        for (int offset = 1; offset < LPC; offset <<= 1) {
            sk += __shfl_xor_sync(0xffffffffu, sk, offset);
            sq += __shfl_xor_sync(0xffffffffu, sq, offset);
        }
        const float u = beta * (vs[stage][col_local] - g * sk);
        if (sub == 0 && valid) *out_at = fmaf(g, sq, u * qk);
#pragma unroll
        for (int i = 0; i < DPL / 4; ++i) {
            const float4 k = k4[i];
            S[4 * i] = fmaf(g, S[4 * i], k.x * u);
            S[4 * i + 1] = fmaf(g, S[4 * i + 1], k.y * u);
            S[4 * i + 2] = fmaf(g, S[4 * i + 2], k.z * u);
            S[4 * i + 3] = fmaf(g, S[4 * i + 3], k.w * u);
        }
    }
    copy_async_wait<0>();
    fwb::pdl_launch_dependents();
    if (VEC) {
#pragma unroll
        for (int i = 0; i < DPL; i += 4) {
            const int dd = sub * DPL + i;
            if (valid && dd < d) *reinterpret_cast<float4*>(S_col + dd) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
        }
    } else {
#pragma unroll
        for (int i = 0; i < DPL; ++i) {
            const int dd = sub * DPL + i;
            if (valid && dd < d) S_col[dd] = S[i];
        }
    }
}

// ---- runs of tokens: chunks of 32 ---------------------------------------------------------------------
// The scan above walks a request token by token: 0.59 us a token whatever the heads, a chain of a copy, a barrier
// and two reductions over lanes.  Over a chunk of C tokens behind the state S0 the same recurrence is
//     u = T r,  r_i = beta_i (v_i - G_i S0^T k_i),  T = (I + A)^-1,  A_ij = beta_i D_ij k_i.k_j  (j < i)
//     o_i = G_i S0^T q_i + sum_{j <= i} P_ij u_j,  P_ij = D_ij q_i.k_j
//     S <- G_C S0 + sum_j D_Cj k_j u_j^T
// with D_ij = g_{j+1} ... g_i and G_i = g_1 ... g_i, all products of decays (no logarithms: a difference of two
// large sums would lose what a product of factors keeps).  T and P need no state: delta_chunk_kernel makes them for
// every chunk and head at once; delta_runs_kernel then walks the chunks, one block per 16 columns of S and head, S
// in shared memory, five small products a chunk.
//
// What the chunk adds to the scan's roundings would be those of T, P, u and of sums over 32 tokens (2.5 times the scan's
// error under strong decays, 1.9 under moderate ones, all in 32 bits).  So the products with T and P, the dot products
// behind those two and the state's update run in 64 bits; only the 128-channel sums S0^T k and S0^T q, S itself and the
// results are 32 bits wide.  Error against 64 bits over the scan's, 600 tokens on B200, keys behind silu, keys that come
// again, keys that nearly coincide and keys of both signs, decays from none to e^-60 a token: 0.76 to 0.90 in the
// read-out, 0.72 to 1.00 in the state (what is left is the inputs' own rounding).  64-bit multiply-adds run at half the
// rate of 32-bit ones here and do not bind; 16 heads of 128, 2,048 tokens, all launches: 302 us in 32 bits, 378 so by
// multiply-adds, 268 with the 64-bit tensor cores, 749 by the scan.
//
// A token reads nothing of a later one: T and P are summed up to the token's own column, so a value that is not finite
// stays where the scan leaves it.
constexpr int CHUNK = 32, CT = 34;                    // rows of T and P: 32 entries, then what a token has besides
constexpr int CHUNK_DOUBLES = 2 * CHUNK * CT;         // T | P of one chunk and head
constexpr int AT_BETA = 32, AT_G = 32, AT_REST = 33;  // T[i][32] = beta_i; P[i][32] = G_i, P[i][33] = D_Ci

__device__ __forceinline__ void fma_pair(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float pair_sum(unsigned long long v) {
    return __uint_as_float((unsigned)v) + __uint_as_float((unsigned)(v >> 32));
}

// d[8][8] += a[8][4] b[4][8]: a lane has a[lane / 4][lane % 4], b[lane % 4][lane / 4], d[lane / 4][2 (lane % 4) + 0, 1].
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1]) : "d"(a), "d"(b));
}

// Chunk c of segment s and head h: scratch + (((seg_start[s] / 32 + s) + c) * H + h) * CHUNK_DOUBLES: chunks of
// different segments never meet, and T / 32 + S of them are enough.  Segments shorter than `from` are the scan's.
// The dot products are 8 x 8 tiles of the 64-bit tensor cores, a warp eight rows of k or q and the tiles up to its own
// tokens; (I + A)^-1 is two inverses of 16 tokens side by side in a warp and T21 = -T22 A21 T11 over the block.  With
// multiply-adds from doubles in shared memory and one substitution of 32 steps, two blocks an SM, it took 57 us a layer
// of 2,048 tokens and 16 heads.
template <int D>
__global__ void __launch_bounds__(256, 4)
delta_chunk_kernel(const float* __restrict__ r, const int* __restrict__ seg_start, double* __restrict__ scratch, int from,
                   DeltaShape sh) {
    fwb::pdl_entry();
    constexpr int ROW = D + 4, DOTS = CHUNK + 1, A_ROW = CHUNK + 2, HALF = CHUNK / 2;
    constexpr int DOUBLES = 2 * CHUNK * DOTS + 2 * CHUNK * A_ROW, LOADED = CHUNK * ROW;      // (floats, two to a double)
    __shared__ __align__(16) double pool[DOUBLES > LOADED ? DOUBLES : LOADED];
    float* rows = reinterpret_cast<float*>(pool);                     // [64][D + 4]: k, then q
    double* dots = pool;                                              // [64][33]: k_i.k_j, q_i.k_j
    double* a_rows = pool + 2 * CHUNK * DOTS;                         // [32][34]
    double* t_rows = a_rows + CHUNK * A_ROW;                          // [32][34]
    double* u = pool;                                                 // [16][16], where k's dot products were
    __shared__ double beta[CHUNK], g[CHUNK];
    const int seg = blockIdx.z, h = blockIdx.y;
    const int begin = seg_start[seg], end = seg_start[seg + 1], t0 = begin + blockIdx.x * CHUNK;
    const int left = end - t0;
    if (left <= 0 || end - begin < from) return;
    const int n = left < CHUNK ? left : CHUNK, R = sh.r_width(), head = h / (sh.H / sh.G);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x < CHUNK) {
        const bool in = (int)threadIdx.x < n;
        const float* row = r + (size_t)(t0 + (in ? threadIdx.x : 0)) * R + sh.channels();
        beta[threadIdx.x] = in ? (double)row[h] : 0.0;
        g[threadIdx.x] = in ? (double)row[sh.H + h] : 1.0;
    }
#pragma unroll
    for (int i = threadIdx.x; i < 2 * CHUNK * (D / 4); i += 256) {
        const int row = i / (D / 4), c = (i % (D / 4)) * 4, token = row % CHUNK;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (token < n)
            v = *reinterpret_cast<const float4*>(r + (size_t)(t0 + token) * R + (row < CHUNK ? sh.cq() : 0) + head * D + c);
        *reinterpret_cast<float4*>(rows + row * ROW + c) = v;
    }
    __syncthreads();
    // warps 0-3 eight k rows each, 4-7 eight q rows; nobody needs the columns of later tokens
    const int own = warp & 3, row0 = (warp >> 2) * CHUNK + own * 8, at = (lane >> 2) * ROW + (lane & 3);
    double acc[4][2];
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j][0] = acc[j][1] = 0.0;
#pragma unroll 4
    for (int k = 0; k < D; k += 4) {
        const double a = rows[row0 * ROW + at + k];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j <= own) mma_f64(acc[j], a, (double)rows[j * 8 * ROW + at + k]);
    }
    __syncthreads();                                                  // k and q have been read: the pool is free
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (j <= own) {
            double* to = dots + (row0 + (lane >> 2)) * DOTS + j * 8 + 2 * (lane & 3);
            to[0] = acc[j][0];
            to[1] = acc[j][1];
        }
    __syncthreads();
    double* out = scratch + ((size_t)(begin / CHUNK + seg + blockIdx.x) * sh.H + h) * CHUNK_DOUBLES;
    double* p_out = out + CHUNK * CT;
    if (warp == 0) {                                                  // A: lane j walks its column down
        double d = 1.0;
#pragma unroll 4
        for (int i = 0; i < CHUNK; ++i) {
            d = i > lane ? d * g[i] : 1.0;
            a_rows[i * A_ROW + lane] = i > lane ? beta[i] * (d * dots[i * DOTS + lane]) : 0.0;
        }
        __syncwarp();
        // column `lane` of the inverse inside its half, forwards
        const int base = lane & HALF, column = lane & (HALF - 1);
        double t[HALF];
#pragma unroll
        for (int i = 0; i < HALF; ++i) {
            const double* row = a_rows + (base + i) * A_ROW + base;
            double s0 = 0.0, s1 = 0.0;
#pragma unroll
            for (int m = 0; m + 1 < i; m += 2) {
                s0 = fma(row[m], t[m], s0);
                s1 = fma(row[m + 1], t[m + 1], s1);
            }
            if (i & 1) s0 = fma(row[i - 1], t[i - 1], s0);
            t[i] = i == column ? 1.0 : (i > column ? -(s0 + s1) : 0.0);
            t_rows[(base + i) * A_ROW + lane] = t[i];
        }
        if (lane >= HALF)
            for (int i = 0; i < HALF; ++i) t_rows[i * A_ROW + lane] = 0.0;
    } else if (warp == 1) {                                           // P
        double d = 1.0;
#pragma unroll 4
        for (int i = 0; i < CHUNK; ++i) {
            d = i > lane ? d * g[i] : 1.0;
            p_out[i * CT + lane] = i >= lane ? d * dots[(CHUNK + i) * DOTS + lane] : 0.0;
        }
        p_out[lane * CT + AT_REST] = d;                               // D_Cj: the last row's factor
    } else if (warp == 2) {                                           // G_i
        double d = 1.0;
        for (int i = 0; i <= lane; ++i) d *= g[i];
        p_out[lane * CT + AT_G] = d;
        out[lane * CT + AT_BETA] = beta[lane];
    }
    __syncthreads();
    const int i = threadIdx.x >> 4, j = threadIdx.x & (HALF - 1);     // an element of the lower left quarter
    double sum = 0.0;
    for (int l = j; l < HALF; ++l) sum = fma(a_rows[(HALF + i) * A_ROW + l], t_rows[l * A_ROW + j], sum);
    u[i * HALF + j] = sum;
    __syncthreads();
    sum = 0.0;
    for (int m = 0; m <= i; ++m) sum = fma(t_rows[(HALF + i) * A_ROW + HALF + m], u[m * HALF + j], sum);
    t_rows[(HALF + i) * A_ROW + j] = -sum;
    __syncthreads();
#pragma unroll
    for (int x = threadIdx.x; x < CHUNK * CHUNK; x += 256) out[(x / CHUNK) * CT + x % CHUNK] = t_rows[(x / CHUNK) * A_ROW + x % CHUNK];
}

constexpr int RUN_COLS = 16;
constexpr int COL = 36, UN_ROW = 20;                   // columns of r and u, rows of D_Cj u_j: a fragment's 16 values on 16 banks

template <int D>
struct RunLayout {                                     // floats (T, P, r and u: two a value, on 16-byte borders)
    static constexpr int ROW = D + 4;
    static constexpr int K = 0, V = 2 * CHUNK * ROW, Q = V + 2 * CHUNK * RUN_COLS, TP = Q + CHUNK * ROW;     // k and v: two chunks
    static constexpr int S = TP + 2 * CHUNK_DOUBLES, RT = S + RUN_COLS * ROW, RED = RT + 2 * RUN_COLS * COL;  // S column by column
    static constexpr int RED_FLOATS = 4 * 2 * CHUNK * 20, FLOATS = RED + RED_FLOATS;
    static constexpr int UT = RED, UN = UT + 2 * RUN_COLS * COL;      // where the quarters' sums lay: they have been read
    static_assert(UN + 2 * CHUNK * UN_ROW <= FLOATS && Q % 4 == 0 && TP % 4 == 0 && RT % 4 == 0 && RED % 4 == 0, "it fits");
    static_assert(FLOATS * 4 <= 112 * 1024, "two blocks an SM");
};

// Bound by latency: five barriers a chunk with little between them, 3.4 us a chunk for a block that has an SM to itself
// (one prompt of 16 heads is 128 blocks; 4.4 us, 281 -> 215 us a layer of 2,048 tokens, while the 64-bit products were
// multiply-adds: a conversion of k for every four of them and rows of T and P of up to 32 steps a thread).  So what a
// chunk needs lies once in shared memory where its place comes free in time (q behind the first products, T and P behind
// the last), k and v twice, and two blocks share an SM where several segments bring them.
template <int D>
__global__ void __launch_bounds__(256, 2)
delta_runs_kernel(const float* __restrict__ r, const float* __restrict__ p, const double* __restrict__ scratch,
                  float* __restrict__ state, long long slot_stride, const int* __restrict__ seg_start,
                  const int* __restrict__ seg_slot, float* __restrict__ o, int from, DeltaShape sh) {
    using Y = RunLayout<D>;
    extern __shared__ __align__(16) float sm[];
    fwb::pdl_wait();
    const int seg = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * RUN_COLS;
    const int t0 = seg_start[seg], t1 = seg_start[seg + 1];
    if (t1 <= t0 || t1 - t0 < from) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, e = sh.e, R = sh.r_width();
    const int head = h / (sh.H / sh.G), chunks = (t1 - t0 + CHUNK - 1) / CHUNK;
    float* slot = state + (size_t)seg_slot[seg] * slot_stride;
    if (blockIdx.x == 0 && h == 0 && sh.L > 1) delta_conv_advance(p, slot, t0, t1 - t0, sh);
    float* S = sm + Y::S;
    float* red = sm + Y::RED;
    double* rt = reinterpret_cast<double*>(sm + Y::RT);               // r, column by column [16][COL]
    double* ut = reinterpret_cast<double*>(sm + Y::UT);               // u, column by column
    double* un = reinterpret_cast<double*>(sm + Y::UN);               // D_Cj u_j, token by token [32][UN_ROW]
    for (int i = tid; i < RUN_COLS * (D / 4); i += 256) {
        const int c = i / (D / 4), k = (i % (D / 4)) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (col0 + c < e) v = *reinterpret_cast<const float4*>(slot + ((size_t)h * e + col0 + c) * D + k);
        *reinterpret_cast<float4*>(S + c * Y::ROW + k) = v;
    }
    const double* tp0 = scratch + ((size_t)(t0 / CHUNK + seg) * sh.H + h) * CHUNK_DOUBLES;
    auto copy = [&](float* dst, const void* src, bool in) {           // 16 bytes, or as many zeros
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                     "l"(src), "r"(in ? 16 : 0) : "memory");
    };
    // rows of k or q (from column `at` of r's rows) of chunk c
    auto fetch_rows = [&](float* to, int c, int at) {
        const int first = t0 + c * CHUNK, n = t1 - first;
        for (int i = tid; i < CHUNK * (D / 4); i += 256) {
            const int token = i / (D / 4), k = (i % (D / 4)) * 4;
            const bool in = token < n;
            copy(to + token * Y::ROW + k, r + (size_t)(in ? first + token : t0) * R + at + head * D + k, in);
        }
    };
    auto fetch_kv = [&](int c) {
        if (c < chunks) {
            fetch_rows(sm + Y::K + (c & 1) * CHUNK * Y::ROW, c, sh.cq());
            const int first = t0 + c * CHUNK, n = t1 - first;
            if (tid < CHUNK * RUN_COLS / 4) {
                const int token = tid / 4, k = (tid % 4) * 4;
                const bool in = token < n && col0 + k < e;
                copy(sm + Y::V + (c & 1) * CHUNK * RUN_COLS + token * RUN_COLS + k,
                     r + (in ? (size_t)(first + token) * R + 2 * sh.cq() + h * e + col0 + k : (size_t)t0 * R), in);
            }
        }
        copy_async_commit();
    };
    auto fetch_q = [&](int c) {
        if (c < chunks) fetch_rows(sm + Y::Q, c, 0);
        copy_async_commit();
    };
    auto fetch_tp = [&](int c) {
        if (c < chunks) {
            const double* tp = tp0 + (size_t)c * sh.H * CHUNK_DOUBLES;
            for (int i = tid * 2; i < CHUNK_DOUBLES; i += 512) copy(sm + Y::TP + 2 * i, tp + i, true);
        }
        copy_async_commit();
    };
    fetch_kv(0);
    fetch_q(0);
    fetch_tp(0);
    const double* T = reinterpret_cast<const double*>(sm + Y::TP);
    const double* P = T + CHUNK * CT;
    for (int c = 0; c < chunks; ++c) {
        copy_async_wait<1>();                          // k, v and q of this chunk; T and P may still be on their way
        __syncthreads();
        fetch_kv(c + 1);                               // (its places were last read in front of the barrier)
        const float* ks_rows = sm + Y::K + (c & 1) * CHUNK * Y::ROW;
        const float* vs = sm + Y::V + (c & 1) * CHUNK * RUN_COLS;
        const int n = t1 - t0 - c * CHUNK < CHUNK ? t1 - t0 - c * CHUNK : CHUNK;
        {   // S0^T k and S0^T q: warps 0-3 the k rows, 4-7 the q rows, a quarter of the channels each
            const int quarter = warp & 3, tm = lane & 7, tn = lane >> 3;
            const float* rows = (warp < 4 ? ks_rows : sm + Y::Q) + tm * Y::ROW + quarter * (D / 4);
            const float* cols = S + tn * Y::ROW + quarter * (D / 4);
            unsigned long long acc[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll
            for (int k = 0; k < D / 4; k += 4) {
                ulonglong2 a[4], b[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(rows + 8 * i * Y::ROW + k);
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(cols + 4 * j * Y::ROW + k);
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        fma_pair(acc[i][j], a[i].x, b[j].x);
                        fma_pair(acc[i][j], a[i].y, b[j].y);
                    }
            }
            float* to = red + quarter * (2 * CHUNK * 20) + ((warp >> 2) * CHUNK + tm) * 20 + tn;
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) to[i * 160 + 4 * j] = pair_sum(acc[i][j]);
        }
        copy_async_wait<1>();                          // T and P; the next chunk's k and v may still be on their way
        __syncthreads();
        fetch_q(c + 1);
        // the middle products: a warp has 8 tokens and 8 columns, a lane a token and two neighbouring columns
        const int g = lane >> 2, t = lane & 3, tokens0 = (warp >> 1) * 8, row = tokens0 + g, cc = (warp & 1) * 8 + 2 * t;
        double from_state[2];
        bool plain = false;
        {
            const double beta = T[row * CT + AT_BETA], G = P[row * CT + AT_G];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float* at = red + row * 20 + cc + j;
                const float ks = (at[0] + at[2 * CHUNK * 20]) + (at[4 * CHUNK * 20] + at[6 * CHUNK * 20]);
                at += CHUNK * 20;
                const float qs = (at[0] + at[2 * CHUNK * 20]) + (at[4 * CHUNK * 20] + at[6 * CHUNK * 20]);
                const double one = beta * ((double)vs[row * RUN_COLS + cc + j] - G * (double)ks);
                rt[(cc + j) * COL + row] = one;
                plain |= !isfinite(one);
                from_state[j] = G * (double)qs;
            }
        }
        // A token's row of T or P times the columns, up to the row's own token: rows end in zeros, which the tensor cores
        // multiply with later tokens' values all the same.  Where one of those is not finite, the row is added up to
        // its end instead.
        auto rows_times = [&](const double* m, const double* columns, bool plain_sums, double (&v)[2]) {
            v[0] = v[1] = 0.0;
            if (!plain_sums) {
                double odd[2] = {0.0, 0.0};
                for (int k = 0; k < tokens0 + 8; k += 8) {
                    const double* a = m + row * CT + k + t;
                    const double* b = columns + ((warp & 1) * 8 + g) * COL + k + t;
                    mma_f64(v, a[0], b[0]);
                    mma_f64(odd, a[4], b[4]);
                }
                v[0] += odd[0], v[1] += odd[1];
            } else {
                for (int k = 0; k <= row; ++k)
                    for (int j = 0; j < 2; ++j) v[j] = fma(m[row * CT + k], columns[(cc + j) * COL + k], v[j]);
            }
        };
        plain = __syncthreads_or(plain);
        {
            double u[2];
            rows_times(T, rt, plain, u);
            const double rest = P[row * CT + AT_REST];
            plain = false;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                ut[(cc + j) * COL + row] = u[j];
                un[row * UN_ROW + cc + j] = rest * u[j];
                plain |= !isfinite(u[j]);
            }
        }
        plain = __syncthreads_or(plain);
        {
            double v[2];
            rows_times(P, ut, plain, v);
            if (row < n) {
                float* at = o + ((size_t)(t0 + c * CHUNK + row) * sh.H + h) * e + col0;
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    if (col0 + cc + j < e) at[cc + j] = (float)(from_state[j] + v[j]);
            }
        }
        {   // S <- G_C S0 + sum_j k_j (D_Cj u_j), all tokens
            constexpr int M_TILES = D / 8, PER_WARP = M_TILES * 2 / 8;      // tiles of 8 channels by 8 columns
            const double last = P[(CHUNK - 1) * CT + AT_G];
            const int n0 = PER_WARP == 2 ? (warp & 1) * 8 : 0, m0 = PER_WARP == 2 ? (warp >> 1) * 16 : warp * 16;
            // D = 128: two tiles of channels, both of columns; D = 64: two of channels, one of columns
            double acc[2][PER_WARP / 2][2];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < PER_WARP / 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll
            for (int k = 0; k < CHUNK; k += 4) {
                const float* a = ks_rows + (k + t) * Y::ROW + m0 + g;
                const double a0 = a[0], a1 = a[8];
#pragma unroll
                for (int j = 0; j < PER_WARP / 2; ++j) {
                    const double b = un[(k + t) * UN_ROW + n0 + 8 * j + g];
                    mma_f64(acc[0][j], a0, b);
                    mma_f64(acc[1][j], a1, b);
                }
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < PER_WARP / 2; ++j)
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        float* at = S + (n0 + 8 * j + 2 * t + x) * Y::ROW + m0 + 8 * i + g;
                        *at = (float)fma(last, (double)*at, acc[i][j][x]);
                    }
        }
        __syncthreads();                               // S is whole, and T and P have been read
        fetch_tp(c + 1);
    }
    copy_async_wait<0>();
    fwb::pdl_launch_dependents();
    for (int i = tid; i < RUN_COLS * (D / 4); i += 256) {
        const int c = i / (D / 4), k = (i % (D / 4)) * 4;
        if (col0 + c < e)
            *reinterpret_cast<float4*>(slot + ((size_t)h * e + col0 + c) * D + k) = *reinterpret_cast<float4*>(S + c * Y::ROW + k);
    }
}

template <int DPL, int LPC, bool VEC>
int launch_scan(const float* r, const float* p, float* state, long long slot_stride, const int* seg_start,
                const int* seg_slot, float* o, int below, int T, int segments, const DeltaShape& sh, cudaStream_t stream) {
    // blocks that fit the SMs one by one must not meet on some of them, where they would land beside the last blocks of the
    // kernel in front: they ask for more than half of an SM's shared memory (16 heads of 128, 128 blocks, all launches, us
    // before and so: 256 tokens 149 117, 512 237 205, 1,024 449 385, 2,048 1,180 749, 4,096 2,580 1,476).  A walk of a few
    // tokens does not pay for waiting until an SM has that much free (a decode step of Diforax, ten such layers: 960 us, 972)
    constexpr int ALONE = 116 * 1024, COLS = 128 / LPC;
    auto kernel = delta_scan_kernel<DPL, LPC, VEC>;
    static bool configured = false;
    if (!configured) {
        cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ALONE);
        if (err != cudaSuccess) return (int)err;
        configured = true;
    }
    const dim3 grid((sh.e + COLS - 1) / COLS, sh.H, segments);
    const bool alone = T >= 64 && (long)grid.x * grid.y * grid.z <= 148;
    fwb::pdl(kernel, grid, 128, alone ? ALONE : 0, stream)(r, p, state, slot_stride, seg_start, seg_slot, o, below, sh);
    return fwb_launch_status();
}

// Segments `first` .. of at least `from` tokens, the longest of `longest`.
template <int D>
int launch_runs(const float* r, const float* p, double* scratch, float* state, long long slot_stride, const int* seg_start,
                const int* seg_slot, float* o, int first, int from, int longest, int n_segments, const DeltaShape& sh,
                cudaStream_t stream) {
    // blocks that fit the SMs one by one must not pair up on some of them (128 blocks, started in the shadow of the kernel
    // in front: 552 us for 2,048 tokens in pairs, 400 apart): they ask for more than half of an SM's shared memory
    constexpr int SMEM = RunLayout<D>::FLOATS * 4, ALONE = 120 * 1024;
    static bool configured = false;
    if (!configured) {
        cudaError_t err = cudaFuncSetAttribute(delta_runs_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, ALONE);
        if (err != cudaSuccess) return (int)err;
        configured = true;
    }
    const dim3 chunks((longest + CHUNK - 1) / CHUNK, sh.H, n_segments - first);
    fwb::pdl(delta_chunk_kernel<D>, chunks, 256, 0, stream)(r, seg_start + first, scratch, from, sh);
    const dim3 grid((sh.e + RUN_COLS - 1) / RUN_COLS, sh.H, n_segments - first);
    const bool alone = (long)grid.x * grid.y * grid.z <= 148;
    fwb::pdl(delta_runs_kernel<D>, grid, 256, alone ? ALONE : SMEM, stream)(r, p, scratch, state, slot_stride, seg_start + first,
                                                            seg_slot + first, o, from, sh);
    return fwb_launch_status();
}

template <typename TO>
__global__ void __launch_bounds__(128)
gated_head_norm_kernel(const float* __restrict__ o, const float* __restrict__ gate, long long gate_stride,
                       const float* __restrict__ weight, float scale, float eps, TO* __restrict__ out, long long out_stride,
                       int rows, int H, int e) {
    fwb::pdl_entry();
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= rows) return;
    const int t = row / H, h = row - t * H;
    const float* src = o + (size_t)row * e;
    const float* g = gate + (size_t)t * gate_stride + (size_t)h * e;
    TO* dst = out + (size_t)t * out_stride + (size_t)h * e;
    float ss = 0.0f;
    for (int i = lane; i < e; i += 32) ss = fmaf(src[i], src[i], ss);
    const float inv = rsqrtf(warp_sum(ss) / (float)e + eps);
    for (int i = lane; i < e; i += 32)
        dst[i] = from_f32<TO>(((src[i] * inv) * (weight ? weight[i] : scale)) * silu_f32(g[i]));
}

}  // namespace

// p: [T][2Gd + 2He + 2H] fp32 (q | k | v | gate | b | a).  taps: [2Gd + He][L] fp32.  a_log, dt_bias: [H].
// state: [slots][slot_stride] fp32 with S at 0 and the convolution's inputs behind it.
// r: [T][2Gd + He + 2H + G rounded up to a multiple of 4] fp32 scratch.  o: [T][H][e] fp32.
// scratch: null (every token through the scan), or [T / 32 + n_segments][H][2][32][34] fp64 on a 16-byte border: segments
// of `from` tokens and more go by chunks, the others through the scan; sizes that the chunks do not take all go through the
// scan.  The caller says where to look: no segment of the first `first` has `from` tokens, none behind the first `scanned`
// has fewer, and the longest has `longest`.
FWB_API int fwb_delta_rule(const float* p, const float* taps, const float* a_log, const float* dt_bias,
                           float* state, long long slot_stride, const int* seg_start, const int* seg_slot,
                           const int* tok_seg, float* r, float* o, double* scratch, int from, int longest, int first,
                           int scanned, int T, int n_segments, int H, int G, int d, int e, int L, cudaStream_t stream) {
    if (T <= 0 || n_segments <= 0) return FWB_OK;
    if (!p || !taps || !a_log || !dt_bias || !state || !seg_start || !seg_slot || !tok_seg || !r || !o)
        return FWB_BAD_ARGUMENT;
    if (H <= 0 || G <= 0 || H % G || d <= 0 || e <= 0 || L < 1) return FWB_BAD_ARGUMENT;
    if (L > MAX_TAPS || d > 256) return FWB_TOO_LARGE;
    const DeltaShape sh{H, G, d, e, L};
    if (slot_stride < (long long)H * d * e + (long long)sh.channels() * (L - 1)) return FWB_BAD_ARGUMENT;
    if (scratch && (from <= 0 || longest <= 0 || longest > T || first < 0 || first > n_segments || scanned < first ||
                    scanned > n_segments))
        return FWB_BAD_ARGUMENT;
    const size_t smem = (size_t)sh.channels() * sizeof(float);
    if (smem > 160 * 1024 || n_segments > 65535 || H > 65535) return FWB_TOO_LARGE;
    // tokens in fours once there are enough of them, where 16-byte loads can read everything
    const size_t window_smem = (size_t)PREP * 2 * sh.cq() * sizeof(float);
    if (T >= 128 && L == 4 && sh.cq() % 2 == 0 && sh.cv() % 4 == 0 && sh.p_width() % 4 == 0 && window_smem <= 100 * 1024 &&
        ((uintptr_t)p & 15) == 0 && ((uintptr_t)taps & 15) == 0 && ((uintptr_t)r & 15) == 0) {
        if (window_smem > 48 * 1024)
            cudaFuncSetAttribute(delta_prepare_window_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
        fwb::pdl(delta_prepare_window_kernel, dim3((T + PREP - 1) / PREP, 2), 256, window_smem, stream)(
            p, taps, a_log, dt_bias, state, slot_stride, seg_start, seg_slot, tok_seg, r, T, sh);
    } else {
        if (smem > 48 * 1024)
            cudaFuncSetAttribute(delta_prepare_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        const int prepare_threads = sh.channels() >= 2048 ? 512 : (sh.channels() >= 512 ? 256 : 128);
        fwb::pdl(delta_prepare_kernel, T, prepare_threads, smem, stream)(p, taps, a_log, dt_bias, state, slot_stride,
                                                                         seg_start, seg_slot, tok_seg, r, sh);
    }
    const bool vec = d % 4 == 0 && e % 4 == 0 && slot_stride % 4 == 0 && ((uintptr_t)state & 15) == 0 &&
                     ((uintptr_t)r & 15) == 0;
    const bool runs = scratch && vec && (d == 64 || d == 128) && ((uintptr_t)scratch & 15) == 0;
    const int below = runs ? from : 2147483647, scans = runs ? scanned : n_segments;
#define FWB_SCAN(DPL, LPC)                                                                                             \
    do {                                                                                                               \
        const int status = vec ? launch_scan<DPL, LPC, true>(r, p, state, slot_stride, seg_start, seg_slot, o, below, T, scans, sh, stream) \
                               : launch_scan<DPL, LPC, false>(r, p, state, slot_stride, seg_start, seg_slot, o, below, T, scans, sh, stream); \
        if (status != FWB_OK) return status;                                                                           \
    } while (0)
    if (scans > 0) {
        if (d <= 16) FWB_SCAN(4, 4);
        else if (d <= 32) FWB_SCAN(8, 4);
        else if (d <= 64) FWB_SCAN(16, 4);
        else if (d <= 128) FWB_SCAN(16, 8);
        else FWB_SCAN(32, 8);
    }
#undef FWB_SCAN
    if (runs && first < n_segments) {
        const int status = d == 64 ? launch_runs<64>(r, p, scratch, state, slot_stride, seg_start, seg_slot, o, first, from,
                                                     longest, n_segments, sh, stream)
                                   : launch_runs<128>(r, p, scratch, state, slot_stride, seg_start, seg_slot, o, first, from,
                                                      longest, n_segments, sh, stream);
        if (status != FWB_OK) return status;
    }
    return fwb_launch_status();
}

// o: [T][H][e] fp32; gate: row t at gate + t * gate_stride, [H][e] fp32; weight: [e], or null: every channel
// counts `scale`; out: row t at out + t * out_stride (0: H e), [H][e].
FWB_API int fwb_gated_head_norm(const float* o, const float* gate, long long gate_stride, const float* weight,
                                float scale, float eps, void* out, int out_bf16, long long out_stride, int T, int H,
                                int e, cudaStream_t stream) {
    if (T <= 0) return FWB_OK;
    if (!o || !gate || !out || H <= 0 || e <= 0) return FWB_BAD_ARGUMENT;
    if (out_stride == 0) out_stride = (long long)H * e;
    if (out_stride < (long long)H * e) return FWB_BAD_ARGUMENT;
    const long long rows = (long long)T * H;
    if (rows > 2147483647LL / 4) return FWB_TOO_LARGE;
    const int blocks = (int)((rows + 3) / 4);
    if (out_bf16)
        fwb::pdl(gated_head_norm_kernel<__nv_bfloat16>, blocks, 128, 0, stream)(
            o, gate, gate_stride, weight, scale, eps, (__nv_bfloat16*)out, out_stride, (int)rows, H, e);
    else
        fwb::pdl(gated_head_norm_kernel<float>, blocks, 128, 0, stream)(
            o, gate, gate_stride, weight, scale, eps, (float*)out, out_stride, (int)rows, H, e);
    return fwb_launch_status();
}
