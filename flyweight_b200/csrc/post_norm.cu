// Kernels for layers that put a weighted RMS norm on a sublayer's output before the residual sum, and
// the gated product of a feed-forward with a choice of activation.
//
//   fwb_rmsnorm_add:   x[t] += w * y[t] / sqrt(mean(y[t]^2) + eps)                 (fp32, in place)
//                      and, when a second weight is given, the norm that the next sublayer reads,
//                      h[t] = w2 * x[t] / sqrt(mean(x[t]^2) + eps2), from the new x in the same pass
//   fwb_gate_act_mul:  out[t][f] = act(gu[t][f]) * gu[t][F + f],  act = silu | gelu (tanh form); or the clamped
//                      swish, min(g, L) sigmoid(1.702 min(g, L)) (clamp(u, -L, L) + 1)
// All arithmetic is fp32; a row is summed in an order that depends on its length alone.
#include "common.cuh"

using namespace fwb;

namespace {

template <typename TO>
__global__ void __launch_bounds__(256)
rmsnorm_add_kernel(float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ w, float eps,
                   const float* __restrict__ w2, float eps2, TO* __restrict__ h, int H) {
    fwb::pdl_entry();
    extern __shared__ float row[];            // the new x of this row
    __shared__ float scratch[33];
    const size_t base = (size_t)blockIdx.x * H;
    float ss = 0.0f;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        const float v = y[base + i];
        ss = fmaf(v, v, ss);
    }
    const float inv = rsqrtf(block_sum(ss, scratch) / (float)H + eps);
    float sx = 0.0f;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        const float v = x[base + i] + (y[base + i] * inv) * w[i];
        x[base + i] = v;
        if (w2) {
            row[i] = v;
            sx = fmaf(v, v, sx);
        }
    }
    if (!w2) return;
    const float inv2 = rsqrtf(block_sum(sx, scratch) / (float)H + eps2);
    for (int i = threadIdx.x; i < H; i += blockDim.x) h[base + i] = from_f32<TO>((row[i] * inv2) * w2[i]);
}

// The same with a row in registers, VEC float4 a thread: y and x are asked for together and read once, the weights
// before the wait (they are nobody's output).  Bound by memory at prompt sizes and by the chain of its two
// reductions in a decode step; the kernel above reads y twice, 4 bytes a load.
template <typename TO, int VEC, bool NEXT>
__global__ void __launch_bounds__(256)
rmsnorm_add_vec_kernel(float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ w, float eps,
                       const float* __restrict__ w2, float eps2, TO* __restrict__ h, int H) {
    fwb::pdl_launch_dependents();
    __shared__ float scratch[33];
    const int n4 = H >> 2;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 wv[VEC], wn[NEXT ? VEC : 1];
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
        const int c = threadIdx.x + i * 256;
        wv[i] = c < n4 ? reinterpret_cast<const float4*>(w)[c] : zero;
        if (NEXT) wn[i] = c < n4 ? reinterpret_cast<const float4*>(w2)[c] : zero;
    }
    fwb::pdl_wait();
    float4* xr = reinterpret_cast<float4*>(x + (size_t)blockIdx.x * H);
    const float4* yr = reinterpret_cast<const float4*>(y + (size_t)blockIdx.x * H);
    float4 v[VEC], r[VEC];
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
        const int c = threadIdx.x + i * 256;
        v[i] = c < n4 ? yr[c] : zero;
        r[i] = c < n4 ? xr[c] : zero;
    }
    float ss = 0.0f;
#pragma unroll
    for (int i = 0; i < VEC; ++i) ss += v[i].x * v[i].x + v[i].y * v[i].y + v[i].z * v[i].z + v[i].w * v[i].w;
    const float inv = rsqrtf(block_sum(ss, scratch) / (float)H + eps);
    float sx = 0.0f;
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
        const int c = threadIdx.x + i * 256;
        r[i].x += (v[i].x * inv) * wv[i].x, r[i].y += (v[i].y * inv) * wv[i].y;
        r[i].z += (v[i].z * inv) * wv[i].z, r[i].w += (v[i].w * inv) * wv[i].w;
        if (c < n4) xr[c] = r[i];
        sx += r[i].x * r[i].x + r[i].y * r[i].y + r[i].z * r[i].z + r[i].w * r[i].w;
    }
    if constexpr (NEXT) {
        const float inv2 = rsqrtf(block_sum(sx, scratch) / (float)H + eps2);
        TO* out = h + (size_t)blockIdx.x * H;
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
            const int c = threadIdx.x + i * 256;
            if (c >= n4) continue;
            const float a = (r[i].x * inv2) * wn[i].x, b = (r[i].y * inv2) * wn[i].y;
            const float cc = (r[i].z * inv2) * wn[i].z, d = (r[i].w * inv2) * wn[i].w;
            if (sizeof(TO) == 4) {
                reinterpret_cast<float4*>(out)[c] = make_float4(a, b, cc, d);
            } else {
                __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(cc, d);
                reinterpret_cast<uint2*>(out)[c] = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
            }
        }
    }
}

template <typename TO, bool NEXT>
void launch_vec(float* x, const float* y, const float* w, float eps, const float* w2, float eps2, TO* h, int T, int H,
                cudaStream_t stream) {
    const int vec = (H / 4 + 255) / 256;
    if (vec == 1) fwb::pdl(rmsnorm_add_vec_kernel<TO, 1, NEXT>, T, 256, 0, stream)(x, y, w, eps, w2, eps2, h, H);
    else if (vec == 2) fwb::pdl(rmsnorm_add_vec_kernel<TO, 2, NEXT>, T, 256, 0, stream)(x, y, w, eps, w2, eps2, h, H);
    else if (vec == 3) fwb::pdl(rmsnorm_add_vec_kernel<TO, 3, NEXT>, T, 256, 0, stream)(x, y, w, eps, w2, eps2, h, H);
    else fwb::pdl(rmsnorm_add_vec_kernel<TO, 4, NEXT>, T, 256, 0, stream)(x, y, w, eps, w2, eps2, h, H);
}

template <typename TI, typename TO>
__global__ void gate_act_mul_kernel(const TI* __restrict__ gu, TO* __restrict__ out, int T, int F, int act,
                                    float limit) {
    fwb::pdl_entry();
    const size_t n = (size_t)T * F;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const size_t t = i / F, f = i - t * F;
        const float g = to_f32<TI>(gu[t * 2 * F + f]);
        const float u = to_f32<TI>(gu[t * 2 * F + F + f]);
        out[i] = from_f32<TO>(gated_f32(act, limit, g, u));
    }
}

}  // namespace

// x, y: [T][H] fp32; w: [H] fp32.  w2 (may be null), eps2, h ([T][H], fp32 or bf16): the next norm.
FWB_API int fwb_rmsnorm_add(float* x, const float* y, const float* w, float eps, const float* w2, float eps2,
                            void* h, int h_bf16, int T, int H, cudaStream_t stream) {
    if (T <= 0) return FWB_OK;
    if (!x || !y || !w || H <= 0 || (w2 && !h)) return FWB_BAD_ARGUMENT;
    const size_t smem = w2 ? (size_t)H * sizeof(float) : 0;
    if (smem > 160 * 1024) return FWB_TOO_LARGE;
    // rows of 16-byte pieces that 256 threads hold in registers (shorter ones leave most of them idle)
    const bool aligned = (((uintptr_t)x | (uintptr_t)y | (uintptr_t)w | (uintptr_t)w2 | (uintptr_t)h) & 15) == 0;
    if ((H & 3) == 0 && H >= 512 && H <= 4096 && aligned) {
        if (!w2) launch_vec<float, false>(x, y, w, eps, nullptr, 0.0f, nullptr, T, H, stream);
        else if (h_bf16) launch_vec<__nv_bfloat16, true>(x, y, w, eps, w2, eps2, (__nv_bfloat16*)h, T, H, stream);
        else launch_vec<float, true>(x, y, w, eps, w2, eps2, (float*)h, T, H, stream);
        return fwb_launch_status();
    }
    if (h_bf16) {
        if (smem > 48 * 1024)
            cudaFuncSetAttribute(rmsnorm_add_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        fwb::pdl(rmsnorm_add_kernel<__nv_bfloat16>, T, 256, smem, stream)(x, y, w, eps, w2, eps2, (__nv_bfloat16*)h, H);
    } else {
        if (smem > 48 * 1024)
            cudaFuncSetAttribute(rmsnorm_add_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        fwb::pdl(rmsnorm_add_kernel<float>, T, 256, smem, stream)(x, y, w, eps, w2, eps2, (float*)h, H);
    }
    return fwb_launch_status();
}

// gu: [T][2F] (gate columns, then up columns); out: [T][F].  act: 0 silu, 1 gelu (tanh form), 2 the clamped
// swish with its `limit`, 3 relu.
FWB_API int fwb_gate_act_mul(const void* gu, int in_bf16, void* out, int out_bf16, int T, int F, int act,
                             float limit, cudaStream_t stream) {
    if (T <= 0) return FWB_OK;
    if (!gu || !out || F <= 0 || act < 0 || act > 3) return FWB_BAD_ARGUMENT;
    const size_t n = (size_t)T * F;
    const int blocks = (int)((n + 255) / 256 > 8192 ? 8192 : (n + 255) / 256);
    if (in_bf16 && out_bf16)
        fwb::pdl(gate_act_mul_kernel<__nv_bfloat16, __nv_bfloat16>, blocks, 256, 0, stream)(
            (const __nv_bfloat16*)gu, (__nv_bfloat16*)out, T, F, act, limit);
    else if (!in_bf16 && out_bf16)
        fwb::pdl(gate_act_mul_kernel<float, __nv_bfloat16>, blocks, 256, 0, stream)(
            (const float*)gu, (__nv_bfloat16*)out, T, F, act, limit);
    else if (!in_bf16 && !out_bf16)
        fwb::pdl(gate_act_mul_kernel<float, float>, blocks, 256, 0, stream)((const float*)gu, (float*)out, T, F, act, limit);
    else
        return FWB_UNSUPPORTED;
    return fwb_launch_status();
}
