// Folding of a net's parameters into the stacks the forward kernels read (kernels/reference.py:68-91): V' = V * rms_w and
// U' = alpha * U, each operand rounded to bf16, products formed in fp32 and rounded once.
//
// Bound by memory: every value is read once and written once.  The layers' tensors are read where they are (their addresses
// travel as a kernel parameter), so that no stacked copy is made first, eight values per load and store, four loads in
// flight per thread.  d = 2048, r = 64, L = 142 (149 MB in and out): about 30 us; one value per thread over a stacked copy,
// with a 64-bit division each, took 250 us with the copies.
#include <cuda_bf16.h>
#include <stdint.h>

#include "fold.h"

namespace dlr {

namespace {

constexpr int kLayersPerLaunch = 128;
constexpr int kThreadsF = 256;
constexpr int kUnroll = 4;

struct Addresses {
    const void* V[kLayersPerLaunch];
    const void* U[kLayersPerLaunch];
    const void* gain[kLayersPerLaunch];
    const void* alpha[kLayersPerLaunch];
};

template <bool F32>
__device__ __forceinline__ float value(const void* p, size_t i) {
    if constexpr (F32) return __bfloat162float(__float2bfloat16_rn(static_cast<const float*>(p)[i]));
    else return __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]);
}

// eight values from an aligned address, rounded to bf16
template <bool F32>
__device__ __forceinline__ uint4 load8(const void* p, size_t i8) {
    if constexpr (F32) {
        const float4 a = __ldg(static_cast<const float4*>(p) + 2 * i8), b = __ldg(static_cast<const float4*>(p) + 2 * i8 + 1);
        uint4 v;
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
        h[0] = __floats2bfloat162_rn(a.x, a.y);
        h[1] = __floats2bfloat162_rn(a.z, a.w);
        h[2] = __floats2bfloat162_rn(b.x, b.y);
        h[3] = __floats2bfloat162_rn(b.z, b.w);
        return v;
    } else {
        return __ldg(static_cast<const uint4*>(p) + i8);
    }
}

__device__ __forceinline__ uint4 times(uint4 a, uint4 g) {
    uint4 o;
    const __nv_bfloat162* x = reinterpret_cast<const __nv_bfloat162*>(&a);
    const __nv_bfloat162* y = reinterpret_cast<const __nv_bfloat162*>(&g);
    __nv_bfloat162* z = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 p = __bfloat1622float2(x[k]), q = __bfloat1622float2(y[k]);
        z[k] = __floats2bfloat162_rn(p.x * q.x, p.y * q.y);
    }
    return o;
}

__device__ __forceinline__ uint4 times(uint4 a, float s) {
    uint4 o;
    const __nv_bfloat162* x = reinterpret_cast<const __nv_bfloat162*>(&a);
    __nv_bfloat162* z = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 p = __bfloat1622float2(x[k]);
        z[k] = __floats2bfloat162_rn(p.x * s, p.y * s);
    }
    return o;
}

// blockIdx = (share of a matrix, layer of this launch, V or U)
template <bool F32, bool VEC>
__global__ void __launch_bounds__(kThreadsF) fold_kernel(const __grid_constant__ Addresses at, bool alpha_f32, bool round_alpha,
                                                         __nv_bfloat16* Vp, __nv_bfloat16* Up, int d, uint32_t n) {
    const int l = blockIdx.y;
    const bool is_u = blockIdx.z != 0;
    const void* src = is_u ? at.U[l] : at.V[l];
    __nv_bfloat16* dst = (is_u ? Up : Vp) + size_t(l) * n;
    float s = 0.f;
    if (is_u) {
        s = alpha_f32 ? *static_cast<const float*>(at.alpha[l]) : __bfloat162float(*static_cast<const __nv_bfloat16*>(at.alpha[l]));
        if (alpha_f32 && round_alpha) s = __bfloat162float(__float2bfloat16_rn(s));
    }
    if constexpr (VEC) {
        const uint32_t n8 = n / 8, d8 = uint32_t(d) / 8, i0 = blockIdx.x * (kThreadsF * kUnroll) + threadIdx.x;
        uint4 v[kUnroll], g[kUnroll];
#pragma unroll
        for (int k = 0; k < kUnroll; ++k) {
            const uint32_t i = i0 + k * kThreadsF;
            if (i < n8) {
                v[k] = load8<F32>(src, i);
                if (!is_u) g[k] = load8<F32>(at.gain[l], i % d8);
            }
        }
#pragma unroll
        for (int k = 0; k < kUnroll; ++k) {
            const uint32_t i = i0 + k * kThreadsF;
            if (i < n8) reinterpret_cast<uint4*>(dst)[i] = is_u ? times(v[k], s) : times(v[k], g[k]);
        }
    } else {
        for (uint32_t i = blockIdx.x * kThreadsF + threadIdx.x; i < n; i += gridDim.x * kThreadsF)
            dst[i] = __float2bfloat16_rn(value<F32>(src, i) * (is_u ? s : value<F32>(at.gain[l], i % uint32_t(d))));
    }
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

bool fold_layers(const void* const* V, const void* const* U, const void* const* gain, const void* const* alpha,
                 bool matrices_f32, bool alpha_f32, bool round_alpha, void* Vp, void* Up, int d, int r, int L,
                 cudaStream_t stream) {
    const size_t n = size_t(r) * d;
    if (n > 0x7fffffffu) return false;
    for (int l0 = 0; l0 < L; l0 += kLayersPerLaunch) {
        const int layers = L - l0 < kLayersPerLaunch ? L - l0 : kLayersPerLaunch;
        Addresses at;
        bool vec = d % 8 == 0 && aligned16(Vp) && aligned16(Up);
        for (int l = 0; l < layers; ++l) {
            at.V[l] = V[l0 + l];
            at.U[l] = U[l0 + l];
            at.gain[l] = gain[l0 + l];
            at.alpha[l] = alpha[l0 + l];
            vec = vec && aligned16(at.V[l]) && aligned16(at.U[l]) && aligned16(at.gain[l]);
        }
        const unsigned per = vec ? kThreadsF * kUnroll * 8 : kThreadsF * 8;
        const dim3 grid(unsigned((n + per - 1) / per), layers, 2);
        __nv_bfloat16* vp = static_cast<__nv_bfloat16*>(Vp) + size_t(l0) * n;
        __nv_bfloat16* up = static_cast<__nv_bfloat16*>(Up) + size_t(l0) * n;
        auto kern = matrices_f32 ? (vec ? fold_kernel<true, true> : fold_kernel<true, false>)
                                 : (vec ? fold_kernel<false, true> : fold_kernel<false, false>);
        kern<<<grid, kThreadsF, 0, stream>>>(at, alpha_f32, round_alpha, vp, up, d, uint32_t(n));
    }
    return true;
}

}  // namespace dlr
