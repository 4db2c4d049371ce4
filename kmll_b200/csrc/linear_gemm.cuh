// What the tcgen05 kernels share, included by linear.cu: activations as two binary16 planes, tcgen05 / TMA helpers.
//
// f16 carries 11 significant bits, f32 activations 24: x = 2^-sh (x_hi + x_lo), x_hi = f16(x 2^sh), x_lo = f16(x 2^sh - x_hi), with
// 2^sh putting the row maximum near 2^14.  The rounding of x_lo is below 2^-22 of the product; all products with integer weights
// are exact in the f32 accumulators.
#pragma once

#include <cuda.h>

namespace kmll {

constexpr int kGMaxN = 256;        // rows of x per unit of work = MMA N (multiple of 16)
constexpr int kGKT = 64;           // columns per k-tile (one 128-byte swizzle atom of f16)
constexpr int kGMaxSplit = 8;

// ---- activations -> f16 planes ----------------------------------------------------------------------------------
// One block per row of x: optional RMSNorm (kmll's order x * inv * w) or SiLU(x) * up, power-of-two scale, hi / lo split.
// Block 0 also clears the split-K counters.  Bound by HBM: the row stays in registers between the pass that finds the scale
// and the one that writes (rows up to 16384 columns; what lies beyond is read again).  With `up` the activation never exists
// in memory: 2048 x 14336 in 67 us instead
// of ~100 through an element-wise kernel and a plain split.  Two blocks of 512 threads per multiprocessor, so that one row's loads
// run behind another's arithmetic (one block: 97 us).
__device__ inline float split_silu_mul(float g, float u) { return (g / (1.0f + expf(-g))) * u; }  // (silu_mul_f32 of elementwise.cu)

__device__ inline void split_load8(const float* xr, const float* ur, int k8, float (&v)[8]) {
    const float4 a = reinterpret_cast<const float4*>(xr)[2 * k8], b = reinterpret_cast<const float4*>(xr)[2 * k8 + 1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    if (ur != nullptr) {
        const float4 c = reinterpret_cast<const float4*>(ur)[2 * k8], d = reinterpret_cast<const float4*>(ur)[2 * k8 + 1];
        const float u[8] = {c.x, c.y, c.z, c.w, d.x, d.y, d.z, d.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = split_silu_mul(v[j], u[j]);
    }
}
// bf16 norm weights of eight columns (two 8-byte loads: callers guarantee no more than that)
__device__ inline void split_norm8(const uint16_t* norm_w, int k8, float (&w)[8]) {
    const uint2 p = reinterpret_cast<const uint2*>(norm_w)[2 * k8], q = reinterpret_cast<const uint2*>(norm_w)[2 * k8 + 1];
    const uint32_t ww[4] = {p.x, p.y, q.x, q.y};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        w[2 * j] = __uint_as_float(ww[j] << 16);
        w[2 * j + 1] = __uint_as_float(ww[j] & 0xffff0000u);
    }
}

// kHold: pieces of eight columns a thread keeps, 1 (up to 4096 columns), 2 or 4.
template <int kHold>
__global__ void __launch_bounds__(512, 2) split_rows_kernel(const float* __restrict__ x, const float* __restrict__ up, int ldx, int K,
                                                         const uint16_t* __restrict__ norm_w, float eps, __half* __restrict__ x_hi,
                                                         __half* __restrict__ x_lo, float* __restrict__ inv_xscale, unsigned int* counters,
                                                         int n_counters, int permute) {
    __shared__ float scratch[40];
    pdl_wait();
    const int m = blockIdx.x;
    if (m == 0)
        for (int i = threadIdx.x; i < n_counters; i += blockDim.x) counters[i] = 0u;
    const float* xr = x + (size_t)m * ldx;
    const float* ur = up != nullptr ? up + (size_t)m * ldx : nullptr;
    const int n8 = K / 8;
    float held[kHold][8];
    float ss = 0.0f, mx = 0.0f;
    auto look = [&](const float (&v)[8], int k8) {
        if (norm_w) {
            float w[8];
            split_norm8(norm_w, k8, w);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                ss += v[j] * v[j];
                mx = fmaxf(mx, fabsf(v[j] * w[j]));
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) mx = fmaxf(mx, fabsf(v[j]));
        }
    };
#pragma unroll
    for (int c = 0; c < kHold; ++c) {
        const int k8 = (int)threadIdx.x + c * 512;
        if (k8 < n8) split_load8(xr, ur, k8, held[c]);
    }
#pragma unroll
    for (int c = 0; c < kHold; ++c) {
        const int k8 = (int)threadIdx.x + c * 512;
        if (k8 < n8) look(held[c], k8);
    }
    for (int k8 = (int)threadIdx.x + kHold * 512; k8 < n8; k8 += 512) {
        float v[8];
        split_load8(xr, ur, k8, v);
        look(v, k8);
    }
    if (norm_w) ss = block_sum(ss, scratch);
    mx = block_max(mx, scratch);
    const float inv = norm_w ? 1.0f / sqrtf(ss / (float)K + eps) : 1.0f;
    const float amax = mx * inv * 1.00001f;
    float xscale = 0.0f, inv_scale = 1.0f;
    if (amax > 0.0f && amax < INFINITY) {
        const int e = (int)((__float_as_uint(amax) >> 23) & 0xff) - 127;
        int sh = 13 - e;  // the row maximum lands in [2^13, 2^14): far from the binary16 overflow
        sh = sh > 126 ? 126 : (sh < -126 ? -126 : sh);
        xscale = __uint_as_float((uint32_t)(sh + 127) << 23);
        inv_scale = __uint_as_float((uint32_t)(127 - sh) << 23);
    }
    // permute != 0 (W4-G128): inside every group of eight columns the planes hold the columns in the order 0 4 1 5 2 6 3 7 - the
    // order in which the weight expansion of linear_gemm_pair_kernel produces the nibbles of a word; a contraction does not care
    // in which order its terms are summed as long as both operands agree
    uint4* hi = reinterpret_cast<uint4*>(x_hi + (size_t)m * K);
    uint4* lo = reinterpret_cast<uint4*>(x_lo + (size_t)m * K);
    auto write = [&](float (&v)[8], int k8) {
        if (norm_w) {
            float w[8];
            split_norm8(norm_w, k8, w);
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = v[j] * inv * w[j];
        }
        uint32_t h[4], l[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float v0 = (permute ? v[q] : v[2 * q]) * xscale, v1 = (permute ? v[q + 4] : v[2 * q + 1]) * xscale;
            const __half2 hh = __floats2half2_rn(v0, v1);
            const float2 hf = __half22float2(hh);
            const __half2 ll = __floats2half2_rn(v0 - hf.x, v1 - hf.y);
            h[q] = *reinterpret_cast<const uint32_t*>(&hh);
            l[q] = *reinterpret_cast<const uint32_t*>(&ll);
        }
        hi[k8] = make_uint4(h[0], h[1], h[2], h[3]);
        lo[k8] = make_uint4(l[0], l[1], l[2], l[3]);
    };
#pragma unroll
    for (int c = 0; c < kHold; ++c) {
        const int k8 = (int)threadIdx.x + c * 512;
        if (k8 < n8) write(held[c], k8);
    }
    for (int k8 = (int)threadIdx.x + kHold * 512; k8 < n8; k8 += 512) {
        float v[8];
        split_load8(xr, ur, k8, v);
        write(v, k8);
    }
    if (threadIdx.x == 0) inv_xscale[m] = inv_scale;
}

}  // namespace kmll
