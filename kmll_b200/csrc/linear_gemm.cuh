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
// One block per row of x: optional RMSNorm (kmll's order x * inv * w), power-of-two scale, hi / lo split.  Block 0
// also clears the split-K counters.
__global__ void __launch_bounds__(512) split_rows_kernel(const float* __restrict__ x, int ldx, int K, const uint16_t* __restrict__ norm_w,
                                                         float eps, __half* __restrict__ x_hi, __half* __restrict__ x_lo,
                                                         float* __restrict__ inv_xscale, unsigned int* counters, int n_counters, int permute) {
    __shared__ float scratch[40];
    pdl_wait();
    const int m = blockIdx.x;
    if (m == 0)
        for (int i = threadIdx.x; i < n_counters; i += blockDim.x) counters[i] = 0u;
    const float4* xr = reinterpret_cast<const float4*>(x + (size_t)m * ldx);
    const uint2* nw = reinterpret_cast<const uint2*>(norm_w);
    float ss = 0.0f, mx = 0.0f;
    for (int k4 = threadIdx.x; k4 < K / 4; k4 += blockDim.x) {
        const float4 v = xr[k4];
        ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
        if (norm_w) {
            const uint2 w = nw[k4];
            mx = fmaxf(mx, fmaxf(fmaxf(fabsf(v.x * __uint_as_float(w.x << 16)), fabsf(v.y * __uint_as_float(w.x & 0xffff0000u))),
                                 fmaxf(fabsf(v.z * __uint_as_float(w.y << 16)), fabsf(v.w * __uint_as_float(w.y & 0xffff0000u)))));
        } else {
            mx = fmaxf(mx, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
        }
    }
    ss = block_sum(ss, scratch);
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
    // eight columns per thread and step.  permute != 0 (W4-G128): inside every group of eight columns the planes hold the
    // columns in the order 0 4 1 5 2 6 3 7 - the order in which the weight expansion of linear_gemm_pair_kernel produces the
    // nibbles of a word; a contraction does not care in which order its terms are summed as long as both operands agree
    uint4* hi = reinterpret_cast<uint4*>(x_hi + (size_t)m * K);
    uint4* lo = reinterpret_cast<uint4*>(x_lo + (size_t)m * K);
    const uint4* nw8 = reinterpret_cast<const uint4*>(norm_w);
    for (int k8 = threadIdx.x; k8 < K / 8; k8 += blockDim.x) {
        const float4 a = xr[2 * k8], b = xr[2 * k8 + 1];
        float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        if (norm_w) {
            const uint4 w = nw8[k8];
            const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                v[2 * q] = v[2 * q] * inv * __uint_as_float(ww[q] << 16);
                v[2 * q + 1] = v[2 * q + 1] * inv * __uint_as_float(ww[q] & 0xffff0000u);
            }
        }
        uint32_t h[4], l[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int i0 = permute ? q : 2 * q, i1 = permute ? q + 4 : 2 * q + 1;
            const float v0 = v[i0] * xscale, v1 = v[i1] * xscale;
            const __half2 hh = __floats2half2_rn(v0, v1);
            const float2 hf = __half22float2(hh);
            const __half2 ll = __floats2half2_rn(v0 - hf.x, v1 - hf.y);
            h[q] = *reinterpret_cast<const uint32_t*>(&hh);
            l[q] = *reinterpret_cast<const uint32_t*>(&ll);
        }
        hi[k8] = make_uint4(h[0], h[1], h[2], h[3]);
        lo[k8] = make_uint4(l[0], l[1], l[2], l[3]);
    }
    if (threadIdx.x == 0) inv_xscale[m] = inv_scale;
}

// ---- tcgen05 / TMA helpers ------------------------------------------------------------------------------------------
__device__ inline void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ inline void tcgen05_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ inline void tcgen05_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ inline void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// shared-memory matrix descriptor: K-major operand tile with 128-byte rows in the 128-byte swizzle (what TMA writes with
// CU_TENSOR_MAP_SWIZZLE_128B): groups of 8 rows are 1024 bytes apart; version 1 (sm_100); layout type 2 = SWIZZLE_128B
__device__ inline uint64_t gemm_smem_desc(uint32_t smem_addr) {
    return (uint64_t)((smem_addr >> 4) & 0x3fffu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// instruction descriptor of kind::f16: D = f32, A = B = binary16, both K-major, N >> 3 at bit 17, M >> 4 at bit 24
__host__ __device__ constexpr uint32_t gemm_idesc_f16(int m, int n) {
    return (1u << 4) | (0u << 7) | (0u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ inline void gemm_mma_f16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}
__device__ inline void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// 2-D tiled TMA load into this block's shared memory (no multicast), completion on an mbarrier
__device__ inline void tma_load_2d(uint32_t smem_dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(smem_dst), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
                 : "memory");
}

// 3-D tiled TMA load (inner, row, plane)
__device__ inline void tma_load_3d(uint32_t smem_dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(smem_dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
                 : "memory");
}

}  // namespace kmll
