// Device-side quantizers and dequantizers.  They restate kmll's host quantizer
// (RowwiseScaledI8Matrix::from_bf16_rows_symmetric, crates/inference/src/rowwise_scaled.rs:21-51)
// with IEEE f32 division and round-half-away-from-zero, so the produced bytes are identical to
// the host result; max() is order-independent, hence the parallel reduction is exact.
#include "internal.cuh"

namespace kmll {

__device__ inline float clamp_f32(float v, float lo, float hi) { return v < lo ? lo : (v > hi ? hi : v); }

// round(v / scale), half away from zero, as the host rule computes it.  An IEEE division per element was what bounded the
// quantizers; v * (1 / scale) differs from the quotient by less than 3e-5 for results up to 127, so the two can only round apart
// within 1e-4 of a tie, and there (and for anything not finite) the division decides.  `inv` = 1 / scale.  The integer is in the low
// bits of the returned word.
__device__ inline uint32_t round_quotient(float v, float scale, float inv, float limit) {
    constexpr float kMagic = 12582912.0f;  // 1.5 2^23: adding it rounds to a whole number, ties aside
    const float t = v * inv, m = t + kMagic;
    if (!(fabsf(t - (m - kMagic)) <= 0.4999f)) return (uint32_t)(int)clamp_f32(roundf(v / scale), -limit, limit);
    return (uint32_t)(__float_as_int(fminf(fmaxf(m, kMagic - limit), kMagic + limit)) - __float_as_int(kMagic));
}

// One block per row.  kHold > 0 (rows of whole 8-column pieces, aligned): bound by HBM, 16-byte loads; a thread keeps up to kHold pieces
// between the maximum and the rounding (with 4: 16384 columns per block, further ones are read again).  14336 x 4096: 65 -> 49 us =
// 3.6 TB/s; what is left is the block reduction between the two halves of a row.  Small matrices are bound by latency, which four
// pieces one after another in a thread add to: 896 x 896 5.0 us with 4 pieces, 2.8 with one (value by value: 3.5).  kHold = 0: value
// by value.
template <int kHold>
__global__ void __launch_bounds__(512, 2) quantize_rs_i8_kernel(const uint16_t* __restrict__ w, int cols,
                                                             int8_t* __restrict__ values, float* __restrict__ scales) {
    __shared__ float scratch[40];
    const size_t base = (size_t)blockIdx.x * cols;
    float mx = 0.0f;
    if constexpr (kHold > 0) {
        const uint4* src = reinterpret_cast<const uint4*>(w + base);
        const int n8 = cols >> 3;
        uint4 held[kHold];
        auto look = [&](const uint4& q) {
            const uint32_t ww[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) mx = fmaxf(mx, fmaxf(fabsf(__uint_as_float(ww[j] << 16)), fabsf(__uint_as_float(ww[j] & 0xffff0000u))));
        };
#pragma unroll
        for (int h = 0; h < kHold; ++h) {
            const int c = threadIdx.x + h * blockDim.x;
            held[h] = c < n8 ? __ldg(src + c) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int h = 0; h < kHold; ++h) look(held[h]);
        if (kHold > 1)
            for (int c = threadIdx.x + kHold * blockDim.x; c < n8; c += blockDim.x) look(__ldg(src + c));
        mx = block_max(mx, scratch);
        const float scale = (mx == 0.0f) ? 1.0f : mx / 127.0f, inv = 1.0f / scale;
        if (threadIdx.x == 0) scales[blockIdx.x] = scale;
        uint2* dst = reinterpret_cast<uint2*>(values + base);
        auto put = [&](const uint4& q, int c) {
            const uint32_t ww[4] = {q.x, q.y, q.z, q.w};
            uint32_t o[2] = {0u, 0u};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                o[j >> 1] |= (round_quotient(__uint_as_float(ww[j] << 16), scale, inv, 127.0f) & 0xffu) << (16 * (j & 1));
                o[j >> 1] |= (round_quotient(__uint_as_float(ww[j] & 0xffff0000u), scale, inv, 127.0f) & 0xffu) << (16 * (j & 1) + 8);
            }
            dst[c] = make_uint2(o[0], o[1]);
        };
#pragma unroll
        for (int h = 0; h < kHold; ++h) {
            const int c = threadIdx.x + h * blockDim.x;
            if (c < n8) put(held[h], c);
        }
        if (kHold > 1)
            for (int c = threadIdx.x + kHold * blockDim.x; c < n8; c += blockDim.x) put(__ldg(src + c), c);
    } else {
        for (int c = threadIdx.x; c < cols; c += 256) mx = fmaxf(mx, fabsf(bf16_bits_to_f32(w[base + c])));
        mx = block_max(mx, scratch);
        const float scale = (mx == 0.0f) ? 1.0f : mx / 127.0f;
        if (threadIdx.x == 0) scales[blockIdx.x] = scale;
        for (int c = threadIdx.x; c < cols; c += 256) {
            const float q = clamp_f32(roundf(bf16_bits_to_f32(w[base + c]) / scale), -127.0f, 127.0f);
            values[base + c] = (int8_t)(int)q;
        }
    }
}

// Dequantizers: bound by the f32 stores; a thread turns four values into 16 bytes, kSteps times, so that several loads are in
// flight and a warp's stores are contiguous (14336 x 4096: RS-I8 167 -> 49 us = 6.0 TB/s, W4 166 -> 47 us = 5.6 TB/s; one value per thread
// was bound by address arithmetic, a 64-bit division per value in the RS-I8 form).  RS-I8 rows that are not a multiple of four columns go one value per thread.
template <int kSteps>
__global__ void __launch_bounds__(256) dequant_rs_i8_quads_kernel(const uint32_t* __restrict__ values, const float* __restrict__ scales, uint32_t quads,
                                                                  uint32_t quads_per_row, float4* __restrict__ out) {
    const uint32_t first = blockIdx.x * (256u * kSteps) + threadIdx.x;
    uint32_t v[kSteps];
    float s[kSteps];
#pragma unroll
    for (int j = 0; j < kSteps; ++j) {
        const uint32_t i = first + 256u * j;
        if (i < quads) {
            v[j] = __ldg(values + i);
            s[j] = __ldg(scales + i / quads_per_row);
        }
    }
#pragma unroll
    for (int j = 0; j < kSteps; ++j) {
        const uint32_t i = first + 256u * j;
        if (i < quads)
            out[i] = make_float4((float)(int8_t)v[j] * s[j], (float)(int8_t)(v[j] >> 8) * s[j], (float)(int8_t)(v[j] >> 16) * s[j], (float)(int8_t)(v[j] >> 24) * s[j]);
    }
}

__global__ void dequant_rs_i8_kernel(const int8_t* __restrict__ values, const float* __restrict__ scales, int rows,
                                     int cols, float* __restrict__ out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)rows * cols) return;
    out[i] = (float)values[i] * scales[i / cols];
}

// kPer consecutive columns of a 128-column group per lane.  16 (eight lanes, 64 bytes in, 8 bytes out): four 16-byte loads in flight per
// lane and three shuffles per group; 14336 x 4096: 74 us (one warp per group, one load per lane, IEEE divisions) -> 44 us = 6.0 TB/s.
// 4 (a warp): a quarter of the work one after another, for matrices that do not fill the chip (896 x 896: 3.1 us with 16, 2.5 with 4).
template <int kPer>
__global__ void __launch_bounds__(256) quantize_w4_kernel(const float* __restrict__ w, size_t n_groups,
                                                          uint8_t* __restrict__ packed, uint16_t* __restrict__ gscales) {
    constexpr int kLanes = 128 / kPer;
    const int part = threadIdx.x & (kLanes - 1);
    const size_t grp = (size_t)blockIdx.x * (256 / kLanes) + threadIdx.x / kLanes;
    const bool live = grp < n_groups;
    float4 v[kPer / 4];
    float mx = 0.0f;
#pragma unroll
    for (int j = 0; j < kPer / 4; ++j) v[j] = live ? reinterpret_cast<const float4*>(w + grp * 128 + part * kPer)[j] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int j = 0; j < kPer / 4; ++j) mx = fmaxf(mx, fmaxf(fmaxf(fabsf(v[j].x), fabsf(v[j].y)), fmaxf(fabsf(v[j].z), fabsf(v[j].w))));
#pragma unroll
    for (int off = 1; off < kLanes; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    if (!live) return;
    const float scale_f32 = (mx == 0.0f) ? 1.0f : mx / 7.0f;
    __half sh = __float2half_rn(scale_f32);
    uint16_t sbits = __half_as_ushort(sh);
    if ((sbits & 0x7fffu) == 0) {
        sbits = 0x0001u;  // never divide by a zero scale
        sh = __ushort_as_half(sbits);
    }
    if (part == 0) gscales[grp] = sbits;
    const float scale = __half2float(sh), inv = 1.0f / scale;
    uint32_t o[2] = {0u, 0u};
#pragma unroll
    for (int j = 0; j < kPer / 4; ++j) {
        const float e[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) o[j >> 1] |= (round_quotient(e[i], scale, inv, 7.0f) + 8u) << (16 * (j & 1) + 4 * i);
    }
    uint8_t* to = packed + grp * 64 + part * (kPer / 2);
    if ((reinterpret_cast<uintptr_t>(packed) & 7u) == 0) {
        if (kPer == 16) *reinterpret_cast<uint2*>(to) = make_uint2(o[0], o[1]);
        else *reinterpret_cast<uint16_t*>(to) = (uint16_t)o[0];
    } else {
#pragma unroll
        for (int i = 0; i < kPer / 2; ++i) to[i] = (uint8_t)(o[i >> 2] >> (8 * (i & 3)));
    }
}

template <int kSteps>
__global__ void __launch_bounds__(256) dequant_w4_quads_kernel(const uint16_t* __restrict__ packed, const uint16_t* __restrict__ gscales, size_t quads,
                                                               float4* __restrict__ out) {
    const size_t first = (size_t)blockIdx.x * (256 * kSteps) + threadIdx.x;
    uint32_t v[kSteps];
    float s[kSteps];
#pragma unroll
    for (int j = 0; j < kSteps; ++j) {
        const size_t i = first + 256 * j;
        if (i < quads) {
            v[j] = __ldg(packed + i);
            s[j] = __half2float(__ushort_as_half(__ldg(gscales + (i >> 5))));
        }
    }
#pragma unroll
    for (int j = 0; j < kSteps; ++j) {
        const size_t i = first + 256 * j;
        if (i < quads)
            out[i] = make_float4((float)((int)(v[j] & 15u) - 8) * s[j], (float)((int)((v[j] >> 4) & 15u) - 8) * s[j], (float)((int)((v[j] >> 8) & 15u) - 8) * s[j],
                                 (float)((int)((v[j] >> 12) & 15u) - 8) * s[j]);
    }
}

__global__ void dequant_w4_kernel(const uint8_t* __restrict__ packed, const uint16_t* __restrict__ gscales, size_t n,
                                  float* __restrict__ out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint8_t byte = packed[i >> 1];
    const int nib = (i & 1) ? (byte >> 4) : (byte & 0xf);
    out[i] = (float)(nib - 8) * __half2float(__ushort_as_half(gscales[i >> 7]));
}

__global__ void f32_to_bf16_kernel(const float* __restrict__ src, size_t n, uint16_t* __restrict__ dst) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = f32_to_bf16_bits(src[i]);
}

__global__ void widen_bf16_kernel(const uint16_t* __restrict__ src, size_t n, float* __restrict__ dst) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = bf16_bits_to_f32(src[i]);
}

__device__ inline uint64_t splitmix64(uint64_t x) {
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}

// Counter-based N(0, std): element i depends only on (seed, i).
__global__ void fill_normal_kernel(float* __restrict__ dst, size_t n, uint64_t seed, float stddev) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t r = splitmix64(seed * 0xd1342543de82ef95ull + i);
    const float u1 = ((float)((r >> 40) & 0xffffffull) + 1.0f) * (1.0f / 16777216.0f);  // (0,1]
    const float u2 = (float)((r >> 16) & 0xffffffull) * (1.0f / 16777216.0f);           // [0,1)
    dst[i] = stddev * sqrtf(-2.0f * logf(u1)) * cospif(2.0f * u2);
}

int widen_bf16(cudaStream_t stream, const uint16_t* src, size_t n, float* dst) {
    if (n == 0) return KMLL_OK;
    widen_bf16_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(src, n, dst);
    return check_launch("widen_bf16");
}

}  // namespace kmll

using namespace kmll;

// One step per thread while that leaves room on the multiprocessors (1024 threads each), else four (128 x 896: 2.0 us with four, 1.6 with one)
template <typename K, typename... A>
static void launch_quads(kmll_stream_t s, size_t quads, K one, K four, A... args) {
    const int steps = quads <= 148 * 1024 ? 1 : 4;
    (steps == 1 ? one : four)<<<(unsigned)((quads + 256 * steps - 1) / (256 * steps)), 256, 0, as_stream(s)>>>(args...);
}

extern "C" {

int kmll_quantize_rs_i8(kmll_stream_t s, const uint16_t* w, int rows, int cols, int8_t* values, float* scales) {
    KMLL_REQUIRE_PTR(w); KMLL_REQUIRE_PTR(values); KMLL_REQUIRE_PTR(scales);
    KMLL_REQUIRE(rows > 0 && cols > 0, "quantize_rs_i8: shape [%d, %d] must be positive", rows, cols);
    const bool vec = cols % 8 == 0 && (reinterpret_cast<uintptr_t>(w) & 15u) == 0 && (reinterpret_cast<uintptr_t>(values) & 7u) == 0;
    // One piece per thread while the rows' threads are no more than two rounds of the chip at 1024 per multiprocessor (2000 x 1024, 1.7
    // rounds: 5.2 us with four pieces, 3.4 with one; at 3.5 rounds 6.1 and 5.3; 4096 x 4096, 14 rounds: 15.0 and 15.8; 14336 x 4096 48 and 56).
    auto whole_warps = [](int n) { n = (n + 31) / 32 * 32; return n > 512 ? 512 : n; };
    const int one = whole_warps((cols + 7) / 8), four = whole_warps((cols + 31) / 32);
    if (!vec) quantize_rs_i8_kernel<0><<<rows, 256, 0, as_stream(s)>>>(w, cols, values, scales);
    else if (one * 8 >= cols && (size_t)rows * one <= 2 * 148 * 1024) quantize_rs_i8_kernel<1><<<rows, one, 0, as_stream(s)>>>(w, cols, values, scales);
    else quantize_rs_i8_kernel<4><<<rows, four, 0, as_stream(s)>>>(w, cols, values, scales);
    return check_launch("quantize_rs_i8");
}
int kmll_dequant_rs_i8(kmll_stream_t s, const int8_t* values, const float* scales, int rows, int cols, float* out) {
    KMLL_REQUIRE_PTR(values); KMLL_REQUIRE_PTR(scales); KMLL_REQUIRE_PTR(out);
    KMLL_REQUIRE(rows > 0 && cols > 0, "dequant_rs_i8: shape [%d, %d] must be positive", rows, cols);
    const size_t n = (size_t)rows * cols;
    if (cols % 4 == 0 && n / 4 < 0xfffffc00ull && (reinterpret_cast<uintptr_t>(values) & 3u) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0)
        launch_quads(s, n / 4, dequant_rs_i8_quads_kernel<1>, dequant_rs_i8_quads_kernel<4>, reinterpret_cast<const uint32_t*>(values), scales, (uint32_t)(n / 4),
                     (uint32_t)(cols / 4), reinterpret_cast<float4*>(out));
    else
        dequant_rs_i8_kernel<<<(unsigned)((n + 255) / 256), 256, 0, as_stream(s)>>>(values, scales, rows, cols, out);
    return check_launch("dequant_rs_i8");
}
int kmll_quantize_w4g128(kmll_stream_t s, const float* w, int rows, int cols, uint8_t* packed, uint16_t* gscales) {
    KMLL_REQUIRE_PTR(w); KMLL_REQUIRE_PTR(packed); KMLL_REQUIRE_PTR(gscales);
    KMLL_REQUIRE(rows > 0 && cols > 0 && cols % 128 == 0, "quantize_w4g128: cols %d must be a positive multiple of 128", cols);
    KMLL_REQUIRE((reinterpret_cast<uintptr_t>(w) & 15u) == 0, "quantize_w4g128: source must be 16-byte aligned");
    const size_t n_groups = (size_t)rows * (cols / 128);
    // a warp per group as long as all of them run at once (64 warps per multiprocessor; 16000 groups: 3.9 us either way)
    if (n_groups <= 148 * 64) quantize_w4_kernel<4><<<(unsigned)((n_groups + 7) / 8), 256, 0, as_stream(s)>>>(w, n_groups, packed, gscales);
    else quantize_w4_kernel<16><<<(unsigned)((n_groups + 31) / 32), 256, 0, as_stream(s)>>>(w, n_groups, packed, gscales);
    return check_launch("quantize_w4g128");
}
int kmll_dequant_w4g128(kmll_stream_t s, const uint8_t* packed, const uint16_t* gscales, int rows, int cols, float* out) {
    KMLL_REQUIRE_PTR(packed); KMLL_REQUIRE_PTR(gscales); KMLL_REQUIRE_PTR(out);
    KMLL_REQUIRE(rows > 0 && cols > 0 && cols % 128 == 0, "dequant_w4g128: cols %d must be a positive multiple of 128", cols);
    const size_t n = (size_t)rows * cols;
    if ((reinterpret_cast<uintptr_t>(packed) & 1u) == 0 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0)
        launch_quads(s, n / 4, dequant_w4_quads_kernel<1>, dequant_w4_quads_kernel<4>, reinterpret_cast<const uint16_t*>(packed), gscales, n / 4,
                     reinterpret_cast<float4*>(out));
    else
        dequant_w4_kernel<<<(unsigned)((n + 255) / 256), 256, 0, as_stream(s)>>>(packed, gscales, n, out);
    return check_launch("dequant_w4g128");
}
int kmll_f32_to_bf16(kmll_stream_t s, const float* src, size_t n, uint16_t* dst) {
    KMLL_REQUIRE_PTR(src); KMLL_REQUIRE_PTR(dst);
    if (n == 0) return KMLL_OK;
    f32_to_bf16_kernel<<<(unsigned)((n + 255) / 256), 256, 0, as_stream(s)>>>(src, n, dst);
    return check_launch("f32_to_bf16");
}
int kmll_fill_normal_f32(kmll_stream_t s, float* dst, size_t n, uint64_t seed, float stddev) {
    KMLL_REQUIRE_PTR(dst);
    if (n == 0) return KMLL_OK;
    fill_normal_kernel<<<(unsigned)((n + 255) / 256), 256, 0, as_stream(s)>>>(dst, n, seed, stddev);
    return check_launch("fill_normal_f32");
}

}  // extern "C"
