// Causal attention of a prompt on tcgen05: one block = 128 query rows of one head; f32 or bf16 operands, f32 softmax and sums.
//
// Serves the batched prompt of the uniform decoders (f32 or bf16 cache) and the latent attention of the layered ones.  An f32 operand
// is split into bf16 planes, x = x0 + x1 (a remainder of 2^-17 of x), and of the products of two split operands the
// one of both remainders is left out; a bf16 operand is one plane and exact.  These are the products of the mma.sync kernels in
// attention.cu and latent_attention.cu, which keep what this file does not serve.
//
// Roles of the 12 warps:
//   warps 0-3, 4-7  softmax of the even and of the odd key tiles: a thread has one query row (one lane of tensor memory); scores come
//                   by tcgen05.ld, twice - a first pass for the maximum, a second for the weights -, and the weights go back as bf16
//                   planes in the place of the scores.  The two are independent streams, each with its own maximum, sum and
//                   O in tensor memory, and are merged at the end.
//   warps 8, 9      TMA of the key tiles and of the value tiles (values as they lie: the B operand of P V is MN-major); warp 9 also looks
//                   through the values of tiles that some row does not see in full (PaHeld)
//   warp 10         issues S = Q K^T (both operands in shared memory) and O += P V (P from tensor memory)
// Bound by the tensor cores with f32 operands (48 MMAs of 61 cycles a tile; a fifth of the issuer's time is waiting), by the second pass of
// the softmax (3460 cycles of its warps per tile, exponentials and conversions) with bf16 ones; all threads are held to 168 registers, and
// the softmax spills 12 to 60 bytes of them.  Profiled against the mma.sync kernel, 32 heads of 128: 2000 tokens, f32 cache 363 -> 125 us, bf16
// cache 279 -> 108; 512 tokens 48 -> 24 and 41 -> 21.  A block costs 11 to 15 us beside its tiles (prompt_attention_pays).  Built before and slower: eight
// warps that convert keys and values of an f32 cache themselves, every block again, instead of TMA of planes written once (262 us).
// Order of the MMAs: S0 S1, P0V0 S2, P1V1 S3, ...  O is rescaled only when a row's maximum has grown by more than 2^8 since the last
// time (larger weights cost no precision: every plane is relative), which after the first tiles hardly happens.
// Blocks with the most keys start first.  Every wait is bounded; a time-out raises the status word, and the block waits for the copies it
// began, frees its tensor memory and returns.
#include <cuda.h>

#include "internal.cuh"
#include "mma_bf16.cuh"
#include "tcgen05.cuh"

namespace kmll {

__device__ int g_prompt_attention_status = 0;

namespace {

constexpr int kPaRows = 128;  // query rows of a block
constexpr int kPaKeys = 128;  // keys of a tile
constexpr int kPaThreads = 12 * 32;
constexpr int kPaBox = 128 * 128;  // a TMA box: 128 rows of 64 bf16 entries in the 128-byte swizzle
// tensor-memory columns: score buffers at 0 and 128, the two streams' O behind them.  A block allocates all 512 columns, so its
// allocation starts at column 0 (a constant address keeps the issuing warp's operands uniform).
constexpr uint32_t kPaTmemO = 256;

// Shared memory: planes of Q [128 rows][DQ] as 64-entry wide blocks; ring of stages with the boxes of K ([128 keys][DQ], NK planes) and of V
// ([128 keys][DV]); each stream's (maximum, sum) per row; barriers; PaHeld.  NQ, NK: planes of Q and of K and V.
template <int DQ, int DV, int NQ, int NK>
struct PaShape {
    static constexpr int kQPlane = kPaRows * DQ * 2, kKBoxes = NK * DQ / 64, kVBoxes = NK * DV / 64;
    static constexpr int kOffK = NQ * kQPlane;
    static constexpr int kStages = kOffK + 2 * (kKBoxes + kVBoxes) * kPaBox <= 216 * 1024 ? 2 : 1;
    static constexpr int kOffV = kOffK + kStages * kKBoxes * kPaBox, kOffStat = kOffV + kStages * kVBoxes * kPaBox;
    static constexpr int kOffBars = kOffStat + 2 * kPaRows * 8;
    static constexpr int kOffHeld = kOffBars + 128;           // PaHeld: [3 tiles][DV][128 bits]
    static constexpr int kSmemBytes = kOffHeld + 3 * DV * 16 + 1024;  // + slack for the 1024-byte alignment
    static constexpr int kStagePitch = DV / 2 + 4;            // rows of half of O on their way out, over the operands
    static_assert(DQ % 64 == 0 && (DV == 64 || DV == 128) && kSmemBytes <= 227 * 1024, "shape");
    static_assert(8 * 32 * kStagePitch * 4 <= kOffStat, "the rows of O fit over the operands");
};

// byte of (row, eight-entry piece c8) in a plane of Q
__device__ inline uint32_t pa_place(int row, int c8) { return (uint32_t)((c8 >> 3) * kPaBox + row * 128 + (((c8 & 7) ^ (row & 7)) << 4)); }
__device__ inline void pa_split8(const float (&v)[8], uint4& hi, uint4& lo) {
    split_bf16x2(v[0], v[1], hi.x, lo.x);
    split_bf16x2(v[2], v[3], hi.y, lo.y);
    split_bf16x2(v[4], v[5], hi.z, lo.z);
    split_bf16x2(v[6], v[7], hi.w, lo.w);
}
// B operand whose N entries lie together (values: 64 dimensions of a key are a 128-byte row): groups of 8 keys are 1024 bytes apart, blocks
// of 64 dimensions a box
__device__ inline uint64_t pa_desc_mn(uint32_t smem_addr) {
    return (uint64_t)((smem_addr >> 4) & 0x3fffu) | ((uint64_t)(kPaBox >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// Values that are not finite.  A key that a row does not attend has weight 0 there, and 0 * infinity is NaN.  So in the tiles that some
// row does not see in full - at most three: the first (window) and the last two (causal) - such entries become zeros ahead of the
// MMAs and are noted, a bit per (column, key); at the end an output whose row attends one of them becomes NaN.
struct PaHeld {
    // slot of tile j; the keys of the tile in the slot
    static __device__ inline int slot(int j, int tiles) { return j == tiles - 1 ? 0 : j == tiles - 2 ? 1 : 2; }
    static __device__ inline int tile(int slot, int tiles) { return slot == 2 ? 0 : tiles - 1 - slot; }
    // The exponent of a half of w is all ones: bit 15 of that half here.  (Of two planes the first one tells: the remainder is finite with it.)
    static __device__ inline uint32_t not_finite(uint32_t w) { return (w & 0x7f807f80u) + 0x00800080u; }
    // key r of the tile, whose 128-byte rows of the first box start at `box`
    template <int DV, int NK>
    static __device__ inline void hold_back(unsigned char* box, int r, uint32_t* bits) {
#pragma unroll 1
        for (int col = 0; col < DV; ++col) {
            unsigned char* const at = box + (col >> 6) * kPaBox + r * 128 + ((((col >> 3) & 7) ^ (r & 7)) << 4) + (col & 7) * 2;
            if ((*reinterpret_cast<const uint16_t*>(at) & 0x7f80u) != 0x7f80u) continue;
            for (int n = 0; n < NK; ++n) *reinterpret_cast<uint16_t*>(at + n * (DV / 64) * kPaBox) = 0u;
            atomicOr(bits + col * 4 + (r >> 5), 1u << (r & 31));
        }
    }
    // whether a bit of keys a .. b is set (either may lie outside the tile)
    static __device__ inline bool any(const uint32_t* bits, int a, int b) {
        for (int w = 0; w < 4; ++w) {
            const int lo = max(a - w * 32, 0), hi = min(b - w * 32, 31);
            if (lo <= hi && (bits[w] & (0xffffffffu >> (31 - hi)) & (0xffffffffu << lo)) != 0u) return true;
        }
        return false;
    }
};
// What a block attends: row r of the block is position pos0 + r and sees the keys max(0, pos - window + 1) .. pos (window 0: from 0);
// keys first .. last are walked in tiles.
struct PaRange {
    int pos0, live_rows, first, last, window;
    float scale2;  // log2(e) times the score scale, positive
    // some row does not see some key of the tile that starts at t0
    __device__ bool partly(int t0) const { return t0 + kPaKeys - 1 > pos0 || (window > 0 && t0 < pos0 + kPaRows - window); }
};

// Src: kDQ, kDV, kNQ, kNK; q_planes(row, c8, planes): eight entries of a query row; load_k(lead, box, pos, dst, bar), load_v: the TMA of one box
// from position pos on (its rows behind the last position are zeros or keys that no row sees).
template <class Src>
__device__ inline void prompt_attention_block(const Src& src, const PaRange& rg, float* out, size_t ldo) {
    constexpr int DQ = Src::kDQ, DV = Src::kDV, NQ = Src::kNQ, NK = Src::kNK, C8 = DQ / 8;
    using S = PaShape<DQ, DV, NQ, NK>;
    constexpr int kStages = S::kStages;
    extern __shared__ unsigned char pa_smem_raw[];
    unsigned char* smem = pa_smem_raw + ((1024u - (smem_u32(pa_smem_raw) & 1023u)) & 1023u);
    uint64_t* const s_full = reinterpret_cast<uint64_t*>(smem + S::kOffBars);  // [2] the scores of a tile are there
    uint64_t* const p_ready = s_full + 2;         // [2] its weights are there (and O is rescaled)
    uint64_t* const pv_done = p_ready + 2;        // [2] O has taken the tile
    uint64_t* const k_full = pv_done + 2;         // [kStages]
    uint64_t* const v_full = k_full + kStages;    // [kStages]
    uint64_t* const v_clean = v_full + kStages;   // [3] PaHeld: the tile of the slot has been looked through
    uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(v_clean + 3);
    uint32_t* const any_held = tmem_slot + 1;
    uint32_t* const held = reinterpret_cast<uint32_t*>(smem + S::kOffHeld);
    const int tid = threadIdx.x, lane = tid & 31, warp = uniform_warp_index();
    if (tid == 0) {
        for (int b = 0; b < 2; ++b) { mbar_init(&s_full[b], 1); mbar_init(&p_ready[b], 4); mbar_init(&pv_done[b], 1); }
        for (int st = 0; st < kStages; ++st) { mbar_init(&k_full[st], 1); mbar_init(&v_full[st], 1); }
        for (int i = 0; i < 3; ++i) mbar_init(&v_clean[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        *any_held = 0u;
    }
    for (int i = tid; i < 3 * DV * 4; i += kPaThreads) held[i] = 0u;
    if (warp == 10) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();  // (columns first, then the dependents: tcgen05.cuh)
    tcgen05_fence_after();
    pdl_wait();
    for (int i = tid; i < kPaRows * C8; i += kPaThreads) {  // (rows beyond the prompt are zeros)
        const int r = i / C8, c8 = i - r * C8;
        uint4 pl[NQ];
#pragma unroll
        for (int n = 0; n < NQ; ++n) pl[n] = make_uint4(0u, 0u, 0u, 0u);
        if (r < rg.live_rows) src.q_planes(r, c8, pl);
#pragma unroll
        for (int n = 0; n < NQ; ++n) *reinterpret_cast<uint4*>(smem + n * S::kQPlane + pa_place(r, c8)) = pl[n];
    }
    fence_proxy_async_smem();
    __syncthreads();
    const int tiles = (rg.last - rg.first) / kPaKeys + 1;
    const uint32_t base = smem_u32(smem);
    bool ok = true;

    if (warp == 8 || warp == 9) {
        // ---- TMA: the place of K(j - kStages) is free once its scores are done, that of V(j - kStages) once O has taken that tile
        const bool keys = warp == 8;
        uint64_t* const full = keys ? k_full : v_full;
        uint64_t* const done = keys ? s_full : pv_done;
        const int boxes = keys ? S::kKBoxes : S::kVBoxes;
        const uint32_t lead = elect_lead();
        // (This warp has seen every earlier use of the stage end, so the parity of v_full means tile j.)
        auto look_through = [&](int j) {
            if (!rg.partly(rg.first + j * kPaKeys)) return true;
            if (!warp_wait(&v_full[j % kStages], (uint32_t)(j / kStages) & 1u)) return false;
            unsigned char* const box = smem + S::kOffV + (j % kStages) * S::kVBoxes * kPaBox;
            uint32_t bad = 0u;
#pragma unroll 8
            for (int i = lane; i < 8 * kPaKeys * (DV / 64); i += 32) {
                const uint4 w = reinterpret_cast<const uint4*>(box)[i];
                bad |= PaHeld::not_finite(w.x) | PaHeld::not_finite(w.y) | PaHeld::not_finite(w.z) | PaHeld::not_finite(w.w);
            }
            const int slot = PaHeld::slot(j, tiles);
            if (__any_sync(0xffffffffu, (bad & 0x80008000u) != 0u)) {
                for (int r = lane; r < kPaKeys; r += 32) PaHeld::hold_back<DV, NK>(box, r, held + slot * DV * 4);
                *any_held = 1u;
                fence_proxy_async_smem();
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&v_clean[slot]);
            return true;
        };
        int issued = 0;
        for (int j = 0; j < tiles; ++j) {
            const int st = j % kStages, before = j - kStages;
            ok = before < 0 || warp_wait(&done[before & 1], (uint32_t)(before >> 1) & 1u);
            if (!ok) break;
            const uint32_t dst = base + (uint32_t)((keys ? S::kOffK : S::kOffV) + st * boxes * kPaBox);
            lead_expect_tx(lead, &full[st], (uint32_t)(boxes * kPaBox));
            for (int b = 0; b < boxes; ++b) {
                if (keys) src.load_k(lead, b, rg.first + j * kPaKeys, dst + b * kPaBox, &full[st]);
                else src.load_v(lead, b, rg.first + j * kPaKeys, dst + b * kPaBox, &full[st]);
            }
            issued = j + 1;
            // (with two stages a tile behind, so that the next one's copies are under way)
            if (!keys && j >= kStages - 1) ok = look_through(j - (kStages - 1));
            if (!ok) break;
        }
        for (int j = max(tiles - (kStages - 1), 0); j < tiles && !keys && ok; ++j) ok = look_through(j);
        ok = ring_landed(full, issued, kStages) && ok;  // (after a time-out too)
    } else if (warp == 10) {
        constexpr uint32_t idesc_s = gemm_idesc_bf16(128, kPaKeys), idesc_o = gemm_idesc_bf16(128, DV) | (1u << 16);  // V is MN-major
        const uint64_t dq = gemm_smem_desc(base), dk = gemm_smem_desc(base + S::kOffK), dv = pa_desc_mn(base + S::kOffV);
        constexpr int NP = NQ > NK ? NQ : NK;
        const uint32_t lead = elect_lead();
        auto scores = [&](int j) {
            const int st = j % kStages;
            if (!warp_wait(&k_full[st], (uint32_t)(j / kStages) & 1u)) return false;
            tcgen05_fence_after();
            const uint64_t dkj = dk + (uint64_t)(st * (S::kKBoxes * kPaBox >> 4));
            const uint32_t d = (uint32_t)(j & 1) * 128u;
            uint32_t acc = 0u;
#pragma unroll
            for (int order = NP - 1; order >= 0; --order)  // the small products first
#pragma unroll
                for (int a = 0; a < NQ; ++a) {
                    const int b = order - a;
                    if (b < 0 || b >= NK) continue;
#pragma unroll
                    for (int ks = 0; ks < DQ / 16; ++ks) {
                        const int at = (ks >> 2) * kPaBox + (ks & 3) * 32;
                        lead_mma_f16(lead, d, dq + (uint64_t)((a * S::kQPlane + at) >> 4), dkj + (uint64_t)((b * (DQ / 64) * kPaBox + at) >> 4), idesc_s, acc);
                        acc = 1u;
                    }
                }
            lead_commit(lead, &s_full[j & 1]);
            return true;
        };
        ok = scores(0) && (tiles < 2 || scores(1));
        for (int j = 0; j < tiles && ok; ++j) {
            const int st = j % kStages;
            ok = warp_wait(&v_full[st], (uint32_t)(j / kStages) & 1u) && warp_wait(&p_ready[j & 1], (uint32_t)(j >> 1) & 1u);
            if (ok && rg.partly(rg.first + j * kPaKeys)) ok = warp_wait(&v_clean[PaHeld::slot(j, tiles)], 0u);
            if (!ok) break;
            tcgen05_fence_after();
            const uint32_t p = (uint32_t)(j & 1) * 128u, d = kPaTmemO + (uint32_t)(j & 1) * 128u;
            const uint64_t dvj = dv + (uint64_t)(st * (S::kVBoxes * kPaBox >> 4));
            uint32_t acc = j >= 2 ? 1u : 0u;
#pragma unroll
            for (int order = 1; order >= 0; --order)  // the weights are two planes
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    const int b = order - a;
                    if (b < 0 || b >= NK) continue;
#pragma unroll
                    for (int ks = 0; ks < kPaKeys / 16; ++ks) {
                        lead_mma_f16_ts(lead, d, p + (uint32_t)(a * (kPaKeys / 2) + ks * 8), dvj + (uint64_t)((b * (DV / 64) * kPaBox + ks * 2048) >> 4), idesc_o, acc);
                        acc = 1u;
                    }
                }
            lead_commit(lead, &pv_done[j & 1]);
            if (j + 2 < tiles) ok = scores(j + 2);
        }
    } else if (warp < 8) {
        // ---- softmax of the tiles j = stream, stream + 2, ..
        const int stream = warp >> 2, r = (warp & 3) * 32 + lane, pos = rg.pos0 + r, lo = rg.window > 0 ? pos - rg.window + 1 : 0;
        const uint32_t rows = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t ts = rows + (uint32_t)stream * 128u, to = rows + kPaTmemO + (uint32_t)stream * 128u;
        float m_ref = -INFINITY, l = 0.0f;
        int n = 0;  // tiles of this stream so far
        for (int j = stream; j < tiles; j += 2, ++n) {
            const int t0 = rg.first + j * kPaKeys;
            const bool masked = rg.partly(t0);
            ok = warp_wait(&s_full[stream], (uint32_t)n & 1u);
            if (!ok) break;
            tcgen05_fence_after();
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < kPaKeys / 32; ++c) {
                uint32_t d[32];
                tmem_load_x32(ts + c * 32, d);
                if (masked) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const int key = t0 + c * 32 + i;
                        mx[i & 3] = fmaxf(mx[i & 3], key <= pos && key >= lo ? __uint_as_float(d[i]) : -INFINITY);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) mx[i & 3] = fmaxf(mx[i & 3], __uint_as_float(d[i]));
                }
            }
            const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * rg.scale2;
            const bool grow = top > m_ref + 8.0f;  // (a row with nothing attended so far has -inf)
            if (__any_sync(0xffffffffu, grow)) {
                const float corr = grow ? ex2_approx(m_ref - top) : 1.0f;
                if (grow) m_ref = top;
                l *= corr;
                if (n > 0) {
                    ok = warp_wait(&pv_done[stream], (uint32_t)(n - 1) & 1u);
                    if (!ok) break;
                    tcgen05_fence_after();
#pragma unroll
                    for (int c = 0; c < DV / 32; ++c) {
                        uint32_t d[32];
                        tmem_load_x32(to + c * 32, d);
#pragma unroll
                        for (int i = 0; i < 32; ++i) d[i] = __float_as_uint(__uint_as_float(d[i]) * corr);
                        tmem_store_x32(to + c * 32, d);
                    }
                }
            }
            const float m = m_ref == -INFINITY ? 0.0f : m_ref;
            float sum[2] = {0.0f, 0.0f};
            uint32_t rest[2][32];  // the second plane, until all scores are read
#pragma unroll
            for (int c = 0; c < kPaKeys / 32; ++c) {
                uint32_t d[32], hi[16];
                tmem_load_x32(ts + c * 32, d);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    float p0 = ex2_approx(fmaf(__uint_as_float(d[2 * i]), rg.scale2, -m)), p1 = ex2_approx(fmaf(__uint_as_float(d[2 * i + 1]), rg.scale2, -m));
                    if (masked) {
                        const int key = t0 + c * 32 + 2 * i;
                        p0 = key <= pos && key >= lo ? p0 : 0.0f;
                        p1 = key + 1 <= pos && key + 1 >= lo ? p1 : 0.0f;
                    }
                    sum[0] += p0;
                    sum[1] += p1;
                    split_bf16x2(p0, p1, hi[i], rest[c >> 1][(c & 1) * 16 + i]);
                }
                tmem_store_x16(ts + c * 16, hi);
            }
            l += sum[0] + sum[1];
            tmem_store_x32(ts + 64, rest[0]);
            tmem_store_x32(ts + 96, rest[1]);
            tmem_store_wait();
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_ready[stream]);
        }
        if (ok && n > 0) ok = warp_wait(&pv_done[stream], (uint32_t)(n - 1) & 1u);
        // ---- both streams of a row, then half of its columns per stream's warps
        float2* const stat = reinterpret_cast<float2*>(smem + S::kOffStat);
        stat[stream * kPaRows + r] = make_float2(m_ref, l);
        tcgen05_fence_before();
        asm volatile("bar.sync 1, 256;" ::: "memory");
        tcgen05_fence_after();
        const float2 st0 = stat[r], st1 = stat[kPaRows + r];
        const float m = fmaxf(st0.x, st1.x);
        const float w0 = ex2_approx(st0.x - m), w1 = tiles > 1 ? ex2_approx(st1.x - m) : 0.0f, inv = 1.0f / (st0.y * w0 + (tiles > 1 ? st1.y * w1 : 0.0f));
        const float f0 = w0 * inv, f1 = w1 * inv;
        // the last MMAs are done and nobody loads: the rows leave over the operands' shared memory, so that a warp writes whole runs
        float* const stage = reinterpret_cast<float*>(smem) + warp * 32 * S::kStagePitch;
#pragma unroll
        for (int c = 0; c < DV / 64; ++c) {
            uint32_t d[32], e[32];
            const uint32_t col = rows + kPaTmemO + (uint32_t)(stream * (DV / 2) + c * 32);
            tmem_load_x32(col, d);
            if (tiles > 1) tmem_load_x32(col + 128u, e);
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
                float y[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    y[k] = __uint_as_float(d[i + k]) * f0;
                    if (tiles > 1) y[k] = fmaf(__uint_as_float(e[i + k]), f1, y[k]);
                }
                *reinterpret_cast<float4*>(stage + lane * S::kStagePitch + c * 32 + i) = make_float4(y[0], y[1], y[2], y[3]);
            }
        }
        __syncwarp();
        for (int i = lane; i < 32 * (DV / 8); i += 32) {
            const int rr = i / (DV / 8), c4 = i - rr * (DV / 8), row = (warp & 3) * 32 + rr;
            if (ok && row < rg.live_rows)
                *reinterpret_cast<float4*>(out + (size_t)row * ldo + stream * (DV / 2) + c4 * 4) = *reinterpret_cast<const float4*>(stage + rr * S::kStagePitch + c4 * 4);
        }
    }
    if (!ok) atomicCAS(&g_prompt_attention_status, 0, 1);
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    if (*any_held != 0u)
        for (int i = tid; i < 3 * rg.live_rows * DV; i += kPaThreads) {
            const int slot = i / (rg.live_rows * DV), row = (i / DV) % rg.live_rows, col = i % DV;
            const int pos = rg.pos0 + row, t0 = rg.first + PaHeld::tile(slot, tiles) * kPaKeys;  // (no bits are set in a slot without a tile)
            if (PaHeld::any(held + (slot * DV + col) * 4, (rg.window > 0 ? pos - rg.window + 1 : 0) - t0, pos - t0)) out[(size_t)row * ldo + col] = __int_as_float(0x7fffffff);
        }
    if (warp == 10) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*tmem_slot), "r"(512u) : "memory");
}

// ---- rows of q in f32; keys and values as bf16 rows: the bf16 cache, or the two planes that the rotation wrote for an f32 cache -------------
template <int HD, bool KVB>
struct DenseSource {
    static constexpr int kDQ = HD, kDV = HD, kNQ = 2, kNK = KVB ? 1 : 2;
    const float* q;  // first query row of the block, this head
    size_t q_len;
    const CUtensorMap *map_k, *map_v;
    int col, kv_len;  // column of this kv head; the second plane lies kv_len columns on
    __device__ void q_planes(int r, int c8, uint4 (&pl)[2]) const {
        const float4* p = reinterpret_cast<const float4*>(q + (size_t)r * q_len + c8 * 8);
        const float4 a = p[0], b = p[1];
        const float x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        pa_split8(x, pl[0], pl[1]);
    }
    __device__ int column(int box) const { return col + (box / (HD / 64)) * kv_len + (box % (HD / 64)) * 64; }
    __device__ void load_k(uint32_t lead, int box, int pos, uint32_t dst, uint64_t* bar) const { lead_tma_2d(lead, dst, map_k, column(box), pos, bar); }
    __device__ void load_v(uint32_t lead, int box, int pos, uint32_t dst, uint64_t* bar) const { lead_tma_2d(lead, dst, map_v, column(box), pos, bar); }
};

template <int HD, bool KVB>
__global__ void __launch_bounds__(kPaThreads, 1) prompt_attention_kernel(const float* __restrict__ q_batch, int prompt_len, int n_heads, int n_kv_heads,
                                                                         float* __restrict__ out, int window, const __grid_constant__ CUtensorMap map_k,
                                                                         const __grid_constant__ CUtensorMap map_v) {
    const int head = blockIdx.x, r0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * kPaRows, kv_head = head / (n_heads / n_kv_heads);
    DenseSource<HD, KVB> src;
    src.q_len = (size_t)n_heads * HD;
    src.q = q_batch + (size_t)r0 * src.q_len + (size_t)head * HD;
    src.map_k = &map_k;
    src.map_v = &map_v;
    src.col = kv_head * HD;
    src.kv_len = n_kv_heads * HD;
    PaRange rg;
    rg.pos0 = r0;
    rg.live_rows = min(kPaRows, prompt_len - r0);
    rg.first = window > 0 ? max(0, r0 - window + 1) : 0;
    rg.last = r0 + rg.live_rows - 1;
    rg.window = window;
    rg.scale2 = 1.4426950408889634f / sqrtf((float)HD);
    prompt_attention_block(src, rg, out + (size_t)r0 * src.q_len + (size_t)head * HD, src.q_len);
}

// ---- latent attention: heads of 128 + 64 rotated entries, values of 128; keys and values from the expanded latents, the rotated key part
// (one for all heads) from the cache --------------------------------------------------------------------------------------------
struct LatentSource {
    static constexpr int kDQ = 192, kDV = 128, kNQ = 1, kNK = 1;
    const uint16_t* q;    // first query row of the block, this head: 128 entries, then 64 unrotated ones
    size_t ld;
    const float2* turns;  // of the first row's position, [position][32]
    const CUtensorMap *map_ex, *map_cache;
    int kcol, vcol, kr_off, first;
    __device__ void q_planes(int r, int c8, uint4 (&pl)[1]) const {
        const uint16_t* row = q + (size_t)r * ld;
        if (c8 < 16) {
            pl[0] = *reinterpret_cast<const uint4*>(row + c8 * 8);
            return;
        }
        const bool second = c8 >= 20;  // entry j of the first half turns with entry j + 32
        const int j0 = (c8 - (second ? 20 : 16)) * 8;
        const uint4 ua = *reinterpret_cast<const uint4*>(row + 128 + j0), va = *reinterpret_cast<const uint4*>(row + 160 + j0);
        const uint32_t uu[4] = {ua.x, ua.y, ua.z, ua.w}, vv[4] = {va.x, va.y, va.z, va.w};
        const float2* cs = turns + (size_t)r * 32 + j0;
        uint32_t y[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float u = bf16_bits_to_f32((uint16_t)(uu[i >> 1] >> (16 * (i & 1)))), v = bf16_bits_to_f32((uint16_t)(vv[i >> 1] >> (16 * (i & 1))));
            const float2 f = cs[i];
            y[i] = f32_to_bf16_bits(second ? v * f.x + u * f.y : u * f.x - v * f.y);
        }
        pl[0] = make_uint4(y[0] | (y[1] << 16), y[2] | (y[3] << 16), y[4] | (y[5] << 16), y[6] | (y[7] << 16));
    }
    // (positions in front of the first expanded one are rows before the map's: zeros)
    __device__ void load_k(uint32_t lead, int box, int pos, uint32_t dst, uint64_t* bar) const {
        if (box < 2) lead_tma_2d(lead, dst, map_ex, kcol + box * 64, pos - first, bar);
        else lead_tma_2d(lead, dst, map_cache, kr_off, pos, bar);
    }
    __device__ void load_v(uint32_t lead, int box, int pos, uint32_t dst, uint64_t* bar) const { lead_tma_2d(lead, dst, map_ex, vcol + box * 64, pos - first, bar); }
};

__global__ void __launch_bounds__(kPaThreads, 1) latent_prompt_kernel(const LatentArgs a, const __grid_constant__ CUtensorMap map_ex, const __grid_constant__ CUtensorMap map_cache) {
    const int head = blockIdx.x, r0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * kPaRows;
    LatentSource src;
    src.ld = (size_t)a.ld;
    src.q = static_cast<const uint16_t*>(a.in) + (size_t)r0 * a.ld + a.q_off + (size_t)head * 192;
    src.turns = a.table + (size_t)(a.pos0 + r0) * 32;
    src.map_ex = &map_ex;
    src.map_cache = &map_cache;
    src.kcol = head * 128;
    src.vcol = a.heads * 128 + head * 128;
    src.kr_off = a.kr_off;
    src.first = a.first;
    PaRange rg;
    rg.pos0 = a.pos0 + r0;
    rg.live_rows = min(kPaRows, a.T - r0);
    rg.first = a.window > 0 ? max(0, rg.pos0 - a.window + 1) : 0;
    rg.last = rg.pos0 + rg.live_rows - 1;
    rg.window = a.window;
    rg.scale2 = 1.4426950408889634f * a.scale;
    prompt_attention_block(src, rg, a.out + (size_t)r0 * a.ldo + (size_t)head * 128, (size_t)a.ldo);
}

}  // namespace

// Whole heads of 128 + 64 / 128 in aligned bf16 rows; a positive scale (the row maximum is taken before it is applied).
bool latent_prompt_serves(const LatentArgs& a) {
    const uintptr_t bits = reinterpret_cast<uintptr_t>(a.in) | reinterpret_cast<uintptr_t>(a.cache) | reinterpret_cast<uintptr_t>(a.expanded) | reinterpret_cast<uintptr_t>(a.out);
    return !a.in_f32 && !a.cache_f32 && a.dim == 128 && a.rot == 64 && a.vdim == 128 && a.scale > 0.0f && (bits & 15u) == 0 &&
           ((a.ld | a.q_off | a.lde | a.pitch | a.kr_off) & 7) == 0 && (a.ldo & 3) == 0 && a.lde >= a.heads * 256;
}

int latent_prompt_launch(cudaStream_t stream, const LatentArgs& a) {
    CUtensorMap map_ex, map_cache;
    KMLL_TRY_RC(make_map_bf16_rows(&map_ex, a.expanded, (uint64_t)a.heads * 256, (uint64_t)(a.pos0 + a.T - a.first), (uint64_t)a.lde * 2, kPaKeys));
    KMLL_TRY_RC(make_map_bf16_rows(&map_cache, a.cache, (uint64_t)a.pitch, (uint64_t)(a.pos0 + a.T), (uint64_t)a.pitch * 2, kPaKeys));
    cudaError_t e = allow_all_dynamic_smem(latent_prompt_kernel);
    if (e == cudaSuccess)
        e = launch(latent_prompt_kernel, dim3(a.heads, (a.T + kPaRows - 1) / kPaRows), dim3(kPaThreads), PaShape<192, 128, 1, 1>::kSmemBytes, stream, true, a, map_ex, map_cache);
    if (e != cudaSuccess) return fail(KMLL_ERR_CUDA, "latent attention (prompt): %s", cudaGetErrorString(e));
    return KMLL_OK;
}

// A block here has 128 rows and costs 11 to 15 us however few keys they see; one of the mma.sync kernel has 64 and costs 3 to 5 a key tile of 64.  So
// that kernel keeps short prompts and narrow windows.  Both with the rotation in front, which writes the planes of an f32 cache; 8 to
// 32 heads, here / there in us: heads of 128, 128 tokens 20.2 / 18.4 and 129 tokens 20.2 / 20.9 (32 heads, f32 cache; bf16 20.4 / 19.0 and 19.9 / 19.9); 1024
// tokens and windows of 64 (two tiles there) 28.3 / 26.5, of 72 (three) 27.9 / 29.0, of 256 32.0 / 46.0.  Heads of 64: 129 tokens 15.9 / 14.8, 192 15.5 /
// 16.0, 200 16.6 / 18.9; 1024 tokens, f32 cache, windows of 128 19.0 / 19.7, 192 23.7 / 23.6 (2000 tokens 40.4 / 35.3), 256 23.2 / 26.5; bf16 cache, 32 heads, 256 38.3 / 30.7,
// 384 40.4 / 34.1, 512 39.9 / 39.8 (2000 tokens 73.6 / 77.0).
bool prompt_attention_pays(int prompt_len, int window, int head_dim, int kv_bf16) {
    const int shortest = head_dim == 128 ? 129 : 193, narrowest = head_dim == 128 ? 66 : kv_bf16 ? 512 : 256;
    return prompt_len >= shortest && (window <= 0 || window >= prompt_len || window >= narrowest);
}

bool prompt_attention_serves(const void* q, const void* k, const void* v, const void* out, int head_dim) {
    const uintptr_t bits = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(out);
    return (head_dim == 64 || head_dim == 128) && (bits & 15u) == 0;
}

int prompt_attention_launch(cudaStream_t stream, const float* q_batch, const void* k, const void* v, int prompt_len, int n_heads, int n_kv_heads,
                            int head_dim, float* out, int kv_bf16, int window) {
    const int kv_len = n_kv_heads * head_dim, inner = kv_bf16 ? kv_len : 2 * kv_len;
    CUtensorMap map_k, map_v;
    KMLL_TRY_RC(make_map_bf16_rows(&map_k, k, (uint64_t)inner, (uint64_t)prompt_len, (uint64_t)inner * 2, kPaKeys));
    KMLL_TRY_RC(make_map_bf16_rows(&map_v, v, (uint64_t)inner, (uint64_t)prompt_len, (uint64_t)inner * 2, kPaKeys));
    auto go = [&](auto kern, size_t smem) {
        cudaError_t e = allow_all_dynamic_smem(kern);
        if (e != cudaSuccess) return e;
        return launch(kern, dim3(n_heads, (prompt_len + kPaRows - 1) / kPaRows), dim3(kPaThreads), smem, stream, true, q_batch, prompt_len, n_heads, n_kv_heads, out,
                      window, map_k, map_v);
    };
    cudaError_t e;
    if (head_dim == 128) e = kv_bf16 ? go(prompt_attention_kernel<128, true>, PaShape<128, 128, 2, 1>::kSmemBytes) : go(prompt_attention_kernel<128, false>, PaShape<128, 128, 2, 2>::kSmemBytes);
    else e = kv_bf16 ? go(prompt_attention_kernel<64, true>, PaShape<64, 64, 2, 1>::kSmemBytes) : go(prompt_attention_kernel<64, false>, PaShape<64, 64, 2, 2>::kSmemBytes);
    if (e != cudaSuccess) return fail(KMLL_ERR_CUDA, "prompt attention: %s", cudaGetErrorString(e));
    return KMLL_OK;
}

int prompt_attention_status(int* status_out) {
    cudaError_t e = cudaMemcpyFromSymbol(status_out, g_prompt_attention_status, sizeof(int));
    if (e != cudaSuccess) return fail(KMLL_ERR_CUDA, "device_status: %s", cudaGetErrorString(e));
    return KMLL_OK;
}

}  // namespace kmll
