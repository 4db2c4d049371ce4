// Batched quantized linear of 33 or more rows of x on pairs of multiprocessors, included by linear.cu.  Serves kmll's batched
// i8 linear (gemm_f32_i8_scaled_tiled_kernel, crates/inference/src/kernels/matmul.rs:116-214) for RS-I8 and W4-G128.
//
// y[m, r] = sum_k dequant(W)[r, k] * x[m, k] as tcgen05.mma.cta_group::2.kind::f16: 256 weight rows (128 in each block of a
// cluster of two) against up to 256 rows of x, half of which lie in each block's shared memory.
//
// What bounds it: the tensor cores.  An f32 row of x counts as two binary16 planes (x = 2^-sh (x_hi + x_lo), 22 bits), so two
// MMAs per useful one are the least; the dequantized W4 weight q * scale has 14 bits and would need two planes of its own (a
// third MMA).  Here the weight operand is the integer q alone, exact in binary16, and the group scale is applied behind the
// contraction, as kmll applies its scales: the 128 columns of a group accumulate in tensor memory, the drain warps
// (tensor-memory lane = weight row = one scale per thread) add scale * D to f32 sums in registers, two accumulators alternate.
// A drain takes ~600 cycles of the ~2000 the group's MMAs take.  RS-I8 rows have one scale: even and odd k-tiles of a unit
// accumulate separately and are drained once.
//
// Why pairs: with one block per tile both planes of 256 rows of x cross L2 -> SM for every 128 weight rows (64 bytes per cycle
// at the MMA rate of two planes, the whole port); a pair brings each row of x into one of the two blocks only.
//
// Measured in a graph of ten calls, split of x included (one block per 128 x 256 tile with three / two MMAs per k-step before): W4 2048 x 14336 x
// 4096 612 -> 355 us (677 TFLOP/s useful, 1353 of MMA work), RS-I8 587 -> 328, W4 300 x 18944 x 3584 131 -> 73, 64 x 14336 x 4096 53 -> 29,
// RS-I8 333 x 4096 x 4096 74 -> 31, W4 33 x 3584 x 3584 28 -> 17.  Issued by whole warps (tcgen05.cuh) instead of single threads: W4 2048 x 14336 x
// 4096 362 -> 334, 300 x 18944 x 3584 72 -> 62, 200 x 28672 x 4096 97 -> 90, 200 x 4096 x 14336 56 -> 50, RS-I8 333 x 4096 x 14336 82 -> 76.  Error against 64 bits 8.4e-6 -> 2.6e-7 (W4: no second weight plane).
//
// Roles of a block (512 threads, one block per SM, persistent over units = (weight row tile, x block, k-split)):
//   warp 0      TMA of x: both planes of n_block / 2 rows, one 3-D box per 64-column k-tile
//   warp 1, 3   tensor memory (warp 1); in the leader block (rank 0) each issues the MMAs of one accumulator, so that one's waits and
//               commits run behind the other's MMAs
//   warp 2      TMA of the raw weight tile (ahead of the grid dependency: weights are constants)
//   warps 4-7   expand raw weights to swizzled binary16 rows of the MMA operand
//   warps 8-15  drain accumulators, epilogue
// setmaxnreg moves registers to the drain warps (40 + 40 + 2 x 216 = 4 x 128 per thread of a warpgroup).
// Barriers: `full` (own block's copies of a stage landed), `a_ready` (in the leader: both blocks' operands of a stage are
// written), `empty` (in each block, multicast commit), `acc_full` (in each block, multicast commit), `acc_empty` (in the leader).
// Every wait is bounded; on a time-out the role raises the device status word and walks to the cluster barrier at the end.
#pragma once

namespace kmll {

constexpr int kPThreads = 512;
constexpr int kPMaxMats = 3;
constexpr int kPClusters = 74;   // pairs of the 148 multiprocessors

struct PairMat {
    const void* scales;        // RS-I8: float[rows]; W4: binary16 [rows, K / 128]
    float* out;                // [M, ldo]
    const float* residual;     // [M, ldo] or null
    int rows, ldo;
    int tile_start;            // first 256-row tile of this matrix
};
struct PairParams {
    PairMat mat[kPMaxMats];
    int nmat, K, M;
    int n_block, x_blocks;     // rows of x per unit (multiple of 16, <= 256)
    int ksplit, units;         // units = row tiles * x blocks * k-splits
    int stages;
    const float* inv_xscale;   // [M] 2^-sh per row of x
    float* partial;            // split-K: [128-row tiles][x blocks][splits][n_block][128] partial sums
    unsigned int* counters;    // split-K: 8 per (128-row tile, x block), zero between launches
};

// Arrival on the leader block's copy of a barrier.  What it orders lies in this block's shared or tensor memory, where the pair's
// MMA reads it through the async proxy: the fences in front of the arrival do that, a cluster-wide release (which waits for every
// store of the thread, ~1000 cycles with copies in flight) is not needed.
__device__ inline void mbar_arrive_leader(uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %0, 0;\n\tmbarrier.arrive.shared::cluster.b64 _, [ra];\n\t}"
        ::"r"(smem_u32(bar)) : "memory");
}
// (issued by the elected lane of a converged warp, see tcgen05.cuh)
__device__ inline void pair_mma_f16(uint32_t lead, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\t"
        "@e tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(lead)
        : "memory");
}
// completion of all earlier MMAs of this thread, signalled on the same barrier of both blocks
__device__ inline void pair_commit(uint32_t lead, uint64_t* bar) {
    asm volatile("{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %2, 0;\n\t"
                 "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
                 ::"r"(smem_u32(bar)), "h"((uint16_t)3), "r"(lead) : "memory");
}
// two f32 sums: acc += s * (lo, hi)
__device__ inline void fma_pair(unsigned long long& acc, unsigned long long s2, uint32_t lo, uint32_t hi) {
    const unsigned long long d = ((unsigned long long)hi << 32) | lo;
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(s2), "l"(d));
}

// The 2^-sh of up to 128 rows of x, one per lane and register.  Loaded at the start of a unit: a load waits behind the tile copies in
// flight (~3000 cycles), and one in front of every 16 columns made the epilogue 23000 cycles long.
struct PairScales {
    float v[4];
    __device__ PairScales(const float* inv_xscale, int m, int n, int lane) {
#pragma unroll
        for (int c = 0; c < 4; ++c) v[c] = c * 32 + lane < n ? __ldg(inv_xscale + m + c * 32 + lane) : 0.0f;
    }
    __device__ float chunk(int c) const { return c < 32 ? v[0] : c < 64 ? v[1] : c < 96 ? v[2] : v[3]; }
};
// 16 columns (rows of x m .. m + n_ok - 1) of one weight row: y = d 2^-sh scale (+ residual); `iv`: the 2^-sh of 32 columns, these from
// lane `iv0`; the loads of the residual are issued together
__device__ inline void store_columns(const PairMat& mat, int row, bool row_ok, int m, int n_ok, float iv, int iv0, float rscale, const uint32_t (&d)[16]) {
    const size_t o = (size_t)m * mat.ldo + row;
    const int ldo = mat.ldo;
    float* out = mat.out + o;
    if (mat.residual != nullptr) {
        const float* res = mat.residual + o;
        float r[16];
#pragma unroll
        for (int j = 0; j < 16; ++j, res += ldo) r[j] = (row_ok && j < n_ok) ? *res : 0.0f;
#pragma unroll
        for (int j = 0; j < 16; ++j, out += ldo) {
            const float v = r[j] + __uint_as_float(d[j]) * __shfl_sync(0xffffffffu, iv, iv0 + j) * rscale;
            if (row_ok && j < n_ok) *out = v;
        }
    } else {
#pragma unroll
        for (int j = 0; j < 16; ++j, out += ldo) {
            const float v = __uint_as_float(d[j]) * __shfl_sync(0xffffffffu, iv, iv0 + j) * rscale;
            if (row_ok && j < n_ok) *out = v;
        }
    }
}
// Position in the ring of stages: counted, not divided (a division by a run-time number per k-tile costs the issuing thread ~600 cycles).
struct PairRing {
    int stage = 0, stages;
    uint32_t phase = 0;  // parity of this stage's next use
    bool wrapped = false;
    __device__ explicit PairRing(int n) : stages(n) {}
    __device__ void next() {
        if (++stage == stages) { stage = 0; phase ^= 1u; wrapped = true; }
    }
};

struct PairUnit {
    int mat, row0;             // first weight row of this block inside its matrix
    int m0;                    // first row of x
    int kt0, KT;               // k-tiles
    int z, slot;               // k-split, index of (128-row tile, x block)
};
template <bool W4>
__device__ inline PairUnit pair_unit(const PairParams& p, int unit, int rank) {
    PairUnit u;
    const int tile = unit / p.ksplit;
    u.z = unit - tile * p.ksplit;
    const int rt = tile / p.x_blocks, xb = tile - rt * p.x_blocks;
    u.mat = (p.nmat > 2 && rt >= p.mat[2].tile_start) ? 2 : (p.nmat > 1 && rt >= p.mat[1].tile_start) ? 1 : 0;
    u.row0 = (rt - p.mat[u.mat].tile_start) * 256 + rank * 128;
    u.m0 = xb * p.n_block;
    // splits fall on whole groups (W4); there are at least as many groups as splits
    constexpr int kUnitTiles = W4 ? 2 : 1;
    const unsigned int items = (unsigned int)p.K / (kGKT * kUnitTiles);
    const int a = (int)(items * (unsigned int)u.z / (unsigned int)p.ksplit), b = (int)(items * (unsigned int)(u.z + 1) / (unsigned int)p.ksplit);
    u.kt0 = a * kUnitTiles;
    u.KT = (b - a) * kUnitTiles;
    u.slot = (rt * 2 + rank) * p.x_blocks + xb;
    return u;
}

// WIDE, up to 128 rows of x: the two planes of a block's rows lie back to back, so one MMA of N = 2 n_block multiplies both.  The
// accumulator columns are then, for each block's half of the rows, [x_hi | x_lo], added by the drain.  (Issuing an MMA takes ~70
// cycles however narrow it is.)
template <int FMT, bool WIDE>
__global__ void __launch_bounds__(kPThreads, 1) linear_gemm_pair_kernel(const PairParams p, const __grid_constant__ CUtensorMap map_w0,
                                                                       const __grid_constant__ CUtensorMap map_w1,
                                                                       const __grid_constant__ CUtensorMap map_w2,
                                                                       const __grid_constant__ CUtensorMap map_x) {
    constexpr bool W4 = FMT == FMT_W4;
    constexpr int kRawBytes = W4 ? 128 * 32 : 128 * 64;
    constexpr int kABytes = 128 * 128;
    constexpr int kChunks = WIDE ? 2 : 4;  // of 32 columns of x per drain warp
    extern __shared__ unsigned char psmem_raw[];
    unsigned char* smem = psmem_raw + ((1024u - (smem_u32(psmem_raw) & 1023u)) & 1023u);  // the same offset in both blocks
    const int n_half = p.n_block / 2;
    const int b_bytes = n_half * 128;  // one plane of this block's rows of x
    const int stage_bytes = kABytes + 2 * b_bytes + kRawBytes;
    const int stages = p.stages;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)stages * stage_bytes);
    uint64_t* a_ready = full + stages;
    uint64_t* empty = a_ready + stages;
    uint64_t* acc_full = empty + stages;
    uint64_t* acc_empty = acc_full + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);

    const int tid = threadIdx.x, lane = tid & 31, warp = uniform_warp_index();
    const int rank = (int)(blockIdx.x & 1u), cluster = (int)(blockIdx.x >> 1), n_clusters = (int)(gridDim.x >> 1);
    if (tid == 0) {
        for (int s = 0; s < stages; ++s) { mbar_init(&full[s], 2); mbar_init(&a_ready[s], 8); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 16); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");  // the other block's barriers exist
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t smem_base = smem_u32(smem);
    bool ok = true;

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp != 2) pdl_wait();  // the planes of x come from the previous kernel
        const uint32_t lead = elect_lead();
        PairRing ring(stages);
        if (warp == 0 || warp == 2) {
            for (int unit = cluster; unit < p.units && ok; unit += n_clusters) {
                const PairUnit u = pair_unit<W4>(p, unit, rank);
                const CUtensorMap* mw = u.mat == 0 ? &map_w0 : u.mat == 1 ? &map_w1 : &map_w2;
#pragma unroll 1
                for (int kt = 0; kt < u.KT; ++kt, ring.next()) {
                    const int stage = ring.stage;
                    if (ring.wrapped && !warp_wait(&empty[stage], ring.phase ^ 1u)) { ok = false; break; }
                    const uint32_t st = smem_base + (uint32_t)stage * stage_bytes;
                    const int k = (u.kt0 + kt) * kGKT;
                    if (warp == 0) {
                        lead_expect_tx(lead, &full[stage], (uint32_t)(2 * b_bytes));
                        lead_tma_3d(lead, st + kABytes, &map_x, k, u.m0 + rank * n_half, 0, &full[stage]);
                    } else {
                        lead_expect_tx(lead, &full[stage], (uint32_t)kRawBytes);
                        lead_tma_2d(lead, st + kABytes + 2 * b_bytes, mw, W4 ? k / 2 : k, u.row0, &full[stage]);
                    }
                }
            }
            // nothing of this block's copies, and no arrival on its barriers, is in flight when it reaches the end
            for (int j = 0; j < stages; ++j, ring.next())
                if (ring.wrapped && !warp_wait(ok ? &empty[ring.stage] : &full[ring.stage], ring.phase ^ 1u)) { ok = false; break; }
        } else if (rank == 0) {
            // ---- two issuing warps, one per accumulator: warp 1 the even spans, warp 3 the odd ones (a span: W4 the two k-tiles of
            // a group, RS-I8 every other k-tile of a unit)
            const uint32_t idesc = gemm_idesc_f16(256, WIDE ? 2 * p.n_block : p.n_block);
            const int own = warp >> 1;
            const uint32_t dst = (uint32_t)own * 256u;  // (all 512 columns are this pair's: they start at 0)
            int span0 = 0;
            uint32_t uses = 0, acc = 0u;
            for (int unit = cluster; unit < p.units && ok; unit += n_clusters) {
                const int KT = pair_unit<W4>(p, unit, 0).KT;
#pragma unroll 1
                for (int kt = 0; kt < KT; ++kt, ring.next()) {
                    if (((W4 ? span0 + (kt >> 1) : kt) & 1) != own) continue;
                    const int stage = ring.stage;
                    if (W4 ? (kt & 1) == 0 : kt < 2) {  // first k-tile of a span
                        if (uses > 0 && !warp_wait(&acc_empty[own], (uses - 1) & 1u)) { ok = false; break; }
                        acc = 0u;
                    }
                    // an odd ring: the stage's use before this one was the other warp's; before it has come, the parity below is that
                    // of the use before it
                    if ((stages & 1) != 0 && ring.wrapped && !warp_wait(&empty[stage], ring.phase ^ 1u)) { ok = false; break; }
                    if (!warp_wait(&a_ready[stage], ring.phase)) { ok = false; break; }
                    tcgen05_fence_after();
                    const uint32_t st = smem_base + (uint32_t)stage * stage_bytes;
                    const uint64_t da = gemm_smem_desc(st), dh = gemm_smem_desc(st + kABytes), dl = gemm_smem_desc(st + kABytes + b_bytes);
#pragma unroll
                    for (int ks = 0; ks < kGKT / 16; ++ks) {  // 32 bytes = 2 descriptor units per k-step
                        pair_mma_f16(lead, dst, da + 2 * ks, dh + 2 * ks, idesc, acc);
                        if (!WIDE) pair_mma_f16(lead, dst, da + 2 * ks, dl + 2 * ks, idesc, 1u);
                        acc = 1u;
                    }
                    pair_commit(lead, &empty[stage]);
                    if (W4 ? (kt & 1) == 1 : kt + 2 >= KT) {  // last one
                        pair_commit(lead, &acc_full[own]);
                        ++uses;
                    }
                }
                span0 += KT >> 1;
            }
        }
    } else if (warp < 8) {
        // ---- weight expansion: thread pair (row, half) turns 32 columns of two raw rows into binary16 in the swizzled tile
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        pdl_wait();
        const int et = tid - 128, h = et & 1;
        PairRing ring(stages);
        for (int unit = cluster; unit < p.units && ok; unit += n_clusters) {
            const int KT = pair_unit<W4>(p, unit, rank).KT;
#pragma unroll 1
            for (int kt = 0; kt < KT; ++kt, ring.next()) {
                const int stage = ring.stage;
                if (!mbar_wait<false>(&full[stage], ring.phase)) { ok = false; break; }
                unsigned char* a = smem + (size_t)stage * stage_bytes;
                const unsigned char* raw = a + kABytes + 2 * b_bytes;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int r = (et >> 1) + 64 * i;
                    if (W4) {
                        const uint4 w = *reinterpret_cast<const uint4*>(raw + r * 32 + h * 16);
                        const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                        for (int c = 0; c < 4; ++c) {  // one word = 8 columns in the order 0 4 1 5 2 6 3 7 (split_rows_kernel permutes x alike)
                            // 0x6400 | n is the binary16 1024 + n, 0x6400 | (n << 4) is 1024 + 16 n: q = n - 8 without a conversion
                            const uint32_t kMagic = 0x64006400u, kSubLo = 0x64086408u /* 1032 */, kMulHi = 0x2c002c00u /* 1/16 */, kAddHi = 0xd480d480u /* -72 */;
                            const uint32_t w0 = ww[c], w8 = ww[c] >> 8;
                            uint32_t qa = lop3_and_or(w0, 0x000f000fu, kMagic), qb = lop3_and_or(w0, 0x00f000f0u, kMagic);
                            uint32_t qc = lop3_and_or(w8, 0x000f000fu, kMagic), qd = lop3_and_or(w8, 0x00f000f0u, kMagic);
                            __half2 q2[4];
                            q2[0] = __hsub2(*reinterpret_cast<__half2*>(&qa), *reinterpret_cast<const __half2*>(&kSubLo));
                            q2[1] = __hfma2(*reinterpret_cast<__half2*>(&qb), *reinterpret_cast<const __half2*>(&kMulHi), *reinterpret_cast<const __half2*>(&kAddHi));
                            q2[2] = __hsub2(*reinterpret_cast<__half2*>(&qc), *reinterpret_cast<const __half2*>(&kSubLo));
                            q2[3] = __hfma2(*reinterpret_cast<__half2*>(&qd), *reinterpret_cast<const __half2*>(&kMulHi), *reinterpret_cast<const __half2*>(&kAddHi));
                            const uint32_t* q = reinterpret_cast<const uint32_t*>(q2);
                            *reinterpret_cast<uint4*>(a + r * 128 + ((4 * h + c) ^ (r & 7)) * 16) = make_uint4(q[0], q[1], q[2], q[3]);
                        }
                    } else {
                        const uint4 w0 = *reinterpret_cast<const uint4*>(raw + r * 64 + h * 32);
                        const uint4 w1 = *reinterpret_cast<const uint4*>(raw + r * 64 + h * 32 + 16);
                        const uint32_t ww[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            uint32_t h2[4];
#pragma unroll
                            for (int e = 0; e < 2; ++e) {  // 4 signed bytes -> 2 half2, exact (bias to unsigned, 1024 + u as a half, minus 1152)
                                const uint32_t v = ww[2 * c + e] ^ 0x80808080u;
                                uint32_t lo = __byte_perm(v, 0x64646464u, 0x4140), hi = __byte_perm(v, 0x64646464u, 0x4342);
                                const uint32_t kSub = 0x64806480u;
                                const __half2 r0 = __hsub2(*reinterpret_cast<__half2*>(&lo), *reinterpret_cast<const __half2*>(&kSub));
                                const __half2 r1 = __hsub2(*reinterpret_cast<__half2*>(&hi), *reinterpret_cast<const __half2*>(&kSub));
                                h2[2 * e] = *reinterpret_cast<const uint32_t*>(&r0);
                                h2[2 * e + 1] = *reinterpret_cast<const uint32_t*>(&r1);
                            }
                            *reinterpret_cast<uint4*>(a + r * 128 + ((4 * h + c) ^ (r & 7)) * 16) = make_uint4(h2[0], h2[1], h2[2], h2[3]);
                        }
                    }
                }
                fence_proxy_async_smem();  // the tensor core reads these tiles through the async proxy
                __syncwarp();
                if (lane == 0) mbar_arrive_leader(&a_ready[stage]);
            }
        }
    } else {
        // ---- drain and epilogue: warp w reads tensor-memory lanes 32 (w % 4) .., warps 8-11 the first half of the columns
        asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
        pdl_wait();
        const int q = warp & 3, half = (warp - 8) >> 2, rl = q * 32 + lane;
        const int c_first = half * n_half;
        const int n_groups = p.K >> 7;
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(WIDE ? 2 * c_first : c_first);
        auto load_columns = [&](uint32_t at, int c, uint32_t (&d)[32]) {
            tmem_load_x32(at + (uint32_t)c * 32u, d);
            if (WIDE) {
                uint32_t lo[32];
                tmem_load_x32(at + (uint32_t)(n_half + c * 32), lo);
#pragma unroll
                for (int j = 0; j < 32; ++j) d[j] = __float_as_uint(__uint_as_float(d[j]) + __uint_as_float(lo[j]));
            }
        };
        uint32_t phases = 0u, buffer = 0u;
        for (int unit = cluster; unit < p.units; unit += n_clusters) {
            const PairUnit u = pair_unit<W4>(p, unit, rank);
            const PairMat& mat = p.mat[u.mat];
            const int row = u.row0 + rl, srow = min(row, mat.rows - 1);
            const int spans = W4 ? u.KT >> 1 : min(u.KT, 2);
            const unsigned short* sc = reinterpret_cast<const unsigned short*>(mat.scales) + (size_t)srow * n_groups + (u.kt0 >> 1);
            unsigned short s0 = 0, s1 = 0;  // a group scale is requested two groups ahead of its use
            if (W4) {
                s0 = __ldg(sc);
                if (spans > 1) s1 = __ldg(sc + 1);
            } else {
                buffer = 0u;
            }
            const PairScales scales(p.inv_xscale, u.m0 + c_first, min(n_half, p.M - (u.m0 + c_first)), lane);
            const float rscale = W4 ? 1.0f : reinterpret_cast<const float*>(mat.scales)[srow];
            unsigned long long acc[16 * kChunks];  // pairs of f32 sums
#pragma unroll
            for (int j = 0; j < 16 * kChunks; ++j) acc[j] = 0ull;
#pragma unroll 1
            for (int g = 0; g < spans; ++g, buffer ^= 1u) {
                const uint32_t sb = __float_as_uint(W4 ? __half2float(__ushort_as_half(s0)) : 1.0f);
                const unsigned long long s2 = ((unsigned long long)sb << 32) | sb;
                s0 = s1;
                if (W4 && g + 2 < spans) s1 = __ldg(sc + g + 2);
                ok = __all_sync(0xffffffffu, mbar_wait<false>(&acc_full[buffer], (phases >> buffer) & 1u));
                if (!ok) break;
                phases ^= 1u << buffer;
                tcgen05_fence_after();
#pragma unroll
                for (int c = 0; c < kChunks; ++c) {
                    if (c * 32 < n_half) {
                        uint32_t d[32];
                        load_columns(taddr + buffer * 256u, c, d);
#pragma unroll
                        for (int j = 0; j < 16; ++j) fma_pair(acc[c * 16 + j], s2, d[2 * j], d[2 * j + 1]);
                    }
                }
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_leader(&acc_empty[buffer]);
            }
            if (!ok) break;
            const bool split = p.ksplit > 1, row_ok = row < mat.rows;
            float* part = p.partial + ((size_t)u.slot * p.ksplit + u.z) * (size_t)p.n_block * 128;
#pragma unroll
            for (int c = 0; c < 32 * kChunks; c += 16) {
                const int n_ok = n_half - c;
                if (n_ok <= 0) break;
                uint32_t d[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) d[j] = (uint32_t)(acc[(c + j) / 2] >> (32 * (j & 1)));
                if (split) {
                    float* to = part + (size_t)(c_first + c) * 128 + rl;
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (j < n_ok) to[j * 128] = __uint_as_float(d[j]);  // scales and residual are applied after the merge
                } else {
                    store_columns(mat, row, row_ok, u.m0 + c_first + c, min(n_ok, p.M - (u.m0 + c_first + c)), scales.chunk(c), c & 31, rscale, d);
                }
            }
            if (split) {
                // every warp merges its own rows and columns: the warp that delivers last adds the splits in split order
                __threadfence();
                __syncwarp();
                unsigned int* counter = p.counters + (size_t)u.slot * 8 + (warp - 8);
                unsigned int prev = 0;
                if (lane == 0) prev = atomicAdd(counter, 1u);
                prev = __shfl_sync(0xffffffffu, prev, 0);
                if (prev == (unsigned int)p.ksplit - 1u) {
                    __threadfence();
                    const float* base = p.partial + (size_t)u.slot * p.ksplit * (size_t)p.n_block * 128;
#pragma unroll 1
                    for (int c = 0; c < n_half; c += 16) {  // four splits' loads in flight (a round of loads costs ~1 us whatever it carries)
                        const int n_ok = n_half - c;
                        const float* from = base + (size_t)(c_first + c) * 128 + rl;
                        uint32_t d[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j) d[j] = 0u;
#pragma unroll 1
                        for (int z0 = 0; z0 < p.ksplit; z0 += 4) {
                            float t[4][16];
#pragma unroll
                            for (int z = 0; z < 4; ++z, from += (size_t)p.n_block * 128)
#pragma unroll
                                for (int j = 0; j < 16; ++j) t[z][j] = (z0 + z < p.ksplit && j < n_ok) ? __ldcg(from + j * 128) : 0.0f;
#pragma unroll
                            for (int z = 0; z < 4; ++z)
#pragma unroll
                                for (int j = 0; j < 16; ++j) d[j] = __float_as_uint(__uint_as_float(d[j]) + t[z][j]);
                        }
                        store_columns(mat, row, row_ok, u.m0 + c_first + c, min(n_ok, p.M - (u.m0 + c_first + c)), scales.chunk(c), c & 31, rscale, d);
                    }
                    if (lane == 0) *counter = 0u;
                }
            }
        }
    }
    // neither block may leave, or free tensor memory, while the other can still signal its barriers or read its operands
    if (!ok) atomicCAS(&g_device_status, 0, 1);
    __syncwarp();
    tcgen05_fence_before();
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
    tcgen05_fence_after();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
}

}  // namespace kmll
