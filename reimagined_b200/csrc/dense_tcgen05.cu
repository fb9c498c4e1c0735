// y[M,N] = x[M,K] (bf16) x w[N,K]^T (bf16) on the 5th-generation tensor cores: the dense counterpart of
// gemm_tcgen05.cu, with the same roles and the same operand geometry (a stage is 128 bytes of K per row, i.e. 64
// bf16, in the 128-byte-swizzled K-major layout TMA writes; an MMA takes 32 bytes of K).
//
// One persistent CTA per SM -- two of them up to 64 rows -- (or, where the tiles would leave SMs idle, a cluster of CTAs per tile that share its K
// range and finish it together), ten warps (six): TMA producer, MMA issuer (tcgen05.mma kind::f16, fp32 accumulators in TMEM,
// two buffers of BN columns), eight (four) epilogue warps.  128 x BN tiles; the two accumulators double-buffer tiles.  (256 x
// 256 tiles, which the int8 kernel uses for large problems, gain nothing here: these epilogues -- residual, gated pair --
// are longer, and a tall tile cannot hide them.)
// The epilogue adds the bias and either adds the fp32 residual and stores fp32, stores bf16, or -- for a gated
// feed-forward, whose weight rows alternate in blocks of 32 gate and 32 up rows -- combines two neighbouring
// 32-column blocks into act(gate) * up and stores that.
// Every wait is bounded: on a timeout the role records the status word and falls through to the common exit, where
// TMEM is released.
#include <cuda.h>

#include <algorithm>

#include "shares.cuh"
#include "stack.cuh"
#include "tc05.cuh"

namespace tbl {
namespace stack {
namespace {

using namespace tc05;

constexpr int BM = 128;             // activation rows per MMA
constexpr int BKB = 128;            // bytes of K per stage
constexpr int BKE = BKB / 2;        // the same in elements
constexpr int kGroupM = 16;         // row tiles per group of the tile walk
constexpr int kMaxStages = 12;
constexpr int kMaxSplit = 4;
__host__ __device__ constexpr int threads_for(int ar) { return 32 * (2 + ar / 16); }

// ar: activation rows of a stage, 128, or 64 for no more than that (see the kernel).  With 64 two CTAs share an SM.
__host__ __device__ constexpr int epi_warps(int ar) { return ar / 16; }
constexpr size_t other_smem(int ar) { return (ar == BM ? 1024 : 0) + epi_warps(ar) * 4096 + 256; }
// deep: where an SM has one CTA anyway, stages to fill it
__host__ __device__ constexpr int stages_for(int bn, int ar, bool deep) {
    return ar == BM ? (bn >= 192 ? 4 : (bn >= 128 ? 6 : 8)) : (bn >= 128 ? 4 : 6) * (deep ? 2 : 1);
}
constexpr size_t smem_for(int bn, int ar, bool deep) { return other_smem(ar) + static_cast<size_t>(stages_for(bn, ar, deep)) * (ar + bn) * BKB; }

struct Params {
    DenseCall c;
    int tiles_m, tiles_n;
    int split;              // shares of K = CTAs of a cluster (SHARED kernel)
    int deep;               // 64 rows: all of an SM's shared memory for one CTA
    int part;               // 64 rows: blocks of K that are added up in the tensor cores' accumulators
    int vec;                // outputs (and residual) take 4-column vector accesses
    int* status;
};

__device__ __forceinline__ bool decode_tile(const Params& p, int t, int& row0, int& tn) {
    if (t >= p.tiles_m * p.tiles_n) return false;
    const int per_group = kGroupM * p.tiles_n;
    const int grp = t / per_group, in_grp = t - grp * per_group;
    const int gm = min(kGroupM, p.tiles_m - grp * kGroupM);
    tn = in_grp / gm;
    row0 = (grp * kGroupM + in_grp % gm) * BM;
    return true;
}

// Stores one 32 x 32 block staged in shared memory (row = lane order, 16-byte chunk j of row r at j ^ (r & 7)).
template <bool RES>
__device__ __forceinline__ void store_block(const Params& p, const uint8_t* stage, int lane, int row0, int valid, int col0,
                                            int ncols) {
    const DenseCall& c = p.c;
    const int chunk = lane & 7, rsub = lane >> 3, col = col0 + 4 * chunk;
    if (col >= ncols) return;
    if (RES && p.vec) {
        // residual rows are requested together: one memory round trip per block, not one per row
        float4 res[8];
        {
#pragma unroll
            for (int i8 = 0; i8 < 8; ++i8) {
                const int rr = 4 * i8 + rsub;
                res[i8] = rr < valid ? *reinterpret_cast<const float4*>(c.residual + static_cast<size_t>(row0 + rr) * c.ldo + col)
                                     : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        }
#pragma unroll
        for (int i8 = 0; i8 < 8; ++i8) {
            const int rr = 4 * i8 + rsub;
            if (rr >= valid) continue;
            float4 f = *reinterpret_cast<const float4*>(stage + rr * 128 + ((chunk ^ (rr & 7)) << 4));
            f.x += res[i8].x; f.y += res[i8].y; f.z += res[i8].z; f.w += res[i8].w;
            *reinterpret_cast<float4*>(c.out_f32 + static_cast<size_t>(row0 + rr) * c.ldo + col) = f;
        }
        return;
    }
#pragma unroll
    for (int i8 = 0; i8 < 8; ++i8) {
        const int rr = 4 * i8 + rsub;
        if (rr >= valid) continue;
        const float4 f = *reinterpret_cast<const float4*>(stage + rr * 128 + ((chunk ^ (rr & 7)) << 4));
        const size_t o = static_cast<size_t>(row0 + rr) * c.ldo + col;
        if (p.vec && c.out_f32) {
            *reinterpret_cast<float4*>(c.out_f32 + o) = f;
        } else if (p.vec) {
            *reinterpret_cast<uint2*>(c.out_b16 + o) = make_uint2(pack_bf16(f.x, f.y), pack_bf16(f.z, f.w));
        } else {
            const float v[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (col + e >= ncols) break;
                if (c.out_f32) c.out_f32[o + e] = RES ? c.residual[o + e] + v[e] : v[e];
                else c.out_b16[o + e] = __float2bfloat16_rn(v[e]);
            }
        }
    }
}

// SHARED: a CTA takes one share of the K range of one tile, the CTAs of a cluster finish the tile together.
// AR: activation rows of a stage, 128, or 64 for no more rows than that: the MMA still takes 128, the upper half of them from the weights behind (of the
// same stage), and nobody reads those sums.
// With so few rows a layer is the stream of its weights, and what held that up was the chain of a K block in the two issuing warps (0.33 us a block however
// narrow the tile; one elected lane, places counted instead of divided for, descriptors by addition: 0.18) and that nothing streams while a block of one CTA
// to an SM starts up or stores.  So two CTAs share an SM, each with half of its memory, except where there are no more CTAs than SMs and K is long: then one
// has twice the stages.  us before | after at 64 rows, cold weights: 24576 gated x 4096 53.2 | 43.1, 32000 x 4096 53.9 | 47.3, 8192 x 4096 18.9 | 17.4,
// 4096 x 12288 24.6 | 23.2, 2048 x 6144 13.2 | 10.8, 10304 x 2048 15.4 | 12.1.  A step of 64 sequences of the width-4096 Guselix 803 | 762, of 32 of the
// width-2048 Goguvik 577 | 523, of 24 of the width-2048 Guselix 746 | 642.
// The accumulators drop the bits that they shift out, which adds up with K (1.1e-9 of the result per number of K).  Few rows have no shares of K to speak of,
// and went through a kernel that cuts K into eight before; so the accumulators hold a part of K at a time, in two buffers, and the epilogue's warps add the
// parts up in registers, rounding to nearest.  TMEM is free for the next tile before this one is stored.
template <int BN, int AR, bool RES, bool SHARED>
__global__ void __launch_bounds__(threads_for(AR), AR == BM ? 1 : 2)
dense_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ Params p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // (nothing else is in shared memory, which starts on a 1024-byte boundary as declared; with two CTAs there is no room to round up)
    uint8_t* smem = AR == BM ? reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023)) : smem_raw;
    constexpr int kThreads = threads_for(AR), kEpiWarps = epi_warps(AR);
    const int kStages = AR == BM ? stages_for(BN, AR, false) : stages_for(BN, AR, p.deep);
    constexpr int kLoadWarp = AR == BM ? 0 : 2, kMmaWarp = kLoadWarp + 1;   // the others are epilogue warps, which reach the TMEM lanes of their number mod 4
    constexpr int kABytes = AR * BKB;
    constexpr int kBBytes = BN * BKB;
    constexpr int kStageBytes = kABytes + kBBytes;
    constexpr uint32_t kTmemCols = BN == 192 ? 512 : 2 * BN;          // a power of two
    constexpr int LDS = BN + 4;                                        // floats per row of a share's sums
    static_assert(AR + BN >= BM, "the rows an MMA takes lie within the stage");
    static_assert(!SHARED || sizeof(float) * AR * LDS <= stages_for(BN, AR, false) * kStageBytes, "the sums take the stages' place");
    uint8_t* epi_stage = smem + kStages * kStageBytes;                 // 4 KB a warp
    uint64_t* full = reinterpret_cast<uint64_t*>(epi_stage + kEpiWarps * 4096);
    uint64_t* empty = full + kMaxStages;
    uint64_t* tmem_full = empty + kMaxStages;
    uint64_t* tmem_empty = tmem_full + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);

    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int all_blocks = (p.c.K + BKE - 1) / BKE, per = SHARED ? (all_blocks + p.split - 1) / p.split : all_blocks;
    const int share = SHARED ? blockIdx.x % p.split : 0, first = SHARED ? blockIdx.x / p.split : blockIdx.x;
    const int stride = SHARED ? p.tiles_m * p.tiles_n : gridDim.x;     // SHARED: this tile only
    const int kb0 = SHARED ? min(all_blocks, share * per) : 0, kblocks = SHARED ? min(all_blocks, kb0 + per) - kb0 : all_blocks;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full[b], 1); mbar_init(&tmem_empty[b], kEpiWarps); }
        fence_mbar_init();
        fence_proxy_async();
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (AR == BM) pdl_launch_dependents();
    // Up to 64 rows every tile starts at another block of K: otherwise all of them would ask for the same few lines of the activations at the same time
    // (64 x 24576 x 4096 45.3 and 43.1 us, 64 x 32000 x 4096 49.2 and 47.3; a step of 64 sequences of the width-4096 Goguvik 601 and 583).
    auto k_block = [&](int kb, int tn) {
        if (AR == BM) return kb0 + kb;
        const int at = kb + tn * 7 % kblocks;
        return kb0 + (at < kblocks ? at : at - kblocks);
    };
    // the weights of the first stages do not depend on the kernel before this one, unless the call says so
    int early = 0;
    if (warp == kLoadWarp) {
        int row0, tn;
        if (!p.c.w_computed && decode_tile(p, first, row0, tn)) early = min(kStages, kblocks);
        if (elect_one())
            for (int s = 0; s < early; ++s) {
                mbar_arrive_expect_tx(&full[s], kStageBytes);
                tma_load_2d(smem + s * kStageBytes + kABytes, &map_b, k_block(s, tn) * BKE, tn * BN, &full[s]);
            }
    }
    pdl_wait();
    // Up to 64 rows not before the wait (24 sequences at width 2048 646 and 640 us a step: dense_rows.cu says why), and up to 16, where the layers around are the
    // row-streaming kernel's, whose blocks crowd onto the SMs without one of these, not at all (16 sequences of the width-4096 Guselix 866 and 714,
    // of the width-2048 one 718 and 606).
    if (AR != BM && p.c.M > 16) pdl_launch_dependents();

    const int part = AR == BM ? kblocks : p.part;
    // 64 rows: waits for the parts of a tile one after the other and adds up `blocks` blocks of 32 columns, `step` apart from `col` on, of this warp's
    // rows.  False: a wait ran out.
    auto add_parts = [&](auto& v, int col, int step, int blocks, int& local) {
        constexpr int kBlocks = sizeof(v) / sizeof(v[0]);
#pragma unroll
        for (int i = 0; i < kBlocks; ++i)
#pragma unroll
            for (int e = 0; e < 32; ++e) v[i][e] = 0.0f;
        const uint32_t t_row = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16) + col;
        for (int begin = 0; begin < kblocks; begin += part, ++local) {
            const int buf = local & 1;
            const bool alive = mbar_wait_bounded(&tmem_full[buf], (local >> 1) & 1, p.status);
            if (!__all_sync(0xffffffffu, alive)) return false;
            tc_fence_after();
#pragma unroll
            for (int i = 0; i < kBlocks; ++i) {
                if (i >= blocks) break;
                uint32_t r[32];
                tmem_ld32(t_row + buf * BN + i * step, r);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 32; ++e) v[i][e] += __uint_as_float(r[e]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tmem_empty[buf]);
        }
        return true;
    };
    if (warp == kLoadWarp) {
        // ---------------- TMA producer ----------------
        if (elect_one()) {
            int s = 0, row0, tn;
            uint32_t round = 0;                                // full rounds of the ring so far
            bool alive = true;
            for (int tile = first; alive && decode_tile(p, tile, row0, tn); tile += stride) {
                for (int kb = 0; kb < kblocks; ++kb) {
                    if (round) {
                        alive = mbar_wait_bounded(&empty[s], (round - 1) & 1, p.status);
                        if (!alive) break;
                    }
                    uint8_t* a_dst = smem + s * kStageBytes;
                    const bool whole = round || s >= early;
                    if (whole) mbar_arrive_expect_tx(&full[s], kStageBytes);
                    tma_load_2d(a_dst, &map_a, k_block(kb, tn) * BKE, row0, &full[s]);
                    if (whole) tma_load_2d(a_dst + kABytes, &map_b, k_block(kb, tn) * BKE, tn * BN, &full[s]);
                    if (++s == kStages) { s = 0; ++round; }
                }
            }
        }
    } else if (warp == kMmaWarp) {
        // ---------------- MMA issuer ----------------
        if (elect_one()) {
            const uint32_t idesc = idesc_bf16(BN);
            const uint64_t a_desc = smem_desc_sw128(smem_u32(smem)), b_desc = smem_desc_sw128(smem_u32(smem) + kABytes);
            int s = 0, local = 0, row0, tn;                    // local: parts of tiles so far
            uint32_t phase = 0;
            bool alive = true;
            for (int tile = first; alive && decode_tile(p, tile, row0, tn); tile += stride) {
                for (int begin = 0; alive && begin < kblocks; begin += part, ++local) {
                    const int buf = local & 1, end = min(kblocks, begin + part);
                    if (local >= 2) {
                        alive = mbar_wait_bounded(&tmem_empty[buf], ((local >> 1) - 1) & 1, p.status);
                        if (!alive) break;
                    }
                    tc_fence_after();
                    const uint32_t d_tmem = tmem_base + buf * BN;
                    for (int kb = begin; kb < end; ++kb) {
                        alive = mbar_wait_bounded(&full[s], phase, p.status);
                        if (!alive) break;
                        tc_fence_after();
                        const uint32_t at = static_cast<uint32_t>(s) * (kStageBytes >> 4);     // descriptors count 16 bytes
#pragma unroll
                        for (int kk = 0; kk < BKB / 32; ++kk)
                            umma_f16(d_tmem, a_desc + at + 2 * kk, b_desc + at + 2 * kk, idesc, ((kb - begin) | kk) != 0 ? 1u : 0u);
                        umma_commit(&empty[s]);
                        if (++s == kStages) { s = 0; phase ^= 1; }
                    }
                    if (alive) umma_commit(&tmem_full[buf]);
                }
            }
        }
    } else if (SHARED) {
        // ---------------- sums of this share into the place of the stages (all of which the MMAs have read) ----------------
        const int quarter = warp & 3, half = AR == BM ? (warp - 2) >> 2 : warp >> 2;
        float* row = reinterpret_cast<float*>(smem) + (quarter * 32 + lane) * LDS + half * (BN / 2);
        if constexpr (AR == BM) {
            bool alive = mbar_wait_bounded(&tmem_full[0], 0, p.status);     // (no share is empty: K has four blocks for each)
            alive = __all_sync(0xffffffffu, alive);
            tc_fence_after();
#pragma unroll
            for (int j = 0; j < BN / 2; j += 32) {
                uint32_t r[32];
                tmem_ld32(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + half * (BN / 2) + j, r);
                tmem_ld_wait();
                if (alive)
#pragma unroll
                    for (int e = 0; e < 32; e += 4) *reinterpret_cast<uint4*>(row + j + e) = make_uint4(r[e], r[e + 1], r[e + 2], r[e + 3]);
            }
        } else {
            float v[BN / 64][32];
            int local = 0;
            if (add_parts(v, half * (BN / 2), 32, BN / 64, local))
#pragma unroll
                for (int i = 0; i < BN / 64; ++i)
#pragma unroll
                    for (int e = 0; e < 32; e += 4) *reinterpret_cast<float4*>(row + 32 * i + e) = make_float4(v[i][e], v[i][e + 1], v[i][e + 2], v[i][e + 3]);
        }
    } else if constexpr (AR != BM) {
        // ---------------- epilogue warps, 64 rows ----------------
        // Two blocks of 32 columns a warp: of a gated layer a pair, else every other one.  TMEM is free again before anything is stored.
        const int quarter = warp & 3, half = warp >> 2;
        uint8_t* stage = epi_stage + (2 * half + quarter) * 4096;
        const bool pair = p.c.pair_cols > 0;
        const Activation act = activation_of(p.c.act);
        int local = 0, tile_row0, tn;
        for (int tile = first; decode_tile(p, tile, tile_row0, tn); tile += stride) {
            const int row0 = tile_row0 + quarter * 32, valid = min(32, p.c.M - row0);
            const int nblocks = min(BN / 32, (p.c.N - tn * BN + 31) / 32), b0 = pair ? 2 * half : half, step = pair ? 1 : 2;
            const int mine = valid <= 0 || b0 >= nblocks ? 0 : (b0 + step < nblocks ? 2 : 1);
            float v[2][32];
            if (!add_parts(v, 32 * b0, 32 * step, mine, local)) break;
            const int n0 = tn * BN + 32 * b0;
            if (pair && mine) {                                // (N is a multiple of 64: both blocks are there)
                const float bias_l = p.c.bias ? __ldg(p.c.bias + n0 + lane) : 0.0f, bias_u = p.c.bias ? __ldg(p.c.bias + n0 + 32 + lane) : 0.0f;
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    const float g = v[0][i] + __shfl_sync(0xffffffffu, bias_l, i), u = v[1][i] + __shfl_sync(0xffffffffu, bias_u, i);
                    v[0][i] = activate(act, g) * u;
                }
            }
#pragma unroll 1
            for (int b = 0; b < (pair ? mine / 2 : mine); ++b) {
                const int col = n0 + 64 * b;
                if (p.c.bias && !pair) {
                    const float bias = col + lane < p.c.N ? __ldg(p.c.bias + col + lane) : 0.0f;
#pragma unroll
                    for (int i = 0; i < 32; ++i) v[0][i] += __shfl_sync(0xffffffffu, bias, i);
                }
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    *reinterpret_cast<float4*>(stage + lane * 128 + ((j ^ (lane & 7)) << 4)) =
                        make_float4(v[0][4 * j], v[0][4 * j + 1], v[0][4 * j + 2], v[0][4 * j + 3]);
                __syncwarp();
                store_block<RES>(p, stage, lane, row0, valid, pair ? col >> 1 : col, pair ? p.c.pair_cols : p.c.N);
#pragma unroll
                for (int i = 0; i < 32; ++i) v[0][i] = v[1][i];
            }
        }
    } else {
        // ---------------- epilogue warps ----------------
        const int quarter = warp & 3;          // TMEM lanes 32*quarter .. +31 are this warp's
        const int half = (warp - 2) >> 2;      // which of the two warps of the quarter
        uint8_t* stage = epi_stage + (warp - 2) * 4096;
        const bool pair = p.c.pair_cols > 0;
        const Activation act = activation_of(p.c.act);
        int local = 0, tile_row0, tn;
        bool alive = true;
        for (int tile = first; alive && decode_tile(p, tile, tile_row0, tn); tile += stride, ++local) {
            const int buf = local & 1;
            alive = mbar_wait_bounded(&tmem_full[buf], (local >> 1) & 1, p.status);
            alive = __all_sync(0xffffffffu, alive);
            if (!alive) break;
            tc_fence_after();
            const int row0 = tile_row0 + quarter * 32;
            const int valid = min(32, p.c.M - row0);
            const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buf * BN;
            const int nblocks = min(BN / 32, (p.c.N - tn * BN + 31) / 32);
            // blocks of 32 columns: every other one is this warp's -- of a gated layer every other pair
            const int step = pair ? 2 : 1;
            uint32_t r[32], rn[32];
            if (half * step < nblocks) tmem_ld32(t_row + half * step * 32, r);
#pragma unroll 1
            for (int b = half * step; b < nblocks; b += 2 * step) {
                const int n0 = tn * BN + b * 32;
                const float bias_l = p.c.bias && n0 + lane < p.c.N ? __ldg(p.c.bias + n0 + lane) : 0.0f;
                int col0 = n0, ncols = p.c.N;
                float v[32];
                tmem_ld_wait();
                if (pair) {
                    tmem_ld32(t_row + (b + 1) * 32, rn);      // N is a multiple of 64
                    const float bias_u = p.c.bias ? __ldg(p.c.bias + n0 + 32 + lane) : 0.0f;
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const float g = __uint_as_float(r[i]) + __shfl_sync(0xffffffffu, bias_l, i);
                        const float u = __uint_as_float(rn[i]) + __shfl_sync(0xffffffffu, bias_u, i);
                        v[i] = activate(act, g) * u;
                    }
                    if (b + 4 < nblocks) tmem_ld32(t_row + (b + 4) * 32, r);
                    col0 = n0 >> 1;
                    ncols = p.c.pair_cols;
                } else {
                    if (b + 2 < nblocks) tmem_ld32(t_row + (b + 2) * 32, rn);   // in flight while this block is stored
                    if (p.c.bias) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]) + __shfl_sync(0xffffffffu, bias_l, i);
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
                    }
                }
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    *reinterpret_cast<float4*>(stage + lane * 128 + ((j ^ (lane & 7)) << 4)) =
                        make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                __syncwarp();
                if (valid > 0) store_block<RES>(p, stage, lane, row0, valid, col0, ncols);
                if (!pair) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) r[i] = rn[i];
                }
            }
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tmem_empty[buf]);
        }
    }

    if constexpr (SHARED) {
        int row0, tn;
        decode_tile(p, first, row0, tn);
        __syncwarp();
        cluster_sync_all();
        finish_shares<BN, LDS, kThreads>(p.c, smem_u32(smem), p.split, share, tn, row0, AR, p.vec, [](int, int, float v) { return v; });
        cluster_sync_all();                                // nobody leaves while a neighbour may still read its sums
    }

    // common exit: all roles meet, then the allocating warp releases TMEM
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
}

template <int BN, int AR, bool RES, bool SHARED>
cudaError_t launch_kernel(const CUtensorMap& ma, const CUtensorMap& mb, const Params& p, cudaStream_t st) {
    static bool done[64] = {};
    constexpr size_t most = smem_for(BN, AR, true);
    static_assert(most <= 227 * 1024 && (AR == BM || smem_for(BN, AR, false) <= 113 * 1024), "shared memory of a CTA");
    const size_t smem = smem_for(BN, AR, p.deep);
    const cudaError_t e = allow_smem(dense_tcgen05_kernel<BN, AR, RES, SHARED>, most, done);
    if (e != cudaSuccess) return e;
    const int tiles = p.tiles_m * p.tiles_n;
    constexpr int kThreads = threads_for(AR), room = AR == BM ? kNumSm : 2 * kNumSm;
    if (SHARED) return launch_dependent_cluster(dense_tcgen05_kernel<BN, AR, RES, SHARED>, dim3(tiles * p.split), p.split, dim3(kThreads), smem, st, ma, mb, p);
    return launch_dependent(dense_tcgen05_kernel<BN, AR, RES, SHARED>, dim3(tiles < room ? tiles : room), dim3(kThreads), smem, st, ma, mb, p);
}
template <int BN, int AR>
cudaError_t launch_bn(const CUtensorMap& ma, const CUtensorMap& mb, const Params& p, cudaStream_t st) {
    if constexpr (BN != 192)
        if (p.split > 1) return launch_kernel<BN, AR, false, true>(ma, mb, p, st);
    return p.c.residual ? launch_kernel<BN, AR, true, false>(ma, mb, p, st) : launch_kernel<BN, AR, false, false>(ma, mb, p, st);
}
template <int AR>
cudaError_t launch_ar(const CUtensorMap& ma, const CUtensorMap& mb, const Params& p, int bn, cudaStream_t st) {
    if constexpr (AR == BM) {
        if (bn == 256) return launch_bn<256, AR>(ma, mb, p, st);
        if (bn == 192) return launch_bn<192, AR>(ma, mb, p, st);
    }
    return bn == 128 ? launch_bn<128, AR>(ma, mb, p, st) : launch_bn<64, AR>(ma, mb, p, st);
}

}  // namespace

bool dense_tensor_supported(const DenseCall& c) {
    return c.K % 8 == 0 && c.ldx % 8 == 0 && c.ldw % 8 == 0 && (reinterpret_cast<uintptr_t>(c.x) & 15) == 0 &&
           (reinterpret_cast<uintptr_t>(c.w) & 15) == 0 && (!c.pair_cols || c.N % 64 == 0);
}

cudaError_t launch_dense_tensor(const DenseCall& c, cudaStream_t st) {
    Params p{};
    p.c = c;
    p.status = device_status_ptr();
    if (!p.status) return cudaErrorUnknown;
    const int cols = c.pair_cols ? c.pair_cols : c.N;
    p.vec = (cols % 4 == 0) && (c.ldo % 4 == 0) && (reinterpret_cast<uintptr_t>(c.out_f32) & 15) == 0 &&
            (reinterpret_cast<uintptr_t>(c.out_b16) & 7) == 0 && (reinterpret_cast<uintptr_t>(c.residual) & 15) == 0;
    const long long tm = (c.M + BM - 1) / BM, kb = (c.K + BKE - 1) / BKE;
    const int a_rows = c.M < BM ? static_cast<int>(c.M) : BM;         // (more than 64)
    int bn = 64, split = 1;
    double best = 0.0;
    if (c.M <= 64) {
        // The chain of a CTA's K blocks (0.17 us and more each) against the weights' bytes at 6 TB/s, both felt where they are alike; plus storing the
        // tile or exchanging the sums of shares.  us, fitted to 23 shapes at 64 and 24 rows: within a tenth of the best choice on 19 of them.  Beyond two CTAs an SM the last
        // round counts whole.
        const double mem = 2.0 * c.N * c.K / 6.0e6;
        for (const int b : {128, 64}) {
            if (b > 64 && c.N <= b / 2) continue;
            const long long tiles = (c.N + b - 1) / b;
            for (int s = 1; s <= kMaxSplit; s *= 2) {
                const long long n = tiles * s;
                if (s > 1 && (kb < 4 * s || n > cluster_room<dense_tcgen05_kernel<128, 64, false, true>>(s, threads_for(64), smem_for(128, 64, false)))) break;
                // (up to 16 blocks of K the memory is better left to the kernel that comes next: 24 sequences at width 1024 397 and 378 us a step)
                const bool deep = n <= (s > 1 ? 128 : kNumSm) && (kb + s - 1) / s > 16;
                const long long waves = (n + 2 * kNumSm - 1) / (2 * kNumSm);
                const double chain = static_cast<double>(waves * ((kb + s - 1) / s)) * (deep ? (b == 128 ? 0.18 : 0.17) : (b == 128 ? 0.29 : 0.2));
                const double m = waves > 1 ? mem * (2.0 * kNumSm * waves) / n : mem;
                const double us = sqrt(chain * chain + m * m) + (s > 1 ? 1.2 + 0.025 * b / s : 0.02 * b);
                if (best == 0.0 || us < best) { best = us; bn = b; split = s; p.deep = deep; }
            }
        }
        // Blocks of K that the accumulators take at a time: eight, and no more than a warp of the row-streaming kernel has where that is the other choice.
        // us and error against 64 bits at 4, 8 and all blocks: 64 x 24576 gated x 4096 38.1, 37.8, 37.8; 64 x 12288 gated x 2048 16.1, 15.4, 14.9;
        // 64 x 6208 x 4096 15.0, 14.7, 14.5 and 2.4e-7, 4.7e-7, 2.1e-6; 64 x 10368 x 2048 13.2, 12.0, 11.3; 16 x 32000 x 4096 43.7, 43.6, 43.6 and 2.4e-7, 4.8e-7, 4.4e-6.
        const bool rows_too = c.M <= 16 || (c.M <= 32 && c.N <= 4096) || (c.M <= 48 && c.N <= 2048);
        p.part = rows_too ? static_cast<int>(std::min(8LL, std::max(2LL, kb / 8))) : 8;
    } else {
        // More than 64 rows: tile width and shares of K by the blocks of K that a CTA takes one after another (an SM takes in about 100 GB/s, and
        // 0.12 us pass all the same) against what it costs to exchange the sums of shared tiles; constants in us, fitted to
        // measurements.  Whole and shared: 512 x 2048 x 6144 33 and 19; 128 x 3072 x 3072 19 and 11; 900 x 2048 x 2048 15 and 19.  192 columns, whole tiles only,
        // where 256 leave much of a last wave empty and 128 take one more (us without and with: 900 x 10368 x 2048 41.3 and 38.4, 900 x 3072 x 3072 22.5 and 19.7,
        // 251 x 20736 x 4096 58.9 and 53.6, 512 x 5184 x 1024 11.6 and 10.0, 100 x 24576 gated x 4096 42.4 and 41.3).
        for (const int b : {256, 192, 128, 64}) {
            if (b > 64 && c.N <= b / 2) continue;
            const long long tiles = tm * ((c.N + b - 1) / b);
            for (int s = 1; s <= kMaxSplit; s *= 2) {
                if (s > 1 && (b == 192 || kb < 4 * s || tiles * s > cluster_room<dense_tcgen05_kernel<256, BM, false, true>>(s, threads_for(BM), smem_for(256, BM, true)))) break;
                const double blocks = static_cast<double>((tiles + kNumSm - 1) / kNumSm) * ((kb + s - 1) / s);
                const double us = blocks * (0.12 + 0.95e-3 * (a_rows + b)) + (s > 1 ? 1.7 + 3.9e-4 * a_rows * b / s : 0.0);
                if (best == 0.0 || us < best) { best = us; bn = b; split = s; }
            }
        }
    }
    p.split = split;
    const int ar = c.M <= 64 ? 64 : BM;
    p.tiles_m = static_cast<int>(tm);
    p.tiles_n = (c.N + bn - 1) / bn;
    CUtensorMap ma, mb;
    if (!make_map(&ma, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, c.x, c.M, c.K, BKE, ar, CU_TENSOR_MAP_SWIZZLE_128B, c.ldx))
        return cudaErrorUnknown;
    if (!make_map(&mb, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, c.w, c.N, c.K, BKE, bn, CU_TENSOR_MAP_SWIZZLE_128B, c.ldw)) return cudaErrorUnknown;
    return ar == 64 ? launch_ar<64>(ma, mb, p, bn, st) : launch_ar<BM>(ma, mb, p, bn, st);
}

}  // namespace stack
}  // namespace tbl
