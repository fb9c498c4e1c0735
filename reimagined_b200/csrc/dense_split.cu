// y[M,N] = x[M,K] (fp32) x w[N,K]^T (bf16) at fp32 accuracy on the 5th-generation tensor cores.
//
// An fp32 number down to 2^-110 is the exact sum of three bf16 numbers (24 bits of significand, cut after 8 and 16), the weights
// are bf16 already and products of two bf16 are exact in fp32: three MMAs per step of K give every product exactly.  What remains is
// the accumulation, and there the tensor cores cut off what an addend or the sum loses in alignment, always towards zero.
// So no accumulator runs for long: the high parts have one of their own, both are taken over into registers after every
// kSlab blocks of K, where the sums are ordinary rounded fp32 additions.
//
// One CTA per tile of 128 rows x BN columns and share of K (the shares of a tile are a cluster, so that short matrices fill
// the GPU too), nineteen warps: TMA producers of the weights and of x, MMA issuer, eight warps that add up, eight that cut
// rows of x up and store the three pieces as 128-byte-swizzled operand rows.  (x comes by TMA too: the fence behind the
// stores waits for all loads its warp has under way, so that loads ahead of their time would be waited for at once.)  At the end the sums of all shares meet in shared
// memory (distributed, in the order of the shares) and all warps finish the rows: bias, residual, gated pair.
// A sum that is not finite is worked out once more the plain way, since infinities have no such pieces, and so is a small one of
// rows some number of which lost bits below bf16's smallest.
// 251 x 6144 x 2048: 58 us (0.33 PFLOP/s of bf16 MMAs), one of them for watching the lost bits; the SIMT kernel 700 us; relative
// error 1.5e-7, the SIMT kernel's 1.4e-6.  What bounds it is the round of a block through the cutting warps, their fence and the MMAs with two places for
// the pieces: 1.2 us a block of 64, where the MMAs alone take 0.3.
// Every wait is bounded: on a timeout the role records the status word and falls through to the common exit.
#include <cuda.h>

#include "shares.cuh"
#include "stack.cuh"
#include "tc05.cuh"

namespace tbl {
namespace stack {
namespace {

using namespace tc05;

constexpr int BM = 128;
constexpr int BKE = 64;             // elements of K per block: 128 bytes of each operand row
constexpr int kA = 2, kB = 4;       // blocks of operand A (three pieces) and B in shared memory
constexpr int kSlab = 2;            // blocks per accumulation in tensor memory
constexpr int kSumWarps = 8, kCutWarps = 8;
constexpr int kThreads = 32 * (3 + kSumWarps + kCutWarps);
constexpr int kPieceBytes = BM * 128;
constexpr int kXBytes = BM * BKE * 4;                      // a block of x on its way
constexpr int kMaxSplit = 8;

__host__ __device__ constexpr int x_blocks(int bn) { return bn == 128 ? 2 : 3; }
__host__ __device__ constexpr int operands(int bn) { return kA * 3 * kPieceBytes + kB * bn * 128; }
__host__ __device__ constexpr size_t smem_for(int bn) { return 1024 + operands(bn) + static_cast<size_t>(x_blocks(bn)) * kXBytes + 256; }

struct Params {
    DenseCall c;
    int split;               // shares of K = CTAs of a cluster
    int tma_x, vec_out;      // rows of x start on 16 bytes / outputs take 16-byte accesses
    int* status;
};

// high halves of two words: the bf16 numbers nearest to them towards zero, packed
__device__ __forceinline__ uint32_t high_halves(float lo, float hi) { return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632); }
__device__ __forceinline__ float beyond_bf16(float v) { return v - __uint_as_float(__float_as_uint(v) & 0xffff0000u); }

// Bits that the pieces of a row lost are worth less than K * 2^-133 * |w|: nothing beside a sum from here on, for weights up to 2^50.
constexpr float kSmallSum = 9.094947e-13f;                 // 2^-40

// lost: address of the flag of these rows, one per share of K
__device__ __noinline__ float rechecked(const DenseCall& c, int m, int n, float sum, uint32_t lost, int split) {
    if (fabsf(sum) < kSmallSum) {
        uint32_t any = 0;
        for (int k = 0; k < split; ++k) any |= peer_load_u32(lost, k);
        if (!any) return sum;
    }
    const float* x = static_cast<const float*>(c.x) + static_cast<size_t>(m) * c.ldx;
    const bf16* w = c.w + static_cast<size_t>(n) * c.ldw;
    float v = 0.0f;
    for (int k = 0; k < c.K; ++k) v = fmaf(x[k], to_f(w[k]), v);
    return v;
}

template <int BN>
__global__ void __launch_bounds__(kThreads, 1) dense_split_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_b, const __grid_constant__ Params p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr int X = x_blocks(BN);
    constexpr uint32_t kTmemCols = 4 * BN;                 // two buffers of two accumulators
    constexpr int LDS = BN + 4;                            // floats per row of the sums in shared memory
    constexpr int COLS = BN / 2;                           // columns per summing warp
    static_assert(sizeof(float) * BM * LDS <= kA * 3 * kPieceBytes, "the sums take the pieces' place");
    uint8_t *smem_b = smem + kA * 3 * kPieceBytes, *smem_x = smem + operands(BN);
    uint64_t* full_a = reinterpret_cast<uint64_t*>(smem_x + X * kXBytes);
    uint64_t *empty_a = full_a + kA, *full_b = empty_a + kA, *empty_b = full_b + kB, *full_x = empty_b + kB, *empty_x = full_x + X,
             *tmem_full = empty_x + X, *tmem_empty = tmem_full + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2), *lost_rows = tmem_slot + 1;     // [cutting warps]
    const DenseCall& c = p.c;
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int share = blockIdx.x % p.split, tn = blockIdx.x / p.split, m0 = blockIdx.y * BM;
    const int kblocks = (c.K + BKE - 1) / BKE, per = (kblocks + p.split - 1) / p.split;
    const int kb0 = min(kblocks, share * per), count = min(kblocks, kb0 + per) - kb0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kA; ++s) { mbar_init(&full_a[s], kCutWarps); mbar_init(&empty_a[s], 1); }
        for (int s = 0; s < kB; ++s) { mbar_init(&full_b[s], 1); mbar_init(&empty_b[s], 1); }
        for (int s = 0; s < X; ++s) { mbar_init(&full_x[s], 1); mbar_init(&empty_x[s], kCutWarps); }
        for (int b = 0; b < 2; ++b) { mbar_init(&tmem_full[b], 1); mbar_init(&tmem_empty[b], kSumWarps); }
        fence_mbar_init();
        fence_proxy_async();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();

    // The limit of a bounded wait is meant for this kernel's own pipeline, so nobody waits for a barrier while the kernel before
    // still runs: only the weights' producer goes ahead, by the places of its ring.
    if (warp != 0) pdl_wait();
    // TMA producer: `count` blocks through a ring of n places of `bytes` each
    auto produce = [&](const CUtensorMap* map, uint8_t* ring, int n, int bytes, int row, uint64_t* full, uint64_t* empty) {
        int i = 0;
        bool alive = true;
        for (; i < count; ++i) {
            const int s = i % n;
            if (i == n) pdl_wait();
            if (i >= n) alive = mbar_wait_bounded(&empty[s], ((i / n) - 1) & 1, p.status);
            if (!alive) break;
            mbar_arrive_expect_tx(&full[s], bytes);
            tma_load_2d(ring + s * bytes, map, (kb0 + i) * BKE, row, &full[s]);
        }
        if (!alive)                                        // nobody else may be waiting for the copies in flight
            for (int j = max(0, i - n); j < i; ++j) mbar_wait_bounded(&full[j % n], (j / n) & 1, p.status);
    };
    if (warp == 0) {
        // the weights depend on no kernel before this one, unless the call says so
        pdl_wait_for_weights(c.w_computed);
        if (lane == 0) produce(&map_b, smem_b, kB, BN * 128, tn * BN, full_b, empty_b);
        __syncwarp();
    } else if (warp == 2 + kSumWarps + kCutWarps) {
        if (lane == 0 && p.tma_x) produce(&map_x, smem_x, X, kXBytes, m0, full_x, empty_x);
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        const uint32_t idesc = idesc_bf16(BN);
        bool alive = true;
        for (int i = 0; i < count; ++i) {
            const int sa = i % kA, sb = i % kB, slab = i / kSlab, in_slab = i - slab * kSlab, buf = slab & 1;
            if (in_slab == 0 && slab >= 2) alive = mbar_wait_bounded(&tmem_empty[buf], ((slab >> 1) - 1) & 1, p.status);
            if (alive) alive = mbar_wait_bounded(&full_b[sb], (i / kB) & 1, p.status);
            if (alive) alive = mbar_wait_bounded(&full_a[sa], (i / kA) & 1, p.status);
            alive = __all_sync(0xffffffffu, alive);
            if (!alive) break;
            tc_fence_after();
            if (elect_one()) {
                const uint32_t a = smem_u32(smem + sa * 3 * kPieceBytes), b = smem_u32(smem_b + sb * BN * 128);
                const uint32_t high = tmem_base + buf * 2 * BN, low = high + BN;
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    const uint64_t bd = smem_desc_sw128(b + kk * 32);
                    const uint32_t on = (in_slab | kk) != 0 ? 1u : 0u;
                    umma_f16(high, smem_desc_sw128(a + kk * 32), bd, idesc, on);
                    umma_f16(low, smem_desc_sw128(a + kPieceBytes + kk * 32), bd, idesc, on);
                    umma_f16(low, smem_desc_sw128(a + 2 * kPieceBytes + kk * 32), bd, idesc, 1u);
                }
                umma_commit(&empty_a[sa]);
                umma_commit(&empty_b[sb]);
                if (in_slab == kSlab - 1 || i == count - 1) umma_commit(&tmem_full[buf]);
            }
            __syncwarp();
        }
    } else if (warp < 2 + kSumWarps) {
        // ---------------- sums ----------------
        const int quarter = warp & 3, half = (warp - 2) >> 2;      // TMEM lanes and columns of this warp
        float acc[COLS];
#pragma unroll
        for (int j = 0; j < COLS; ++j) acc[j] = 0.0f;
        const int slabs = (count + kSlab - 1) / kSlab;
        bool alive = true;
        for (int slab = 0; slab < slabs; ++slab) {
            const int buf = slab & 1;
            alive = mbar_wait_bounded(&tmem_full[buf], (slab >> 1) & 1, p.status);
            alive = __all_sync(0xffffffffu, alive);
            if (!alive) break;
            tc_fence_after();
            const uint32_t at = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + buf * 2 * BN + half * COLS;
#pragma unroll
            for (int j = 0; j < COLS; j += 8) {
                uint32_t h[8], l[8];
                tmem_ld8(at + j, h);
                tmem_ld8(at + BN + j, l);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[j + e] += __uint_as_float(h[e]) + __uint_as_float(l[e]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&tmem_empty[buf]);
        }
        // the last slab's MMAs are done, so nothing reads or writes the pieces any more
        if (alive) {
            float* row = reinterpret_cast<float*>(smem) + (quarter * 32 + lane) * LDS + half * COLS;
#pragma unroll
            for (int j = 0; j < COLS; j += 4) *reinterpret_cast<float4*>(row + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
        }
    } else {
        // ---------------- rows of x, cut into three pieces: sixteen lanes a row, four elements each ----------------
        const int w = warp - 2 - kSumWarps, q = lane & 15;
        const float* x = static_cast<const float*>(c.x);
        uint32_t lost = 0;                                             // low halves of third pieces: bits that those do not hold
        for (int i = 0; i < count; ++i) {
            const int s = i % kA, sx = i % X;
            bool alive = i < kA || mbar_wait_bounded(&empty_a[s], ((i / kA) - 1) & 1, p.status);
            if (alive && p.tma_x) alive = mbar_wait_bounded(&full_x[sx], (i / X) & 1, p.status);
            if (!__all_sync(0xffffffffu, alive)) break;
            float4 v[8];
            const bool live = m0 + w * 16 < c.M || i < kA;             // (rows past the end stay zero)
            if (live) {
                uint8_t* dst = smem + s * 3 * kPieceBytes;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int r = w * 16 + 2 * j + (lane >> 4), k = (kb0 + i) * BKE + 4 * q;
                    if (p.tma_x) {
                        v[j] = *reinterpret_cast<const float4*>(smem_x + sx * kXBytes + r * 256 + q * 16);
                    } else {
                        v[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        if (m0 + r < c.M && k < c.K) {                 // K is a multiple of 8
                            const float* src = x + static_cast<size_t>(m0 + r) * c.ldx + k;
                            v[j] = make_float4(src[0], src[1], src[2], src[3]);
                        }
                    }
                }
#pragma unroll
                for (int piece = 0; piece < 3; ++piece)
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int r = w * 16 + 2 * j + (lane >> 4);
                        *reinterpret_cast<uint2*>(dst + piece * kPieceBytes + r * 128 + (((q >> 1) ^ (r & 7)) << 4) + (q & 1) * 8) =
                            make_uint2(high_halves(v[j].x, v[j].y), high_halves(v[j].z, v[j].w));
                        if (piece == 2)
                            lost |= __float_as_uint(v[j].x) | __float_as_uint(v[j].y) | __float_as_uint(v[j].z) | __float_as_uint(v[j].w);
                        else
                            v[j] = make_float4(beyond_bf16(v[j].x), beyond_bf16(v[j].y), beyond_bf16(v[j].z), beyond_bf16(v[j].w));
                    }
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&full_a[s]);
                if (p.tma_x) mbar_arrive(&empty_x[sx]);
            }
        }
        lost = __any_sync(0xffffffffu, (lost & 0xffff) != 0);
        if (lane == 0) lost_rows[w] = lost;
    }

    // ---------------- all shares' sums, a part of the rows per CTA ----------------
    pdl_wait();
    if (p.split > 1) cluster_sync_all(); else __syncthreads();
    const uint32_t lost_at = smem_u32(lost_rows);
    finish_shares<BN, LDS, kThreads>(c, smem_u32(smem), p.split, share, tn, m0, BM, p.vec_out, [&](int m, int n, float v) {
        const float size = fabsf(v);
        return (size >= kSmallSum && size <= 3.402823466e38f) || n >= c.N ? v : rechecked(c, m, n, v, lost_at + 4 * ((m - m0) >> 4), p.split);
    });
    // nobody leaves while a neighbour may still read its sums; then the allocating warp releases TMEM
    tc_fence_before();
    if (p.split > 1) cluster_sync_all(); else __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
}

template <int BN>
cudaError_t launch_bn(Params p, cudaStream_t st) {
    static bool done[64] = {};
    static_assert(smem_for(BN) <= 227 * 1024, "shared memory of a CTA");
    cudaError_t e = allow_smem(dense_split_kernel<BN>, smem_for(BN), done);
    if (e != cudaSuccess) return e;
    const DenseCall& c = p.c;
    CUtensorMap mx{}, mb;
    if (p.tma_x && !make_map(&mx, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, c.x, c.M, c.K, BKE, BM, CU_TENSOR_MAP_SWIZZLE_NONE, c.ldx)) return cudaErrorUnknown;
    if (!make_map(&mb, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, c.w, c.N, c.K, BKE, BN, CU_TENSOR_MAP_SWIZZLE_128B, c.ldw)) return cudaErrorUnknown;
    const int tiles_m = ceil_div(c.M, BM), tiles_n = ceil_div(c.N, BN), kblocks = ceil_div(c.K, BKE);
    // shares of K until the SMs are taken, of at least four blocks each
    p.split = 1;
    while (p.split < kMaxSplit && kblocks >= 8 * p.split &&
           2LL * p.split * tiles_m * tiles_n <= cluster_room<dense_split_kernel<BN>>(2 * p.split, kThreads, smem_for(BN)))
        p.split *= 2;
    return launch_dependent_cluster(dense_split_kernel<BN>, dim3(tiles_n * p.split, tiles_m), p.split, dim3(kThreads), smem_for(BN), st, mx, mb, p);
}

}  // namespace

bool dense_split_supported(const DenseCall& c) {
    return c.K % 8 == 0 && c.ldw % 8 == 0 && (reinterpret_cast<uintptr_t>(c.w) & 15) == 0 && (!c.pair_cols || c.N % 64 == 0) &&
           c.out_f32 && c.batch == 0 && !c.gate && ceil_div(c.M, BM) <= 65535;
}

cudaError_t launch_dense_split(const DenseCall& c, cudaStream_t st) {
    Params p{};
    p.c = c;
    p.status = device_status_ptr();
    if (!p.status) return cudaErrorUnknown;
    const int cols = c.pair_cols ? c.pair_cols : c.N;
    p.tma_x = c.ldx % 4 == 0 && (reinterpret_cast<uintptr_t>(c.x) & 15) == 0;
    p.vec_out = cols % 4 == 0 && c.ldo % 4 == 0 && (reinterpret_cast<uintptr_t>(c.out_f32) & 15) == 0 && (reinterpret_cast<uintptr_t>(c.residual) & 15) == 0;
    // the wider tile where it fills the SMs too: it cuts up every row of x half as often
    const bool wide = static_cast<long long>(ceil_div(c.M, BM)) * ceil_div(c.N, 128) >= 100;
    return wide ? launch_bn<128>(p, st) : launch_bn<64>(p, st);
}

}  // namespace stack
}  // namespace tbl
