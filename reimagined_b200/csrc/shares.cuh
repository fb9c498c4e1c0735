// The end of a linear layer whose K range is shared by the CTAs of a cluster: every CTA has its sums of a tile in shared
// memory, and each finishes a part of the rows -- adds the shares up in their order, then bias, residual or gated pair.
#pragma once

#include <atomic>

#include "stack.cuh"

namespace tbl {
namespace stack {

__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 peer_load(uint32_t addr, int rank) {
    uint32_t a;
    float4 v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t peer_load_u32(uint32_t addr, int rank) {
    uint32_t a, v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}

// `sums`: shared-memory address of this tile's sums, LDS floats per row, the same in every CTA of the cluster.  vec: outputs
// and residual take accesses of four columns.  check(m, weight row, sum) returns the sum to use.
template <int BN, int LDS, int THREADS, typename Check>
__device__ __forceinline__ void finish_shares(const DenseCall& c, uint32_t sums, int split, int share, int tn, int m0, int tile_rows, int vec, Check check) {
    const bool pair = c.pair_cols > 0;
    const int rows = min(tile_rows, c.M - m0), each = (rows + split - 1) / split;
    const int r0 = share * each, r1 = min(rows, r0 + each);
    const int groups = pair ? BN / 8 : BN / 4;             // of four output columns
    const int ncols = pair ? c.pair_cols : c.N;
    const Activation act = activation_of(c.act);
    auto total = [&](int r, int col) {
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (int k = 0; k < split; ++k) {
            const float4 a = peer_load(sums + 4 * (r * LDS + col), k);
            v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
        }
        return v;
    };
    for (int e = threadIdx.x; e < (r1 - r0) * groups; e += THREADS) {
        const int r = r0 + e / groups, gq = e % groups, m = m0 + r;
        const int col = pair ? gq / 8 * 64 + gq % 8 * 4 : 4 * gq;            // of the (first) weight row within the tile
        const int row_w = tn * BN + col, n = pair ? tn * (BN / 2) + 4 * gq : row_w;
        if (n >= ncols) continue;
        const float4 t = total(r, col);
        float v[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (n + j >= ncols) continue;
            v[j] = check(m, row_w + j, v[j]);
            if (c.bias) v[j] += __ldg(c.bias + row_w + j);
        }
        if (pair) {
            const float4 tu = total(r, col + 32);
            const float u[4] = {tu.x, tu.y, tu.z, tu.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (n + j >= ncols) continue;
                float up = check(m, row_w + 32 + j, u[j]);
                if (c.bias) up += __ldg(c.bias + row_w + 32 + j);
                v[j] = activate(act, v[j]) * up;
            }
        }
        const size_t o = static_cast<size_t>(m) * c.ldo + n;
        if (vec && c.out_f32) {
            if (c.residual) {
                const float4 res = *reinterpret_cast<const float4*>(c.residual + o);
                v[0] += res.x; v[1] += res.y; v[2] += res.z; v[3] += res.w;
            }
            *reinterpret_cast<float4*>(c.out_f32 + o) = make_float4(v[0], v[1], v[2], v[3]);
        } else if (vec) {
            *reinterpret_cast<uint2*>(c.out_b16 + o) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (n + j >= ncols) continue;
                if (c.out_f32) c.out_f32[o + j] = c.residual ? c.residual[o + j] + v[j] : v[j];
                else c.out_b16[o + j] = __float2bfloat16_rn(v[j]);
            }
        }
    }
}

// CTAs that run at the same time when they come in clusters of 2, 4 or 8 and take an SM each (a cluster lies within one group
// of SMs, so that some of these stay empty: 148, 132 and 120 on a B200 with 148 SMs).  One more and the launch takes twice as long.
// Asked once for every kernel, device and cluster size; a kernel has one number of threads and bytes.
template <auto Kernel>
int cluster_room(int cluster, int threads, size_t smem) {
    static std::atomic<int> known[64][4];
    int dev = 0;
    cudaGetDevice(&dev);
    const int at = cluster >= 8 ? 3 : (cluster >= 4 ? 2 : (cluster >= 2 ? 1 : 0));
    if (dev >= 0 && dev < 64)
        if (const int n = known[dev][at].load(std::memory_order_relaxed)) return n;
    static bool done[64] = {};
    if (allow_smem(Kernel, smem, done) != cudaSuccess) return 0;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(cluster * kNumSm); cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, Kernel, &cfg) != cudaSuccess) { cudaGetLastError(); return 0; }
    if (dev >= 0 && dev < 64) known[dev][at].store(n * cluster, std::memory_order_relaxed);
    return n * cluster;
}

// Launch as a programmatic dependent whose CTAs come in clusters of `cluster` along x.
template <typename... Params, typename... Args>
cudaError_t launch_dependent_cluster(void (*kernel)(Params...), dim3 grid, int cluster, dim3 block, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
    note_launch();
    return e;
}

}  // namespace stack
}  // namespace tbl
