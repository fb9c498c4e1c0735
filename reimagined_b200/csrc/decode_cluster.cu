// The blocks of a decode step in one launch.
//
// A step of the hybrid is a chain: every projection needs the whole row its predecessor made, and at 24 MB of packed weights (which stay in L2)
// neither bytes nor operations bound it, only the hand-over from one operator to the next.  As separate launches a hand-over costs 5.3 us
// (D768, 61 launches, 323 us a token).  Here a thread-block cluster of 16 or 8 CTAs takes a few sequences through all the blocks on
// its own: a projection's rows are spread over the CTAs, and a row that the next projection reads as a whole is gathered into every CTA's
// shared memory by st.async, which counts its bytes on the receiver's mbarrier -- no launch, no trip through L2, no grid-wide barrier.
// Clusters share nothing but the weights, so a batch is as many clusters as it needs.  D768, 16 blocks, us a step with the head, separate launches and
// this: batch 1 318 and 173, 8 417 and 248, 16 408 and 263, 32 530 and 361, 64 649 and 494 (64 cached tokens); 1 338 and 188, 64 819 and 745 (900).
// The results are the same bit for bit, but for the attention over more than 256 cached tokens, whose dot products and sums of values are taken in another order.
//
// Passes of a block (the row each of them reads is normed and quantised by every CTA for itself, with the arithmetic of the kernels
// in decode.cu and gemv_strip.cu):
//   A  x, z, B, C, dt [q, k, v] of the CTA's own channels and heads; conv step, SSD step, gate [attention] -> gather
//   B  out [and attention out] -> residual stream, gather
//   C  FFN up, squared ReLU -> gather          (hybrid blocks)
//   D  FFN down -> residual stream, gather     (hybrid blocks)
// B and C (16 rows each) are made by every CTA, the step sizes by every CTA that owns one of a head's channels.
//
// What bounds it now is the chain of dependent instructions of a pass, 3 to 4 us of them at batch 1: norm and quantise 1.2 (the sum in the order of the
// other route, three barriers, four correctly rounded divisions and roots), products 0.7 to 1.3 (int8 MMAs of a warp follow each other at 40 cycles),
// convolution and step size 0.5, SSD step 0.5, the gather 0.5.
#include "decode_cluster.cuh"

#include <cmath>
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"

namespace tbl {
namespace {

// Threads of a CTA.  One sequence a cluster runs as straight code, held up by chains of dependent instructions: 256 threads with 255 registers as fast as
// 512 with 128.  More sequences: 512 threads spill (batch 64 593 us a step), 256 leave too few warps (665), 320 549, 384 513, 448 582.
constexpr int kOneThreads = 256, kRowsThreads = 384;
constexpr int kMaxWarps = 16;
constexpr int kDepth = 4;            // weight blocks a warp holds ahead: a piece of a strip
constexpr int kMaxRows = 8;          // sequences of a cluster: the columns of an MMA
constexpr int kMaxParts = 64;        // parts of a row's sum of squares
constexpr int kMaxBlocks = 32;       // blocks of a launch (kernel parameters)
constexpr int kTaps = 3;             // tokens before this one that the convolution sees
constexpr int kJobs = 8;             // projections of a pass
constexpr int kStripParts = 8;       // parts of a row's sum in the order kSumStrips

struct Linear {
    const uint8_t* strips;
    const float* magnitude;
    const float* bias;
    float scale;
    int pad;
};
enum { kX, kZ, kB, kC, kDt, kOut, kQ, kKv, kAttnOut, kUp, kDown, kLinears };
enum { kPassA, kPassB, kPassC, kPassD, kPasses };

// what differs from block to block
struct Block {
    Linear lin[kLinears];
    const float *core_norm_w, *A_log, *D, *conv_w, *conv_b, *norm_w, *attn_norm_w, *ff_norm_w, *mamba_gate, *attn_gate, *ffn_gate, *rope_cos, *rope_sin;
    float *ring, *ssm, *k_cache, *v_cache;
    float core_eps, norm_eps;
    int hybrid, window, rope_positions, pad;
};
static_assert(sizeof(Block) % 16 == 0 && sizeof(Block) <= 64 * 16, "copied by a warp, two 16-byte pieces a lane");

// what all blocks share
struct Dims {
    int D, inner, n_heads, d_head, ff, a_heads, a_kv_heads, head_dim;
};

// byte offsets into dynamic shared memory
struct Layout {
    int x0, x1, codes, acc, xs, zs, bc, bcring, decay, skip, heads_of, norm, scores, partial, qkv, table, total;
    int acc_stride;          // ints between two sequences' accumulators
    int score_len;
    int pieces;              // room in the table
    int partial_all;         // room for all of attention_decode_kernel's partial sums
    int state, taps;         // sequences' states and windows, brought in ahead (-1: not)
};

// What a CTA of a cluster owns: channels (rows of x and z), the heads they belong to, attention heads and their key/value heads, rows of the residual stream and of the FFN's hidden layer.
struct Range { uint16_t lo, hi; };
__host__ __device__ __forceinline__ int size_of(const Range& r) { return r.hi - r.lo; }
struct Owned { Range chan, head, attn, kv, row, ff; };

struct Params {
    Dims d;
    Owned own[16];
    int batch, rows, n_blocks, capacity, vocab, advance;
    int row_order, gate_order, gate_share;       // SumOrder of the residual stream's norms and of the gated one
    const int32_t* ids;
    const float* embedding;
    const float* hidden_in;
    float* hidden_out;
    float* trace;
    int32_t* positions;
    int* status;
    Layout L;
    Block blk[kMaxBlocks];
};

// A projection's share of a pass: `cnt` strips from `lo` of a matrix of `total` strips of `nblk` weight blocks
struct Job {
    int total, lo, nblk, slabs, begin, end;      // slabs: pieces a strip is cut into; begin, end: among the pass's pieces
    int cut;                 // blocks of a piece (the last ones of a slab may be fewer)
    int codes;               // byte offset of its input codes
    int acc;                 // column of its first row among the accumulators
    int lin;
};

struct Static {
    Block blk[2];
    Job job[kPasses][kJobs];
    int first[kPasses];      // where a pass's pieces begin in the table of them
    int count[2][kPasses];   // how many it has, in a plain and in a hybrid block
    uint64_t bar[2];
    alignas(16) float red[kMaxRows * kMaxParts];      // sums of squares by row and part
    float inv[kMaxRows];     // the norms' factors
    uint32_t span[kMaxParts];        // of the gated norm's parts
    alignas(16) float redm[kMaxWarps];
    int dead;                // a wait ran out
    float act_scale[2][kMaxRows];
    int q_sum[2][2][kMaxRows];           // [pass & 1]: as the accumulators
    int pos[kMaxRows];
};

__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
    uint32_t d;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(addr), "r"(rank));
    return d;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ uint4 load_weights(const uint8_t* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ void mma_u8s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// x sigmoid(x); for the convolution and for the gate (both branches of decode.cu's silu_stable are this)
__device__ __forceinline__ float silu(float g) {
    const float e = expf(-fabsf(g));
    return __fmul_rn(g, __fdiv_rn(g >= 0.0f ? 1.0f : e, __fadd_rn(1.0f, e)));
}

// one copy of the code for its three uses
__device__ __noinline__ double exp64(double x) { return exp(x); }

// This CTA's share of every pass, by one warp: lane 8 p + j takes projection j of pass p.
template <int T>
__device__ __forceinline__ void plan_jobs(const Params& P, Static& S, int rank, int R) {
    const Dims& d = P.d;
    const int lane = threadIdx.x & 31, pass = lane >> 3, j = lane & 7, D = d.D;
    int lin = -1, lo = 0, hi = 0, K = D, N = 0, codes = 0;
    const Owned& o = P.own[rank];
    if (pass == kPassA) {
        const int per = d.head_dim >> 4;
        if (j <= 1) { lin = j == 0 ? kX : kZ; lo = o.chan.lo >> 4; hi = o.chan.hi >> 4; N = d.inner; }
        if (j == 2 || j == 3) { lin = j == 2 ? kB : kC; hi = 1; N = 16; }
        if (j == 4) { lin = kDt; lo = o.head.lo >> 4; hi = (o.head.hi + 15) >> 4; N = d.n_heads; }
        if (j >= 5) codes = R * D;
        if (j == 5) { lin = kQ; lo = o.attn.lo * per; hi = o.attn.hi * per; N = d.a_heads * d.head_dim; }
        if (j >= 6) { lin = kKv; N = 2 * d.a_kv_heads * d.head_dim; lo = ((j - 6) * d.a_kv_heads + o.kv.lo) * per; hi = ((j - 6) * d.a_kv_heads + o.kv.hi) * per; }
    } else if (pass == kPassB && j < 2) {
        lin = j == 0 ? kOut : kAttnOut; N = D; lo = o.row.lo >> 4; hi = o.row.hi >> 4;
        if (j == 0) K = d.inner; else codes = R * d.inner;
        if (j == 1 && d.a_heads == 0) hi = lo;
    } else if (pass >= kPassC && j == 0 && d.ff) {
        const Range r = pass == kPassC ? o.ff : o.row;
        lin = pass == kPassC ? kUp : kDown; N = pass == kPassC ? d.ff : D; lo = r.lo >> 4; hi = r.hi >> 4;
        if (pass == kPassD) K = d.ff;
    }
    // Pieces of up to `cut` blocks, within a slab of four: as short as leaves every warp one piece (or one after the other where there are more).
    const int cnt = lin < 0 ? 0 : hi - lo, nblk = K >> 8;
    int cut = 0, slabs = 0, pieces = 0;
    const int plain = pass == kPassA ? 4 : (pass == kPassB ? 0 : kJobs - 1);        // last projection of a block without attention
#pragma unroll
    for (int c = 1; c <= kDepth; ++c) {
        const int per_strip = (nblk >> 2) * ((4 + c - 1) / c) + ((nblk & 3) + c - 1) / c;
        int all = cnt * per_strip;
#pragma unroll
        for (int k = 1; k < kJobs; k <<= 1) all += __shfl_xor_sync(0xffffffffu, all, k, kJobs);
        if (cut == 0 && (all <= T / 32 || c == kDepth)) { cut = c; slabs = per_strip; pieces = cnt * per_strip; }
    }
    int cols = cnt * 16, end = pieces;
#pragma unroll
    for (int k = 1; k < kJobs; k <<= 1) {
        const int pp = __shfl_up_sync(0xffffffffu, end, k, kJobs), pc = __shfl_up_sync(0xffffffffu, cols, k, kJobs);
        if (j >= k) { end += pp; cols += pc; }
    }
    S.job[pass][j] = Job{(N + 15) >> 4, lo, nblk, slabs, end - pieces, end, cut, codes, cols - cnt * 16, max(lin, 0)};
    if (j == plain) S.count[0][pass] = end;
    if (j == kJobs - 1) S.count[1][pass] = end;
    __syncwarp();
    if (lane == 0) {
        int at = 0;
        for (int p = 0; p < kPasses; ++p) { S.first[p] = at; at += S.count[1][p]; }
    }
}

// The table of pieces: x = index of the first weight block in its matrix (the slab-major order of gemv_strip.cu) | projection << 24,
// y = input codes / 256 << 16 | accumulator column / 16 << 3 | blocks.  The same for every block of the model.
template <int T>
__device__ __forceinline__ void plan_pieces(const Static& S, uint2* table, int R) {
    const int count = S.first[kPassD] + S.count[1][kPassD];
    for (int i = threadIdx.x; i < count; i += T) {
        int p = 0, k = 0;
        while (p < kPassD && S.first[p + 1] <= i) ++p;
        const int j = i - S.first[p];
        while (S.job[p][k].end <= j) ++k;
        const Job& job = S.job[p][k];
        const uint32_t rel = j - job.begin, strip = rel / static_cast<uint32_t>(job.slabs), piece = rel - strip * job.slabs;
        const uint32_t per_slab = (4 + job.cut - 1) / static_cast<uint32_t>(job.cut), slab = piece / per_slab, at = (piece - slab * per_slab) * job.cut;
        const int bs = min(4, job.nblk - 4 * static_cast<int>(slab));        // a slab: four blocks of K of every strip, the last one what is left
        const uint32_t index = 4 * slab * job.total + (job.lo + strip) * bs + at, codes = (job.codes >> 8) + (4 * slab + at) * R;
        table[i] = make_uint2(index | static_cast<uint32_t>(job.lin) << 24, codes << 16 | ((job.acc >> 4) + strip) << 3 | min(job.cut, bs - static_cast<int>(at)));
    }
}

// A warp's piece of a pass, requested ahead
struct Stream {
    uint4 lo[kDepth], hi[kDepth];
    uint32_t y;              // of the table
};

__device__ __forceinline__ const uint8_t* piece_address(const Block& b, const uint2& d) {
    return b.lin[d.x >> 24].strips + (static_cast<size_t>(d.x & 0xffffffu) << 10) + (threadIdx.x & 31) * 16;
}
__device__ __forceinline__ void request(const Block& b, const uint2* table, int count, int piece, Stream& s) {
    s.y = 0;
    if (piece >= count) return;
    const uint2 d = table[piece];
    s.y = d.y;
    const uint8_t* p = piece_address(b, d);
    const int n = d.y & 7;
#pragma unroll
    for (int i = 0; i < kDepth; ++i) {
        if (i < n) {
            s.lo[i] = load_weights(p + i * 1024);
            s.hi[i] = load_weights(p + i * 1024 + 512);
        }
    }
}

// The warp's pieces (every (T / 32)-th of the pass) against the codes: sums into acc[row][column].
template <bool ONE, int T>
__device__ __forceinline__ void multiply(const Block& b, const uint2* table, int count, Stream& s, uint32_t codes, int* acc, int acc_stride, int R) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    // one row: all eight columns of the MMA are that row (its codes are read once)
    const uint32_t a0 = codes + (ONE ? t * 16 : g * 256 + t * 16), flip = ONE ? 0 : (g & 1) << 6;
#pragma unroll 1
    for (int piece = warp; piece < count; piece += (T / 32)) {
        const uint32_t y = s.y;
        const int n = y & 7;
        uint32_t ablk = a0 + (y >> 16 << 8);
        // the next piece's blocks take the place of this one's as they are used
        const uint2 d = piece + T / 32 < count ? table[piece + T / 32] : make_uint2(0, 0);
        const uint8_t* next = piece_address(b, d);
        const int n_next = d.y & 7;
        s.y = d.y;
        int sum[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) sum[j][0] = sum[j][1] = sum[j][2] = sum[j][3] = 0;
#pragma unroll
        for (int i = 0; i < kDepth; ++i) {
            if (i < n) {
                const uint32_t lw[4] = {s.lo[i].x, s.lo[i].y, s.lo[i].z, s.lo[i].w}, hw[4] = {s.hi[i].x, s.hi[i].y, s.hi[i].z, s.hi[i].w};
#pragma unroll
                for (int xp = 0; xp < 2; ++xp) {
                    const uint4 b0 = lds128(ablk + ((128 * xp) ^ flip)), b1 = lds128(ablk + ((128 * xp + 64) ^ flip));
                    const uint32_t u0[4] = {b0.x, b0.y, b0.z, b0.w}, u1[4] = {b1.x, b1.y, b1.z, b1.w};
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        const uint32_t mk = 0x03030303u << (2 * p);
                        mma_u8s8(sum[p], lw[2 * xp] & mk, hw[2 * xp] & mk, lw[2 * xp + 1] & mk, hw[2 * xp + 1] & mk, u0[p], u1[p]);
                    }
                }
                ablk += ONE ? 256 : R * 256;
            }
            if (i < n_next) {
                s.lo[i] = load_weights(next + i * 1024);
                s.hi[i] = load_weights(next + i * 1024 + 512);
            }
        }
        // plane p holds 4^p times its sum
        int* at = acc + (y & 0xfff8u) * 2 + g;
        if constexpr (ONE) {
            if (t == 0) {
                atomicAdd(at, sum[0][0] + (sum[1][0] >> 2) + (sum[2][0] >> 4) + (sum[3][0] >> 6));
                atomicAdd(at + 8, sum[0][2] + (sum[1][2] >> 2) + (sum[2][2] >> 4) + (sum[3][2] >> 6));
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int m = 2 * t + (e & 1);
                if (m < R) atomicAdd(at + m * acc_stride + 4 * (e & 2), sum[0][e] + (sum[1][e] >> 2) + (sum[2][e] >> 4) + (sum[3][e] >> 6));
            }
        }
    }
}

// A row's sum of squares is taken in the very order of the kernel that takes it where the step is made of separate launches: 107 layers that round their
// input to 8 bits would carry another last place into other codes, and a hundred tokens on into other logits.  A part is one of that kernel's warps.
enum SumOrder {
    kSumStrips,      // gemv_strip_kernel's prologue: a thread takes 16 numbers, the batch's rows one after the other over its 512 threads
    kSumStrided,     // residual_norm_kernel, mamba_mix_kernel: thread t of 512 takes numbers t, t + 512, ...
    kSumClusters,    // mamba_mix_cluster_kernel: eight CTAs, `share` numbers each, one a thread
};
struct Sums { int order, share, row0; };      // row0: of the batch, the cluster's first
// The most of that kernel's warps (32 threads of 16 numbers) that a row of K numbers lies in
__host__ __device__ __forceinline__ int sum_strips_parts(int K) { return (K >> 9) + 2; }

// The sums over the lanes of eight numbers a lane, each added up like a butterfly (lanes 16, 8, 4, 2, 1 apart), in nine exchanges: at each of the first
// three steps a lane keeps half of its numbers and sends the others.  Lane l has number l / 4 in the end.
__device__ __forceinline__ float butterfly8(const float (&v)[8], int lane) {
    float a[4], b[2];
    const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] = __fadd_rn(h16 ? v[k + 4] : v[k], __shfl_xor_sync(0xffffffffu, h16 ? v[k] : v[k + 4], 16));
#pragma unroll
    for (int k = 0; k < 2; ++k) b[k] = __fadd_rn(h8 ? a[k + 2] : a[k], __shfl_xor_sync(0xffffffffu, h8 ? a[k] : a[k + 2], 8));
    float c = __fadd_rn(h4 ? b[1] : b[0], __shfl_xor_sync(0xffffffffu, h4 ? b[0] : b[1], 4));
    c = __fadd_rn(c, __shfl_xor_sync(0xffffffffu, c, 2));
    return __fadd_rn(c, __shfl_xor_sync(0xffffffffu, c, 1));
}
// The parts of rows src [R][K], into part [row][kMaxParts].  span (kSumClusters): a part's place there | its numbers << 8 | its first number << 16.
template <bool ONE, int T>
__device__ __forceinline__ void sum_parts(const Sums& o, const float* src, int K, int R, const uint32_t* span, float* part) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (o.order == kSumStrips) {
        // its warps in order: of a row that goes on at the first warp, the parts there come first
        static_assert(kStripParts == 8, "sum_total() adds eight");
        const int n = sum_strips_parts(K);
#pragma unroll 1
        for (int i = warp; i < R * kStripParts; i += T / 32) {
            const int r = ONE ? 0 : i / kStripParts, p = i % kStripParts;
            const int g0 = (o.row0 + r) * (K >> 4), w0 = g0 >> 5, g = (w0 + p) * 32 + lane - g0, wrap = 16 - (w0 & 15);
            float ss = 0.0f;
            if (p < n) {
                if (g >= 0 && g < K >> 4) {
                    const float4* x4 = reinterpret_cast<const float4*>(src + r * K) + 4 * g;
                    float q = 0.0f;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const float4 x = x4[k];
                        q += x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
                    }
                    ss += q;
                }
                ss = warp_sum(ss);
            }
            if (lane == 0) part[r * kMaxParts + (p >= n ? p : (p >= wrap ? p - wrap : p + max(n - wrap, 0)))] = ss;
        }
        return;
    }
    const bool strided = o.order == kSumStrided;
    const int chunks = strided ? 2 : (o.share + 31) >> 5;          // of eight parts
#pragma unroll 1
    for (int i = warp; i < R * chunks; i += T / 32) {
        const int r = ONE ? 0 : i / chunks, p = (i - r * chunks) * 8;
        const float* row = src + r * K;
        float ss[8];
        if (strided) {
#pragma unroll
            for (int k = 0; k < 8; ++k) ss[k] = 0.0f;
#pragma unroll 1
            for (int d = p * 32 + lane; d < K; d += 512) {
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const float v = d + 32 * k < K ? row[d + 32 * k] : 0.0f;
                    ss[k] += v * v;
                }
            }
        } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const uint32_t at = span[p + k];
                const float v = lane < static_cast<int>(at >> 8 & 0xff) ? row[(at >> 16) + lane] : 0.0f;
                ss[k] = __fmul_rn(v, v);
            }
        }
        const float sum = butterfly8(ss, lane);
        const int at = p + (lane >> 2);
        if ((lane & 3) == 0) part[r * kMaxParts + (strided ? at : span[at] & 0xff)] = sum;
    }
}
__device__ __forceinline__ float sum_total(const Sums& o, const float* part) {
    float total = 0.0f;
    const float4* v4 = reinterpret_cast<const float4*>(part);
    if (o.order == kSumStrips) {
        const float4 a = v4[0], b = v4[1];
        return ((((((a.x + a.y) + a.z) + a.w) + b.x) + b.y) + b.z) + b.w;
    }
    if (o.order == kSumStrided) {
        float4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = v4[i];
#pragma unroll
        for (int i = 0; i < 4; ++i) total = (((total + v[i].x) + v[i].y) + v[i].z) + v[i].w;
        return total;
    }
    // parts lie [warp of its CTA][CTA]: eight lanes add up a CTA each
    float cta = 0.0f;
#pragma unroll 2
    for (int w = 0; w < (o.share + 31) >> 5; ++w) cta += part[8 * w + (threadIdx.x & 7)];
#pragma unroll
    for (int c = 0; c < 8; ++c) total += __shfl_sync(0xffffffffu, cta, c);
    return total;
}

// Rows src [R][K] in shared memory -> 8-bit codes in the order the weights are paired in; with norm weights w the row is normed first (`again`: by the
// factors of the call before).  The row's code sum and scale, which only the results of the products need, follow behind the barrier that hands the
// codes over.  ONE: the row is at most kHeld * 4 * T long, and a thread holds its part of w.  Else w is in shared memory, and a row is the work of
// (T / 32) / R warps.  False where a wait ran out in some thread (S.dead; a barrier that votes takes 150 cycles more).
template <bool ONE, int T, int kHeld>
__device__ __forceinline__ bool quantise_rows(Static& S, const float* src, int K, int R, const float* w, const float4 (&held)[kHeld], float eps, uint8_t* codes,
                                              float* act_scale, int* q_sum, float inv_k, const Sums& order, bool again) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wpr = ONE ? (T / 32) : (T / 32) / R, row = ONE ? 0 : warp / wpr, first = (warp - row * wpr) * 32 + lane, step = wpr * 32;
    const int n4 = ONE || row < R ? K >> 2 : 0;
    const bool on = first - lane < n4;         // this warp has a part of the row
    const float4* v4 = reinterpret_cast<const float4*>(src + (ONE || row >= R ? 0 : row * K));
    const float4* w4 = reinterpret_cast<const float4*>(w);
    float4 v[kHeld];
    float inv = 1.0f;
    if (on) {
#pragma unroll
        for (int i = 0; i < kHeld; ++i) v[i] = first + i * step < n4 ? v4[first + i * step] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    if (w && again) {
        inv = S.inv[row < R ? row : 0];
    } else if (w) {
        sum_parts<ONE, T>(order, src, K, R, S.span, S.red);
        __syncthreads();
        if (*reinterpret_cast<volatile int*>(&S.dead)) return false;
        if (on) {
            const float sum = sum_total(order, S.red + row * kMaxParts);
            // sum / K, correctly rounded: one residual against the rounded reciprocal of K (Markstein 1990)
            const float k = static_cast<float>(K), q0 = sum * inv_k, mean = __fmaf_rn(__fmaf_rn(-q0, k, sum), inv_k, q0);
            inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(isfinite(q0) ? mean : q0, eps)));
            if (lane == 0 && warp == row * wpr) S.inv[row] = inv;
        }
    }
    auto scaled = [&](const float4& a, const float4& b) {
        return w ? make_float4(__fmul_rn(__fmul_rn(a.x, inv), b.x), __fmul_rn(__fmul_rn(a.y, inv), b.y), __fmul_rn(__fmul_rn(a.z, inv), b.z),
                               __fmul_rn(__fmul_rn(a.w, inv), b.w))
                 : a;
    };
    auto weights = [&](int q) { return w ? w4[q] : make_float4(1.0f, 1.0f, 1.0f, 1.0f); };
    auto top = [](float m, const float4& a) { return fmaxf(m, fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w)))); };
    if (on) {
        float mx = 0.0f;
#pragma unroll
        for (int i = 0; i < kHeld; ++i) {
            if (ONE || first + i * step < n4) v[i] = scaled(v[i], ONE ? held[i] : weights(first + i * step));
            mx = top(mx, v[i]);
        }
        if constexpr (!ONE) {
#pragma unroll 1
            for (int q = first + kHeld * step; q < n4; q += step) mx = top(mx, scaled(v4[q], weights(q)));
        }
        const uint32_t wm = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
        if (lane == 0) S.redm[warp] = __uint_as_float(wm);
    } else if (lane == 0) {
        S.redm[warp] = 0.0f;
    }
    __syncthreads();
    if (*reinterpret_cast<volatile int*>(&S.dead)) return false;
    float denom = 0.0f;
    int total = 0;
    if (on) {
        float m = 0.0f;
        if constexpr (ONE) {
            const float4 a = reinterpret_cast<const float4*>(S.redm)[0], c = reinterpret_cast<const float4*>(S.redm)[1];
            m = fmaxf(fmaxf(fmaxf(a.x, a.y), fmaxf(a.z, a.w)), fmaxf(fmaxf(c.x, c.y), fmaxf(c.z, c.w)));
        } else {
#pragma unroll 1
            for (int k = 0; k < wpr; ++k) m = fmaxf(m, S.redm[row * wpr + k]);
        }
        denom = __fadd_rn(m, 1e-8f);
        const float scale = __fdiv_rn(127.0f, denom);
        auto store = [&](const float4& a, int q) {
            auto code = [&](float x) { return static_cast<uint32_t>(round_code(__fmul_rn(x, scale), false)); };
            const uint32_t c0 = code(a.x), c1 = code(a.y), c2 = code(a.z), c3 = code(a.w);
            total = dp4a_ss(static_cast<int>(__byte_perm(__byte_perm(c0, c1, 0x0040), __byte_perm(c2, c3, 0x0040), 0x5410)), 0x01010101, total);
            // qp_offset() of four elements of one of its 16-element groups
            uint8_t* at = codes + (q >> 6) * (R * 256) + row * 256 + (((((q >> 2) & 3) ^ (row & 1)) << 6) | (q & 48) | (q & 3));
            at[0] = static_cast<uint8_t>(c0); at[4] = static_cast<uint8_t>(c1); at[8] = static_cast<uint8_t>(c2); at[12] = static_cast<uint8_t>(c3);
        };
#pragma unroll
        for (int i = 0; i < kHeld; ++i)
            if (first + i * step < n4) store(v[i], first + i * step);
        if constexpr (!ONE) {
#pragma unroll 1
            for (int q = first + kHeld * step; q < n4; q += step) store(scaled(v4[q], weights(q)), q);
        }
    }
    __syncthreads();
    if (on) {
        total = __reduce_add_sync(0xffffffffu, total);
        if (lane == 0) {
            atomicAdd(q_sum + row, total);
            if (warp == row * wpr) act_scale[row] = __fdiv_rn(denom, 127.0f);
        }
    }
    return true;
}

// Sends a value to the same place of every CTA of the cluster (dst and bar: this CTA's addresses).  One value per thread, as the thread has it:
// a gather of 768 / 1536 numbers over 16 CTAs takes 0.45 / 0.57 us this way, 0.65 / 0.78 as staged float4s, 0.93 by bulk copies, 1.05 / 1.20 by
// plain stores and a cluster barrier.
// Peers first, first + step, ...: several lanes can share the work.
__device__ __forceinline__ void send(uint32_t dst, uint32_t bar, float v, int ctas, int first = 0, int step = 1) {
#pragma unroll 4
    for (int peer = first; peer < ctas; peer += step)
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(map_rank(dst, peer)), "r"(__float_as_uint(v)),
                     "r"(map_rank(bar, peer))
                     : "memory");
}
// Half of the peers
__device__ __forceinline__ void send_half(uint32_t dst, uint32_t bar, float v, int ctas, int half) {
#pragma unroll
    for (int k = 0; k < 8; ++k)
        if (2 * k < ctas)
            asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(map_rank(dst, 2 * k + half)),
                         "r"(__float_as_uint(v)), "r"(map_rank(bar, 2 * k + half))
                         : "memory");
}

// Rotated queries and keys, and the values, of the CTA's heads: qkv [row][q | k | v] in shared memory.
template <bool ONE, int T>
__device__ __noinline__ void rotate(const Params& P, const Static& S, const Block& b, uint8_t* smem, int rank, int R, const int* acc, const int (*q_sum)[kMaxRows]) {
    const Owned& o = P.own[rank];
    const Job* ja = S.job[kPassA];
    float* qkv = reinterpret_cast<float*>(smem + P.L.qkv);
    const int dim = P.d.head_dim, half = dim >> 1, nq = size_of(o.attn), nkv = size_of(o.kv);
    const int width = (nq + 2 * nkv) * dim, kv_dim = P.d.a_kv_heads * dim;
    auto value = [&](const Linear& v, const Job& job, int r, int local, int n) {
        return epilogue(acc[r * P.L.acc_stride + job.acc + local] - q_sum[1][r], __fmul_rn(S.act_scale[1][r], v.scale), v.magnitude, v.bias, n);
    };
    const int n_rot = (nq + nkv) * half, items = n_rot + nkv * half;
    for (int i = threadIdx.x; i < R * items; i += T) {
        const int r = i / items, k = i - r * items;
        const int pos = min(max(S.pos[r], 0), b.rope_positions - 1);
        float* out = qkv + r * width;
        if (k < n_rot) {
            const int h = k / half, e = k - h * half;
            const bool is_q = h < nq;
            const int hl = is_q ? h : h - nq, n = (is_q ? o.attn.lo + hl : o.kv.lo + hl) * dim + e;
            const Linear& v = b.lin[is_q ? kQ : kKv];
            const Job& job = ja[is_q ? 5 : 6];
            const float v0 = value(v, job, r, hl * dim + e, n), v1 = value(v, job, r, hl * dim + e + half, n + half);
            const float cv = __ldg(b.rope_cos + static_cast<size_t>(pos) * half + e), sv = __ldg(b.rope_sin + static_cast<size_t>(pos) * half + e);
            out[h * dim + e] = __fsub_rn(__fmul_rn(v0, cv), __fmul_rn(v1, sv));
            out[h * dim + e + half] = __fadd_rn(__fmul_rn(v0, sv), __fmul_rn(v1, cv));
        } else {
            const int hl = (k - n_rot) / half, e = (k - n_rot) - hl * half, n = kv_dim + (o.kv.lo + hl) * dim + e;
            out[(nq + nkv + hl) * dim + e] = value(b.lin[kKv], ja[7], r, hl * dim + e, n);
            out[(nq + nkv + hl) * dim + e + half] = value(b.lin[kKv], ja[7], r, hl * dim + e + half, n + half);
        }
    }
}

// Single-token attention of the CTA's heads (attention_decode_kernel's arithmetic and orders; a sequence's head is the work of (T / 32) / R warps);
// the results go to dst [row][d_model] of every CTA.
template <bool ONE, int T>
__device__ __noinline__ void attend(const Params& P, Static& S, const Block& b, uint8_t* smem, int rank, int ctas, int row0, int R, uint32_t dst, uint32_t bar) {
    const Owned& own = P.own[rank];
    const int group = max(P.d.a_heads / P.d.a_kv_heads, 1);
    float* qkv = reinterpret_cast<float*>(smem + P.L.qkv);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int dim = P.d.head_dim, nq = size_of(own.attn), nkv = size_of(own.kv), width = (nq + 2 * nkv) * dim, kv_dim = P.d.a_kv_heads * dim;
    // the new key and value join the cache
    for (int i = tid; i < R * nkv * dim; i += T) {
        const int r = i / (nkv * dim), k = i - r * (nkv * dim), hl = k / dim, e = k - hl * dim, kvh = own.kv.lo + hl, pos = S.pos[r];
        const bool ok = pos >= 0 && pos < P.capacity && pos < b.rope_positions;
        if (ok && kvh * group >= own.attn.lo && kvh * group < own.attn.hi) {
            const size_t at = (static_cast<size_t>(row0 + r) * P.capacity + pos) * kv_dim + kvh * dim + e;
            b.k_cache[at] = qkv[r * width + (nq + hl) * dim + e];
            b.v_cache[at] = qkv[r * width + (nq + nkv + hl) * dim + e];
        }
    }
    float* scores = reinterpret_cast<float*>(smem + P.L.scores);
    float4* partial = reinterpret_cast<float4*>(smem + P.L.partial);
    const int wpr = (T / 32) / R, row = warp / wpr, nthr = wpr * 32, lr = tid - row * nthr;
    const int pos = row < R ? S.pos[row] : -1;
    const bool on = pos >= 0 && pos < P.capacity && pos < b.rope_positions;
    if (row < R && !on && lr == 0) atomicOr(P.status, TBL_DEV_CACHE_FULL);
    const int cached = on ? pos + 1 : 0, first = max(0, cached - b.window);
    float* sc = scores + (row < R ? row : 0) * P.L.score_len;
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn(static_cast<float>(dim)));
    for (int hl = 0; hl < nq; ++hl) {
        const int kvh = min((own.attn.lo + hl) / group, P.d.a_kv_heads - 1), kl = kvh - own.kv.lo;
        const float* q = qkv + (row < R ? row : 0) * width + hl * dim;
        const float* knew = qkv + (row < R ? row : 0) * width + (nq + kl) * dim;
        const float* vnew = knew + nkv * dim;
        const size_t head_base = static_cast<size_t>(row0 + (row < R ? row : 0)) * P.capacity * kv_dim + static_cast<size_t>(kvh) * dim;
        float top = -1e30f;
        const bool long_context = cached - first > 256;
        if (long_context) {
            // A long context: four lanes a token, 64 bytes of its key a load, dot products in four parts.  A thread a token reads 16 bytes here and there of
            // as many keys as there are threads, whose other halves the L1 beside this kernel's shared memory does not hold.
            const int sub = lane & 3, stride = wpr * 8;
            const float4* q4 = reinterpret_cast<const float4*>(q) + sub;
            constexpr int kTokens = 2, kParts = 4;
            for (int base = first + (lr >> 5) * 8; base < cached; base += kTokens * stride) {
                float dot[kTokens];
#pragma unroll
                for (int u = 0; u < kTokens; ++u) dot[u] = 0.0f;
                for (int c = 0; c < dim / 16; c += kParts) {
                    float4 k[kTokens][kParts];
#pragma unroll
                    for (int u = 0; u < kTokens; ++u) {
                        const int t = base + u * stride + (lane >> 2);
                        const float4* key = (t == pos ? reinterpret_cast<const float4*>(knew) : reinterpret_cast<const float4*>(b.k_cache + head_base + static_cast<size_t>(t) * kv_dim)) + sub;
#pragma unroll
                        for (int v = 0; v < kParts; ++v) k[u][v] = t < cached && c + v < dim / 16 ? key[4 * (c + v)] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    }
#pragma unroll
                    for (int v = 0; v < kParts; ++v) {
                        if (c + v < dim / 16) {
                            const float4 a = q4[4 * (c + v)];
#pragma unroll
                            for (int u = 0; u < kTokens; ++u) dot[u] += (a.x * k[u][v].x + a.y * k[u][v].y) + (a.z * k[u][v].z + a.w * k[u][v].w);
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < kTokens; ++u) {
                    const int t = base + u * stride + (lane >> 2);
                    dot[u] += __shfl_xor_sync(0xffffffffu, dot[u], 1);
                    dot[u] += __shfl_xor_sync(0xffffffffu, dot[u], 2);
                    if (t < cached) {
                        const float s = __fmul_rn(dot[u], scale);
                        if (sub == 0) sc[t - first] = s;
                        top = fmaxf(top, s);
                    }
                }
            }
        } else
        for (int t = first + lr; t < cached; t += nthr) {
            // the dot product in dimension order; the new token's key is the one in shared memory
            const float4* key = t == pos ? reinterpret_cast<const float4*>(knew) : reinterpret_cast<const float4*>(b.k_cache + head_base + static_cast<size_t>(t) * kv_dim);
            float dot = 0.0f;
            constexpr int kParts = 8;
            for (int d = 0; d < dim / 4; d += kParts) {
                float4 k4[kParts];
#pragma unroll
                for (int u = 0; u < kParts; ++u) k4[u] = d + u < dim / 4 ? key[d + u] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                for (int u = 0; u < kParts; ++u) {
                    if (d + u < dim / 4) {
                        const float4 q4 = reinterpret_cast<const float4*>(q)[d + u];
                        dot = __fadd_rn(dot, __fmul_rn(q4.x, k4[u].x));
                        dot = __fadd_rn(dot, __fmul_rn(q4.y, k4[u].y));
                        dot = __fadd_rn(dot, __fmul_rn(q4.z, k4[u].z));
                        dot = __fadd_rn(dot, __fmul_rn(q4.w, k4[u].w));
                    }
                }
            }
            const float s = __fmul_rn(dot, scale);
            sc[t - first] = s;
            top = fmaxf(top, s);
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        if (lane == 0) S.redm[warp] = top;
        __syncthreads();
        if (row < R)
            for (int w = 0; w < wpr; ++w) top = fmaxf(top, S.redm[row * wpr + w]);
        // the exponentials' sum by attention_decode_kernel's eight warps: thread t of 256 takes tokens t, t + 256, ...
        if (row < R) {
            for (int vw = lr >> 5; vw < 8; vw += wpr) {
                float sum = 0.0f;
                for (int t = first + vw * 32 + lane; t < cached; t += 256) {
                    const float e = expf(__fsub_rn(sc[t - first], top));
                    sc[t - first] = e;
                    sum += e;
                }
                sum = warp_sum(sum);
                if (lane == 0) S.red[row * kMaxParts + vw] = sum;
            }
        }
        __syncthreads();
        float total = S.red[(row < R ? row : 0) * kMaxParts];
        for (int w = 1; w < 8; ++w) total += S.red[(row < R ? row : 0) * kMaxParts + w];
        const float inv_sum = __fdiv_rn(1.0f, fmaxf(total, 1e-9f));
        // Its groups of dim / 4 threads take the tokens round-robin, and their sums are added in order: so do ours, in rounds where we have fewer.  (Over a
        // long context our own groups: 64 sequences with 900 tokens 740 us a step, as against 847 in its order and 812 as separate launches.  These are
        // fewer, and longer sums err more: so eight tokens are added up by themselves, and a sum errs a little less than in its order instead of three times.)
        const int row_threads = dim / 4, groups = nthr / row_threads, all = 256 / row_threads;
        const int its_groups = long_context ? groups : all, g0 = lr / row_threads, d4 = lr - g0 * row_threads;
        const int hold = P.L.partial_all ? max(all, groups) : groups, rounds = (max(all, groups) + hold - 1) / hold;       // groups' sums there is room for
        float4* mine = partial + (row < R ? row : 0) * hold * row_threads;
        const float4* vrow = reinterpret_cast<const float4*>(b.v_cache + head_base) + d4;
        const size_t step = static_cast<size_t>(kv_dim / 4);
        float* sums = const_cast<float*>(q);           // (the query has done its work)
        for (int round = 0; round < rounds; ++round) {
            const int n_groups = min(hold, its_groups - round * hold);
            if (g0 < groups && row < R) {
#pragma unroll 1
                for (int local = g0; local < n_groups; local += groups) {
                    const int g = round * hold + local;
                    float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (long_context) mine[local * row_threads + d4] = o;
                    auto add = [&](const float4& v, float p) {
                        o.x = __fadd_rn(o.x, __fmul_rn(p, v.x)); o.y = __fadd_rn(o.y, __fmul_rn(p, v.y));
                        o.z = __fadd_rn(o.z, __fmul_rn(p, v.z)); o.w = __fadd_rn(o.w, __fmul_rn(p, v.w));
                    };
                    constexpr int kInFlight = 8;
                    for (int t = first + g; t < cached; t += kInFlight * its_groups) {
                        float4 v[kInFlight];
#pragma unroll
                        for (int j = 0; j < kInFlight; ++j) {
                            const int at = t + j * its_groups;
                            v[j] = at < pos ? vrow[static_cast<size_t>(at) * step] : reinterpret_cast<const float4*>(vnew)[d4];
                        }
#pragma unroll
                        for (int j = 0; j < kInFlight; ++j)
                            if (t + j * its_groups < cached) add(v[j], __fmul_rn(sc[t + j * its_groups - first], inv_sum));
                        if (long_context) {
                            float4& sum = mine[local * row_threads + d4];        // (in shared memory: there are no registers to spare)
                            sum = make_float4(__fadd_rn(sum.x, o.x), __fadd_rn(sum.y, o.y), __fadd_rn(sum.z, o.z), __fadd_rn(sum.w, o.w));
                            o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        }
                    }
                    if (!long_context) mine[local * row_threads + d4] = o;
                }
            }
            __syncthreads();
            if (row < R && n_groups > 0) {
                const float* m = reinterpret_cast<const float*>(mine);
                for (int d = lr; d < dim; d += nthr) {
                    float v = round ? __fadd_rn(sums[d], m[d]) : m[d];
#pragma unroll 4
                    for (int j = 1; j < n_groups; ++j) v = __fadd_rn(v, m[j * dim + d]);
                    sums[d] = v;
                    if (round * hold + n_groups == its_groups) send(dst + 4u * (row * P.d.D + (own.attn.lo + hl) * dim + d), bar, v, ctas);
                }
            }
            if (round + 1 < rounds) __syncthreads();
        }
    }
}

template <bool ONE, int T>
__global__ void __launch_bounds__(T, 1) decode_cluster_kernel(const __grid_constant__ Params P) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(16) Static S;
    constexpr int kHeld = ONE ? 4 : 2;  // float4s of a row that a thread norms and quantises in registers
    constexpr int kDtFirst = T - 32;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint32_t rank_u, ctas_u;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank_u));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ctas_u));
    const int rank = static_cast<int>(rank_u), ctas = static_cast<int>(ctas_u);
    const int row0 = (blockIdx.x / ctas) * P.rows;
    const int R = ONE ? 1 : min(P.rows, P.batch - row0);
    const int D = P.d.D, DI = P.d.inner;
    const Layout& L = P.L;
    float* x0 = reinterpret_cast<float*>(smem + L.x0);
    float* x1 = reinterpret_cast<float*>(smem + L.x1);
    uint8_t* codes = smem + L.codes;
    int* acc_all = reinterpret_cast<int*>(smem + L.acc);       // two sets: a pass fills one, the other is emptied
    float* zs = reinterpret_cast<float*>(smem + L.zs);
    float* xs = reinterpret_cast<float*>(smem + L.xs);
    float* bc = reinterpret_cast<float*>(smem + L.bc);
    float* bcring = reinterpret_cast<float*>(smem + L.bcring);
    float* decay_s = reinterpret_cast<float*>(smem + L.decay);
    float* normw = reinterpret_cast<float*>(smem + L.norm);
    float* skip_s = reinterpret_cast<float*>(smem + L.skip);       // D of the CTA's heads
    uint16_t* heads_of = reinterpret_cast<uint16_t*>(smem + L.heads_of);       // a channel's head
    uint2* table = reinterpret_cast<uint2*>(smem + L.table);
    const int acc_stride = L.acc_stride, acc_quads = acc_stride * P.rows / 4;

    // the kernel behind this one (final norm, head) may set up and fetch its weights meanwhile
    pdl_launch_dependents();

    // a block's description comes to shared memory by the last warp, while the others are at the SSD step of the block before
    constexpr int kPieces = sizeof(Block) / 16;
    auto fetch_block = [&](int index) {
        const uint4* src = reinterpret_cast<const uint4*>(&P.blk[index]);
        uint4* dst = reinterpret_cast<uint4*>(&S.blk[index & 1]);
        const uint4 a = src[lane], c = lane + 32 < kPieces ? src[lane + 32] : make_uint4(0, 0, 0, 0);
        dst[lane] = a;
        if (lane + 32 < kPieces) dst[lane + 32] = c;
    };
    if (tid == 0) {
        S.dead = 0;
        mbar_init(&S.bar[0], 1);
        mbar_init(&S.bar[1], 1);
        fence_mbar_init();
    }
    if (warp == T / 32 - 1) fetch_block(0);
    if (warp == 0) plan_jobs<T>(P, S, rank, R);
    for (int i = tid; i < 2 * acc_quads; i += T) reinterpret_cast<int4*>(acc_all)[i] = make_int4(0, 0, 0, 0);
    if (tid < 4 * kMaxRows) (&S.q_sum[0][0][0])[tid] = 0;
    if (tid >= 128 && tid < 128 + kMaxParts) {
        const int a_cta = (P.gate_share + 31) >> 5, p = tid - 128, cta = p / a_cta, w = p - cta * a_cta, c = cta * P.gate_share + 32 * w;
        S.span[p] = static_cast<uint32_t>(w * 8 + cta) | static_cast<uint32_t>(max(0, min(32, min(P.gate_share - 32 * w, DI - c)))) << 8 | static_cast<uint32_t>(c) << 16;
    }
    if (tid >= 64 && tid < 64 + R) S.pos[tid - 64] = P.positions[row0 + tid - 64];
    for (int i = tid; i < R * (D >> 2); i += T) {
        const int r = ONE ? 0 : i / (D >> 2), q = i - r * (D >> 2);
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (P.ids) {
            const int id = P.ids[row0 + r];
            if (id >= 0 && id < P.vocab) {
                const float* e = P.embedding + static_cast<size_t>(id) * D + 4 * q;
                v = make_float4(e[0], e[1], e[2], e[3]);
            }
        } else {
            v = reinterpret_cast<const float4*>(P.hidden_in + static_cast<size_t>(row0 + r) * D)[q];
        }
        reinterpret_cast<float4*>(x0)[i] = v;
        if (P.trace && rank == 0) {
            float* tr = P.trace + static_cast<size_t>(row0 + r) * D + 4 * q;
            tr[0] = v.x; tr[1] = v.y; tr[2] = v.z; tr[3] = v.w;
        }
    }

    __syncthreads();
    plan_pieces<T>(S, table, R);

    // ---- threads' parts in what follows the products: the same in every block ----
    const Owned& own = P.own[rank];
    const int conv_dim = DI + 32, ring_row = kTaps * conv_dim;
    const int chan_lo = own.chan.lo, per = size_of(own.chan), head_lo = own.head.lo, nh = size_of(own.head);
    // Items: convolution of the CTA's channels and of B and C, gates.  A thread keeps one item (and its parameters) and takes every c_step-th
    // sequence.  From the last threads down, since the first ones also finish the residual stream.  Step sizes: the last warp.
    struct Item { int lin, row, channel, acc; };          // its projection, row there, channel of the convolution (-1: a gate), accumulator
    auto item_of = [&](int c) {
        if (c < per) return Item{kX, chan_lo + c, chan_lo + c, S.job[kPassA][0].acc + c};
        if (c >= per + 32) return Item{kZ, chan_lo + c - per - 32, -1, S.job[kPassA][1].acc + c - per - 32};
        const int e = c - per;
        return Item{e < 16 ? kB : kC, e & 15, DI + e, S.job[kPassA][e < 16 ? 2 : 3].acc + (e & 15)};
    };
    const int n_items = 2 * per + 32, item = kDtFirst - 1 - tid, c_wide = min(n_items, kDtFirst), c_step = ONE ? 1 : min(R, kDtFirst / c_wide);
    const int c0 = ONE ? item : item % c_wide, cr0 = item < 0 || (ONE ? item >= c_wide : item / c_wide >= c_step) ? R : (ONE ? 0 : item / c_wide);
    Item it = cr0 < R ? item_of(c0) : Item{0, 0, 0, 0};
    const bool dtt = tid >= kDtFirst && (!ONE || tid - kDtFirst < nh);
    const int dt0 = ONE ? tid - kDtFirst : (tid - kDtFirst) % nh;
    // SSD step: four lanes share a channel's sixteen numbers.  ONE: a pair of warps takes 32 channels, eight a warp and round; else T / 4 channels a round
    const int s_lane = tid & 3, s_first = ONE ? (warp >> 1) * 32 + (warp & 1) * 16 + (lane >> 2) : tid >> 2;
    // rows of the residual stream
    const int n_lo = own.row.lo, n_own = size_of(own.row);
    // ONE: a pair of warps sends 32 numbers, each warp to every other peer: 128 bytes a packet (sent as they come from the quads, 32 bytes each, a gather
    // took a microsecond longer)
    const int s_own = (warp >> 1) * 32 + lane;
    const float inv_d = 1.0f / static_cast<float>(D), inv_inner = 1.0f / static_cast<float>(DI);

    if constexpr (!ONE)
        for (int i = tid; i < per; i += T) heads_of[i] = static_cast<uint16_t>((chan_lo + i) / P.d.d_head - head_lo);
    const int s_head[2] = {(chan_lo + s_first) / P.d.d_head - head_lo, (chan_lo + s_first + 8) / P.d.d_head - head_lo};       // ONE
    cluster_sync();          // barriers of all CTAs are up before anybody sends; the tables are there

    int gathers = 0;         // how many gathers this CTA has waited for
    // expects the next gather (all CTAs' parts, this one's too)
    auto expect = [&](int floats) {
        if (tid == 0) mbar_arrive_expect_tx(&S.bar[gathers & 1], 4u * R * floats);
    };
    auto norm_weights = [&](const float* w, int n, int at) {
#pragma unroll 1
        for (int i = tid; i < n >> 2; i += T) cp_async16(smem_u32(normw + at + 4 * i), w + 4 * i);
    };
    float stream = ONE && s_own < n_own ? x0[n_lo + s_own] : 0.0f;       // ONE: its number of the residual stream
    Stream ws;
    // what a thread's results of pass A meet, requested ahead of the products (a projection without magnitudes or biases: 1 and 0)
    float cw[kTaps + 1], tap[kTaps], cb = 0.0f, mg = 1.0f, bs = 0.0f, a_log = 0.0f, Dv[2] = {0.0f, 0.0f};
    double rate = 0.0;                            // exp(A_log)
    float4 hv[2];

    int pass = kPassA, bi = 0, turn = 0;         // turn: passes so far
    bool alive = true;
#pragma unroll 1
    for (;; ++turn) {
        const Block& b = S.blk[bi & 1];
        const bool hybrid = b.hybrid != 0, last = bi + 1 == P.n_blocks;
        int* acc = acc_all + (turn & 1) * acc_stride * P.rows;
        int (*q_sum)[kMaxRows] = S.q_sum[turn & 1];
        const uint2* pieces = table + S.first[pass];
        const int n_pieces = S.count[hybrid ? 1 : 0][pass];
        // ---- while the row is on its way: weights, norm weights, the state ----
        request(b, pieces, n_pieces, warp, ws);
        const float* norm_w = pass == kPassA ? b.core_norm_w : (pass == kPassB ? b.norm_w : (pass == kPassC ? b.ff_norm_w : nullptr));
        const int K = pass == kPassB ? DI : (pass == kPassD ? P.d.ff : D);
        float4 held[kHeld];
        auto hold = [&](const float* w, int k) {
#pragma unroll
            for (int i = 0; i < kHeld; ++i) {
                held[i] = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
                if (ONE && w && tid + i * T < k >> 2) held[i] = __ldg(reinterpret_cast<const float4*>(w) + tid + i * T);
            }
        };
        hold(norm_w, K);
        if constexpr (!ONE) {
            if (norm_w) norm_weights(norm_w, K, 0);
            if (hybrid && pass == kPassA) norm_weights(b.attn_norm_w, D, D);
        }
        auto conv_params = [&](const Item& t) {
            const Linear& v = b.lin[t.lin];
            if (v.magnitude) mg = __ldg(v.magnitude + t.row);
            if (v.bias) bs = __ldg(v.bias + t.row);
            if (t.channel < 0) return;
#pragma unroll
            for (int j = 0; j <= kTaps; ++j) cw[j] = __ldg(b.conv_w + t.channel * (kTaps + 1) + j);
            cb = __ldg(b.conv_b + t.channel);
        };
        auto window_of = [&](const Item& t, int r) { return b.ring + static_cast<size_t>(row0 + r) * ring_row + t.channel; };
        auto state_of = [&](int ch) { return reinterpret_cast<float4*>(b.ssm) + (static_cast<size_t>(row0) * DI + chan_lo + ch) * 4 + s_lane; };       // ONE
        auto dt_params = [&](int head) {
            mg = b.lin[kDt].magnitude ? __ldg(b.lin[kDt].magnitude + head) : 1.0f;
            bs = b.lin[kDt].bias ? __ldg(b.lin[kDt].bias + head) : 0.0f;
            a_log = __ldg(b.A_log + head);
        };
        if (pass == kPassA) {
            if (cr0 < R) {
                mg = 1.0f; bs = 0.0f;
                conv_params(it);
                if (ONE && c_wide == n_items && it.channel >= 0) {
#pragma unroll
                    for (int j = 0; j < kTaps; ++j) tap[j] = window_of(it, 0)[j * conv_dim];
                }
            } else if (ONE && dtt) {
                dt_params(head_lo + dt0);
                rate = exp64(a_log);
            }
            if constexpr (ONE) {
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    if (s_first + 8 * k < per) {
                        hv[k] = *state_of(s_first + 8 * k);
                        Dv[k] = __ldg(b.D + head_lo + s_head[k]);
                    }
                }
            } else if (L.state >= 0) {
                // a thread fetches what it will itself read: no barrier, only its own wait
                if (it.channel >= 0 && c_wide == n_items) {
#pragma unroll 1
                    for (int r = cr0; r < R; r += c_step)
#pragma unroll
                        for (int j = 0; j < kTaps; ++j) cp_async4(smem_u32(smem + L.taps) + 4 * ((r * kTaps + j) * (per + 32) + c0), window_of(it, r) + j * conv_dim);
                }
#pragma unroll 1
                for (int i = s_first, r = 0, ch = s_first; i < R * per; i += T / 4, ch += T / 4) {
                    while (ch >= per) { ch -= per; ++r; }
                    cp_async16(smem_u32(smem + L.state) + 16 * (4 * i + s_lane), b.ssm + ((static_cast<size_t>(row0 + r) * DI + chan_lo + ch) * 4 + s_lane) * 4);
                }
            }
        }
        if (turn) {
            if (!mbar_wait_bounded(&S.bar[gathers & 1], (gathers >> 1) & 1, P.status)) S.dead = 1;
            ++gathers;
        }
        if constexpr (!ONE) {
            cp_async_wait();
            if (norm_w) __syncthreads();          // the norm's weights are there
        }

        // ---- the row(s) as codes, the products ----
        // (the first row of a step is normed by residual_norm_kernel there: it comes from the embedding)
        const Sums order = pass == kPassB ? Sums{P.gate_order, P.gate_share, row0} : Sums{turn == 0 && P.ids ? kSumStrided : P.row_order, 0, row0};
#pragma unroll 1
        for (int set = 0;; ++set) {
            // the second set: the attention's input row, or its heads' result
            const float* w = set == 0 ? norm_w : (pass == kPassA ? b.attn_norm_w : nullptr);
            if (set && ONE) hold(w, D);
            alive = quantise_rows<ONE, T, kHeld>(S, pass == kPassA || pass == kPassC ? x0 : x1 + (set ? R * DI : 0), set ? D : K, R, ONE || !w ? w : normw + (set ? D : 0), held,
                                              pass == kPassA ? b.core_eps : (pass == kPassB ? b.norm_eps : 1e-5f), codes + (set ? R * K : 0), S.act_scale[set],
                                              q_sum[set], set || K == D ? inv_d : inv_inner, order, set != 0);
            if (set || !hybrid || pass > kPassB || !alive) break;
        }
        if (!alive) break;                        // some CTA of the cluster does not answer
        multiply<ONE, T>(b, pieces, n_pieces, ws, smem_u32(codes), acc, acc_stride, R);
        // empty accumulators for the next pass: everybody has read what the pass before left there
        {
            int4* other = reinterpret_cast<int4*>(acc_all + ((turn & 1) ^ 1) * acc_stride * P.rows);
#pragma unroll 1
            for (int i = T - 1 - tid; i < acc_quads; i += T) other[i] = make_int4(0, 0, 0, 0);
            if (tid >= T - 2 * kMaxRows) (&S.q_sum[(turn & 1) ^ 1][0][0])[T - 1 - tid] = 0;
        }
        __syncthreads();
        const uint32_t bar = smem_u32(&S.bar[gathers & 1]);
        // a product's result: the sum of codes x (code + 1) less the sum of codes, scaled
        auto affine = [&](int sum, int set, int r, float scale, float magnitude, float bias) {
            return __fadd_rn(__fmul_rn(__fmul_rn(static_cast<float>(sum - q_sum[set][r]), __fmul_rn(S.act_scale[set][r], scale)), magnitude), bias);
        };

        if (pass == kPassA) {
            // The convolution's window moves on: for the CTA's own channels at once, for B and C (every CTA reads the old window) behind the next gather.
            // N sequences at a time: a chain of dependent steps each.
            auto convolve = [&](auto n, int c, int r, const float (&t)[decltype(n)::value][kTaps]) {
                constexpr int N = decltype(n)::value;
                float in[N], y[N];
#pragma unroll
                for (int k = 0; k < N; ++k) y[k] = in[k] = affine(acc[(r + k * c_step) * acc_stride + it.acc], 0, r + k * c_step, b.lin[it.lin].scale, mg, bs);
                if (it.channel >= 0) {
#pragma unroll
                    for (int k = 0; k < N; ++k) {
                        y[k] = cb;
#pragma unroll
                        for (int j = 0; j < kTaps; ++j) y[k] = __fadd_rn(y[k], __fmul_rn(cw[j], t[k][j]));
                        y[k] = __fadd_rn(y[k], __fmul_rn(cw[kTaps], in[k]));
                    }
                }
#pragma unroll
                for (int k = 0; k < N; ++k) y[k] = silu(y[k]);
                // x, gates and [B | C] each have their place: [row][channel]
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const int rr = r + k * c_step;
                    if (c < per) {
                        float* w = window_of(it, rr);
                        w[0] = t[k][1]; w[conv_dim] = t[k][2]; w[2 * conv_dim] = in[k];
                        xs[rr * per + c] = y[k];
                    } else if (it.channel >= 0) {
                        float* w = bcring + (rr * 32 + c - per) * kTaps;
                        w[0] = t[k][1]; w[1] = t[k][2]; w[2] = in[k];
                        bc[rr * 32 + c - per] = y[k];
                    } else {
                        zs[rr * per + c - per - 32] = y[k];
                    }
                }
            };
#pragma unroll 1
            for (int c = c0; cr0 < R && c < n_items; c += c_wide) {
                const bool there = !ONE && L.state >= 0 && c_wide == n_items;
                if (c_wide < n_items && (c != c0 || turn)) {
                    it = item_of(c);
                    mg = 1.0f; bs = 0.0f;
                    conv_params(it);
                }
                auto load_taps = [&](int r, float (&t)[kTaps]) {
                    const float* from = there ? reinterpret_cast<const float*>(smem + L.taps) + r * kTaps * (per + 32) + c : window_of(it, r);
#pragma unroll
                    for (int j = 0; j < kTaps; ++j) t[j] = it.channel >= 0 ? from[j * (there ? per + 32 : conv_dim)] : 0.0f;
                };
                if constexpr (ONE) {
                    float t[1][kTaps];
                    if (c_wide < n_items) load_taps(0, t[0]);
                    else { t[0][0] = tap[0]; t[0][1] = tap[1]; t[0][2] = tap[2]; }
                    convolve(std::integral_constant<int, 1>{}, c, 0, t);
                    if (c_wide == n_items) break;
                } else {
                    int r = cr0;
#pragma unroll 1
                    for (; r + c_step < R; r += 2 * c_step) {
                        float t[2][kTaps];
                        load_taps(r, t[0]);
                        load_taps(r + c_step, t[1]);
                        convolve(std::integral_constant<int, 2>{}, c, r, t);
                    }
                    if (r < R) {
                        float t[1][kTaps];
                        load_taps(r, t[0]);
                        convolve(std::integral_constant<int, 1>{}, c, r, t);
                    }
                }
            }
            if (dtt) {
#pragma unroll 1
                for (int i = tid - kDtFirst, have = -1; i < R * nh; i += 32) {
                    const int r = ONE ? 0 : i / nh, h = i - r * nh, head = head_lo + h;
                    if (!ONE && h != have) {
                        dt_params(head);
                        rate = exp64(a_log);
                        have = h;
                    }
                    const float dt = affine(acc[r * acc_stride + S.job[kPassA][4].acc + head - 16 * (head_lo >> 4)], 0, r, b.lin[kDt].scale, mg, bs);
                    const float delta = dt > 20.0f ? dt : (dt < -20.0f ? expf(dt) : log1pf(expf(dt)));
                    // decay = exp(-delta exp(A_log)) in double; below -20 the step size itself has lost what its logarithm holds
                    float decay;
                    if (!isfinite(dt) || !isfinite(a_log)) decay = nanf("");
                    else decay = static_cast<float>(exp64(-(dt < -20.0f ? exp64(static_cast<double>(dt) + static_cast<double>(a_log)) : static_cast<double>(delta) * rate)));
                    decay_s[i * 2] = delta;
                    decay_s[i * 2 + 1] = decay;
                    if (!ONE && r == 0) skip_s[h] = __ldg(b.D + head);
                    if (ONE) break;
                }
            }
            expect(DI + (hybrid ? D : 0));
            if (hybrid) rotate<ONE, T>(P, S, b, smem, rank, R, acc, q_sum);
            __syncthreads();
            // SSD step: four numbers of the state a lane; the sum over them goes from lane to lane in order
            struct Chan { int r, ch, hl; float skip; float4 h; float4* to; };
            auto step = [&](auto n, Chan (&a)[decltype(n)::value]) {
                constexpr int N = decltype(n)::value;
                float y[N];
                float4 t[N];
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const float2 dd = reinterpret_cast<const float2*>(decay_s)[a[k].r * nh + a[k].hl];
                    const float delta = dd.x, decay = dd.y, input = xs[a[k].r * per + a[k].ch];
                    const float4 B = reinterpret_cast<const float4*>(bc + a[k].r * 32)[s_lane], C = reinterpret_cast<const float4*>(bc + a[k].r * 32 + 16)[s_lane];
                    float4& h = a[k].h;
                    h.x = __fadd_rn(__fmul_rn(decay, h.x), __fmul_rn(__fmul_rn(delta, B.x), input));
                    h.y = __fadd_rn(__fmul_rn(decay, h.y), __fmul_rn(__fmul_rn(delta, B.y), input));
                    h.z = __fadd_rn(__fmul_rn(decay, h.z), __fmul_rn(__fmul_rn(delta, B.z), input));
                    h.w = __fadd_rn(__fmul_rn(decay, h.w), __fmul_rn(__fmul_rn(delta, B.w), input));
                    t[k] = make_float4(__fmul_rn(h.x, C.x), __fmul_rn(h.y, C.y), __fmul_rn(h.z, C.z), __fmul_rn(h.w, C.w));
                    y[k] = __fmul_rn(a[k].skip, input);
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) {
#pragma unroll
                    for (int k = 0; k < N; ++k) {
                        const float z = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(y[k], t[k].x), t[k].y), t[k].z), t[k].w);
                        y[k] = __shfl_sync(0xffffffffu, z, (lane & ~3) + q);
                    }
                }
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    float* out = zs + a[k].r * per + a[k].ch;
                    if (s_lane == 0) *out = __fmul_rn(y[k], *out);
                    *a[k].to = a[k].h;
                }
            };
            if constexpr (ONE) {
                Chan a[2] = {{0, s_first, s_head[0], Dv[0], hv[0], state_of(s_first)}, {0, s_first + 8, s_head[1], Dv[1], hv[1], state_of(s_first + 8)}};
                if (s_first < per) step(std::integral_constant<int, 2>{}, a);         // (shares are multiples of sixteen channels)
                asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp >> 1)) : "memory");
                if (s_own < per) send_half(smem_u32(x1 + chan_lo + s_own), bar, zs[s_own], ctas, warp & 1);
            } else {
                auto chan_at = [&](int i, int& r, int& ch) {
                    while (ch >= per) { ch -= per; ++r; }
                    const int hl = heads_of[ch];
                    float4* st = reinterpret_cast<float4*>(b.ssm) + (static_cast<size_t>(row0 + r) * DI + chan_lo + ch) * 4 + s_lane;
                    Chan a{r, ch, hl, skip_s[hl], L.state >= 0 ? reinterpret_cast<const float4*>(smem + L.state)[4 * i + s_lane] : *st, st};
                    ch += T / 4;
                    return a;
                };
                int i = s_first, r = 0, ch = s_first;
#pragma unroll 1
                for (; i + T / 4 < R * per; i += T / 2) {
                    Chan a[2];
                    a[0] = chan_at(i, r, ch);
                    a[1] = chan_at(i + T / 4, r, ch);
                    step(std::integral_constant<int, 2>{}, a);
                }
                if (i < R * per) {
                    Chan a[1];
                    a[0] = chan_at(i, r, ch);
                    step(std::integral_constant<int, 1>{}, a);
                }
                __syncthreads();
#pragma unroll 1
                for (int i = tid, r = 0, ch = tid; i < R * per; i += T, ch += T) {
                    while (ch >= per) { ch -= per; ++r; }
                    send(smem_u32(x1 + r * DI + chan_lo + ch), bar, zs[i], ctas);
                }
            }
            if (warp == T / 32 - 1 && !last) fetch_block(bi + 1);
            if (hybrid) attend<ONE, T>(P, S, b, smem, rank, ctas, row0, R, smem_u32(x1 + R * DI), bar);
            pass = kPassB;
            continue;
        }
        if (pass == kPassC) {
            expect(P.d.ff);
            const int f_lo = own.ff.lo, f_own = size_of(own.ff);
            const Linear& v = b.lin[kUp];
#pragma unroll 1
            for (int i = tid; i < R * f_own; i += T) {
                const int r = ONE ? 0 : i / f_own, c = i - r * f_own;
                const float y = fmaxf(affine(acc[r * acc_stride + c], 0, r, v.scale, v.magnitude ? __ldg(v.magnitude + f_lo + c) : 1.0f, v.bias ? __ldg(v.bias + f_lo + c) : 0.0f), 0.0f);
                send(smem_u32(x1 + r * P.d.ff + f_lo + c), bar, __fmul_rn(y, y), ctas);
            }
            pass = kPassD;
            continue;
        }
        // ---- B and D: the residual stream of this CTA's rows, on its way to everybody unless this was the model's last pass ----
        const bool ends = pass == kPassD || !hybrid;
        if (!(ends && last)) expect(D);
        const Linear& v = b.lin[pass == kPassB ? kOut : kDown];
        const float* gate = pass == kPassD ? b.ffn_gate : (hybrid ? b.mamba_gate : nullptr);
#pragma unroll 1
        for (int i = ONE ? s_own : tid, r = 0, c = i; i < R * n_own; i += T, c += T) {
            if constexpr (!ONE)
                while (c >= n_own) { c -= n_own; ++r; }
            const int n = n_lo + c;
            float y = affine(acc[r * acc_stride + c], 0, r, v.scale, v.magnitude ? __ldg(v.magnitude + n) : 1.0f, v.bias ? __ldg(v.bias + n) : 0.0f);
            if (gate) y = __fmul_rn(y, __ldg(gate + n));
            if (pass == kPassB && hybrid) {
                const Linear& va = b.lin[kAttnOut];
                const float a = affine(acc[r * acc_stride + S.job[kPassB][1].acc + c], 1, r, va.scale, va.magnitude ? __ldg(va.magnitude + n) : 1.0f,
                                       va.bias ? __ldg(va.bias + n) : 0.0f);
                y = __fadd_rn(y, __fmul_rn(a, __ldg(b.attn_gate + n)));
            }
            y = __fadd_rn(ONE ? stream : x0[r * D + n], y);
            if (ONE) stream = y;
            if (!(ends && last)) {
                if constexpr (ONE) {
                    send_half(smem_u32(x0 + n), bar, y, ctas, warp & 1);
                } else {
                    send(smem_u32(x0 + r * D + n), bar, y, ctas);
                }
            }
            if (ends && (!ONE || (warp & 1) == 0)) {
                const size_t at = static_cast<size_t>(row0 + r) * D + n;
                if (last) P.hidden_out[at] = y;
                else if (P.trace) P.trace[static_cast<size_t>(bi + 1) * P.batch * D + at] = y;
            }
        }
        if (pass == kPassB && rank == 0) {
            // every CTA is past its convolution: the window of B and C moves on
#pragma unroll 1
            for (int i = T - 1 - tid; i < R * 32 * kTaps; i += T) {
                const int k = i / kTaps, j = i - k * kTaps;
                b.ring[static_cast<size_t>(row0 + (k >> 5)) * ring_row + j * conv_dim + DI + (k & 31)] = bcring[i];
            }
        }
        if (!ends) { pass = kPassC; continue; }
        if (last) break;
        pass = kPassA;
        ++bi;
    }
    if (P.advance && rank == 0 && tid < R) P.positions[row0 + tid] = S.pos[tid] + 1;
    // nobody leaves while a peer may still send to it
    if (!alive) __nanosleep(100000);
    cp_async_wait();
    __syncthreads();
    cluster_sync();
}

inline int round_up_int(int v, int a) { return (v + a - 1) / a * a; }

bool plain_view(const tbl_linear_view& v, int inputs, int outputs) {
    return v.strips && !(reinterpret_cast<uintptr_t>(v.strips) & 15) && v.packed && !(reinterpret_cast<uintptr_t>(v.packed) & 15) && !v.weight &&
           v.inputs == inputs && v.outputs == outputs && v.activation_bits == 8 && !v.rms_input && inputs % 256 == 0 && std::isfinite(v.weight_scale) &&
           v.weight_scale > 0.0f;
}
// CTA `rank`'s share
Owned owned(const Dims& d, int rank, int ctas) {
    auto share = [&](int n) { return Range{static_cast<uint16_t>(n * rank / ctas), static_cast<uint16_t>(n * (rank + 1) / ctas)}; };
    auto sixteens = [&](int n) { const Range r = share(n >> 4); return Range{static_cast<uint16_t>(r.lo * 16), static_cast<uint16_t>(r.hi * 16)}; };
    auto over = [](int lo, int hi) { return Range{static_cast<uint16_t>(lo), static_cast<uint16_t>(hi)}; };
    Owned o{};
    o.chan = sixteens(d.inner); o.row = sixteens(d.D); o.ff = sixteens(d.ff); o.attn = share(d.a_heads);
    o.head = over(o.chan.lo / d.d_head, (o.chan.hi - 1) / d.d_head + 1);
    if (size_of(o.attn)) {
        const int group = d.a_heads / d.a_kv_heads > 0 ? d.a_heads / d.a_kv_heads : 1;
        auto kv = [&](int h) { return h / group < d.a_kv_heads - 1 ? h / group : d.a_kv_heads - 1; };
        o.kv = over(kv(o.attn.lo), kv(o.attn.hi - 1) + 1);
    }
    return o;
}

bool aligned(const float* p) { return p && !(reinterpret_cast<uintptr_t>(p) & 15); }

Linear linear_of(const tbl_linear_view& v) { return Linear{static_cast<const uint8_t*>(v.strips), v.magnitude, v.bias, v.weight_scale, 0}; }

constexpr int kRoom = 227 * 1024 - (static_cast<int>(sizeof(Static)) + 127) / 128 * 128;     // dynamic shared memory of a CTA

// Shared memory of a CTA for `rows` sequences in clusters of `ctas`
Layout layout_with(const Dims& d, int rows, int ctas, int score_len, int room, bool partial_all) {
    Layout L{};
    const int D = d.D;
    auto share_max = [&](int n) { return (n + ctas - 1) / ctas; };
    auto larger = [](int a, int b) { return a > b ? a : b; };
    const int per = share_max(d.inner >> 4) * 16, nh = (per + d.d_head - 2) / d.d_head + 1;
    int own = 0, kv = 0;
    if (d.a_heads) {
        const int group = d.a_heads / d.a_kv_heads > 0 ? d.a_heads / d.a_kv_heads : 1;
        own = share_max(d.a_heads);
        kv = (own + group - 2) / group + 1 < d.a_kv_heads ? (own + group - 2) / group + 1 : d.a_kv_heads;
    }
    const int cols_a = 2 * per + 32 + round_up_int(nh + 15, 16) + (own + 2 * kv) * d.head_dim, rows_d = share_max(D >> 4) * 16, rows_f = share_max(d.ff >> 4) * 16;
    const int heads = d.a_heads ? D : 0;
    L.acc_stride = round_up_int(larger(larger(cols_a, 2 * rows_d), rows_f), 32) + 4;
    L.score_len = round_up_int(score_len, 4);
    L.pieces = (cols_a >> 4) * (D >> 8) + (rows_d >> 4) * ((d.inner + heads + d.ff) >> 8) + (rows_f >> 4) * (D >> 8);       // if every piece were one block
    long long off = 0;
    auto take = [&](long long bytes) { const long long at = off; off += (bytes + 127) / 128 * 128; return static_cast<int>(at < (1 << 28) ? at : 1 << 28); };
    L.x0 = take(4ll * rows * D);
    L.x1 = take(4ll * rows * larger(d.inner + heads, d.ff));
    // (MMA columns past the last sequence read on behind the codes)
    L.codes = take(static_cast<long long>(rows) * larger(larger(2 * D, d.inner + heads), d.ff) + kMaxRows * 256);
    L.acc = take(8ll * rows * L.acc_stride);
    L.xs = take(4ll * rows * per);
    L.zs = take(4ll * rows * per);
    L.bc = take(4ll * rows * 32);
    L.bcring = take(4ll * rows * 32 * kTaps);
    L.decay = take(8ll * rows * nh);
    L.skip = take(4ll * nh);
    L.heads_of = take(2ll * per);
    L.norm = take(4ll * larger(2 * D, d.inner));
    L.scores = take(4ll * rows * L.score_len);
    L.partial_all = partial_all;
    L.partial = take(d.a_heads ? (partial_all && rows > 2 ? 4096ll * rows : 512 * 16) : 0);
    L.qkv = take(4ll * rows * (own + 2 * kv) * d.head_dim);
    L.table = take(8ll * L.pieces);
    // several sequences: what their steps read of the state comes ahead of time where there is room
    L.state = L.taps = -1;
    const long long state = 64ll * rows * per, windows = 4ll * rows * kTaps * (per + 32);
    if (rows > 1 && off + state + windows + 256 <= room) { L.state = take(state); L.taps = take(windows); }
    L.total = static_cast<int>(off < (1 << 28) ? off : 1 << 28);
    return L;
}

// The dimensions all blocks of the model share; false: they do not, or some are not this kernel's
bool common_dims(const tbl_decode_model& m, int capacity, Dims* dims, int* score_len) {
    Dims d{};
    d.D = m.d_model;
    *score_len = 0;
    if (d.D % 256) return false;
    auto same = [](int& a, int b, bool first) { if (first) a = b; return a == b; };
    bool first_hybrid = true;
    for (int i = 0; i < m.n_blocks; ++i) {
        const tbl_decode_block& b = m.blocks[i];
        const tbl_mamba_block& mm = b.mamba;
        if (mm.d_state != 16 || mm.n_groups != 1 || mm.conv_kernel != kTaps + 1 || mm.d_inner % 256 || !aligned(b.core_norm_w) || !aligned(mm.norm_w)) return false;
        if (!same(d.inner, mm.d_inner, i == 0) || !same(d.n_heads, mm.n_heads, i == 0) || !same(d.d_head, mm.d_head, i == 0))
            return false;
        if (!plain_view(mm.x, d.D, mm.d_inner) || !plain_view(mm.z, d.D, mm.d_inner) || !plain_view(mm.B, d.D, 16) || !plain_view(mm.C, d.D, 16) ||
            !plain_view(mm.dt, d.D, mm.n_heads) || !plain_view(mm.out, mm.d_inner, d.D))
            return false;
        if (!b.hybrid) continue;
        const tbl_attention_block& a = b.attn;
        if (a.head_dim % 16 || a.head_dim > 128 || !aligned(b.attn_norm_w) || !aligned(b.ff_norm_w) || b.ffn_up.outputs % 256) return false;
        if (!same(d.ff, b.ffn_up.outputs, first_hybrid) || !same(d.a_heads, a.n_heads, first_hybrid) || !same(d.a_kv_heads, a.n_kv_heads, first_hybrid) ||
            !same(d.head_dim, a.head_dim, first_hybrid))
            return false;
        if (!plain_view(a.q, d.D, d.D) || !plain_view(a.kv, d.D, 2 * a.n_kv_heads * a.head_dim) || !plain_view(a.out, d.D, d.D) ||
            !plain_view(b.ffn_up, d.D, b.ffn_up.outputs) || !plain_view(b.ffn_down, b.ffn_up.outputs, d.D))
            return false;
        const int len = capacity < a.sliding_window ? capacity : a.sliding_window;
        if (len > *score_len) *score_len = len;
        first_hybrid = false;
    }
    *dims = d;
    return true;
}


// One sequence a cluster, and no row, share of channels or of heads longer than one sweep of the threads: straight code
bool one_sweep(const Dims& d, int rows, int ctas) {
    const int per = (d.inner / 16 + ctas - 1) / ctas * 16, longest = d.ff > d.inner ? d.ff : d.inner;
    return rows == 1 && longest <= 16 * 256 && per <= 128 && (d.D / 16 + ctas - 1) / ctas * 16 <= 128 && (per + d.d_head - 2) / d.d_head + 1 <= 32;
}

template <bool ONE, int T>
cudaError_t configure(int* max_clusters, int ctas, size_t smem) {
    static bool done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (!max_clusters && dev >= 0 && dev < 64 && done[dev]) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(decode_cluster_kernel<ONE, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, kRoom);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(decode_cluster_kernel<ONE, T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev] = true;
    if (e != cudaSuccess || !max_clusters) return e;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = ctas; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    cfg.gridDim = dim3(ctas); cfg.blockDim = dim3(T); cfg.dynamicSmemBytes = smem; cfg.attrs = &attr; cfg.numAttrs = 1;
    return cudaOccupancyMaxActiveClusters(max_clusters, decode_cluster_kernel<ONE, T>, &cfg);
}

}  // namespace

Layout layout_of(const Dims& d, int rows, int ctas, int score_len, int room) {
    const Layout L = layout_with(d, rows, ctas, score_len, room, true);
    return L.total <= room ? L : layout_with(d, rows, ctas, score_len, room, false);
}

// How many clusters of `ctas` run at once on this device
int clusters_at_once(int ctas) {
    static int known[64][2] = {};
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    int& k = known[dev][ctas == 16];
    if (k) return k;
    if (configure<true, kOneThreads>(&n, ctas, 120 * 1024) != cudaSuccess) { cudaGetLastError(); return 0; }
    return k = n;
}

// Whether clusters of this shape still pay over `len` cached tokens.  Here a CTA attends for its heads and all its cluster's sequences, by itself; separate
// launches have a block per head and sequence, on every SM: us a cached token on the busiest SM, by 64-wide heads, fitted to widths of 256 to 2048, batches
// of 1 to 256 and 64 to 10000 tokens.  Against that stands what a step over few tokens is shorter by, a block: 10 to 14 us, 18 to 30 from width 1024 on where
// a CTA's share of the weights is small; past 64 sequences 50 and more, 23 to 50.  us a step, clusters and launches, width 768, 16 blocks of which two
// attend: 64 sequences, 1084 tokens 807 and 848, 1284 864 and 866, 2000 1082 and 973, 3000 1377 and 1123; 48, 1684 740 and 816, 3000 981 and 959; 32, 2584 759 and 780,
// 3000 823 and 814.  A cache is taken to be as full as it can get: a step's positions are on the device.
bool context_pays(const Dims& d, int rows, int ctas, int waves, int batch, int len, int attending, int n_blocks, long long share) {
    const double heads = d.head_dim / 64.0, here = 0.0145 * rows * ((d.a_heads + ctas - 1) / ctas) * waves * heads, there = 0.0175 + 7.2e-5 * batch * d.a_heads * heads;
    const double lead = batch > 64 ? (d.D >= 1024 ? 25.0 : 50.0) : (d.D >= 1024 && share <= 256 * 1024 ? 18.0 : 10.0);
    return attending * len * (here - there) <= lead * n_blocks;
}

// Clusters of sixteen CTAs (seven at once on a B200, up to eight sequences each) where they hold the batch, else of eight (fifteen at once); as few
// sequences a cluster as lets all run at once.  A CTA streams its share of the weights by itself, so that wide models are better off with every SM at
// every matrix, one launch each: us a step of 8 blocks at batch 1 / 7 / 16, this kernel and separate launches, by width: 1536 256 / 271 / 284 and 330 / 407 /
// 490; 2048 359 / 347 / 386 and 421 / 556 / 619; 3072 735 / 674 / 2799 and 706 / 759 / 844; 4096 1263 / 1131 / - and 869 / 944 / 1065; in clusters of
// eight, 60 sequences of 1024 290 and 442, 40 of 1280 378 and 468, 64 of 1536 871 and 609.  Hence the line at 400 KB of a block's three large matrices.  Several waves of
// clusters only where the separate launches leave their GEMV and GEMM of up to 64 rows (768: batch 100 680 and 1841, batch 1024 7018 and 16807).
bool decode_cluster_shape(const tbl_decode_model& m, int batch, int capacity, ClusterShape* shape) {
    Dims d;
    int score_len, attending = 0;
    if (!common_dims(m, capacity, &d, &score_len)) return false;
    for (int i = 0; i < m.n_blocks; ++i) attending += m.blocks[i].hybrid != 0;
    // the parts that gemv_strip_kernel takes a row's sum of squares in: more than sum_parts() has places for
    if (batch <= gemv_strip_fused_rows(d.D) && sum_strips_parts(d.D) > kStripParts) return false;
    for (int ctas = 16; ctas >= 8; ctas >>= 1) {
        const int most = clusters_at_once(ctas);
        if (most <= 0) continue;
        int rows = (batch + most - 1) / most;
        if (rows > kMaxRows) {
            if (ctas == 16) continue;
            rows = kMaxRows;
        }
        Layout L = layout_of(d, rows, ctas, score_len, kRoom);
        while (L.total > kRoom && rows > 1 && ctas == 8) L = layout_of(d, --rows, ctas, score_len, kRoom);
        const int waves = (batch + rows * most - 1) / (rows * most);
        const long long share = 3ll * d.D * d.inner / 4 / ctas;
        if (share > (waves > 1 ? 200 : 400) * 1024 || (waves > 1 && batch <= 64)) continue;
        if (waves > 1) {
            rows = (batch + waves * most - 1) / (waves * most);
            L = layout_of(d, rows, ctas, score_len, kRoom);
        }
        // limits: what the separate launches refuse, shared memory, the fields of the table of pieces, an mbarrier's byte count
        if (d.inner > 16 * 1024 || d.ff > 32768 || L.total > kRoom || L.acc_stride > 32767 || L.x1 - L.x0 > 1 << 19 || L.codes - L.x1 > 1 << 19) continue;
        if (!context_pays(d, rows, ctas, waves, batch, score_len, attending, m.n_blocks, share)) continue;
        shape->ctas = ctas; shape->rows = rows; shape->clusters = (batch + rows - 1) / rows; shape->smem = L.total;
        return true;
    }
    return false;
}

cudaError_t launch_decode_cluster(const tbl_decode_model& m, const ClusterShape& shape, int batch, int capacity, const ClusterBlockState* state,
                                  int32_t* positions, const int32_t* token_ids, float* hidden_out, float* trace, int* status, cudaStream_t st) {
    Params P{};
    int score_len;
    if (!common_dims(m, capacity, &P.d, &score_len)) return cudaErrorInvalidValue;
    const bool one = one_sweep(P.d, shape.rows, shape.ctas);
    cudaError_t e = one ? configure<true, kOneThreads>(nullptr, 0, 0) : configure<false, kRowsThreads>(nullptr, 0, 0);
    if (e != cudaSuccess) return e;
    // the orders of the kernels of the general route
    P.row_order = batch <= gemv_strip_fused_rows(P.d.D) ? kSumStrips : kSumStrided;
    P.gate_share = (P.d.inner + 7) / 8;
    P.gate_order = P.gate_share + 32 <= 256 ? kSumClusters : kSumStrided;
    P.batch = batch; P.rows = shape.rows; P.capacity = capacity; P.vocab = m.vocab;
    P.embedding = m.embedding; P.hidden_out = hidden_out; P.positions = positions; P.status = status;
    P.L = layout_of(P.d, shape.rows, shape.ctas, score_len, kRoom);
    for (int i = 0; i < shape.ctas; ++i) P.own[i] = owned(P.d, i, shape.ctas);
    for (int first = 0; first < m.n_blocks; first += kMaxBlocks) {
        P.n_blocks = m.n_blocks - first < kMaxBlocks ? m.n_blocks - first : kMaxBlocks;
        P.ids = first == 0 ? token_ids : nullptr;
        P.hidden_in = first == 0 ? nullptr : hidden_out;
        P.trace = trace ? trace + static_cast<size_t>(first) * batch * m.d_model : nullptr;
        P.advance = first + P.n_blocks == m.n_blocks;
        for (int i = 0; i < P.n_blocks; ++i) {
            const tbl_decode_block& s = m.blocks[first + i];
            const tbl_mamba_block& mm = s.mamba;
            Block& b = P.blk[i];
            b = Block{};
            b.lin[kX] = linear_of(mm.x); b.lin[kZ] = linear_of(mm.z); b.lin[kB] = linear_of(mm.B); b.lin[kC] = linear_of(mm.C);
            b.lin[kDt] = linear_of(mm.dt); b.lin[kOut] = linear_of(mm.out);
            b.core_norm_w = s.core_norm_w; b.A_log = mm.A_log; b.D = mm.D; b.conv_w = mm.conv_w; b.conv_b = mm.conv_b; b.norm_w = mm.norm_w;
            b.ring = state[first + i].ring; b.ssm = state[first + i].ssm; b.k_cache = state[first + i].k_cache; b.v_cache = state[first + i].v_cache;
            b.core_eps = s.core_norm_eps; b.norm_eps = mm.norm_eps;
            b.hybrid = s.hybrid != 0;
            if (!s.hybrid) continue;
            const tbl_attention_block& a = s.attn;
            b.lin[kQ] = linear_of(a.q); b.lin[kKv] = linear_of(a.kv); b.lin[kAttnOut] = linear_of(a.out);
            b.lin[kUp] = linear_of(s.ffn_up); b.lin[kDown] = linear_of(s.ffn_down);
            b.attn_norm_w = s.attn_norm_w; b.ff_norm_w = s.ff_norm_w; b.mamba_gate = s.mamba_gate; b.attn_gate = s.attn_gate; b.ffn_gate = s.ffn_gate;
            b.rope_cos = a.rope_cos; b.rope_sin = a.rope_sin; b.window = a.sliding_window; b.rope_positions = a.rope_positions;
        }
        cudaLaunchConfig_t cfg{};
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = shape.ctas; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
        cfg.gridDim = dim3(shape.ctas * shape.clusters); cfg.blockDim = dim3(one ? kOneThreads : kRowsThreads); cfg.dynamicSmemBytes = shape.smem; cfg.stream = st;
        cfg.attrs = &attr; cfg.numAttrs = 1;
        e = one ? cudaLaunchKernelEx(&cfg, decode_cluster_kernel<true, kOneThreads>, P) : cudaLaunchKernelEx(&cfg, decode_cluster_kernel<false, kRowsThreads>, P);
        note_launch();
        if (e != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

}  // namespace tbl
