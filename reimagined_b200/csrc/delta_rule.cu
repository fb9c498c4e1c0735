// The generalized delta rule (per head: S <- diag(w) S - (a*u)(u^T S) + k v^T, o = S^T r) with its decays, removal
// rates, unit keys, head norm and output gate.  Everything here is fp32; states are stored [head][value][key].
//
// A value column j of a state evolves on its own:  s_j <- w*s_j + (k v_j - (a*u) (u.s_j)),  o_j = r.s_j,  so the
// columns are spread over threads and CTAs and only the dot products over the keys cross lanes: eight or sixteen lanes
// share a column, each holding its groups of four keys in registers, and the arithmetic runs on packed fp32 pairs.
//
//   delta_records_kernel  turns the raw projections of two tokens into a record: everything a round of the scan multiplies
//                       with, once per head instead of once per block of columns.
//   delta_scan_kernel   a sequence of tokens, two per round: a CTA owns 8, 16 or 32 columns of a head.  A producer brings the
//                       records by bulk copies (or, of short sequences, eight make them), four warps walk them with the state in registers.
//   delta_step_kernel   one token: a CTA per head also computes the low-rank decay product, the head norm and the gate.
#include "stack.cuh"

namespace tbl {
namespace stack {
namespace {

using pair2 = unsigned long long;      // two packed fp32

__device__ __forceinline__ pair2 dup2(float v) { pair2 r; asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v)); return r; }
__device__ __forceinline__ pair2 make2(float a, float b) { pair2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void split2(pair2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ pair2 fma2(pair2 a, pair2 b, pair2 c) { pair2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ pair2 mul2(pair2 a, pair2 b) { pair2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ pair2 add2(pair2 a, pair2 b) { pair2 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ float sum2(pair2 v) { float a, b; split2(v, a, b); return a + b; }
__device__ __forceinline__ float sum8lanes(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    return v;
}

// The sums of eight columns over the LANES lanes that hold them, each in the order of sum8lanes: three exchanges that halve the number of values, then
// plain ones (nine for 32 lanes, where every column by itself takes five).  Lane l has the sum of column l % 8, bits reversed.
__device__ __forceinline__ constexpr int bits3(int n) { return (n & 1) << 2 | (n & 2) | (n & 4) >> 2; }
template <int LANES>
__device__ __forceinline__ float sum_columns8(const float* v, int lane) {
    float a[4], b[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = (lane & 1 ? v[i + 4] : v[i]) + __shfl_xor_sync(0xffffffffu, lane & 1 ? v[i] : v[i + 4], 1);
#pragma unroll
    for (int i = 0; i < 2; ++i) b[i] = (lane & 2 ? a[i + 2] : a[i]) + __shfl_xor_sync(0xffffffffu, lane & 2 ? a[i] : a[i + 2], 2);
    float r = (lane & 4 ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, lane & 4 ? b[0] : b[1], 4);
#pragma unroll
    for (int o = 8; o < LANES; o <<= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
    return r;
}

// Four keys of one column (key index c .. c+3, clipped at dim): state <-> registers.
__device__ __forceinline__ ulonglong2 load_state4(const float* col, int c, int dim) {
    if ((dim & 3) == 0) {
        if (c >= dim) return make_ulonglong2(0, 0);
        return *reinterpret_cast<const ulonglong2*>(col + c);
    }
    const float a = c < dim ? col[c] : 0.0f, b = c + 1 < dim ? col[c + 1] : 0.0f;
    const float d = c + 2 < dim ? col[c + 2] : 0.0f, e = c + 3 < dim ? col[c + 3] : 0.0f;
    return make_ulonglong2(make2(a, b), make2(d, e));
}
__device__ __forceinline__ void store_state4(float* col, int c, int dim, ulonglong2 v) {
    if ((dim & 3) == 0) {
        if (c < dim) *reinterpret_cast<ulonglong2*>(col + c) = v;
        return;
    }
    float f[4];
    split2(v.x, f[0], f[1]);
    split2(v.y, f[2], f[3]);
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (c + i < dim) col[c + i] = f[i];
}

struct DeltaParams {
    const float* proj;       // [rows][ld]: r | k | v | g | a | w1 (raw products, biases added)
    const float* z;          // [rows][heads*dim] decay products W_w2 tanh(.) (scan kernel)
    const bf16* w2;          // [heads*dim][rank] (step kernel)
    const float* w0;         // [heads*dim]
    const float* norm;       // [heads*dim]
    float* states;           // [slots][heads][dim][dim]
    const int32_t* slots;
    float* o;                // [rows][heads*dim] raw readouts (scan kernel)
    float* records;          // [seq][head][round][record] (scan kernel)
    int* status;
    void* out;
    int ld, heads, dim, rank, n_tok;
    int seq0, tok0, some;    // scan kernel: first sequence and token of this launch, and how many tokens of each
    float rate, key_eps, eps;
    int w_computed;          // host: of w2, as in DenseCall
};

constexpr int kScanLanes = 8;          // groups of sixteen lanes in the consumer warps; each has NC value columns
// warps beside the four consumers: one that starts bulk copies, or as many to make records as there are registers for
__host__ __device__ constexpr int producers(int dkp, int nc, bool own) { return !own ? 1 : (dkp == 256 && nc == 4 ? 4 : 8); }
__host__ __device__ constexpr int scan_threads(int dkp, int nc, bool own) { return 32 * (4 + producers(dkp, nc, own)); }
constexpr int kStageRounds = 8;        // rounds per bulk copy
constexpr int kOwnTokens = 32;         // most tokens of a sequence whose records the scan makes itself

// The scan takes two tokens per round.  With w, u, q = a * u, k, r, v of the two tokens (0 and 1) and the state S before
// them, everything the round needs from S are four dot products per column, taken together:
//     d0 = u0.S,   e1 = (u1 w0).S,   p0 = (r0 w0).S,   p1 = (r1 w0 w1).S
// and the rest are products of the tokens with each other, the same for every column, which the producers work out:
//     d1 = e1 + (u1.k0) v0 - (u1.q0) d0
//     o0 = p0 + (r0.k0) v0 - (r0.q0) d0
//     o1 = p1 + (r1.w1 k0) v0 - (r1.w1 q0) d0 + (r1.k1) v1 - (r1.q1) d1
//     S  <- (w0 w1) S + (w1 k0) v0 - (w1 q0) d0 + k1 v1 - q1 d1
// An odd last token is followed by one that changes nothing (w = 1, the others 0).
template <int DKP>
struct Record {
    static constexpr int kScalars = 9 * DKP;                           // 12 products of the tokens with each other
    static constexpr int kValues = kScalars + 16;                      // v of both tokens
    static constexpr int kFloats = kValues + 2 * DKP;
    static constexpr int kStageBytes = 4 * kStageRounds * kFloats;
    static constexpr int kStages = DKP == 256 ? 2 : 4;                 // bulk copies on their way or in use
};
// Bytes of records at a time: longer sequences are scanned in pieces, more sequences in groups, so that the workspace stays small and
// the records mostly in the 126 MB of L2 (16 heads of 128: 1104 rounds of all heads; by twice the bytes 6001 tokens of 32 heads take
// 1577 us, by these 1584).
constexpr size_t kRecordBytes = size_t(96) << 20;
inline int padded_dim(int dim) { return dim <= 64 ? 64 : (dim <= 128 ? 128 : 256); }
inline size_t record_floats(int dim) { return 11 * static_cast<size_t>(padded_dim(dim)) + 16; }
// rounds of all heads at a time, at least a bulk copy's worth
inline int max_rounds(int heads, int dim) {
    const size_t n = kRecordBytes / (sizeof(float) * record_floats(dim) * heads);
    return n < kStageRounds ? kStageRounds : (n > 1000000 ? 1000000 : static_cast<int>(n));
}

__device__ __forceinline__ float pick4(const float (&v)[4], int n) {
    const float a = n & 1 ? v[1] : v[0], b = n & 1 ? v[3] : v[2];
    return n & 2 ? b : a;
}
__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float dot4(float4 a, float4 b, float c) { return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, c)))); }
// (a division good to two units in the last place)
__device__ __forceinline__ float sigmoid_near(float z) { return __fdividef(1.0f, 1.0f + expf(-z)); }

// The record of a head's tokens at row `at` and, where `second`, the one behind it, by one warp; lane l has channels 4l .. 4l + 3
// (+ 128).
template <int DKP>
__device__ __forceinline__ void make_record(const DeltaParams& p, int head, size_t at, bool second, float* rec) {
    using R = Record<DKP>;
    constexpr int NI = (DKP + 127) / 128;      // groups of four channels per lane
    const int lane = threadIdx.x & 31, dim = p.dim, HD = p.heads * dim;
    // every row and head starts on 16 bytes
    const bool vec = ((dim | p.ld) & 3) == 0 && ((reinterpret_cast<uintptr_t>(p.proj) | reinterpret_cast<uintptr_t>(p.w0)) & 15) == 0;
    auto load4 = [&](const float* base, int c, bool live) {
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (!live || c >= dim) return v;
        if (vec) return *reinterpret_cast<const float4*>(base + c);
        v.x = base[c];
        if (c + 1 < dim) v.y = base[c + 1];
        if (c + 2 < dim) v.z = base[c + 2];
        if (c + 3 < dim) v.w = base[c + 3];
        return v;
    };
    float4 r[2][NI], k[2][NI], u[2][NI], q[2][NI], w[2][NI], v[2][NI];
    float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        const bool live = s == 0 || second;
        const float* row = p.proj + (at + (live ? s : 0)) * p.ld + head * dim;
        const float* zr = p.z + (at + (live ? s : 0)) * HD + head * dim;
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const int c = 4 * lane + 128 * i;
            r[s][i] = load4(row, c, live);
            k[s][i] = load4(row + HD, c, live);
            v[s][i] = load4(row + 2 * HD, c, live);
            q[s][i] = load4(row + 4 * HD, c, live);
            w[s][i] = load4(zr, c, live);
        }
    }
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        s0 = dot4(k[0][i], k[0][i], s0);
        s1 = dot4(k[1][i], k[1][i], s1);
    }
    const float i0 = 1.0f / sqrtf(warp_sum(s0) + p.key_eps), i1 = 1.0f / sqrtf(warp_sum(s1) + p.key_eps);
    auto decay = [&](float z) { return expf(-p.rate * sigmoid_near(z)); };
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const float n = s ? i1 : i0;
            const float4 w0 = load4(p.w0 + head * dim, 4 * lane + 128 * i, true), a = q[s][i], z = w[s][i];
            u[s][i] = mul4(k[s][i], make_float4(n, n, n, n));
            q[s][i] = mul4(make_float4(sigmoid_near(a.x), sigmoid_near(a.y), sigmoid_near(a.z), sigmoid_near(a.w)), u[s][i]);
            w[s][i] = make_float4(decay(z.x + w0.x), decay(z.y + w0.y), decay(z.z + w0.z), decay(z.w + w0.w));
            if (s == 1 && !second) w[s][i] = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
        }
    float m[8] = {};
#pragma unroll
    for (int i = 0; i < NI; ++i) {
        const int c = 4 * lane + 128 * i;
        const float4 k0w = mul4(w[1][i], k[0][i]), q0w = mul4(w[1][i], q[0][i]), ww = mul4(w[0][i], w[1][i]);
        m[0] = dot4(r[0][i], k[0][i], m[0]); m[1] = dot4(r[0][i], q[0][i], m[1]);
        m[2] = dot4(r[1][i], k0w, m[2]);     m[3] = dot4(r[1][i], q0w, m[3]);
        m[4] = dot4(r[1][i], k[1][i], m[4]); m[5] = dot4(r[1][i], q[1][i], m[5]);
        m[6] = dot4(u[1][i], k[0][i], m[6]); m[7] = dot4(u[1][i], q[0][i], m[7]);
        if (c >= DKP) continue;
        *reinterpret_cast<float4*>(rec + c) = u[0][i];
        *reinterpret_cast<float4*>(rec + DKP + c) = mul4(u[1][i], w[0][i]);
        *reinterpret_cast<float4*>(rec + 2 * DKP + c) = mul4(r[0][i], w[0][i]);
        *reinterpret_cast<float4*>(rec + 3 * DKP + c) = mul4(r[1][i], ww);
        *reinterpret_cast<float4*>(rec + 4 * DKP + c) = ww;
        *reinterpret_cast<float4*>(rec + 5 * DKP + c) = k0w;
        *reinterpret_cast<float4*>(rec + 6 * DKP + c) = q0w;
        *reinterpret_cast<float4*>(rec + 7 * DKP + c) = k[1][i];
        *reinterpret_cast<float4*>(rec + 8 * DKP + c) = q[1][i];
        *reinterpret_cast<float4*>(rec + R::kValues + c) = v[0][i];
        *reinterpret_cast<float4*>(rec + R::kValues + DKP + c) = v[1][i];
    }
    // the eight products over the lanes: after three exchanges a lane holds one of them, number lane / 4
    float m4[4], m2[2];
#pragma unroll
    for (int e = 0; e < 4; ++e)
        m4[e] = (lane & 16 ? m[e + 4] : m[e]) + __shfl_xor_sync(0xffffffffu, lane & 16 ? m[e] : m[e + 4], 16);
#pragma unroll
    for (int e = 0; e < 2; ++e)
        m2[e] = (lane & 8 ? m4[e + 2] : m4[e]) + __shfl_xor_sync(0xffffffffu, lane & 8 ? m4[e] : m4[e + 2], 8);
    float m1 = (lane & 4 ? m2[1] : m2[0]) + __shfl_xor_sync(0xffffffffu, lane & 4 ? m2[0] : m2[1], 4);
    m1 += __shfl_xor_sync(0xffffffffu, m1, 2);
    m1 += __shfl_xor_sync(0xffffffffu, m1, 1);
    // token 0: factors of v0, d0, v1, d1; token 1: the same; then those of d1 (and nothing)
    float* sc = rec + R::kScalars;
    if ((lane & 3) == 0) {
        const int e = lane >> 2;
        sc[e < 2 ? e : e + 2] = m1;
        if (e < 2) sc[2 + e] = 0.0f;
    }
    if (lane < 6) sc[10 + lane] = 0.0f;
}

template <int DKP>
__global__ void __launch_bounds__(256) delta_records_kernel(const DeltaParams p, const int n_seq) {
    const int rounds = (p.some + 1) / 2;
    // neighbouring warps take neighbouring heads of the same tokens: their rows are one piece of memory
    const size_t unit = static_cast<size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    const int head = static_cast<int>(unit % p.heads);
    const size_t round = unit / p.heads;
    const int seq = static_cast<int>(round / rounds), t0 = 2 * static_cast<int>(round - static_cast<size_t>(seq) * rounds);
    pdl_launch_dependents();
    if (seq >= n_seq) return;
    pdl_wait();
    make_record<DKP>(p, head, static_cast<size_t>(p.seq0 + seq) * p.n_tok + p.tok0 + t0, t0 + 1 < p.some,
                     p.records + ((static_cast<size_t>(seq) * p.heads + head) * rounds + t0 / 2) * Record<DKP>::kFloats);
}

// What bounds it is a round's chain from the state through the dot products and their sums over sixteen lanes back to the
// state (350 ns a round at 16 columns, of which the vectors' way out of shared memory takes 160), so the columns are spread
// over as many SMs as there are, and whatever does not wait for the sums is done while they travel.  6001 tokens, 16 heads of
// 128: 1743 us with the records made by each block of columns for itself on 64 SMs, 1070 now and 75 for the records.
// Every wait is bounded.
// OWN: the records are not in memory, warps of the CTA make them where the bulk copies would leave them.
template <int DKP, int NC, bool OWN>
__global__ void __launch_bounds__(scan_threads(DKP, NC, OWN)) delta_scan_kernel(const DeltaParams p, const int stages) {
    using R = Record<DKP>;
    constexpr int COLS = kScanLanes * NC;      // value columns per CTA
    constexpr int G = DKP / 64;                // groups of four keys per consumer lane: 4 (l + 16 g), l = lane % 16
    extern __shared__ __align__(128) float sm[];
    __shared__ __align__(8) uint64_t full[R::kStages], empty[R::kStages];
    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int head = blockIdx.y, seq = blockIdx.z, j0 = blockIdx.x * COLS;
    const int dim = p.dim, HD = p.heads * dim;
    const int rounds = (p.some + 1) / 2, chunks = (rounds + kStageRounds - 1) / kStageRounds;
    const size_t row0 = static_cast<size_t>(p.seq0 + seq) * p.n_tok + p.tok0;
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) { mbar_init(&full[s], producers(DKP, NC, OWN)); mbar_init(&empty[s], 4); }
        fence_mbar_init();
        fence_proxy_async();
    }
    __syncthreads();
    pdl_launch_dependents();
    pdl_wait();
    if (OWN && warp >= 4) {
        for (int ch = 0; ch < chunks; ++ch) {
            const int s = ch % stages, n = min(kStageRounds, rounds - ch * kStageRounds);
            const bool alive = ch < stages || mbar_wait_bounded(&empty[s], ((ch / stages) - 1) & 1, p.status);
            if (!__all_sync(0xffffffffu, alive)) break;
            for (int i = warp - 4; i < n; i += producers(DKP, NC, OWN)) {
                const int t0 = 2 * (ch * kStageRounds + i);
                make_record<DKP>(p, head, row0 + t0, t0 + 1 < p.some, sm + static_cast<size_t>(s * kStageRounds + i) * R::kFloats);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
        }
        return;
    }
    if (warp == 4) {
        if (lane == 0) {
            const float* src = p.records + (static_cast<size_t>(seq) * p.heads + head) * rounds * R::kFloats;
            int ch = 0;
            bool alive = true;
            for (; ch < chunks; ++ch) {
                const int s = ch % stages, n = min(kStageRounds, rounds - ch * kStageRounds);
                if (ch >= stages) alive = mbar_wait_bounded(&empty[s], ((ch / stages) - 1) & 1, p.status);
                if (!alive) break;
                mbar_arrive_expect_tx(&full[s], 4 * n * R::kFloats);
                bulk_g2s(sm + s * kStageRounds * R::kFloats, src + static_cast<size_t>(ch) * kStageRounds * R::kFloats, 4 * n * R::kFloats, &full[s]);
            }
            if (!alive)                                    // nobody else may be waiting for the copies in flight
                for (int j = max(0, ch - stages); j < ch; ++j) mbar_wait_bounded(&full[j % stages], (j / stages) & 1, p.status);
        }
        return;
    }
    // ---- consumers: sixteen lanes share the keys of NC columns ----
    const int l = lane & 15, base = lane & 16, cl = (2 * warp + (base >> 4)) * NC;       // first of this lane's columns within the CTA
    float* st = p.states + (static_cast<size_t>(p.slots[p.seq0 + seq]) * p.heads + head) * dim * dim;
    ulonglong2 S[NC][G];
#pragma unroll
    for (int n = 0; n < NC; ++n)
#pragma unroll
        for (int g = 0; g < G; ++g)
            S[n][g] = j0 + cl + n < dim ? load_state4(st + static_cast<size_t>(j0 + cl + n) * dim, 4 * (l + 16 * g), dim) : make_ulonglong2(0, 0);
    // after the sums over the lanes, lane l holds dot product l / 4 of column l % 4 * NC / 4: lanes 8 .. 15 finish the two readouts
    constexpr int STEP = 4 / NC;                           // lanes that hold the same sum
    const int mine = (l & 3) / STEP, token = (l >> 2) & 1;
    const bool writes = l >= 8 && l % STEP == 0 && j0 + cl + mine < dim;
    float* o = p.o + (row0 + token) * HD + head * dim + j0 + cl + mine;
    auto pick = [&](const float (&v)[NC]) {
        if constexpr (NC == 4) return pick4(v, mine);
        else if constexpr (NC == 2) return mine ? v[1] : v[0];
        else return v[0];
    };
    for (int ch = 0; ch < chunks; ++ch) {
        const int b = ch % stages;
        const bool alive = mbar_wait_bounded(&full[b], (ch / stages) & 1, p.status);
        if (!__all_sync(0xffffffffu, alive)) break;
        const int t0 = 2 * ch * kStageRounds, n_rounds = min(kStageRounds, rounds - ch * kStageRounds);
        constexpr int V = DKP / 4;                         // 16-byte units per vector
        ulonglong2 c[4][G];                                // the dot products' vectors, a round ahead
        auto load_dots = [&](int i) {
            const ulonglong2* q = reinterpret_cast<const ulonglong2*>(sm + static_cast<size_t>(b * kStageRounds + i) * R::kFloats) + l;
#pragma unroll
            for (int d = 0; d < 4; ++d)
#pragma unroll
                for (int g = 0; g < G; ++g) c[d][g] = q[d * V + 16 * g];
        };
        load_dots(0);
#pragma unroll 1
        for (int i = 0; i < n_rounds; ++i) {
            const float* rec = sm + static_cast<size_t>(b * kStageRounds + i) * R::kFloats;
            const ulonglong2* q = reinterpret_cast<const ulonglong2*>(rec) + l;
            float x[4][NC];
#pragma unroll
            for (int d = 0; d < 4; ++d) {
#pragma unroll
                for (int n = 0; n < NC; ++n) {
                    pair2 a = mul2(c[d][0].x, S[n][0].x), e = mul2(c[d][0].y, S[n][0].y);
#pragma unroll
                    for (int g = 1; g < G; ++g) { a = fma2(c[d][g].x, S[n][g].x, a); e = fma2(c[d][g].y, S[n][g].y, e); }
                    x[d][n] = sum2(add2(a, e));
                }
            }
            float v0[NC], v1[NC];
#pragma unroll
            for (int n = 0; n < NC; ++n) { v0[n] = rec[R::kValues + min(j0 + cl + n, DKP - 1)]; v1[n] = rec[R::kValues + DKP + min(j0 + cl + n, DKP - 1)]; }
            const float4 f = *reinterpret_cast<const float4*>(rec + R::kScalars + 4 * token);
            const float2 fd = *reinterpret_cast<const float2*>(rec + R::kScalars + 8);
            // what the update does not need the dot products for, while those are on their way through the lanes
            pair2 p0[NC], p1[NC];
#pragma unroll
            for (int n = 0; n < NC; ++n) { p0[n] = dup2(v0[n]); p1[n] = dup2(v1[n]); }
            ulonglong2 q0[G], q1[G];
#pragma unroll
            for (int g = 0; g < G; ++g) {
                const ulonglong2 w = q[4 * V + 16 * g], k0 = q[5 * V + 16 * g], k1 = q[7 * V + 16 * g];
                q0[g] = q[6 * V + 16 * g];
                q1[g] = q[8 * V + 16 * g];
#pragma unroll
                for (int n = 0; n < NC; ++n) {
                    S[n][g].x = fma2(k1.x, p1[n], fma2(k0.x, p0[n], mul2(w.x, S[n][g].x)));
                    S[n][g].y = fma2(k1.y, p1[n], fma2(k0.y, p0[n], mul2(w.y, S[n][g].y)));
                }
            }
            if (i + 1 < n_rounds) load_dots(i + 1);
            float y[2][NC], z[NC], r;
#pragma unroll
            for (int d = 0; d < 2; ++d)
#pragma unroll
                for (int n = 0; n < NC; ++n) y[d][n] = (l & 8 ? x[d + 2][n] : x[d][n]) + __shfl_xor_sync(0xffffffffu, l & 8 ? x[d][n] : x[d + 2][n], 8);
#pragma unroll
            for (int n = 0; n < NC; ++n) z[n] = (l & 4 ? y[1][n] : y[0][n]) + __shfl_xor_sync(0xffffffffu, l & 4 ? y[0][n] : y[1][n], 4);
            if constexpr (NC == 4) {
                float h[2];
#pragma unroll
                for (int n = 0; n < 2; ++n) h[n] = (l & 2 ? z[n + 2] : z[n]) + __shfl_xor_sync(0xffffffffu, l & 2 ? z[n] : z[n + 2], 2);
                r = (l & 1 ? h[1] : h[0]) + __shfl_xor_sync(0xffffffffu, l & 1 ? h[0] : h[1], 1);
            } else {
                if constexpr (NC == 2) r = (l & 2 ? z[1] : z[0]) + __shfl_xor_sync(0xffffffffu, l & 2 ? z[0] : z[1], 2);
                else r = z[0] + __shfl_xor_sync(0xffffffffu, z[0], 2);
                r += __shfl_xor_sync(0xffffffffu, r, 1);
            }
            float d0[NC], d1[NC];
#pragma unroll
            for (int n = 0; n < NC; ++n) {
                d0[n] = __shfl_sync(0xffffffffu, r, base + n * STEP);
                d1[n] = __shfl_sync(0xffffffffu, r, base + 4 + n * STEP);
            }
#pragma unroll
            for (int n = 0; n < NC; ++n) d1[n] = fmaf(fd.x, v0[n], fmaf(-fd.y, d0[n], d1[n]));
            pair2 m0[NC], m1[NC];
#pragma unroll
            for (int n = 0; n < NC; ++n) { m0[n] = dup2(-d0[n]); m1[n] = dup2(-d1[n]); }
#pragma unroll
            for (int g = 0; g < G; ++g)
#pragma unroll
                for (int n = 0; n < NC; ++n) {
                    S[n][g].x = fma2(q1[g].x, m1[n], fma2(q0[g].x, m0[n], S[n][g].x));
                    S[n][g].y = fma2(q1[g].y, m1[n], fma2(q0[g].y, m0[n], S[n][g].y));
                }
            const float out = fmaf(f.x, pick(v0), fmaf(-f.y, pick(d0), fmaf(f.z, pick(v1), fmaf(-f.w, pick(d1), r))));
            if (writes && t0 + 2 * i + token < p.some) o[static_cast<size_t>(t0 + 2 * i) * HD] = out;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[b]);
    }
#pragma unroll
    for (int n = 0; n < NC; ++n)
#pragma unroll
        for (int g = 0; g < G; ++g)
            if (j0 + cl + n < dim) store_state4(st + static_cast<size_t>(j0 + cl + n) * dim, 4 * (l + 16 * g), dim, S[n][g]);
}

// tanh of the low-rank decay projection, in the precision's type, for the GEMM with W_w2
template <typename T>
__global__ void __launch_bounds__(256) delta_tanh_kernel(const float* __restrict__ proj, int ld, int offset, int rows, int rank,
                                                         int ldt, T* __restrict__ out) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t i = static_cast<size_t>(blockIdx.x) * 256 + threadIdx.x;
    const size_t row = i / rank;
    const int c = static_cast<int>(i - row * rank);
    if (row < static_cast<size_t>(rows)) out[row * ldt + c] = from_f<T>(tanhf(proj[row * ld + offset + c]));
}

// head norm, weight and output gate of the scan's readouts: one warp per (row, head)
template <typename T>
__global__ void __launch_bounds__(256) delta_out_kernel(const DeltaParams p, int rows) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t unit = static_cast<size_t>(blockIdx.x) * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31, dim = p.dim, HD = p.heads * dim;
    if (unit >= static_cast<size_t>(rows) * p.heads) return;
    const size_t row = unit / p.heads;
    const int head = static_cast<int>(unit - row * p.heads);
    const float* o = p.o + row * HD + head * dim;
    const float* g = p.proj + row * p.ld + 3 * HD + head * dim;
    T* out = static_cast<T*>(p.out) + row * HD + head * dim;
    float ov[TBL_MAX_DELTA_DIM / 32], gv[TBL_MAX_DELTA_DIM / 32], ss = 0.0f;
#pragma unroll
    for (int i = 0; i < TBL_MAX_DELTA_DIM / 32; ++i) {
        const int c = lane + 32 * i;
        ov[i] = c < dim ? o[c] : 0.0f;
        gv[i] = c < dim ? g[c] : 0.0f;
        ss = fmaf(ov[i], ov[i], ss);
    }
    const float inv = 1.0f / sqrtf(warp_sum(ss) / static_cast<float>(dim) + p.eps);
#pragma unroll
    for (int i = 0; i < TBL_MAX_DELTA_DIM / 32; ++i) {
        const int c = lane + 32 * i;
        if (c < dim) out[c] = from_f<T>(ov[i] * inv * __ldg(p.norm + head * dim + c) * sigmoid_f(gv[i]));
    }
}

// ---- one token ------------------------------------------------------------------------------------------------------
// LANES lanes share a column, NCP columns of a group of lanes are in flight; a group's columns are its number + i * THREADS / LANES.
template <typename T, int DKP, int THREADS, int LANES, int NCP, int BLOCKS, bool FUSED>
__global__ void __launch_bounds__(THREADS, BLOCKS) delta_step_kernel(const DeltaParams p) {
    constexpr int G = DKP / (4 * LANES), GROUPS = THREADS / LANES, PASSES = DKP / (GROUPS * NCP);
    static_assert(NCP % 8 == 0 || LANES == 8, "columns are added eight at a time");
    static_assert(PASSES >= 1 && PASSES * GROUPS * NCP == DKP, "columns of a head");
    __shared__ __align__(16) float su[DKP], sw[DKP], sau[DKP], sk[DKP], sr[DKP], sv[DKP], so[DKP], part[FUSED ? THREADS : 1];
    extern __shared__ float st_tanh[];         // [rank]
    const int tid = threadIdx.x, lane = tid & 31;
    const int head = blockIdx.x, row = blockIdx.y;
    const int dim = p.dim, HD = p.heads * dim;
    pdl_launch_dependents();
    float* st = p.states + (static_cast<size_t>(p.slots[row]) * p.heads + head) * dim * dim;
    for (int e = tid * 32; e < dim * dim; e += THREADS * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(st + e));
    pdl_wait();
    const float* pr = p.proj + static_cast<size_t>(row) * p.ld;
    const int lg = tid & (LANES - 1), group = tid / LANES;
    ulonglong2 S[NCP][G];
    auto load_pass = [&](int ps) {
#pragma unroll
        for (int n = 0; n < NCP; ++n) {
            const int j = (ps * NCP + n) * GROUPS + group;
#pragma unroll
            for (int g = 0; g < G; ++g)
                S[n][g] = j < dim ? load_state4(st + static_cast<size_t>(j) * dim, 4 * (lg + LANES * g), dim) : make_ulonglong2(0, 0);
        }
    };
    // everything that depends on this step's projections is requested first, then the state
    const int hc = head * dim + tid;
    const bool ch = tid < dim;
    const float k_in = ch ? pr[HD + hc] : 0.0f, r_in = ch ? pr[hc] : 0.0f, v_in = ch ? pr[2 * HD + hc] : 0.0f;
    const float g_in = ch ? pr[3 * HD + hc] : 0.0f, a_in = ch ? pr[4 * HD + hc] : 0.0f;
    float z_in = !FUSED && ch ? p.z[static_cast<size_t>(row) * HD + hc] : 0.0f;
    float kn[DKP / 32];
#pragma unroll
    for (int i = 0; i < DKP / 32; ++i) kn[i] = lane + 32 * i < dim ? pr[HD + head * dim + lane + 32 * i] : 0.0f;
    load_pass(0);
    if constexpr (FUSED) {
        for (int e = tid; e < p.rank; e += THREADS) st_tanh[e] = tanhf(pr[5 * HD + e]);
        __syncthreads();
        // decay products: THREADS / DKP threads per channel
        constexpr int TPC = THREADS / DKP;
        const int c = tid / TPC, sub = tid % TPC;
        float z = 0.0f;
        if (c < dim) {
            const bf16* w2 = p.w2 + static_cast<size_t>(head * dim + c) * p.rank;
            if ((p.rank & 7) == 0) {
#pragma unroll 4
                for (int e = sub * 8; e < p.rank; e += TPC * 8) {
                    const uint4 w = __ldg(reinterpret_cast<const uint4*>(w2 + e));
                    z = fmaf(bf_lo(w.x), st_tanh[e], z); z = fmaf(bf_hi(w.x), st_tanh[e + 1], z);
                    z = fmaf(bf_lo(w.y), st_tanh[e + 2], z); z = fmaf(bf_hi(w.y), st_tanh[e + 3], z);
                    z = fmaf(bf_lo(w.z), st_tanh[e + 4], z); z = fmaf(bf_hi(w.z), st_tanh[e + 5], z);
                    z = fmaf(bf_lo(w.w), st_tanh[e + 6], z); z = fmaf(bf_hi(w.w), st_tanh[e + 7], z);
                }
            } else {
                for (int e = sub; e < p.rank; e += TPC) z = fmaf(to_f(w2[e]), st_tanh[e], z);
            }
        }
        part[tid] = z;
        __syncthreads();
        if (ch) {
#pragma unroll
            for (int s = 0; s < TPC; ++s) z_in += part[tid * TPC + s];
        }
    }
    float ss = 0.0f;                            // every warp takes the key's norm for itself
#pragma unroll
    for (int i = 0; i < DKP / 32; ++i) ss = fmaf(kn[i], kn[i], ss);
    const float inv_key = 1.0f / sqrtf(warp_sum(ss) + p.key_eps);
    if (tid < DKP) {
        const float u = k_in * inv_key;
        su[tid] = u;
        sk[tid] = k_in;
        sr[tid] = r_in;
        sv[tid] = v_in;
        sw[tid] = ch ? expf(-p.rate * sigmoid_f(z_in + __ldg(p.w0 + hc))) : 0.0f;
        sau[tid] = sigmoid_f(a_in) * u;
    }
    __syncthreads();
    const ulonglong2 *qu = reinterpret_cast<const ulonglong2*>(su) + lg, *qw = reinterpret_cast<const ulonglong2*>(sw) + lg,
                     *qa = reinterpret_cast<const ulonglong2*>(sau) + lg, *qk = reinterpret_cast<const ulonglong2*>(sk) + lg,
                     *qr = reinterpret_cast<const ulonglong2*>(sr) + lg;
#pragma unroll 1
    for (int ps = 0; ps < PASSES; ++ps) {
        asm volatile("" ::: "memory");         // the head's vectors stay in shared memory, not in registers across the passes
        if (ps > 0) load_pass(ps);
        float sums[NCP];
#pragma unroll
        for (int n = 0; n < NCP; ++n) {
            pair2 d = 0, e = 0;
#pragma unroll
            for (int g = 0; g < G; ++g) { d = fma2(qu[LANES * g].x, S[n][g].x, d); e = fma2(qu[LANES * g].y, S[n][g].y, e); }
            sums[n] = sum2(add2(d, e));
        }
        if constexpr (NCP % 8 == 0) {
#pragma unroll
            for (int b = 0; b < NCP; b += 8) {
                const float r = sum_columns8<LANES>(sums + b, lane);
#pragma unroll
                for (int n = 0; n < 8; ++n) sums[b + n] = __shfl_sync(0xffffffffu, r, bits3(n), LANES);
            }
        } else {
#pragma unroll
            for (int n = 0; n < NCP; ++n) sums[n] = sum8lanes(sums[n]);
        }
#pragma unroll
        for (int n = 0; n < NCP; ++n) {
            const int j = (ps * NCP + n) * GROUPS + group;
            const pair2 m = dup2(-sums[n]), vv = dup2(sv[j]);
            pair2 o = 0, f = 0;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                S[n][g].x = fma2(qw[LANES * g].x, S[n][g].x, fma2(qa[LANES * g].x, m, mul2(qk[LANES * g].x, vv)));
                S[n][g].y = fma2(qw[LANES * g].y, S[n][g].y, fma2(qa[LANES * g].y, m, mul2(qk[LANES * g].y, vv)));
                o = fma2(qr[LANES * g].x, S[n][g].x, o);
                f = fma2(qr[LANES * g].y, S[n][g].y, f);
                if (j < dim) store_state4(st + static_cast<size_t>(j) * dim, 4 * (lg + LANES * g), dim, S[n][g]);
            }
            sums[n] = sum2(add2(o, f));
        }
        if constexpr (NCP % 8 == 0) {
#pragma unroll
            for (int b = 0; b < NCP; b += 8) {
                const float r = sum_columns8<LANES>(sums + b, lane);
                if (lg < 8) so[(ps * NCP + b + bits3(lg)) * GROUPS + group] = r;
            }
        } else {
#pragma unroll
            for (int n = 0; n < NCP; ++n) {
                const float r = sum8lanes(sums[n]);
                if (lg == 0) so[(ps * NCP + n) * GROUPS + group] = r;
            }
        }
    }
    __syncthreads();
    float sq = 0.0f;
#pragma unroll
    for (int i = 0; i < DKP / 32; ++i) { const float v = so[lane + 32 * i]; sq = fmaf(v, v, sq); }   // zero past dim
    const float inv = 1.0f / sqrtf(warp_sum(sq) / static_cast<float>(dim) + p.eps);
    if (ch) static_cast<T*>(p.out)[static_cast<size_t>(row) * HD + hc] = from_f<T>(so[tid] * inv * __ldg(p.norm + hc) * sigmoid_f(g_in));
}

// From this many rows on W_w2 is one product over all of them instead of a part of every head's CTA.
constexpr int kStepFusedRows = 4;

// z = W_w2 tanh(low-rank part), fp32 [rows][heads*dim]
template <typename T>
int decay_products(const tbl_delta_mixer& m, const DeltaParams& p, int precision, int rows, T* th, float* z, cudaStream_t st) {
    const int HD = p.heads * p.dim, ldt = static_cast<int>(round_up(p.rank, 8));
    if (launch_dependent(delta_tanh_kernel<T>, dim3(ceil_div(static_cast<long long>(rows) * p.rank, 256)), dim3(256), 0, st, p.proj, p.ld, 5 * HD,
                         rows, p.rank, ldt, th) != cudaSuccess)
        return TBL_ERR_CUDA;
    DenseCall c{};
    c.x = th; c.w = static_cast<const bf16*>(m.decay_up.weight); c.ldx = ldt; c.M = rows; c.K = p.rank; c.N = HD;
    c.out_f32 = z; c.ldo = HD; c.w_computed = p.w_computed;
    return launch_dense(precision, kDenseAuto, c, st);
}

template <typename T, int DKP, int THREADS, int LANES, int NCP, int BLOCKS>
cudaError_t launch_step_d(const DeltaParams& p, dim3 grid, cudaStream_t st) {
    return p.z ? launch_dependent(delta_step_kernel<T, DKP, THREADS, LANES, NCP, BLOCKS, false>, grid, dim3(THREADS), 0, st, p)
               : launch_dependent(delta_step_kernel<T, DKP, THREADS, LANES, NCP, BLOCKS, true>, grid, dim3(THREADS), sizeof(float) * p.rank, st, p);
}

struct Workspace {
    float *z, *o, *records;
    void* th;
    size_t bytes;
};
Workspace carve(const tbl_delta_mixer& m, int precision, size_t rows, void* base) {
    Workspace w{};
    const size_t HD = static_cast<size_t>(m.heads) * m.dim, e = precision == TBL_BF16 ? 2 : 4;
    uint8_t* p = static_cast<uint8_t*>(base);
    auto take = [&](size_t bytes) { uint8_t* r = p + w.bytes; w.bytes += round_up(bytes, 256); return r; };
    w.z = reinterpret_cast<float*>(take(sizeof(float) * rows * HD));
    w.o = reinterpret_cast<float*>(take(sizeof(float) * rows * HD));
    w.th = take(e * rows * round_up(m.rank, 8));
    // (up to a round per row: a sequence of an odd number of tokens has half a round more)
    const size_t most = max_rounds(m.heads, m.dim);
    w.records = reinterpret_cast<float*>(take(sizeof(float) * record_floats(m.dim) * m.heads * (rows < most ? rows : most)));
    return w;
}

template <typename T>
int launch_step(const tbl_delta_mixer& m, DeltaParams p, int precision, int n_seq, void* ws, cudaStream_t st) {
    const dim3 grid(p.heads, n_seq);
    if (n_seq > 65535 || p.rank > 8192) return TBL_ERR_SHAPE;
    if (n_seq >= kStepFusedRows) {
        const Workspace w = carve(m, precision, n_seq, ws);
        const int rc = decay_products<T>(m, p, precision, n_seq, static_cast<T*>(w.th), w.z, st);
        if (rc != TBL_OK) return rc;
        p.z = w.z;
    }
    cudaError_t e;
    // Bound by the states' bytes once the heads fill the chip, by the chain through one head before that.  A few heads: all of a head's columns in flight
    // at once (at 128: 8 lanes a column, two blocks an SM).  More heads than fit at once: fewer columns and registers a thread and more blocks, so that
    // one block's sums and stores run under the others' loads.  us for heads x dim x sequences, with the decay products of 256 channels ahead
    // (before | after): 32x128x64 70.8 | 57.3 (states alone 41), 32x100x64 60.5 | 49.6, 32x128x16 23.7 | 22.1, 32x64x64 28.9 | 22.5, 12x64x64 15.4 | 11.9;
    // not below it: 32x128x4 11.3 | 14.9, 32x64x8 7.7 | 9.3.  Heads of 256 with a warp a column need no spills: 16x256x32 68.9 | 59.8, 8x256x1 15.1 | 13.0.
    const long long heads = static_cast<long long>(p.heads) * n_seq;
    if (p.dim <= 32) e = launch_step_d<T, 32, 256, 8, 1, 1>(p, grid, st);
    else if (p.dim <= 64) e = heads > 4 * kNumSm ? launch_step_d<T, 64, 128, 8, 4, 6>(p, grid, st) : launch_step_d<T, 64, 256, 8, 2, 1>(p, grid, st);
    else if (p.dim <= 128) e = heads > 2 * kNumSm ? launch_step_d<T, 128, 256, 8, 1, 4>(p, grid, st) : launch_step_d<T, 128, 256, 8, 4, 2>(p, grid, st);
    else e = launch_step_d<T, 256, 512, 32, 8, 1>(p, grid, st);
    return e == cudaSuccess ? TBL_OK : TBL_ERR_CUDA;
}

template <int DKP>
int scan_stages(int tokens) {
    const int chunks = ceil_div((tokens + 1) / 2, kStageRounds);
    return chunks < Record<DKP>::kStages ? chunks : Record<DKP>::kStages;
}
// CTAs of the scan that run at once: one or two to an SM, by shared memory.  (Short sequences leave room for more, but gain
// nothing by it: 16 heads of 128, 24 tokens, 17.5 us by 128 CTAs of 16 columns and 22.5 by 256 of eight.)
constexpr int scan_room(int dkp) { return dkp <= 64 ? 2 * kNumSm : kNumSm; }

template <int DKP, int NC, bool OWN>
int launch_scan_n(const DeltaParams& p, int n_seq, cudaStream_t st) {
    static bool done[64] = {};
    using R = Record<DKP>;
    const int stages = scan_stages<DKP>(p.some);
    if (allow_smem(delta_scan_kernel<DKP, NC, OWN>, static_cast<size_t>(R::kStages) * R::kStageBytes, done) != cudaSuccess) return TBL_ERR_CUDA;
    const dim3 grid(ceil_div(p.dim, kScanLanes * NC), p.heads, n_seq);
    if (!OWN) {
        const long long units = static_cast<long long>(n_seq) * p.heads * ((p.some + 1) / 2);
        if (launch_dependent(delta_records_kernel<DKP>, dim3(ceil_div(units, 8)), dim3(256), 0, st, p, n_seq) != cudaSuccess) return TBL_ERR_CUDA;
    }
    return launch_dependent(delta_scan_kernel<DKP, NC, OWN>, grid, dim3(scan_threads(DKP, NC, OWN)), static_cast<size_t>(stages) * R::kStageBytes, st, p,
                            stages) == cudaSuccess ? TBL_OK : TBL_ERR_CUDA;
}

template <int DKP>
int launch_scan_d(const DeltaParams& p, int n_seq, cudaStream_t st) {
    // Narrow blocks of columns take less time a round (2000 tokens of 128 channels by 32, 16 and 8 columns: 8 heads 463, 364
    // and 305 us, in one wave each), a second wave of CTAs as long again (16 heads 480, 380 and 580; 32 heads 547, 766 and
    // 1159), and two to an SM a fifth longer than one.
    constexpr int room = scan_room(DKP);
    auto cost = [&](int cols, int us) {
        const long long ctas = static_cast<long long>(ceil_div(p.dim, cols)) * p.heads * n_seq;
        return (ctas > kNumSm && room > kNumSm ? 6 : 5) * us * ((ctas + room - 1) / room);
    };
    const long long wide = cost(32, 480), half = cost(16, 380), narrow = cost(8, 305);
    const int cols = narrow <= half && narrow <= wide ? 8 : (half <= wide ? 16 : 32);
    // Records made in place take no launch of their own and no way through memory, but are made once per block of columns: 16
    // heads of 128, 2, 16, 28 and 33 tokens 8.9, 15.5, 17.3 and 19.0 us, from memory 10.8, 18.5, 19.7 and 18.1; in more than one wave
    // (8 such sequences, 16 tokens) 35.3 and 27.1.
    const bool own = p.n_tok <= kOwnTokens && static_cast<long long>(ceil_div(p.dim, cols)) * p.heads * n_seq <= kNumSm;
    if (cols == 8) return own ? launch_scan_n<DKP, 1, true>(p, n_seq, st) : launch_scan_n<DKP, 1, false>(p, n_seq, st);
    if (cols == 16) return own ? launch_scan_n<DKP, 2, true>(p, n_seq, st) : launch_scan_n<DKP, 2, false>(p, n_seq, st);
    return own ? launch_scan_n<DKP, 4, true>(p, n_seq, st) : launch_scan_n<DKP, 4, false>(p, n_seq, st);
}

template <typename T>
int launch_scan(const tbl_delta_mixer& m, DeltaParams p, int precision, int n_seq, void* ws, cudaStream_t st) {
    if (p.heads > 65535 || n_seq > 65535) return TBL_ERR_SHAPE;
    const int rows = n_seq * p.n_tok;
    const Workspace w = carve(m, precision, rows, ws);
    p.o = w.o;
    int rc = decay_products<T>(m, p, precision, rows, static_cast<T*>(w.th), w.z, st);
    if (rc != TBL_OK) return rc;
    p.z = w.z;
    p.records = w.records;
    p.status = device_status_ptr();
    if (!p.status) return TBL_ERR_CUDA;
    // Whole sequences, as many as there is room for (in whole waves of blocks of 32 columns), or, where that would leave SMs
    // idle, pieces of enough sequences side by side: a scan takes as long by itself (4 sequences of 1100 tokens, 8 heads of
    // 128, one after the other: 659 us).
    const int rounds = (p.n_tok + 1) / 2, most = max_rounds(p.heads, p.dim);
    const int room = static_cast<int>(scan_room(padded_dim(p.dim)) / (static_cast<long long>(ceil_div(p.dim, 32)) * p.heads)), side = room < 1 ? 1 : room;
    int group = most / rounds, piece = p.n_tok;
    if (group >= n_seq) {
        group = n_seq;
    } else if (group >= side) {
        group -= group % side;
    } else {
        group = side < n_seq ? side : n_seq;
        const int per = most / group / kStageRounds * kStageRounds;
        piece = 2 * (per < kStageRounds ? kStageRounds : per);
    }
    for (p.seq0 = 0; p.seq0 < n_seq; p.seq0 += group) {
        const int n = n_seq - p.seq0 < group ? n_seq - p.seq0 : group;
        for (p.tok0 = 0; p.tok0 < p.n_tok; p.tok0 += piece) {
            p.some = p.n_tok - p.tok0 < piece ? p.n_tok - p.tok0 : piece;
            if (p.dim <= 64) rc = launch_scan_d<64>(p, n, st);
            else if (p.dim <= 128) rc = launch_scan_d<128>(p, n, st);
            else rc = launch_scan_d<256>(p, n, st);
            if (rc != TBL_OK) return rc;
        }
    }
    const cudaError_t e = launch_dependent(delta_out_kernel<T>, dim3(ceil_div(static_cast<long long>(rows) * p.heads, 8)), dim3(256), 0, st, p, rows);
    return e == cudaSuccess ? TBL_OK : TBL_ERR_CUDA;
}

}  // namespace

int check_delta(const tbl_delta_mixer& m, int width) {
    if (m.heads <= 0 || m.dim <= 0 || m.dim > TBL_MAX_DELTA_DIM || m.rank <= 0) return TBL_ERR_SHAPE;
    const int HD = m.heads * m.dim;
    if (m.in.inputs != width || m.in.outputs != 5 * HD + m.rank || m.decay_up.inputs != m.rank || m.decay_up.outputs != HD ||
        m.out.inputs != HD || m.out.outputs != width)
        return TBL_ERR_SHAPE;
    if (!m.in.weight || !m.in.bias || !m.decay_up.weight || !m.decay_up.bias || !m.out.weight || !m.norm) return TBL_ERR_INVALID_ARG;
    return TBL_OK;
}

size_t delta_workspace(const tbl_delta_mixer& m, int precision, int rows) { return carve(m, precision, rows, nullptr).bytes; }

int launch_delta(const tbl_delta_mixer& m, int precision, int route, float eps, const float* proj, float* states,
                 const int32_t* slots, int n_seq, int n_tok, void* out, void* ws, int w_computed, cudaStream_t st) {
    DeltaParams p{};
    p.proj = proj; p.w2 = static_cast<const bf16*>(m.decay_up.weight); p.w0 = m.decay_up.bias; p.norm = m.norm;
    p.states = states; p.slots = slots; p.out = out; p.ld = m.in.outputs; p.heads = m.heads; p.dim = m.dim; p.rank = m.rank;
    p.n_tok = n_tok; p.rate = m.decay_rate; p.key_eps = m.key_eps; p.eps = eps; p.w_computed = w_computed;
    if (route == 0) route = n_tok == 1 ? 2 : 1;
    if (route == 2) {
        if (n_tok != 1) return TBL_ERR_SHAPE;
        return precision == TBL_BF16 ? launch_step<bf16>(m, p, precision, n_seq, ws, st) : launch_step<float>(m, p, precision, n_seq, ws, st);
    }
    if (route != 1) return TBL_ERR_INVALID_ARG;
    return precision == TBL_BF16 ? launch_scan<bf16>(m, p, precision, n_seq, ws, st) : launch_scan<float>(m, p, precision, n_seq, ws, st);
}

}  // namespace stack
}  // namespace tbl

using namespace tbl;
using namespace tbl::stack;

extern "C" {

size_t tbl_delta_workspace_bytes(const tbl_delta_mixer* mixer, int precision, int rows) {
    return mixer && rows > 0 ? delta_workspace(*mixer, precision, rows) : 0;
}

int tbl_delta_forward(const tbl_delta_mixer* mixer, int precision, int route, float eps, const float* proj_dev, float* states_dev,
                      const int32_t* slots_dev, int n_seq, int n_tok, void* out_dev, void* workspace_dev, size_t workspace_bytes,
                      void* stream) {
    if (!mixer || !proj_dev || !states_dev || !slots_dev || !out_dev || n_seq <= 0 || n_tok <= 0 ||
        (precision != TBL_F32 && precision != TBL_BF16))
        return TBL_ERR_INVALID_ARG;
    const int rc = check_delta(*mixer, mixer->in.inputs);
    if (rc != TBL_OK) return rc;
    if (!workspace_dev || workspace_bytes < delta_workspace(*mixer, precision, n_seq * n_tok)) return TBL_ERR_WORKSPACE;
    if ((reinterpret_cast<uintptr_t>(workspace_dev) & 255) || (reinterpret_cast<uintptr_t>(states_dev) & 15)) return TBL_ERR_ALIGNMENT;
    return launch_delta(*mixer, precision, route, eps, proj_dev, states_dev, slots_dev, n_seq, n_tok, out_dev, workspace_dev, 1,
                        static_cast<cudaStream_t>(stream));
}

}  // extern "C"
