// Recurrences with one decay per head and no correction (state space, matrix memory) over prompt portions, in segments of 128 tokens that all run at once.  With S
// the state before a segment, u_i = beta_i v_i, c_j the product of the decays of its tokens up to j and D(i, j) that of tokens i + 1 .. j:
//     o_j = c_j S^T q_j + sum_{i <= j} D(i, j) (q_j . k_i) u_i,     S <- c_end S + sum_i k_i (D(i, end) u_i)^T.
//   * segment_sums_kernel: a block per (segment, head, 64 columns) forms the segment's own end state, sum_i k_i (D(i, end) u_i)^T, and blocks in front of them, one
//     per (segment, key head), the products q_j . k_i, i up to the end of j's 16 tokens, which all heads of a group share;
//   * scan_prefix_kernel chains the segments' start states;
//   * segment_outputs_kernel: a block per (segment, head, 64 columns), a warp per 16 tokens: S^T q and the products times their decays times u.
// All of it are products on mma.sync with split operands (seq_chunk.cuh).  An operand that several warps need is split once and lies in shared memory; the other one comes
// from memory straight into the lanes that use it and is split there.  Decays are products of factors, never quotients or differences of logarithms: within 16 tokens as
// they come, beyond that D(i, j) = (those behind i in its 16) (whole 16s between) (those of j's 16 up to j).
// The matrix unit cuts its sums off, so a chain of six products (16 k) starts from zero, the small terms first, and is added to the sum by an addition that rounds.
// What bounds it: a third each the matrix unit (8 clk per m16n8k8 and SM quarter), the operands' way from L2 (170 KB a block of the outputs, in bursts where blocks begin
// together), and the latencies of a block's few phases, two blocks an SM.  Measured (40 heads over 5, 128 x 64, one sequence of 2048 tokens), with what the launches
// overlap taken off: 173 us 16 tokens at a time (records 30, two passes 48 + 76, their chain 26), 131 so (sums 46, chain 14, outputs 65).
// Numbers that are not finite: everything read and formed is watched, and what is marked is taken again by chunk_redo_kernel, as in seq_chunk.cu.
#include "seq_chunk.cuh"
#include <math.h>

namespace wf {
namespace seq {

namespace {

constexpr int SG = SCAN_CHUNK, SG_THREADS = 256, SG_COLS = 64, SG_BLK = SG / 16, SG_VECS = SG * (SG_COLS / 4) / SG_THREADS;
static_assert(SG == 128, "eight warps take 16 tokens each");
constexpr int SG_G = SG * SG;                                // floats of a segment's products q k
// An operand tile [up to 128 k][64 columns] in shared memory as pairs (hi, lo), split once for all warps that use it: rows of SG_US pairs, so that the 8-byte reads of
// half a warp (four rows two apart, four columns) meet different banks.
constexpr int SG_US = SG_COLS + 2;
// shared memory in floats: decay products and write strengths; D within each 16 tokens; the split tile; the values as they came (outputs) - or a segment's keys
constexpr int SG_DEC = 4 * SG + 2 * SG_BLK;                  // c within 16, behind within 16, raw or weights, write strengths; products of the 16s
constexpr int SG_DIAG = SG_BLK * 16 * 17;                    // [16s][j][i]
constexpr int SG_TILE = 2 * SG * SG_US;
__host__ __device__ constexpr int sg_sum_floats(int DS) { return SG_DEC + (SG_TILE > SG * (DS + 8) ? SG_TILE : SG * (DS + 8)); }
constexpr int SG_OUT_FLOATS = SG_DEC + SG_DIAG + SG_TILE + SG * SG_COLS;

struct SegArgs { int n; float *local, *prod; const float* start; };

// Where this block works: entry of the workspaces, first token, tokens
struct SegAt { int sq, seg, start, len; size_t entry; };
__device__ __forceinline__ SegAt sg_at(const Batch& b, int n) {
    SegAt a;
    a.sq = blockIdx.x / n; a.seg = blockIdx.x - a.sq * n;
    const int seq0 = b.seq_start[a.sq];
    a.start = seq0 + a.seg * SG;
    a.len = min(SG, b.seq_len[a.sq] - a.seg * SG);
    a.entry = (size_t)(seq0 / SG + a.sq + a.seg);
    return a;
}

// decays of one head's segment: a token's factor and write strength (threads of the first 128), requested early
struct SgDecay { float g = 1.f, bt = 1.f; };
__device__ __forceinline__ SgDecay sg_decay(const ChunkView& w, int H, int h, const SegAt& a) {
    SgDecay d;
    const size_t at = (size_t)(a.start + threadIdx.x) * H + h;
    if ((int)threadIdx.x < a.len) { d.g = w.decay[at]; if (w.beta) d.bt = w.beta[at]; }      // (a.len <= 128)
    return d;
}
__device__ __forceinline__ void sg_decay_put(const SgDecay& d, float* dec, float& watch) {
    if (threadIdx.x < SG) { dec[2 * SG + threadIdx.x] = d.g; dec[3 * SG + threadIdx.x] = d.bt; cr_watch(watch, d.g); }
}
// products: cum[j] within j's 16 up to j, suf[i] within i's 16 behind i, blk[16s]; DIAG: D within each 16
template <bool DIAG>
__device__ __forceinline__ void sg_decay_form(float* dec, float* diag) {
    float *cum = dec, *suf = dec + SG, *blk = dec + 4 * SG;
    const float* raw = dec + 2 * SG;
    const int tid = threadIdx.x;
    if (tid >= SG) return;
    const int bk = tid >> 4, i = tid & 15;
    float c = 1.f, s = 1.f;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const float g = raw[bk * 16 + j];
        if (j <= i) c *= g; else s *= g;
        if (DIAG) diag[(bk * 16 + j) * 17 + i] = j < i ? 0.f : s;
    }
    cum[tid] = c; suf[tid] = s;
    if (i == 15) blk[bk] = c;
}

// vector k of this thread: token (or key row) and first column
__device__ __forceinline__ int sg_row(int k) { return (threadIdx.x + k * SG_THREADS) / (SG_COLS / 4); }
__device__ __forceinline__ int sg_col() { return (threadIdx.x % (SG_COLS / 4)) * 4; }
__device__ __forceinline__ float4 sg_value(const DeltaDims& D, const ChunkView& w, const SegAt& a, int h, int c, int tk) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (tk >= a.len) return v;
    const float* row = w.qkv + (size_t)(a.start + tk) * w.ld + w.v_off + h * D.dv;
    auto one = [&](int x) { return x < D.dv ? row[x] : x == D.dv && D.ones_col ? 1.f : 0.f; };
    if (c + 4 <= D.dv && ((uintptr_t)(row + c) & 15) == 0) return *reinterpret_cast<const float4*>(row + c);
    v.x = one(c); v.y = one(c + 1); v.z = one(c + 2); v.w = one(c + 3);
    return v;
}
__device__ __forceinline__ void sg_put(uint32_t* tile, int row, int col, const float4& v) {
    uint4 x, y;
    cr_split(v.x, x.x, x.y); cr_split(v.y, x.z, x.w); cr_split(v.z, y.x, y.y); cr_split(v.w, y.z, y.w);
    uint4* to = reinterpret_cast<uint4*>(tile + 2 * (row * SG_US + col));
    to[0] = x; to[1] = y;
}
__device__ __forceinline__ void sg_watch4(float& watch, const float4& v) { cr_watch(watch, v.x); cr_watch(watch, v.y); cr_watch(watch, v.z); cr_watch(watch, v.w); }

// tot += A B over 16 k: A as two 8-k tiles of float values (accumulator order: columns 2 t and 2 t + 1 are k = t and t + 4), b(nt, s) the B operand of column
// tile nt and 8-k tile s.  Four column tiles side by side, so that no product waits for the one before it; of NT tiles the first nn are wanted.
template <int NT, typename B>
__device__ __forceinline__ void sg_step(float (&tot)[NT][4], const float (&x)[2][4], int nn, const B& b) {
    const CrA a0 = cr_a(x[0]), a1 = cr_a(x[1]);
#pragma unroll
    for (int n0 = 0; n0 < NT; n0 += 4) {
        if (n0 >= nn) break;
        CrB b0[4], b1[4];
        float d[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) { b0[i] = b(n0 + i, 0); b1[i] = b(n0 + i, 1); }
#pragma unroll
        for (int i = 0; i < 4; ++i) cr_mma0(d[i], a0.l, b0[i].h);
#pragma unroll
        for (int i = 0; i < 4; ++i) cr_mma(d[i], a0.h, b0[i].l);
#pragma unroll
        for (int i = 0; i < 4; ++i) cr_mma(d[i], a1.l, b1[i].h);
#pragma unroll
        for (int i = 0; i < 4; ++i) cr_mma(d[i], a1.h, b1[i].l);
#pragma unroll
        for (int i = 0; i < 4; ++i) cr_mma(d[i], a0.h, b0[i].h);
#pragma unroll
        for (int i = 0; i < 4; ++i) cr_mma(d[i], a1.h, b1[i].h);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) tot[n0 + i][e] += d[i][e];
    }
}
// rows k0 .. of a split tile
struct SgRows {
    const uint2* p;
    __device__ __forceinline__ SgRows(const uint32_t* tile, int k0, int c0, int g, int t) : p(reinterpret_cast<const uint2*>(tile) + (k0 + 2 * t) * SG_US + c0 + g) {}
    __device__ __forceinline__ CrB operator()(int nt, int s) const {
        const uint2 x = p[8 * s * SG_US + 8 * nt], y = p[(8 * s + 1) * SG_US + 8 * nt];
        CrB b;
        b.h[0] = x.x; b.l[0] = x.y; b.h[1] = y.x; b.l[1] = y.y;
        return b;
    }
};

__device__ __forceinline__ void sg_cp16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ void sg_next(float (&x)[2][4], const float (&y)[2][4]) {
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int e = 0; e < 4; ++e) x[s][e] = y[s][e];
}

// the 16 tokens of a warp: tiles w and 7 - w meet on one quarter of the SM, so that each quarter has as many products to form
__device__ __forceinline__ int sg_tile(int warp) { return warp < 4 ? warp : 11 - warp; }

__device__ __forceinline__ void sg_mark(const DeltaDims& D, const ChunkView& w, int sq, int h0, int heads) {
    for (int z = 0; z < heads * w.cols; ++z) w.redo[((size_t)sq * D.H + h0) * w.cols + z] = 1;
}

// blocks y < Hk: products q k of a key head -> rec [entry][Hk][128 j][128 i], columns up to the end of j's 16; the others: head y - Hk
template <int DS>
__global__ void __launch_bounds__(SG_THREADS, 2) segment_sums_kernel(Batch b, DeltaDims D, ChunkView w, SegArgs sg) {
    extern __shared__ __align__(16) float sm[];
    const SegAt a = sg_at(b, sg.n);
    if (a.len <= 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    float watch = 0.f;
    if ((int)blockIdx.y < D.Hk) {
        if (blockIdx.z) return;
        constexpr int KS = DS + 8;
        const int kh = blockIdx.y, tile = sg_tile(warp), j0 = 16 * tile + g;
        float* ks = sm;
        for (int i = tid; i < SG * (DS / 4); i += SG_THREADS) {
            const int r = i / (DS / 4), c = (i - r * (DS / 4)) * 4;
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < a.len && c < D.d) x = *reinterpret_cast<const float4*>(w.qkv + (size_t)(a.start + r) * w.ld + w.k_off + kh * D.d + c);
            cr_watch(watch, x.x); cr_watch(watch, x.y); cr_watch(watch, x.z); cr_watch(watch, x.w);
            *reinterpret_cast<float4*>(ks + r * KS + c) = x;
        }
        __syncthreads();
        if (16 * tile < a.len) {
            const float* q0 = w.qkv + (size_t)(a.start + j0) * w.ld + w.q_off + kh * D.d + 2 * t;
            const float* q1 = q0 + (size_t)8 * w.ld;
            const bool ok0 = j0 < a.len, ok1 = j0 + 8 < a.len;
            float* G = w.rec + (a.entry * D.Hk + kh) * SG_G + (size_t)j0 * SG + 2 * t;
            for (int n0 = 0; n0 <= tile; n0 += 4) {                       // 64 earlier tokens at a time
                float tot[8][4];
#pragma unroll
                for (int nt = 0; nt < 8; ++nt) tot[nt][0] = tot[nt][1] = tot[nt][2] = tot[nt][3] = 0.f;
                const int nn = 2 * min(4, tile + 1 - n0);
                float x[2][2][4];
                auto rows = [&](int c, float (&y)[2][4]) {
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        const bool in = c + 8 * s + 2 * t < D.d;
                        const float2 u = in && ok0 ? *reinterpret_cast<const float2*>(q0 + c + 8 * s) : make_float2(0.f, 0.f);
                        const float2 v = in && ok1 ? *reinterpret_cast<const float2*>(q1 + c + 8 * s) : make_float2(0.f, 0.f);
                        y[s][0] = u.x; y[s][1] = u.y; y[s][2] = v.x; y[s][3] = v.y;
                    }
                };
                rows(0, x[0]);
#pragma unroll
                for (int k = 0; k < DS / 16; ++k) {
                    if (k + 1 < DS / 16) rows(16 * k + 16, x[(k + 1) & 1]);
#pragma unroll
                    for (int s = 0; s < 2; ++s)
#pragma unroll
                        for (int e = 0; e < 4; ++e) cr_watch(watch, x[k & 1][s][e]);
                    const float* p = ks + (16 * n0 + g) * KS + 16 * k + 2 * t;
                    // these are split once more on their way to the outputs: all four terms, and a chain from zero for every 8 k
#pragma unroll
                    for (int m0 = 0; m0 < 8; m0 += 4) {
                        if (m0 >= nn) break;
#pragma unroll
                        for (int s = 0; s < 2; ++s) {
                            const CrA q = cr_a(x[k & 1][s]);
                            CrB kk[4];
                            float d[4][4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) { kk[i] = cr_b2(p + 8 * (m0 + i) * KS + 8 * s); cr_mma0(d[i], q.l, kk[i].l); }
#pragma unroll
                            for (int i = 0; i < 4; ++i) cr_mma(d[i], q.l, kk[i].h);
#pragma unroll
                            for (int i = 0; i < 4; ++i) cr_mma(d[i], q.h, kk[i].l);
#pragma unroll
                            for (int i = 0; i < 4; ++i) cr_mma(d[i], q.h, kk[i].h);
#pragma unroll
                            for (int i = 0; i < 4; ++i)
#pragma unroll
                                for (int e = 0; e < 4; ++e) tot[m0 + i][e] += d[i][e];
                        }
                    }
                }
#pragma unroll
                for (int nt = 0; nt < 8; ++nt) {
                    if (nt >= nn) break;
                    *reinterpret_cast<float2*>(G + 16 * n0 + 8 * nt) = make_float2(tot[nt][0], tot[nt][1]);
                    *reinterpret_cast<float2*>(G + 8 * SG + 16 * n0 + 8 * nt) = make_float2(tot[nt][2], tot[nt][3]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) cr_watch(watch, tot[nt][e]);
                }
            }
        }
        if (!(watch == 0.f)) sg_mark(D, w, a.sq, kh * (D.H / D.Hk), D.H / D.Hk);
        return;
    }
    const int h = blockIdx.y - D.Hk, kh = h / (D.H / D.Hk), col0 = blockIdx.z * SG_COLS, dvs = D.dv + D.ones_col;
    float *suf = sm + SG, *weight = sm + 2 * SG, *bt = sm + 3 * SG, *blk = sm + 4 * SG;
    uint32_t* tile = reinterpret_cast<uint32_t*>(sm + SG_DEC);
    const SgDecay dec = sg_decay(w, D.H, h, a);
    float4 v[SG_VECS];
#pragma unroll
    for (int k = 0; k < SG_VECS; ++k) v[k] = sg_value(D, w, a, h, col0 + sg_col(), sg_row(k));
    // 128 key rows: a warp takes 16 of them and all columns; 64: 16 of them and half of the columns
    constexpr int NT = DS == 128 ? 8 : 4;
    const int r0 = 16 * (DS == 128 ? warp : warp & 3) + g, c0 = DS == 128 ? 0 : 32 * (warp >> 2);
    const float* k0 = w.qkv + (size_t)a.start * w.ld + w.k_off + kh * D.d + r0;
    const bool ok0 = r0 < D.d, ok1 = r0 + 8 < D.d;
    auto keys = [&](int k, float (&y)[2][4]) {
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int tk = 16 * k + 8 * s + 2 * t + e;
                const float* p = k0 + (size_t)tk * w.ld;
                y[s][e] = tk < a.len && ok0 ? p[0] : 0.f;
                y[s][2 + e] = tk < a.len && ok1 ? p[8] : 0.f;
            }
    };
    float x[2][4], y[2][4];
    keys(0, x);
    sg_decay_put(dec, sm, watch);
    __syncthreads();
    sg_decay_form<false>(sm, nullptr);
    __syncthreads();
    if (tid < SG) {
        float f = suf[tid];
        for (int k = (tid >> 4) + 1; k < SG_BLK; ++k) f *= blk[k];
        weight[tid] = f;
        if (tid == 0 && blockIdx.z == 0) {
            float p = 1.f;
            for (int k = 0; k < SG_BLK; ++k) p *= blk[k];
            sg.prod[a.entry * D.H + h] = p;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < SG_VECS; ++k) {
        const int r = sg_row(k);
        const float b = bt[r], f = weight[r];
        float4 x = make_float4(v[k].x * b, v[k].y * b, v[k].z * b, v[k].w * b);
        sg_watch4(watch, x);
        x.x *= f; x.y *= f; x.z *= f; x.w *= f;
        sg_put(tile, r, sg_col(), x);
    }
    __syncthreads();
    const int nn = min(NT, (dvs - col0 - c0 + 7) / 8);
    if (16 * (DS == 128 ? warp : warp & 3) < D.d && nn > 0) {
        float tot[NT][4];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) tot[nt][0] = tot[nt][1] = tot[nt][2] = tot[nt][3] = 0.f;
        const int steps = (a.len + 15) / 16;
#pragma unroll 1
        for (int k = 0; k < steps; ++k) {
            if (k + 1 < steps) keys(k + 1, y);
            sg_step<NT>(tot, x, nn, SgRows(tile, 16 * k, c0, g, t));
            sg_next(x, y);
        }
        float* S = sg.local + (a.entry * D.H + h) * D.d * dvs;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = r0 + 8 * (e >> 1), c = col0 + c0 + 8 * nt + 2 * t + (e & 1);
                cr_watch(watch, tot[nt][e]);
                if (r < D.d && c < dvs) S[(size_t)r * dvs + c] = tot[nt][e];
            }
    }
    if (!(watch == 0.f)) sg_mark(D, w, a.sq, h, 1);
}

template <int DS>
__global__ void __launch_bounds__(SG_THREADS, 2) segment_outputs_kernel(Batch b, DeltaDims D, ChunkView w, SegArgs sg, float* __restrict__ o) {
    extern __shared__ __align__(16) float sm[];
    const SegAt a = sg_at(b, sg.n);
    if (a.len <= 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int h = blockIdx.y, kh = h / (D.H / D.Hk), col0 = blockIdx.z * SG_COLS, dvs = D.dv + D.ones_col, nn = min(8, (dvs - col0 + 7) / 8);
    float *cum = sm, *suf = sm + SG, *bt = sm + 3 * SG, *blk = sm + 4 * SG, *diag = sm + SG_DEC, *vals = diag + SG_DIAG + SG_TILE;
    uint32_t* tile = reinterpret_cast<uint32_t*>(diag + SG_DIAG);
    float watch = 0.f;
    const SgDecay dec = sg_decay(w, D.H, h, a);
    const int mine = sg_tile(warp), j0 = 16 * mine + g;
    const bool some = 16 * mine < a.len, ok0 = j0 < a.len, ok1 = j0 + 8 < a.len;
    const float* q0 = w.qkv + (size_t)(a.start + j0) * w.ld + w.q_off + kh * D.d + 2 * t;
    const float* q1 = q0 + (size_t)8 * w.ld;
    auto rows = [&](int c, float (&y)[2][4]) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const bool in = c + 8 * s + 2 * t < D.d;
            const float2 u = in && ok0 ? *reinterpret_cast<const float2*>(q0 + c + 8 * s) : make_float2(0.f, 0.f);
            const float2 v = in && ok1 ? *reinterpret_cast<const float2*>(q1 + c + 8 * s) : make_float2(0.f, 0.f);
            y[s][0] = u.x; y[s][1] = u.y; y[s][2] = v.x; y[s][3] = v.y;
        }
    };
    const float* G = w.rec + (a.entry * D.Hk + kh) * SG_G + (size_t)j0 * SG + 2 * t;
    auto products = [&](int k, float (&y)[2][4]) {
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const float2 u = *reinterpret_cast<const float2*>(G + 16 * k + 8 * s), v = *reinterpret_cast<const float2*>(G + 8 * SG + 16 * k + 8 * s);
            y[s][0] = u.x; y[s][1] = u.y; y[s][2] = v.x; y[s][3] = v.y;
        }
    };
    float x[2][4], y[2][4];
    {   // the start state's columns; the values on their way meanwhile
        const float* S = sg.start + (a.entry * D.H + h) * D.d * dvs;
        const int c = col0 + sg_col();
        float4 v[DS * SG_VECS / SG];
#pragma unroll
        for (int k = 0; k < DS * SG_VECS / SG; ++k) {
            const int r = sg_row(k);
            const float* p = S + (size_t)r * dvs + c;
            v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r >= D.d) continue;
            if (dvs % 4 == 0 && c + 4 <= dvs) v[k] = *reinterpret_cast<const float4*>(p);
            else {
                if (c < dvs) v[k].x = p[0];
                if (c + 1 < dvs) v[k].y = p[1];
                if (c + 2 < dvs) v[k].z = p[2];
                if (c + 3 < dvs) v[k].w = p[3];
            }
        }
#pragma unroll
        for (int k = 0; k < SG_VECS; ++k) {
            const int tk = sg_row(k);
            float* to = vals + tk * SG_COLS + sg_col();
            const float* from = w.qkv + (size_t)(a.start + tk) * w.ld + w.v_off + h * D.dv + c;
            if (tk < a.len && c + 4 <= D.dv && ((uintptr_t)from & 15) == 0) sg_cp16(to, from);
            else *reinterpret_cast<float4*>(to) = sg_value(D, w, a, h, c, tk);
        }
        cp_async_commit();
#pragma unroll
        for (int k = 0; k < DS * SG_VECS / SG; ++k) { sg_watch4(watch, v[k]); sg_put(tile, sg_row(k), sg_col(), v[k]); }
    }
    sg_decay_put(dec, sm, watch);
    __syncthreads();
    float tot[8][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) tot[nt][0] = tot[nt][1] = tot[nt][2] = tot[nt][3] = 0.f;
    if (some) {                                              // ---- S^T q
        rows(0, x);
#pragma unroll 1
        for (int k = 0; k < DS / 16; ++k) {
            if (k + 1 < DS / 16) rows(16 * k + 16, y);
            sg_step<8>(tot, x, nn, SgRows(tile, 16 * k, 0, g, t));
            sg_next(x, y);
        }
    }
    sg_decay_form<true>(sm, diag);
    cp_async_wait<0>();
    __syncthreads();                                         // the start state has been read
#pragma unroll
    for (int k = 0; k < SG_VECS; ++k) {
        const int r = sg_row(k);
        const float4 x = *reinterpret_cast<const float4*>(vals + r * SG_COLS + sg_col());
        const float b = bt[r];
        const float4 u = make_float4(x.x * b, x.y * b, x.z * b, x.w * b);
        sg_watch4(watch, u);
        sg_put(tile, r, sg_col(), u);
    }
    __syncthreads();
    if (some) {
        float c0 = cum[j0], c1 = cum[j0 + 8];
        {   // S^T q times the decays up to the token
            float f0 = c0, f1 = c1;
            for (int k = 0; k < mine; ++k) { f0 *= blk[k]; f1 *= blk[k]; }
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) { tot[nt][0] *= f0; tot[nt][1] *= f0; tot[nt][2] *= f1; tot[nt][3] *= f1; }
        }
        {   // ---- the segment's own tokens, from the token's 16 back
            products(mine, x);
#pragma unroll 1
            for (int k = mine; k >= 0; --k) {
                if (k > 0) products(k - 1, y);
                if (k == mine) {
                    const float* d0 = diag + j0 * 17 + 2 * t;
#pragma unroll
                    for (int s = 0; s < 2; ++s)
#pragma unroll
                        for (int e = 0; e < 2; ++e) { x[s][e] *= d0[8 * s + e]; x[s][2 + e] *= d0[8 * 17 + 8 * s + e]; }
                } else {
#pragma unroll
                    for (int s = 0; s < 2; ++s)
#pragma unroll
                        for (int e = 0; e < 2; ++e) { const float f = suf[16 * k + 8 * s + 2 * t + e]; x[s][e] *= c0 * f; x[s][2 + e] *= c1 * f; }
                    c0 *= blk[k]; c1 *= blk[k];
                }
                sg_step<8>(tot, x, nn, SgRows(tile, 16 * k, 0, g, t));
                sg_next(x, y);
            }
        }
#pragma unroll
        for (int nt = 0; nt < 8; ++nt)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int tk = j0 + 8 * (e >> 1), c = col0 + 8 * nt + 2 * t + (e & 1);
                cr_watch(watch, tot[nt][e]);
                if (tk < a.len && c < dvs) o[((size_t)(a.start + tk) * D.H + h) * dvs + c] = tot[nt][e] * D.o_scale;
            }
    }
    if (!(watch == 0.f)) sg_mark(D, w, a.sq, h, 1);
}

template <int DS>
int sg_launch(const Batch& b, const DeltaDims& D, const ChunkView& w, const float* decay, float* state, size_t slot_stride, float* o, cudaStream_t s, const ScanWorkspace* scan) {
    static DevOnce once;
    constexpr int sum_bytes = sg_sum_floats(DS) * 4, out_bytes = SG_OUT_FLOATS * 4;
    if (once.need() && (cuda_check(cudaFuncSetAttribute(segment_sums_kernel<DS>, cudaFuncAttributeMaxDynamicSharedMemorySize, sum_bytes), "segment shared memory") ||
                        cuda_check(cudaFuncSetAttribute(segment_outputs_kernel<DS>, cudaFuncAttributeMaxDynamicSharedMemorySize, out_bytes), "segment shared memory"))) return WF_ERR_CUDA;
    SegArgs sg;
    sg.n = (b.max_len + SG - 1) / SG;
    sg.local = scan->local; sg.start = scan->start; sg.prod = scan->prod;
    const int z = (D.dv + D.ones_col + SG_COLS - 1) / SG_COLS;
    // (behind the end of the kernel before, like the scans: see cr_scan)
    segment_sums_kernel<DS><<<dim3(b.nseq * sg.n, D.Hk + D.H, z), SG_THREADS, sum_bytes, s>>>(b, D, w, sg);
    if (int rc = launch_check(cudaGetLastError(), "segment_sums")) return rc;
    if (int rc = launch_scan_prefix(b, D, decay, state, slot_stride, scan, sg.n, s)) return rc;
    segment_outputs_kernel<DS><<<dim3(b.nseq * sg.n, D.H, z), SG_THREADS, out_bytes, s>>>(b, D, w, sg, o);
    return launch_check(cudaGetLastError(), "segment_outputs");
}

}  // namespace

size_t segment_workspace_floats(const DeltaDims& D, int max_step_tokens, int slots) {
    return D.no_delta && !D.vec_decay && max_step_tokens >= 4 * SG ? (size_t)scan_chunks_needed(max_step_tokens, slots) * D.Hk * SG_G : 0;
}

// Whether portions are taken in segments, by what 22 sets of portions of 19 sizes of heads took in both forms (us, 16 tokens at a time / so).  Long portions only: a segment moves
// its state five times through memory and its blocks cost their latencies however few the tokens; 40 heads of 128 x 64 over 5, one portion of 256 tokens 38 / 48.
//   * The longest well beyond the average: the other form waits for it with SMs idle.  40 heads over 5, 1700 and 100 tokens 1.9 times as fast so; matrix memory, 16 heads of
//     64 x 128, 1500, 400 and 100 tokens 1.35.  Not where heads have keys of their own, 128 wide, and the other form cuts its portions, too (other_in_passes): matrix memory, 4
//     heads of 128 x 128, 900 and 3 x 300 tokens 0.86.
//   * About one length: only where several heads share a key head's products q k.  With keys of their own segments lose more often than they gain (matrix memory, whose normaliser
//     column takes 64 columns for itself besides: 16 heads of 128 x 128, 2 of 512 tokens 0.68, 2 of 2048 0.79; at best 32 heads of 64 x 64, 1024 tokens 1.14).  Shared, by the
//     times of both: rounds of blocks over the SMs, each kernel to about 15 %.  40 heads of 128 x 64 over 5, 512 tokens 1.09, 2048 1.32; 16 of 128 x 128 over 2, 1024 1.23; but 8 of
//     128 x 64 over 1, 1024 tokens 0.79, 16 of 128 x 128 over 2, 4 of 512 0.81.
// Of those 418 sets five are slower so than the other form by more than 2 %, the worst by 10 (16 heads of 128 x 128 over 2, one portion of 512).
bool segments_faster(const DeltaDims& D, int nseq, int n, int max_len) {
    const long long sms = sm_count();
    const int dvs = D.dv + D.ones_col, cols = (dvs + CR_COLS - 1) / CR_COLS, z = (dvs + SG_COLS - 1) / SG_COLS;
    if (!D.no_delta || D.vec_decay || nseq < 1 || max_len < 4 * SG || n < 3LL * SG * nseq) return false;
    const long long tiles = (long long)nseq * D.H * cols, pairs = (long long)nseq * D.H * ((cols + 1) / 2);
    const bool big = D.d > 64, shared = D.H >= 4 * D.Hk, other_in_passes = 2 * tiles < 3 * sms;
    if (5LL * max_len * nseq > 7LL * n) return shared || !big || !other_in_passes;
    if (!shared) return false;
    auto rounds = [&](double blocks) { return ceil(blocks / (double)sms); };
    const double segs = n / (double)SG + 0.5 * nseq, heads = segs * D.H;
    double so = big ? 21. + 17. * rounds(heads * z) + 12. * segs * D.Hk / sms : 15. + 12. * rounds(heads * z) + 7. * segs * D.Hk / sms;
    double other = 4. + (big ? 5e-3 : 3.7e-3) * n / CHUNK_TOKENS * D.H;          // the preparation, then the scan
    if (other_in_passes) {
        const double one = 0.84 * heads * cols / sms, two = 1.3 * heads * ((cols + 1) / 2) / sms, chunks = SG / CHUNK_TOKENS * (one < two ? one : two);
        other += big ? 19. + 1.3 * chunks : 17. + 0.85 * chunks;                  // (the chain of the passes is the same kernel as here)
    } else {
        auto chunk = [&](long long blocks, double one, double two, double more) { const long long k = (blocks + sms - 1) / sms; return k <= 1 ? one : k == 2 ? two : more * (double)k; };
        const double one = chunk(tiles, 1.2, 1.7, 0.84), two = chunk(pairs, 1.5, 2.6, 1.3);
        other += 8. + (big ? 0.91 : 0.67) * max_len / CHUNK_TOKENS * (one < two ? one : two);
        so += 3. + 2.2e-6 * heads * D.d * dvs;
    }
    return so < 0.95 * other;
}

bool segments_usable(const Batch& b, const DeltaDims& D, const ScanWorkspace* scan) {
    const long long segs = b.n / SG + b.nseq + 1;
    return segments_faster(D, b.nseq, b.n, b.max_len) && scan->local && segs <= scan->chunks && (size_t)segs * D.Hk * SG_G <= scan->rec_floats && D.H + D.Hk <= 65535;
}

int launch_segments(const Batch& b, const DeltaDims& D, const ChunkView& w, const float* decay, float* state, size_t slot_stride, float* o, cudaStream_t s, const ScanWorkspace* scan) {
    return D.d <= 64 ? sg_launch<64>(b, D, w, decay, state, slot_stride, o, s, scan) : sg_launch<128>(b, D, w, decay, state, slot_stride, o, s, scan);
}

}  // namespace seq
}  // namespace wf
