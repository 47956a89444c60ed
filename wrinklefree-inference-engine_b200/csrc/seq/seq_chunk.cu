// The matrix-state recurrences of seq_delta.cu over prompt portions, 16 tokens at a time instead of one by one.  With S the state before a chunk, c_j the
// product of the decays of tokens 1 .. j and D(i, j) that of tokens i + 1 .. j (diagonal over the key rows, or a number):
//     R_j = S^T (c_j k_j),   A_ji = k_i^T D(i, j) k_j (i < j),   u_j = beta_j (v_j - R_j - sum_{i<j} A_ji u_i)      -> U = T (V - R),
//     o_j = S^T (c_j q_j) + sum_{i<=j} B_ji u_i with B_ji = k_i^T D(i, j) q_j,   S <- c_16 S + sum_j (D(j, 16) k_j) u_j^T.
// Without the correction (state-space, gated linear attention, matrix memory) U = beta V.
//   * chunk_prep_kernel, a block per (chunk, head): T = (I + beta A)^-1 beta and B, and with a decay per key row the decayed k and q rows;
//   * chunk_scan_kernel, a block per (sequence, head, 16 columns): walks the chunks in order, the next one's rows under way by cp.async.  All products run
//     on mma.sync m16n8k8 with every operand as a sum of two tf32 numbers (hi hi + hi lo + lo hi, 22 to 24 bits of each product) and float sums; the
//     state stays in float registers, as S^T in accumulator layout, which with the key rows of an 8-row tile taken in the order 0 2 4 6 1 3 5 7 is also
//     the operand layout of S^T k, so it is never moved.  The four warps share the 16 columns and split the key rows; their partial R and S^T q meet in
//     shared memory once per chunk.
// What bounded the forms before: token by token, a chain of multiply-adds, shuffles and shared-memory reads of about 1000 clk per token; chunks on
// the multiply-add units, shared-memory bandwidth (every thread of a column reads every key: 5 wavefronts per request, 450 us for the case below).
// Measured: delta rule (20 heads, 128 x 128, two sequences, 1801 tokens) 569 -> 236 us, since then 183 (the longer sequence in blocks of its own kind, four blocks an SM in the
// preparation); state space (40 heads, 128 x 64, one sequence, 2048 tokens) 307 -> 179 us, 131 in segments, which it now takes (seq_segment.cu);
// with eight warps of half the rows each 287 and 257 us (both in one pass).  Left: the chain of a chunk, about 3000 clk of products, one exchange of partial
// sums and two barriers.  Error against 64 bits (2-norm of a mixer's output, up to 2048 tokens): in float32 engines 4.47e-7 against 4.36e-7 token by token (delta rule),
// 3.35e-7 / 3.33e-7 (state space), 4.82e-7 / 4.94e-7 (matrix memory); float32 engines keep the token form all the same.  In bf16 engines both 2.05e-3, 1.67e-3, 1.66e-3.
// Numbers that are not finite: in a product with the zeros of T and B, or as a sum of two tf32 numbers, an infinity or a NaN would reach tokens and rows
// that never meet it (and the rounding of cr_split takes the bit pattern of a NaN past the exponent, to zero).  So the preparation marks the heads in which
// anything that it reads or forms is not finite, the scan those in which U or the state is not, and chunk_redo_kernel takes the marked portions again from
// their start, token by token as the recurrence is stated: a launch of blocks that leave at once where nothing is marked (about 2 us; deciding chunk by
// chunk inside the scan cost it 15 to 30 %).
#include "seq_chunk.cuh"

namespace wf {
namespace seq {

namespace {

constexpr int CR = CHUNK_TOKENS, CR_WARPS = 4, CR_THREADS = 32 * CR_WARPS;
static_assert(CR == 16, "a chunk is two 8-token tiles");

__device__ __forceinline__ void cr_cp16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// one of the two passes over segments of SCAN_CHUNK tokens in parallel (recurrences linear in the state): pass 1 leaves each segment's own end state (from a
// zero one) and, with one decay per head, the product of its decays; pass 3 reads the segments' start states, chained by scan_prefix_kernel; 0: whole portions
struct Segments { int pass = 0, n = 1; float *local = nullptr, *prod = nullptr; const float* start = nullptr; };

// a record: [T 256][B 256] then, decay per row: [c_j q_j 16 DS][c_j k_j 16 DS][D(j, 16) k_j 16 DS][c_16 DS]; one decay: [c_j 16][D(j, 16) 16][c_16, padding]
// (DS: the key rows, padded to 64 or 128)
__host__ __device__ constexpr int cr_rec_floats(int DS, bool vec) { return vec ? 512 + (3 * CR + 1) * DS : 512 + 48; }

// transposed sum over 16 lanes: v[t] of all of them -> the sum of t = p for lane p
__device__ __forceinline__ float cr_reduce(float (&v)[CR], int p) {
#pragma unroll
    for (int w = 8; w >= 1; w >>= 1) {
        const bool up = (p & w) != 0;
#pragma unroll
        for (int k = 0; k < w; ++k) {
            const float send = up ? v[k] : v[w + k], keep = up ? v[w + k] : v[k];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, send, w);
        }
    }
    return v[0];
}

// (128 registers in place of 167, a few of them spilled, where the correction takes most: four blocks an SM instead of three; 20 heads of 128 x 128, 1801 tokens 47 -> 40 us)
template <int DS, bool VEC, bool DELTA>
__global__ void __launch_bounds__(CR_THREADS, DS == 128 && DELTA ? 4 : 0) chunk_prep_kernel(Batch b, DeltaDims D, ChunkView w) {
    pdl_enter();
    constexpr int Q4 = DS / 64;             // float4 per lane part
    __shared__ __align__(16) float ks[CR][DS], qs[CR][DS], gs[VEC ? CR : 1][VEC ? DS : 4];
    __shared__ float As[CR][CR + 1], Bs[CR][CR + 1], gsc[CR], bt[CR];
    const int sq = blockIdx.x / w.nchunks, ch = blockIdx.x - sq * w.nchunks, h = blockIdx.y;
    const int len = b.seq_len[sq], start = b.seq_start[sq] + ch * CR, left = min(CR, len - ch * CR);
    if (left <= 0) return;
    const int tid = threadIdx.x, kh = h / (D.H / D.Hk);
    float watch = 0.f;
    float* rec = w.rec + ((size_t)(b.seq_start[sq] / CR + sq + ch) * D.H + h) * cr_rec_floats(DS, VEC);
    for (int i = tid; i < CR * (DS / 4); i += CR_THREADS) {
        const int t = i / (DS / 4), c = (i - t * (DS / 4)) * 4;
        float4 k = make_float4(0.f, 0.f, 0.f, 0.f), q = k, g = make_float4(1.f, 1.f, 1.f, 1.f);
        if (t < left && c < D.d) {
            const float* row = w.qkv + (size_t)(start + t) * w.ld;
            k = *reinterpret_cast<const float4*>(row + w.k_off + kh * D.d + c);
            q = *reinterpret_cast<const float4*>(row + w.q_off + kh * D.d + c);
            if (VEC) g = *reinterpret_cast<const float4*>(w.decay + ((size_t)(start + t) * D.H + h) * D.d + c);
            else {
                cr_watch(watch, k.x); cr_watch(watch, k.y); cr_watch(watch, k.z); cr_watch(watch, k.w);
                cr_watch(watch, q.x); cr_watch(watch, q.y); cr_watch(watch, q.z); cr_watch(watch, q.w);
            }
        }
        *reinterpret_cast<float4*>(&ks[t][c]) = k;
        *reinterpret_cast<float4*>(&qs[t][c]) = q;
        if (VEC) *reinterpret_cast<float4*>(&gs[t][c]) = g;
    }
    if (tid < CR) {
        bt[tid] = tid < left ? (w.beta ? w.beta[(size_t)(start + tid) * D.H + h] : 1.f) : 0.f;
        if (!VEC) gsc[tid] = tid < left ? w.decay[(size_t)(start + tid) * D.H + h] : 1.f;
    }
    __syncthreads();
    // ---- A and B: a thread takes the earlier tokens i and 15 - i and a sixteenth of the key rows, and runs over the later tokens j with the decayed keys in hand
    {
        const int p = tid & 15, i0 = tid >> 4, i1 = CR - 1 - i0;      // i0 < i1
        float a0[CR], a1[CR], b0[CR], b1[CR];
#pragma unroll
        for (int j = 0; j < CR; ++j) a0[j] = a1[j] = b0[j] = b1[j] = 0.f;
#pragma unroll
        for (int m = 0; m < Q4; ++m) {
            const int c = (p + 16 * m) * 4;
            float4 x = *reinterpret_cast<const float4*>(&ks[i0][c]), y = *reinterpret_cast<const float4*>(&ks[i1][c]);
#pragma unroll
            for (int j = 0; j < CR; ++j) {
                if (j < i0) continue;
                const float4 q = *reinterpret_cast<const float4*>(&qs[j][c]);
                float4 g, k;
                if (VEC) g = *reinterpret_cast<const float4*>(&gs[j][c]);
                if (DELTA) k = *reinterpret_cast<const float4*>(&ks[j][c]);
                if (j > i0) {
                    if (VEC) { x.x *= g.x; x.y *= g.y; x.z *= g.z; x.w *= g.w; }
                    if (DELTA) a0[j] = fmaf(x.x, k.x, fmaf(x.y, k.y, fmaf(x.z, k.z, fmaf(x.w, k.w, a0[j]))));
                }
                b0[j] = fmaf(x.x, q.x, fmaf(x.y, q.y, fmaf(x.z, q.z, fmaf(x.w, q.w, b0[j]))));
                if (j < i1) continue;
                if (j > i1) {
                    if (VEC) { y.x *= g.x; y.y *= g.y; y.z *= g.z; y.w *= g.w; }
                    if (DELTA) a1[j] = fmaf(y.x, k.x, fmaf(y.y, k.y, fmaf(y.z, k.z, fmaf(y.w, k.w, a1[j]))));
                }
                b1[j] = fmaf(y.x, q.x, fmaf(y.y, q.y, fmaf(y.z, q.z, fmaf(y.w, q.w, b1[j]))));
            }
        }
        float s0 = DELTA ? cr_reduce(a0, p) : 0.f, s1 = DELTA ? cr_reduce(a1, p) : 0.f, t0 = cr_reduce(b0, p), t1 = cr_reduce(b1, p);   // token j = p
        if (!VEC) {
            float pr = 1.f;
            for (int j = CR - 1; j > i0; --j) if (j <= p) pr *= gsc[j];
            s0 *= pr; t0 *= pr;
            pr = 1.f;
            for (int j = CR - 1; j > i1; --j) if (j <= p) pr *= gsc[j];
            s1 *= pr; t1 *= pr;
        }
        if (DELTA) { As[p][i0] = s0; As[p][i1] = s1; }
        Bs[p][i0] = t0; Bs[p][i1] = t1;
    }
    __syncthreads();
    if (DELTA && tid < CR) {                              // column tid of (I + beta A)^-1, by forward substitution, times beta
        float x[CR];
#pragma unroll
        for (int j = 0; j < CR; ++j) {
            float v = 0.f;
#pragma unroll
            for (int l = 0; l < j; ++l) v = fmaf(As[j][l], x[l], v);     // x[l] = 0 for l < tid
            x[j] = j == tid ? 1.f : j > tid ? -bt[j] * v : 0.f;
            rec[j * CR + tid] = x[j] * bt[tid];
            cr_watch(watch, x[j] * bt[tid]);
        }
    }
    for (int i = tid; i < CR * CR; i += CR_THREADS) { rec[256 + i] = Bs[i >> 4][i & 15]; cr_watch(watch, Bs[i >> 4][i & 15]); }
    if (VEC) {
        float *qt = rec + 512, *kt = qt + CR * DS, *kn = kt + CR * DS, *ge = kn + CR * DS;
        for (int c = tid; c < DS; c += CR_THREADS) {
            float cum = 1.f;
#pragma unroll
            for (int t = 0; t < CR; ++t) {
                cum *= gs[t][c];
                const float q = qs[t][c] * cum;
                qt[t * DS + c] = q;
                cr_watch(watch, q);
                if (DELTA) { const float k = ks[t][c] * cum; kt[t * DS + c] = k; cr_watch(watch, k); }
            }
            ge[c] = cum;
            cr_watch(watch, cum);
            float suf = 1.f;
#pragma unroll
            for (int t = CR - 1; t >= 0; --t) { const float k = ks[t][c] * suf; kn[t * DS + c] = k; cr_watch(watch, k); suf *= gs[t][c]; }
        }
    } else if (tid < CR) {
        float cum = 1.f, suf = 1.f;
        for (int t = 0; t <= tid; ++t) cum *= gsc[t];
        for (int t = tid + 1; t < CR; ++t) suf *= gsc[t];
        rec[512 + tid] = cum; rec[528 + tid] = suf;
        if (tid == CR - 1) rec[544] = cum;
        cr_watch(watch, cum); cr_watch(watch, suf);
    }
    if (!(watch == 0.f))
        for (int z = 0; z < w.cols; ++z) w.redo[((size_t)sq * D.H + h) * w.cols + z] = 1;
}

template <int DS, bool VEC, bool DELTA> struct CrStage {
    static constexpr int QS = DS + 8, KS = DS + 4;        // row strides: pairs of rows 8 tokens apart, single rows 2 tokens apart, each without bank conflicts
    static constexpr int TS = 24;                         // of T and B
    static constexpr int T = 0, B = T + (DELTA ? CR * TS : 0), Q = B + CR * TS, K = Q + CR * QS, N = K + (DELTA ? CR * QS : 0), G = N + CR * KS,
                         FLOATS = G + (VEC ? DS : 48);    // G: c_16 per row, or [c_j][D(j, 16)][c_16]
};
constexpr int CR_RS = 24;                                 // row stride of the partial sums [16 columns][16 tokens]

// CT: tiles of 16 columns that a block takes.  The key and query rows that the products need as sums of two numbers are split once for all of them; without the
// correction that splitting was the larger part of the work (the two passes over 40 heads of 128 x 64, 2048 tokens: 63 + 97 us with one, 48 + 78 with two).
// Which one: two_tiles.
// sq, seg: the sequence and its segment; tile0: the first of the block's column tiles.
template <int DS, bool VEC, bool DELTA, int CT>
__device__ __forceinline__ void chunk_scan(const Batch b, const DeltaDims D, const ChunkView w, float* __restrict__ state, size_t slot_stride, float* __restrict__ o, const Segments sg,
                                           const int sq, const int seg, const int h, const int tile0) {
#include "seq_chunk_scan.cuh"
}

template <int DS, bool VEC, bool DELTA, int CT>
__global__ void __launch_bounds__(CR_THREADS) chunk_scan_kernel(Batch b, DeltaDims D, ChunkView w, float* __restrict__ state, size_t slot_stride, float* __restrict__ o, Segments sg) {
    pdl_enter();
    const int sq = blockIdx.x / sg.n, seg = blockIdx.x - sq * sg.n, h = blockIdx.y, tile0 = blockIdx.z * CT;
#include "seq_chunk_scan.cuh"
}

// The longest portion in blocks of one column tile, handed out first, the others in blocks of two (mixed_tiles): the sequence that the scan waits for goes its chain with
// less beside it, and two blocks fit every SM.
template <int DS, bool VEC, bool DELTA>
__global__ void __launch_bounds__(CR_THREADS, 2) chunk_scan_mixed_kernel(Batch b, DeltaDims D, ChunkView w, float* __restrict__ state, size_t slot_stride, float* __restrict__ o) {
    pdl_enter();
    int longest = 0;
    for (int s = 1; s < b.nseq; ++s) if (b.seq_len[s] > b.seq_len[longest]) longest = s;
    const Segments whole;
    int i = blockIdx.x;
    const int ones = D.H * w.cols, pairs = (w.cols + 1) / 2;
    if (i < ones) {
        const int h = i / w.cols;
        chunk_scan<DS, VEC, DELTA, 1>(b, D, w, state, slot_stride, o, whole, longest, 0, h, i - h * w.cols);
        return;
    }
    i -= ones;
    int sq = i / (D.H * pairs);
    i -= sq * D.H * pairs;
    const int h = i / pairs;
    if (sq >= longest) ++sq;
    chunk_scan<DS, VEC, DELTA, 2>(b, D, w, state, slot_stride, o, whole, sq, 0, h, 2 * (i - h * pairs));
}

// The marked portions again, token by token (see above), a block per (sequence, head, 16 columns); their start state is still in the slot, or, with segments,
// that of the first one.  A thread holds the part of the state that it holds in chunk_scan_kernel; rows come straight from memory.
template <int DS, bool VEC, bool DELTA>
__global__ void __launch_bounds__(CR_THREADS) chunk_redo_kernel(Batch b, DeltaDims D, ChunkView w, float* __restrict__ state, size_t slot_stride, float* __restrict__ o, Segments sg) {
    pdl_enter();
    constexpr int NT = DS / (8 * CR_WARPS);
    __shared__ float rs[CR_WARPS][CR_COLS], os[CR_WARPS][CR_COLS];
    const int sq = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3, row0 = warp * 8 * NT;
    int* mark = w.redo + ((size_t)sq * D.H + h) * w.cols + blockIdx.z;
    if (!*mark) return;
    const int col0 = blockIdx.z * CR_COLS, c0 = col0 + g, dvs = D.dv + D.ones_col, kh = h / (D.H / D.Hk), start = b.seq_start[sq], len = b.seq_len[sq];
    float* S1 = state + (size_t)b.seq_slot[sq] * slot_stride + (size_t)h * D.d * dvs;
    const float* S0 = sg.start ? sg.start + ((size_t)(start / SCAN_CHUNK + sq) * D.H + h) * D.d * dvs : S1;
    float s[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = row0 + 8 * nt + 2 * t + (e & 1), c = c0 + 8 * (e >> 1);
            s[nt][e] = r < D.d && c < dvs ? S0[(size_t)r * dvs + c] : 0.f;
        }
#pragma unroll 1
    for (int tk = 0; tk < len; ++tk) {
        const size_t at = (size_t)(start + tk) * D.H + h;
        const float *row = w.qkv + (size_t)(start + tk) * w.ld, *kr = row + w.k_off + kh * D.d, *qr = row + w.q_off + kh * D.d, *vr = row + w.v_off + h * D.dv;
        const float *gr = w.decay + at * (VEC ? D.d : 1), gg = VEC ? 1.f : gr[0], bt = w.beta ? w.beta[at] : 1.f;
        float r0 = 0.f, r1 = 0.f;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = row0 + 8 * nt + 2 * t + e;
                if (r >= D.d) continue;
                if (VEC) { s[nt][e] *= gr[r]; s[nt][2 + e] *= gr[r]; }
                if (DELTA) { r0 = fmaf(s[nt][e], kr[r], r0); r1 = fmaf(s[nt][2 + e], kr[r], r1); }
            }
        if (DELTA) {
            r0 += __shfl_xor_sync(0xffffffffu, r0, 1); r1 += __shfl_xor_sync(0xffffffffu, r1, 1);
            r0 += __shfl_xor_sync(0xffffffffu, r0, 2); r1 += __shfl_xor_sync(0xffffffffu, r1, 2);
            if (t == 0) { rs[warp][g] = r0; rs[warp][g + 8] = r1; }
            __syncthreads();                              // (the next token writes rs behind this token's second barrier)
            r0 = r1 = 0.f;
#pragma unroll
            for (int k = 0; k < CR_WARPS; ++k) { r0 += rs[k][g]; r1 += rs[k][g + 8]; }
        }
        const float v0 = c0 >= dvs ? 0.f : c0 == D.dv ? 1.f : vr[c0], v1 = c0 + 8 >= dvs ? 0.f : c0 + 8 == D.dv ? 1.f : vr[c0 + 8];
        const float u0 = bt * (v0 - gg * r0), u1 = bt * (v1 - gg * r1);
        float o0 = 0.f, o1 = 0.f;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int r = row0 + 8 * nt + 2 * t + e;
                if (r >= D.d) continue;
                s[nt][e] = fmaf(kr[r], u0, gg * s[nt][e]); o0 = fmaf(s[nt][e], qr[r], o0);
                s[nt][2 + e] = fmaf(kr[r], u1, gg * s[nt][2 + e]); o1 = fmaf(s[nt][2 + e], qr[r], o1);
            }
        o0 += __shfl_xor_sync(0xffffffffu, o0, 1); o1 += __shfl_xor_sync(0xffffffffu, o1, 1);
        o0 += __shfl_xor_sync(0xffffffffu, o0, 2); o1 += __shfl_xor_sync(0xffffffffu, o1, 2);
        if (!DELTA) __syncthreads();                      // the token before has been written out
        if (t == 0) { os[warp][g] = o0; os[warp][g + 8] = o1; }
        __syncthreads();
        if (tid < CR_COLS && col0 + tid < dvs) {
            float x = 0.f;
#pragma unroll
            for (int k = 0; k < CR_WARPS; ++k) x += os[k][tid];
            o[at * dvs + col0 + tid] = x * D.o_scale;
        }
    }
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int r = row0 + 8 * nt + 2 * t + (e & 1), c = c0 + 8 * (e >> 1);
            if (r < D.d && c < dvs) S1[(size_t)r * dvs + c] = s[nt][e];
        }
    if (tid == 0) *mark = 0;
}

// Whether a recurrence takes two column tiles a block, where tiles is the number of 16-column tiles and pairs that of blocks of two.  A scan
// takes as long as its fullest SM.  us a chunk with n blocks there, 128-row states: one tile a block 1.2, 1.7, 2.5, 3.3, 4.4 (n = 1 .. 5), two tiles 1.5, 2.6, 3.9.
// So 16 heads of 128 x 64 (64 tiles), one sequence of 256 tokens 36 / 41 us, 40 heads, 2 sequences of 2048 (320 tiles) 317 / 338, but 4 of 1024 (640) 287 / 259;
// an odd tile is a block of its own: matrix memory, 16 heads of 64 x 129, 4 of 1024 (576 tiles, 320 pairs) 147 / 163.
// The same with the correction: 20 heads of 128 x 128, 1801 tokens in 1 sequence (160 tiles) 280 / 259, 2 (320) 209 / 224, 3 (480) 203 / 169, 4 (640) 190 / 192;
// 20 heads of 64 x 64 in 1 (80 tiles) 142 / 190.
bool two_tiles(long long tiles, long long pairs) {
    const long long sms = sm_count(), one = (tiles + sms - 1) / sms, two = (pairs + sms - 1) / sms;
    return 3 * two < 2 * one;
}

// Whether the longest of a few portions is taken in blocks of one column tile and the others in blocks of two, by the same times: with 2.1 us a chunk where one of each share
// an SM.  us, all blocks alike -> so: 20 heads of 128 x 128, 741 and 1060 tokens 231 / 191, 100 and 1700 336 / 272, 2 of 1024 228 / 213; 8 heads of 64 x 128, 400, 600 and
// 801 tokens 89 / 68.
bool mixed_tiles(const Batch& b, int H, int cols) {
    const long long sms = sm_count(), ones = (long long)H * cols, pairs = (long long)H * ((cols + 1) / 2), blocks = ones + (b.nseq - 1) * pairs;
    if (b.nseq < 2 || b.nseq > 16 || blocks > 2 * sms || b.max_len <= 0) return false;
    const double rest = (double)(b.n - b.max_len) / (b.nseq - 1), len = b.max_len;
    auto alone = [](double one, double two, double more, long long n) { return n <= 1 ? one : n == 2 ? two : more * n; };
    const double t1 = len * alone(1.2, 1.7, 0.84, (b.nseq * ones + sms - 1) / sms), t2 = len * alone(1.5, 2.6, 1.3, (b.nseq * pairs + sms - 1) / sms);
    const double shared = blocks > sms ? 2.1 * rest + 1.2 * (len - rest) : 1.5 * rest, own = len * (ones > sms ? 1.7 : 1.2);
    return (shared > own ? shared : own) < 0.95 * (t1 < t2 ? t1 : t2);
}

template <int DS, bool VEC, bool DELTA, int CT>
int cr_scan(const Batch& b, const DeltaDims& D, const ChunkView& w, float* state, size_t slot_stride, float* o, const Segments& sg, cudaStream_t s) {
    const int cols = w.cols;
    constexpr size_t smem = (size_t)(2 * CrStage<DS, VEC, DELTA>::FLOATS + CR_WARPS * (DELTA ? 2 * CT : 2) * CR_COLS * CR_RS) * sizeof(float);
    static DevOnce once;
    if (once.need() && cuda_check(cudaFuncSetAttribute(chunk_scan_kernel<DS, VEC, DELTA, CT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "chunk shared memory")) return WF_ERR_CUDA;
    // Behind the end of the kernel before, not by launch_pdl: blocks that come while that kernel still holds most SMs gather on the few that are free, several
    // to one, and a scan is as slow as its fullest SM.  us by launch_pdl / so: delta rule, 8 heads of 64 x 128, one sequence of 2048 tokens (64 blocks) 300 / 146,
    // 20 heads of 128 x 128 (160 blocks) 395 / 313; state space, 80 heads of 64 x 64 (160 blocks) 383 / 241, 16 heads, 4 sequences (128 blocks) 104 / 57.
    chunk_scan_kernel<DS, VEC, DELTA, CT><<<dim3(b.nseq * sg.n, D.H, (cols + CT - 1) / CT), CR_THREADS, smem, s>>>(b, D, w, state, slot_stride, o, sg);
    return launch_check(cudaGetLastError(), "chunk_scan");
}

template <int DS, bool VEC, bool DELTA>
int cr_launch(const Batch& b, const DeltaDims& D, const ChunkView& w, const float* decay, float* state, size_t slot_stride, float* o, cudaStream_t s, const ScanWorkspace* scan) {
    Segments sg;
    const int cols = w.cols;
    auto redo = [&]() {
        launch_pdl(chunk_redo_kernel<DS, VEC, DELTA>, dim3(b.nseq, D.H, cols), CR_THREADS, 0, s, b, D, w, state, slot_stride, o, sg);
        return launch_check(cudaGetLastError(), "chunk_redo");
    };
    if (!VEC && !DELTA && segments_usable(b, D, scan)) {
        if (int rc = launch_segments(b, D, w, decay, state, slot_stride, o, s, scan)) return rc;
        sg.start = scan->start;
        return redo();
    }
    launch_pdl(chunk_prep_kernel<DS, VEC, DELTA>, dim3(b.nseq * w.nchunks, D.H), CR_THREADS, 0, s, b, D, w);
    if (int rc = launch_check(cudaGetLastError(), "chunk_prep")) return rc;
    if constexpr (DELTA) {
        if (mixed_tiles(b, D.H, cols)) {
            constexpr size_t smem = (size_t)(2 * CrStage<DS, VEC, DELTA>::FLOATS + CR_WARPS * 4 * CR_COLS * CR_RS) * sizeof(float);
            static DevOnce once;
            if (once.need() && cuda_check(cudaFuncSetAttribute(chunk_scan_mixed_kernel<DS, VEC, DELTA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "chunk shared memory")) return WF_ERR_CUDA;
            chunk_scan_mixed_kernel<DS, VEC, DELTA><<<D.H * cols + (b.nseq - 1) * D.H * ((cols + 1) / 2), CR_THREADS, smem, s>>>(b, D, w, state, slot_stride, o);
            if (int rc = launch_check(cudaGetLastError(), "chunk_scan_mixed")) return rc;
            return redo();
        }
    }
    auto scan_pass = [&](int pass) {
        sg.pass = pass;
        const long long chains = (long long)b.nseq * sg.n * D.H, tiles = chains * cols;
        return two_tiles(tiles, chains * ((cols + 1) / 2)) ? cr_scan<DS, VEC, DELTA, 2>(b, D, w, state, slot_stride, o, sg, s) : cr_scan<DS, VEC, DELTA, 1>(b, D, w, state, slot_stride, o, sg, s);
    };
    // (Portions that launch_segments leaves.)  Segments in parallel where the recurrence is linear in the state, one portion is long and the chains of whole portions leave the machine idle: the two
    // passes cost half as much work again.  us, whole -> segments, each with the better number of tiles a block: 4 heads of 128 x 64, 1024 tokens 88 -> 40, 600 tokens
    // 59 -> 39; 16 heads, 2048 tokens 171 -> 93; 40 heads (160 tiles) 230 -> 175; 24 heads, 2 sequences of 1024 (192 tiles) 126 -> 121, 16 heads, 4 sequences of
    // 1024 (256 tiles) 131 -> 147.
    if (DELTA || !scan->local || b.max_len < 4 * SCAN_CHUNK || b.n / SCAN_CHUNK + b.nseq + 1 > scan->chunks || 2LL * b.nseq * D.H * cols >= 3LL * sm_count())
    {
        if (int rc = scan_pass(0)) return rc;
        return redo();
    }
    sg.n = (b.max_len + SCAN_CHUNK - 1) / SCAN_CHUNK;
    sg.local = scan->local; sg.start = scan->start; sg.prod = scan->prod;
    if (int rc = scan_pass(1)) return rc;
    if (int rc = launch_scan_prefix(b, D, decay, state, slot_stride, scan, sg.n, s)) return rc;
    if (int rc = scan_pass(3)) return rc;
    return redo();
}

}  // namespace

size_t chunk_workspace_floats(const DeltaDims& D, int max_step_tokens, int slots) {
    if (D.d > 128) return 0;
    const size_t rec = cr_rec_floats(D.d <= 64 ? 64 : 128, D.vec_decay != 0);
    return (size_t)(max_step_tokens / CR + slots + 1) * D.H * rec;
}

size_t chunk_redo_words(const DeltaDims& D, int slots) { return (size_t)slots * D.H * ((D.dv + 1 + CR_COLS - 1) / CR_COLS); }

bool chunk_usable(const Batch& b, const DeltaDims& D, const float* qkv, int ld, const ScanWorkspace* scan) {
    const int qo = D.q_off >= 0 ? D.q_off : 0, ko = D.k_off >= 0 ? D.k_off : D.Hk * D.d;
    return scan && scan->rec && b.max_len >= 2 * CR && D.d <= 128 && D.d % 4 == 0 && ld % 4 == 0 && qo % 4 == 0 && ko % 4 == 0 && ((uintptr_t)qkv & 15) == 0 && D.H <= 65535 &&
           chunk_workspace_floats(D, b.n, b.nseq) <= scan->rec_floats && chunk_redo_words(D, b.nseq) <= scan->redo_words;
}

int launch_chunk_recurrence(const Batch& b, const DeltaDims& D, const float* qkv, int ld, const float* beta, const float* decay, float* state, size_t slot_stride,
                            float* o, cudaStream_t s, const ScanWorkspace* scan) {
    ChunkView w;
    w.qkv = qkv; w.beta = beta; w.decay = decay; w.ld = ld;
    w.q_off = D.q_off >= 0 ? D.q_off : 0; w.k_off = D.k_off >= 0 ? D.k_off : D.Hk * D.d; w.v_off = D.v_off >= 0 ? D.v_off : 2 * D.Hk * D.d;
    w.redo = scan->redo; w.cols = (D.dv + D.ones_col + CR_COLS - 1) / CR_COLS;
    w.rec = scan->rec; w.nchunks = (b.max_len + CR - 1) / CR;
#define CR_PICK(vec, delta) (D.d <= 64 ? cr_launch<64, vec, delta>(b, D, w, decay, state, slot_stride, o, s, scan) : cr_launch<128, vec, delta>(b, D, w, decay, state, slot_stride, o, s, scan))
    if (D.no_delta) return D.vec_decay ? CR_PICK(true, false) : CR_PICK(false, false);
    return D.vec_decay ? CR_PICK(true, true) : CR_PICK(false, true);
#undef CR_PICK
}

}  // namespace seq
}  // namespace wf
