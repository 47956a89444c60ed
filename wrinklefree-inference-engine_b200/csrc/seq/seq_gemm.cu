// Dense, batched and grouped matrix products of the sequence models: C[m, n] = sum_k A[m, k] * B[n, k] with float accumulation.
//   * gemm_simt_kernel — any storage type, plain FMA (the all-32-bit mode; the tests compare the tensor-core forms with it);
//   * gemm_mma_kernel  — bf16 operands on mma.sync.m16n8k16 with a cp.async double buffer (the serving mode).
// Both take the same GemmArgs: grid.z batches with strides (per-head up-projections), or the grouped form in which every 64-row tile
// names its own weight matrix (routed experts) and A rows may be gathered through an index list.
#include "seq_kernels.cuh"
#include <stdlib.h>

namespace wf {
namespace seq {

namespace {

constexpr int BM = 64, BN = 64, BK = 16;       // kernel tile; GEMM_BM (the grouped form's row granule) is a multiple of BM

template <typename T, bool AF32, bool CF32>
__global__ void __launch_bounds__(256) gemm_simt_kernel(GemmArgs g) {
    pdl_enter();
    __shared__ float As[BK][BM + 4];
    __shared__ float Bs[BK][BN + 4];
    const int tile_m = blockIdx.y, tile_n = blockIdx.x, z = blockIdx.z;
    long long grp = 0;
    if (g.tile_group) {
        const int e = g.tile_group[tile_m * BM / GEMM_BM];
        if (e < 0) return;
        grp = (long long)e * g.group_stride;
    }
    const T* B = (const T*)g.B + grp + (long long)z * g.sB;
    const char* Abase = (const char*)g.A;
    const size_t a_elt = AF32 ? 4 : sizeof(T);
    Abase += (size_t)z * g.sA * a_elt;
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;          // 16 x 16 threads, 4 x 4 outputs each
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    // loader mapping: 64 rows x 16 k = 1024 elements, 4 per thread: row = idx / 16, k = idx % 16
    int a_src[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int idx = tid + q * 256;
        const int m = tile_m * BM + idx / BK;
        int r = -1;
        if (m < g.M) r = g.a_rows ? g.a_rows[m] : m;
        a_src[q] = r;
    }
    for (int k0 = 0; k0 < g.K; k0 += BK) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int idx = tid + q * 256;
            const int row = idx / BK, kk = idx % BK, k = k0 + kk;
            float av = 0.f;
            if (a_src[q] >= 0 && k < g.K) {
                const size_t off = (size_t)a_src[q] * g.lda + k;
                av = AF32 ? ((const float*)Abase)[off] : to_f(((const T*)Abase)[off]);
            }
            As[kk][row] = av;
            const int n = tile_n * BN + row;
            Bs[kk][row] = (n < g.N && k < g.K) ? to_f(B[(size_t)n * g.ldb + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = tile_m * BM + ty * 4 + i;
        if (m >= g.M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = tile_n * BN + tx * 4 + j;
            if (n >= g.N) continue;
            const size_t off = (size_t)z * g.sC + (size_t)m * g.ldc + n;
            const float v = epilogue_f(g.ep, acc[i][j]);
            if (CF32) ((float*)g.C)[off] = v;
            else ((T*)g.C)[off] = from_f<T>(v);
        }
    }
}

// ---- bf16 tensor-core form: 64 x 64 x 32 tiles, 4 warps (2 x 2), each warp 32 x 32 = 2 x 4 m16n8k16 tiles -----------------------------
constexpr int MK = 32, MPAD = 8;

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

template <bool AF32, bool CF32>
__global__ void __launch_bounds__(128) gemm_mma_kernel(GemmArgs g) {
    pdl_enter();
    __shared__ __align__(16) __nv_bfloat16 As[2][BM][MK + MPAD];
    __shared__ __align__(16) __nv_bfloat16 Bs[2][BN][MK + MPAD];
    const int tile_m = blockIdx.y, tile_n = blockIdx.x, z = blockIdx.z;
    long long grp = 0;
    if (g.tile_group) {
        const int e = g.tile_group[tile_m * BM / GEMM_BM];
        if (e < 0) return;
        grp = (long long)e * g.group_stride;
    }
    const __nv_bfloat16* B = (const __nv_bfloat16*)g.B + grp + (long long)z * g.sB;
    const char* Abase = (const char*)g.A + (size_t)z * g.sA * (AF32 ? 4 : 2);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp >> 1, wn = warp & 1;
    // loader: 64 rows x 32 k = 256 chunks of 8 elements; 2 chunks per thread per operand
    int a_src[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int ch = tid + q * 128;
        const int m = tile_m * BM + ch / 4;
        a_src[q] = m < g.M ? (g.a_rows ? g.a_rows[m] : m) : -1;
    }
    const bool a_vec = !AF32 && (g.lda % 8 == 0) && (((uintptr_t)Abase & 15) == 0) && (g.K % 8 == 0);
    const bool b_vec = (g.ldb % 8 == 0) && (((uintptr_t)B & 15) == 0) && (g.K % 8 == 0);
    auto load_tile = [&](int buf, int k0) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int ch = tid + q * 128;
            const int row = ch / 4, kc = (ch % 4) * 8, k = k0 + kc;
            __nv_bfloat16* da = &As[buf][row][kc];
            if (a_vec && a_src[q] >= 0 && k + 8 <= g.K) {
                cp_async16(da, (const __nv_bfloat16*)Abase + (size_t)a_src[q] * g.lda + k);
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    float v = 0.f;
                    if (a_src[q] >= 0 && k + e < g.K) {
                        const size_t off = (size_t)a_src[q] * g.lda + k + e;
                        v = AF32 ? ((const float*)Abase)[off] : __bfloat162float(((const __nv_bfloat16*)Abase)[off]);
                    }
                    da[e] = __float2bfloat16_rn(v);
                }
            }
            const int n = tile_n * BN + row;
            __nv_bfloat16* db = &Bs[buf][row][kc];
            if (b_vec && n < g.N && k + 8 <= g.K) {
                cp_async16(db, B + (size_t)n * g.ldb + k);
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e) db[e] = (n < g.N && k + e < g.K) ? B[(size_t)n * g.ldb + k + e] : __float2bfloat16_rn(0.f);
            }
        }
        cp_async_commit();
    };
    float acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[i][j][c] = 0.f;
    const int nk = (g.K + MK - 1) / MK;
    load_tile(0, 0);
    for (int kt = 0; kt < nk; ++kt) {
        const int buf = kt & 1;
        if (kt + 1 < nk) { load_tile(buf ^ 1, (kt + 1) * MK); cp_async_wait<1>(); } else { cp_async_wait<0>(); }
        __syncthreads();
#pragma unroll
        for (int ks = 0; ks < MK; ks += 16) {
            uint32_t a[2][4], b[4][2];
            const int r = lane >> 2, c = (lane & 3) * 2;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int m0 = wm * 32 + i * 16;
                a[i][0] = *(const uint32_t*)&As[buf][m0 + r][ks + c];
                a[i][1] = *(const uint32_t*)&As[buf][m0 + r + 8][ks + c];
                a[i][2] = *(const uint32_t*)&As[buf][m0 + r][ks + c + 8];
                a[i][3] = *(const uint32_t*)&As[buf][m0 + r + 8][ks + c + 8];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int n0 = wn * 32 + j * 8;
                b[j][0] = *(const uint32_t*)&Bs[buf][n0 + r][ks + c];
                b[j][1] = *(const uint32_t*)&Bs[buf][n0 + r][ks + c + 8];
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) mma_bf16_16816(acc[i][j], a[i], b[j]);
        }
        __syncthreads();
    }
    const int r = lane >> 2, c = (lane & 3) * 2;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int m = tile_m * BM + wm * 32 + i * 16 + r + h * 8;
                if (m >= g.M) continue;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int n = tile_n * BN + wn * 32 + j * 8 + c + e;
                    if (n >= g.N) continue;
                    const size_t off = (size_t)z * g.sC + (size_t)m * g.ldc + n;
                    const float v = epilogue_f(g.ep, acc[i][j][h * 2 + e]);
                    if (CF32) ((float*)g.C)[off] = v;
                    else ((__nv_bfloat16*)g.C)[off] = __float2bfloat16_rn(v);
                }
            }
}

// ---- few-row form (decoding): the weight matrix is streamed once, 16 bytes per lane per load; a warp owns GV_RPW output columns and
// all MR <= 8 activation rows, which every warp re-reads through L1.  With `pair_expert` set, grid.y walks (token, expert) pairs instead:
// pair p multiplies ONE activation row (p / pair_div) with the weight matrix of expert pair_expert[p] (routed experts while decoding).
constexpr int GV_WARPS = 8, GV_RPW = 2;

template <typename T> struct Vec16;
template <> struct Vec16<__nv_bfloat16> { static constexpr int N = 8; };
template <> struct Vec16<float> { static constexpr int N = 4; };

template <typename T>
__device__ __forceinline__ void load_vec(const T* p, float (&out)[Vec16<T>::N]);
template <>
__device__ __forceinline__ void load_vec<__nv_bfloat16>(const __nv_bfloat16* p, float (&out)[8]) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { out[2 * i] = __uint_as_float(w[i] << 16); out[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u); }
}
template <>
__device__ __forceinline__ void load_vec<float>(const float* p, float (&out)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
}

struct PairArgs { const int32_t* pair_expert; int n_experts; int pair_div; };

template <typename T, int MR, bool AF32, bool CF32>
__global__ void __launch_bounds__(GV_WARPS * 32) gemv_rows_kernel(GemmArgs g, PairArgs pa) {
    pdl_enter();
    constexpr int VN = Vec16<T>::N;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const T* B = (const T*)g.B;
    int a_row0 = 0, c_row0 = 0, rows = g.M;
    if (pa.pair_expert) {
        const int pr = blockIdx.y;
        const int e = pa.pair_expert[pr];
        if (e < 0 || e >= pa.n_experts) return;
        B += (long long)e * g.group_stride;
        a_row0 = pr / pa.pair_div; c_row0 = pr; rows = 1;
    }
    const int n0 = (blockIdx.x * GV_WARPS + warp) * GV_RPW;
    if (n0 >= g.N) return;
    float acc[GV_RPW][MR];
#pragma unroll
    for (int r = 0; r < GV_RPW; ++r)
#pragma unroll
        for (int m = 0; m < MR; ++m) acc[r][m] = 0.f;
    const int kvec = g.K / VN;                       // the launcher guarantees K % VN == 0 and 16-byte aligned rows
    for (int kv = lane; kv < kvec; kv += 32) {
        const int k = kv * VN;
        float b[GV_RPW][VN];
#pragma unroll
        for (int r = 0; r < GV_RPW; ++r) {
            const int n = n0 + r < g.N ? n0 + r : g.N - 1;
            load_vec<T>(B + (size_t)n * g.ldb + k, b[r]);
        }
#pragma unroll
        for (int m = 0; m < MR; ++m) {
            if (m < rows) {
                float a[VN];
                if (AF32) {
#pragma unroll
                    for (int i = 0; i < VN; ++i) a[i] = ((const float*)g.A)[(size_t)(a_row0 + m) * g.lda + k + i];
                } else {
                    load_vec<T>((const T*)g.A + (size_t)(a_row0 + m) * g.lda + k, a);
                }
#pragma unroll
                for (int r = 0; r < GV_RPW; ++r)
#pragma unroll
                    for (int i = 0; i < VN; ++i) acc[r][m] = fmaf(a[i], b[r][i], acc[r][m]);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < GV_RPW; ++r)
#pragma unroll
        for (int m = 0; m < MR; ++m) {
            float v = acc[r][m];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0 && m < rows && n0 + r < g.N) {
                const size_t off = (size_t)(c_row0 + m) * g.ldc + n0 + r;
                v = epilogue_f(g.ep, v);
                if (CF32) ((float*)g.C)[off] = v; else ((T*)g.C)[off] = from_f<T>(v);
            }
        }
}

template <typename T, int MR>
void gemv_dispatch(const GemmArgs& g, const PairArgs& pa, dim3 grid, cudaStream_t s) {
    if (g.a_f32) { if (g.c_f32) launch_pdl(gemv_rows_kernel<T, MR, true, true>, grid, GV_WARPS * 32, 0, s, g, pa); else launch_pdl(gemv_rows_kernel<T, MR, true, false>, grid, GV_WARPS * 32, 0, s, g, pa); }
    else { if (g.c_f32) launch_pdl(gemv_rows_kernel<T, MR, false, true>, grid, GV_WARPS * 32, 0, s, g, pa); else launch_pdl(gemv_rows_kernel<T, MR, false, false>, grid, GV_WARPS * 32, 0, s, g, pa); }
}

template <typename T>
bool gemv_ok(const GemmArgs& g) {
    constexpr int VN = Vec16<T>::N;
    const size_t ea = g.a_f32 ? 4 : sizeof(T);
    return g.K % VN == 0 && g.ldb % VN == 0 && (((uintptr_t)g.B) & 15) == 0 && (g.lda * ea) % 16 == 0 && (((uintptr_t)g.A) & 15) == 0 &&
           (g.group_stride * (long long)sizeof(T)) % 16 == 0;
}

template <typename T>
void gemv_launch(const GemmArgs& g, const PairArgs& pa, int rows, int ny, cudaStream_t s) {
    dim3 grid((g.N + GV_WARPS * GV_RPW - 1) / (GV_WARPS * GV_RPW), ny);
    if (rows <= 1) gemv_dispatch<T, 1>(g, pa, grid, s);
    else if (rows <= 2) gemv_dispatch<T, 2>(g, pa, grid, s);
    else if (rows <= 4) gemv_dispatch<T, 4>(g, pa, grid, s);
    else gemv_dispatch<T, 8>(g, pa, grid, s);
}

// ---- few-row form on tensor cores (bf16 operands, decoding): 16 weight rows per warp as the M side of mma.sync.m16n8k16, the activation rows as its N
// side, so that a loaded weight serves all rows in two MMAs per 32 k instead of being multiplied row by row.  A lane loads 16 consecutive bytes of a
// row: the four lanes of a row hold k 8 t .. 8 t + 7, and weights and activations are permuted over k alike, so no shuffle is needed.  The WK
// warps of a tile take 64-k steps in turn (a short, wide product has too few rows to cover the machine otherwise) and meet in shared memory.
// The matrix unit cuts off what it adds.  Up to 8 rows (before: the multiply-add kernel) it therefore never adds more than 16 products: those sums meet
// pairwise in float, the warps' in double, and the error against 64 bits stays below the multiply-add kernel's (2-norm, K = 1024 / 2560 / 6912 / 28672: 5.7e-8 / 6.6e-8 /
// 7.5e-8 / 9.4e-8 against 7.0e-8 / 8.4e-8 / 1.2e-7 / 2.4e-7; at K = 64, where every order rounds once or twice, 4.4e-8 against 4.0e-8).  From 9 rows on (before: one
// running sum in gemm_mma_kernel, 2.7e-6 at K = 2560) four running sums per warp are close enough: 1.1e-7.
// Bound: the weight stream, by latency on small matrices.  Measured with 8 rows against gemv_rows_kernel: 1024 x 2304 23.1 -> 9.3 us, 2560 x 6912
// 64.6 -> 12.5, 13824 x 2560 43.7 -> 14.8, 128256 x 2560 298 -> 102; with 16 rows against gemm_mma_kernel: 2560 x 6912 131 -> 12.6.
constexpr int FR_WARPS = 8;
constexpr int FR_CARVEOUT = 14;                           // per cent of an SM's memory: four blocks' sums (0, which leaves room for less, takes twice as long)

// U: 32-k blocks in flight per warp; OCC: blocks per SM
// Weights that no kernel of the stream has written (b_const) are requested before the kernel waits for the one before it, as many as a warp has in flight: a
// decode step of 8 sequences through four layers, 21 such products, 154 -> 146 us.
// glu: a tile's rows 0 .. 7 are gate rows and 8 .. 15 the up rows of the same outputs, so that a pair meets where the tile's sums do.
template <int NT, int WK, int U, int OCC, bool CF32>
__global__ void __launch_bounds__(FR_WARPS * 32, OCC) gemm_few_kernel(GemmArgs g) {
    // (with more blocks per SM, or two of 9 to 16 rows, there are no registers for it, and one another's loads to wait under: 16 rows x 13824 x 2560, gated, on two blocks 30 us, 25 without)
    constexpr bool AHEAD = OCC == 1 || (OCC == 2 && NT == 1);
    const bool early = AHEAD && g.b_const;
    if (!early) pdl_enter();
    constexpr int TILES = FR_WARPS / WK;                  // 16-row tiles per block
    constexpr int C = NT == 1 ? 1 : 4;                    // running sums
    __shared__ float part[FR_WARPS][NT * 8][16 + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g4 = lane >> 2, t4 = lane & 3;
    const int tile = warp / WK, kw = warp % WK;
    const int n0 = (blockIdx.x * TILES + tile) * 16;
    const __nv_bfloat16 *B = (const __nv_bfloat16*)g.B, *A = (const __nv_bfloat16*)g.A;
    const int ff = g.N / 2, gr = min(n0 / 2 + g4, ff - 1);
    const int ra = g.glu ? gr : min(n0 + g4, g.N - 1), rb = g.glu ? ff + gr : min(n0 + g4 + 8, g.N - 1);          // rows past N repeat the last one; they are not stored
    const __nv_bfloat16 *wa = B + (size_t)ra * g.ldb + 8 * t4, *wb = B + (size_t)rb * g.ldb + 8 * t4;
    const __nv_bfloat16* xa[NT];
    bool x_ok[NT];
#pragma unroll
    for (int j = 0; j < NT; ++j) { const int m = j * 8 + g4; x_ok[j] = m < g.M; xa[j] = A + (size_t)(x_ok[j] ? m : 0) * g.lda + 8 * t4; }
    float acc[C][NT][4];
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
        for (int j = 0; j < NT; ++j) acc[c][j][0] = acc[c][j][1] = acc[c][j][2] = acc[c][j][3] = 0.f;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    const int blocks = (g.K + 31) / 32;                   // block i of this warp: steps of 64 k (two blocks) dealt to the WK warps in turn
    uint4 a[U], b[U];
    auto weights = [&](int i0) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int blk = (((i0 + u) >> 1) * WK + kw) * 2 + ((i0 + u) & 1), k = blk * 32;
            const bool ok = blk < blocks && k + 8 * t4 + 8 <= g.K;
            a[u] = ok ? __ldg(reinterpret_cast<const uint4*>(wa + k)) : zero;
            b[u] = ok ? __ldg(reinterpret_cast<const uint4*>(wb + k)) : zero;
        }
    };
    if (AHEAD) weights(0);
    if (early) pdl_enter();
    for (int i0 = 0; ; i0 += U) {
        const int first = ((i0 >> 1) * WK + kw) * 2;
        if (first >= blocks) break;
        if (!AHEAD || i0) weights(i0);
        uint4 x[U][NT];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int blk = (((i0 + u) >> 1) * WK + kw) * 2 + ((i0 + u) & 1), k = blk * 32;
            const bool ok = blk < blocks && k + 8 * t4 + 8 <= g.K;
#pragma unroll
            for (int j = 0; j < NT; ++j) x[u][j] = ok && x_ok[j] ? *reinterpret_cast<const uint4*>(xa[j] + k) : zero;
        }
        float sum[U][4];                                      // NT = 1
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t f0[4] = {a[u].x, b[u].x, a[u].y, b[u].y}, f1[4] = {a[u].z, b[u].z, a[u].w, b[u].w};
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const uint32_t x0[2] = {x[u][j].x, x[u][j].y}, x1[2] = {x[u][j].z, x[u][j].w};
                if (NT > 1) {
                    mma_bf16_16816(acc[u % C][j], f0, x0);
                    mma_bf16_16816(acc[u % C][j], f1, x1);
                    continue;
                }
                float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
                mma_bf16_16816(s0, f0, x0);
                mma_bf16_16816(s1, f1, x1);
#pragma unroll
                for (int e = 0; e < 4; ++e) sum[u][e] = s0[e] + s1[e];
            }
        }
        if (NT == 1) {
#pragma unroll
            for (int half = U / 2; half >= 1; half /= 2)
#pragma unroll
                for (int u = 0; u < half; ++u)
#pragma unroll
                    for (int e = 0; e < 4; ++e) sum[u][e] += sum[u + half][e];
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[0][0][e] += sum[0][e];
        }
    }
    // acc: rows g4 (0, 1) and g4 + 8 (2, 3), activation rows 2 t4 and 2 t4 + 1
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) part[warp][j * 8 + 2 * t4 + (e & 1)][g4 + 8 * (e >> 1)] = C == 1 ? acc[0][j][e] : (acc[0][j][e] + acc[C / 2][j][e]) + (acc[C / 4][j][e] + acc[C - 1][j][e]);
    __syncthreads();
    if (g.glu) {
        for (int i = threadIdx.x; i < TILES * NT * 8 * 8; i += FR_WARPS * 32) {
            const int r = i & 7, m = (i >> 3) % (NT * 8), t = (i >> 3) / (NT * 8);
            const int n = (blockIdx.x * TILES + t) * 8 + r;
            if (n >= ff || m >= g.M) continue;
            double gate = 0., up = 0.;
#pragma unroll
            for (int w = 0; w < WK; ++w) { gate += part[t * WK + w][m][r]; up += part[t * WK + w][m][r + 8]; }
            ((__nv_bfloat16*)g.C)[(size_t)m * g.ldc + n] = __float2bfloat16_rn(glu_f(g.glu - 1, (float)gate, (float)up, g.limit));
        }
        return;
    }
    for (int i = threadIdx.x; i < TILES * NT * 8 * 16; i += FR_WARPS * 32) {
        const int r = i & 15, m = (i >> 4) % (NT * 8), t = (i >> 4) / (NT * 8);
        const int n = (blockIdx.x * TILES + t) * 16 + r;
        if (n >= g.N || m >= g.M) continue;
        double all = 0.;
#pragma unroll
        for (int w = 0; w < WK; ++w) all += part[t * WK + w][m][r];
        const float v = epilogue_f(g.ep, (float)all);
        if (CF32) ((float*)g.C)[(size_t)m * g.ldc + n] = v;
        else ((__nv_bfloat16*)g.C)[(size_t)m * g.ldc + n] = __float2bfloat16_rn(v);
    }
}

template <int NT, int WK, int U, int OCC>
void few_launch(const GemmArgs& g, cudaStream_t s) {
    const int tiles = g.glu ? (g.N / 2 + 7) / 8 : (g.N + 15) / 16, per = FR_WARPS / WK, blocks = (tiles + per - 1) / per;
    // An SM that kernels overlap on keeps the split between cache and shared memory that the first of them had.  Behind an attention its cache would be what 200 KB of shared
    // memory leave, too little for the loads of four blocks under way: a decode step of 8 sequences, 6440 x 2560 behind the attention's output product 18.4 us, 9.7 with a split stated.
    static DevOnce once;
    if (once.need()) {
        if (cudaFuncSetAttribute(gemm_few_kernel<NT, WK, U, OCC, true>, cudaFuncAttributePreferredSharedMemoryCarveout, FR_CARVEOUT) != cudaSuccess ||
            cudaFuncSetAttribute(gemm_few_kernel<NT, WK, U, OCC, false>, cudaFuncAttributePreferredSharedMemoryCarveout, FR_CARVEOUT) != cudaSuccess) cudaGetLastError();      // a preference only
    }
    if (g.c_f32) launch_pdl(gemm_few_kernel<NT, WK, U, OCC, true>, blocks, FR_WARPS * 32, 0, s, g); else launch_pdl(gemm_few_kernel<NT, WK, U, OCC, false>, blocks, FR_WARPS * 32, 0, s, g);
}
// Which split.  8 rows, weights from memory, back to back; us with blocks of one tile and eight warps: one block an SM with 8 loads a warp under way / two with 4 / four with 4; and four
// blocks of two tiles with 4 warps each.  Up to a tile an SM a warp wants many loads under way: 1024 x 4096 4.3 / 5.6 / 7.7; 12.8, 2304 x 6912 8.3 / 9.7 / 12.8; 21.2.  Up to two
// tiles two blocks share an SM: 2560 x 6912 14.8 / 10.5 / 13.1; 21.3, 4608 x 2560 8.2 / 5.7 / 7.0; 9.4 (a decode step of four layers 2560 wide 283 -> 266 us against blocks of two
// tiles alone on an SM, 12.4 and 6.4 here).  Beyond, resident blocks cover the latency, and as a block of one tile takes half the time of one of two, the fuller rounds decide: one
// round of single tiles 4800 x 2560 11.4 / 9.0 / 7.5; 9.5, 9472 x 6912 32.1 / 24.0 / 22.6; 27.7; two rounds either way 13824 x 2560 23.5 / 16.0 / 15.0; 13.5; three for four
// 20000 x 2560 34.3 / 24.3 / 20.8; 22.9; as many 32768 x 2560 54.1 / 35.2 / 30.3; 28.4; seven for eight 65536 x 6912 205 / 154 / 139; 145; 128256 x 2560 204 / 134 / 106; 103.
// With 9 to 16 rows the registers hold half as much in flight and a second block stays resident.
template <int NT>
void few_dispatch(const GemmArgs& g, cudaStream_t s) {
    const int tiles = (g.N + 15) / 16, sms = sm_count();
    if (NT == 1) {
        if (tiles <= sms) few_launch<1, 8, 8, 1>(g, s);
        else if (tiles <= 2 * sms) few_launch<1, 8, 4, 2>(g, s);
        else {
            const int slots = 4 * sms, tiles_a_block = (tiles + slots - 1) / slots, pairs_a_block = ((tiles + 1) / 2 + slots - 1) / slots;
            if (tiles_a_block < 2 * pairs_a_block) few_launch<1, 8, 4, 4>(g, s); else few_launch<1, 4, 4, 4>(g, s);
        }
    } else {
        if (tiles <= 4 * sms) few_launch<2, 8, 4, 1>(g, s);
        else few_launch<2, 2, 4, 2>(g, s);
    }
}

template <typename T>
void simt_dispatch(const GemmArgs& g, dim3 grid, cudaStream_t s) {
    if (g.a_f32) { if (g.c_f32) launch_pdl(gemm_simt_kernel<T, true, true>, grid, 256, 0, s, g); else launch_pdl(gemm_simt_kernel<T, true, false>, grid, 256, 0, s, g); }
    else { if (g.c_f32) launch_pdl(gemm_simt_kernel<T, false, true>, grid, 256, 0, s, g); else launch_pdl(gemm_simt_kernel<T, false, false>, grid, 256, 0, s, g); }
}

int g_force_simt = -1, g_tc_min = -1;

}  // namespace

static void read_env() {
    if (g_tc_min < 0) { const char* e = getenv("WF_SEQ_TC_MIN"); g_tc_min = e ? atoi(e) : 17; }
    if (g_force_simt < 0) { const char* e = getenv("WF_SEQ_GEMM_SIMT"); g_force_simt = (e && atoi(e)) ? 1 : 0; }
}
// few rows on mma.sync, as launch_gemm chooses it by itself (9 to 16 rows go to the tcgen05 form where WF_SEQ_TC_MIN asks for it)
static bool few_rows(int dt, const GemmArgs& g) {
    return (g.M <= 8 || g.M < g_tc_min || !gemm_tc_usable(g)) && g.batch == 1 && !g.tile_group && !g.a_rows && g.M <= 16 && dt == WF_BF16 && !g.a_f32 && gemv_ok<__nv_bfloat16>(g);
}
bool gemm_glu_usable(int dt, const GemmArgs& g) {
    read_env();
    if (dt != WF_BF16 || g.algo != 0 || g_force_simt || g.c_f32 || g.ep != EP_NONE || g.N % 2) return false;
    return few_rows(dt, g) || (g.M >= g_tc_min && gemm_tc_usable(g));
}

int launch_gemm(int dt, const GemmArgs& g, cudaStream_t s) {
    if (g.M <= 0 || g.N <= 0 || g.batch <= 0) return WF_OK;
    if (g.glu && !gemm_glu_usable(dt, g)) { set_error("gemm: no gated form takes this shape"); return WF_ERR_UNSUPPORTED; }
    if (g.K <= 0 || !g.A || !g.B || !g.C) { set_error("gemm: bad arguments (M %d N %d K %d)", g.M, g.N, g.K); return WF_ERR_INVALID; }
    read_env();
    const bool few = g.batch == 1 && !g.tile_group && !g.a_rows && g.M <= 8;
    const bool few_mma = g.algo == 5 || (g.algo == 0 && !g_force_simt && few_rows(dt, g));
    if (few_mma && g.batch == 1 && !g.tile_group && !g.a_rows && g.M <= 16 && dt == WF_BF16 && !g.a_f32 && gemv_ok<__nv_bfloat16>(g)) {
        if (g.M <= 8) few_dispatch<1>(g, s); else few_dispatch<2>(g, s);
        return launch_check(cudaGetLastError(), "gemm_few");
    }
    if (g.algo == 5) { set_error("gemm: the few-row tensor-core form does not take this shape"); return WF_ERR_UNSUPPORTED; }
    if ((g.algo == 0 && few) || g.algo == 4) {      // decoding: stream the weights once
        const PairArgs none{nullptr, 0, 1};
        if (few && dt == WF_F32 && gemv_ok<float>(g)) { gemv_launch<float>(g, none, g.M, 1, s); return launch_check(cudaGetLastError(), "gemv_rows"); }
        if (few && dt == WF_BF16 && gemv_ok<__nv_bfloat16>(g)) { gemv_launch<__nv_bfloat16>(g, none, g.M, 1, s); return launch_check(cudaGetLastError(), "gemv_rows"); }
        if (g.algo == 4) { set_error("gemm: the few-row form does not take this shape"); return WF_ERR_UNSUPPORTED; }
    }
    dim3 grid((g.N + BN - 1) / BN, (g.M + BM - 1) / BM, g.batch);
    if (grid.y > 65535u || grid.z > 65535u) { set_error("gemm: grid too large"); return WF_ERR_UNSUPPORTED; }
    if (g.algo == 3 && (dt != WF_BF16 || !gemm_tc_usable(g))) { set_error("gemm: the tcgen05 form does not take this shape"); return WF_ERR_UNSUPPORTED; }
    if (dt == WF_F32) simt_dispatch<float>(g, grid, s);
    else if (g.algo == 1 || (g.algo == 0 && g_force_simt)) simt_dispatch<__nv_bfloat16>(g, grid, s);
    else if (g.algo == 3 || (g.algo == 0 && g.M >= g_tc_min && gemm_tc_usable(g))) return launch_gemm_tc(g, g.n_groups, s);
    else {
        if (g.a_f32) { if (g.c_f32) launch_pdl(gemm_mma_kernel<true, true>, grid, 128, 0, s, g); else launch_pdl(gemm_mma_kernel<true, false>, grid, 128, 0, s, g); }
        else { if (g.c_f32) launch_pdl(gemm_mma_kernel<false, true>, grid, 128, 0, s, g); else launch_pdl(gemm_mma_kernel<false, false>, grid, 128, 0, s, g); }
    }
    return launch_check(cudaGetLastError(), "gemm");
}

bool gemv_pairs_usable(int dt, const GemmArgs& g) {
    return dt == WF_F32 ? gemv_ok<float>(g) : gemv_ok<__nv_bfloat16>(g);
}

int launch_gemv_pairs(int dt, const GemmArgs& g, const int32_t* pair_expert, int n_experts, int pairs, int pair_div, cudaStream_t s) {
    if (pairs <= 0 || g.N <= 0) return WF_OK;
    if (pairs > 65535 || !gemv_pairs_usable(dt, g)) { set_error("gemv_pairs: unsupported shape"); return WF_ERR_UNSUPPORTED; }
    const PairArgs pa{pair_expert, n_experts, pair_div};
    if (dt == WF_F32) gemv_launch<float>(g, pa, 1, pairs, s); else gemv_launch<__nv_bfloat16>(g, pa, 1, pairs, s);
    return launch_check(cudaGetLastError(), "gemv_pairs");
}

}  // namespace seq
}  // namespace wf
