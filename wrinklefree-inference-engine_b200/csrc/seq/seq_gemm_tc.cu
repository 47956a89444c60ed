// bf16 matrix product on the 5th-generation tensor cores for prompt-sized row counts:  C[m, n] = sum_k A[m, k] * B[n, k], fp32 accumulate.
//
// A pair of CTAs (cta_group::2) works on one tile of 256 weight rows (UMMA M, 128 TMEM lanes in each CTA) x TN tokens (UMMA N, TN a multiple of 16 up
// to 256): each CTA holds its own 128 weight rows and HALF of the tokens in shared memory, so a stage of 64 k costs it 16 KB + TN / 2 * 128 bytes.
// That is the reason for the pair: a 128 x 128 tile of one CTA writes and reads 256 bytes of shared memory per clock of tensor time against 128 that
// the SM moves, and measured 40 to 55 % of the cuBLAS rate; at 256 x 256 the pair needs 128.
//   * persistent pairs, 10 warps: 8 epilogue (two per TMEM lane quarter), 1 TMA producer, 1 MMA issuer (first CTA only);
//   * six stages; the TMA loads of both CTAs report to the first CTA's barrier, tcgen05.commit hands a stage back to both producers;
//   * accumulators double-buffered in TMEM (2 x 256 columns): the epilogue of tile i overlaps the stream of tile i + 1;
//   * rows past the tensor and k past K are zero-filled by the TMA unit, so no shape needs padding;
//   * epilogue: tcgen05.ld 32x32b.x32 -> a thread holds its weight row's values for 32 tokens; a warp's store of one token covers 32
//     consecutive n (one 128-byte line of float, or 64 bytes of bf16);
//   * consecutive tiles share the token tile and walk the weight rows, so activations are re-read from L2, weights streamed;
//   * grouped form (routed experts): every 128-token tile names its expert; the weight tensor map covers all experts' rows stacked.
// Every wait is bounded: a wait that runs out records an error word the host checks, and the CTAs drain and leave.
#include "seq_kernels.cuh"
#include <cuda.h>

namespace wf {
namespace seq {

namespace {

constexpr int TC_ROWS = 128;                       // weight rows per CTA (256 per pair = UMMA M)
constexpr int TC_MAX_TOK = 256;                    // most tokens per tile (UMMA N)
constexpr int TC_KC = 64;                          // k per stage: 128 bytes of bf16 = one swizzle atom row
constexpr int TC_STAGES = 6;
constexpr int TC_W_BYTES = TC_ROWS * 128;          // 16 KB
constexpr int TC_STAGE_BYTES = TC_W_BYTES + TC_MAX_TOK / 2 * 128;
constexpr int TC_SMEM = TC_STAGES * TC_STAGE_BYTES + 1024;
constexpr int TC_EPW = 8;
constexpr int TC_THREADS = (TC_EPW + 2) * 32;
constexpr int TC_TMEM_COLS = 512;
constexpr unsigned long long TC_LIMIT_NS = 1000000000ull;   // a wait that lasts this long has failed

struct TcParams {
    int M, N, K;
    int tn;                        // tokens per tile
    int n_tiles, tiles;            // tiles of 256 weight rows; all tiles
    void* C; int ldc, c_f32, ep;
    int glu; float limit;          // > 0: rows [gate | up] (N = 2 ff), stored as activation glu - 1 of the pair in bf16 [M, ff]; its clamp
    const int32_t* tile_group;     // per 128-token tile: expert, or < 0 = skip (null: dense)
    int group_w_rows;              // weight rows between consecutive experts in the stacked tensor
    int* err;
};

__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {   // K-major tile, 128-byte rows, 8-row groups 1024 B apart
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3ffffu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// D f32, A bf16 (K-major), B bf16 (K-major), N, M
__device__ __forceinline__ uint32_t make_idesc(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void mma_bf16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// arrival at the same barrier of both CTAs of the pair once every MMA issued so far is done
__device__ __forceinline__ void commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ uint32_t of_first_cta(uint32_t saddr) {        // the pair's first CTA's copy of a shared-memory address
    uint32_t ra;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(ra) : "r"(saddr));
    return ra;
}
__device__ __forceinline__ bool try_wait_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// bounded wait on an mbarrier phase; false when it ran out
__device__ __forceinline__ bool wait_bounded(uint32_t bar, uint32_t parity) {
    for (int i = 0; i < 64; ++i) if (try_wait_cluster(bar, parity)) return true;
    unsigned long long t0, t1;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    do {
        if (try_wait_cluster(bar, parity)) return true;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t1));
    } while (t1 - t0 < TC_LIMIT_NS);
    return false;
}
#define TC_LD32(taddr, v)                                                                                              \
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"       \
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"                            \
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),      \
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), \
                   "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]),           \
                   "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]),           \
                   "=r"(v[30]), "=r"(v[31])                                                                             \
                 : "r"(taddr) : "memory")

// GLU: a CTA's 128 weight rows are four blocks of 16 gate rows and the 16 up rows that belong to them (one box of a four-dimensional map), so that a pair
// meets in the lanes of one warp and only the activation's result is stored.  A form of its own: the plain form's epilogue keeps its registers.
template <bool GLU>
__global__ void __launch_bounds__(TC_THREADS, 1) gemm_tc_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a,
                                                                const TcParams p) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[TC_STAGES], empty_bar[TC_STAGES], tfull_bar[2], tempty_bar[2], drained;
    __shared__ uint32_t tmem_base_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int rank = (int)(blockIdx.x & 1), pair = (int)(blockIdx.x >> 1), pairs = (int)(gridDim.x >> 1);
    const int my_tiles = p.tiles > pair ? (p.tiles - pair + pairs - 1) / pairs : 0;
    const int kchunks = (p.K + TC_KC - 1) / TC_KC;

    if (tid == 0) {
        for (int s = 0; s < TC_STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&tfull_bar[b], 1); mbar_init(&tempty_bar[b], 2 * TC_EPW); }
        mbar_init(&drained, 1);
        fence_mbar_init();
    }
    if (warp == TC_EPW + 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "n"(TC_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");      // the other CTA's barriers are initialised
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_s;
    pdl_wait_prior();                                  // barriers, TMEM and the pair's meeting above overlap the kernel before

    // every role of both CTAs walks the same list of tiles and skips the same ones; `it` counts ring items, `done` counts tiles that were computed
    if (warp == TC_EPW) {
        // ------------------------------------------------------------ TMA producer
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_w) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_a) : "memory");
            const uint32_t full0 = of_first_cta(smem_u32(&full_bar[0]));
            const int half = p.tn / 2;
            int it = 0;
            bool ok = true;
            for (int tl = 0; tl < my_tiles && ok; ++tl) {
                const int tile = pair + tl * pairs;
                const int mt = tile / p.n_tiles, nt = tile - mt * p.n_tiles;
                int w_row = nt * 2 * TC_ROWS + rank * TC_ROWS;
                if (p.tile_group) {
                    const int e = p.tile_group[mt];
                    if (e < 0) continue;
                    w_row += e * p.group_w_rows;
                }
                for (int kc = 0; kc < kchunks; ++kc, ++it) {
                    const int s = it % TC_STAGES;
                    if (it >= TC_STAGES && !wait_bounded(smem_u32(&empty_bar[s]), (uint32_t)(((it / TC_STAGES) & 1) ^ 1))) { ok = false; break; }
                    if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * (TC_W_BYTES + half * 128));      // both CTAs' loads report here
                    if (GLU)
                        asm volatile("cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
                                     ::"r"(ring + s * TC_STAGE_BYTES), "l"(&tmap_w), "r"(kc * TC_KC), "r"(0), "r"(0), "r"(w_row / 32), "r"(full0 + s * 8) : "memory");
                    else
                        asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                                     ::"r"(ring + s * TC_STAGE_BYTES), "l"(&tmap_w), "r"(kc * TC_KC), "r"(w_row), "r"(full0 + s * 8) : "memory");
                    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                                 ::"r"(ring + s * TC_STAGE_BYTES + TC_W_BYTES), "l"(&tmap_a), "r"(kc * TC_KC), "r"(mt * p.tn + rank * half), "r"(full0 + s * 8) : "memory");
                }
            }
            // the last stages' hand-backs come from the other CTA too: none may be under way when this CTA leaves
            for (int j = it > TC_STAGES ? it - TC_STAGES : 0; ok && j < it; ++j) ok = wait_bounded(smem_u32(&empty_bar[j % TC_STAGES]), (uint32_t)((j / TC_STAGES) & 1));
            if (!ok) {                                                     // the pair leaves early, but not before its copies have landed (both CTAs' report to the first)
                atomicExch(p.err, 1);
                for (int j = it > TC_STAGES ? it - TC_STAGES : 0; rank == 0 && j < it; ++j) wait_bounded(smem_u32(&full_bar[j % TC_STAGES]), (uint32_t)((j / TC_STAGES) & 1));
            }
        }
        __syncwarp();
    } else if (warp == TC_EPW + 1) {
        // ------------------------------------------------------------ MMA issuer: one elected thread of the first CTA runs the whole loop
        const uint32_t idesc = make_idesc(2 * TC_ROWS, p.tn);
        const uint64_t adesc0 = smem_desc_sw128(ring);
        const uint64_t bdesc0 = smem_desc_sw128(ring + TC_W_BYTES);
        uint32_t elected;
        asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(elected));
        if (elected && rank == 0) {
            int it = 0, done = 0;
            bool ok = true;
            for (int tl = 0; tl < my_tiles && ok; ++tl) {
                const int tile = pair + tl * pairs;
                const int mt = tile / p.n_tiles;
                if (p.tile_group && p.tile_group[mt] < 0) continue;
                const int buf = done & 1;
                if (done >= 2 && !wait_bounded(smem_u32(&tempty_bar[buf]), (uint32_t)(((done >> 1) & 1) ^ 1))) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d_tmem = tmem + buf * TC_MAX_TOK;
                for (int kc = 0; kc < kchunks; ++kc, ++it) {
                    const int s = it % TC_STAGES;
                    if (!wait_bounded(smem_u32(&full_bar[s]), (uint32_t)((it / TC_STAGES) & 1))) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t ad = adesc0 + (uint64_t)(s * (TC_STAGE_BYTES >> 4));
                    const uint64_t bd = bdesc0 + (uint64_t)(s * (TC_STAGE_BYTES >> 4));
                    mma_bf16_pair(d_tmem, ad, bd, idesc, kc != 0 ? 1u : 0u);          // 16 k per instruction = 32 bytes = +2 in the descriptor
                    mma_bf16_pair(d_tmem, ad + 2, bd + 2, idesc, 1u);
                    mma_bf16_pair(d_tmem, ad + 4, bd + 4, idesc, 1u);
                    mma_bf16_pair(d_tmem, ad + 6, bd + 6, idesc, 1u);
                    commit_pair(smem_u32(&empty_bar[s]));
                }
                if (!ok) break;
                commit_pair(smem_u32(&tfull_bar[buf]));
                ++done;
            }
            if (!ok) {                                                     // nor while a product still reads shared memory
                atomicExch(p.err, 2);
                commit_pair(smem_u32(&drained));
                wait_bounded(smem_u32(&drained), 0);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue warps: TMEM -> C
        const int q = warp & 3, part = warp >> 2;                          // lane quarter; the two warps of a quarter take alternate 32-token chunks
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        const uint32_t tempty0 = of_first_cta(smem_u32(&tempty_bar[0]));
        const int chunks = (p.tn + 31) / 32;
        int done = 0;
        bool ok = true;
        for (int tl = 0; tl < my_tiles && ok; ++tl) {
            const int tile = pair + tl * pairs;
            const int mt = tile / p.n_tiles, nt = tile - mt * p.n_tiles;
            if (p.tile_group && p.tile_group[mt] < 0) continue;
            const int buf = done & 1;
            const int n = nt * 2 * TC_ROWS + rank * TC_ROWS + q * 32 + lane;   // this thread's weight row = output column
            const bool n_ok = n < p.N;
            if (!__all_sync(0xffffffffu, wait_bounded(smem_u32(&tfull_bar[buf]), (uint32_t)((done >> 1) & 1)))) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int c = part; c < chunks; c += 2) {
                uint32_t r[32];
                TC_LD32(tmem + lane_base + buf * TC_MAX_TOK + c * 32, r);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                const int m0 = mt * p.tn + c * 32;
                int mcnt = p.M - m0 < 32 ? p.M - m0 : 32;                  // tokens of this chunk that exist and belong to this tile (warp-uniform)
                if (p.tn - c * 32 < mcnt) mcnt = p.tn - c * 32;
                if (GLU) {
                    // lanes 0 .. 15 hold gate rows and keep the chunk's tokens 0 .. 15, lanes 16 .. 31 the up rows and keep the others; they swap the rest
                    const bool up = lane >= 16;
                    __nv_bfloat16* dst = (__nv_bfloat16*)p.C + (size_t)(m0 + (up ? 16 : 0)) * p.ldc + (n >> 5) * 16 + (n & 15);
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const float got = __shfl_xor_sync(0xffffffffu, __uint_as_float(up ? r[j] : r[16 + j]), 16), mine = __uint_as_float(up ? r[16 + j] : r[j]);
                        const float a = glu_f(p.glu - 1, up ? got : mine, up ? mine : got, p.limit);
                        if (n_ok && (up ? 16 : 0) + j < mcnt) *dst = __float2bfloat16_rn(a);
                        dst += p.ldc;
                    }
                    __syncwarp();
                    continue;
                }
                if (p.ep != EP_NONE) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(epilogue_f(p.ep, __uint_as_float(r[j])));
                }
                if (n_ok) {
                    if (p.c_f32) {
                        float* dst = (float*)p.C + (size_t)m0 * p.ldc + n;
#pragma unroll
                        for (int j = 0; j < 32; ++j) { if (j < mcnt) *dst = __uint_as_float(r[j]); dst += p.ldc; }
                    } else {
                        __nv_bfloat16* dst = (__nv_bfloat16*)p.C + (size_t)m0 * p.ldc + n;
#pragma unroll
                        for (int j = 0; j < 32; ++j) { if (j < mcnt) *dst = __float2bfloat16_rn(__uint_as_float(r[j])); dst += p.ldc; }
                    }
                }
                __syncwarp();
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(tempty0 + buf * 8) : "memory");
            ++done;
        }
        if (!ok && lane == 0) atomicExch(p.err, 3);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");      // nobody leaves while the other CTA may still signal or read here
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (warp == TC_EPW + 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TC_TMEM_COLS) : "memory");
    }
}

// Tokens per tile.  A tile's stage takes 2 tn clk on the tensor cores, or the time of the pair's loads where that is longer (256 weight rows and tn
// tokens of 128 bytes into two SMs at about 64 bytes a clock each); its start and end cost about as much as four stages.  The whole takes as many
// rounds as the pairs need for all tiles: of the sizes with the least of both, the largest.
int tokens_per_tile(int M, int N, int K, int pairs) {
    const int rows = (N + 2 * TC_ROWS - 1) / (2 * TC_ROWS), stages = (K + TC_KC - 1) / TC_KC;
    int best = TC_MAX_TOK;
    double best_t = 1e30;
    for (int tn = TC_MAX_TOK; tn >= 32; tn -= 16) {
        const long long tiles = (long long)rows * ((M + tn - 1) / tn);
        const long long rounds = (tiles + pairs - 1) / pairs;
        const double stage = 2. * tn > 256. + tn ? 2. * tn : 256. + tn;
        const double t = (double)rounds * stage * (stages + 1) + 4. * stage;
        if (t < best_t * 0.995) { best_t = t; best = tn; }
    }
    return best;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn g_encode = nullptr;
DevOnce g_attr;
int* g_err_dev[64] = {nullptr};

int encode_2d(CUtensorMap* tm, const void* base, uint64_t rows, uint64_t cols, uint64_t row_stride_elems, uint32_t box_rows) {
    const cuuint64_t gdim[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t gstride[1] = {(cuuint64_t)row_stride_elems * 2};
    const cuuint32_t box[2] = {TC_KC, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult cr = g_encode(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)base, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                 CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) { set_error("gemm_tc: tensor map failed (%d)", (int)cr); return WF_ERR_CUDA; }
    return WF_OK;
}

}  // namespace

bool gemm_tc_usable(const GemmArgs& g) {
    if (g.a_f32 || g.batch != 1 || g.a_rows) return false;
    if (g.lda % 8 || g.ldb % 8 || ((uintptr_t)g.A & 15) || ((uintptr_t)g.B & 15) || g.K < 8 || g.lda < g.K || g.ldb < g.K) return false;
    if (g.tile_group && (g.group_stride % g.ldb)) return false;
    if (g.glu && (g.tile_group || g.c_f32 || g.ep != EP_NONE || g.N % 32)) return false;
    return true;
}

void* tensor_map_encoder() {
    if (!g_encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult qr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qr) == cudaSuccess && qr == cudaDriverEntryPointSuccess)
            g_encode = (EncodeTiledFn)fn;
    }
    return (void*)g_encode;
}

int* tc_error_word(bool make) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev > 63) dev = 0;
    if (!g_err_dev[dev] && make) {
        if (cuda_check(cudaMalloc((void**)&g_err_dev[dev], 4), "cudaMalloc")) { g_err_dev[dev] = nullptr; return nullptr; }
        if (cuda_check(cudaMemset(g_err_dev[dev], 0, 4), "memset")) return nullptr;
    }
    return g_err_dev[dev];
}

int gemm_tc_error(cudaStream_t s) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev > 63 || !g_err_dev[dev]) return 0;
    int h = 0;
    if (cudaMemcpyAsync(&h, g_err_dev[dev], 4, cudaMemcpyDeviceToHost, s) != cudaSuccess) return -1;
    if (cudaStreamSynchronize(s) != cudaSuccess) return -1;
    return h;
}

// n_groups: number of stacked weight matrices (1 when dense)
int launch_gemm_tc(const GemmArgs& g, int n_groups, cudaStream_t s) {
    if (g_attr.need()) {
        cudaFuncSetAttribute(gemm_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM);
        cudaFuncSetAttribute(gemm_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM);
    }
    if (!tensor_map_encoder()) { set_error("gemm_tc: cuTensorMapEncodeTiled unavailable"); return WF_ERR_CUDA; }
    int* err = tc_error_word();
    if (!err) return WF_ERR_CUDA;
    CUtensorMap tw, ta;
    const int group_w_rows = g.tile_group ? (int)(g.group_stride / g.ldb) : 0;
    const uint64_t w_rows = g.tile_group ? (uint64_t)(n_groups - 1) * group_w_rows + g.N : (uint64_t)g.N;
    if (g.glu) {
        const cuuint64_t dim[4] = {(cuuint64_t)g.K, 16, 2, (cuuint64_t)(g.N / 32)}, row = (cuuint64_t)g.ldb * 2, stride[3] = {row, row * (g.N / 2), row * 16};
        const cuuint32_t box[4] = {TC_KC, 16, 2, TC_ROWS / 32}, one[4] = {1, 1, 1, 1};
        const CUresult cr = g_encode(&tw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, (void*)g.B, dim, stride, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (cr != CUDA_SUCCESS) { set_error("gemm_tc: tensor map failed (%d)", (int)cr); return WF_ERR_CUDA; }
    } else if (int rc = encode_2d(&tw, g.B, w_rows, g.K, g.ldb, TC_ROWS)) return rc;
    const int sms = sm_count(), pairs = sms / 2;
    const int tn = g.tile_group ? GEMM_BM : tokens_per_tile(g.M, g.N, g.K, pairs);
    if (int rc = encode_2d(&ta, g.A, g.M, g.K, g.lda, tn / 2)) return rc;
    TcParams p;
    p.M = g.M; p.N = g.N; p.K = g.K;
    p.tn = tn;
    p.n_tiles = (g.N + 2 * TC_ROWS - 1) / (2 * TC_ROWS);
    p.tiles = p.n_tiles * ((g.M + tn - 1) / tn);
    p.C = g.C; p.ldc = g.ldc; p.c_f32 = g.c_f32; p.ep = g.ep;
    p.glu = g.glu; p.limit = g.limit;
    p.tile_group = g.tile_group; p.group_w_rows = group_w_rows;
    p.err = err;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (p.tiles < pairs ? p.tiles : pairs));
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = TC_SMEM;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    return launch_check(g.glu ? cudaLaunchKernelEx(&cfg, gemm_tc_kernel<true>, tw, ta, p) : cudaLaunchKernelEx(&cfg, gemm_tc_kernel<false>, tw, ta, p), "gemm_tc");
}

}  // namespace seq
}  // namespace wf
