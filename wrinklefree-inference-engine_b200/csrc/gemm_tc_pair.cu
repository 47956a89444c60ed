// Ternary product on CTA pairs (tcgen05, cta_group::2, kind::i8):  S[m,n] = sum_k code[n,k] * a[m,k],  exact int32.
//
// Two CTAs work on one tile of 256 weight rows (UMMA M: 128 TMEM lanes in each) x TN tokens (UMMA N, 32 .. 256).
//   * An MMA of 32 k takes about 100 clk up to 128 tokens, 113 at 192 and 131 at 256 (64 .. 128 clk are its work; two accumulators in turn made it 140), so
//     a tile is as wide as the token count lets it be: 256 rows x 192 tokens are 3.8 times the work of gemm_tc.cu's 128 x 128 for 1.2 times its clocks.
//   * Each CTA holds HALF of the tile's activations.  One load brings 2 or 4 k-blocks: at one block a load the issuing thread paced the kernel (420 clk a block).
//   * Packed weights come by TMA, four k-blocks (16 KB) at a time, swizzled so that the unpack warps' 16-byte reads meet no bank twice.  (Read from
//     global memory row by row, the checkpoint layout costs the load unit 256 clk of each 128-k stage.)
//   * NU groups of four unpack warps expand 2-bit codes to bytes into a TMEM operand ring, as the A operand of the MMAs; the next item's codes are read
//     while the present one waits for its TMEM stage.  Three groups: an item takes a group 900 clk, most of it latency.
//   * Up to 192 tokens two accumulators and a ring of four stages fill TMEM and the epilogue of a tile overlaps the next one's stream; at 256 there is one
//     accumulator and eight stages, and the epilogue stands alone (2.5 us a tile, the rate at which L2 takes what all SMs write at once).
// Roles of a CTA: 8 epilogue warps, 4 * NU unpack warps, one warp loading activations, one loading weights, one issuing MMAs (first CTA of the pair).
// Measured without / with it (us): 6912 x 2560, 1987 tokens 44.8 / 34.8; 2560 x 6912, 16384 tokens 246 / 177 (3.3 PTOP/s); gate | up of 13824 x 2560, 512
// tokens 43 / 24; 14336 x 4096, 48 tokens 17.4 / 13.1.
// Every wait is bounded: one that runs out leaves a code in the device's wait word (tc_wait_word), and the CTAs wait for their own copies and products and
// leave.  The word is host memory, so that the next ternary call on the device and the engine's waits see it without a copy: they fail with WF_ERR_CUDA once.
#include "gemm_tc_common.cuh"
#include "gemm_tc_pair_walk.h"
#include "kernels.cuh"
#include <string.h>
#include <atomic>
#include <mutex>

namespace wf {

namespace {

constexpr int TP_ROWS = 128;                        // weight rows per CTA
constexpr int TP_MAX_TOK = 256;                     // most tokens per tile (UMMA N)
constexpr int TP_BK = 128;                          // k per stage
constexpr int TP_AS_MAX = 16;                       // most activation loads in flight
constexpr int TP_W_BYTES = TP_ROWS * TP_WKB * 32;
constexpr int TP_A_COLS = TP_BK / 4;
constexpr int TP_EPW = 8;
constexpr int TP_EP_CHUNKS = TP_MAX_TOK / 32 / (TP_EPW / 4);   // 32-token chunks per epilogue warp
constexpr int TP_TOK_BYTES = TP_EPW * TP_EP_CHUNKS * 32 * 8;
constexpr int TP_SMEM = 220 * 1024;                 // weights, token table, the rest is the activation ring: 163 KB
constexpr int TP_ACT_RING = TP_SMEM - 1024 - TP_WS * TP_W_BYTES - TP_TOK_BYTES;
constexpr int tp_threads(int nu) { return (TP_EPW + 4 * nu + 3) * 32; }
constexpr unsigned long long TP_LIMIT_NS = 1000000000ull;      // a wait that lasts this long has failed

struct TpParams {
    int M, N, K, KB;
    int tn, n_tiles, tiles;
    int i2s;
    int akb, as;         // k-blocks per activation load, loads in flight
    int ahead;           // the weights were complete long before: their loads and expansion do not wait for the kernel before, and the next one may come early
    int* err;            // the wait word
    EpiParams ep;
};

__device__ __forceinline__ void gave_up(const TpParams& p, int role) {
    *(volatile int*)p.err = role;
    __threadfence_system();
}
__device__ __forceinline__ uint32_t of_first_cta(uint32_t saddr) {        // the pair's first CTA's copy of a shared-memory address
    uint32_t ra;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(ra) : "r"(saddr));
    return ra;
}
__device__ __forceinline__ bool try_wait_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __noinline__ bool wait_long(uint32_t bar, uint32_t parity) {
    unsigned long long t0, t1;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    do {
        if (try_wait_cluster(bar, parity)) return true;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t1));
    } while (t1 - t0 < TP_LIMIT_NS);
    return try_wait_cluster(bar, parity);              // the time may have passed between the look and the clock, with the SM in other hands
}
// (one look inline and the rest out of line: the issuing thread's loop paces a stage when it is long)
__device__ __forceinline__ bool wait_bounded(uint32_t bar, uint32_t parity) { return try_wait_cluster(bar, parity) || wait_long(bar, parity); }
__device__ __forceinline__ void arrive_remote(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory"); }
// D[tmem] (+)= A[tmem] * B[smem], rows of both CTAs
__device__ __forceinline__ void mma_i8_pair(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// arrival at the same barrier of both CTAs once every MMA issued so far is done
__device__ __forceinline__ void commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}

// The linear epilogue of 32 tokens (m0 ..) of one weight row per lane: the rounding sequence of linear_value (linear_common.cuh).
// tk[j]: {fl(w_s * Sigma a) where one scale serves the matrix, the bits of Sigma a for whole-number results, else (float) Sigma a; activation scale} of token m0 + j.
struct PairEp {
    int mode;
    bool relu2, resid, obf16, fold;
    __device__ __forceinline__ explicit PairEp(const EpiParams& e) {
        mode = e.out_mode;
        const bool lin = mode == WF_OUT_LINEAR;
        relu2 = lin && (e.epi_flags & WF_EPI_RELU2_MUL);
        resid = lin && (e.epi_flags & WF_EPI_RESIDUAL);
        obf16 = lin && e.out_dtype == WF_BF16;
        fold = lin && !relu2 && !resid && e.nseg <= 1;
    }
};

__device__ __forceinline__ void pair_store(const EpiParams& ep, const PairEp& e, const uint32_t (&v)[32], const float2* tk, int m0, int mcnt, int n, float ws, int lane) {
    const size_t ldo = (size_t)ep.ldo;
    auto folded = [&](int j) { const float2 t = tk[j]; return __fmul_rn(__fsub_rn(__fmul_rn((float)(int)v[j], ws), t.x), t.y); };
    auto plain = [&](int j) { const float2 t = tk[j]; return __fmul_rn(__fsub_rn(__fmul_rn((float)(int)v[j], ws), __fmul_rn(ws, t.x)), t.y); };
    if (e.relu2) {
        // rows alternate in blocks of 16 gate and 16 up rows: lanes 0 .. 15 keep tokens 0 .. 15 and hand over the others, lanes 16 .. 31 the reverse
        const bool up = lane >= 16;
        uint32_t h[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) h[i] = pack_bf16x2(plain(2 * i), plain(2 * i + 1));
        const int col = (n >> 5) * 16 + (n & 15), first = up ? 16 : 0;
        __nv_bfloat16* ob = reinterpret_cast<__nv_bfloat16*>(ep.out) + (size_t)(m0 + first) * ldo + col;
        float* of = reinterpret_cast<float*>(ep.out) + (size_t)(m0 + first) * ldo + col;
        const bool n_ok = n < ep.N;                                        // N is a multiple of 32: the same for the whole warp
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? h[i] : h[8 + i], 16), mine = up ? h[8 + i] : h[i];
            const uint32_t g2 = up ? got : mine, u2 = up ? mine : got;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const float g = k ? bf16hi(g2) : bf16lo(g2), u = k ? bf16hi(u2) : bf16lo(u2);
                const float r = fmaxf(g, 0.f), y = bf16_round(r * r) * u;
                if (n_ok && first + 2 * i + k < mcnt) {
                    if (e.obf16) *ob = __float2bfloat16_rn(y);
                    else *of = bf16_round(y);
                }
                ob += ldo; of += ldo;
            }
        }
        return;
    }
    if (n >= ep.N) return;
    auto each = [&](auto* op, auto value) {
        op += (size_t)m0 * ldo + n;
        if (mcnt == 32) {
#pragma unroll
            for (int j = 0; j < 32; ++j) { *op = value(j); op += ldo; }
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) { if (j < mcnt) *op = value(j); op += ldo; }
        }
    };
    float* const of = reinterpret_cast<float*>(ep.out);
    __nv_bfloat16* const ob = reinterpret_cast<__nv_bfloat16*>(ep.out);
    if (e.mode == WF_OUT_COMPAT_F32) each(of, [&](int j) { return __fmul_rn((float)(int)v[j], ep.host_scale); });
    else if (e.mode == WF_OUT_I32_PLUS1) each(reinterpret_cast<int32_t*>(ep.out), [&](int j) { return (int32_t)v[j]; });
    else if (e.mode == WF_OUT_I32) each(reinterpret_cast<int32_t*>(ep.out), [&](int j) { return (int32_t)v[j] - __float_as_int(tk[j].x); });
    else if (e.resid) {
        const __nv_bfloat16* rp = ep.residual + (size_t)m0 * ldo + n;
        auto added = [&](int j) { return __bfloat162float(rp[(size_t)j * ldo]) + bf16_round(plain(j)); };
        if (e.obf16) each(ob, [&](int j) { return __float2bfloat16_rn(added(j)); });
        else each(of, added);
    } else if (e.obf16) {
        if (e.fold) each(ob, [&](int j) { return __float2bfloat16_rn(folded(j)); });
        else each(ob, [&](int j) { return __float2bfloat16_rn(plain(j)); });
    } else if (e.fold) each(of, folded);
    else each(of, plain);
}

template <int NU, int NBUF, bool RAGGED>
__global__ void __launch_bounds__(tp_threads(NU), 1) ternary_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_w,
                                                                              const TpParams p) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t act_full[TP_AS_MAX];   // first CTA: both CTAs' activation bytes of a load are there
    __shared__ __align__(8) uint64_t act_empty[TP_AS_MAX];  // both: the MMAs of a load are done
    __shared__ __align__(8) uint64_t a_full[8];             // first CTA: the unpack warps of both CTAs have written a TMEM stage
    __shared__ __align__(8) uint64_t a_empty[8];            // both: the MMAs of a TMEM stage are done
    __shared__ __align__(8) uint64_t w_full[TP_WS], w_empty[TP_WS];
    __shared__ __align__(8) uint64_t tfull_bar[2];          // both: an accumulator is complete
    __shared__ __align__(8) uint64_t tempty_bar[2];         // first CTA: the epilogue warps of both CTAs have read an accumulator
    __shared__ __align__(8) uint64_t drained;
    __shared__ uint32_t tmem_base_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t wring = ring, aring = ring + TP_WS * TP_W_BYTES;
    const int AS = p.as, akb = p.akb, act_bytes = p.tn / 2 * TP_BK;
    const int rank = (int)(blockIdx.x & 1), pair = (int)(blockIdx.x >> 1), pairs = (int)(gridDim.x >> 1);
    const int my_tiles = p.tiles > pair ? (p.tiles - pair + pairs - 1) / pairs : 0;
    const int KB = p.KB, n_items = my_tiles * KB, wloads = (KB + TP_WKB - 1) / TP_WKB, aloads = (KB + p.akb - 1) / p.akb;
    constexpr int TP_ACC = NBUF == 2 ? 192 : 256, TP_A_COL0 = NBUF * TP_ACC;      // columns of an accumulator; where the operand ring starts
    constexpr int TP_TS = (512 - TP_A_COL0) / TP_A_COLS;                          // stages of that ring
    constexpr int W_ACT = TP_EPW + 4 * NU, W_WGT = W_ACT + 1, W_MMA = W_ACT + 2;

    if (tid == 0) {
        for (int s = 0; s < AS; ++s) { mbar_init(&act_full[s], 1); mbar_init(&act_empty[s], 1); }
        for (int s = 0; s < TP_TS; ++s) { mbar_init(&a_full[s], 8); mbar_init(&a_empty[s], 1); }
        for (int s = 0; s < TP_WS; ++s) { mbar_init(&w_full[s], 1); mbar_init(&w_empty[s], 4 * TP_WKB); }
        for (int b = 0; b < 2; ++b) { mbar_init(&tfull_bar[b], 1); mbar_init(&tempty_bar[b], 2 * TP_EPW); }
        mbar_init(&drained, 1);
        fence_mbar_init();
    }
    if (warp == W_MMA) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "n"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");      // the other CTA's barriers are initialised
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    if (p.ahead) pdl_launch_dependents();
    if (!p.ahead || warp < TP_EPW || warp == W_ACT) pdl_wait_prior();   // barriers, TMEM and the pair's meeting above overlap the kernel before

    if (warp == W_ACT) {
        // ------------------------------------------------------------ activations: this CTA's half of the tile's tokens
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_q) : "memory");
            const uint32_t full0 = of_first_cta(smem_u32(&act_full[0]));
            const int half = p.tn / 2;
            int it = 0, s = 0;
            uint32_t ph = 1;                          // parity of the hand-back that slot s waits for
            bool ok = true;
            for (int tl = 0; tl < my_tiles && ok; ++tl) {
                const int m0 = (pair + tl * pairs) / p.n_tiles * p.tn + rank * half;
                for (int l = 0; l < aloads; ++l, ++it) {
                    if (it >= AS && !wait_bounded(smem_u32(&act_empty[s]), ph)) { ok = false; break; }
                    if (rank == 0) mbar_expect_tx(&act_full[s], 2 * akb * act_bytes);       // both CTAs' loads report here
                    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                                 ::"r"(aring + s * akb * act_bytes), "l"(&tmap_q), "r"(0), "r"(m0), "r"(l * akb), "r"(full0 + s * 8) : "memory");
                    if (++s == AS) { s = 0; ph ^= 1u; }
                }
            }
            // the last stages' hand-backs come from the first CTA: none may be under way when this CTA leaves
            for (int j = it > AS ? it - AS : 0; ok && j < it; ++j) ok = wait_bounded(smem_u32(&act_empty[j % AS]), (uint32_t)((j / AS) & 1));
            if (!ok) {                                                     // leaves early, but not before the pair's copies have landed
                gave_up(p, 1);
                for (int j = it > AS ? it - AS : 0; rank == 0 && j < it; ++j) wait_bounded(smem_u32(&act_full[j % AS]), (uint32_t)((j / AS) & 1));
            }
        }
        __syncwarp();
    } else if (warp == W_WGT) {
        // ------------------------------------------------------------ packed weights of this CTA's 128 rows, four k-blocks a load
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tmap_w) : "memory");
            int c = 0;
            bool ok = true;
            for (int tl = 0; tl < my_tiles && ok; ++tl) {
                const int tile = pair + tl * pairs;
                const int row = (tile - tile / p.n_tiles * p.n_tiles) * 2 * TP_ROWS + rank * TP_ROWS;
                for (int l = 0; l < wloads; ++l, ++c) {
                    const int s = c % TP_WS;
                    if (c >= TP_WS && !wait_bounded(smem_u32(&w_empty[s]), (uint32_t)(((c / TP_WS) & 1) ^ 1))) { ok = false; break; }
                    mbar_expect_tx(&w_full[s], TP_W_BYTES);
                    if (p.i2s)
                        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                                     ::"r"(wring + s * TP_W_BYTES), "l"(&tmap_w), "r"(l * TP_WKB * 32), "r"(row), "r"(smem_u32(&w_full[s])) : "memory");
                    else
                        asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
                                     ::"r"(wring + s * TP_W_BYTES), "l"(&tmap_w), "r"(0), "r"(0), "r"(l * TP_WKB), "r"(row / 16), "r"(smem_u32(&w_full[s])) : "memory");
                }
            }
            if (!ok) {
                gave_up(p, 2);
                for (int j = c > TP_WS ? c - TP_WS : 0; j < c; ++j) wait_bounded(smem_u32(&w_full[j % TP_WS]), (uint32_t)((j / TP_WS) & 1));
            }
        }
        __syncwarp();
    } else if (warp == W_MMA) {
        // ------------------------------------------------------------ MMA issuer: one elected thread of the first CTA; ring positions are constants
        const uint32_t idesc = tc_idesc(2 * TP_ROWS, p.tn);
        const uint64_t bdesc0 = tc_smem_desc_sw128(aring);
        const uint32_t a_tmem0 = __shfl_sync(0xffffffffu, tmem, 0) + TP_A_COL0;
        const uint32_t act0 = smem_u32(&act_full[0]), actd0 = smem_u32(&act_empty[0]), afull0 = smem_u32(&a_full[0]), aempty0 = smem_u32(&a_empty[0]);
        uint32_t elected;
        asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(elected));
        if (elected && rank == 0) {
            auto stream = [&]() -> bool {
                uint32_t aph = 0, tph = 0, d_tmem = 0, as = 0;
                uint64_t bd = bdesc0;
                int kb = 0, ka = 0, tl = 0;           // k-block in the tile and in its activation load, tile
                for (int left = n_items; left > 0; left -= TP_TS) {
#pragma unroll
                    for (int s = 0; s < TP_TS; ++s) {
                        if (s >= left) return true;
                        if (kb == 0) {   // a new tile: its accumulator must have been read
                            const int buf = tl % NBUF;
                            if (!wait_bounded(smem_u32(&tempty_bar[buf]), (uint32_t)(((tl / NBUF) & 1) ^ 1))) return false;
                            d_tmem = a_tmem0 - TP_A_COL0 + buf * TP_ACC;
                        }
                        if (ka == 0) {   // a new load of activations
                            if (!wait_bounded(act0 + as * 8, aph)) return false;
                            bd = bdesc0 + (uint64_t)(as * (uint32_t)(akb * act_bytes >> 4));
                        }
                        if (!wait_bounded(afull0 + s * 8, tph)) return false;
                        tc_fence_after();
                        const uint32_t at = a_tmem0 + s * TP_A_COLS;
                        mma_i8_pair(d_tmem, at, bd, idesc, kb != 0 ? 1u : 0u);
                        mma_i8_pair(d_tmem, at + 8, bd + 2, idesc, 1u);
                        mma_i8_pair(d_tmem, at + 16, bd + 4, idesc, 1u);
                        mma_i8_pair(d_tmem, at + 24, bd + 6, idesc, 1u);
                        commit_pair(aempty0 + s * 8);
                        bd += (uint64_t)(act_bytes >> 4);
                        ++ka; ++kb;
                        if (ka == akb || kb == KB) {
                            commit_pair(actd0 + as * 8);
                            ka = 0;
                            if (++as == (uint32_t)AS) { as = 0; aph ^= 1u; }
                        }
                        if (kb == KB) {
                            commit_pair(smem_u32(&tfull_bar[tl % NBUF]));
                            kb = 0; ++tl;
                        }
                    }
                    tph ^= 1u;
                }
                return true;
            };
            if (!stream()) {                                               // not while a product still reads shared memory
                gave_up(p, 3);
                commit_pair(smem_u32(&drained));
                wait_bounded(smem_u32(&drained), 0);
            }
        }
        __syncwarp();
    } else if (warp >= TP_EPW) {
        // ------------------------------------------------------------ unpack warps: 2-bit weights -> byte codes -> TMEM
        const int q = warp & 3, grp = (warp - TP_EPW) >> 2;
        const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16) + TP_A_COL0;
        const uint32_t afull0 = of_first_cta(smem_u32(&a_full[0]));
        const int row = q * 32 + lane;
        // packed layout: 128-byte rows of four k-blocks, 16-byte chunk c at c ^ (row & 7).  Tile layout: [row / 16][k-block][row % 8] of 64 bytes, chunk c
        // (packed bytes 4c .. and 16 + 4c .. of rows r and r + 8) at c ^ (row % 8 / 2)
        const uint32_t rbase = p.i2s ? (uint32_t)(row * 128) : (uint32_t)((row >> 4) * (TP_WKB * 512) + (row & 7) * 64);
        const uint32_t rx = p.i2s ? (uint32_t)(row & 7) : (uint32_t)((row & 7) >> 1);
        const bool odd = (row >> 3) & 1;
        const bool i2s = p.i2s != 0;
        PairWeightWalk<RAGGED> walk(grp, NU, KB);
        bool ok = true;
        uint32_t pk[8], empty = 0;                    // an item's packed codes, and the hand-back barrier of their buffer
        auto landed = [&](int load) { return __all_sync(0xffffffffu, wait_bounded(smem_u32(&w_full[load % TP_WS]), (uint32_t)((load / TP_WS) & 1))) != 0; };
        auto pass_by = [&](int load) { if (lane == 0) mbar_arrive(&w_empty[load % TP_WS]); };
        auto fetch = [&]() -> bool {
            if (!walk.next(landed, pass_by)) return false;
            const int ws = walk.load % TP_WS, j = walk.part;
            empty = smem_u32(&w_empty[ws]);
            const uint32_t src = wring + ws * TP_W_BYTES + rbase;
            if (i2s) {
#pragma unroll
                for (int c = 0; c < 2; ++c)
                    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(pk[4 * c]), "=r"(pk[4 * c + 1]), "=r"(pk[4 * c + 2]), "=r"(pk[4 * c + 3])
                                 : "r"(src + (((uint32_t)(2 * j + c) ^ rx) << 4)) : "memory");
            } else {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint32_t a, b, d, e;
                    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(a), "=r"(b), "=r"(d), "=r"(e) : "r"(src + (uint32_t)(j * 512) + (((uint32_t)c ^ rx) << 4)) : "memory");
                    pk[c] = odd ? b : a;
                    pk[4 + c] = odd ? e : d;
                }
            }
            return true;
        };
        if (grp < n_items) ok = fetch();
        for (int it = grp; it < n_items && ok; it += NU) {
            uint32_t v[32];
#pragma unroll
            for (int g = 0; g < 4; ++g)
#pragma unroll
                for (int i = 0; i < 8; ++i) v[8 * g + i] = (pk[i] >> (6 - 2 * g)) & 0x03030303u;   // k = 32g + 4i .. +3
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(empty), "r"((uint32_t)walk.count) : "memory");
            if (it + NU < n_items && !fetch()) { ok = false; break; }       // the next item's codes arrive while this one waits for its TMEM stage
            const int ts = it % TP_TS;
            if (it >= TP_TS && !__all_sync(0xffffffffu, wait_bounded(smem_u32(&a_empty[ts]), (uint32_t)((it / TP_TS - 1) & 1)))) { ok = false; break; }   // its last MMAs are done
            tc_fence_after();
            TC_ST32(tbase + ts * TP_A_COLS, v);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_remote(afull0 + ts * 8);
        }
        if (!ok && lane == 0) gave_up(p, 4);
    } else {
        // ------------------------------------------------------------ epilogue warps: TMEM -> registers -> global
        const int q = warp & 3, part = warp >> 2;                          // lane quarter; its two warps take alternate 32-token chunks
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        const uint32_t tempty0 = of_first_cta(smem_u32(&tempty_bar[0]));
        float2* tok = reinterpret_cast<float2*>(smem_raw + (aring - smem_u32(smem_raw)) + TP_ACT_RING) + warp * (TP_EP_CHUNKS * 32);
        const PairEp e(p.ep);
        const bool staged = e.mode == WF_OUT_LINEAR || e.mode == WF_OUT_I32;
        const float ws_all = e.fold ? w_scale_of(p.ep, 0) : 1.f;
        const int chunks = p.tn / 32;
        bool ok = true;
        for (int tl = 0; tl < my_tiles; ++tl) {
            const int tile = pair + tl * pairs, buf = tl % NBUF;
            const int mt = tile / p.n_tiles, nt = tile - mt * p.n_tiles;
            if (staged) {
                __syncwarp();                                               // the previous tile's readers are done
                for (int c = part, i = 0; c < chunks; c += 2, ++i) {
                    const int m = min(mt * p.tn + c * 32 + lane, p.M - 1);
                    const int rs = p.ep.rowsum ? p.ep.rowsum[m] : 0;
                    const float sa = e.mode == WF_OUT_LINEAR ? p.ep.act_scale[p.ep.act_scale_per_token ? m : 0] : 1.f;
                    tok[i * 32 + lane] = make_float2(e.mode == WF_OUT_I32 ? __int_as_float(rs) : e.fold ? __fmul_rn(ws_all, (float)rs) : (float)rs, sa);
                }
                __syncwarp();
            }
            const int n = nt * 2 * TP_ROWS + rank * TP_ROWS + q * 32 + lane;
            float ws = 1.f;
            if (e.mode == WF_OUT_LINEAR) ws = e.relu2 ? w_scale_of(p.ep, (lane >= 16 && p.ep.nseg > 1) ? 1 : 0) : seg_scale(p.ep, min(n, p.N - 1));
            ok = __all_sync(0xffffffffu, wait_bounded(smem_u32(&tfull_bar[buf]), (uint32_t)((tl / NBUF) & 1)));
            if (!ok) break;
            tc_fence_after();
#pragma unroll 1
            for (int c = part, i = 0; c < chunks; c += 2, ++i) {
                uint32_t v[32];
                TC_LD32(tmem + lane_base + buf * TP_ACC + c * 32, v);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                const int m0 = mt * p.tn + c * 32, mcnt = min(32, p.M - m0);
                pair_store(p.ep, e, v, tok + i * 32, m0, mcnt, n, ws, lane);
                __syncwarp();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) arrive_remote(tempty0 + buf * 8);
        }
        if (!ok && lane == 0) gave_up(p, 5);
    }
    tc_fence_before();
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");      // nobody leaves while the other CTA may still signal or read here
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (warp == W_MMA) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
    }
}

// us of the pair form at tn tokens per tile: what was measured over N 2560 .. 14336, K 2560 .. 14336, 20 .. 4000 tokens, to about 5 %.  A round of tiles takes
// 0.21 (32 tokens) to 0.29 us (256) a k-block; the one accumulator of 256 tokens leaves 2 us of the first and 4.2 us of each further epilogue uncovered.
double pair_time(int M, int N, int KB, int tn, int pairs) {
    const long long tiles = (long long)((N + 2 * TP_ROWS - 1) / (2 * TP_ROWS)) * ((M + tn - 1) / tn), rounds = (tiles + pairs - 1) / pairs;
    return 5.5 + 0.006 * tn + (double)rounds * KB * (0.203 + 0.00036 * tn) + (tn > 192 ? 2. + 4.2 * (double)(rounds - 1) : 0.);
}

int tokens_per_tile(int M, int N, int KB, int pairs) {
    int best = 32;
    for (int tn = 64; tn <= TP_MAX_TOK; tn += 32)
        if (tn != 224 && pair_time(M, N, KB, tn, pairs) < pair_time(M, N, KB, best, pairs)) best = tn;      // 224: 256's uncovered epilogue without its width
    return best;
}

DevOnce g_attr;

// The wait words: a page of the library's own memory that every device may write.  Nothing is allocated; locking the page is also allowed to a call that is
// being captured.
constexpr int WAIT_WORDS = 64;
alignas(4096) int g_wait_page[4096 / sizeof(int)];
std::atomic<int> g_wait_state{0};                      // 1: usable; -1: the page cannot be locked

bool wait_page_usable() {
    if (const int st = g_wait_state.load(std::memory_order_acquire)) return st > 0;
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    if (const int st = g_wait_state.load(std::memory_order_acquire)) return st > 0;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    const bool swapped = cudaThreadExchangeStreamCaptureMode(&mode) == cudaSuccess;
    void* dev = nullptr;
    const bool ok = cudaHostRegister(g_wait_page, sizeof g_wait_page, cudaHostRegisterPortable | cudaHostRegisterMapped) == cudaSuccess &&
                    cudaHostGetDevicePointer(&dev, g_wait_page, 0) == cudaSuccess && dev == (void*)g_wait_page;
    if (!ok) cudaGetLastError();
    if (swapped) cudaThreadExchangeStreamCaptureMode(&mode);
    g_wait_state.store(ok ? 1 : -1, std::memory_order_release);
    return ok;
}

}  // namespace

int* tc_wait_word() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= WAIT_WORDS || !wait_page_usable()) return nullptr;
    return g_wait_page + dev;
}

int check_wait_word(const char* who) {
    if (g_wait_state.load(std::memory_order_acquire) <= 0) return WF_OK;
    int* word = tc_wait_word();
    if (!word || !*(volatile int*)word) return WF_OK;
    if (const int role = __atomic_exchange_n(word, 0, __ATOMIC_ACQ_REL)) {
        set_error("%s: a bounded wait of an earlier ternary product on this device ran out (%d); that product's output is not complete", who, role);
        return WF_ERR_CUDA;
    }
    return WF_OK;
}

int gemm_tc_pair_tokens(int M, int N, int K) { return tokens_per_tile(M, N, K / WF_QK, sm_count() / 2); }

double gemm_tc_pair_time(int M, int N, int K, bool relu2) {
    const int pairs = sm_count() / 2, tn = gemm_tc_pair_tokens(M, N, K);
    const long long tiles = (long long)((N + 2 * TP_ROWS - 1) / (2 * TP_ROWS)) * ((M + tn - 1) / tn);
    return pair_time(M, N, K / WF_QK, tn, pairs) + (relu2 ? 0.4 * (double)((tiles + pairs - 1) / pairs) : 0.);      // the pairs' exchange of gate and up
}

int launch_gemm_tc_pair(const wf_linear_args* a, const EpiParams& ep, cudaStream_t s, bool ahead) {
    constexpr int NU = 3;
    EncodeTiledFn enc = tc_encoder();
    if (!enc) { set_error("gemm_tc_pair: cuTensorMapEncodeTiled unavailable"); return WF_ERR_CUDA; }
    typedef void (*Kernel)(CUtensorMap, CUtensorMap, TpParams);
    static const Kernel kernels[2][2] = {{ternary_gemm_pair_kernel<NU, 2, false>, ternary_gemm_pair_kernel<NU, 2, true>},       // [one accumulator][ragged]
                                         {ternary_gemm_pair_kernel<NU, 1, false>, ternary_gemm_pair_kernel<NU, 1, true>}};
    if (g_attr.need()) {
        for (const auto& row : kernels)
            for (Kernel k : row)
                if (cuda_check(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, TP_SMEM), "gemm_tc_pair attribute")) return WF_ERR_CUDA;
    }
    TpParams p;
    memset(&p, 0, sizeof p);
    p.M = a->M; p.N = a->N; p.K = a->K; p.KB = a->K / WF_QK;
    p.i2s = a->w_layout == WF_W_I2S;
    const int pairs = sm_count() / 2;
    p.tn = tokens_per_tile(p.M, p.N, p.KB, pairs);
    p.n_tiles = (p.N + 2 * TP_ROWS - 1) / (2 * TP_ROWS);
    p.tiles = p.n_tiles * ((p.M + p.tn - 1) / p.tn);
    p.akb = p.tn <= 128 ? 4 : 2;
    p.as = TP_ACT_RING / (p.akb * p.tn / 2 * TP_BK);
    if (p.as > TP_AS_MAX) p.as = TP_AS_MAX;
    p.err = tc_wait_word();
    if (!p.err) { set_error("gemm_tc_pair: no wait word"); return WF_ERR_CUDA; }
    p.ep = ep;
    p.ahead = ahead;
    CUtensorMap tq, tw;
    const cuuint32_t one[4] = {1, 1, 1, 1};
    {
        const cuuint64_t dim[3] = {TP_BK, (cuuint64_t)a->M, (cuuint64_t)p.KB}, stride[2] = {(cuuint64_t)a->ldq, TP_BK};
        const cuuint32_t box[3] = {TP_BK, (cuuint32_t)(p.tn / 2), (cuuint32_t)p.akb};
        const CUresult cr = enc(&tq, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, (void*)a->q, dim, stride, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (cr != CUDA_SUCCESS) { set_error("gemm_tc_pair: tensor map of the activations failed (%d)", (int)cr); return WF_ERR_CUDA; }
    }
    CUresult cr;
    if (p.i2s) {
        const cuuint64_t dim[2] = {(cuuint64_t)(a->K / 4), (cuuint64_t)a->N}, stride[1] = {(cuuint64_t)(a->K / 4)};
        const cuuint32_t box[2] = {TP_WKB * 32, TP_ROWS};
        cr = enc(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)a->w, dim, stride, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                 CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    } else {
        const cuuint64_t dim[4] = {16, 8, (cuuint64_t)p.KB, (cuuint64_t)((a->N + 15) / 16)};
        const cuuint64_t stride[3] = {64, WF_TILE_BYTES, (cuuint64_t)p.KB * WF_TILE_BYTES};
        const cuuint32_t box[4] = {16, 8, TP_WKB, TP_ROWS / 16};
        cr = enc(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, (void*)a->w, dim, stride, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                 CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    if (cr != CUDA_SUCCESS) { set_error("gemm_tc_pair: tensor map of the weights failed (%d)", (int)cr); return WF_ERR_CUDA; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (p.tiles < pairs ? p.tiles : pairs));
    cfg.blockDim = dim3(tp_threads(NU));
    cfg.dynamicSmemBytes = TP_SMEM;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    return launch_check(cudaLaunchKernelEx(&cfg, kernels[p.tn > 192][pair_ragged(p.KB, NU)], tq, tw, p), "ternary_gemm_pair");
}

}  // namespace wf
