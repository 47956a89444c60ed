// Prompt attention on the 5th-generation tensor cores (tcgen05, scores and outputs in TMEM): softmax attention with per-head keys and values,
// causal and windowed, with an optional linear distance penalty, head or element gates and a softmax sink.  Keys and values come either from the
// paged cache (grouped-query attention) or from a dense per-token buffer (latent attention whose latents were expanded to per-head keys and values).
//
// A CTA owns one key/value head and TWO tiles of 128 query rows (a row = a token and one of the query heads that share the key/value head), so that
// one tile's softmax runs while the tensor cores work for the other:
//   * warps 0..3 / 4..7: softmax of tile 0 / 1, one thread per row; they also load their queries and write the results;
//   * warp 8: TMA producer, 128 keys x 64 dims per box (paged: one box per page), two stages each of keys and values;
//   * warp 9: one elected thread issues S = Q K^T (both operands in shared memory, 128B swizzle) and O += P V (P in TMEM, V as the MN-major operand).
// TMEM: per tile 128 columns of scores, overwritten in place by the weights, and 128 columns of output: 512 in all.  With grouped-query attention
// the weights enter the value product as a two-term bf16 split (hi + lo), so that it sees the float weights to 2^-17, like the mma.sync kernel;
// latent attention rounds them to bf16, like its mma.sync kernel.  The output is rescaled only when a row's maximum has grown by more than 2^8 since
// the scale was last fixed (exact: the sum carries the same scale).
// What bounds it: per pair of 128 x 128 tiles the tensor cores take 6 x 128^3 multiply-adds (about 3060 clk, 2040 without the split) and the eight
// softmax warps about 5 instructions per score (1280 issue slots of each SM quarter's share), hence the packed float pairs and the scale folded
// into the exponent's multiply-add.  Measured, 2048 tokens causal, 20 heads of 128: grouped-query attention 181 -> 67 us (mma.sync kernel before),
// latent attention 895 -> 49 us (one CTA per token before; plus 24 us for the expansion; 61 us with the heads' tiles handed out head after head).
// Every wait is bounded: one that runs out records an error word that the host checks, and the CTA drains and leaves.
// A value that is infinite or NaN meets the zero weights of the rows of its key tile that do not see it, too: a row whose sum of weights is finite and
// whose output is not is taken again by its warp, over the keys that it sees (at_row).
#include "seq_attn_mma.cuh"
#include <cuda.h>
#include <math.h>

namespace wf {
namespace seq {

namespace {

constexpr int AT_ROWS = 128, AT_KEYS = 128;
constexpr int AT_HALF = 128 * 128;                    // bytes of a 128-row x 64-element bf16 block (one swizzle atom wide)
constexpr int AT_TILE = 2 * AT_HALF;
constexpr int AT_SMEM = 2 * AT_TILE + 4 * AT_TILE + 1024;   // queries of two tiles, two stages of keys and of values
constexpr int AT_THREADS = 10 * 32;
constexpr unsigned long long AT_LIMIT_NS = 1000000000ull;   // a wait that lasts this long has failed
constexpr float AT_LAZY = 8.f;                        // growth of a row's maximum (in log 2) that the fixed scale tolerates

struct AtParams {
    GqaDims D;
    const __nv_bfloat16* qn;       // [n, H, d]
    const float* gate;
    void* out; int out_f32;        // [n, H, dv]
    const int32_t* block_table; int max_blocks, page_size;
    const int32_t* key_row;        // dense keys: a sequence's first row in the buffer (null: paged)
    int rep, tq;                   // query heads per key/value head, tokens per row tile
    int box;                       // keys per TMA box
    const __nv_bfloat16 *k, *v;    // what the tensor maps cover, and their strides in elements
    long long k_row, k_head, v_row, v_head, page_stride;
    int* err;
};

__device__ __forceinline__ uint64_t at_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3ffffu) >> 4);
    d |= (uint64_t)(lbo >> 4) << 16;
    d |= (uint64_t)(sbo >> 4) << 32;
    d |= (uint64_t)1 << 46;                           // descriptor version (sm_100)
    d |= (uint64_t)2 << 61;                           // 128-byte swizzle
    return d;
}
// D f32, A bf16, B bf16; b_mn: B is MN-major
constexpr uint32_t at_idesc(int m, int n, int b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)b_mn << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void at_mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void at_mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void at_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool at_wait(uint64_t* bar, uint32_t parity) {
    for (int i = 0; i < 64; ++i) if (mbar_try_wait(bar, parity)) return true;
    unsigned long long t0, t1;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    do {
        if (mbar_try_wait(bar, parity)) return true;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t1));
    } while (t1 - t0 < AT_LIMIT_NS);
    return false;
}
// the same for a whole warp: one answer, and the warp together again
__device__ __forceinline__ bool at_wait_warp(uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, at_wait(bar, parity)); }
__device__ __forceinline__ void at_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void at_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }

#define AT_R32(v, o)                                                                                                     \
    "r"(v[o + 0]), "r"(v[o + 1]), "r"(v[o + 2]), "r"(v[o + 3]), "r"(v[o + 4]), "r"(v[o + 5]), "r"(v[o + 6]), "r"(v[o + 7]), \
    "r"(v[o + 8]), "r"(v[o + 9]), "r"(v[o + 10]), "r"(v[o + 11]), "r"(v[o + 12]), "r"(v[o + 13]), "r"(v[o + 14]), "r"(v[o + 15]), \
    "r"(v[o + 16]), "r"(v[o + 17]), "r"(v[o + 18]), "r"(v[o + 19]), "r"(v[o + 20]), "r"(v[o + 21]), "r"(v[o + 22]), "r"(v[o + 23]), \
    "r"(v[o + 24]), "r"(v[o + 25]), "r"(v[o + 26]), "r"(v[o + 27]), "r"(v[o + 28]), "r"(v[o + 29]), "r"(v[o + 30]), "r"(v[o + 31])
#define AT_W32(v, o)                                                                                                     \
    "=r"(v[o + 0]), "=r"(v[o + 1]), "=r"(v[o + 2]), "=r"(v[o + 3]), "=r"(v[o + 4]), "=r"(v[o + 5]), "=r"(v[o + 6]), "=r"(v[o + 7]), \
    "=r"(v[o + 8]), "=r"(v[o + 9]), "=r"(v[o + 10]), "=r"(v[o + 11]), "=r"(v[o + 12]), "=r"(v[o + 13]), "=r"(v[o + 14]), "=r"(v[o + 15]), \
    "=r"(v[o + 16]), "=r"(v[o + 17]), "=r"(v[o + 18]), "=r"(v[o + 19]), "=r"(v[o + 20]), "=r"(v[o + 21]), "=r"(v[o + 22]), "=r"(v[o + 23]), \
    "=r"(v[o + 24]), "=r"(v[o + 25]), "=r"(v[o + 26]), "=r"(v[o + 27]), "=r"(v[o + 28]), "=r"(v[o + 29]), "=r"(v[o + 30]), "=r"(v[o + 31])
#define AT_LD32(taddr, v, o)                                                                                             \
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"          \
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];" : AT_W32(v, o) : "r"(taddr) : "memory")
#define AT_ST32(taddr, v, o)                                                                                             \
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"    \
                 "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr), AT_R32(v, o) : "memory")

// two floats in one 64-bit register pair (the packed float units take both at once)
__device__ __forceinline__ uint64_t at_pair(uint32_t a, uint32_t b) { uint64_t v; asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(a), "r"(b)); return v; }
__device__ __forceinline__ void at_unpair(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t at_fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t v; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c)); return v; }
__device__ __forceinline__ uint64_t at_add2(uint64_t a, uint64_t b) { uint64_t v; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b)); return v; }
__device__ __forceinline__ float at_ex2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }   // weights below 2^-126 are zero

// One row of one head, key by key over what it sees, with a whole warp: a lane per key for the scores, then a lane per 4 output columns.  Not inlined: its
// registers would come out of the kernel's.
__device__ __noinline__ void at_row(const Batch& b, const AtParams& p, int head, int tok) {
    const GqaDims& D = p.D;
    const int kvh = blockIdx.x % D.G, sq = b.tok_seq[tok], pos = b.tok_pos[tok], row0 = p.key_row ? p.key_row[sq] : 0;
    const int32_t* bt = p.key_row ? nullptr : p.block_table + (size_t)b.seq_slot[sq] * p.max_blocks;
    const int lane = threadIdx.x & 31;
    const __nv_bfloat16* q = p.qn + ((size_t)tok * D.H + head) * D.d;
    const float slope2 = D.dist_exp > 0.f ? exp2f(-D.dist_exp * (float)(head + 1) / (float)D.H) * LOG2E : 0.f, scale2 = D.scale * LOG2E;
    float m = -INFINITY, l = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
    auto place = [&](const __nv_bfloat16* base, long long row_stride, long long head_stride, int j) {
        const int pg = bt ? j / p.page_size : 0;
        return base + (bt ? (long long)bt[pg] * p.page_stride + (long long)(j - pg * p.page_size) * row_stride : (long long)(row0 + j) * row_stride) + kvh * head_stride;
    };
    for (int j0 = max(0, pos - D.window + 1); j0 <= pos; j0 += 32) {
        const int j = j0 + lane;
        float x = -INFINITY;
        if (j <= pos) {
            const __nv_bfloat16* kr = place(p.k, p.k_row, p.k_head, j);
            float dot = 0.f;
            for (int c = 0; c < D.d; ++c) dot = fmaf(__bfloat162float(q[c]), __bfloat162float(kr[c]), dot);
            x = fmaf(dot, scale2, -slope2 * (float)(pos - j));
        }
        float top = x;
#pragma unroll
        for (int w = 16; w; w >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, w));
        top = fmaxf(m, top);
        const float f = top == -INFINITY ? 1.f : exp2f(m - top), e = x == -INFINITY ? 0.f : exp2f(x - top);
        m = top;
        l *= f;
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[k] *= f;
        const int n = min(32, pos - j0 + 1);
        for (int i = 0; i < n; ++i) {
            const float w = __shfl_sync(0xffffffffu, e, i);
            const __nv_bfloat16* vr = place(p.v, p.v_row, p.v_head, j0 + i);
            l += w;
#pragma unroll
            for (int k = 0; k < 4; ++k) { const int c = lane + 32 * k; if (c < D.dv) acc[k] = fmaf(w, __bfloat162float(vr[c]), acc[k]); }
        }
    }
    const float mul = (p.gate && !D.gate_elem ? p.gate[(size_t)tok * D.H + head] : 1.f) * am_inv_sum(D, head, m, l);
    const size_t at = ((size_t)tok * D.H + head) * D.dv;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int c = lane + 32 * k;
        if (c >= D.dv) continue;
        float y = acc[k] * mul;
        if (p.gate && D.gate_elem) y *= p.gate[at + c];
        if (p.out_f32) ((float*)p.out)[at + c] = y; else ((__nv_bfloat16*)p.out)[at + c] = __float2bfloat16_rn(y);
    }
}

// SPLIT: the weights as a two-term bf16 split (grouped-query attention); without it rounded to bf16 (latent attention)
template <bool SPLIT>
__global__ void __launch_bounds__(AT_THREADS, 1) attn_tc_kernel(const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ Batch b,
                                                                const __grid_constant__ AtParams p) {
    pdl_wait_prior();
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t q_full[2], k_full[2], k_empty[2], v_full[2], v_empty[2], v_fixed, s_full[2], p_full[2], o_full[2], drained;
    __shared__ uint32_t tmem_base_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const GqaDims& D = p.D;
    const int kvh = blockIdx.x % D.G;
    // ---- which sequence and which of its tokens: the last tiles of a sequence see the most keys and are handed out first, those of all heads before the others
    int sq = -1, tok0 = 0, left = 0;
    {
        int t = (int)((gridDim.x - 1 - blockIdx.x) / D.G);
        for (int s = 0; s < b.nseq; ++s) {
            const int units = (b.seq_len[s] + 2 * p.tq - 1) / (2 * p.tq);
            if (t < units) { sq = s; tok0 = t * 2 * p.tq; left = b.seq_len[s] - tok0; break; }
            t -= units;
        }
    }
    if (sq < 0) return;
    const int pos0 = b.seq_pos0[sq] + tok0, flat0 = b.seq_start[sq] + tok0;
    int ntok[2], lo_t[2], hi_t[2];                        // tokens of each tile; its first and last 128-key tile (last < first: no tokens)
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        ntok[t] = min(p.tq, max(0, left - t * p.tq));
        const int first = pos0 + t * p.tq;
        lo_t[t] = max(0, first - D.window + 1) / AT_KEYS;
        hi_t[t] = ntok[t] > 0 ? (first + ntok[t] - 1) / AT_KEYS : -1;
    }
    const int lo = lo_t[0], hi = max(hi_t[0], hi_t[1]), nt = hi - lo + 1;
    const int pos_last = pos0 + ntok[0] + ntok[1] - 1;
    const int fix_row = pos_last + 1 - hi * AT_KEYS;      // rows of the last value tile from here on hold no key: zeroed (a weight of zero times NaN is NaN)
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t q_s = base, k_s = base + 2 * AT_TILE, v_s = k_s + 2 * AT_TILE;

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&q_full[i], 4); mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
            mbar_init(&s_full[i], 1); mbar_init(&p_full[i], 4); mbar_init(&o_full[i], 1);
        }
        mbar_init(&v_fixed, 1);
        mbar_init(&drained, 1);
        fence_mbar_init();
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "n"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    at_fence_before();
    __syncthreads();
    at_fence_after();
    const uint32_t tmem = tmem_base_s;

    if (warp == 8) {
        // ------------------------------------------------------------ producer
        const int32_t* bt = p.block_table + (size_t)b.seq_slot[sq] * p.max_blocks;
        const int kh = D.d > 64 ? 2 : 1, vh = D.dv > 64 ? 2 : 1, nbox = AT_KEYS / p.box;
        const int row0 = p.key_row ? p.key_row[sq] : 0;
        bool ok = true;
        int issued[2] = {0, 0};                           // tiles of keys and of values under way or landed
        for (int i = 0; i < nt && ok; ++i) {
            const int st = i & 1, u = lo + i, j = u * AT_KEYS + lane * p.box;
            const bool mine = lane < nbox && j <= pos_last;
            const uint32_t boxes = __popc(__ballot_sync(0xffffffffu, mine));
            int slot = row0 + j, page = 0;
            if (!p.key_row && mine) { const int pg = j / p.page_size; slot = j - pg * p.page_size; page = bt[pg]; }
#pragma unroll
            for (int kv = 0; kv < 2; ++kv) {
                uint64_t* full = kv ? &v_full[st] : &k_full[st];
                uint64_t* empty = kv ? &v_empty[st] : &k_empty[st];
                if (i >= 2 && !at_wait_warp(empty, (uint32_t)(((i >> 1) & 1) ^ 1))) { ok = false; break; }
                const int halves = kv ? vh : kh;
                if (lane == 0) mbar_expect_tx(full, boxes * (uint32_t)(halves * p.box * 128));
                __syncwarp();
                if (mine) {
                    const uint32_t dst = (kv ? v_s : k_s) + st * AT_TILE + lane * p.box * 128;
                    for (int h = 0; h < halves; ++h)
                        asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
                                     ::"r"(dst + h * AT_HALF), "l"(kv ? &tmap_v : &tmap_k), "r"(h * 64), "r"(slot), "r"(kvh), "r"(page), "r"(smem_u32(full)) : "memory");
                }
                __syncwarp();
                issued[kv] = i + 1;
            }
            if (ok && u == hi && fix_row < AT_KEYS) {
                if (!at_wait_warp(&v_full[st], (uint32_t)((i >> 1) & 1))) { ok = false; break; }
                for (int c = lane; c < (AT_KEYS - fix_row) * 8 * vh; c += 32) {
                    const int h = c / ((AT_KEYS - fix_row) * 8), r = c - h * (AT_KEYS - fix_row) * 8;
                    asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(v_s + st * AT_TILE + h * AT_HALF + (fix_row * 8 + r) * 16), "r"(0u) : "memory");
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(&v_fixed);
            }
        }
        if (!ok) {                                        // the CTA leaves early, but not before its copies have landed
            if (lane == 0) atomicExch(p.err, 4);
            for (int kv = 0; kv < 2; ++kv)
                for (int i = max(0, issued[kv] - 2); i < issued[kv]; ++i) at_wait_warp(kv ? &v_full[i & 1] : &k_full[i & 1], (uint32_t)((i >> 1) & 1));
        }
    } else if (warp == 9) {
        // ------------------------------------------------------------ MMA issuer
        uint32_t elected;
        asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(elected));
        if (elected) {
            const uint32_t idesc_s = at_idesc(AT_ROWS, AT_KEYS, 0), idesc_o = at_idesc(AT_ROWS, (D.dv + 15) / 16 * 16, 1);
            const int ksteps = (D.d + 15) / 16;
            uint32_t np[2] = {0, 0};                      // weight tiles consumed per row tile
            bool ok = true;
            for (int i = -1; i < nt && ok; ++i) {
                const int u = lo + i, st = i & 1, st1 = (i + 1) & 1;
                bool v_ready = false, k_ready = false;
                for (int t = 0; t < 2 && ok; ++t) {
                    const uint32_t s_t = tmem + t * 256, o_t = s_t + 128;
                    if (i >= 0 && u >= lo_t[t] && u <= hi_t[t]) {
                        if (!v_ready) {
                            ok = at_wait(&v_full[st], (uint32_t)((i >> 1) & 1)) && !(u == hi && fix_row < AT_KEYS && !at_wait(&v_fixed, 0));
                            if (!ok) break;
                            v_ready = true;
                        }
                        if (!at_wait(&p_full[t], np[t] & 1)) { ok = false; break; }
                        at_fence_after();
                        const uint64_t vd = at_desc(v_s + st * AT_TILE, AT_HALF, 1024);
#pragma unroll
                        for (int ks = 0; ks < 8; ++ks) at_mma_ts(o_t, s_t + ks * 8, vd + (uint64_t)(ks * 128), idesc_o, np[t] || ks ? 1u : 0u);   // 16 keys = 2048 bytes
                        if (SPLIT) {
#pragma unroll
                            for (int ks = 0; ks < 8; ++ks) at_mma_ts(o_t, s_t + 64 + ks * 8, vd + (uint64_t)(ks * 128), idesc_o, 1u);
                        }
                        ++np[t];
                        if (u == hi_t[t]) at_commit(&o_full[t]);
                    }
                    if (i + 1 < nt && u + 1 >= lo_t[t] && u + 1 <= hi_t[t]) {
                        if (!k_ready) { if (!at_wait(&k_full[st1], (uint32_t)(((i + 1) >> 1) & 1))) { ok = false; break; } k_ready = true; }
                        if (u + 1 == lo_t[t] && !at_wait(&q_full[t], 0)) { ok = false; break; }
                        at_fence_after();
                        const uint64_t qd = at_desc(q_s + t * AT_TILE, 16, 1024), kd = at_desc(k_s + st1 * AT_TILE, 16, 1024);
                        for (int ks = 0; ks < ksteps; ++ks) {
                            const uint64_t off = (uint64_t)((ks >> 2) * (AT_HALF >> 4) + (ks & 3) * 2);
                            at_mma_ss(s_t, qd + off, kd + off, idesc_s, ks ? 1u : 0u);
                        }
                        at_commit(&s_full[t]);
                    }
                }
                if (!ok) break;
                if (i >= 0) at_commit(&v_empty[st]);
                if (i + 1 < nt) at_commit(&k_empty[st1]);
            }
            if (!ok) atomicExch(p.err, 5);
            at_commit(&drained);                          // nor while a product still reads shared memory or TMEM
            at_wait(&drained, 0);
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ softmax: a thread per row
        const int t = warp >> 2, row = (warp & 3) * 32 + lane;
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t s_t = tmem + t * 256 + lane_base, o_t = s_t + 128;
        const int tk = row / p.rep, head = kvh * p.rep + (row - tk * p.rep);
        const bool r_ok = tk < ntok[t];
        const int tok = flat0 + t * p.tq + tk, pos = pos0 + t * p.tq + tk;
        const int pos_min = pos0 + t * p.tq, pos_max = pos_min + ntok[t] - 1;
        if (ntok[t] > 0) {
            // the row's query into the swizzled operand tile (zero where there is no row and beyond d)
            const uint32_t qrow = q_s + t * AT_TILE + row * 128;
            const uint4* src = reinterpret_cast<const uint4*>(p.qn + ((size_t)(r_ok ? tok : 0) * D.H + (r_ok ? head : 0)) * D.d);
            const int chunks = D.d > 64 ? 16 : 8;
            for (int c = 0; c < chunks; ++c) {
                uint4 v = make_uint4(0u, 0u, 0u, 0u);
                if (r_ok && c * 8 < D.d) v = src[c];
                asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(qrow + (c >> 3) * AT_HALF + (((c & 7) ^ (row & 7)) << 4)), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&q_full[t]);
        }
        const float scale2 = D.scale * LOG2E;
        const float slope2 = D.dist_exp > 0.f ? exp2f(-D.dist_exp * (float)(head + 1) / (float)D.H) * LOG2E : 0.f;
        // scores are kept in units of log 2: raw ones take the scale in the exponent's own multiply-add, with a penalty they take it before
        const bool pre = D.dist_exp > 0.f || !(D.scale > 0.f);
        const float unit = pre ? 1.f : scale2;
        float m_ref = -INFINITY, l = 0.f;
        bool ok = true;
        uint32_t it = 0;
        for (int u = lo_t[t]; u <= hi_t[t] && ok; ++u, ++it) {
            if (!at_wait_warp(&s_full[t], it & 1)) { ok = false; break; }     // also: every earlier product of this tile is done
            at_fence_after();
            uint32_t r[128];
            AT_LD32(s_t, r, 0);
            AT_LD32(s_t + 32, r, 32);
            AT_LD32(s_t + 64, r, 64);
            AT_LD32(s_t + 96, r, 96);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            const int j0 = u * AT_KEYS;
            if (pre) {
                const float nb = -slope2 * (float)(pos - j0);
#pragma unroll
                for (int c = 0; c < 128; ++c) r[c] = __float_as_uint(fmaf(__uint_as_float(r[c]), scale2, fmaf(slope2, (float)c, nb)));
            }
            if (j0 + AT_KEYS - 1 > pos_min || j0 < pos_max - D.window + 1) {         // some row of the tile does not see the whole key tile
                const int last = r_ok ? pos - j0 : -1, first = last - D.window + 1;      // visible columns of this row
#pragma unroll
                for (int c = 0; c < 128; ++c) if (c > last || c < first) r[c] = 0xff800000u;
            }
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < 128; c += 8)
#pragma unroll
                for (int k = 0; k < 4; ++k) mx4[k] = fmaxf(fmaxf(mx4[k], __uint_as_float(r[c + k])), __uint_as_float(r[c + 4 + k]));
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * unit;
            float corr = 1.f;
            if (mx > m_ref + AT_LAZY) {                    // also the first time anything is seen
                corr = m_ref == -INFINITY ? 0.f : exp2f(m_ref - mx);
                m_ref = mx;
                l *= corr;
            }
            const uint32_t nm = __float_as_uint(m_ref == -INFINITY ? 0.f : -m_ref);
            const uint64_t nm2 = at_pair(nm, nm), unit2 = at_pair(__float_as_uint(unit), __float_as_uint(unit)), minus2 = at_pair(0xbf800000u, 0xbf800000u);
            uint64_t ls[2] = {0ull, 0ull};
            // hi of columns (2c, 2c + 1) goes to r[c], an entry whose score has been read
            uint32_t lo32[SPLIT ? 64 : 1];
#pragma unroll
            for (int c = 0; c < 64; ++c) {
                float a, d;
                at_unpair(at_fma2(at_pair(r[2 * c], r[2 * c + 1]), unit2, nm2), a, d);
                a = at_ex2(a); d = at_ex2(d);
                const uint64_t w = at_pair(__float_as_uint(a), __float_as_uint(d));
                ls[c & 1] = at_add2(ls[c & 1], w);
                const uint32_t h = pack_bf16(a, d);
                if (SPLIT) {
                    at_unpair(at_fma2(at_pair(h << 16, h & 0xffff0000u), minus2, w), a, d);
                    lo32[c] = pack_bf16(a, d);
                }
                r[c] = h;
            }
            float l0, l1;
            at_unpair(at_add2(ls[0], ls[1]), l0, l1);
            l += l0 + l1;
            AT_ST32(s_t, r, 0);
            AT_ST32(s_t + 32, r, 32);
            if (SPLIT) {
                AT_ST32(s_t + 64, lo32, 0);
                AT_ST32(s_t + 96, lo32, 32);
            }
            if (it > 0 && __any_sync(0xffffffffu, corr != 1.f)) {
#pragma unroll 1
                for (int c = 0; c < D.dv; c += 32) {
                    uint32_t o[32];
                    AT_LD32(o_t + c, o, 0);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int k = 0; k < 32; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * corr);
                    AT_ST32(o_t + c, o, 0);
                }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            at_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[t]);
        }
        if (ok && ntok[t] > 0) {
            if (at_wait_warp(&o_full[t], 0)) {
                at_fence_after();
                const float mul = r_ok ? (p.gate && !D.gate_elem ? p.gate[(size_t)tok * D.H + head] : 1.f) * am_inv_sum(D, head, m_ref, l) : 0.f;
                const size_t at = ((size_t)(r_ok ? tok : 0) * D.H + head) * D.dv;
                const float* ge = p.gate && D.gate_elem ? p.gate + at : nullptr;
                float watch = 0.f;                         // times zero: NaN from the first sum that is not finite on
#pragma unroll 1
                for (int c = 0; c < D.dv; c += 32) {
                    uint32_t o[32];
                    __syncwarp();
                    AT_LD32(o_t + c, o, 0);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (r_ok) {
#pragma unroll
                        for (int k = 0; k < 32; k += 8) {
                            if (c + k >= D.dv) break;
                            float v[8];
#pragma unroll
                            for (int e = 0; e < 8; ++e) { watch = fmaf(__uint_as_float(o[k + e]), 0.f, watch); v[e] = __uint_as_float(o[k + e]) * mul; }
                            if (ge) {
                                const float4 g0 = *reinterpret_cast<const float4*>(ge + c + k), g1 = *reinterpret_cast<const float4*>(ge + c + k + 4);
                                v[0] *= g0.x; v[1] *= g0.y; v[2] *= g0.z; v[3] *= g0.w; v[4] *= g1.x; v[5] *= g1.y; v[6] *= g1.z; v[7] *= g1.w;
                            }
                            if (p.out_f32) {
                                float4* dst = reinterpret_cast<float4*>((float*)p.out + at + c + k);
                                dst[0] = make_float4(v[0], v[1], v[2], v[3]);
                                dst[1] = make_float4(v[4], v[5], v[6], v[7]);
                            } else {
                                *reinterpret_cast<uint4*>((__nv_bfloat16*)p.out + at + c + k) = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
                            }
                        }
                    }
                }
                __syncwarp();
                for (uint32_t redo = __ballot_sync(0xffffffffu, r_ok && !(watch == 0.f) && l * 0.f == 0.f); redo; redo &= redo - 1) {
                    const int r = __ffs(redo) - 1;
                    at_row(b, p, __shfl_sync(0xffffffffu, head, r), __shfl_sync(0xffffffffu, tok, r));
                    __syncwarp();
                }
            } else ok = false;
        }
        if (!ok && lane == 0) atomicExch(p.err, 6);
    }
    __syncwarp();
    at_fence_before();
    __syncthreads();
    if (warp == 9) {
        at_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// [d][rows][heads][pages], strides in elements
int at_encode(CUtensorMap* tm, const void* base, int d, uint64_t rows, uint64_t row_stride, int heads, uint64_t head_stride, uint64_t pages, uint64_t page_stride, int box) {
    EncodeTiledFn fn = (EncodeTiledFn)tensor_map_encoder();
    if (!fn) { set_error("attention: cuTensorMapEncodeTiled unavailable"); return WF_ERR_CUDA; }
    const cuuint64_t gdim[4] = {(cuuint64_t)d, rows, (cuuint64_t)heads, pages};
    const cuuint64_t gstride[3] = {row_stride * 2, head_stride * 2, page_stride * 2};
    const cuuint32_t bx[4] = {64, (cuuint32_t)box, 1, 1}, es[4] = {1, 1, 1, 1};
    const CUresult cr = fn(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, (void*)base, gdim, gstride, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (cr != CUDA_SUCCESS) { set_error("attention: tensor map failed (%d)", (int)cr); return WF_ERR_CUDA; }
    return WF_OK;
}

DevOnce g_at_attr;

int at_launch(const Batch& b, const AtParams& p, bool split, const CUtensorMap& tk, const CUtensorMap& tv, cudaStream_t s) {
    if (g_at_attr.need() && (cuda_check(cudaFuncSetAttribute(attn_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, AT_SMEM), "attention shared memory") ||
                             cuda_check(cudaFuncSetAttribute(attn_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, AT_SMEM), "attention shared memory"))) return WF_ERR_CUDA;
    // every sequence's tokens are cut into units of 2 tq; n / (2 tq) + nseq bounds their number (CTAs beyond the last unit return at once)
    const dim3 grid((b.n / (2 * p.tq) + b.nseq) * p.D.G);
    if (split) launch_pdl(attn_tc_kernel<true>, grid, AT_THREADS, AT_SMEM, s, tk, tv, b, p);
    else launch_pdl(attn_tc_kernel<false>, grid, AT_THREADS, AT_SMEM, s, tk, tv, b, p);
    return launch_check(cudaGetLastError(), "attn_tc");
}

bool at_sizes_ok(const GqaDims& D) {
    return D.G > 0 && D.H % D.G == 0 && D.H / D.G <= AT_ROWS && D.d % 8 == 0 && D.dv % 8 == 0 && D.d <= 128 && D.dv <= 128 && D.G <= 65535 &&
           D.chunk <= 0 && D.keep_first <= 0 && !D.talk && !(D.softcap > 0.f) && !D.rel && !D.dist_r1 && !D.v_is_k;
}

}  // namespace

bool attn_tc_usable(const GqaDims& D, const PagedCache& pc) {
    const int ps = pc.page_size;
    return at_sizes_ok(D) && ps >= 8 && (ps & (ps - 1)) == 0 && pc.layer_off % 8 == 0 && pc.page_stride % 8 == 0 && ((uintptr_t)pc.pool & 15) == 0;
}

int launch_attn_tc(const Batch& b, const GqaDims& D, const void* qn, const float* gate, const PagedCache& pc, int max_pages, void* out, cudaStream_t s) {
    if (b.n <= 0) return WF_OK;
    if (!attn_tc_usable(D, pc)) { set_error("attention: the tcgen05 form does not take these sizes"); return WF_ERR_UNSUPPORTED; }
    AtParams p;
    p.D = D; p.qn = (const __nv_bfloat16*)qn; p.gate = gate; p.out = out; p.out_f32 = 0;
    p.block_table = pc.block_table; p.max_blocks = pc.max_blocks; p.page_size = pc.page_size;
    p.key_row = nullptr;
    p.rep = D.H / D.G; p.tq = AT_ROWS / p.rep;
    p.box = pc.page_size < AT_KEYS ? pc.page_size : AT_KEYS;
    p.err = tc_error_word();
    if (!p.err) return WF_ERR_CUDA;
    CUtensorMap tk, tv;
    const __nv_bfloat16* k = (const __nv_bfloat16*)pc.pool + pc.layer_off;
    const uint64_t ps = pc.page_size;
    p.k = k; p.v = k + (size_t)D.G * ps * D.d;
    p.k_row = D.d; p.k_head = (long long)ps * D.d; p.v_row = D.dv; p.v_head = (long long)ps * D.dv; p.page_stride = pc.page_stride;
    if (int rc = at_encode(&tk, p.k, D.d, ps, p.k_row, D.G, p.k_head, max_pages, pc.page_stride, p.box)) return rc;
    if (int rc = at_encode(&tv, p.v, D.dv, ps, p.v_row, D.G, p.v_head, max_pages, pc.page_stride, p.box)) return rc;
    return at_launch(b, p, true, tk, tv, s);
}

bool attn_tc_dense_usable(const GqaDims& D) { return at_sizes_ok(D); }

int launch_attn_tc_dense(const Batch& b, const GqaDims& D, const void* qn, const float* gate, const void* k, const void* v, int row_stride, int rows,
                         const int32_t* key_row, void* out, int out_f32, cudaStream_t s) {
    if (b.n <= 0) return WF_OK;
    if (!at_sizes_ok(D) || row_stride % 8 || ((uintptr_t)k & 15) || ((uintptr_t)v & 15)) { set_error("attention: the tcgen05 form does not take these sizes"); return WF_ERR_UNSUPPORTED; }
    AtParams p;
    p.D = D; p.qn = (const __nv_bfloat16*)qn; p.gate = gate; p.out = out; p.out_f32 = out_f32;
    p.block_table = nullptr; p.max_blocks = 0; p.page_size = 1;
    p.key_row = key_row;
    p.rep = D.H / D.G; p.tq = AT_ROWS / p.rep;
    p.box = AT_KEYS;
    p.err = tc_error_word();
    if (!p.err) return WF_ERR_CUDA;
    CUtensorMap tk, tv;
    p.k = (const __nv_bfloat16*)k; p.v = (const __nv_bfloat16*)v;
    p.k_row = p.v_row = row_stride; p.k_head = D.d; p.v_head = D.dv; p.page_stride = 0;
    if (int rc = at_encode(&tk, k, D.d, rows, row_stride, D.G, D.d, 1, (uint64_t)rows * row_stride, AT_KEYS)) return rc;
    if (int rc = at_encode(&tv, v, D.dv, rows, row_stride, D.G, D.dv, 1, (uint64_t)rows * row_stride, AT_KEYS)) return rc;
    return at_launch(b, p, false, tk, tv, s);
}

}  // namespace seq
}  // namespace wf
