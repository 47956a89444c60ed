/* TEST INFRASTRUCTURE ONLY.
 *
 * CPU restatement (plain C, scalar, exact integer arithmetic) of the reference's
 * BitNet b1.58 decode hot path.  Nothing under oracle/ may be imported, linked or
 * executed by the product (the CUDA library + its Python host); only tests/,
 * __graft_entry__.smoke() and bench.py's cpu_baseline / --impl reference legs use it,
 * and only as the checker / CPU baseline.
 *
 * Parity status: PINNED.  tests/test_oracle_golden.py checks every function here
 * against (a) golden vectors generated by importing the reference's own Python
 * (tests/golden/make_golden.py -> tests/golden/*.npz) and (b) the unmodified
 * reference SIMD kernel built into oracle/_ref/libwf_ref.so (oracle/Makefile).
 *
 * Each function cites the reference file:line it follows (paths relative to
 * /root/reference).
 */
#include <stdint.h>
#include <stddef.h>
#include <string.h>
#include <math.h>
#include <stdlib.h>

#define WFO_QK 128 /* QK_I2_S, extern/BitNet/src/ggml-bitnet-mad.cpp:9 */

/* ------------------------------------------------------------------------- */
/* Weight packing                                                            */
/* ------------------------------------------------------------------------- */

/* Block geometry shared by pack and unpack: tests/test_bitnet_core.py:83-90
 * (block_size = 32 bytes = 128 weights; if K < 128 a single block of K/4 bytes). */
static void wfo_block_geom(int K, int* block_bytes, int* num_blocks) {
    int bb = 32;
    int nb = K / (bb * 4);
    if (nb == 0) { bb = K / 4; nb = 1; }
    *block_bytes = bb;
    *num_blocks = nb;
}

/* _pack_ternary_weights: src/wrinklefree_inference/cache/bitnet_converter.py:26-77
 * == tests/test_bitnet_core.py:56-106.  round-half-even (torch.round), clamp to
 * [-1,1], code = w+1, blocked layout: byte (b*bb + k) = c[base+k]<<6 | c[base+k+bb]<<4 |
 * c[base+k+2bb]<<2 | c[base+k+3bb].  scale = max|w| (1.0 if < 1e-6).
 * Returns 0, or -1 if K % 4 != 0 (the reference raises ValueError). */
int wfo_pack_ternary(const float* w, int N, int K, uint8_t* packed, float* scale) {
    if (K % 4 != 0) return -1;
    int bb, nb;
    wfo_block_geom(K, &bb, &nb);
    float amax = 0.f;
    for (size_t i = 0; i < (size_t)N * K; ++i) {
        float a = fabsf(w[i]);
        if (a > amax) amax = a;
    }
    for (int n = 0; n < N; ++n) {
        const float* row = w + (size_t)n * K;
        uint8_t* prow = packed + (size_t)n * (K / 4);
        memset(prow, 0, (size_t)K / 4);
        for (int b = 0; b < nb; ++b) {
            int base = b * bb * 4;
            for (int k = 0; k < bb; ++k) {
                uint8_t byte = 0;
                for (int g = 0; g < 4; ++g) {
                    float t = nearbyintf(row[base + k + g * bb]); /* ties-to-even like torch.round */
                    if (t < -1.f) t = -1.f;
                    if (t > 1.f) t = 1.f;
                    uint8_t code = (uint8_t)((int)t + 1);
                    byte |= (uint8_t)(code << (6 - 2 * g));
                }
                prow[b * bb + k] = byte;
            }
        }
    }
    *scale = (amax < 1e-6f) ? 1.0f : amax;
    return 0;
}

/* quantize_i2_s: extern/BitNet/src/ggml-bitnet-mad.cpp:46-92.  |x|<1e-6 -> code 1;
 * x*max > 0 -> 2 else 0; flat 128-blocking over the whole tensor (coincides with
 * per-row blocking when K % 128 == 0).  Returns scale = max|x|. */
float wfo_quantize_i2_s(const float* src, int N, int K, uint8_t* dst) {
    size_t n = (size_t)N * K;
    double mx = 0;
    for (size_t i = 0; i < n; ++i) mx = fmax(mx, fabs((double)src[i]));
    memset(dst, 0, n / 4);
    for (size_t i = 0; i < n / WFO_QK; ++i) {
        for (int j = 0; j < WFO_QK; ++j) {
            double x = (double)src[i * WFO_QK + j];
            uint8_t q = (fabs(x) < 1e-6) ? 1 : ((x * mx > 0) ? 2 : 0);
            dst[i * 32 + (j % 32)] |= (uint8_t)(q << (6 - 2 * (j / 32)));
        }
    }
    return (float)mx;
}

/* _unpack_i2_to_ternary: tests/test_bitnet_core.py:109-136. */
void wfo_unpack_i2s(const uint8_t* packed, int N, int K, float* w) {
    int bb, nb;
    wfo_block_geom(K, &bb, &nb);
    for (int n = 0; n < N; ++n) {
        const uint8_t* prow = packed + (size_t)n * (K / 4);
        float* row = w + (size_t)n * K;
        for (int b = 0; b < nb; ++b) {
            int base = b * bb * 4;
            for (int k = 0; k < bb; ++k) {
                uint8_t byte = prow[b * bb + k];
                for (int g = 0; g < 4; ++g)
                    row[base + k + g * bb] = (float)((byte >> (6 - 2 * g)) & 3) - 1.0f;
            }
        }
    }
}

/* _unpack_ternary_weights (HF checkpoint layout u8 [N/4, K], blocked along N):
 * tests/test_bitnet_core.py:21-53; extern/BitNet/utils/convert-hf-to-gguf-bitnet.py:731-739. */
void wfo_unpack_hf(const uint8_t* hf, int N4, int K, float* w) {
    for (int i = 0; i < 4; ++i)
        for (int r = 0; r < N4; ++r)
            for (int k = 0; k < K; ++k)
                w[((size_t)i * N4 + r) * K + k] = (float)((hf[(size_t)r * K + k] >> (2 * i)) & 3) - 1.0f;
}

/* HF [N/4,K] -> I2_S [N,K/4] without the float detour (composition of the two above;
 * DirectBitNetInference._repack_hf_weight, scripts/direct_inference_full.py:113-117). */
void wfo_hf_to_i2s(const uint8_t* hf, int N4, int K, uint8_t* packed) {
    int bb, nb;
    wfo_block_geom(K, &bb, &nb);
    for (int i = 0; i < 4; ++i)
        for (int r = 0; r < N4; ++r) {
            const uint8_t* src = hf + (size_t)r * K;
            uint8_t* prow = packed + ((size_t)i * N4 + r) * (K / 4);
            for (int b = 0; b < nb; ++b)
                for (int k = 0; k < bb; ++k) {
                    uint8_t byte = 0;
                    for (int g = 0; g < 4; ++g)
                        byte |= (uint8_t)(((src[b * bb * 4 + k + g * bb] >> (2 * i)) & 3) << (6 - 2 * g));
                    prow[b * bb + k] = byte;
                }
        }
}

/* kernels/native.py pack_weights / unpack_weights (LSB-sequential; :181-216):
 * byte j bits (2i+1..2i) = code of w[4j+i]. */
void wfo_native_pack(const float* w, int N, int K, uint8_t* packed) {
    for (int n = 0; n < N; ++n)
        for (int j = 0; j < K / 4; ++j) {
            uint8_t byte = 0;
            for (int i = 0; i < 4; ++i) {
                int c = (int)w[(size_t)n * K + 4 * j + i] + 1; /* astype(int32) truncation, :195 */
                if (c < 0) c = 0;
                if (c > 2) c = 2;
                byte |= (uint8_t)(c << (2 * i));
            }
            packed[(size_t)n * (K / 4) + j] = byte;
        }
}

/* ------------------------------------------------------------------------- */
/* Activation quantisation                                                   */
/* ------------------------------------------------------------------------- */

/* quantize_activations_i8: tests/test_bitnet_core.py:139-146 (copy of
 * sgl_kernel/quantization/bitnet.py).  max_val is an fp32 value read out with
 * .item() (-> Python double); scale = max_val / 127.0 is a DOUBLE division; torch
 * then divides the fp32 tensor by that scalar cast to fp32; .round() is
 * ties-to-even; clamp(-128,127).  Returns the scale as the fp32 value the tensor op
 * used; *scale_f64 (optional) receives the Python-float the reference returns. */
float wfo_quantize_act_i8(const float* x, size_t n, int8_t* q, double* scale_f64) {
    float amax = 0.f;
    for (size_t i = 0; i < n; ++i) {
        float a = fabsf(x[i]);
        if (a > amax) amax = a; /* NaN never wins, like at::max on non-NaN data */
    }
    double mv = (double)amax;
    if (mv < 1e-6) mv = 1.0;
    double sd = mv / 127.0;
    float s = (float)sd;
    for (size_t i = 0; i < n; ++i) {
        float r = nearbyintf(x[i] / s);
        if (r < -128.f) r = -128.f;
        if (r > 127.f) r = 127.f;
        q[i] = (int8_t)r;
    }
    if (scale_f64) *scale_f64 = sd;
    return s;
}

/* per-token variant: the same function applied to each row on its own
 * (what bitnet_linear sees at M == 1, scripts/direct_inference_full.py:196). */
void wfo_quantize_act_i8_rows(const float* x, int M, int K, int8_t* q, float* scales, int32_t* rowsum) {
    for (int m = 0; m < M; ++m) {
        scales[m] = wfo_quantize_act_i8(x + (size_t)m * K, (size_t)K, q + (size_t)m * K, NULL);
        if (rowsum) {
            int32_t s = 0;
            for (int k = 0; k < K; ++k) s += q[(size_t)m * K + k];
            rowsum[m] = s;
        }
    }
}

/* ------------------------------------------------------------------------- */
/* Dot products / GEMV / GEMM                                                */
/* ------------------------------------------------------------------------- */

/* ggml_vec_dot_i2_i8_s: extern/BitNet/src/ggml-bitnet-mad.cpp:94-186.
 * sumi = sum_k code[k] * y[k] with code in {0,1,2} read from the blocked layout:
 * byte j of 128-block b carries k = b*128 + {j, 32+j, 64+j, 96+j} in bits 7-6, 5-4,
 * 3-2, 1-0.  Exact int64 here; the AVX2 kernel's int16 lane partials can wrap on
 * adversarial data — wfo_vec_dot_i2_i8_avx2model models that. */
int64_t wfo_vec_dot_i2_i8(int K, const uint8_t* x, const int8_t* y) {
    int64_t sum = 0;
    int nb = K / WFO_QK;
    for (int b = 0; b < nb; ++b) {
        /* one block's 128 terms fit an int32 exactly (|term| <= 3 * 128); the inner loops run over contiguous bytes so that the
         * compiler can vectorise them */
        int32_t part = 0;
        for (int g = 0; g < 4; ++g) {
            const int sh = 6 - 2 * g;
            for (int j = 0; j < 32; ++j) part += (int32_t)((x[b * 32 + j] >> sh) & 3) * (int32_t)y[b * WFO_QK + g * 32 + j];
        }
        sum += part;
    }
    return sum;
}

/* Bit-faithful scalar model of the AVX2 data path (same file, :103-186): per group of
 * up to 32 blocks, 16 int16 lanes accumulate maddubs pair sums with wrap-around
 * (_mm256_add_epi16); maddubs itself saturates (cannot trigger: |2*128*2| < 32768);
 * then madd_epi16 widens to int32.  Used to document where the reference wraps. */
int32_t wfo_vec_dot_i2_i8_avx2model(int K, const uint8_t* x, const int8_t* y) {
    int nb = K / WFO_QK;
    int32_t total = 0;
    for (int g0 = 0; g0 < nb; g0 += 32) {
        int gcount = nb - g0 < 32 ? nb - g0 : 32;
        int16_t lanes[16];
        memset(lanes, 0, sizeof lanes);
        for (int jb = 0; jb < gcount; ++jb) {
            int b = g0 + jb;
            for (int l = 0; l < 16; ++l) {
                int32_t acc = 0;
                for (int g = 0; g < 4; ++g)
                    for (int e = 0; e < 2; ++e) {
                        int j = 2 * l + e;
                        uint8_t code = (x[b * 32 + j] >> (6 - 2 * g)) & 3;
                        acc += (int32_t)code * (int32_t)y[b * WFO_QK + g * 32 + j];
                    }
                /* the four maddubs results are added pairwise in int16 (wrapping) */
                lanes[l] = (int16_t)(uint16_t)((uint16_t)lanes[l] + (uint16_t)(int16_t)acc);
            }
        }
        for (int l = 0; l < 16; ++l) total += lanes[l];
    }
    return total;
}

/* bitnet_gemv(packed, x_i8, scale) -> f32[N]; semantic reference
 * tests/test_bitnet_core.py:149-167: y[n] = scale * sum_k (w[n,k]+1) * a[k].
 * The fp32 value is (float)sumi * scale, one rounding (mad.cpp:186 then the op's scale). */
void wfo_gemv(const uint8_t* packed, const int8_t* act, float scale, int N, int K, float* out) {
    /* rows are independent and each is an exact integer sum: splitting them over threads changes nothing */
#pragma omp parallel for schedule(static) if (N >= 64)
    for (int n = 0; n < N; ++n)
        out[n] = (float)wfo_vec_dot_i2_i8(K, packed + (size_t)n * (K / 4), act) * scale;
}

/* bitnet_gemm(packed, X_i8[M,K], scale) -> f32[M,N] (bitnet_patch.py:73). */
void wfo_gemm(const uint8_t* packed, const int8_t* act, float scale, int M, int N, int K, float* out) {
    for (int m = 0; m < M; ++m)
        wfo_gemv(packed, act + (size_t)m * K, scale, N, K, out + (size_t)m * N);
}

/* Raw int32 accumulators: mode 0 = sum (w+1)*a (what the kernel returns),
 * mode 1 = sum w*a (= mode 0 minus sum a; what kernels/native.py:27-41 computes). */
void wfo_gemm_i32(const uint8_t* packed, const int8_t* act, int M, int N, int K, int mode, int32_t* out) {
    for (int m = 0; m < M; ++m) {
        const int8_t* a = act + (size_t)m * K;
        int64_t asum = 0;
        for (int k = 0; k < K; ++k) asum += a[k];
        for (int n = 0; n < N; ++n) {
            int64_t s = wfo_vec_dot_i2_i8(K, packed + (size_t)n * (K / 4), a);
            out[(size_t)m * N + n] = (int32_t)(mode ? s - asum : s);
        }
    }
}

/* kernels/native.py bitnet_dot (:27-41): LSB-sequential layout, sum (code-1)*a. */
int32_t wfo_native_dot(int K, const uint8_t* packed, const int8_t* act) {
    int32_t sum = 0;
    for (int i = 0; i < K / 4; ++i) {
        uint8_t byte = packed[i];
        for (int j = 0; j < 4; ++j) sum += (((byte >> (2 * j)) & 3) - 1) * (int32_t)act[i * 4 + j];
    }
    return sum;
}

/* ------------------------------------------------------------------------- */
/* bitnet_linear: quant -> gemv -> Sigma-a correction -> dequant              */
/* ------------------------------------------------------------------------- */

/* scripts/direct_inference_full.py:186-208 (one row; the reference loops rows):
 *   x_i8, s_a = quantize_activations_i8(x.float())
 *   out = bitnet_gemv(W, x_i8, s_w)               # fp32: s_w * sum (w+1) a
 *   out = (out - s_w * act_sum) * s_a             # python-double scalars cast to fp32 by torch
 * out_f32[n] is returned; the caller rounds to bf16 (:208). */
void wfo_bitnet_linear(const float* x, const uint8_t* packed, float w_scale, int N, int K, float* out) {
    int8_t* q = (int8_t*)malloc((size_t)K);
    double s_a64;
    wfo_quantize_act_i8(x, (size_t)K, q, &s_a64);
    int64_t asum = 0;
    for (int k = 0; k < K; ++k) asum += q[k];
    float corr = (float)((double)w_scale * (double)asum); /* Python float product, then cast */
    float s_a = (float)s_a64;
#pragma omp parallel for schedule(static) if (N >= 64)
    for (int n = 0; n < N; ++n) {
        float y = (float)wfo_vec_dot_i2_i8(K, packed + (size_t)n * (K / 4), q) * w_scale;
        out[n] = (y - corr) * s_a;
    }
    free(q);
}
