// Activation quantisation and the RMSNorm that precedes it.
//
// Reference arithmetic: quantize_activations_i8, tests/test_bitnet_core.py:139-146 (copy of the
// missing sgl_kernel/quantization/bitnet.py); rms_norm, scripts/direct_inference_full.py:181-184.
// HBM/L2-bound elementwise + reduction work: one CTA per token row, 16-byte vector loads, the row is
// read twice (absmax pass, quantise pass) — the second read hits L2/L1.
#include "common.cuh"
#include "wf_bitnet.h"
#include <cuda_fp16.h>

namespace wf {

constexpr int QT = 256;  // threads per CTA

template <typename T> struct Vec;  // 16-byte vector of T
template <> struct Vec<float> {
    static constexpr int N = 4;
    __device__ static void load(const float* p, float (&v)[8]) {
        unpack(*reinterpret_cast<const uint4*>(p), v);
    }
    __device__ static void unpack(const uint4& t, float (&v)[8]) {
        v[0] = __uint_as_float(t.x); v[1] = __uint_as_float(t.y); v[2] = __uint_as_float(t.z); v[3] = __uint_as_float(t.w);
    }
};
template <> struct Vec<__nv_bfloat16> {
    static constexpr int N = 8;
    __device__ static void load(const __nv_bfloat16* p, float (&v)[8]) {
        unpack(*reinterpret_cast<const uint4*>(p), v);
    }
    __device__ static void unpack(const uint4& t, float (&v)[8]) {
        v[0] = bf16lo(t.x); v[1] = bf16hi(t.x); v[2] = bf16lo(t.y); v[3] = bf16hi(t.y);
        v[4] = bf16lo(t.z); v[5] = bf16hi(t.z); v[6] = bf16lo(t.w); v[7] = bf16hi(t.w);
    }
};
template <> struct Vec<__half> {
    static constexpr int N = 8;
    __device__ static void load(const __half* p, float (&v)[8]) {
        unpack(*reinterpret_cast<const uint4*>(p), v);
    }
    __device__ static void unpack(const uint4& t, float (&v)[8]) {
        const __half2* h = reinterpret_cast<const __half2*>(&t);
#pragma unroll
        for (int i = 0; i < 4; ++i) { const float2 f = __half22float2(h[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
    }
};

// f(values, k) over a thread's share of a row, QU vectors in flight: four for the maximum, which only reads (16384 x 6912 bf16: 45 -> 37 us against one);
// one for the quantisation, where more registers mean fewer rows in flight (72 us, 78 with four)
template <int QU, typename T, typename F>
__device__ __forceinline__ void row_vectors(const T* row, int K, F f) {
    constexpr int VN = Vec<T>::N;
    for (int k0 = threadIdx.x * VN; k0 < K; k0 += QU * QT * VN) {
        uint4 raw[QU];
#pragma unroll
        for (int u = 0; u < QU; ++u)
            if (k0 + u * QT * VN < K) raw[u] = *reinterpret_cast<const uint4*>(row + k0 + u * QT * VN);
#pragma unroll
        for (int u = 0; u < QU; ++u) {
            const int k = k0 + u * QT * VN;
            if (k >= K) break;
            float v[8];
            Vec<T>::unpack(raw[u], v);
            f(v, k);
        }
    }
}

template <typename T>
__device__ __forceinline__ float row_absmax(const T* row, int K) {
    float amax = 0.f;
    row_vectors<4>(row, K, [&](const float (&v)[8], int) {
#pragma unroll
        for (int i = 0; i < Vec<T>::N; ++i) amax = fmaxf(amax, fabsf(v[i]));
    });
    return amax;
}

// quantise one row with a known scale; returns this thread's partial sum of q
template <typename T>
__device__ __forceinline__ int row_quant(const T* row, int K, float scale, int8_t* q) {
    int psum = 0;
    const QDiv qd = make_qdiv(scale);
    row_vectors<1>(row, K, [&](const float (&v)[8], int k) {
        const uint32_t w0 = quant_i8x4(v[0], v[1], v[2], v[3], qd);
        psum = __dp4a((int)w0, 0x01010101, psum);
        if (Vec<T>::N == 4) { *reinterpret_cast<uint32_t*>(q + k) = w0; return; }
        const uint32_t w1 = quant_i8x4(v[4], v[5], v[6], v[7], qd);
        psum = __dp4a((int)w1, 0x01010101, psum);
        *reinterpret_cast<uint2*>(q + k) = make_uint2(w0, w1);
    });
    return psum;
}

// per-token: grid = M
template <typename T>
__global__ void __launch_bounds__(QT) act_quant_rows_kernel(const T* x, int K, int ldx, int8_t* __restrict__ q,
                                                            float* __restrict__ scale_out, int32_t* __restrict__ rowsum) {
    __shared__ float fs[33];
    __shared__ int is[33];
    const int m = blockIdx.x;
    const T* row = x + (size_t)m * ldx;
    pdl_wait_prior();
    pdl_launch_dependents();
    const float amax = block_max<QT>(row_absmax(row, K), fs);
    const float scale = act_scale_from_absmax(amax);
    const int total = block_sum_i<QT>(row_quant(row, K, scale, q + (size_t)m * K), is);
    if (threadIdx.x == 0) {
        scale_out[m] = scale;
        if (rowsum) rowsum[m] = total;
    }
}

// per-tensor pass 1: grid-stride absmax -> atomicMax on the float bit pattern (values are >= 0)
template <typename T>
__global__ void __launch_bounds__(QT) act_absmax_kernel(const T* x, int M, int K, int ldx,
                                                        unsigned int* __restrict__ amax_bits) {
    pdl_wait_prior();
    pdl_launch_dependents();
    float amax = 0.f;
    for (int m = blockIdx.x; m < M; m += gridDim.x) amax = fmaxf(amax, row_absmax(x + (size_t)m * ldx, K));
    amax = warp_max(amax);
    if ((threadIdx.x & 31) == 0 && amax > 0.f) atomicMax(amax_bits, __float_as_uint(amax));
}
// The same over rows that follow one another without a gap, as one vector: AU vectors of a thread in flight, whatever the row length leaves over (row by row
// every row ends with a wait for its last loads).  16384 x 6912 bf16, 226 MB: 46 -> 38 us, 5.9 TB/s.
constexpr int AU = 8;
template <typename T>
__global__ void __launch_bounds__(QT) act_absmax_flat_kernel(const T* x, size_t vectors, unsigned int* __restrict__ amax_bits) {
    pdl_wait_prior();
    pdl_launch_dependents();
    const uint4* p = reinterpret_cast<const uint4*>(x);
    const size_t step = (size_t)gridDim.x * QT;
    float amax = 0.f;
    for (size_t i = (size_t)blockIdx.x * QT + threadIdx.x; i < vectors; i += AU * step) {
        uint4 raw[AU];
#pragma unroll
        for (int u = 0; u < AU; ++u) raw[u] = i + u * step < vectors ? p[i + u * step] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int u = 0; u < AU; ++u) {
            float v[8];
            Vec<T>::unpack(raw[u], v);
#pragma unroll
            for (int k = 0; k < Vec<T>::N; ++k) amax = fmaxf(amax, fabsf(v[k]));
        }
    }
    amax = warp_max(amax);
    if ((threadIdx.x & 31) == 0 && amax > 0.f) atomicMax(amax_bits, __float_as_uint(amax));
}
// Per-tensor pass 2: grid = M, last rows first: pass 1 has left those in L2 (with quant_i8x4 79 -> 72 us at 16384 x 6912 bf16; the bytes
// alone are 51; a warp per row with three vectors in flight 91).
template <typename T>
__global__ void __launch_bounds__(QT) act_quant_tensor_kernel(const T* x, int K, int ldx,
                                                              const unsigned int* amax_bits,
                                                              int8_t* __restrict__ q, float* __restrict__ scale_out,
                                                              int32_t* __restrict__ rowsum) {
    __shared__ int is[QT / 32];
    pdl_wait_prior();
    pdl_launch_dependents();
    const int m = gridDim.x - 1 - blockIdx.x;
    const float scale = act_scale_from_absmax(__uint_as_float(*amax_bits));
    const int part = warp_sum_i(row_quant(x + (size_t)m * ldx, K, scale, q + (size_t)m * K));
    if ((threadIdx.x & 31) == 0) is[threadIdx.x >> 5] = part;
    __syncthreads();
    if (threadIdx.x == 0) {
        int total = 0;
#pragma unroll
        for (int i = 0; i < QT / 32; ++i) total += is[i];
        if (m == 0) scale_out[0] = scale;
        if (rowsum) rowsum[m] = total;
    }
}

// RMSNorm (+ optional store) + per-token quant.  Rounding points follow the reference on bf16 tensors:
//   variance = mean(float(x)^2)                         (fp32)
//   r        = bf16( rsqrt(variance + eps) )            (`.to(x.dtype)`)
//   y        = bf16( bf16(x * r) * gamma )              (two bf16 multiplies)
//   q        = quantize_activations_i8(float(y))        (per token)
// The normalised row is kept in shared memory as bf16 (K*2 bytes, dynamic).
__global__ void __launch_bounds__(QT) rmsnorm_quant_kernel(const __nv_bfloat16* x,
                                                           const __nv_bfloat16* gamma, float eps, int K,
                                                           __nv_bfloat16* __restrict__ y_out, int8_t* __restrict__ q,
                                                           float* __restrict__ scale_out, int32_t* __restrict__ rowsum) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __nv_bfloat16* ys = reinterpret_cast<__nv_bfloat16*>(smem_raw);
    __shared__ float fs[33];
    __shared__ int is[33];
    const int m = blockIdx.x;
    const __nv_bfloat16* row = x + (size_t)m * K;
    pdl_wait_prior();
    float ss = 0.f;
    float v[8];
    for (int k = threadIdx.x * 8; k < K; k += QT * 8) {
        Vec<__nv_bfloat16>::load(row + k, v);
#pragma unroll
        for (int i = 0; i < 8; ++i) ss += v[i] * v[i];
    }
    ss = block_sum<QT>(ss, fs);
    const float var = ss / (float)K;
    const float r = bf16_round(1.0f / sqrtf(var + eps));
    float amax = 0.f;
    for (int k = threadIdx.x * 8; k < K; k += QT * 8) {
        float g[8];
        Vec<__nv_bfloat16>::load(row + k, v);
        Vec<__nv_bfloat16>::load(gamma + k, g);
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
            const float y0 = bf16_round(bf16_round(v[i] * r) * g[i]);
            const float y1 = bf16_round(bf16_round(v[i + 1] * r) * g[i + 1]);
            amax = fmaxf(amax, fmaxf(fabsf(y0), fabsf(y1)));
            w[i >> 1] = pack_bf16x2(y0, y1);
        }
        *reinterpret_cast<uint4*>(ys + k) = make_uint4(w[0], w[1], w[2], w[3]);
        if (y_out) *reinterpret_cast<uint4*>(y_out + (size_t)m * K + k) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    amax = block_max<QT>(amax, fs);  // contains __syncthreads: ys is complete
    const float scale = act_scale_from_absmax(amax);
    const int total = block_sum_i<QT>(row_quant<__nv_bfloat16>(ys, K, scale, q + (size_t)m * K), is);
    if (threadIdx.x == 0) {
        scale_out[m] = scale;
        if (rowsum) rowsum[m] = total;
    }
    pdl_launch_dependents();
}

constexpr int QR_T = 512, QR_W = QR_T / 32;
inline int qr_its(int K) { return (K / 8 + QR_T - 1) / QR_T; }
inline int qr_threads(int K) { const int n = K / 8, it = qr_its(K); return ((n + it - 1) / it + 31) & ~31; }
__device__ __forceinline__ float qr_max(float v, float* scratch) {
    v = warp_max(v);
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
    __syncthreads();
    v = (threadIdx.x & 31) < blockDim.x / 32 ? scratch[threadIdx.x & 31] : 0.f;   // of magnitudes
    return warp_max(v);
}
__device__ __forceinline__ float qr_sum(float v, float* scratch) {
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
    __syncthreads();
    v = (threadIdx.x & 31) < blockDim.x / 32 ? scratch[threadIdx.x & 31] : 0.f;
    return warp_sum(v);
}
template <int IT>
__device__ __forceinline__ void qr_load(const __nv_bfloat16* row, int K, uint4 (&raw)[IT]) {
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int k = (it * (int)blockDim.x + (int)threadIdx.x) * 8;
        raw[it] = k < K ? *reinterpret_cast<const uint4*>(row + k) : make_uint4(0u, 0u, 0u, 0u);
    }
}
// The same for rows of up to 8192, which wait in registers: a block of just the warps that the row's vectors fill, up to IT a thread, the row and its gains requested
// before anything is used, one barrier a reduction (each has its own scratch), and the two products in bf16 as packed multiplications, which round the same way (the product
// of two bf16 is exact in 32 bits).  What bounds it is instructions: 40 an element before, about 26 now.  L2 cold: 512 x 6912 14.3 -> 12.3 us, 4096 x 6912 45 -> 41.
template <int IT>
__global__ void __launch_bounds__(QR_T) rmsnorm_quant_regs_kernel(const __nv_bfloat16* x, const __nv_bfloat16* gamma, float eps, int K, __nv_bfloat16* __restrict__ y_out, int8_t* __restrict__ q,
                                                                  float* __restrict__ scale_out, int32_t* __restrict__ rowsum) {
    __shared__ float fs[2][QR_W];
    __shared__ int is[QR_W];
    const int m = blockIdx.x;
    pdl_wait_prior();
    uint4 xv[IT], gv[IT];
    qr_load<IT>(x + (size_t)m * K, K, xv);
    qr_load<IT>(gamma, K, gv);
    float ss = 0.f;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const uint32_t w[4] = {xv[it].x, xv[it].y, xv[it].z, xv[it].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) { const float a = bf16lo(w[i]), b = bf16hi(w[i]); ss += a * a; ss += b * b; }
    }
    const __nv_bfloat162 r2 = __float2bfloat162_rn(1.0f / sqrtf(qr_sum(ss, fs[0]) / (float)K + eps));
    __nv_bfloat162 am = __float2bfloat162_rn(0.f);
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int k = (it * (int)blockDim.x + (int)threadIdx.x) * 8;
        __nv_bfloat162* xh = reinterpret_cast<__nv_bfloat162*>(&xv[it]);
        const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&gv[it]);
#pragma unroll
        for (int i = 0; i < 4; ++i) { xh[i] = __hmul2_rn(__hmul2_rn(xh[i], r2), gh[i]); am = __hmax2(am, __habs2(xh[i])); }
        if (y_out && k < K) *reinterpret_cast<uint4*>(y_out + (size_t)m * K + k) = xv[it];
    }
    const float scale = act_scale_from_absmax(qr_max(fmaxf(__low2float(am), __high2float(am)), fs[1]));
    const QDiv qd = make_qdiv(scale);
    int psum = 0;
#pragma unroll
    for (int it = 0; it < IT; ++it) {
        const int k = (it * (int)blockDim.x + (int)threadIdx.x) * 8;
        if (k >= K) break;
        float v[8];
        Vec<__nv_bfloat16>::unpack(xv[it], v);
        const uint32_t w0 = quant_i8x4(v[0], v[1], v[2], v[3], qd), w1 = quant_i8x4(v[4], v[5], v[6], v[7], qd);
        psum = __dp4a((int)w1, 0x01010101, __dp4a((int)w0, 0x01010101, psum));
        *reinterpret_cast<uint2*>(q + (size_t)m * K + k) = make_uint2(w0, w1);
    }
    psum = warp_sum_i(psum);
    if ((threadIdx.x & 31) == 0) is[threadIdx.x >> 5] = psum;
    __syncthreads();
    if (threadIdx.x < 32) {
        psum = warp_sum_i(threadIdx.x < blockDim.x / 32 ? is[threadIdx.x] : 0);
        if (threadIdx.x == 0) {
            scale_out[m] = scale;
            if (rowsum) rowsum[m] = psum;
        }
    }
    pdl_launch_dependents();
}

}  // namespace wf

using namespace wf;

template <typename T>
static int launch_act_quant(const T* x, int M, int K, int ldx, int per_token, int8_t* q, float* scale_out, int32_t* rowsum,
                            void* workspace, cudaStream_t s) {
    if (per_token) {
        launch_pdl(act_quant_rows_kernel<T>, M, QT, 0, s, x, K, ldx, q, scale_out, rowsum);
    } else {
        if (cuda_check(cudaMemsetAsync(workspace, 0, 4, s), "memset absmax")) return WF_ERR_CUDA;
        const int sms = sm_count();
        const size_t vectors = (size_t)M * K / Vec<T>::N;
        if (ldx == K && vectors >= (size_t)sms * 4 * QT * AU) launch_pdl(act_absmax_flat_kernel<T>, sms * 4, QT, 0, s, x, vectors, (unsigned int*)workspace);
        else launch_pdl(act_absmax_kernel<T>, M < sms * 4 ? M : sms * 4, QT, 0, s, x, M, K, ldx, (unsigned int*)workspace);
        launch_pdl(act_quant_tensor_kernel<T>, M, QT, 0, s, x, K, ldx, (const unsigned int*)workspace, q, scale_out, rowsum);
    }
    return launch_check(cudaGetLastError(), "wf_act_quant_i8");
}

extern "C" int wf_act_quant_i8(const void* x, int x_dtype, int M, int K, int ldx, int per_token, int8_t* q, float* scale_out,
                               int32_t* rowsum_out, void* workspace, void* stream) {
    if (!x || !q || !scale_out) { set_error("wf_act_quant_i8: null pointer"); return WF_ERR_INVALID; }
    if (M < 0 || K <= 0) { set_error("wf_act_quant_i8: bad shape M=%d K=%d", M, K); return WF_ERR_INVALID; }
    if (M == 0) return WF_OK;
    if (K % 8 != 0 || ldx % 8 != 0) { set_error("wf_act_quant_i8: K (%d) and ldx (%d) must be multiples of 8", K, ldx); return WF_ERR_UNSUPPORTED; }
    if (!per_token && !workspace) { set_error("wf_act_quant_i8: per-tensor mode needs a 4-byte workspace"); return WF_ERR_INVALID; }
    cudaStream_t s = (cudaStream_t)stream;
    switch (x_dtype) {
        case WF_F32: return launch_act_quant((const float*)x, M, K, ldx, per_token, q, scale_out, rowsum_out, workspace, s);
        case WF_BF16: return launch_act_quant((const __nv_bfloat16*)x, M, K, ldx, per_token, q, scale_out, rowsum_out, workspace, s);
        case WF_F16: return launch_act_quant((const __half*)x, M, K, ldx, per_token, q, scale_out, rowsum_out, workspace, s);
    }
    set_error("wf_act_quant_i8: bad dtype %d", x_dtype);
    return WF_ERR_INVALID;
}

namespace wf {
int launch_rmsnorm_quant(const void* x, const void* gamma, float eps, int M, int K, void* y_out, int8_t* q, float* scale_out,
                         int32_t* rowsum_out, cudaStream_t s, bool pdl) {
    const size_t smem = (size_t)K * 2;
    static DevOnce attr_set;
    if (attr_set.need()) cudaFuncSetAttribute(rmsnorm_quant_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
    const int it = qr_its(K);   // measured up to two vectors a thread; wider rows keep the form with the row in shared memory
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(M);
    cfg.blockDim = dim3(it <= 2 ? qr_threads(K) : QT);
    cfg.dynamicSmemBytes = it <= 2 ? 0 : smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    return launch_check(cudaLaunchKernelEx(&cfg, it == 1 ? rmsnorm_quant_regs_kernel<1> : it == 2 ? rmsnorm_quant_regs_kernel<2> : rmsnorm_quant_kernel, (const __nv_bfloat16*)x, (const __nv_bfloat16*)gamma, eps, K,
                                         (__nv_bfloat16*)y_out, q, scale_out, rowsum_out),
                      "wf_rmsnorm_quant");
}
}  // namespace wf

extern "C" int wf_rmsnorm_quant(const void* x, const void* gamma, float eps, int M, int K, void* y_out, int8_t* q,
                                float* scale_out, int32_t* rowsum_out, void* stream) {
    if (!x || !gamma || !q || !scale_out) { set_error("wf_rmsnorm_quant: null pointer"); return WF_ERR_INVALID; }
    if (M <= 0 || K <= 0 || K % 8 != 0) { set_error("wf_rmsnorm_quant: bad shape M=%d K=%d (K %% 8 == 0)", M, K); return WF_ERR_INVALID; }
    if ((size_t)K * 2 > 128 * 1024) { set_error("wf_rmsnorm_quant: K=%d exceeds the 64K-element row limit", K); return WF_ERR_UNSUPPORTED; }
    return launch_rmsnorm_quant(x, gamma, eps, M, K, y_out, q, scale_out, rowsum_out, (cudaStream_t)stream, true);
}

namespace wf {
void quant_init_attrs() { cudaFuncSetAttribute(rmsnorm_quant_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024); }
}
