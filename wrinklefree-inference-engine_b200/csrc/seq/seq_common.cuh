// Shared pieces of the sequence-model kernels (hybrid stacks of attention / recurrent mixers with routed feed-forwards): element types,
// the flat ragged batch every kernel indexes, small reductions.  Storage type T is __nv_bfloat16 or float (the all-32-bit mode); residual
// stream, norms, softmax, rotary angles, routers and recurrent state are float in both.
#pragma once
#include "../common.cuh"

namespace wf {
namespace seq {

template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// four consecutive elements (16-byte aligned floats, 8-byte aligned bf16)
template <typename T> __device__ __forceinline__ float4 load4(const T* p);
template <> __device__ __forceinline__ float4 load4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 load4<__nv_bfloat16>(const __nv_bfloat16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
}
__device__ __forceinline__ void store4(float* p, const float (&v)[4]) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void store4(__nv_bfloat16* p, const float (&v)[4]) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}
inline bool vec_ok(const void* p, size_t align) { return ((uintptr_t)p & (align - 1)) == 0; }

// One step's ragged batch: n tokens laid out sequence after sequence.  All arrays live on the device.
struct Batch {
    int n = 0;                 // tokens
    int nseq = 0;              // sequences
    const int32_t* tok_seq;    // [n] index of the token's sequence in this step
    const int32_t* tok_pos;    // [n] absolute position in its sequence
    const int32_t* seq_start;  // [nseq] first token of the sequence in the flat batch
    const int32_t* seq_len;    // [nseq] tokens of the sequence in this step
    const int32_t* seq_pos0;   // [nseq] position of its first token
    const int32_t* seq_slot;   // [nseq] state slot = block-table row
    int max_len = 0;           // longest portion of the step (known on the host; sizes grids that cut portions into chunks)
    const int32_t* key_row = nullptr;   // [nseq] first row of the sequence where all its positions so far lie one sequence after another
    int max_ctx = 0;           // most positions that a sequence holds behind the step (known on the host)
    int ctx_total = 0;         // those rows: the sum over sequences of the positions behind the step (known on the host)
};

// Every kernel of the engine but the scans of the recurrences is launched by launch_pdl and begins with pdl_enter (the CTA pairs' product: behind its set-up): its launch overlaps the kernel
// before it in the stream, whose results, and whose reads of what this one overwrites, are complete behind pdl_enter.  A decode step is a chain of some 40
// kernels of 2 to 6 us, a prompt layer one of 15 to 25, at about 1 us of launch each.  Measured without / with: a decode step of 8 sequences, four layers
// 182 / 159 us (221 where a kernel lets the next one in before its own wait: the CTAs of several waiting kernels then hold slots); layers 524 / 491, 940 / 918, 1060 / 1019 us.
__device__ __forceinline__ void pdl_enter() { pdl_wait_prior(); pdl_launch_dependents(); }
// Kernels of one short block a row do so (their last argument) up to eight blocks an SM: the two instructions cost a block some 0.5 us, which beyond that is more than
// the overlap gives.  16128 padded rows of a routed feed-forward: their activation (384 wide) 22.5 us with them, 16 without; plan and gathering (2560 wide) 28.5 / 23.
inline bool few_blocks(dim3 grid) { return (long long)grid.x * grid.y * grid.z <= 8LL * sm_count(); }
template <typename... P, typename... A>
inline cudaError_t launch_rows(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
    if (few_blocks(grid)) return launch_pdl(kernel, grid, block, smem, s, std::forward<A>(args)..., true);
    kernel<<<grid, block, smem, s>>>(std::forward<A>(args)..., false);
    return cudaPeekAtLastError();
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
// sum over a block of up to 1024 threads; every thread gets the result (every warp adds the warps' sums for itself).  scratch: 33 floats of shared memory
__device__ __forceinline__ float block_sum(float v, float* scratch) {
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    __syncthreads();
    if (lane == 0) scratch[w] = v;
    __syncthreads();
    return warp_sum(lane < nw ? scratch[lane] : 0.f);
}
// the same where nothing else uses the scratch before.  many: of more blocks than SMs hold, where instructions count and not a block's latency, one warp adds for all (rows of 1024,
// 4000 of them 12.4 -> 11.6 us; 300 2.4 / 2.6)
__device__ __forceinline__ float block_sum_once(float v, float* scratch, bool many = false) {
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    if (lane == 0) scratch[w] = v;
    __syncthreads();
    if (many) {
        if (w == 0) {
            v = warp_sum(lane < nw ? scratch[lane] : 0.f);
            if (lane == 0) scratch[32] = v;
        }
        __syncthreads();
        return scratch[32];
    }
    return warp_sum(lane < nw ? scratch[lane] : 0.f);
}
__device__ __forceinline__ float gelu_erf_f(float z) { return 0.5f * z * (1.f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float epilogue_f(int ep, float v) {        // GemmArgs::ep
    if (ep == 1) { v = fmaxf(v, 0.f); return v * v; }
    return ep == 2 ? gelu_erf_f(v) : v;
}
__device__ __forceinline__ float sigmoid_f(float z) { return 1.f / (1.f + expf(-z)); }
__device__ __forceinline__ float silu_f(float z) { return z / (1.f + expf(-z)); }
// gated activations (launch_silu_mul's act): silu(g) u; 1: clamped, with u + 1; 2: tanh-gelu(g) u
__device__ __forceinline__ float glu_f(int act, float g, float u, float limit) {
    if (act == 1) {
        const float gg = fminf(g, limit), uu = fminf(fmaxf(u, -limit), limit);
        return gg * sigmoid_f(1.702f * gg) * (uu + 1.f);
    }
    if (act == 2) return 0.5f * g * (1.f + tanhf(0.7978845608028654f * (g + 0.044715f * g * g * g))) * u;
    return silu_f(g) * u;
}
__device__ __forceinline__ float softplus_f(float z) { return z > 20.f ? z : log1pf(expf(z)); }

}  // namespace seq
}  // namespace wf
