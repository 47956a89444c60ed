// What the forms of the matrix-state recurrences over many tokens share (seq_chunk.cu, seq_segment.cu): float products on mma.sync m16n8k8 with every operand as
// a sum of two tf32 numbers (hi hi + hi lo + lo hi, 22 to 24 bits of each product), and the watch for numbers that are not finite.
#pragma once
#include "seq_kernels.cuh"

namespace wf {
namespace seq {

constexpr int CR_COLS = 16;        // columns of a mark of chunk_redo_kernel

struct ChunkView {
    const float *qkv, *beta, *decay; int ld, q_off, k_off, v_off;
    float* rec;
    int nchunks;
    int *redo, cols;               // [sequence][head][CR_COLS columns]: marked; zero between launches
};

// x * 0 summed up: zero while everything is finite, NaN from the first infinity or NaN on
__device__ __forceinline__ void cr_watch(float& w, float x) { w = fmaf(x, 0.f, w); }

// Recurrences with one decay per head and no correction, in segments of SCAN_CHUNK tokens (seq_segment.cu): the segments' own end states and products q k in w.rec,
// the chain between them, the outputs.  What it marks is left to chunk_redo_kernel.
bool segments_faster(const DeltaDims& D, int nseq, int n, int max_len);          // n tokens in nseq portions
bool segments_usable(const Batch& b, const DeltaDims& D, const ScanWorkspace* scan);
int launch_segments(const Batch& b, const DeltaDims& D, const ChunkView& w, const float* decay, float* state, size_t slot_stride, float* o, cudaStream_t s, const ScanWorkspace* scan);

__device__ __forceinline__ void cr_split(float x, uint32_t& hi, uint32_t& lo) {
    // round to 10 stored bits by integer arithmetic (the conversion instruction runs at a fraction of its rate); the instruction drops the low 13 bits of lo
    hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(x - __uint_as_float(hi)) + 0x1000u;
}
__device__ __forceinline__ void cr_mma(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void cr_mma0(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {       // the first of a chain: the sum begins with it
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}
struct CrA { uint32_t h[4], l[4]; };
struct CrB { uint32_t h[2], l[2]; };
// an accumulator tile as the A operand: columns 2 t and 2 t + 1 become k = t and t + 4
__device__ __forceinline__ CrA cr_a(const float (&c)[4]) {
    CrA a;
    cr_split(c[0], a.h[0], a.l[0]); cr_split(c[2], a.h[1], a.l[1]); cr_split(c[1], a.h[2], a.l[2]); cr_split(c[3], a.h[3], a.l[3]);
    return a;
}
__device__ __forceinline__ CrB cr_b(float x, float y) {
    CrB b;
    cr_split(x, b.h[0], b.l[0]); cr_split(y, b.h[1], b.l[1]);
    return b;
}
__device__ __forceinline__ CrB cr_b2(const float* p) { const float2 v = *reinterpret_cast<const float2*>(p); return cr_b(v.x, v.y); }
__device__ __forceinline__ void cr_mma3(float (&d)[4], const CrA& a, const CrB& b) { cr_mma(d, a.l, b.h); cr_mma(d, a.h, b.l); cr_mma(d, a.h, b.h); }

}  // namespace seq
}  // namespace wf
