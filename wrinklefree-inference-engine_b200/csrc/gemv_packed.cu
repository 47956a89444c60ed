// One or two tokens on the packed (checkpoint) weight layout: a warp per R weight rows, packed bytes straight from memory into registers, products with dp4a.
//
//   S[m,n] = sum_k code[n,k] * a[m,k], exact int32; then any output form of the linear epilogue but relu^2 * up.
//
// What bounds it is the weight stream.  The tiled kernel (gemm_mma.cu) pads one token to eight, stages 16-byte pieces through shared memory and spends about
// three times the instructions per weight byte.  Measured there / here, one token: 28672 x 8192 (59 MB) 26.3 / 14.3 us (4.1 TB/s), 8192 x 8192 10.5 / 4.9,
// 2560 x 2560 4.9 / 2.4; two tokens 27.7 / 20.8, 10.3 / 6.9, 5.1 / 2.8.  Here a lane holds 16 bytes (64 codes) of R rows and the next 16 bytes of
// each under way; the activations lie in shared memory as [k group][16-byte piece], so that a warp's reads meet no bank twice and serve R rows.
#include "linear_common.cuh"

namespace wf {

constexpr int GP_WARPS = 8;

struct PackedParams {
    const uint8_t* w;
    const int8_t* q;
    int N, K, ldq;
    EpiParams ep;
};

template <int M, int R>
__global__ void __launch_bounds__(GP_WARPS * 32) ternary_gemv_packed_kernel(const PackedParams p) {
    extern __shared__ __align__(16) uint4 xs[];            // [M][4 groups][K / 64]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int pieces = p.K / 64, row0 = (blockIdx.x * GP_WARPS + warp) * R;
    pdl_wait_prior();
    const uint4* wr[R];                                    // rows past N repeat the last one; they are not stored
#pragma unroll
    for (int r = 0; r < R; ++r) wr[r] = reinterpret_cast<const uint4*>(p.w + (size_t)min(row0 + r, p.N - 1) * (p.K / 4));
    uint4 w[R];
    int c = lane;
    if (c < pieces) {
#pragma unroll
        for (int r = 0; r < R; ++r) w[r] = __ldg(wr[r] + c);
    }
    // byte j of a 32-byte block holds the codes of k = j, j + 32, j + 64, j + 96 from its high bits down: group g of piece c starts at k = c / 2 * 128 + 32 g + c % 2 * 16
    for (int i = tid; i < M * 4 * pieces; i += GP_WARPS * 32) {
        const int m = i / (4 * pieces), s = i - m * 4 * pieces, blk = s >> 3, g = (s >> 1) & 3, half = s & 1;
        xs[(m * 4 + g) * pieces + blk * 2 + half] = reinterpret_cast<const uint4*>(p.q + (size_t)m * p.ldq)[s];
    }
    __syncthreads();
    int acc[M][R];
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
        for (int r = 0; r < R; ++r) acc[m][r] = 0;
    for (; c < pieces; c += 32) {
        uint4 cur[R];
#pragma unroll
        for (int r = 0; r < R; ++r) cur[r] = w[r];
        if (c + 32 < pieces) {
#pragma unroll
            for (int r = 0; r < R; ++r) w[r] = __ldg(wr[r] + c + 32);
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            uint4 x[M];
#pragma unroll
            for (int m = 0; m < M; ++m) x[m] = xs[(m * 4 + g) * pieces + c];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const uint32_t k0 = (cur[r].x >> (6 - 2 * g)) & 0x03030303u, k1 = (cur[r].y >> (6 - 2 * g)) & 0x03030303u;
                const uint32_t k2 = (cur[r].z >> (6 - 2 * g)) & 0x03030303u, k3 = (cur[r].w >> (6 - 2 * g)) & 0x03030303u;
#pragma unroll
                for (int m = 0; m < M; ++m)
                    acc[m][r] = __dp4a((int)k0, (int)x[m].x, __dp4a((int)k1, (int)x[m].y, __dp4a((int)k2, (int)x[m].z, __dp4a((int)k3, (int)x[m].w, acc[m][r]))));
            }
        }
    }
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int s = warp_sum_i(acc[m][r]);
            if (lane == 0 && row0 + r < p.N) epilogue_store(p.ep, m, row0 + r, s);
        }
}

template <int M, int R>
static int launch_packed(const PackedParams& p, cudaStream_t s) {
    const int rows = GP_WARPS * R;
    return launch_check(launch_pdl(ternary_gemv_packed_kernel<M, R>, (p.N + rows - 1) / rows, GP_WARPS * 32, (size_t)M * p.K, s, p), "ternary_gemv_packed");
}

// the activations have to fit the shared memory that every kernel has
bool gemv_packed_usable(const wf_linear_args* a) {
    return a->w_layout == WF_W_I2S && a->M >= 1 && a->M <= 2 && (size_t)a->M * a->K <= 48 * 1024 && !(a->out_mode == WF_OUT_LINEAR && (a->epi_flags & WF_EPI_RELU2_MUL));
}

int launch_gemv_packed(const wf_linear_args* a, const EpiParams& ep, cudaStream_t s) {
    PackedParams p;
    p.w = a->w; p.q = a->q; p.N = a->N; p.K = a->K; p.ldq = a->ldq; p.ep = ep;
    // rows per warp: as many as leave the SMs 16 warps each
    const long long warps = 16LL * sm_count();
    if (a->M == 1) return a->N >= 4 * warps ? launch_packed<1, 4>(p, s) : a->N >= 2 * warps ? launch_packed<1, 2>(p, s) : launch_packed<1, 1>(p, s);
    return a->N >= 4 * warps ? launch_packed<2, 4>(p, s) : a->N >= 2 * warps ? launch_packed<2, 2>(p, s) : launch_packed<2, 1>(p, s);
}

}  // namespace wf
