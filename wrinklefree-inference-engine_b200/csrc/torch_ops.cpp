// The tensor-level ops under torch's dispatcher, natively: argument checks, output tensors and the launches of one call without a pass through Python.
//   sgl_kernel::bitnet_gemv_cpu / bitnet_gemm_cpu / bitnet_quantize_activations_cpu and their aliases (schemas: sgl_kernel/_ops.py; the names are the
//   reference's, docs/research/sglang_optimization_plan.md:59-75): CUDA kernels of those ops;
//   wf_native::linear, wf_native::mlp: the calls behind BitNetLinearNative and bitnet_mlp_forward (several launches each);
//   wf_native::paged_decode_attn: wf_bitnet.ops.paged_decode_attn.
// A call through ctypes spent 20 us of host time on what takes the GPU 6 (one token, 2560 x 2560), and the feed-forward op waited twice for a copy of
// its weight scales to the device; here a call costs about 8 us and the scales travel as kernel parameters.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <pybind11/pybind11.h>
#include <torch/library.h>

#include <map>
#include <mutex>
#include <utility>

#include "wf_bitnet.h"

namespace {

using at::Tensor;

// wf_bitnet._lib.WfError, as the calls through ctypes raise it: callers tell a failed launch from a bad argument by its type
[[noreturn]] void raise_wf_error(const std::string& msg) {
    if (Py_IsInitialized()) {
        pybind11::gil_scoped_acquire gil;
        const pybind11::object type = pybind11::module_::import("wf_bitnet._lib").attr("WfError");
        PyErr_SetString(type.ptr(), msg.c_str());
        throw pybind11::error_already_set();
    }
    TORCH_CHECK(false, msg);
}

void check(int rc) {          // the Python side's mapping of the C status
    if (rc == 0) return;
    const char* msg = wf_last_error();
    TORCH_CHECK_VALUE(rc != -1, msg);
    TORCH_CHECK_NOT_IMPLEMENTED(rc != -2, msg);
    raise_wf_error(msg);
}

void need_gpu(std::initializer_list<const Tensor*> ts) {
    if (!wf_bitnet_available()) raise_wf_error("no compute-capability-10.x CUDA device visible; the BitNet kernels are sm_100a-only and there is no CPU fallback");
    for (const Tensor* t : ts) TORCH_CHECK_VALUE(t->is_cuda(), "expected a CUDA tensor (the B200 BitNet ops have no CPU path)");
}

void* stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }

int code_of(at::ScalarType t) {
    switch (t) {
        case at::kFloat: return 0;
        case at::kBFloat16: return 1;
        case at::kHalf: return 2;
        default: TORCH_CHECK_VALUE(false, "unsupported dtype ", t);
    }
    return -1;
}

// Scratch per device and stream, grown to the largest request.  zeroed: the split-K workspace that kernels leave zero; its contents are only ever
// touched by launches on that stream.  The map itself is never destroyed: tensors outlive the CUDA context at exit otherwise.
Tensor workspace(const Tensor& like, int64_t bytes, bool zeroed) {
    static std::mutex& mu = *new std::mutex;
    static auto& all = *new std::map<std::tuple<int, void*, bool>, Tensor>;
    const auto key = std::make_tuple((int)like.get_device(), stream(), zeroed);
    std::lock_guard<std::mutex> lk(mu);
    Tensor& t = all[key];
    if (!t.defined() || t.numel() < bytes) {
        const auto opt = like.options().dtype(at::kByte);
        bytes = std::max<int64_t>(bytes, 1 << 20);
        t = zeroed ? at::zeros({bytes}, opt) : at::empty({bytes}, opt);
    }
    return t;
}

Tensor bitnet_gemv(const Tensor& packed_weights, const Tensor& activations, double scale) {
    need_gpu({&packed_weights, &activations});
    const c10::cuda::CUDAGuard guard(packed_weights.device());
    TORCH_CHECK_VALUE(packed_weights.dim() == 2, "packed_weights must be 2-D");
    const Tensor p = packed_weights.contiguous(), x = activations.contiguous();
    const int N = (int)p.size(0), K = (int)p.size(1) * 4;
    Tensor y = at::empty({N}, p.options().dtype(at::kFloat));
    const size_t need = wf_bitnet_gemm_workspace_bytes(1, N, K);
    Tensor ws = workspace(p, (int64_t)need, true);
    check(wf_bitnet_gemv((const uint8_t*)p.data_ptr(), (const int8_t*)x.data_ptr(), (float)scale, N, K, (float*)y.data_ptr(), ws.data_ptr(), (size_t)ws.numel(), stream()));
    return y;
}

Tensor bitnet_gemm(const Tensor& packed_weights, const Tensor& activations, double scale) {
    need_gpu({&packed_weights, &activations});
    const c10::cuda::CUDAGuard guard(packed_weights.device());
    TORCH_CHECK_VALUE(packed_weights.dim() == 2 && activations.dim() >= 1, "packed_weights must be 2-D");
    const Tensor p = packed_weights.contiguous(), x = activations.contiguous();
    const int M = (int)x.size(0), N = (int)p.size(0), K = (int)p.size(1) * 4;
    Tensor y = at::empty({M, N}, p.options().dtype(at::kFloat));
    const size_t need = wf_bitnet_gemm_workspace_bytes(M, N, K);
    Tensor ws;
    if (need) ws = workspace(p, (int64_t)need, true);
    check(wf_bitnet_gemm((const uint8_t*)p.data_ptr(), (const int8_t*)x.data_ptr(), (float)scale, M, N, K, (float*)y.data_ptr(), need ? ws.data_ptr() : nullptr,
                         need ? (size_t)ws.numel() : 0, stream()));
    return y;
}

struct Quant { Tensor q, scale, rowsum; };

// x2: [M, K] contiguous
Quant quantize(const Tensor& x2, bool per_token) {
    const int M = (int)x2.size(0), K = (int)x2.size(1);
    const int dt = code_of(x2.scalar_type());
    Quant o;
    o.q = at::empty({M, K}, x2.options().dtype(at::kChar));
    o.scale = at::empty({per_token ? M : 1}, x2.options().dtype(at::kFloat));
    o.rowsum = at::empty({std::max(M, 1) + 1}, x2.options().dtype(at::kInt));       // the last entry: the per-tensor absmax cell
    check(wf_act_quant_i8(x2.data_ptr(), dt, M, K, K, per_token ? 1 : 0, (int8_t*)o.q.data_ptr(), (float*)o.scale.data_ptr(), (int32_t*)o.rowsum.data_ptr(),
                          (int32_t*)o.rowsum.data_ptr() + std::max(M, 1), stream()));
    return o;
}

std::tuple<Tensor, Tensor> bitnet_quantize_activations(const Tensor& activations) {
    need_gpu({&activations});
    const c10::cuda::CUDAGuard guard(activations.device());
    const Tensor x2 = (activations.dim() == 1 ? activations.reshape({1, -1}) : activations.reshape({-1, activations.size(-1)})).contiguous();
    Quant o = quantize(x2, false);
    return {o.q.reshape(activations.sizes()), o.scale};
}

void fill_linear(wf_linear_args& a, const Tensor& w, bool tile, int N, int K, const Quant& x, Tensor& out, int out_dtype, Tensor& ws) {
    memset(&a, 0, sizeof a);
    const int M = (int)x.q.size(0);
    a.w = (const uint8_t*)w.data_ptr(); a.w_layout = tile ? 1 : 0; a.N = N; a.K = K;
    a.q = (const int8_t*)x.q.data_ptr(); a.M = M; a.ldq = K;
    a.rowsum = (const int32_t*)x.rowsum.data_ptr();
    a.act_scale = (const float*)x.scale.data_ptr(); a.act_scale_per_token = x.scale.numel() > 1 || M == 1 ? 1 : 0;
    a.nseg = 1; a.seg_end[0] = N;
    a.host_scale = 1.f;
    a.out_mode = 3; a.out_dtype = out_dtype;
    a.out = out.data_ptr(); a.ldo = (int)out.size(1);
    size_t need = M > 8 ? wf_bitnet_gemm_workspace_bytes(M, N, K) : wf_linear_workspace_bytes(M, N, K);
    if (need) {
        need += 4 * (size_t)((N + 15) / 16) + 256;
        ws = workspace(w, (int64_t)need, true);
        a.workspace = ws.data_ptr(); a.workspace_bytes = (size_t)ws.numel();
    }
}

// y [M, N] float = w_scale * W x, x [M, K] quantised with one scale for all of it; w: tile (tile = true) or packed layout
Tensor linear(const Tensor& x, const Tensor& w, bool tile, int64_t N, int64_t K, const Tensor& w_scale) {
    need_gpu({&x, &w, &w_scale});
    const c10::cuda::CUDAGuard guard(w.device());
    TORCH_CHECK_VALUE(x.dim() == 2 && x.size(1) == K, "activations.shape[-1] != in_features");
    const Tensor x2 = x.contiguous(), wc = w.contiguous(), sc = w_scale.contiguous();
    TORCH_CHECK_VALUE(sc.scalar_type() == at::kFloat && sc.numel() >= 1, "w_scale must be float32");
    Quant q = quantize(x2, false);
    Tensor out = at::empty({x2.size(0), N}, x2.options().dtype(at::kFloat)), ws;
    wf_linear_args a;
    fill_linear(a, wc, tile, (int)N, (int)K, q, out, 0, ws);
    a.w_scale = (const float*)sc.data_ptr();
    check(wf_ternary_linear(&a, stream()));
    return out;
}

// quantise -> [gate | up] with relu(gate)^2 * up -> norm + quantise -> down; x [M, K], y bf16 [M, down rows]
Tensor mlp(const Tensor& x, const Tensor& gate_up_tile, int64_t N2, const Tensor& down_w, double gate_scale, double up_scale, double down_scale, const Tensor& norm, double eps) {
    need_gpu({&x, &gate_up_tile, &down_w, &norm});
    const c10::cuda::CUDAGuard guard(x.device());
    const Tensor x2 = x.contiguous(), dw = down_w.contiguous(), g = norm.contiguous();
    TORCH_CHECK_VALUE(dw.dim() == 2, "packed weights must be 2-D");
    const int M = (int)x2.size(0), K = (int)x2.size(1), F = (int)N2 / 2, D = (int)dw.size(0);
    TORCH_CHECK_VALUE(dw.size(1) * 4 == F, "activations.shape[-1] != in_features");
    TORCH_CHECK_VALUE(g.scalar_type() == at::kBFloat16 && g.numel() >= F, "ffn_sub_norm must have one weight per feed-forward row");
    Quant q = quantize(x2, true);
    const auto bf = x2.options().dtype(at::kBFloat16);
    Tensor h = at::empty({M, F}, bf), ws, ws2;
    wf_linear_args a;
    fill_linear(a, gate_up_tile, true, (int)N2, K, q, h, 1, ws);
    const float gu[2] = {(float)gate_scale, (float)up_scale};
    a.nseg = 2; a.epi_flags = 2;
    check(wf_ternary_linear_scales(&a, gu, stream()));
    Quant q2;
    q2.q = at::empty({M, F}, x2.options().dtype(at::kChar));
    q2.scale = at::empty({M}, x2.options().dtype(at::kFloat));
    q2.rowsum = at::empty({M}, x2.options().dtype(at::kInt));
    check(wf_rmsnorm_quant(h.data_ptr(), g.data_ptr(), (float)eps, M, F, nullptr, (int8_t*)q2.q.data_ptr(), (float*)q2.scale.data_ptr(), (int32_t*)q2.rowsum.data_ptr(), stream()));
    Tensor y = at::empty({M, D}, bf);
    fill_linear(a, dw, false, D, F, q2, y, 1, ws2);
    const float ds[1] = {(float)down_scale};
    check(wf_ternary_linear_scales(&a, ds, stream()));
    return y;
}

Tensor paged_decode_attn(const Tensor& q, const Tensor& pool, int64_t max_pages, int64_t layers, int64_t kv_heads, int64_t page_size, int64_t head_dim, int64_t kv_dtype,
                         int64_t layer, const Tensor& block_table, const Tensor& seq_lens, double scale, at::ScalarType out_dtype) {
    need_gpu({&q, &block_table, &seq_lens});
    const c10::cuda::CUDAGuard guard(q.device());
    TORCH_CHECK_VALUE(q.dim() == 3 && block_table.dim() == 2, "q must be [B, H, D] and block_table [B, blocks]");
    const Tensor qc = q.contiguous();
    const int B = (int)q.size(0), H = (int)q.size(1), D = (int)q.size(2), blocks = (int)block_table.size(1);
    Tensor out = at::empty({B, H, D}, q.options().dtype(out_dtype));
    wf_kv_layout kv;
    memset(&kv, 0, sizeof kv);
    kv.pool = pool.data_ptr();
    kv.max_pages = (int)max_pages; kv.layers = (int)layers; kv.kv_heads = (int)kv_heads; kv.page_size = (int)page_size; kv.head_dim = (int)head_dim; kv.dtype = (int)kv_dtype;
    Tensor ws = workspace(q, (int64_t)wf_attn_workspace_bytes(B, H, D, blocks * (int)page_size), false);
    check(wf_paged_decode_attn(qc.data_ptr(), &kv, (int)layer, (const int32_t*)block_table.data_ptr(), blocks, (const int32_t*)seq_lens.data_ptr(), B, H, (float)scale, out.data_ptr(),
                               code_of(out_dtype), ws.data_ptr(), (size_t)ws.numel(), stream()));
    return out;
}

}  // namespace

TORCH_LIBRARY(wf_native, m) {
    m.def("linear(Tensor x, Tensor w, bool tile, int N, int K, Tensor w_scale) -> Tensor");
    m.def("mlp(Tensor x, Tensor gate_up_tile, int N2, Tensor down_w, float gate_scale, float up_scale, float down_scale, Tensor norm, float eps) -> Tensor");
    m.def("paged_decode_attn(Tensor q, Tensor pool, int max_pages, int layers, int kv_heads, int page_size, int head_dim, int kv_dtype, int layer, Tensor block_table, "
          "Tensor seq_lens, float scale, ScalarType out_dtype) -> Tensor");
}
// CPU: the same functions, for their errors (a missing GPU, a tensor that is not on it).  Autograd: passed through, so that the outputs are plain tensors
// whatever the inputs require, as behind the calls through ctypes.
#define WF_NATIVE_IMPL(key)                    \
    TORCH_LIBRARY_IMPL(wf_native, key, m) {    \
        m.impl("linear", linear);              \
        m.impl("mlp", mlp);                    \
        m.impl("paged_decode_attn", paged_decode_attn); \
    }
WF_NATIVE_IMPL(CUDA)
WF_NATIVE_IMPL(CPU)
TORCH_LIBRARY_IMPL(wf_native, Autograd, m) {
    m.impl("linear", torch::CppFunction::makeFallthrough());
    m.impl("mlp", torch::CppFunction::makeFallthrough());
    m.impl("paged_decode_attn", torch::CppFunction::makeFallthrough());
}
TORCH_LIBRARY_IMPL(sgl_kernel, CUDA, m) {
    m.impl("bitnet_gemv_cpu", bitnet_gemv);
    m.impl("bitnet_gemv", bitnet_gemv);
    m.impl("bitnet_gemm_cpu", bitnet_gemm);
    m.impl("bitnet_gemm", bitnet_gemm);
    m.impl("bitnet_quantize_activations_cpu", bitnet_quantize_activations);
    m.impl("bitnet_quantize_activations", bitnet_quantize_activations);
}
