// The calls whose kernels take a few microseconds, from tensors to launch in C++: output allocation, argument struct and the
// C ABI's entry point in one step.  The Python forms of the same calls (turbopi_b200/ops.py and the modules) stay the
// reference for what is accepted: whatever a function here does not recognise as its plain case (a CPU tensor, another
// device, a dtype or a stride that needs a conversion) returns None and takes the Python form, which converts or refuses.
// A non-zero status of the C ABI comes back as an int.  Time to issue a call (us, Python form -> here): one-token INT4 linear
// 13.1 -> 7.1, 50-token MLP 31.2 -> 17.4, attention 18.2 -> 8.2, W4A4 linear 21.7 -> 12.4, FP8 quantiser + W4A8 launcher 24.4 -> 18.1.
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <optional>

#include "turbopi_b200.h"

namespace {

struct Entries {
    decltype(&tpb200_w4_gemm) w4_gemm;
    decltype(&tpb200_w4a16_gemv) w4a16_gemv;
    decltype(&tpb200_w4a16_gemm) w4a16_gemm;
    decltype(&tpb200_attention) attention;
    decltype(&quantizeActivationToFP8) quantize_fp8;
    decltype(&tpb200_last_error) last_error;
    decltype(&tpb200_nvfp4_tiled_a_bytes) tiled_a_bytes;
    decltype(&tpb200_nvfp4_quantize_act_tiled) quantize_act_tiled;
    decltype(&tpb200_nvfp4_gemm_ex) gemm_ex;
} g;

using OptTensor = std::optional<at::Tensor>;

// the entry points of the library that turbopi_b200/_lib.py has loaded, in the order of Entries
void bind(const std::vector<uint64_t>& a) {
    TORCH_CHECK(a.size() * sizeof(void*) == sizeof(Entries), "calls.bind: wrong number of entry points");
    memcpy(&g, a.data(), sizeof(Entries));
}

int code_of(at::ScalarType t) {
    return t == at::kBFloat16 ? TPB200_BF16 : t == at::kHalf ? TPB200_F16 : t == at::kFloat ? TPB200_F32 : -1;
}
at::ScalarType type_of(int code) { return code == TPB200_BF16 ? at::kBFloat16 : code == TPB200_F16 ? at::kHalf : at::kFloat; }

void* ptr(const OptTensor& t) { return t.has_value() ? t->data_ptr() : nullptr; }
bool on(const at::Tensor& t, int dev) { return t.is_cuda() && t.get_device() == dev; }
bool on(const OptTensor& t, int dev) { return !t.has_value() || on(*t, dev); }

// the device of `t` if it is the current one, else -1
int here(const at::Tensor& t) {
    if (!t.is_cuda()) return -1;
    const int d = t.get_device();
    return d == c10::cuda::current_device() ? d : -1;
}
tpb200_stream_t stream_of(int dev) { return reinterpret_cast<tpb200_stream_t>(c10::cuda::getCurrentCUDAStream(dev).stream()); }

template <class F>
int launch(F&& f) {                                       // without the interpreter lock, as through ctypes
    py::gil_scoped_release nogil;
    return f();
}

py::object done(int status, const at::Tensor& out) { return status == 0 ? py::cast(out) : py::int_(status); }

int w4(const at::Tensor& x, int64_t M, int64_t K, const at::Tensor& w, int64_t N, int format, const OptTensor& w_scales,
       const OptTensor& w_zeros, double alpha, double beta, const OptTensor& bias, int activation, bool gated, const at::Tensor& out,
       int flags, int dev) {
    tpb200_w4_gemm_args a = {};
    a.x = x.data_ptr();
    a.ldx = static_cast<int>(M > 1 ? x.stride(0) : K);
    a.format = format;
    a.w = w.data_ptr();
    a.w_pitch = format == TPB200_W4_NVFP4_ROWMAJOR ? static_cast<int>(w.stride(0)) : 0;
    a.w_scales = ptr(w_scales);
    a.w_zeros = ptr(w_zeros);
    a.alpha = static_cast<float>(alpha);
    a.beta = static_cast<float>(beta);
    a.bias = ptr(bias);
    a.bias_dtype = bias.has_value() ? code_of(bias->scalar_type()) : TPB200_F32;
    a.activation = activation;
    a.gated = gated;
    a.out = out.data_ptr();
    a.out_dtype = code_of(out.scalar_type());
    a.ldo = static_cast<int>(M > 1 ? out.stride(0) : out.size(1));
    a.M = static_cast<int>(M);
    a.N = static_cast<int>(N);
    a.K = static_cast<int>(K);
    a.flags = flags;
    const tpb200_stream_t s = stream_of(dev);
    return launch([&] { return g.w4_gemm(&a, s); });
}

// ops.w4_gemm
py::object w4_gemm(const at::Tensor& x, const at::Tensor& w, int64_t N, int format, const OptTensor& w_scales, const OptTensor& w_zeros,
                   double alpha, double beta, const OptTensor& bias, int activation, bool gated, const OptTensor& out, int out_code,
                   int flags) {
    const int dev = here(x);
    if (dev < 0 || x.dim() != 2 || x.scalar_type() != at::kBFloat16 || x.stride(1) != 1 || !on(w, dev) || !on(w_scales, dev) ||
        !on(w_zeros, dev) || !on(bias, dev) || !on(out, dev) || (bias.has_value() && code_of(bias->scalar_type()) < 0) ||
        (out.has_value() ? out->dim() != 2 || code_of(out->scalar_type()) < 0 : out_code < 0)) {
        return py::none();
    }
    const int64_t M = x.size(0), K = x.size(1);
    const at::Tensor y = out.has_value() ? *out : at::empty({M, gated ? N / 2 : N}, x.options().dtype(type_of(out_code)));
    return done(w4(x, M, K, w, N, format, w_scales, w_zeros, alpha, beta, bias, activation, gated, y, flags, dev), y);
}

// NVFP4PackedMLP's two launches on tiled images: gate_up with act(gate) * up in its epilogue, down on its bf16 result
py::object mlp(const at::Tensor& x, const at::Tensor& gate_up, const at::Tensor& down, const OptTensor& bias, int64_t I, int64_t H,
               double alpha_gu, double alpha_d, int activation, int flags_first, int flags_second) {
    const int dev = here(x);
    if (dev < 0 || x.dim() != 2 || x.scalar_type() != at::kBFloat16 || !x.is_contiguous() || x.size(1) != H || !on(gate_up, dev) ||
        !on(down, dev) || !on(bias, dev)) {
        return py::none();
    }
    const int64_t M = x.size(0);
    const at::Tensor h = at::empty({M, I}, x.options()), y = at::empty({M, H}, x.options());
    const int st = w4(x, M, H, gate_up, 2 * I, TPB200_W4_NVFP4_TILED, {}, {}, alpha_gu, 0.0, {}, activation, true, h, flags_first, dev);
    if (st != 0) return py::int_(st);
    return done(w4(h, M, I, down, H, TPB200_W4_NVFP4_TILED, {}, {}, alpha_d, 0.0, bias, TPB200_ACT_NONE, false, y, flags_second, dev), y);
}

// W4A16Linear.forward on its buffers
py::object w4a16_linear(const at::Tensor& input, const at::Tensor& packed, const at::Tensor& scales, const OptTensor& bias, int64_t N,
                        int flags) {
    const int dev = here(input);
    const int code = code_of(input.scalar_type());
    if (dev < 0 || code < 0 || input.dim() < 1 || !input.is_contiguous() || !on(packed, dev) || !on(scales, dev) || !on(bias, dev) ||
        packed.dim() != 3 || packed.size(0) == 0 || input.size(-1) != packed.size(0) * 32 ||
        (bias.has_value() && (code_of(bias->scalar_type()) < 0 || !bias->is_contiguous())) || scales.scalar_type() != at::kHalf) {
        return py::none();
    }
    const int64_t K = input.size(-1), T = input.numel() / K;
    if (T < 1 || (T > 16 && (K % 128 != 0 || N % 8 != 0))) return py::none();
    std::vector<int64_t> shape(input.sizes().begin(), input.sizes().end());
    shape.back() = N;
    const at::Tensor y = at::empty(shape, input.options());
    const at::Tensor x = T <= 16 || code == TPB200_BF16 ? input : input.to(at::kBFloat16);
    const void *xp = x.data_ptr(), *wp = packed.data_ptr(), *sp = scales.data_ptr(), *bp = ptr(bias);
    void* yp = y.data_ptr();
    const int bias_code = bias.has_value() ? code_of(bias->scalar_type()) : TPB200_F32;
    const tpb200_stream_t s = stream_of(dev);
    const int m = static_cast<int>(T), n = static_cast<int>(N), k = static_cast<int>(K);
    const int st = launch([&] {
        return T <= 16 ? g.w4a16_gemv(xp, code, wp, sp, TPB200_SCALE_F16, bp, bias_code, yp, code, m, n, k, 32, TPB200_INT4_KBLOCK, 0, s)
                       : g.w4a16_gemm(xp, wp, sp, nullptr, bp, bias_code, yp, code, m, n, k, n, TPB200_INT4_KBLOCK, 1.0f, 0.0f, flags, s);
    });
    return done(st, y);
}

// ops.attention without a fused quantiser
py::object attention(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& out, double scale,
                     const OptTensor& key_bias, const at::Tensor& workspace, int flags) {
    const int dev = here(q);
    const int64_t nd = q.dim();
    if (dev < 0 || (nd != 2 && nd != 4) || !on(workspace, dev) || !on(key_bias, dev)) return py::none();
    for (const at::Tensor* t : {&q, &k, &v, &out}) {
        if (!on(*t, dev) || t->dim() != nd || t->scalar_type() != at::kBFloat16 || t->stride(-1) != 1) return py::none();
    }
    const int64_t A = nd == 4 ? q.size(0) : 1, B = nd == 4 ? q.size(1) : 1, R = q.size(-2), D = q.size(-1), S = k.size(-2);
    if (out.sizes() != q.sizes() || v.sizes() != k.sizes() || k.size(-1) != D || (nd == 4 && (k.size(0) != A || k.size(1) != B)) ||
        (key_bias.has_value() &&
         (key_bias->scalar_type() != at::kBFloat16 || key_bias->numel() < S || !key_bias->is_contiguous()))) {
        return py::none();
    }
    tpb200_attention_args a = {};
    a.q = q.data_ptr();
    a.k = k.data_ptr();
    a.v = v.data_ptr();
    a.out = out.data_ptr();
    a.key_bias = ptr(key_bias);
    a.n_rows = static_cast<int>(R);
    a.n_keys = static_cast<int>(S);
    a.head_dim = static_cast<int>(D);
    a.ldq = static_cast<int>(q.stride(-2));
    a.ldk = static_cast<int>(k.stride(-2));
    a.ldv = static_cast<int>(v.stride(-2));
    a.ldo = static_cast<int>(out.stride(-2));
    a.groups_outer = static_cast<int>(A);
    a.groups_inner = static_cast<int>(B);
    if (nd == 4) {
        for (int i = 0; i < 2; ++i) {
            a.q_stride[i] = q.stride(i);
            a.k_stride[i] = k.stride(i);
            a.v_stride[i] = v.stride(i);
            a.o_stride[i] = out.stride(i);
        }
    }
    a.scale = static_cast<float>(scale);
    a.workspace = workspace.data_ptr();
    a.workspace_bytes = static_cast<size_t>(workspace.numel());
    a.flags = flags;
    a.quant_rows_per_token = 1;
    const tpb200_stream_t s = stream_of(dev);
    const int st = launch([&] { return g.attention(&a, s); });
    if (st != 0) return py::int_(st);
    return py::cast(nd == 4 ? out : out.unsqueeze(0).unsqueeze(0));
}

// ops.quantize_activation_to_fp8
py::object quantize_fp8(const at::Tensor& x) {
    const int dev = here(x);
    if (dev < 0 || x.dim() != 2 || x.scalar_type() != at::kBFloat16 || !x.is_contiguous()) return py::none();
    const int64_t M = x.size(0), K = x.size(1);
    const auto bytes = x.options().dtype(at::kByte);
    const at::Tensor out = at::empty({M, K}, bytes), scales = at::empty({M, K / 16}, bytes);
    const void* xp = x.data_ptr();
    void *op = out.data_ptr(), *sp = scales.data_ptr();
    const tpb200_stream_t s = stream_of(dev);
    const int st = launch([&] {
        g.quantize_fp8(xp, op, sp, static_cast<int>(M), static_cast<int>(K), s);
        return g.last_error();
    });
    return st == 0 ? py::object(py::make_tuple(out, scales)) : py::int_(st);
}

// ops.nvfp4_linear_tiled on row-major weights
py::object nvfp4_linear(const at::Tensor& x, const at::Tensor& w, int64_t N, double alpha, const OptTensor& bias, int activation,
                        int out_code, const at::Tensor& w_sf) {
    const int dev = here(x);
    const int code = code_of(x.scalar_type());
    if (dev < 0 || code < 0 || out_code < 0 || x.dim() != 2 || !x.is_contiguous() || !on(w, dev) || !on(w_sf, dev) || !on(bias, dev) || w.dim() != 2 ||
        (bias.has_value() && (bias->scalar_type() != at::kFloat || !bias->is_contiguous()))) {
        return py::none();
    }
    const int M = static_cast<int>(x.size(0)), K = static_cast<int>(x.size(1));
    const at::Tensor a = at::empty({static_cast<int64_t>(g.tiled_a_bytes(M, K, 1))}, x.options().dtype(at::kByte));
    const at::Tensor y = at::empty({M, N}, x.options().dtype(type_of(out_code)));
    tpb200_nvfp4_gemm_args p = {};
    p.a_packed = a.data_ptr();
    p.a_pieces = 1;
    p.b_packed = w.data_ptr();
    p.b_pitch = static_cast<int>(w.stride(0));
    p.b_sf = w_sf.data_ptr();
    p.alpha = static_cast<float>(alpha);
    p.bias = static_cast<decltype(p.bias)>(ptr(bias));
    p.activation = activation;
    p.out = y.data_ptr();
    p.out_dtype = out_code;
    p.ldo = static_cast<int>(N);
    p.M = M;
    p.N = static_cast<int>(N);
    p.K = K;
    p.layout = TPB200_OPERANDS_TILED_A;
    // the quantiser is a plain launch, so what wrote the weights is complete when it starts: their blocks travel while it runs
    p.flags = TPB200_FLAG_PDL;
    const void* xp = x.data_ptr();
    void* ap = a.data_ptr();
    const tpb200_stream_t s = stream_of(dev);
    const int st = launch([&] {
        const int q = g.quantize_act_tiled(xp, code, K, ap, M, K, s);
        return q != 0 ? q : g.gemm_ex(&p, s);
    });
    return done(st, y);
}

}  // namespace

PYBIND11_MODULE(_calls, m) {
    m.def("bind", &bind);
    m.def("w4_gemm", &w4_gemm);
    m.def("mlp", &mlp);
    m.def("w4a16_linear", &w4a16_linear);
    m.def("attention", &attention);
    m.def("quantize_fp8", &quantize_fp8);
    m.def("nvfp4_linear", &nvfp4_linear);
}
