// Host side of the calls whose device time is a few microseconds: argument checks, output allocation and the parameter block
// of one C ABI call, on torch tensors, in C++.  In Python the same steps cost 25-30 us per call (a ctypes structure of some
// thirty fields, as many tensor attributes, a device context, a stream object), which is what a decode step of a small batch
// or a short prompt then waited for.  The library's functions are handed over as addresses (bind), so that this module and
// the ctypes binding drive the same loaded library; checks and messages are those of the Python wrappers (ops.py).
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/types.h>

#include "../../include/vortex_b200.h"

namespace py = pybind11;
using at::Tensor;
using Opt = std::optional<Tensor>;

namespace {

decltype(&vtx_decode_layer) p_decode_layer;
decltype(&vtx_fused_fir_fwd) p_fused_fir_fwd;
decltype(&vtx_fused_iir_fwd) p_fused_iir_fwd;
decltype(&vtx_fused_iir_scratch_bytes) p_fused_iir_scratch_bytes;
decltype(&vtx_last_error) p_last_error;

// The entry points run without the GIL (see the module definition); an error is made with it.
[[noreturn]] void raise(PyObject* type, const std::string& msg) {
    const py::gil_scoped_acquire gil;
    PyErr_SetString(type, msg.c_str());
    throw py::error_already_set();
}
void check(int rc) {
    if (rc == 0) return;
    char buf[512];
    p_last_error(buf, sizeof buf);
    PyObject* type = rc == VTX_ERR_BAD_ARG || rc == VTX_ERR_ALIGNMENT ? PyExc_ValueError
                     : rc == VTX_ERR_UNSUPPORTED ? PyExc_NotImplementedError : PyExc_RuntimeError;
    raise(type, "vortex_b200: " + std::string(buf) + " (status " + std::to_string(rc) + ")");
}
void need_cuda(const Tensor& t) {
    if (!t.is_cuda()) raise(PyExc_RuntimeError, "vortex_b200 kernels need CUDA tensors (there is no CPU path)");
}
void need_cuda(const Opt& t) { if (t) need_cuda(*t); }
bool known(at::ScalarType t) { return t == at::kFloat || t == at::kBFloat16 || t == at::kHalf; }
int64_t code(const Tensor& t) {
    switch (t.scalar_type()) {
        case at::kFloat: return VTX_F32;
        case at::kBFloat16: return VTX_BF16;
        case at::kHalf: return VTX_F16;
        default: raise(PyExc_TypeError, std::string("vortex_b200: unsupported dtype ") + c10::toString(t.scalar_type()));
    }
}
// parameters are read with their own dtype; dense and beside the activations
Tensor param(const Tensor& t, const Tensor& like) {
    if (t.device() != like.device()) raise(PyExc_RuntimeError, "vortex_b200: parameter on a different device than the activations");
    Tensor r = t;
    if (!known(r.scalar_type())) r = r.detach().to(at::kFloat);
    return r.is_contiguous() ? r : r.detach().contiguous();
}
Opt param(const Opt& t, const Tensor& like) { return t ? Opt(param(*t, like)) : Opt(); }
const void* ptr(const Tensor& t) { return t.const_data_ptr(); }
const void* ptr(const Opt& t) { return t ? t->const_data_ptr() : nullptr; }
void* out(const Tensor& t) { return t.mutable_data_ptr(); }
int64_t code_or_0(const Opt& t) { return t ? code(*t) : 0; }
Tensor empty(at::IntArrayRef size, const Tensor& like, at::ScalarType dtype) { return at::empty(size, at::TensorOptions().device(like.device()).dtype(dtype)); }
void* stream_of(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
std::string str(const Tensor& t) {
    std::string s = "(";
    for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
    return s + (t.dim() == 1 ? ",)" : ")");
}

const Tensor& have(const Opt& t, const char* use) {
    if (!t) raise(PyExc_AttributeError, std::string("'NoneType' object has no attribute '") + use + "'");
    return *t;
}

// fp32 [G, S] parameter block; the tensors stay alive until the call has been issued
struct Modal {
    vtx_modal_params m{};
    Tensor lp, res;
    Opt th, ri;
    Modal(const Tensor& log_poles, const Tensor& residues, const Tensor& like, const Opt& theta, const Opt& res_im) {
        auto f32 = [&](const Tensor& t) {
            if (t.scalar_type() == at::kFloat && t.device() == like.device() && t.is_contiguous()) return t;
            return t.detach().to(like.device(), at::kFloat).contiguous();
        };
        res = f32(residues);
        if (res.dim() != 2) raise(PyExc_ValueError, "residues must be [G, S]");
        m.G = res.size(0); m.S = res.size(1);
        auto gs = [&](const Tensor& t) {
            Tensor r = f32(t);
            return r.numel() == m.G * m.S ? r : r.reshape({m.G, m.S});      // (raises as reshape does)
        };
        lp = gs(log_poles);
        if (theta) th = gs(*theta);
        if (res_im) ri = gs(*res_im);
        m.log_poles = ptr(lp); m.theta = ptr(th); m.res_re = ptr(res); m.res_im = ptr(ri);
    }
};

std::tuple<Tensor, Tensor, Tensor> decode_layer(Tensor u, const Tensor& w3_, const Opt& b3_, const Tensor& fir_state, int64_t D, const Opt& h_,
                                                const Opt& inner_state, const Opt& bias_, bool flip_filter, bool gated_bias, const Opt& log_poles,
                                                const Opt& residues, const Opt& iir_state, const Opt& theta, const Opt& res_im, int64_t layout,
                                                int64_t num_heads, bool flip) {
    need_cuda(u); need_cuda(w3_); need_cuda(fir_state);
    u = u.contiguous();
    if (u.dim() != 2) raise(PyExc_ValueError, "u must be [B, 3D]");
    const int64_t B = u.size(0), C3 = u.size(1);
    if (C3 != 3 * D) raise(PyExc_ValueError, "expected " + std::to_string(3 * D) + " packed channels, got " + std::to_string(C3));
    const Tensor w3 = param(w3_, u);
    const int64_t K3 = C3 ? w3.numel() / C3 : 0;
    if (K3 * C3 != w3.numel()) raise(PyExc_RuntimeError, "shape '[" + std::to_string(C3) + ", -1]' is invalid for input of size " + std::to_string(w3.numel()));
    const Opt b3 = param(b3_, u), bias = param(bias_, u);
    const Tensor fs = fir_state.contiguous();
    if (fs.size(-1) != K3 - 1) raise(PyExc_NotImplementedError, "decode_layer needs a full featurizer cache (prompt of at least K3-1 tokens)");
    vtx_decode_layer_params p{};
    p.io_dtype = code(u);
    Tensor fs_out = empty({B, C3, K3 - 1}, u, at::kFloat), y = empty({B, D}, u, u.scalar_type()), state;
    p.u = ptr(u); p.w3 = ptr(w3); p.w3_dtype = code(w3); p.b3 = ptr(b3); p.b3_dtype = code_or_0(b3);
    p.fir_state_in = ptr(fs); p.fir_state_dtype = code(fs); p.fir_state_out = static_cast<float*>(out(fs_out));
    p.bias = ptr(bias); p.bias_dtype = code_or_0(bias); p.y = out(y);
    p.B = B; p.D = D; p.K3 = K3; p.layout = layout; p.num_heads = num_heads; p.flip_x1x2 = flip; p.flip_filter = flip_filter;
    std::optional<Modal> modal;
    Tensor h, in;
    if (h_) {
        h = param(*h_, u);
        p.G = h.size(0);
        p.K = p.G ? h.numel() / p.G : 0;
        in = have(inner_state, "contiguous").contiguous();
        if (in.size(-1) != p.K - 1) raise(PyExc_NotImplementedError, "decode_layer needs a full inner cache (prompt of at least K-1 tokens)");
        state = empty({B, D, p.K - 1}, u, at::kFloat);
        p.h = ptr(h); p.h_dtype = code(h);
        p.inner_state_in = ptr(in); p.inner_state_dtype = code(in); p.inner_state_out = static_cast<float*>(out(state));
        p.bias_mode = bias ? (gated_bias ? VTX_BIAS_GATED : VTX_BIAS_ADD) : VTX_BIAS_NONE;
    } else {
        have(residues, "detach");
        modal.emplace(have(log_poles, "detach"), *residues, u, theta, res_im);
        in = have(iir_state, "contiguous").contiguous();
        if (in.scalar_type() != at::kFloat) in = in.to(at::kFloat);
        state = at::empty_like(in);
        p.modal = modal->m; p.K = 0; p.G = modal->m.G;
        p.iir_state_in = static_cast<const float*>(ptr(in)); p.iir_state_out = static_cast<float*>(out(state));
    }
    const c10::cuda::CUDAGuard on(u.device());
    check(p_decode_layer(&p, stream_of(u)));
    return {y, fs_out, state};
}

std::tuple<Tensor, Opt, Opt> fused_fir_fwd(Tensor u, const Tensor& w3_, const Opt& b3_, const Tensor& h_, const Opt& bias_, int64_t D, int64_t taps,
                                           int64_t bias_mode, int64_t layout, int64_t num_heads, bool flip, bool want_state, int64_t hist_rows) {
    need_cuda(u); need_cuda(w3_); need_cuda(b3_); need_cuda(h_); need_cuda(bias_);
    if (u.dim() != 3) raise(PyExc_ValueError, "u must be [B, L, 3D]");
    if (u.stride(2) != 1) {
        if (hist_rows) raise(PyExc_ValueError, "hist_rows needs u with unit channel stride (a view into the buffer that holds the history)");
        u = u.contiguous();
    }
    const int64_t B = u.size(0), L = u.size(1), C3 = u.size(2);
    if (C3 != 3 * D) raise(PyExc_ValueError, "expected " + std::to_string(3 * D) + " packed channels, got " + std::to_string(C3));
    const Tensor w3 = param(w3_, u), h = param(h_, u);
    const int64_t K3 = C3 ? w3.numel() / C3 : 0, G = h.size(0), K = G ? h.numel() / G : 0;
    if (K3 * C3 != w3.numel()) raise(PyExc_RuntimeError, "shape '[" + std::to_string(C3) + ", -1]' is invalid for input of size " + std::to_string(w3.numel()));
    const Opt b3 = param(b3_, u), bias = param(bias_, u);
    if (hist_rows && u.storage_offset() < hist_rows * u.stride(1))
        raise(PyExc_ValueError, "hist_rows=" + std::to_string(hist_rows) + ": u starts " +
                                    std::to_string(u.storage_offset() / std::max<int64_t>(u.stride(1), 1)) + " rows into its storage");
    vtx_fused_fir_params p{};
    p.io_dtype = code(u);
    Tensor y = empty({B, L, D}, u, u.scalar_type());
    Opt fs, ist;
    if (want_state) {
        fs = empty({B, C3, hist_rows ? K3 - 1 : std::min(L, K3 - 1)}, u, u.scalar_type());
        ist = empty({B, D, hist_rows ? K - 1 : std::min(L, K - 1)}, u, u.scalar_type());
        p.fir_state = fs->numel() ? out(*fs) : nullptr;
        p.inner_state = ist->numel() ? out(*ist) : nullptr;
    }
    p.u = ptr(u); p.u_stride_b = u.stride(0); p.u_stride_l = u.stride(1);
    p.w3 = ptr(w3); p.w3_dtype = code(w3); p.b3 = ptr(b3); p.b3_dtype = code_or_0(b3);
    p.h = ptr(h); p.h_dtype = code(h); p.bias = ptr(bias); p.bias_dtype = code_or_0(bias);
    p.y = out(y); p.y_stride_b = L * D; p.y_stride_l = D;
    p.B = B; p.L = L; p.D = D; p.G = G; p.K3 = K3; p.K = K;
    p.layout = layout; p.num_heads = num_heads; p.flip_x1x2 = flip;
    p.taps = taps; p.bias_mode = bias ? bias_mode : VTX_BIAS_NONE; p.u_hist_rows = hist_rows;
    const c10::cuda::CUDAGuard on(u.device());
    check(p_fused_fir_fwd(&p, stream_of(u)));
    return {y, fs, ist};
}

std::tuple<Tensor, Opt> fused_iir_fwd(Tensor u, const Tensor& w3_, const Tensor& log_poles, const Tensor& residues, const Opt& bias_, int64_t D,
                                      int64_t layout, int64_t num_heads, bool flip, const Opt& theta, const Opt& res_im, bool want_state,
                                      const Opt& b3_, Opt state_in, Opt fir_state_in, int64_t hist_rows, const Opt& out_) {
    need_cuda(u); need_cuda(w3_); need_cuda(residues); need_cuda(bias_); need_cuda(b3_); need_cuda(state_in); need_cuda(fir_state_in);
    if (u.dim() != 3) raise(PyExc_ValueError, "u must be [B, L, 3D]");
    if (u.stride(2) != 1) {
        if (hist_rows) raise(PyExc_ValueError, "hist_rows needs u with unit channel stride (a view into the buffer that holds the history)");
        u = u.contiguous();
    }
    if (hist_rows) {
        if (hist_rows < 2 || fir_state_in) raise(PyExc_ValueError, "hist_rows must be >= 2 and excludes fir_state_in");
        if (u.storage_offset() < hist_rows * u.stride(1))
            raise(PyExc_ValueError, "hist_rows=" + std::to_string(hist_rows) + ": u starts " +
                                        std::to_string(u.storage_offset() / std::max<int64_t>(u.stride(1), 1)) + " rows into its storage");
    }
    const int64_t B = u.size(0), L = u.size(1), C3 = u.size(2);
    if (C3 != 3 * D) raise(PyExc_ValueError, "expected " + std::to_string(3 * D) + " packed channels, got " + std::to_string(C3));
    const Tensor w3 = param(w3_, u);
    const int64_t K3 = C3 ? w3.numel() / C3 : 0;
    if (K3 * C3 != w3.numel()) raise(PyExc_RuntimeError, "shape '[" + std::to_string(C3) + ", -1]' is invalid for input of size " + std::to_string(w3.numel()));
    const Opt bias = param(bias_, u), b3 = param(b3_, u);
    const Modal m(log_poles, residues, u, theta, res_im);
    vtx_fused_iir_params p{};
    p.io_dtype = code(u);
    Tensor y;
    if (out_) {       // a [B, L, D] view with unit channel stride (e.g. a range of rows of a larger output)
        y = *out_;
        if (y.dim() != 3 || y.size(0) != B || y.size(1) != L || y.size(2) != D || y.scalar_type() != u.scalar_type() || y.stride(2) != 1 || y.device() != u.device())
            raise(PyExc_ValueError, "out must be a [B, L, D] tensor of u's dtype and device with unit channel stride");
    } else {
        y = empty({B, L, D}, u, u.scalar_type());
    }
    auto shape = [&] { return theta ? std::vector<int64_t>{B, D, m.m.S, 2} : std::vector<int64_t>{B, D, m.m.S}; };
    Opt st;
    if (want_state) { st = empty(shape(), u, at::kFloat); p.state = static_cast<float*>(out(*st)); }
    if (state_in) {
        if (state_in->sizes() != at::IntArrayRef(shape())) raise(PyExc_ValueError, "state_in has shape " + str(*state_in));
        state_in = state_in->to(at::kFloat).contiguous();
    }
    if (fir_state_in) {
        if (fir_state_in->sizes() != at::IntArrayRef({B, C3, 2}))
            raise(PyExc_ValueError, "fir_state_in has shape " + str(*fir_state_in) + ", expected (" + std::to_string(B) + ", " + std::to_string(C3) + ", 2)");
        fir_state_in = fir_state_in->contiguous();
    }
    p.u = ptr(u); p.u_stride_b = u.stride(0); p.u_stride_l = u.stride(1);
    p.w3 = ptr(w3); p.w3_dtype = code(w3); p.b3 = ptr(b3); p.b3_dtype = code_or_0(b3);
    p.modal = m.m; p.bias = ptr(bias); p.bias_dtype = code_or_0(bias);
    p.y = out(y); p.y_stride_b = y.stride(0); p.y_stride_l = y.stride(1);
    p.B = B; p.L = L; p.D = D; p.K3 = K3; p.layout = layout; p.num_heads = num_heads; p.flip_x1x2 = flip;
    p.state_in = static_cast<const float*>(ptr(state_in)); p.fir_state_in = ptr(fir_state_in); p.fir_state_dtype = code_or_0(fir_state_in);
    p.u_hist_rows = hist_rows;
    const int64_t need = p_fused_iir_scratch_bytes(&p);
    Tensor scratch;
    if (need > 0) { scratch = empty({need}, u, at::kByte); p.scratch = out(scratch); }
    const c10::cuda::CUDAGuard on(u.device());
    check(p_fused_iir_fwd(&p, stream_of(u)));
    return {y, st};
}

}  // namespace

PYBIND11_MODULE(_vtx_host, m) {
    m.def("abi_version", [] { return VTX_ABI_VERSION; });
    m.def("bind", [](uintptr_t decode, uintptr_t fir, uintptr_t iir, uintptr_t iir_scratch, uintptr_t last_error) {
        p_decode_layer = reinterpret_cast<decltype(p_decode_layer)>(decode);
        p_fused_fir_fwd = reinterpret_cast<decltype(p_fused_fir_fwd)>(fir);
        p_fused_iir_fwd = reinterpret_cast<decltype(p_fused_iir_fwd)>(iir);
        p_fused_iir_scratch_bytes = reinterpret_cast<decltype(p_fused_iir_scratch_bytes)>(iir_scratch);
        p_last_error = reinterpret_cast<decltype(p_last_error)>(last_error);
    });
    // Without the GIL, as torch's own calls and calls through ctypes are: an allocation or a launch into a full queue can
    // block, and the process's other threads go on meanwhile.
    m.def("decode_layer", &decode_layer, py::call_guard<py::gil_scoped_release>());
    m.def("fused_fir_fwd", &fused_fir_fwd, py::call_guard<py::gil_scoped_release>());
    m.def("fused_iir_fwd", &fused_iir_fwd, py::call_guard<py::gil_scoped_release>());
}
