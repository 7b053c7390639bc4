// host.cpp — the host path of the ops in native code: argument checks, output and workspace allocation, autograd nodes and
// the calls into the C ABI.  A call of a small problem is bound by this path, not by the GPU: through Python autograd
// Functions and ctypes one fused forward took 29 us on the host for a kernel of 8 us, and a forward + backward of the
// separate ops 214 us for 66 us of kernels; this path costs a few microseconds per op.
//
// The kernels stay behind the C ABI of libsapa_b200.so, whose functions are looked up in the library file that Python
// names (bind), so that one build of the library serves both this module and ctypes.
#include <torch/extension.h>

#include <ATen/cuda/CUDAContext.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAGuard.h>

#include <dlfcn.h>

#include <string>

#include "../../include/sapa_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

// ---------------------------------------------------------------------------------- the C ABI
struct Api {
#define SAPA_FN(name) decltype(&::name) name = nullptr;
#define SAPA_FNS                                                                                                          \
    SAPA_FN(sapa_last_error) SAPA_FN(sapa_qk_forward) SAPA_FN(sapa_qk_backward) SAPA_FN(sapa_av_forward)                  \
    SAPA_FN(sapa_av_backward) SAPA_FN(sapa_fused_forward_slab) SAPA_FN(sapa_fused_backward_workspace)                     \
    SAPA_FN(sapa_fused_forward_part) SAPA_FN(sapa_fused_forward_scratch)                                                                                 \
    SAPA_FN(sapa_fused_backward) SAPA_FN(sapa_deform_qk_forward) SAPA_FN(sapa_deform_qk_backward)                         \
    SAPA_FN(sapa_deform_av_forward) SAPA_FN(sapa_deform_av_backward) SAPA_FN(sapa_deform_fused_forward)                   \
    SAPA_FN(sapa_deform_fused_backward) SAPA_FN(sapa_deform_qk_forward_dense) SAPA_FN(sapa_deform_qk_backward_dense)      \
    SAPA_FN(sapa_deform_av_forward_dense) SAPA_FN(sapa_deform_av_backward_dense) SAPA_FN(sapa_deform_fused_forward_dense) \
    SAPA_FN(sapa_deform_fused_backward_dense) SAPA_FN(sapa_deform_fused_forward_workspace)                                \
    SAPA_FN(sapa_deform_fused_backward_workspace) SAPA_FN(sapa_deform_fused_backward_scatter_bytes)                       \
    SAPA_FN(sapa_project_workspace) SAPA_FN(sapa_project_forward) SAPA_FN(sapa_project_list_workspace)                    \
    SAPA_FN(sapa_project_list_forward) SAPA_FN(sapa_projections_workspace) SAPA_FN(sapa_projections_forward)              \
    SAPA_FN(sapa_projections_backward_workspace) SAPA_FN(sapa_projections_backward)
    SAPA_FNS
#undef SAPA_FN
};
Api api;

void bind(const std::string &path) {
    void *handle = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
    TORCH_CHECK(handle != nullptr, "cannot load ", path, ": ", dlerror());
#define SAPA_FN(name)                                                                       \
    api.name = reinterpret_cast<decltype(api.name)>(dlsym(handle, #name));                  \
    TORCH_CHECK(api.name != nullptr, path, " does not export " #name "; rebuild it");
    SAPA_FNS
#undef SAPA_FN
}

// ---------------------------------------------------------------------------------- checks and small helpers
[[noreturn]] void raise(PyObject *type, const char *text) {
    pybind11::gil_scoped_acquire gil;
    PyErr_SetString(type, text);
    throw pybind11::error_already_set();
}
#define PY_ASSERT(cond) do { if (!(cond)) raise(PyExc_AssertionError, #cond); } while (0)

// The ops mean the same inside torch.autocast as outside (the modules are given its type as an argument): the torch ops on their
// way must not cast.  softmax and sum come out in float32 there, and the kernels would read that as 16-bit elements.
struct NoAutocast {
    c10::impl::ExcludeDispatchKeyGuard off{c10::autocast_dispatch_keyset};
};
// An entry point as Python calls it: without the interpreter lock, which other threads may need while a launch waits for room in
// the queue or an allocation for the device.
template <typename R, typename... A>
auto native(R (*f)(A...)) {
    return [f](A... a) -> R {
        const pybind11::gil_scoped_release no_lock;
        const NoAutocast no_autocast;
        return f(a...);
    };
}

void need_cuda(const Tensor &t) {
    if (!t.is_cuda()) raise(PyExc_NotImplementedError, "");
}

struct Named { const char *name; const Tensor *t; };

// CUDA + contiguous (the reference's CHECK_INPUT, qk_cuda.cpp:34-39), plus one dtype and one device per call
void check_tensors(std::initializer_list<Named> named) {
    const Tensor &first = *named.begin()->t;
    for (const Named &n : named) {
        const Tensor &t = *n.t;
        TORCH_CHECK(t.is_cuda(), n.name, " must be a CUDA tensor");
        TORCH_CHECK(t.is_contiguous(), n.name, " must be contiguous");
        TORCH_CHECK(t.scalar_type() == first.scalar_type(), n.name, " has dtype ", t.scalar_type(), ", expected ",
                    first.scalar_type(), " (all tensors of a call share one dtype)");
        TORCH_CHECK(t.device() == first.device(), n.name, " is on ", t.device(), ", expected ", first.device());
    }
}

// an intermediate that the kernels read as elements of `like`'s type
void same_type(const Tensor &t, const Tensor &like, const char *name) {
    TORCH_CHECK(t.scalar_type() == like.scalar_type(), name, " has dtype ", t.scalar_type(), ", expected ", like.scalar_type());
}

int dtype_code(const Tensor &t) {
    switch (t.scalar_type()) {
        case at::kFloat: return SAPA_F32;
        case at::kHalf: return SAPA_F16;
        case at::kBFloat16: return SAPA_BF16;
        case at::kDouble: return SAPA_F64;
        default: TORCH_CHECK(false, "sapa_b200: unsupported dtype ", t.scalar_type());
    }
}

void done(int status, const char *name) {
    TORCH_CHECK(status == SAPA_OK, name, " failed with status ", status, ": ", api.sapa_last_error());
}

bool aligned16(const Tensor &t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }
// the fused kernels need a 16-byte aligned first element; a contiguous view with an odd storage offset is copied
Tensor aligned(const Tensor &t) { return aligned16(t) ? t : t.clone(); }
template <typename... Ts> bool all_aligned16(const Ts &...ts) { return (aligned16(ts) && ...); }

void *ptr(const Tensor &t) { return t.defined() ? t.data_ptr() : nullptr; }
void *stream() { return at::cuda::getCurrentCUDAStream().stream(); }
Tensor bytes(size_t n, const Tensor &like) { return at::empty({(int64_t)n}, like.options().dtype(at::kByte)); }
bool fast_type(const Tensor &t) {
    return t.scalar_type() == at::kFloat || t.scalar_type() == at::kHalf || t.scalar_type() == at::kBFloat16;
}
// scatter targets accumulate with atomics in float32 (float64 for float64 inputs)
at::ScalarType acc_type(const Tensor &t) { return t.scalar_type() == at::kDouble ? at::kDouble : at::kFloat; }
int dim(const Tensor &t, int i) { return (int)t.size(i); }
template <typename... Ts> bool wants_grad(const Ts &...ts) {
    return at::GradMode::is_enabled() && (ts.requires_grad() || ...);
}

void check_window(int64_t K, int64_t s) {
    const int64_t scale_factor = s, kernel_size = K;
    PY_ASSERT(scale_factor >= 1);
    PY_ASSERT((kernel_size - 1) % 2 == 0 && kernel_size >= 1);
}

#include "host_sapa.inc"
#include "host_deform.inc"
#include "host_module.inc"

}  // namespace

PYBIND11_MODULE(_host, m) {
    m.def("bind", &bind);
    m.def("qk", native(&qk));
    m.def("av", native(&av));
    m.def("sapa_fused", native(&sapa_fused));
    m.def("fused_forward_raw", native(&fused_forward_raw));
    m.def("qk_backward", native(&qk_bwd));
    m.def("av_backward", native(&av_bwd));
    m.def("sapa_fused_forward", native(&fused_forward_with_map));
    m.def("sapa_fused_backward", native(&fused_bwd));
    m.def("deform_qk_backward", native(&deform_qk_bwd));
    m.def("deform_av_backward", native(&deform_av_bwd));
    m.def("deform_fused_forward", native(&deform_fused_forward));
    m.def("deform_fused_backward", native(&deform_fused_bwd));
    m.def("deform_qk", native(&deform_qk));
    m.def("deform_av", native(&deform_av));
    m.def("deform_sapa_fused", native(&deform_fused));
    m.def("sapa_module", native(&sapa_module));
    m.def("deform_module", native(&deform_module));
    m.def("project_module", native(&project_module));
    m.def("project", native(&project));
    m.def("project_workspace", native(&project_workspace));
}
