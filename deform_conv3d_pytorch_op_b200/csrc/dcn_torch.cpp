// Native host path of the autograd Functions: argument checks, output and workspace allocation, the call into the
// C ABI (include/dcn.h) and the graph node that runs the backward pass, in one C++ call per direction.
//
// Why native: a training step of a small layer is a few kernels of 5-20 us, and the same work done through a Python
// autograd.Function over ctypes took 170-370 us of host time a step on a B200 box (problem structs, workspace queries,
// pointer wrapping, context managers), so that everything below ~10 GFLOP a step was bound by the host.
//
// It holds no state: sizes and layout are read from the tensors on every call, memory comes from torch's allocator
// on the current stream, and the environment switches (DCN_PRECISION, DCN_OOB_OFFSET_GRAD, DCN_CHECK_STATUS,
// DCN_NVTX) are read when a call needs them.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/DynamicTypes.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <cuda_runtime_api.h>
#include <nvtx3/nvToolsExt.h>

#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>

#include "../../include/dcn.h"

namespace {

using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

PyObject* g_error = nullptr;            // the package's DcnError

struct DcnFailure {
    std::string text;
};
[[noreturn]] void fail(const std::string& text) { throw DcnFailure{text}; }

void check(int status, const char* what) {
    if (status != DCN_OK)
        fail(std::string(what) + " failed: " + dcn_status_string(status) + " (status " + std::to_string(status) + ")");
}

bool env_set(const char* name) {
    const char* e = getenv(name);
    return e != nullptr && e[0] != '\0' && strcmp(e, "0") != 0;
}

struct Range {
    bool on;
    explicit Range(const char* name) : on(env_set("DCN_NVTX")) {
        if (on) nvtxRangePushA(name);
    }
    ~Range() {
        if (on) nvtxRangePop();
    }
};

enum Kind { kDeform, kPlain, kLayer };

struct Spec {                            // what a call says beside its tensors
    Kind kind = kDeform;
    bool std_rule = false;               // output size under the dilation-aware rule
    int channels_last = -1;              // -1: as the input is stored
    int ndim = 0;
    int stride[3] = {1, 1, 1}, pad[3] = {0, 0, 0}, dil[3] = {1, 1, 1};
    int64_t cpg = 1, group = 1;
    int oob = -1;                        // -1: DCN_OOB_OFFSET_GRAD decides
    std::string precision;               // empty: DCN_PRECISION decides
};

struct Problem {
    dcn_problem p;
    bool cl = false;
    at::MemoryFormat act = at::MemoryFormat::Contiguous;
    int64_t out[3] = {1, 1, 1};          // the last ndim hold the output size
};

std::string dtype_name(const Tensor& t) { return std::string("torch.") + torch::getTHPDtype(t.scalar_type())->name; }

std::string lower(std::string s) {
    for (char& c : s) c = (char)tolower((unsigned char)c);
    return s;
}

void fill_problem(dcn_problem& p, const Spec& s, const Tensor& x, const Tensor& w, int precision, bool cl) {
    memset(&p, 0, sizeof(p));
    p.ndim = s.ndim;
    p.dtype = x.scalar_type() == at::kDouble ? DCN_F64 : DCN_F32;
    p.precision = precision;
    p.deformable = s.kind != kPlain;
    p.std_size_rule = s.std_rule ? 1 : 0;
    if (s.oob >= 0) {
        p.oob_offset_grad = s.oob;
    } else {
        const char* e = getenv("DCN_OOB_OFFSET_GRAD");
        p.oob_offset_grad = !(e != nullptr && lower(e) == "zero");
    }
    p.N = (int32_t)x.size(0);
    p.C = (int32_t)x.size(1);
    p.O = (int32_t)w.size(0);
    p.G = (int32_t)s.group;
    p.cpg = (int32_t)(s.kind == kPlain ? x.size(1) : s.cpg);
    for (int a = 0; a < 3; ++a) {
        const int d = a - (3 - s.ndim);
        p.in[a] = d < 0 ? 1 : (int32_t)x.size(2 + d);
        p.k[a] = d < 0 ? 1 : (int32_t)w.size(2 + d);
        p.stride[a] = d < 0 ? 1 : s.stride[d];
        p.pad[a] = d < 0 ? 0 : s.pad[d];
        p.dil[a] = d < 0 ? 1 : s.dil[d];
    }
    p.channels_last = cl ? 1 : 0;
}

Problem make_problem(const Spec& s, const Tensor& x, const Tensor& w) {
    if (w.dim() != s.ndim + 2) fail("kernel dim");
    if (x.size(1) != w.size(1) * s.group) fail("input c != kernel c");
    if (x.scalar_type() != at::kFloat && x.scalar_type() != at::kDouble)
        fail("tensors must be float32 or float64, got " + dtype_name(x));
    Problem r;
    const at::MemoryFormat cl_format = s.ndim == 2 ? at::MemoryFormat::ChannelsLast : at::MemoryFormat::ChannelsLast3d;
    const bool cl = s.channels_last < 0 ? !x.is_contiguous() && x.is_contiguous(cl_format) : s.channels_last != 0;
    std::string prec = s.precision;
    if (prec.empty()) {
        const char* e = getenv("DCN_PRECISION");
        prec = e != nullptr ? e : "exact";
    }
    prec = lower(prec);
    if (prec == "auto") {
        // the tensor cores where the shape allows them and the problem pays for their layout pre-passes
        double flops = 2.0 * x.size(0) * w.size(0) * w.size(1);
        for (int d = 0; d < s.ndim; ++d) {
            const int64_t o = (x.size(2 + d) + 2 * s.pad[d] - w.size(2 + d)) / s.stride[d] + 1;
            flops *= (double)w.size(2 + d) * (o > 1 ? o : 1);
        }
        bool tc = x.scalar_type() == at::kFloat && flops >= 1e8;
        if (tc) {
            fill_problem(r.p, s, x, w, DCN_PREC_BF16, cl);
            tc = dcn_precision_supported(&r.p) != 0;
        }
        if (!tc) fill_problem(r.p, s, x, w, DCN_PREC_EXACT, false);
    } else if (prec == "bf16") {
        fill_problem(r.p, s, x, w, DCN_PREC_BF16, cl);
    } else if (prec == "exact" || prec == "fp32") {
        fill_problem(r.p, s, x, w, DCN_PREC_EXACT, false);
    } else {
        fail("unknown precision '" + prec + "' (exact | bf16 | auto)");
    }
    check(dcn_validate(&r.p), "shape check");
    if (!dcn_precision_supported(&r.p))
        fail("precision '" + prec + "' is not available for this problem (needs float32 tensors and channel counts per "
             "group that are multiples of 8); there is no silent fallback");
    r.cl = r.p.channels_last != 0;
    if (r.cl) r.act = cl_format;
    int32_t out[3];
    check(dcn_output_size(&r.p, out), "dcn_output_size");
    for (int a = 0; a < 3; ++a) r.out[a] = out[a];
    return r;
}

// A tensor of the call as the kernels read it: on x's device, of its type, dense in `format`.
Tensor prep(const Tensor& t, const char* name, const Tensor& x, at::MemoryFormat format = at::MemoryFormat::Contiguous) {
    if (!t.defined()) return t;
    if (!t.is_cuda()) fail(std::string(name) + " must be a CUDA tensor (there is no CPU implementation)");
    if (t.device() != x.device())
        fail(std::string(name) + " is on " + t.device().str() + " but input is on " + x.device().str());
    if (t.scalar_type() != x.scalar_type())
        fail(std::string(name) + " has dtype " + dtype_name(t) + " but input has " + dtype_name(x));
    return t.is_contiguous(format) ? t : t.contiguous(format);
}

void check_shape(const Tensor& t, const char* name, const std::vector<int64_t>& want) {
    if (t.sizes() != at::IntArrayRef(want)) {
        std::string a, b;
        for (int64_t v : t.sizes()) a += (a.empty() ? "" : ", ") + std::to_string(v);
        for (int64_t v : want) b += (b.empty() ? "" : ", ") + std::to_string(v);
        fail(std::string(name) + " shape (" + a + "), expected (" + b + ")");
    }
}

std::vector<int64_t> with_out(const Problem& q, int64_t n, int64_t c) {
    std::vector<int64_t> v{n, c};
    for (int a = 3 - q.p.ndim; a < 3; ++a) v.push_back(q.out[a]);
    return v;
}

int64_t offset_channels(const Problem& q) {
    return (int64_t)(q.p.C / q.p.cpg) * q.p.k[0] * q.p.k[1] * q.p.k[2] * q.p.ndim;
}

const void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
void* wptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

Tensor scratch(size_t bytes, const Tensor& x) {
    return bytes == 0 ? Tensor() : at::empty({(int64_t)bytes}, x.options().dtype(at::kByte));
}

// Workspace of a pass.  The exact precision also runs without one, on slower kernels that need no memory beside the tensors:
// where the allocator has no room for `bytes` the call goes on with the `least` that it cannot do without.
Tensor workspace(const Problem& q, size_t& bytes, size_t least, const Tensor& x) {
    if (q.p.precision != DCN_PREC_EXACT) return scratch(bytes, x);
    try {
        return scratch(bytes, x);
    } catch (const c10::OutOfMemoryError&) {
        bytes = least;
    }
    return scratch(bytes, x);
}

struct CallTensors {
    Tensor x, off, w, b, ow, ob;         // off: kDeform; ow, ob: kLayer
};

// Forward pass; on the bf16 path `keep` (if not null) receives the input copy, half the input's size, that the backward pass
// takes over.  For a layer t.off receives the offsets.
Tensor run_forward(const Problem& q, Kind kind, CallTensors& t, Tensor* keep) {
    const Tensor x = prep(t.x, "input", t.x, q.act);
    const Tensor w = prep(t.w, "weight", x), b = prep(t.b, "bias", x);
    Tensor off, ow, ob;
    size_t bytes;
    if (kind == kLayer) {
        ow = prep(t.ow, "offset_weight", x);
        ob = prep(t.ob, "offset_bias", x);
        std::vector<int64_t> want = w.sizes().vec();
        want[0] = offset_channels(q);
        want[1] = q.p.C;
        check_shape(ow, "offset_weight", want);
        bytes = dcn_layer_workspace_bytes(&q.p, DCN_PASS_FORWARD);
    } else {
        if (kind == kDeform) {
            off = prep(t.off, "offset", x);
            check_shape(off, "offset", with_out(q, q.p.N, offset_channels(q)));
        }
        bytes = dcn_workspace_bytes(&q.p, DCN_PASS_FORWARD);
    }
    const c10::cuda::CUDAGuard guard(x.device());
    void* st = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
    Tensor y = at::empty(with_out(q, q.p.N, q.p.O), x.options().memory_format(q.act));
    const size_t copy = keep != nullptr ? dcn_input_copy_bytes(&q.p) : 0;
    if (copy != 0) {
        *keep = scratch(copy, x);
        bytes -= copy;
    }
    void* xcl = copy != 0 ? wptr(*keep) : nullptr;
    if (kind == kLayer) off = at::empty(with_out(q, q.p.N, offset_channels(q)), x.options());
    const Tensor ws = workspace(q, bytes, 0, x);
    if (kind == kLayer) {
        Range range("dcn_layer_forward");
        check(dcn_layer_forward_keep(&q.p, ptr(x), ptr(ow), ptr(ob), ptr(w), ptr(b), wptr(off), wptr(y), xcl, wptr(ws), bytes,
                                     st), "dcn_layer_forward");
        t.off = off;
    } else {
        Range range("dcn_forward");
        check(dcn_forward_keep(&q.p, ptr(x), ptr(off), ptr(w), ptr(b), wptr(y), xcl, wptr(ws), bytes, st), "dcn_forward");
    }
    return y;
}

// Gradient slots, in the order of the node's edges.
enum Slot { kGx, kGoff, kGw, kGb, kGow, kGob, kSlots };

void run_backward(const Problem& q, Kind kind, const CallTensors& t, const Tensor& grad, const Tensor& xcl,
                  const bool (&want)[kSlots], Tensor (&g)[kSlots]) {
    const Tensor x = prep(t.x, "input", t.x, q.act);
    const Tensor w = prep(t.w, "weight", x), off = prep(t.off, "offset", x), ow = prep(t.ow, "offset_weight", x);
    const Tensor dy = prep(grad, "grad_output", x, q.act);
    const c10::cuda::CUDAGuard guard(x.device());
    const auto stream = c10::cuda::getCurrentCUDAStream(x.device().index());
    const auto opts = x.options();
    if (want[kGx]) g[kGx] = at::empty(x.sizes(), opts.memory_format(q.act));
    if (want[kGoff]) g[kGoff] = at::empty(off.sizes(), opts);
    if (want[kGw]) g[kGw] = at::empty(w.sizes(), opts);
    if (want[kGb]) g[kGb] = at::empty({q.p.O}, opts);
    if (want[kGow]) g[kGow] = at::empty(ow.sizes(), opts);
    if (want[kGob]) g[kGob] = at::empty({offset_channels(q)}, opts);
    if (kind == kLayer) {
        size_t bytes = dcn_layer_workspace_bytes(&q.p, DCN_PASS_BACKWARD);
        const Tensor ws = workspace(q, bytes, (off.nbytes() + 255) / 256 * 256, x);        // (the offset gradient)
        Range range("dcn_layer_backward");
        check(dcn_layer_backward(&q.p, ptr(x), ptr(off), ptr(ow), ptr(w), ptr(dy), ptr(xcl), wptr(g[kGx]), wptr(g[kGow]),
                                 wptr(g[kGob]), wptr(g[kGw]), wptr(g[kGb]), wptr(ws), bytes, stream.stream()),
              "dcn_layer_backward");
    } else {
        size_t bytes = dcn_workspace_bytes(&q.p, DCN_PASS_BACKWARD);
        const Tensor ws = workspace(q, bytes, 0, x);
        Range range("dcn_backward");
        check(dcn_backward(&q.p, ptr(x), ptr(off), ptr(w), ptr(dy), ptr(xcl), wptr(g[kGx]), wptr(g[kGoff]),
                           wptr(g[kGw]), wptr(g[kGb]), wptr(ws), bytes, stream.stream()),
              "dcn_backward");
    }
    if (kind != kPlain && env_set("DCN_CHECK_STATUS")) {
        cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
        cudaStreamIsCapturing(stream.stream(), &capturing);
        if (capturing == cudaStreamCaptureStatusNone) check(dcn_check_status(stream.stream()), "device status");
    }
}

struct DcnBackward : public Node {
    Problem q;
    Kind kind = kDeform;
    bool has[kSlots] = {};               // inputs the call had; their edges come in slot order
    SavedVariable x, off, w, ow;
    Tensor xcl;
    bool freed = false;

    std::string name() const override {
        if (kind == kLayer) return "DeformLayerFunctionBackward";
        return std::string(kind == kPlain ? "Conv" : "ConvOffset") + (q.p.ndim == 2 ? "2d" : "3d") + "FunctionBackward";
    }

    variable_list apply(variable_list&& grads) override {
        const std::lock_guard<std::mutex> lock(mutex_);
        if (freed)
            throw std::runtime_error("Trying to backward through the graph a second time (the saved tensors have already "
                                     "been freed). Specify retain_graph=True if you need to backward a second time.");
        Tensor g[kSlots];
        bool want[kSlots] = {};
        size_t edge = 0;
        for (int s = 0; s < kSlots; ++s)
            if (has[s]) want[s] = task_should_compute_output(edge++);
        bool differentiated = false;
        try {
            const auto self = shared_from_this();
            CallTensors t;
            t.x = x.unpack(self);
            t.w = w.unpack(self);
            t.off = off.unpack(self);
            t.ow = ow.unpack(self);
            Tensor dy = grads[0];
            differentiated = at::GradMode::is_enabled() && dy.defined() && dy.requires_grad();
            at::NoGradGuard no_grad;
            if (!dy.defined()) dy = at::zeros(with_out(q, q.p.N, q.p.O), t.x.options());
            run_backward(q, kind, t, dy, xcl, want, g);
        } catch (const DcnFailure& e) {
            pybind11::gil_scoped_acquire gil;
            PyErr_SetString(g_error, e.text.c_str());
            python_error err;
            err.persist();
            throw std::move(err);
        }
        variable_list out;
        for (int s = 0; s < kSlots; ++s)
            if (has[s]) out.push_back(g[s]);
        if (differentiated) {            // gradients of gradients are refused when they are asked for
            auto later = std::make_shared<torch::autograd::DelayedError>(
                "trying to differentiate twice a function that was marked with @once_differentiable", (int64_t)out.size());
            for (auto& v : out)
                if (v.defined()) v.requires_grad_(true);
            out = (*later)(std::move(out));
        }
        return out;
    }

    void release_variables() override {
        const std::lock_guard<std::mutex> lock(mutex_);
        freed = true;
        x.reset_data();
        off.reset_data();
        w.reset_data();
        ow.reset_data();
        xcl.reset();
    }
};

Tensor call(const Spec& s, CallTensors& t) {
    if (t.x.dim() != s.ndim + 2) throw std::runtime_error("input dim");
    const Tensor* slot[kSlots] = {&t.x, &t.off, &t.w, &t.b, &t.ow, &t.ob};
    bool has[kSlots], need = false;
    for (int i = 0; i < kSlots; ++i) {
        has[i] = slot[i]->defined();
        need = need || (has[i] && slot[i]->requires_grad());
    }
    need = need && at::GradMode::is_enabled();
    const Problem q = make_problem(s, t.x, t.w);
    if (!need) {
        at::NoGradGuard no_grad;
        return run_forward(q, s.kind, t, nullptr);
    }
    auto node = std::shared_ptr<DcnBackward>(new DcnBackward(), torch::autograd::deleteNode);
    torch::autograd::edge_list edges;
    for (int i = 0; i < kSlots; ++i)
        if (has[i])
            edges.push_back(slot[i]->requires_grad() ? torch::autograd::impl::gradient_edge(*slot[i]) : torch::autograd::Edge());
    node->set_next_edges(std::move(edges));
    node->q = q;
    node->kind = s.kind;
    memcpy(node->has, has, sizeof(has));
    Tensor y;
    {
        at::NoGradGuard no_grad;
        // the input copy is kept only where a gradient needs it, and never past saved-tensor hooks: a program that moves or
        // drops what is saved (offloading, checkpoints) gets the tensors named below and nothing beside them
        bool kept = t.w.requires_grad();
        if (s.kind != kPlain)
            for (int i : {kGx, kGoff, kGow, kGob}) kept = kept || (has[i] && slot[i]->requires_grad());
        kept = kept && !at::SavedTensorDefaultHooks::get_hooks().has_value();
        y = run_forward(q, s.kind, t, kept ? &node->xcl : nullptr);
    }
    node->x = SavedVariable(t.x, false);
    node->w = SavedVariable(t.w, false);
    if (t.off.defined()) node->off = SavedVariable(t.off, false);
    if (t.ow.defined()) node->ow = SavedVariable(t.ow, false);
    torch::autograd::set_history(y, node);
    return y;
}

// Calls that have to go through a torch.autograd.Function: a trace records it as one operation (a direct call would leave
// its result in the trace as a constant), and function transforms and forward-mode derivatives ask it for rules.
bool transformed(const CallTensors& t) {
    if (torch::jit::tracer::isTracing() ||
        c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode))
        return true;
    for (const Tensor* v : {&t.x, &t.off, &t.w, &t.b, &t.ow, &t.ob})
        if (v->defined() && torch::autograd::isFwGradDefined(*v)) return true;
    return false;
}

// ---- arguments ------------------------------------------------------------------------------------------------
Tensor tensor_arg(PyObject* o, const char* name, bool optional = false) {
    if (optional && o == Py_None) return Tensor();
    if (!THPVariable_Check(o)) {
        PyErr_Format(PyExc_TypeError, "%s must be a Tensor, not %s", name, Py_TYPE(o)->tp_name);
        throw python_error();
    }
    return THPVariable_Unpack(o);
}

int64_t int_arg(PyObject* o) {
    PyObject* i = PyNumber_Index(o);
    if (i == nullptr) throw python_error();
    const int64_t v = PyLong_AsLongLong(i);
    Py_DECREF(i);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return v;
}

int small_int(int64_t v) {
    if (v < -2147483647ll || v > 2147483647ll) fail("value out of range");
    return (int)v;
}

// an int for every axis, or one int per axis
void axes_arg(PyObject* o, int ndim, int (&out)[3]) {
    if (PyTuple_Check(o) || PyList_Check(o)) {
        const Py_ssize_t n = PySequence_Fast_GET_SIZE(o);
        if (n != ndim) fail("expected " + std::to_string(ndim) + " values, got " + std::to_string(n));
        for (int i = 0; i < ndim; ++i) out[i] = small_int(int_arg(PySequence_Fast_GET_ITEM(o, i)));
    } else {
        const int v = small_int(int_arg(o));
        for (int i = 0; i < ndim; ++i) out[i] = v;
    }
}

void precision_arg(PyObject* o, Spec& s) {
    if (o == Py_None) return;
    const char* text = PyUnicode_AsUTF8(o);
    if (text == nullptr) throw python_error();
    s.precision = text;
}

void oob_arg(PyObject* o, Spec& s) {
    if (o == Py_None) return;
    s.oob = PyObject_IsTrue(o);
    if (s.oob < 0) throw python_error();
}

void count_arg(Py_ssize_t n, Py_ssize_t lo, Py_ssize_t hi) {
    if (n >= lo && n <= hi) return;
    PyErr_Format(PyExc_TypeError, "expected %zd to %zd arguments, got %zd", lo, hi, n);
    throw python_error();
}

template <typename Parse>
PyObject* entry(Parse&& parse) {
    HANDLE_TH_ERRORS
    try {
        Spec s;
        CallTensors t;
        parse(s, t);
        if (transformed(t)) Py_RETURN_NOTIMPLEMENTED;          // functions.py takes the other way
        Tensor y;
        {
            pybind11::gil_scoped_release no_gil;
            y = call(s, t);
        }
        return THPVariable_Wrap(std::move(y));
    } catch (const DcnFailure& e) {
        PyErr_SetString(g_error, e.text.c_str());
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

// (inputs, offset, weight, bias, stride, padding, dilation, channel_per_group, group, precision, oob_offset_grad)
template <int ND>
PyObject* conv_offset(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return entry([&](Spec& s, CallTensors& t) {
        count_arg(n, 3, 11);
        s.kind = kDeform;
        s.ndim = ND;
        t.x = tensor_arg(a[0], "inputs");
        t.off = tensor_arg(a[1], "offset");
        t.w = tensor_arg(a[2], "weight");
        if (n > 3) t.b = tensor_arg(a[3], "bias", true);
        if (n > 4) axes_arg(a[4], ND, s.stride);
        if (n > 5) axes_arg(a[5], ND, s.pad);
        if (n > 6) axes_arg(a[6], ND, s.dil);
        if (n > 7) s.cpg = small_int(int_arg(a[7]));
        if (n > 8) s.group = small_int(int_arg(a[8]));
        if (n > 9) precision_arg(a[9], s);
        if (n > 10) oob_arg(a[10], s);
    });
}

// (inputs, weight, bias, stride, padding, dilation, group, precision)
template <int ND>
PyObject* conv(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return entry([&](Spec& s, CallTensors& t) {
        count_arg(n, 2, 8);
        s.kind = kPlain;
        s.std_rule = true;
        s.ndim = ND;
        t.x = tensor_arg(a[0], "inputs");
        t.w = tensor_arg(a[1], "weight");
        if (n > 2) t.b = tensor_arg(a[2], "bias", true);
        if (n > 3) axes_arg(a[3], ND, s.stride);
        if (n > 4) axes_arg(a[4], ND, s.pad);
        if (n > 5) axes_arg(a[5], ND, s.dil);
        if (n > 6) s.group = small_int(int_arg(a[6]));
        if (n > 7) precision_arg(a[7], s);
    });
}

// (inputs, offset_weight, offset_bias, weight, bias, stride, padding, dilation, channel_per_group, group, precision,
//  oob_offset_grad); 2-D or 3-D by the input's rank
PyObject* deform_layer(PyObject*, PyObject* const* a, Py_ssize_t n) {
    return entry([&](Spec& s, CallTensors& t) {
        count_arg(n, 8, 12);
        s.kind = kLayer;
        t.x = tensor_arg(a[0], "inputs");
        s.ndim = (int)t.x.dim() - 2;
        if (s.ndim != 2 && s.ndim != 3) fail("input dim");
        t.ow = tensor_arg(a[1], "offset_weight");
        t.ob = tensor_arg(a[2], "offset_bias", true);
        t.w = tensor_arg(a[3], "weight");
        t.b = tensor_arg(a[4], "bias", true);
        axes_arg(a[5], s.ndim, s.stride);
        axes_arg(a[6], s.ndim, s.pad);
        axes_arg(a[7], s.ndim, s.dil);
        if (n > 8) s.cpg = small_int(int_arg(a[8]));
        if (n > 9) s.group = small_int(int_arg(a[9]));
        if (n > 10) precision_arg(a[10], s);
        if (n > 11) oob_arg(a[11], s);
    });
}

// The dcn_problem of a call, as bytes: every check and rule on sizes, types, precision and storage that the Functions apply,
// for ops.py.  (x, weight, stride, padding, dilation, channel_per_group, group, deformable, std_size_rule, oob_offset_grad,
// precision, channels_last); the last three may be None
PyObject* problem(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    try {
        count_arg(n, 12, 12);
        const Tensor x = tensor_arg(a[0], "x"), w = tensor_arg(a[1], "weight");
        Spec s;
        s.ndim = (int)x.dim() - 2;
        if (s.ndim != 2 && s.ndim != 3) fail("input dim");
        axes_arg(a[2], s.ndim, s.stride);
        axes_arg(a[3], s.ndim, s.pad);
        axes_arg(a[4], s.ndim, s.dil);
        s.cpg = small_int(int_arg(a[5]));
        s.group = small_int(int_arg(a[6]));
        s.kind = PyObject_IsTrue(a[7]) ? kDeform : kPlain;
        s.std_rule = PyObject_IsTrue(a[8]) != 0;
        oob_arg(a[9], s);
        precision_arg(a[10], s);
        if (a[11] != Py_None) s.channels_last = PyObject_IsTrue(a[11]);
        const Problem q = make_problem(s, x, w);
        return PyBytes_FromStringAndSize(reinterpret_cast<const char*>(&q.p), sizeof(q.p));
    } catch (const DcnFailure& e) {
        PyErr_SetString(g_error, e.text.c_str());
        return nullptr;
    }
    END_HANDLE_TH_ERRORS
}

PyObject* set_error(PyObject*, PyObject* cls) {
    Py_INCREF(cls);
    Py_XDECREF(g_error);
    g_error = cls;
    Py_RETURN_NONE;
}

#define DCN_FAST(fn) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL
PyMethodDef methods[] = {
    {"conv_offset2d", DCN_FAST(conv_offset<2>), nullptr},
    {"conv_offset3d", DCN_FAST(conv_offset<3>), nullptr},
    {"conv2d", DCN_FAST(conv<2>), nullptr},
    {"conv3d", DCN_FAST(conv<3>), nullptr},
    {"deform_layer", DCN_FAST(deform_layer), nullptr},
    {"problem", DCN_FAST(problem), nullptr},
    {"set_error", set_error, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_dcn_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__dcn_torch(void) { return PyModule_Create(&module); }
