// The Python-facing calls of the library: argument checks, allocation, stream lookup and the C ABI call, and the
// differentiable forms of the two ops as native autograd nodes.  Everything here is host work per call; it bounds every
// layer that runs for less than a few tens of microseconds, which is why it is not Python (one image through the
// 64 x 64 x 56 x 56 layer took 24 us to enqueue from Python for 12 us of kernel).  The arithmetic, and every decision about
// how a shape is computed, stays behind include/winograd2x2_b200.h.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>

#include <mutex>

#include "../../include/winograd2x2_b200.h"

namespace {

using at::Tensor;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

PyObject *g_error = nullptr;     // wg2x2.Wg2x2Error, handed over by set_error

// ---------------------------------------------------------------------------------------
// Errors: the types and texts that the callers of the Python functions see
// ---------------------------------------------------------------------------------------
void check(int status, const char *what)
{
    if (status == WG2X2_OK) return;
    pybind11::gil_scoped_acquire gil;      // also reached from the autograd engine's threads
    PyObject *e = g_error ? PyObject_CallFunction(g_error, "is", status, what) : nullptr;
    if (e) {
        PyErr_SetObject(g_error, e);
        Py_DECREF(e);
    } else if (!PyErr_Occurred()) {
        PyErr_Format(PyExc_RuntimeError, "%s: status %d", what, status);
    }
    python_error err;                      // carries the exception over to whichever thread reports it
    err.persist();
    throw std::move(err);
}
[[noreturn]] void value_error(const std::string &msg) { TORCH_CHECK_VALUE(false, msg); __builtin_unreachable(); }
[[noreturn]] void type_error(const std::string &msg) { throw torch::TypeError(msg); }
[[noreturn]] void not_a_tensor(const char *name) { type_error(std::string(name) + " must be a contiguous float32 CUDA tensor"); }

void require(const Tensor &t, const char *name)
{
    if (!(t.is_cuda() && t.scalar_type() == at::kFloat && t.is_contiguous()))
        not_a_tensor(name);
}
std::string shape_text(at::IntArrayRef s)
{
    std::string o = "(";
    for (size_t i = 0; i < s.size(); ++i) o += (i ? ", " : "") + std::to_string(s[i]);
    return o + (s.size() == 1 ? ",)" : ")");
}

// a float32 CUDA tensor argument; `None` gives an undefined tensor where that is allowed
Tensor arg(PyObject *o, const char *name, bool optional = false)
{
    if (optional && o == Py_None) return Tensor();
    if (!THPVariable_Check(o)) not_a_tensor(name);
    const Tensor &t = THPVariable_Unpack(o);
    require(t, name);
    return t;
}
Tensor arg_shaped(PyObject *o, at::IntArrayRef shape, const char *name)
{
    Tensor t = arg(o, name, true);
    if (t.defined() && t.sizes() != shape)
        value_error(std::string(name) + " has shape " + shape_text(t.sizes()) + ", expected " + shape_text(shape));
    return t;
}
// a tensor whose memory is used as it is: an output or a workspace of the caller
Tensor arg_raw(PyObject *o, const char *name)
{
    if (o == Py_None) return Tensor();
    if (!THPVariable_Check(o)) type_error(std::string(name) + " must be a tensor");
    return THPVariable_Unpack(o);
}
int arg_int(PyObject *o)
{
    const long v = PyLong_AsLong(o);
    if (v == -1 && PyErr_Occurred()) throw python_error();
    return (int)v;
}
bool arg_bool(PyObject *o)
{
    const int v = PyObject_IsTrue(o);
    if (v < 0) throw python_error();
    return v != 0;
}
int arg_int_or(PyObject *o, int otherwise) { return o == Py_None ? otherwise : arg_int(o); }

void need_dims(const Tensor &t, int dims, const char *name)
{
    if (t.dim() != dims) value_error(std::string(name) + " must have " + std::to_string(dims) + " dimensions, got " + shape_text(t.sizes()));
}

struct Img { int64_t B, H, W, C; };
Img img_of(const Tensor &t, int layout, const char *name)
{
    need_dims(t, 4, name);
    const auto s = t.sizes();
    return layout == WG2X2_NHWC ? Img{s[0], s[1], s[2], s[3]} : Img{s[0], s[2], s[3], s[1]};
}
std::array<int64_t, 4> img_shape(int64_t B, int64_t H, int64_t W, int64_t C, int layout)
{
    if (layout == WG2X2_NHWC) return {B, H, W, C};
    return {B, C, H, W};
}

// The opaque buffer of prepare_weights for exactly (C, K): the kernels build their TMA maps over it from C and K alone, so
// a buffer made for other sizes would be read past its end.
Tensor arg_prepared(PyObject *o, int64_t C, int64_t K)
{
    if (!THPVariable_Check(o)) type_error("prepared must be the buffer returned by prepare_weights");
    const Tensor &t = THPVariable_Unpack(o);
    if (!t.is_cuda() || t.scalar_type() != at::kByte) type_error("prepared must be the buffer returned by prepare_weights");
    static PyObject *ck_name = PyUnicode_InternFromString("_wg_ck");
    if (PyObject *ck = PyObject_GetAttr(o, ck_name)) {
        long c = 0, k = 0;
        const bool pair = PyTuple_Check(ck) && PyTuple_GET_SIZE(ck) == 2;
        if (pair) { c = PyLong_AsLong(PyTuple_GET_ITEM(ck, 0)); k = PyLong_AsLong(PyTuple_GET_ITEM(ck, 1)); }
        Py_DECREF(ck);
        if (pair && (c != C || k != K))
            value_error("prepared weights are for (C, K) = (" + std::to_string(c) + ", " + std::to_string(k) + "), the call has (" +
                        std::to_string(C) + ", " + std::to_string(K) + ")");
    } else {
        PyErr_Clear();
    }
    if ((size_t)t.numel() < wg2x2_prepared_weights_bytes((int)C, (int)K))
        value_error("prepared weight buffer too small for C=" + std::to_string(C) + " K=" + std::to_string(K));
    return t;
}

// ---------------------------------------------------------------------------------------
// Memory and launch context
// ---------------------------------------------------------------------------------------
const float *cptr(const Tensor &t) { return t.defined() ? static_cast<const float *>(t.data_ptr()) : nullptr; }
float *ptr(const Tensor &t) { return t.defined() ? static_cast<float *>(t.data_ptr()) : nullptr; }

Tensor new_float(at::IntArrayRef shape, const Tensor &like)
{
    return Tensor(at::detail::empty_cuda(shape, at::kFloat, like.device(), std::nullopt));
}

// Scratch memory of one call: from torch's caching allocator, whose blocks belong to the stream they were taken on, so that
// the block may be handed on while the kernels that use it are still queued.
struct Scratch {
    c10::DataPtr block;
    size_t bytes = 0;
    void take(size_t n)
    {
        if (!n) return;
        block = c10::cuda::CUDACachingAllocator::get()->allocate(n);
        bytes = n;
    }
    void *get() const { return block.get(); }
};

// The tensor's device, current, and its current stream
struct OnDevice {
    c10::cuda::CUDAGuard guard;
    void *stream;
    explicit OnDevice(const Tensor &t) : guard(t.device()), stream(c10::cuda::getCurrentCUDAStream(t.device().index()).stream()) {}
};

// ---------------------------------------------------------------------------------------
// The ops
// ---------------------------------------------------------------------------------------
Tensor imtrans_fwd(const Tensor &x, bool relu, int layout, const Tensor &out, const Tensor &in_scale, const Tensor &in_shift)
{
    const Img d = img_of(x, layout, "x");
    OnDevice on(x);
    Tensor V = out.defined() ? out : new_float({16, d.B, (d.H + 1) / 2, (d.W + 1) / 2, d.C}, x);
    if (in_scale.defined())
        check(wg2x2_imtrans_fwd_affine(cptr(x), cptr(in_scale), cptr(in_shift), ptr(V), d.B, d.H, d.W, d.C, layout, relu, on.stream),
              "wg2x2_imtrans_fwd_affine");
    else
        check(wg2x2_imtrans_fwd(cptr(x), ptr(V), d.B, d.H, d.W, d.C, layout, relu, on.stream), "wg2x2_imtrans_fwd");
    return V;
}

Tensor imtrans_bwd(const Tensor &dV, int64_t H, int64_t W, const Tensor &V_relu, int layout)
{
    need_dims(dV, 5, "dV");
    const int64_t B = dV.size(1), nH = dV.size(2), nW = dV.size(3), C = dV.size(4);
    if ((H + 1) / 2 != nH || (W + 1) / 2 != nW) value_error("H, W do not match the tile grid of dV");
    OnDevice on(dV);
    Tensor dX = new_float(img_shape(B, H, W, C, layout), dV);
    check(wg2x2_imtrans_bwd(cptr(dV), cptr(V_relu), ptr(dX), B, H, W, C, layout, on.stream), "wg2x2_imtrans_bwd");
    return dX;
}

Tensor conv_fwd(const Tensor &V, const Tensor &Wt, int out_h, int out_w, int layout, int math, const Tensor &out, const Tensor &workspace)
{
    need_dims(V, 5, "V");
    const int64_t B = V.size(1), nH = V.size(2), nW = V.size(3), C = V.size(4);
    if (Wt.dim() != 3 || Wt.size(0) != 16 || Wt.size(1) != C) value_error("Wt must be (16, C, K)");
    const int64_t K = Wt.size(2);
    if (out_h < 0) out_h = (int)(2 * nH);
    if (out_w < 0) out_w = (int)(2 * nW);
    OnDevice on(V);
    Tensor Y = out.defined() ? out : new_float(img_shape(B, out_h, out_w, K, layout), V);
    Scratch ws;
    void *wp = nullptr;
    size_t wn = 0;
    if (workspace.defined()) { wp = workspace.data_ptr(); wn = (size_t)workspace.numel(); }
    else { ws.take(wg2x2_conv_fwd_workspace_bytes(B, nH, nW, C, K, math)); wp = ws.get(); wn = ws.bytes; }
    check(wg2x2_conv_fwd(cptr(V), cptr(Wt), ptr(Y), B, nH, nW, C, K, out_h, out_w, layout, math, wp, wn, on.stream), "wg2x2_conv_fwd");
    return Y;
}

std::pair<Tensor, Tensor> conv_bwd(const Tensor &V, const Tensor &Wt, const Tensor &dY, const Tensor &mask, int layout, bool relu, int math,
                                   bool need_dV, bool need_dW)
{
    need_dims(V, 5, "V");
    const int64_t B = V.size(1), nH = V.size(2), nW = V.size(3), C = V.size(4);
    need_dims(Wt, 3, "Wt");
    const int64_t K = Wt.size(2);
    const Img d = img_of(dY, layout, "dY");
    if (d.B != B || d.C != K || (d.H + 1) / 2 != nH || (d.W + 1) / 2 != nW) value_error("dY does not match V / Wt");
    OnDevice on(V);
    Tensor dV, dW;
    if (need_dV) dV = new_float(V.sizes(), V);
    if (need_dW) dW = new_float(Wt.sizes(), V);
    Scratch ws;
    ws.take(wg2x2_conv_bwd_workspace_bytes(B, d.H, d.W, C, K, math, need_dW));
    check(wg2x2_conv_bwd(cptr(V), cptr(Wt), cptr(dY), cptr(mask), ptr(dV), ptr(dW), B, d.H, d.W, C, K, layout, relu, math, ws.get(), ws.bytes,
                         on.stream),
          "wg2x2_conv_bwd");
    return {dV, dW};
}

// ---------------------------------------------------------------------------------------
// Autograd nodes of the two ops (the reference pairs each op with its gradient op by RegisterGradient:
// winograd2x2_imTrans.py:29-33, winograd2x2_conv.py:32-36).  Several threads may run backward over one graph: what a node saved is read
// and released under its lock.
// ---------------------------------------------------------------------------------------
struct ImTransBackward : public torch::autograd::Node {
    SavedVariable bits_;       // where the output is positive, kept only where the ReLU was applied
    int64_t H = 0, W = 0;
    int layout = 0;
    bool relu = false;
    std::string name() const override { return "Winograd2x2ImTransBackward"; }
    void release_variables() override
    {
        const std::lock_guard<std::mutex> lock(mutex_);
        bits_.reset_data();
    }
    variable_list apply(variable_list &&grads) override
    {
        if (!grads[0].defined()) return {Tensor()};
        Tensor bits;
        if (relu) {
            const std::lock_guard<std::mutex> lock(mutex_);
            bits = bits_.unpack();
        }
        const Tensor g = grads[0].contiguous();
        require(g, "dV");
        if (!relu) return {imtrans_bwd(g, H, W, Tensor(), layout)};
        OnDevice on(g);
        const int64_t B = g.size(1), C = g.size(4);
        Tensor dX = new_float(img_shape(B, H, W, C, layout), g);
        check(wg2x2_imtrans_bwd_relu_bits(cptr(g), bits.data_ptr(), ptr(dX), B, H, W, C, layout, on.stream), "wg2x2_imtrans_bwd_relu_bits");
        return {dX};
    }
};

struct ConvBackward : public torch::autograd::Node {
    SavedVariable I_, W_, mask_;      // W with the mask applied
    int layout = 0, math = 0;
    std::string name() const override { return "Winograd2x2ConvBackward"; }
    void release_variables() override
    {
        const std::lock_guard<std::mutex> lock(mutex_);
        I_.reset_data();
        W_.reset_data();
        mask_.reset_data();
    }
    variable_list apply(variable_list &&grads) override
    {
        if (!grads[0].defined()) return {Tensor(), Tensor()};
        const bool dI = task_should_compute_output(0), dW = task_should_compute_output(1);
        const Tensor g = grads[0].contiguous();
        require(g, "dY");
        Tensor I, Wt, mask;
        {
            const std::lock_guard<std::mutex> lock(mutex_);
            I = I_.unpack();
            Wt = W_.unpack();
            mask = mask_.unpack();
        }
        auto r = conv_bwd(I, Wt, g, mask, layout, false, math, dI, dW);
        return {r.first, r.second};
    }
};

template <class N>
std::shared_ptr<N> new_node(torch::autograd::edge_list edges)
{
    std::shared_ptr<N> n(new N(), torch::autograd::deleteNode);
    n->set_next_edges(std::move(edges));
    return n;
}

// There is no forward-mode rule: a tangent is refused, as torch.autograd.Function refuses it, not dropped.
void no_tangent(const Tensor &t)
{
    TORCH_CHECK_NOT_IMPLEMENTED(!t.defined() || !t._fw_grad(0).defined(), "forward-mode automatic differentiation is not implemented for the Winograd ops");
}

Tensor imtrans_op(const Tensor &in, bool relu, int layout)
{
    no_tangent(in);
    const Tensor I = in.contiguous();
    require(I, "x");
    const bool grad = torch::autograd::compute_requires_grad(I);
    Tensor V, bits;
    if (grad && relu) {
        const Img d = img_of(I, layout, "x");
        OnDevice on(I);
        V = new_float({16, d.B, (d.H + 1) / 2, (d.W + 1) / 2, d.C}, I);
        bits = Tensor(at::detail::empty_cuda({d.B, (d.H + 1) / 2, (d.W + 1) / 2, d.C}, at::kShort, I.device(), std::nullopt));
        check(wg2x2_imtrans_fwd_relu_bits(cptr(I), ptr(V), bits.data_ptr(), d.B, d.H, d.W, d.C, layout, on.stream), "wg2x2_imtrans_fwd_relu_bits");
    } else {
        V = imtrans_fwd(I, relu, layout, Tensor(), Tensor(), Tensor());
    }
    if (grad) {
        auto n = new_node<ImTransBackward>(torch::autograd::collect_next_edges(I));
        const Img d = img_of(I, layout, "x");
        n->H = d.H; n->W = d.W; n->layout = layout; n->relu = relu;
        if (relu) n->bits_ = SavedVariable(bits, false);
        torch::autograd::set_history(V, n);
    }
    return V;
}

// With a mask the weights are win * mask.  The product is made here, not by the caller, so that neither it nor its gradient (the
// mask on dW, which the dW kernels apply anyway) is a node and a kernel of its own: 12 + 10 us of host time in a training step.
Tensor conv_op(const Tensor &in, const Tensor &win, const Tensor &mask, int out_h, int out_w, int layout, int math)
{
    no_tangent(in);
    no_tangent(win);
    no_tangent(mask);
    const Tensor I = in.contiguous();
    Tensor Wt = win.contiguous();
    require(I, "V");
    require(Wt, "Wt");
    const Tensor W0 = Wt;
    if (mask.defined()) {
        if (Wt.dim() != 3 || Wt.size(0) != 16 || mask.sizes() != Wt.sizes() || mask.device() != Wt.device())
            value_error("mask must have the weights' shape (16, C, K) and be on their device");
        OnDevice on(Wt);
        Wt = new_float(W0.sizes(), W0);
        check(wg2x2_weights_mask(cptr(W0), cptr(mask), ptr(Wt), (int)W0.size(1), (int)W0.size(2), on.stream), "wg2x2_weights_mask");
    }
    Tensor Y = conv_fwd(I, Wt, out_h, out_w, layout, math, Tensor(), Tensor());
    if (torch::autograd::compute_requires_grad(I, W0)) {
        auto n = new_node<ConvBackward>(torch::autograd::collect_next_edges(I, W0));
        n->layout = layout; n->math = math;
        n->I_ = SavedVariable(I, false);
        n->W_ = SavedVariable(Wt, false);
        if (mask.defined()) n->mask_ = SavedVariable(mask, false);
        torch::autograd::set_history(Y, n);
    }
    return Y;
}

// ---------------------------------------------------------------------------------------
// Python entry points (positional arguments, all given; the keyword forms and defaults are in ops.py)
// ---------------------------------------------------------------------------------------
void want(Py_ssize_t got, Py_ssize_t n)
{
    if (got != n) type_error("expected " + std::to_string(n) + " arguments, got " + std::to_string(got));
}
#define WG_ARGS PyObject *, PyObject *const *a, Py_ssize_t n
// The GIL is given up while a call allocates and launches, as a foreign call would do it
#define WG_NOGIL pybind11::gil_scoped_release nogil

PyObject *py_set_error(PyObject *, PyObject *cls)
{
    Py_XINCREF(cls);
    Py_XSETREF(g_error, cls);
    Py_RETURN_NONE;
}

// x, relu, layout, out, in_scale, in_shift
PyObject *py_imtrans_fwd(WG_ARGS)
{
    HANDLE_TH_ERRORS
    want(n, 6);
    const Tensor x = arg(a[0], "x");
    const bool relu = arg_bool(a[1]);
    const int layout = arg_int(a[2]);
    const Tensor out = arg_raw(a[3], "out");
    Tensor sc, sh;
    if (a[4] != Py_None) { sc = arg(a[4], "in_scale"); sh = arg(a[5], "in_shift"); }
    Tensor V;
    { WG_NOGIL; V = imtrans_fwd(x, relu, layout, out, sc, sh); }
    return THPVariable_Wrap(V);
    END_HANDLE_TH_ERRORS
}

// dV, H, W, V_relu, layout
PyObject *py_imtrans_bwd(WG_ARGS)
{
    HANDLE_TH_ERRORS
    want(n, 5);
    const Tensor dV = arg(a[0], "dV");
    const int H = arg_int(a[1]), W = arg_int(a[2]);
    const Tensor Vr = arg(a[3], "V_relu", true);
    const int layout = arg_int(a[4]);
    Tensor dX;
    { WG_NOGIL; dX = imtrans_bwd(dV, H, W, Vr, layout); }
    return THPVariable_Wrap(dX);
    END_HANDLE_TH_ERRORS
}

// V, Wt, out_h, out_w, layout, math, out, workspace
PyObject *py_conv_fwd(WG_ARGS)
{
    HANDLE_TH_ERRORS
    want(n, 8);
    const Tensor V = arg(a[0], "V"), Wt = arg(a[1], "Wt");
    const int oh = arg_int_or(a[2], -1), ow = arg_int_or(a[3], -1), layout = arg_int(a[4]), math = arg_int(a[5]);
    const Tensor out = arg_raw(a[6], "out"), ws = arg_raw(a[7], "workspace");
    Tensor Y;
    { WG_NOGIL; Y = conv_fwd(V, Wt, oh, ow, layout, math, out, ws); }
    return THPVariable_Wrap(Y);
    END_HANDLE_TH_ERRORS
}

// V, prepared, K, out_h, out_w, layout, out, out_scale, out_shift, residual, workspace, wide
PyObject *py_conv_fwd_prepared(WG_ARGS)
{
    HANDLE_TH_ERRORS
    want(n, 12);
    const Tensor V = arg(a[0], "V");
    need_dims(V, 5, "V");
    const int64_t B = V.size(1), nH = V.size(2), nW = V.size(3), C = V.size(4), K = arg_int(a[2]);
    const Tensor prep = arg_prepared(a[1], C, K);
    const int oh = arg_int_or(a[3], (int)(2 * nH)), ow = arg_int_or(a[4], (int)(2 * nW)), layout = arg_int(a[5]);
    const auto ys = img_shape(B, oh, ow, K, layout);
    Tensor Y = arg_shaped(a[6], ys, "out");
    const Tensor sc = arg_shaped(a[7], {K}, "out_scale"), sh = arg_shaped(a[8], {K}, "out_shift"), res = arg_shaped(a[9], ys, "residual");
    const Tensor uws = arg_raw(a[10], "workspace");
    const bool wide = arg_bool(a[11]);
    {
        WG_NOGIL;
        OnDevice on(V);
        if (!Y.defined()) Y = new_float(ys, V);
        const size_t nws = wide ? wg2x2_conv_fwd_prepared_workspace_bytes(B, nH, nW, C, K) : 0;
        if (nws) {       // many channels: products as wide GEMMs into scratch memory, then the output transform
            Scratch ws;
            void *wp;
            size_t wn;
            if (uws.defined() && (size_t)uws.numel() >= nws) { wp = uws.data_ptr(); wn = (size_t)uws.numel(); }
            else { ws.take(nws); wp = ws.get(); wn = nws; }
            check(wg2x2_conv_fwd_prepared_ws(cptr(V), prep.data_ptr(), ptr(Y), B, nH, nW, C, K, oh, ow, layout, cptr(sc), cptr(sh), cptr(res),
                                             wp, wn, on.stream),
                  "wg2x2_conv_fwd_prepared_ws");
        } else if (!sc.defined() && !res.defined()) {
            check(wg2x2_conv_fwd_prepared(cptr(V), prep.data_ptr(), ptr(Y), B, nH, nW, C, K, oh, ow, layout, on.stream), "wg2x2_conv_fwd_prepared");
        } else {
            check(wg2x2_conv_fwd_prepared_fused(cptr(V), prep.data_ptr(), ptr(Y), B, nH, nW, C, K, oh, ow, layout, cptr(sc), cptr(sh), cptr(res),
                                                on.stream),
                  "wg2x2_conv_fwd_prepared_fused");
        }
    }
    return THPVariable_Wrap(Y);
    END_HANDLE_TH_ERRORS
}

// V, Wt, dY, mask, layout, relu, math, need_dV, need_dW
PyObject *py_conv_bwd(WG_ARGS)
{
    HANDLE_TH_ERRORS
    want(n, 9);
    const Tensor V = arg(a[0], "V"), Wt = arg(a[1], "Wt"), dY = arg(a[2], "dY"), mask = arg(a[3], "mask", true);
    const int layout = arg_int(a[4]);
    const bool relu = arg_bool(a[5]);
    const int math = arg_int(a[6]);
    const bool ndv = arg_bool(a[7]), ndw = arg_bool(a[8]);
    std::pair<Tensor, Tensor> r;
    { WG_NOGIL; r = conv_bwd(V, Wt, dY, mask, layout, relu, math, ndv, ndw); }
    PyObject *t = PyTuple_New(2);
    if (!t) throw python_error();
    PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(r.first));       // an undefined tensor wraps to None
    PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(r.second));
    return t;
    END_HANDLE_TH_ERRORS
}

// x, Wt, relu, layout, math, keep_V, out, workspace
PyObject *py_layer_fwd(WG_ARGS)
{
    HANDLE_TH_ERRORS
    want(n, 8);
    const Tensor x = arg(a[0], "x"), Wt = arg(a[1], "Wt");
    const bool relu = arg_bool(a[2]);
    const int layout = arg_int(a[3]), math = arg_int(a[4]);
    const bool keep = arg_bool(a[5]);
    const Img d = img_of(x, layout, "x");
    if (Wt.dim() != 3 || Wt.size(0) != 16 || Wt.size(1) != d.C) value_error("Wt must be (16, C, K)");
    const int64_t K = Wt.size(2);
    Tensor Y = arg_raw(a[6], "out"), V;
    const Tensor uws = arg_raw(a[7], "workspace");
    {
        WG_NOGIL;
        OnDevice on(x);
        if (!Y.defined()) Y = new_float(img_shape(d.B, d.H, d.W, K, layout), x);
        if (keep) V = new_float({16, d.B, (d.H + 1) / 2, (d.W + 1) / 2, d.C}, x);
        Scratch ws;
        void *wp;
        size_t wn;
        if (uws.defined()) { wp = uws.data_ptr(); wn = (size_t)uws.numel(); }
        else { ws.take(wg2x2_layer_fwd_workspace_bytes(d.B, d.H, d.W, d.C, K, math, keep)); wp = ws.get(); wn = ws.bytes; }
        check(wg2x2_layer_fwd(cptr(x), cptr(Wt), ptr(Y), ptr(V), d.B, d.H, d.W, d.C, K, layout, relu, math, wp, wn, on.stream), "wg2x2_layer_fwd");
    }
    if (!keep) return THPVariable_Wrap(Y);
    PyObject *t = PyTuple_New(2);
    if (!t) throw python_error();
    PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(Y));
    PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(V));
    return t;
    END_HANDLE_TH_ERRORS
}

// The scratch buffers of a layer call, taken here where the caller gives none (or too little)
struct LayerScratch {
    Scratch vs, ws;
    float *v = nullptr;
    void *w = nullptr;
    size_t wn = 0;
    LayerScratch(const Img &d, int64_t K, int layout, bool aligned, bool none, const Tensor &V, const Tensor &uws)
    {
        size_t nv = 0, nw = 0;
        if (!none) wg2x2_layer_fwd_prepared_scratch(d.B, d.H, d.W, d.C, K, layout, aligned, &nv, &nw);
        v = ptr(V);
        if (!v && nv) { vs.take(nv); v = static_cast<float *>(vs.get()); }
        if (nw) {
            if (uws.defined() && (size_t)uws.numel() >= nw) w = uws.data_ptr();
            else { ws.take(nw); w = ws.get(); }
            wn = nw;
        }
    }
};
bool on16(const Tensor &t) { return !t.defined() || (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) == 0; }

void layer_fwd_prepared(const Tensor &x, const Tensor &prep, const Tensor &Y, const Img &d, int64_t K, bool relu, int layout, const Tensor &in_scale,
                        const Tensor &in_shift, const Tensor &out_scale, const Tensor &out_shift, const Tensor &residual, bool residual_relu,
                        const Tensor &V, const Tensor &uws, void *stream)
{
    const bool apart = x.const_data_ptr<float>() + x.numel() <= Y.const_data_ptr<float>() || Y.const_data_ptr<float>() + Y.numel() <= x.const_data_ptr<float>();
    const bool xy = on16(x) && on16(Y) && apart, extras = on16(out_scale) && on16(out_shift) && on16(residual);
    // (Y over X needs V in between; extras off 16 bytes are the one-kernel layer's, or without the residual the cluster's and the pairs'; none
    // of them reads scratch.  C, K >= 256: refused off 16 bytes, by the path through scratch)
    const bool one_kernel = xy && !extras && (d.C < 256 || K < 256) && wg2x2_layer_fwd_fused_supported(d.B, d.H, d.W, d.C, K, layout);
    const bool own = xy && on16(residual) && (extras || d.C < 256 || K < 256);
    const int shortcut = !residual.defined() ? 0 : residual.data_ptr() == Y.data_ptr() ? 2 : 1;
    const bool none = one_kernel || (own && wg2x2_layer_fwd_pair_preferred_for(d.B, d.H, d.W, d.C, K, layout, in_scale.defined(), shortcut));
    const LayerScratch s(d, K, layout, own && on16(in_scale) && on16(in_shift), none, V, uws);
    check(wg2x2_layer_fwd_prepared_ex(cptr(x), cptr(in_scale), cptr(in_shift), prep.data_ptr(), ptr(Y), s.v, d.B, d.H, d.W, d.C, K, layout, relu,
                                      cptr(out_scale), cptr(out_shift), cptr(residual), residual_relu, s.w, s.wn, stream),
          "wg2x2_layer_fwd_prepared_ex");
}

// x, prepared, K, relu, layout, out, V_scratch, out_scale, out_shift, residual, workspace, in_scale, in_shift, residual_relu
PyObject *py_layer_fwd_prepared(WG_ARGS)
{
    HANDLE_TH_ERRORS
    want(n, 14);
    const Tensor x = arg(a[0], "x");
    const int layout = arg_int(a[4]);
    const Img d = img_of(x, layout, "x");
    const int64_t K = arg_int(a[2]);
    const Tensor prep = arg_prepared(a[1], d.C, K);
    const bool relu = arg_bool(a[3]);
    const auto ys = img_shape(d.B, d.H, d.W, K, layout);
    Tensor Y = arg_shaped(a[5], ys, "out");
    const Tensor sc = arg_shaped(a[7], {K}, "out_scale"), sh = arg_shaped(a[8], {K}, "out_shift"), res = arg_shaped(a[9], ys, "residual");
    const Tensor V = arg_shaped(a[6], {16, d.B, (d.H + 1) / 2, (d.W + 1) / 2, d.C}, "V_scratch");
    const Tensor uws = arg_raw(a[10], "workspace");
    const Tensor isc = arg_shaped(a[11], {d.C}, "in_scale"), ish = arg_shaped(a[12], {d.C}, "in_shift");
    const bool res_relu = arg_bool(a[13]);
    {
        WG_NOGIL;
        OnDevice on(x);
        if (!Y.defined()) Y = new_float(ys, x);
        layer_fwd_prepared(x, prep, Y, d, K, relu, layout, isc, ish, sc, sh, res, res_relu, V, uws, on.stream);
    }
    return THPVariable_Wrap(Y);
    END_HANDLE_TH_ERRORS
}

// x, shortcut, K, prepared_a, in_scale_a, in_shift_a, prepared_b, in_scale_b, in_shift_b, out_scale, out_shift, layout: the two
// layers of a residual block in one call.  The shortcut is added in place where there is one, else it is relu(x).
PyObject *py_residual_block(WG_ARGS)
{
    HANDLE_TH_ERRORS
    want(n, 12);
    const Tensor x = arg(a[0], "x");
    const int layout = arg_int(a[11]);
    const Img d = img_of(x, layout, "x");
    const int64_t K = arg_int(a[2]);
    const auto ys = img_shape(d.B, d.H, d.W, K, layout);
    const Tensor shortcut = arg_shaped(a[1], ys, "shortcut");
    if (!shortcut.defined() && d.C != K) value_error("a block that changes the channel count needs a shortcut");
    const Tensor pa = arg_prepared(a[3], d.C, K), pb = arg_prepared(a[6], K, K);
    const Tensor sa = arg_shaped(a[4], {d.C}, "in_scale_a"), ta = arg_shaped(a[5], {d.C}, "in_shift_a");
    const Tensor sb = arg_shaped(a[7], {K}, "in_scale_b"), tb = arg_shaped(a[8], {K}, "in_shift_b");
    const Tensor so = arg_shaped(a[9], {K}, "out_scale"), to = arg_shaped(a[10], {K}, "out_shift");
    Tensor y;
    {
        WG_NOGIL;
        OnDevice on(x);
        const Tensor mid = new_float(ys, x), none;
        layer_fwd_prepared(x, pa, mid, d, K, true, layout, sa, ta, none, none, none, false, none, none, on.stream);
        y = shortcut.defined() ? shortcut : new_float(ys, x);
        layer_fwd_prepared(mid, pb, y, Img{d.B, d.H, d.W, K}, K, true, layout, sb, tb, so, to, shortcut.defined() ? shortcut : x,
                           !shortcut.defined(), none, none, on.stream);
    }
    return THPVariable_Wrap(y);
    END_HANDLE_TH_ERRORS
}

// x (B,C,H,W), w (K,C) rounded to TF32 -> (B,K,H,W), or None where the kernel is not worth taking
PyObject *py_conv1x1(WG_ARGS)
{
    HANDLE_TH_ERRORS
    want(n, 2);
    const Tensor x = arg(a[0], "x"), w = arg(a[1], "w");
    const Img d = img_of(x, WG2X2_NCHW, "x");
    if (w.dim() < 2 || w.numel() != w.size(0) * d.C || w.size(1) != d.C) value_error("w must be (K, C)");
    if (!wg2x2_conv1x1_preferred(d.B, d.C, w.size(0), (int)(d.H * d.W)) || (reinterpret_cast<uintptr_t>(w.data_ptr()) & 15u)) Py_RETURN_NONE;
    Tensor y;
    {
        WG_NOGIL;
        OnDevice on(x);
        y = new_float({d.B, w.size(0), d.H, d.W}, x);
        check(wg2x2_conv1x1(cptr(x), cptr(w), ptr(y), d.B, d.C, w.size(0), (int)(d.H * d.W), on.stream), "wg2x2_conv1x1");
    }
    return THPVariable_Wrap(y);
    END_HANDLE_TH_ERRORS
}

// x (B,C,H,W) -> (B,C): mean of relu(x) over the pixels
PyObject *py_relu_mean(PyObject *, PyObject *o)
{
    HANDLE_TH_ERRORS
    const Tensor x = arg(o, "x");
    const Img d = img_of(x, WG2X2_NCHW, "x");
    Tensor y;
    {
        WG_NOGIL;
        OnDevice on(x);
        y = new_float({d.B, d.C}, x);
        check(wg2x2_relu_mean(cptr(x), ptr(y), d.B * d.C, (int)(d.H * d.W), on.stream), "wg2x2_relu_mean");
    }
    return THPVariable_Wrap(y);
    END_HANDLE_TH_ERRORS
}

// x, prepared, K, relu, out, out_scale, out_shift, residual, in_scale, in_shift
PyObject *py_layer_fwd_fused(WG_ARGS)
{
    HANDLE_TH_ERRORS
    want(n, 10);
    const Tensor x = arg(a[0], "x");
    const Img d = img_of(x, WG2X2_NCHW, "x");
    const int64_t K = arg_int(a[2]);
    const Tensor prep = arg_prepared(a[1], d.C, K);
    const bool relu = arg_bool(a[3]);
    const auto ys = img_shape(d.B, d.H, d.W, K, WG2X2_NCHW);
    Tensor Y = arg_shaped(a[4], ys, "out");
    const Tensor sc = arg_shaped(a[5], {K}, "out_scale"), sh = arg_shaped(a[6], {K}, "out_shift"), res = arg_shaped(a[7], ys, "residual");
    const Tensor isc = arg_shaped(a[8], {d.C}, "in_scale"), ish = arg_shaped(a[9], {d.C}, "in_shift");
    {
        WG_NOGIL;
        OnDevice on(x);
        if (!Y.defined()) Y = new_float(ys, x);
        if (!isc.defined() && !ish.defined())
            check(wg2x2_layer_fwd_fused(cptr(x), prep.data_ptr(), ptr(Y), d.B, d.H, d.W, d.C, K, relu, cptr(sc), cptr(sh), cptr(res), on.stream),
                  "wg2x2_layer_fwd_fused");
        else
            check(wg2x2_layer_fwd_fused_affine(cptr(x), prep.data_ptr(), ptr(Y), d.B, d.H, d.W, d.C, K, relu, cptr(isc), cptr(ish), cptr(sc),
                                               cptr(sh), cptr(res), on.stream),
                  "wg2x2_layer_fwd_fused_affine");
    }
    return THPVariable_Wrap(Y);
    END_HANDLE_TH_ERRORS
}

PyObject *pair_or_one(const Tensor &y, const Tensor &yr)
{
    if (!yr.defined()) return THPVariable_Wrap(y);
    PyObject *t = PyTuple_New(2);
    if (!t) throw python_error();
    PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(y));
    PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(yr));
    return t;
}

// x, with_relu, relu_scale, relu_shift
PyObject *py_maxpool(WG_ARGS)
{
    HANDLE_TH_ERRORS
    want(n, 4);
    if (!THPVariable_Check(a[0])) not_a_tensor("x");
    const Tensor x = THPVariable_Unpack(a[0]);
    const Img d = img_of(x, WG2X2_NCHW, "x");
    const bool nhwc = !x.is_contiguous() && x.is_contiguous(at::MemoryFormat::ChannelsLast) && x.is_cuda() && x.scalar_type() == at::kFloat;
    if (!nhwc) require(x, "x");
    const bool with_relu = arg_bool(a[1]);
    const Tensor sc = arg_shaped(a[2], {d.C}, "relu_scale"), sh = arg_shaped(a[3], {d.C}, "relu_shift");
    Tensor y, yr;
    {
        WG_NOGIL;
        OnDevice on(x);
        y = new_float({d.B, d.C, (d.H + 1) / 2, (d.W + 1) / 2}, x);
        if (with_relu) yr = new_float(y.sizes(), x);
        if (nhwc)
            check(wg2x2_maxpool3x3s2_same_nhwc_in(cptr(x), ptr(y), ptr(yr), cptr(sc), cptr(sh), d.B, d.C, d.H, d.W, on.stream),
                  "wg2x2_maxpool3x3s2_same_nhwc_in");
        else
            check(wg2x2_maxpool3x3s2_same(cptr(x), ptr(y), ptr(yr), cptr(sc), cptr(sh), d.B, d.C, d.H, d.W, on.stream), "wg2x2_maxpool3x3s2_same");
    }
    return pair_or_one(y, yr);
    END_HANDLE_TH_ERRORS
}

// x, prepared, with_relu, relu_scale, relu_shift (sizes checked by the caller)
PyObject *py_stem_pool(WG_ARGS)
{
    HANDLE_TH_ERRORS
    want(n, 5);
    const Tensor x = arg(a[0], "x");
    const Img d = img_of(x, WG2X2_NCHW, "x");
    const Tensor prep = arg_shaped(a[1], {(int64_t)wg2x2_stem_prepared_floats()}, "prepared");
    const bool with_relu = arg_bool(a[2]);
    const Tensor sc = arg_shaped(a[3], {64}, "relu_scale"), sh = arg_shaped(a[4], {64}, "relu_shift");
    Tensor y, yr;
    {
        WG_NOGIL;
        OnDevice on(x);
        y = new_float({d.B, 64, d.H / 4, d.W / 4}, x);
        if (with_relu) yr = new_float(y.sizes(), x);
        check(wg2x2_stem7x7s2_pool(cptr(x), cptr(prep), ptr(y), ptr(yr), cptr(sc), cptr(sh), d.B, d.H, d.W, on.stream), "wg2x2_stem7x7s2_pool");
    }
    return pair_or_one(y, yr);
    END_HANDLE_TH_ERRORS
}

// I, relu, layout: differentiable; NotImplemented while torch.jit.trace is on, which does not see native calls
PyObject *py_imtrans_op(WG_ARGS)
{
    HANDLE_TH_ERRORS
    want(n, 3);
    if (torch::jit::tracer::isTracing()) Py_RETURN_NOTIMPLEMENTED;
    if (!THPVariable_Check(a[0])) not_a_tensor("x");
    const Tensor I = THPVariable_Unpack(a[0]);
    const bool relu = arg_bool(a[1]);
    const int layout = arg_int(a[2]);
    Tensor V;
    { WG_NOGIL; V = imtrans_op(I, relu, layout); }
    return THPVariable_Wrap(V);
    END_HANDLE_TH_ERRORS
}

// I, W, out_h, out_w, layout, math, mask: differentiable in I and W; NotImplemented as above
PyObject *py_conv_op(WG_ARGS)
{
    HANDLE_TH_ERRORS
    want(n, 7);
    if (torch::jit::tracer::isTracing()) Py_RETURN_NOTIMPLEMENTED;
    if (!THPVariable_Check(a[0])) not_a_tensor("V");
    if (!THPVariable_Check(a[1])) not_a_tensor("Wt");
    const Tensor I = THPVariable_Unpack(a[0]), Wt = THPVariable_Unpack(a[1]);
    const int oh = arg_int_or(a[2], -1), ow = arg_int_or(a[3], -1), layout = arg_int(a[4]), math = arg_int(a[5]);
    Tensor Y;
    const Tensor mask = arg(a[6], "mask", true);
    { WG_NOGIL; Y = conv_op(I, Wt, mask, oh, ow, layout, math); }
    return THPVariable_Wrap(Y);
    END_HANDLE_TH_ERRORS
}

#define WG_FN(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"set_error", py_set_error, METH_O, nullptr},
    WG_FN("imtrans_fwd", py_imtrans_fwd),
    WG_FN("imtrans_bwd", py_imtrans_bwd),
    WG_FN("conv_fwd", py_conv_fwd),
    WG_FN("conv_fwd_prepared", py_conv_fwd_prepared),
    WG_FN("conv_bwd", py_conv_bwd),
    WG_FN("layer_fwd", py_layer_fwd),
    WG_FN("layer_fwd_prepared", py_layer_fwd_prepared),
    WG_FN("layer_fwd_fused", py_layer_fwd_fused),
    WG_FN("residual_block", py_residual_block),
    WG_FN("conv1x1", py_conv1x1),
    {"relu_mean", py_relu_mean, METH_O, nullptr},
    WG_FN("maxpool", py_maxpool),
    WG_FN("stem_pool", py_stem_pool),
    WG_FN("imtrans_op", py_imtrans_op),
    WG_FN("conv_op", py_conv_op),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native() { return PyModule_Create(&module); }
