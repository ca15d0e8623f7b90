// The autograd node of a layer call and its Python entry points.
//
// Why native: on a short sequence a call is nothing but launches.  Driving the C ABI from Python (ctypes structs, a dozen torch.empty
// calls, a Python autograd function) took 145 us per forward and 380 us per forward + backward of a 77- / 256-token call whose kernels
// need 45 / 120 us.  A C++ node has none of the checks of a Python autograd function: saved-tensor hooks, forward-mode AD and a second
// differentiation are seen to below.
#include <Python.h>

#include "layer.h"

#include <c10/cuda/CUDAGuard.h>
#include <pybind11/pybind11.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/edge.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/grad_mode.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <memory>
#include <string>

using namespace mkda_host;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

namespace {

// An error of the library is a mogankda_b200._lib.MkdaError, in the forward call and out of the autograd engine.  Called without the GIL.
template <typename F>
auto library_call(F f) {
    try {
        return f();
    } catch (const LibraryError& e) {
        pybind11::gil_scoped_acquire gil;
        PyObject* mod = PyImport_ImportModule("mogankda_b200._lib");
        PyObject* type = mod ? PyObject_GetAttrString(mod, "MkdaError") : nullptr;
        if (type) PyErr_SetString(type, e.what());
        Py_XDECREF(type);
        Py_XDECREF(mod);
        python_error err;
        err.persist();
        throw err;
    }
}

// Inputs and intermediates are saved as variables: in-place changes are detected, a second backward pass is refused once the buffers are gone,
// and saved-tensor hooks (activation checkpointing, offloading) get all of it.  The blocks that hold the intermediates may come back from a hook
// at another place: the pointers into them are taken again.
constexpr int NUM_INPUTS = 10;
struct DeltaRuleBackward : public torch::autograd::Node {
    Call call;
    SavedVariable vars[NUM_INPUTS];
    std::vector<SavedVariable> blocks;                     // saved->arena.keep
    std::vector<int64_t> block_bytes;
    std::unique_ptr<Saved> saved;

    std::string name() const override { return "DeltaRuleBackward"; }
    void release_variables() override {
        for (auto& v : vars) v.reset_data();
        for (auto& b : blocks) b.reset_data();
        saved.reset();
    }
    void save(std::unique_ptr<Saved> s) {
        saved = std::move(s);
        for (const Tensor& t : saved->arena.keep) {
            blocks.emplace_back(t, false);
            block_bytes.push_back(t.numel());
        }
        saved->arena.keep.clear();
    }
    variable_list apply(variable_list&& grads) override {
        std::lock_guard<std::mutex> lock(mutex_);
        Inputs in;
        Tensor* slots[NUM_INPUTS] = {&in.q, &in.k, &in.v, &in.x, &in.beta, &in.A_log, &in.dt_bias, &in.h0, &in.ep_w, &in.ep_gate};
        for (int i = 0; i < NUM_INPUTS; ++i) *slots[i] = vars[i].unpack();
        TORCH_CHECK(saved, torch::autograd::ERR_BACKWARD_TWICE);
        c10::cuda::CUDAGuard guard(call.dev);
        std::vector<Tensor>& keep = saved->arena.keep;
        struct Release { std::vector<Tensor>& t; ~Release() { t.clear(); } } release{keep};      // the saved variables hold the blocks
        for (size_t i = 0; i < blocks.size(); ++i) {
            const Tensor t = blocks[i].unpack();
            TORCH_CHECK(t.scalar_type() == at::kByte && t.numel() == block_bytes[i] && t.device() == call.dev,
                        "chunk_delta_rule: a saved-tensor hook returned another tensor than was saved");
            keep.push_back(aligned(t, 256));
        }
        saved->arena.point();
        const Tensor dy = grads[0], dht = grads.size() > 1 ? grads[1] : Tensor();
        const bool twice = c10::GradMode::is_enabled() && ((dy.defined() && dy.requires_grad()) || (dht.defined() && dht.requires_grad()));
        Grads g;
        {
            at::AutoGradMode off(false);
            g = library_call([&] {
                return run_backward(call, in, *saved, dy, dht, in.A_log.defined() && task_should_compute_output(5),
                                    in.dt_bias.defined() && task_should_compute_output(6), task_should_compute_output(7));
            });
        }
        variable_list out = {g.q, g.k, g.v, g.x, g.beta, g.A_log, g.dt_bias, g.h0, g.ep_w, g.ep_gate};
        for (int i = 0; i < NUM_INPUTS; ++i)
            if (!task_should_compute_output(i)) out[i] = Tensor();
        if (twice) {      // gradients of these gradients are not provided: using them has to fail, not to give zeros
            auto err = std::make_shared<torch::autograd::Error>("chunk_delta_rule: double backward is not supported", torch::autograd::edge_list());
            for (auto& t : out)
                if (t.defined()) torch::autograd::set_history(t, err);
        }
        return out;
    }
};

PyObject* fail(PyObject* type, const std::string& msg) {
    PyErr_SetString(type, msg.c_str());
    return nullptr;
}
#define REQUIRE(cond, msg) do { if (!(cond)) return fail(PyExc_AssertionError, msg); } while (0)

bool tensor_arg(PyObject* o, Tensor& t) {
    if (o == Py_None) return true;
    if (!THPVariable_Check(o)) { PyErr_Format(PyExc_TypeError, "expected a tensor, got %s", Py_TYPE(o)->tp_name); return false; }
    t = THPVariable_Unpack(o);
    return true;
}
const char NEED_CUDA[] = "mogankda_b200 kernels need CUDA tensors (there is no CPU fallback)";

// check(q, k, v, g, beta, initial_state, cu_seqlens) -> (B, T, HV, device index); raises what the call has to raise
PyObject* check(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 7) return fail(PyExc_TypeError, "check takes 7 arguments");
    Tensor q, k, v, g, beta, h0, cu;
    Tensor* t[7] = {&q, &k, &v, &g, &beta, &h0, &cu};
    for (int i = 0; i < 7; ++i) {
        if (!tensor_arg(a[i], *t[i])) return nullptr;
        if (i < 5 && !t[i]->defined()) return fail(PyExc_TypeError, "q, k, v, g and beta must be tensors");
    }
    if (!(q.is_cuda() && k.is_cuda() && v.is_cuda())) return fail(PyExc_RuntimeError, "mogankda_b200 runs on CUDA tensors only (no CPU fallback)");
    REQUIRE(q.scalar_type() == k.scalar_type() && q.scalar_type() == v.scalar_type(), "q, k, v must share a dtype");
    REQUIRE(q.scalar_type() == at::kBFloat16 || q.scalar_type() == at::kHalf || q.scalar_type() == at::kFloat, "q, k, v must be bfloat16, float16 or float32");
    REQUIRE(q.dim() == 4 && v.dim() == 4 && q.sizes() == k.sizes(), "q, k [B,T,HK,K]; v [B,T,HV,V]");
    REQUIRE(q.size(3) == 128 && v.size(3) == 128, "head dims must be 128");
    REQUIRE(v.size(0) == q.size(0) && v.size(1) == q.size(1), "q and v disagree on [B,T]");
    REQUIRE(q.size(2) > 0 && v.size(2) % q.size(2) == 0, "GVA needs HV % HK == 0");
    REQUIRE((g.dim() == 3 || (g.dim() == 4 && g.size(3) == 128)) && g.size(0) == v.size(0) && g.size(1) == v.size(1) && g.size(2) == v.size(2),
            "g must be [B,T,HV] or [B,T,HV,128]");
    REQUIRE(beta.dim() == 3 && beta.size(0) == v.size(0) && beta.size(1) == v.size(1) && beta.size(2) == v.size(2), "beta must be [B,T,HV]");
    int64_t rows = q.size(0);
    if (cu.defined()) {
        if (rows != 1)
            return fail(PyExc_ValueError, "The batch size is expected to be 1 rather than " + std::to_string(rows) + " when using `cu_seqlens`.");
        rows = cu.numel() - 1;
    }
    if (h0.defined()) {
        REQUIRE(h0.scalar_type() == at::kFloat, "initial_state must be float32");
        if (h0.dim() < 1 || h0.size(0) != rows)
            return fail(PyExc_ValueError, "The number of initial states is expected to be equal to the number of input sequences, i.e., " +
                                              std::to_string(rows) + " rather than " + std::to_string(h0.dim() ? h0.size(0) : 0) + ".");
        REQUIRE(h0.dim() == 4 && h0.size(1) == v.size(2) && h0.size(2) == 128 && h0.size(3) == 128, "initial_state must be [N,HV,128,128]");
    }
    return Py_BuildValue("(LLLi)", (long long)q.size(0), (long long)q.size(1), (long long)v.size(2), (int)q.device().index());
    END_HANDLE_TH_ERRORS
}

// check_params(v, g, A_log, dt_bias, norm weight, norm gate): the kernels take the sizes of these tensors from v and g, for reading them and
// for writing their gradients
PyObject* check_params(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 6) return fail(PyExc_TypeError, "check_params takes 6 arguments");
    Tensor v, g, alog, bias, w, gate;
    Tensor* t[6] = {&v, &g, &alog, &bias, &w, &gate};
    for (int i = 0; i < 6; ++i)
        if (!tensor_arg(a[i], *t[i])) return nullptr;
    const int64_t HV = v.size(2);
    REQUIRE(!alog.defined() || alog.numel() == HV, "A_log must have one element per v-head");
    REQUIRE(!bias.defined() || bias.numel() == (g.dim() == 3 ? HV : HV * 128), "dt_bias must have one element per v-head and, for a per-channel gate, key channel");
    REQUIRE(!w.defined() || w.numel() == 128, "the weight of the gated norm must have 128 elements");
    REQUIRE(!gate.defined() || gate.numel() == v.numel(), "the gate of the gated norm must have as many elements as v");
    Py_RETURN_NONE;
    END_HANDLE_TH_ERRORS
}

// layer(q, k, v, g, beta, A_log, dt_bias, initial_state, norm weight, norm gate, tables, (NC, NS, N, segmented, covers_all, longest, chain, few), scale, want_ht,
//       v_first, gate mode, lower bound or None, beta sigmoid, beta scale, l2, act or None, eps, warm-up threshold or None) -> (o, ht or None)
PyObject* layer(PyObject*, PyObject* const* a, Py_ssize_t n) {
    HANDLE_TH_ERRORS
    if (n != 23) return fail(PyExc_TypeError, "layer takes 23 arguments");
    Inputs in;
    Tensor* slots[NUM_INPUTS] = {&in.q, &in.k, &in.v, &in.x, &in.beta, &in.A_log, &in.dt_bias, &in.h0, &in.ep_w, &in.ep_gate};
    for (int i = 0; i < NUM_INPUTS; ++i)
        if (!tensor_arg(a[i], *slots[i])) return nullptr;
    Tensor tables;
    if (!tensor_arg(a[10], tables)) return nullptr;
    Call c;
    int seg, all;
    if (!PyArg_ParseTuple(a[11], "iiiiiiii", &c.NC, &c.NS, &c.N, &seg, &all, &c.longest, &c.chain, &c.few)) return nullptr;
    c.segmented = seg; c.covers_all = all;
    c.B = (int)in.q.size(0); c.T = (int)in.q.size(1); c.HK = (int)in.q.size(2); c.HV = (int)in.v.size(2); c.TT = c.B * c.T;
    c.dev = in.q.device();
    c.scale = (float)PyFloat_AsDouble(a[12]);
    c.want_ht = PyObject_IsTrue(a[13]); c.vf = PyObject_IsTrue(a[14]);
    c.mode = (int)PyLong_AsLong(a[15]);
    c.lower_bound = a[16] == Py_None ? -3.0e38f : (float)PyFloat_AsDouble(a[16]);
    c.beta_sigmoid = PyObject_IsTrue(a[17]); c.beta_scale = (float)PyFloat_AsDouble(a[18]); c.l2 = PyObject_IsTrue(a[19]);
    c.has_ep = a[20] != Py_None;
    c.act = c.has_ep ? (int)PyLong_AsLong(a[20]) : 0;
    c.eps = c.has_ep ? (float)PyFloat_AsDouble(a[21]) : 0.f;
    c.warm = a[22] != Py_None;
    c.warm_log2 = c.warm ? (float)(PyFloat_AsDouble(a[22]) * 1.4426950408889634) : 0.f;
    if (PyErr_Occurred()) return nullptr;
    c.scalar_gate = in.x.dim() == 3;
    c.qkv_dtype = dtype_code(in.q);
    dtype_code(in.x); dtype_code(in.beta);
    if (c.has_ep) {
        REQUIRE(in.ep_gate.defined(), "the gated norm needs a gate tensor");
        dtype_code(in.ep_gate);
        if (in.ep_w.defined()) dtype_code(in.ep_w);
    }
    for (Tensor* t : slots) {
        if (t->defined() && !t->is_cuda()) return fail(PyExc_RuntimeError, NEED_CUDA);
        // a node without a forward-mode formula would drop the tangent without a word
        if (t->defined() && t->_fw_grad(0).defined()) return fail(PyExc_NotImplementedError, "chunk_delta_rule: forward-mode AD is not supported");
    }
    c.set_tables(tables);

    Tensor out, ht;
    {
        pybind11::gil_scoped_release nogil;
        c10::cuda::CUDAGuard guard(c.dev);
        for (Tensor* t : {&in.q, &in.k, &in.v, &in.x, &in.beta, &in.ep_gate}) *t = aligned(*t);
        in.h0 = aligned(in.h0, 32);
        bool any = false;
        if (c10::GradMode::is_enabled())
            for (Tensor* t : slots) any = any || (t->defined() && t->requires_grad());
        auto saved = std::make_unique<Saved>();
        std::shared_ptr<DeltaRuleBackward> node;
        if (any) {
            node = std::shared_ptr<DeltaRuleBackward>(new DeltaRuleBackward(), torch::autograd::deleteNode);
            node->set_next_edges(torch::autograd::collect_next_edges(in.q, in.k, in.v, in.x, in.beta, in.A_log, in.dt_bias, in.h0, in.ep_w, in.ep_gate));
            for (int i = 0; i < NUM_INPUTS; ++i) node->vars[i] = SavedVariable(*slots[i], false);
        }
        {
            at::AutoGradMode off(false);
            // Running sequences continued by a handful of tokens, nothing to differentiate: the recurrence itself is cheaper than a 64-row chunk
            // (step.cu).  The choice is made for each sequence by itself, so that its results do not depend on what else is in the batch: in
            // a mixed batch the steps go over the chunk kernels' results.  Sequences that start from zero keep to the chunk algebra, whose results
            // for a prefix of a sequence are those of the whole sequence bit for bit.
            const bool steps = !any && in.h0.defined();
            library_call([&] {
                if (!steps || c.longest > MKDA_STEP_MAX_TOKENS) std::tie(out, ht) = run_forward(c, in, any, *saved);
                if (steps && (!out.defined() || c.few)) run_step(c, in, out, ht);
            });
        }
        if (any) {
            node->call = c;
            node->save(std::move(saved));
            torch::autograd::set_history(out, node);
            if (ht.defined()) torch::autograd::set_history(ht, node);
        }
    }
    PyObject* po = THPVariable_Wrap(out);
    if (!po) return nullptr;
    PyObject* ph = Py_None;
    if (ht.defined()) ph = THPVariable_Wrap(ht);
    else Py_INCREF(ph);
    PyObject* res = ph ? PyTuple_Pack(2, po, ph) : nullptr;
    Py_DECREF(po);
    Py_XDECREF(ph);
    return res;
    END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"check", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(check)), METH_FASTCALL, "argument checks of a call"},
    {"check_params", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(check_params)), METH_FASTCALL, "sizes of the parameter tensors"},
    {"layer", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(layer)), METH_FASTCALL, "one layer call"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "host path of a layer call over libmkda", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() {
#define MKDA_SIZE(S) (int)sizeof(S),
    const int built[] = {MKDA_STRUCTS(MKDA_SIZE)};
    constexpr int n = sizeof(built) / sizeof(built[0]);
    int have[n];
    if (mkda_struct_sizes(have, n) != n || !std::equal(have, have + n, built)) {
        PyErr_SetString(PyExc_ImportError, "_host.so and libmkda.so were built from different include/mkda.h (struct sizes differ): rebuild with "
                                           "`python -m mogankda_b200.build --force`");
        return nullptr;
    }
    return PyModule_Create(&module);
}
