// The host path of the operator's calls, in C++: argument checks, output and workspace tensors and the C-ABI call(s)
// of one forward or one incremental step.  The Python wrappers spend 40-60 us on the same work (a one-token step of
// eight streams keeps the GPU busy for 4 us); here it is 5-10 us.
//
// Every function returns None for anything but the plain case (host tensors, other types or geometries, wrong shapes):
// the Python wrapper then runs its general path, which also words the errors.  So nothing is decided here that the
// wrapper does not decide itself.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdlib>
#include <cstring>
#include <exception>

#include "race_b200.h"

namespace {

// tensors and parameters; subclasses take the general path, which gives their type back
const at::Tensor* tensor_of(PyObject* o) { return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr; }

// a contiguous CUDA tensor of one of the two element types
bool plain(const at::Tensor& t) {
    return t.is_cuda() && t.layout() == at::kStrided && t.is_contiguous() &&
           (t.scalar_type() == at::kFloat || t.scalar_type() == at::kBFloat16);
}
bool like(const at::Tensor& t, const at::Tensor& ref) {
    return plain(t) && t.scalar_type() == ref.scalar_type() && t.device() == ref.device() && t.sizes() == ref.sizes();
}
bool state_ok(const at::Tensor& t, const at::Tensor& ref, int64_t floats) {
    return t.is_cuda() && t.device() == ref.device() && t.scalar_type() == at::kFloat && t.is_contiguous() &&
           t.numel() == floats;
}
int dtype_of(const at::Tensor& t) { return t.scalar_type() == at::kFloat ? RACE_DTYPE_F32 : RACE_DTYPE_BF16; }

at::Tensor floats(std::initializer_list<int64_t> size, const at::Tensor& like) {
    return at::empty(at::IntArrayRef(size.begin(), size.size()), like.options().dtype(at::kFloat));
}
at::Tensor bytes(size_t n, const at::Tensor& like) {
    return at::empty({(int64_t)(n < 256 ? 256 : n)}, like.options().dtype(at::kByte));
}

// planes_T [d_k, L K] (any type, strides) -> the same in fp32 with the memory of rows, [L K, d_k]; usually the buffer is the
// transposed view of exactly that, and is returned as it is (a view of it would take a third of a microsecond of a step's six)
at::Tensor planes_rows(const at::Tensor& planes_T, const at::Tensor& ref) {
    if (planes_T.scalar_type() == at::kFloat && planes_T.device() == ref.device() && planes_T.layout() == at::kStrided &&
        planes_T.stride(0) == 1 && planes_T.stride(1) == planes_T.size(0))
        return planes_T;
    at::Tensor p = planes_T.t();
    if (p.device() != ref.device() || p.scalar_type() != at::kFloat)
        p = p.to(ref.options().dtype(at::kFloat));
    return p.contiguous().t();
}

// The kernels want 16-byte boundaries.  A contiguous tensor off them is refused by the C entries, except where this package
// has always copied it on the way: then it is copied here.
at::Tensor on_boundary(const at::Tensor& t, bool copies) {
    return copies && (reinterpret_cast<uintptr_t>(t.const_data_ptr()) & 15) ? t.clone() : t;
}

struct Fail : std::exception {
    std::string msg;
    explicit Fail(std::string m) : msg(std::move(m)) {}
    const char* what() const noexcept override { return msg.c_str(); }
};
void check(int rc, const char* what) {
    if (rc) throw Fail(std::string(what) + ": " + race_b200_error_string(rc) + " (code " + std::to_string(rc) + ")");
}
// with RACE_B200_CHECK_STATUS=1: synchronise and fail if a kernel gave up a bounded wait
void raise_on_wait(int* status, const char* what) {
    const char* e = std::getenv("RACE_B200_CHECK_STATUS");
    if (!e || std::strcmp(e, "1") != 0 || !status) return;
    int code = 0;
    if (cudaDeviceSynchronize() != cudaSuccess || cudaMemcpy(&code, status, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
        throw Fail(std::string(what) + ": " + cudaGetErrorString(cudaGetLastError()));
    if (code) {
        cudaMemset(status, 0, sizeof(int));
        throw Fail(std::string(what) + ": a bounded device-side wait ran out (code " + std::to_string(code) + ")");
    }
}

PyObject* none() { Py_RETURN_NONE; }

// Other Python threads run while a call allocates and launches (a full launch queue, or the synchronisation with
// RACE_B200_CHECK_STATUS=1, would hold them up), as they did when the calls went through ctypes.  No Python object may be
// touched meanwhile; hooks and modes of torch take the lock for themselves.
struct WithoutGil {
    PyThreadState* state = PyEval_SaveThread();
    WithoutGil() = default;
    WithoutGil(const WithoutGil&) = delete;
    ~WithoutGil() { PyEval_RestoreThread(state); }
};

// out, or (out, A [N,L,R], B [N,L,R,d_k]) as views of the packed state
PyObject* result(const at::Tensor& out, const at::Tensor& state, int64_t N, int64_t L, int64_t R, int64_t dk) {
    if (!state.defined()) return THPVariable_Wrap(out);
    const int64_t S = L * R, sf = S * (dk + 1);
    PyObject* o = THPVariable_Wrap(out);
    PyObject* a = THPVariable_Wrap(state.as_strided({N, L, R}, {sf, R, 1}, S * dk));
    PyObject* b = THPVariable_Wrap(state.as_strided({N, L, R, dk}, {sf, R * dk, dk, 1}, 0));
    return (o && a && b) ? Py_BuildValue("(NNN)", o, a, b) : nullptr;
}

// step(planes_T, K, V, Q, state, L, n_planes, eps) -> out | None
PyObject* step_impl(PyObject* const* args, Py_ssize_t nargs) {
    if (nargs != 8) throw Fail("step takes 8 arguments");
    const at::Tensor *pt = tensor_of(args[0]), *k = tensor_of(args[1]), *v = tensor_of(args[2]), *q = tensor_of(args[3]),
                     *st = tensor_of(args[4]);
    if (!pt || !k || !v || !q || !st || k->dim() != 5 || !plain(*k) || !like(*v, *k) || !like(*q, *k)) return none();
    const int64_t L = PyLong_AsLongLong(args[5]), P = PyLong_AsLongLong(args[6]);
    if (L < 1 || P < 1 || P > 12) return none();
    const int64_t MB = k->size(0) * k->size(1), T = k->size(2), H = k->size(3), dk = k->size(4), N = MB * H;
    RaceShape sh{N, T, (int32_t)L, (int32_t)(1 << P), (int32_t)dk, dtype_of(*k), (float)PyFloat_AsDouble(args[7]), (int32_t)H};
    if (pt->dim() != 2 || pt->size(0) != dk || pt->size(1) != L * P || !state_ok(*st, *k, N * (L << P) * (dk + 1)) ||
        N == 0 || T == 0 || !race_b200_decode_qkv_is_supported(&sh, (int)P))
        return none();
    at::Tensor out;
    {
        WithoutGil unlocked;
        c10::cuda::CUDAGuard guard(k->device());
        const at::Tensor planes = planes_rows(*pt, *k), va = on_boundary(*v, H > 1 && T > 1);
        out = at::empty(k->sizes(), k->options());
        float* state = st->data_ptr<float>();
        check(race_b200_decode_step_qkv(k->const_data_ptr(), va.const_data_ptr(), q->const_data_ptr(), planes.const_data_ptr<float>(),
                                        out.data_ptr(), state, state, &sh, (int)P, c10::cuda::getCurrentCUDAStream().stream()),
              "race_b200_decode_step_qkv");
    }
    return THPVariable_Wrap(out);
}

// forward(planes_T, K, V, Q, L, n_planes, eps, carry | None, return_state, fuse, status pointer) -> out | (out, A, B) | None
PyObject* forward_impl(PyObject* const* args, Py_ssize_t nargs) {
    if (nargs != 11) throw Fail("forward takes 11 arguments");
    const at::Tensor *pt = tensor_of(args[0]), *k = tensor_of(args[1]), *v = tensor_of(args[2]), *q = tensor_of(args[3]);
    const at::Tensor* carry = tensor_of(args[7]);
    if (!pt || !k || !v || !q || k->dim() != 5 || !plain(*k) || !like(*v, *k) || !like(*q, *k) ||
        (!carry && args[7] != Py_None))
        return none();
    const int64_t L = PyLong_AsLongLong(args[4]), P = PyLong_AsLongLong(args[5]);
    const bool want_state = args[8] == Py_True, fuse = args[9] == Py_True;
    if (L < 1 || P < 1 || P > 12) return none();
    const int64_t MB = k->size(0) * k->size(1), T = k->size(2), H = k->size(3), dk = k->size(4), N = MB * H, R = 1ll << P;
    RaceShape sh{N, T, (int32_t)L, (int32_t)R, (int32_t)dk, dtype_of(*k), (float)PyFloat_AsDouble(args[6]), (int32_t)H};
    if (pt->dim() != 2 || pt->size(0) != dk || pt->size(1) != L * P || N == 0 || T == 0 ||
        (carry && !state_ok(*carry, *k, N * L * R * (dk + 1))))
        return none();
    const bool qkv = fuse && race_b200_qkv_is_supported(&sh, (int)P);
    const size_t wb = qkv ? race_b200_causal_workspace_bytes(&sh, 0, RACE_VARIANT_TENSOR)
                          : race_b200_causal_heads_workspace_bytes(&sh);
    if (!qkv && !wb) return none();
    int* status = (int*)PyLong_AsVoidPtr(args[10]);
    at::Tensor out, state;
    {
        WithoutGil unlocked;
        c10::cuda::CUDAGuard guard(k->device());
        void* stream = c10::cuda::getCurrentCUDAStream().stream();
        const at::Tensor planes = planes_rows(*pt, *k);
        out = at::empty(v->sizes(), v->options());
        if (want_state) state = floats({N, L * R * (dk + 1)}, *k);
        const float* carry_p = carry ? carry->const_data_ptr<float>() : nullptr;
        float* state_p = want_state ? state.data_ptr<float>() : nullptr;
        at::Tensor ws = bytes(wb, *k);
        if (qkv) {
            check(race_b200_causal_fwd_qkv(q->const_data_ptr(), k->const_data_ptr(), v->const_data_ptr(), planes.const_data_ptr<float>(),
                                           out.data_ptr(), carry_p, state_p, ws.data_ptr(), wb, &sh, (int)P, 0, 0, stream, status),
                  "race_b200_causal_fwd_qkv");
        } else {
            at::Tensor pk = at::empty({N, T, L, R}, k->options()), pq = at::empty({N, T, L, R}, k->options());
            const at::Tensor va = on_boundary(*v, H > 1 && T > 1 && !race_b200_is_supported(&sh, RACE_VARIANT_AUTO));
            check(race_b200_bucket_probs_streams_pair(k->const_data_ptr(), q->const_data_ptr(), planes.const_data_ptr<float>(),
                                                      pk.data_ptr(), pq.data_ptr(), MB, T, (int32_t)H, (int32_t)dk, (int32_t)L,
                                                      (int32_t)P, sh.dtype, 0, stream),
                  "race_b200_bucket_probs_streams_pair");
            check(race_b200_causal_fwd_heads(pq.const_data_ptr(), pk.const_data_ptr(), va.const_data_ptr(), out.data_ptr(), carry_p,
                                             state_p, ws.data_ptr(), wb, &sh, stream, status),
                  "race_b200_causal_fwd_heads");
        }
        raise_on_wait(status, "BatchedACE.forward");
    }
    return result(out, state, N, L, R, dk);
}

// causal_prefix(probsQ, probsK, V [N,T,d_k], eps, carry | None, return_state, status pointer) -> out | (out, A, B) | None
PyObject* prefix_impl(PyObject* const* args, Py_ssize_t nargs) {
    if (nargs != 7) throw Fail("causal_prefix takes 7 arguments");
    const at::Tensor *pq = tensor_of(args[0]), *pk = tensor_of(args[1]), *v = tensor_of(args[2]), *carry = tensor_of(args[4]);
    if (!pq || !pk || !v || pk->dim() != 4 || v->dim() != 3 || !plain(*v) || !plain(*pk) || !like(*pq, *pk) ||
        pk->scalar_type() != v->scalar_type() || pk->device() != v->device() || (!carry && args[4] != Py_None))
        return none();
    const int64_t N = pk->size(0), T = pk->size(1), L = pk->size(2), R = pk->size(3), dk = v->size(2);
    const bool want_state = args[5] == Py_True;
    if (v->size(0) != N || v->size(1) != T || N == 0 || T == 0 || L < 1 || R < 1 || L * R > 4096 || dk < 1 || dk > 4096 ||
        (carry && !state_ok(*carry, *v, N * L * R * (dk + 1))))
        return none();
    RaceShape sh{N, T, (int32_t)L, (int32_t)R, (int32_t)dk, dtype_of(*v), (float)PyFloat_AsDouble(args[3]), 0};
    if (!race_b200_is_supported(&sh, RACE_VARIANT_AUTO)) return none();
    int* status = (int*)PyLong_AsVoidPtr(args[6]);
    at::Tensor out, state;
    {
        WithoutGil unlocked;
        c10::cuda::CUDAGuard guard(v->device());
        out = at::empty(v->sizes(), v->options());
        if (want_state) state = floats({N, L * R * (dk + 1)}, *v);
        const size_t wb = race_b200_causal_workspace_bytes(&sh, 0, RACE_VARIANT_AUTO);
        at::Tensor ws = bytes(wb, *v);
        check(race_b200_causal_fwd(pq->const_data_ptr(), pk->const_data_ptr(), v->const_data_ptr(), out.data_ptr(),
                                   carry ? carry->const_data_ptr<float>() : nullptr,
                                   want_state ? state.data_ptr<float>() : nullptr, ws.data_ptr(), wb, &sh, 0, RACE_VARIANT_AUTO,
                                   c10::cuda::getCurrentCUDAStream().stream(), status),
              "race_b200_causal_fwd");
        raise_on_wait(status, "race_b200_causal_fwd");
    }
    return result(out, state, N, L, R, dk);
}

// The operator with gradients for K, V and Q as one autograd node: producers, prefix forward; causal backward, producer
// backward.  Saved are the inputs and the two probability tensors.
struct TrainOp : torch::autograd::Function<TrainOp> {
    static RaceShape shape(const at::Tensor& k, int64_t L, int64_t P, double eps) {
        return RaceShape{k.size(0) * k.size(1) * k.size(3), k.size(2), (int32_t)L, (int32_t)(1 << P), (int32_t)k.size(4),
                         dtype_of(k), (float)eps, (int32_t)k.size(3)};
    }

    static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& k_in, const at::Tensor& v_in,
                              const at::Tensor& q_in, const at::Tensor& planes_in, int64_t L, int64_t P, double eps, int64_t status) {
        c10::cuda::CUDAGuard guard(k_in.device());
        void* stream = c10::cuda::getCurrentCUDAStream().stream();
        const RaceShape sh = shape(k_in, L, P, eps);
        const at::Tensor k = on_boundary(k_in, true), q = on_boundary(q_in, true), planes = on_boundary(planes_in, true),
                         v = on_boundary(v_in, sh.heads > 1 && sh.seq_len > 1);
        at::Tensor pk = at::empty({sh.n_streams, sh.seq_len, L, 1ll << P}, k.options()), pq = at::empty_like(pk);
        check(race_b200_bucket_probs_streams_pair(k.const_data_ptr(), q.const_data_ptr(), planes.const_data_ptr<float>(),
                                                  pk.data_ptr(), pq.data_ptr(), k.size(0) * k.size(1), sh.seq_len, sh.heads,
                                                  sh.head_dim, (int32_t)L, (int32_t)P, sh.dtype, 1, stream),
              "race_b200_bucket_probs_streams_pair");
        at::Tensor out = at::empty(v.sizes(), v.options());
        const size_t wb = race_b200_causal_heads_workspace_bytes(&sh);
        at::Tensor ws = bytes(wb, k);
        check(race_b200_causal_fwd_heads(pq.const_data_ptr(), pk.const_data_ptr(), v.const_data_ptr(), out.data_ptr(), nullptr,
                                         nullptr, ws.data_ptr(), wb, &sh, stream, (int*)status),
              "race_b200_causal_fwd_heads");
        raise_on_wait((int*)status, "BatchedACE.forward");
        ctx->save_for_backward({k, v, q, planes, pk, pq});
        ctx->saved_data["dims"] = std::vector<int64_t>{L, P, status};
        ctx->saved_data["eps"] = eps;
        return out;
    }

    static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        const auto dims = ctx->saved_data["dims"].toIntVector();
        const int64_t L = dims[0], P = dims[1];
        int* status = (int*)dims[2];
        torch::autograd::variable_list res(8);
        {
            at::AutoGradMode no_grad(false);
            c10::cuda::CUDAGuard guard(saved[0].device());
            // (hooks on saved tensors may hand back other memory: the kernels need dense rows)
            auto dense = [](const at::Tensor& t) { return on_boundary(t.contiguous(), true); };
            const at::Tensor k = dense(saved[0]), v = dense(saved[1]), q = dense(saved[2]), pk = dense(saved[4]), pq = dense(saved[5]);
            const at::Tensor planes = on_boundary(planes_rows(saved[3], k), true);
            void* stream = c10::cuda::getCurrentCUDAStream().stream();
            const RaceShape sh = shape(k, L, P, ctx->saved_data["eps"].toDouble());
            const at::Tensor g = on_boundary(grads[0].to(v.scalar_type()).contiguous(), true);   // may come expanded (stride 0)
            at::Tensor dpq = at::empty_like(pq), dpk = at::empty_like(pk), dv = at::empty(v.sizes(), v.options());
            const size_t wb = race_b200_causal_bwd_workspace_bytes(&sh);
            at::Tensor ws = bytes(wb, k);
            check(race_b200_causal_bwd_heads(pq.const_data_ptr(), pk.const_data_ptr(), v.const_data_ptr(), g.const_data_ptr(), nullptr,
                                             nullptr, dpq.data_ptr(), dpk.data_ptr(), dv.data_ptr(), nullptr, ws.data_ptr(), wb,
                                             &sh, stream, status),
                  "race_b200_causal_bwd_heads");
            const int64_t MB = k.size(0) * k.size(1);
            const at::Tensor* x[2] = {&k, &q};
            const at::Tensor* dp[2] = {&dpk, &dpq};
            for (int i = 0; i < 2; ++i)
                if (ctx->needs_input_grad(i ? 2 : 0)) res[i ? 2 : 0] = at::empty(x[i]->sizes(), x[i]->options());
            if (res[0].defined() && res[2].defined()) {
                check(race_b200_bucket_probs_streams_bwd_pair(k.const_data_ptr(), q.const_data_ptr(), planes.const_data_ptr<float>(),
                                                              dpk.const_data_ptr(), dpq.const_data_ptr(), res[0].data_ptr(),
                                                              res[2].data_ptr(), MB, sh.seq_len, sh.heads, sh.head_dim,
                                                              (int32_t)L, (int32_t)P, sh.dtype, stream),
                      "race_b200_bucket_probs_streams_bwd_pair");
            } else {
                for (int i = 0; i < 2; ++i)
                    if (res[i ? 2 : 0].defined())
                        check(race_b200_bucket_probs_streams_bwd(x[i]->const_data_ptr(), planes.const_data_ptr<float>(),
                                                                 dp[i]->const_data_ptr(), res[i ? 2 : 0].data_ptr(), MB, sh.seq_len,
                                                                 sh.heads, sh.head_dim, (int32_t)L, (int32_t)P, sh.dtype, stream),
                              "race_b200_bucket_probs_streams_bwd");
            }
            if (ctx->needs_input_grad(1)) res[1] = dv;
            raise_on_wait(status, "BatchedACE backward");
        }
        if (at::GradMode::is_enabled()) {   // the backward has no derivative of its own
            torch::autograd::variable_list first{res[0], res[1], res[2]};
            auto err = std::make_shared<torch::autograd::DelayedError>(
                "trying to differentiate twice a function that was marked with @once_differentiable", 3);
            for (auto& t : first)
                if (t.defined()) t.requires_grad_(true);
            first = (*err)(std::move(first));
            for (int i = 0; i < 3; ++i) res[i] = first[i];
        }
        return res;
    }
};

// train_forward(planes_T, K, V, Q, L, n_planes, eps, status pointer) -> out | None
PyObject* train_impl(PyObject* const* args, Py_ssize_t nargs) {
    if (nargs != 8) throw Fail("train_forward takes 8 arguments");
    const at::Tensor *pt = tensor_of(args[0]), *k = tensor_of(args[1]), *v = tensor_of(args[2]), *q = tensor_of(args[3]);
    if (!pt || pt->requires_grad() || !k || !v || !q || k->dim() != 5 || !plain(*k) || !like(*v, *k) || !like(*q, *k)) return none();
    const int64_t L = PyLong_AsLongLong(args[4]), P = PyLong_AsLongLong(args[5]);
    if (L < 1 || P < 1 || P > 12 || k->numel() == 0) return none();
    const double eps = PyFloat_AsDouble(args[6]);
    const RaceShape sh = TrainOp::shape(*k, L, P, eps);
    if (pt->dim() != 2 || pt->size(0) != sh.head_dim || pt->size(1) != L * P ||
        !race_b200_bucket_probs_bwd_is_supported(sh.head_dim, (int32_t)L, (int32_t)P, sh.dtype) ||
        !race_b200_causal_heads_workspace_bytes(&sh) || !race_b200_causal_bwd_workspace_bytes(&sh))
        return none();
    const int64_t status = (int64_t)PyLong_AsVoidPtr(args[7]);
    at::Tensor out;
    {
        WithoutGil unlocked;
        out = TrainOp::apply(*k, *v, *q, planes_rows(*pt, *k), L, P, eps, status);
    }
    return THPVariable_Wrap(out);
}

template <PyObject* (*kImpl)(PyObject* const*, Py_ssize_t)>
PyObject* guarded(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
    try {
        PyObject* r = kImpl(args, nargs);
        if (r && PyErr_Occurred()) {   // an argument that was not the number it should be
            Py_DECREF(r);
            return nullptr;
        }
        return r;
    } catch (python_error& e) {   // raised by a hook or a mode in Python: on as it is (a checkpoint ends its second run so)
        e.restore();
        if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, e.what());
    } catch (const c10::OutOfMemoryError& e) {
        PyObject* mod = PyImport_ImportModule("torch");   // raise the class torch's own allocations raise
        PyObject* cls = mod ? PyObject_GetAttrString(mod, "OutOfMemoryError") : nullptr;
        PyErr_Clear();
        PyErr_SetString(cls ? cls : PyExc_RuntimeError, e.what_without_backtrace());
        Py_XDECREF(cls);
        Py_XDECREF(mod);
    } catch (const c10::Error& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
    } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
    }
    return nullptr;
}

PyMethodDef kMethods[] = {
    {"step", (PyCFunction)(void (*)(void))guarded<step_impl>, METH_FASTCALL, nullptr},
    {"forward", (PyCFunction)(void (*)(void))guarded<forward_impl>, METH_FASTCALL, nullptr},
    {"train_forward", (PyCFunction)(void (*)(void))guarded<train_impl>, METH_FASTCALL, nullptr},
    {"causal_prefix", (PyCFunction)(void (*)(void))guarded<prefix_impl>, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&kModule); }
