// The differentiable layers of the training path (linear, embedding, RMSNorm, SwiGLU, SwiGLU MLP, cross-entropy,
// rotary split of the fused projection) as autograd functions in native code: shape checks, output allocation, the calls into
// libb200ops.so and the weight-gradient hand-over run without the interpreter. A layer's launches are
// a few microseconds of device time each at small sizes, and the interpreter's share of a forward and
// backward call was several times that: a linear layer of 256 x 768 x 256 took 148 us a pass through
// Python functions and ctypes, 70 us here, of which the kernels are 20.
//
// Weight gradients follow the convention of the Python side: a parameter that carries `main_grad` (a
// view of the flat gradient buffer) has its gradient written there, `grad_written` is set, and the
// parameter's `grad_ready` hook is called; other parameters receive an ordinary gradient.
#include <torch/extension.h>

#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/library.h>

#include <atomic>
#include <climits>

#include "b200ops.h"

namespace {

namespace py = pybind11;
using torch::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;

std::atomic<int64_t> g_launches{0};
PyObject* g_error = nullptr;   // the package's B200OpsError (a RuntimeError), looked up when the module is loaded

// Raises a Python exception with or without the interpreter lock: with it as error_already_set, without (in a
// layer's body, forward or on an autograd thread) in torch's own carrier.
[[noreturn]] void raise(PyObject* type, const std::string& what) {
  if (PyGILState_Check()) {
    PyErr_SetString(type, what.c_str());
    throw py::error_already_set();
  }
  py::gil_scoped_acquire gil;
  PyErr_SetString(type, what.c_str());
  python_error err;
  err.persist();
  throw err;
}
void require(bool ok, const char* what) {
  if (!ok) raise(PyExc_AssertionError, what);
}
// Rows of `width` elements; an empty row is the error that the division is in Python, not a signal.
int64_t rows_of(const Tensor& t, int64_t width) {
  if (width == 0) raise(PyExc_ZeroDivisionError, "the last dimension holds no element of a row");
  return t.numel() / width;
}
void check(int rc, const char* what) {
  if (rc != 0) raise(g_error, std::string(what) + " failed with code " + std::to_string(rc));
}
bool bf16_cuda(const Tensor& t) { return t.is_cuda() && t.scalar_type() == at::kBFloat16; }
// An incoming gradient as the kernels read it: contiguous and on a 16-byte boundary, whatever view it is.
Tensor rows16(const Tensor& g) {
  const Tensor c = g.contiguous();
  return reinterpret_cast<uintptr_t>(c.data_ptr()) % 16 ? c.clone() : c;
}
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// C[M,N] (+)= op(A) op(B); the checks of ops.gemm.gemm
void gemm(const Tensor& a, const Tensor& b, bool a_mn, bool b_mn, const Tensor& out, bool accumulate) {
  require(bf16_cuda(a) && bf16_cuda(b), "operands are bfloat16 CUDA tensors");
  require(a.dim() == 2 && b.dim() == 2 && a.stride(1) == 1 && b.stride(1) == 1, "operands are matrices with contiguous rows");
  const int64_t M = a.size(a_mn ? 1 : 0), K = a.size(a_mn ? 0 : 1), N = b.size(b_mn ? 1 : 0);
  require(b.size(b_mn ? 0 : 1) == K, "reduction dims differ");
  require(out.dim() == 2 && out.size(0) == M && out.size(1) == N && out.stride(1) == 1 &&
              (out.scalar_type() == at::kBFloat16 || out.scalar_type() == at::kFloat),
          "the output is an [M, N] bfloat16 or float32 matrix with contiguous rows");
  g_launches.fetch_add(1, std::memory_order_relaxed);
  check(b200_gemm_bf16(a.data_ptr(), b.data_ptr(), out.data_ptr(), static_cast<int>(M), static_cast<int>(N), static_cast<int>(K),
                       a.stride(0), b.stride(0), out.stride(0), a_mn, b_mn, out.scalar_type() == at::kFloat, accumulate, 0, 0,
                       stream()),
        "b200_gemm_bf16");
}

// dx = dy W and dw (+)= dy^T x, in one launch where that pays
void linear_grads(const Tensor& dy, const Tensor& x, const Tensor& w, const Tensor& dx, const Tensor& dw, bool accumulate) {
  if (dw.scalar_type() != at::kBFloat16) {   // a gradient buffer of 32 bits
    gemm(dy, w, false, true, dx, false);
    gemm(dy, x, true, true, dw, accumulate);
    return;
  }
  require(bf16_cuda(dy) && bf16_cuda(x) && bf16_cuda(w), "operands are bfloat16 CUDA tensors");
  require(dy.dim() == 2 && x.dim() == 2 && w.dim() == 2 && dy.stride(1) == 1 && x.stride(1) == 1 && w.stride(1) == 1,
          "operands are matrices with contiguous rows");
  const int64_t M = dy.size(0), N = dy.size(1), K = w.size(1);
  require(w.size(0) == N && x.size(0) == M && x.size(1) == K, "reduction dims differ");
  require(dw.is_cuda() && dw.dim() == 2 && dw.size(0) == N && dw.size(1) == K && dw.stride(1) == 1,
          "the output is an [M, N] bfloat16 or float32 matrix with contiguous rows");
  int launches = 2;
  const int rc = b200_linear_grads(dy.data_ptr(), x.data_ptr(), w.data_ptr(), dx.data_ptr(), dw.data_ptr(), static_cast<int>(M),
                                   static_cast<int>(N), static_cast<int>(K), dy.stride(0), x.stride(0), w.stride(0), dx.stride(0),
                                   dw.stride(0), accumulate, &launches, stream());
  g_launches.fetch_add(launches, std::memory_order_relaxed);
  check(rc, "b200_linear_grads");
}

PyObject* interned(const char* name) { return PyUnicode_InternFromString(name); }
PyObject* name_written() {
  static PyObject* const name = interned("grad_written");
  return name;
}

// An attribute, or nothing where there is none; needs the interpreter lock.
py::object attribute(const py::object& of, PyObject* name) {
  PyObject* v = PyObject_GetAttr(of.ptr(), name);
  if (!v) {
    if (!PyErr_ExceptionMatches(PyExc_AttributeError)) throw py::error_already_set();
    PyErr_Clear();
  }
  return py::reinterpret_steal<py::object>(v);
}

// Runs produce(out, accumulate) into weight.main_grad when the parameter has one (and returns an
// undefined tensor), else into a new tensor of the weight's shape.
template <class Produce>
Tensor write_param_grad(const Tensor& weight, Produce produce) {
  Tensor main;
  bool accumulate = false;
  {
    py::gil_scoped_acquire gil;
    static PyObject* const kMain = interned("main_grad");
    const py::object w = py::reinterpret_steal<py::object>(THPVariable_Wrap(weight));
    const py::object buffer = attribute(w, kMain);
    if (buffer && !buffer.is_none()) {
      const py::object written = attribute(w, name_written());
      const int truth = written ? PyObject_IsTrue(written.ptr()) : 0;
      if (truth < 0) throw py::error_already_set();
      accumulate = truth == 1;
      main = buffer.cast<Tensor>();
    }
  }
  if (!main.defined()) {
    const Tensor dw = at::empty_like(weight);
    produce(dw, false);
    return dw;
  }
  produce(main, accumulate);   // without the interpreter lock: a launch may wait for the GPU
  py::gil_scoped_acquire gil;
  static PyObject* const kReady = interned("grad_ready");
  const py::object w = py::reinterpret_steal<py::object>(THPVariable_Wrap(weight));
  if (PyObject_SetAttr(w.ptr(), name_written(), Py_True) != 0) throw py::error_already_set();
  const py::object ready = attribute(w, kReady);
  if (ready && !ready.is_none()) ready(w);
  return {};
}

// pybind's exception cannot cross the autograd engine's threads; torch's carrier can.
template <class F>
auto on_engine_thread(F f) {
  try {
    return f();
  } catch (py::error_already_set& e) {
    py::gil_scoped_acquire gil;
    e.restore();
    python_error err;
    err.persist();
    throw err;
  }
}

// y = x W^T
struct Linear : public Function<Linear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight) {
    ctx->save_for_backward({x, weight});
    require(x.dim() >= 1 && weight.dim() == 2, "x has a last dimension and the weight is a matrix");
    auto shape = x.sizes().vec();
    shape.back() = weight.size(0);
    // allocated with the final shape: a custom function must not return a view that it made, or later
    // in-place ops on the output are refused
    Tensor y = at::empty(shape, x.options().dtype(at::kBFloat16));
    gemm(x.reshape({-1, x.size(-1)}), weight, false, false, y.view({-1, weight.size(0)}), false);
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return on_engine_thread([&]() -> variable_list {
      const auto saved = ctx->get_saved_variables();
      const Tensor &x = saved[0], &weight = saved[1];
      const Tensor dy = grads[0].reshape({-1, grads[0].size(-1)}).contiguous();
      const Tensor x2 = x.reshape({-1, x.size(-1)});
      Tensor dx, dw;
      const bool want_dx = ctx->needs_input_grad(0);
      if (want_dx) dx = at::empty_like(x2, x2.options(), at::MemoryFormat::Contiguous);
      if (ctx->needs_input_grad(1))
        dw = write_param_grad(weight, [&](const Tensor& out, bool accumulate) {
          if (want_dx)
            linear_grads(dy, x2, weight, dx, out, accumulate);
          else
            gemm(dy, x2, true, true, out, accumulate);
        });
      else if (want_dx)
        gemm(dy, weight, false, true, dx, false);
      return {want_dx ? dx.view(x.sizes()) : dx, dw};
    });
  }
};

// Rows of the table by token id; the gradient is added up in the table's. What bounds a few hundred tokens is the host: a
// forward and backward pass of the two-layer model of 256 channels on 256 tokens takes 923 us, and took 1011 with this layer in
// Python (five processes of each in turn, within 2 %).
struct Embedding : public Function<Embedding> {
  static Tensor forward(AutogradContext* ctx, const Tensor& ids, const Tensor& table) {
    require(ids.scalar_type() == at::kLong && ids.is_contiguous() && (ids.is_cuda() || ids.is_pinned()),
            "ids are contiguous 64-bit integers that the GPU can read");
    require(bf16_cuda(table) && table.dim() == 2 && table.is_contiguous(), "the table is a contiguous bfloat16 CUDA matrix");
    ctx->save_for_backward({ids, table});
    const int64_t H = table.size(1);
    auto shape = ids.sizes().vec();
    shape.push_back(H);
    Tensor out = at::empty(shape, table.options());
    g_launches.fetch_add(1, std::memory_order_relaxed);
    check(b200_embedding_fwd(static_cast<const long long*>(ids.data_ptr()), table.data_ptr(), out.data_ptr(), ids.numel(),
                             static_cast<int>(H), stream()),
          "embedding_fwd");
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return on_engine_thread([&]() -> variable_list {
      const auto saved = ctx->get_saved_variables();
      const Tensor &ids = saved[0], &table = saved[1];
      const Tensor dout = rows16(grads[0]);
      return {Tensor(), write_param_grad(table, [&](const Tensor& out, bool accumulate) {
                require(bf16_cuda(out) && out.sizes() == table.sizes() && out.is_contiguous(),
                        "the table's gradient buffer is a contiguous bfloat16 CUDA matrix of its size");
                if (!accumulate) out.zero_();
                g_launches.fetch_add(1, std::memory_order_relaxed);
                check(b200_embedding_bwd(static_cast<const long long*>(ids.data_ptr()), dout.data_ptr(), out.data_ptr(), ids.numel(),
                                         static_cast<int>(table.size(1)), stream()),
                      "embedding_bwd");
              })};
    });
  }
};

// y = rmsnorm(h) * w with h = x (+ res), h a new tensor when there is a residual
struct RMSNorm : public Function<RMSNorm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const c10::optional<Tensor>& res, const Tensor& weight,
                               double eps) {
    const int64_t H = x.size(-1), T = rows_of(x, H);
    require(x.is_contiguous() && (!res || res->is_contiguous()), "x and the residual are contiguous");
    require(bf16_cuda(x) && (!res || (bf16_cuda(*res) && res->numel() == x.numel())),
            "x and the residual are bfloat16 CUDA tensors of one size");
    require(bf16_cuda(weight) && weight.is_contiguous() && weight.numel() == H, "the weight is a bfloat16 CUDA tensor of one row");
    Tensor y = at::empty_like(x), h = res ? at::empty_like(x) : x;
    Tensor rstd = at::empty({T}, x.options().dtype(at::kFloat));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    check(b200_rmsnorm_fwd(x.data_ptr(), res ? res->data_ptr() : nullptr, res ? h.data_ptr() : nullptr, weight.data_ptr(),
                           y.data_ptr(), rstd.data_ptr<float>(), static_cast<int>(T), static_cast<int>(H),
                           static_cast<float>(eps), stream()),
          "b200_rmsnorm_fwd");
    ctx->save_for_backward({h, weight, rstd});
    ctx->saved_data["res"] = res.has_value();
    if (res) return {y, h};
    return {y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return on_engine_thread([&]() -> variable_list {
      const auto saved = ctx->get_saved_variables();
      const Tensor &x = saved[0], &weight = saved[1], &rstd = saved[2];
      const bool has_res = ctx->saved_data["res"].toBool();
      const int64_t H = x.size(-1), T = rows_of(x, H);
      const Tensor dy = rows16(grads[0]);
      const Tensor dres = has_res ? rows16(grads[1]) : Tensor();
      Tensor dx = at::empty_like(x);
      const Tensor partial = at::empty({b200_rmsnorm_bwd_partial_rows(), H}, rstd.options());
      const Tensor dw = write_param_grad(weight, [&](const Tensor& out, bool accumulate) {
        require(bf16_cuda(out) && out.is_contiguous() && out.numel() == H, "the gradient buffer is a bfloat16 CUDA tensor of one row");
        g_launches.fetch_add(2, std::memory_order_relaxed);
        check(b200_rmsnorm_bwd(dy.data_ptr(), x.data_ptr(), weight.data_ptr(), rstd.data_ptr<float>(),
                               has_res ? dres.data_ptr() : nullptr, dx.data_ptr(), partial.data_ptr<float>(), out.data_ptr(),
                               accumulate, static_cast<int>(T), static_cast<int>(H), stream()),
              "b200_rmsnorm_bwd");
      });
      return {dx, has_res ? dx : Tensor(), dw, Tensor()};
    });
  }
};

// silu(gate) * up of a [..., 2F] tensor laid out as gate | up
struct SwiGLU : public Function<SwiGLU> {
  static Tensor forward(AutogradContext* ctx, const Tensor& gu) {
    const int64_t F = gu.size(-1) / 2, T = rows_of(gu, 2 * F);
    require(gu.is_contiguous(), "gate_up is contiguous");
    require(bf16_cuda(gu) && gu.size(-1) == 2 * F, "gate_up is a bfloat16 CUDA tensor with two halves");
    auto shape = gu.sizes().vec();
    shape.back() = F;
    Tensor out = at::empty(shape, gu.options());
    g_launches.fetch_add(1, std::memory_order_relaxed);
    check(b200_swiglu_fwd(gu.data_ptr(), out.data_ptr(), T, static_cast<int>(F), stream()), "swiglu_fwd");
    ctx->save_for_backward({gu});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return on_engine_thread([&]() -> variable_list {
      const auto saved = ctx->get_saved_variables();
      const Tensor& gu = saved[0];
      const int64_t F = gu.size(-1) / 2, T = rows_of(gu, 2 * F);
      const Tensor dout = rows16(grads[0]);
      Tensor dgu = at::empty_like(gu);
      g_launches.fetch_add(1, std::memory_order_relaxed);
      check(b200_swiglu_bwd(dout.data_ptr(), gu.data_ptr(), dgu.data_ptr(), T, static_cast<int>(F), stream()), "swiglu_bwd");
      return {dgu};
    });
  }
};

// The SwiGLU MLP of a decoder layer, gate over up in w_gu. One layer instead of three, so that the activation and its
// gradient ride in the products beside them.
struct SwiGLUMLP : public Function<SwiGLUMLP> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w_gu, const Tensor& w_down) {
    require(bf16_cuda(x) && bf16_cuda(w_gu) && bf16_cuda(w_down), "x and the weights are bfloat16 CUDA tensors");
    require(x.dim() >= 1 && w_gu.dim() == 2 && w_down.dim() == 2 && w_gu.is_contiguous() && w_down.is_contiguous(),
            "x has a last dimension and the weights are contiguous matrices");
    const int64_t F = w_down.size(1), K = w_gu.size(1);
    require(w_gu.size(0) == 2 * F && x.size(-1) == K, "the weights are [2F, hidden] and [out, F]");
    const Tensor x2 = x.reshape({-1, K});
    require(x2.stride(1) == 1, "x has contiguous rows");
    const int T = static_cast<int>(x2.size(0));
    const Tensor gu = at::empty({T, 2 * F}, x.options()), act = at::empty({T, F}, x.options());
    g_launches.fetch_add(b200_gemm_swiglu_launches(x2.data_ptr(), w_gu.data_ptr(), T, static_cast<int>(F), static_cast<int>(K), x2.stride(0)),
                         std::memory_order_relaxed);
    check(b200_gemm_swiglu(x2.data_ptr(), w_gu.data_ptr(), gu.data_ptr(), act.data_ptr(), T, static_cast<int>(F), static_cast<int>(K),
                           x2.stride(0), stream()),
          "b200_gemm_swiglu");
    auto shape = x.sizes().vec();
    shape.back() = w_down.size(0);
    Tensor y = at::empty(shape, x.options());
    gemm(act, w_down, false, false, y.view({-1, w_down.size(0)}), false);
    ctx->save_for_backward({x, w_gu, w_down, gu, act});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return on_engine_thread([&]() -> variable_list {
      const auto saved = ctx->get_saved_variables();
      const Tensor &x = saved[0], &w_gu = saved[1], &w_down = saved[2], &gu = saved[3], &act = saved[4];
      const Tensor dy = rows16(grads[0].reshape({-1, grads[0].size(-1)}));
      const int T = static_cast<int>(dy.size(0)), F = static_cast<int>(act.size(1)), H = static_cast<int>(dy.size(1));
      Tensor dgu, dx, dw_gu, dw_down;
      if (ctx->needs_input_grad(0) || ctx->needs_input_grad(1)) {
        const int launches = b200_gemm_swiglu_bwd_launches(dy.data_ptr(), w_down.data_ptr(), T, F, H, dy.stride(0));
        const Tensor scratch = launches == 1 ? Tensor() : at::empty_like(act);
        dgu = at::empty_like(gu);
        g_launches.fetch_add(launches, std::memory_order_relaxed);
        check(b200_gemm_swiglu_bwd(dy.data_ptr(), w_down.data_ptr(), gu.data_ptr(), dgu.data_ptr(),
                                   scratch.defined() ? scratch.data_ptr() : nullptr, T, F, H, dy.stride(0), stream()),
              "b200_gemm_swiglu_bwd");
      }
      if (ctx->needs_input_grad(2))
        dw_down = write_param_grad(w_down, [&](const Tensor& out, bool accumulate) { gemm(dy, act, true, true, out, accumulate); });
      const Tensor x2 = x.reshape({-1, x.size(-1)});
      const bool want_dx = ctx->needs_input_grad(0);
      if (want_dx) dx = at::empty_like(x2, x2.options(), at::MemoryFormat::Contiguous);
      if (ctx->needs_input_grad(1))
        dw_gu = write_param_grad(w_gu, [&](const Tensor& out, bool accumulate) {
          if (want_dx)
            linear_grads(dgu, x2, w_gu, dx, out, accumulate);
          else
            gemm(dgu, x2, true, true, out, accumulate);
        });
      else if (want_dx)
        gemm(dgu, w_gu, false, true, dx, false);
      return {want_dx ? dx.view(x.sizes()) : dx, dw_gu, dw_down};
    });
  }
};

// Whether the gradient that comes into the cross-entropy's backward pass is taken for one: `assume_unit_grad` of the Python class, which a
// program may clear at any time before the backward pass.
bool unit_grad_assumed() {
  py::gil_scoped_acquire gil;
  static PyObject* const module = py::module_::import("aws_ofi_nccl_b200.ops.llm").release().ptr();
  static PyObject *const cls_name = interned("_CrossEntropy"), *const flag_name = interned("assume_unit_grad");
  const py::object cls = attribute(py::reinterpret_borrow<py::object>(module), cls_name);
  const py::object flag = cls ? attribute(cls, flag_name) : py::object();
  const int truth = flag ? PyObject_IsTrue(flag.ptr()) : 1;
  if (truth < 0) throw py::error_already_set();
  return truth == 1;
}

// Mean cross-entropy of a matrix of logits, which are overwritten with its gradient: the backward pass hands them on. In Python this was
// 60 us of a forward and backward pass, 30 here: a head of 300 x 512 x 4096 takes 97 us for 130, the two-layer model of 256 channels on
// 256 tokens 860 for 970 (three processes of each in turn, within 5 %).
struct CrossEntropy : public Function<CrossEntropy> {
  static variable_list forward(AutogradContext* ctx, const Tensor& logits, const Tensor& targets) {
    if (logits.dim() != 2) raise(PyExc_ValueError, "the logits are a matrix");
    const int64_t T = logits.size(0), V = logits.size(1);
    require(logits.stride(1) == 1, "the logits have contiguous rows");
    if (T == 0) raise(PyExc_ZeroDivisionError, "the mean of no rows");
    require(bf16_cuda(logits), "the logits are a bfloat16 CUDA tensor");
    require(targets.scalar_type() == at::kLong && targets.is_contiguous() && targets.numel() >= T &&
                (targets.device() == logits.device() || targets.is_pinned()),
            "the targets are contiguous 64-bit integers that the GPU can read, one for every row");
    require(T <= INT_MAX && V <= INT_MAX, "rows and columns are numbers of 32 bits");
    const Tensor loss = at::empty({T}, logits.options().dtype(at::kFloat));
    g_launches.fetch_add(1, std::memory_order_relaxed);
    check(b200_cross_entropy(logits.data_ptr(), static_cast<const long long*>(targets.data_ptr()), loss.data_ptr<float>(), static_cast<int>(T),
                             static_cast<int>(V), logits.stride(0), static_cast<float>(1.0 / static_cast<double>(T)), stream()),
          "cross_entropy");
    ctx->save_for_backward({logits});
    ctx->mark_dirty({logits});
    // nobody differentiates through the overwritten logits: no zero-filled [T, V] gradient for them
    ctx->set_materialize_grads(false);
    return {loss.mean(), logits};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return on_engine_thread([&]() -> variable_list {
      const Tensor dlogits = ctx->get_saved_variables()[0];
      if (grads[1].defined())
        raise(PyExc_RuntimeError, "cross_entropy overwrites its logits with their gradient: nothing can be differentiated through them afterwards");
      if (!grads[0].defined()) return {Tensor(), Tensor()};   // the loss was not differentiated
      // the gradient is one in a training loop: no pass over all logits for it
      return {unit_grad_assumed() ? dlogits : dlogits * grads[0], Tensor()};
    });
  }
};

// q, k (rotated) and v as [B, S, heads, hd] tensors of their own from the fused projection [B*S, (nq+2nkv)*hd]
struct RopeQKV : public Function<RopeQKV> {
  static void launch(const Tensor& qkv, const Tensor (&part)[3], const Tensor& cos, const Tensor& sin, int64_t S, bool backward) {
    long long strides[9];
    for (int i = 0; i < 3; ++i)
      for (int d = 0; d < 3; ++d) strides[3 * i + d] = part[i].size(d) == 1 ? 0 : part[i].stride(d);   // no step, no alignment
    g_launches.fetch_add(1, std::memory_order_relaxed);
    check(b200_rope_qkv(qkv.data_ptr(), qkv.size(0) == 1 ? 0 : qkv.stride(0), part[0].data_ptr(), part[1].data_ptr(), part[2].data_ptr(), strides,
                        cos.data_ptr<float>(), sin.data_ptr<float>(), qkv.size(0), static_cast<int>(part[0].size(2)),
                        static_cast<int>(part[1].size(2)), static_cast<int>(part[0].size(3)), static_cast<int>(S), backward,
                        stream()),
          "rope_qkv");
  }
  static variable_list forward(AutogradContext* ctx, const Tensor& qkv, const Tensor& cos, const Tensor& sin, int64_t B, int64_t S,
                               int64_t nq, int64_t nkv, int64_t hd) {
    require(qkv.is_cuda() && qkv.scalar_type() == at::kBFloat16 && qkv.dim() == 2 && qkv.stride(1) == 1 && qkv.size(0) == B * S &&
                qkv.size(1) == (nq + 2 * nkv) * hd,
            "the projection is a [B*S, (nq+2nkv)*hd] bfloat16 CUDA matrix");
    require(cos.is_contiguous() && sin.is_contiguous() && cos.size(0) >= S && sin.size(0) >= S && cos.size(-1) == hd / 2 &&
                sin.size(-1) == hd / 2,
            "cos and sin are [>= S, hd/2] tables");
    const Tensor part[3] = {at::empty({B, S, nq, hd}, qkv.options()), at::empty({B, S, nkv, hd}, qkv.options()),
                            at::empty({B, S, nkv, hd}, qkv.options())};
    launch(qkv, part, cos, sin, S, false);
    ctx->save_for_backward({cos, sin});
    return {part[0], part[1], part[2]};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    return on_engine_thread([&]() -> variable_list {
      const auto saved = ctx->get_saved_variables();
      // attention returns its gradients as transposed views: any layout with contiguous heads is read in place
      auto rows = [](const Tensor& g) {
        const bool fits = g.stride(3) == 1 && g.stride(0) % 8 == 0 && g.stride(1) % 8 == 0 && g.stride(2) % 8 == 0 &&
                          reinterpret_cast<uintptr_t>(g.data_ptr()) % 16 == 0;
        return fits ? g : g.clone(at::MemoryFormat::Contiguous);
      };
      const Tensor part[3] = {rows(grads[0]), rows(grads[1]), rows(grads[2])};
      const int64_t B = part[0].size(0), S = part[0].size(1), hd = part[0].size(3);
      Tensor d = at::empty({B * S, (part[0].size(2) + 2 * part[1].size(2)) * hd}, part[0].options());
      launch(d, part, saved[0], saved[1], S, true);
      return {d, Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    });
  }
};

Tensor linear(const Tensor& x, const Tensor& w) { return Linear::apply(x, w); }
variable_list rmsnorm(const Tensor& x, const c10::optional<Tensor>& res, const Tensor& w, double eps) {
  return RMSNorm::apply(x, res, w, eps);
}
Tensor swiglu(const Tensor& gu) { return SwiGLU::apply(gu); }
Tensor embedding(const Tensor& ids, const Tensor& table) { return Embedding::apply(ids, table); }
Tensor swiglu_mlp(const Tensor& x, const Tensor& w_gu, const Tensor& w_down) { return SwiGLUMLP::apply(x, w_gu, w_down); }
variable_list cross_entropy(const Tensor& logits, const Tensor& targets) { return CrossEntropy::apply(logits, targets); }
variable_list rope_qkv(const Tensor& qkv, const Tensor& cos, const Tensor& sin, int64_t B, int64_t S, int64_t nq, int64_t nkv,
                       int64_t hd) {
  return RopeQKV::apply(qkv, cos, sin, B, S, nq, nkv, hd);
}

// The call itself, or under torch.jit.trace the operator of the same name: the tracer records operators,
// and of the bodies above it would see nothing but the allocation of their outputs.
template <class R, class... A, class... Args>
R traced_or_direct(const char* name, R (*fn)(A...), const Args&... args) {
  if (!torch::jit::tracer::isTracing()) return fn(args...);
  return c10::Dispatcher::singleton().findSchemaOrThrow(name, "").typed<R(A...)>().call(args...);
}

}  // namespace

TORCH_LIBRARY(b200ops, m) {
  m.def("linear(Tensor x, Tensor weight) -> Tensor", linear);
  m.def("embedding(Tensor ids, Tensor table) -> Tensor", embedding);
  m.def("rmsnorm(Tensor x, Tensor? res, Tensor weight, float eps) -> Tensor[]", rmsnorm);
  m.def("swiglu(Tensor gate_up) -> Tensor", swiglu);
  m.def("swiglu_mlp(Tensor x, Tensor w_gate_up, Tensor w_down) -> Tensor", swiglu_mlp);
  m.def("rope_qkv(Tensor qkv, Tensor cos, Tensor sin, int batch, int seq, int heads, int kv_heads, int head_dim) -> Tensor[]",
        rope_qkv);
}

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  g_error = py::object(py::module_::import("aws_ofi_nccl_b200.ops._lib").attr("B200OpsError")).release().ptr();
  // Like torch's own operators these run without the interpreter lock, which a launch into a full queue would
  // otherwise hold for as long as it waits; the wrapper takes exceptions back to Python.
  m.def("linear", torch::wrap_pybind_function_no_gil(
                      [](const Tensor& x, const Tensor& w) { return traced_or_direct("b200ops::linear", linear, x, w); }));
  m.def("embedding", torch::wrap_pybind_function_no_gil([](const Tensor& ids, const Tensor& table) {
          return traced_or_direct("b200ops::embedding", embedding, ids, table);
        }));
  m.def("rmsnorm", torch::wrap_pybind_function_no_gil(
                       [](const Tensor& x, const c10::optional<Tensor>& res, const Tensor& w, double eps) {
                         return traced_or_direct("b200ops::rmsnorm", rmsnorm, x, res, w, eps);
                       }));
  m.def("swiglu", torch::wrap_pybind_function_no_gil(
                      [](const Tensor& gu) { return traced_or_direct("b200ops::swiglu", swiglu, gu); }));
  m.def("swiglu_mlp", torch::wrap_pybind_function_no_gil([](const Tensor& x, const Tensor& w_gu, const Tensor& w_down) {
          return traced_or_direct("b200ops::swiglu_mlp", swiglu_mlp, x, w_gu, w_down);
        }));
  m.def("rope_qkv", torch::wrap_pybind_function_no_gil([](const Tensor& qkv, const Tensor& cos, const Tensor& sin, int64_t B, int64_t S,
                                                          int64_t nq, int64_t nkv, int64_t hd) {
          return traced_or_direct("b200ops::rope_qkv", rope_qkv, qkv, cos, sin, B, S, nq, nkv, hd);
        }));
  m.def("cross_entropy", torch::wrap_pybind_function_no_gil(cross_entropy));
  m.def("launches", [] { return g_launches.load(std::memory_order_relaxed); });
}
