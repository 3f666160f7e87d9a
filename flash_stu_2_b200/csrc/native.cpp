// The C-ABI of include/stu_b200.h as functions of a Python extension module, and the two calls that every layer makes most, the
// linear layer and the norm, from tensors in one step.  A launch through ctypes costs 4 us of argument conversion and 5 more of
// checks in the interpreter, as much as the launch itself; token steps of small batches and short prefills are bound by that.
//
// Arguments are positional.  A pointer parameter takes a CUDA tensor (its first element), an address or None.  The lock of the
// interpreter is released around the call.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <atomic>
#include <stdexcept>
#include <tuple>
#include <utility>

#include "../../include/stu_b200.h"

namespace {

struct BadArgument : std::runtime_error {
  using std::runtime_error::runtime_error;
};

template <typename T> T value_of(PyObject* o);
template <> long long value_of<long long>(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw BadArgument("");
  return v;
}
template <> int value_of<int>(PyObject* o) {
  const long long v = value_of<long long>(o);
  if (v != (int)v) {
    PyErr_SetString(PyExc_OverflowError, "an int argument does not fit 32 bits");
    throw BadArgument("");
  }
  return (int)v;
}
template <> float value_of<float>(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw BadArgument("");
  return (float)v;
}
void* address_of(PyObject* o) {
  if (o == Py_None) return nullptr;
  if (THPVariable_Check(o)) {
    const at::Tensor& t = THPVariable_Unpack(o);
    if (!t.is_cuda()) {
      PyErr_SetString(PyExc_RuntimeError, "flash_stu_2_b200 has no CPU path: tensors must live on a CUDA device");
      throw BadArgument("");
    }
    return t.data_ptr();
  }
  void* p = PyLong_AsVoidPtr(o);
  if (!p && PyErr_Occurred()) throw BadArgument("");
  return p;
}
template <typename T> struct Convert {
  static T from(PyObject* o) { return value_of<T>(o); }
};
template <typename T> struct Convert<T*> {
  static T* from(PyObject* o) { return static_cast<T*>(const_cast<typename std::remove_const<T>::type*>(
      static_cast<const T*>(address_of(o)))); }
};

template <auto F> struct Call;
template <typename R, typename... A, R (*F)(A...)> struct Call<F> {
  template <size_t... I>
  static R run(PyObject* const* args, std::index_sequence<I...>) {
    std::tuple<A...> a{Convert<A>::from(args[I])...};
    R r;
    Py_BEGIN_ALLOW_THREADS
    r = F(std::get<I>(a)...);
    Py_END_ALLOW_THREADS
    return r;
  }
  static PyObject* call(PyObject*, PyObject* const* args, Py_ssize_t n) {
    if (n != (Py_ssize_t)sizeof...(A)) {
      PyErr_Format(PyExc_TypeError, "%zd arguments expected, %zd given", (Py_ssize_t)sizeof...(A), n);
      return nullptr;
    }
    try {
      return PyLong_FromLongLong((long long)run(args, std::make_index_sequence<sizeof...(A)>()));
    } catch (const BadArgument&) {
      return nullptr;
    } catch (const std::exception& e) {
      PyErr_SetString(PyExc_RuntimeError, e.what());
      return nullptr;
    }
  }
};

// Devices whose status word has been registered (ops.status_word)
std::atomic<unsigned long long> g_ready{0};
PyObject* status_ready(PyObject*, PyObject* const* args, Py_ssize_t n) {
  const long dev = n == 1 ? PyLong_AsLong(args[0]) : -1;
  if (dev < 0 || dev >= 64) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "a device index is expected");
    return nullptr;
  }
  g_ready.fetch_or(1ull << dev);
  Py_RETURN_NONE;
}

int dtype_code(const at::Tensor& t) {
  return t.scalar_type() == at::kBFloat16 ? 1 : t.scalar_type() == at::kFloat ? 0 : -1;
}
// A plain CUDA tensor or None (null); anything else: the caller's other path decides.
bool plain(PyObject* o, const at::Tensor** t) {
  *t = nullptr;
  if (o == Py_None) return true;
  if (!THPVariable_Check(o)) return false;
  *t = &THPVariable_Unpack(o);
  return (*t)->is_cuda();
}
void* data_of(const at::Tensor* t) { return t ? t->data_ptr() : nullptr; }

// A CUDA error (rc > 0) raises as _lib.check does: the kernel may have gone out all the same (the error can be one that an earlier
// call left behind), so the call must not be made a second time.  Refusals (rc < 0) come before any launch.
bool raised(int rc, const char* what) {
  if (rc <= 0) return false;
  PyErr_Format(PyExc_RuntimeError, "%s: CUDA error %d", what, rc);
  return true;
}

// K from which the layers let a product's K be cut (stu_linear_split): the contractions of all filters' features (filters * d), not an MLP's.  A cut sum is
// rounded other than one chain, and how K is cut depends on the rows of the call: with it a model drew other tokens in another batch or a prefill in chunks
// (28 prompts of 1033 tokens, 512 channels: 3 of 1036), for 1 % of a prefill.
constexpr long long CUT_K = 16384;

// linear(x, W, W2, resid, out, epilogue, norm_w, eps, backend, transposed, hist_T, hist_t0, hist_Lh) -> y, or (y,) where K was cut
// and there were two launches, or None where a check fails or the library refuses: ops.linear then goes through its own checks, which raise what they raise.
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 13) {
    PyErr_SetString(PyExc_TypeError, "13 arguments expected");
    return nullptr;
  }
  try {
    const at::Tensor *x, *W, *W2, *resid, *out, *norm_w;
    if (!plain(args[0], &x) || !plain(args[1], &W) || !plain(args[2], &W2) || !plain(args[3], &resid) || !plain(args[4], &out) ||
        !plain(args[6], &norm_w) || !x || !W)
      Py_RETURN_NONE;
    const int epi = value_of<int>(args[5]), code = dtype_code(*x), dev = x->device().index();
    if (code < 0 || x->dim() != 2 || W->dim() != 2 || x->stride(1) != 1 || !(g_ready.load(std::memory_order_relaxed) >> dev & 1))
      Py_RETURN_NONE;
    const long long M = x->size(0), K = x->size(1);
    const bool transposed = value_of<int>(args[9]) != 0;
    if (W->size(transposed ? 0 : 1) != K) Py_RETURN_NONE;
    const long long N = W->size(transposed ? 1 : 0), w_rs = W->stride(transposed ? 1 : 0), w_ks = W->stride(transposed ? 0 : 1);
    if (M > INT32_MAX || N > INT32_MAX || K > INT32_MAX) Py_RETURN_NONE;
    if (W2 && (W2->sizes() != W->sizes() || W2->strides() != W->strides())) Py_RETURN_NONE;
    if (resid && (resid->dim() != 2 || resid->size(0) != M || resid->size(1) != N || resid->stride(1) != 1)) Py_RETURN_NONE;
    const bool hist = (epi & 0xff) == 3;
    at::Tensor made;
    long long y_rs = 0;
    if (hist) {
      if (!out) Py_RETURN_NONE;
    } else {
      if (!out) {
        made = at::empty({M, N}, x->options());
        out = &made;
      }
      if (out->dim() != 2 || out->size(0) != M || out->size(1) != N || out->stride(1) != 1) Py_RETURN_NONE;
      y_rs = out->stride(0);
    }
    const float eps = value_of<float>(args[7]);
    const int backend = value_of<int>(args[8]), hT = value_of<int>(args[10]), ht0 = value_of<int>(args[11]), hLh = value_of<int>(args[12]);
    void *px = data_of(x), *pW = data_of(W), *pW2 = data_of(W2), *pr = data_of(resid), *py = data_of(out), *pn = data_of(norm_w);
    const long long lda = x->stride(0), r_rs = resid ? resid->stride(0) : 0;
    void* stream = (void*)c10::cuda::getCurrentCUDAStream().stream();
    // backends that may come to the tcgen05 GEMM: 0 and 2
    const long long parts = K >= CUT_K && (backend == 0 || backend == 2) ? stu_linear_workspace_elems((int)M, (int)N, (int)K, epi, code) : 0;
    at::Tensor workspace;
    if (parts > 0) workspace = at::empty({parts}, x->options().dtype(at::kFloat));
    float* pw = parts > 0 ? workspace.data_ptr<float>() : nullptr;
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = stu_linear_split(px, lda, pW, w_rs, w_ks, pW2, pr, r_rs, py, y_rs, (int)M, (int)N, (int)K, epi, hT, ht0, hLh, pn, eps, code, backend, pw, parts, stream);
    Py_END_ALLOW_THREADS
    if (raised(rc, "stu_linear")) return nullptr;
    if (rc != 0) Py_RETURN_NONE;
    PyObject* y = made.defined() ? THPVariable_Wrap(std::move(made)) : Py_NewRef(args[4]);
    if (parts > 0 && y && stu_linear_launches() == 2) {
      PyObject* pair = PyTuple_Pack(1, y);
      Py_DECREF(y);
      y = pair;
    }
    return y;
  } catch (const BadArgument&) {
    PyErr_Clear();
  } catch (const std::exception&) {
  }
  Py_RETURN_NONE;
}

// rmsnorm(x, weight, eps) -> y, or None as above.
PyObject* rmsnorm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 3) {
    PyErr_SetString(PyExc_TypeError, "3 arguments expected");
    return nullptr;
  }
  try {
    const at::Tensor *x, *w;
    if (!plain(args[0], &x) || !plain(args[1], &w) || !x || !w) Py_RETURN_NONE;
    const int code = dtype_code(*x);
    if (code < 0 || x->dim() < 1 || !x->is_contiguous() || x->numel() == 0) Py_RETURN_NONE;
    const long long d = x->size(-1), rows = x->numel() / d;
    if (rows > INT32_MAX || d > INT32_MAX) Py_RETURN_NONE;
    at::Tensor y = at::empty(x->sizes(), x->options());
    void *px = data_of(x), *pw = data_of(w), *py = y.data_ptr(), *stream = (void*)c10::cuda::getCurrentCUDAStream().stream();
    const float eps = value_of<float>(args[2]);
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = stu_rmsnorm(px, pw, py, (int)rows, (int)d, d, d, eps, code, stream);
    Py_END_ALLOW_THREADS
    if (raised(rc, "stu_rmsnorm")) return nullptr;
    if (rc == 0) return THPVariable_Wrap(std::move(y));
  } catch (const BadArgument&) {
    PyErr_Clear();
  } catch (const std::exception&) {
  }
  Py_RETURN_NONE;
}

// layer_step_f32(x, norm_w, MinT, hist, taps, pos, mid, mlp_norm_w, gate, up, down, eps, mlp_eps, decode_flags, gate_flags, down_flags,
// status): one cached token of an approx layer in fp32, three launches: mid = x + STU(norm(x)); x = mid + MLP(norm(mid)).  Returns 3,
// or 1 where the MLP was refused (mid is done; its kernels write nothing that they read, so the caller may run both again), or None
// where nothing was launched.
PyObject* layer_step_f32(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 17) {
    PyErr_SetString(PyExc_TypeError, "17 arguments expected");
    return nullptr;
  }
  try {
    const at::Tensor* t[11];
    for (int i = 0; i < 11; i++)
      if (!plain(args[i], &t[i]) || !t[i] || !t[i]->is_contiguous() || t[i]->device() != t[0]->device() ||
          t[i]->scalar_type() != (i == 5 ? at::kInt : at::kFloat))
        Py_RETURN_NONE;
    const at::Tensor &x = *t[0], &hist = *t[3], &gate = *t[8];
    const int dev = x.device().index();
    if (x.dim() != 2 || hist.dim() != 4 || gate.dim() != 2 || dev != c10::cuda::current_device() ||
        !(g_ready.load(std::memory_order_relaxed) >> dev & 1))
      Py_RETURN_NONE;
    const int64_t B = x.size(0), d = x.size(1), Lh = hist.size(3), I = gate.size(0);
    const auto is = [&](int i, at::IntArrayRef want) { return t[i]->sizes() == want; };
    if (B < 1 || B > INT32_MAX || d > INT32_MAX || I > INT32_MAX || Lh > INT32_MAX || !is(1, {d}) || !is(2, {d, d}) || !is(3, {B, d, 2, Lh}) ||
        !is(4, {d, Lh}) || !is(5, {B, 2}) || !is(6, {B, d}) || !is(7, {d}) || !is(8, {I, d}) || !is(9, {I, d}) || !is(10, {d, I}) ||
        x.data_ptr() == t[6]->data_ptr())
      Py_RETURN_NONE;
    const float eps = value_of<float>(args[11]), mlp_eps = value_of<float>(args[12]);
    const int decode_flags = value_of<int>(args[13]), gate_flags = value_of<int>(args[14]), down_flags = value_of<int>(args[15]);
    int* status = static_cast<int*>(address_of(args[16]));
    const at::Tensor h = at::empty({B, I}, x.options());
    void* p[11];
    for (int i = 0; i < 11; i++) p[i] = t[i]->data_ptr();
    void *ph = h.data_ptr(), *stream = (void*)c10::cuda::getCurrentCUDAStream().stream();
    int rc, done = 0;
    Py_BEGIN_ALLOW_THREADS
    rc = stu_decode_approx(p[0], d, p[1], p[2], p[3], p[4], nullptr, (int*)p[5], p[6], d, (int)B, (int)d, (int)Lh, eps, status, decode_flags,
                           stream);
    if (rc == 0) {
      done = 1;
      rc = stu_linear(p[6], d, p[8], d, 1, p[9], nullptr, 0, ph, I, (int)B, (int)I, (int)d, 2 | gate_flags, 0, 0, 0, p[7], mlp_eps, 0, 0, stream);
    }
    if (rc == 0)
      rc = stu_linear(ph, I, p[10], I, 1, nullptr, p[6], d, p[0], d, (int)B, (int)d, (int)I, 1 | down_flags, 0, 0, 0, nullptr, 0.f, 0, 0, stream);
    Py_END_ALLOW_THREADS
    if (raised(rc, "layer_step_f32")) return nullptr;
    if (rc == 0) done = 3;
    if (done) return PyLong_FromLong(done);
  } catch (const BadArgument&) {
    PyErr_Clear();
  } catch (const std::exception&) {
  }
  Py_RETURN_NONE;
}

// layer_prefill(x, norm_w, MinT, hist, taps, pos, mlp_norm_w, gate, up, down, eps, mlp_eps, t0, fresh, kind, status): new positions of an
// approx layer, in place on x [B, T, d]: x += STU(norm(x)); x += MLP(norm(x)), seven launches.  kind and taps as in
// stu_conv_prefill_positions; pos may be None.  Returns 3 (7: the last product took two launches), or 1 where the MLP was refused (the STU
// is done), or None where the STU was (x is as it was, and so are the positions).
PyObject* layer_prefill(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 16) {
    PyErr_SetString(PyExc_TypeError, "16 arguments expected");
    return nullptr;
  }
  try {
    const at::Tensor* t[10];
    for (int i = 0; i < 10; i++) {
      if (!plain(args[i], &t[i]) || (!t[i] && i != 5)) Py_RETURN_NONE;
      if (t[i] && (!t[i]->is_contiguous() || t[i]->device() != t[0]->device() || t[i]->scalar_type() != (i == 5 ? at::kInt : t[0]->scalar_type())))
        Py_RETURN_NONE;
    }
    const at::Tensor &x = *t[0], &hist = *t[3], &gate = *t[7];
    const int dev = x.device().index(), code = dtype_code(x);
    if (code < 0 || x.dim() != 3 || x.numel() == 0 || hist.dim() != 4 || gate.dim() != 2 || dev != c10::cuda::current_device() ||
        !(g_ready.load(std::memory_order_relaxed) >> dev & 1))
      Py_RETURN_NONE;
    const int64_t B = x.size(0), T = x.size(1), d = x.size(2), Lh = hist.size(3), I = gate.size(0);
    const float eps = value_of<float>(args[10]), mlp_eps = value_of<float>(args[11]);
    const int t0 = value_of<int>(args[12]), fresh = value_of<int>(args[13]), kind = value_of<int>(args[14]);
    int* status = static_cast<int*>(address_of(args[15]));
    const auto is = [&](int i, at::IntArrayRef want) { return t[i]->sizes() == want; };
    if (B * T > INT32_MAX || d > INT32_MAX || I > INT32_MAX || Lh > INT32_MAX || t0 < 0 || t0 + T > 2 * Lh || !is(1, {d}) || !is(2, {d, d}) ||
        !is(3, {B, d, 2, Lh}) || (kind == 2 ? !is(4, {8, d, Lh + 8}) : !is(4, {d, Lh})) || (t[5] && !is(5, {B, 2})) || !is(6, {d}) ||
        !is(7, {I, d}) || !is(8, {I, d}) || !is(9, {d, I}))
      Py_RETURN_NONE;
    const int64_t yLh = ((t0 + T + 1) / 2 + 7) / 8 * 8;
    const int M = (int)(B * T), t_end = (int)(t0 + T);
    at::Tensor xn = at::empty({M, d}, x.options()), yT = at::empty({B, d, 2, yLh}, x.options()), h = at::empty({M, I}, x.options());
    const long long parts = I >= CUT_K ? stu_linear_workspace_elems(M, (int)d, (int)I, 1, code) : 0;
    at::Tensor workspace;
    if (parts > 0) workspace = at::empty({parts}, x.options().dtype(at::kFloat));
    float* pw = parts > 0 ? workspace.data_ptr<float>() : nullptr;
    void* p[10];
    for (int i = 0; i < 10; i++) p[i] = data_of(t[i]);
    void *pn = xn.data_ptr(), *py = yT.data_ptr(), *ph = h.data_ptr(), *stream = (void*)c10::cuda::getCurrentCUDAStream().stream();
    int rc, done = 0;
    Py_BEGIN_ALLOW_THREADS
    rc = stu_rmsnorm(p[0], p[1], pn, M, (int)d, d, d, eps, code, stream);
    if (rc == 0)
      rc = stu_linear(pn, d, p[2], d, 1, nullptr, nullptr, 0, p[3], 0, M, (int)d, (int)d, 3, (int)T, t0, (int)Lh, nullptr, 0.f, code, 0, stream);
    if (rc == 0)
      rc = stu_conv_prefill_positions(p[3], p[4], py, p[0], T * d, d, (int)B, (int)d, (int)Lh, (int)yLh, t0, t_end, (int*)p[5], fresh, kind,
                                      status, code, stream);
    if (rc == 0) {
      done = 1;
      rc = stu_rmsnorm(p[0], p[6], pn, M, (int)d, d, d, mlp_eps, code, stream);
    }
    if (rc == 0)
      rc = stu_linear(pn, d, p[7], d, 1, p[8], nullptr, 0, ph, I, M, (int)I, (int)d, 2, 0, 0, 0, nullptr, 0.f, code, 0, stream);
    if (rc == 0)
      rc = stu_linear_split(ph, I, p[9], I, 1, nullptr, p[0], d, p[0], d, M, (int)d, (int)I, 1, 0, 0, 0, nullptr, 0.f, code, 0, pw, parts, stream);
    Py_END_ALLOW_THREADS
    if (raised(rc, "layer_prefill")) return nullptr;
    if (rc == 0) done = stu_linear_launches() == 2 ? 7 : 3;
    if (done) return PyLong_FromLong(done);
  } catch (const BadArgument&) {
    PyErr_Clear();
  } catch (const std::exception&) {
  }
  Py_RETURN_NONE;
}

// what ops.py launches
#define ENTRY(name) {#name, (PyCFunction)(void (*)(void))Call<&name>::call, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    ENTRY(stu_bias_act),
    ENTRY(stu_block_decode_step),
    ENTRY(stu_block_step_workspace_bytes),
    ENTRY(stu_conv_prefill_approx),
    ENTRY(stu_conv_prefill_approx_static),
    ENTRY(stu_conv_prefill_approx_tc5),
    ENTRY(stu_decode_approx),
    ENTRY(stu_decode_approx_pipelined),
    ENTRY(stu_decode_approx_projected), ENTRY(stu_stream_ahead), ENTRY(stu_stream_finish),
    ENTRY(stu_decode_approx_push),
    ENTRY(stu_decode_approx_shard),
    ENTRY(stu_embed),
    ENTRY(stu_full_combine),
    ENTRY(stu_full_conv),
    ENTRY(stu_full_decode_combine),
    ENTRY(stu_full_conv_tc5),
    ENTRY(stu_full_conv_f32_tc5),
    ENTRY(stu_full_conv_f32_tc5_pays),
    ENTRY(stu_full_decode_prepare),
    ENTRY(stu_full_decode_step),
    ENTRY(stu_full_decode_step_tc5),
    ENTRY(stu_lds_chunk_scan),
    ENTRY(stu_lds_decode_step),
    ENTRY(stu_lds_final_state),
    ENTRY(stu_linear),
    ENTRY(stu_linear_split),
    ENTRY(stu_linear_workspace_elems),
    ENTRY(stu_linear_can_fuse_norm),
    ENTRY(stu_linear_launches),
    ENTRY(stu_linear_tile_cost),
    ENTRY(stu_linear_push),
    ENTRY(stu_peer_combine),
    ENTRY(stu_peer_exchange),
    ENTRY(stu_rmsnorm),
    ENTRY(stu_sample),
    ENTRY(stu_swa_forward),
    ENTRY(stu_swa_prefill_scratch_elems),
    ENTRY(stu_swa_prefill_tc5),
    ENTRY(stu_taps_even),
    ENTRY(stu_taps_rev8),
    ENTRY(stu_to_history),
    ENTRY(stu_toeplitz),
    {"status_ready", (PyCFunction)(void (*)(void))status_ready, METH_FASTCALL, nullptr},
    {"linear", (PyCFunction)(void (*)(void))linear, METH_FASTCALL, nullptr},
    {"layer_step_f32", (PyCFunction)(void (*)(void))layer_step_f32, METH_FASTCALL, nullptr},
    {"layer_prefill", (PyCFunction)(void (*)(void))layer_prefill, METH_FASTCALL, nullptr},
    {"rmsnorm", (PyCFunction)(void (*)(void))rmsnorm, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&module); }
