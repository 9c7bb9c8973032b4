// The Python surface's usual calls in native code: exact torch.Tensor arguments on the GPU, the library's own scratch, the
// current stream.  A call that looks like anything else (a subclass, a wrapped or traced tensor, another type, a shape that an
// assertion refuses, a workspace that has to grow) is answered with None, and the Python path, which says what is wrong with
// it, serves it.  Arguments are read with the interpreter lock; the output is allocated and the library called without it
// (Unlocked): an allocation and a launch into a full queue may wait, and other threads go on meanwhile.
// Bound: the host.  A call's Python attribute look-ups, struct packing and ctypes conversions took 5 to 10 us, where the kernels of
// the smallest calls take 8 to 15.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cstring>

#include "dtattn.h"

namespace {

// The library's entry points, from the handle that Python has loaded (bind)
decltype(&dt_sdpa_workspace_size) f_workspace_size;
decltype(&dt_sdpa_kernel_name) f_kernel_name;
decltype(&dt_sdpa_forward) f_forward;
decltype(&dt_sdpa_decode_step_workspace_size) f_step_workspace_size;
decltype(&dt_sdpa_decode_step) f_step;
decltype(&dt_qk_prologue) f_prologue;
decltype(&dt_sparse_indexed_attention) f_sparse;

// Thrown where a call is for the Python path.
struct NotMine {};

[[noreturn]] void decline() { throw NotMine(); }

// Without the interpreter lock as long as it lives: no Python object is touched then.
struct Unlocked {
  PyThreadState* const state = PyEval_SaveThread();
  Unlocked() = default;
  Unlocked(const Unlocked&) = delete;
  Unlocked& operator=(const Unlocked&) = delete;
  ~Unlocked() { PyEval_RestoreThread(state); }
};

const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_CheckExact(o)) decline();
  const at::Tensor& t = THPVariable_Unpack(o);
  const c10::TensorImpl* impl = t.unsafeGetTensorImpl();
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || !impl->has_storage() || impl->is_python_dispatch() ||
      impl->key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::FuncTorchGradWrapper,
                                                   c10::DispatchKey::Functionalize, c10::DispatchKey::Negative, c10::DispatchKey::Conjugate})))
    decline();
  return t;
}
bool none(PyObject* o) { return o == Py_None; }
double number(PyObject* o) {
  if (!PyFloat_CheckExact(o)) decline();
  return PyFloat_AS_DOUBLE(o);
}
long long whole(PyObject* o, long long lo, long long hi) {
  if (!PyLong_CheckExact(o)) decline();
  int over = 0;
  const long long x = PyLong_AsLongLongAndOverflow(o, &over);
  if (over || x < lo || x > hi) decline();
  return x;
}
bool truth(PyObject* o) {
  if (o != Py_True && o != Py_False) decline();
  return o == Py_True;
}
int32_t dtype_of(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kHalf: return DT_F16;
    case at::kBFloat16: return DT_BF16;
    case at::kFloat: return DT_F32;
    default: decline();
  }
}
int32_t dim(const at::Tensor& t, int i) {
  const int64_t n = t.size(i);
  if (n > 0x7fffffff) decline();
  return (int32_t)n;
}
dt_tensor4 quad(const at::Tensor& t) {
  if (t.dim() != 4 || (t.stride(3) != 1 && t.size(3) != 1)) decline();
  return {t.data_ptr(), t.stride(0), t.stride(1), t.stride(2)};
}
// a [n] vector in the type of `like`
const void* vector(PyObject* o, const at::Tensor& like, int64_t n) {
  if (none(o)) return nullptr;
  const at::Tensor& t = tensor(o);
  if (t.scalar_type() != like.scalar_type() || !t.is_contiguous() || t.numel() != n) decline();
  return t.data_ptr();
}
void same_kind(const at::Tensor& t, const at::Tensor& q) {
  if (t.scalar_type() != q.scalar_type() || t.device() != q.device()) decline();
}
// the caller's output tensor, or an undefined one where it is for the call to allocate
at::Tensor given(PyObject* o) { return none(o) ? at::Tensor() : tensor(o); }
at::Tensor new_output(const at::Tensor& q) {
  return q.is_contiguous() ? at::empty_like(q) : at::empty(q.sizes(), q.options().requires_grad(false));
}

// All but the output (place)
dt_sdpa_params attention(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, double scale, bool causal, PyObject* mask,
                         PyObject* lse, uint32_t flags, PyObject* sinks, int32_t window, int32_t Sk) {
  dt_sdpa_params p;
  memset(&p, 0, sizeof(p));
  p.q = quad(q);
  p.k = quad(k);
  p.v = quad(v);
  same_kind(k, q);
  same_kind(v, q);
  p.B = dim(q, 0);
  p.Sq = dim(q, 1);
  p.Hq = dim(q, 2);
  p.D = dim(q, 3);
  p.Sk = Sk < 0 ? dim(k, 1) : Sk;
  p.Hkv = dim(k, 2);
  p.dtype = dtype_of(q);
  p.scale = (float)scale;
  p.is_causal = causal ? 1 : 0;
  p.flags = flags;
  if (!none(mask)) {
    const at::Tensor& m = tensor(mask);
    same_kind(m, q);
    if (m.dim() != 4 || m.size(2) != p.Sq || m.size(3) != p.Sk || (m.stride(3) != 1 && p.Sk != 1)) decline();
    p.mask = m.data_ptr();
    p.mask_stride_b = m.size(0) > 1 ? m.stride(0) : 0;
    p.mask_stride_h = m.size(1) > 1 ? m.stride(1) : 0;
    p.mask_stride_q = m.stride(2);
  }
  if (!none(lse)) {
    const at::Tensor& t = tensor(lse);
    if (t.scalar_type() != at::kFloat || !t.is_contiguous() || t.dim() != 3 || t.size(0) != p.B || t.size(1) != p.Hq || t.size(2) != p.Sq)
      decline();
    p.lse = t.data_ptr<float>();
  }
  p.sinks = vector(sinks, q, p.Hq);
  p.sliding_window = window;
  return p;
}

// The output of a call, allocated where there is none yet
void place(dt_sdpa_params& p, at::Tensor& out, const at::Tensor& q) {
  if (!out.defined()) out = new_output(q);
  p.o = quad(out);
  same_kind(out, q);
}

// The status of a failed call as a number, its output otherwise.
PyObject* answer(int status, const at::Tensor& out, PyObject* given) {
  if (status != DT_OK) return PyLong_FromLong(status);
  return none(given) ? THPVariable_Wrap(out) : Py_NewRef(given);
}

// Runs `body`, with what it throws turned into None.  (Nothing is called before bind, whose last assignment is f_sparse.)
template <typename F>
PyObject* guarded(Py_ssize_t n, Py_ssize_t want, F body) {
  if (n != want) {
    PyErr_Format(PyExc_TypeError, "%zd arguments, %zd wanted", n, want);
    return nullptr;
  }
  try {
    if (!f_sparse) decline();
    return body();
  } catch (const NotMine&) {
  } catch (const std::exception&) {  // (no room for the output, a tensor without data: the Python path raises the same)
  }
  PyErr_Clear();  // what a dispatch mode raised while the output was allocated comes with the error indicator set
  Py_RETURN_NONE;
}

// sdpa(q, k, v, out, scale, is_causal, mask, lse, flags, sinks, window, stream, workspace, workspace_bytes): the output, or, for
// a call with scratch of its own, (output, parameters, scratch bytes, whether it can do without) for run
PyObject* py_sdpa(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 14, [&]() -> PyObject* {
    const at::Tensor &q = tensor(a[0]), &k = tensor(a[1]), &v = tensor(a[2]);
    if (q.dim() != 4 || k.dim() != 4) decline();
    const uint32_t flags = (uint32_t)whole(a[8], 0, 0xffffffffll);
    const int32_t window = (int32_t)whole(a[10], -0x7fffffffll, 0x7fffffffll);
    void* const stream = PyLong_AsVoidPtr(a[11]);
    void* const ws = PyLong_AsVoidPtr(a[12]);
    const size_t bytes = (size_t)whole(a[13], 0, 1ll << 62);
    at::Tensor out = given(a[3]);
    dt_sdpa_params p = attention(q, k, v, number(a[4]), truth(a[5]), a[6], a[7], flags, a[9], window, -1);
    size_t need = 0;
    const char* name = "";
    int status = DT_OK;
    bool done = true;
    {
      Unlocked here;
      place(p, out, q);
      if (f_workspace_size(&p, &need) != DT_OK) decline();
      if (need != 0 && f_kernel_name(&p, &name) != DT_OK) decline();
      if (need == 0) {
        status = f_forward(&p, nullptr, 0, stream);
      } else if (strcmp(name, "decode_splitkv") == 0) {  // (its tickets have to start at zero: the device's own workspace, if it is large enough)
        if (!ws || bytes < need) decline();
        status = f_forward(&p, ws, bytes, stream);
      } else {
        done = false;
      }
    }
    if (done) return answer(status, out, a[3]);
    PyObject* o = none(a[3]) ? THPVariable_Wrap(out) : Py_NewRef(a[3]);
    return Py_BuildValue("(Ny#nO)", o, reinterpret_cast<const char*>(&p), (Py_ssize_t)sizeof(p), (Py_ssize_t)need,
                         none(a[6]) || strcmp(name, "generic") == 0 ? Py_True : Py_False);
  });
}

// run(parameters, out, scratch, scratch_bytes, stream): a call that sdpa has asked scratch for
PyObject* py_run(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 5, [&]() -> PyObject* {
    dt_sdpa_params p;
    if (!PyBytes_CheckExact(a[0]) || PyBytes_GET_SIZE(a[0]) != (Py_ssize_t)sizeof(p)) decline();
    memcpy(&p, PyBytes_AS_STRING(a[0]), sizeof(p));
    void* const scratch = PyLong_AsVoidPtr(a[2]);
    const size_t bytes = (size_t)whole(a[3], 0, 1ll << 62);
    void* const stream = PyLong_AsVoidPtr(a[4]);
    int status;
    {
      Unlocked here;
      status = f_forward(&p, scratch, bytes, stream);
    }
    return status == DT_OK ? Py_NewRef(a[1]) : PyLong_FromLong(status);
  });
}

// step(q, k_cache, v_cache, k_new, v_new, rotary, out, scale, total, lse, flags, q_weight, k_weight, eps, sinks, window, stream,
//      workspace, workspace_bytes)
PyObject* py_step(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 19, [&]() -> PyObject* {
    const at::Tensor &q = tensor(a[0]), &k = tensor(a[1]), &v = tensor(a[2]), &kn = tensor(a[3]), &vn = tensor(a[4]);
    if (q.dim() != 4 || k.dim() != 4 || v.dim() != 4) decline();
    const int32_t total = (int32_t)whole(a[8], 1, std::min<int64_t>(0x7fffffff, std::min(k.size(1), v.size(1))));
    const uint32_t flags = (uint32_t)whole(a[10], 0, 0xffffffffll);
    const int32_t window = (int32_t)whole(a[15], -0x7fffffffll, 0x7fffffffll);
    void* const stream = PyLong_AsVoidPtr(a[16]);
    void* const ws = PyLong_AsVoidPtr(a[17]);
    const size_t bytes = (size_t)whole(a[18], 0, 1ll << 62);
    at::Tensor out = given(a[6]);
    dt_decode_step_params s;
    memset(&s, 0, sizeof(s));
    s.attn = attention(q, k, v, number(a[7]), true, Py_None, a[9], flags, a[14], window, total);
    s.k_new = quad(kn);
    s.v_new = quad(vn);
    same_kind(kn, q);
    same_kind(vn, q);
    s.T_new = dim(kn, 1);
    if (!none(a[5])) {
      const at::Tensor& r = tensor(a[5]);
      same_kind(r, q);
      if (r.dim() != 3 || r.size(1) != s.T_new || r.stride(2) != 1) decline();
      s.rotary = r.data_ptr();
      s.rotary_stride_b = r.size(0) > 1 ? r.stride(0) : 0;
      s.rotary_stride_s = r.stride(1);
    }
    s.q_norm_weight = vector(a[11], q, q.size(3));
    s.k_norm_weight = vector(a[12], q, q.size(3));
    s.norm_eps = (float)number(a[13]);
    int status;
    {
      Unlocked here;
      place(s.attn, out, q);
      size_t need = 0;
      if (f_step_workspace_size(&s, &need) != DT_OK) decline();
      if (need && (!ws || bytes < need)) decline();
      status = f_step(&s, need ? ws : nullptr, need ? bytes : 0, stream);
    }
    return answer(status, out, a[6]);
  });
}

// All but the output
dt_qk_prologue_params prologue(const at::Tensor& x, PyObject* weight, PyObject* rotary, double eps, bool per_token, double post_scale) {
  dt_qk_prologue_params p;
  memset(&p, 0, sizeof(p));
  p.x = quad(x);
  p.B = dim(x, 0);
  p.S = dim(x, 1);
  p.H = dim(x, 2);
  p.D = dim(x, 3);
  p.dtype = dtype_of(x);
  p.norm_weight = vector(weight, x, per_token ? x.size(2) * x.size(3) : x.size(3));
  p.norm_per_token = per_token ? 1 : 0;
  p.eps = (float)eps;
  if (!none(rotary)) {
    const at::Tensor& r = tensor(rotary);
    if (r.dim() != 4 || r.scalar_type() != x.scalar_type() || r.stride(3) != 1 || r.size(1) != p.S || r.size(3) != p.D) decline();
    p.rotary = r.data_ptr();
    p.rotary_stride_b = r.size(0) > 1 ? r.stride(0) : 0;
    p.rotary_stride_s = r.stride(1);
    p.rotary_stride_h = r.size(2) > 1 ? r.stride(2) : 0;
  }
  p.post_scale = (float)post_scale;
  return p;
}

// prologue(q, k, q_out, k_out, q_weight, k_weight, rotary, rotary_k, eps, norm_per_token, post_scale, stream): (q_out, k_out)
PyObject* py_prologue(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 12, [&]() -> PyObject* {
    const at::Tensor &q = tensor(a[0]), &k = tensor(a[1]);
    if (q.dim() != 4 || k.dim() != 4) decline();
    const double eps = number(a[8]), post_scale = number(a[10]);
    const bool per_token = truth(a[9]);
    void* const stream = PyLong_AsVoidPtr(a[11]);
    at::Tensor q_out = given(a[2]), k_out = given(a[3]);
    dt_qk_prologue_params pq = prologue(q, a[4], a[6], eps, per_token, post_scale);
    dt_qk_prologue_params pk = prologue(k, a[5], none(a[7]) ? a[6] : a[7], eps, per_token, post_scale);
    int status;
    {
      Unlocked here;
      if (!q_out.defined()) q_out = at::empty_like(q);
      if (!k_out.defined()) k_out = at::empty_like(k);
      pq.y = quad(q_out);
      pk.y = quad(k_out);
      status = f_prologue(&pq, &pk, stream);
    }
    if (status != DT_OK) return PyLong_FromLong(status);
    PyObject* first = none(a[2]) ? THPVariable_Wrap(q_out) : Py_NewRef(a[2]);
    PyObject* second = none(a[3]) ? THPVariable_Wrap(k_out) : Py_NewRef(a[3]);
    PyObject* both = first && second ? PyTuple_Pack(2, first, second) : nullptr;
    Py_XDECREF(first);
    Py_XDECREF(second);
    return both;
  });
}

// sparse(q, k_raw, v_raw, k_comp, v_comp, selected, scale, sinks, window, is_causal, out, lse, flags, stream)
PyObject* py_sparse(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded(n, 14, [&]() -> PyObject* {
    const at::Tensor &q = tensor(a[0]), &kr = tensor(a[1]), &vr = tensor(a[2]);
    if (q.dim() != 4 || kr.dim() != 4) decline();
    dt_sparse_indexed_params p;
    memset(&p, 0, sizeof(p));
    at::Tensor out = given(a[10]);
    void* const stream = PyLong_AsVoidPtr(a[13]);
    p.q = quad(q);
    p.k_raw = quad(kr);
    p.v_raw = quad(vr);
    p.B = dim(q, 0);
    p.Sq = dim(q, 1);
    p.Hq = dim(q, 2);
    p.D = dim(q, 3);
    p.Hkv = dim(kr, 2);
    p.Sr = dim(kr, 1);
    p.dtype = dtype_of(q);
    if (!none(a[3])) {
      const at::Tensor &kc = tensor(a[3]), &vc = tensor(a[4]);
      if (kc.dim() != 4) decline();
      p.Sc = dim(kc, 1);
      if (p.Sc > 0) {
        p.k_comp = quad(kc);
        p.v_comp = quad(vc);
      }
    }
    if (!none(a[5])) {
      const at::Tensor& sel = tensor(a[5]);
      if (sel.scalar_type() != at::kInt || sel.dim() != 3 || sel.size(1) != p.Sq || sel.stride(2) != 1) decline();
      p.selected = sel.data_ptr<int32_t>();
      p.n_selected = dim(sel, 2);
      p.selected_stride_b = sel.size(0) > 1 ? sel.stride(0) : 0;
      p.selected_stride_q = sel.stride(1);
    }
    p.scale = (float)number(a[6]);
    p.sinks = vector(a[7], q, p.Hq);
    p.sliding_window = (int32_t)whole(a[8], -0x7fffffffll, 0x7fffffffll);
    p.is_causal = truth(a[9]) ? 1 : 0;
    if (!none(a[11])) {
      const at::Tensor& t = tensor(a[11]);
      if (t.scalar_type() != at::kFloat || !t.is_contiguous() || t.dim() != 3 || t.size(0) != p.B || t.size(1) != p.Hq || t.size(2) != p.Sq)
        decline();
      p.lse = t.data_ptr<float>();
    }
    p.flags = (uint32_t)whole(a[12], 0, 0xffffffffll);
    int status;
    {
      Unlocked here;
      if (!out.defined()) out = at::empty_like(q);
      p.o = quad(out);
      status = f_sparse(&p, stream);
    }
    return answer(status, out, a[10]);
  });
}

// bind(addresses of the seven entry points, in the order of the declarations above)
PyObject* py_bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 7) {
    PyErr_SetString(PyExc_TypeError, "seven addresses");
    return nullptr;
  }
  void* f[7];
  for (int i = 0; i < 7; ++i) {
    f[i] = PyLong_AsVoidPtr(a[i]);
    if (!f[i]) {
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "no address");
      return nullptr;
    }
  }
  f_workspace_size = reinterpret_cast<decltype(f_workspace_size)>(f[0]);
  f_kernel_name = reinterpret_cast<decltype(f_kernel_name)>(f[1]);
  f_forward = reinterpret_cast<decltype(f_forward)>(f[2]);
  f_step_workspace_size = reinterpret_cast<decltype(f_step_workspace_size)>(f[3]);
  f_step = reinterpret_cast<decltype(f_step)>(f[4]);
  f_prologue = reinterpret_cast<decltype(f_prologue)>(f[5]);
  f_sparse = reinterpret_cast<decltype(f_sparse)>(f[6]);
  Py_RETURN_NONE;
}

#define DT_METHOD(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {DT_METHOD("sdpa", py_sdpa), DT_METHOD("run", py_run), DT_METHOD("step", py_step), DT_METHOD("prologue", py_prologue),
                         DT_METHOD("sparse", py_sparse), DT_METHOD("bind", py_bind), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "dtattn_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_dtattn_calls() { return PyModule_Create(&module); }
