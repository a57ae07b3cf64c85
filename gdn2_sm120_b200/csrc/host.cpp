// The usual calls of the Python API as one native function each: argument checks, buffers, launch.
//
// A decode step at batch 1 keeps the GPU busy for 3 us; the same checks and the ctypes call in Python
// took 25.  Every function here handles the plain case completely (CUDA tensors of the documented
// shapes and types, one wave, no overlap of buffers) and returns None for anything else: the Python
// wrappers then go through their own checks, which raise what is documented or take the rarer way.
// The kernels are those of libgdn2_b200.so, reached through its C ABI.

#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/core/GradMode.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <cstring>

#include "../../include/gdn2_b200.h"

namespace {

struct Api {
  decltype(&gdn2_token_forward) token_forward;
  decltype(&gdn2_token_forward_fused) token_forward_fused;
  decltype(&gdn2_token_forward_t1_zero) token_forward_t1_zero;
  decltype(&gdn2_token_forward_t1_zero_fused) token_forward_t1_zero_fused;
  decltype(&gdn2_token_dstate_scan) token_dstate_scan;
  decltype(&gdn2_token_chunk_vjp) token_chunk_vjp;
  decltype(&gdn2_chunk_forward) chunk_forward;
  decltype(&gdn2_chunk_forward_fused) chunk_forward_fused;
  decltype(&gdn2_chunk_forward_kernels) chunk_forward_kernels;
  decltype(&gdn2_chunk_backward) chunk_backward;
  decltype(&gdn2_chunk_backward_kernels) chunk_backward_kernels;
  decltype(&gdn2_chunk_workspace_bytes) chunk_workspace_bytes;
  decltype(&gdn2_chunk_scratch_bytes) chunk_scratch_bytes;
  decltype(&gdn2_gate_prologue) gate_prologue;
  decltype(&gdn2_gate_prologue_vjp) gate_prologue_vjp;
} api;
PyObject* g_check = nullptr;     // _lib.check(status, name): raises
PyObject* g_launches = nullptr;  // _lib.LAUNCHES
PyObject* g_oom = nullptr;       // torch.cuda.OutOfMemoryError
bool g_bound = false;

constexpr int64_t kDim = GDN2_DIM, kChunk = GDN2_CHUNK, kInterval = GDN2_TOKEN_INTERVAL;
constexpr int64_t kStateBytes = kDim * kDim * 4;
// requests of this size are left to the Python wrappers, which look at the free memory first
constexpr int64_t kCheckedBytes = int64_t(16) << 30;

// ---- small helpers -----------------------------------------------------------------------------------
inline PyObject* none() { Py_RETURN_NONE; }

inline const at::Tensor* tensor(PyObject* o) {
  return THPVariable_CheckExact(o) ? &THPVariable_Unpack(o) : nullptr;
}

inline int dtype_code(at::ScalarType t) {
  return t == at::kBFloat16 ? GDN2_BF16 : t == at::kHalf ? GDN2_FP16 : t == at::kFloat ? GDN2_FP32 : -1;
}

inline bool aligned(const at::Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }

bool b200(int index) {
  static int8_t known[64] = {0};
  if (index < 0 || index >= 64) return false;
  if (known[index] == 0) known[index] = at::cuda::getDeviceProperties(index)->major == 10 ? 1 : -1;
  return known[index] == 1;
}

struct Seq {
  const at::Tensor* t[6];  // q k v g beta w
  int64_t batch, time, heads;
  int dtype, g_dtype;
  bool all_aligned;
  const void* ptr(int i) const { return t[i]->data_ptr(); }
};

// The six sequence tensors as the kernels take them; false for anything unusual.
bool read_seq(PyObject* const* a, Seq* s) {
  for (int i = 0; i < 6; ++i) {
    s->t[i] = tensor(a[i]);
    if (s->t[i] == nullptr) return false;
  }
  const at::Tensor& q = *s->t[0];
  if (!q.defined() || q.dim() != 4 || !q.is_cuda()) return false;
  const auto shape = q.sizes();
  s->batch = shape[0]; s->time = shape[1]; s->heads = shape[2];
  if (shape[3] != kDim || s->batch <= 0 || s->time <= 0 || s->heads <= 0) return false;
  s->dtype = dtype_code(q.scalar_type());
  s->g_dtype = dtype_code(s->t[3]->scalar_type());
  if (s->dtype != GDN2_BF16 && s->dtype != GDN2_FP16) return false;
  if (s->g_dtype != s->dtype && s->g_dtype != GDN2_FP32) return false;
  s->all_aligned = true;
  for (int i = 0; i < 6; ++i) {
    const at::Tensor& x = *s->t[i];
    if (i > 0 && (x.dim() != 4 || x.sizes() != shape || x.device() != q.device())) return false;
    if (i > 0 && i != 3 && x.scalar_type() != q.scalar_type()) return false;
    if (!x.is_contiguous() || x.layout() != at::kStrided || x.is_neg() || x.is_conj()) return false;
    s->all_aligned = s->all_aligned && aligned(x);
  }
  return b200(q.device().index());
}

// an optional tensor argument: 0 = None, 1 = given and as expected, -1 = anything else
int read_state(PyObject* o, const Seq& s, const at::Tensor** out) {
  *out = nullptr;
  if (o == Py_None) return 0;
  const at::Tensor* t = tensor(o);
  if (t == nullptr || t->dim() != 4 || t->scalar_type() != at::kFloat || t->device() != s.t[0]->device() ||
      !t->is_contiguous() || t->size(0) != s.batch || t->size(1) != s.heads || t->size(2) != kDim ||
      t->size(3) != kDim) {
    return -1;
  }
  *out = t;
  return 1;
}

bool read_scale(PyObject* o, float* scale) {
  double value = 1.0 / std::sqrt(double(kDim));
  if (o != Py_None) {
    if (!PyFloat_Check(o)) return false;
    value = PyFloat_AS_DOUBLE(o);
  }
  *scale = static_cast<float>(value);
  return std::isfinite(value) && std::isfinite(*scale);
}

// the scratch budget, a module variable that callers set: a float or a huge number is left to Python
bool read_budget(PyObject* o, int64_t* budget) {
  int overflow = 1;
  if (PyLong_Check(o)) *budget = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0;
}

struct Span {
  uintptr_t lo, hi;
  explicit Span(const at::Tensor& t)
      : lo(reinterpret_cast<uintptr_t>(t.data_ptr())), hi(lo + t.numel() * t.element_size()) {}
  bool meets(const Span& o) const { return lo < o.hi && o.lo < hi; }
};

// buffers the caller owns must not overlap what is read (`final_state` may be the initial state itself)
bool apart(const Seq& s, const at::Tensor* init, const at::Tensor& out, const at::Tensor& fin, bool check_out,
           bool check_fin) {
  const Span o(out), f(fin);
  for (int i = 0; i < 6; ++i) {
    const Span x(*s.t[i]);
    if ((check_out && o.meets(x)) || (check_fin && f.meets(x))) return false;
  }
  if (init != nullptr) {
    const Span x(*init);
    if ((check_out && o.meets(x)) || (check_fin && f.meets(x) && f.lo != x.lo)) return false;
  }
  return !(check_out && o.meets(f));
}

void count(long kernels) {
  PyObject* old = PyList_GET_ITEM(g_launches, 0);
  PyObject* now = PyLong_FromLong(PyLong_AsLong(old) + kernels);
  if (now != nullptr) PyList_SetItem(g_launches, 0, now);
}

// Other Python threads run while a call allocates and launches: an allocation may go to the driver and a launch
// waits where the launch queue is full or its kernel is loaded for the first time.
struct WithoutGil {
  PyThreadState* state = PyEval_SaveThread();
  void end() {
    if (state != nullptr) PyEval_RestoreThread(state);
    state = nullptr;
  }
  ~WithoutGil() { end(); }
};

// false with a Python exception set when the entry point failed
bool ok(int status, const char* name, long kernels) {
  if (status == GDN2_OK) { count(kernels); return true; }
  PyObject* r = PyObject_CallFunction(g_check, "is", status, name);
  Py_XDECREF(r);
  if (r != nullptr) PyErr_SetString(PyExc_RuntimeError, name);
  return false;
}

inline float* fptr(const at::Tensor* t) { return t == nullptr ? nullptr : static_cast<float*>(t->data_ptr()); }
inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }
inline PyObject* wrap(at::Tensor t) { return THPVariable_Wrap(std::move(t)); }

inline at::Tensor floats(at::IntArrayRef shape, const at::Tensor& like) {
  return at::empty(shape, like.options().dtype(at::kFloat));
}
inline at::Tensor bytes(int64_t n, const at::Tensor& like) { return at::empty({n}, like.options().dtype(at::kByte)); }

#define GDN2_TRY try {
#define GDN2_CATCH                                                    \
  }                                                                   \
  catch (const c10::Error& e) { PyErr_SetString(                      \
      std::strstr(e.what(), "out of memory") ? g_oom : PyExc_RuntimeError, e.what_without_backtrace()); return nullptr; } \
  catch (const std::exception& e) { PyErr_SetString(PyExc_RuntimeError, e.what()); return nullptr; }

// ---- inference ---------------------------------------------------------------------------------------
// forward(q, k, v, g, beta, w, initial_state, scale, out, final_state_out, inplace, prologue, chunk_api, budget)
// -> (output, final_state) or None
PyObject* forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  GDN2_TRY
  Seq s;
  float scale;
  if (!g_bound || n != 14 || !read_seq(a, &s) || !read_scale(a[7], &scale)) return none();
  const at::Tensor *init = nullptr, *fin_given = nullptr;
  if (read_state(a[6], s, &init) < 0 || read_state(a[9], s, &fin_given) < 0) return none();
  const int truth = PyObject_IsTrue(a[10]);  // (any object is a flag in Python: 1, a NumPy bool)
  if (truth < 0) return nullptr;
  const bool inplace = truth != 0, chunk_api = a[12] == Py_True;
  const int prologue = int(PyLong_AsLong(a[11]));
  int64_t budget;
  if (!read_budget(a[13], &budget)) return none();
  if (inplace && (init == nullptr || fin_given != nullptr)) return none();
  if (chunk_api && c10::GradMode::is_enabled()) {
    bool grad = init != nullptr && init->requires_grad();
    for (int i = 0; i < 6; ++i) grad = grad || s.t[i]->requires_grad();
    if (grad) return none();
  }
  const at::Tensor* out_given = nullptr;
  if (a[8] != Py_None) {
    out_given = tensor(a[8]);
    if (out_given == nullptr || out_given->sizes() != s.t[0]->sizes() || !out_given->is_contiguous() ||
        out_given->scalar_type() != s.t[0]->scalar_type() || out_given->device() != s.t[0]->device()) {
      return none();
    }
  }
  const bool chunked = s.time >= kChunk;
  if (chunked) {
    if (!s.all_aligned || (init && !aligned(*init)) || (fin_given && !aligned(*fin_given)) ||
        (out_given && !aligned(*out_given))) {
      return none();
    }
  }
  const int64_t full = ceil_div(s.time, kChunk) * kChunk;
  int64_t ws_bytes = 0, sc_bytes = 0;
  if (chunked) {
    ws_bytes = api.chunk_workspace_bytes(s.batch, full, s.heads, 0);
    sc_bytes = api.chunk_scratch_bytes(s.batch, full, s.heads, 0);
    if (ws_bytes <= 0 || sc_bytes <= 0 || sc_bytes > budget || ws_bytes + sc_bytes >= kCheckedBytes) return none();
  }
  at::Tensor out, fin;
  int status;
  const char* name;
  bool distinct = true;
  WithoutGil others;
  const c10::cuda::CUDAGuard guard(s.t[0]->device());
  out = out_given ? *out_given : at::empty(s.t[0]->sizes(), s.t[0]->options());
  fin = inplace ? *init : fin_given ? *fin_given : floats({s.batch, s.heads, kDim, kDim}, *s.t[0]);
  if (out_given || fin_given || inplace) {
    // (an exact alias is spelled inplace_final_state, a final_state_out that meets initial_state is refused)
    distinct = apart(s, init, out, fin, out_given, fin_given || inplace) &&
               !(fin_given && init && Span(fin).meets(Span(*init)));
  }
  void* stream = at::cuda::getCurrentCUDAStream().stream();
  if (!distinct) {
    others.end();
    return none();
  }
  if (chunked) {
    name = "gdn2_chunk_forward";
    const at::Tensor buffer = bytes(ws_bytes + sc_bytes, *s.t[0]);
    uint8_t* ws = static_cast<uint8_t*>(buffer.data_ptr());
    if (prologue) {
      status = api.chunk_forward_fused(s.ptr(0), s.ptr(1), s.ptr(2), s.ptr(3), s.ptr(4), s.ptr(5), fptr(init),
                                       out.data_ptr(), fptr(&fin), ws, ws + ws_bytes, s.batch, s.time, s.heads, full,
                                       s.dtype, s.g_dtype, scale, prologue, stream);
    } else {
      status = api.chunk_forward(s.ptr(0), s.ptr(1), s.ptr(2), s.ptr(3), s.ptr(4), s.ptr(5), fptr(init),
                                 out.data_ptr(), fptr(&fin), nullptr, ws, ws + ws_bytes, s.batch, s.time, s.heads,
                                 full, 0, s.dtype, s.g_dtype, scale, stream);
    }
  } else if (s.time == 1 && init == nullptr) {
    name = "gdn2_token_forward_t1_zero";
    status = prologue ? api.token_forward_t1_zero_fused(s.ptr(0), s.ptr(1), s.ptr(2), s.ptr(5), out.data_ptr(),
                                                        fptr(&fin), s.batch, s.heads, s.dtype, scale, prologue, stream)
                      : api.token_forward_t1_zero(s.ptr(0), s.ptr(1), s.ptr(2), s.ptr(5), out.data_ptr(), fptr(&fin),
                                                  s.batch, s.heads, s.dtype, scale, stream);
  } else {
    name = "gdn2_token_forward";
    status = prologue ? api.token_forward_fused(s.ptr(0), s.ptr(1), s.ptr(2), s.ptr(3), s.ptr(4), s.ptr(5), fptr(init),
                                                out.data_ptr(), fptr(&fin), s.batch, s.time, s.heads, 0, s.time,
                                                s.dtype, s.g_dtype, scale, prologue, stream)
                      : api.token_forward(s.ptr(0), s.ptr(1), s.ptr(2), s.ptr(3), s.ptr(4), s.ptr(5), fptr(init),
                                          out.data_ptr(), fptr(&fin), nullptr, s.batch, s.time, s.heads, 0, s.time,
                                          s.dtype, s.g_dtype, scale, stream);
  }
  others.end();
  if (!ok(status, name, chunked ? api.chunk_forward_kernels() : 1)) return nullptr;
  PyObject* first = out_given ? Py_NewRef(a[8]) : wrap(out);
  PyObject* second = inplace ? Py_NewRef(a[6]) : fin_given ? Py_NewRef(a[9]) : wrap(fin);
  PyObject* result = PyTuple_New(2);
  PyTuple_SET_ITEM(result, 0, first);
  PyTuple_SET_ITEM(result, 1, second);
  return result;
  GDN2_CATCH
}

// ---- training ------------------------------------------------------------------------------------------
// train_forward(q, k, v, g, beta, w, initial_state, scale, budget)
// -> (output, final_state, workspace or None, boundaries) or None
PyObject* train_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  GDN2_TRY
  Seq s;
  float scale;
  const at::Tensor* init = nullptr;
  if (!g_bound || n != 9 || !read_seq(a, &s) || !read_scale(a[7], &scale) || read_state(a[6], s, &init) < 0) {
    return none();
  }
  int64_t budget;
  if (!read_budget(a[8], &budget)) return none();
  const bool chunked = s.time >= kChunk;
  const at::Tensor& q = *s.t[0];
  int64_t full = 0, ws_bytes = 0;
  if (chunked) {
    if (!s.all_aligned || (init && !aligned(*init))) return none();
    full = ceil_div(s.time, kChunk) * kChunk;
    ws_bytes = api.chunk_workspace_bytes(s.batch, full, s.heads, 1);
    const int64_t states = s.batch * (full / kChunk + 1) * s.heads * kStateBytes;
    // one wave: what backward needs for all batch rows fits the budget
    const int64_t wave = api.chunk_scratch_bytes(s.batch, full, s.heads, 1) + states;
    if (ws_bytes <= 0 || (wave > budget && s.batch > 1) || ws_bytes + states + wave >= kCheckedBytes) return none();
  }
  at::Tensor out, fin, boundaries, workspace;
  int status;
  WithoutGil others;
  const c10::cuda::CUDAGuard guard(q.device());
  out = at::empty(q.sizes(), q.options());
  fin = floats({s.batch, s.heads, kDim, kDim}, q);
  const int64_t slots = chunked ? full / kChunk + 1 : ceil_div(s.time, kInterval) + 1;
  boundaries = floats({s.batch, slots, s.heads, kDim, kDim}, q);
  void* stream = at::cuda::getCurrentCUDAStream().stream();
  if (chunked) {
    workspace = bytes(ws_bytes, q);
    status = api.chunk_forward(s.ptr(0), s.ptr(1), s.ptr(2), s.ptr(3), s.ptr(4), s.ptr(5), fptr(init), out.data_ptr(),
                               fptr(&fin), fptr(&boundaries), workspace.data_ptr(), nullptr, s.batch, s.time, s.heads,
                               full, 1, s.dtype, s.g_dtype, scale, stream);
  } else {
    status = api.token_forward(s.ptr(0), s.ptr(1), s.ptr(2), s.ptr(3), s.ptr(4), s.ptr(5), fptr(init), out.data_ptr(),
                               fptr(&fin), fptr(&boundaries), s.batch, s.time, s.heads, 0, s.time, s.dtype, s.g_dtype,
                               scale, stream);
  }
  others.end();
  if (!ok(status, chunked ? "gdn2_chunk_forward" : "gdn2_token_forward", chunked ? api.chunk_forward_kernels() : 1)) {
    return nullptr;
  }
  PyObject* result = PyTuple_New(4);
  PyTuple_SET_ITEM(result, 0, wrap(out));
  PyTuple_SET_ITEM(result, 1, wrap(fin));
  PyTuple_SET_ITEM(result, 2, chunked ? wrap(workspace) : Py_NewRef(Py_None));
  PyTuple_SET_ITEM(result, 3, wrap(boundaries));
  return result;
  GDN2_CATCH
}

// train_backward(q, k, v, g, beta, w, d_output or None, d_final_state or None, workspace or None, boundaries, scale)
// -> (dq, dk, dv, dg, dbeta, dw, d_initial_state) or None.  The first five of the saved tensors are what
// train_forward saw and returned (one wave).
PyObject* train_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  GDN2_TRY
  Seq s;
  float scale;
  if (!g_bound || n != 11 || !read_seq(a, &s) || !read_scale(a[10], &scale)) return none();
  const bool chunked = s.time >= kChunk;
  const at::Tensor& q = *s.t[0];
  const at::Tensor* workspace = chunked ? tensor(a[8]) : nullptr;
  const at::Tensor* boundaries = tensor(a[9]);
  if (boundaries == nullptr || (chunked && (workspace == nullptr || !s.all_aligned))) return none();
  const at::Tensor *out_given = nullptr, *fin_given = nullptr;
  if (a[6] != Py_None) {
    out_given = tensor(a[6]);
    if (out_given == nullptr || out_given->sizes() != q.sizes() || out_given->scalar_type() != q.scalar_type() ||
        out_given->device() != q.device()) {
      return none();
    }
  }
  if (a[7] != Py_None) {
    fin_given = tensor(a[7]);
    if (fin_given == nullptr || fin_given->dim() != 4 || fin_given->numel() != s.batch * s.heads * kDim * kDim ||
        fin_given->scalar_type() != at::kFloat || fin_given->device() != q.device()) {
      return none();
    }
  }
  const int64_t full = chunked ? ceil_div(s.time, kChunk) * kChunk : 0;
  const int64_t states = s.batch * (full / kChunk + 1) * s.heads * kStateBytes;
  if (chunked && boundaries->numel() * 4 != states) return none();
  at::Tensor grads[6], d_init;
  int status, scan_status = GDN2_OK;
  WithoutGil others;
  const c10::cuda::CUDAGuard guard(q.device());
  auto dense = [](const at::Tensor& t) {
    at::Tensor d = t.contiguous();
    return aligned(d) ? d : d.clone();
  };
  const at::Tensor d_out = out_given ? dense(*out_given) : at::zeros(q.sizes(), q.options());
  const at::Tensor d_fin = fin_given ? dense(*fin_given) : at::Tensor();
  for (int i = 0; i < 6; ++i) grads[i] = at::empty(s.t[i]->sizes(), s.t[i]->options());
  d_init = floats({s.batch, s.heads, kDim, kDim}, q);
  const float* df = d_fin.defined() ? static_cast<const float*>(d_fin.data_ptr()) : nullptr;
  void* stream = at::cuda::getCurrentCUDAStream().stream();
  void* g[6];
  for (int i = 0; i < 6; ++i) g[i] = grads[i].data_ptr();
  if (chunked) {
    const int64_t sc_bytes = api.chunk_scratch_bytes(s.batch, full, s.heads, 1);
    const at::Tensor buffer = bytes(states + sc_bytes, q);
    uint8_t* base = static_cast<uint8_t*>(buffer.data_ptr());
    status = api.chunk_backward(
        s.ptr(0), s.ptr(1), s.ptr(2), s.ptr(3), s.ptr(4), s.ptr(5), d_out.data_ptr(), df, fptr(boundaries),
        reinterpret_cast<float*>(base), workspace->data_ptr(), base + states, g[0], g[1], g[2], g[3], g[4], g[5],
        fptr(&d_init), s.batch, s.time, s.heads, full, s.dtype, s.g_dtype, scale, stream);
  } else {
    const at::Tensor d_bnd = at::empty(boundaries->sizes(), boundaries->options());
    status = scan_status = api.token_dstate_scan(s.ptr(0), s.ptr(1), s.ptr(3), s.ptr(4), d_out.data_ptr(), df,
                                                 fptr(&d_bnd), fptr(&d_init), s.batch, s.time, s.heads, 0, s.time,
                                                 s.dtype, s.g_dtype, scale, stream);
    if (scan_status == GDN2_OK) {
      status = api.token_chunk_vjp(s.ptr(0), s.ptr(1), s.ptr(2), s.ptr(3), s.ptr(4), s.ptr(5), d_out.data_ptr(),
                                   fptr(boundaries), fptr(&d_bnd), g[0], g[1], g[2], g[3], g[4], g[5], s.batch, s.time,
                                   s.heads, 0, s.time, s.dtype, s.g_dtype, scale, stream);
    }
  }
  others.end();
  if (chunked) {
    if (!ok(status, "gdn2_chunk_backward", api.chunk_backward_kernels())) return nullptr;
  } else if (!ok(scan_status, "gdn2_token_dstate_scan", 1) || !ok(status, "gdn2_token_chunk_vjp", 1)) {
    return nullptr;
  }
  PyObject* result = PyTuple_New(7);
  for (int i = 0; i < 6; ++i) PyTuple_SET_ITEM(result, i, wrap(grads[i]));
  PyTuple_SET_ITEM(result, 6, wrap(d_init));
  return result;
  GDN2_CATCH
}

// ---- input prologue of a training call -----------------------------------------------------------------
// prologue_forward(q, k, g, beta, w, normalize, activate) -> (q, k, g, beta, w, inv_q or None, inv_k or None) or None
PyObject* prologue_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  GDN2_TRY
  if (!g_bound || n != 7) return none();
  PyObject* order[6] = {a[0], a[1], a[4], a[2], a[3], a[4]};  // w in the place of v
  Seq s;
  if (!read_seq(order, &s) || !s.all_aligned) return none();
  const bool norm = a[5] == Py_True, gate = a[6] == Py_True;
  if (!norm && !gate) return none();
  const at::Tensor& q = *s.t[0];
  const int which[5] = {0, 1, 3, 4, 5};  // q k g beta w
  at::Tensor out[5], inv[2];
  int status;
  WithoutGil others;
  const c10::cuda::CUDAGuard guard(q.device());
  const void* in[5];
  void* to[5];
  for (int i = 0; i < 5; ++i) {
    const bool on = i < 2 ? norm : gate;
    const at::Tensor& x = *s.t[which[i]];
    if (on) out[i] = at::empty(x.sizes(), x.options());
    in[i] = on ? x.data_ptr() : nullptr;
    to[i] = on ? out[i].data_ptr() : nullptr;
  }
  if (norm) {
    for (int i = 0; i < 2; ++i) inv[i] = floats({s.batch, s.time, s.heads}, q);
  }
  status = api.gate_prologue(in[0], in[1], in[2], in[3], in[4], to[0], to[1], to[2], to[3], to[4],
                             norm ? fptr(&inv[0]) : nullptr, norm ? fptr(&inv[1]) : nullptr, s.batch, s.time, s.heads,
                             s.dtype, s.g_dtype, at::cuda::getCurrentCUDAStream().stream());
  others.end();
  if (!ok(status, "gdn2_gate_prologue", 1)) return nullptr;
  PyObject* result = PyTuple_New(7);
  for (int i = 0; i < 5; ++i) PyTuple_SET_ITEM(result, i, out[i].defined() ? wrap(out[i]) : Py_NewRef(a[i]));
  for (int i = 0; i < 2; ++i) PyTuple_SET_ITEM(result, 5 + i, norm ? wrap(inv[i]) : Py_NewRef(Py_None));
  return result;
  GDN2_CATCH
}

// prologue_backward(q, k, g, beta, w, inv_q, inv_k, dq, dk, dg, dbeta, dw, normalize, activate)
// -> the five cotangents of the raw tensors, or None
PyObject* prologue_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  GDN2_TRY
  if (!g_bound || n != 14) return none();
  PyObject* order[6] = {a[0], a[1], a[4], a[2], a[3], a[4]};
  Seq s;
  if (!read_seq(order, &s) || !s.all_aligned) return none();
  const bool norm = a[12] == Py_True, gate = a[13] == Py_True;
  const at::Tensor *inv[2] = {nullptr, nullptr}, *in[5];
  for (int i = 0; i < 2 && norm; ++i) {
    inv[i] = tensor(a[5 + i]);
    if (inv[i] == nullptr) return none();
  }
  const int which[5] = {0, 1, 3, 4, 5};
  for (int i = 0; i < 5; ++i) {
    in[i] = tensor(a[7 + i]);  // None (no cotangent) and other layouts are the wrapper's
    const at::Tensor& x = *s.t[which[i]];
    if (in[i] == nullptr || in[i]->sizes() != x.sizes() || in[i]->scalar_type() != x.scalar_type() ||
        !in[i]->is_contiguous() || !aligned(*in[i]) || in[i]->device() != x.device()) {
      return none();
    }
  }
  at::Tensor out[5];
  int status;
  WithoutGil others;
  const c10::cuda::CUDAGuard guard(s.t[0]->device());
  const void *raw[5], *from[5];
  void* to[5];
  for (int i = 0; i < 5; ++i) {
    const bool on = i < 2 ? norm : gate;
    if (on) out[i] = at::empty(in[i]->sizes(), in[i]->options());
    raw[i] = on ? s.t[which[i]]->data_ptr() : nullptr;
    from[i] = on ? in[i]->data_ptr() : nullptr;
    to[i] = on ? out[i].data_ptr() : nullptr;
  }
  status = api.gate_prologue_vjp(raw[0], raw[1], raw[2], raw[3], raw[4], fptr(inv[0]), fptr(inv[1]), from[0], from[1],
                                 from[2], from[3], from[4], to[0], to[1], to[2], to[3], to[4], s.batch, s.time, s.heads,
                                 s.dtype, s.g_dtype, at::cuda::getCurrentCUDAStream().stream());
  others.end();
  if (!ok(status, "gdn2_gate_prologue_vjp", 1)) return nullptr;
  PyObject* result = PyTuple_New(5);
  for (int i = 0; i < 5; ++i) PyTuple_SET_ITEM(result, i, out[i].defined() ? wrap(out[i]) : Py_NewRef(a[7 + i]));
  return result;
  GDN2_CATCH
}

// bind({entry point: address}, _lib.check, _lib.LAUNCHES, torch.cuda.OutOfMemoryError)
PyObject* bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 4 || !PyDict_Check(a[0]) || !PyList_Check(a[2])) {
    PyErr_SetString(PyExc_TypeError, "bind(addresses, check, launches, out_of_memory)");
    return nullptr;
  }
  bool missing = false;
  auto get = [&](const char* name) -> void* {
    PyObject* v = PyDict_GetItemString(a[0], name);
    if (v == nullptr) { missing = true; return nullptr; }
    return PyLong_AsVoidPtr(v);
  };
#define GDN2_BIND(f) api.f = reinterpret_cast<decltype(api.f)>(get("gdn2_" #f))
  GDN2_BIND(token_forward);
  GDN2_BIND(token_forward_fused);
  GDN2_BIND(token_forward_t1_zero);
  GDN2_BIND(token_forward_t1_zero_fused);
  GDN2_BIND(token_dstate_scan);
  GDN2_BIND(token_chunk_vjp);
  GDN2_BIND(chunk_forward);
  GDN2_BIND(chunk_forward_fused);
  GDN2_BIND(chunk_forward_kernels);
  GDN2_BIND(chunk_backward);
  GDN2_BIND(chunk_backward_kernels);
  GDN2_BIND(chunk_workspace_bytes);
  GDN2_BIND(chunk_scratch_bytes);
  GDN2_BIND(gate_prologue);
  GDN2_BIND(gate_prologue_vjp);
#undef GDN2_BIND
  if (missing) {
    PyErr_SetString(PyExc_RuntimeError, "libgdn2_b200.so lacks an entry point");
    return nullptr;
  }
  g_check = Py_NewRef(a[1]);
  g_launches = Py_NewRef(a[2]);
  g_oom = Py_NewRef(a[3]);
  g_bound = true;
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(bind), METH_FASTCALL, nullptr},
    {"forward", reinterpret_cast<PyCFunction>(forward), METH_FASTCALL, nullptr},
    {"train_forward", reinterpret_cast<PyCFunction>(train_forward), METH_FASTCALL, nullptr},
    {"train_backward", reinterpret_cast<PyCFunction>(train_backward), METH_FASTCALL, nullptr},
    {"prologue_forward", reinterpret_cast<PyCFunction>(prologue_forward), METH_FASTCALL, nullptr},
    {"prologue_backward", reinterpret_cast<PyCFunction>(prologue_backward), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Native host path of gdn2_sm120_b200.", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
