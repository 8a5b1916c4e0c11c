// Native front of the short calls in ops.py.
//
// A back-to-back GEMM of 2 MB or one attention head block runs for 5..10 us on the device, while the
// checks, attribute reads, context managers and ctypes conversions of the Python path cost 17 us of
// host time per call: such a call was bound by the host, whatever the kernel did.  The functions here
// take the call's objects as they are, read shapes, types and pointers from the tensors in C++,
// allocate the result through the same caching allocator and enter the C ABI with the current
// stream of the inputs' device (4..6 us per call, most of it the allocation and the launch).  The calls of the word
// program (lookup, packing, ragged LSTM, projection) are here too: a pass of a small model was bound by their host time.
//
// They are the accepting half only: whatever is not the plain, valid call (a wrong type or shape, a
// tensor on the CPU, no workspace on that device yet, no memory for the result) is answered with
// None before the library is entered, and ops.py goes through its Python checks, which raise.  An error of
// the library is answered with its status number: it may come after a launch, and the call is not made again.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/version.h>

#include <algorithm>
#include <vector>

#include "../../include/ftb200.h"

namespace {

// A contiguous CUDA tensor, or nullptr.
const at::Tensor* cuda_tensor(PyObject* o) {
  if (!THPVariable_Check(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.is_contiguous() ? &t : nullptr;
}

int dtype_code(const at::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return FTB_DTYPE_F32;
    case at::kHalf: return FTB_DTYPE_F16;
    case at::kBFloat16: return FTB_DTYPE_BF16;
    default: return -1;
  }
}

bool same_kind(const at::Tensor& a, const at::Tensor& b) {
  return a.scalar_type() == b.scalar_type() && a.device() == b.device();
}

bool get_int(PyObject* o, int64_t* v) {
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  *v = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0 && *v >= -0x7fffffffLL && *v <= 0x7fffffffLL;
}

bool get_float(PyObject* o, float* v) {
  if (!PyFloat_CheckExact(o)) return false;
  *v = static_cast<float>(PyFloat_AS_DOUBLE(o));
  return true;
}

void* stream_of(c10::DeviceIndex dev) { return c10::cuda::getCurrentCUDAStream(dev).stream(); }

// The workspace ops.py keeps for the current stream of `dev` in its dictionary {(device index, stream
// handle): uint8 tensor}; undefined when there is none yet or it is smaller than `bytes`.  (Held by value:
// another thread may put a larger one in its place while this call runs.)
at::Tensor workspace_of(PyObject* dict, c10::DeviceIndex dev, size_t bytes) {
  PyObject* key = Py_BuildValue("(iK)", static_cast<int>(dev), reinterpret_cast<unsigned long long>(stream_of(dev)));
  PyObject* t = key != nullptr && PyDict_Check(dict) ? PyDict_GetItemWithError(dict, key) : nullptr;
  Py_XDECREF(key);
  if (t == nullptr) {
    PyErr_Clear();
    return at::Tensor();
  }
  const at::Tensor* ws = cuda_tensor(t);
  return ws != nullptr && static_cast<size_t>(ws->numel()) >= bytes ? *ws : at::Tensor();
}

// What follows runs without the GIL: allocating may free memory and wait, and a launch waits while the
// stream's queue is full.  Other Python threads go on meanwhile, as they do around a ctypes call.
class WithoutGil {
 public:
  WithoutGil() : state_(PyEval_SaveThread()) {}
  ~WithoutGil() { PyEval_RestoreThread(state_); }
  WithoutGil(const WithoutGil&) = delete;
  WithoutGil& operator=(const WithoutGil&) = delete;

 private:
  PyThreadState* state_;
};

// *o: `out` if the caller gave one, undefined for None; false when the given one does not fit.
bool given_result(PyObject* out, const at::Tensor& like, at::IntArrayRef shape, at::Tensor* o) {
  if (out == Py_None) return true;
  const at::Tensor* t = cuda_tensor(out);
  if (t == nullptr || !same_kind(*t, like) || t->sizes() != shape) return false;
  *o = *t;
  return true;
}
at::Tensor new_result(const at::Tensor& like, at::IntArrayRef shape) {
  return at::empty(shape, at::TensorOptions().dtype(like.scalar_type()).device(like.device()));
}

#define DECLINE_UNLESS(cond) \
  do {                       \
    if (!(cond)) Py_RETURN_NONE; \
  } while (0)

template <typename F>
PyObject* guarded(F f) {
  try {
    return f();
  } catch (const std::exception&) {
    // No memory for the result, or an error of earlier work: the Python path meets it too and raises torch's type.
    PyErr_Clear();
    Py_RETURN_NONE;
  }
}

// (A, B, C, out, workspaces)
PyObject* b2b_gemm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    DECLINE_UNLESS(n == 5);
    const at::Tensor *A = cuda_tensor(args[0]), *B = cuda_tensor(args[1]), *C = cuda_tensor(args[2]);
    DECLINE_UNLESS(A && B && C && same_kind(*A, *B) && same_kind(*A, *C));
    DECLINE_UNLESS(A->dim() == 3 && B->dim() == 3 && C->dim() == 3);
    const int64_t batch = A->size(0), M = A->size(1), K = A->size(2), N = B->size(1), P = C->size(1);
    DECLINE_UNLESS(B->size(0) == batch && B->size(2) == K && C->size(0) == batch && C->size(2) == N);
    DECLINE_UNLESS(batch <= 0x7fffffff && M <= 0x7fffffff);
    const int dt = dtype_code(*A);
    DECLINE_UNLESS(dt >= 0);
    const c10::DeviceIndex dev = A->device().index();
    const at::Tensor ws = workspace_of(args[4], dev, ftb_workspace_bytes());
    DECLINE_UNLESS(ws.defined());
    at::Tensor out;
    DECLINE_UNLESS(given_result(args[3], *A, {batch, M, P}, &out));
    int rc;
    {
      const WithoutGil released;
      const c10::cuda::CUDAGuard guard(dev);
      if (!out.defined()) out = new_result(*A, {batch, M, P});
      rc = ftb_b2b_gemm(A->data_ptr(), B->data_ptr(), C->data_ptr(), out.data_ptr(), static_cast<int>(batch),
                        static_cast<int>(M), static_cast<int>(N), static_cast<int>(K), static_cast<int>(P), dt,
                        ws.data_ptr(), ws.numel(), stream_of(dev));
    }
    return rc == 0 ? THPVariable_Wrap(out) : PyLong_FromLong(rc);
  });
}

// (q, k, v, out, scale, mode, left, right, workspaces); mode 0 full, 1 causal, 2 window (`left` keys
// that end at the query), 3 local
PyObject* flash_attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    DECLINE_UNLESS(n == 9);
    const at::Tensor *q = cuda_tensor(args[0]), *k = cuda_tensor(args[1]), *v = cuda_tensor(args[2]);
    DECLINE_UNLESS(q && k && v && same_kind(*q, *k) && same_kind(*q, *v) && q->dim() == 4);
    DECLINE_UNLESS(k->sizes() == q->sizes() && v->sizes() == q->sizes());
    float scale;
    int64_t mode, left, right;
    DECLINE_UNLESS(get_float(args[4], &scale) && get_int(args[5], &mode) && get_int(args[6], &left) &&
                   get_int(args[7], &right));
    for (int i = 0; i < 4; ++i) DECLINE_UNLESS(q->size(i) <= 0x7fffffff);
    const int B = static_cast<int>(q->size(0)), h = static_cast<int>(q->size(1)), S = static_cast<int>(q->size(2)),
              d = static_cast<int>(q->size(3)), dt = dtype_code(*q);
    DECLINE_UNLESS(dt >= 0);
    const c10::DeviceIndex dev = q->device().index();
    const at::Tensor ws = workspace_of(args[8], dev, ftb_workspace_bytes());
    DECLINE_UNLESS(ws.defined());
    at::Tensor out;
    DECLINE_UNLESS(given_result(args[3], *q, q->sizes(), &out));
    int rc;
    {
      const WithoutGil released;
      const c10::cuda::CUDAGuard guard(dev);
      if (!out.defined()) out = new_result(*q, q->sizes());
      const void *qp = q->data_ptr(), *kp = k->data_ptr(), *vp = v->data_ptr();
      void *op = out.data_ptr(), *wp = ws.data_ptr(), *st = stream_of(dev);
      const size_t wb = ws.numel();
      switch (mode) {
        case 0: rc = ftb_flash_attn_fwd(qp, kp, vp, op, B, h, S, d, scale, dt, wp, wb, st); break;
        case 1: rc = ftb_flash_attn_causal_fwd(qp, kp, vp, op, B, h, S, d, scale, dt, wp, wb, st); break;
        case 2:
          rc = ftb_flash_attn_window_fwd(qp, kp, vp, op, B, h, S, d, static_cast<int>(left), scale, dt, wp, wb, st);
          break;
        default:
          rc = ftb_flash_attn_local_fwd(qp, kp, vp, op, B, h, S, d, static_cast<int>(left), static_cast<int>(right),
                                        scale, dt, wp, wb, st);
      }
    }
    return rc == 0 ? THPVariable_Wrap(out) : PyLong_FromLong(rc);
  });
}

// (q, k, v, rand_pos | None, out, window, dilation, n_global, scale, as_shipped, workspaces)
PyObject* sparse_attention(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    DECLINE_UNLESS(n == 11);
    const at::Tensor *q = cuda_tensor(args[0]), *k = cuda_tensor(args[1]), *v = cuda_tensor(args[2]);
    DECLINE_UNLESS(q && k && v && same_kind(*q, *k) && same_kind(*q, *v) && q->dim() == 4);
    DECLINE_UNLESS(k->sizes() == q->sizes() && v->sizes() == q->sizes());
    int64_t window, dilation, ng;
    float scale;
    DECLINE_UNLESS(get_int(args[5], &window) && get_int(args[6], &dilation) && get_int(args[7], &ng) &&
                   get_float(args[8], &scale) && (args[9] == Py_True || args[9] == Py_False));
    for (int i = 0; i < 4; ++i) DECLINE_UNLESS(q->size(i) <= 0x7fffffff);
    const int64_t S = q->size(2), inner = S - 2 * ng;
    DECLINE_UNLESS(ng >= 0 && inner >= 0);
    int64_t R = 0;
    const int* pos = nullptr;
    if (args[3] != Py_None) {
      const at::Tensor* p = cuda_tensor(args[3]);
      DECLINE_UNLESS(p && p->scalar_type() == at::kInt && p->device() == q->device() && p->dim() == 4);
      DECLINE_UNLESS(p->size(0) == q->size(0) && p->size(1) == q->size(1) && p->size(2) == inner);
      R = p->size(3);
      DECLINE_UNLESS(R <= 0x7fffffff);
      if (R > 0) pos = static_cast<const int*>(p->data_ptr());
    }
    const int dt = dtype_code(*q);
    DECLINE_UNLESS(dt >= 0);
    const c10::DeviceIndex dev = q->device().index();
    const int as_shipped = args[9] == Py_True ? 1 : 0;
    const at::Tensor ws = workspace_of(args[10], dev, ftb_workspace_bytes());
    DECLINE_UNLESS(ws.defined());
    at::Tensor out;
    DECLINE_UNLESS(given_result(args[4], *q, q->sizes(), &out));
    int rc;
    {
      const WithoutGil released;
      const c10::cuda::CUDAGuard guard(dev);
      if (!out.defined()) out = new_result(*q, q->sizes());
      rc = ftb_sparse_attn_fwd(q->data_ptr(), k->data_ptr(), v->data_ptr(), pos, out.data_ptr(),
                               static_cast<int>(q->size(0)), static_cast<int>(q->size(1)), static_cast<int>(S),
                               static_cast<int>(q->size(3)), static_cast<int>(window), static_cast<int>(dilation),
                               static_cast<int>(ng), static_cast<int>(R), scale, as_shipped, dt, ws.data_ptr(),
                               ws.numel(), stream_of(dev));
    }
    return rc == 0 ? THPVariable_Wrap(out) : PyLong_FromLong(rc);
  });
}

// (table, ids, out, workspaces)
PyObject* embedding_gather(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    DECLINE_UNLESS(n == 4);
    const at::Tensor *table = cuda_tensor(args[0]), *ids = cuda_tensor(args[1]);
    DECLINE_UNLESS(table && ids && table->dim() == 2 && ids->scalar_type() == at::kLong && ids->device() == table->device());
    const int64_t V = table->size(0), H = table->size(1), T = ids->numel();
    const int dt = dtype_code(*table);
    DECLINE_UNLESS(dt >= 0 && H <= 0x7fffffff);
    const c10::DeviceIndex dev = table->device().index();
    const at::Tensor ws = workspace_of(args[3], dev, ftb_workspace_bytes());
    DECLINE_UNLESS(ws.defined());
    at::Tensor out;
    DECLINE_UNLESS(given_result(args[2], *table, {T, H}, &out));
    int rc;
    {
      const WithoutGil released;
      const c10::cuda::CUDAGuard guard(dev);
      if (!out.defined()) out = new_result(*table, {T, H});
      rc = ftb_embedding_gather(table->data_ptr(), static_cast<const long long*>(ids->data_ptr()), out.data_ptr(), T, V,
                                static_cast<int>(H), dt, ws.data_ptr(), ws.numel(), stream_of(dev));
    }
    return rc == 0 ? THPVariable_Wrap(out) : PyLong_FromLong(rc);
  });
}

// (W, U, bias | None) -> (Wp, bias_p | None)
PyObject* lstm_pack_weights(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    DECLINE_UNLESS(n == 3);
    const at::Tensor *W = cuda_tensor(args[0]), *U = cuda_tensor(args[1]);
    DECLINE_UNLESS(W && U && same_kind(*W, *U) && W->dim() == 4 && U->dim() == 4);
    const int64_t D = W->size(0), I = W->size(2), H = W->size(3);
    DECLINE_UNLESS(W->size(1) == 4 && U->size(0) == D && U->size(1) == 4 && U->size(2) == H && U->size(3) == H);
    DECLINE_UNLESS(D <= 0x7fffffff && I <= 0x7fffffff && H <= 0x7fffffff);
    const at::Tensor* b = nullptr;
    if (args[2] != Py_None) {
      b = cuda_tensor(args[2]);
      DECLINE_UNLESS(b && same_kind(*b, *W) && b->numel() == D * 4 * H);
    }
    const int dt = dtype_code(*W);
    DECLINE_UNLESS(dt >= 0);
    at::Tensor Wp, bias_p;
    int rc;
    {
      const WithoutGil released;
      const c10::DeviceIndex dev = W->device().index();
      const c10::cuda::CUDAGuard guard(dev);
      Wp = new_result(*W, {D, 4 * H, I + H});
      if (b) bias_p = at::empty({D, 4 * H}, at::TensorOptions().dtype(at::kFloat).device(W->device()));
      rc = ftb_lstm_pack_weights(W->data_ptr(), U->data_ptr(), b ? b->data_ptr() : nullptr, Wp.data_ptr(),
                                 b ? static_cast<float*>(bias_p.data_ptr()) : nullptr, static_cast<int>(D), static_cast<int>(I),
                                 static_cast<int>(H), dt, stream_of(dev));
    }
    if (rc != 0) return PyLong_FromLong(rc);
    PyObject* bias = Py_None;
    if (b) bias = THPVariable_Wrap(bias_p); else Py_INCREF(bias);
    return Py_BuildValue("(NN)", THPVariable_Wrap(Wp), bias);
  });
}

// (x, lens, Wp, bias_p | None, workspace): the caller holds the workspace's turn
PyObject* lstm_stacked_ragged(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    DECLINE_UNLESS(n == 5);
    const at::Tensor *x = cuda_tensor(args[0]), *Wp = cuda_tensor(args[2]), *ws = cuda_tensor(args[4]);
    DECLINE_UNLESS(x && Wp && ws && same_kind(*x, *Wp) && ws->device() == x->device() && ws->scalar_type() == at::kByte);
    DECLINE_UNLESS(x->dim() == 2 && Wp->dim() == 3 && PyList_CheckExact(args[1]));
    const Py_ssize_t N = PyList_GET_SIZE(args[1]);
    DECLINE_UNLESS(N > 0 && N <= 0x7fffffff);
    std::vector<int> lens(static_cast<size_t>(N));
    int64_t T = 0;
    int L = 0;
    for (Py_ssize_t i = 0; i < N; ++i) {
      int64_t v;
      DECLINE_UNLESS(get_int(PyList_GET_ITEM(args[1], i), &v) && v > 0);
      lens[i] = static_cast<int>(v);
      L = std::max(L, lens[i]);
      T += v;
    }
    const int64_t D = Wp->size(0), H = Wp->size(1) / 4, I = x->size(1);
    DECLINE_UNLESS(x->size(0) == T && Wp->size(1) == 4 * H && Wp->size(2) == I + H && D <= 0x7fffffff && I + H <= 0x7fffffff);
    const at::Tensor* b = nullptr;
    if (args[3] != Py_None) {
      b = cuda_tensor(args[3]);
      DECLINE_UNLESS(b && b->scalar_type() == at::kFloat && b->device() == x->device() && b->dim() == 2 && b->size(0) == D &&
                     b->size(1) == 4 * H);
    }
    const int dt = dtype_code(*x);
    DECLINE_UNLESS(dt >= 0);
    at::Tensor out;
    int rc;
    {
      const WithoutGil released;
      const c10::DeviceIndex dev = x->device().index();
      const c10::cuda::CUDAGuard guard(dev);
      const auto bytes = at::TensorOptions().dtype(at::kByte).device(x->device());
      // the packed input, and behind it the rows' tables, the call's own: they are read again behind the LSTM
      const int64_t rows = x->numel() * x->element_size();
      const size_t tables = ftb_lstm_stacked_ragged_scratch_bytes(L, static_cast<int>(N));
      const at::Tensor xt = at::empty({rows + static_cast<int64_t>(tables)}, bytes);
      const at::Tensor hs = new_result(*x, {D, T, H});
      const at::Tensor c = at::empty({D, N, H}, bytes.dtype(at::kFloat));
      out = new_result(*x, {T, H});
      rc = ftb_lstm_stacked_ragged_fwd_scratch(x->data_ptr(), Wp->data_ptr(), b ? static_cast<const float*>(b->data_ptr()) : nullptr,
                                               lens.data(), xt.data_ptr(), hs.data_ptr(), static_cast<float*>(c.data_ptr()),
                                               out.data_ptr(), static_cast<int>(D), static_cast<int>(N), static_cast<int>(I),
                                               static_cast<int>(H), dt, static_cast<char*>(xt.data_ptr()) + rows, tables,
                                               ws->data_ptr(), ws->numel(), stream_of(dev));
    }
    return rc == 0 ? THPVariable_Wrap(out) : PyLong_FromLong(rc);
  });
}

// (h, P, workspaces): probabilities from P [H, V] as it is
PyObject* project_softmax(PyObject*, PyObject* const* args, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    DECLINE_UNLESS(n == 3);
    const at::Tensor *h = cuda_tensor(args[0]), *P = cuda_tensor(args[1]);
    DECLINE_UNLESS(h && P && same_kind(*h, *P) && P->dim() == 2 && h->dim() > 0);
    const int64_t H = P->size(0), V = P->size(1);
    DECLINE_UNLESS(h->size(-1) == H && H > 0 && H % 64 == 0 && V > 0 && V % 8 == 0 && V <= 48 * 1024);
    const int64_t T = h->numel() / H;
    const int dt = dtype_code(*h);
    DECLINE_UNLESS(dt >= 0 && T > 0 && (reinterpret_cast<uintptr_t>(h->data_ptr()) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(P->data_ptr()) & 15) == 0);
    const size_t bytes = ftb_project_softmax_scratch_bytes(T, static_cast<int>(V), static_cast<int>(H), dt, 1);
    DECLINE_UNLESS(bytes > 0);
    const c10::DeviceIndex dev = h->device().index();
    const at::Tensor ws = workspace_of(args[2], dev, ftb_workspace_bytes());
    DECLINE_UNLESS(ws.defined());
    at::Tensor probs;
    int rc;
    {
      const WithoutGil released;
      const c10::cuda::CUDAGuard guard(dev);
      probs = at::empty({T, V}, at::TensorOptions().dtype(at::kFloat).device(h->device()));
      const at::Tensor scratch = at::empty({static_cast<int64_t>(bytes)}, at::TensorOptions().dtype(at::kByte).device(h->device()));
      rc = ftb_project_softmax_fwd(h->data_ptr(), P->data_ptr(), 1, static_cast<float*>(probs.data_ptr()), V, T, static_cast<int>(V),
                                   static_cast<int>(H), dt, scratch.data_ptr(), bytes, ws.data_ptr(), ws.numel(), stream_of(dev));
    }
    return rc == 0 ? THPVariable_Wrap(probs) : PyLong_FromLong(rc);
  });
}

// (device index, -1: the current one) -> handle of its current stream.  (torch.cuda.current_stream makes a
// stream object for it: 2 us, three times in a call of the word program.)
PyObject* current_stream(PyObject*, PyObject* const* args, Py_ssize_t n) {
  int64_t dev;
  if (n != 1 || !get_int(args[0], &dev) || dev < -1 || dev > 127) {
    PyErr_SetString(PyExc_TypeError, "current_stream: expected a device index");
    return nullptr;
  }
  try {
    return PyLong_FromVoidPtr(stream_of(static_cast<c10::DeviceIndex>(dev)));
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

template <typename F>
PyCFunction as_method(F f) { return reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(f)); }

PyMethodDef kMethods[] = {
    {"b2b_gemm", as_method(b2b_gemm), METH_FASTCALL, nullptr},
    {"flash_attention", as_method(flash_attention), METH_FASTCALL, nullptr},
    {"sparse_attention", as_method(sparse_attention), METH_FASTCALL, nullptr},
    {"embedding_gather", as_method(embedding_gather), METH_FASTCALL, nullptr},
    {"lstm_pack_weights", as_method(lstm_pack_weights), METH_FASTCALL, nullptr},
    {"lstm_stacked_ragged", as_method(lstm_stacked_ragged), METH_FASTCALL, nullptr},
    {"project_softmax", as_method(project_softmax), METH_FASTCALL, nullptr},
    {"current_stream", as_method(current_stream), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_host", "Native front of the short calls in ops.py.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  PyObject* m = PyModule_Create(&kModule);
  // the torch whose headers this was built against: _lib.py uses the module with that one only
  if (m != nullptr && PyModule_AddStringConstant(m, "torch_version", TORCH_VERSION) < 0) Py_CLEAR(m);
  return m;
}
