// The operators' call path in native code: a CPython module over the C ABI for torch tensors.
//
// A call on one short sequence is a few microseconds of device time; argument checks, output allocation and the
// ctypes call in Python took 13 of the 15 us such a call cost.  The functions here do the same checks on the C++
// tensors, allocate the result (and scratch memory) from torch's caching allocator and call the C ABI: about 4 us,
// half of it the launch itself.
//
// Only the straight path lives here.  Whatever is out of the ordinary -- a wrong type or shape, a tensor on another
// device, an error code -- makes a function return None without having launched anything (or after a failed
// launch), and the caller in ops.py goes through its checks again and reports what is wrong.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <initializer_list>

namespace {

using SoftmaxFn = int (*)(const void*, const void*, const void*, void*, int, int, int, int, int, int, int, float, int, void*,
                          size_t, int*, void*);
using MhaFn = int (*)(const void*, void*, int, int, int, int, int, float, int, int*, void*);
using GemmFn = int (*)(const void*, const void*, const void*, void*, int, int, int, int, int, int, int, int, void*, size_t,
                       int*, void*);
using FfnFn = int (*)(const void*, const void*, const void*, const void*, const void*, void*, int, int, int, int, int, int,
                      int, int, int, void*, size_t, int*, void*);
using BytesFn = size_t (*)(int, int, int, int, int, int, int);

SoftmaxFn g_softmax = nullptr;
MhaFn g_mha = nullptr;
GemmFn g_gemm = nullptr;
FfnFn g_ffn = nullptr;
BytesFn g_bytes = nullptr;
constexpr int kDevices = 64;
int* g_status[kDevices] = {};       // device status words, registered by ops.py

constexpr int kOpGemmReluGemm = 1, kOpLessScratch = 0x2000;

// What all tensors of a call have in common.
struct Common {
  int device = -1;
  at::ScalarType type = at::ScalarType::Undefined;
  int code = 0;
};

// The tensor behind `o` if it is a contiguous CUDA tensor that fits the call so far (the first one decides type and
// device: 16-bit floating point, on the current device).
const at::Tensor* take(PyObject* o, Common& c) {
  if (!THPVariable_Check(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.is_cuda() || t.layout() != at::kStrided || !t.is_contiguous()) return nullptr;
  const int dev = t.device().index();
  const at::ScalarType st = t.scalar_type();
  if (c.device < 0) {
    if (st == at::kHalf) c.code = 0;
    else if (st == at::kBFloat16) c.code = 1;
    else return nullptr;
    if (dev < 0 || dev >= kDevices || g_status[dev] == nullptr || dev != c10::cuda::current_device()) return nullptr;
    c.device = dev;
    c.type = st;
  } else if (dev != c.device || st != c.type) {
    return nullptr;
  }
  return &t;
}

bool fits(std::initializer_list<int64_t> v) {
  for (int64_t x : v)
    if (x < 0 || x > INT_MAX) return false;
  return true;
}

bool is_text(PyObject* o, const char* s) { return PyUnicode_Check(o) && PyUnicode_CompareWithASCIIString(o, s) == 0; }

at::Tensor make(at::IntArrayRef shape, at::ScalarType type, int device) {
  return at::detail::empty_cuda(shape, type, c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(device)), std::nullopt);
}

void* stream_of(int device) { return c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream(); }

bool shape_is(const at::Tensor& t, int64_t a, int64_t b, int64_t c) {
  return t.dim() == 3 && t.size(0) == a && t.size(1) == b && t.size(2) == c;
}

// Lets other Python threads run: around allocations and launches, which can block (a full launch queue, cudaMalloc, a queue that
// waits for a Python host callback).  Everything taken from Python objects -- addresses, shapes, texts -- is read before.
struct WithoutLock {
  PyThreadState* state = PyEval_SaveThread();
  WithoutLock() = default;
  WithoutLock(const WithoutLock&) = delete;
  WithoutLock& operator=(const WithoutLock&) = delete;
  ~WithoutLock() { PyEval_RestoreThread(state); }
};

// Runs `body` and returns what it returns; None for nullptr or an exception.
template <class F>
PyObject* guarded(F body) {
  try {
    PyObject* r = body();
    if (r != nullptr) return r;
  } catch (...) {
  }
  PyErr_Clear();
  Py_RETURN_NONE;
}

// The result: `given`, checked by the caller, or a new tensor.
class Result {
 public:
  Result(PyObject* given, const at::Tensor* t) : given_(given), address_(t ? t->data_ptr() : nullptr) {}
  // its address; allocates a new one (without the lock)
  void* address(const Common& c, at::IntArrayRef shape) {
    if (given_ != Py_None) return address_;
    fresh_ = make(shape, c.type, c.device);
    return fresh_.data_ptr();
  }
  PyObject* give() {
    if (given_ == Py_None) return THPVariable_Wrap(fresh_);
    Py_INCREF(given_);
    return given_;
  }

 private:
  PyObject* given_;
  void* address_;
  at::Tensor fresh_;
};

// Whether `given` can be the result; `t` is the tensor behind it (null for None).
bool result_ok(PyObject* given, Common& c, at::IntArrayRef shape, const at::Tensor** t) {
  *t = nullptr;
  if (given == Py_None) return true;
  *t = take(given, c);
  return *t != nullptr && (*t)->sizes() == shape;
}

// softmax(query, key, value, out, scale, key_layout, flags)
PyObject* py_softmax(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 7 || g_softmax == nullptr) return nullptr;
    Common c;
    const at::Tensor *q = take(a[0], c), *k = q ? take(a[1], c) : nullptr, *v = k ? take(a[2], c) : nullptr;
    if (v == nullptr || q->dim() != 3 || k->dim() != 3 || v->dim() != 3) return nullptr;
    int layout;
    if (is_text(a[5], "LK")) layout = 1;
    else if (is_text(a[5], "KL")) layout = 0;
    else return nullptr;
    const int64_t b = q->size(0), M = q->size(1), K = q->size(2), L = v->size(1), N = v->size(2);
    if (!(layout ? shape_is(*k, b, L, K) : shape_is(*k, b, K, L)) || v->size(0) != b || !fits({b, M, N, K, L})) return nullptr;
    const double scale = PyFloat_AsDouble(a[4]);
    const long flags = PyLong_AsLong(a[6]);
    if (PyErr_Occurred() || flags < INT_MIN || flags > INT_MAX) return nullptr;
    const int64_t shape[3] = {b, M, N};
    const at::Tensor* given;
    if (!result_ok(a[3], c, shape, &given)) return nullptr;
    const void *qp = q->data_ptr(), *kp = k->data_ptr(), *vp = v->data_ptr();
    Result out(a[3], given);
    int rc;
    {
      WithoutLock unlocked;
      rc = g_softmax(qp, kp, vp, out.address(c, shape), b, M, N, K, L, c.code, layout, static_cast<float>(scale),
                     static_cast<int>(flags), nullptr, 0, g_status[c.device], stream_of(c.device));
    }
    return rc ? nullptr : out.give();
  });
}

// mha(qkv, num_heads, out, scale, flags)
PyObject* py_mha(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 5 || g_mha == nullptr) return nullptr;
    Common c;
    const at::Tensor* x = take(a[0], c);
    if (x == nullptr || x->dim() != 3) return nullptr;
    const long heads = PyLong_AsLong(a[1]), flags = PyLong_AsLong(a[4]);
    const double scale = PyFloat_AsDouble(a[3]);
    if (PyErr_Occurred() || heads <= 0 || heads > INT_MAX || flags < INT_MIN || flags > INT_MAX) return nullptr;
    const int64_t b = x->size(0), M = x->size(1), k3 = x->size(2);
    if (k3 % (3 * heads) || !fits({b, M, k3})) return nullptr;
    const int64_t hidden = k3 / 3;
    const int64_t shape[3] = {b, M, hidden};
    const at::Tensor* given;
    if (!result_ok(a[2], c, shape, &given)) return nullptr;
    const void* xp = x->data_ptr();
    Result out(a[2], given);
    int rc;
    {
      WithoutLock unlocked;
      rc = g_mha(xp, out.address(c, shape), b, M, heads, hidden / heads, c.code, static_cast<float>(scale), static_cast<int>(flags),
                 g_status[c.device], stream_of(c.device));
    }
    return rc ? nullptr : out.give();
  });
}

// The operands of the MLP chain and the feed-forward block: x [M, K] or [batch, M, K], weights likewise.
struct Chain {
  const at::Tensor *x, *w1, *w2;
  const void *xp, *w1p, *w2p;     // their addresses
  int64_t b, M, N, K, L;
  int layout;                     // 1: weights [out, in]
  bool flat;                      // x is a matrix, and so is the result
};
bool chain_of(PyObject* px, PyObject* pw1, PyObject* pw2, PyObject* layout, Common& c, Chain& r) {
  r.x = take(px, c);
  r.w1 = r.x ? take(pw1, c) : nullptr;
  r.w2 = r.w1 ? take(pw2, c) : nullptr;
  if (r.w2 == nullptr) return false;
  if (is_text(layout, "OI")) r.layout = 1;
  else if (is_text(layout, "IO")) r.layout = 0;
  else return false;
  auto dims = [](const at::Tensor& t, int64_t (&d)[3]) {
    if (t.dim() != 2 && t.dim() != 3) return false;
    d[0] = t.dim() == 3 ? t.size(0) : 1;
    d[1] = t.size(t.dim() - 2);
    d[2] = t.size(t.dim() - 1);
    return true;
  };
  int64_t x[3], u[3], v[3];
  if (!dims(*r.x, x) || !dims(*r.w1, u) || !dims(*r.w2, v)) return false;
  r.flat = r.x->dim() == 2;
  r.b = x[0];
  r.M = x[1];
  r.K = x[2];
  r.L = r.layout ? u[1] : u[2];
  r.N = r.layout ? v[1] : v[2];
  r.xp = r.x->data_ptr();
  r.w1p = r.w1->data_ptr();
  r.w2p = r.w2->data_ptr();
  return u[0] == r.b && v[0] == r.b && (r.layout ? u[2] : u[1]) == r.K && (r.layout ? v[2] : v[1]) == r.L &&
         fits({r.b, r.M, r.N, r.K, r.L});
}
// As the operators' Python path takes it: a given result may be a matrix or have a batch dimension of its own.
bool chain_result_ok(PyObject* given, Common& c, const Chain& r, const at::Tensor** t) {
  *t = nullptr;
  if (given == Py_None) return true;
  *t = take(given, c);
  return *t != nullptr && (((*t)->dim() == 2 && r.b == 1 && (*t)->size(0) == r.M && (*t)->size(1) == r.N) || shape_is(**t, r.b, r.M, r.N));
}
// The shape of a new result.
struct ChainShape {
  int64_t d[3];
  bool flat;
  explicit ChainShape(const Chain& r) : d{r.b, r.M, r.N}, flat(r.flat) {}
  operator at::IntArrayRef() const { return flat ? at::IntArrayRef(d + 1, 2) : at::IntArrayRef(d, 3); }
};
// Whether the caching allocator can be expected to have `bytes` more in one piece: cached, or free on the device and within the process's share.
// Asked before a large request, because one that fails is dear: the allocator gives all its cached blocks back first, waiting for the device
// (16384 x 1024 -> 4096 -> 1024 with 100 MB left and no such question: 1073 us a call, 209 with it).
// An allocator that cannot tell is asked for the memory itself.
bool room_for(int device, size_t bytes) {
  if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) return true;
  try {
    const auto index = static_cast<c10::DeviceIndex>(device);
    const auto s = c10::cuda::CUDACachingAllocator::getDeviceStats(index);
    const size_t reserved = static_cast<size_t>(s.reserved_bytes[0].current);
    // what the allocator can give back: cached segments of which no part is in use
    const size_t whole = reserved - static_cast<size_t>(s.allocated_bytes[0].current) - static_cast<size_t>(s.inactive_split_bytes[0].current);
    if (whole >= bytes) return true;
    size_t free = 0, total = 0, largest = 1;       // (a largest block of 0 would ask the device)
    if (cudaMemGetInfo(&free, &total) != cudaSuccess) {
      cudaGetLastError();
      return true;
    }
    const double share = c10::cuda::CUDACachingAllocator::getMemoryFraction(index) * static_cast<double>(total);
    const size_t allowed = share > static_cast<double>(reserved) ? static_cast<size_t>(share) - reserved : 0;
    if (whole + std::min(free, allowed) >= bytes) return true;
    c10::cuda::CUDACachingAllocator::cacheInfo(index, &largest);       // (walks all cached blocks)
    return largest >= bytes;
  } catch (const std::exception&) {
    return true;
  }
}
constexpr size_t kLargeScratch = 48u << 20;      // (what the question costs counts in small calls)

// Scratch memory of a call, in stream order from the caching allocator: its own for every stream, thread and captured graph.
// Where there is no memory left for the whole hidden layer of a large call, the ring of the next best form; none where there is
// none for that: the call then takes the form that needs none.
at::Tensor scratch_for(const Common& c, int64_t b, int64_t M, int64_t N, int64_t K, int64_t L, size_t* bytes) {
  for (const int op : {kOpGemmReluGemm, kOpGemmReluGemm | kOpLessScratch}) {
    *bytes = g_bytes(op, b, M, N, K, L, c.code);
    if (*bytes == 0) break;
    if (*bytes <= kLargeScratch || room_for(c.device, *bytes)) {
      try {
        return make({static_cast<int64_t>(*bytes)}, at::kByte, c.device);
      } catch (const c10::OutOfMemoryError&) {
      }
    }
    *bytes = 0;
  }
  return at::Tensor();
}

// gemm(x, w1, w2, out, activation, weight_layout, scratch)
PyObject* py_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 7 || g_gemm == nullptr) return nullptr;
    int act;
    if (is_text(a[4], "relu")) act = 1;
    else if (is_text(a[4], "identity")) act = 0;
    else return nullptr;
    Common c;
    Chain r;
    if (!chain_of(a[0], a[1], a[2], a[5], c, r)) return nullptr;
    const at::Tensor* given;
    if (!chain_result_ok(a[3], c, r, &given)) return nullptr;
    const bool scratch = a[6] == Py_True;
    Result out(a[3], given);
    int rc;
    {
      WithoutLock unlocked;
      size_t bytes = 0;
      at::Tensor ws;
      void* y = out.address(c, ChainShape(r));
      if (scratch) ws = scratch_for(c, r.b, r.M, r.N, r.K, r.L, &bytes);
      rc = g_gemm(r.xp, r.w1p, r.w2p, y, r.b, r.M, r.N, r.K, r.L, c.code, r.layout, act, bytes ? ws.data_ptr() : nullptr, bytes,
                  g_status[c.device], stream_of(c.device));
    }
    return rc ? nullptr : out.give();
  });
}

int act_code(PyObject* o) { return is_text(o, "identity") ? 0 : is_text(o, "relu") ? 1 : is_text(o, "gelu") ? 2 : -1; }

// ffn(x, w1, b1, w2, b2, out, act1, act2, weight_layout)
PyObject* py_ffn(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n != 9 || g_ffn == nullptr) return nullptr;
    const int act1 = act_code(a[6]), act2 = act_code(a[7]);
    if (act1 < 0 || act2 < 0) return nullptr;
    Common c;
    Chain r;
    if (!chain_of(a[0], a[1], a[3], a[8], c, r)) return nullptr;
    const void* bias[2] = {nullptr, nullptr};
    for (int i = 0; i < 2; ++i) {
      PyObject* o = a[i == 0 ? 2 : 4];
      if (o == Py_None) continue;
      const at::Tensor* t = take(o, c);
      if (t == nullptr || t->numel() != r.b * (i == 0 ? r.L : r.N)) return nullptr;
      bias[i] = t->data_ptr();
    }
    const at::Tensor* given;
    if (!chain_result_ok(a[5], c, r, &given)) return nullptr;
    Result out(a[5], given);
    int rc;
    {
      WithoutLock unlocked;
      size_t bytes = 0;
      void* y = out.address(c, ChainShape(r));
      at::Tensor ws = scratch_for(c, r.b, r.M, r.N, r.K, r.L, &bytes);
      rc = g_ffn(r.xp, r.w1p, bias[0], r.w2p, bias[1], y, r.b, r.M, r.N, r.K, r.L, c.code, r.layout, act1, act2,
                 bytes ? ws.data_ptr() : nullptr, bytes, g_status[c.device], stream_of(c.device));
    }
    return rc ? nullptr : out.give();
  });
}

// A built module's compiled shape: plan(kind, batch, M, N, K, L, type code, heads, scale, act1, act2, bias1, bias2).
struct Plan {
  int kind;                       // 0 softmax, 1 GEMM chain, 2 packed attention, 3 feed-forward
  int64_t b, M, N, K, L;
  int code, heads, act1, act2, bias1, bias2;
  float scale;
};
constexpr const char* kPlanName = "ditto_b200.plan";
void free_plan(PyObject* cap) { delete static_cast<Plan*>(PyCapsule_GetPointer(cap, kPlanName)); }
PyObject* py_plan(PyObject*, PyObject* args) {
  Plan p;
  long long b, M, N, K, L;
  if (!PyArg_ParseTuple(args, "iLLLLLiifiiii", &p.kind, &b, &M, &N, &K, &L, &p.code, &p.heads, &p.scale, &p.act1, &p.act2, &p.bias1,
                        &p.bias2))
    return nullptr;
  p.b = b, p.M = M, p.N = N, p.K = K, p.L = L;
  return PyCapsule_New(new Plan(p), kPlanName, free_plan);
}

// call(plan, *tensors) -> True, or None where the checked path has to look at the arguments
PyObject* py_call(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    if (n < 3 || !PyCapsule_IsValid(a[0], kPlanName)) return nullptr;
    const Plan& p = *static_cast<const Plan*>(PyCapsule_GetPointer(a[0], kPlanName));
    const at::Tensor* t[6];
    void* ptr[6];
    const int count = static_cast<int>(n - 1);
    if (count > 6) return nullptr;
    Common c;
    for (int i = 0; i < count; ++i) {
      if ((t[i] = take(a[i + 1], c)) == nullptr) return nullptr;
      ptr[i] = t[i]->data_ptr();
    }
    if (c.code != p.code) return nullptr;
    int* status = g_status[c.device];
    if (p.kind <= 1) {
      if (count != 4 || !shape_is(*t[0], p.b, p.M, p.K) || !shape_is(*t[1], p.b, p.K, p.L) || !shape_is(*t[2], p.b, p.L, p.N) ||
          !shape_is(*t[3], p.b, p.M, p.N))
        return nullptr;
    } else if (p.kind == 2) {
      if (count != 2 || !shape_is(*t[0], p.b, p.M, 3 * p.N) || !shape_is(*t[1], p.b, p.M, p.N)) return nullptr;
    } else {
      // x, w1 [L, K], (b1 [L]), w2 [N, L], (b2 [N]), out; x and out keep whatever leading dimensions the layer has
      if (count != 4 + p.bias1 + p.bias2) return nullptr;
      const int i2 = 2 + p.bias1;                      // w2
      auto matrix = [](const at::Tensor& m, int64_t r, int64_t k) { return m.dim() == 2 && m.size(0) == r && m.size(1) == k; };
      auto vector = [](const at::Tensor& v, int64_t k) { return v.dim() == 1 && v.size(0) == k; };
      if (t[0]->numel() != p.M * p.K || t[count - 1]->numel() != p.M * p.N || !matrix(*t[1], p.L, p.K) || !matrix(*t[i2], p.N, p.L) ||
          (p.bias1 && !vector(*t[2], p.L)) || (p.bias2 && !vector(*t[i2 + 1], p.N)))
        return nullptr;
    }
    int rc = -1;
    {
      WithoutLock unlocked;
      void* stream = stream_of(c.device);
      size_t bytes = 0;
      at::Tensor ws;
      if (p.kind == 0) {
        rc = g_softmax(ptr[0], ptr[1], ptr[2], ptr[3], p.b, p.M, p.N, p.K, p.L, p.code, 0, p.scale, 0, nullptr, 0, status, stream);
      } else if (p.kind == 1) {
        ws = scratch_for(c, p.b, p.M, p.N, p.K, p.L, &bytes);
        rc = g_gemm(ptr[0], ptr[1], ptr[2], ptr[3], p.b, p.M, p.N, p.K, p.L, p.code, 0, p.act1, bytes ? ws.data_ptr() : nullptr, bytes,
                    status, stream);
      } else if (p.kind == 2) {
        rc = g_mha(ptr[0], ptr[1], p.b, p.M, p.heads, p.N / p.heads, p.code, p.scale, 0, status, stream);
      } else {
        const int i2 = 2 + p.bias1;
        ws = scratch_for(c, 1, p.M, p.N, p.K, p.L, &bytes);
        rc = g_ffn(ptr[0], ptr[1], p.bias1 ? ptr[2] : nullptr, ptr[i2], p.bias2 ? ptr[i2 + 1] : nullptr, ptr[count - 1], 1, p.M, p.N, p.K,
                   p.L, p.code, 1, p.act1, p.act2, bytes ? ws.data_ptr() : nullptr, bytes, status, stream);
      }
    }
    if (rc != 0) return nullptr;
    Py_RETURN_TRUE;
  });
}

// bind(softmax, mha, gemm, ffn, bytes): addresses of the C entry points
PyObject* py_bind(PyObject*, PyObject* args) {
  unsigned long long s, m, g, f, b;
  if (!PyArg_ParseTuple(args, "KKKKK", &s, &m, &g, &f, &b)) return nullptr;
  g_softmax = reinterpret_cast<SoftmaxFn>(s);
  g_mha = reinterpret_cast<MhaFn>(m);
  g_gemm = reinterpret_cast<GemmFn>(g);
  g_ffn = reinterpret_cast<FfnFn>(f);
  g_bytes = reinterpret_cast<BytesFn>(b);
  Py_RETURN_NONE;
}
// status(device index, address of its status word)
PyObject* py_status(PyObject*, PyObject* args) {
  int dev;
  unsigned long long p;
  if (!PyArg_ParseTuple(args, "iK", &dev, &p)) return nullptr;
  if (dev >= 0 && dev < kDevices) g_status[dev] = reinterpret_cast<int*>(p);
  Py_RETURN_NONE;
}

#define DITTO_FAST(name, fn) {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(fn)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {DITTO_FAST("softmax", py_softmax),
                          DITTO_FAST("mha", py_mha),
                          DITTO_FAST("gemm", py_gemm),
                          DITTO_FAST("ffn", py_ffn),
                          DITTO_FAST("call", py_call),
                          {"plan", py_plan, METH_VARARGS, nullptr},
                          {"bind", py_bind, METH_VARARGS, nullptr},
                          {"status", py_status, METH_VARARGS, nullptr},
                          {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_fastcall", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fastcall(void) { return PyModule_Create(&kModule); }
