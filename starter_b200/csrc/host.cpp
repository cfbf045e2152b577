// The host side of a launch as native code: entry points that take tensors, the check that stands in front of every operand, an
// output's allocation and the current stream.  A step of a few hundred tokens is ten launches of a few microseconds each on the
// device; written in Python with ctypes a launch took 8 to 11 us on the host (rmsnorm: 8.2, now 5.9), of which the driver's own part is
// under 3: a latent layer of 78 tokens 139 -> 78 us, a window layer of 466 90 -> 59, a dense layer of 300 behind 1,000 107 -> 87.
//
// An Entry calls a library's entry point by its address.  The kernels' entry points take integers, addresses and floats only, and
// return an integer or nothing; on the calling conventions of x86-64 (System V) and of 64-bit ARM arguments of the two classes are
// handed out independently, in order (first registers, then eight-byte places on the stack), a float in the low half of its
// register, and the caller clears the stack.  So one call with every place filled serves all signatures; Entry counts what it is
// given against the declared arguments.
#include <Python.h>

#include <ATen/Context.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/autocast_mode.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/core/LegacyTypeDispatch.h>
#include <ATen/record_function.h>
#include <ATen/ops/mm_cuda_dispatch.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cstring>
#include <functional>
#include <utility>
#include <vector>

namespace {

constexpr int MAX_INTS = 40, MAX_FLOATS = 8;
typedef unsigned long long word;
typedef word (*Function)(word, word, word, word, word, word, double, double, double, double, double, double, double, double, word, word,
                         word, word, word, word, word, word, word, word, word, word, word, word, word, word, word, word, word, word,
                         word, word, word, word, word, word, word, word, word, word, word, word, word, word);

struct Entry {
  PyObject_HEAD
  vectorcallfunc call;
  Function function;
  char result;                     // 'i': int, 'l': long long, 'v': nothing
  int count;
  char kinds[MAX_INTS + MAX_FLOATS];       // 'p': address (or a tensor, or None), 'i': integer, 'f': float
};

// An argument as a word; false with an exception set.
bool as_word(PyObject* o, char kind, word& out) {
  if (PyLong_Check(o)) {
    out = PyLong_AsUnsignedLongLongMask(o);
    return !(out == ~0ull && PyErr_Occurred());
  }
  if (kind == 'p') {
    if (o == Py_None) {
      out = 0;
      return true;
    }
    if (THPVariable_Check(o)) {
      try {
        out = (word)THPVariable_Unpack(o).data_ptr();
        return true;
      } catch (const std::exception& e) {
        PyErr_SetString(PyExc_RuntimeError, e.what());
        return false;
      }
    }
  }
  // what stands for an integer (numpy's, a tensor of one), or a ctypes number
  PyObject* inner = kind == 'i' && PyIndex_Check(o) ? PyNumber_Index(o) : PyObject_GetAttrString(o, "value");
  if (inner && (PyLong_Check(inner) || (kind == 'p' && inner == Py_None))) {
    const bool done = as_word(inner, kind, out);
    Py_DECREF(inner);
    return done;
  }
  Py_XDECREF(inner);
  PyErr_Clear();
  PyErr_Format(PyExc_TypeError, "a kernel's entry point takes an integer%s here, not %s", kind == 'p' ? ", a tensor or None" : "",
               Py_TYPE(o)->tp_name);
  return false;
}

bool as_float(PyObject* o, double& out) {
  double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) {
    PyErr_Clear();
    PyObject* inner = PyObject_GetAttrString(o, "value");      // a ctypes number
    v = inner ? PyFloat_AsDouble(inner) : -1.0;
    Py_XDECREF(inner);
    if (PyErr_Occurred()) {
      PyErr_Clear();
      PyErr_Format(PyExc_TypeError, "a kernel's entry point takes a number here, not %s", Py_TYPE(o)->tp_name);
      return false;
    }
  }
  const float f = (float)v;
  word bits = 0;
  std::memcpy(&bits, &f, sizeof f);
  std::memcpy(&out, &bits, sizeof bits);
  return true;
}

PyObject* entry_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  Entry* e = reinterpret_cast<Entry*>(self);
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  if (n != e->count || (kwnames && PyTuple_GET_SIZE(kwnames))) {
    PyErr_Format(PyExc_TypeError, "this entry point takes %d arguments in order, not %zd", e->count, n);
    return nullptr;
  }
  word w[MAX_INTS] = {};
  double f[MAX_FLOATS] = {};
  int nw = 0, nf = 0;
  for (Py_ssize_t i = 0; i < n; ++i)
    if (!(e->kinds[i] == 'f' ? as_float(args[i], f[nf++]) : as_word(args[i], e->kinds[i], w[nw++]))) return nullptr;
  word r;
  Py_BEGIN_ALLOW_THREADS             // (a launch waits while the queue is full)
  r = e->function(w[0], w[1], w[2], w[3], w[4], w[5], f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[7], w[6], w[7], w[8], w[9], w[10],
                  w[11], w[12], w[13], w[14], w[15], w[16], w[17], w[18], w[19], w[20], w[21], w[22], w[23], w[24], w[25], w[26], w[27],
                  w[28], w[29], w[30], w[31], w[32], w[33], w[34], w[35], w[36], w[37], w[38], w[39]);
  Py_END_ALLOW_THREADS
  if (e->result == 'i') return PyLong_FromLong((int)r);
  if (e->result == 'l') return PyLong_FromLongLong((long long)r);
  Py_RETURN_NONE;
}

// Entry(address, kinds, result)
PyObject* entry_new(PyTypeObject* type, PyObject* args, PyObject*) {
  unsigned long long address;
  const char *kinds, *result;
  if (!PyArg_ParseTuple(args, "Kss", &address, &kinds, &result)) return nullptr;
  int ints = 0, floats = 0;
  for (const char* k = kinds; *k; ++k) ++(*k == 'f' ? floats : ints);
  if (ints > MAX_INTS || floats > MAX_FLOATS || !address) {
    PyErr_Format(PyExc_ValueError, "no call with %d integers and %d floats", ints, floats);
    return nullptr;
  }
  Entry* e = reinterpret_cast<Entry*>(type->tp_alloc(type, 0));
  if (!e) return nullptr;
  e->call = entry_call;
  e->function = (Function)address;
  e->result = result[0];
  e->count = ints + floats;
  std::memcpy(e->kinds, kinds, e->count);
  return reinterpret_cast<PyObject*>(e);
}

PyTypeObject entry_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyObject* refuse = nullptr;        // need()'s way out: says what is wrong with an operand, or accepts it

// need(t, name, dtype=None, ndim=None): a contiguous CUDA tensor of this type and number of dimensions.
PyObject* need(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n >= 1 && n <= 4 && THPVariable_Check(args[0])) {
    try {
      const at::Tensor& t = THPVariable_Unpack(args[0]);
      if (t.is_cuda() && t.layout() == at::kStrided && t.is_contiguous() &&
          (n < 3 || args[2] == Py_None || (THPDtype_Check(args[2]) && reinterpret_cast<THPDtype*>(args[2])->scalar_type == t.scalar_type())) &&
          (n < 4 || args[3] == Py_None || (PyLong_Check(args[3]) && PyLong_AsLong(args[3]) == t.dim())))
        Py_RETURN_NONE;
    } catch (const std::exception&) {
    }
  }
  PyErr_Clear();
  return PyObject_Vectorcall(refuse, args, n, nullptr);
}

// empty(like, shape, dtype=None): like.new_empty(shape, dtype=dtype).
PyObject* empty(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if ((n == 2 || n == 3) && THPVariable_Check(args[0]) && PyTuple_Check(args[1]) && PyTuple_GET_SIZE(args[1]) <= 6) {
    try {
      const at::Tensor& like = THPVariable_Unpack(args[0]);
      if (like.is_cuda() && !at::globalContext().deterministicAlgorithms() && (n == 2 || args[2] == Py_None || THPDtype_Check(args[2]))) {
        int64_t sizes[6];
        const Py_ssize_t dims = PyTuple_GET_SIZE(args[1]);
        bool plain = true;
        for (Py_ssize_t i = 0; i < dims && plain; ++i) {
          PyObject* o = PyTuple_GET_ITEM(args[1], i);
          plain = PyLong_Check(o);
          if (plain) sizes[i] = PyLong_AsLongLong(o);
        }
        if (plain && !PyErr_Occurred()) {
          const at::ScalarType type =
              n == 2 || args[2] == Py_None ? like.scalar_type() : reinterpret_cast<THPDtype*>(args[2])->scalar_type;
          return THPVariable_Wrap(at::Tensor(at::detail::empty_cuda(at::IntArrayRef(sizes, dims), type, like.device(), std::nullopt)));
        }
        PyErr_Clear();
      }
    } catch (const std::exception&) {
    }
  }
  // everything else, errors among it, the general way
  PyObject* made = PyObject_GetAttrString(args[0], "new_empty");
  if (!made) return nullptr;
  PyObject* kw = nullptr;
  PyObject* call[2] = {args[1], n > 2 ? args[2] : nullptr};
  if (n > 2 && args[2] != Py_None) kw = Py_BuildValue("(s)", "dtype");
  PyObject* out = PyObject_Vectorcall(made, call, 1, kw);
  Py_XDECREF(kw);
  Py_DECREF(made);
  return out;
}

// Whether an operation on these tensors would go straight to its CUDA kernel: plain tensors, nothing recorded, cast, mapped or traced.
bool plain(const at::Tensor& t) {
  static const c10::DispatchKeySet usual =
      c10::DispatchKeySet({c10::DispatchKey::CUDA, c10::DispatchKey::ADInplaceOrView, c10::DispatchKey::AutogradCUDA, c10::DispatchKey::AutocastCUDA});
  return t.is_cuda() && t.layout() == at::kStrided && !(t.key_set().raw_repr() & ~usual.raw_repr()) && !(t.requires_grad() && c10::GradMode::is_enabled()) &&
         !t._fw_grad(0).defined();           // (a dual number's tangent shows in neither: torch's one level of them)
}
bool plain_thread() {
  return !(c10::impl::tls_local_dispatch_key_set().included_.raw_repr() & ~c10::default_included_set.raw_repr()) && !at::autocast::is_autocast_enabled(at::kCUDA) &&
         !at::impl::torch_function_mode_enabled() && !at::hasCallbacks();      // (a profiler sees the operation at the dispatcher)
}

// product(x, w, low, high): x @ w.T by the library for contiguous bfloat16 matrices of low < rows < high on one device, as torch.mm(x, w.t()) calls
// it (the dispatcher and the Python bindings of a view and a product less: a product of 300 rows keeps the host busy for 9.7 us in place of 10.9).  None where it is
// not that plain a call, or fails: torch.mm does it then, or says why not.
PyObject* product(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n == 4 && THPVariable_CheckExact(args[0]) && THPVariable_CheckExact(args[1]) && PyLong_Check(args[2]) && PyLong_Check(args[3])) {
    const at::Tensor &x = THPVariable_Unpack(args[0]), &w = THPVariable_Unpack(args[1]);
    if (x.dim() == 2 && w.dim() == 2 && x.scalar_type() == at::kBFloat16 && w.scalar_type() == at::kBFloat16 && plain(x) && plain(w) &&
        x.device() == w.device() && x.is_contiguous() && w.is_contiguous() && !at::globalContext().deterministicAlgorithms() && plain_thread()) {
      const int64_t rows = x.size(0), k = x.size(1), width = w.size(0);
      if (rows > PyLong_AsLongLong(args[2]) && rows < PyLong_AsLongLong(args[3]) && w.size(1) == k && k > 0 && width > 0) {
        at::Tensor out;
        bool done = false;
        Py_BEGIN_ALLOW_THREADS
        try {
          const c10::cuda::CUDAGuard device(x.device());
          const at::AutoDispatchBelowADInplaceOrView below;
          out = at::cuda::mm(x, w.t());
          done = true;
        } catch (const std::exception&) {
        }
        Py_END_ALLOW_THREADS
        if (done) return THPVariable_Wrap(out);
      }
    }
  }
  PyErr_Clear();
  Py_RETURN_NONE;
}

// A sequence of integers; false with an exception set.
bool integers(PyObject* o, std::vector<long long>& out) {
  PyObject* fast = PySequence_Fast(o, "a sequence of integers is wanted here");
  if (!fast) return false;
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(fast);
  out.resize(n);
  for (Py_ssize_t i = 0; i < n; ++i) out[i] = PyLong_AsLongLong(PySequence_Fast_GET_ITEM(fast, i));
  Py_DECREF(fast);
  return !PyErr_Occurred();
}

// block_steps(kv lengths, new tokens, window): see latent_block_steps in ops.py.
PyObject* block_steps(PyObject*, PyObject* const* args, Py_ssize_t n) try {
  std::vector<long long> kv, q, steps;
  if (n != 3 || !integers(args[0], kv) || !integers(args[1], q)) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "block_steps(kv lengths, new tokens, window)");
    return nullptr;
  }
  const long long window = PyLong_AsLongLong(args[2]);
  if (PyErr_Occurred()) return nullptr;
  for (size_t i = 0; i < kv.size() && i < q.size(); ++i) {
    const long long past = kv[i] - q[i], base = window ? std::max(0ll, past - window + 1) : 0;
    for (long long first = 0; first < q[i]; first += 256) {
      const long long low = window ? std::max(0ll, past + first - window + 1) : 0;
      steps.push_back((past + std::min(first + 256, q[i]) - 1 - base) / 64 - (low - base) / 64 + 1);
    }
  }
  std::sort(steps.begin(), steps.end(), std::greater<long long>());
  PyObject* out = PyTuple_New((Py_ssize_t)steps.size());
  for (size_t i = 0; out && i < steps.size(); ++i) PyTuple_SET_ITEM(out, i, PyLong_FromLongLong(steps[i]));
  return out;
} catch (const std::exception& e) {
  PyErr_SetString(PyExc_RuntimeError, e.what());
  return nullptr;
}

// mixed_splits(steps, heads, SMs): see latent_mixed_splits in ops.py.  At most sixteen of the lengths are tried: 2 us with 16 heads, 21 with one (148 blocks).
PyObject* mixed_splits(PyObject*, PyObject* const* args, Py_ssize_t n) try {
  std::vector<long long> steps;
  if (n != 3 || !integers(args[0], steps)) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_TypeError, "mixed_splits(steps, heads, SMs)");
    return nullptr;
  }
  const long long heads = PyLong_AsLongLong(args[1]), sms = PyLong_AsLongLong(args[2]);
  if (PyErr_Occurred()) return nullptr;
  if (steps.empty() || heads < 1 || sms < 1 || *std::min_element(steps.begin(), steps.end()) < 1) return PyLong_FromLong(1);
  std::sort(steps.begin(), steps.end(), std::greater<long long>());
  std::vector<std::pair<long long, long long>> runs;         // (steps, blocks of all heads)
  for (long long s : steps) {
    if (runs.empty() || runs.back().first != s) runs.push_back({s, 0});
    runs.back().second += heads;
  }
  const size_t apart = (runs.size() + 15) / 16;
  long long best = 0, from = 0;
  std::vector<long long> jobs;
  for (size_t last = (runs.size() - 1) / apart * apart;; last -= apart) {      // blocks of runs[.. last] in two, the shortest such first
    // the jobs, the longest first, as many as the estimate looks at
    long long all = 0;
    for (size_t k = 0; k < runs.size(); ++k) all += (k <= last ? 2 : 1) * runs[k].second;
    jobs.clear();
    size_t a = 0, b = last + 1;
    while ((long long)jobs.size() < std::min(all, 2 * sms)) {
      const long long half = a <= last ? (runs[a].first + 1) / 2 + 9 : -1, whole = b < runs.size() ? runs[b].first + 3 : -1;
      const bool split = half >= whole;
      const long long many = split ? 2 * runs[a].second : runs[b].second;
      jobs.insert(jobs.end(), (size_t)std::min(many, 2 * sms - (long long)jobs.size()), split ? half : whole);
      ++(split ? a : b);
    }
    long long time = jobs[0];
    for (long long i = 0; i < std::min(sms, all - sms); ++i) time = std::max(time, jobs[sms - 1 - i] + jobs[sms + i] + 10);
    if (!from || time < best) {
      best = time;
      from = runs[last].first;
    }
    if (!last) break;
  }
  return PyLong_FromLongLong((double)best <= 0.93 * (double)(steps[0] + 3) ? 2 | from << 8 : 1);
} catch (const std::exception& e) {
  PyErr_SetString(PyExc_RuntimeError, e.what());
  return nullptr;
}

// stream(): the current CUDA stream's address.
PyObject* stream(PyObject*, PyObject*) {
  try {
    return PyLong_FromUnsignedLongLong((word)c10::cuda::getCurrentCUDAStream().stream());
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

PyObject* refuse_with(PyObject*, PyObject* function) {
  Py_INCREF(function);
  Py_XSETREF(refuse, function);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"need", (PyCFunction)(void (*)(void))need, METH_FASTCALL, nullptr},
    {"empty", (PyCFunction)(void (*)(void))empty, METH_FASTCALL, nullptr},
    {"product", (PyCFunction)(void (*)(void))product, METH_FASTCALL, nullptr},
    {"block_steps", (PyCFunction)(void (*)(void))block_steps, METH_FASTCALL, nullptr},
    {"mixed_splits", (PyCFunction)(void (*)(void))mixed_splits, METH_FASTCALL, nullptr},
    {"stream", stream, METH_NOARGS, nullptr},
    {"refuse_with", refuse_with, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "sb_host", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit_sb_host() {
  entry_type.tp_name = "sb_host.Entry";
  entry_type.tp_basicsize = sizeof(Entry);
  entry_type.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL;
  entry_type.tp_vectorcall_offset = offsetof(Entry, call);
  entry_type.tp_call = PyVectorcall_Call;
  entry_type.tp_new = entry_new;
  if (PyType_Ready(&entry_type) < 0) return nullptr;
  PyObject* m = PyModule_Create(&module);
  if (m && PyModule_AddObjectRef(m, "Entry", reinterpret_cast<PyObject*>(&entry_type)) < 0) Py_CLEAR(m);
  return m;
}
