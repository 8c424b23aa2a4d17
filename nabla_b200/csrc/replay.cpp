// Compiled calls without Python in between.
//
// A compiled function's second call is written down (`transforms/tape.py`): which exported launch functions it called, with
// which numbers, and which of their pointers lie in an argument, in a result or in scratch. `call` then does the whole of a later
// call here: it looks at the arguments (structure, shape, type, strides, device, alignment), allocates the results and one
// block of scratch from torch's allocator on the current stream, calls the same launch functions with the pointers of this
// call, and wraps the results. A function that replays a CUDA graph goes the same way around one launch each for the copies in and out.
// Anything that does not match what was written down returns NotImplemented, and the caller takes the general path.
//
// What bounded such calls was Python: 20 to 40 us per launch in wrappers and 1 to 5 us per argument and result (attention of one query
// over 4001 keys 53 us a call for 29 us of kernels, a layer norm with its gradient 102 for 81).
#include <Python.h>
#include <structmember.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstdlib>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#if !defined(__x86_64__) || !defined(__linux__)
#error "call_launcher relies on the System V calling convention of x86-64"
#endif

namespace {

constexpr int REG_INTS = 6, STACK_INTS = 56, FLOATS = 8;

// Integers and pointers go to six registers and then to the stack, eight bytes each, floating-point numbers to eight
// registers, each class in its own order: one call through this type serves every launch function with at most that many.
typedef int (*Launcher)(long, long, long, long, long, long, double, double, double, double, double, double, double, double,
#define L8 long, long, long, long, long, long, long, long
                        L8, L8, L8, L8, L8, L8, L8);
#undef L8
int call_launcher(void* fn, const long* i, const double* d) {
  const long* s = i + REG_INTS;
#define S8(k) s[k], s[k + 1], s[k + 2], s[k + 3], s[k + 4], s[k + 5], s[k + 6], s[k + 7]
  return reinterpret_cast<Launcher>(fn)(i[0], i[1], i[2], i[3], i[4], i[5], d[0], d[1], d[2], d[3], d[4], d[5], d[6], d[7], S8(0), S8(8),
                                        S8(16), S8(24), S8(32), S8(40), S8(48));
#undef S8
}

struct Ref {                                         // owned reference
  PyObject* p = nullptr;
  Ref() = default;
  explicit Ref(PyObject* o) : p(o) {}
  static Ref borrow(PyObject* o) { Py_XINCREF(o); return Ref(o); }
  Ref(Ref&& o) noexcept : p(o.p) { o.p = nullptr; }
  Ref& operator=(Ref&& o) noexcept { std::swap(p, o.p); return *this; }
  Ref(const Ref&) = delete;
  ~Ref() { Py_XDECREF(p); }
};

// Launches wait for the device when the stream's queue is full, and allocations may; other threads of Python run meanwhile (and so does
// a host function on the stream that needs Python), as they do while ctypes or torch calls a library.
struct WithoutGil {
  PyThreadState* state = PyEval_SaveThread();
  ~WithoutGil() { PyEval_RestoreThread(state); }
};

struct Tree {                                        // structure of an argument or of the result
  char kind = 'n';                                   // n None, x a leaf, l list, t tuple, d dict
  Ref keys;                                          // tuple
  std::vector<Tree> ch;
};

struct Leaf {
  Ref shape, dtype, device, batch_dims;
  at::ScalarType scalar;
  std::vector<int64_t> sizes, strides;
  unsigned align;                                    // address modulo 16; 16: any (arguments that are copied)
};
struct Pin {                                         // a tensor that the function captured, as it was
  Ref impl;
  void* ptr;
  std::vector<int64_t> sizes, strides;
};

enum ArgKind { INT = 0, FLOAT = 1, DOUBLE = 2, POINTER = 3, STREAM = 4, BLOB = 5 };
struct Patch { size_t at; int base; long offset; };
struct Arg {
  int kind;
  long value = 0;                                    // INT: the number; POINTER: the offset from its base
  double number = 0;
  int base = 0;
  std::string bytes;                                 // BLOB: a host array; the pointers in it are patched
  std::vector<Patch> patches;
};
struct Launch {
  void* fn;
  long rc;
  std::string name;
  std::vector<Arg> args;
};

struct Out {
  bool is_static = false;
  Ref value;                                         // static
  std::vector<int64_t> sizes, strides;
  at::TensorOptions options;
  std::vector<std::pair<Py_ssize_t, Ref>> slots;     // what a result's impl holds besides its buffer
};

struct Tape {
  std::vector<Tree> args;
  std::vector<Leaf> leaves;
  std::vector<std::pair<std::string, Ref>> env;      // (name, bytes or None)
  std::vector<Pin> pins;
  std::vector<at::Tensor> kept;                      // what the launches' fixed addresses lie in: alive as long as a call is at it
  int device = 0;
  bool deterministic = false;
  std::vector<Launch> launches;
  size_t scratch = 0;
  std::vector<Out> outs;
  Tree out_tree;
  // CUDA graph
  Ref replay;                                        // its replay method; null: none
  void* copy_batch = nullptr;
  std::vector<void*> in_ptrs, out_ptrs;
  std::vector<unsigned long long> in_bytes, out_bytes;
};

// classes and the offsets of their slots
PyTypeObject *g_tensor = nullptr, *g_impl = nullptr;
Py_ssize_t o_impl, o_buffers, o_shape, o_dtype, o_device, o_sharding, o_batch;

Py_ssize_t slot_offset(PyObject* type, const char* name) {
  Ref d(PyObject_GetAttrString(type, name));
  if (d.p == nullptr || !PyObject_TypeCheck(d.p, &PyMemberDescr_Type)) {
    if (!PyErr_Occurred()) PyErr_Format(PyExc_TypeError, "%s is not a slot", name);
    return -1;
  }
  return reinterpret_cast<PyMemberDescrObject*>(d.p)->d_member->offset;
}
inline PyObject* slot(PyObject* o, Py_ssize_t at) { return *reinterpret_cast<PyObject**>(reinterpret_cast<char*>(o) + at); }
inline void set_slot(PyObject* o, Py_ssize_t at, PyObject* v) {       // steals v; the slot is empty
  *reinterpret_cast<PyObject**>(reinterpret_cast<char*>(o) + at) = v;
}

struct Fail {};                                      // a Python error is set
PyObject* item(PyObject* seq, Py_ssize_t i) {
  PyObject* o = PyTuple_Check(seq) ? PyTuple_GetItem(seq, i) : PyList_GetItem(seq, i);
  if (o == nullptr) throw Fail();
  return o;
}
Py_ssize_t size(PyObject* seq) {
  const Py_ssize_t n = PyTuple_Check(seq) ? PyTuple_GET_SIZE(seq) : PyList_Check(seq) ? PyList_GET_SIZE(seq) : -1;
  if (n < 0) { PyErr_SetString(PyExc_TypeError, "a list or tuple"); throw Fail(); }
  return n;
}
long integer(PyObject* o) {
  const unsigned long long v = PyLong_AsUnsignedLongLongMask(o);
  if (PyErr_Occurred()) throw Fail();
  return static_cast<long>(v);
}
std::string text(PyObject* o) {
  char* p;
  Py_ssize_t n;
  if (PyBytes_AsStringAndSize(o, &p, &n) < 0) throw Fail();
  return std::string(p, static_cast<size_t>(n));
}
const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) { PyErr_SetString(PyExc_TypeError, "a torch tensor"); throw Fail(); }
  return THPVariable_Unpack(o);
}
Tree read_tree(PyObject* o) {                        // (kind, keys or None, children)
  Tree t;
  t.kind = text(item(o, 0)).at(0);
  t.keys = Ref::borrow(item(o, 1));
  PyObject* ch = item(o, 2);
  for (Py_ssize_t i = 0; i < size(ch); ++i) t.ch.push_back(read_tree(item(ch, i)));
  return t;
}

void release(PyObject* cap) { delete static_cast<Tape*>(PyCapsule_GetPointer(cap, "nb_tape")); }

// make(args, leaves, env, device, deterministic, launches, scratch, outs, out_tree, graph, captured impls, kept tensors): see transforms/tape.py
PyObject* make(PyObject*, PyObject* a) {
  auto t = std::make_unique<Tape>();
  try {
    PyObject* o = item(a, 0);
    for (Py_ssize_t i = 0; i < size(o); ++i) t->args.push_back(read_tree(item(o, i)));
    o = item(a, 1);
    for (Py_ssize_t i = 0; i < size(o); ++i) {       // (shape, dtype, batch dims, device, torch tensor)
      PyObject* l = item(o, i);
      Leaf f;
      f.shape = Ref::borrow(item(l, 0));
      f.dtype = Ref::borrow(item(l, 1));
      f.batch_dims = Ref::borrow(item(l, 2));
      f.device = Ref::borrow(item(l, 3));
      const at::Tensor& x = tensor(item(l, 4));
      f.scalar = x.scalar_type();
      f.sizes = x.sizes().vec();
      f.strides = x.strides().vec();
      f.align = static_cast<unsigned>(reinterpret_cast<uintptr_t>(x.data_ptr()) & 15);
      t->leaves.push_back(std::move(f));
    }
    o = item(a, 2);
    for (Py_ssize_t i = 0; i < size(o); ++i) t->env.emplace_back(text(item(item(o, i), 0)), Ref::borrow(item(item(o, i), 1)));
    t->device = static_cast<int>(integer(item(a, 3)));
    t->deterministic = PyObject_IsTrue(item(a, 4)) == 1;
    o = item(a, 5);
    for (Py_ssize_t i = 0; i < size(o); ++i) {       // (address, expected code, name, [(kind, ...)])
      PyObject* l = item(o, i);
      Launch r;
      r.fn = reinterpret_cast<void*>(integer(item(l, 0)));
      r.rc = integer(item(l, 1));
      r.name = text(item(l, 2));
      PyObject* as = item(l, 3);
      int ints = 0, floats = 0;
      for (Py_ssize_t j = 0; j < size(as); ++j) {
        PyObject* e = item(as, j);
        Arg g;
        g.kind = static_cast<int>(integer(item(e, 0)));
        if (g.kind == FLOAT || g.kind == DOUBLE) {
          const double v = PyFloat_AsDouble(item(e, 1));
          if (PyErr_Occurred()) throw Fail();
          if (g.kind == FLOAT) {                     // a float is the low half of its register
            const float f = static_cast<float>(v);
            std::memcpy(&g.number, &f, sizeof(f));
          } else {
            g.number = v;
          }
          ++floats;
        } else {
          ++ints;
          if (g.kind == INT) {
            g.value = integer(item(e, 1));
          } else if (g.kind == POINTER) {
            g.base = static_cast<int>(integer(item(e, 1)));
            g.value = integer(item(e, 2));
          } else if (g.kind == BLOB) {
            g.bytes = text(item(e, 1));
            PyObject* ps = item(e, 2);
            for (Py_ssize_t k = 0; k < size(ps); ++k) {
              PyObject* p = item(ps, k);
              g.patches.push_back({static_cast<size_t>(integer(item(p, 0))), static_cast<int>(integer(item(p, 1))), integer(item(p, 2))});
            }
          }
        }
        r.args.push_back(std::move(g));
      }
      if (ints > REG_INTS + STACK_INTS || floats > FLOATS) { PyErr_SetString(PyExc_ValueError, "too many arguments"); throw Fail(); }
      t->launches.push_back(std::move(r));
    }
    t->scratch = static_cast<size_t>(integer(item(a, 6)));
    o = item(a, 7);
    for (Py_ssize_t i = 0; i < size(o); ++i) {       // (value,) or (torch tensor, example impl)
      PyObject* l = item(o, i);
      Out r;
      if (size(l) == 1) {
        r.is_static = true;
        r.value = Ref::borrow(item(l, 0));
      } else {
        const at::Tensor& x = tensor(item(l, 0));
        r.sizes = x.sizes().vec();
        r.strides = x.strides().vec();
        r.options = x.options();
        PyObject* like = item(l, 1);
        Ref names(PyObject_GetAttrString(reinterpret_cast<PyObject*>(g_impl), "__slots__"));
        if (names.p == nullptr) throw Fail();
        for (Py_ssize_t k = 0; k < size(names.p); ++k) {
          const char* name = PyUnicode_AsUTF8(item(names.p, k));
          if (name == nullptr) throw Fail();
          if (std::strcmp(name, "_buffers") == 0 || std::strcmp(name, "__weakref__") == 0) continue;
          const Py_ssize_t at = slot_offset(reinterpret_cast<PyObject*>(g_impl), name);
          if (at < 0) throw Fail();
          if (slot(like, at) != nullptr) r.slots.emplace_back(at, Ref::borrow(slot(like, at)));
        }
      }
      t->outs.push_back(std::move(r));
    }
    t->out_tree = read_tree(item(a, 8));
    o = item(a, 9);
    if (o != Py_None) {                              // (replay, copy_batch address, [(ptr, bytes)] in, [(ptr, bytes)] out)
      t->replay = Ref::borrow(item(o, 0));
      t->copy_batch = reinterpret_cast<void*>(integer(item(o, 1)));
      for (int k = 0; k < 2; ++k) {
        PyObject* l = item(o, 2 + k);
        for (Py_ssize_t i = 0; i < size(l); ++i) {
          (k ? t->out_ptrs : t->in_ptrs).push_back(reinterpret_cast<void*>(integer(item(item(l, i), 0))));
          (k ? t->out_bytes : t->in_bytes).push_back(static_cast<unsigned long long>(integer(item(item(l, i), 1))));
        }
      }
    }
    for (Leaf& f : t->leaves)
      if (o != Py_None) f.align = 16;
    o = item(a, 10);
    for (Py_ssize_t i = 0; i < size(o); ++i) {
      Pin p;
      p.impl = Ref::borrow(item(o, i));
      const at::Tensor& x = tensor(item(slot(p.impl.p, o_buffers), 0));
      p.ptr = x.data_ptr();
      p.sizes = x.sizes().vec();
      p.strides = x.strides().vec();
      t->pins.push_back(std::move(p));
    }
    o = item(a, 11);
    for (Py_ssize_t i = 0; i < size(o); ++i) t->kept.push_back(tensor(item(o, i)));
  } catch (const Fail&) {
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
  PyObject* cap = PyCapsule_New(t.get(), "nb_tape", release);
  if (cap != nullptr) t.release();
  return cap;
}

// The leaves of `o` in the order of `t`; false for another structure.
bool gather(const Tree& t, PyObject* o, std::vector<PyObject*>& out) {
  switch (t.kind) {
    case 'x':
      out.push_back(o);
      return true;
    case 'n':
      return o == Py_None;
    case 'd': {
      if (!PyDict_CheckExact(o) || PyDict_GET_SIZE(o) != static_cast<Py_ssize_t>(t.ch.size())) return false;
      for (size_t i = 0; i < t.ch.size(); ++i) {
        PyObject* v = PyDict_GetItemWithError(o, PyTuple_GET_ITEM(t.keys.p, i));
        if (v == nullptr) { PyErr_Clear(); return false; }
        if (!gather(t.ch[i], v, out)) return false;
      }
      return true;
    }
    default: {
      const bool list = t.kind == 'l';
      if (list ? !PyList_CheckExact(o) : !PyTuple_CheckExact(o)) return false;
      if ((list ? PyList_GET_SIZE(o) : PyTuple_GET_SIZE(o)) != static_cast<Py_ssize_t>(t.ch.size())) return false;
      for (size_t i = 0; i < t.ch.size(); ++i)
        if (!gather(t.ch[i], list ? PyList_GET_ITEM(o, i) : PyTuple_GET_ITEM(o, i), out)) return false;
      return true;
    }
  }
}

// The torch tensor of an argument that is what was written down, else null.
const at::Tensor* buffer(const Leaf& f, PyObject* o, int device) {
  if (Py_TYPE(o) != g_tensor) return nullptr;
  PyObject* im = slot(o, o_impl);
  if (im == nullptr || Py_TYPE(im) != g_impl || slot(im, o_sharding) != Py_None || slot(im, o_dtype) != f.dtype.p) return nullptr;
  PyObject *bufs = slot(im, o_buffers), *shape = slot(im, o_shape), *dev = slot(im, o_device), *bd = slot(im, o_batch);
  if (bufs == nullptr || !PyList_CheckExact(bufs) || PyList_GET_SIZE(bufs) != 1 || shape == nullptr || dev == nullptr || bd == nullptr) return nullptr;
  if ((shape != f.shape.p && PyObject_RichCompareBool(shape, f.shape.p, Py_EQ) != 1) ||
      (dev != f.device.p && PyObject_RichCompareBool(dev, f.device.p, Py_EQ) != 1) ||
      (bd != f.batch_dims.p && PyObject_RichCompareBool(bd, f.batch_dims.p, Py_EQ) != 1)) {
    PyErr_Clear();
    return nullptr;
  }
  PyObject* b = PyList_GET_ITEM(bufs, 0);
  if (reinterpret_cast<PyObject*>(Py_TYPE(b)) != THPVariableClass) return nullptr;
  const at::Tensor& x = THPVariable_Unpack(b);
  if (x.layout() != at::kStrided || x.scalar_type() != f.scalar || !x.is_cuda() || x.get_device() != device || x.sizes() != at::IntArrayRef(f.sizes) ||
      x.strides() != at::IntArrayRef(f.strides) || x.is_conj() || x.is_neg() ||
      (f.align < 16 && (reinterpret_cast<uintptr_t>(x.data_ptr()) & 15) != f.align))
    return nullptr;
  return &x;
}

PyObject* build(const Tree& t, std::vector<Ref>& leaves, size_t& at) {
  switch (t.kind) {
    case 'n':
      Py_RETURN_NONE;
    case 'x': {
      PyObject* o = leaves[at].p;
      leaves[at++].p = nullptr;
      return o;
    }
    case 'd': {
      Ref d(PyDict_New());
      if (d.p == nullptr) return nullptr;
      for (size_t i = 0; i < t.ch.size(); ++i) {
        Ref v(build(t.ch[i], leaves, at));
        if (v.p == nullptr || PyDict_SetItem(d.p, PyTuple_GET_ITEM(t.keys.p, i), v.p) < 0) return nullptr;
      }
      return std::exchange(d.p, nullptr);
    }
    default: {
      const Py_ssize_t n = static_cast<Py_ssize_t>(t.ch.size());
      Ref s(t.kind == 'l' ? PyList_New(n) : PyTuple_New(n));
      if (s.p == nullptr) return nullptr;
      for (Py_ssize_t i = 0; i < n; ++i) {
        PyObject* v = build(t.ch[i], leaves, at);
        if (v == nullptr) return nullptr;
        if (t.kind == 'l') PyList_SET_ITEM(s.p, i, v); else PyTuple_SET_ITEM(s.p, i, v);
      }
      return std::exchange(s.p, nullptr);
    }
  }
}

// The launches in their order. Returns the first that failed (`code`: with what), else null.
const Launch* run_launches(const Tape& t, const std::vector<char*>& bases, cudaStream_t stream, int& code) {
  long ints[REG_INTS + STACK_INTS];
  double floats[FLOATS];
  std::vector<std::string> blobs;
  for (const Launch& l : t.launches) {
    std::memset(ints, 0, sizeof(ints));
    std::memset(floats, 0, sizeof(floats));
    blobs.clear();
    blobs.reserve(l.args.size());
    int ni = 0, nf = 0;
    for (const Arg& g : l.args) {
      switch (g.kind) {
        case FLOAT:
        case DOUBLE:
          floats[nf++] = g.number;
          break;
        case INT:
          ints[ni++] = g.value;
          break;
        case POINTER:
          ints[ni++] = reinterpret_cast<long>(bases[static_cast<size_t>(g.base)] + g.value);
          break;
        case STREAM:
          ints[ni++] = reinterpret_cast<long>(stream);
          break;
        default: {
          blobs.push_back(g.bytes);
          char* b = blobs.back().data();
          for (const Patch& p : g.patches) {
            const long v = reinterpret_cast<long>(bases[static_cast<size_t>(p.base)] + p.offset);
            std::memcpy(b + p.at, &v, sizeof(v));
          }
          ints[ni++] = reinterpret_cast<long>(b);
        }
      }
    }
    code = call_launcher(l.fn, ints, floats);
    if (code != l.rc) return &l;
  }
  return nullptr;
}

// One launch that copies for a graph; a negative code when it failed.
int run_copies(void* copy_batch, void* const* dst, void* const* src, const unsigned long long* bytes, size_t n, cudaStream_t stream) {
  long ints[REG_INTS + STACK_INTS] = {reinterpret_cast<long>(dst), reinterpret_cast<long>(src), reinterpret_cast<long>(bytes), static_cast<long>(n),
                                      reinterpret_cast<long>(stream)};
  double floats[FLOATS] = {};
  return call_launcher(copy_batch, ints, floats);
}

// call(tape, args, deterministic) -> result, or NotImplemented when the call is not the one that was written down
PyObject* call(PyObject*, PyObject* const* argv, Py_ssize_t argc) {
  HANDLE_TH_ERRORS
  if (argc != 3 || !PyTuple_CheckExact(argv[1])) { PyErr_SetString(PyExc_TypeError, "call(tape, args, deterministic)"); return nullptr; }
  Tape* t = static_cast<Tape*>(PyCapsule_GetPointer(argv[0], "nb_tape"));
  if (t == nullptr) return nullptr;
  if (PyTuple_GET_SIZE(argv[1]) != static_cast<Py_ssize_t>(t->args.size()) || (argv[2] == Py_True) != t->deterministic) Py_RETURN_NOTIMPLEMENTED;
  std::vector<PyObject*> leaves;
  leaves.reserve(t->leaves.size());
  for (size_t i = 0; i < t->args.size(); ++i)
    if (!gather(t->args[i], PyTuple_GET_ITEM(argv[1], i), leaves)) Py_RETURN_NOTIMPLEMENTED;
  if (leaves.size() != t->leaves.size()) Py_RETURN_NOTIMPLEMENTED;
  if (c10::cuda::current_device() != t->device) Py_RETURN_NOTIMPLEMENTED;
  for (const auto& e : t->env) {
    const char* v = std::getenv(e.first.c_str());
    if (v == nullptr ? e.second.p != Py_None : (e.second.p == Py_None || std::strcmp(v, PyBytes_AS_STRING(e.second.p)) != 0)) Py_RETURN_NOTIMPLEMENTED;
  }
  std::vector<at::Tensor> held;                      // stay alive whatever else runs while this waits
  held.reserve(leaves.size() + t->pins.size());
  for (const Pin& p : t->pins) {
    PyObject* b = slot(p.impl.p, o_buffers);
    if (b == nullptr || !PyList_CheckExact(b) || PyList_GET_SIZE(b) != 1 || !THPVariable_Check(PyList_GET_ITEM(b, 0))) Py_RETURN_NOTIMPLEMENTED;
    const at::Tensor& x = THPVariable_Unpack(PyList_GET_ITEM(b, 0));
    if (x.data_ptr() != p.ptr || x.sizes() != at::IntArrayRef(p.sizes) || x.strides() != at::IntArrayRef(p.strides)) Py_RETURN_NOTIMPLEMENTED;
    held.push_back(x);
  }
  std::vector<char*> bases(leaves.size() + t->outs.size() + 1, nullptr);
  for (size_t i = 0; i < leaves.size(); ++i) {
    const at::Tensor* x = buffer(t->leaves[i], leaves[i], t->device);
    if (x == nullptr) Py_RETURN_NOTIMPLEMENTED;
    held.push_back(*x);
    bases[i] = static_cast<char*>(x->data_ptr());
  }
  cudaStream_t stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(t->device)).stream();
  int code = 0;
  if (t->replay.p != nullptr) {
    const size_t n = leaves.size();
    std::vector<void*> src(n, nullptr);
    std::vector<unsigned long long> bytes(n, 0);
    bool any = false;
    for (size_t i = 0; i < n; ++i)
      if (bases[i] != t->in_ptrs[i]) {
        src[i] = bases[i];
        bytes[i] = t->in_bytes[i];
        any = any || bytes[i] > 0;
      }
    if (any) {
      WithoutGil free;
      code = run_copies(t->copy_batch, t->in_ptrs.data(), src.data(), bytes.data(), n, stream);
    }
    if (code < 0) return PyErr_Format(PyExc_RuntimeError, "copy_batch failed with code %d", code);
    Ref r(PyObject_CallNoArgs(t->replay.p));
    if (r.p == nullptr) return nullptr;
  }
  std::vector<at::Tensor> results;
  results.reserve(t->outs.size());
  at::Tensor scratch;
  const Launch* failed = nullptr;
  {
    WithoutGil free;
    at::AutoDispatchBelowAutograd guard;
    for (size_t i = 0; i < t->outs.size(); ++i) {
      const Out& o = t->outs[i];
      if (o.is_static) { results.emplace_back(); continue; }
      results.push_back(at::empty_strided(o.sizes, o.strides, o.options));
      bases[leaves.size() + i] = static_cast<char*>(results.back().data_ptr());
    }
    if (t->scratch) {
      scratch = at::empty({static_cast<int64_t>(t->scratch)}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, t->device));
      bases.back() = static_cast<char*>(scratch.data_ptr());
    }
    if (t->replay.p != nullptr && !t->out_ptrs.empty()) {
      std::vector<void*> dst;
      for (size_t i = 0; i < t->outs.size(); ++i)
        if (!t->outs[i].is_static) dst.push_back(bases[leaves.size() + i]);
      code = run_copies(t->copy_batch, dst.data(), t->out_ptrs.data(), t->out_bytes.data(), dst.size(), stream);
    }
    if (code >= 0) failed = run_launches(*t, bases, stream, code);
  }
  if (failed == nullptr && code < 0) return PyErr_Format(PyExc_RuntimeError, "copy_batch failed with code %d", code);
  if (failed != nullptr) {
    PyErr_Format(PyExc_RuntimeError, "%s failed with code %d", failed->name.c_str(), code);
    return nullptr;
  }
  std::vector<Ref> wrapped;
  wrapped.reserve(t->outs.size());
  for (size_t i = 0; i < t->outs.size(); ++i) {
    const Out& o = t->outs[i];
    if (o.is_static) { wrapped.push_back(Ref::borrow(o.value.p)); continue; }
    Ref im(g_impl->tp_alloc(g_impl, 0)), x(g_tensor->tp_alloc(g_tensor, 0)), l(PyList_New(1));
    if (im.p == nullptr || x.p == nullptr || l.p == nullptr) return nullptr;
    PyObject* v = THPVariable_Wrap(std::move(results[i]));
    if (v == nullptr) return nullptr;
    PyList_SET_ITEM(l.p, 0, v);
    for (const auto& s : o.slots) {
      Py_INCREF(s.second.p);
      set_slot(im.p, s.first, s.second.p);
    }
    set_slot(im.p, o_buffers, std::exchange(l.p, nullptr));
    set_slot(x.p, o_impl, std::exchange(im.p, nullptr));
    wrapped.push_back(std::move(x));
  }
  size_t at = 0;
  return build(t->out_tree, wrapped, at);
  END_HANDLE_TH_ERRORS
}

// classes(Tensor, TensorImpl)
PyObject* classes(PyObject*, PyObject* a) {
  PyObject *x, *im;
  if (!PyArg_ParseTuple(a, "O!O!", &PyType_Type, &x, &PyType_Type, &im)) return nullptr;
  if ((o_impl = slot_offset(x, "_impl")) < 0 || (o_buffers = slot_offset(im, "_buffers")) < 0 || (o_shape = slot_offset(im, "_shape")) < 0 ||
      (o_dtype = slot_offset(im, "_dtype")) < 0 || (o_device = slot_offset(im, "_device")) < 0 ||
      (o_sharding = slot_offset(im, "sharding")) < 0 || (o_batch = slot_offset(im, "batch_dims")) < 0)
    return nullptr;
  Py_INCREF(x);
  Py_INCREF(im);
  g_tensor = reinterpret_cast<PyTypeObject*>(x);
  g_impl = reinterpret_cast<PyTypeObject*>(im);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {{"make", make, METH_O, nullptr},
                         {"call", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(call)), METH_FASTCALL, nullptr},
                         {"classes", classes, METH_VARARGS, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "libnb_replay", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

#define NB_TEXT_(x) #x
#define NB_TEXT(x) NB_TEXT_(x)
PyMODINIT_FUNC PyInit_libnb_replay() {
  PyObject* m = PyModule_Create(&module);
  if (m != nullptr && PyModule_AddStringConstant(m, "built_for", NB_TEXT(NB_BUILT_FOR)) < 0) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
