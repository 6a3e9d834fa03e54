// CPython extension under the host layer: the objects every operator touches (device buffers, the
// fields of a tensor) and the calls into liblitenn_b200.so.
//
// A training step of a small network is some sixty operator calls whose kernels take two to four
// microseconds each, so the time between two launches is the host's.  Written in Python with ctypes
// a launch cost seven to nine microseconds: an object per buffer, four nested calls per pointer, the
// conversion of ten arguments.  Here a pointer argument is the tensor itself, resolved in C.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>
#include <stdint.h>
#include <string.h>
#include <vector>

namespace {

typedef int (*AllocFn)(int, uint64_t, uint64_t*);
typedef int (*FreeFn)(int, uint64_t, uint64_t);
AllocFn g_alloc = nullptr;
FreeFn g_free = nullptr;
PyObject* g_error = nullptr;          // error(status, function name): raises
PyObject *s_ensure, *s_inited, *s_initialize_buffer, *s_size, *s_index, *s_get_buffers, *s_before_write;
long g_buffers = 0, g_tensors = 0;
long long g_seq_id = 0;

// ---- device buffers --------------------------------------------------------------------------
// Memory of `size` bytes on one device, taken from the library's pool on first use.  `init` is
// nullptr, a callable init(buffer), or (with init_arg) an initializer whose
// initialize_buffer(buffer, init_arg) fills it.
struct Buffer {
  PyObject_HEAD
  PyObject *device, *init, *init_arg;
  uint64_t ptr;
  unsigned long long size;
  int index;
  char must_init;                     // the initializer may not be skipped by a kernel that overwrites
  long shares;                        // gradients that use this buffer besides its first holder
};

int raise_status(int rc, const char* name) {
  if (g_error) {
    PyObject* r = PyObject_CallFunction(g_error, "is", rc, name);
    Py_XDECREF(r);
  }
  if (!PyErr_Occurred()) PyErr_Format(PyExc_RuntimeError, "%s failed with status %d", name, rc);
  return -1;
}

int buffer_setup(Buffer* b, PyObject* device, unsigned long long size, PyObject* init, PyObject* init_arg, int must_init) {
  PyObject* idx = PyObject_GetAttr(device, s_index);
  if (!idx) return -1;
  b->index = (int)PyLong_AsLong(idx);
  Py_DECREF(idx);
  if (PyErr_Occurred()) return -1;
  Py_INCREF(device);
  Py_XSETREF(b->device, device);
  if (init == Py_None) init = nullptr;
  Py_XINCREF(init);
  Py_XSETREF(b->init, init);
  Py_XINCREF(init_arg);
  Py_XSETREF(b->init_arg, init_arg);
  b->size = size;
  b->must_init = (char)must_init;
  return 0;
}

// The memory's address (0 and an exception on failure); overwrite: the caller's kernel writes all of it.
uint64_t buffer_address(Buffer* b, bool overwrite) {
  if (b->ptr) return b->ptr;
  PyObject* inited = PyObject_GetAttr(b->device, s_inited);
  if (!inited) return 0;
  const int ready = PyObject_IsTrue(inited);
  Py_DECREF(inited);
  if (!ready || !g_alloc) {
    PyObject* r = PyObject_CallMethodNoArgs(b->device, s_ensure);
    if (!r) return 0;
    Py_DECREF(r);
  }
  if (!g_alloc) { PyErr_SetString(PyExc_RuntimeError, "the device library is not loaded"); return 0; }
  uint64_t p = 0;
  const int rc = g_alloc(b->index, b->size, &p);
  if (rc != 0) { raise_status(rc, "lnn_alloc"); return 0; }
  b->ptr = p;
  if (b->init && (!overwrite || b->must_init)) {
    PyObject* r = b->init_arg ? PyObject_CallMethodObjArgs(b->init, s_initialize_buffer, (PyObject*)b, b->init_arg, nullptr)
                              : PyObject_CallOneArg(b->init, (PyObject*)b);
    if (!r) return 0;
    Py_DECREF(r);
  }
  return b->ptr;
}

void buffer_release(Buffer* b) {
  if (b->ptr && g_free) g_free(b->index, b->ptr, b->size);
  b->ptr = 0;
}

PyObject* buffer_new(PyTypeObject* type, PyObject*, PyObject*) {
  Buffer* b = (Buffer*)type->tp_alloc(type, 0);
  if (b) ++g_buffers;
  return (PyObject*)b;
}
int buffer_init(PyObject* self, PyObject* args, PyObject* kw) {
  static const char* names[] = {"device", "size", "init_func", "must_init", nullptr};
  PyObject *device, *init = Py_None;
  long long size;
  int must_init = 1;
  if (!PyArg_ParseTupleAndKeywords(args, kw, "OL|Op", (char**)names, &device, &size, &init, &must_init)) return -1;
  if (size <= 0) { PyErr_Format(PyExc_ValueError, "Create DeviceBuffer with %lld size.", size); return -1; }
  return buffer_setup((Buffer*)self, device, (unsigned long long)size, init, nullptr, must_init);
}
int buffer_traverse(PyObject* self, visitproc visit, void* arg) {
  Buffer* b = (Buffer*)self;
  Py_VISIT(Py_TYPE(self));
  Py_VISIT(b->device); Py_VISIT(b->init); Py_VISIT(b->init_arg);
  return 0;
}
int buffer_clear(PyObject* self) {
  Buffer* b = (Buffer*)self;
  Py_CLEAR(b->init); Py_CLEAR(b->init_arg);
  return 0;
}
void buffer_dealloc(PyObject* self) {
  Buffer* b = (Buffer*)self;
  PyTypeObject* type = Py_TYPE(self);
  PyObject_GC_UnTrack(self);
  buffer_release(b);
  --g_buffers;
  Py_CLEAR(b->device); Py_CLEAR(b->init); Py_CLEAR(b->init_arg);
  type->tp_free(self);
  Py_DECREF(type);
}
PyObject* buffer_ptr(PyObject* self, PyObject*) {
  const uint64_t p = buffer_address((Buffer*)self, false);
  return p ? PyLong_FromUnsignedLongLong(p) : nullptr;
}
PyObject* buffer_ptr_to_overwrite(PyObject* self, PyObject*) {
  const uint64_t p = buffer_address((Buffer*)self, true);
  return p ? PyLong_FromUnsignedLongLong(p) : nullptr;
}
PyObject* buffer_free(PyObject* self, PyObject*) { buffer_release((Buffer*)self); Py_RETURN_NONE; }
PyObject* buffer_has_mem(PyObject* self, PyObject*) { return PyBool_FromLong(((Buffer*)self)->ptr != 0); }
PyObject* buffer_get_ptr(PyObject* self, void*) {
  const uint64_t p = ((Buffer*)self)->ptr;
  if (!p) Py_RETURN_NONE;
  return PyLong_FromUnsignedLongLong(p);
}
PyMethodDef buffer_methods[] = {
    {"ptr", buffer_ptr, METH_NOARGS, "Address of the memory, allocated and initialised on first use."},
    {"ptr_to_overwrite", buffer_ptr_to_overwrite, METH_NOARGS,
     "The same for a kernel that writes every element: an initializer without effects of its own is skipped."},
    {"free", buffer_free, METH_NOARGS, "Return the memory to the pool."},
    {"has_mem", buffer_has_mem, METH_NOARGS, "Whether memory has been allocated."},
    {nullptr, nullptr, 0, nullptr}};
PyMemberDef buffer_members[] = {
    {"device", T_OBJECT, offsetof(Buffer, device), READONLY, nullptr},
    {"size", T_ULONGLONG, offsetof(Buffer, size), READONLY, nullptr},
    {"shares", T_LONG, offsetof(Buffer, shares), 0, nullptr},
    {nullptr, 0, 0, 0, nullptr}};
PyGetSetDef buffer_getset[] = {{"_ptr", buffer_get_ptr, nullptr, nullptr, nullptr}, {nullptr, nullptr, nullptr, nullptr, nullptr}};
PyType_Slot buffer_slots[] = {{Py_tp_new, (void*)buffer_new}, {Py_tp_init, (void*)buffer_init},
                              {Py_tp_dealloc, (void*)buffer_dealloc}, {Py_tp_traverse, (void*)buffer_traverse},
                              {Py_tp_clear, (void*)buffer_clear}, {Py_tp_methods, buffer_methods},
                              {Py_tp_members, buffer_members}, {Py_tp_getset, buffer_getset}, {0, nullptr}};
PyType_Spec buffer_spec = {"litenn_b200._native.BufferBase", sizeof(Buffer), 0,
                           Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE | Py_TPFLAGS_HAVE_GC, buffer_slots};
PyTypeObject* BufferType = nullptr;

// ---- tensors ---------------------------------------------------------------------------------
struct Tensor {
  PyObject_HEAD
  PyObject *shape, *seq_id, *grad_t, *gradfns, *op_name, *op, *parent_module_w, *pending, *chain, *deps, *buffers, *t;
  char freezed, trainable, shared;
};

PyObject* tensor_new(PyTypeObject* type, PyObject*, PyObject*) {
  Tensor* t = (Tensor*)type->tp_alloc(type, 0);
  if (t) ++g_tensors;
  return (PyObject*)t;
}
int tensor_traverse(PyObject* self, visitproc visit, void* arg) {
  Tensor* t = (Tensor*)self;
  Py_VISIT(Py_TYPE(self));
  Py_VISIT(t->shape); Py_VISIT(t->grad_t); Py_VISIT(t->gradfns); Py_VISIT(t->op_name); Py_VISIT(t->op);
  Py_VISIT(t->parent_module_w); Py_VISIT(t->pending); Py_VISIT(t->chain); Py_VISIT(t->deps); Py_VISIT(t->buffers); Py_VISIT(t->t);
  return 0;
}
int tensor_clear(PyObject* self) {
  Tensor* t = (Tensor*)self;
  Py_CLEAR(t->grad_t); Py_CLEAR(t->gradfns); Py_CLEAR(t->op); Py_CLEAR(t->parent_module_w); Py_CLEAR(t->pending);
  Py_CLEAR(t->chain); Py_CLEAR(t->deps); Py_CLEAR(t->t);
  return 0;
}
void tensor_dealloc(PyObject* self) {
  Tensor* t = (Tensor*)self;
  PyTypeObject* type = Py_TYPE(self);
  PyObject_GC_UnTrack(self);
  if (t->shared && t->buffers && PyList_Check(t->buffers))
    for (Py_ssize_t i = 0; i < PyList_GET_SIZE(t->buffers); ++i) --((Buffer*)PyList_GET_ITEM(t->buffers, i))->shares;
  tensor_clear(self);
  Py_CLEAR(t->shape); Py_CLEAR(t->seq_id); Py_CLEAR(t->op_name); Py_CLEAR(t->buffers);
  if (--g_tensors == 0) g_seq_id = 0;
  type->tp_free(self);
  Py_DECREF(type);
}
PyTypeObject* TensorType = nullptr;

// The tensor that owns the buffers of a (reference to a reference to a ...) tensor.
inline Tensor* top_of(PyObject* o) {
  Tensor* t = (Tensor*)o;
  while (t->t && t->t != Py_None) t = (Tensor*)t->t;
  return t;
}

// Buffer number i of a tensor, borrowed.  A tensor whose work has been put off launches it first.
Buffer* tensor_buffer(PyObject* o, Py_ssize_t i) {
  Tensor* t = top_of(o);
  PyObject* list = t->buffers;
  PyObject* got = nullptr;
  if (t->pending && t->pending != Py_None) {
    got = PyObject_CallMethodNoArgs((PyObject*)t, s_get_buffers);
    if (!got) return nullptr;
    list = got;
  }
  Buffer* b = nullptr;
  if (!list || !PyList_Check(list) || i < 0 || i >= PyList_GET_SIZE(list))
    PyErr_SetString(PyExc_IndexError, "tensor has no buffer for this device");
  else
    b = (Buffer*)PyList_GET_ITEM(list, i);        // the tensor keeps the list's buffers alive
  Py_XDECREF(got);
  return b;
}

PyObject* tensor_ptr(PyObject* self, PyObject* arg) {
  const long i = PyLong_AsLong(arg);
  if (i == -1 && PyErr_Occurred()) return nullptr;
  Buffer* b = tensor_buffer(self, i);
  if (!b) return nullptr;
  const uint64_t p = buffer_address(b, false);
  return p ? PyLong_FromUnsignedLongLong(p) : nullptr;
}
PyObject* tensor_top(PyObject* self, PyObject*) {
  PyObject* t = (PyObject*)top_of(self);
  Py_INCREF(t);
  return t;
}
// Nothing has touched the memory of this tensor on any device yet.
PyObject* tensor_untouched(PyObject* self, PyObject*) {
  Tensor* t = top_of(self);
  if (!t->buffers || !PyList_Check(t->buffers)) Py_RETURN_FALSE;
  for (Py_ssize_t i = 0; i < PyList_GET_SIZE(t->buffers); ++i)
    if (((Buffer*)PyList_GET_ITEM(t->buffers, i))->ptr) Py_RETURN_FALSE;
  Py_RETURN_TRUE;
}
PyMethodDef tensor_methods[] = {
    {"_ptr", tensor_ptr, METH_O, "Device pointer of this tensor's buffer on current device number device_id."},
    {"_get_top_reference_source", tensor_top, METH_NOARGS, "The tensor that owns the buffers."},
    {"_untouched", tensor_untouched, METH_NOARGS, "Whether no memory has been allocated yet."},
    {nullptr, nullptr, 0, nullptr}};
PyMemberDef tensor_members[] = {
    {"shape", T_OBJECT, offsetof(Tensor, shape), 0, nullptr},
    {"_seq_id", T_OBJECT, offsetof(Tensor, seq_id), 0, nullptr},
    {"_grad_t", T_OBJECT, offsetof(Tensor, grad_t), 0, nullptr},
    {"_gradfns", T_OBJECT, offsetof(Tensor, gradfns), 0, nullptr},
    {"_op_name", T_OBJECT, offsetof(Tensor, op_name), 0, nullptr},
    {"_op", T_OBJECT, offsetof(Tensor, op), 0, nullptr},
    {"_parent_module_w", T_OBJECT, offsetof(Tensor, parent_module_w), 0, nullptr},
    {"_pending", T_OBJECT, offsetof(Tensor, pending), 0, nullptr},
    {"_chain", T_OBJECT, offsetof(Tensor, chain), 0, nullptr},
    {"_deps", T_OBJECT, offsetof(Tensor, deps), 0, nullptr},
    {"_buffers", T_OBJECT, offsetof(Tensor, buffers), 0, nullptr},
    {"_t", T_OBJECT, offsetof(Tensor, t), 0, nullptr},
    {"_freezed", T_BOOL, offsetof(Tensor, freezed), 0, nullptr},
    {"_trainable", T_BOOL, offsetof(Tensor, trainable), 0, nullptr},
    {"_shared", T_BOOL, offsetof(Tensor, shared), 0, nullptr},
    {nullptr, 0, 0, 0, nullptr}};
PyType_Slot tensor_slots[] = {{Py_tp_new, (void*)tensor_new}, {Py_tp_dealloc, (void*)tensor_dealloc},
                              {Py_tp_traverse, (void*)tensor_traverse}, {Py_tp_clear, (void*)tensor_clear},
                              {Py_tp_methods, tensor_methods}, {Py_tp_members, tensor_members}, {0, nullptr}};
PyType_Spec tensor_spec = {"litenn_b200._native.TensorBase", sizeof(Tensor), 0,
                           Py_TPFLAGS_DEFAULT | Py_TPFLAGS_BASETYPE | Py_TPFLAGS_HAVE_GC, tensor_slots};

// setup_tensor(tensor, buffer class, devices, shape, init or None, must_init, freezed): the fields of a
// tensor with memory of its own.  `shape` is a TensorShape.
int setup_tensor(Tensor* t, PyTypeObject* buffer_type, PyObject* devices, PyObject* shape, PyObject* init, int must_init,
                 int freezed) {
  PyObject* size_o = PyObject_GetAttr(shape, s_size);
  if (!size_o) return -1;
  const unsigned long long bytes = PyLong_AsUnsignedLongLong(size_o) * 4ull;
  Py_DECREF(size_o);
  if (PyErr_Occurred()) return -1;
  if (!PyTuple_Check(devices)) { PyErr_SetString(PyExc_TypeError, "devices must be a tuple"); return -1; }
  const Py_ssize_t n = PyTuple_GET_SIZE(devices);
  PyObject* list = PyList_New(n);
  if (!list) return -1;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* b = buffer_new(buffer_type, nullptr, nullptr);
    if (!b) { Py_DECREF(list); return -1; }
    PyList_SET_ITEM(list, i, b);
    if (buffer_setup((Buffer*)b, PyTuple_GET_ITEM(devices, i), bytes, init, init == Py_None ? nullptr : shape, must_init)) {
      Py_DECREF(list);
      return -1;
    }
  }
  Py_XSETREF(t->buffers, list);
  Py_INCREF(shape);
  Py_XSETREF(t->shape, shape);
  Py_XSETREF(t->seq_id, PyLong_FromLongLong(++g_seq_id));
  t->freezed = (char)freezed;
  return 0;
}
PyObject* py_setup_tensor(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 7) { PyErr_SetString(PyExc_TypeError, "setup_tensor takes 7 arguments"); return nullptr; }
  if (setup_tensor((Tensor*)a[0], (PyTypeObject*)a[1], a[2], a[3], a[4], PyObject_IsTrue(a[5]), PyObject_IsTrue(a[6])))
    return nullptr;
  Py_RETURN_NONE;
}
// new_tensor(tensor class, buffer class, devices, shape, freezed, op name[, record, members]): the result of an
// operator, whose kernel writes every element.  With a record the kernel has not been launched: the tensor's
// `_pending` is the record, and `members`, the list of its watch, gets a weak reference to the tensor.
PyObject* py_new_tensor(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 6 && n != 8) { PyErr_SetString(PyExc_TypeError, "new_tensor takes 6 or 8 arguments"); return nullptr; }
  PyObject* t = tensor_new((PyTypeObject*)a[0], nullptr, nullptr);
  if (!t) return nullptr;
  if (setup_tensor((Tensor*)t, (PyTypeObject*)a[1], a[2], a[3], Py_None, 0, PyObject_IsTrue(a[4]))) {
    Py_DECREF(t);
    return nullptr;
  }
  Py_INCREF(a[5]);
  ((Tensor*)t)->op_name = a[5];
  if (n == 8) {
    PyObject* ref = PyWeakref_NewRef(t, nullptr);
    if (!ref || PyList_Append(a[7], ref)) { Py_XDECREF(ref); Py_DECREF(t); return nullptr; }
    Py_DECREF(ref);
    Py_INCREF(a[6]);
    ((Tensor*)t)->pending = a[6];
  }
  return t;
}
// observe(tensor, watch): the owner of the tensor's memory refers weakly to work that still has to read it.
PyObject* py_observe(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2 || !PyObject_TypeCheck(a[0], TensorType)) {
    PyErr_SetString(PyExc_TypeError, "observe takes a tensor and a watch");
    return nullptr;
  }
  Tensor* t = top_of(a[0]);
  PyObject* ref = PyWeakref_NewRef(a[1], nullptr);
  if (!ref) return nullptr;
  PyObject* deps = t->deps && PyList_Check(t->deps) ? t->deps : nullptr;
  const Py_ssize_t have = deps ? PyList_GET_SIZE(deps) : 0;
  // what has died leaves when the length reaches a power of two: many that live are not looked at over and over
  if (!deps || (have >= 8 && (have & (have - 1)) == 0)) {
    PyObject* kept = PyList_New(0);
    if (!kept) { Py_DECREF(ref); return nullptr; }
    for (Py_ssize_t i = 0; i < have; ++i) {
      PyObject* r = PyList_GET_ITEM(deps, i);
      if (PyWeakref_GetObject(r) != Py_None && PyList_Append(kept, r)) { Py_DECREF(kept); Py_DECREF(ref); return nullptr; }
    }
    Py_XSETREF(t->deps, kept);
    deps = kept;
  }
  const int rc = PyList_Append(deps, ref);
  Py_DECREF(ref);
  if (rc) return nullptr;
  Py_RETURN_NONE;
}

// ---- library functions -----------------------------------------------------------------------
// Function(address, name, signature)(i, ...): one call of the C ABI for current device number i.  One letter
// per C argument:
//   n      integer                               f  float
//   p      device pointer that is read (a tensor, an address or None)
//   m / w  pointer to memory that is modified / overwritten
//   o      the one or the other, depending on the a argument, the accumulate flag
//   l / L  a list of tensors that are read / modified, passed as an array of their device pointers
// Integers travel in general registers and on the stack in order, floats in vector registers, so one call form
// serves every signature (at most 20 integers, 4 floats).
constexpr int kMaxInts = 20, kMaxFloats = 4, kMaxArgs = 24, kMaxLists = 4;
struct Function {
  PyObject_HEAD
  vectorcallfunc call;
  void* address;
  char name[48];
  char sig[kMaxArgs + 1];
  int n, acc_at;
};
typedef int (*AnyFn)(uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t,
                     uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t,
                     float, float, float, float);

enum Access { READ, MODIFY, OVERWRITE };
int resolve(PyObject* o, Py_ssize_t i, Access access, uint64_t* out) {
  if (PyLong_Check(o)) {
    *out = PyLong_AsUnsignedLongLongMask(o);
    return *out == (uint64_t)-1 && PyErr_Occurred() ? -1 : 0;
  }
  if (o == Py_None) { *out = 0; return 0; }
  if (PyObject_TypeCheck(o, TensorType)) {
    if (access != READ) {
      // work that was put off and reads this tensor has to see the values it has now
      Tensor* t = top_of(o);
      if (t->deps && t->deps != Py_None) {
        PyObject* r = PyObject_CallMethodNoArgs((PyObject*)t, s_before_write);
        if (!r) return -1;
        Py_DECREF(r);
      }
    }
    Buffer* b = tensor_buffer(o, i);
    if (!b) return -1;
    *out = buffer_address(b, access == OVERWRITE);
    return *out ? 0 : -1;
  }
  PyErr_Format(PyExc_TypeError, "expected a tensor or an address, got %s", Py_TYPE(o)->tp_name);
  return -1;
}

// Whether this overwritten argument runs its initializer all the same (it may draw from the host's random stream).
bool initialized_first(PyObject* o, Py_ssize_t i) {
  if (!PyObject_TypeCheck(o, TensorType)) return false;
  PyObject* list = top_of(o)->buffers;
  if (!list || !PyList_Check(list) || i < 0 || i >= PyList_GET_SIZE(list)) return false;
  const Buffer* b = (const Buffer*)PyList_GET_ITEM(list, i);
  return !b->ptr && b->init && b->must_init;
}

PyObject* function_call(PyObject* self, PyObject* const* args, size_t nargsf, PyObject* kwnames) {
  Function* f = (Function*)self;
  const Py_ssize_t n = PyVectorcall_NARGS(nargsf);
  if (n != f->n + 1 || (kwnames && PyTuple_GET_SIZE(kwnames))) {
    PyErr_Format(PyExc_TypeError, "%s takes a device number and %d arguments, got %zd", f->name, f->n, n);
    return nullptr;
  }
  const Py_ssize_t slot = PyLong_AsSsize_t(args[0]);
  if (slot == -1 && PyErr_Occurred()) return nullptr;
  ++args;
  int acc = 0;
  if (f->acc_at >= 0) {
    acc = PyObject_IsTrue(args[f->acc_at]);
    if (acc < 0) return nullptr;
  }
  uint64_t iv[kMaxInts] = {0};
  float fv[kMaxFloats] = {0};
  int ni = 0, nf = 0;
  std::vector<uint64_t> lists[kMaxLists];
  int nl = 0;
  // Memory that is overwritten is looked up last: a tensor nobody has touched skips its initializer there, and
  // the call may read it too, as an argument or through work that has been put off.
  struct { PyObject* tensor; uint64_t* out; } later[kMaxArgs];
  int nlater = 0;
  for (int k = 0; k < f->n; ++k) {
    PyObject* o = args[k];
    switch (f->sig[k]) {
      case 'f': {
        const double v = PyFloat_AsDouble(o);
        if (v == -1.0 && PyErr_Occurred()) return nullptr;
        fv[nf++] = (float)v;
        break;
      }
      case 'n': {
        const long long v = PyLong_AsLongLong(o);
        if (v == -1 && PyErr_Occurred()) return nullptr;
        iv[ni++] = (uint64_t)v;
        break;
      }
      case 'a': iv[ni++] = (uint64_t)acc; break;
      case 'p':
        if (resolve(o, slot, READ, &iv[ni++])) return nullptr;
        break;
      case 'm':
        if (resolve(o, slot, MODIFY, &iv[ni++])) return nullptr;
        break;
      case 'l':
      case 'L': {
        if (!PyList_Check(o)) { PyErr_SetString(PyExc_TypeError, "expected a list of tensors"); return nullptr; }
        std::vector<uint64_t>& v = lists[nl++];
        v.resize((size_t)PyList_GET_SIZE(o) + 1);
        for (Py_ssize_t k2 = 0; k2 < PyList_GET_SIZE(o); ++k2)
          if (resolve(PyList_GET_ITEM(o, k2), slot, f->sig[k] == 'l' ? READ : MODIFY, &v[(size_t)k2])) return nullptr;
        iv[ni++] = (uint64_t)(uintptr_t)v.data();
        break;
      }
      default:                                       // 'w', 'o'
        if (f->sig[k] == 'o' && acc) {
          if (resolve(o, slot, MODIFY, &iv[ni++])) return nullptr;
        } else if (initialized_first(o, slot)) {     // an initializer that always runs keeps its place in the order
          if (resolve(o, slot, OVERWRITE, &iv[ni++])) return nullptr;
        } else {
          later[nlater].tensor = o;
          later[nlater++].out = &iv[ni++];
        }
    }
  }
  for (int k = 0; k < nlater; ++k)
    if (resolve(later[k].tensor, slot, OVERWRITE, later[k].out)) return nullptr;
  int rc;
  AnyFn fn = (AnyFn)f->address;
  Py_BEGIN_ALLOW_THREADS
  rc = fn(iv[0], iv[1], iv[2], iv[3], iv[4], iv[5], iv[6], iv[7], iv[8], iv[9], iv[10], iv[11], iv[12], iv[13], iv[14],
          iv[15], iv[16], iv[17], iv[18], iv[19], fv[0], fv[1], fv[2], fv[3]);
  Py_END_ALLOW_THREADS
  if (rc != 0) { raise_status(rc, f->name); return nullptr; }
  Py_RETURN_NONE;
}

PyObject* function_new(PyTypeObject* type, PyObject* args, PyObject*) {
  unsigned long long address;
  const char *name, *sig;
  if (!PyArg_ParseTuple(args, "Kss", &address, &name, &sig)) return nullptr;
  const size_t n = strlen(sig);
  int ints = 0, floats = 0, lists = 0;
  for (size_t k = 0; k < n; ++k) {
    (sig[k] == 'f' ? floats : ints)++;
    lists += sig[k] == 'l' || sig[k] == 'L';
  }
  if (n > (size_t)kMaxArgs || ints > kMaxInts || floats > kMaxFloats || lists > kMaxLists || strspn(sig, "nfpmwoalL") != n) {
    PyErr_Format(PyExc_ValueError, "bad signature '%s' of %s", sig, name);
    return nullptr;
  }
  Function* f = (Function*)type->tp_alloc(type, 0);
  if (!f) return nullptr;
  f->call = function_call;
  f->address = (void*)(uintptr_t)address;
  snprintf(f->name, sizeof(f->name), "%s", name);
  snprintf(f->sig, sizeof(f->sig), "%s", sig);
  f->n = (int)n;
  const char* a = strchr(sig, 'a');
  f->acc_at = a ? (int)(a - sig) : -1;
  return (PyObject*)f;
}
void function_dealloc(PyObject* self) {
  PyTypeObject* type = Py_TYPE(self);
  type->tp_free(self);
  Py_DECREF(type);
}
PyMemberDef function_members[] = {
    {"__vectorcalloffset__", T_PYSSIZET, offsetof(Function, call), READONLY, nullptr}, {nullptr, 0, 0, 0, nullptr}};
PyType_Slot function_slots[] = {{Py_tp_new, (void*)function_new}, {Py_tp_dealloc, (void*)function_dealloc},
                                {Py_tp_call, (void*)PyVectorcall_Call}, {Py_tp_members, function_members}, {0, nullptr}};
PyType_Spec function_spec = {"litenn_b200._native.Function", sizeof(Function), 0,
                             Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_VECTORCALL, function_slots};

PyObject* py_bind(PyObject*, PyObject* args) {
  unsigned long long alloc, release;
  PyObject* error;
  if (!PyArg_ParseTuple(args, "KKO", &alloc, &release, &error)) return nullptr;
  g_alloc = (AllocFn)(uintptr_t)alloc;
  g_free = (FreeFn)(uintptr_t)release;
  Py_INCREF(error);
  Py_XSETREF(g_error, error);
  Py_RETURN_NONE;
}
PyObject* py_buffer_count(PyObject*, PyObject*) { return PyLong_FromLong(g_buffers); }
PyObject* py_tensor_count(PyObject*, PyObject*) { return PyLong_FromLong(g_tensors); }

PyMethodDef module_methods[] = {
    {"bind", py_bind, METH_VARARGS, "bind(lnn_alloc, lnn_free, error): addresses and the function that raises for a status."},
    {"setup_tensor", (PyCFunction)(void (*)(void))py_setup_tensor, METH_FASTCALL, nullptr},
    {"new_tensor", (PyCFunction)(void (*)(void))py_new_tensor, METH_FASTCALL, nullptr},
    {"observe", (PyCFunction)(void (*)(void))py_observe, METH_FASTCALL, nullptr},
    {"buffer_count", py_buffer_count, METH_NOARGS, "Live device buffers."},
    {"tensor_count", py_tensor_count, METH_NOARGS, "Live tensors."},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, module_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
  s_ensure = PyUnicode_InternFromString("_ensure");
  s_inited = PyUnicode_InternFromString("_inited");
  s_initialize_buffer = PyUnicode_InternFromString("initialize_buffer");
  s_size = PyUnicode_InternFromString("size");
  s_index = PyUnicode_InternFromString("index");
  s_before_write = PyUnicode_InternFromString("_before_write");
  s_get_buffers = PyUnicode_InternFromString("_get_buffers");
  PyObject* m = PyModule_Create(&module_def);
  if (!m) return nullptr;
  PyObject* b = PyType_FromSpec(&buffer_spec);
  PyObject* t = PyType_FromSpec(&tensor_spec);
  PyObject* f = PyType_FromSpec(&function_spec);
  if (!b || !t || !f) return nullptr;
  BufferType = (PyTypeObject*)b;
  TensorType = (PyTypeObject*)t;
  PyModule_AddObject(m, "BufferBase", b);
  PyModule_AddObject(m, "TensorBase", t);
  PyModule_AddObject(m, "Function", f);
  return m;
}
