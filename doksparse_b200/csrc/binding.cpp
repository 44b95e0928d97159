// _native: the map's and the DOK tensor's hot calls from Python in one step each.
//
// A call of the C ABI through ctypes spends more time around the launch than in it: checking the tensors, allocating the
// outputs, packing the structs and entering the device took 14 us of a 16 us lookup of 1000 rows.  A Plan holds what does
// not change between calls on one table (the packed structs, the expected shapes and types) and does the rest in C++.
// Every method answers None for arguments that it does not take as they are (another device, a view that is not
// contiguous, a type to convert, ...); the Python methods then go their general way, which raises the documented errors.
#define PY_SSIZE_T_CLEAN
#include <ATen/Functions.h>
#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <structmember.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/doksparse.h"

namespace {

struct Plan {
  PyObject_HEAD
  dok_table table;
  dok_hash_params hash;
  int64_t *state;              // counter blocks of the table (device)
  int device;
  int key_ndim, value_ndim;    // dims of one row
  int64_t key_shape[8], value_shape[8];
  at::ScalarType key_type, value_type;
};

enum { STATE_SET = 0, STATE_REMOVE = 8, STATE_BULK = 24, STATE_ADJUST = 7, STATE_WORDS = 32 };   // int64 offsets of the counter blocks

PyObject *dok_error = nullptr;
extern PyTypeObject plan_type;

// -> true, or sets DokError with the wording of the ctypes path
bool check(int status, const char *what) {
  if (status == DOK_OK) return true;
  const char *name = status == DOK_BAD_ARG ? "DOK_BAD_ARG" : status == DOK_CUDA_ERROR ? "DOK_CUDA_ERROR" : "DOK_TOO_LARGE";
  if (status == DOK_CUDA_ERROR) PyErr_Format(dok_error, "%s failed: %s (cudaError %d)", what, name, dok_last_cuda_error());
  else PyErr_Format(dok_error, "%s failed: %s", what, name);
  return false;
}

bool rows_match(const at::Tensor &t, int device, at::ScalarType type, int ndim, const int64_t *shape) {
  if (!t.is_cuda() || t.scalar_type() != type || t.layout() != at::kStrided || t.get_device() != device) return false;
  const auto sizes = t.sizes();
  if ((int)sizes.size() != ndim + 1) return false;
  for (int i = 0; i < ndim; i++) if (sizes[i + 1] != shape[i]) return false;
  return t.is_contiguous();
}

const at::Tensor *tensor_of(PyObject *o) { return THPVariable_Check(o) ? &THPVariable_Unpack(o) : nullptr; }

at::TensorOptions on_device(const Plan *p, at::ScalarType type) {
  return at::TensorOptions().dtype(type).device(at::Device(at::kCUDA, (c10::DeviceIndex)p->device));
}

// C++ exceptions (out of memory, most of all) become Python's
template <class F>
PyObject *guarded(F f) {
  HANDLE_TH_ERRORS
  return f();
  END_HANDLE_TH_ERRORS
}

int shape_from(PyObject *tuple, int64_t *out, int most = 7) {
  if (!PyTuple_Check(tuple) || PyTuple_GET_SIZE(tuple) > most) return -1;
  const int n = (int)PyTuple_GET_SIZE(tuple);
  for (int i = 0; i < n; i++) {
    out[i] = PyLong_AsLongLong(PyTuple_GET_ITEM(tuple, i));
    if (out[i] == -1 && PyErr_Occurred()) return -1;
  }
  return n;
}

// Plan(table: bytes, hash: bytes, state address, device index, key shape, key dtype, value shape, value dtype)
int plan_init(Plan *self, PyObject *args, PyObject *) {
  const char *table, *hash;
  Py_ssize_t table_bytes, hash_bytes;
  unsigned long long state;
  int device;
  PyObject *key_shape, *key_type, *value_shape, *value_type;
  if (!PyArg_ParseTuple(args, "y#y#KiOOOO", &table, &table_bytes, &hash, &hash_bytes, &state, &device, &key_shape, &key_type,
                        &value_shape, &value_type))
    return -1;
  self->key_ndim = shape_from(key_shape, self->key_shape);
  self->value_ndim = shape_from(value_shape, self->value_shape);
  if (table_bytes != sizeof(dok_table) || hash_bytes != sizeof(dok_hash_params) || self->key_ndim < 0 || self->value_ndim < 0 ||
      !THPDtype_Check(key_type) || !THPDtype_Check(value_type)) {
    PyErr_SetString(PyExc_ValueError, "Plan: bad arguments");
    return -1;
  }
  memcpy(&self->table, table, sizeof(dok_table));
  memcpy(&self->hash, hash, sizeof(dok_hash_params));
  self->state = (int64_t *)state;
  self->device = device;
  self->key_type = reinterpret_cast<THPDtype *>(key_type)->scalar_type;
  self->value_type = reinterpret_cast<THPDtype *>(value_type)->scalar_type;
  return 0;
}

// allocate(device index, buckets, key shape, key dtype, value shape, value dtype, state tensor or None) ->
// (plan without hash parameters, slots, state, layout): a new slot array with empty tags and zero counters
PyObject *plan_allocate(PyObject *, PyObject *args) {
  return guarded([&]() -> PyObject * {
    int device;
    long long buckets;
    PyObject *key_shape, *key_type, *value_shape, *value_type, *given_state;
    if (!PyArg_ParseTuple(args, "iLOOOOO", &device, &buckets, &key_shape, &key_type, &value_shape, &value_type, &given_state)) return nullptr;
    Plan *p = PyObject_New(Plan, &plan_type);
    if (!p) return nullptr;
    struct Drop { Plan *p; ~Drop() { Py_XDECREF((PyObject *)p); } } drop{p};
    memset(&p->table, 0, sizeof(p->table));
    memset(&p->hash, 0, sizeof(p->hash));
    p->device = device;
    p->key_ndim = shape_from(key_shape, p->key_shape);
    p->value_ndim = shape_from(value_shape, p->value_shape);
    if (p->key_ndim < 0 || p->value_ndim < 0 || !THPDtype_Check(key_type) || !THPDtype_Check(value_type)) {
      if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "allocate: bad arguments");
      return nullptr;
    }
    p->key_type = reinterpret_cast<THPDtype *>(key_type)->scalar_type;
    p->value_type = reinterpret_cast<THPDtype *>(value_type)->scalar_type;
    int64_t key_bytes = c10::elementSize(p->key_type), value_bytes = c10::elementSize(p->value_type);
    for (int i = 0; i < p->key_ndim; i++) key_bytes *= p->key_shape[i];
    for (int i = 0; i < p->value_ndim; i++) value_bytes *= p->value_shape[i];
    dok_layout_info lay;
    if (!check(dok_table_layout((int)value_bytes, (int)key_bytes, buckets, &lay), "dok_table_layout")) return nullptr;
    const c10::cuda::CUDAGuard guard((c10::DeviceIndex)device);
    at::Tensor slots = at::empty({lay.total_bytes}, on_device(p, at::kByte));
    const at::Tensor *given = tensor_of(given_state);
    at::Tensor state = given ? *given : at::empty({STATE_WORDS}, on_device(p, at::kLong));
    p->table.slots = slots.data_ptr();
    p->table.n_buckets = buckets;
    p->table.slot_bytes = lay.slot_bytes;
    p->table.value_bytes = (int32_t)value_bytes;
    p->table.key_bytes = (int32_t)key_bytes;
    p->state = (int64_t *)state.data_ptr();
    if (!check(dok_map_init_state(&p->table, p->state, STATE_WORDS, c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream()),
               "dok_map_init_state"))
      return nullptr;
    drop.p = nullptr;
    return Py_BuildValue("(NNN(iiiiiLL))", (PyObject *)p, THPVariable_Wrap(std::move(slots)), THPVariable_Wrap(std::move(state)), lay.slot_bytes,
                         lay.slots_per_group, lay.value_offset, lay.key_offset, lay.stamp_offset, (long long)lay.n_slots,
                         (long long)lay.total_bytes);
  });
}

// set_hash(dtype code, alpha2, beta2, prime2, alpha1, beta1, prime1, key_perm): lists of one integer per key element
PyObject *plan_set_hash(Plan *self, PyObject *const *args, Py_ssize_t nargs) {
  if (nargs != 8) { PyErr_SetString(PyExc_TypeError, "set_hash takes 8 arguments"); return nullptr; }
  self->hash.key_dtype = (int32_t)PyLong_AsLong(args[0]);
  const Py_ssize_t n = PyList_Check(args[1]) ? PyList_GET_SIZE(args[1]) : 0;
  int64_t *to[6] = {self->hash.alpha2, self->hash.beta2, self->hash.prime2, self->hash.alpha1, self->hash.beta1, self->hash.prime1};
  for (int k = 1; k < 8; k++) {
    if (!PyList_Check(args[k]) || PyList_GET_SIZE(args[k]) != n || n < 1 || n > DOK_MAX_KEY_SIZE) {
      PyErr_SetString(PyExc_ValueError, "set_hash: one value per key element");
      return nullptr;
    }
    for (Py_ssize_t i = 0; i < n; i++) {
      const long long v = PyLong_AsLongLong(PyList_GET_ITEM(args[k], i));
      if (k < 7) to[k - 1][i] = v; else self->hash.key_perm[i] = (int32_t)v;
    }
  }
  if (PyErr_Occurred()) return nullptr;
  self->hash.key_size = (int32_t)n;
  Py_RETURN_NONE;
}

// ---- what sets leave behind in one slot array ---------------------------------------------------------------

// For as long as there is the slot array: every map that writes it has these marks, a new one gets new ones.  They are changed
// with the interpreter's lock held, so that sets from several threads and on several streams never share an epoch or numbers.
struct Marks {
  PyObject_HEAD
  PyObject *stamp;             // the stamps (a tensor), where the slots have no room for them and a set has needed them
  long long epoch;             // largest one in a stamp
  long long numbered;          // largest number of a row that shares its value's word with it
  long long renumbered;        // ... that sets in graphs use again and again
  cudaStream_t stream;         // of the numbered sets so far
  bool any, several;           // there were some; on more than one stream
};

void marks_dealloc(Marks *self) {
  Py_XDECREF(self->stamp);
  Py_TYPE(self)->tp_free((PyObject *)self);
}

// Marks(), or Marks(other, stamp): for a copy of other's slots, `stamp` the copy of its stamps or None
int marks_init(Marks *self, PyObject *args, PyObject *) {
  PyObject *other = nullptr, *stamp = Py_None;
  if (!PyArg_ParseTuple(args, "|OO", &other, &stamp)) return -1;
  if (other && Py_TYPE(other) != Py_TYPE(self)) { PyErr_SetString(PyExc_TypeError, "Marks: other marks expected"); return -1; }
  if (other) {
    const Marks *m = (const Marks *)other;
    self->epoch = m->epoch;
    self->numbered = m->numbered;
  }
  Py_INCREF(stamp);
  Py_XSETREF(self->stamp, stamp);
  return 0;
}

// in the slots, or in an array that the marks have
bool add_stamps(const Marks *m, dok_table *table) {
  const at::Tensor *stamp = m->stamp ? tensor_of(m->stamp) : nullptr;
  table->stamp = stamp ? (int64_t *)stamp->data_ptr() : nullptr;
  dok_layout_info lay;
  return stamp || (dok_table_layout(table->value_bytes, table->key_bytes, table->n_buckets, &lay) == DOK_OK && lay.stamp_offset >= 0);
}

// A new start for the numbers: nothing that numbers rows of these slots is on its way, and nothing starts before they are
// cleared.  false where there is no quiet moment for it (or, with several streams, where one of them captures); the caller
// stamps its rows then.
bool start_over(const Plan *p, Marks *m, cudaStream_t stream) {
  for (int i = 0; i < 4; i++) {
    const int64_t launched = dok_launch_count();
    cudaError_t e;
    Py_BEGIN_ALLOW_THREADS
    e = m->several || m->stream != stream ? cudaDeviceSynchronize() : cudaStreamSynchronize(stream);
    Py_END_ALLOW_THREADS
    if (e == cudaErrorStreamCaptureUnsupported) { (void)cudaGetLastError(); return false; }
    C10_CUDA_CHECK(e);
    if (dok_launch_count() != launched) continue;            // another thread had the interpreter meanwhile
    if (dok_map_clear_numbers(&p->table, stream) != DOK_OK) return false;
    C10_CUDA_CHECK(cudaStreamSynchronize(stream));
    m->numbered = 0;
    m->any = m->several = false;
    return true;
  }
  return false;
}

// Numbers for n rows, to `base`; false where their set has to be stamped.
bool take_numbers(const Plan *p, Marks *m, int64_t n, cudaStream_t stream, int64_t *base) {
  if (!dok_set_takes_numbers(&p->table, &p->hash, n)) return false;
  cudaStreamCaptureStatus capturing;
  C10_CUDA_CHECK(cudaStreamIsCapturing(stream, &capturing));
  if (capturing != cudaStreamCaptureStatusNone) {
    m->renumbered = std::max<long long>(m->renumbered, n);
    m->numbered = std::max(m->numbered, m->renumbered);
    *base = DOK_RENUMBER;
    return true;
  }
  // (sets in graphs are replayed without anybody asking here, so with them no moment is quiet for certain)
  if (m->numbered > DOK_MAX_NUMBER - n && (m->renumbered > 0 || !start_over(p, m, stream))) return false;
  m->several = m->several || (m->any && m->stream != stream);
  m->any = true;
  m->stream = stream;
  *base = m->numbered;
  m->numbered += n;
  return true;
}

// An epoch for a stamped set, and its table with the stamps; false where the stamps have yet to be made or epochs are used up
bool take_epoch(Marks *m, dok_table *table, int64_t *epoch) {
  if (!add_stamps(m, table) || m->epoch >= DOK_MAX_EPOCH - 1) return false;
  *epoch = ++m->epoch;
  return true;
}

Marks *marks_of(PyObject *o);

// ---- counts that travel to the host by themselves -----------------------------------------------------------

// Eight landing places for copies of a table's counters, in pinned memory that the caller provides, with an event each.
struct Ring {
  PyObject_HEAD
  PyObject *memory;            // keeps the pinned words alive
  int64_t *words;
  int device;
  cudaEvent_t events[8];
  unsigned used;
};

// Ring(pinned int64 tensor of 8 * STATE_WORDS, device index)
int ring_init(Ring *self, PyObject *args, PyObject *) {
  PyObject *memory;
  if (!PyArg_ParseTuple(args, "Oi", &memory, &self->device)) return -1;
  const at::Tensor *t = tensor_of(memory);
  if (!t || t->scalar_type() != at::kLong || t->numel() != 8 * STATE_WORDS || !t->is_contiguous()) {
    PyErr_SetString(PyExc_ValueError, "Ring: pinned words expected");
    return -1;
  }
  Py_INCREF(memory);
  self->memory = memory;
  self->words = (int64_t *)t->data_ptr();
  return 0;
}
void ring_dealloc(Ring *self) {
  // a copy on its way would land in memory that the allocator has given to somebody else
  Py_BEGIN_ALLOW_THREADS
  for (int i = 0; i < 8; i++) if ((self->used >> i) & 1u) (void)cudaEventSynchronize(self->events[i]);
  Py_END_ALLOW_THREADS
  for (int i = 0; i < 8; i++) if (self->events[i]) cudaEventDestroy(self->events[i]);
  Py_XDECREF(self->memory);
  Py_TYPE(self)->tp_free((PyObject *)self);
}

// copy(plan, place): enqueues a copy of the plan's counters
PyObject *ring_copy(Ring *self, PyObject *const *args, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject * {
    if (nargs != 2 || Py_TYPE(args[0]) != &plan_type) { PyErr_SetString(PyExc_TypeError, "copy takes a Plan and a place"); return nullptr; }
    const Plan *plan = (const Plan *)args[0];
    const long i = PyLong_AsLong(args[1]);
    if (i < 0 || i > 7 || plan->device != self->device) { PyErr_SetString(PyExc_ValueError, "copy: no such place"); return nullptr; }
    const c10::cuda::CUDAGuard guard((c10::DeviceIndex)self->device);
    const auto stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)self->device);
    if (!self->events[i]) C10_CUDA_CHECK(cudaEventCreateWithFlags(&self->events[i], cudaEventDisableTiming));
    C10_CUDA_CHECK(cudaMemcpyAsync(self->words + i * STATE_WORDS, plan->state, STATE_WORDS * sizeof(int64_t), cudaMemcpyDeviceToHost, stream.stream()));
    C10_CUDA_CHECK(cudaEventRecord(self->events[i], stream.stream()));
    self->used |= 1u << i;
    Py_RETURN_NONE;
  });
}
// landed(place) -> bool
PyObject *ring_landed(Ring *self, PyObject *arg) {
  return guarded([&]() -> PyObject * {
    const long i = PyLong_AsLong(arg);
    if (i < 0 || i > 7 || !self->events[i]) { PyErr_SetString(PyExc_ValueError, "landed: no such copy"); return nullptr; }
    const cudaError_t e = cudaEventQuery(self->events[i]);
    if (e == cudaErrorNotReady) { (void)cudaGetLastError(); Py_RETURN_FALSE; }
    C10_CUDA_CHECK(e);
    Py_RETURN_TRUE;
  });
}
// wait(place), or wait(-1) for every copy so far
PyObject *ring_wait(Ring *self, PyObject *arg) {
  return guarded([&]() -> PyObject * {
    const long i = PyLong_AsLong(arg);
    cudaError_t e = cudaSuccess;
    Py_BEGIN_ALLOW_THREADS
    for (int k = 0; k < 8; k++) if ((i < 0 || i == k) && ((self->used >> k) & 1u) && e == cudaSuccess) e = cudaEventSynchronize(self->events[k]);
    Py_END_ALLOW_THREADS
    C10_CUDA_CHECK(e);
    Py_RETURN_NONE;
  });
}
// read(place) -> the counters
PyObject *ring_read(Ring *self, PyObject *arg) {
  const long i = PyLong_AsLong(arg);
  if (i < 0 || i > 7) { PyErr_SetString(PyExc_ValueError, "read: no such place"); return nullptr; }
  PyObject *list = PyList_New(STATE_WORDS);
  for (int k = 0; list && k < STATE_WORDS; k++) PyList_SET_ITEM(list, k, PyLong_FromLongLong(self->words[i * STATE_WORDS + k]));
  return list;
}

// ---- the map ------------------------------------------------------------------------------------------------

// get(keys) -> (values, is_found) or None
PyObject *plan_get(Plan *self, PyObject *arg) {
  return guarded([&]() -> PyObject * {
    const at::Tensor *keys = tensor_of(arg);
    if (!keys || !rows_match(*keys, self->device, self->key_type, self->key_ndim, self->key_shape)) Py_RETURN_NONE;
    const int64_t n = keys->size(0);
    if (n == 0) Py_RETURN_NONE;
    const c10::cuda::CUDAGuard guard((c10::DeviceIndex)self->device);
    int64_t shape[8] = {n};
    for (int i = 0; i < self->value_ndim; i++) shape[i + 1] = self->value_shape[i];
    at::Tensor values = at::empty(at::IntArrayRef(shape, self->value_ndim + 1), on_device(self, self->value_type));
    at::Tensor found = at::empty({n}, on_device(self, at::kBool));
    if (!check(dok_map_get(&self->table, &self->hash, keys->data_ptr(), n, values.data_ptr(), (uint8_t *)found.data_ptr(), nullptr,
                           nullptr, c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)self->device).stream()),
               "dok_map_get"))
      return nullptr;
    PyObject *v = THPVariable_Wrap(std::move(values)), *f = THPVariable_Wrap(std::move(found));
    PyObject *out = v && f ? PyTuple_Pack(2, v, f) : nullptr;
    Py_XDECREF(v);
    Py_XDECREF(f);
    return out;
  });
}

// set(keys, values, assume_unique, marks) -> the number of rows, or None
PyObject *plan_set(Plan *self, PyObject *const *args, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject * {
    Marks *marks = nargs == 4 ? marks_of(args[3]) : nullptr;
    if (!marks) { PyErr_SetString(PyExc_TypeError, "set takes keys, values, assume_unique and Marks"); return nullptr; }
    const at::Tensor *keys = tensor_of(args[0]), *values = tensor_of(args[1]);
    if (!keys || !values || !rows_match(*keys, self->device, self->key_type, self->key_ndim, self->key_shape) ||
        !rows_match(*values, self->device, self->value_type, self->value_ndim, self->value_shape) || keys->size(0) != values->size(0) ||
        keys->size(0) == 0)
      Py_RETURN_NONE;
    const int64_t n = keys->size(0);
    const int unique = PyObject_IsTrue(args[2]);
    if (unique < 0) return nullptr;
    const c10::cuda::CUDAGuard guard((c10::DeviceIndex)self->device);
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)self->device).stream();
    dok_table table = self->table;
    int64_t base, epoch;
    if (unique) {
      add_stamps(marks, &table);         // (windows are cut by the bytes of slots and stamps)
      if (!check(dok_map_set_unique(&table, &self->hash, keys->data_ptr(), values->data_ptr(), n, nullptr, self->state + STATE_SET, stream),
                 "dok_map_set_unique"))
        return nullptr;
    } else if (take_numbers(self, marks, n, stream, &base)) {
      if (!check(dok_map_set_numbered(&table, &self->hash, keys->data_ptr(), values->data_ptr(), n, base, self->state + STATE_SET, stream),
                 "dok_map_set_numbered"))
        return nullptr;
    } else {
      if (!take_epoch(marks, &table, &epoch)) Py_RETURN_NONE;
      const int64_t words = dok_set_scratch_words(&table, n);
      at::Tensor scratch;
      if (words > 0) scratch = at::empty({words}, on_device(self, at::kLong));
      if (!check(dok_map_set_with(&table, &self->hash, keys->data_ptr(), values->data_ptr(), n,
                                  words > 0 ? (int64_t *)scratch.data_ptr() : nullptr, words, epoch, self->state + STATE_SET, stream),
                 "dok_map_set_with"))
        return nullptr;
    }
    return PyLong_FromLongLong(n);
  });
}

// remove_rows(keys) -> is_removed or None
PyObject *plan_remove_rows(Plan *self, PyObject *arg) {
  return guarded([&]() -> PyObject * {
    const at::Tensor *keys = tensor_of(arg);
    if (!keys || !rows_match(*keys, self->device, self->key_type, self->key_ndim, self->key_shape)) Py_RETURN_NONE;
    const int64_t n = keys->size(0);
    if (n == 0) Py_RETURN_NONE;
    const c10::cuda::CUDAGuard guard((c10::DeviceIndex)self->device);
    at::Tensor removed = at::empty({n}, on_device(self, at::kBool));
    if (!check(dok_map_remove(&self->table, &self->hash, keys->data_ptr(), n, (uint8_t *)removed.data_ptr(), self->state + STATE_REMOVE,
                              c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)self->device).stream()),
               "dok_map_remove"))
      return nullptr;
    return THPVariable_Wrap(std::move(removed));
  });
}

// A few words of pinned memory per thread, for counts that a call has to wait for.
int64_t *pinned_words() {
  static thread_local at::Tensor words;
  if (!words.defined()) words = at::empty({STATE_WORDS}, at::TensorOptions().dtype(at::kLong).pinned_memory(true));
  return (int64_t *)words.data_ptr();
}

void wait_for(const c10::cuda::CUDAStream &stream) {           // other Python threads run meanwhile
  struct Released {
    PyThreadState *state = PyEval_SaveThread();
    ~Released() { PyEval_RestoreThread(state); }
  } released;
  stream.synchronize();
}

PyObject *read_state(Plan *self, const c10::cuda::CUDAStream &stream) {
  int64_t *words = pinned_words();
  C10_CUDA_CHECK(cudaMemcpyAsync(words, self->state, STATE_WORDS * sizeof(int64_t), cudaMemcpyDeviceToHost, stream.stream()));
  wait_for(stream);
  PyObject *list = PyList_New(STATE_WORDS);
  for (int i = 0; list && i < STATE_WORDS; i++) PyList_SET_ITEM(list, i, PyLong_FromLongLong(words[i]));
  return list;
}

// read() -> the counters of the table
PyObject *plan_read(Plan *self, PyObject *) {
  return guarded([&]() -> PyObject * {
    const c10::cuda::CUDAGuard guard((c10::DeviceIndex)self->device);
    return read_state(self, c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)self->device));
  });
}

// count_new(keys, word, exact, empty table): adds the number of distinct new keys to the counter `word`; exact: sets it, and
// answers the counters
PyObject *plan_count_new(Plan *self, PyObject *const *args, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject * {
    if (nargs != 4) { PyErr_SetString(PyExc_TypeError, "count_new takes 4 arguments"); return nullptr; }
    const at::Tensor *keys = tensor_of(args[0]);
    const long word = PyLong_AsLong(args[1]);
    const int exact = PyObject_IsTrue(args[2]), empty = PyObject_IsTrue(args[3]);
    if (PyErr_Occurred()) return nullptr;
    if (!keys || word < 0 || word >= STATE_WORDS || !rows_match(*keys, self->device, self->key_type, self->key_ndim, self->key_shape)) {
      PyErr_SetString(PyExc_ValueError, "count_new: not a batch of this table");
      return nullptr;
    }
    const c10::cuda::CUDAGuard guard((c10::DeviceIndex)self->device);
    const auto stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)self->device);
    const int64_t n = keys->size(0);
    at::Tensor scratch = at::empty({2 * n}, on_device(self, at::kLong));
    if (exact) C10_CUDA_CHECK(cudaMemsetAsync(self->state + word, 0, sizeof(int64_t), stream.stream()));
    const auto count = at::isFloatingType(self->key_type) ? dok_map_count_new_rows : dok_map_count_new;
    if (!check(count(empty ? nullptr : &self->table, &self->hash, keys->data_ptr(), n, (int64_t *)scratch.data_ptr(), 2 * n, self->state + word, stream.stream()),
               "dok_map_count_new"))
      return nullptr;
    if (exact) return read_state(self, stream);
    Py_RETURN_NONE;
  });
}

// reinsert(plan): the live rows of another table of the same row shape
PyObject *plan_reinsert(Plan *self, PyObject *arg) {
  return guarded([&]() -> PyObject * {
    if (Py_TYPE(arg) != &plan_type) { PyErr_SetString(PyExc_TypeError, "reinsert takes a Plan"); return nullptr; }
    const c10::cuda::CUDAGuard guard((c10::DeviceIndex)self->device);
    if (!check(dok_map_reinsert(&((Plan *)arg)->table, &self->table, &self->hash, self->state + STATE_BULK,
                                c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)self->device).stream()),
               "dok_map_reinsert"))
      return nullptr;
    Py_RETURN_NONE;
  });
}

// remove(keys) -> flags of the sorted unique rows, or None
PyObject *plan_remove(Plan *self, PyObject *arg) {
  return guarded([&]() -> PyObject * {
    const at::Tensor *keys = tensor_of(arg);
    if (!keys || !rows_match(*keys, self->device, self->key_type, self->key_ndim, self->key_shape)) Py_RETURN_NONE;
    const int64_t n = keys->size(0), bytes = n ? dok_map_remove_unique_bytes(n) : -1;
    if (bytes < 0) Py_RETURN_NONE;
    const c10::cuda::CUDAGuard guard((c10::DeviceIndex)self->device);
    const auto stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)self->device);
    at::Tensor removed = at::empty({n}, on_device(self, at::kBool)), work;
    if (bytes) work = at::empty({bytes}, on_device(self, at::kByte));
    volatile int64_t *count = pinned_words();
    *count = -2;
    int status = dok_map_remove_unique(&self->table, &self->hash, keys->data_ptr(), n, (uint8_t *)removed.data_ptr(),
                                       bytes ? work.data_ptr() : nullptr, (int64_t *)count, self->state + STATE_REMOVE, stream.stream());
    if (status == DOK_TOO_LARGE) Py_RETURN_NONE;
    if (!check(status, "dok_map_remove_unique")) return nullptr;
    wait_for(stream);
    if (*count < -DOK_SORT_ALL_WORDS) {
      const int words = (int)(-*count - DOK_SORT_ALL_WORDS);
      *count = -2;
      status = dok_map_remove_unique_words(&self->table, &self->hash, keys->data_ptr(), n, (uint8_t *)removed.data_ptr(), work.data_ptr(), words,
                                           (int64_t *)count, self->state + STATE_REMOVE, stream.stream());
      if (!check(status, "dok_map_remove_unique_words")) return nullptr;
      wait_for(stream);
    }
    if (*count == -1) Py_RETURN_NONE;
    if (*count < 0) { PyErr_SetString(dok_error, "dok_map_remove_unique: a wait between blocks ran out"); return nullptr; }
    at::Tensor flags = removed.narrow(0, 0, *count);
    // flags of a large batch with few different rows do not hold the memory of all of them; a copy costs 6 us
    if (n - *count >= 1 << 20) flags = flags.clone();
    return THPVariable_Wrap(std::move(flags));
  });
}

// ---- selectors of a DOK tensor ------------------------------------------------------------------------------

struct Selection {
  dok_selectors sel;
  int64_t n;                          // selected positions
  c10::SmallVector<int64_t, 8> shape; // their common shape
  int scalars[DOK_MAX_KEY_SIZE];      // positions of the scalar selectors
  int n_scalars;
  c10::SmallVector<at::Tensor, 4> keep;
};

struct One { bool slice; int64_t start, stop; const at::Tensor *tensor; };   // tensor null and not a slice: the scalar `start`

// integer member of a slice, or its default; false for anything but None and int
bool bound_of(PyObject *o, int64_t size, int64_t none, int64_t *out) {
  if (o == Py_None) { *out = none; return true; }
  if (!PyLong_CheckExact(o)) return false;
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  *out = v < 0 ? std::max<int64_t>(v + size, 0) : v;
  return true;
}

// What selectors.normalise_selectors computes, for ints, slices and index or mask tensors on the table's device, without
// an index tensor for a slice or a scalar.  false: leave it to the general way.
bool parse_selection(PyObject *selectors, const int64_t *size, int ndim, int device, Selection *out) {
  One list[DOK_MAX_KEY_SIZE];
  int count = 0;
  const bool many = PyTuple_Check(selectors);
  const Py_ssize_t given = many ? PyTuple_GET_SIZE(selectors) : 1;
  out->keep.reserve(2 * DOK_MAX_KEY_SIZE);                     // `list` points into it
  for (Py_ssize_t i = 0; i < given; i++) {
    PyObject *o = many ? PyTuple_GET_ITEM(selectors, i) : selectors;
    if (count >= ndim) return false;
    if (PyLong_CheckExact(o)) {
      const long long v = PyLong_AsLongLong(o);
      if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
      list[count++] = One{false, v, 0, nullptr};
    } else if (PySlice_Check(o)) {
      const PySliceObject *s = (const PySliceObject *)o;
      const int64_t extent = size[count];
      int64_t start, stop;
      if (!bound_of(s->start, extent, 0, &start) || !bound_of(s->stop, extent, extent, &stop)) return false;
      list[count++] = One{true, start, std::max(std::min(stop, extent), start), nullptr};
    } else if (const at::Tensor *t = tensor_of(o)) {
      if (!t->is_cuda() || t->get_device() != device || t->layout() != at::kStrided) return false;
      if (t->scalar_type() == at::kLong) {
        out->keep.push_back(*t);
        list[count++] = One{false, 0, 0, &out->keep.back()};
      } else if (t->scalar_type() == at::kBool && t->dim() > 0) {
        if (count + t->dim() > ndim) return false;
        const at::Tensor where = at::nonzero(*t);
        for (int64_t d = 0; d < t->dim(); d++) {
          out->keep.push_back(where.select(1, d));
          list[count++] = One{false, 0, 0, &out->keep.back()};
        }
      } else {
        return false;
      }
    } else {
      return false;
    }
  }
  for (; count < ndim; count++) list[count] = One{true, 0, size[count], nullptr};

  // the broadcast block of the tensors, and where it sits among the slices
  int64_t block[DOK_MAX_SELECTOR_NDIM];
  int block_ndim = 0, n_slices = 0, first = -1;
  for (int i = 0; i < ndim; i++) {
    if (list[i].slice) { n_slices++; continue; }
    if (first < 0) first = i;
    if (list[i].tensor) block_ndim = std::max<int>(block_ndim, (int)list[i].tensor->dim());
  }
  if (block_ndim + n_slices > DOK_MAX_SELECTOR_NDIM) return false;
  for (int j = 0; j < block_ndim; j++) block[j] = 1;
  for (int i = 0; i < ndim; i++) {
    if (!list[i].tensor) continue;
    const auto sizes = list[i].tensor->sizes();
    const int off = block_ndim - (int)sizes.size();
    for (int j = 0; j < (int)sizes.size(); j++) {
      if (sizes[j] == 1 || sizes[j] == block[off + j]) continue;
      if (block[off + j] != 1) return false;
      block[off + j] = sizes[j];
    }
  }
  dok_selectors &sel = out->sel;
  memset(&sel, 0, sizeof(sel));
  sel.ndim = ndim;
  sel.selector_ndim = block_ndim + n_slices;
  out->n_scalars = 0;
  int axis = 0;
  for (int i = 0; i < ndim; i++) {
    if (list[i].slice) {
      sel.sizes[axis] = list[i].stop - list[i].start;
      sel.strides[i][axis] = 1;
      sel.base[i] = list[i].start;
      axis++;
      continue;
    }
    if (i == first) {
      for (int j = 0; j < block_ndim; j++) sel.sizes[first + j] = block[j];
      axis += block_ndim;
    }
    if (const at::Tensor *t = list[i].tensor) {
      sel.ptr[i] = (const int64_t *)t->data_ptr();
      const int off = block_ndim - (int)t->dim();
      for (int j = 0; j < (int)t->dim(); j++)
        if (t->size(j) != 1) sel.strides[i][first + off + j] = t->stride(j);
    } else {
      sel.base[i] = list[i].start;
    }
    if (!list[i].tensor || list[i].tensor->dim() == 0) out->scalars[out->n_scalars++] = i;
  }
  out->n = 1;
  for (int j = 0; j < sel.selector_ndim; j++) {
    out->shape.push_back(sel.sizes[j]);
    out->n *= sel.sizes[j];
  }
  return true;
}

// index(selectors, size) -> the dense gather, or None
PyObject *plan_index(Plan *self, PyObject *const *args, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject * {
    if (nargs != 2) { PyErr_SetString(PyExc_TypeError, "index takes 2 arguments"); return nullptr; }
    int64_t size[DOK_MAX_KEY_SIZE];
    const int ndim = shape_from(args[1], size, DOK_MAX_KEY_SIZE);
    if (ndim < 1 || ndim > DOK_MAX_KEY_SIZE || ndim != self->hash.key_size || self->value_ndim != 1 || self->value_shape[0] != 1) {
      PyErr_Clear();
      Py_RETURN_NONE;
    }
    const c10::cuda::CUDAGuard guard((c10::DeviceIndex)self->device);
    Selection s;
    if (!parse_selection(args[0], size, ndim, self->device, &s)) Py_RETURN_NONE;
    at::Tensor values = at::empty(s.shape, on_device(self, self->value_type));
    if (s.n > 0 &&
        !check(dok_dok_get(&self->table, &self->hash, &s.sel, values.data_ptr(), nullptr, nullptr, nullptr,
                           c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)self->device).stream()),
               "dok_dok_get"))
      return nullptr;
    for (int k = s.n_scalars - 1; k >= 0; k--) {
      const int i = s.scalars[k];
      if (i < values.dim() && values.size(i) == 1) values = values.squeeze(i);
    }
    return THPVariable_Wrap(std::move(values));
  });
}

// assign(selectors, size, values, room, marks) -> the number of positions, or None; its negative, and nothing done, when it
// is more than `room`, so that the table might have to grow
PyObject *plan_assign(Plan *self, PyObject *const *args, Py_ssize_t nargs) {
  return guarded([&]() -> PyObject * {
    Marks *marks = nargs == 5 ? marks_of(args[4]) : nullptr;
    if (!marks) { PyErr_SetString(PyExc_TypeError, "assign takes selectors, size, values, room and Marks"); return nullptr; }
    int64_t size[DOK_MAX_KEY_SIZE];
    const int ndim = shape_from(args[1], size, DOK_MAX_KEY_SIZE);
    const at::Tensor *given = tensor_of(args[2]);
    const bool number = PyFloat_CheckExact(args[2]) ? at::isFloatingType(self->value_type)
                                                    : PyLong_CheckExact(args[2]) && (at::isFloatingType(self->value_type) || self->value_type == at::kLong);
    if (ndim < 1 || ndim > DOK_MAX_KEY_SIZE || ndim != self->hash.key_size || self->value_ndim != 1 || self->value_shape[0] != 1 ||
        (given ? given->layout() != at::kStrided || !given->is_cuda() || given->get_device() != self->device ||
                     given->scalar_type() != self->value_type
               : !number)) {
      PyErr_Clear();
      Py_RETURN_NONE;
    }
    const double room = PyFloat_AsDouble(args[3]);
    if (PyErr_Occurred()) return nullptr;
    const c10::cuda::CUDAGuard guard((c10::DeviceIndex)self->device);
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)self->device).stream();
    dok_table table = self->table;
    int64_t base, epoch;
    Selection s;
    if (!parse_selection(args[0], size, ndim, self->device, &s)) Py_RETURN_NONE;
    if ((double)s.n > room) return PyLong_FromLongLong(-s.n);
    at::Tensor values;
    if (given) {
      values = given->expand(s.shape);
    } else {
      at::Scalar value;
      if (PyFloat_CheckExact(args[2])) value = PyFloat_AS_DOUBLE(args[2]);
      else {
        const long long v = PyLong_AsLongLong(args[2]);
        if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); Py_RETURN_NONE; }
        value = (int64_t)v;
      }
      values = at::full({}, value, on_device(self, self->value_type)).expand(s.shape);
    }
    if (take_numbers(self, marks, s.n, stream, &base)) {
      if (!check(dok_dok_assign_numbered(&table, &self->hash, &s.sel, values.data_ptr(), values.strides().data(), base, self->state + STATE_SET,
                                         self->state + STATE_ADJUST, stream),
                 "dok_dok_assign_numbered"))
        return nullptr;
    } else if (s.n > 0) {
      if (!take_epoch(marks, &table, &epoch)) Py_RETURN_NONE;
      const int64_t words = dok_set_scratch_words(&table, s.n);
      at::Tensor scratch;
      if (words > 0) scratch = at::empty({words}, on_device(self, at::kLong));
      if (!check(dok_dok_assign(&table, &self->hash, &s.sel, values.data_ptr(), values.strides().data(),
                                words > 0 ? (int64_t *)scratch.data_ptr() : nullptr, words, epoch, self->state + STATE_SET, self->state + STATE_ADJUST, stream),
                 "dok_dok_assign"))
        return nullptr;
    }
    return PyLong_FromLongLong(s.n);
  });
}

PyMethodDef ring_methods[] = {
    {"copy", (PyCFunction)(void *)ring_copy, METH_FASTCALL, nullptr},
    {"landed", (PyCFunction)ring_landed, METH_O, nullptr},
    {"wait", (PyCFunction)ring_wait, METH_O, nullptr},
    {"read", (PyCFunction)ring_read, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyTypeObject ring_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyMemberDef marks_members[] = {{"stamp", T_OBJECT, offsetof(Marks, stamp), 0, nullptr},
                               {"epoch", T_LONGLONG, offsetof(Marks, epoch), 0, nullptr},
                               {"numbered", T_LONGLONG, offsetof(Marks, numbered), 0, nullptr},
                               {"renumbered", T_LONGLONG, offsetof(Marks, renumbered), READONLY, nullptr},
                               {nullptr, 0, 0, 0, nullptr}};

PyTypeObject marks_type = {PyVarObject_HEAD_INIT(nullptr, 0)};

Marks *marks_of(PyObject *o) { return Py_TYPE(o) == &marks_type ? (Marks *)o : nullptr; }

PyMethodDef module_methods[] = {{"allocate", (PyCFunction)plan_allocate, METH_VARARGS, nullptr}, {nullptr, nullptr, 0, nullptr}};

PyMethodDef plan_methods[] = {
    {"set_hash", (PyCFunction)(void *)plan_set_hash, METH_FASTCALL, nullptr},
    {"get", (PyCFunction)plan_get, METH_O, nullptr},
    {"set", (PyCFunction)(void *)plan_set, METH_FASTCALL, nullptr},
    {"remove_rows", (PyCFunction)plan_remove_rows, METH_O, nullptr},
    {"remove", (PyCFunction)plan_remove, METH_O, nullptr},
    {"read", (PyCFunction)plan_read, METH_NOARGS, nullptr},
    {"count_new", (PyCFunction)(void *)plan_count_new, METH_FASTCALL, nullptr},
    {"reinsert", (PyCFunction)plan_reinsert, METH_O, nullptr},
    {"index", (PyCFunction)(void *)plan_index, METH_FASTCALL, nullptr},
    {"assign", (PyCFunction)(void *)plan_assign, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyTypeObject plan_type = {  // filled in below
    PyVarObject_HEAD_INIT(nullptr, 0)};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, module_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) {
  plan_type.tp_name = "doksparse_b200._native.Plan";
  plan_type.tp_basicsize = sizeof(Plan);
  plan_type.tp_flags = Py_TPFLAGS_DEFAULT;
  plan_type.tp_new = PyType_GenericNew;
  plan_type.tp_init = (initproc)plan_init;
  plan_type.tp_methods = plan_methods;
  ring_type.tp_name = "doksparse_b200._native.Ring";
  ring_type.tp_basicsize = sizeof(Ring);
  ring_type.tp_flags = Py_TPFLAGS_DEFAULT;
  ring_type.tp_new = PyType_GenericNew;
  ring_type.tp_init = (initproc)ring_init;
  ring_type.tp_dealloc = (destructor)ring_dealloc;
  ring_type.tp_methods = ring_methods;
  marks_type.tp_name = "doksparse_b200._native.Marks";
  marks_type.tp_basicsize = sizeof(Marks);
  marks_type.tp_flags = Py_TPFLAGS_DEFAULT;
  marks_type.tp_new = PyType_GenericNew;
  marks_type.tp_init = (initproc)marks_init;
  marks_type.tp_dealloc = (destructor)marks_dealloc;
  marks_type.tp_members = marks_members;
  if (PyType_Ready(&plan_type) < 0 || PyType_Ready(&ring_type) < 0 || PyType_Ready(&marks_type) < 0) return nullptr;
  PyObject *lib = PyImport_ImportModule("doksparse_b200._lib");
  if (!lib) return nullptr;
  dok_error = PyObject_GetAttrString(lib, "DokError");
  Py_DECREF(lib);
  PyObject *m = dok_error ? PyModule_Create(&module) : nullptr;
  if (m && (PyModule_AddObjectRef(m, "Plan", (PyObject *)&plan_type) < 0 || PyModule_AddObjectRef(m, "Ring", (PyObject *)&ring_type) < 0 ||
            PyModule_AddObjectRef(m, "Marks", (PyObject *)&marks_type) < 0)) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
