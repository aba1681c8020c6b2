// The ten page tables of build_page_lists as torch tensors over one allocation, and the pools of an encode.
//
// Host time between the read of the table sizes and the next launch is what bounds a short prompt; ten
// allocations, or ten views made from Python, cost 1.3-2 us each, and as much the three of an encode.  Everything
// that computes is in libsphkv_b200.so behind the C ABI; this module only makes tensors.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

namespace {

constexpr int kTables = 10;
constexpr int64_t kAlign = 64;  // i32 values: every table starts on a 256-byte boundary

// make(pointers, device index or -1, P, N, U, max_blocks, n_bundles): a tuple of the tables in the order of
// PageListsParams; their addresses go to the ten consecutive pointers at `pointers`.
PyObject* make(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 7) {
    PyErr_SetString(PyExc_TypeError, "make: seven integers");
    return nullptr;
  }
  long long v[7];
  for (int i = 0; i < 7; ++i) {
    v[i] = PyLong_AsLongLong(args[i]);
    if (v[i] == -1 && PyErr_Occurred()) return nullptr;
  }
  const int64_t P = v[2], N = v[3], U = v[4], mb = v[5], nb = v[6];
  const int64_t rows[kTables] = {P, P, P, P, P, P, U, U, U, nb};
  const int64_t cols[kTables] = {N, N, 0, 0, 0, 3, mb, mb, 0, 8};  // 0: one dimension
  int64_t at[kTables + 1] = {0};
  for (int i = 0; i < kTables; ++i)
    at[i + 1] = at[i] + (rows[i] * (cols[i] ? cols[i] : 1) + kAlign - 1) / kAlign * kAlign;
  HANDLE_TH_ERRORS
  const at::AutoDispatchBelowADInplaceOrView plain;  // integer tables: nothing for autograd to follow
  const at::Device dev = v[1] < 0 ? at::Device(at::kCPU) : at::Device(at::kCUDA, (c10::DeviceIndex)v[1]);
  at::Tensor buf;
  {
    const pybind11::gil_scoped_release no_gil;  // an allocation can wait for the device, and other threads go on
    buf = at::empty({at[kTables]}, at::TensorOptions().dtype(at::kInt).device(dev));
  }
  int32_t* base = buf.data_ptr<int32_t>();
  void** out = reinterpret_cast<void**>(static_cast<intptr_t>(v[0]));
  PyObject* tables = PyTuple_New(kTables);
  if (tables == nullptr) return nullptr;
  for (int i = 0; i < kTables; ++i) {
    out[i] = base + at[i];
    PyObject* t = THPVariable_Wrap(cols[i] ? buf.as_strided({rows[i], cols[i]}, {cols[i], 1}, at[i])
                                           : buf.as_strided({rows[i]}, {1}, at[i]));
    if (t == nullptr) {
      Py_DECREF(tables);
      return nullptr;
    }
    PyTuple_SET_ITEM(tables, i, t);
  }
  return tables;
  END_HANDLE_TH_ERRORS
}

// pools(device index or -1, pool_bytes, P, N, dh, V pool is bf16 (else f16), V pool is zeroed, scratch_bytes): the zeroed
// byte pool, the V pool [P, N, dh], bytes of scratch (None for no bytes), and the three addresses.
PyObject* pools(PyObject*, PyObject* const* args, Py_ssize_t n) {
  if (n != 8) {
    PyErr_SetString(PyExc_TypeError, "pools: eight integers");
    return nullptr;
  }
  long long v[8];
  for (int i = 0; i < 8; ++i) {
    v[i] = PyLong_AsLongLong(args[i]);
    if (v[i] == -1 && PyErr_Occurred()) return nullptr;
  }
  HANDLE_TH_ERRORS
  const at::AutoDispatchBelowADInplaceOrView plain;  // made here, nothing for autograd to follow
  const at::Device dev = v[0] < 0 ? at::Device(at::kCPU) : at::Device(at::kCUDA, (c10::DeviceIndex)v[0]);
  const at::TensorOptions bytes = at::TensorOptions().dtype(at::kByte).device(dev);
  const at::TensorOptions vo = bytes.dtype(v[5] ? at::kBFloat16 : at::kHalf);
  at::Tensor k_pages, v_pool, scratch;
  {
    const pybind11::gil_scoped_release no_gil;  // as in make(); the zeroing is a launch, which waits where the queue is full
    k_pages = at::zeros({v[1]}, bytes);
    v_pool = v[6] ? at::zeros({v[2], v[3], v[4]}, vo) : at::empty({v[2], v[3], v[4]}, vo);
    if (v[7] > 0) scratch = at::empty({v[7]}, bytes);
  }
  auto address = [](const at::Tensor& t) { return (unsigned long long)reinterpret_cast<uintptr_t>(t.defined() ? t.data_ptr() : nullptr); };
  PyObject* k = THPVariable_Wrap(k_pages);
  PyObject* vp = THPVariable_Wrap(v_pool);
  PyObject* s = scratch.defined() ? THPVariable_Wrap(scratch) : Py_NewRef(Py_None);
  if (k == nullptr || vp == nullptr || s == nullptr) {
    Py_XDECREF(k);
    Py_XDECREF(vp);
    Py_XDECREF(s);
    return nullptr;
  }
  return Py_BuildValue("(NNNKKK)", k, vp, s, address(k_pages), address(v_pool), address(scratch));
  END_HANDLE_TH_ERRORS
}

PyMethodDef kMethods[] = {
    {"pools", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(pools)), METH_FASTCALL, nullptr},
    {"make", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(make)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "host_tables", nullptr, -1, kMethods};

}  // namespace

PyMODINIT_FUNC PyInit_host_tables() { return PyModule_Create(&kModule); }
