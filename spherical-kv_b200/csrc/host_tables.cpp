// The ten page tables of build_page_lists as torch tensors over one allocation.
//
// Host time between the read of the table sizes and the next launch is what bounds a short prompt; ten
// allocations, or ten views made from Python, cost 1.3-2 us each.  Everything that computes is in
// libsphkv_b200.so behind the C ABI; this module only makes tensors.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

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
  const at::Tensor buf = at::empty({at[kTables]}, at::TensorOptions().dtype(at::kInt).device(dev));
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

PyMethodDef kMethods[] = {
    {"make", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(make)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "host_tables", nullptr, -1, kMethods};

}  // namespace

PyMODINIT_FUNC PyInit_host_tables() { return PyModule_Create(&kModule); }
