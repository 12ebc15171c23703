// The host path of `flash_kda.fwd`: argument checks, scratch memory and the launch in one native call.
//
// A decode step costs a few microseconds on the GPU; the checks written in Python (some ninety attribute reads), a
// torch.empty, a ctypes structure and a device guard cost 20 of the 26 us that such a call took.  The same conditions are
// read here from the tensor objects directly.  This file only decides "everything is in order" and then calls the C ABI
// (include/fkda.h); whenever anything is not, it reports that and the caller walks the Python checks, which own the order
// and the wording of the errors (the reference's TORCH_CHECKs, csrc/flash_kda.cpp:44-174).
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/fkda.h"

namespace {

// A plain tensor (no subclass with behaviour of its own) on the GPU, contiguous; nullptr otherwise.
const at::Tensor* cuda_tensor(PyObject* o, at::ScalarType type) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.scalar_type() == type && t.is_contiguous() && t.has_storage() ? &t : nullptr;
}

// fwd_fast(q, k, v, g, beta, scale, out, A_log, dt_bias, lower_bound, initial_state, final_state, cu_seqlens)
// -> True: launched; False: not an ordinary call, nothing was done; str: the library's error message.
PyObject* fwd_fast(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 13) Py_RETURN_FALSE;
  const at::Tensor* main[6];
  const int at_main[6] = {0, 1, 2, 3, 4, 6};      // q k v g beta out
  for (int i = 0; i < 6; ++i)
    if ((main[i] = cuda_tensor(a[at_main[i]], at::kBFloat16)) == nullptr) Py_RETURN_FALSE;
  const at::Tensor *A_log = cuda_tensor(a[7], at::kFloat), *dt_bias = cuda_tensor(a[8], at::kFloat);
  if (A_log == nullptr || dt_bias == nullptr) Py_RETURN_FALSE;
  const at::Tensor& q = *main[0];
  if (q.dim() != 4) Py_RETURN_FALSE;
  const int64_t B = q.size(0), T = q.size(1), H = q.size(2), D = q.size(3);
  for (int i : {1, 2, 3, 5})
    if (main[i]->sizes() != q.sizes()) Py_RETURN_FALSE;
  const at::Tensor& beta = *main[4];
  if (D != 128 || beta.dim() != 3 || beta.size(0) != B || beta.size(1) != T || beta.size(2) != H) Py_RETURN_FALSE;
  if (A_log->dim() != 1 || A_log->size(0) != H || dt_bias->dim() != 2 || dt_bias->size(0) != H || dt_bias->size(1) != D) Py_RETURN_FALSE;
  const c10::Device dev = q.device();
  for (const at::Tensor* t : {main[1], main[2], main[3], main[4], main[5], A_log, dt_bias})
    if (t->device() != dev) Py_RETURN_FALSE;
  int64_t N = B;
  const at::Tensor* cu = nullptr;
  if (a[12] != Py_None) {
    if ((cu = cuda_tensor(a[12], at::kLong)) == nullptr || B != 1 || cu->dim() != 1 || cu->numel() < 2 || cu->device() != dev) Py_RETURN_FALSE;
    N = cu->numel() - 1;
  }
  const at::Tensor* state[2] = {nullptr, nullptr};
  int state_dtype = FKDA_STATE_NONE;
  for (int i = 0; i < 2; ++i) {
    if (a[10 + i] == Py_None) continue;
    const at::Tensor* s = cuda_tensor(a[10 + i], at::kFloat);
    const int type = s != nullptr ? FKDA_STATE_FP32 : FKDA_STATE_BF16;
    if (s == nullptr && (s = cuda_tensor(a[10 + i], at::kBFloat16)) == nullptr) Py_RETURN_FALSE;
    if (state_dtype != FKDA_STATE_NONE && state_dtype != type) Py_RETURN_FALSE;
    if (s->dim() != 4 || s->size(0) != N || s->size(1) != H || s->size(2) != D || s->size(3) != D || s->device() != dev) Py_RETURN_FALSE;
    state[i] = s;
    state_dtype = type;
  }
  if (!PyFloat_CheckExact(a[5]) || !PyFloat_CheckExact(a[9])) Py_RETURN_FALSE;

  fkda_fwd_params p{};
  p.q = q.data_ptr();
  p.k = main[1]->data_ptr();
  p.v = main[2]->data_ptr();
  p.g = main[3]->data_ptr();
  p.beta = beta.data_ptr();
  p.out = main[5]->data_ptr();
  p.A_log = static_cast<const float*>(A_log->data_ptr());
  p.dt_bias = static_cast<const float*>(dt_bias->data_ptr());
  p.initial_state = state[0] != nullptr ? state[0]->data_ptr() : nullptr;
  p.final_state = state[1] != nullptr ? state[1]->data_ptr() : nullptr;
  p.cu_seqlens = cu != nullptr ? static_cast<const int64_t*>(cu->data_ptr()) : nullptr;
  p.B = B;
  p.T = T;
  p.H = H;
  p.N = N;
  p.scale = static_cast<float>(PyFloat_AS_DOUBLE(a[5]));
  p.lower_bound = static_cast<float>(PyFloat_AS_DOUBLE(a[9]));
  p.state_dtype = state_dtype;
  p.flags = FKDA_FLAG_STATUS_UNREAD;      // the scratch memory is not the caller's: nobody can read its status word

  char message[512];
  bool failed = false;
  try {
    c10::cuda::CUDAGuard guard(dev);
    int64_t bytes = 0;
    if (fkda_fwd_scratch_bytes(&p, &bytes) != FKDA_OK) Py_RETURN_FALSE;
    // freed when the call returns: the caching allocator hands a block only to later work of the same stream
    // (none for a decode step, where asking for it would be a tenth of the call)
    c10::DataPtr ws;
    if (bytes > 0) ws = c10::cuda::CUDACachingAllocator::get()->allocate(static_cast<size_t>(bytes));
    p.workspace = ws.get();
    p.workspace_bytes = bytes;
    void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    int rc;
    Py_BEGIN_ALLOW_THREADS
    rc = fkda_fwd(&p, stream);
    Py_END_ALLOW_THREADS
    if (rc != FKDA_OK) {
      snprintf(message, sizeof(message), "flash_kda: %s (code %d)", fkda_last_error(), rc);
      failed = true;
    }
  } catch (const c10::OutOfMemoryError&) {
    Py_RETURN_FALSE;                       // the Python path meets the same and raises torch's own exception
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
  if (failed) return PyUnicode_FromString(message);
  Py_RETURN_TRUE;
}

PyMethodDef methods[] = {
    {"fwd_fast", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fwd_fast)), METH_FASTCALL,
     "checks an ordinary flash_kda.fwd call and launches it"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_fkda_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__fkda_host(void) {
  PyObject* m = PyModule_Create(&module);
  // the torch whose headers this was compiled against: another one may lay out a tensor differently (checked by the loader)
  if (m != nullptr && PyModule_AddStringConstant(m, "torch_version", FKDA_TORCH_VERSION) != 0) Py_CLEAR(m);
  return m;
}
