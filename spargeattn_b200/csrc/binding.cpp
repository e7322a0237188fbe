// Python binding of the whole path: one function, no interpreter work between a model's call and the launches.
//
//   forward(q, k, v, mask, simthreshd1, cdfthreshd, topk, pvthreshd, scale, is_causal, kernel_causal, attention_sink,
//           smooth_k, pv_fp16, tensor_layout, q_block_ranges, q_blocks_max, want_valid)
//
// returns the output (with want_valid: (output, live-block counts [B,H,nq])), or None for arguments that it leaves to the
// Python front end: tensors that need a conversion or a complaint, knobs that are neither a number nor a ready [H] fp32
// tensor on the device. Output and workspace come from PyTorch's caching allocator on the current stream, so they are
// ordered, shared between streams and given back like any other tensor; nothing else outlives a call but the per-head
// copies of scalar knobs (at most 256 of them) and one status word per device.
//
// Cost on the host, a [1,4,2048,64] call: the ctypes wrappers spent about 20 us in the interpreter before the launches.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAFunctions.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>

#include "forward.cuh"

namespace {

using at::Tensor;

// Scalar knobs as [H] tensors, materialised once per (value, H, device) for every caller, Python's general path included:
// a value that one entry has seen can be captured into a graph by another. Built on the host and copied with a blocking
// transfer, so that a cached tensor is complete before any stream can read it.
Tensor knob_tensor(double value, int64_t H, c10::Device dev) {
  static std::mutex mu;
  static auto* cache = new std::map<std::tuple<double, int64_t, int>, Tensor>();   // never destroyed: CUDA may be gone at exit
  const auto key = std::make_tuple(value, H, (int)dev.index());
  const bool cacheable = !std::isnan(value);                 // NaN has no place in an ordered map
  if (cacheable) {
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache->find(key);
    if (it != cache->end()) return it->second;
  }
  Tensor t = at::full({H}, value, at::TensorOptions().dtype(at::kFloat)).to(dev);   // may run Python: not under the lock
  std::lock_guard<std::mutex> lock(mu);
  if (!cacheable || cache->size() >= 256) return t;
  return cache->emplace(key, t).first->second;
}

// A knob argument: None -> null, number or ready tensor -> pointer; false: not one of these.
bool knob(PyObject* o, int64_t H, c10::Device dev, const float** out, Tensor& keep) {
  *out = nullptr;
  if (o == Py_None) return true;
  if (PyFloat_CheckExact(o) || PyLong_CheckExact(o)) {
    const double v = PyFloat_CheckExact(o) ? PyFloat_AS_DOUBLE(o) : PyLong_AsDouble(o);
    if (PyErr_Occurred() || std::isnan(v)) {
      PyErr_Clear();
      return false;
    }
    keep = knob_tensor(v, H, dev);
    *out = keep.data_ptr<float>();
    return true;
  }
  if (!THPVariable_Check(o)) return false;
  const Tensor& t = THPVariable_Unpack(o);
  if (t.dim() != 1 || t.numel() != H || t.scalar_type() != at::kFloat || t.device() != dev || !t.is_contiguous()) return false;
  *out = t.data_ptr<float>();
  return true;
}

int dtype_code(const Tensor& t) {
  return t.scalar_type() == at::kHalf ? SPARGE_F16 : t.scalar_type() == at::kBFloat16 ? SPARGE_BF16 : -1;
}

// [B,H,N,D] strides (batch, head, token) of a tensor in the given layout; false if it cannot be read in place.
bool view_strides(const Tensor& t, bool nhd, long long* st) {
  const auto s = t.strides();
  st[0] = s[0], st[1] = s[nhd ? 2 : 1], st[2] = s[nhd ? 1 : 2];
  return s[3] == 1 && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0 && st[0] >= 0 && st[1] >= 0 && st[2] > 0 &&
         st[0] % 8 == 0 && st[1] % 8 == 0 && st[2] % 8 == 0;
}

Tensor* status_words[64];   // kept for the life of the process: kernels write to them

PyObject* py_knob_tensor(PyObject*, PyObject* const* args, Py_ssize_t nargs) {   // (value, H, device index) -> [H] fp32
  HANDLE_TH_ERRORS
  if (nargs != 3) {
    PyErr_SetString(PyExc_TypeError, "knob_tensor takes 3 arguments");
    return nullptr;
  }
  const double value = PyFloat_AsDouble(args[0]);
  const long H = PyLong_AsLong(args[1]), index = PyLong_AsLong(args[2]);
  if (PyErr_Occurred()) return nullptr;
  return THPVariable_Wrap(knob_tensor(value, H, c10::Device(c10::kCUDA, (c10::DeviceIndex)index)));
  END_HANDLE_TH_ERRORS
}

PyObject* set_status_word(PyObject*, PyObject* o) {   // the int32 word of its device that expired waits are written to
  if (!THPVariable_Check(o) || THPVariable_Unpack(o).get_device() < 0 || THPVariable_Unpack(o).get_device() >= 64) {
    PyErr_SetString(PyExc_ValueError, "expected a CUDA tensor");
    return nullptr;
  }
  status_words[THPVariable_Unpack(o).get_device()] = new Tensor(THPVariable_Unpack(o));
  Py_RETURN_NONE;
}

const char* kErrors[] = {"ok", "invalid argument", "a required pointer is NULL", "a CUDA call failed",
                         "a size exceeds what the kernel supports", "not implemented in this build"};

PyObject* forward(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 18) {
    PyErr_SetString(PyExc_TypeError, "forward takes 18 arguments");
    return nullptr;
  }
  for (int i = 0; i < 3; i++)
    if (!THPVariable_Check(args[i])) Py_RETURN_NONE;
  const Tensor &q = THPVariable_Unpack(args[0]), &k = THPVariable_Unpack(args[1]), &v = THPVariable_Unpack(args[2]);
  const c10::Device dev = q.device();
  if (!q.is_cuda() || k.device() != dev || v.device() != dev || q.dim() != 4 || k.sizes() != q.sizes() || v.sizes() != q.sizes())
    Py_RETURN_NONE;
  if (!PyUnicode_Check(args[14])) Py_RETURN_NONE;
  const bool nhd = PyUnicode_CompareWithASCIIString(args[14], "NHD") == 0;
  if (!nhd && PyUnicode_CompareWithASCIIString(args[14], "HND") != 0) Py_RETURN_NONE;

  sparge::ForwardArgs a = {};
  const int64_t B = q.size(0), H = q.size(nhd ? 2 : 1), N = q.size(nhd ? 1 : 2), D = q.size(3);
  a.dtype = dtype_code(q), a.v_dtype = dtype_code(v);
  if (a.dtype < 0 || a.v_dtype < 0 || dtype_code(k) != a.dtype || (D != 64 && D != 128) || N < 128 || B < 1 || H < 1 ||
      B * H > 65535 || N > (1 << 30))
    Py_RETURN_NONE;
  if (!view_strides(q, nhd, a.q_st) || !view_strides(k, nhd, a.k_st) || !view_strides(v, nhd, a.v_st)) Py_RETURN_NONE;
  if (dev.index() >= 64 || !status_words[dev.index()]) Py_RETURN_NONE;
  a.B = (int)B, a.H = (int)H, a.N = (int)N, a.D = (int)D;
  a.pv_fp16 = PyObject_IsTrue(args[13]);

  Tensor keep[4];
  const float* pv = nullptr;
  // from this scalar threshold on the skip test cannot change the output: see core.PV_SKIP_NEVER_FIRES_FROM
  const bool pv_off = (PyFloat_CheckExact(args[7]) && PyFloat_AS_DOUBLE(args[7]) >= 30.0) ||
                      (PyLong_CheckExact(args[7]) && PyLong_AsDouble(args[7]) >= 30.0);
  if (args[7] == Py_None || (!pv_off && !knob(args[7], H, dev, &pv, keep[0]))) Py_RETURN_NONE;
  a.pvthr = pv;
  if (args[3] != Py_None) {   // block mask
    if (!THPVariable_Check(args[3])) Py_RETURN_NONE;
    const Tensor& m = THPVariable_Unpack(args[3]);
    if (m.dim() != 4 || m.size(0) != B || m.size(1) != H || m.size(2) != (N + 127) / 128 || m.size(3) != (N + 63) / 64 ||
        m.device() != dev || !m.is_contiguous() || m.is_floating_point() || m.is_complex())
      Py_RETURN_NONE;
    a.mask = m.data_ptr();
    a.mask_elem_size = (int)m.element_size();
  } else {
    if (!knob(args[4], H, dev, &a.simthr, keep[1]) || !knob(args[5], H, dev, &a.cdf, keep[2]) ||
        !knob(args[6], H, dev, &a.topk, keep[3]) || !a.simthr || (a.cdf == nullptr) == (a.topk == nullptr))
      Py_RETURN_NONE;
  }
  if (args[8] == Py_None) a.sm_scale = D == 64 ? 0.125f : (float)(1.0 / std::sqrt(128.0));
  else if (PyFloat_Check(args[8]) || PyLong_Check(args[8])) a.sm_scale = (float)PyFloat_AsDouble(args[8]);
  else Py_RETURN_NONE;
  a.is_causal = PyObject_IsTrue(args[9]), a.kernel_causal = PyObject_IsTrue(args[10]);
  a.sink = PyObject_IsTrue(args[11]), a.smooth_k = PyObject_IsTrue(args[12]);
  if (PyErr_Occurred()) return nullptr;
  if (args[15] != Py_None) {
    if (!THPVariable_Check(args[15])) Py_RETURN_NONE;
    const Tensor& r = THPVariable_Unpack(args[15]);
    if (r.scalar_type() != at::kInt || r.numel() != 2 * B * H || !r.is_contiguous() || r.device() != dev) Py_RETURN_NONE;
    a.q_ranges = r.data_ptr<int32_t>();
    a.q_blocks_max = (int)PyLong_AsLong(args[16]);
    if (PyErr_Occurred()) return nullptr;
    if (a.q_blocks_max <= 0) Py_RETURN_NONE;
  }

  c10::cuda::set_device(dev.index());
  const auto opts = q.options();
  // output in q's memory format
  const bool out_nhd = a.q_st[1] == D && a.q_st[2] == H * D && a.q_st[0] == N * H * D;
  Tensor out = at::empty(out_nhd ? at::IntArrayRef{B, N, H, D} : at::IntArrayRef{B, H, N, D}, opts);
  if (out_nhd) a.o_st[0] = N * H * D, a.o_st[1] = D, a.o_st[2] = H * D;
  else a.o_st[0] = H * N * D, a.o_st[1] = N * D, a.o_st[2] = D;
  const bool copies = sparge::forward_copies_v(a.pv_fp16, a.v_dtype, a.v_st);
  size_t off[sparge::kWsCount];
  a.workspace_bytes = sparge::forward_layout(a.B, a.H, a.N, a.D, copies ? 2 : a.pv_fp16 ? 0 : 1, off);
  Tensor ws = at::empty({(int64_t)a.workspace_bytes}, opts.dtype(at::kByte));
  a.q = q.data_ptr(), a.k = k.data_ptr(), a.v = v.data_ptr(), a.o = out.data_ptr(), a.workspace = ws.data_ptr();
  a.dev_status = status_words[dev.index()]->data_ptr<int32_t>();
  const cudaStream_t st = at::cuda::getCurrentCUDAStream(dev.index()).stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = sparge::forward(a, st);
  Py_END_ALLOW_THREADS
  if (rc != SPARGE_OK) {
    PyErr_Format(rc == SPARGE_ERR_INVALID_ARG || rc == SPARGE_ERR_TOO_LARGE ? PyExc_ValueError : PyExc_RuntimeError,
                 "sparge forward: %s (status %d)", rc > 0 && rc < 6 ? kErrors[rc] : "unknown status", rc);
    return nullptr;
  }
  if (out_nhd != nhd) out = out.transpose(1, 2);
  if (!PyObject_IsTrue(args[17])) return THPVariable_Wrap(std::move(out));
  const int64_t nq = (N + 127) / 128;
  Tensor valid = ws.narrow(0, (int64_t)off[sparge::kWsValid], B * H * nq * 4).view(at::kInt).view({B, H, nq});
  PyObject *po = THPVariable_Wrap(std::move(out)), *pvld = THPVariable_Wrap(std::move(valid));
  PyObject* r = PyTuple_Pack(2, po, pvld);
  Py_XDECREF(po);
  Py_XDECREF(pvld);
  return r;
  END_HANDLE_TH_ERRORS
}

PyMethodDef kMethods[] = {
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(forward)), METH_FASTCALL,
     "The whole path in one call; None for arguments that are left to the caller."},
    {"knob_tensor", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_knob_tensor)), METH_FASTCALL,
     "A scalar knob as an [H] tensor on a CUDA device, materialised once."},
    {"set_status_word", set_status_word, METH_O, "Registers the device status word of a CUDA device."},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_binding", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__binding() { return PyModule_Create(&kModule); }
