// quantized_matmul of a few rows, from Python objects to the launch in one native call. The Python form of the same steps
// (ops.py) took 9 of the 14 us that a one-row product costs the host: attribute lookups, shape tuples, a ctypes call of
// sixteen arguments. It stays for every other form: this one answers None to whatever it does not know - subclasses of
// Tensor, tensors without storage of their own (vmap, tracing), CPU tensors, another device than the current one, operands
// that want a copy, more than sixteen rows, and all that is refused with a message.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/kquant_b200.h"

namespace {

// entry points of the library, handed over by address: this module links to torch alone
decltype(&kq_codec_find) codec_find;
decltype(&kq_codec_info) codec_info;
decltype(&kq_quantized_matmul_workspace_bytes) workspace_bytes;
decltype(&kq_quantized_matmul) matmul;

PyObject* init(PyObject*, PyObject* args) {
  unsigned long long p[4];
  if (!PyArg_ParseTuple(args, "KKKK", &p[0], &p[1], &p[2], &p[3])) return nullptr;
  codec_find = reinterpret_cast<decltype(codec_find)>(p[0]);
  codec_info = reinterpret_cast<decltype(codec_info)>(p[1]);
  workspace_bytes = reinterpret_cast<decltype(workspace_bytes)>(p[2]);
  matmul = reinterpret_cast<decltype(matmul)>(p[3]);
  Py_RETURN_NONE;
}

bool plain(const at::Tensor& t) {  // a dense CUDA tensor and nothing around it
  return t.layout() == at::kStrided && t.is_cuda() && t.has_storage() && !t.is_conj() && !t.is_neg() &&
         !t.key_set().has_any(c10::DispatchKeySet({c10::DispatchKey::Python, c10::DispatchKey::FuncTorchBatched,
                                                   c10::DispatchKey::FuncTorchGradWrapper, c10::DispatchKey::Functionalize}));
}

// qmm(x, w, kquant_type, transpose) -> the product, an error code of the library, or None: not for this path
PyObject* qmm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 4 || matmul == nullptr || !THPVariable_CheckExact(args[0]) || !THPVariable_CheckExact(args[1]) ||
      !PyUnicode_Check(args[2]) || args[3] != Py_True)
    Py_RETURN_NONE;
  const at::Tensor& x = THPVariable_Unpack(args[0]);
  const at::Tensor& w = THPVariable_Unpack(args[1]);
  if (!plain(x) || !plain(w) || w.scalar_type() != at::kByte || w.dim() != 2 || !w.is_contiguous() || x.dim() < 1 ||
      x.numel() == 0 || x.device() != w.device() || x.device().index() != c10::cuda::current_device())
    Py_RETURN_NONE;
  int type;
  at::ScalarType out = x.scalar_type();
  switch (out) {
    case at::kFloat: type = KQ_F32, out = at::kBFloat16; break;
    case at::kHalf: type = KQ_F16; break;
    case at::kBFloat16: type = KQ_BF16; break;
    default: Py_RETURN_NONE;
  }
  const char* codec = PyUnicode_AsUTF8(args[2]);
  if (codec == nullptr) return nullptr;
  const int index = codec_find(codec);
  int wpb = 0, bpb = 0;
  if (index < 0 || codec_info(index, nullptr, &wpb, &bpb, nullptr, nullptr) != 0) Py_RETURN_NONE;
  const int64_t K = x.size(-1), rows = x.numel() / K, N = w.size(0), row_bytes = w.size(1);
  if (rows > 16 || N <= 0 || N > INT32_MAX || K > INT32_MAX || row_bytes % bpb != 0 || row_bytes / bpb * wpb != K)
    Py_RETURN_NONE;
  int64_t stride = K;
  if (x.dim() == 2) {
    if (x.stride(1) != 1) Py_RETURN_NONE;
    stride = x.stride(0);
  } else if (!x.is_contiguous()) {
    Py_RETURN_NONE;
  }
  if (stride < 0 || stride * (int64_t)x.element_size() % 16 != 0 || reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 != 0)
    Py_RETURN_NONE;
  at::Tensor y = at::empty({rows, N}, x.options().dtype(out).requires_grad(false)), ws;
  const size_t need = rows > 1 ? workspace_bytes(type, rows, K) : 0;
  if (need != 0) ws = at::empty({(int64_t)need}, w.options().requires_grad(false));
  if (!plain(y) || (need != 0 && !plain(ws))) Py_RETURN_NONE;  // (under a dispatch mode)
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = matmul(x.data_ptr(), type, rows, K, stride, w.data_ptr(), row_bytes, N, codec, 1, y.data_ptr(), N,
              need != 0 ? ws.data_ptr() : nullptr, need, stream);
  Py_END_ALLOW_THREADS
  if (rc != 0) return PyLong_FromLong(rc);
  if (x.dim() != 2) {
    std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = N;
    y = y.view(shape);
  }
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {{"init", init, METH_VARARGS, nullptr},
                         {"qmm", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(qmm)), METH_FASTCALL, nullptr},
                         {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_kq_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// torch_version: of the torch that this was compiled against, whose classes it takes apart; _lib.py uses it with no other
PyMODINIT_FUNC PyInit__kq_torch() {
  PyObject* m = PyModule_Create(&module);
  if (m != nullptr && PyModule_AddStringConstant(m, "torch_version", KQ_TORCH_VERSION) != 0) Py_CLEAR(m);
  return m;
}
