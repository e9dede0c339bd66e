// The calls of a quantized linear layer (quantization/fp8_kernel.py act_quant, fp8_gemm; quantization/w4a8_kernel.py act_quant,
// w4a8_gemm) from Python to the library in one step: checks, outputs, scratch and launches.
//
// A decode step's linear layer is two or three kernels of 2 to 12 us; asked for from Python, each call spent 9 to 15 us of
// interpreter time on attribute look-ups, allocator calls and argument conversion, and the GPU waited for it (fp8 layer of 16 x 7168 x
// 7168: 26.7 -> 18.0 us, 15 us of which are kernels).
//
// Every function returns None for operands that are not what the launches take as they are (other types, shapes, strides or
// devices, tensor subclasses, CPU tensors); the Python functions then go through their own checks and messages.  A non-zero
// status of the library is returned as a number and raised by the caller.
//
// The interpreter is released around allocations and launches: an allocation can wait for the device, a launch for room in the
// launch queue, and other threads, also those that the queued work itself waits for, go on meanwhile.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/DynamicTypes.h>
#include <torch/csrc/Dtype.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>

#include <algorithm>
#include <vector>

#include "../../include/b200moe.h"

namespace {

// The operand as a tensor that a launch can take: a plain contiguous tensor on the current device; undefined otherwise.  A
// reference of the call's own, since other threads run meanwhile.
at::Tensor plain(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return {};
  const at::Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.get_device() == c10::cuda::current_device() && t.layout() == at::kStrided && t.is_contiguous() &&
                 !t.is_neg() && t.dim() > 0
             ? t : at::Tensor();
}

class ReleasedInterpreter {
 public:
  ReleasedInterpreter() : state_(PyEval_SaveThread()) {}
  ~ReleasedInterpreter() { PyEval_RestoreThread(state_); }
  ReleasedInterpreter(const ReleasedInterpreter&) = delete;

 private:
  PyThreadState* state_;
};

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return B200MOE_F32;
    case at::kHalf: return B200MOE_F16;
    case at::kBFloat16: return B200MOE_BF16;
    default: return -1;
  }
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

std::vector<int64_t> with_last(const at::Tensor& t, int64_t last) {
  std::vector<int64_t> s(t.sizes().begin(), t.sizes().end());
  s.back() = last;
  return s;
}

PyObject* none() { Py_RETURN_NONE; }

// A Python integer that fits the library's int.
bool to_int(PyObject* o, int* out) {
  const long v = PyLong_AsLong(o);
  if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); return false; }
  *out = static_cast<int>(v);
  return *out == v;
}

// act_quant(x, kind): kind 0 fp8, 1 int8 with f16 scales and floor(v + 0.5)
PyObject* act_quant(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 2) return none();
  const at::Tensor x = plain(args[0]);
  int kind;
  if (!to_int(args[1], &kind) || !x.defined() || dtype_code(x.scalar_type()) < 0) return none();
  const int64_t cols = x.size(-1);
  if (cols == 0 || cols % 128 != 0) return none();
  const int64_t rows = x.numel() / cols;
  at::Tensor y, s;
  int rc;
  {
    ReleasedInterpreter released;
    y = at::empty(x.sizes(), x.options().dtype(kind == 0 ? at::kFloat8_e4m3fn : at::kChar));
    s = at::empty(with_last(x, cols / 128), x.options().dtype(kind == 0 ? at::kFloat : at::kHalf));
    rc = kind == 0 ? b200moe_act_quant_fp8(x.data_ptr(), dtype_code(x.scalar_type()), rows, cols, y.data_ptr(), cols,
                                           static_cast<float*>(s.data_ptr()), cols / 128, stream())
                   : b200moe_act_quant_int8(x.data_ptr(), dtype_code(x.scalar_type()), rows, cols, y.data_ptr(), s.data_ptr(), 1, stream());
  }
  if (rc) return PyLong_FromLong(rc);
  PyObject* out = PyTuple_New(2);
  PyTuple_SET_ITEM(out, 0, THPVariable_Wrap(std::move(y)));
  PyTuple_SET_ITEM(out, 1, THPVariable_Wrap(std::move(s)));
  return out;
  END_HANDLE_TH_ERRORS
}

// fp8_gemm(a, a_s, b, b_s, out_dtype, ksplits)
PyObject* fp8_gemm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 6 || !THPDtype_Check(args[4])) return none();
  const at::Tensor a = plain(args[0]), a_s = plain(args[1]), b = plain(args[2]), b_s = plain(args[3]);
  if (!a.defined() || !a_s.defined() || !b.defined() || !b_s.defined() || a.scalar_type() != at::kFloat8_e4m3fn ||
      b.scalar_type() != at::kFloat8_e4m3fn || a_s.scalar_type() != at::kFloat || b_s.scalar_type() != at::kFloat) return none();
  const at::ScalarType out_t = reinterpret_cast<THPDtype*>(args[4])->scalar_type;
  const int code = dtype_code(out_t);
  const int64_t K = a.size(-1), N = b.size(0);
  if (code < 0 || K == 0 || a.numel() == 0) return none();
  const int64_t M = a.numel() / K;
  int ks;
  if (!to_int(args[5], &ks)) return none();
  at::Tensor c;
  int rc;
  {
    ReleasedInterpreter released;
    c = at::empty(with_last(a, N), a.options().dtype(out_t));
    const auto *as = static_cast<const float*>(a_s.data_ptr()), *bs = static_cast<const float*>(b_s.data_ptr());
    if (ks > 1) {
      // the call's own, as in the Python function
      at::Tensor part = at::empty({M * N * ks}, a_s.options());
      rc = b200moe_gemm_fp8_block_splitk(a.data_ptr(), as, b.data_ptr(), bs, c.data_ptr(), code, M, N, K, ks,
                                         static_cast<float*>(part.data_ptr()), part.numel() * 4, stream());
    } else {
      rc = b200moe_gemm_fp8_block(a.data_ptr(), as, b.data_ptr(), bs, c.data_ptr(), code, M, N, K, stream());
    }
  }
  return rc ? PyLong_FromLong(rc) : THPVariable_Wrap(std::move(c));
  END_HANDLE_TH_ERRORS
}

// w4a8_gemm(a, a_s, b, b_s, s4, z4, out_dtype, ksplits) for operands that agree on M, N and K
PyObject* w4a8_gemm(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 8 || !THPDtype_Check(args[6])) return none();
  at::Tensor t[6];
  for (int i = 0; i < 6; ++i) if (!(t[i] = plain(args[i])).defined()) return none();
  const at::Tensor &a = t[0], &a_s = t[1], &b = t[2], &b_s = t[3], &s4 = t[4], &z4 = t[5];
  auto scales = [](const at::Tensor& s) { return s.scalar_type() == at::kHalf || s.scalar_type() == at::kFloat; };
  if (a.scalar_type() != at::kChar || b.scalar_type() != at::kInt || s4.scalar_type() != at::kChar || z4.scalar_type() != at::kChar ||
      !scales(a_s) || !scales(b_s) || b.dim() != 2) return none();
  const at::ScalarType out_t = reinterpret_cast<THPDtype*>(args[6])->scalar_type;
  const int code = dtype_code(out_t);
  const int64_t K = a.size(-1), N = b.size(0) * 8;
  if (code < 0 || K == 0 || a.numel() == 0 || b.size(1) != K) return none();
  const int64_t M = a.numel() / K;
  if (a_s.numel() * 128 != M * K) return none();
  int ks;
  if (!to_int(args[7], &ks)) return none();
  const int64_t na = a_s.scalar_type() == at::kHalf ? a_s.numel() : 0, nb = b_s.scalar_type() == at::kHalf ? b_s.numel() : 0;
  auto up = [](int64_t v) { return (v + 255) / 256 * 256; };
  const int64_t w8 = up(N * K), fa = up(na * 4), fb = up(nb * 4), part = ks > 1 ? M * N * ks * 4 : 0;
  at::Tensor c;
  int rc;
  {
    ReleasedInterpreter released;
    c = at::empty(with_last(a, N), a.options().dtype(out_t));
    at::Tensor scratch = at::empty({w8 + fa + fb + part}, a.options().dtype(at::kByte));
    char* base = static_cast<char*>(scratch.data_ptr());
    float *pa = reinterpret_cast<float*>(base + w8), *pb = reinterpret_cast<float*>(base + w8 + fa);
    rc = b200moe_w4a8_gemm_operands(b.data_ptr(), static_cast<const int8_t*>(s4.data_ptr()), static_cast<const int8_t*>(z4.data_ptr()),
                                    base, N, K, a_s.data_ptr(), pa, na, b_s.data_ptr(), pb, nb, stream());
    const float* as = na ? pa : static_cast<const float*>(a_s.data_ptr());
    const float* bs = nb ? pb : static_cast<const float*>(b_s.data_ptr());
    if (!rc)
      rc = ks > 1 ? b200moe_gemm_i8_block_splitk(a.data_ptr(), as, base, bs, c.data_ptr(), code, M, N, K, ks,
                                                 reinterpret_cast<float*>(base + w8 + fa + fb), part, stream())
                  : b200moe_gemm_i8_block(a.data_ptr(), as, base, bs, c.data_ptr(), code, M, N, K, stream());
  }
  return rc ? PyLong_FromLong(rc) : THPVariable_Wrap(std::move(c));
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"act_quant", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(act_quant)), METH_FASTCALL, nullptr},
    {"fp8_gemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fp8_gemm)), METH_FASTCALL, nullptr},
    {"w4a8_gemm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(w4a8_gemm)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__calls() {
  PyObject* m = PyModule_Create(&module);
  if (m && PyModule_AddStringConstant(m, "stamp", CALLS_STAMP) < 0) { Py_DECREF(m); return nullptr; }   // looked up by build.py
  return m;
}
