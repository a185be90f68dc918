// Native host path of the layer-level entry points: one call from Python per layer instead of one per op.
//
// At decode sizes a linear layer is 8-50 us of GPU work, and the Python route to it (argument checks, three torch
// allocations, two ctypes calls with ten to nineteen converted arguments each) took 55-60 us, so the host set the rate.
// Here the same steps are compiled: checks on the tensors, one allocation for everything that does not outlive the
// call (codes, scales, split-K scratch) and one for the result, then the C-ABI entry points on the current stream.
//
// Every function answers None when its arguments are not of the plain form it handles (another dtype, a view that needs
// a copy, a bad shape, ...); the caller then takes the Python route, which handles or refuses them.  Nothing is launched
// before all checks have passed.  The temporaries come from torch's caching allocator on the current stream and go back
// to it when the call returns, which is stream-ordered like any tensor that goes out of scope.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>

#include "../../../include/sglb200.h"

namespace {

// A C-ABI call that failed after the checks here: reported like the Python route does.
struct LibraryError {
  int rc;
  const char* what;
};

inline void check_rc(int rc, const char* what) {
  if (rc != 0) throw LibraryError{rc, what};
}

PyObject* raise(const LibraryError& e) {
  PyErr_Format(PyExc_RuntimeError, "%s: %s (%s)", e.what, sglb200_status_string(e.rc), sglb200_last_error_detail());
  return nullptr;
}

// The tensor behind `o`, or NULL where its sizes or its memory cannot simply be asked for (sparse and nested tensors, symbolic
// sizes, tracing subclasses): those are left to the Python route.
inline const at::Tensor* tensor_or_null(PyObject* o) {
  if (!THPVariable_CheckExact(o) && !THPVariable_Check(o)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || t.layout() != at::kStrided || t.is_nested() || t.key_set().has(c10::DispatchKey::Python) ||
      t.unsafeGetTensorImpl()->has_symbolic_sizes_strides())
    return nullptr;
  return &t;
}

inline int64_t up(int64_t x, int64_t a) { return (x + a - 1) / a * a; }

inline bool is16(at::ScalarType t) { return t == at::kBFloat16 || t == at::kHalf; }
inline int code16(at::ScalarType t) { return t == at::kBFloat16 ? SGLB200_BF16 : SGLB200_F16; }

// eps rounded to the input dtype, as the torch-native quantiser clamps; fp16 keeps the fp32 value where it rounds to 0
inline float eps_in_dtype(double eps, at::ScalarType t) {
  if (t == at::kFloat) return (float)eps;
  const float v = t == at::kBFloat16 ? static_cast<float>(c10::BFloat16((float)eps)) : static_cast<float>(c10::Half((float)eps));
  return v == 0.f && eps > 0. ? (float)eps : v;
}

inline at::Tensor empty(at::IntArrayRef sizes, at::ScalarType t, c10::Device dev) {
  return at::Tensor(at::detail::empty_cuda(sizes, t, dev, c10::nullopt));
}

using Function = PyObject*(PyObject* const* args, Py_ssize_t n);

// The C entry of `f`, checks included: what it throws becomes the Python exception that torch or the Python route would raise.
template <Function* f>
PyObject* entry(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    return f(args, n);
  } catch (const LibraryError& e) {
    return raise(e);
  }
  END_HANDLE_TH_ERRORS
}

// ---------------------------------------------------------------------------------------------- quantiser
// quant(x, group_size, eps, fp8_min, fp8_max, column_major, tma_aligned, ue8m0, fuse_silu, masked_m) -> (codes, scales)
PyObject* quant(PyObject* const* args, Py_ssize_t n) {
  if (n != 10) Py_RETURN_NONE;
  const at::Tensor* xp = tensor_or_null(args[0]);
  const at::Tensor* mp = args[9] == Py_None ? nullptr : tensor_or_null(args[9]);
  if (!xp || !PyLong_Check(args[1]) || (args[9] != Py_None && !mp)) Py_RETURN_NONE;
  const at::Tensor& x = *xp;
  const int64_t gs = PyLong_AsLong(args[1]);
  const double eps = PyFloat_AsDouble(args[2]);
  const double lo = PyFloat_AsDouble(args[3]), hi = PyFloat_AsDouble(args[4]);
  if (PyErr_Occurred()) return nullptr;
  const bool col = PyObject_IsTrue(args[5]) == 1, tma = PyObject_IsTrue(args[6]) == 1;
  const bool ue = PyObject_IsTrue(args[7]) == 1, silu = PyObject_IsTrue(args[8]) == 1;
  const int64_t dim = x.dim();
  const at::ScalarType t = x.scalar_type();
  if (!x.is_cuda() || !(dim == 2 || dim == 3) || !x.is_contiguous() || x.numel() == 0) Py_RETURN_NONE;
  if (!(is16(t) || (t == at::kFloat && dim == 2)) || (ue && !(col && tma))) Py_RETURN_NONE;
  const int64_t hidden_in = x.size(dim - 1), hidden = silu ? hidden_in / 2 : hidden_in;
  if (gs <= 0 || hidden_in % gs != 0 || (silu && hidden_in % 2 != 0) || hidden % gs != 0) Py_RETURN_NONE;
  const int64_t E = dim == 3 ? x.size(0) : 1, M = x.size(dim - 2), G = hidden / gs;
  // a 3-D tensor with plain column-major scales keeps the Python route's shape rules
  if (dim == 3 && col && !tma) Py_RETURN_NONE;
  const int32_t* mptr = nullptr;
  if (mp) {
    if (dim != 3 || !mp->is_cuda() || mp->scalar_type() != at::kInt || !mp->is_contiguous() || mp->numel() != E) Py_RETURN_NONE;
    mptr = mp->const_data_ptr<int32_t>();
  }
  const c10::Device dev = x.device();
  const c10::cuda::OptionalCUDAGuard guard(dev);
  void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  const int64_t W = ue ? (G + 3) / 4 : G;                       // scale words per row
  const int64_t ld = col ? (tma ? up(M, 4) : M) : W;            // stride between word columns (or rows)
  const at::ScalarType st = ue ? at::kInt : at::kFloat;
  at::Tensor q, s;
  if (dim == 2) {
    q = empty({M, hidden}, at::kFloat8_e4m3fn, dev);
    s = col ? empty({W, ld}, st, dev) : empty({M, W}, st, dev);
    if (col) s.unsafeGetTensorImpl()->set_sizes_and_strides(at::IntArrayRef({M, W}), at::IntArrayRef({1, ld}));
  } else {
    q = empty({E, M, hidden}, at::kFloat8_e4m3fn, dev);
    s = col ? empty({E, W, ld}, st, dev) : empty({E, M, W}, st, dev);
    if (col) s.unsafeGetTensorImpl()->set_sizes_and_strides(at::IntArrayRef({E, M, W}), at::IntArrayRef({W * ld, 1, ld}));
  }
  const int code = t == at::kFloat ? SGLB200_F32 : code16(t);
  const float e = eps_in_dtype(eps, t);
  if (dim == 3)
    check_rc(sglb200_group_quant_fp8_batched(x.const_data_ptr(), code, q.mutable_data_ptr(), s.mutable_data_ptr(), E, M, hidden,
                                             (int)gs, e, (float)lo, (float)hi, ue, silu, mptr, s.stride(0), s.stride(1),
                                             s.stride(2), stream),
             "sgl_per_token_group_quant_8bit(masked)");
  else if (silu)
    check_rc(sglb200_silu_mul_group_quant_fp8(x.const_data_ptr(), code, q.mutable_data_ptr(), s.mutable_data_ptr(), nullptr, M,
                                              hidden, (int)gs, e, (float)lo, (float)hi, ue, s.stride(0), s.stride(1), stream),
             "sgl_per_token_group_quant_8bit(fuse_silu_and_mul)");
  else
    check_rc(sglb200_per_token_group_quant_fp8(x.const_data_ptr(), code, q.mutable_data_ptr(), s.mutable_data_ptr(), M, hidden,
                                               (int)gs, e, (float)lo, (float)hi, ue, s.stride(0), s.stride(1), stream),
             "sgl_per_token_group_quant_8bit");
  PyObject* out = PyTuple_New(2);
  if (!out) return nullptr;
  PyTuple_SET_ITEM(out, 0, THPVariable_Wrap(std::move(q)));
  PyTuple_SET_ITEM(out, 1, THPVariable_Wrap(std::move(s)));
  return out;
}

// ---------------------------------------------------------------------------------------------- linear layer
// block_linear(x, weight, weight_scale, bias, ue8m0) -> out: quantise the activations, multiply, add the bias.
// weight_scale is fp32 [ceil(N/128), K/128], or with ue8m0 the packed int32 words [ceil(N/128), ceil(K/512)].
PyObject* block_linear(PyObject* const* args, Py_ssize_t n) {
  if (n != 5) Py_RETURN_NONE;
  const at::Tensor *xp = tensor_or_null(args[0]), *wp = tensor_or_null(args[1]), *sp = tensor_or_null(args[2]);
  const at::Tensor* bp = args[3] == Py_None ? nullptr : tensor_or_null(args[3]);
  if (!xp || !wp || !sp || (args[3] != Py_None && !bp)) Py_RETURN_NONE;
  const at::Tensor &x = *xp, &w = *wp, &ws = *sp;
  const bool ue = args[4] == Py_True;
  const at::ScalarType t = x.scalar_type();
  const int64_t dim = x.dim();
  if (!x.is_cuda() || !is16(t) || dim < 1 || !x.is_contiguous() || x.numel() == 0) Py_RETURN_NONE;
  if (w.scalar_type() != at::kFloat8_e4m3fn || w.dim() != 2 || !w.is_contiguous() || w.device() != x.device()) Py_RETURN_NONE;
  const int64_t N = w.size(0), K = w.size(1), KB = K / 128, NB = (N + 127) / 128, KG = (KB + 3) / 4;
  if (N == 0 || N % 8 != 0 || K == 0 || K % 128 != 0 || x.size(dim - 1) != K) Py_RETURN_NONE;
  if (ws.scalar_type() != (ue ? at::kInt : at::kFloat) || ws.dim() != 2 || ws.size(0) != NB || ws.size(1) != (ue ? KG : KB) ||
      ws.device() != x.device())
    Py_RETURN_NONE;
  if (bp && (bp->device() != x.device() || bp->scalar_type() != t || bp->requires_grad() ||
             bp->dim() != 1 || bp->size(0) != N || bp->stride(0) != 1 || reinterpret_cast<uintptr_t>(bp->const_data_ptr()) % 16 != 0))
    Py_RETURN_NONE;
  const int64_t M = x.numel() / K;
  const c10::Device dev = x.device();
  const c10::cuda::OptionalCUDAGuard guard(dev);
  const c10::cuda::CUDAStream cs = c10::cuda::getCurrentCUDAStream(dev.index());
  void* stream = cs.stream();
  at::DimVector shape(x.sizes().begin(), x.sizes().end());
  shape[dim - 1] = N;
  at::Tensor out = empty(shape, t, dev);
  const int64_t bytes = sglb200_fp8_block_linear_scratch_bytes(M, N, K, ue);
  c10::DataPtr scratch;
  if (bytes > 0) scratch = c10::cuda::CUDACachingAllocator::get()->allocate((size_t)bytes);
  check_rc(sglb200_fp8_block_linear(x.const_data_ptr(), w.const_data_ptr(), ws.const_data_ptr(),
                                    bp ? bp->const_data_ptr() : nullptr, out.mutable_data_ptr(), M, N, K, ws.stride(0),
                                    ws.stride(1), ue, eps_in_dtype(1e-10, t), code16(t), scratch.get(), bytes, stream),
           "fp8_block_linear");
  return THPVariable_Wrap(std::move(out));
}

// ---------------------------------------------------------------------------------------------- router
// topk_softmax(logits, topk, renormalize) -> (weights, ids)
PyObject* topk_softmax(PyObject* const* args, Py_ssize_t n) {
  if (n != 3) Py_RETURN_NONE;
  const at::Tensor* lp = tensor_or_null(args[0]);
  if (!lp || !PyLong_Check(args[1])) Py_RETURN_NONE;
  const at::Tensor& x = *lp;
  const int64_t topk = PyLong_AsLong(args[1]);
  if (PyErr_Occurred()) return nullptr;
  const at::ScalarType t = x.scalar_type();
  if (!x.is_cuda() || x.dim() != 2 || !x.is_contiguous() || !(is16(t) || t == at::kFloat) || x.numel() == 0) Py_RETURN_NONE;
  if (topk < 1 || topk > x.size(1)) Py_RETURN_NONE;
  const bool renorm = PyObject_IsTrue(args[2]) == 1;
  const c10::Device dev = x.device();
  const c10::cuda::OptionalCUDAGuard guard(dev);
  void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  const int64_t M = x.size(0);
  at::Tensor w = empty({M, topk}, at::kFloat, dev), ids = empty({M, topk}, at::kInt, dev);
  check_rc(sglb200_topk_softmax(x.const_data_ptr(), t == at::kFloat ? SGLB200_F32 : code16(t), w.mutable_data_ptr<float>(),
                                ids.mutable_data_ptr<int32_t>(), M, x.size(1), topk, renorm, stream),
           "topk_softmax");
  PyObject* out = PyTuple_New(2);
  if (!out) return nullptr;
  PyTuple_SET_ITEM(out, 0, THPVariable_Wrap(std::move(w)));
  PyTuple_SET_ITEM(out, 1, THPVariable_Wrap(std::move(ids)));
  return out;
}

// ---------------------------------------------------------------------------------------------- expert layer
// fused_experts(x, w1, w2, s1, s2, topk_weights, topk_ids, weight_factor, out or None, ue8m0) -> out
PyObject* fused_experts(PyObject* const* args, Py_ssize_t n) {
  if (n != 10) Py_RETURN_NONE;
  const at::Tensor* t[7];
  for (int i = 0; i < 7; ++i)
    if (!(t[i] = tensor_or_null(args[i]))) Py_RETURN_NONE;
  const at::Tensor &x = *t[0], &w1 = *t[1], &w2 = *t[2], &s1 = *t[3], &s2 = *t[4], &tw = *t[5], &ids = *t[6];
  const double factor = PyFloat_AsDouble(args[7]);
  if (PyErr_Occurred()) return nullptr;
  const at::Tensor* op = args[8] == Py_None ? nullptr : tensor_or_null(args[8]);
  if (args[8] != Py_None && !op) Py_RETURN_NONE;
  const bool ue = args[9] == Py_True;
  const at::ScalarType dt = x.scalar_type();
  if (!x.is_cuda() || !is16(dt) || x.dim() != 2 || !x.is_contiguous() || x.numel() == 0) Py_RETURN_NONE;
  for (int i = 1; i < 7; ++i)
    if (t[i]->device() != x.device()) Py_RETURN_NONE;
  if (w1.dim() != 3 || w2.dim() != 3 || !w1.is_contiguous() || !w2.is_contiguous() || w1.scalar_type() != at::kFloat8_e4m3fn ||
      w2.scalar_type() != at::kFloat8_e4m3fn)
    Py_RETURN_NONE;
  const int64_t M = x.size(0), H = x.size(1), E = w1.size(0), I = w1.size(1) / 2, topk = ids.dim() == 2 ? ids.size(1) : 0;
  if (E < 1 || E > 1024 || w1.size(1) != 2 * I || w1.size(2) != H || w2.size(0) != E || w2.size(1) != H || w2.size(2) != I)
    Py_RETURN_NONE;
  if (H % 128 != 0 || I == 0 || I % 128 != 0) Py_RETURN_NONE;
  const at::ScalarType st = ue ? at::kInt : at::kFloat;
  const int64_t k1 = ue ? (H / 128 + 3) / 4 : H / 128, k2 = ue ? (I / 128 + 3) / 4 : I / 128;
  if (s1.scalar_type() != st || s2.scalar_type() != st || s1.dim() != 3 || s2.dim() != 3 || s1.size(0) != E || s2.size(0) != E ||
      s1.size(1) != 2 * I / 128 || s1.size(2) != k1 || s2.size(1) != H / 128 || s2.size(2) != k2)
    Py_RETURN_NONE;
  if (topk < 1 || topk > 32 || M * topk > (1 << 24) || tw.dim() != 2 || tw.size(0) != M || tw.size(1) != topk || ids.size(0) != M ||
      tw.scalar_type() != at::kFloat || ids.scalar_type() != at::kInt || !tw.is_contiguous() || !ids.is_contiguous())
    Py_RETURN_NONE;
  if (op && (op->device() != x.device() || op->scalar_type() != dt || op->dim() != 2 || op->size(0) != M || op->size(1) != H ||
             !op->is_contiguous()))
    Py_RETURN_NONE;
  const c10::Device dev = x.device();
  const c10::cuda::OptionalCUDAGuard guard(dev);
  void* stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  at::Tensor out = op ? *op : empty({M, H}, dt, dev);
  const int64_t bytes = sglb200_fused_experts_scratch_bytes(M, H, I, E, topk, ue);
  c10::DataPtr scratch = c10::cuda::CUDACachingAllocator::get()->allocate((size_t)bytes);
  check_rc(sglb200_fused_experts(x.const_data_ptr(), code16(dt), w1.const_data_ptr(), w2.const_data_ptr(), s1.const_data_ptr(),
                                 s2.const_data_ptr(), s1.strides().data(), s2.strides().data(), tw.const_data_ptr<float>(),
                                 ids.const_data_ptr<int32_t>(), (float)factor, out.mutable_data_ptr(), M, H, I, E, topk, ue,
                                 eps_in_dtype(1e-10, dt), scratch.get(), bytes, stream),
           "fused_experts");
  return THPVariable_Wrap(std::move(out));
}

// grouped_masked(a, a_s, w, w_s, out, masked_m, expected_m) -> True
PyObject* grouped_masked(PyObject* const* args, Py_ssize_t n) {
  if (n != 7) Py_RETURN_NONE;
  const at::Tensor* t[6];
  for (int i = 0; i < 6; ++i)
    if (!(t[i] = tensor_or_null(args[i]))) Py_RETURN_NONE;
  const at::Tensor &a = *t[0], &as = *t[1], &w = *t[2], &ws = *t[3], &out = *t[4], &mm = *t[5];
  if (!PyLong_Check(args[6])) Py_RETURN_NONE;
  const int64_t expected = PyLong_AsLong(args[6]);
  if (PyErr_Occurred()) return nullptr;
  if (!a.is_cuda() || a.dim() != 3 || w.dim() != 3 || a.scalar_type() != at::kFloat8_e4m3fn || w.scalar_type() != at::kFloat8_e4m3fn ||
      !a.is_contiguous() || w.stride(2) != 1)
    Py_RETURN_NONE;
  for (int i = 1; i < 6; ++i)
    if (t[i]->device() != a.device()) Py_RETURN_NONE;
  const int64_t G = a.size(0), max_m = a.size(1), K = a.size(2), N = w.size(1), kt = (K + 127) / 128, nt = (N + 127) / 128;
  if (G == 0 || max_m == 0 || N == 0 || w.size(0) != G || w.size(2) != K) Py_RETURN_NONE;
  if (out.dim() != 3 || out.size(0) != G || out.size(1) != max_m || out.size(2) != N || !out.is_contiguous() || !is16(out.scalar_type()))
    Py_RETURN_NONE;
  if (as.scalar_type() != at::kFloat || as.dim() != 3 || as.size(0) != G || as.size(1) != max_m || as.size(2) != kt ||
      ws.scalar_type() != at::kFloat || ws.dim() != 3 || ws.size(0) != G || ws.size(1) != nt || ws.size(2) != kt)
    Py_RETURN_NONE;
  if (mm.scalar_type() != at::kInt || !mm.is_contiguous() || mm.numel() != G) Py_RETURN_NONE;
  const c10::Device dev = a.device();
  const c10::cuda::OptionalCUDAGuard guard(dev);
  check_rc(sglb200_fp8_blockwise_scaled_masked_grouped_mm_expected(
               a.const_data_ptr(), w.const_data_ptr(), as.const_data_ptr<float>(), ws.const_data_ptr<float>(), out.mutable_data_ptr(),
               mm.const_data_ptr<int32_t>(), G, max_m, expected, N, K, a.stride(1), w.stride(1), w.stride(0), out.stride(1),
               as.stride(0), as.stride(1), as.stride(2), ws.stride(0), ws.stride(1), ws.stride(2), code16(out.scalar_type()),
               c10::cuda::getCurrentCUDAStream(dev.index()).stream()),
           "grouped_gemm_nt_f8f8bf16_masked");
  Py_RETURN_TRUE;
}

#define SGLB_METHOD(name) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)(void)>(entry<name>)), METH_FASTCALL, nullptr}
PyMethodDef kMethods[] = {
    SGLB_METHOD(quant),         SGLB_METHOD(block_linear),   SGLB_METHOD(topk_softmax),
    SGLB_METHOD(fused_experts), SGLB_METHOD(grouped_masked),
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_sglb200_host", nullptr, -1, kMethods};

}  // namespace

PyMODINIT_FUNC PyInit__sglb200_host() { return PyModule_Create(&kModule); }
