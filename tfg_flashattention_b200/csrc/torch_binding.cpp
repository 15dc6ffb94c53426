// Python binding of the library's entry points that a program calls per layer or per token: the
// compiled counterpart of the reference's src/cpp/torch_bind.cpp:21-49 (`PYBIND11_MODULE ...
// m.def("forward", ...)`), in front of this library's C ABI (include/fa_b200.h) instead of the
// reference's launcher template.
//
//   forward(Q, K_mat, V, causal=True, return_lse=False, softmax_scale=None, out=None)
//   decode(Q, K_cache, V_cache, kv_len, return_lse=False, softmax_scale=None, out=None,
//          k_new=None, v_new=None)
//   add_layernorm(a, resid, scale, shift, eps=1e-5, return_sum=True, sum_out=None, norm_out=None)
//
// Three positional tensors behave as the reference's binding: CUDA + bfloat16 checked the same way
// (CHECK_CUDA / the dtype branch, torch_bind.cpp:13-19, 33-42), O = empty_like(Q) (:31), causal,
// scale 1/sqrt(64), returns O.  Differences: size(3) is checked (the reference assumes 64), tensors
// need not be contiguous (strides go to the library, which reads `[B,N,H,d]` views in place), the
// launch goes to the current stream of Q's device, the GIL is released around the library call,
// and the library's error code becomes a RuntimeError (the reference drops its cudaError_t).
// PyTorch is used for what it owns: tensors, the current device and stream.
//
// The functions are plain CPython vector calls: for the smallest problems the call IS the time, and
// pybind11's argument casters cost about as much as the launch (a decode call through ctypes: 31-38
// us of host time for 4-9 us of GPU work).
#include <algorithm>
#include <ATen/cuda/CUDAContextLight.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cublasLt.h>
#include <dlfcn.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/extension.h>

#include "../../include/fa_b200.h"

namespace {

// Argument and library errors leave as std::runtime_error, which `guarded` turns into the same
// Python RuntimeError that TORCH_CHECK produces in the reference binding.
#define FA_CHECK(cond, ...)                                        \
  do {                                                             \
    if (!(cond)) throw std::runtime_error(c10::str(__VA_ARGS__)); \
  } while (0)

struct TypeError : std::runtime_error {
  using std::runtime_error::runtime_error;
};
struct PythonError {};      // the Python error is set already

template <class F>
PyObject* guarded(F f) {
  try {
    return f();
  } catch (const PythonError&) {
    return nullptr;
  } catch (const TypeError& e) {
    PyErr_SetString(PyExc_TypeError, e.what());
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

// Positional and keyword arguments into `out` by the order of `names`; missing ones stay null.
template <size_t kN>
void take_args(const char* fn, const char* const (&names)[kN], size_t required, PyObject* const* args, Py_ssize_t nargs,
               PyObject* kwnames, PyObject* (&out)[kN]) {
  if (nargs > static_cast<Py_ssize_t>(kN)) throw TypeError(c10::str(fn, "() takes at most ", kN, " arguments"));
  for (size_t i = 0; i < kN; ++i) out[i] = i < static_cast<size_t>(nargs) ? args[i] : nullptr;
  const Py_ssize_t nkw = kwnames ? PyTuple_GET_SIZE(kwnames) : 0;
  for (Py_ssize_t k = 0; k < nkw; ++k) {
    PyObject* name = PyTuple_GET_ITEM(kwnames, k);
    size_t i = 0;
    while (i < kN && PyUnicode_CompareWithASCIIString(name, names[i]) != 0) ++i;
    if (i == kN) throw TypeError(c10::str(fn, "() got an unexpected keyword argument"));
    if (out[i] != nullptr) throw TypeError(c10::str(fn, "() got multiple values for argument '", names[i], "'"));
    out[i] = args[nargs + k];
  }
  for (size_t i = 0; i < required; ++i)
    if (out[i] == nullptr) throw TypeError(c10::str(fn, "() missing required argument '", names[i], "'"));
}
const at::Tensor& tensor_arg(PyObject* o, const char* name) {
  if (!THPVariable_Check(o)) throw TypeError(c10::str(name, " must be a torch.Tensor"));
  return THPVariable_Unpack(o);
}
bool given(PyObject* o) { return o != nullptr && o != Py_None; }
bool flag_arg(PyObject* o, bool absent) {
  if (o == nullptr) return absent;
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw PythonError();
  return v != 0;
}
double number_arg(PyObject* o, double absent) {
  if (!given(o)) return absent;
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PythonError();
  return v;
}
PyObject* pair(const at::Tensor& a, const at::Tensor& b) {
  PyObject* t = PyTuple_New(2);
  if (t == nullptr) throw PythonError();
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(a));
  PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(b));
  return t;
}
// Outputs come from the allocator directly: the dispatcher's way to it (autograd, device guards, the
// factory function's own dispatch) costs as much as the allocation, and nothing here is differentiated.
at::Tensor empty_cuda(at::IntArrayRef sizes, at::ScalarType type, const at::Device& device) {
  return at::detail::empty_cuda(sizes, type, device, std::nullopt);
}
at::Tensor empty_like_cuda(const at::Tensor& t) {
  if (!t.is_non_overlapping_and_dense()) return at::empty_like(t);      // chooses the strides itself
  return at::detail::empty_strided_cuda(t.sizes(), t.strides(), t.scalar_type(), t.device());
}

template <class Call>
void launch(const char* what, Call call) {
  int rc;
  {
    py::gil_scoped_release release;
    rc = call();
  }
  FA_CHECK(rc == 0, what, " failed (", rc, "): ", fa_b200_strerror(rc));
}

void check_input(const at::Tensor& t, const char* name) {
  FA_CHECK(t.device().is_cuda(), name, " must be a CUDA tensor");
  FA_CHECK(t.scalar_type() == torch::kBFloat16, "Unsupported tensor dtype. Use bfloat16.");
  FA_CHECK(t.dim() == 4, name, " must have shape [B, H, N, d]");
}

// Element strides {batch, head, row}; strides of size-1 dimensions are never dereferenced, so they
// are replaced by a canonical value that always passes the library's checks.
void strides3(const at::Tensor& t, const char* name, int64_t out[3]) {
  const int64_t H = t.size(1), N = t.size(2), d = t.size(3);
  FA_CHECK(d <= 1 || t.stride(3) == 1, name, ": the last dimension must be dense (stride 1)");
  int64_t sb = t.stride(0), sh = t.stride(1), sn = t.stride(2);
  if (N == 1) sn = d;
  if (H == 1) sh = std::max<int64_t>(N * sn, 8);
  if (t.size(0) == 1) sb = std::max<int64_t>(std::max(H * sh, N * sn), 8);
  out[0] = sb; out[1] = sh; out[2] = sn;
}

PyObject* forward(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
  return guarded([&]() -> PyObject* {
    static const char* const names[] = {"Q", "K_mat", "V", "causal", "return_lse", "softmax_scale", "out"};
    PyObject* a[7];
    take_args("forward", names, 3, args, nargs, kwnames, a);
    const at::Tensor &Q = tensor_arg(a[0], "Q"), &K_mat = tensor_arg(a[1], "K_mat"), &V = tensor_arg(a[2], "V");
    const bool return_lse = flag_arg(a[4], false);
    check_input(Q, "Q");
    check_input(K_mat, "K_mat");
    check_input(V, "V");
    FA_CHECK(K_mat.sizes() == Q.sizes() && V.sizes() == Q.sizes(),
             "Q, K_mat and V must have the same shape [B, H, N, d]");
    FA_CHECK(K_mat.device() == Q.device() && V.device() == Q.device(),
             "Q, K_mat and V must be on the same device");
    at::Tensor O;
    if (given(a[6])) {
      O = tensor_arg(a[6], "out");
      check_input(O, "out");
      FA_CHECK(O.sizes() == Q.sizes() && O.device() == Q.device(), "out must match Q in shape and device");
    } else {
      O = empty_like_cuda(Q);   // same allocation rule as the reference (torch_bind.cpp:31)
    }
    at::Tensor lse;
    if (return_lse) lse = empty_cuda({Q.size(0), Q.size(1), Q.size(2)}, torch::kFloat32, Q.device());

    fa_b200_params p{};
    p.B = static_cast<int32_t>(Q.size(0));
    p.H = static_cast<int32_t>(Q.size(1));
    p.N = static_cast<int32_t>(Q.size(2));
    p.d = static_cast<int32_t>(Q.size(3));
    if (Q.numel() > 0) {
      p.q = Q.data_ptr(); p.k = K_mat.data_ptr(); p.v = V.data_ptr(); p.o = O.data_ptr();
      strides3(Q, "Q", p.q_strides);
      strides3(K_mat, "K_mat", p.k_strides);
      strides3(V, "V", p.v_strides);
      strides3(O, "out", p.o_strides);
    } else {            // empty problem: nothing is read, any valid pointers and strides do
      p.q = p.k = p.v = p.o = reinterpret_cast<void*>(16);
      for (int i = 0; i < 3; ++i) p.q_strides[i] = p.k_strides[i] = p.v_strides[i] = p.o_strides[i] = 8;
    }
    p.lse = return_lse && Q.numel() > 0 ? lse.data_ptr<float>() : nullptr;
    p.softmax_scale = static_cast<float>(number_arg(a[5], 0.0));
    p.causal = flag_arg(a[3], true) ? 1 : 0;
    p.device = Q.device().index();
    p.stream = c10::cuda::getCurrentCUDAStream(Q.device().index()).stream();
    launch("custom_flash_attn.forward", [&] { return fa_b200_fwd(&p); });
    return return_lse ? pair(O, lse) : THPVariable_Wrap(O);
  });
}

// Whether t is [B, H, 64] or [B, H, n, 64] (its first row is meant then), dense in the last dimension.  (No
// view is made of it: three of them cost more host time than the launch's arguments.)
bool is_row(const at::Tensor& t, int64_t B, int64_t H, int64_t d) {
  const int64_t n = t.dim();
  return (n == 3 || (n == 4 && t.size(2) >= 1)) && t.size(0) == B && t.size(1) == H && t.size(n - 1) == d && t.stride(n - 1) == 1;
}
// {batch, head} strides of it; size-1 dimensions get a canonical stride
void strides2(const at::Tensor& t, int64_t out[2]) {
  out[1] = t.size(1) == 1 ? 64 : t.stride(1);
  out[0] = t.size(0) == 1 ? std::max<int64_t>(t.size(1) * out[1], 64) : t.stride(0);
}
void cache_strides(const at::Tensor& t, int64_t out[3]) {
  out[2] = t.size(2) == 1 ? 64 : t.stride(2);
  out[1] = t.size(1) == 1 ? std::max<int64_t>(t.size(2) * out[2], 64) : t.stride(1);
  out[0] = t.size(0) == 1 ? std::max<int64_t>(t.size(1) * out[1], 64) : t.stride(0);
}

PyObject* decode(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
  return guarded([&]() -> PyObject* {
    static const char* const names[] = {"Q", "K_cache", "V_cache", "kv_len", "return_lse", "softmax_scale", "out",
                                        "k_new", "v_new"};
    PyObject* a[9];
    take_args("decode", names, 4, args, nargs, kwnames, a);
    const at::Tensor &Q = tensor_arg(a[0], "Q"), &K = tensor_arg(a[1], "K_cache"), &V = tensor_arg(a[2], "V_cache");
    const bool squeeze = Q.dim() == 4;
    for (const auto& [t, name] : {std::pair<const at::Tensor&, const char*>{Q, "Q"}, {K, "K_cache"}, {V, "V_cache"}}) {
      FA_CHECK(t.device().is_cuda(), name, " must be a CUDA tensor");
      FA_CHECK(t.scalar_type() == torch::kBFloat16, "Unsupported tensor dtype. Use bfloat16.");
    }
    FA_CHECK(!squeeze || Q.size(2) == 1, "Q must hold one query row per head: [B, H, 64] or [B, H, 1, 64]");
    FA_CHECK((squeeze || Q.dim() == 3) && K.dim() == 4 && V.dim() == 4, "expected Q [B, H, d] and caches [B, H, N, d]");
    const int64_t B = Q.size(0), H = Q.size(1), d = Q.size(Q.dim() - 1), rows = K.size(2);
    FA_CHECK(K.size(0) == B && K.size(1) == H && V.sizes() == K.sizes() && K.size(3) == d,
             "Q, K_cache and V_cache disagree on B, H or d");
    fa_b200_decode_params p{};
    int64_t kv_len = rows;
    if (THPVariable_Check(a[3])) {
      // the length lives on the device (an int32 scalar that the caller advances between steps): the
      // launch is sized for the whole cache and the kernel reads the length when it runs, which is
      // what lets one recorded CUDA-graph launch serve every step of a generation loop
      const at::Tensor& n = THPVariable_Unpack(a[3]);
      FA_CHECK(n.is_cuda() && n.scalar_type() == torch::kInt32 && n.numel() == 1,
               "a tensor kv_len must be one int32 on the GPU");
      p.kv_len_device = n.data_ptr<int32_t>();
    } else {
      kv_len = PyLong_Check(a[3]) ? PyLong_AsLongLong(a[3]) : static_cast<int64_t>(number_arg(a[3], 0.0));
      if (kv_len == -1 && PyErr_Occurred()) throw PythonError();
    }
    FA_CHECK(kv_len >= 1 && kv_len <= rows, "kv_len must be between 1 and the cache length");
    FA_CHECK(Q.stride(Q.dim() - 1) == 1, "Q: the last dimension must be dense (stride 1)");
    FA_CHECK(K.stride(3) == 1, "K_cache: the last dimension must be dense (stride 1)");
    FA_CHECK(V.stride(3) == 1, "V_cache: the last dimension must be dense (stride 1)");
    at::Tensor O;
    if (given(a[6])) {
      O = tensor_arg(a[6], "out");
      FA_CHECK(O.scalar_type() == torch::kBFloat16 && O.device() == Q.device() && is_row(O, B, H, d),
               "out must match Q in shape, dtype and device");
    } else {
      const int64_t sizes[4] = {B, H, 1, d}, flat[3] = {B, H, d};
      O = squeeze ? empty_cuda(sizes, torch::kBFloat16, Q.device()) : empty_cuda(flat, torch::kBFloat16, Q.device());
    }
    const bool return_lse = flag_arg(a[4], false);
    at::Tensor lse;
    if (return_lse) lse = empty_cuda({B, H}, torch::kFloat32, Q.device());
    p.B = static_cast<int32_t>(B); p.H = static_cast<int32_t>(H);
    p.kv_len = static_cast<int32_t>(kv_len); p.d = static_cast<int32_t>(d);
    if (B * H > 0) {
      p.q = Q.data_ptr(); p.k_cache = K.data_ptr(); p.v_cache = V.data_ptr(); p.o = O.data_ptr();
      strides2(Q, p.q_strides);
      strides2(O, p.o_strides);
      cache_strides(K, p.k_strides);
      cache_strides(V, p.v_strides);
    } else {
      p.q = p.k_cache = p.v_cache = p.o = reinterpret_cast<void*>(16);
      for (int i = 0; i < 2; ++i) p.q_strides[i] = p.o_strides[i] = 64;
      for (int i = 0; i < 3; ++i) p.k_strides[i] = p.v_strides[i] = 64;
    }
    p.lse = return_lse ? lse.data_ptr<float>() : nullptr;
    p.softmax_scale = static_cast<float>(number_arg(a[5], 0.0));
    FA_CHECK(given(a[7]) == given(a[8]), "k_new and v_new go together");
    if (given(a[7])) {
      const at::Tensor &kn = tensor_arg(a[7], "k_new"), &vn = tensor_arg(a[8], "v_new");
      for (const auto& [t, name] : {std::pair<const at::Tensor&, const char*>{kn, "k_new"}, {vn, "v_new"}})
        FA_CHECK(t.is_cuda() && t.scalar_type() == torch::kBFloat16 && is_row(t, B, H, d),
                 name, " must be a CUDA bfloat16 tensor [B, H, 64] with a dense last dimension");
      int64_t vs[2];
      strides2(kn, p.new_strides);
      strides2(vn, vs);
      FA_CHECK(vs[0] == p.new_strides[0] && vs[1] == p.new_strides[1], "k_new and v_new must have the same strides");
      p.k_new = kn.data_ptr();
      p.v_new = vn.data_ptr();
    }
    p.device = Q.device().index();
    p.stream = c10::cuda::getCurrentCUDAStream(Q.device().index()).stream();
    launch("custom_flash_attn.decode", [&] { return fa_b200_decode_direct(&p); });
    return return_lse ? pair(O, lse) : THPVariable_Wrap(O);
  });
}

const at::Tensor& dense2d(PyObject* o, const char* name, int64_t cols) {
  FA_CHECK(THPVariable_Check(o), name, " must be a CUDA bfloat16 tensor");
  const at::Tensor& t = THPVariable_Unpack(o);
  FA_CHECK(t.is_cuda() && t.scalar_type() == torch::kBFloat16, name, " must be a CUDA bfloat16 tensor");
  FA_CHECK(t.dim() > 0 && t.size(-1) == cols && t.is_contiguous(), name, " must be contiguous with ", cols, " columns");
  return t;
}

PyObject* add_layernorm(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
  return guarded([&]() -> PyObject* {
    static const char* const names[] = {"a", "resid", "scale", "shift", "eps", "return_sum", "sum_out", "norm_out"};
    PyObject* v[8];
    take_args("add_layernorm", names, 4, args, nargs, kwnames, v);
    const at::Tensor& a = tensor_arg(v[0], "a");
    FA_CHECK(a.dim() > 0, "a must have at least one dimension");
    const int64_t cols = a.size(-1);
    dense2d(v[0], "a", cols);
    fa_b200_add_layernorm_params p{};
    p.a = a.data_ptr();
    if (given(v[1])) {
      const at::Tensor& resid = dense2d(v[1], "resid", cols);
      FA_CHECK(resid.sizes() == a.sizes(), "a and resid must have the same shape");
      p.resid = resid.data_ptr();
    }
    const at::Tensor &scale = dense2d(v[2], "scale", cols), &shift = dense2d(v[3], "shift", cols);
    FA_CHECK(scale.numel() == cols, "scale must have ", cols, " elements");
    FA_CHECK(shift.numel() == cols, "shift must have ", cols, " elements");
    const bool keep = flag_arg(v[5], true) && given(v[1]);
    at::Tensor sum, norm;
    if (keep) sum = given(v[6]) ? tensor_arg(v[6], "sum_out") : empty_like_cuda(a);
    norm = given(v[7]) ? tensor_arg(v[7], "norm_out") : empty_like_cuda(a);
    p.scale = scale.data_ptr();
    p.shift = shift.data_ptr();
    p.sum_out = keep ? sum.data_ptr() : nullptr;
    p.norm_out = norm.data_ptr();
    p.rows = cols ? a.numel() / cols : 0;
    p.cols = static_cast<int32_t>(cols);
    p.eps = static_cast<float>(number_arg(v[4], 1e-5));
    p.device = a.device().index();
    p.stream = c10::cuda::getCurrentCUDAStream(a.device().index()).stream();
    int rc;
    {
      py::gil_scoped_release release;
      rc = fa_b200_add_layernorm(&p);
    }
    FA_CHECK(rc == 0, fa_b200_strerror(rc));
    return keep ? pair(sum, norm) : THPVariable_Wrap(norm);
  });
}

// ---- GEMMs of the block loop: cuBLASLt, which torch's linear calls too, but asked for an algorithm once
// per shape.  Torch asks on every call: 17 us of host time per GEMM, four per layer, more than the
// kernels themselves take for a few hundred tokens; with the plan kept it is a launch.
// The library is the one torch has loaded; where it cannot be found the loop uses at::linear.
struct LtApi {
  decltype(&cublasLtMatmulDescCreate) desc_create = nullptr;
  decltype(&cublasLtMatmulDescDestroy) desc_destroy = nullptr;
  decltype(&cublasLtMatmulDescSetAttribute) desc_set = nullptr;
  decltype(&cublasLtMatrixLayoutCreate) layout_create = nullptr;
  decltype(&cublasLtMatrixLayoutDestroy) layout_destroy = nullptr;
  decltype(&cublasLtMatmulPreferenceCreate) pref_create = nullptr;
  decltype(&cublasLtMatmulPreferenceSetAttribute) pref_set = nullptr;
  decltype(&cublasLtMatmulPreferenceDestroy) pref_destroy = nullptr;
  decltype(&cublasLtMatmulAlgoGetHeuristic) heuristic = nullptr;
  decltype(&cublasLtMatmul) matmul = nullptr;
  bool ok = false;
  LtApi() {
    void* lib = dlopen("libcublasLt.so.12", RTLD_NOW | RTLD_NOLOAD);
    if (lib == nullptr) return;
    auto get = [&](auto& fn, const char* name) { fn = reinterpret_cast<std::decay_t<decltype(fn)>>(dlsym(lib, name)); return fn != nullptr; };
    ok = get(desc_create, "cublasLtMatmulDescCreate") && get(desc_destroy, "cublasLtMatmulDescDestroy") &&
         get(desc_set, "cublasLtMatmulDescSetAttribute") && get(layout_destroy, "cublasLtMatrixLayoutDestroy") &&
         get(layout_create, "cublasLtMatrixLayoutCreate") && get(pref_create, "cublasLtMatmulPreferenceCreate") &&
         get(pref_set, "cublasLtMatmulPreferenceSetAttribute") && get(pref_destroy, "cublasLtMatmulPreferenceDestroy") &&
         get(heuristic, "cublasLtMatmulAlgoGetHeuristic") && get(matmul, "cublasLtMatmul");
  }
};
const LtApi& lt() {
  static const LtApi api;
  return api;
}
// With 1 to 16 MB the library picks the kernels that it picks for torch; with 32 MB or none it takes others
// for some GELU GEMMs (GPT-2 medium, 750 rows: 14.3 us instead of 11.1).
constexpr size_t kLtWorkspace = 8u << 20;
struct LtKey {
  int device;
  int64_t m, n, k;
  int epilogue;
  uint32_t align[3];      // of w, x and y: an algorithm may rely on them
  bool operator==(const LtKey& o) const {
    return device == o.device && m == o.m && n == o.n && k == o.k && epilogue == o.epilogue && align[0] == o.align[0] &&
           align[1] == o.align[1] && align[2] == o.align[2];
  }
};
// The largest power of two up to 256 (what the library assumes unless told) that the address is a multiple of.
uint32_t alignment(const at::Tensor& t) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(t.data_ptr()) | 256u;
  return static_cast<uint32_t>(a & (~a + 1));
}
struct LtPlan {
  LtKey key;
  bool usable = false;
  cublasLtMatmulDesc_t desc = nullptr;
  cublasLtMatrixLayout_t w = nullptr, x = nullptr, y = nullptr;
  cublasLtMatmulAlgo_t algo;
  void clear() {
    for (cublasLtMatrixLayout_t* l : {&w, &x, &y})
      if (*l != nullptr) { lt().layout_destroy(*l); *l = nullptr; }
    if (desc != nullptr) { lt().desc_destroy(desc); desc = nullptr; }
  }
  ~LtPlan() { clear(); }
};
// y [m, n] = x [m, k] w [n, k]^T + bias, tanh-GELU with `gelu`.  Plans are per host thread (a descriptor
// is written on every call: the bias address), the last 64 of them.
bool lt_linear(const at::Tensor& x, const at::Tensor& w, const at::Tensor* bias, bool gelu, at::Tensor& y, void* workspace,
               void* stream) {
  const LtApi& api = lt();
  if (!api.ok || !w.is_contiguous() || !x.is_contiguous() || (gelu && bias == nullptr)) return false;
  const uint32_t align[3] = {alignment(w), alignment(x), alignment(y)};
  if (std::min({align[0], align[1], align[2], bias ? alignment(*bias) : 256u}) < 16) return false;
  constexpr int kPlans = 64;
  static thread_local LtPlan plans[kPlans];
  static thread_local int next = 0;
  const int64_t k = w.size(1), n = w.size(0), m = x.numel() / k;
  const int epilogue = gelu ? CUBLASLT_EPILOGUE_GELU_BIAS : (bias ? CUBLASLT_EPILOGUE_BIAS : CUBLASLT_EPILOGUE_DEFAULT);
  const LtKey key{x.device().index(), m, n, k, epilogue, {align[0], align[1], align[2]}};
  LtPlan* plan = nullptr;
  for (LtPlan& p : plans)
    if (p.desc != nullptr && p.key == key) { plan = &p; break; }
  const cublasLtHandle_t handle = at::cuda::getCurrentCUDABlasLtHandle();
  if (plan == nullptr) {
    plan = &plans[next];
    next = (next + 1) % kPlans;
    plan->clear();
    plan->key = key;
    plan->usable = false;
    // (row-major operands are column-major transposes: y^T [n, m] = w [n, k] x^T [k, m])
    auto ok = [](cublasStatus_t s) { return s == CUBLAS_STATUS_SUCCESS; };
    const cublasOperation_t trans = CUBLAS_OP_T;
    const cublasLtEpilogue_t ep = static_cast<cublasLtEpilogue_t>(epilogue);
    const cudaDataType_t type = CUDA_R_16BF;
    cublasLtMatmulPreference_t pref = nullptr;
    cublasLtMatmulHeuristicResult_t found[1];
    int count = 0;
    const uint64_t limit = kLtWorkspace;
    const void* any = reinterpret_cast<const void*>(256);
    plan->usable = ok(api.desc_create(&plan->desc, CUBLAS_COMPUTE_32F, CUDA_R_32F)) &&
                   ok(api.desc_set(plan->desc, CUBLASLT_MATMUL_DESC_TRANSA, &trans, sizeof(trans))) &&
                   ok(api.desc_set(plan->desc, CUBLASLT_MATMUL_DESC_EPILOGUE, &ep, sizeof(ep))) &&
                   (bias == nullptr || (ok(api.desc_set(plan->desc, CUBLASLT_MATMUL_DESC_BIAS_DATA_TYPE, &type, sizeof(type))) &&
                                        ok(api.desc_set(plan->desc, CUBLASLT_MATMUL_DESC_BIAS_POINTER, &any, sizeof(any))))) &&
                   ok(api.layout_create(&plan->w, type, k, n, k)) && ok(api.layout_create(&plan->x, type, k, m, k)) &&
                   ok(api.layout_create(&plan->y, type, n, m, n)) && ok(api.pref_create(&pref)) &&
                   ok(api.pref_set(pref, CUBLASLT_MATMUL_PREF_MAX_WORKSPACE_BYTES, &limit, sizeof(limit))) &&
                   ok(api.pref_set(pref, CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_A_BYTES, &align[0], sizeof(uint32_t))) &&
                   ok(api.pref_set(pref, CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_B_BYTES, &align[1], sizeof(uint32_t))) &&
                   ok(api.pref_set(pref, CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_C_BYTES, &align[2], sizeof(uint32_t))) &&
                   ok(api.pref_set(pref, CUBLASLT_MATMUL_PREF_MIN_ALIGNMENT_D_BYTES, &align[2], sizeof(uint32_t))) &&
                   ok(api.heuristic(handle, plan->desc, plan->w, plan->x, plan->y, plan->y, pref, 1, found, &count)) && count > 0;
    if (pref != nullptr) api.pref_destroy(pref);
    if (plan->usable) plan->algo = found[0].algo;
  }
  if (!plan->usable) return false;
  if (bias != nullptr) {
    const void* at = bias->data_ptr();
    if (api.desc_set(plan->desc, CUBLASLT_MATMUL_DESC_BIAS_POINTER, &at, sizeof(at)) != CUBLAS_STATUS_SUCCESS) return false;
  }
  const float one = 1.f, zero = 0.f;
  return api.matmul(handle, plan->desc, &one, w.data_ptr(), plan->w, x.data_ptr(), plan->x, &zero, y.data_ptr(), plan->y,
                    y.data_ptr(), plan->y, &plan->algo, workspace, kLtWorkspace, static_cast<cudaStream_t>(stream)) ==
         CUBLAS_STATUS_SUCCESS;
}

// The block stack of a prompt, one native loop instead of a dozen Python calls per layer (those cost
// more than their kernels for a few hundred tokens: GPT-2 small, 72 tokens: 0.9 ms of host time for
// 0.57 ms of kernels).  The same operations in the same order as GPTModel._blocks_fused.
void add_ln(const at::Tensor& a, const at::Tensor* resid, const at::Tensor& g, const at::Tensor& b, double eps,
            void* sum_out, at::Tensor& norm, void* stream) {
  fa_b200_add_layernorm_params p{};
  const int64_t cols = a.size(-1);
  p.a = a.data_ptr();
  p.resid = resid ? resid->data_ptr() : nullptr;
  p.scale = g.data_ptr();
  p.shift = b.data_ptr();
  p.sum_out = sum_out;
  p.norm_out = norm.data_ptr();
  p.rows = a.numel() / cols;
  p.cols = static_cast<int32_t>(cols);
  p.eps = static_cast<float>(eps);
  p.device = a.device().index();
  p.stream = stream;
  const int rc = fa_b200_add_layernorm(&p);
  FA_CHECK(rc == 0, fa_b200_strerror(rc));
}

// blocks(x, layers, caches, heads, eps, lnf_scale, lnf_shift, last_token_only): x [B, n, C] is the
// residual stream (overwritten); layers a list of tuples (ln1 scale, shift, qkv weight, bias or None, proj
// weight, bias, ln2 scale, shift, fc weight, bias, out weight, bias); caches a list of (K, V) pairs
// [B, N_max, H, 64] whose rows 0 .. n-1 are written, or None.  Returns the final LayerNorm's output.
PyObject* blocks(PyObject*, PyObject* const* args, Py_ssize_t nargs, PyObject* kwnames) {
  return guarded([&]() -> PyObject* {
    static const char* const names[] = {"x", "layers", "caches", "heads", "eps", "lnf_scale", "lnf_shift", "last_token_only"};
    PyObject* a[8];
    take_args("blocks", names, 8, args, nargs, kwnames, a);
    at::Tensor x = tensor_arg(a[0], "x");
    FA_CHECK(x.is_cuda() && x.scalar_type() == torch::kBFloat16 && x.dim() == 3 && x.is_contiguous(), "x must be a contiguous bfloat16 CUDA tensor [B, n, C]");
    FA_CHECK(PyList_Check(a[1]) && (a[2] == Py_None || PyList_Check(a[2])), "layers and caches are lists");
    const int64_t B = x.size(0), n = x.size(1), C = x.size(2), H = PyLong_AsLongLong(a[3]);
    FA_CHECK(H > 0 && C == 64 * H, "the width must be 64 * heads");
    const double eps = number_arg(a[4], 1e-5);
    const at::Tensor lnf_g = tensor_arg(a[5], "lnf_scale"), lnf_b = tensor_arg(a[6], "lnf_shift");
    const bool last_only = flag_arg(a[7], false), cached = a[2] != Py_None;
    struct Layer { at::Tensor t[12], k, v; };
    std::vector<Layer> layers(static_cast<size_t>(PyList_GET_SIZE(a[1])));
    FA_CHECK(!cached || PyList_GET_SIZE(a[2]) == static_cast<Py_ssize_t>(layers.size()), "one cache per layer");
    for (size_t l = 0; l < layers.size(); ++l) {
      PyObject* t = PyList_GET_ITEM(a[1], l);
      FA_CHECK(PyTuple_Check(t) && PyTuple_GET_SIZE(t) == 12, "a layer has twelve tensors");
      for (int i = 0; i < 12; ++i)
        if (PyTuple_GET_ITEM(t, i) != Py_None) layers[l].t[i] = tensor_arg(PyTuple_GET_ITEM(t, i), "a layer's parameter");
      const at::Tensor &qkv_w = layers[l].t[2], &proj_w = layers[l].t[4], &fc_w = layers[l].t[8], &out_w = layers[l].t[10];
      FA_CHECK(qkv_w.defined() && proj_w.defined() && fc_w.defined() && out_w.defined() && qkv_w.dim() == 2 && proj_w.dim() == 2 &&
                   fc_w.dim() == 2 && out_w.dim() == 2 && qkv_w.size(0) == 3 * C && qkv_w.size(1) == C && proj_w.size(0) == C &&
                   proj_w.size(1) == C && fc_w.size(1) == C && out_w.size(0) == C && out_w.size(1) == fc_w.size(0),
               "a layer's weights are [3C, C], [C, C], [hidden, C] and [C, hidden]");
      if (cached) {
        PyObject* kv = PyList_GET_ITEM(a[2], l);
        FA_CHECK(PyTuple_Check(kv) && PyTuple_GET_SIZE(kv) == 2, "a cache is a pair");
        for (int i = 0; i < 2; ++i) {
          const at::Tensor& c = tensor_arg(PyTuple_GET_ITEM(kv, i), "a cache");
          FA_CHECK(c.is_cuda() && c.scalar_type() == torch::kBFloat16 && c.dim() == 4 && c.size(0) == B && c.size(1) >= n &&
                       c.size(2) == H && c.size(3) == 64 && c.stride(3) == 1 &&
                       (i == 0 || c.strides() == layers[l].k.strides()),
                   "the caches must be bfloat16 [B, >= n, H, 64] with the same strides");
          (i ? layers[l].v : layers[l].k) = c;
        }
      }
    }
    at::Tensor result;
    {
      py::gil_scoped_release release;
      const at::AutoDispatchBelowADInplaceOrView below_autograd;
      const c10::cuda::CUDAGuard guard(x.device());
      void* stream = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
      // Buffers for all layers.  The hidden layer lies where the projection and the attention's output lay,
      // which are dead by then: 7 instead of 11 widths per row, so that more of a prompt stays in L2.
      const int64_t rows = B * n;
      const int64_t ctx_at = (rows * 3 * C + 127) / 128 * 128;       // 256 bytes: any GEMM takes it
      int64_t size = ctx_at + rows * C;
      for (const Layer& L : layers) size = std::max(size, rows * L.t[8].size(0));
      const at::Tensor arena = empty_cuda({size}, torch::kBFloat16, x.device());
      at::Tensor qkv = arena.narrow(0, 0, rows * 3 * C).view({B, n, 3 * C});
      at::Tensor ctx = arena.narrow(0, ctx_at, rows * C).view({B, n, C}), mid;
      at::Tensor branch, added = empty_like_cuda(x), h = empty_like_cuda(x);
      const at::Tensor workspace = empty_cuda({static_cast<int64_t>(kLtWorkspace)}, torch::kUInt8, x.device());
      auto linear = [&](const at::Tensor& in, const at::Tensor& w, const at::Tensor& bias, at::Tensor& y) {
        if (!lt_linear(in, w, bias.defined() ? &bias : nullptr, false, y, workspace.data_ptr(), stream))
          y.copy_(at::linear(in, w, bias.defined() ? std::optional<at::Tensor>(bias) : std::nullopt));
      };
      for (const Layer& L : layers) {
        if (branch.defined()) add_ln(branch, &x, L.t[0], L.t[1], eps, x.data_ptr(), h, stream);
        else add_ln(x, nullptr, L.t[0], L.t[1], eps, nullptr, h, stream);
        linear(h, L.t[2], L.t[3], qkv);
        auto* base = static_cast<at::BFloat16*>(qkv.data_ptr());
        fa_b200_params p{};
        p.B = static_cast<int32_t>(B); p.H = static_cast<int32_t>(H); p.N = static_cast<int32_t>(n); p.d = 64;
        p.q = base; p.k = base + C; p.v = base + 2 * C; p.o = ctx.data_ptr();
        for (int64_t* s : {p.q_strides, p.k_strides, p.v_strides}) { s[0] = 3 * C * n; s[1] = 64; s[2] = 3 * C; }
        p.o_strides[0] = C * n; p.o_strides[1] = 64; p.o_strides[2] = C;
        p.causal = 1;
        p.device = x.device().index();
        p.stream = stream;
        int rc = 0;
        if (cached) {
          fa_b200_cache_write_params c{};
          c.k = p.k; c.v = p.v; c.k_cache = L.k.data_ptr(); c.v_cache = L.v.data_ptr();
          c.strides[0] = 3 * C * n; c.strides[1] = 3 * C; c.strides[2] = 64;
          for (int i = 0; i < 3; ++i) c.cache_strides[i] = L.k.size(i) == 1 ? 64 : L.k.stride(i);   // (size 1: never used)
          c.B = p.B; c.N = p.N; c.H = p.H; c.device = p.device; c.stream = stream;
          rc = fa_b200_cache_write(&c);
          FA_CHECK(rc == 0, "cache write failed (", rc, "): ", fa_b200_strerror(rc));
        }
        rc = fa_b200_fwd(&p);
        FA_CHECK(rc == 0, "custom_flash_attn.forward failed (", rc, "): ", fa_b200_strerror(rc));
        branch = added;
        linear(ctx, L.t[4], L.t[5], branch);
        add_ln(branch, &x, L.t[6], L.t[7], eps, x.data_ptr(), h, stream);
        const int64_t hidden = L.t[8].size(0);
        if (!mid.defined() || mid.size(2) != hidden) mid = arena.narrow(0, 0, rows * hidden).view({B, n, hidden});
        if (!lt_linear(h, L.t[8], &L.t[9], true, mid, workspace.data_ptr(), stream))
          mid.copy_(at::_addmm_activation(L.t[9], h.view({rows, C}), L.t[8].t(), 1, 1, /*use_gelu=*/true).view({B, n, hidden}));
        linear(mid, L.t[10], L.t[11], branch);
      }
      if (last_only) {                 // what generate() consumes
        x = x.slice(1, n - 1, n).contiguous();
        if (branch.defined()) branch = branch.slice(1, n - 1, n).contiguous();
      }
      result = empty_like_cuda(x);
      if (branch.defined()) add_ln(branch, &x, lnf_g, lnf_b, eps, nullptr, result, stream);
      else add_ln(x, nullptr, lnf_g, lnf_b, eps, nullptr, result, stream);
    }
    return THPVariable_Wrap(result);
  });
}

PyMethodDef methods[] = {
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&forward)), METH_FASTCALL | METH_KEYWORDS,
     "FlashAttention forward on B200 (libfa_b200.so)"},
    {"decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&decode)), METH_FASTCALL | METH_KEYWORDS,
     "Single-query attention against a K/V cache"},
    {"add_layernorm", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&add_layernorm)),
     METH_FASTCALL | METH_KEYWORDS, "Shortcut addition and LayerNorm in one pass"},
    {"blocks", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(&blocks)), METH_FASTCALL | METH_KEYWORDS,
     "The transformer blocks of a prompt"},
    {nullptr, nullptr, 0, nullptr}};

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  if (PyModule_AddFunctions(m.ptr(), methods) != 0) throw py::error_already_set();
  m.attr("abi_version") = FA_B200_ABI_VERSION;   // the header this module was compiled against
}
