// Python entry points of the kernel library that take tensors (module cosmos_rl_b200.ops._host).
//
// A small call is bound by the host, and most of that is the way from Python to a launch: every argument converted by ctypes,
// every pointer and stride asked for by a method call, results allocated through Python. Here a launcher takes its tensors as they
// are (wrap: one entry for each launcher named below, argument types from its declaration), and the calls that every layer makes
// check their operands, allocate their results and launch in one step. us a call on the host, with ctypes and here: a projection
// of 57 rows 11.9 and 6.7 (its two launches take 4.3), residual add + RMSNorm 9.3 and 7.4, SwiGLU 7.9 and 5.6, rotary embedding
// 13.7 and 4.3, attention 16.2 and 8.6, a dense GEMM 13.3 and 6.9.
//
// A launcher's answer (0, or a code of api.h) is returned as an int; the steps return their tensors, or the int if it is not 0.
// Nothing is kept between calls. The interpreter lock is released around allocations and launches, as ctypes does; C++ exceptions
// become the Python exceptions that torch's own functions raise.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <ATen/ATen.h>

#include <climits>
#include <utility>

#include "api.h"

namespace {

using at::Tensor;

struct Unlocked {   // the interpreter lock is released while this lives
  PyThreadState* state = PyEval_SaveThread();
  ~Unlocked() { PyEval_RestoreThread(state); }
};

// ---- arguments ---------------------------------------------------------------------------------------------------
const Tensor& tensor(PyObject* o) {
  TORCH_CHECK_TYPE(THPVariable_Check(o), "expected a tensor, got ", Py_TYPE(o)->tp_name);
  return THPVariable_Unpack(o);
}
const Tensor& tensor_or_none(PyObject* o) {
  static const Tensor none;
  return o == Py_None ? none : tensor(o);
}
long long integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}
double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw python_error();
  return v;
}
// a tensor's memory; tensors that have elements but no memory (traced, fake) never get to a launch
void* mem(const Tensor& t) {
  void* p = t.data_ptr();
  TORCH_CHECK(p != nullptr || t.numel() == 0, "a tensor without memory cannot be given to a kernel");
  return p;
}
void* address(PyObject* o) {   // None, an address or a tensor
  if (o == Py_None) return nullptr;
  if (THPVariable_Check(o)) return mem(THPVariable_Unpack(o));
  void* p = PyLong_AsVoidPtr(o);
  if (p == nullptr && PyErr_Occurred()) throw python_error();
  return p;
}
template <class T>
struct Arg;
template <class T>
struct Arg<T*> {
  static T* of(PyObject* o) { return static_cast<T*>(address(o)); }
};
template <>
struct Arg<long long> {
  static long long of(PyObject* o) { return integer(o); }
};
template <>
struct Arg<int> {
  static int of(PyObject* o) {
    const long long v = integer(o);
    TORCH_CHECK_VALUE(v >= INT_MIN && v <= INT_MAX, v, " does not fit the launcher's argument");
    return (int)v;
  }
};
template <>
struct Arg<float> {
  static float of(PyObject* o) { return (float)real(o); }
};
bool flag(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw python_error();
  return v != 0;
}
void want(Py_ssize_t n, Py_ssize_t count) {
  TORCH_CHECK_TYPE(n == count, "expected ", count, " arguments, got ", n);
}

// ---- one entry for a launcher ------------------------------------------------------------------------------------
template <class R, class... A, size_t... I>
PyObject* launch(R (*fn)(A...), PyObject* const* args, std::index_sequence<I...>) {
  const std::tuple<A...> a{Arg<A>::of(args[I])...};
  R rc;
  {
    Unlocked unlocked;
    rc = std::apply(fn, a);
  }
  return PyLong_FromLongLong(rc);
}
template <class R, class... A>
PyObject* launch_all(R (*fn)(A...), PyObject* const* args, Py_ssize_t n) {
  want(n, sizeof...(A));
  return launch(fn, args, std::index_sequence_for<A...>{});
}
template <auto FN>
PyObject* wrap(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  return launch_all(FN, args, n);
  END_HANDLE_TH_ERRORS
}

// ---- steps -------------------------------------------------------------------------------------------------------
// what a step refuses, as the assertions of the Python functions around it do
#define REQUIRE(cond)                                          \
  if (!(cond)) {                                               \
    PyErr_SetString(PyExc_AssertionError, #cond);              \
    throw python_error();                                      \
  }

bool bf16(const Tensor& t) { return t.scalar_type() == at::kBFloat16; }
Tensor like(const Tensor& t, at::IntArrayRef shape) { return at::empty(shape, t.options().dtype(at::kBFloat16)); }
Tensor floats(const Tensor& t, at::IntArrayRef shape) { return at::empty(shape, t.options().dtype(at::kFloat)); }
void* data(const Tensor& t) { return t.defined() ? mem(t) : nullptr; }
int i32(int64_t v) {
  TORCH_CHECK_VALUE(v <= INT_MAX, "a size of ", v, " is beyond what the kernels take");
  return (int)v;
}
PyObject* give(const Tensor& t) {
  if (t.defined()) return THPVariable_Wrap(t);
  Py_RETURN_NONE;
}
PyObject* give2(const Tensor& a, const Tensor& b) {
  PyObject* r = PyTuple_New(2);
  if (r == nullptr) throw python_error();
  PyTuple_SET_ITEM(r, 0, give(a));
  PyTuple_SET_ITEM(r, 1, give(b));
  return r;
}
cudaStream_t stream_of(PyObject* o) { return static_cast<cudaStream_t>(address(o)); }

// (x [T, H], weight, eps, residual or None, rstd or None, stream) -> (y, x + residual or None); rows contiguous
PyObject* rmsnorm_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  want(n, 6);
  const Tensor &x = tensor(a[0]), &w = tensor(a[1]), &res = tensor_or_none(a[3]), &rstd = tensor_or_none(a[4]);
  const float eps = (float)real(a[2]);
  const cudaStream_t s = stream_of(a[5]);
  REQUIRE(x.dim() == 2);
  Tensor y, res_out;
  int rc;
  {
    Unlocked unlocked;
    y = at::empty_like(x);
    if (res.defined()) res_out = at::empty_like(x);
    rc = b200_rmsnorm_fwd(mem(x), data(res), mem(w), mem(y), data(res_out), (float*)data(rstd), i32(x.size(0)),
                          i32(x.size(1)), eps, s);
  }
  return rc ? PyLong_FromLong(rc) : give2(y, res_out);
  END_HANDLE_TH_ERRORS
}

// (dy, h [T, H], weight, rstd, dres or None, with dw, rows of scratch, stream) -> (dx, dw or None)
PyObject* rmsnorm_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  want(n, 8);
  const Tensor &h = tensor(a[1]), &w = tensor(a[2]), &rstd = tensor(a[3]);
  Tensor dy = tensor(a[0]), dres = tensor_or_none(a[4]);
  const bool with_dw = flag(a[5]);
  const int64_t rows = integer(a[6]), H = h.size(1);
  const cudaStream_t s = stream_of(a[7]);
  Tensor dx, dw, ws;
  int rc;
  {
    Unlocked unlocked;
    dy = dy.contiguous();
    if (dres.defined()) dres = dres.contiguous();
    dx = at::empty_like(h);
    if (with_dw) {
      dw = like(h, {H});
      ws = floats(h, {rows * std::max<int64_t>(H, 1024)});
    }
    rc = b200_rmsnorm_bwd2(mem(dy), mem(h), mem(w), (const float*)mem(rstd), data(dres), mem(dx),
                           data(dw), (float*)data(ws), h.size(0), i32(H), s);
  }
  return rc ? PyLong_FromLong(rc) : give2(dx, dw);
  END_HANDLE_TH_ERRORS
}

// (gate_up [T, 2 I], stream) -> [T, I]; rows contiguous
PyObject* swiglu_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  want(n, 2);
  const Tensor& gu = tensor(a[0]);
  const cudaStream_t s = stream_of(a[1]);
  REQUIRE(gu.dim() == 2);
  const int64_t T = gu.size(0), I = gu.size(1) / 2;
  Tensor out;
  int rc;
  {
    Unlocked unlocked;
    out = at::empty({T, I}, gu.options());
    rc = b200_swiglu_fwd(mem(gu), mem(out), T, i32(I), nullptr, s);
  }
  return rc ? PyLong_FromLong(rc) : give(out);
  END_HANDLE_TH_ERRORS
}

// (gradient of the product, gate_up [T, 2 I], stream) -> gradient of gate_up
PyObject* swiglu_bwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  want(n, 3);
  Tensor d = tensor(a[0]);
  const Tensor& gu = tensor(a[1]);
  const cudaStream_t s = stream_of(a[2]);
  Tensor dgu;
  int rc;
  {
    Unlocked unlocked;
    d = d.contiguous();
    dgu = at::empty_like(gu);
    rc = b200_swiglu_bwd(mem(d), mem(gu), mem(dgu), gu.size(0), i32(gu.size(1) / 2), nullptr, s);
  }
  return rc ? PyLong_FromLong(rc) : give(dgu);
  END_HANDLE_TH_ERRORS
}

// (qkv [T, >= (hq + hkv) d], positions, hq, hkv, d, theta, backward, stream) -> answer of the launcher: q and k columns in place.
// None: not a matrix of adjacent columns; nothing was done.
PyObject* rope_qkv(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  want(n, 8);
  const Tensor &qkv = tensor(a[0]), &pos = tensor(a[1]);
  const int hq = Arg<int>::of(a[2]), hkv = Arg<int>::of(a[3]), d = Arg<int>::of(a[4]), backward = flag(a[6]);
  const float theta = (float)real(a[5]);
  const cudaStream_t s = stream_of(a[7]);
  if (qkv.dim() != 2 || qkv.stride(1) != 1 || hq <= 0 || hkv <= 0 || qkv.size(1) < (int64_t)(hq + hkv) * d) Py_RETURN_NONE;
  char* q = (char*)mem(qkv);
  const long long *p = (const long long*)mem(pos), stride = qkv.stride(0);
  int rc;
  {
    Unlocked unlocked;
    rc = b200_rope_inplace(q, q + (int64_t)hq * d * qkv.element_size(), p, i32(qkv.size(0)), hq, hkv, d, stride, stride, theta,
                           backward, s);
  }
  return PyLong_FromLong(rc);
  END_HANDLE_TH_ERRORS
}

// (qkv [T, (hq + 2 hkv) d], positions, hq, hkv, d, theta, backward, stream) -> a new tensor, q and k columns rotated. None: not a
// matrix that the kernel takes.
PyObject* rope_qkv_new(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  want(n, 8);
  const Tensor &qkv = tensor(a[0]), &pos = tensor(a[1]);
  const int hq = Arg<int>::of(a[2]), hkv = Arg<int>::of(a[3]), d = Arg<int>::of(a[4]), backward = flag(a[6]);
  const float theta = (float)real(a[5]);
  const cudaStream_t s = stream_of(a[7]);
  if (qkv.dim() != 2 || !bf16(qkv) || qkv.stride(1) != 1 || hq <= 0 || hkv <= 0 || d <= 0 || d % 16 || d > 512 ||
      qkv.size(1) != (int64_t)(hq + 2 * hkv) * d || qkv.stride(0) % 8 || ((uintptr_t)mem(qkv) & 15))
    Py_RETURN_NONE;
  Tensor out;
  int rc;
  {
    Unlocked unlocked;
    out = like(qkv, qkv.sizes());
    rc = b200_rope_qkv(mem(qkv), mem(out), (const long long*)mem(pos), i32(qkv.size(0)), hq, hkv, d, qkv.stride(0), out.stride(0), theta,
                       backward, s);
  }
  return rc ? PyLong_FromLong(rc) : give(out);
  END_HANDLE_TH_ERRORS
}

// whether the tensor-core GEMMs take x and weight: they move rows with TMA, feature dimensions must give 16-byte rows
PyObject* linear_ok(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  want(n, 2);
  const Tensor &x = tensor(a[0]), &w = tensor(a[1]);
  return PyBool_FromLong(x.is_cuda() && w.device() == x.device() && bf16(x) && bf16(w) && w.dim() == 2 && w.stride(1) == 1 && w.size(0) % 8 == 0 &&
                         w.size(1) % 8 == 0 && w.stride(0) % 8 == 0);
  END_HANDLE_TH_ERRORS
}

// (x [M <= max_m, K], weight [N, K], bias or None, out or None, workspace or None, max_m, status, SMs, stream) -> out
PyObject* skinny_linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  want(n, 9);
  const Tensor &x = tensor(a[0]), &w = tensor(a[1]), &bias = tensor_or_none(a[2]), &ws = tensor_or_none(a[4]);
  Tensor out = tensor_or_none(a[3]);
  const int max_m = Arg<int>::of(a[5]), sms = Arg<int>::of(a[7]);
  uint32_t* status = (uint32_t*)address(a[6]);
  const cudaStream_t s = stream_of(a[8]);
  REQUIRE(x.dim() == 2 && x.is_cuda() && bf16(x) && bf16(w) && x.size(0) <= max_m);
  REQUIRE(w.dim() == 2 && x.stride(1) == 1 && w.stride(1) == 1);
  REQUIRE(x.size(1) == w.size(1));
  int rc;
  {
    Unlocked unlocked;
    if (!out.defined()) out = like(x, {x.size(0), w.size(0)});
    rc = b200_skinny_linear(mem(x), mem(w), data(bias), bias.defined() && bf16(bias), mem(out), (float*)data(ws),
                            ws.defined() ? ws.numel() : 0, i32(x.size(0)), i32(w.size(0)), i32(x.size(1)), x.stride(0), w.stride(0),
                            out.stride(0), status, sms, s);
  }
  return rc ? PyLong_FromLong(rc) : give(out);
  END_HANDLE_TH_ERRORS
}

// (a, b, a_mn, b_mn, out or None, fp32 result, accumulate, bias or None, swiglu, path, scratch or None, its floats, status, SMs,
// stream) -> out. floats < 0: not known yet; a call that wants scratch then answers how much (more than any code of api.h).
PyObject* gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  want(n, 15);
  const Tensor &A = tensor(a[0]), &B = tensor(a[1]), &bias = tensor_or_none(a[7]), &ws = tensor_or_none(a[10]);
  const bool a_mn = flag(a[2]), b_mn = flag(a[3]), accumulate = flag(a[6]), swiglu = flag(a[8]);
  Tensor out = tensor_or_none(a[4]);
  bool fp32 = flag(a[5]);
  const int path = Arg<int>::of(a[9]), sms = Arg<int>::of(a[13]);
  const long long ws_floats = integer(a[11]);
  uint32_t* status = (uint32_t*)address(a[12]);
  const cudaStream_t s = stream_of(a[14]);
  REQUIRE(A.is_cuda() && bf16(A) && bf16(B));
  REQUIRE(A.dim() == 2 && B.dim() == 2 && A.stride(1) == 1 && B.stride(1) == 1);
  const int64_t M = A.size(a_mn), K = A.size(!a_mn), N = B.size(b_mn), cols = swiglu ? N / 2 : N;
  if (K != B.size(!b_mn)) {
    PyErr_Format(PyExc_AssertionError, "contraction of %lld and %lld", (long long)K, (long long)B.size(!b_mn));
    throw python_error();
  }
  if (bias.defined()) REQUIRE(bias.is_contiguous() && bias.numel() == N && (bf16(bias) || bias.scalar_type() == at::kFloat));
  long long need = 0;
  int rc = 0;
  {
    Unlocked unlocked;
    if (out.defined()) fp32 = out.scalar_type() == at::kFloat;
    else out = at::empty({M, cols}, A.options().dtype(fp32 ? at::kFloat : at::kBFloat16));
    if (ws_floats < 0) {
      const bool rows16 = (((uintptr_t)mem(out) | (uintptr_t)(out.stride(0) * out.element_size())) & 15) == 0;
      need = b200_gemm_scratch(i32(M), i32(N), i32(K), a_mn, rows16, fp32, accumulate, bias.defined(), swiglu, path, sms);
    }
    if (need == 0) {
      auto call = [&](int cut) {
        return b200_gemm_bf16_ws(mem(A), mem(B), mem(out), i32(M), i32(N), i32(K), A.stride(0), B.stride(0),
                                 out.stride(0), a_mn, b_mn, fp32, accumulate, data(bias), bias.defined() && bf16(bias), swiglu,
                                 swiglu ? i32(N / 2) : 0, path, cut, (float*)data(ws), ws_floats < 0 ? 0 : ws_floats, status, sms, s);
      };
      rc = call(1);
      if (rc == B200_NEED_WORKSPACE) rc = call(0);
    }
  }
  if (need) return PyLong_FromLongLong(need);
  return rc ? PyLong_FromLong(rc) : give(out);
  END_HANDLE_TH_ERRORS
}

// whether the attention kernels take q, k and v [T, heads, 128]
PyObject* flash_ok(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  want(n, 3);
  const Tensor *t[3] = {&tensor(a[0]), &tensor(a[1]), &tensor(a[2])};
  const Tensor& q = *t[0];
  bool ok = q.is_cuda() && bf16(q) && q.size(-1) == 128;
  for (int i = 0; i < 3 && ok; ++i) ok = t[i]->stride(-1) == 1 && t[i]->stride(1) == 128 && t[i]->stride(0) % 8 == 0;
  if (ok && t[1]->size(1) == 0) {
    PyErr_SetString(PyExc_ZeroDivisionError, "attention without kv heads");
    throw python_error();
  }
  return PyBool_FromLong(ok && q.size(1) % t[1]->size(1) == 0);
  END_HANDLE_TH_ERRORS
}

// (q, k, v, cu_q, cu_k, max_q, causal, scale, status, SMs, stream) -> (out [Tq, hq, d], lse [hq, Tq])
PyObject* flash_fwd(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  want(n, 11);
  const Tensor &q = tensor(a[0]), &k = tensor(a[1]), &v = tensor(a[2]), &cu_q = tensor(a[3]), &cu_k = tensor(a[4]);
  const int max_q = Arg<int>::of(a[5]), causal = flag(a[6]), sms = Arg<int>::of(a[9]);
  const float scale = (float)real(a[7]);
  uint32_t* status = (uint32_t*)address(a[8]);
  const cudaStream_t s = stream_of(a[10]);
  REQUIRE(q.dim() == 3 && k.dim() == 3 && v.dim() == 3);
  const int64_t Tq = q.size(0), hq = q.size(1), d = q.size(2);
  Tensor out, lse;
  int rc;
  {
    Unlocked unlocked;
    out = at::empty({Tq, hq, d}, q.options());
    lse = floats(q, {hq, Tq});
    rc = b200_flash_fwd(mem(q), mem(k), mem(v), mem(out), (float*)mem(lse),
                        (const int*)mem(cu_q), (const int*)mem(cu_k), i32(cu_q.numel() - 1), i32(Tq), i32(k.size(0)),
                        i32(hq), i32(k.size(1)), i32(d), q.stride(0), k.stride(0), v.stride(0), hq * d, max_q, causal, scale, status,
                        sms, s);
  }
  return rc ? PyLong_FromLong(rc) : give2(out, lse);
  END_HANDLE_TH_ERRORS
}

#define ENTRY(name, fn) {name, (PyCFunction)(void (*)(void))(fn), METH_FASTCALL, nullptr}
#define LAUNCHER(fn) ENTRY(#fn, wrap<fn>)
PyMethodDef methods[] = {
    ENTRY("rmsnorm_fwd", rmsnorm_fwd),
    ENTRY("rmsnorm_bwd", rmsnorm_bwd),
    ENTRY("swiglu_fwd", swiglu_fwd),
    ENTRY("swiglu_bwd", swiglu_bwd),
    ENTRY("rope_qkv", rope_qkv),
    ENTRY("rope_qkv_new", rope_qkv_new),
    ENTRY("linear_ok", linear_ok),
    ENTRY("skinny_linear", skinny_linear),
    ENTRY("gemm", gemm),
    ENTRY("flash_ok", flash_ok),
    ENTRY("flash_fwd", flash_fwd),
    LAUNCHER(b200_swiglu_fwd),
    LAUNCHER(b200_rope_inplace),
    LAUNCHER(b200_flash_bwd),
    LAUNCHER(b200_gemm_gate_up),
    LAUNCHER(b200_gemm_dgate_up),
    LAUNCHER(b200_gemm_gated_scratch),
    LAUNCHER(b200_gemm_skinny_splits),
    LAUNCHER(b200_gemm_skinny),
    LAUNCHER(b200_splitk_reduce_residual_rmsnorm),
    LAUNCHER(b200_splitk_reduce_qkv_rope_append),
    LAUNCHER(b200_paged_decode_tc),
    LAUNCHER(b200_lmhead_logprob_partial),
    LAUNCHER(b200_logprob_combine),
    LAUNCHER(b200_lmhead_dlogits),
    LAUNCHER(b200_quant_fp8_block),
    LAUNCHER(b200_gemm_fp8_block),
    LAUNCHER(b200_moe_route_topk),
    LAUNCHER(b200_moe_offsets),
    LAUNCHER(b200_moe_permute),
    LAUNCHER(b200_moe_zero_padding),
    LAUNCHER(b200_moe_spread),
    LAUNCHER(b200_moe_swiglu_bwd),
    LAUNCHER(b200_moe_combine),
    LAUNCHER(b200_grouped_gate_up),
    LAUNCHER(b200_grouped_gemm_rows),
    LAUNCHER(b200_grouped_wgrad_filled),
    {nullptr, nullptr, 0, nullptr},
};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Launchers of libb200rl that take tensors.", -1, methods};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit__host() { return PyModule_Create(&module); }
