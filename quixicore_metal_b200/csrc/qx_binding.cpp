// Native side of the Python binding for the operators a decode step calls: argument checks, output
// allocation, stream and workspace handling and the C ABI call in one C++ function, so that an eager call
// costs the interpreter one argument tuple instead of some forty Python-level operations (an M = 1
// projection: 14 us of host time per call through ctypes, of which the launch is 3).  Same checks in the
// same order and the same RuntimeError texts as the Python layer documents; torch supplies device memory
// and the current stream only.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "../../include/quixicore_cuda.h"

namespace {

struct CheckFailed { std::string msg; };
struct StatusFailed { qx_status st; };

[[noreturn]] void fail(std::string m) { throw CheckFailed{std::move(m)}; }
inline void check(bool ok, const char* op, const char* what) { if (!ok) fail(std::string(op) + ": " + what); }
inline void check_status(const qx_status& st) { if (st.code != QX_OK) throw StatusFailed{st}; }

PyObject* g_raise_status = nullptr;      // Python callable (code, operation, detail) -> raises

template <class F>
PyObject* guarded(F&& f) {
  try {
    return f();
  } catch (const CheckFailed& e) {
    PyErr_SetString(PyExc_RuntimeError, e.msg.c_str());
  } catch (const StatusFailed& e) {
    PyObject* r = PyObject_CallFunction(g_raise_status, "iss", (int)e.st.code, e.st.operation ? e.st.operation : "",
                                        e.st.detail ? e.st.detail : "");
    Py_XDECREF(r);
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "library status");
  } catch (const c10::Error& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

// The interpreter is released while a call copies operands, allocates and enqueues: a launch blocks when the queue
// is full, and other threads (and host functions on the stream) go on meanwhile.  No Python object is touched inside;
// the caller's argument tuple keeps the operands alive.
struct Released {
  PyThreadState* state = PyEval_SaveThread();
  ~Released() { PyEval_RestoreThread(state); }
};

// ---- arguments -----------------------------------------------------------------------------------------
const at::Tensor& tensor(PyObject* o, const char* op) {
  if (!THPVariable_Check(o)) fail(std::string(op) + ": a tensor was expected");
  return THPVariable_Unpack(o);
}
const at::Tensor* tensor_or_null(PyObject* o, const char* op) { return o == Py_None ? nullptr : &tensor(o, op); }   // only None is absent
int64_t integer(PyObject* o) {
  const int64_t v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) { PyErr_Clear(); fail("an integer was expected"); }
  return v;
}
double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) { PyErr_Clear(); fail("a number was expected"); }
  return v;
}
const char* text(PyObject* o) {
  const char* s = PyUnicode_AsUTF8(o);
  if (!s) { PyErr_Clear(); fail("a string was expected"); }
  return s;
}
bool truth(PyObject* o) { return PyObject_IsTrue(o) == 1; }

struct Format { const char* name; int bk, bb; };
const Format* format_of(const char* s) {
  static const Format f[] = {{"q4_0", 32, 18}, {"q8_0", 32, 34}, {"q6_K", 256, 210}, {"mxfp8", 32, 33}, {"nvfp4", 16, 9}, {"mxfp4", 32, 17}};
  for (const Format& x : f) if (std::strcmp(x.name, s) == 0) return &x;
  return nullptr;
}
int dtype_of(at::ScalarType t) {
  return t == at::kBFloat16 ? QX_DTYPE_BF16 : t == at::kHalf ? QX_DTYPE_F16 : t == at::kFloat ? QX_DTYPE_F32 : 0;
}
void same_device(const char* op, const at::Tensor& first, const at::Tensor* t) {
  if (t && t->device() != first.device())
    fail(std::string(op) + ": all tensors must be on the same device (got " + first.device().str() + " and " + t->device().str() + ")");
}
at::Tensor empty(at::IntArrayRef shape, at::ScalarType t, const at::Tensor& like) {
  return at::empty(shape, like.options().dtype(t).requires_grad(false));
}
inline at::Tensor dense(const at::Tensor& t) { return t.is_contiguous() ? t : t.contiguous(); }

// ---- workspace: one growing scratch tensor per stream ----------------------------------------------------
// Calls on one stream are ordered, so they share it.  A captured graph keeps the addresses that its calls used for
// as long as it lives, so memory once handed out is never given to anyone else: a tensor that became too small stays
// (each is at least twice as large as the one before, the total below twice the largest), and streams past
// the 64th get a tensor for the one call - a capture keeps what it allocated itself.
struct Key { int dev; cudaStream_t st; bool operator==(const Key& o) const { return dev == o.dev && st == o.st; } };
struct KeyHash { size_t operator()(const Key& k) const { return std::hash<void*>()((void*)k.st) * 31u + (size_t)k.dev; } };
std::mutex g_ws_mu;
using Sizes = std::vector<at::Tensor>;             // ascending; the last one serves the calls
std::unordered_map<Key, Sizes, KeyHash>& ws_map() { static auto* m = new std::unordered_map<Key, Sizes, KeyHash>(); return *m; }
at::Tensor workspace(at::Device device, cudaStream_t st, size_t bytes) {      // `device` is current, the interpreter released
  const Key key{(int)device.index(), st};
  int64_t size = std::max<int64_t>((int64_t)bytes, 1 << 20);
  {
    const std::lock_guard<std::mutex> lock(g_ws_mu);
    const auto it = ws_map().find(key);
    if (it != ws_map().end()) {
      if ((size_t)it->second.back().numel() >= bytes) return it->second.back();
      size = std::max<int64_t>(size, 2 * it->second.back().numel());
    }
  }
  const at::Tensor t = at::empty({size}, at::TensorOptions().dtype(at::kByte).device(device));
  const std::lock_guard<std::mutex> lock(g_ws_mu);
  if (ws_map().size() < 64 || ws_map().count(key)) {
    Sizes& s = ws_map()[key];
    if (s.empty() || s.back().numel() < size) s.push_back(t);
  }
  return t;
}

// ---- packed projections ----------------------------------------------------------------------------------
// The reference's check_decode_epilogue_weight (torch_kernels.mm:6376-6405): returns N.
int64_t check_weight(const at::Tensor& x, const at::Tensor& w, const Format* f, const char* op) {
  check(x.is_cuda() && w.is_cuda() && dtype_of(x.scalar_type()) && x.dim() == 2 && x.size(0) > 0 && x.size(1) > 0, op,
        "x must be non-empty (B,K) fp32/fp16/bf16");
  check(f != nullptr, op, "format must be q4_0, q8_0, q6_K, mxfp8, nvfp4, or mxfp4 (dense weights are routed to the framework "
                          "matmul, not to this backend)");
  const int64_t K = x.size(1);
  check(w.scalar_type() == at::kByte && w.dim() == 3 && w.size(0) > 0 && K % f->bk == 0 && w.size(1) == K / f->bk && w.size(2) == f->bb,
        op, "packed weight must be uint8 (N,K/block_k,block_bytes)");
  return w.size(0);
}
struct Quant { at::Tensor codes, scale; };
Quant quant_outputs(const at::Tensor& x, int64_t B, int64_t N, int kind) {
  Quant q;
  if (kind < 0) fail("output_quant must be None, 'fp8', 'int8', or 'mxfp8'");
  if (kind == 3) {
    if (N % 32 != 0) fail("output_quant='mxfp8' needs N to be a multiple of 32");
    q.codes = empty({B, N / 32, 33}, at::kByte, x);
  } else if (kind) {
    q.codes = empty({B, N}, kind == 1 ? at::kByte : at::kChar, x);
    q.scale = empty({B}, at::kFloat, x);
  }
  return q;
}
PyObject* wrap(const at::Tensor& t) { return THPVariable_Wrap(t); }
PyObject* wrap_or_none(const at::Tensor& t) {
  if (t.defined()) return wrap(t);
  Py_RETURN_NONE;
}
PyObject* quant_result(const at::Tensor& out, int kind, const Quant& q, bool with_output) {
  if (kind == 0) return wrap(out);
  PyObject* r = kind == 3 ? wrap(q.codes) : Py_BuildValue("(NN)", wrap(q.codes), wrap(q.scale));
  return with_output ? Py_BuildValue("(NN)", wrap(out), r) : r;
}
void* ptr(const at::Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

// (x, weight, bias, residual, format, activation, use_bias, use_residual, quant_kind, with_output, ordered)
PyObject* decode_linear_epilogue(PyObject*, PyObject* const* a, Py_ssize_t) {
  return guarded([&]() -> PyObject* {
    static const char* op = "decode_linear_epilogue";
    const int64_t act = integer(a[5]);
    check(act >= 0 && act <= 2, op, "activation must be 0, 1, or 2");
    const at::Tensor &x = tensor(a[0], op), &w = tensor(a[1], op);
    const Format* f = format_of(text(a[4]));
    const int64_t N = check_weight(x, w, f, op), B = x.size(0), K = x.size(1);
    const bool ub = truth(a[6]), ur = truth(a[7]);
    const at::Tensor *b = ub ? &tensor(a[2], op) : nullptr, *r = ur ? &tensor(a[3], op) : nullptr;
    same_device(op, x, &w); same_device(op, x, b); same_device(op, x, r);
    check(!ub || (b->is_cuda() && b->dim() == 1 && b->size(0) == N && b->scalar_type() == x.scalar_type()), op,
          "bias must be (N,) with x dtype");
    check(!ur || (r->is_cuda() && r->dim() == 2 && r->size(0) == B && r->size(1) == N && r->scalar_type() == x.scalar_type()), op,
          "residual must be (B,N) with x dtype");
    const int kind = (int)integer(a[8]);
    const bool with_output = truth(a[9]), ordered = truth(a[10]);
    at::Tensor out;
    Quant q;
    {
      const Released released;
      const c10::cuda::OptionalCUDAGuard guard(x.device());
      const at::Tensor xc = dense(x), wc = dense(w);
      at::Tensor bc, rc;
      if (ub) bc = dense(*b);
      if (ur) rc = dense(*r);
      out = empty({B, N}, x.scalar_type(), x);
      if (ordered) {
        check(kind == 0, op, "the ordered form has no output_quant");
        check_status(qx_cuda_decode_linear_epilogue_ordered(at::cuda::getCurrentCUDAStream().stream(), ptr(xc), ptr(wc), ptr(bc), ptr(rc),
                                                            ptr(out), B, K, N, f->name, (qx_dtype)dtype_of(x.scalar_type()), (int)act, ub,
                                                            ur, nullptr, 0));
      } else {
        q = quant_outputs(x, B, N, kind);
        check_status(qx_cuda_decode_linear_epilogue(at::cuda::getCurrentCUDAStream().stream(), ptr(xc), ptr(wc), ptr(bc), ptr(rc),
                                                    ptr(out), B, K, N, f->name, (qx_dtype)dtype_of(x.scalar_type()), (int)act, ub, ur,
                                                    kind, ptr(q.codes), (float*)ptr(q.scale), nullptr, 0));
      }
    }
    return quant_result(out, kind, q, with_output);
  });
}

// (x, weight, format)
PyObject* decode_linear_partial(PyObject*, PyObject* const* a, Py_ssize_t) {
  return guarded([&]() -> PyObject* {
    static const char* op = "decode_linear_partial";
    const at::Tensor &x = tensor(a[0], op), &w = tensor(a[1], op);
    const Format* f = format_of(text(a[2]));
    const int64_t N = check_weight(x, w, f, op);
    same_device(op, x, &w);
    at::Tensor out;
    {
      const Released released;
      const c10::cuda::OptionalCUDAGuard guard(x.device());
      const at::Tensor xc = dense(x), wc = dense(w);
      out = empty({x.size(0), N}, at::kFloat, x);
      check_status(qx_cuda_decode_linear_partial(at::cuda::getCurrentCUDAStream().stream(), ptr(xc), ptr(wc), (float*)ptr(out), x.size(0),
                                                 x.size(1), N, f->name, (qx_dtype)dtype_of(x.scalar_type()), nullptr, 0));
    }
    return wrap(out);
  });
}

// (x, gate, up, gate_bias, up_bias, format, use_bias, quant_kind, with_output, ordered)
PyObject* decode_swiglu(PyObject*, PyObject* const* a, Py_ssize_t) {
  return guarded([&]() -> PyObject* {
    static const char* op = "decode_swiglu";
    const at::Tensor &x = tensor(a[0], op), &g = tensor(a[1], op), &u = tensor(a[2], op);
    const Format* f = format_of(text(a[5]));
    const int64_t N = check_weight(x, g, f, op), UN = check_weight(x, u, f, op), B = x.size(0), K = x.size(1);
    check(UN == N && u.sizes() == g.sizes(), op, "gate and up weights must have identical shapes");
    const bool ub = truth(a[6]);
    const at::Tensor *gb = ub ? &tensor(a[3], op) : nullptr, *bb = ub ? &tensor(a[4], op) : nullptr;
    same_device(op, x, &g); same_device(op, x, &u); same_device(op, x, gb); same_device(op, x, bb);
    check(!ub || (gb->is_cuda() && bb->is_cuda() && gb->scalar_type() == x.scalar_type() && bb->scalar_type() == x.scalar_type() &&
                  gb->dim() == 1 && bb->dim() == 1 && gb->size(0) == N && bb->size(0) == N), op, "both biases must be (N,) with x dtype");
    const int kind = (int)integer(a[7]);
    const bool with_output = truth(a[8]), ordered = truth(a[9]);
    at::Tensor out;
    Quant q;
    {
      const Released released;
      const c10::cuda::OptionalCUDAGuard guard(x.device());
      const at::Tensor xc = dense(x), gc = dense(g), uc = dense(u);
      at::Tensor gbc, bbc;
      if (ub) { gbc = dense(*gb); bbc = dense(*bb); }
      out = empty({B, N}, x.scalar_type(), x);
      if (ordered) {
        check(kind == 0, op, "the ordered form has no output_quant");
        check_status(qx_cuda_decode_swiglu_ordered(at::cuda::getCurrentCUDAStream().stream(), ptr(xc), ptr(gc), ptr(uc), ptr(gbc), ptr(bbc),
                                                   ptr(out), B, K, N, f->name, (qx_dtype)dtype_of(x.scalar_type()), ub, nullptr, 0));
      } else {
        q = quant_outputs(x, B, N, kind);
        check_status(qx_cuda_decode_swiglu(at::cuda::getCurrentCUDAStream().stream(), ptr(xc), ptr(gc), ptr(uc), ptr(gbc), ptr(bbc),
                                           ptr(out), B, K, N, f->name, (qx_dtype)dtype_of(x.scalar_type()), ub, kind, ptr(q.codes),
                                           (float*)ptr(q.scale), nullptr, 0));
      }
    }
    return quant_result(out, kind, q, with_output);
  });
}

// (h, Wq, bias or None, V, K, format, mode, topk, temperature, seed, top_p)
PyObject* lm_head_sample_q(PyObject*, PyObject* const* a, Py_ssize_t) {
  return guarded([&]() -> PyObject* {
    static const char* op = "lm_head_sample_q";
    const at::Tensor &h = tensor(a[0], op), &w = tensor(a[1], op);
    const at::Tensor* b = tensor_or_null(a[2], op);
    const int64_t V = integer(a[3]), K = integer(a[4]), mode = integer(a[6]), topk = integer(a[7]);
    const Format* f = format_of(text(a[5]));
    const double temperature = real(a[8]), top_p = real(a[10]);
    check(h.is_cuda() && w.is_cuda() && (!b || b->is_cuda()) && dtype_of(h.scalar_type()), op,
          "inputs must be CUDA and h must be floating point");
    const bool ub = b && b->numel() > 1;
    same_device(op, h, &w);
    if (ub) same_device(op, h, b);
    check(h.dim() == 2 && h.size(1) == K, op, "h must be (T, K)");
    check(mode >= 0 && mode <= 3, op, "mode 0=argmax, 1=categorical, 2=topk, 3=topp");
    check(temperature > 0.0, op, "temperature must be positive");
    check(f != nullptr, op, "format must be q8_0, q4_0, q6_K, mxfp8, nvfp4, or mxfp4");
    check(K % f->bk == 0 && w.scalar_type() == at::kByte && w.dim() == 3 && w.size(0) == V && w.size(1) == K / f->bk && w.size(2) == f->bb,
          op, "packed weight shape does not match V/K/format");
    check(h.size(0) > 0 && V > 0 && K > 0, op, "T, V, and K must be positive");
    if (mode >= 2) {
      check(topk >= 1 && topk <= 64, op, "k must be in [1, 64]");
      check(mode != 3 || (top_p > 0.0 && top_p <= 1.0), op, "topp requires top_p in (0, 1]");
      check(topk <= V, op, "k must be <= vocab size V");
    }
    if (ub) check(b->numel() == V, op, "bias must be (V,)");
    const uint32_t seed = (uint32_t)PyLong_AsUnsignedLongLongMask(a[9]);
    at::Tensor ids;
    {
      const Released released;
      const c10::cuda::OptionalCUDAGuard guard(h.device());
      const at::Tensor hc = dense(h), wc = dense(w);
      at::Tensor bc;
      if (ub) bc = b->to(at::kFloat).contiguous();
      const int64_t T = h.size(0);
      const cudaStream_t st = at::cuda::getCurrentCUDAStream().stream();
      ids = empty({T}, at::kInt, h);
      const size_t bytes = qx_cuda_lm_head_workspace_bytes(T, V, K, (int)mode, (int)topk);
      const at::Tensor ws = workspace(h.device(), st, bytes);
      check_status(qx_cuda_lm_head_sample_q(st, ptr(hc), ptr(wc), (const float*)ptr(bc), (int32_t*)ptr(ids), ptr(ws), bytes, T, V, K,
                                            f->name, (qx_dtype)dtype_of(h.scalar_type()), (int)mode, (int)topk, temperature, seed, top_p));
    }
    return wrap(ids);
  });
}

// (x, residual, weight, eps, quant, static_scale, group, ue8m0, op) -> (y or None, codes or None, added, scale or None)
PyObject* rms_norm_add(PyObject*, PyObject* const* a, Py_ssize_t) {
  return guarded([&]() -> PyObject* {
    const char* op = text(a[8]);
    const at::Tensor &x = tensor(a[0], op), &r = tensor(a[1], op), &w = tensor(a[2], op);
    check(x.is_cuda() && dtype_of(x.scalar_type()) && x.dim() >= 1 && x.numel() > 0, op, "x must be a non-empty CUDA fp32/fp16/bf16 tensor");
    const int64_t D = x.size(-1), rows = x.numel() / D;
    check(r.sizes() == x.sizes() && r.scalar_type() == x.scalar_type() && w.dim() == 1 && w.size(0) == D && w.scalar_type() == x.scalar_type(),
          op, "residual must match x, weight must be (D,) with x dtype");
    same_device(op, x, &r); same_device(op, x, &w);
    const int quant = (int)integer(a[4]), group = (int)integer(a[6]);
    const double eps = real(a[3]), static_scale = real(a[5]);
    const bool ue8m0 = truth(a[7]);
    at::Tensor added, y, codes, scale;
    {
      const Released released;
      const c10::cuda::OptionalCUDAGuard guard(x.device());
      const at::Tensor xc = dense(x), rc = dense(r), wc = dense(w);
      added = at::empty_like(xc);
      if (quant == 0) y = at::empty_like(xc);
      else codes = empty(x.sizes(), quant == 3 || quant == 5 ? at::kChar : at::kByte, x);
      if (quant == 2 || quant == 3) {
        scale = empty(x.sizes().slice(0, x.dim() - 1), at::kFloat, x);
      } else if (quant >= 4) {
        std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
        shape.back() = D / group;
        scale = empty(shape, at::kFloat, x);
      }
      check_status(qx_cuda_rms_norm_add(at::cuda::getCurrentCUDAStream().stream(), ptr(xc), ptr(rc), ptr(wc), ptr(y), ptr(codes),
                                        ptr(added), (float*)ptr(scale), rows, D, (qx_dtype)dtype_of(x.scalar_type()), eps, quant,
                                        static_scale, group, ue8m0));
    }
    return Py_BuildValue("(NNNN)", wrap_or_none(y), wrap_or_none(codes), wrap(added), wrap_or_none(scale));
  });
}

// (x, gate, act, alpha, limit, quant, group, ue8m0, op) -> (codes, scale)
PyObject* silu_mul_quant(PyObject*, PyObject* const* a, Py_ssize_t) {
  return guarded([&]() -> PyObject* {
    const char* op = text(a[8]);
    const int64_t act = integer(a[2]);
    check(act >= 0, op, "act must be 'swiglu' or 'swiglu_oai'");
    const at::Tensor &x = tensor(a[0], op), &g = tensor(a[1], op);
    check(x.is_cuda() && dtype_of(x.scalar_type()) && x.dim() >= 1 && x.numel() > 0 && g.sizes() == x.sizes() &&
              g.scalar_type() == x.scalar_type(), op, "x and gate must be matching non-empty CUDA float tensors");
    same_device(op, x, &g);
    const int64_t D = x.size(-1), rows = x.numel() / D;
    const int quant = (int)integer(a[5]), group = (int)integer(a[6]);
    if (quant == 4) check(group > 0 && group % 4 == 0 && D % group == 0, op, "group_size must be a multiple of 4 that divides D");
    const double alpha = real(a[3]), limit = real(a[4]);
    const bool ue8m0 = truth(a[7]);
    at::Tensor codes, scale;
    {
      const Released released;
      const c10::cuda::OptionalCUDAGuard guard(x.device());
      const at::Tensor xc = dense(x), gc = dense(g);
      codes = empty(x.sizes(), quant == 3 ? at::kChar : at::kByte, x);
      if (quant == 4) {
        std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
        shape.back() = D / group;
        scale = empty(shape, at::kFloat, x);
      } else {
        scale = empty(x.sizes().slice(0, x.dim() - 1), at::kFloat, x);
      }
      check_status(qx_cuda_silu_mul_quant(at::cuda::getCurrentCUDAStream().stream(), ptr(xc), ptr(gc), ptr(codes), (float*)ptr(scale),
                                          rows, D, (qx_dtype)dtype_of(x.scalar_type()), (int)act, alpha, limit, quant, group, ue8m0));
    }
    return Py_BuildValue("(NN)", wrap(codes), wrap(scale));
  });
}

// (codes, scales, biases or None, x, bits, group_size, scale_dtype, symmetric, layout, op, gemv_only)
PyObject* base_q_matmul(PyObject*, PyObject* const* a, Py_ssize_t) {
  return guarded([&]() -> PyObject* {
    const char* op = text(a[9]);
    const int64_t bits = integer(a[4]), group = integer(a[5]);
    const char *sd = text(a[6]), *layout = text(a[8]);
    const bool sym = truth(a[7]);
    // the descriptor and storage checks of kernels/common/base_q_descriptor.h:34-68 and base_q.cpp:57-131
    if (!(bits == 2 || bits == 3 || bits == 4 || bits == 5 || bits == 6 || bits == 8)) fail("BaseQN: bits must be one of 2, 3, 4, 5, 6, or 8");
    if (!(group == 32 || group == 64 || group == 128)) fail("BaseQN: group_size must be 32, 64, or 128");
    const bool bf = !std::strcmp(sd, "bf16") || !std::strcmp(sd, "bfloat16"), hf = !std::strcmp(sd, "f16") || !std::strcmp(sd, "float16");
    const bool e8 = !std::strcmp(sd, "e8m0"), e4 = !std::strcmp(sd, "e4m3");
    if (!(bf || hf || e8 || e4)) fail("BaseQN: scale_dtype must be bf16, f16, e8m0, or e4m3");
    if (e4 && bits != 8) fail("BaseQN: e4m3 scale storage is valid only for q8");
    const std::string lane = "metal_lane_strided_q" + std::to_string(bits);
    if (std::strcmp(layout, "metal") && std::strcmp(layout, "metal_lane_strided") && lane != layout)
      fail("BaseQN: layout must be metal or metal_lane_strided_q" + std::to_string(bits));
    const at::Tensor &c = tensor(a[0], op), &s = tensor(a[1], op), &x = tensor(a[3], op);
    const at::Tensor* b = tensor_or_null(a[2], op);
    const at::ScalarType st = bf ? at::kBFloat16 : hf ? at::kHalf : at::kByte;
    check(c.is_cuda() && c.scalar_type() == at::kByte && c.dim() == 2, op, "codes must be uint8 (rows, packed_bytes)");
    check(s.is_cuda() && s.scalar_type() == st && s.dim() == 2, op, "scales must be a rank-2 tensor with the declared scale_dtype");
    check(s.size(0) > 0 && s.size(1) > 0 && s.size(0) == c.size(0), op, "codes/scales rows and group count must be positive and match");
    const int64_t K = s.size(1) * group, rows = c.size(0);
    check(K * bits % 8 == 0 && c.size(1) == K * bits / 8, op, "codes.shape[1] must equal columns * bits / 8");
    check(sym || b, op, "biases are required for asymmetric BaseQN");
    check(!b || (b->scalar_type() == s.scalar_type() && b->sizes() == s.sizes()), op, "biases must match scales shape and dtype");
    same_device(op, c, &s); same_device(op, c, b);
    check(x.is_cuda() && x.dim() == 2 && x.size(0) == K, op, "x must be (K, M) with K matching the packed weights");
    if (truth(a[10]) && x.size(1) != 1) fail("base_qgemv: x must be (K, 1)");
    if (!dtype_of(x.scalar_type())) fail("BaseQN matmul: x must be float16, bfloat16, or float32");
    if (x.size(1) <= 0) fail("BaseQN matmul: M must be positive");
    same_device(op, c, &x);
    const int64_t M = x.size(1);
    at::Tensor out;
    {
      const Released released;
      const c10::cuda::OptionalCUDAGuard guard(x.device());
      const at::Tensor cc = dense(c), sc = dense(s), xc = dense(x);
      at::Tensor bc, ws;
      if (b) bc = dense(*b);
      out = empty({rows, M}, x.scalar_type(), x);
      const cudaStream_t stream = at::cuda::getCurrentCUDAStream().stream();
      const qx_dtype dt = (qx_dtype)dtype_of(x.scalar_type());
      const size_t bytes = qx_cuda_base_q_workspace_bytes(K, M, 0, dt);
      if (bytes) ws = workspace(x.device(), stream, bytes);
      const qx_base_q_planes planes{ptr(cc), ptr(sc), ptr(bc)};
      const qx_base_q_desc desc{(int32_t)bits, (int32_t)group, sd, sym, layout};
      check_status(qx_cuda_base_qgemm(stream, &planes, &desc, ptr(xc), ptr(out), rows, K, M, dt, ptr(ws), bytes));
    }
    return wrap(out);
  });
}

// (device index, bytes) -> uint8 tensor of at least that size for calls on the current stream
PyObject* stream_workspace(PyObject*, PyObject* const* a, Py_ssize_t) {
  return guarded([&]() -> PyObject* {
    const at::Device device(at::kCUDA, (c10::DeviceIndex)integer(a[0]));
    const int64_t bytes = integer(a[1]);
    at::Tensor ws;
    {
      const Released released;
      const c10::cuda::OptionalCUDAGuard guard(device);
      ws = workspace(device, at::cuda::getCurrentCUDAStream(device.index()).stream(), (size_t)bytes);
    }
    return wrap(ws);
  });
}

PyObject* set_status_handler(PyObject*, PyObject* f) {
  Py_XINCREF(f);
  Py_XSETREF(g_raise_status, f);
  Py_RETURN_NONE;
}

template <PyObject* (*F)(PyObject*, PyObject* const*, Py_ssize_t), int N>
PyObject* counted(PyObject* m, PyObject* const* a, Py_ssize_t n) {
  if (n != N) { PyErr_SetString(PyExc_TypeError, "wrong number of arguments"); return nullptr; }
  return F(m, a, n);
}
#define QX_METHOD(name, n) {#name, (PyCFunction)(void (*)(void))counted<name, n>, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    QX_METHOD(decode_linear_epilogue, 11),
    QX_METHOD(decode_linear_partial, 3),
    QX_METHOD(decode_swiglu, 10),
    QX_METHOD(lm_head_sample_q, 11),
    QX_METHOD(rms_norm_add, 9),
    QX_METHOD(silu_mul_quant, 9),
    QX_METHOD(base_q_matmul, 11),
    QX_METHOD(stream_workspace, 2),
    {"set_status_handler", set_status_handler, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_qx_native", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__qx_native() { return PyModule_Create(&module); }
