// The per-call host path of the operators as a CPython extension (awq_b200/_native.so): argument
// checks, output allocation, the choice of weight layout and the call into the C ABI of
// libawq_b200.so, without interpreter work in between.
//
// What bounds it: a decode-size call keeps the GPU busy for 4 - 20 us, so the time until the launch
// is on the critical path of an eager loop.  The same steps in Python (tensor attribute reads, shape
// tuples, ctypes conversion of 14 arguments) took 22 us for one linear of K 2048 x N 5120 at M = 1 and
// 44 us for a router + experts pair; tensors are read here through their C++ objects instead.
//
// The functions take positional arguments only (METH_FASTCALL); the signatures users see are those
// of ops.py and linear.py.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <map>
#include <utility>
#include <vector>

#include "../../include/awq_b200.h"

namespace {

// Thrown with the Python error already set.
struct PyFailure {};

[[noreturn]] void fail(PyObject* type, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  PyErr_FormatV(type, fmt, ap);
  va_end(ap);
  throw PyFailure{};
}

// A negative status of the C ABI, raised by _lib.check so that the exception types live in one place.
[[noreturn]] void fail_status(const char* fn, int rc) {
  PyObject* mod = PyImport_ImportModule("awq_b200._lib");
  if (mod != nullptr) {
    PyObject* r = PyObject_CallMethod(mod, "check", "si", fn, rc);
    Py_XDECREF(r);
    Py_DECREF(mod);
  }
  if (!PyErr_Occurred()) PyErr_Format(PyExc_RuntimeError, "%s failed (code %d)", fn, rc);
  throw PyFailure{};
}

const char* dtype_name(at::ScalarType t) {
  switch (t) {
    case at::kInt: return "torch.int32";
    case at::kHalf: return "torch.float16";
    case at::kFloat: return "torch.float32";
    case at::kByte: return "torch.uint8";
    case at::kLong: return "torch.int64";
    case at::kBFloat16: return "torch.bfloat16";
    default: return c10::toString(t);
  }
}

const at::Tensor& tensor_arg(PyObject* o, const char* name) {
  if (!THPVariable_Check(o)) fail(PyExc_TypeError, "%s must be a torch.Tensor", name);
  return THPVariable_Unpack(o);
}

void require_kind(const at::Tensor& t, const char* name, at::ScalarType dtype, int ndim) {
  if (!t.is_cuda())
    fail(PyExc_ValueError, "%s must live on a CUDA device (there is no CPU path)", name);
  if (t.scalar_type() != dtype)
    fail(PyExc_ValueError, "%s must be %s, got %s", name, dtype_name(dtype),
         dtype_name(t.scalar_type()));
  if (ndim >= 0 && t.dim() != ndim)
    fail(PyExc_ValueError, "%s must have %d dimensions, got %d", name, ndim, (int)t.dim());
}

void require(const at::Tensor& t, const char* name, at::ScalarType dtype, int ndim) {
  require_kind(t, name, dtype, ndim);
  if (!t.is_contiguous()) fail(PyExc_ValueError, "%s must be contiguous", name);
}

const at::Tensor& require_arg(PyObject* o, const char* name, at::ScalarType dtype, int ndim) {
  const at::Tensor& t = tensor_arg(o, name);
  require(t, name, dtype, ndim);
  return t;
}

long long int_arg(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw PyFailure{};
  return v;
}

bool truth_arg(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw PyFailure{};
  return v != 0;
}

void expect_args(const char* fn, Py_ssize_t n, Py_ssize_t want) {
  if (n != want) fail(PyExc_TypeError, "%s takes %zd arguments, got %zd", fn, want, n);
}

void* stream_now() { return c10::cuda::getCurrentCUDAStream().stream(); }

template <typename... Sizes>
at::Tensor empty_like_device(const at::Tensor& ref, at::ScalarType dtype, Sizes... sizes) {
  const int64_t dims[] = {(int64_t)sizes...};
  return at::detail::empty_cuda(at::IntArrayRef(dims, sizeof...(sizes)), dtype, ref.device(),
                                std::nullopt);
}

PyObject* wrap(at::Tensor t) { return THPVariable_Wrap(std::move(t)); }

// ---- scratch: one buffer per (device, stream), one per call while the stream is captured ----------
// The partial tiles of a call and the flags that announce them lie in its scratch, so calls that may
// overlap must not share one.  Calls of one stream never overlap; captured on one stream, they do as
// soon as their graphs are replayed on several.  A captured call therefore takes its scratch from the
// graph's own memory pool and gives it back to the pool at the end of the call, like any temporary
// tensor of a captured operator.
constexpr int64_t kMinWorkspace = 24 << 20;  // covers every dense kernel's scratch need

// Callers hold the GIL, which is what makes the table safe with several threads.  Growing replaces a
// buffer; the old one goes back to the caching allocator, which hands it on in stream order.
std::map<std::pair<int, void*>, at::Tensor>& workspaces() {
  // never destroyed: tensors must not be freed after the interpreter and CUDA are gone
  static auto* w = new std::map<std::pair<int, void*>, at::Tensor>;
  return *w;
}

at::Tensor workspace(const at::Device& device, int64_t nbytes) {
  const int dev = device.has_index() ? device.index() : c10::cuda::current_device();
  const auto fresh = [&](int64_t size) {
    return at::detail::empty_cuda({size}, at::kByte, at::Device(at::kCUDA, dev), std::nullopt);
  };
  if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None)
    return fresh(nbytes);
  at::Tensor& ws = workspaces()[{dev, stream_now()}];
  if (!ws.defined() || ws.numel() < nbytes) ws = fresh(nbytes > kMinWorkspace ? nbytes : kMinWorkspace);
  return ws;
}

// ---- dense linear -----------------------------------------------------------------------------

struct AwqDims {
  int64_t k, n, group;
};

AwqDims awq_dims(const at::Tensor& qweight, const at::Tensor& scales, const at::Tensor& qzeros,
                 bool kmajor) {
  require(qweight, "qweight", at::kInt, 2);
  require(scales, "scales", at::kHalf, 2);
  require(qzeros, "qzeros", at::kInt, 2);
  const int64_t k = qweight.size(0);
  int64_t words = qweight.size(1);
  if (kmajor) {
    // output of awq_repack_kmajor: [K, ceil(N / 256) * 256 / 8], the true N is that of scales
    const int64_t n = scales.size(1);
    if (n % 8 != 0 || words != (n + 255) / 256 * 32)
      fail(PyExc_ValueError, "qweight is not the k-major copy of a matrix with scales' width");
    words = n / 8;
  }
  const int64_t n = words * 8, groups = scales.size(0);
  if (groups == 0 || k == 0 || k % groups != 0)
    fail(PyExc_ValueError, "K=%lld is not a multiple of the number of groups %lld", (long long)k,
         (long long)groups);
  if (scales.size(1) != n)
    fail(PyExc_ValueError, "scales must be [%lld, %lld], got (%lld, %lld)", (long long)groups,
         (long long)n, (long long)scales.size(0), (long long)scales.size(1));
  if (qzeros.size(0) != groups || qzeros.size(1) != words)
    fail(PyExc_ValueError, "qzeros must be [%lld, %lld], got (%lld, %lld)", (long long)groups,
         (long long)words, (long long)qzeros.size(0), (long long)qzeros.size(1));
  return {k, n, k / groups};
}

// y = x @ dequant(qweight) (+ bias) into `out`, both contiguous with m rows.
void gemm_into(const at::Tensor& x, int64_t m, const at::Tensor& qweight, const at::Tensor& scales,
               const at::Tensor& qzeros, const at::Tensor* bias, const AwqDims& d, int kernel,
               const at::Tensor& out) {
  if (m == 0) return;
  const size_t need = awq_b200_gemm_workspace_bytes((int)m, (int)d.n, (int)d.k, (int)d.group, kernel);
  at::Tensor ws;
  if (need > 0) ws = workspace(x.device(), (int64_t)need);
  void* stream = stream_now();
  const void* xp = x.const_data_ptr();
  const void* wp = qweight.const_data_ptr();
  const void* sp = scales.const_data_ptr();
  const void* zp = qzeros.const_data_ptr();
  const void* bp = bias ? bias->const_data_ptr() : nullptr;
  void* op = out.data_ptr();
  void* wsp = need > 0 ? ws.data_ptr() : nullptr;
  const size_t wsn = need > 0 ? (size_t)ws.numel() : 0;
  int rc;
  Py_BEGIN_ALLOW_THREADS
  rc = awq_b200_gemm(xp, wp, sp, zp, bp, op, (int)m, (int)d.n, (int)d.k, (int)d.group, kernel, wsp,
                     wsn, stream);
  Py_END_ALLOW_THREADS
  if (rc != AWQ_B200_OK) fail_status("awq_b200_gemm", rc);
}

const at::Tensor* bias_arg(PyObject* o, int64_t n) {
  if (o == Py_None) return nullptr;
  const at::Tensor& b = require_arg(o, "bias", at::kHalf, 1);
  if (b.size(0) != n) fail(PyExc_ValueError, "bias must have %lld elements", (long long)n);
  return &b;
}

// gemm(input, qweight, scales, qzeros, bias | None, kernel, out | None)
PyObject* gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    expect_args("gemm", n, 7);
    const int kernel = (int)int_arg(a[5]);
    const at::Tensor& qweight = tensor_arg(a[1], "qweight");
    const at::Tensor& scales = tensor_arg(a[2], "scales");
    const at::Tensor& qzeros = tensor_arg(a[3], "qzeros");
    const AwqDims d = awq_dims(qweight, scales, qzeros, kernel == AWQ_B200_KERNEL_Q8);
    const at::Tensor& x = require_arg(a[0], "input", at::kHalf, 2);
    if (x.size(1) != d.k)
      fail(PyExc_ValueError, "input has K=%lld, qweight has K=%lld", (long long)x.size(1),
           (long long)d.k);
    const at::Tensor* bias = bias_arg(a[4], d.n);
    const int64_t m = x.size(0);
    if (a[6] != Py_None) {
      const at::Tensor& out = require_arg(a[6], "out", at::kHalf, 2);
      if (out.size(0) != m || out.size(1) != d.n)
        fail(PyExc_ValueError, "out must be [%lld, %lld]", (long long)m, (long long)d.n);
      gemm_into(x, m, qweight, scales, qzeros, bias, d, kernel, out);
      Py_INCREF(a[6]);
      return a[6];
    }
    at::Tensor out = empty_like_device(x, at::kHalf, m, d.n);
    gemm_into(x, m, qweight, scales, qzeros, bias, d, kernel, out);
    return wrap(std::move(out));
  } catch (const PyFailure&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// linear(x, qweight, scales, qzeros, bias | None): x of any rank
PyObject* linear(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    expect_args("linear", n, 5);
    const at::Tensor& x_arg = tensor_arg(a[0], "input");
    const at::Tensor& qweight = tensor_arg(a[1], "qweight");
    const at::Tensor& scales = tensor_arg(a[2], "scales");
    const at::Tensor& qzeros = tensor_arg(a[3], "qzeros");
    require_kind(x_arg, "input", at::kHalf, -1);
    if (x_arg.dim() < 1) fail(PyExc_ValueError, "input must have at least one dimension");
    const int64_t kx = x_arg.size(-1);
    const int64_t m = kx > 0 ? x_arg.numel() / kx : 0;
    const AwqDims d = awq_dims(qweight, scales, qzeros, false);
    if (kx != d.k)
      fail(PyExc_ValueError, "input has K=%lld, qweight has K=%lld", (long long)kx, (long long)d.k);
    const at::Tensor* bias = bias_arg(a[4], d.n);
    const bool dense = x_arg.is_contiguous();
    const at::Tensor kept = dense ? at::Tensor() : x_arg.contiguous();
    const at::Tensor& x = dense ? x_arg : kept;
    c10::SmallVector<int64_t, 4> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = d.n;
    at::Tensor out = at::detail::empty_cuda(shape, at::kHalf, x.device(), std::nullopt);
    gemm_into(x, m, qweight, scales, qzeros, bias, d, AWQ_B200_KERNEL_AUTO, out);
    return wrap(std::move(out));
  } catch (const PyFailure&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// dequantize(qweight, scales, qzeros)
PyObject* dequantize(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    expect_args("dequantize", n, 3);
    const at::Tensor& qweight = tensor_arg(a[0], "qweight");
    const at::Tensor& scales = tensor_arg(a[1], "scales");
    const at::Tensor& qzeros = tensor_arg(a[2], "qzeros");
    const AwqDims d = awq_dims(qweight, scales, qzeros, false);
    at::Tensor out = empty_like_device(qweight, at::kHalf, d.k, d.n);
    const int rc =
        awq_b200_dequantize(qweight.const_data_ptr(), scales.const_data_ptr(),
                            qzeros.const_data_ptr(), out.data_ptr(), (int)d.k, (int)d.n,
                            (int)d.group, stream_now());
    if (rc != AWQ_B200_OK) fail_status("awq_b200_dequantize", rc);
    return wrap(std::move(out));
  } catch (const PyFailure&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// ---- MoE ------------------------------------------------------------------------------------------

// topk(hidden_states, gating, topk, renormalize) -> (weights, ids, token_expert_indices)
PyObject* topk(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    expect_args("topk", n, 4);
    const at::Tensor& x = tensor_arg(a[0], "hidden_states");
    const at::Tensor& g = tensor_arg(a[1], "gating_output");
    if (x.dim() < 1 || g.dim() < 1 || x.size(0) != g.size(0))
      fail(PyExc_ValueError, "Number of tokens mismatch");
    const at::ScalarType dt = g.scalar_type();
    if (dt != at::kFloat && dt != at::kHalf)
      fail(PyExc_ValueError, "gating_output must be float32 or float16");
    require(g, "gating_output", dt, 2);
    const int64_t t = g.size(0), e = g.size(1), k = int_arg(a[2]);
    at::Tensor w = empty_like_device(g, at::kFloat, t, k);
    at::Tensor ids = empty_like_device(g, at::kInt, t, k);
    at::Tensor tok = empty_like_device(g, at::kInt, t, k);
    if (t > 0) {
      const int renorm = truth_arg(a[3]);
      const void* gp = g.const_data_ptr();
      float* wp = w.data_ptr<float>();
      int32_t* ip = ids.data_ptr<int32_t>();
      int32_t* tp = tok.data_ptr<int32_t>();
      void* stream = stream_now();
      int rc;
      Py_BEGIN_ALLOW_THREADS
      rc = awq_b200_topk_softmax(gp, dt == at::kFloat ? 0 : 1, (int)t, (int)e, (int)k, renorm, wp, ip,
                                 tp, stream);
      Py_END_ALLOW_THREADS
      if (rc != AWQ_B200_OK) fail_status("awq_b200_topk_softmax", rc);
    }
    PyObject* r = PyTuple_New(3);
    if (r == nullptr) return nullptr;
    PyTuple_SET_ITEM(r, 0, wrap(std::move(w)));
    PyTuple_SET_ITEM(r, 1, wrap(std::move(ids)));
    PyTuple_SET_ITEM(r, 2, wrap(std::move(tok)));
    return r;
  } catch (const PyFailure&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

struct Expert {
  const at::Tensor *q, *s, *z;
};

Expert expert_arg(PyObject* o, const char* nq, const char* ns, const char* nz) {
  if (!PyTuple_Check(o) || PyTuple_GET_SIZE(o) != 3)
    fail(PyExc_ValueError, "expert weights are (qweight, scales, qzeros) triples");
  return {&require_arg(PyTuple_GET_ITEM(o, 0), nq, at::kInt, 3),
          &require_arg(PyTuple_GET_ITEM(o, 1), ns, at::kHalf, 3),
          &require_arg(PyTuple_GET_ITEM(o, 2), nz, at::kInt, 3)};
}

bool has_shape(const at::Tensor& t, int64_t a, int64_t b, int64_t c) {
  return t.size(0) == a && t.size(1) == b && t.size(2) == c;
}

// experts(hidden_states, w1 triple, w2 triple, topk_weights, topk_ids, inplace, global_num_experts,
//         expert_map | None, group_size, w1_decode | None, w2_decode | None, direct_max_pairs)
PyObject* experts(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    expect_args("experts", n, 12);
    const at::Tensor& x = require_arg(a[0], "hidden_states", at::kHalf, 2);
    const Expert w1 = expert_arg(a[1], "w1.qweight", "w1.scales", "w1.qzeros");
    const Expert w2 = expert_arg(a[2], "w2.qweight", "w2.scales", "w2.qzeros");
    const at::Tensor& tw = require_arg(a[3], "topk_weights", at::kFloat, 2);
    const at::Tensor& ids = require_arg(a[4], "topk_ids", at::kInt, 2);
    const int64_t t = x.size(0), h = x.size(1), e = w1.q->size(0), inter = w2.q->size(1);
    const int64_t k = ids.size(1), g = int_arg(a[8]), global_e = int_arg(a[6]);
    if (g <= 0) fail(PyExc_ValueError, "group_size must be positive");
    if (!has_shape(*w1.q, e, h, 2 * inter / 8) || !has_shape(*w2.q, e, inter, h / 8))
      fail(PyExc_ValueError, "expert weight shapes do not match hidden/intermediate sizes");
    if (!has_shape(*w1.s, e, h / g, 2 * inter) || !has_shape(*w1.z, e, h / g, 2 * inter / 8))
      fail(PyExc_ValueError, "w1 scales/zeros shapes do not match group size");
    if (!has_shape(*w2.s, e, inter / g, h) || !has_shape(*w2.z, e, inter / g, h / 8))
      fail(PyExc_ValueError, "w2 scales/zeros shapes do not match group size");
    if (tw.size(0) != t || tw.size(1) != k || ids.size(0) != t)
      fail(PyExc_ValueError, "topk_weights / topk_ids shape mismatch");
    const at::Tensor* emap = nullptr;
    if (a[7] != Py_None) emap = &require_arg(a[7], "expert_map", at::kInt, 1);
    if (global_e != -1 && global_e != e && emap == nullptr)
      fail(PyExc_ValueError, "global_num_experts differs from the stacked expert count");
    if ((a[9] == Py_None) != (a[10] == Py_None))
      fail(PyExc_ValueError, "w1_decode and w2_decode go together");
    if (a[9] != Py_None) {
      // checked for the caller's sake; the expert kernels read the checkpoint layout
      const at::Tensor& d1 = require_arg(a[9], "w1_decode", at::kInt, 3);
      const at::Tensor& d2 = require_arg(a[10], "w2_decode", at::kInt, 3);
      if (d1.sizes() != w1.q->sizes() || d2.sizes() != w2.q->sizes())
        fail(PyExc_ValueError, "decode-layout copies must have the shapes of the qweights");
    }
    const bool inplace = truth_arg(a[5]);
    at::Tensor fresh;
    if (!inplace) fresh = empty_like_device(x, at::kHalf, t, h);
    const at::Tensor& out = inplace ? x : fresh;
    if (t > 0) {
      const int T = (int)t, K = (int)k, H = (int)h, I = (int)inter, G = (int)g;
      const int ng = (int)(global_e == -1 ? e : global_e);
      const int64_t pairs = t * k;
      const int block = awq_b200_moe_block_size(T, K, ng, H, I, G);
      const at::Tensor ws =
          workspace(x.device(), (int64_t)awq_b200_moe_workspace_bytes(T, K, ng, H, I));
      // A handful of pairs: one row block per pair straight from topk_ids, no permutation (3 to 5 us
      // less).  Up to half as many pairs as experts, where most pairs have their expert to themselves:
      // the permutation makes an expert's matrices be read once for all of its rows.  64 experts of
      // 4096 x 1536, direct / permuted: 20.5 / 25.0 us at 4 pairs, 41.9 / 46.5 at 16, 64.8 / 64.4 at 32;
      // 128 of 2048 x 768: 17.3 / 21.1 at 8, 42.3 / 45.5 at 64.  (The last condition: the scratch bound of
      // awq_b200_moe_workspace_bytes covers one 8-row block per pair only while the pairs are few
      // compared with the experts.)
      const bool direct = block == 8 && pairs <= int_arg(a[11]) && 2 * pairs <= ng &&
                          pairs * 8 <= awq_b200_moe_sorted_capacity(pairs, ng, 16);
      int64_t cap = pairs * 8;
      int flags;
      at::Tensor tables;  // sorted_ids [cap] | expert_ids [nblk] | num_post [1]; direct: local ids
      const int32_t *sorted = nullptr, *blocks = ids.const_data_ptr<int32_t>(), *post = nullptr;
      void* stream = stream_now();
      const int32_t* map = emap ? emap->const_data_ptr<int32_t>() : nullptr;
      int rc = AWQ_B200_OK;
      if (!direct) {
        flags = emap ? 1 : 0;
        cap = awq_b200_moe_sorted_capacity(pairs, ng, block);
        const int64_t nblk = (cap + block - 1) / block;
        tables = empty_like_device(x, at::kInt, cap + nblk + 1);
        int32_t* base = tables.data_ptr<int32_t>();
        rc = awq_b200_moe_align_block_size(blocks, T, K, ng, block, map, base, cap, base + cap,
                                           base + cap + nblk, stream);
        if (rc != AWQ_B200_OK) fail_status("awq_b200_moe_align_block_size", rc);
        sorted = base;
        blocks = base + cap;
        post = base + cap + nblk;
      } else {
        flags = 4;
        if (emap) {
          tables = empty_like_device(x, at::kInt, pairs);
          rc = awq_b200_moe_local_ids(blocks, T, K, ng, map, tables.data_ptr<int32_t>(), stream);
          if (rc != AWQ_B200_OK) fail_status("awq_b200_moe_local_ids", rc);
          blocks = tables.const_data_ptr<int32_t>();
          flags |= 8;
        }
      }
      void* xp = x.data_ptr();
      void* op = out.data_ptr();
      Py_BEGIN_ALLOW_THREADS
      rc = awq_b200_moe_experts(
          xp, w1.q->const_data_ptr(), w1.s->const_data_ptr(), w1.z->const_data_ptr(),
          w2.q->const_data_ptr(), w2.s->const_data_ptr(), w2.z->const_data_ptr(),
          tw.const_data_ptr<float>(), sorted, blocks, post, op, T, K, (int)e, H, I, G, block, flags,
          cap, ws.data_ptr(), (size_t)ws.numel(), stream);
      Py_END_ALLOW_THREADS
      if (rc != AWQ_B200_OK) fail_status("awq_b200_moe_experts", rc);
    }
    if (inplace) {
      Py_INCREF(a[0]);
      return a[0];
    }
    return wrap(std::move(fresh));
  } catch (const PyFailure&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

// workspace(device_index, nbytes) -> the current stream's scratch tensor, grown to nbytes
PyObject* workspace_py(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  try {
    expect_args("workspace", n, 2);
    const int dev = (int)int_arg(a[0]);
    return wrap(workspace(at::Device(at::kCUDA, (c10::DeviceIndex)dev), int_arg(a[1])));
  } catch (const PyFailure&) {
    return nullptr;
  }
  END_HANDLE_TH_ERRORS
}

#define AWQ_METHOD(name, fn) \
  { name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL, nullptr }

PyMethodDef kMethods[] = {AWQ_METHOD("gemm", gemm),
                          AWQ_METHOD("linear", linear),
                          AWQ_METHOD("dequantize", dequantize),
                          AWQ_METHOD("topk", topk),
                          AWQ_METHOD("experts", experts),
                          AWQ_METHOD("workspace", workspace_py),
                          {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "_native", "Per-call host path of the operators.", -1,
                       kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__native(void) { return PyModule_Create(&kModule); }
