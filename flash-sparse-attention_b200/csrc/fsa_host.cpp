// Native launcher of the common operator calls (module flash_sparse_attn._host): argument checks, result and workspace
// allocation through ATen and ONE call into the C ABI. The Python launchers (ops/triton/flash_dec.py, flash_fwd.py)
// do the same in Python, which took 36 us (decode) and 44 us (forward) per call on the build machine, several times
// what the kernels of a small call take; the functions here answer in a few microseconds.
//
// They take a call only when every argument is of the ordinary kind checked below and return None otherwise: the Python
// launcher then runs, raises the contract's errors, and serves the rest (gated kind, tensor subclasses, tensors on
// another device than the current one, default windows, debug outputs). Nothing is kept between calls but the function
// addresses of the library and the per-device status words.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/version.h>

#include <cmath>
#include <optional>

#include "../../include/fsa_b200.h"

namespace {

decltype(&fsa_decode) g_decode = nullptr;
decltype(&fsa_fwd) g_fwd = nullptr;
decltype(&fsa_topk_indices) g_topk = nullptr;
decltype(&fsa_pack_scales) g_pack = nullptr;
constexpr int MAX_DEVICES = 64;
at::Tensor* g_status[MAX_DEVICES] = {};  // registered by the package, one int32 word per device, never replaced
int g_sms[MAX_DEVICES] = {};

using at::Tensor;

// Held around the allocations and the launch: an allocation may wait for the device, a launch for room in the stream's
// queue, and other Python threads (one of which may have to feed what is waited for) go on meanwhile.
struct NoGil {
  PyThreadState* state = PyEval_SaveThread();
  ~NoGil() { PyEval_RestoreThread(state); }
};

// Optional tensor argument: None -> undefined. Returns false for anything but None or an exact torch.Tensor.
bool opt_tensor(PyObject* o, Tensor* t) {
  if (o == Py_None) return true;
  if (!THPVariable_CheckExact(o)) return false;
  *t = THPVariable_Unpack(o);
  return true;
}
int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kBFloat16: return FSA_DT_BF16;
    case at::kHalf: return FSA_DT_FP16;
    case at::kFloat8_e4m3fn: return FSA_DT_E4M3;
    case at::kFloat8_e5m2: return FSA_DT_E5M2;
    default: return -1;
  }
}
// The de-quantisation scales: None, one fp32 tensor of three, or a tuple of three tensors of one element and one type, which a
// kernel packs.
struct Scales {
  Tensor packed, one[3];
  bool defined() const { return packed.defined() || one[0].defined(); }
  bool get(PyObject* o) {
    if (!PyTuple_CheckExact(o)) return opt_tensor(o, &packed);
    if (PyTuple_GET_SIZE(o) != 3) return false;
    for (int i = 0; i < 3; ++i)
      if (PyTuple_GET_ITEM(o, i) == Py_None || !opt_tensor(PyTuple_GET_ITEM(o, i), &one[i])) return false;
    return true;
  }
  int type() const { return one[0].scalar_type() == at::kFloat ? FSA_DT_F32 : dtype_code(one[0].scalar_type()); }
  bool ok(const at::Device& dev) const {
    if (packed.defined())
      return packed.scalar_type() == at::kFloat && packed.numel() == 3 && packed.device() == dev && packed.is_contiguous();
    for (const Tensor& t : one)
      if (t.scalar_type() != one[0].scalar_type() || t.numel() != 1 || t.device() != dev) return false;
    return g_pack && type() >= 0 && type() != FSA_DT_E4M3 && type() != FSA_DT_E5M2;
  }
  int pack(cudaStream_t stream) {
    if (!one[0].defined()) return FSA_OK;
    packed = at::empty({3}, one[0].options().dtype(at::kFloat));
    return g_pack(one[0].data_ptr(), one[1].data_ptr(), one[2].data_ptr(), type(), packed.data_ptr<float>(), stream);
  }
};
bool opt_double(PyObject* o, double dflt, double* v) {
  if (o == Py_None) {
    *v = dflt;
    return true;
  }
  if (PyFloat_CheckExact(o)) {
    *v = PyFloat_AS_DOUBLE(o);
    return true;
  }
  if (PyLong_CheckExact(o)) {
    *v = PyLong_AsDouble(o);
    if (!PyErr_Occurred()) return true;
    PyErr_Clear();
  }
  return false;
}
bool get_int(PyObject* o, int64_t* v) {
  if (!PyLong_CheckExact(o)) return false;
  int overflow = 0;
  *v = PyLong_AsLongLongAndOverflow(o, &overflow);
  return !overflow && *v >= 0 && *v <= INT32_MAX;
}

bool is_fp8(int code) { return code == FSA_DT_E4M3 || code == FSA_DT_E5M2; }

// An int32 vector / matrix on the device with unit inner stride (undefined passes).
bool int_ok(const Tensor& t, const at::Device& dev, int64_t ndim) {
  return !t.defined() || (t.scalar_type() == at::kInt && t.device() == dev && t.dim() == ndim &&
                          (t.size(ndim - 1) <= 1 || t.stride(ndim - 1) == 1));
}
template <typename T>
T* ptr(const Tensor& t) {
  return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr;
}

// q, k, v and the scales: one device (the current one), one type the kernels take as it is, a head size they take.
// Returns the type code or -1.
int check_qkv(const Tensor& q, const Tensor& k, const Tensor& v, const Scales& scale, int64_t hq, int64_t hkv, int64_t d) {
  if (!q.is_cuda() || k.device() != q.device() || v.device() != q.device()) return -1;
  const int dev = q.device().index();
  if (dev < 0 || dev >= MAX_DEVICES || !g_status[dev] || c10::cuda::current_device() != dev) return -1;
  const int code = dtype_code(q.scalar_type());
  if (code < 0 || k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type()) return -1;
  if (is_fp8(code) != scale.defined()) return -1;
  if (scale.defined() && (!scale.ok(q.device()) || d != 128)) return -1;
  if (hkv <= 0 || hq % hkv != 0 || d % 16 != 0 || d <= 0 || d > 256) return -1;
  if (q.stride(-1) != 1 || k.stride(-1) != 1 || k.sizes() != v.sizes() || k.strides() != v.strides()) return -1;
  return code;
}

// The rule of flash_dec.py::decode_num_splits.
int64_t decode_splits(int64_t batch, int64_t heads_kv, int64_t keys, int64_t sms) {
  const int64_t slots = 2 * std::max<int64_t>(sms, 1), ctas = std::max<int64_t>(batch * heads_kv, 1);
  const int64_t fill = std::min(slots / ctas, keys / 512);
  const int64_t balance = std::min<int64_t>({32, keys / 2048, (6 * slots + ctas - 1) / ctas});
  return std::max<int64_t>({1, fill, balance});
}

PyObject* none() { Py_RETURN_NONE; }

PyObject* pair(Tensor out, Tensor lse) {
  PyObject* a = THPVariable_Wrap(std::move(out));
  PyObject* b = a ? THPVariable_Wrap(std::move(lse)) : nullptr;
  PyObject* r = b ? PyTuple_Pack(2, a, b) : nullptr;
  Py_XDECREF(a);
  Py_XDECREF(b);
  return r;
}

// decode(kind, q, k, v, softmax_scale, window_sizes, softmax_threshold, is_local, num_splits, page_table, gather,
//        seqused_k, cu_seqlens_k, max_seqlen_k, out, lse, scales) -> (out, lse), an error code, or None
PyObject* decode(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 17 || !g_decode) return none();
  HANDLE_TH_ERRORS  // torch's own translation: an allocation that fails raises torch.OutOfMemoryError
    Tensor q, k, v, win, table, gather, used, cu, out, lse;
    Scales scale;
    if (a[1] == Py_None || a[2] == Py_None || a[3] == Py_None) return none();
    if (!opt_tensor(a[1], &q) || !opt_tensor(a[2], &k) || !opt_tensor(a[3], &v) || !opt_tensor(a[5], &win) ||
        !opt_tensor(a[9], &table) || !opt_tensor(a[10], &gather) || !opt_tensor(a[11], &used) ||
        !opt_tensor(a[12], &cu) || !opt_tensor(a[14], &out) || !opt_tensor(a[15], &lse) || !scale.get(a[16]))
      return none();
    int64_t kind, splits = 0, max_k = 0;
    if (!get_int(a[0], &kind)) return none();
    if (!PyBool_Check(a[7])) return none();
    const bool local = a[7] == Py_True;
    if (local != win.defined()) return none();
    const bool varlen = cu.defined();
    if (q.dim() != 3 || k.dim() != (varlen ? 3 : 4) || (varlen && (table.defined() || !get_int(a[13], &max_k)))) return none();
    const int64_t batch = q.size(0), hq = q.size(1), d = q.size(2), hkv = k.size(-2);
    if (batch <= 0 || hq <= 0 || k.size(-1) != d || v.dim() != k.dim()) return none();
    const int code = check_qkv(q, k, v, scale, hq, hkv, d);
    if (code < 0) return none();
    const at::Device dev = q.device();
    if (!int_ok(win, dev, 2) || !int_ok(table, dev, 2) || !int_ok(gather, dev, 2) || !int_ok(used, dev, 1) || !int_ok(cu, dev, 1))
      return none();
    if (win.defined() && (win.size(1) != 4 || win.size(0) < hkv)) return none();
    if (gather.defined() && gather.size(0) != batch) return none();
    if (used.defined() && used.size(0) < batch) return none();
    if (varlen && cu.size(0) != batch + 1) return none();
    int64_t page = 0, seqlen_k;
    if (table.defined()) {
      page = k.size(1);
      if ((page != 32 && page != 64 && page != 128 && page != 256) || table.size(0) != batch) return none();
      seqlen_k = table.size(1) * page;
    } else if (varlen) {
      seqlen_k = max_k;
    } else {
      if (k.size(0) != batch) return none();
      seqlen_k = k.size(1);
    }
    const auto out_type = is_fp8(code) ? at::kBFloat16 : q.scalar_type();
    if (out.defined() && (out.sizes() != q.sizes() || out.scalar_type() != out_type || out.device() != dev || out.stride(2) != 1))
      return none();
    if (lse.defined() && (lse.dim() != 2 || lse.size(0) != batch || lse.size(1) != hq || lse.scalar_type() != at::kFloat ||
                          lse.device() != dev || lse.stride(1) != 1))
      return none();
    double sm_scale, thr;
    if (!opt_double(a[4], 1.0 / std::sqrt((double)d), &sm_scale) || !opt_double(a[6], 1.0, &thr)) return none();
    const int64_t keys = gather.defined() ? gather.size(1) : seqlen_k;
    if (a[8] == Py_None)
      splits = decode_splits(batch, hkv, keys, g_sms[dev.index()]);
    else if (!get_int(a[8], &splits))
      return none();
    splits = std::max<int64_t>(splits, 1);
    int32_t* const status = ptr<int32_t>(*g_status[dev.index()]);
    std::optional<NoGil> no_gil(std::in_place);
    if (!out.defined()) out = at::empty(q.sizes(), q.options().dtype(out_type));
    if (!lse.defined()) lse = at::empty({batch, hq}, q.options().dtype(at::kFloat));

    FsaDecArgs x = {};
    Tensor partial;
    if (splits > 1) {
      partial = at::empty({splits * batch * hq * (d + 1)}, q.options().dtype(at::kFloat));
      x.out_partial = ptr<float>(partial);
      x.lse_partial = x.out_partial + splits * batch * hq * d;
    }
    x.q = q.data_ptr();
    x.k = k.data_ptr();
    x.v = v.data_ptr();
    x.out = out.data_ptr();
    x.lse = ptr<float>(lse);
    x.cu_seqlens_k = ptr<int32_t>(cu);
    x.seqused_k = ptr<int32_t>(used);
    x.page_table = ptr<int32_t>(table);
    x.gather_kv_indices = ptr<int32_t>(gather);
    x.window_sizes = ptr<int32_t>(win);
    x.status = status;
    x.q_stride_b = q.stride(0);
    x.q_stride_h = q.stride(1);
    x.k_stride_b = varlen ? 0 : k.stride(0);
    x.k_stride_s = k.stride(-3);
    x.k_stride_h = k.stride(-2);
    x.o_stride_b = out.stride(0);
    x.o_stride_h = out.stride(1);
    x.lse_stride_b = lse.stride(0);
    x.lse_stride_h = lse.stride(1);
    x.batch = (int)batch;
    x.seqlen_k = (int)seqlen_k;
    x.total_k = varlen ? (int)k.size(0) : 0;
    x.heads_q = (int)hq;
    x.heads_kv = (int)hkv;
    x.head_dim = (int)d;
    if (gather.defined()) {
      x.topk = (int)gather.size(1);
      x.gather_stride = (int)gather.stride(0);
    }
    if (table.defined()) {
      x.num_pages = (int)k.size(0);
      x.page_size = (int)page;
      x.page_table_stride = (int)table.stride(0);
    }
    x.window_stride = win.defined() ? (int)win.stride(0) : 0;
    x.num_splits = (int)splits;
    x.kind = (int)kind;
    x.dtype = code;
    x.flags = (local ? FSA_F_LOCAL : 0) | FSA_F_LOGSIGMOID | FSA_F_SCRATCH_PARTIALS;
    x.softmax_scale = (float)sm_scale;
    x.softmax_threshold = (float)thr;
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    int rc = scale.pack(stream);
    x.qkv_scale = ptr<float>(scale.packed);
    if (rc == FSA_OK) rc = g_decode(&x, stream);
    no_gil.reset();
    if (rc != FSA_OK) return PyLong_FromLong(rc);
    return pair(std::move(out), std::move(lse));
  END_HANDLE_TH_ERRORS
}

// forward(kind, q, k, v, is_causal, softmax_scale, window_sizes, softmax_threshold, is_local, num_splits, pack_gqa,
//         cu_seqlens_q, cu_seqlens_k, max_seqlen_q, max_seqlen_k, page_table, seqused_q, seqused_k, out, lse, scales)
//         -> (out, lse), an error code, or None. num_splits: what the launcher settled on (1: unsplit).
PyObject* forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 21 || !g_fwd) return none();
  HANDLE_TH_ERRORS  // torch's own translation: an allocation that fails raises torch.OutOfMemoryError
    Tensor q, k, v, win, cu_q, cu_k, table, used_q, used_k, out, lse;
    Scales scale;
    if (a[1] == Py_None || a[2] == Py_None || a[3] == Py_None) return none();
    if (!opt_tensor(a[1], &q) || !opt_tensor(a[2], &k) || !opt_tensor(a[3], &v) || !opt_tensor(a[6], &win) ||
        !opt_tensor(a[11], &cu_q) || !opt_tensor(a[12], &cu_k) || !opt_tensor(a[15], &table) ||
        !opt_tensor(a[16], &used_q) || !opt_tensor(a[17], &used_k) || !opt_tensor(a[18], &out) ||
        !opt_tensor(a[19], &lse) || !scale.get(a[20]))
      return none();
    int64_t kind, splits, max_q = 0, max_k = 0;
    if (!get_int(a[0], &kind) || !get_int(a[9], &splits) || splits < 1) return none();
    if (!PyBool_Check(a[4]) || !PyBool_Check(a[8]) || !PyBool_Check(a[10])) return none();
    const bool causal = a[4] == Py_True, local = a[8] == Py_True, pack = a[10] == Py_True;
    if (local != win.defined()) return none();
    const bool varlen = cu_q.defined();
    if (varlen != cu_k.defined() || (varlen && (table.defined() || !get_int(a[13], &max_q) || !get_int(a[14], &max_k))))
      return none();
    if (q.dim() != (varlen ? 3 : 4) || k.dim() != q.dim() || v.dim() != k.dim()) return none();
    const int64_t hq = q.size(-2), d = q.size(-1), hkv = k.size(-2);
    if (hq <= 0 || k.size(-1) != d) return none();
    const int code = check_qkv(q, k, v, scale, hq, hkv, d);
    if (code < 0 || !q.is_contiguous() || !k.is_contiguous()) return none();
    const at::Device dev = q.device();
    if (!int_ok(win, dev, 2) || !int_ok(table, dev, 2) || !int_ok(used_q, dev, 1) || !int_ok(used_k, dev, 1) ||
        !int_ok(cu_q, dev, 1) || !int_ok(cu_k, dev, 1))
      return none();
    if (win.defined() && (win.size(1) != 4 || win.size(0) < hkv)) return none();
    int64_t batch, seqlen_q, seqlen_k, total_q = 0, total_k = 0, page = 0;
    if (varlen) {
      batch = cu_q.size(0) - 1;
      if (cu_k.size(0) != batch + 1) return none();
      seqlen_q = max_q;
      seqlen_k = max_k;
      total_q = q.size(0);
      total_k = k.size(0);
    } else {
      batch = q.size(0);
      seqlen_q = q.size(1);
      if (table.defined()) {
        page = k.size(1);
        if ((page != 32 && page != 64 && page != 128 && page != 256) || table.size(0) != batch) return none();
        seqlen_k = table.size(1) * page;
      } else {
        if (k.size(0) != batch) return none();
        seqlen_k = k.size(1);
      }
    }
    if (batch <= 0 || seqlen_q <= 0 || seqlen_k <= 0) return none();
    if ((used_q.defined() && used_q.size(0) < batch) || (used_k.defined() && used_k.size(0) < batch)) return none();
    if (splits > 1 && varlen && used_q.defined()) return none();  // the partials' unused rows want a fill there
    const auto out_type = is_fp8(code) ? at::kBFloat16 : q.scalar_type();
    if (out.defined() && (out.sizes() != q.sizes() || out.scalar_type() != out_type || out.device() != dev || out.stride(-1) != 1))
      return none();
    const int64_t l0 = varlen ? hq : batch, l1 = varlen ? total_q : hq;
    if (lse.defined() && (lse.dim() != (varlen ? 2 : 3) || lse.size(0) != l0 || lse.size(1) != l1 ||
                          (!varlen && lse.size(2) != seqlen_q) || lse.scalar_type() != at::kFloat || lse.device() != dev ||
                          lse.stride(-1) != 1))
      return none();
    double sm_scale, thr;
    if (!opt_double(a[5], 1.0 / std::sqrt((double)d), &sm_scale) || !opt_double(a[7], 1.0, &thr)) return none();
    int32_t* const status = ptr<int32_t>(*g_status[dev.index()]);
    std::optional<NoGil> no_gil(std::in_place);
    if (!out.defined()) out = at::empty(q.sizes(), q.options().dtype(out_type));
    if (!lse.defined())
      lse = varlen ? at::empty({hq, total_q}, q.options().dtype(at::kFloat))
                   : at::empty({batch, hq, seqlen_q}, q.options().dtype(at::kFloat));

    FsaFwdArgs x = {};
    Tensor partial;
    if (splits > 1) {
      const int64_t rows = varlen ? total_q : batch * seqlen_q;
      partial = at::empty({splits * rows * hq * (d + 1)}, q.options().dtype(at::kFloat));
      x.out_partial = ptr<float>(partial);
      x.lse_partial = x.out_partial + splits * rows * hq * d;
    }
    x.q = q.data_ptr();
    x.k = k.data_ptr();
    x.v = v.data_ptr();
    x.out = out.data_ptr();
    x.lse = ptr<float>(lse);
    x.cu_seqlens_q = ptr<int32_t>(cu_q);
    x.cu_seqlens_k = ptr<int32_t>(cu_k);
    x.seqused_q = ptr<int32_t>(used_q);
    x.seqused_k = ptr<int32_t>(used_k);
    x.page_table = ptr<int32_t>(table);
    x.window_sizes = ptr<int32_t>(win);
    x.status = status;
    x.q_stride_b = varlen ? 0 : q.stride(0);
    x.q_stride_s = q.stride(-3);
    x.q_stride_h = q.stride(-2);
    x.k_stride_b = x.v_stride_b = varlen ? 0 : k.stride(0);
    x.k_stride_s = x.v_stride_s = k.stride(-3);
    x.k_stride_h = x.v_stride_h = k.stride(-2);
    x.o_stride_b = varlen ? 0 : out.stride(0);
    x.o_stride_s = out.stride(-3);
    x.o_stride_h = out.stride(-2);
    x.lse_stride_b = varlen ? 0 : lse.stride(0);
    x.lse_stride_h = varlen ? lse.stride(0) : lse.stride(1);
    x.batch = (int)batch;
    x.seqlen_q = (int)seqlen_q;
    x.seqlen_k = (int)seqlen_k;
    x.total_q = (int)total_q;
    x.total_k = (int)total_k;
    x.heads_q = (int)hq;
    x.heads_kv = (int)hkv;
    x.head_dim = (int)d;
    if (table.defined()) {
      x.num_pages = (int)k.size(0);
      x.page_size = (int)page;
      x.page_table_stride = (int)table.stride(0);
    }
    x.window_stride = win.defined() ? (int)win.stride(0) : 0;
    x.num_splits = (int)splits;
    x.tile_m = x.tile_n = 128;
    x.kind = (int)kind;
    x.dtype = code;
    x.flags = (causal ? FSA_F_CAUSAL : 0) | (local ? FSA_F_LOCAL : 0) | (splits > 1 ? FSA_F_SPLIT : 0) |
              (pack && hq > hkv ? FSA_F_PACK_GQA : 0) | FSA_F_LOGSIGMOID | FSA_F_ADAPT_GATE;
    x.softmax_scale = (float)sm_scale;
    x.softmax_threshold = (float)thr;
    const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
    int rc = scale.pack(stream);
    x.qkv_scale = ptr<float>(scale.packed);
    if (rc == FSA_OK) rc = g_fwd(&x, stream);
    no_gil.reset();
    if (rc != FSA_OK) return PyLong_FromLong(rc);
    return pair(std::move(out), std::move(lse));
  END_HANDLE_TH_ERRORS
}

// topk(scores, k, positions as int64) -> positions, an error code, or None. Scores of 16 or 32 bits whose rows are equally far apart.
PyObject* topk(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 3 || !g_topk || !THPVariable_CheckExact(a[0]) || !PyBool_Check(a[2])) return none();
  HANDLE_TH_ERRORS
    int64_t k;
    const Tensor x = THPVariable_Unpack(a[0]);
    if (!get_int(a[1], &k) || !x.is_cuda() || x.dim() < 1) return none();
    const int dev = x.device().index();
    if (dev < 0 || dev >= MAX_DEVICES || c10::cuda::current_device() != dev) return none();
    const int type = x.scalar_type() == at::kFloat ? FSA_DT_F32 : dtype_code(x.scalar_type());
    const int64_t len = x.size(-1);
    if (type < 0 || is_fp8(type) || k <= 0 || k > len || len > INT32_MAX || x.numel() == 0) return none();
    if (!x.is_contiguous() && (x.dim() != 2 || x.stride(1) != 1 || x.stride(0) < len)) return none();
    const int64_t rows = x.numel() / len, pitch = x.is_contiguous() ? len : x.stride(0);
    if (rows > INT32_MAX) return none();
    auto shape = x.sizes().vec();
    shape.back() = k;
    const bool wide = a[2] == Py_True;
    std::optional<NoGil> no_gil(std::in_place);
    Tensor out = at::empty(shape, x.options().dtype(wide ? at::kLong : at::kInt));
    const int rc = g_topk(x.data_ptr(), type, (int)rows, (int)len, pitch, (int)k, out.data_ptr(), wide ? 1 : 0,
                          c10::cuda::getCurrentCUDAStream(dev).stream());
    no_gil.reset();
    if (rc != FSA_OK) return PyLong_FromLong(rc);
    return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// init(addresses of fsa_decode, fsa_fwd[, fsa_topk_indices, fsa_pack_scales])
PyObject* init(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2 && n != 4) {
    PyErr_SetString(PyExc_TypeError, "init takes two or four addresses");
    return nullptr;
  }
  void* at[4] = {};
  for (Py_ssize_t i = 0; i < n && !PyErr_Occurred(); ++i) at[i] = PyLong_AsVoidPtr(a[i]);
  if (PyErr_Occurred()) return nullptr;
  if (n == 4) {
    g_topk = reinterpret_cast<decltype(g_topk)>(at[2]);
    g_pack = reinterpret_cast<decltype(g_pack)>(at[3]);
  }
  g_decode = reinterpret_cast<decltype(g_decode)>(at[0]);
  g_fwd = reinterpret_cast<decltype(g_fwd)>(at[1]);
  return none();
}

// set_status(device index, int32 status tensor, number of SMs)
PyObject* set_status(PyObject*, PyObject* const* a, Py_ssize_t n) {
  int64_t dev, sms;
  if (n != 3 || !get_int(a[0], &dev) || dev >= MAX_DEVICES || !THPVariable_CheckExact(a[1]) || !get_int(a[2], &sms)) {
    PyErr_SetString(PyExc_TypeError, "set_status takes a device index, a tensor and a number of SMs");
    return nullptr;
  }
  g_sms[dev] = (int)sms;
  if (!g_status[dev]) g_status[dev] = new Tensor(THPVariable_Unpack(a[1]));
  return none();
}

PyObject* decode_num_splits(PyObject*, PyObject* const* a, Py_ssize_t n) {
  int64_t v[4];
  for (int i = 0; i < 4; ++i)
    if (n != 4 || !get_int(a[i], &v[i])) {
      PyErr_SetString(PyExc_TypeError, "decode_num_splits takes four non-negative integers");
      return nullptr;
    }
  return PyLong_FromLongLong(decode_splits(v[0], v[1], v[2], v[3]));
}

PyMethodDef methods[] = {
    {"init", reinterpret_cast<PyCFunction>(init), METH_FASTCALL, nullptr},
    {"set_status", reinterpret_cast<PyCFunction>(set_status), METH_FASTCALL, nullptr},
    {"decode", reinterpret_cast<PyCFunction>(decode), METH_FASTCALL, nullptr},
    {"forward", reinterpret_cast<PyCFunction>(forward), METH_FASTCALL, nullptr},
    {"topk", reinterpret_cast<PyCFunction>(topk), METH_FASTCALL, nullptr},
    {"decode_num_splits", reinterpret_cast<PyCFunction>(decode_num_splits), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// ABI_VERSION and TORCH_VERSION: what this was compiled against (the argument blocks of the header, ATen's classes).
PyMODINIT_FUNC PyInit__host(void) {
  PyObject* m = PyModule_Create(&module);
  if (m && (PyModule_AddIntConstant(m, "ABI_VERSION", FSA_ABI_VERSION) < 0 ||
            PyModule_AddStringConstant(m, "TORCH_VERSION", TORCH_VERSION) < 0)) {
    Py_DECREF(m);
    return nullptr;
  }
  return m;
}
