// Tensor plumbing of the Python layer, in C++: argument checks, device memory, streams, and the calls of the C ABI.
//
// A short call (a decode step, the prefill of a chat prompt) is bound by the host: in Python its plumbing took 40 to 100 us,
// against 8 to 60 us of kernels.  These functions do the same work in a few microseconds.  They are plain CPython functions
// on torch tensors, no operator registration and no dispatch; all of them enqueue on torch's current stream and return.
// Once the arguments are read the interpreter lock is given back (without_gil): an allocation may wait for the device, and a
// launch does while its queue is full; other Python threads run on meanwhile.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <optional>
#include <string>

#include "../../../include/xattn_b200.h"

namespace {

using at::Tensor;

PyObject* g_error = nullptr;        // XattnB200Error
PyObject* g_status_of = nullptr;    // device index -> address of the device's status word
int* g_status[64] = {};

// An error on its way to Python, thrown with or without the interpreter lock (see END_PY).
struct Refused {
  PyObject* type;
  std::string text;
};
[[noreturn]] void fail(PyObject* type, const char* format, ...) {
  char text[256];
  va_list args;
  va_start(args, format);
  std::vsnprintf(text, sizeof text, format, args);
  va_end(args);
  throw Refused{type, text};
}
void check(int code, const char* what) {
  if (code != 0) fail(g_error, "%s: %s (status %d)", what, xattn_b200_error_string(code), code);
}
#define BEGIN_PY HANDLE_TH_ERRORS try {
#define END_PY                                      \
  }                                                 \
  catch (const Refused& r) {                        \
    PyErr_SetString(r.type, r.text.c_str());        \
    return nullptr;                                 \
  }                                                 \
  END_HANDLE_TH_ERRORS

// f() without the interpreter lock: no Python object is touched in it (torch takes the lock itself where a tensor needs it)
template <typename F>
auto without_gil(F&& f) {
  struct Release {
    PyThreadState* state = PyEval_SaveThread();
    ~Release() { PyEval_RestoreThread(state); }
  } release;
  return f();
}

// ---------------------------------------------------------------------------------------------- arguments
struct Args {
  PyObject* const* v;
  Py_ssize_t n;
  const char* name;
  void count(Py_ssize_t want) const {
    if (n != want) fail(PyExc_TypeError, "%s: %zd arguments, %zd wanted", name, n, want);
  }
  const Tensor& tensor(int i) const {
    if (!THPVariable_Check(v[i])) fail(PyExc_TypeError, "a tensor is wanted");
    return THPVariable_Unpack(v[i]);
  }
  bool none(int i) const { return v[i] == Py_None; }
  long long integer(int i) const {
    const long long x = PyLong_AsLongLong(v[i]);
    if (x == -1 && PyErr_Occurred()) throw python_error();
    return x;
  }
  double real(int i) const {
    PyObject* f = PyNumber_Float(v[i]);            // what float() takes
    if (!f) throw python_error();
    const double x = PyFloat_AS_DOUBLE(f);
    Py_DECREF(f);
    return x;
  }
  bool flag(int i) const {
    const int x = PyObject_IsTrue(v[i]);
    if (x < 0) throw python_error();
    return x != 0;
  }
};

void need_cuda(const Tensor& t) {
  if (!t.is_cuda()) fail(g_error, "xattn_b200 ops need CUDA tensors: there is no CPU path");
}
void need_4d(const Tensor& t) {
  if (t.dim() != 4) fail(PyExc_ValueError, "tensors of four dimensions [batch, heads, length, head_dim] are wanted");
}
// `x` as the kernels read it: [batch, heads, len, dim] of the sizes that the call takes from q and k, on q's device.  What is
// smaller would be read past its end; of what is larger the leading part counts.
Tensor fit(const Tensor& x, int64_t batch, int64_t heads, int64_t len, int64_t dim, const Tensor& q, const char* name) {
  if (x.device() != q.device()) fail(PyExc_ValueError, "%s must be on the device of the query tensor", name);
  if (x.size(0) == batch && x.size(1) == heads && x.size(2) == len && x.size(3) == dim) return x;
  if (x.size(0) < batch || x.size(1) < heads || x.size(2) < len || x.size(3) < dim)
    fail(PyExc_ValueError, "%s is [%lld, %lld, %lld, %lld], at least [%lld, %lld, %lld, %lld] is wanted", name, (long long)x.size(0),
         (long long)x.size(1), (long long)x.size(2), (long long)x.size(3), (long long)batch, (long long)heads, (long long)len, (long long)dim);
  return x.narrow(0, 0, batch).narrow(1, 0, heads).narrow(2, 0, len).narrow(3, 0, dim);
}
Tensor fit_k(const Tensor& k, const Tensor& q) { return fit(k, q.size(0), k.size(1), k.size(2), q.size(3), q, "the key tensor"); }
Tensor fit_v(const Tensor& v, const Tensor& k, const Tensor& q) {
  return fit(v, q.size(0), k.size(1), k.size(2), q.size(3), q, "the value tensor");
}
// unit inner stride, 16-byte aligned rows; otherwise a contiguous copy
bool is_aligned16(const Tensor& x) {
  const int64_t e = x.element_size();
  return x.stride(3) == 1 && (reinterpret_cast<uintptr_t>(x.data_ptr()) & 15) == 0 && (x.stride(0) * e) % 16 == 0 &&
         (x.stride(1) * e) % 16 == 0 && (x.stride(2) * e) % 16 == 0;
}
Tensor aligned16(const Tensor& x) { return is_aligned16(x) ? x : x.contiguous(); }
// The same for tensors which any strides and any alignment will do for: what the tensor maps cannot express (rows of a
// contiguous tensor that starts off a 16-byte boundary, expanded dimensions) is copied, too.
Tensor aligned16_any(const Tensor& x) {
  bool ok = is_aligned16(x);
  for (int i = 0; i < 3; ++i) ok = ok && (x.size(i) == 1 || x.stride(i) > 0);
  return ok ? x : x.clone(at::MemoryFormat::Contiguous);
}
Tensor empty(at::IntArrayRef sizes, at::ScalarType type, const at::Device& dev) {
  return at::detail::empty_cuda(sizes, type, dev, std::nullopt);
}

// Where a call runs: the tensors' device, torch's current stream of it, the device's status word.
struct Place {
  c10::cuda::CUDAGuard guard;
  at::Device dev;
  void* stream;
  int* status;
  explicit Place(const Tensor& t) : guard(t.device()), dev(t.device()) {
    const int i = dev.index();
    stream = c10::cuda::getCurrentCUDAStream(i).stream();
    if (i < 0 || i >= 64) fail(g_error, "device index out of range");
    if (!g_status[i]) {
      PyObject* r = PyObject_CallFunction(g_status_of, "i", i);
      if (!r) throw python_error();
      g_status[i] = static_cast<int*>(PyLong_AsVoidPtr(r));
      Py_DECREF(r);
      if (!g_status[i]) throw python_error();
    }
    status = g_status[i];
  }
};

int dtype_code(at::ScalarType t) {
  return t == at::kBFloat16 ? XATTN_B200_BF16 : (t == at::kHalf ? XATTN_B200_F16 : -1);
}

// ---------------------------------------------------------------------------------------------- phases
struct Geometry {
  int lq, lk, qb, kb, q_chunks, k_chunks, bpc, block_offset;
};
Geometry geometry(int64_t q_len, int64_t k_len, int chunk, int stride, int block) {
  Geometry g;
  check(xattn_b200_estimate_geometry(static_cast<int>(q_len), static_cast<int>(k_len), chunk, stride, block,
                                     reinterpret_cast<int*>(&g)),
        "estimate_geometry");
  return g;
}

struct EstimateArgs {
  int stride, block, chunk, semantics;
  double norm;
  bool causal, band;
};
// fp32 block sums [B, Hq, q_blocks_pad, k_blocks_pad or blocks_per_chunk]
// q16, k16 (fp32 inputs, null: not wanted): set to the bf16 roundings of q and k.
// then: null, or what follows the estimate in the same call of the library: the fields of the selection, the others are set here.
Tensor estimate(const Tensor& q_, const Tensor& k_, const Geometry& g, const EstimateArgs& a, Tensor* q16, Tensor* k16, const Place& at_,
                xattn_b200_estimate_select_args* then = nullptr) {
  int dtype = q_.scalar_type() == at::kFloat ? XATTN_B200_F32 : dtype_code(q_.scalar_type());
  const bool f32 = dtype == XATTN_B200_F32;
  // any memory: fp32, and 16-bit rows of another head_dim than 128 whose length is no multiple of the stride
  const bool any = f32 || (q_.size(3) != 128 && (q_.size(2) % a.stride || k_.size(2) % a.stride));
  auto operand = [&](const Tensor& x) { return any ? aligned16_any(x) : aligned16(x); };
  Tensor q = operand(q_), k = operand(f32 && k_.scalar_type() != at::kFloat ? k_.to(at::kFloat) : k_);
  const int64_t B = q.size(0), Hq = q.size(1), Hkv = k.size(1), D = q.size(3);
  int64_t Lq = q.size(2), Lk = k.size(2);
  const int sem = a.band ? XATTN_B200_SEMANTICS_TORCH_BAND : a.semantics;
  if (f32 && D % 64 == 0 && xattn_b200_estimate_f32_terms(Hq, Hkv, Lq, Lk, a.stride, a.block, a.chunk, a.causal, sem)) {
    dtype = XATTN_B200_F32_TERMS;
    const auto split = [&](const Tensor& x) {
      const int64_t len = (x.size(2) + a.stride - 1) / a.stride * a.stride;
      Tensor t = empty({B, x.size(1), len, 3 * D}, at::kBFloat16, at_.dev);
      check(xattn_b200_split_f32_terms(static_cast<const float*>(x.data_ptr()), B, x.size(1), len, x.size(2), D, x.stride(0), x.stride(1),
                                 x.stride(2), 3, t.data_ptr(), at_.stream),
            "split_f32_terms");
      return t;
    };
    q = split(q);
    k = split(k);
    // (the first terms ARE the roundings)
    if (q16) *q16 = q.narrow(3, 0, D).narrow(2, 0, Lq);
    if (k16) *k16 = k.narrow(3, 0, D).narrow(2, 0, Lk);
    Lq = q.size(2);
    Lk = k.size(2);
  } else if (f32 && q16) {
    *q16 = empty(q.sizes(), at::kBFloat16, at_.dev);
    *k16 = empty(k.sizes(), at::kBFloat16, at_.dev);
  }
  const size_t bytes = xattn_b200_estimate_workspace_bytes_ex(B, Hq, Lq, Lk, a.stride, a.block, a.chunk, a.causal, sem);
  if (bytes == 0)
    fail(PyExc_ValueError, "unsupported estimate geometry (stride must be 4/8/16/32, block_size 128, chunk_size a multiple of 128)");
  const Tensor ws = empty({static_cast<int64_t>(bytes)}, at::kByte, at_.dev);
  Tensor sums = empty({B, Hq, g.qb, a.band ? g.bpc : g.kb}, at::kFloat, at_.dev);
  if (D == 0 || a.norm == 0.0) fail(PyExc_ZeroDivisionError, "the scale of the scores is 1 / (sqrt(head_dim) * stride * norm)");
  const double scale = 1.0 / std::sqrt(static_cast<double>(D)) / a.stride / a.norm;
  if (then) {
    xattn_b200_estimate_select_args& t = *then;
    t.q = q.data_ptr(); t.k = k.data_ptr();
    t.dtype = dtype; t.batch = B; t.hq = Hq; t.hkv = Hkv; t.q_len = Lq; t.k_len = Lk; t.head_dim = D;
    t.q_stride_b = q.stride(0); t.q_stride_h = q.stride(1); t.q_stride_l = q.stride(2);
    t.k_stride_b = k.stride(0); t.k_stride_h = k.stride(1); t.k_stride_l = k.stride(2);
    t.stride = a.stride; t.block_size = a.block; t.chunk_size = a.chunk;
    t.scale = static_cast<float>(scale);
    t.causal = a.causal; t.semantics = sem;
    t.attn_sums = static_cast<float*>(sums.data_ptr());
    t.workspace = ws.data_ptr(); t.workspace_bytes = bytes;
    t.q_bf16 = dtype == XATTN_B200_F32 && q16 ? q16->data_ptr() : nullptr;
    t.k_bf16 = dtype == XATTN_B200_F32 && k16 ? k16->data_ptr() : nullptr;
    t.status = at_.status;
    check(xattn_b200_estimate_select(then, at_.stream), "estimate");
    return sums;
  }
  if (dtype == XATTN_B200_F32)
    check(xattn_b200_estimate_f32(static_cast<const float*>(q.data_ptr()), static_cast<const float*>(k.data_ptr()), B, Hq, Hkv, Lq, Lk, D,
                                  q.stride(0), q.stride(1), q.stride(2), k.stride(0), k.stride(1), k.stride(2), a.stride, a.block, a.chunk,
                                  static_cast<float>(scale), a.causal, sem, static_cast<float*>(sums.data_ptr()), ws.data_ptr(), bytes,
                                  q16 ? q16->data_ptr() : nullptr, k16 ? k16->data_ptr() : nullptr, at_.status, at_.stream),
          "estimate_f32");
  else
    check(xattn_b200_estimate(q.data_ptr(), k.data_ptr(), dtype, B, Hq, Hkv, Lq, Lk, D, q.stride(0), q.stride(1), q.stride(2), k.stride(0),
                              k.stride(1), k.stride(2), a.stride, a.block, a.chunk, static_cast<float>(scale), a.causal, sem,
                              static_cast<float*>(sums.data_ptr()), ws.data_ptr(), bytes, at_.status, at_.stream),
          "estimate");
  return sums;
}

struct Threshold {
  Tensor per_head;              // undefined: `value` for all
  double value;
};
Threshold threshold_of(const Args& a, int i) {
  if (THPVariable_Check(a.v[i])) return {a.tensor(i), 0.0};
  return {Tensor(), a.real(i)};
}
struct Selection {
  Tensor mask, idx, cnt;
};
struct SelectArgs {
  int bpc, block_offset;
  bool causal, cleanup, sink, recent, want_mask;
  int64_t list_q, list_k;       // 0: no lists
  int64_t band_kb;              // > 0: the sums are the chunk band of rows of that many key blocks
};
// What a selection writes, allocated, and its threshold per head as the kernels read it (undefined: `value` for all).
Selection new_selection(const SelectArgs& a, int64_t B, int64_t H, int64_t QB, int64_t KB, const Threshold& threshold, Tensor& thr, const Place& at_) {
  if (threshold.per_head.defined()) {
    thr = threshold.per_head.detach();
    if (thr.device() != at_.dev || thr.scalar_type() != at::kFloat) thr = thr.to(at_.dev, at::kFloat);
    thr = thr.reshape({-1}).contiguous();
    if (thr.numel() != H) fail(PyExc_ValueError, "per-head threshold needs one entry per head");
  }
  Selection r;
  if (a.want_mask) r.mask = empty({B, H, QB, KB}, at::kBool, at_.dev);
  if (a.list_q > 0) {
    const int64_t lqb = (a.list_q + 127) / 128, lkb = (a.list_k + 127) / 128;
    r.idx = empty({B, H, lqb, lkb}, at::kInt, at_.dev);
    r.cnt = empty({B, H, lqb}, at::kInt, at_.dev);
  }
  return r;
}
template <typename T>
T* data(const Tensor& t) { return t.defined() ? static_cast<T*>(t.data_ptr()) : nullptr; }

Selection select(const Tensor& sums, const Threshold& threshold, const SelectArgs& a, const Place& at_) {
  const int64_t B = sums.size(0), H = sums.size(1), QB = sums.size(2), KB = a.band_kb > 0 ? a.band_kb : sums.size(3);
  if (a.band_kb > 0 && sums.size(3) != a.bpc) fail(PyExc_ValueError, "band sums must have blocks_per_chunk columns");
  Tensor thr;
  Selection r = new_selection(a, B, H, QB, KB, threshold, thr, at_);
  auto fn = a.band_kb > 0 ? xattn_b200_select_band : xattn_b200_select;
  check(fn(static_cast<const float*>(sums.data_ptr()), B, H, QB, KB, a.bpc, a.block_offset, a.causal, a.cleanup, threshold.value,
           data<float>(thr), a.sink, a.recent, data<uint8_t>(r.mask), data<int32_t>(r.idx), data<int32_t>(r.cnt), (a.list_q + 127) / 128,
           (a.list_k + 127) / 128, a.list_q, a.list_k, at_.status, at_.stream),
        "select");
  return r;
}

// The estimate and the selection on it.  rounded (mask only): the sums in that tensor's type, null: not wanted.
struct Estimated {
  Tensor sums;
  Selection s;
};
Estimated estimate_and_select(const Tensor& q, const Tensor& k, const Geometry& g, const EstimateArgs& e, const Threshold& threshold,
                              const SelectArgs& a, Tensor* q16, Tensor* k16, const Tensor* rounded, const Place& at_) {
  Tensor thr;
  Estimated r;
  r.s = new_selection(a, q.size(0), q.size(1), g.qb, g.kb, threshold, thr, at_);
  xattn_b200_estimate_select_args t = {};
  t.threshold = threshold.value;
  t.threshold_per_head = data<float>(thr);
  t.keep_sink = a.sink; t.keep_recent = a.recent;
  t.mask = data<uint8_t>(r.s.mask); t.block_idx = data<int32_t>(r.s.idx); t.block_cnt = data<int32_t>(r.s.cnt);
  t.list_q_len = a.list_q; t.list_k_len = a.list_k;
  if (rounded) {
    t.rounded = rounded->data_ptr();
    t.rounded_dtype = dtype_code(rounded->scalar_type());
  }
  r.sums = estimate(q, k, g, e, q16, k16, at_, &t);
  return r;
}

// Attention over block lists (undefined: dense).  q, k, v 16 bit.  `out`: undefined, or [B, Hq, Lq, 128] with unit inner
// stride.  out_f32: write fp32 (bf16 inputs only).  Returns a transposed view of [B, Lq, Hq, D] storage, or `out`.
Tensor attention(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& idx, const Tensor& cnt, bool causal, double scale,
                 Tensor out, bool out_f32, bool use_workspace, const Place& at_, int max_blocks = 0) {
  const Tensor q = aligned16(q_), k = aligned16(k_), v = aligned16(v_);
  const int64_t B = q.size(0), Hq = q.size(1), Lq = q.size(2), D = q.size(3), Hkv = k.size(1), Lk = k.size(2);
  if (!out.defined()) out = empty({B, Lq, Hq, D}, out_f32 ? at::kFloat : q.scalar_type(), at_.dev).transpose(1, 2);
  const size_t bytes = use_workspace ? xattn_b200_block_sparse_attn_workspace_bytes(B, Hq, Hkv, Lq, Lk) : 0;
  Tensor ws;
  if (bytes) ws = empty({static_cast<int64_t>(bytes)}, at::kByte, at_.dev);
  check(xattn_b200_block_sparse_attn_bounded(
            q.data_ptr(), k.data_ptr(), v.data_ptr(), out_f32 ? XATTN_B200_BF16_OUT_F32 : dtype_code(q.scalar_type()), B, Hq, Hkv, Lq, Lk,
            D, q.stride(0), q.stride(1), q.stride(2), k.stride(0), k.stride(1), k.stride(2), v.stride(0), v.stride(1), v.stride(2),
            idx.defined() ? static_cast<const int32_t*>(idx.data_ptr()) : nullptr,
            cnt.defined() ? static_cast<const int32_t*>(cnt.data_ptr()) : nullptr, causal, static_cast<float>(scale), out.data_ptr(),
            out.stride(0), out.stride(1), out.stride(2), bytes ? ws.data_ptr() : nullptr, bytes, max_blocks, at_.status, at_.stream),
        "block_sparse_attn");
  return out;
}
// Non-causal calls: sorting the units by list length is one launch of 4 to 15 us.  What it saves is the chain of a long list that would be
// begun near the end, 1.5 us per block: worth it with many items per SM, or with a few whose lists may be long (24 heads, video
// diffusion, us without and with it: 7456 tokens, 58 key blocks, 9 items per SM, 250 and 199; 11056 tokens, 14 items, 430 and 349; 12
// heads of 7400, 5 items, 189 and 170; but 3800 tokens, 30 key blocks, 5 or 10 items, 138 and 142, 177 and 183).  Lists that are all
// alike, whose lengths the host does not know, gain nothing (lists of two blocks or so, the whole prefill: 5500 tokens 62 and 67, 7400 93 and
// 100, 11000 163 and 169, 12 heads of 7400 51.5 and 56; the attention alone, two full rows of lists among those of five blocks, 200 and 128).
constexpr int64_t kOrderItemsPerSm = 16, kOrderFewItemsPerSm = 4, kOrderKeys = 40 * 128;
bool default_workspace(bool causal, bool dense, const Tensor& q, int64_t k_len) {
  if (dense) return false;
  const char* forced = std::getenv("XATTN_B200_ATTN_WORKSPACE");       // "0" / "1": overrides the rule (for measurements)
  if (forced && (forced[0] == '0' || forced[0] == '1') && forced[1] == 0) return forced[0] == '1';
  const int64_t per_sm = k_len > kOrderKeys ? kOrderFewItemsPerSm : kOrderItemsPerSm;
  return !causal && q.size(0) * q.size(1) * ((q.size(2) + 127) / 128) >= per_sm * at::cuda::getDeviceProperties(q.get_device())->multiProcessorCount;
}

void need_16bit_or_f32(const Tensor& q, const Tensor& k, const char* text) {
  if ((dtype_code(q.scalar_type()) < 0 && q.scalar_type() != at::kFloat) || (q.scalar_type() != at::kFloat && k.scalar_type() != q.scalar_type()))
    fail(PyExc_TypeError, text);
}
bool band_applies(int64_t k_len, int chunk, bool causal, int semantics) {
  return causal && semantics == XATTN_B200_SEMANTICS_TORCH && k_len % chunk == 0 && (chunk / 128) % 4 == 0;
}

// ---------------------------------------------------------------------------------------------- Python functions
PyObject* wrap(Tensor t) { return t.defined() ? THPVariable_Wrap(std::move(t)) : Py_NewRef(Py_None); }

// estimate(q, k, stride, block, chunk, norm, causal, semantics, band) -> sums
PyObject* py_estimate(PyObject*, PyObject* const* v, Py_ssize_t n) {
  BEGIN_PY
  const Args a{v, n, "estimate"};
  a.count(9);
  const Tensor q = a.tensor(0);
  need_cuda(q); need_cuda(a.tensor(1)); need_4d(q); need_4d(a.tensor(1));
  const Tensor k = fit_k(a.tensor(1), q);
  need_16bit_or_f32(q, k, "q/k must both be bf16, fp16 or fp32");
  const Place at_(q);
  const EstimateArgs e{(int)a.integer(2), (int)a.integer(3), (int)a.integer(4), (int)a.integer(7), a.real(5), a.flag(6), a.flag(8)};
  const Geometry g = geometry(q.size(2), k.size(2), e.chunk, e.stride, e.block);
  return wrap(without_gil([&] { return estimate(q, k, g, e, nullptr, nullptr, at_); }));
  END_PY
}

// select(sums, bpc, block_offset, threshold, causal, cleanup, sink, recent, want_mask, list_q, list_k, band_kb) -> (mask, idx, cnt)
PyObject* py_select(PyObject*, PyObject* const* v, Py_ssize_t n) {
  BEGIN_PY
  const Args a{v, n, "select"};
  a.count(12);
  Tensor sums = a.tensor(0);
  need_cuda(sums); need_4d(sums);
  const Place at_(sums);
  const Threshold threshold = threshold_of(a, 3);
  const SelectArgs sel{(int)a.integer(1), (int)a.integer(2), a.flag(4), a.flag(5), a.flag(6), a.flag(7), a.flag(8), a.integer(9), a.integer(10),
                       a.integer(11)};
  Selection r = without_gil([&] {
    if (sums.scalar_type() != at::kFloat) sums = sums.to(at::kFloat);
    sums = sums.contiguous();
    return select(sums, threshold, sel, at_);
  });
  PyObject* t = PyTuple_New(3);
  if (!t) throw python_error();
  PyTuple_SET_ITEM(t, 0, wrap(r.mask));
  PyTuple_SET_ITEM(t, 1, wrap(r.idx));
  PyTuple_SET_ITEM(t, 2, wrap(r.cnt));
  return t;
  END_PY
}

Tensor attention_any(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& idx, const Tensor& cnt, bool causal, double scale,
                     Tensor out, std::optional<bool> use_workspace, const Place& at_, int max_blocks = 0) {
  const int64_t D = q.size(3);
  if (D != 128) fail(PyExc_ValueError, "head_dim must be 128");
  const bool f32 = q.scalar_type() == at::kFloat, dense = !idx.defined();
  Tensor q16 = q, k16 = k, v16 = v;
  if (f32) { q16 = q.to(at::kBFloat16); k16 = k.to(at::kBFloat16); v16 = v.to(at::kBFloat16); }
  if (dtype_code(q16.scalar_type()) < 0 || k16.scalar_type() != q16.scalar_type() || v16.scalar_type() != q16.scalar_type())
    fail(PyExc_TypeError, "q/k/v must share one of bf16, fp16, fp32");
  if (out.defined() && (out.sizes() != q.sizes() || out.scalar_type() != q16.scalar_type() || out.stride(3) != 1 || out.device() != q.device()))
    fail(PyExc_ValueError, "out must be a CUDA tensor [B,Hq,Lq,D] of the compute dtype with unit inner stride");
  const int64_t lqb = (q.size(2) + 127) / 128, lkb = (k.size(2) + 127) / 128;
  if (!dense && (idx.sizes() != at::IntArrayRef({q.size(0), q.size(1), lqb, lkb}) || cnt.sizes() != at::IntArrayRef({q.size(0), q.size(1), lqb})))
    fail(PyExc_ValueError, "block lists have the wrong shape");
  const bool ws = dense ? false : use_workspace.value_or(default_workspace(causal, dense, q, k.size(2)));
  return attention(q16, k16, v16, dense ? idx : idx.contiguous(), dense ? cnt : cnt.contiguous(), causal, scale, out, f32 && !out.defined(), ws, at_, max_blocks);
}

// attention(q, k, v, idx, cnt, causal, scale, out, use_workspace) -> out
PyObject* py_attention(PyObject*, PyObject* const* v, Py_ssize_t n) {
  BEGIN_PY
  const Args a{v, n, "attention"};
  a.count(9);
  const Tensor q = a.tensor(0), k_ = a.tensor(1), v_ = a.tensor(2);
  Tensor idx, cnt, out;
  if (!a.none(3)) idx = a.tensor(3);
  if (!a.none(4)) cnt = a.tensor(4);
  if (idx.defined() != cnt.defined()) fail(PyExc_ValueError, "block lists have the wrong shape");
  if (!a.none(7)) out = a.tensor(7);
  need_cuda(q); need_cuda(k_); need_cuda(v_); need_4d(q); need_4d(k_); need_4d(v_);
  const Tensor k = fit_k(k_, q), vv = fit_v(v_, k_, q);
  if (idx.defined()) {
    need_cuda(idx); need_cuda(cnt);
    if (idx.device() != q.device() || cnt.device() != q.device() || idx.element_size() != 4 || cnt.element_size() != 4)
      fail(PyExc_ValueError, "block lists are 32-bit integers on the device of the query tensor");
  }
  const Place at_(q);
  const double scale = a.none(6) ? 1.0 / std::sqrt(static_cast<double>(q.size(3))) : a.real(6);
  std::optional<bool> ws;
  if (!a.none(8)) ws = a.flag(8);
  const bool causal = a.flag(5);
  return wrap(without_gil([&] { return attention_any(q, k, vv, idx, cnt, causal, scale, out, ws, at_); }));
  END_PY
}

// decode(q, k, v, scale) -> out: one query token per sequence against its whole cache
PyObject* py_decode(PyObject*, PyObject* const* pv, Py_ssize_t n) {
  BEGIN_PY
  const Args a{pv, n, "decode"};
  a.count(4);
  const Tensor q_ = a.tensor(0);
  need_cuda(q_); need_cuda(a.tensor(1)); need_cuda(a.tensor(2)); need_4d(q_); need_4d(a.tensor(1)); need_4d(a.tensor(2));
  const Tensor k_ = fit_k(a.tensor(1), q_), v_ = fit_v(a.tensor(2), k_, q_);
  const Place at_(q_);
  const int64_t B = q_.size(0), Hq = q_.size(1), D = q_.size(3), Hkv = k_.size(1), Lk = k_.size(2);
  const double scale = a.none(3) ? 1.0 / std::sqrt(static_cast<double>(D)) : a.real(3);
  const int code = dtype_code(q_.scalar_type());
  // what the decode kernel does not cover (batch and kv heads are dimensions of its grid)
  if (q_.size(2) != 1 || D != 128 || code < 0 || Hkv == 0 || Hq % Hkv || Hq / Hkv > 16 || B > 65535 || Hkv > 65535)
    return wrap(without_gil([&] { return attention_any(q_, k_, v_, Tensor(), Tensor(), true, scale, Tensor(), false, at_); }));
  if (k_.scalar_type() != q_.scalar_type() || v_.scalar_type() != q_.scalar_type())
    fail(PyExc_TypeError, "q/k/v must share one of bf16, fp16, fp32");
  return wrap(without_gil([&] {
    const Tensor q = aligned16(q_), k = aligned16(k_), v = aligned16(v_);
    const size_t bytes = xattn_b200_decode_workspace_bytes(B, Hq, Hkv, Lk);
    Tensor ws;
    if (bytes) ws = empty({static_cast<int64_t>(bytes)}, at::kByte, at_.dev);
    Tensor out = empty({B, 1, Hq, D}, q.scalar_type(), at_.dev);
    check(xattn_b200_decode_attn(q.data_ptr(), k.data_ptr(), v.data_ptr(), code, B, Hq, Hkv, Lk, D, q.stride(0), q.stride(1), k.stride(0),
                                 k.stride(1), k.stride(2), v.stride(0), v.stride(1), v.stride(2), static_cast<float>(scale), out.data_ptr(),
                                 Hq * D, D, bytes ? ws.data_ptr() : nullptr, bytes, at_.status, at_.stream),
          "decode_attn");
    return out.transpose(1, 2);
  }));
  END_PY
}

// prefill(q, k, v, stride, norm, threshold, block, causal, chunk, sink, recent, semantics, out) -> out: all three phases
PyObject* py_prefill(PyObject*, PyObject* const* pv, Py_ssize_t n) {
  BEGIN_PY
  const Args a{pv, n, "prefill"};
  a.count(13);
  const Tensor q = a.tensor(0);
  Tensor k = a.tensor(1), v = a.tensor(2), out;
  need_cuda(q); need_4d(q); need_4d(k); need_4d(v);
  const Place at_(q);
  const int64_t Lq = q.size(2), Lk = k.size(2), D = q.size(3);
  EstimateArgs e{(int)a.integer(3), (int)a.integer(6), a.none(8) ? xattn_b200_default_chunk_size(Lk) : (int)a.integer(8), (int)a.integer(11),
                 a.real(4), a.flag(7), false};
  const Threshold threshold = threshold_of(a, 5);
  const bool sink = a.flag(9), recent = a.flag(10);
  if (!a.none(12)) out = a.tensor(12);
  return wrap(without_gil([&] {
    if (k.device() != q.device()) k = k.to(q.device());
    if (v.device() != q.device()) v = v.to(q.device());
    v = fit_v(v, k, q);
    k = fit_k(k, q);
    need_16bit_or_f32(q, k, "q/k must both be bf16, fp16 or fp32");
    const Geometry g = geometry(Lq, Lk, e.chunk, e.stride, e.block);       // (refuses a chunk of no blocks)
    // un-padded causal keys under the torch branch: the sums outside a row's own chunk are zero and are not kept
    e.band = band_applies(Lk, e.chunk, e.causal, e.semantics);
    // fp32: the attention phase computes with the bf16 roundings, those of q and k come from the estimate
    const bool f32 = q.scalar_type() == at::kFloat && D == 128 && !out.defined() && v.scalar_type() == at::kFloat;
    Tensor q16, k16;
    const Selection s = estimate_and_select(q, k, g, e, threshold, {g.bpc, g.block_offset, e.causal, true, sink, recent, false, Lq, Lk, 0},
                                            f32 ? &q16 : nullptr, f32 ? &k16 : nullptr, nullptr, at_).s;
    const double scale = 1.0 / std::sqrt(static_cast<double>(D));
    // (a row's own chunk and block 0; keep_sink sets a whole row, of the first block)
    const int max_blocks = e.band && !sink ? g.bpc + 1 : 0;
    if (!f32) return attention_any(q, k, v, s.idx, s.cnt, e.causal, scale, out, std::nullopt, at_, max_blocks);
    const Tensor vc = v.stride(3) == 1 ? v : v.contiguous();
    const Tensor v16 = empty(v.sizes(), at::kBFloat16, at_.dev);
    check(xattn_b200_split_f32_terms(static_cast<const float*>(vc.data_ptr()), v.size(0), v.size(1), Lk, Lk, D, vc.stride(0), vc.stride(1),
                                     vc.stride(2), 1, v16.data_ptr(), at_.stream),
          "split_f32_terms");
    return attention(q16, k16, v16, s.idx, s.cnt, e.causal, scale, out, true, default_workspace(e.causal, false, q, Lk), at_, max_blocks);
  }));
  END_PY
}

// estimate_and_select(q, k, stride, block, chunk, norm, causal, semantics, threshold, sink, recent) -> (sums in q's type, mask)
PyObject* py_estimate_and_select(PyObject*, PyObject* const* pv, Py_ssize_t n) {
  BEGIN_PY
  const Args a{pv, n, "estimate_and_select"};
  a.count(11);
  const Tensor q = a.tensor(0);
  need_cuda(q); need_cuda(a.tensor(1)); need_4d(q); need_4d(a.tensor(1));
  const Tensor k = fit_k(a.tensor(1), q);
  need_16bit_or_f32(q, k, "q/k must both be bf16, fp16 or fp32");
  const Place at_(q);
  const EstimateArgs e{(int)a.integer(2), (int)a.integer(3), (int)a.integer(4), (int)a.integer(7), a.real(5), a.flag(6), false};
  const Geometry g = geometry(q.size(2), k.size(2), e.chunk, e.stride, e.block);
  const Threshold threshold = threshold_of(a, 8);
  const bool sink = a.flag(9), recent = a.flag(10);
  Tensor result;
  Selection s = without_gil([&] {
    const bool f32 = q.scalar_type() == at::kFloat;
    // the sums in q's type: rounded by the selection where it holds a row in registers (up to 1024 key blocks)
    const bool in_select = !f32 && g.kb <= 1024;
    if (in_select) result = empty({q.size(0), q.size(1), g.qb, g.kb}, q.scalar_type(), at_.dev);
    Estimated r = estimate_and_select(q, k, g, e, threshold, {g.bpc, g.block_offset, e.causal, true, sink, recent, true, 0, 0, 0}, nullptr,
                                      nullptr, in_select ? &result : nullptr, at_);
    if (!in_select) result = f32 ? r.sums : r.sums.to(q.scalar_type());
    return r.s;
  });
  PyObject* t = PyTuple_New(2);
  if (!t) throw python_error();
  PyTuple_SET_ITEM(t, 0, wrap(result));
  PyTuple_SET_ITEM(t, 1, wrap(s.mask));
  return t;
  END_PY
}

// init(error class, status word callback)
PyObject* py_init(PyObject*, PyObject* const* v, Py_ssize_t n) {
  BEGIN_PY
  const Args a{v, n, "init"};
  a.count(2);
  g_error = Py_NewRef(v[0]);
  g_status_of = Py_NewRef(v[1]);
  Py_RETURN_NONE;
  END_PY
}

PyMethodDef methods[] = {
    {"init", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_init)), METH_FASTCALL, nullptr},
    {"estimate", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_estimate)), METH_FASTCALL, nullptr},
    {"estimate_and_select", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_estimate_and_select)), METH_FASTCALL, nullptr},
    {"select", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_select)), METH_FASTCALL, nullptr},
    {"attention", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_attention)), METH_FASTCALL, nullptr},
    {"decode", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_decode)), METH_FASTCALL, nullptr},
    {"prefill", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_prefill)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Tensor plumbing of xattn_b200", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
