// Host front of the operators: takes a call's tensors, checks that a kernel covers it, fills the C-ABI parameters, allocates
// the outputs and launches, all in one trip out of Python.
//
// The Python operators (ops/fmha, ops/rope_padded.py) do the same with every check spelled out and every message; at 60-70 us a
// call they, and not the GPU, set the pace of a decoding step or a short prompt.  A rope_padded + attention step of 4 sequences
// (3 kernels of 21 us together): 105 us through Python, 27 through here; a prompt of 333 tokens (one kernel of 11 us): 64 and 13.
// This file only says yes: a function returns None for whatever it does not recognise or would reject, and the caller then takes the
// Python path, which runs the call or raises its error.  What is accepted here is therefore a subset of what is accepted there,
// with the same operator chosen, and the same kernels run with the same arguments.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <cmath>
#include <cstdlib>
#include <limits>
#include <optional>
#include <vector>

#include "../../include/xfb200.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

// The C ABI of the library that Python has loaded (which one is Python's choice: XFB200_LIBRARY).
decltype(&xfb200_prefill_forward) g_prefill = nullptr;
decltype(&xfb200_decode_forward) g_decode = nullptr;
decltype(&xfb200_decode_scratch_bytes) g_scratch_bytes = nullptr;
decltype(&xfb200_decode_split_k) g_split_k = nullptr;
decltype(&xfb200_merge_attentions) g_merge = nullptr;
decltype(&xfb200_rope_padded) g_rope = nullptr;

void bind(uintptr_t prefill, uintptr_t decode, uintptr_t scratch_bytes, uintptr_t split_k, uintptr_t merge, uintptr_t rope) {
  g_prefill = reinterpret_cast<decltype(g_prefill)>(prefill);
  g_decode = reinterpret_cast<decltype(g_decode)>(decode);
  g_scratch_bytes = reinterpret_cast<decltype(g_scratch_bytes)>(scratch_bytes);
  g_split_k = reinterpret_cast<decltype(g_split_k)>(split_k);
  g_merge = reinterpret_cast<decltype(g_merge)>(merge);
  g_rope = reinterpret_cast<decltype(g_rope)>(rope);
}

// XFB200_CHECK_STATUS / XFB200_DEBUG_CHECKS: the Python path does that.
bool checks_wanted() {
  for (const char* name : {"XFB200_CHECK_STATUS", "XFB200_DEBUG_CHECKS"}) {
    const char* v = std::getenv(name);
    if (v != nullptr && v[0] != 0 && !(v[0] == '0' && v[1] == 0)) return true;
  }
  return false;
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kBFloat16: return XFB200_BF16;
    case at::kHalf: return XFB200_F16;
    case at::kFloat: return XFB200_F32;
    default: return -1;
  }
}

// A plain dense CUDA tensor on a B200.
bool plain_cuda(const Tensor& t, c10::DeviceIndex dev) { return t.is_cuda() && t.get_device() == dev && t.layout() == at::kStrided; }
bool on_b200(c10::DeviceIndex dev) {
  const cudaDeviceProp* p = at::cuda::getDeviceProperties(dev);
  return p->major == 10 && p->minor == 0;
}
void* stream_of(c10::DeviceIndex dev) { return at::cuda::getCurrentCUDAStream(dev).stream(); }

// A [B, M, H, D] or [B, M, G, H, D] tensor in BMGHK terms.
struct View {
  const Tensor& t;
  bool five;
  int64_t B, M, G, H, D, sb, sm, sg, sh, sd;
  explicit View(const Tensor& x) : t(x), five(x.dim() == 5) {
    const auto n = x.sizes(), s = x.strides();
    const int o = five ? 1 : 0;
    B = n[0], M = n[1], G = five ? n[2] : 1, H = n[2 + o], D = n[3 + o];
    // (the stride of the axis that unsqueeze(2) would add)
    sb = s[0], sm = s[1], sg = five ? s[2] : n[2] * s[2], sh = s[2 + o], sd = s[3 + o];
  }
  bool same_axes(const View& o) const { return five == o.five && B == o.B && G == o.G && H == o.H; }
  // rows that 16-byte loads and tensor maps can take, 16-bit elements
  bool rows16() const {
    if (D % 8 != 0 || (D > 1 && sd != 1)) return false;
    if (sb % 8 || sm % 8 || sh % 8 || (five && sg % 8)) return false;
    return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
  }
  xfb200_strides strides() const { return {sb, sm, sg, sh}; }
};

// What a bias object tells about its sequences.
struct Sequences {
  const Tensor* start_q = nullptr;
  const Tensor* start_k = nullptr;
  const Tensor* len_k = nullptr;
  const Tensor* tables = nullptr;
  int64_t n = 0, max_q = 0, min_q = 0, padding = 0, page = 0;
  bool gappy = false;
};

// How a call is to be served: the flags the Python wrapper passes.
enum : int64_t { kWantLse = 1, kPartial = 2, kDecodeTakesBias = 4, kPrefillTakesBias = 8, kForceDecode = 16, kForcePrefill = 32 };

struct Call {
  int64_t flags = 0, mask = 0, window_left = -1, window_right = 0;
  float scale = 0.f;
  at::ScalarType out_dtype = at::kFloat;
  const Tensor* bias = nullptr;       // additive
  const Tensor* k_words = nullptr;    // fp8: scale / shift words
  const Tensor* v_words = nullptr;
};

py::object result(const Tensor& out, const OptTensor& lse) { return py::make_tuple(out, lse.has_value() ? py::cast(*lse) : py::none()); }

Tensor new_out(const View& q, at::ScalarType dt) { return at::empty(q.t.sizes(), q.t.options().dtype(dt)); }

py::object prefill(const View& q, const View& k, const View& v, const Sequences* s, const Call& c) {
  const int64_t D = q.D;
  if (!(c.flags & kPrefillTakesBias)) return py::none();
  const int dt = dtype_code(q.t.scalar_type()), odt = dtype_code(c.out_dtype);
  if (dt == XFB200_F32 || dt < 0 || k.t.scalar_type() != q.t.scalar_type() || v.t.scalar_type() != q.t.scalar_type()) return py::none();
  if (k.D != D || v.D != D || D < 8 || D > 256 || !q.rows16() || !k.rows16() || !v.rows16()) return py::none();
  if (k.M == 0 || q.t.numel() == 0) return py::none();
  constexpr int64_t kMax = std::numeric_limits<int32_t>::max();
  if (q.M > kMax || k.M > kMax || q.B > kMax) return py::none();
  xfb200_prefill_params p{};
  if (c.bias != nullptr) {
    const Tensor& b = *c.bias;
    if (s != nullptr || !plain_cuda(b, q.t.get_device()) || b.dim() != (q.five ? 5 : 4) || b.stride(-1) != 1 || dtype_code(b.scalar_type()) < 0) return py::none();
    const int o = q.five ? 1 : 0;
    if (b.size(0) != q.B || (q.five && b.size(1) != q.G) || b.size(1 + o) != q.H || b.size(2 + o) != q.M || b.size(3 + o) != k.M) return py::none();
    p.bias = b.data_ptr(), p.bias_dtype = dtype_code(b.scalar_type());
    p.bias_stride_b = b.stride(0), p.bias_stride_g = q.five ? b.stride(1) : b.size(1) * b.stride(1), p.bias_stride_h = b.stride(1 + o), p.bias_stride_m = b.stride(2 + o);
  }
  const bool lse_wanted = (c.flags & (kWantLse | kPartial)) != 0;
  Tensor out = new_out(q, c.out_dtype);
  OptTensor lse;
  const auto f32 = q.t.options().dtype(at::kFloat);
  if (lse_wanted) lse = q.five ? at::empty({q.B, q.G, q.H, q.M}, f32) : at::empty({q.B, q.H, q.M}, f32);
  p.q = q.t.data_ptr(), p.k = k.t.data_ptr(), p.v = v.t.data_ptr(), p.out = out.data_ptr();
  p.lse = lse_wanted ? lse->data_ptr<float>() : nullptr;
  p.dtype = dt, p.out_dtype = odt;
  if (s != nullptr) {
    p.seqstart_q = s->start_q->data_ptr<int32_t>(), p.seqstart_k = s->start_k->data_ptr<int32_t>();
    p.seqlen_k = s->len_k != nullptr ? s->len_k->data_ptr<int32_t>() : nullptr;
    p.batch = int32_t(s->n), p.mq = int32_t(std::max<int64_t>(s->max_q, 0));
  } else {
    p.batch = int32_t(q.B), p.mq = int32_t(q.M);
  }
  p.mkv = int32_t(k.M), p.total_q = int32_t(q.M);
  p.groups = int32_t(q.G), p.heads_per_group = int32_t(q.H), p.head_dim = int32_t(D);
  p.q_strides = q.strides(), p.k_strides = k.strides(), p.v_strides = v.strides();
  p.o_strides = {q.M * q.G * q.H * D, q.G * q.H * D, q.H * D, D};
  p.lse_stride_b = q.G * q.H * q.M, p.lse_stride_g = q.H * q.M, p.lse_stride_h = q.M;
  p.mask_type = int32_t(c.mask), p.window_left = int32_t(c.window_left), p.window_right = int32_t(c.window_right);
  p.scale = c.scale;
  void* st = stream_of(q.t.get_device());
  int rc;
  {
    py::gil_scoped_release nogil;
    rc = g_prefill(&p, st);
  }
  return rc == XFB200_OK ? result(out, lse) : py::none();
}

py::object decode(const View& q, const View& k, const View& v, const Sequences* s, const Call& c) {
  const int64_t D = q.D;
  if (!(c.flags & kDecodeTakesBias) || c.bias != nullptr || (D != 64 && D != 128) || !q.rows16()) return py::none();
  const int dt = dtype_code(q.t.scalar_type());
  if (dt == XFB200_F32 || dt < 0 || q.t.numel() == 0 || k.t.numel() == 0) return py::none();
  const bool fp8 = c.k_words != nullptr, words = k.t.scalar_type() == at::kInt, int4 = words && !fp8;
  if (v.t.scalar_type() != k.t.scalar_type() || (!words && k.t.scalar_type() != q.t.scalar_type())) return py::none();
  if (fp8 ? (!words || D != 128 || k.D != D / 4) : int4 ? k.D != D / 8 + 1 : k.D != D) return py::none();
  if (v.D != k.D || k.sd != 1 || v.sd != 1) return py::none();
  if (!words && (!k.rows16() || !v.rows16())) return py::none();
  const bool broadcast = q.H > 1 && k.sh == 0 && v.sh == 0;
  const bool window = s != nullptr && c.window_left >= 0;
  int64_t mq = q.M, batch = q.B;
  if (s != nullptr) {
    if (s->len_k == nullptr || s->max_q != s->min_q || s->max_q < 1 || q.B != 1) return py::none();
    mq = s->max_q, batch = s->n;
    if (q.M != batch * mq) return py::none();
    if (window && ((mq != 1 && words) || (fp8 && s->tables != nullptr))) return py::none();
  } else if (q.B > 1 && (q.sb != q.M * q.sm || k.sb != k.M * k.sm || v.sb != v.M * v.sm)) {
    return py::none();
  }
  if (mq * (broadcast ? q.H : 1) > 64) return py::none();
  if (!broadcast && q.G > 1 && q.H > 1 && (k.sg != q.H * k.sh || v.sg != q.H * v.sh || q.sg != q.H * q.sh)) return py::none();

  xfb200_decode_params p{};
  p.kv_format = fp8 ? XFB200_KV_FP8_ROWWISE : int4 ? XFB200_KV_INT4_ROWWISE : XFB200_KV_PLAIN;
  p.num_quant_groups = int4 ? 1 : 0;
  p.dtype = dt, p.out_dtype = dtype_code(c.out_dtype), p.head_dim = int32_t(D);
  p.batch = int32_t(batch), p.mq = int32_t(mq);
  const int64_t osm = q.G * q.H * D, osg = q.H * D, osh = D, total = q.B * q.M;
  p.q_stride_m = q.sm, p.k_stride_m = k.sm, p.v_stride_m = v.sm, p.o_stride_m = osm;
  if (broadcast) {
    p.kv_heads = int32_t(q.G), p.q_per_kv = int32_t(q.H);
    p.q_stride_g = q.sg, p.q_stride_h = q.sh, p.k_stride_g = k.sg, p.v_stride_g = v.sg, p.o_stride_g = osg, p.o_stride_h = osh;
    p.lse_stride_g = q.H * total, p.lse_stride_h = total;
  } else {
    p.kv_heads = int32_t(q.G * q.H), p.q_per_kv = 1;
    p.q_stride_g = q.H > 1 ? q.sh : q.sg, p.k_stride_g = q.H > 1 ? k.sh : k.sg, p.v_stride_g = q.H > 1 ? v.sh : v.sg;
    p.o_stride_g = q.H > 1 ? osh : osg, p.lse_stride_g = total;
  }
  if (fp8) {
    const Tensor &kw = *c.k_words, &vw = *c.v_words;
    for (const Tensor* w : {&kw, &vw})
      if (!plain_cuda(*w, q.t.get_device()) || w->scalar_type() != at::kInt || w->dim() != k.t.dim() - 1 || w->sizes() != k.t.sizes().slice(0, k.t.dim() - 1)) return py::none();
    auto sg = [&](const Tensor& w) { return q.five ? w.stride(2) : w.size(2) * w.stride(2); };
    auto sh = [&](const Tensor& w) { return q.five ? w.stride(3) : w.stride(2); };
    p.k_scale_shift = kw.data_ptr<int32_t>(), p.v_scale_shift = vw.data_ptr<int32_t>();
    p.ks_stride_m = kw.stride(1), p.vs_stride_m = vw.stride(1);
    if (broadcast) {
      p.ks_stride_g = sg(kw), p.vs_stride_g = sg(vw);
      p.ss_words = sh(kw) == 1 && sh(vw) == 1 ? int32_t(q.H) : 1;
    } else {
      p.ks_stride_g = q.H > 1 ? sh(kw) : sg(kw), p.vs_stride_g = q.H > 1 ? sh(vw) : sg(vw);
    }
  }
  p.kv_padding = int32_t(k.M);
  if (s != nullptr) {
    p.seqlen_k = s->len_k->data_ptr<int32_t>();
    p.kv_padding = int32_t(s->padding);
    if (s->tables != nullptr) {
      const Tensor& t = *s->tables;
      if (!plain_cuda(t, q.t.get_device()) || t.scalar_type() != at::kInt || t.dim() != 2 || t.stride(1) != 1 || s->page < 1 || k.M % s->page) return py::none();
      p.block_tables = t.data_ptr<int32_t>(), p.page_size = int32_t(s->page), p.block_table_stride = int32_t(t.stride(0));
      p.kv_padding = int32_t(t.size(1) * s->page);
    } else if (s->gappy) {
      p.kv_seqstart = s->start_k->data_ptr<int32_t>();
    }
    p.mask_type = int32_t(c.mask);
    if (window) p.window_size = int32_t(c.window_left + 1);
  }
  if (p.kv_padding < 1) return py::none();
  p.kv_rows = q.B * k.M;
  p.split_k = g_split_k(p.batch, window ? std::min<int64_t>(p.kv_padding, p.window_size + mq - 1) : p.kv_padding, p.kv_heads, p.mq * p.q_per_kv,
                        int32_t(k.D * k.t.element_size()), words);
  p.scale = c.scale;
  Tensor out = new_out(q, c.out_dtype), lse;
  if (c.flags & (kWantLse | kPartial)) lse = at::empty({q.G, q.H, total}, q.t.options().dtype(at::kFloat));
  const size_t bytes = g_scratch_bytes(p.batch, p.mq, p.kv_heads, p.q_per_kv, p.head_dim, p.split_k);
  Tensor scratch;
  if (bytes) scratch = at::empty({int64_t(bytes)}, q.t.options().dtype(at::kByte));
  p.q = q.t.data_ptr(), p.k = k.t.data_ptr(), p.v = v.t.data_ptr(), p.out = out.data_ptr();
  p.lse = lse.defined() ? lse.data_ptr<float>() : nullptr;
  p.scratch = bytes ? scratch.data_ptr() : nullptr;
  void* st = stream_of(q.t.get_device());
  int rc;
  {
    py::gil_scoped_release nogil;
    rc = g_decode(&p, st);
  }
  if (rc != XFB200_OK) return py::none();
  OptTensor lse_out;
  if (lse.defined())  // packed [G, H, sequences * queries], viewed as [B, (G,) H, Mq]
    lse_out = q.five ? lse.view({q.G, q.H, q.B, q.M}).permute({2, 0, 1, 3}) : lse.view({q.H, q.B, q.M}).permute({1, 0, 2});
  return result(out, lse_out);
}

// The dispatcher's rule (ops/fmha/dispatch.py): decode first when the input looks like decoding.
py::object attention(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Sequences* s, Call& c, std::optional<double> scale,
                     std::optional<at::ScalarType> out_dtype) {
  const auto dim = q_.dim();
  if ((dim != 4 && dim != 5) || k_.dim() != dim || v_.dim() != dim || !q_.is_cuda() || checks_wanted()) return py::none();
  const auto dev = q_.get_device();
  if (!plain_cuda(q_, dev) || !plain_cuda(k_, dev) || !plain_cuda(v_, dev) || !on_b200(dev)) return py::none();
  const View q(q_), k(k_), v(v_);
  if (!q.same_axes(k) || !q.same_axes(v) || k.M != v.M || q.D == 0) return py::none();
  if (s != nullptr) {
    if (q.B != 1 || s->n < 1) return py::none();
    for (const Tensor* t : {s->start_q, s->start_k, s->len_k})
      if (t != nullptr && (!plain_cuda(*t, dev) || t->scalar_type() != at::kInt || !t->is_contiguous())) return py::none();
  }
  c.out_dtype = out_dtype.value_or(q_.scalar_type());
  if (dtype_code(c.out_dtype) < 0) return py::none();
  c.scale = float(scale.has_value() ? *scale : std::pow(double(q.D), -0.5));
  const c10::cuda::CUDAGuard guard(dev);
  const bool decode_only = k_.scalar_type() == at::kInt || (s != nullptr && s->tables != nullptr);
  if (c.flags & kForceDecode) return decode(q, k, v, s, c);
  if (c.flags & kForcePrefill) return decode_only ? py::none() : prefill(q, k, v, s, c);
  if (decode_only) return decode(q, k, v, s, c);
  const int64_t mq = s != nullptr ? s->max_q : q.M, batch = s != nullptr ? s->n : q.B;
  const bool shared_kv = q.H > 1 && k.sh == 0 && v.sh == 0;
  const bool for_grad = (c.flags & kWantLse) && !(c.flags & kPartial);
  if (shared_kv && mq <= 16 && batch <= 64 && !for_grad && (c.flags & kDecodeTakesBias)) return decode(q, k, v, s, c);
  return prefill(q, k, v, s, c);
}

py::object dense(const Tensor& q, const Tensor& k, const Tensor& v, const OptTensor& bias, int64_t flags, int64_t mask, int64_t window_left,
                 int64_t window_right, std::optional<double> scale, std::optional<at::ScalarType> out_dtype) {
  Call c;
  c.flags = flags, c.mask = mask, c.window_left = window_left, c.window_right = window_right;
  c.bias = bias.has_value() ? &*bias : nullptr;
  return attention(q, k, v, nullptr, c, scale, out_dtype);
}

py::object varlen(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& start_q, const Tensor& start_k, const OptTensor& len_k, int64_t n,
                  int64_t max_q, int64_t min_q, int64_t padding, bool gappy, int64_t flags, int64_t mask, int64_t window_left, int64_t window_right,
                  std::optional<double> scale, std::optional<at::ScalarType> out_dtype, const OptTensor& tables, int64_t page, const OptTensor& k_words,
                  const OptTensor& v_words) {
  Sequences s;
  s.start_q = &start_q, s.start_k = &start_k, s.len_k = len_k.has_value() ? &*len_k : nullptr;
  s.tables = tables.has_value() ? &*tables : nullptr;
  s.n = n, s.max_q = max_q, s.min_q = min_q, s.padding = padding, s.page = page, s.gappy = gappy;
  Call c;
  c.flags = flags, c.mask = mask, c.window_left = window_left, c.window_right = window_right;
  if (k_words.has_value() != v_words.has_value()) return py::none();
  if (k_words.has_value()) c.k_words = &*k_words, c.v_words = &*v_words;
  return attention(q, k, v, &s, c, scale, out_dtype);
}

// merge_attentions of a list of partials that share one layout.
py::object merge(const std::vector<Tensor>& attn, const std::vector<Tensor>& lse, bool write_lse, std::optional<at::ScalarType> out_dtype) {
  const size_t n = attn.size();
  if (n == 0 || n != lse.size() || n > XFB200_MERGE_MAX_PTRS) return py::none();
  const Tensor &a0 = attn[0], &l0 = lse[0];
  if (!a0.is_cuda() || (a0.dim() != 4 && a0.dim() != 5) || l0.dim() != a0.dim() - 1) return py::none();
  const auto dev = a0.get_device();
  const void* ap[XFB200_MERGE_MAX_PTRS];
  const float* lp[XFB200_MERGE_MAX_PTRS];
  for (size_t i = 0; i < n; ++i) {
    if (!plain_cuda(attn[i], dev) || !plain_cuda(lse[i], dev) || attn[i].scalar_type() != a0.scalar_type() || lse[i].scalar_type() != at::kFloat) return py::none();
    if (attn[i].sizes() != a0.sizes() || attn[i].strides() != a0.strides() || lse[i].sizes() != l0.sizes() || lse[i].strides() != l0.strides()) return py::none();
    ap[i] = attn[i].data_ptr(), lp[i] = lse[i].data_ptr<float>();
  }
  const View a(a0);
  const int o = a.five ? 1 : 0;
  if (l0.size(0) != a.B || (a.five && l0.size(1) != a.G) || l0.size(1 + o) != a.H || l0.size(2 + o) != a.M) return py::none();
  if ((a.M > 1 && l0.stride(2 + o) != 1) || (a.D > 1 && a.sd != 1) || a0.numel() == 0) return py::none();
  const auto odt = out_dtype.value_or(a0.scalar_type());
  if (dtype_code(a0.scalar_type()) < 0 || dtype_code(odt) < 0) return py::none();
  const c10::cuda::CUDAGuard guard(dev);
  Tensor out = new_out(a, odt);
  OptTensor lse_out;
  if (write_lse) lse_out = at::empty(l0.sizes(), l0.options());
  xfb200_merge_params p{};
  p.attn_ptrs = ap, p.lse_ptrs = lp, p.num_splits = int32_t(n);
  p.attn_strides = a.strides();
  p.lse_in_stride_b = l0.stride(0), p.lse_in_stride_g = a.five ? l0.stride(1) : l0.size(1) * l0.stride(1), p.lse_in_stride_h = l0.stride(1 + o);
  p.out = out.data_ptr(), p.lse_out = write_lse ? lse_out->data_ptr<float>() : nullptr;
  p.out_strides = {a.M * a.G * a.H * a.D, a.G * a.H * a.D, a.H * a.D, a.D};
  p.lse_out_stride_b = a.G * a.H * a.M, p.lse_out_stride_g = a.H * a.M, p.lse_out_stride_h = a.M;
  p.B = int32_t(a.B), p.M = int32_t(a.M), p.G = int32_t(a.G), p.H = int32_t(a.H), p.D = int32_t(a.D);
  p.in_dtype = dtype_code(a0.scalar_type()), p.out_dtype = dtype_code(odt);
  void* st = stream_of(dev);
  int rc;
  {
    py::gil_scoped_release nogil;
    rc = g_merge(&p, st);
  }
  return rc == XFB200_OK ? result(out, lse_out) : py::none();
}

struct RopeOptions {
  double theta, linear_scale, old_context_len, scale_factor, low_freq, high_freq;
};

// rope_padded into a cache of the inputs' type or an int4 row-wise one; returns out_q.
py::object rope(const Tensor& xq, const Tensor& xk, const Tensor& xv, const Tensor& ck, const Tensor& cv, const OptTensor& out_q_, const Tensor& start_q,
                const Tensor& start_k, const Tensor& len_k, int64_t n, int64_t total_q, int64_t total_k, int64_t max_q, const OptTensor& tables, int64_t page,
                bool adjacents, bool dynamic, bool f64, double theta, double linear_scale, double old_context_len, double scale_factor, double low_freq,
                double high_freq) {
  const auto dim = xq.dim();
  if ((dim != 4 && dim != 5) || xk.dim() != dim || xv.dim() != dim || ck.dim() != dim || cv.dim() != dim || !xq.is_cuda()) return py::none();
  const auto dev = xq.get_device();
  for (const Tensor* t : {&xq, &xk, &xv, &ck, &cv, &start_q, &start_k, &len_k})
    if (!plain_cuda(*t, dev)) return py::none();
  for (const Tensor* t : {&start_q, &start_k, &len_k})
    if (t->scalar_type() != at::kInt || !t->is_contiguous()) return py::none();
  const View q(xq), k(xk), v(xv), c(ck), d(cv);
  const int dt = dtype_code(xq.scalar_type());
  if (dt < 0 || xk.scalar_type() != xq.scalar_type() || xv.scalar_type() != xq.scalar_type() || cv.scalar_type() != ck.scalar_type()) return py::none();
  const bool int4 = ck.scalar_type() == at::kInt;
  if (!int4 && ck.scalar_type() != xq.scalar_type()) return py::none();
  if (int4 && (dt == XFB200_F32 || q.D % 8)) return py::none();
  if (q.B != 1 || k.B != 1 || v.B != 1 || c.B != 1 || d.B != 1 || q.M != total_q || k.M != total_q || v.M != total_q || n < 1) return py::none();
  if (k.G != q.G || v.G != q.G || c.G != q.G || d.G != q.G || k.D != q.D || v.D != q.D || v.H != k.H) return py::none();
  const int64_t row = int4 ? 1 + q.D / 8 : q.D;
  if (c.D != row || d.D != row) return py::none();
  const int64_t kv_heads = k.sh == 0 ? 1 : k.H;
  const int64_t cache_heads = kv_heads == 1 && c.sh == 0 ? c.H : kv_heads;
  if (c.H != cache_heads || d.H != cache_heads || c.M != d.M) return py::none();
  if (q.sd != 1 || k.sd != 1 || v.sd != 1 || c.sd != 1 || d.sd != 1) return py::none();
  xfb200_rope_params p{};
  if (tables.has_value()) {
    const Tensor& t = *tables;
    if (!plain_cuda(t, dev) || t.scalar_type() != at::kInt || t.dim() != 2 || t.size(0) != n || t.stride(1) != 1 || page < 1 || c.M % page) return py::none();
    p.block_tables = t.data_ptr<int32_t>(), p.block_tables_stride = t.stride(0), p.page_size = int32_t(page), p.pages_per_seq = int32_t(t.size(1));
  } else if (c.M != total_k) {
    return py::none();
  }
  const c10::cuda::CUDAGuard guard(dev);
  Tensor out_q;
  if (out_q_.has_value()) {
    out_q = *out_q_;
    if (!plain_cuda(out_q, dev) || out_q.scalar_type() != xq.scalar_type() || out_q.sizes() != xq.sizes() || out_q.stride(-1) != 1) return py::none();
  } else {
    out_q = at::empty(xq.sizes(), xq.options());
  }
  const View o(out_q);
  p.xq = xq.data_ptr(), p.xk = xk.data_ptr(), p.xv = xv.data_ptr(), p.out_q = out_q.data_ptr(), p.cache_k = ck.data_ptr(), p.cache_v = cv.data_ptr();
  p.seqstart_q = start_q.data_ptr<int32_t>(), p.seqstart_k = start_k.data_ptr<int32_t>(), p.seqlen_k = len_k.data_ptr<int32_t>();
  p.dtype = dt, p.batch = int32_t(n), p.max_q_per_seq = int32_t(max_q);
  p.q_heads = int32_t(q.H), p.kv_heads = int32_t(kv_heads), p.groups = int32_t(q.G), p.dim = int32_t(q.D);
  p.adjacents = adjacents, p.use_dynamic_scaling = dynamic, p.internal_f64 = f64, p.cache_format = int4 ? 1 : 0;
  p.theta = float(theta), p.linear_scale = float(linear_scale);
  p.dynamic_old_context_len = float(old_context_len), p.dynamic_scale_factor = float(scale_factor);
  p.dynamic_low_freq_factor = float(low_freq), p.dynamic_high_freq_factor = float(high_freq);
  auto put = [](const View& w, int64_t& m, int64_t& g, int64_t& h) { m = w.sm, g = w.five ? w.sg : 0, h = w.sh; };
  put(q, p.xq_m, p.xq_g, p.xq_h), put(k, p.xk_m, p.xk_g, p.xk_h), put(v, p.xv_m, p.xv_g, p.xv_h);
  put(o, p.oq_m, p.oq_g, p.oq_h), put(c, p.ck_m, p.ck_g, p.ck_h), put(d, p.cv_m, p.cv_g, p.cv_h);
  void* st = stream_of(dev);
  int rc;
  {
    py::gil_scoped_release nogil;
    rc = g_rope(&p, st);
  }
  return rc == XFB200_OK ? py::cast(out_q) : py::none();
}

}  // namespace

PYBIND11_MODULE(_front, m) {
  m.doc() = "Host front of the xformers_b200 operators (see csrc/front.cpp)";
  m.def("bind", &bind);
  m.def("split_k", [](int32_t batch, int64_t kv_bound, int32_t kv_heads, int32_t rows, int32_t row_bytes, bool quantised) {
    return g_split_k(batch, kv_bound, kv_heads, rows, row_bytes, quantised);
  });
  m.def("dense", &dense);
  m.def("varlen", &varlen);
  m.def("merge", &merge);
  m.def("rope", &rope);
  m.attr("WANT_LSE") = py::int_(int64_t(kWantLse));
  m.attr("PARTIAL") = py::int_(int64_t(kPartial));
  m.attr("DECODE_TAKES_BIAS") = py::int_(int64_t(kDecodeTakesBias));
  m.attr("PREFILL_TAKES_BIAS") = py::int_(int64_t(kPrefillTakesBias));
  m.attr("FORCE_DECODE") = py::int_(int64_t(kForceDecode));
  m.attr("FORCE_PREFILL") = py::int_(int64_t(kForcePrefill));
}
