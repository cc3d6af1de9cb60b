// Host side of the T5 block's ops, from tensors to kernel launches.
//
// What bounds it: a training step of a small model, and a forward pass of one sentence, are
// limited by the host: through ctypes a GEMM took some 20 us from the Python call to the launch
// (28 converted arguments, a dozen tensor attributes, the current stream, an output allocation)
// while the kernel runs for 4 to 8 us. (T5.1.1 small with 8 + 8 layers, one sentence scored: 9.7 ms
// through ctypes, 3.8 so, 2.0 with the blocks of a layer as one call each, of which the device
// works 1.2.) These functions do the same from C++ for the plain case, contiguous activations and
// row-major bf16 weights, one call per op and direction. They return None for anything else, before
// doing anything; the Python wrappers then take their general path, which handles or rejects the call.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <optional>
#include <string>
#include <tuple>
#include <vector>

#include "t5x_b200.h"
#include "t5x_ops.h"

namespace {

using at::Tensor;
using std::optional;

void check(int rc, const char* what) {
  if (rc != 0) throw std::runtime_error(std::string(what) + ": " + t5x_last_error());
}

void* stream_of() { return at::cuda::getCurrentCUDAStream().stream(); }

bool aligned(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }

// Contiguous bf16 activations [..., k] on the current device.
bool plain(const Tensor& x) {
  return x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() >= 1 && x.is_contiguous() &&
         x.numel() > 0 && x.get_device() == c10::cuda::current_device() && aligned(x);
}

struct Weight {
  Tensor t;
  int64_t k, n, ld;  // row-major [k, n], rows ld apart
  bool ok;
  // [k, out...] as a [k, n] matrix
  explicit Weight(const Tensor& w, int64_t k_) : t(w), k(k_), n(0), ld(0), ok(false) {
    if (!w.is_cuda() || w.scalar_type() != at::kBFloat16 || w.dim() < 2 || w.size(0) != k || !aligned(w))
      return;
    if (w.dim() == 2 && w.stride(1) == 1) {
      n = w.size(1);
      ld = w.stride(0);
    } else if (w.is_contiguous()) {
      n = w.numel() / k;
      ld = n;
    } else {
      return;
    }
    // (a dimension below 8 can have the strides of either order)
    ok = k >= 8 && n >= 8 && k % 8 == 0 && n % 8 == 0 && ld % 8 == 0 && ld >= n;
  }
};

std::vector<int64_t> with_last(const Tensor& x, int64_t n) {
  std::vector<int64_t> s(x.sizes().begin(), x.sizes().end());
  s.back() = n;
  return s;
}

bool fits(int64_t v) { return v <= 0x7fffffff; }

// y[M, n] = x[M, k] @ w (+ residual)
void forward(const Tensor& x, int64_t m, const Weight& w, const Tensor* residual, Tensor& y, void* st) {
  check(t5x_gemm_bf16(x.data_ptr(), w.t.data_ptr(), nullptr, y.data_ptr(), m, w.n, w.k, 1, w.k, w.ld,
                      w.n, 0, 0, 0, 0, 1, 0, 0, residual ? 2 : 0,
                      residual ? residual->data_ptr() : nullptr, residual ? w.n : 0, 0, nullptr,
                      nullptr, 0, 1.f, 0, st),
        "gemm");
}
// dx[M, k] (+)= dy[M, n] @ w^T; dy rows ld_dy apart
void input_grad(const void* dy, int64_t ld_dy, int64_t m, const Weight& w, Tensor& dx, bool accumulate,
                void* st) {
  check(t5x_gemm_bf16(dy, w.t.data_ptr(), nullptr, dx.data_ptr(), m, w.k, w.n, 1, ld_dy, w.ld, w.k, 0,
                      0, 0, 0, 0, 0, accumulate, 0, nullptr, 0, 0, nullptr, nullptr, 0, 1.f, 0, st),
        "gemm");
}
// grad[k, n] (fp32) (+)= x^T @ dy
void weight_grad(const Tensor& x, const void* dy, int64_t ld_dy, int64_t m, const Weight& w,
                 Tensor& grad, bool accumulate, void* st) {
  check(t5x_gemm_wgrad_bf16(x.data_ptr(), dy, grad.data_ptr(), w.k, w.n, m, 1, w.k, ld_dy, w.n, 0, 0, 0,
                            1, 1, accumulate, 0, st),
        "gemm_wgrad");
}

// Products that share their input go out as one launch where there are two or three of them: fewer
// launches and last waves, rows read once, and an input gradient written once instead of read back
// and rounded between the products. us, as separate launches / as one, for three projections:
// 65536 tokens, 768 x 768, forward 189 / 174, input gradient 239 / 157, weight gradients 196 / 170;
// 16384 tokens, 1472 x 384, 85 / 69, 126 / 58, 108 / 73; 16384 tokens, 4096 x 4096, 1179 / 1139,
// 1175 / 1123, 1318 / 1276; 512 tokens, 512 x 384, 40 / 16, 39 / 20, 41 / 15.
constexpr size_t kGroup = 3;
bool groups(size_t n) { return n >= 2 && n <= kGroup; }

// y_i[M, n_i] = x[M, k] @ w_i
void forward_group(const Tensor& x, int64_t m, const std::vector<Weight>& w, std::vector<Tensor>& y,
                   void* st) {
  const void* b[kGroup];
  void* c[kGroup];
  int width[kGroup];
  long long ldb[kGroup], ldc[kGroup];
  for (size_t i = 0; i < w.size(); ++i) {
    b[i] = w[i].t.data_ptr();
    c[i] = y[i].data_ptr();
    width[i] = w[i].n;
    ldb[i] = w[i].ld;
    ldc[i] = w[i].n;
  }
  check(t5x_gemm_shared_bf16(x.data_ptr(), b, c, width, w.size(), m, w[0].k, w[0].k, ldb, ldc, 0, 1, 0, 0,
                             1, st),
        "gemm_shared");
}
// dx[M, k] = dy_0[M, n_0] @ w_0^T + dy_1 @ w_1^T + ...
void input_grad_group(const std::vector<const void*>& dy, const std::vector<long long>& ld_dy, int64_t m,
                      const std::vector<Weight>& w, Tensor& dx, void* st) {
  const void* b[kGroup];
  int width[kGroup];
  long long ldb[kGroup];
  for (size_t i = 0; i < w.size(); ++i) {
    b[i] = w[i].t.data_ptr();
    width[i] = w[i].n;
    ldb[i] = w[i].ld;
  }
  check(t5x_gemm_sum_bf16(dy.data(), b, dx.data_ptr(), width, w.size(), m, w[0].k, ld_dy.data(), ldb,
                          w[0].k, 0, 0, st),
        "gemm_sum");
}
// grad_i[k, n_i] (fp32) (+)= x^T @ dy_i
void weight_grad_group(const Tensor& x, const std::vector<const void*>& dy,
                       const std::vector<long long>& ld_dy, int64_t m, const std::vector<Weight>& w,
                       const std::vector<Tensor>& grad, bool accumulate, void* st) {
  void* c[kGroup];
  int width[kGroup];
  long long ldc[kGroup];
  for (size_t i = 0; i < w.size(); ++i) {
    c[i] = grad[i].data_ptr();
    width[i] = w[i].n;
    ldc[i] = w[i].n;
  }
  check(t5x_gemm_shared_bf16(x.data_ptr(), dy.data(), c, width, w.size(), w[0].k, m, w[0].k, ld_dy.data(),
                             ldc, 1, 1, 1, accumulate, 0, st),
        "gemm_shared");
}

// Whether two contiguous tensors share memory.
bool overlap(const Tensor& a, const Tensor& b) {
  const char *pa = static_cast<const char*>(a.data_ptr()), *pb = static_cast<const char*>(b.data_ptr());
  return pa < pb + b.nbytes() && pb < pa + a.nbytes();
}

// The gradients of x @ w_i, i < n: into `dx` (if wanted) and `grads` (if wanted).
void backward_products(const Tensor& x, int64_t m, const std::vector<const void*>& dy,
                       const std::vector<long long>& ld_dy, const std::vector<Weight>& w,
                       optional<Tensor>& dx, const std::vector<Tensor>& grads,
                       const std::vector<bool>& accumulate, void* st) {
  const bool one_launch = groups(w.size());
  if (dx && one_launch)
    input_grad_group(dy, ld_dy, m, w, *dx, st);
  else if (dx)
    for (size_t i = 0; i < w.size(); ++i) input_grad(dy[i], ld_dy[i], m, w[i], *dx, i > 0, st);
  if (grads.empty()) return;
  // One launch writes its outputs side by side: a weight that stands in for two (tied projections) has
  // one gradient buffer, to which the products have to be added one after the other.
  bool apart = true;
  for (size_t i = 0; i < w.size(); ++i) {
    apart = apart && accumulate[i] == accumulate[0];
    for (size_t j = 0; j < i; ++j) apart = apart && !overlap(grads[i], grads[j]);
  }
  if (one_launch && apart) {
    weight_grad_group(x, dy, ld_dy, m, w, grads, accumulate[0], st);
  } else {
    for (size_t i = 0; i < w.size(); ++i) {
      Tensor g = grads[i];
      weight_grad(x, dy[i], ld_dy[i], m, w[i], g, accumulate[i], st);
    }
  }
}

// A gradient buffer the weight-gradient GEMM can write whole; narrow outputs over many rows are
// cut into K slices by the caller's general path.
bool grad_ok(const optional<Tensor>& g, const Weight& w, int64_t m) {
  return g.has_value() && g->is_cuda() && g->scalar_type() == at::kFloat && g->is_contiguous() &&
         g->numel() == w.k * w.n && ((w.k >= 256 && w.n >= 256) || m < 8192);
}

optional<Tensor> linear(const Tensor& x, const Tensor& weight, const optional<Tensor>& residual) {
  if (!plain(x)) return std::nullopt;
  const int64_t k = x.size(-1), m = x.numel() / k;
  const Weight w(weight, k);
  if (!w.ok || !fits(m)) return std::nullopt;
  if (residual && !(plain(*residual) && residual->numel() == m * w.n)) return std::nullopt;
  Tensor y = at::empty(with_last(x, w.n), x.options());
  forward(x, m, w, residual ? &*residual : nullptr, y, stream_of());
  return y;
}

optional<std::vector<Tensor>> multi_linear(const Tensor& x, const std::vector<Tensor>& weights) {
  if (!plain(x)) return std::nullopt;
  const int64_t k = x.size(-1), m = x.numel() / k;
  if (!fits(m)) return std::nullopt;
  for (const Tensor& t : weights)
    if (!Weight(t, k).ok) return std::nullopt;
  std::vector<Tensor> out;
  std::vector<Weight> w;
  for (const Tensor& t : weights) {
    w.emplace_back(t, k);
    out.push_back(at::empty(with_last(x, w.back().n), x.options()));
  }
  if (groups(w.size()))
    forward_group(x, m, w, out, stream_of());
  else
    for (size_t i = 0; i < w.size(); ++i) forward(x, m, w[i], nullptr, out[i], stream_of());
  return out;
}

// Input gradient (None unless wanted) of x @ W_0, x @ W_1, ...; the weight gradients go into
// `grads` (cleared of what was there unless `accumulate`). The outer value tells whether the call
// was covered.
optional<std::tuple<optional<Tensor>>> multi_linear_bwd(
    const std::vector<Tensor>& dys, const Tensor& x, const std::vector<Tensor>& weights,
    const std::vector<optional<Tensor>>& grads, const std::vector<bool>& accumulate, bool need_dx,
    bool need_dw) {
  if (!plain(x)) return std::nullopt;
  const int64_t k = x.size(-1), m = x.numel() / k;
  if (!fits(m)) return std::nullopt;
  for (size_t i = 0; i < dys.size(); ++i) {
    const Weight w(weights[i], k);
    if (!w.ok || !plain(dys[i]) || dys[i].numel() != m * w.n) return std::nullopt;
    if (need_dw && !grad_ok(grads[i], w, m)) return std::nullopt;
  }
  optional<Tensor> dx;
  if (need_dx) dx = at::empty_like(x);
  std::vector<const void*> dy;
  std::vector<long long> ld;
  std::vector<Weight> w;
  std::vector<Tensor> g;
  for (size_t i = 0; i < dys.size(); ++i) {
    w.emplace_back(weights[i], k);
    dy.push_back(dys[i].data_ptr());
    ld.push_back(w.back().n);
    if (need_dw) g.push_back(*grads[i]);
  }
  backward_products(x, m, dy, ld, w, dx, g, accumulate, stream_of());
  return std::make_tuple(dx);
}

// (gelu(x @ w0) * (x @ w1), the two pre-activations side by side if they are to be kept)
optional<std::tuple<Tensor, optional<Tensor>>> gated_in(const Tensor& x, const Tensor& w0, const Tensor& w1,
                                                        bool keep) {
  if (!plain(x)) return std::nullopt;
  const int64_t k = x.size(-1), m = x.numel() / k;
  const Weight a(w0, k), b(w1, k);
  if (!a.ok || !b.ok || !fits(m) || w0.dim() != 2 || w1.dim() != 2 || a.n != b.n || a.ld != b.ld)
    return std::nullopt;
  Tensor g = at::empty(with_last(x, a.n), x.options());
  optional<Tensor> h;
  char* h0 = nullptr;
  if (keep) {
    h = at::empty({m, 2 * a.n}, x.options());
    h0 = static_cast<char*>(h->data_ptr());
  }
  check(t5x_gemm_bf16(x.data_ptr(), w0.data_ptr(), w1.data_ptr(), g.data_ptr(), m, a.n, k, 1, k, a.ld,
                      a.n, 0, 0, 0, 0, 1, 0, 0, 1, nullptr, 0, 0, h0, keep ? h0 + a.n * 2 : nullptr, 2 * a.n,
                      1.f, 0, stream_of()),
        "gemm");
  return std::make_tuple(g, h);
}

// Backward of gated_in; `h` is overwritten with the gradients of the pre-activations.
optional<std::tuple<optional<Tensor>>> gated_in_bwd(const Tensor& dg, const Tensor& x,
                                                    const Tensor& w0, const Tensor& w1, Tensor h,
                                                    const optional<Tensor>& grad0,
                                                    const optional<Tensor>& grad1, bool acc0,
                                                    bool acc1, bool need_dx, bool need_dw) {
  if (!plain(x) || !plain(dg) || !plain(h)) return std::nullopt;
  const int64_t k = x.size(-1), m = x.numel() / k;
  const Weight a(w0, k), b(w1, k);
  if (!a.ok || !b.ok || !fits(m) || a.n != b.n || dg.numel() != m * a.n || h.numel() != 2 * m * a.n)
    return std::nullopt;
  if (need_dw && !(grad_ok(grad0, a, m) && grad_ok(grad1, b, m))) return std::nullopt;
  void* st = stream_of();
  optional<Tensor> dx;
  if (need_dx) dx = at::empty_like(x);  // what can run out of memory comes before `h` is overwritten
  check(t5x_gated_gelu_bwd(dg.data_ptr(), h.data_ptr(), m, a.n, 2 * a.n, a.n, 0, st),
        "gated_gelu_bwd");
  const char* d0 = static_cast<const char*>(h.data_ptr());
  const char* d1 = d0 + a.n * 2;
  std::vector<Tensor> g;
  if (need_dw) g = {*grad0, *grad1};
  backward_products(x, m, {d0, d1}, {2 * a.n, 2 * a.n}, {a, b}, dx, g, {acc0, acc1}, st);
  return std::make_tuple(dx);
}

optional<std::tuple<Tensor, Tensor>> rmsnorm(const Tensor& x, const Tensor& scale, double eps) {
  if (!plain(x) || scale.scalar_type() != at::kFloat || !scale.is_contiguous() ||
      scale.numel() != x.size(-1) || !scale.is_cuda())
    return std::nullopt;
  const int64_t d = x.size(-1), rows = x.numel() / d;
  if (!fits(rows)) return std::nullopt;
  Tensor y = at::empty_like(x);
  Tensor rstd = at::empty({rows}, x.options().dtype(at::kFloat));
  check(t5x_rmsnorm_fwd(x.data_ptr(), scale.data_ptr(), y.data_ptr(), rstd.data_ptr(), rows, d, eps,
                        stream_of()),
        "rmsnorm_fwd");
  return std::make_tuple(y, rstd);
}

// Scratch for the partial sums of a norm's scale gradient.
Tensor norm_partial(const Tensor& x, int64_t rows, int64_t d) {
  return at::empty({static_cast<int64_t>(t5x_rmsnorm_bwd_partial(rows, d))}, x.options().dtype(at::kFloat));
}

// dx (+ dres); adds to `dscale`
optional<Tensor> rmsnorm_bwd(const Tensor& dy, const Tensor& x, const Tensor& scale,
                             const Tensor& rstd, const optional<Tensor>& dres, Tensor dscale) {
  if (!plain(x) || !plain(dy) || dy.numel() != x.numel() || scale.scalar_type() != at::kFloat ||
      !scale.is_contiguous() || scale.numel() != x.size(-1) || dscale.scalar_type() != at::kFloat ||
      !dscale.is_contiguous() || dscale.numel() != scale.numel())
    return std::nullopt;
  if (dres && !(plain(*dres) && dres->numel() == x.numel())) return std::nullopt;
  const int64_t d = x.size(-1), rows = x.numel() / d;
  if (!fits(rows)) return std::nullopt;
  Tensor dx = at::empty_like(x), partial = norm_partial(x, rows, d);
  check(t5x_rmsnorm_bwd(dy.data_ptr(), x.data_ptr(), scale.data_ptr(), rstd.data_ptr(),
                        dres ? dres->data_ptr() : nullptr, dx.data_ptr(), dscale.data_ptr(),
                        partial.data_ptr(), rows, d, stream_of()),
        "rmsnorm_bwd");
  return dx;
}

// [B, L, H, D] bf16 on the current device, channels contiguous, rows on 16-byte boundaries.
bool heads_ok(const Tensor& t) {
  return t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.dim() == 4 && t.numel() > 0 &&
         t.stride(3) == 1 && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 && t.stride(2) % 8 == 0 &&
         aligned(t) && t.get_device() == c10::cuda::current_device();
}

const void* data_or_null(const optional<Tensor>& t) { return t ? t->data_ptr() : nullptr; }

// What the caller has prepared for flash attention: an fp32 bias table with int32 buckets, a uint8
// key mask, int32 segment codes, all contiguous (checked where they are made).
struct Masks {
  optional<Tensor> rel_bias, buckets, key_mask, q_seg, kv_seg;
  int64_t causal, causal_off, rel_off;
  int num_buckets() const { return rel_bias ? rel_bias->size(1) : 0; }
  int nrel() const { return rel_bias ? buckets->size(0) : 0; }
  const void* bucket_data() const { return rel_bias ? buckets->data_ptr() : nullptr; }
};

// `kernel`: 0, 1 or 2, of KERNELS in t5x_b200/ops/attention.py.
void attention_into(const Tensor& q, const Tensor& k, const Tensor& v, const Masks& m, int64_t kernel,
                    Tensor& o, Tensor& lse, void* st) {
  const int B = q.size(0), Lq = q.size(1), H = q.size(2), D = q.size(3), Lk = k.size(1);
  if (kernel != 0)
    check((kernel == 2 ? t5x_attention_fwd_few : t5x_attention_fwd)(
              q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(), B,
              H, Lq, Lk, q.stride(0), q.stride(1), q.stride(2), k.stride(0),
              k.stride(1), k.stride(2), v.stride(0), v.stride(1), v.stride(2),
              o.stride(0), o.stride(1), o.stride(2), data_or_null(m.rel_bias),
              m.bucket_data(), m.num_buckets(), m.nrel(), m.rel_off,
              data_or_null(m.key_mask), data_or_null(m.q_seg), data_or_null(m.kv_seg),
              m.causal, m.causal_off, st),
          "attention_fwd");
  else
    check(t5x_attention_fwd_stream(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(),
                                   lse.data_ptr(), B, H, Lq, Lk, D, q.stride(0), q.stride(1),
                                   q.stride(2), k.stride(0), k.stride(1), k.stride(2), v.stride(0),
                                   v.stride(1), v.stride(2), o.stride(0), o.stride(1), o.stride(2),
                                   data_or_null(m.rel_bias), m.bucket_data(), m.num_buckets(),
                                   m.nrel(), m.rel_off, data_or_null(m.key_mask),
                                   data_or_null(m.q_seg), data_or_null(m.kv_seg), m.causal,
                                   m.causal_off, st),
          "attention_fwd");
}

optional<std::tuple<Tensor, Tensor>> attention(
    const Tensor& q, const Tensor& k, const Tensor& v, const optional<Tensor>& rel_bias,
    const optional<Tensor>& buckets, const optional<Tensor>& key_mask, const optional<Tensor>& q_seg,
    const optional<Tensor>& kv_seg, int64_t causal, int64_t causal_off, int64_t rel_off,
    int64_t kernel) {
  if (!heads_ok(q) || !heads_ok(k) || !heads_ok(v)) return std::nullopt;
  Tensor o = at::empty(q.sizes(), q.options());
  Tensor lse = at::empty({q.size(0), q.size(2), q.size(1)}, q.options().dtype(at::kFloat));
  attention_into(q, k, v, {rel_bias, buckets, key_mask, q_seg, kv_seg, causal, causal_off, rel_off},
                 kernel, o, lse, stream_of());
  return std::make_tuple(o, lse);
}

// (dq, dk, dv); dq, dk and dv are the column blocks of one buffer when q, k and v are (`packed`).
std::tuple<Tensor, Tensor, Tensor> attention_gradients(const Tensor& d_o, const Tensor& q,
                                                       const Tensor& k, const Tensor& v,
                                                       const Tensor& o, const Tensor& lse,
                                                       const Masks& m, const optional<Tensor>& d_rel,
                                                       bool packed, void* st) {
  const int B = q.size(0), Lq = q.size(1), H = q.size(2), D = q.size(3), Lk = k.size(1);
  const auto f32 = q.options().dtype(at::kFloat);
  const int head = t5x_attention_bwd_head_covers(B, H, Lq, Lk, D, m.num_buckets());
  Tensor dq, dk, dv;
  if (packed) {
    Tensor all = at::empty({B, Lq, 3, H, D}, q.options());
    dq = all.select(2, 0);
    dk = all.select(2, 1);
    dv = all.select(2, 2);
  } else {
    if (head) dq = at::empty({B, Lq, H, D}, q.options());
    dk = at::empty({B, Lk, H, D}, q.options());
    dv = at::empty({B, Lk, H, D}, q.options());
  }
  if (head) {
    optional<Tensor> dk32, dv32;  // what parts of the queries add to
    if (head == 2) {
      dk32 = at::zeros({B, Lk, H, D}, f32);
      dv32 = at::zeros({B, Lk, H, D}, f32);
    }
    check(t5x_attention_bwd_head(
              q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), d_o.data_ptr(), lse.data_ptr(),
              dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), dk32 ? dk32->data_ptr() : nullptr,
              dv32 ? dv32->data_ptr() : nullptr, B, H, Lq, Lk, q.stride(0), q.stride(1),
              q.stride(2), k.stride(0), k.stride(1), k.stride(2), v.stride(0), v.stride(1), v.stride(2),
              o.stride(0), o.stride(1), o.stride(2), d_o.stride(0), d_o.stride(1), d_o.stride(2),
              dq.stride(0), dq.stride(1), dq.stride(2), dk.stride(0), dk.stride(1), dk.stride(2),
              data_or_null(m.rel_bias), m.bucket_data(), d_rel ? d_rel->data_ptr() : nullptr,
              m.num_buckets(), m.nrel(), m.rel_off, data_or_null(m.key_mask), data_or_null(m.q_seg),
              data_or_null(m.kv_seg), m.causal, m.causal_off, st),
          "attention_bwd");
    if (dk32) {
      dk.copy_(*dk32);
      dv.copy_(*dv32);
    }
    return std::make_tuple(dq, dk, dv);
  }
  Tensor dq32 = at::zeros({B, Lq, H, D}, f32), delta = at::empty({B, H, Lq}, f32);
  check(t5x_attention_bwd(
            q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), d_o.data_ptr(), lse.data_ptr(),
            delta.data_ptr(), dq32.data_ptr(), dk.data_ptr(), dv.data_ptr(), B, H, Lq, Lk, D,
            q.stride(0), q.stride(1), q.stride(2), k.stride(0), k.stride(1), k.stride(2), v.stride(0),
            v.stride(1), v.stride(2), o.stride(0), o.stride(1), o.stride(2), d_o.stride(0),
            d_o.stride(1), d_o.stride(2), dk.stride(0), dk.stride(1), dk.stride(2),
            data_or_null(m.rel_bias), m.bucket_data(), d_rel ? d_rel->data_ptr() : nullptr,
            m.num_buckets(), m.nrel(), m.rel_off, data_or_null(m.key_mask), data_or_null(m.q_seg),
            data_or_null(m.kv_seg), m.causal, m.causal_off, st),
        "attention_bwd");
  if (packed)
    dq.copy_(dq32);
  else
    dq = dq32.to(at::kBFloat16);
  return std::make_tuple(dq, dk, dv);
}

optional<std::tuple<Tensor, Tensor, Tensor>> attention_bwd(
    const Tensor& d_o, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o,
    const Tensor& lse, const optional<Tensor>& rel_bias, const optional<Tensor>& buckets,
    const optional<Tensor>& key_mask, const optional<Tensor>& q_seg, const optional<Tensor>& kv_seg,
    const optional<Tensor>& d_rel, int64_t causal, int64_t causal_off, int64_t rel_off, bool packed) {
  if (!heads_ok(d_o) || !heads_ok(q) || !heads_ok(k) || !heads_ok(v) || !heads_ok(o))
    return std::nullopt;
  return attention_gradients(d_o, q, k, v, o, lse,
                             {rel_bias, buckets, key_mask, q_seg, kv_seg, causal, causal_off, rel_off},
                             d_rel, packed, stream_of());
}

// ------------------------------------------------------------------------------------------------
// Whole blocks: a norm, the products around it and the residual, one call per direction. A layer
// is then two or three calls instead of a module call, an autograd node and an op each for seven
// or eleven kernels; what a step of a small model waits for is this (see ops/blocks.py for what is
// covered, and the times).
// ------------------------------------------------------------------------------------------------
bool norm_ok(const Tensor& scale, const Tensor& x) {
  return scale.is_cuda() && scale.scalar_type() == at::kFloat && scale.is_contiguous() &&
         scale.numel() == x.size(-1);
}
bool rows_fit(const Tensor& x) { return fits(x.numel() / x.size(-1)); }
int64_t rows_of(const Tensor& x) { return x.numel() / x.size(-1); }

std::tuple<Tensor, Tensor> norm_forward(const Tensor& x, const Tensor& scale, double eps, void* st) {
  const int64_t d = x.size(-1), rows = rows_of(x);
  Tensor y = at::empty_like(x), rstd = at::empty({rows}, x.options().dtype(at::kFloat));
  check(t5x_rmsnorm_fwd(x.data_ptr(), scale.data_ptr(), y.data_ptr(), rstd.data_ptr(), rows, d, eps, st),
        "rmsnorm_fwd");
  return std::make_tuple(y, rstd);
}
// The norm's input gradient plus that of the residual branch.
Tensor norm_backward(const Tensor& dh, const Tensor& x, const Tensor& scale, const Tensor& rstd,
                     const Tensor& dres, Tensor& dscale, void* st) {
  Tensor dx = at::empty_like(x), partial = norm_partial(x, rows_of(x), x.size(-1));
  check(t5x_rmsnorm_bwd(dh.data_ptr(), x.data_ptr(), scale.data_ptr(), rstd.data_ptr(), dres.data_ptr(),
                        dx.data_ptr(), dscale.data_ptr(), partial.data_ptr(), rows_of(x), x.size(-1), st),
        "rmsnorm_bwd");
  return dx;
}

// Weights wq, wk, wv, wo of an attention block over x [B, Lq, d] and (cross attention) kv, of `heads`
// heads, as many as the bias table was checked for.
bool attention_weights_ok(const Tensor& x, const Tensor& kv, const std::vector<Tensor>& w, int64_t heads,
                          int64_t head_dim) {
  if (w.size() != 4) return false;
  const Weight q(w[0], x.size(-1)), k(w[1], kv.size(-1)), v(w[2], kv.size(-1));
  if (!q.ok || !k.ok || !v.ok || q.n != k.n || q.n != v.n || q.n != heads * head_dim) return false;
  const Weight o(w[3], q.n);
  return o.ok && o.n == x.size(-1);
}
bool mlp_weights_ok(const Tensor& x, const std::vector<Tensor>& w) {
  if (w.size() != 3 || w[0].dim() != 2 || w[1].dim() != 2) return false;
  const Weight a(w[0], x.size(-1)), b(w[1], x.size(-1));
  if (!a.ok || !b.ok || a.n != b.n || a.ld != b.ld) return false;
  const Weight o(w[2], a.n);
  return o.ok && o.n == x.size(-1);
}

bool attention_block_ok(const Tensor& x, const optional<Tensor>& kv, const Tensor& scale,
                        const std::vector<Tensor>& w, int64_t heads, int64_t head_dim) {
  const Tensor& in = kv ? *kv : x;
  return x.dim() == 3 && plain(x) && rows_fit(x) && norm_ok(scale, x) &&
         (!kv || (kv->dim() == 3 && plain(*kv) && rows_fit(*kv) && kv->size(0) == x.size(0))) &&
         attention_weights_ok(x, in, w, heads, head_dim);
}
bool mlp_block_ok(const Tensor& x, const Tensor& scale, const std::vector<Tensor>& w) {
  return x.dim() >= 2 && plain(x) && rows_fit(x) && norm_ok(scale, x) && mlp_weights_ok(x, w);
}
// Gradient buffers that the weight-gradient kernels can write whole, for the weights above.
bool attention_grads_ok(const Tensor& x, const optional<Tensor>& kv, const std::vector<Tensor>& w,
                        const std::vector<optional<Tensor>>& g) {
  const Tensor& in = kv ? *kv : x;
  const Weight q(w[0], x.size(-1)), k(w[1], in.size(-1)), v(w[2], in.size(-1)), o(w[3], q.n);
  return grad_ok(g[0], q, rows_of(x)) && grad_ok(g[1], k, rows_of(in)) && grad_ok(g[2], v, rows_of(in)) &&
         grad_ok(g[3], o, rows_of(x));
}
bool mlp_grads_ok(const Tensor& x, const std::vector<Tensor>& w, const std::vector<optional<Tensor>>& g) {
  const Weight a(w[0], x.size(-1)), b(w[1], x.size(-1)), o(w[2], a.n);
  return grad_ok(g[0], a, rows_of(x)) && grad_ok(g[1], b, rows_of(x)) && grad_ok(g[2], o, rows_of(x));
}

// y = x + attention(rmsnorm(x)) wo, and what the backward pass needs: (y, h, rstd, q, k, v, o, lse).
// The keys and values come from `kv` where there is one, else from h.
std::vector<Tensor> attention_block(const Tensor& x, const optional<Tensor>& kv, const Tensor& scale,
                                    double eps, const std::vector<Tensor>& weights, int64_t heads,
                                    int64_t head_dim, const optional<Tensor>& rel_bias,
                                    const optional<Tensor>& buckets, const optional<Tensor>& key_mask,
                                    const optional<Tensor>& q_seg,
                                    const optional<Tensor>& kv_seg, int64_t causal, int64_t causal_off,
                                    int64_t rel_off, int64_t kernel) {
  if (!attention_block_ok(x, kv, scale, weights, heads, head_dim))
    throw std::invalid_argument("attention_block: operands are not covered");
  void* st = stream_of();
  auto [h, rstd] = norm_forward(x, scale, eps, st);
  const Tensor& in = kv ? *kv : h;
  const int64_t B = x.size(0), Lq = x.size(1), Lk = in.size(1), d = x.size(-1);
  const Weight wq(weights[0], d), wk(weights[1], in.size(-1)), wv(weights[2], in.size(-1)), wo(weights[3], wq.n);
  std::vector<Tensor> out;
  for (int64_t l : {Lq, Lk, Lk}) out.push_back(at::empty({B, l, heads, head_dim}, x.options()));
  if (kv) {
    forward(h, B * Lq, wq, nullptr, out[0], st);
    std::vector<Tensor> pair = {out[1], out[2]};
    forward_group(in, B * Lk, {wk, wv}, pair, st);
  } else {
    forward_group(h, B * Lq, {wq, wk, wv}, out, st);
  }
  Tensor o = at::empty({B, Lq, heads, head_dim}, x.options());
  Tensor lse = at::empty({B, heads, Lq}, x.options().dtype(at::kFloat));
  attention_into(out[0], out[1], out[2],
                 {rel_bias, buckets, key_mask, q_seg, kv_seg, causal, causal_off, rel_off}, kernel, o,
                 lse, st);
  Tensor y = at::empty_like(x);
  forward(o, B * Lq, wo, &x, y, st);
  return {y, h, rstd, out[0], out[1], out[2], o, lse};
}

// Gradients of attention_block: (dx, dkv or None). Weight gradients go into `grads` (cleared first
// unless `accumulate`), the norm's are added to `dscale`, the bias table's to `d_rel`.
std::tuple<Tensor, optional<Tensor>> attention_block_bwd(
    const Tensor& dy, const Tensor& x, const optional<Tensor>& kv, const Tensor& scale,
    const std::vector<Tensor>& weights, const std::vector<Tensor>& saved, const std::vector<Tensor>& grads,
    const std::vector<bool>& accumulate, Tensor dscale, const optional<Tensor>& d_rel, bool need_dkv,
    const optional<Tensor>& rel_bias, const optional<Tensor>& buckets, const optional<Tensor>& key_mask,
    const optional<Tensor>& q_seg, const optional<Tensor>& kv_seg, int64_t causal, int64_t causal_off,
    int64_t rel_off) {
  const Tensor &h = saved[0], &rstd = saved[1], &q = saved[2], &k = saved[3], &v = saved[4], &o = saved[5],
               &lse = saved[6];
  const std::vector<optional<Tensor>> g(grads.begin(), grads.end());
  if (!plain(dy) || dy.numel() != x.numel() ||
      !attention_block_ok(x, kv, scale, weights, q.size(2), q.size(3)) || !attention_grads_ok(x, kv, weights, g))
    throw std::invalid_argument("attention_block_bwd: operands are not covered");
  void* st = stream_of();
  const Tensor& in = kv ? *kv : h;
  const int64_t m = rows_of(x), mk = rows_of(in);
  const Weight wq(weights[0], x.size(-1)), wk(weights[1], in.size(-1)), wv(weights[2], in.size(-1)),
      wo(weights[3], wq.n);
  Tensor d_o = at::empty_like(o);
  input_grad(dy.data_ptr(), wo.n, m, wo, d_o, false, st);
  Tensor gwo = grads[3];
  weight_grad(o, dy.data_ptr(), wo.n, m, wo, gwo, accumulate[3], st);
  auto [dq, dk, dv] = attention_gradients(
      d_o, q, k, v, o, lse, {rel_bias, buckets, key_mask, q_seg, kv_seg, causal, causal_off, rel_off}, d_rel,
      false, st);
  optional<Tensor> dh = at::empty_like(x), dkv;
  if (kv) {
    if (need_dkv) dkv = at::empty_like(in);
    backward_products(in, mk, {dk.data_ptr(), dv.data_ptr()}, {wk.n, wv.n}, {wk, wv}, dkv,
                      {grads[1], grads[2]}, {accumulate[1], accumulate[2]}, st);
    backward_products(h, m, {dq.data_ptr()}, {wq.n}, {wq}, dh, {grads[0]}, {accumulate[0]}, st);
  } else {
    backward_products(h, m, {dq.data_ptr(), dk.data_ptr(), dv.data_ptr()}, {wq.n, wk.n, wv.n},
                      {wq, wk, wv}, dh, {grads[0], grads[1], grads[2]},
                      {accumulate[0], accumulate[1], accumulate[2]}, st);
  }
  return std::make_tuple(norm_backward(*dh, x, scale, rstd, dy, dscale, st), dkv);
}

// y = x + (gelu(h w0) * (h w1)) wo with h = rmsnorm(x): (y, h, rstd, g, pre-activations side by side).
std::vector<Tensor> mlp_block(const Tensor& x, const Tensor& scale, double eps,
                              const std::vector<Tensor>& weights, bool keep) {
  if (!mlp_block_ok(x, scale, weights)) throw std::invalid_argument("mlp_block: operands are not covered");
  void* st = stream_of();
  auto [h, rstd] = norm_forward(x, scale, eps, st);
  const int64_t m = rows_of(x), d = x.size(-1);
  const Weight a(weights[0], d), b(weights[1], d), wo(weights[2], a.n);
  Tensor g = at::empty({m, a.n}, x.options()), pre;
  char* h0 = nullptr;
  if (keep) {
    pre = at::empty({m, 2 * a.n}, x.options());
    h0 = static_cast<char*>(pre.data_ptr());
  }
  check(t5x_gemm_bf16(h.data_ptr(), a.t.data_ptr(), b.t.data_ptr(), g.data_ptr(), m, a.n, d, 1, d, a.ld, a.n, 0,
                      0, 0, 0, 1, 0, 0, 1, nullptr, 0, 0, h0, keep ? h0 + a.n * 2 : nullptr, 2 * a.n, 1.f, 0,
                      st),
        "gemm");
  Tensor y = at::empty_like(x);
  forward(g, m, wo, &x, y, st);
  if (!keep) return {y};
  return {y, h, rstd, g, pre};
}

// The same with one ReLU: y = x + relu(h wi) wo, weights wi, wo; (y, h, rstd, g). Covered where the products can
// do the activation and its gradient themselves.
bool relu_operands_ok(const Tensor& x, const Tensor& scale, const std::vector<Tensor>& w) {
  if (x.dim() < 2 || !plain(x) || !rows_fit(x) || !norm_ok(scale, x) || w.size() != 2 || w[0].dim() != 2)
    return false;
  const Weight a(w[0], x.size(-1));
  if (!a.ok) return false;
  const Weight o(w[1], a.n);
  return o.ok && o.n == x.size(-1);
}
bool relu_block_ok(const Tensor& x, const Tensor& scale, const std::vector<Tensor>& w) {
  return relu_operands_ok(x, scale, w) && t5x_gemm_relu_covers(rows_of(x), Weight(w[0], x.size(-1)).n);
}
bool relu_grads_ok(const Tensor& x, const std::vector<Tensor>& w, const std::vector<optional<Tensor>>& g) {
  const Weight a(w[0], x.size(-1)), o(w[1], a.n);
  return grad_ok(g[0], a, rows_of(x)) && grad_ok(g[1], o, rows_of(x)) && !overlap(*g[0], *g[1]);
}
std::vector<Tensor> relu_block(const Tensor& x, const Tensor& scale, double eps, const std::vector<Tensor>& weights,
                               bool keep) {
  if (!relu_block_ok(x, scale, weights)) throw std::invalid_argument("relu_block: operands are not covered");
  void* st = stream_of();
  auto [h, rstd] = norm_forward(x, scale, eps, st);
  const int64_t m = rows_of(x), d = x.size(-1);
  const Weight a(weights[0], d), wo(weights[1], a.n);
  Tensor g = at::empty({m, a.n}, x.options());
  check(t5x_gemm_relu(h.data_ptr(), a.t.data_ptr(), g.data_ptr(), nullptr, m, a.n, d, d, a.ld, a.n, 0, 1, st),
        "gemm_relu");
  Tensor y = at::empty_like(x);
  forward(g, m, wo, &x, y, st);
  if (!keep) return {y};
  return {y, h, rstd, g};
}
Tensor relu_block_bwd(const Tensor& dy, const Tensor& x, const Tensor& scale, const std::vector<Tensor>& weights,
                      const std::vector<Tensor>& saved, const std::vector<Tensor>& grads,
                      const std::vector<bool>& accumulate, Tensor dscale) {
  const Tensor &h = saved[0], &rstd = saved[1], &g = saved[2];
  const std::vector<optional<Tensor>> have(grads.begin(), grads.end());
  if (!plain(dy) || dy.numel() != x.numel() || !relu_operands_ok(x, scale, weights) ||
      !relu_grads_ok(x, weights, have))
    throw std::invalid_argument("relu_block_bwd: operands are not covered");
  void* st = stream_of();
  const int64_t m = rows_of(x), d = x.size(-1);
  const Weight a(weights[0], d), wo(weights[1], a.n);
  Tensor dg = at::empty_like(g);
  optional<Tensor> dh = at::empty_like(x);
  // (CTA pairs may have been switched off since the forward pass)
  if (t5x_gemm_relu_covers(m, a.n)) {
    check(t5x_gemm_relu(dy.data_ptr(), wo.t.data_ptr(), dg.data_ptr(), g.data_ptr(), m, a.n, wo.n, wo.n, wo.ld, a.n,
                        a.n, 0, st),
          "gemm_relu");
  } else {
    input_grad(dy.data_ptr(), wo.n, m, wo, dg, false, st);
    dg = at::threshold_backward(dg, g, 0);
  }
  Tensor gwo = grads[1];
  weight_grad(g, dy.data_ptr(), wo.n, m, wo, gwo, accumulate[1], st);
  backward_products(h, m, {dg.data_ptr()}, {a.n}, {a}, dh, {grads[0]}, {accumulate[0]}, st);
  return norm_backward(*dh, x, scale, rstd, dy, dscale, st);
}

// Input gradient of mlp_block; the saved pre-activations are overwritten with their gradients.
Tensor mlp_block_bwd(const Tensor& dy, const Tensor& x, const Tensor& scale,
                     const std::vector<Tensor>& weights, const std::vector<Tensor>& saved,
                     const std::vector<Tensor>& grads, const std::vector<bool>& accumulate, Tensor dscale) {
  const Tensor &h = saved[0], &rstd = saved[1], &g = saved[2], &pre = saved[3];
  const std::vector<optional<Tensor>> have(grads.begin(), grads.end());
  if (!plain(dy) || dy.numel() != x.numel() || !mlp_block_ok(x, scale, weights) ||
      !mlp_grads_ok(x, weights, have))
    throw std::invalid_argument("mlp_block_bwd: operands are not covered");
  void* st = stream_of();
  const int64_t m = rows_of(x), d = x.size(-1);
  const Weight a(weights[0], d), b(weights[1], d), wo(weights[2], a.n);
  const bool fused = t5x_gemm_gated_grad_covers(m, a.n) != 0;
  Tensor dg;
  if (!fused) dg = at::empty_like(g);
  optional<Tensor> dh = at::empty_like(x);  // what can run out of memory comes before `pre` is overwritten
  char* d0 = static_cast<char*>(pre.data_ptr());
  Tensor gwo = grads[2];
  if (fused) {
    weight_grad(g, dy.data_ptr(), wo.n, m, wo, gwo, accumulate[2], st);
    check(t5x_gemm_gated_grad(dy.data_ptr(), wo.t.data_ptr(), d0, d0 + a.n * 2, m, a.n, wo.n, wo.n, wo.ld, 2 * a.n,
                              0, st),
          "gemm_gated_grad");
  } else {
    input_grad(dy.data_ptr(), wo.n, m, wo, dg, false, st);
    weight_grad(g, dy.data_ptr(), wo.n, m, wo, gwo, accumulate[2], st);
    check(t5x_gated_gelu_bwd(dg.data_ptr(), pre.data_ptr(), m, a.n, 2 * a.n, a.n, 0, st), "gated_gelu_bwd");
  }
  backward_products(h, m, {d0, d0 + a.n * 2}, {2 * a.n, 2 * a.n}, {a, b}, dh, {grads[0], grads[1]},
                    {accumulate[0], accumulate[1]}, st);
  return norm_backward(*dh, x, scale, rstd, dy, dscale, st);
}

}  // namespace

// The GIL is released for the duration of a call: a launch waits when the device's queue is full,
// and the threads that prepare batches have to go on meanwhile.
PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("linear", torch::wrap_pybind_function_no_gil(linear));
  m.def("multi_linear", torch::wrap_pybind_function_no_gil(multi_linear));
  m.def("multi_linear_bwd", torch::wrap_pybind_function_no_gil(multi_linear_bwd));
  m.def("gated_in", torch::wrap_pybind_function_no_gil(gated_in));
  m.def("gated_in_bwd", torch::wrap_pybind_function_no_gil(gated_in_bwd));
  m.def("rmsnorm", torch::wrap_pybind_function_no_gil(rmsnorm));
  m.def("attention", torch::wrap_pybind_function_no_gil(attention));
  m.def("attention_bwd", torch::wrap_pybind_function_no_gil(attention_bwd));
  m.def("rmsnorm_bwd", torch::wrap_pybind_function_no_gil(rmsnorm_bwd));
  m.def("attention_block_ok", attention_block_ok);
  m.def("attention_grads_ok", attention_grads_ok);
  m.def("attention_block", torch::wrap_pybind_function_no_gil(attention_block));
  m.def("attention_block_bwd", torch::wrap_pybind_function_no_gil(attention_block_bwd));
  m.def("mlp_block_ok", mlp_block_ok);
  m.def("mlp_grads_ok", mlp_grads_ok);
  m.def("mlp_block", torch::wrap_pybind_function_no_gil(mlp_block));
  m.def("mlp_block_bwd", torch::wrap_pybind_function_no_gil(mlp_block_bwd));
  m.def("relu_block_ok", relu_block_ok);
  m.def("relu_grads_ok", relu_grads_ok);
  m.def("relu_block", torch::wrap_pybind_function_no_gil(relu_block));
  m.def("relu_block_bwd", torch::wrap_pybind_function_no_gil(relu_block_bwd));
}
