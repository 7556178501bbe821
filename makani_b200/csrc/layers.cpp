// Forward and backward passes of whole layers on the GPU: allocations and launches without a return to Python in between.
//
// One launch from Python took 15 - 20 us of host time (operand objects, 40 converted integers, the binding), and the small networks
// and filters, whose kernels take 5 - 20 us each, waited for it (a training pass of a 32 x 64 network of 16 channels 2589 -> 1786 us,
// the AFNO filter of 90 x 180 tokens 461 -> 281).  Python says launch by launch what each pass does: `forward_stages` and
// `backward_stages` of ops/spectral.py and ops/afno.py, which also run the passes on the CPU (emulated), and `_conv_fwd`, `_conv_dgrad`
// and `_conv_wgrad` of ops/conv.py, of which convolutions, linear layers (tokens are a channels-last image) and MLPs are made.
// The instance norm is two launches in either direction, as for several GPUs in ops/norm.py.  Strides, and rules that pick among
// launches, are in both: tests/test_gpu_native_passes.py compares the two on the same tensors, bit by bit.
#include "host.h"

#include <pybind11/stl.h>

#include <algorithm>

#include "fused_ops.cuh"

namespace {

using mkh::Gemm;
using mkh::Tensor;
using OptTensor = c10::optional<Tensor>;

const __nv_bfloat16* bf(const Tensor& t) { return reinterpret_cast<const __nv_bfloat16*>(t.data_ptr()); }
__nv_bfloat16* bf_mut(const Tensor& t) { return reinterpret_cast<__nv_bfloat16*>(t.data_ptr()); }
const float* f32_or_null(const Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; }
float* f32_mut(const Tensor& t) { return t.defined() ? t.data_ptr<float>() : nullptr; }
Tensor empty_f32(at::IntArrayRef shape, const Tensor& like) { return at::empty(shape, like.options().dtype(at::kFloat)); }
// zeros in one or two tensors, one launch
void clear(Tensor& a, Tensor* b = nullptr) {
  ++mkh::launches();
  mkh::check(mk::clear_f32(a.data_ptr<float>(), a.numel(), b ? b->data_ptr<float>() : nullptr, b ? b->numel() : 0, mkh::stream()), "clear");
}
Tensor zeros_f32(at::IntArrayRef shape, const Tensor& like) {
  Tensor t = empty_f32(shape, like);
  clear(t);
  return t;
}
Tensor value(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }
OptTensor maybe(const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); }
// (a parameter on the host or another GPU is refused: its address would reach a kernel, or its copy be paid for on every call)
Tensor as_f32(const OptTensor& t, const Tensor& like) {
  if (!t.has_value() || !t->defined()) return Tensor();
  MK_CHECK(t->device() == like.device(), "layers: tensors must be on one CUDA device");
  return t->detach().to(at::kFloat).contiguous();
}

// ------------------------------------------------------------------------------------------ pointwise convolutions and linear layers

// An activation: tokens x channels, or [B, C, H, W] in one of its two dense layouts
struct Act {
  Tensor t;
  bool cl = true;
  int64_t B = 1, C = 0, T = 0;
};

Act act_of(const Tensor& t) {
  MK_CHECK(t.is_cuda() && t.scalar_type() == at::kBFloat16, "layers: bf16 CUDA activations expected");
  Act a;
  a.t = t;
  if (t.dim() == 2) {
    MK_CHECK(t.is_contiguous(), "layers: contiguous tokens expected");
    a.T = t.size(0);
    a.C = t.size(1);
    return a;
  }
  MK_CHECK(t.dim() == 4, "layers: tokens or [B, C, H, W] expected");
  a.B = t.size(0);
  a.C = t.size(1);
  a.T = t.size(2) * t.size(3);
  a.cl = !t.is_contiguous();
  MK_CHECK(!a.cl || t.is_contiguous(at::MemoryFormat::ChannelsLast), "layers: dense activation expected");
  return a;
}

// (an extent of 1 can make one tensor both layouts: the caller's choice is kept, as the strides of the launch go by it)
Act empty_act(const Act& like, int64_t C, bool cl) {
  const Tensor& t = like.t;
  Act a = like;
  a.C = C;
  if (t.dim() == 2) {
    a.t = at::empty({like.T, C}, t.options());
    return a;
  }
  a.cl = cl;
  a.t = at::empty({t.size(0), C, t.size(2), t.size(3)}, t.options(), cl ? at::MemoryFormat::ChannelsLast : at::MemoryFormat::Contiguous);
  return a;
}

mkh::Operand token_rows(const Act& x) {
  return x.cl ? mkh::Operand{&x.t, x.C, false, 0, x.T * x.C, 0} : mkh::Operand{&x.t, x.T, true, 0, x.C * x.T, 0};
}
mkh::Operand channel_rows(const Act& x) {
  return x.cl ? mkh::Operand{&x.t, x.C, true, 0, x.T * x.C, 0} : mkh::Operand{&x.t, x.T, false, 0, x.C * x.T, 0};
}

// fp32 [Co, Ci(, 1, 1)] -> bf16 [Co, pad8(Ci)], of one or two layers in one launch; bf16 weights of a linear layer as they are
void prep_weights(std::initializer_list<const Tensor*> ws, const Tensor& like, Tensor* out) {
  Tensor held[2];
  mk::CastPad jobs[2] = {};
  int n = 0;
  for (const Tensor* w : ws) {
    MK_CHECK(w->device() == like.device(), "layers: tensors must be on one CUDA device");
    const Tensor w2 = w->detach().reshape({w->size(0), -1});
    const int64_t co = w2.size(0), ci = w2.size(1), pitch = (ci + 7) / 8 * 8;
    if (like.dim() == 2 && w->dim() == 2 && w2.scalar_type() == like.scalar_type() && ci % 8 == 0) {
      *out++ = w2.contiguous();
    } else if (w2.scalar_type() == at::kFloat && w2.is_contiguous()) {
      *out = at::empty({co, pitch}, like.options());
      jobs[n] = {w2.data_ptr<float>(), bf_mut(*out), co, static_cast<int>(ci), static_cast<int>(pitch)};
      held[n++] = w2;
      ++out;
    } else {
      *out = at::zeros({co, pitch}, like.options());
      out->narrow(1, 0, ci).copy_(w2);
      ++out;
    }
  }
  if (n == 0) return;
  ++mkh::launches();
  mkh::check(n == 2 ? mk::cast_pad_bf16(jobs[0], jobs[1], mkh::stream()) : mk::cast_pad_bf16(jobs[0], mkh::stream()), "cast_pad");
}
Tensor prep_weight(const Tensor& w, const Tensor& like) {
  Tensor out;
  prep_weights({&w}, like, &out);
  return out;
}

void product(const Act& x, const mkh::Operand& w, int64_t ci, Act& y, Gemm g) {
  g.K = ci;
  g.zlo_n = x.B;
  if (y.cl) {
    g.M = y.T;
    g.N = y.C;
    g.A = token_rows(x);
    g.B = w;
    g.D.rs_lo = y.C;
    g.bias_mode = mkh::BIAS_COL;
  } else {
    g.M = y.C;
    g.N = y.T;
    g.A = w;
    g.B = token_rows(x);
    g.D.rs_lo = y.T;
    g.bias_mode = mkh::BIAS_ROW;
  }
  g.D.t = &y.t;
  g.D.d_zlo = y.C * y.T;
  if (!g.bias || !g.bias->defined()) g.bias_mode = mkh::BIAS_NONE;
  mkh::run(g);
}

// y = act(W x + b) (+ resid); `pre`: the second output
Act forward(const Act& x, const Tensor& wq, int64_t ci, const Tensor& bias, int act, const Tensor& resid, Tensor* pre, bool deriv, bool cl) {
  MK_CHECK(x.C == ci, "layers: the weight does not match the activation");
  Act y = empty_act(x, wq.size(0), cl);
  if (resid.defined()) MK_CHECK(act_of(resid).cl == cl && resid.sizes() == y.t.sizes(), "residual must have the layout of the output");
  Gemm g;
  g.bias = &bias;
  g.act = act;
  g.resid = &resid;
  if (pre) *pre = at::empty_like(y.t);
  g.preact = pre;
  g.preact_deriv = deriv;
  product(x, mkh::Operand{&wq, wq.size(1), false, 0, 0, 0}, ci, y, g);
  return y;
}

// dx = W^T dy (times `aux`)
Act data_gradient(const Act& dy, const Tensor& wq, int64_t ci, int act, const Tensor& aux, bool cl) {
  Act dx = empty_act(dy, ci, cl);
  Gemm g;
  g.act = act;
  g.resid = &aux;
  product(dy, mkh::Operand{&wq, wq.size(1), true, 0, 0, 0}, dy.C, dx, g);
  return dx;
}

// sums over batch and tokens, a pass of their own
Tensor channel_sums(const Act& x) {
  if (x.cl && x.C % 8 == 0 && (reinterpret_cast<uintptr_t>(x.t.data_ptr()) & 15) == 0) {
    Tensor out = empty_f32({x.C}, x.t);
    const int64_t n = mk::colsum_scratch(x.B * x.T, static_cast<int>(x.C), 1);
    Tensor part = empty_f32({n}, x.t);
    ++mkh::launches();
    mkh::check(mk::colsum(bf(x.t), out.data_ptr<float>(), n ? part.data_ptr<float>() : nullptr, x.B * x.T, static_cast<int>(x.C), mkh::stream()),
               "colsum");
    return out;
  }
  if (!x.cl) {
    Tensor sums = empty_f32({x.B * x.C, 2}, x.t);
    ++mkh::launches();
    mkh::check(mk::inorm_partial_stats(bf(x.t), sums.data_ptr<float>(), static_cast<int>(x.B * x.C), x.T, mkh::stream()), "inorm_partial_stats");
    return sums.select(1, 0).view({x.B, x.C}).sum(0);
  }
  return x.t.dim() == 2 ? x.t.to(at::kFloat).sum(0) : x.t.to(at::kFloat).sum(at::IntArrayRef{0, 2, 3});
}

// dw[co, ci] (cleared before) += sum over batch and tokens of dy x, and the sums of dy beside it: complete, or (`later`) once their slabs are
// added up
void weight_gradient(const Act& dy, const Act& x, Tensor& dw, Tensor* db, mkh::SumsLater* later = nullptr) {
  Gemm g;
  g.M = dy.C;
  g.N = x.C;
  g.K = x.T;
  g.A = channel_rows(dy);
  g.B = channel_rows(x);
  g.D.t = &dw;
  g.D.rs_lo = x.C;
  g.zlo_n = x.B;
  g.accumulate = true;
  g.splits = 0;
  Tensor sums;
  if (db) {
    sums = empty_f32({dy.C}, dy.t);
    g.row_sums = &sums;
    g.sums_later = later;
  }
  const bool done = mkh::run(g);
  if (db) *db = done ? sums : channel_sums(dy);
}

bool default_cl(int64_t co) { return co % 8 == 0; }
// layout codes: -1 that of the residual or the default, 0 NCHW, 1 channels-last
bool out_cl(int64_t layout, const Tensor& resid, int64_t co) {
  if (layout >= 0) return layout != 0;
  return resid.defined() ? act_of(resid).cl : default_cl(co);
}

std::tuple<Tensor, Tensor, OptTensor> conv_forward(const Tensor& x, const Tensor& w, const OptTensor& bias, const OptTensor& resid, int64_t act,
                                                   int64_t layout, bool want_pre) {
  c10::cuda::CUDAGuard guard(x.device());
  const Tensor wq = prep_weight(w, x), b = as_f32(bias, x), r = value(resid);
  Tensor pre;
  const Act y = forward(act_of(x), wq, w.size(1), b, static_cast<int>(act), r, want_pre ? &pre : nullptr, false, out_cl(layout, r, w.size(0)));
  return {y.t, wq, maybe(pre)};
}

std::tuple<OptTensor, OptTensor, OptTensor> conv_backward(const Tensor& dy, const Tensor& x, const Tensor& wq, int64_t ci, bool need_x, bool need_w,
                                                          bool need_b) {
  c10::cuda::CUDAGuard guard(x.device());
  const Act g = act_of(dy), xa = act_of(x);
  Tensor dx, dw, db;
  if (need_x) dx = data_gradient(g, wq, ci, mkh::ACT_NONE, Tensor(), xa.cl).t;
  if (need_w) {
    dw = zeros_f32({g.C, xa.C}, x);
    weight_gradient(g, xa, dw, need_b ? &db : nullptr);
  } else if (need_b) {
    db = channel_sums(g);
  }
  return {maybe(dx), maybe(dw), maybe(db)};
}

// y = W2 gelu(W1 x + b1) + b2 (+ resid); with `train` also what the backward pass reads: GELU' and the hidden activations
std::tuple<Tensor, Tensor, Tensor, OptTensor, OptTensor> mlp_forward(const Tensor& x, const Tensor& w1, const OptTensor& b1, const Tensor& w2,
                                                                     const OptTensor& b2, const OptTensor& resid, int64_t layout, bool train) {
  c10::cuda::CUDAGuard guard(x.device());
  Tensor wq[2];
  prep_weights({&w1, &w2}, x, wq);
  const Tensor &w1q = wq[0], &w2q = wq[1], b1f = as_f32(b1, x), b2f = as_f32(b2, x), r = value(resid);
  const int64_t ch = w1.size(0);
  Tensor dact;
  const Act h = forward(act_of(x), w1q, w1.size(1), b1f, mkh::ACT_GELU, Tensor(), train ? &dact : nullptr, train, default_cl(ch));
  const Act y = forward(h, w2q, ch, b2f, mkh::ACT_NONE, r, nullptr, false, out_cl(layout, r, w2.size(0)));
  return {y.t, w1q, w2q, maybe(dact), maybe(h.t)};
}

std::tuple<OptTensor, Tensor, OptTensor, Tensor, OptTensor> mlp_backward(const Tensor& dy, const Tensor& x, const Tensor& w1q, const Tensor& w2q,
                                                                         const Tensor& dact, const Tensor& h, int64_t ci, bool need_x, bool has_b1,
                                                                         bool has_b2) {
  c10::cuda::CUDAGuard guard(x.device());
  const Act g = act_of(dy), xa = act_of(x), ha = act_of(h);
  Tensor db1, db2, dx, dw1 = empty_f32({ha.C, xa.C}, x), dw2 = empty_f32({g.C, ha.C}, x);
  // (one launch each that clears both gradients, casts both weights, adds up both sums: at 16200 tokens every small launch costs some 4 us)
  clear(dw1, &dw2);
  const Act dpre = data_gradient(g, w2q, ha.C, mkh::ACT_MULAUX, dact, ha.cl);
  mkh::SumsLater s1, s2;
  weight_gradient(g, ha, dw2, has_b2 ? &db2 : nullptr, &s2);
  if (need_x) dx = data_gradient(dpre, w1q, ci, mkh::ACT_NONE, Tensor(), xa.cl).t;
  weight_gradient(dpre, xa, dw1, has_b1 ? &db1 : nullptr, &s1);
  if (s1.slabs.C > 0 || s2.slabs.C > 0)
    mkh::check(s1.slabs.C > 0 && s2.slabs.C > 0 ? mk::colsum_add_slabs(s1.slabs, s2.slabs, mkh::stream())
                                                : mk::colsum_add_slabs(s1.slabs.C > 0 ? s1.slabs : s2.slabs, mkh::stream()),
               "colsum_add_slabs");
  return {maybe(dx), dw1, maybe(db1), dw2, maybe(db2)};
}

// ------------------------------------------------------------------------------------------ instance norm, channels-last

std::tuple<Tensor, Tensor, OptTensor, OptTensor> norm_forward(const Tensor& x, const OptTensor& weight, const OptTensor& bias, double eps, int64_t act,
                                                              double count) {
  MK_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 4 && x.is_contiguous(at::MemoryFormat::ChannelsLast),
           "norm_forward: channels-last bf16 CUDA expected");
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t B = x.size(0), C = x.size(1), T = x.size(2) * x.size(3);
  Tensor y = at::empty_like(x), sums = zeros_f32({B, C, 2}, x), stats = empty_f32({B, C, 2}, x);
  const Tensor w = as_f32(weight, x), b = as_f32(bias, x);
  MK_CHECK((!w.defined() || w.numel() == C) && (!b.defined() || b.numel() == C), "norm_forward: one weight and bias per channel expected");
  mkh::launches() += 2;
  // statistics local to this device are accumulated around the first token (mode bit 1): no cancellation in E[x^2] - E[x]^2 for
  // fields with |mean| >> std
  mkh::check(mk::inorm_cl_sums(bf(x), nullptr, nullptr, nullptr, nullptr, sums.data_ptr<float>(), nullptr, nullptr, static_cast<int>(B),
                               static_cast<int>(C), T, 0, 2, mkh::error_word(x), mkh::stream()),
             "inorm_cl_sums");
  mkh::check(mk::inorm_cl_apply(bf(x), nullptr, bf_mut(y), f32_or_null(w), f32_or_null(b), sums.data_ptr<float>(), stats.data_ptr<float>(),
                                static_cast<int>(B), static_cast<int>(C), T, count, static_cast<float>(eps), static_cast<int>(act), 2, mkh::error_word(x),
                                mkh::stream()),
             "inorm_cl_apply");
  return {y, stats, maybe(w), maybe(b)};
}

std::tuple<Tensor, OptTensor, OptTensor> norm_backward(const Tensor& x, const Tensor& dy, const OptTensor& weight, const OptTensor& bias,
                                                       const Tensor& stats, bool affine, int64_t act, double count) {
  MK_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && dy.is_cuda() && dy.scalar_type() == at::kBFloat16 && dy.sizes() == x.sizes() &&
               x.is_contiguous(at::MemoryFormat::ChannelsLast) && dy.is_contiguous(at::MemoryFormat::ChannelsLast),
           "norm_backward: channels-last bf16 CUDA expected");
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t B = x.size(0), C = x.size(1), T = x.size(2) * x.size(3);
  const Tensor acc = zeros_f32({2 * B + (affine ? 2 : 0), C}, x), w = value(weight), b = value(bias);      // one clearing launch
  Tensor dx = at::empty_like(x), dw, db;
  if (affine) {
    dw = acc.select(0, 2 * B);
    db = acc.select(0, 2 * B + 1);
  }
  mkh::launches() += 2;
  mkh::check(mk::inorm_cl_sums(bf(x), bf(dy), f32_or_null(w), f32_or_null(b), stats.data_ptr<float>(), acc.data_ptr<float>(), f32_mut(dw), f32_mut(db),
                               static_cast<int>(B), static_cast<int>(C), T, static_cast<int>(act), 1, mkh::error_word(x), mkh::stream()),
             "inorm_cl_sums");
  mkh::check(mk::inorm_cl_apply(bf(x), bf(dy), bf_mut(dx), f32_or_null(w), f32_or_null(b), acc.data_ptr<float>(), stats.data_ptr<float>(),
                                static_cast<int>(B), static_cast<int>(C), T, count, 0.f, static_cast<int>(act), 1, mkh::error_word(x),
                                mkh::stream()),
             "inorm_cl_apply");
  return {dx, maybe(dw), maybe(db)};
}

// ------------------------------------------------------------------------------------------ spherical convolution

// `SHTPlan.native`: matrices [f, gt, pw, p, synthesis tables forward / inverse, analysis tables forward / inverse (or empty)] and
// extents [nlat, nlon, lmax, mmax]
struct Plan {
  const std::vector<Tensor>& t;
  int64_t nlat, nlon, k2;
  Plan(const std::vector<Tensor>& tables, const std::vector<int64_t>& n) : t(tables) {
    MK_CHECK(tables.size() == 8 && n.size() == 4, "spectral plan: eight tables and four extents expected");
    nlat = n[0];
    nlon = n[1];
    k2 = 2 * n[3];
  }
};

// (the rule of `folding_pays` in ops/spectral.py, which says why)
bool folding_pays(int64_t rows, int64_t folded_rows, int64_t k, int64_t folded_k, int64_t C) {
  auto up = [](int64_t a, int64_t b) { return (a + b - 1) / b; };
  auto tiles = [&](int64_t r, int64_t w) { return up(r, 128) * up(C, w) * w; };
  return tiles(folded_rows, 128) * (2 * up(folded_k, 64) + 1) < tiles(rows, mk::gemm_plain_columns(static_cast<int>(C))) * (up(k, 64) + 1);
}

Tensor analyse(const Tensor& x, const Plan& p, bool forward) {
  const int64_t B = x.size(0), C = x.size(1), H = x.size(2), W = x.size(3), k2 = p.k2;
  MK_CHECK(H == p.nlat && W == p.nlon, "spectral plan: the grid does not match the field");
  Tensor t1 = at::empty({B, H, k2, C}, x.options());
  const Tensor& fold = p.t[forward ? 6 : 7];
  if (fold.numel() && (folding_pays(k2, 2 * (W / 4 + 1), W, W / 2, C) || (forward && W % 8 != 0))) {
    mkh::folded_product(fold, x, t1, {5, k2, 2 * (W / 4 + 1), C, W / 2, W, B * H, fold.size(1), fold.size(1) / 2, 0, 1, 2 * C, W * C, C, 0, C, k2 * C});
    return t1;
  }
  const Tensor& m = p.t[forward ? 0 : 1];
  Gemm g;
  g.M = k2; g.N = C; g.K = W;
  g.A = {&m, m.size(1), !forward, 0, 0, 0};
  g.B = {&x, C, true, 0, W * C, H * W * C};
  g.D.t = &t1; g.D.rs_lo = C; g.D.d_zlo = k2 * C; g.D.d_zhi = H * k2 * C;
  g.zlo_n = H; g.zhi_n = B;
  mkh::run(g);
  return t1;
}

Tensor synthesise(const Tensor& t4, const Plan& p, bool forward) {
  const int64_t B = t4.size(0), H = t4.size(1), k2 = t4.size(2), C = t4.size(3), W = p.nlon;
  Tensor y = at::empty({B, C, H, W}, t4.options(), at::MemoryFormat::ChannelsLast);
  const Tensor& fold = p.t[forward ? 4 : 5];
  if (fold.numel() && (folding_pays(W, W / 2 + 1, k2, k2 / 2, C) || (forward && W % 8 != 0))) {
    mkh::folded_product(fold, t4, y, {4, W, W / 2 + 1, C, k2 / 2, W, B * H, fold.size(1), fold.size(1) / 2, 0, 1, 2 * C, k2 * C, C, 0, C, W * C});
    return y;
  }
  const Tensor& m = p.t[forward ? 0 : 1];
  Gemm g;
  g.M = W; g.N = C; g.K = k2;
  g.A = {&m, m.size(1), forward, 0, 0, 0};
  g.B = {&t4, C, true, 0, k2 * C, H * k2 * C};
  g.D.t = &y; g.D.rs_lo = C; g.D.d_zlo = W * C; g.D.d_zhi = H * W * C;
  g.zlo_n = H; g.zhi_n = B;
  mkh::run(g);
  return y;
}

Tensor legendre_analysis(const Tensor& t1, const Tensor& table, bool by_order) {
  const int64_t B = t1.size(0), H = t1.size(1), k2 = t1.size(2), C = t1.size(3), n2 = 2 * C;
  const int64_t mmax = table.size(0), lmax = table.size(1), pitch = table.size(2);
  Tensor t2 = by_order ? at::empty({B, mmax, lmax, n2}, t1.options()) : at::empty({B, lmax, mmax, n2}, t1.options());
  Gemm g;
  g.M = lmax; g.N = n2; g.K = H;
  g.A = {&table, pitch, false, 0, 0, lmax * pitch};
  g.B = {&t1, k2 * C, true, 0, H * k2 * C, n2};
  g.D.t = &t2; g.D.rs_lo = by_order ? n2 : mmax * n2; g.D.d_zhi = by_order ? lmax * n2 : n2; g.D.d_zlo = lmax * mmax * n2;
  g.zhi_n = mmax; g.zlo_n = B;
  g.tri.rmin_a = 1;
  mkh::run(g);
  return t2;
}

Tensor legendre_synthesis(const Tensor& t, bool lm_order, const Tensor& table, int64_t H) {
  const int64_t B = t.size(0), lmax = t.size(lm_order ? 1 : 2), mmax = t.size(lm_order ? 2 : 1), n2 = t.size(3), pitch = table.size(2);
  Tensor t4 = at::empty({B, H, 2 * mmax, n2 / 2}, t.options());
  Gemm g;
  g.M = H; g.N = n2; g.K = lmax;
  g.A = {&table, pitch, true, 0, 0, lmax * pitch};
  g.B = {&t, lm_order ? mmax * n2 : n2, true, 0, lmax * mmax * n2, lm_order ? n2 : lmax * n2};
  g.D.t = &t4; g.D.rs_lo = mmax * n2; g.D.d_zhi = n2; g.D.d_zlo = H * mmax * n2;
  g.zhi_n = mmax; g.zlo_n = B;
  g.tri.kmin_a = 1;
  mkh::run(g);
  return t4;
}

// wx: the planes [l, 2, Co, Ci] of the weights
Tensor contract(const Tensor& t2, const Tensor& wx, bool adjoint, const Tensor& resid) {
  const int64_t B = t2.size(0), lmax = t2.size(1), mmax = t2.size(2), kin = t2.size(3), co = wx.size(2), ci = wx.size(3);
  const int64_t n = adjoint ? ci : co, k = adjoint ? co : ci;
  Tensor t3 = at::empty({B, mmax, lmax, 2 * n}, t2.options());
  mkh::complex_product(t2, wx, t3, &resid,
                       {adjoint ? 2 : 1, mmax, n, k, B, lmax, 1, 1, 0, mkh::BIG, 0, 0, kin, lmax * mmax * kin, mmax * kin, 0, 0, adjoint ? 1 : 0, ci,
                        2 * co * ci, co * ci, 0, lmax * 2 * n, n, mmax * lmax * 2 * n, 2 * n, 0});
  return t3;
}

// dw[c, o, l] from dt [B, l, m, (ri, o)] and t2 [B, l, m, (ri, c)]: each sample a sum of its own
Tensor spectral_weight_gradient(const Tensor& dt, const Tensor& t2) {
  MK_CHECK(dt.is_cuda() && t2.is_cuda() && dt.device() == t2.device() && dt.scalar_type() == at::kBFloat16 && t2.scalar_type() == at::kBFloat16 &&
               dt.dim() == 4 && t2.dim() == 4 && dt.is_contiguous() && t2.is_contiguous() && dt.sizes().slice(0, 3) == t2.sizes().slice(0, 3) &&
               dt.size(3) % 16 == 0 && t2.size(3) % 16 == 0,
           "spectral weight gradient: contiguous bf16 CUDA coefficients of a multiple of 8 channels expected");
  c10::cuda::CUDAGuard guard(dt.device());
  const int64_t B = dt.size(0), L = dt.size(1), M = dt.size(2), co = dt.size(3) / 2, ci = t2.size(3) / 2;
  Tensor dw = at::empty({ci, co, L}, dt.options().dtype(at::kComplexFloat));
  if (mk::spectral_wgrad_pays(static_cast<int>(co), static_cast<int>(ci), static_cast<int>(L), static_cast<int>(B))) {
    ++mkh::launches();
    mkh::check(mk::spectral_wgrad(bf(dt), bf(t2), reinterpret_cast<float*>(dw.data_ptr()), static_cast<int>(co), static_cast<int>(ci), static_cast<int>(L),
                                  static_cast<int>(M), mkh::error_word(dt), mkh::stream()),
               "spectral_wgrad");
    return dw;
  }
  Tensor planes = B > 1 ? zeros_f32({2, L, co, ci}, dt) : empty_f32({2, L, co, ci}, dt);
  for (int64_t b = 0; b < B; ++b)
    mkh::complex_product(dt, t2, planes, nullptr,
                         {3, co, ci, M, 1, L, 0, mkh::BIG, 1, 1, b * L * M * 2 * co, 1, 2 * co, 0, M * 2 * co, co,
                          b * L * M * 2 * ci, 1, 2 * ci, M * 2 * ci, ci, 0, ci, L * co * ci, 0, co * ci, B > 1 ? 1 : 0});
  ++mkh::launches();
  mkh::check(mk::spectral_fold(planes.data_ptr<float>(), reinterpret_cast<float*>(dw.data_ptr()), static_cast<int>(ci), static_cast<int>(co),
                               static_cast<int>(L), mkh::stream(), 1, 1),
             "spectral_fold");
  return dw;
}

std::tuple<Tensor, OptTensor, Tensor> spectral_forward(const Tensor& x, const Tensor& wx, const std::vector<Tensor>& in, const std::vector<int64_t>& in_n,
                                                       const std::vector<Tensor>& out, const std::vector<int64_t>& out_n, bool want_resid) {
  MK_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 4 && x.is_contiguous(at::MemoryFormat::ChannelsLast),
           "spectral_forward: channels-last bf16 CUDA expected");
  c10::cuda::CUDAGuard guard(x.device());
  const Plan pi(in, in_n), po(out, out_n);
  MK_CHECK(wx.dim() == 4 && wx.size(3) == x.size(1) && wx.size(0) == in[2].size(1), "spectral_forward: the weights do not match the field");
  const Tensor t2 = legendre_analysis(analyse(x, pi, true), in[2], false);
  Tensor t3 = contract(t2, wx, false, Tensor());
  Tensor t4 = legendre_synthesis(t3, false, out[3], po.nlat);
  t3.reset();
  const Tensor y = synthesise(t4, po, false);
  t4.reset();
  Tensor r;
  if (want_resid) r = synthesise(legendre_synthesis(t2, true, out[3], po.nlat), po, false);
  return {y, maybe(r), t2};
}

std::tuple<OptTensor, OptTensor> spectral_backward(const Tensor& dy, const OptTensor& dr, const Tensor& t2, const Tensor& wx, const std::vector<Tensor>& in,
                                                   const std::vector<int64_t>& in_n, const std::vector<Tensor>& out,
                                                   const std::vector<int64_t>& out_n, bool need_x, bool need_w) {
  MK_CHECK(dy.is_cuda() && dy.scalar_type() == at::kBFloat16 && dy.dim() == 4 && dy.is_contiguous(at::MemoryFormat::ChannelsLast),
           "spectral_backward: channels-last bf16 CUDA expected");
  c10::cuda::CUDAGuard guard(dy.device());
  const Plan pi(in, in_n), po(out, out_n);
  const Tensor dt3 = legendre_analysis(analyse(dy, po, false), out[3], false);
  Tensor dw, dx, dr2;
  if (need_w) dw = spectral_weight_gradient(dt3, t2);
  if (need_x) {
    if (dr.has_value() && dr->defined()) {
      // laid out by order, as the contraction writes: its epilogue adds the residual's share
      MK_CHECK(dr->is_cuda() && dr->scalar_type() == dy.scalar_type() && dr->dim() == 4 && dr->is_contiguous(at::MemoryFormat::ChannelsLast),
               "spectral_backward: the residual's gradient must be laid out like the output's");
      dr2 = legendre_analysis(analyse(*dr, po, false), out[3], true);
    }
    Tensor dt2 = contract(dt3, wx, true, dr2);
    dr2.reset();
    dx = synthesise(legendre_synthesis(dt2, false, in[2], pi.nlat), pi, true);
  }
  return {maybe(dx), maybe(dw)};
}

// ------------------------------------------------------------------------------------------ AFNO filter

// DFT matrices of an `AFNOPlan` [fw, fw_t, gw, gw_t, fh, gh] and extents [H, W, kept rows, kept columns, blocks]
struct Afno {
  const std::vector<Tensor>& t;
  int64_t H, W, nkx, nc, nb, B, C, bs;
  Afno(const std::vector<Tensor>& tables, const std::vector<int64_t>& n, const Tensor& x) : t(tables) {
    MK_CHECK(tables.size() == 6 && n.size() == 5, "AFNO plan: six matrices and five extents expected");
    H = n[0]; W = n[1]; nkx = n[2]; nc = n[3]; nb = n[4];
    B = x.size(0); C = x.size(3);
    bs = C / nb;
    MK_CHECK(x.size(1) == H && x.size(2) == W && bs * nb == C, "AFNO plan: the grid or the blocks do not match the tokens");
  }
  mkh::Operand table(int i) const { return {&t[i], t[i].size(1), false, 0, 0, 0}; }
};

// x [B, H, W, C] -> [B, ncols, H, 2, C]
Tensor afno_w_analysis(const Tensor& x, int matrix, const Afno& p) {
  Tensor out = at::empty({p.B, p.nc, p.H, 2, p.C}, x.options());
  Gemm g;
  g.M = 2 * p.nc; g.N = p.C; g.K = p.W;
  g.A = p.table(matrix);
  g.B = {&x, p.C, true, 0, p.W * p.C, p.H * p.W * p.C};
  g.D.t = &out; g.D.rs_lo = p.C; g.D.rdiv = 2; g.D.rs_hi = p.H * 2 * p.C; g.D.d_zlo = 2 * p.C; g.D.d_zhi = p.nc * p.H * 2 * p.C;
  g.zlo_n = p.H; g.zhi_n = p.B;
  mkh::run(g);
  return out;
}

// src [B ncols, nb, nkx, 2, bs] -> [H, B ncols, 2, C]
Tensor afno_h_blocks(const Tensor& src, const Afno& p) {
  Tensor out = at::empty({p.H, p.B * p.nc, 2, p.C}, src.options());
  Gemm g;
  g.M = 2 * p.H; g.N = p.bs; g.K = 2 * p.nkx;
  g.A = p.table(5);
  g.B = {&src, p.bs, true, 0, p.nkx * 2 * p.bs, p.nb * p.nkx * 2 * p.bs};
  g.D.t = &out; g.D.rs_lo = p.C; g.D.rdiv = 2; g.D.rs_hi = p.B * p.nc * 2 * p.C; g.D.d_zlo = p.bs; g.D.d_zhi = 2 * p.C;
  g.zlo_n = p.nb; g.zhi_n = p.B * p.nc;
  mkh::run(g);
  return out;
}

// src [H, B ncols, 2, C] -> [B, H, W, C], + resid
Tensor afno_w_synthesis(const Tensor& src, int matrix, const Afno& p, const Tensor& resid) {
  Tensor out = at::empty({p.B, p.H, p.W, p.C}, src.options());
  if (resid.defined()) MK_CHECK(resid.sizes() == out.sizes(), "AFNO filter: the skip must have the shape of the tokens");
  Gemm g;
  g.M = p.W; g.N = p.C; g.K = 2 * p.nc;
  g.A = p.table(matrix);
  g.B = {&src, p.C, true, 0, p.B * p.nc * 2 * p.C, p.nc * 2 * p.C};
  g.D.t = &out; g.D.rs_lo = p.C; g.D.d_zlo = p.W * p.C; g.D.d_zhi = p.H * p.W * p.C;
  g.zlo_n = p.H; g.zhi_n = p.B;
  g.resid = &resid;
  mkh::run(g);
  return out;
}

// t1 [B, ncols, H, 2, C] -> [B ncols nkx, nb, 2, bs] (the rule is that of `_stage_h_tokens` in ops/afno.py)
Tensor afno_h_tokens(const Tensor& t1, const Afno& p) {
  Tensor y = at::empty({p.B * p.nc * p.nkx, p.nb, 2, p.bs}, t1.options());
  Gemm g;
  g.M = 2 * p.nkx; g.K = 2 * p.H;
  g.A = p.table(4);
  g.D.t = &y; g.D.rs_lo = p.bs; g.D.rdiv = 2; g.D.rs_hi = 2 * p.C;
  if (p.bs >= 64 || p.nb * p.B * p.nc * ((2 * p.nkx + 127) / 128) <= 3 * mk::sm_count()) {
    g.N = p.bs;
    g.B = {&t1, p.C, true, 0, p.bs, p.H * 2 * p.C};
    g.D.d_zlo = 2 * p.bs; g.D.d_zhi = p.nkx * 2 * p.C;
    g.zlo_n = p.nb; g.zhi_n = p.B * p.nc;
  } else {
    g.N = p.C;
    g.B = {&t1, p.C, true, 0, p.H * 2 * p.C, p.nc * p.H * 2 * p.C};
    g.D.ndiv = p.bs; g.D.ns_hi = 2 * p.bs; g.D.d_zlo = p.nkx * 2 * p.C; g.D.d_zhi = p.nc * p.nkx * 2 * p.C;
    g.zlo_n = p.nc; g.zhi_n = p.B;
  }
  mkh::run(g);
  return y;
}

// src [B ncols nkx, nb, k] times the weights of each block -> [B ncols, nb, nkx, n] (the rule is that of `_tokens_to_blocks`)
void afno_tokens_to_blocks(const Tensor& src, const mkh::Operand& w, Tensor& out, const Afno& p, int64_t n, int64_t k, Gemm g) {
  const int64_t rows = (p.nkx + 127) / 128 * 128, cols = std::max<int64_t>(128, (n + 63) / 64 * 64);
  g.N = n; g.K = k;
  g.B = w;
  g.D.t = &out; g.D.rs_lo = n;
  g.zlo_n = p.nb;
  if (n > 128 || p.nkx * n >= 0.45 * rows * cols) {
    g.M = p.nkx;
    g.A = {&src, p.nb * k, false, 0, k, p.nkx * p.nb * k};
    g.D.d_zlo = p.nkx * n; g.D.d_zhi = p.nb * p.nkx * n;
    g.zhi_n = p.B * p.nc;
  } else {
    g.M = p.B * p.nc * p.nkx;
    g.A = {&src, p.nb * k, false, 0, k, 0};
    g.D.rdiv = p.nkx; g.D.rs_hi = p.nb * p.nkx * n; g.D.d_zlo = p.nkx * n;
  }
  mkh::run(g);
}

std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> afno_forward(const Tensor& x, const Tensor& w1, const OptTensor& b1, const Tensor& w2,
                                                                        const OptTensor& b2, const OptTensor& skip, const std::vector<Tensor>& tables,
                                                                        const std::vector<int64_t>& extents, double lam) {
  MK_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 4 && x.is_contiguous(), "afno_forward: contiguous bf16 CUDA tokens expected");
  c10::cuda::CUDAGuard guard(x.device());
  const Afno p(tables, extents, x);
  const int64_t nb = p.nb, bs = p.bs, hid = w1.size(3);
  MK_CHECK(nb <= 32767, "afno_forward: at most 32767 blocks");
  const Tensor w[2] = {w1.detach().to(at::kFloat).contiguous(), w2.detach().to(at::kFloat).contiguous()};
  const Tensor b[2] = {as_f32(b1, x), as_f32(b2, x)};
  Tensor wq[2], bq[2];
  mk::AfnoLayer l[2];
  for (int k = 0; k < 2; ++k) {
    const int64_t ni = k ? hid : bs, no = k ? bs : hid;
    MK_CHECK(w[k].is_cuda() && w[k].numel() == 2 * nb * ni * no && (!b[k].defined() || (b[k].is_cuda() && b[k].numel() == 2 * nb * no)),
             "afno_forward: weights [2, nb, in, out] and biases [2, nb, out] expected");
    wq[k] = at::empty({nb, 2 * no, 2 * ni}, x.options());
    if (b[k].defined()) bq[k] = empty_f32({nb, 2 * no}, x);
    l[k] = {w[k].data_ptr<float>(), f32_or_null(b[k]), bf_mut(wq[k]), f32_mut(bq[k]), static_cast<int>(ni), static_cast<int>(no)};
  }
  ++mkh::launches();
  mkh::check(mk::afno_pack(l[0], l[1], static_cast<int>(nb), mkh::stream()), "afno_pack");
  const Tensor y = afno_h_tokens(afno_w_analysis(x, 0, p), p);
  const int64_t T = p.B * p.nc * p.nkx;
  Tensor o1 = at::empty({T, nb, 2 * hid}, x.options()), o2 = at::empty({p.B * p.nc, nb, p.nkx, 2, bs}, x.options());
  Gemm g;
  g.M = T; g.N = 2 * hid; g.K = 2 * bs;
  g.A = {&y, 2 * p.C, false, 0, 2 * bs, 0};
  g.B = {&wq[0], 2 * bs, false, 0, 2 * hid * 2 * bs, 0};
  g.D.t = &o1; g.D.rs_lo = nb * 2 * hid; g.D.d_zlo = 2 * hid;
  g.zlo_n = nb;
  g.bias = &bq[0]; g.bias_mode = bq[0].defined() ? mkh::BIAS_COL : mkh::BIAS_NONE; g.bias_zs = 2 * hid;
  g.act = mkh::ACT_RELU;
  mkh::run(g);
  Gemm e;
  e.bias = &bq[1]; e.bias_mode = bq[1].defined() ? mkh::BIAS_COL : mkh::BIAS_NONE; e.bias_zs = 2 * bs;
  e.act = mkh::ACT_SHRINK;
  e.act_param = static_cast<float>(lam);
  afno_tokens_to_blocks(o1, {&wq[1], 2 * hid, false, 0, 2 * bs * 2 * hid, 0}, o2, p, 2 * bs, 2 * hid, e);
  const Tensor added = skip.has_value() && skip->defined() ? skip->contiguous() : Tensor();
  const Tensor out = afno_w_synthesis(afno_h_blocks(o2, p), 2, p, added);
  return {out, y, o1, o2, wq[0], wq[1]};
}

std::tuple<Tensor, Tensor, OptTensor, Tensor, OptTensor> afno_backward(const Tensor& dy, const Tensor& y, const Tensor& o1, const Tensor& o2,
                                                                       const Tensor& w1q, const Tensor& w2q, const std::vector<Tensor>& tables,
                                                                       const std::vector<int64_t>& extents, bool has_b1, bool has_b2, bool add_dy) {
  MK_CHECK(dy.is_cuda() && dy.scalar_type() == at::kBFloat16 && dy.dim() == 4 && dy.is_contiguous(), "afno_backward: contiguous bf16 CUDA tokens expected");
  c10::cuda::CUDAGuard guard(dy.device());
  const Afno p(tables, extents, dy);
  const int64_t nb = p.nb, bs = p.bs, nkx = p.nkx, hid = o1.size(2) / 2, Z = p.B * p.nc, T = Z * nkx;
  // fp32 sums of the packed weights and biases, cleared together
  const int64_t n1 = 2 * hid * 2 * bs * nb, n2 = 2 * hid * nb, n3 = 2 * bs * nb;
  const Tensor acc = zeros_f32({2 * n1 + n2 + n3}, dy);
  Tensor dw1 = acc.narrow(0, 0, n1), dw2 = acc.narrow(0, n1, n1), db1 = acc.narrow(0, 2 * n1, n2), db2 = acc.narrow(0, 2 * n1 + n2, n3);
  // adjoint of the synthesis along W, then along H with the shrinkage mask (saved output != 0) in the epilogue
  const Tensor dt4 = afno_w_analysis(dy, 3, p);
  Tensor do2 = at::empty_like(o2), do1 = at::empty_like(o1);
  {
    Gemm g;
    g.M = 2 * nkx; g.N = bs; g.K = 2 * p.H;
    g.A = p.table(4);
    g.B = {&dt4, p.C, true, 0, bs, p.H * 2 * p.C};
    g.D.t = &do2; g.D.rs_lo = bs; g.D.d_zlo = nkx * 2 * bs; g.D.d_zhi = nb * nkx * 2 * bs;
    g.zlo_n = nb; g.zhi_n = Z;
    g.act = mkh::ACT_DSHRINK; g.resid = &o2;
    mkh::run(g);
  }
  // second layer: data gradient with the ReLU mask (saved output > 0), weight gradient summed over the (b, ky) batches
  {
    Gemm g;
    g.M = nkx; g.N = 2 * hid; g.K = 2 * bs;
    g.A = {&do2, 2 * bs, false, 0, nkx * 2 * bs, nb * nkx * 2 * bs};
    g.B = {&w2q, 2 * hid, true, 0, 2 * bs * 2 * hid, 0};
    g.D.t = &do1; g.D.rs_lo = nb * 2 * hid; g.D.d_zlo = 2 * hid; g.D.d_zhi = nkx * nb * 2 * hid;
    g.zlo_n = nb; g.zhi_n = Z;
    g.act = mkh::ACT_DRELU; g.resid = &o1;
    mkh::run(g);
  }
  bool done;
  {
    Gemm g;
    g.M = 2 * bs; g.N = 2 * hid; g.K = nkx;
    g.A = {&do2, 2 * bs, true, 0, nkx * 2 * bs, nb * nkx * 2 * bs};
    g.B = {&o1, nb * 2 * hid, true, 0, 2 * hid, nkx * nb * 2 * hid};
    g.D.t = &dw2; g.D.rs_lo = 2 * hid; g.D.d_zlo = 2 * bs * 2 * hid;
    g.zlo_n = nb; g.zhi_n = Z;
    g.accumulate = true; g.splits = 0;
    g.row_sums = has_b2 ? &db2 : nullptr;
    done = mkh::run(g);
  }
  if (has_b2 && !done) {
    const int64_t n = mk::colsum_scratch(Z * nkx, static_cast<int>(2 * bs), static_cast<int>(nb));
    Tensor part = empty_f32({n}, dy);
    ++mkh::launches();
    mkh::check(mk::colsum(bf(do2), db2.data_ptr<float>(), n ? part.data_ptr<float>() : nullptr, Z * nkx, static_cast<int>(2 * bs), mkh::stream(),
                          static_cast<int>(nb), nkx * 2 * bs, static_cast<int>(nkx), nb * nkx * 2 * bs),
               "colsum_groups");
  }
  // first layer
  Tensor dyt = at::empty({Z, nb, nkx, 2, bs}, dy.options());
  afno_tokens_to_blocks(do1, {&w1q, 2 * bs, true, 0, 2 * hid * 2 * bs, 0}, dyt, p, 2 * bs, 2 * hid, Gemm());
  {
    Gemm g;
    g.M = 2 * hid; g.N = 2 * bs; g.K = T;
    g.A = {&do1, nb * 2 * hid, true, 0, 2 * hid, 0};
    g.B = {&y, 2 * p.C, true, 0, 2 * bs, 0};
    g.D.t = &dw1; g.D.rs_lo = 2 * bs; g.D.d_zlo = 2 * hid * 2 * bs;
    g.zlo_n = nb;
    g.accumulate = true; g.splits = 0;
    g.row_sums = has_b1 ? &db1 : nullptr;
    done = mkh::run(g);
  }
  if (has_b1 && !done) {
    const int64_t n = mk::colsum_scratch(T, static_cast<int>(n2), 1);
    Tensor part = empty_f32({n}, dy);
    ++mkh::launches();
    mkh::check(mk::colsum(bf(do1), db1.data_ptr<float>(), n ? part.data_ptr<float>() : nullptr, T, static_cast<int>(n2), mkh::stream()), "colsum");
  }
  // gradients of the parameters as they are stored
  const Tensor gw1 = empty_f32({2, nb, bs, hid}, dy), gw2 = empty_f32({2, nb, hid, bs}, dy);
  Tensor gb1, gb2;
  if (has_b1) gb1 = empty_f32({2, nb, hid}, dy);
  if (has_b2) gb2 = empty_f32({2, nb, bs}, dy);
  mk::AfnoGrad l[2] = {{dw1.data_ptr<float>(), has_b1 ? db1.data_ptr<float>() : nullptr, gw1.data_ptr<float>(), f32_mut(gb1), static_cast<int>(bs),
                        static_cast<int>(hid)},
                       {dw2.data_ptr<float>(), has_b2 ? db2.data_ptr<float>() : nullptr, gw2.data_ptr<float>(), f32_mut(gb2), static_cast<int>(hid),
                        static_cast<int>(bs)}};
  ++mkh::launches();
  mkh::check(mk::afno_fold(l[0], l[1], static_cast<int>(nb), mkh::stream()), "afno_fold");
  // adjoint of the analysis along H and along W; the skip's gradient joins in the last epilogue
  const Tensor dx = afno_w_synthesis(afno_h_blocks(dyt, p), 1, p, add_dy ? dy : Tensor());
  return {dx, gw1, maybe(gb1), gw2, maybe(gb2)};
}

}  // namespace

namespace mkh {

void bind_layers(pybind11::module_& m) {
  m.def("conv_forward", &conv_forward);
  m.def("conv_backward", &conv_backward);
  m.def("mlp_forward", &mlp_forward);
  m.def("mlp_backward", &mlp_backward);
  m.def("norm_forward", &norm_forward);
  m.def("norm_backward", &norm_backward);
  m.def("spectral_forward", &spectral_forward);
  m.def("spectral_backward", &spectral_backward);
  m.def("spectral_weight_gradient", &spectral_weight_gradient);
  m.def("afno_forward", &afno_forward);
  m.def("afno_backward", &afno_backward);
}

}  // namespace mkh
