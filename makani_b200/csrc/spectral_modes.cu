// Mode-wise complex contractions of the spectral filters whose weights differ per (l, m) mode ("diagonal" operator)
// or act per channel ("separable"): for every mode a [B, Cin] x [Cin, Cout] complex product.  At batch sizes of one
// or two there is no tile shape for the tensor cores here; the work is streaming the weights once, so these are
// bandwidth kernels: threads run along the mode index (the contiguous one in activations and weights), every weight
// element is read exactly once per pair of batch samples and the activations of a block of modes are re-read from L2.
//
//   diag fwd : out[b, o, s] = sum_i a[b, i, s] w[i, o, s]
//   diag dA  : da[b, i, s]  = sum_o dy[b, o, s] conj(w[i, o, s])
//   diag dW  : dw[i, o, s]  = sum_b conj(a[b, i, s]) dy[b, o, s]
//   separable: out[b, i, s] = a[b, i, s] w[i, s'] with s' = s ("diagonal") or s' = s / M (per degree, "dhconv")
#include "spectral_modes.cuh"

#include <stdint.h>

namespace mk {

namespace {

__device__ __forceinline__ float2 cmul(float2 a, float2 b) { return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {   // a * conj(b)
  return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}
__device__ __forceinline__ void cfma(float2& acc, float2 a, float2 b) {
  acc.x = fmaf(a.x, b.x, fmaf(-a.y, b.y, acc.x));
  acc.y = fmaf(a.x, b.y, fmaf(a.y, b.x, acc.y));
}
__device__ __forceinline__ void cfmac(float2& acc, float2 a, float2 b) {   // acc += a * conj(b)
  acc.x = fmaf(a.x, b.x, fmaf(a.y, b.y, acc.x));
  acc.y = fmaf(a.y, b.x, fmaf(-a.x, b.y, acc.y));
}

constexpr int TS = 128;   // threads per CTA along the mode index
constexpr int TU = 8;     // steps of the channel sum whose loads are in flight together

// NV neighbouring modes of one thread: one 16-byte access (NV = 2) where rows keep that alignment, else 8 bytes.
template <int NV>
struct Modes {
  float2 v[NV];
};
template <int NV>
__device__ __forceinline__ Modes<NV> ld_modes(const float2* p) {
  Modes<NV> m;
  if constexpr (NV == 2) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(p));
    m.v[0] = make_float2(q.x, q.y);
    m.v[1] = make_float2(q.z, q.w);
  } else {
    m.v[0] = __ldg(p);
  }
  return m;
}
template <int NV>
__device__ __forceinline__ Modes<NV> ld_modes_once(const float2* p) {      // streaming: weights pass through once
  Modes<NV> m;
  if constexpr (NV == 2) {
    const float4 q = __ldcs(reinterpret_cast<const float4*>(p));
    m.v[0] = make_float2(q.x, q.y);
    m.v[1] = make_float2(q.z, q.w);
  } else {
    m.v[0] = __ldcs(p);
  }
  return m;
}
template <int NV>
__device__ __forceinline__ void st_modes(float2* p, const Modes<NV>& m, bool stream) {
  if constexpr (NV == 2) {
    const float4 q = make_float4(m.v[0].x, m.v[0].y, m.v[1].x, m.v[1].y);
    if (stream) __stcs(reinterpret_cast<float4*>(p), q);
    else *reinterpret_cast<float4*>(p) = q;
  } else {
    if (stream) __stcs(p, m.v[0]);
    else *p = m.v[0];
  }
}

// The sum over one channel index of the weights, forward (over i) or input gradient (over o):
//   CONJ 0: out[b, o, s] = sum_i a[b, i, s] w[i, o, s]        P = O outputs, Q = I summed
//   CONJ 1: out[b, i, s] = sum_o a[b, o, s] conj(w[i, o, s])  P = I outputs, Q = O summed
// with w at (q * wq + p * wp) rows of S modes.  Bound by reading w once (8 bytes per complex product): one output per thread with
// the loads of TU steps in flight, and a pair of samples (NB = 2) shares one pass over w.  Four outputs per thread, which
// load the activations once for four, leave too few CTAs where there are few channels or modes, and their loads go to four
// distant rows.  us, one output / four / one thread per output and sample without loads in flight, input gradient (forward):
//   64 channels, 180 x 180 modes  173 / 185 / 177 (174 / 187 / 242)      two samples  199 / 225 / 342 (200 / 223 / 420)
//   16 x 64, 90 x 90               27 /  61 /  45  (21 /  25 /  26)      24, 24 x 24   12 /  26 /  21  (12 /  27 /  31)
// grid (ceil(S / (TS NV)), P, ceil(B / NB))
template <int NV, int NB, int CONJ>
__global__ void __launch_bounds__(TS) diag_sum_kernel(const float2* __restrict__ a, const float2* __restrict__ w,
                                                      float2* __restrict__ out, int B, int P, int Q, long long wp, long long wq,
                                                      long long S) {
  const long long s = (static_cast<long long>(blockIdx.x) * TS + threadIdx.x) * NV;
  const int p = blockIdx.y, b0 = blockIdx.z * NB;
  if (s >= S) return;
  const int nb = min(NB, B - b0);
  Modes<NV> acc[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b)
#pragma unroll
    for (int h = 0; h < NV; ++h) acc[b].v[h] = make_float2(0.f, 0.f);
  const float2* const ap = a + static_cast<long long>(b0) * Q * S + s;
  const float2* const wr = w + p * wp * S + s;
  auto step = [&](const Modes<NV> (&av)[NB], const Modes<NV>& wv) {
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
      for (int h = 0; h < NV; ++h) {
        if (CONJ) cfmac(acc[b].v[h], av[b].v[h], wv.v[h]);
        else cfma(acc[b].v[h], av[b].v[h], wv.v[h]);
      }
  };
  auto load = [&](int q, Modes<NV> (&av)[NB], Modes<NV>& wv) {
    wv = ld_modes_once<NV>(wr + q * wq * S);
#pragma unroll
    for (int b = 0; b < NB; ++b) av[b] = ld_modes<NV>(ap + (static_cast<long long>(b < nb ? b : 0) * Q + q) * S);
  };
  int q = 0;
  for (; q + TU <= Q; q += TU) {
    Modes<NV> av[TU][NB], wv[TU];
#pragma unroll
    for (int u = 0; u < TU; ++u) load(q + u, av[u], wv[u]);
#pragma unroll
    for (int u = 0; u < TU; ++u) step(av[u], wv[u]);
  }
  for (; q < Q; ++q) {
    Modes<NV> av[NB], wv;
    load(q, av, wv);
    step(av, wv);
  }
#pragma unroll
  for (int b = 0; b < NB; ++b)
    if (b < nb) st_modes<NV>(out + (static_cast<long long>(b0 + b) * P + p) * S + s, acc[b], false);
}

// dw[i, o, s] = sum_b conj(a[b, i, s]) dy[b, o, s]: bound by writing dw; a thread makes TI x TO weights from TI + TO loads (one
// weight from two loads before, with 8-byte stores: 538 -> 165 us for the 1.06 GB above, 6.4 TB/s).
// grid (ceil(S / (TS NV)), ceil(O / TO), ceil(I / TI))
constexpr int TI = 4, TO = 4;
template <int NV>
__global__ void __launch_bounds__(TS) diag_wgrad_kernel(const float2* __restrict__ a, const float2* __restrict__ dy,
                                                        float2* __restrict__ dw, int B, int I, int O, long long S) {
  const long long s = (static_cast<long long>(blockIdx.x) * TS + threadIdx.x) * NV;
  const int o0 = blockIdx.y * TO, i0 = blockIdx.z * TI;
  if (s >= S) return;
  const int no = min(TO, O - o0), ni = min(TI, I - i0);
  Modes<NV> acc[TI][TO];
#pragma unroll
  for (int i = 0; i < TI; ++i)
#pragma unroll
    for (int j = 0; j < TO; ++j)
#pragma unroll
      for (int h = 0; h < NV; ++h) acc[i][j].v[h] = make_float2(0.f, 0.f);
  for (int b = 0; b < B; ++b) {
    Modes<NV> av[TI], gv[TO];
#pragma unroll
    for (int i = 0; i < TI; ++i) av[i] = ld_modes<NV>(a + (static_cast<long long>(b) * I + i0 + (i < ni ? i : 0)) * S + s);
#pragma unroll
    for (int j = 0; j < TO; ++j) gv[j] = ld_modes<NV>(dy + (static_cast<long long>(b) * O + o0 + (j < no ? j : 0)) * S + s);
#pragma unroll
    for (int i = 0; i < TI; ++i)
#pragma unroll
      for (int j = 0; j < TO; ++j)
#pragma unroll
        for (int h = 0; h < NV; ++h) cfmac(acc[i][j].v[h], gv[j].v[h], av[i].v[h]);
  }
#pragma unroll
  for (int i = 0; i < TI; ++i)
#pragma unroll
    for (int j = 0; j < TO; ++j)
      if (i < ni && j < no) st_modes<NV>(dw + (static_cast<long long>(i0 + i) * O + o0 + j) * S + s, acc[i][j], true);
}

// separable: grid (ceil(S / TS), I, B); wdiv = 1 (weight per mode) or M (weight per degree, s' = s / M)
__global__ void __launch_bounds__(TS) sep_mul_kernel(const float2* __restrict__ a, const float2* __restrict__ w,
                                                     float2* __restrict__ out, int I, long long S, int wdiv, int conj_w) {
  const long long s = static_cast<long long>(blockIdx.x) * TS + threadIdx.x;
  const int i = blockIdx.y, b = blockIdx.z;
  if (s >= S) return;
  const long long ws = S / wdiv;
  const float2 wv = w[static_cast<long long>(i) * ws + s / wdiv];
  const float2 av = a[(static_cast<long long>(b) * I + i) * S + s];
  out[(static_cast<long long>(b) * I + i) * S + s] = conj_w ? cmulc(av, wv) : cmul(av, wv);
}

// dw[i, s'] = sum_b sum_{s in s'} conj(a[b, i, s]) dy[b, i, s]; grid (ceil(S' / TS), I); one thread per weight element
__global__ void __launch_bounds__(TS) sep_wgrad_kernel(const float2* __restrict__ a, const float2* __restrict__ dy,
                                                       float2* __restrict__ dw, int B, int I, long long S, int wdiv) {
  const long long ws = S / wdiv;
  const long long sp = static_cast<long long>(blockIdx.x) * TS + threadIdx.x;
  const int i = blockIdx.y;
  if (sp >= ws) return;
  float2 acc = make_float2(0.f, 0.f);
  for (int b = 0; b < B; ++b) {
    const long long base = (static_cast<long long>(b) * I + i) * S + sp * wdiv;
    for (int k = 0; k < wdiv; ++k) cfmac(acc, dy[base + k], a[base + k]);
  }
  dw[static_cast<long long>(i) * ws + sp] = acc;
}

inline unsigned cdiv(long long a, long long b) { return static_cast<unsigned>((a + b - 1) / b); }

}  // namespace

namespace {
// two modes per thread need rows of an even number of modes on 16-byte boundaries
bool pairs_ok(const void* a, const void* b, const void* c, long long S) {
  return (S & 1) == 0 &&
         ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15) == 0;
}

template <int CONJ>
cudaError_t diag_sum(const float* a, const float* w, float* out, int B, int P, int Q, long long wp, long long wq, long long S,
                     cudaStream_t st) {
  if (B <= 0 || P <= 0 || Q <= 0 || S <= 0) return cudaSuccess;
  const float2 *ap = reinterpret_cast<const float2*>(a), *wr = reinterpret_cast<const float2*>(w);
  float2* op = reinterpret_cast<float2*>(out);
  const int nb = B > 1 ? 2 : 1;
  const bool pairs = pairs_ok(a, w, out, S);
  const dim3 grid(cdiv(S, pairs ? 2 * TS : TS), P, cdiv(B, nb));
  if (pairs && nb == 2) diag_sum_kernel<2, 2, CONJ><<<grid, TS, 0, st>>>(ap, wr, op, B, P, Q, wp, wq, S);
  else if (pairs) diag_sum_kernel<2, 1, CONJ><<<grid, TS, 0, st>>>(ap, wr, op, B, P, Q, wp, wq, S);
  else if (nb == 2) diag_sum_kernel<1, 2, CONJ><<<grid, TS, 0, st>>>(ap, wr, op, B, P, Q, wp, wq, S);
  else diag_sum_kernel<1, 1, CONJ><<<grid, TS, 0, st>>>(ap, wr, op, B, P, Q, wp, wq, S);
  return cudaGetLastError();
}
}  // namespace

cudaError_t modes_diag_fwd(const float* a, const float* w, float* out, int B, int I, int O, long long S, cudaStream_t st) {
  return diag_sum<0>(a, w, out, B, O, I, 1, O, S, st);
}

cudaError_t modes_diag_dgrad(const float* dy, const float* w, float* da, int B, int I, int O, long long S, cudaStream_t st) {
  return diag_sum<1>(dy, w, da, B, I, O, O, 1, S, st);
}

cudaError_t modes_diag_wgrad(const float* a, const float* dy, float* dw, int B, int I, int O, long long S, cudaStream_t st) {
  if (I <= 0 || O <= 0 || S <= 0) return cudaSuccess;
  const float2 *ap = reinterpret_cast<const float2*>(a), *gp = reinterpret_cast<const float2*>(dy);
  float2* op = reinterpret_cast<float2*>(dw);
  const bool pairs = pairs_ok(a, dy, dw, S);
  const dim3 grid(cdiv(S, pairs ? 2 * TS : TS), cdiv(O, TO), cdiv(I, TI));
  if (pairs) diag_wgrad_kernel<2><<<grid, TS, 0, st>>>(ap, gp, op, B, I, O, S);
  else diag_wgrad_kernel<1><<<grid, TS, 0, st>>>(ap, gp, op, B, I, O, S);
  return cudaGetLastError();
}

cudaError_t modes_sep_mul(const float* a, const float* w, float* out, int B, int I, long long S, int wdiv, int conj_w, cudaStream_t st) {
  if (B <= 0 || I <= 0 || S <= 0) return cudaSuccess;
  sep_mul_kernel<<<dim3(cdiv(S, TS), I, B), TS, 0, st>>>(reinterpret_cast<const float2*>(a), reinterpret_cast<const float2*>(w),
                                                          reinterpret_cast<float2*>(out), I, S, wdiv, conj_w);
  return cudaGetLastError();
}

cudaError_t modes_sep_wgrad(const float* a, const float* dy, float* dw, int B, int I, long long S, int wdiv, cudaStream_t st) {
  if (I <= 0 || S <= 0) return cudaSuccess;
  sep_wgrad_kernel<<<dim3(cdiv(S / wdiv, TS), I), TS, 0, st>>>(reinterpret_cast<const float2*>(a), reinterpret_cast<const float2*>(dy),
                                                                reinterpret_cast<float2*>(dw), B, I, S, wdiv);
  return cudaGetLastError();
}

}  // namespace mk
