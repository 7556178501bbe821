// GELU and its derivative for the fused epilogues and the normalisation kernels.
//
//   default ("erf form")  : 0.5 x (1 + erf(x / sqrt 2)), the definition of torch.nn.GELU().  These epilogues have a
//                           budget of about a dozen instructions per output element (a 128x256 tile with K = 384 is
//                           done by the tensor cores in 3072 cycles), so erf is not evaluated with erff() (that
//                           doubled the time of the GELU GEMMs) but through the identity
//                           erf(x / sqrt 2) ~= tanh(x (c0 + c1 x^2 + c2 x^4)), a minimax fit of the argument whose
//                           normal-CDF error is below 1.9e-5 everywhere (|GELU error| < 5.5e-5), on the hardware
//                           tanh.approx instruction (relative error 2^-11 on the tanh value).  Both terms are far
//                           below the 2^-8 relative spacing of the bf16 activations the result is rounded to.
//   tanh form (opt-in)    : 0.5 x (1 + tanh(sqrt(2/pi) (x + 0.044715 x^3))), i.e. torch.nn.GELU(approximate="tanh"),
//                           which deviates from the erf form by up to 4.7e-4.
//
// The derivative is that of the function actually evaluated, so forward and backward are consistent.  Which form runs
// is a process-wide setting (mk::set_gelu_tanh) that every launcher reads and passes to its kernel.
#pragma once
#include <cuda_runtime.h>

namespace mk {

// 0: exact erf form, 1: tanh approximation
void set_gelu_tanh(int on);
int gelu_tanh();

__device__ __forceinline__ float gelu_tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Both forms are 0.5 x (1 + tanh(x q(x^2))) with q(u) = c0 + c1 u + c2 u^2; a launcher passes the coefficients of the
// selected form to its kernel, so the device code has no branch on the form.
struct GeluCoef {
  float c0, c1, c2;
};
inline GeluCoef gelu_coef(int tanh_form) {
  if (tanh_form) return GeluCoef{0.7978845608f, 0.0356774081f, 0.f};
  return GeluCoef{0.797717881f, 0.0367982429f, -3.15818913e-4f};
}

// x^2 is clamped at 36: beyond |x| = 6 the tanh is 1 to fp32 precision, and the fitted q (c2 < 0) must not be
// followed to where it turns negative (|x| > 11)
__device__ __forceinline__ float gelu_fwd(float x, const GeluCoef& c) {
  const float u = fminf(x * x, 36.f);
  const float q = fmaf(u, fmaf(u, c.c2, c.c1), c.c0);
  const float hx = 0.5f * x;
  return fmaf(hx, gelu_tanh_approx(x * q), hx);
}

__device__ __forceinline__ float gelu_bwd(float x, const GeluCoef& c) {
  const float u = fminf(x * x, 36.f);
  const float q = fmaf(u, fmaf(u, c.c2, c.c1), c.c0);
  const float dq = fmaf(u, fmaf(u, 5.f * c.c2, 3.f * c.c1), c.c0);   // d(x q(x^2))/dx
  const float t = gelu_tanh_approx(x * q);
  return fmaf(0.5f * x * fmaf(-t, t, 1.0f), dq, fmaf(0.5f, t, 0.5f));
}

// GELU and its derivative at the same point (shared polynomial and tanh): the forward epilogue that saves the
// derivative for the backward pass pays six more instructions than the plain forward.
__device__ __forceinline__ void gelu_fwd_bwd(float x, const GeluCoef& c, float& y, float& dy) {
  const float u = fminf(x * x, 36.f);
  const float q = fmaf(u, fmaf(u, c.c2, c.c1), c.c0);
  const float dq = fmaf(u, fmaf(u, 5.f * c.c2, 3.f * c.c1), c.c0);
  const float t = gelu_tanh_approx(x * q);
  const float hx = 0.5f * x;
  y = fmaf(hx, t, hx);
  dy = fmaf(hx * fmaf(-t, t, 1.0f), dq, fmaf(0.5f, t, 0.5f));
}

#ifdef __CUDACC__
// The same functions on two values at once (sm_100 packed fp32 arithmetic: one instruction, two roundings identical to the
// scalar ones).  The packed derivative carries the opposite sign through t^2 - 1 and -dq, which changes no rounding.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 f2_pack(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void f2_unpack(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 f2_fma(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f32x2 f2_mul(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 f2_add(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// eight fp32 values rounded to one 16-byte vector of bf16
__device__ __forceinline__ uint4 f2_bf16x8(const f32x2 (&f)[4]) {
  uint4 r;
  uint32_t* w = reinterpret_cast<uint32_t*>(&r);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float a, b;
    f2_unpack(f[j], a, b);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w[j]) : "f"(b), "f"(a));
  }
  return r;
}
// eight bf16 of one 16-byte vector as four pairs of fp32
__device__ __forceinline__ void f2_unpack8(const uint4& v, f32x2 (&f)[4]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) f[j] = f2_pack(__uint_as_float(w[j] << 16), __uint_as_float(w[j] & 0xffff0000u));
}
__device__ __forceinline__ f32x2 f2_clamp36(f32x2 u) {
  float a, b;
  f2_unpack(u, a, b);
  return f2_pack(fminf(a, 36.f), fminf(b, 36.f));
}
__device__ __forceinline__ f32x2 f2_tanh(f32x2 u) {
  float a, b;
  f2_unpack(u, a, b);
  return f2_pack(gelu_tanh_approx(a), gelu_tanh_approx(b));
}
// The coefficients as register pairs.  The packed instructions take neither immediates nor constant-bank operands; made by
// volatile moves once per thread, the pairs stay in registers instead of being rebuilt at every use.
struct GeluPairs {
  f32x2 c0, c1, c2, n0, n1, n2, half, neg1;
};
__device__ __forceinline__ f32x2 f2_keep(float a) {
  f32x2 r;
  asm volatile("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ GeluPairs gelu_pairs(const GeluCoef& c) {
  return GeluPairs{f2_keep(c.c0), f2_keep(c.c1), f2_keep(c.c2), f2_keep(-c.c0), f2_keep(-3.f * c.c1), f2_keep(-5.f * c.c2),
                   f2_keep(0.5f), f2_keep(-1.f)};
}
__device__ __forceinline__ f32x2 gelu_fwd2(f32x2 x, const GeluPairs& c) {
  const f32x2 u = f2_clamp36(f2_mul(x, x));
  const f32x2 q = f2_fma(u, f2_fma(u, c.c2, c.c1), c.c0);
  const f32x2 hx = f2_mul(x, c.half);
  return f2_fma(hx, f2_tanh(f2_mul(x, q)), hx);
}
// The derivative by itself, a + a (1 - t) x dq with a = (1 + t) / 2, one instruction less than beside the function: through
// -t = tanh(-x q), as the packed instructions have no negation
struct GeluBwdPairs {
  f32x2 m0, m1, m2, d0, d1, d2, half, nhalf;
};
__device__ __forceinline__ GeluBwdPairs gelu_bwd_pairs(const GeluCoef& c) {
  return GeluBwdPairs{f2_keep(-c.c0), f2_keep(-c.c1), f2_keep(-c.c2), f2_keep(c.c0), f2_keep(3.f * c.c1), f2_keep(5.f * c.c2), f2_keep(0.5f),
                      f2_keep(-0.5f)};
}
__device__ __forceinline__ f32x2 gelu_bwd2(f32x2 x, const GeluBwdPairs& c) {
  const f32x2 u = f2_clamp36(f2_mul(x, x));
  const f32x2 mq = f2_fma(u, f2_fma(u, c.m2, c.m1), c.m0);
  const f32x2 dq = f2_fma(u, f2_fma(u, c.d2, c.d1), c.d0);
  const f32x2 mt = f2_tanh(f2_mul(x, mq));
  const f32x2 a = f2_fma(mt, c.nhalf, c.half);
  return f2_fma(f2_mul(f2_fma(mt, a, a), x), dq, a);
}
__device__ __forceinline__ void gelu_fwd_bwd2(f32x2 x, const GeluPairs& c, f32x2& y, f32x2& dy) {
  const f32x2 u = f2_clamp36(f2_mul(x, x));
  const f32x2 q = f2_fma(u, f2_fma(u, c.c2, c.c1), c.c0);
  const f32x2 ndq = f2_fma(u, f2_fma(u, c.n2, c.n1), c.n0);
  const f32x2 t = f2_tanh(f2_mul(x, q));
  const f32x2 hx = f2_mul(x, c.half);
  const f32x2 s = f2_fma(t, t, c.neg1);
  y = f2_fma(hx, t, hx);
  dy = f2_fma(f2_mul(hx, s), ndq, f2_fma(t, c.half, c.half));
}

#endif  // __CUDACC__

// Activation codes of the GEMM epilogue.  Odd codes act on the value itself (then an optional residual is added); even
// codes multiply the value by the derivative of the matching activation, evaluated at the epilogue operand:
//   1 GELU(x)               2 x * GELU'(aux)          aux = saved pre-activation
//   3 max(x, 0)             4 x * [aux > 0]           aux = saved OUTPUT of the ReLU
//   5 softshrink(x, param)  6 x * [aux != 0]          aux = saved OUTPUT of the soft shrinkage
//                           8 x * aux                 aux = derivative saved by the forward pass
__device__ __forceinline__ float act_fwd(float x, int act, float param, const GeluCoef& gc) {
  if (act == 1) return gelu_fwd(x, gc);
  if (act == 3) return fmaxf(x, 0.f);
  if (act == 5) return x > param ? x - param : (x < -param ? x + param : 0.f);
  return x;
}
__device__ __forceinline__ float act_bwd(float aux, int act, const GeluCoef& gc) {
  if (act == 2) return gelu_bwd(aux, gc);
  if (act == 4) return aux > 0.f ? 1.f : 0.f;
  if (act == 6) return aux != 0.f ? 1.f : 0.f;
  if (act == 8) return aux;
  return 1.f;
}

}  // namespace mk
