// Memory-bound fused kernels for sm_100a: instance norm (+GELU), quadrature-weighted Lp norms, multi-tensor
// AdamW with bf16 shadow weights, spectral-weight re-layout.  Each kernel makes the minimum number of passes
// over HBM (vectorised 16-byte accesses) and keeps reductions in fp32.
#include "fused_ops.cuh"
#include "gelu.cuh"
#include "gemm_tcgen05.cuh"
#include "launch.cuh"
#include "norm_ring.h"
#include "tcgen05.cuh"
#include <cstring>
#include <type_traits>


#include <math.h>

namespace mk {

namespace {
int g_gelu_tanh = 0;
}
void set_gelu_tanh(int on) { g_gelu_tanh = on ? 1 : 0; }
int gelu_tanh() { return g_gelu_tanh; }

// number of SMs of the current device (cached per device index)
int sm_count() {
  static int cache[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cache[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cache[dev] = n;
  }
  return cache[dev];
}

namespace {

constexpr int NT = 512;

// act: 0 none, 1 GELU (exact erf form), 2 GELU (tanh form); the launchers map the caller's on/off flag to 1 or 2
// according to the process-wide setting
__device__ __forceinline__ GeluCoef coef_of(int act) {
  return act == 2 ? GeluCoef{0.7978845608f, 0.0356774081f, 0.f} : GeluCoef{0.797717881f, 0.0367982429f, -3.15818913e-4f};
}
__device__ __forceinline__ float gelu_f(float x, int act) { return gelu_fwd(x, coef_of(act)); }
__device__ __forceinline__ float dgelu_f(float x, int act) { return gelu_bwd(x, coef_of(act)); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// block-wide sum of two values; result valid in all threads
__device__ __forceinline__ void block_sum2(float& a, float& b) {
  __shared__ float sh[2][32];
  __shared__ float res[2];
  a = warp_sum(a);
  b = warp_sum(b);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) {
    sh[0][w] = a;
    sh[1][w] = b;
  }
  __syncthreads();
  if (w == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    float x = l < nw ? sh[0][l] : 0.f;
    float y = l < nw ? sh[1][l] : 0.f;
    x = warp_sum(x);
    y = warp_sum(y);
    if (l == 0) {
      res[0] = x;
      res[1] = y;
    }
  }
  __syncthreads();
  a = res[0];
  b = res[1];
}

__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 x = __bfloat1622float2(h[j]);
    f[2 * j] = x.x;
    f[2 * j + 1] = x.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 v;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
  for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(f[2 * j], f[2 * j + 1]);
  return v;
}

// ------------------------------------------------------------------------------------------ instance norm

// mode 0: full forward; mode 1: partial sums only (sums -> stats[plane] = (sum, sumsq)); mode 2: normalise with given stats
template <bool VEC>
__global__ void __launch_bounds__(NT) inorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y,
                                                       const float* __restrict__ w, const float* __restrict__ b,
                                                       float* __restrict__ stats, int C, long long hw, float eps, int act,
                                                       int mode) {
  const int plane = blockIdx.x;
  const int c = plane % C;
  const __nv_bfloat16* xp = x + static_cast<long long>(plane) * hw;
  float mean, rstd;
  if (mode != 2) {
    float s = 0.f, ss = 0.f;
    if (VEC) {
      const uint4* xv = reinterpret_cast<const uint4*>(xp);
      const long long nv = hw >> 3;
      for (long long i = threadIdx.x; i < nv; i += NT) {
        float f[8];
        unpack8(xv[i], f);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          s += f[j];
          ss += f[j] * f[j];
        }
      }
    } else {
      for (long long i = threadIdx.x; i < hw; i += NT) {
        const float f = __bfloat162float(xp[i]);
        s += f;
        ss += f * f;
      }
    }
    block_sum2(s, ss);
    if (mode == 1) {
      if (threadIdx.x == 0) {
        stats[2 * plane] = s;
        stats[2 * plane + 1] = ss;
      }
      return;
    }
    mean = s / static_cast<float>(hw);
    const float var = fmaxf(ss / static_cast<float>(hw) - mean * mean, 0.f);
    rstd = rsqrtf(var + eps);
    if (threadIdx.x == 0) {
      stats[2 * plane] = mean;
      stats[2 * plane + 1] = rstd;
    }
  } else {
    mean = stats[2 * plane];
    rstd = stats[2 * plane + 1];
  }
  const float ga = (w ? w[c] : 1.f) * rstd;
  const float be = (b ? b[c] : 0.f) - mean * ga;
  __nv_bfloat16* yp = y + static_cast<long long>(plane) * hw;
  if (VEC) {
    const uint4* xv = reinterpret_cast<const uint4*>(xp);
    uint4* yv = reinterpret_cast<uint4*>(yp);
    const long long nv = hw >> 3;
    for (long long i = threadIdx.x; i < nv; i += NT) {
      float f[8];
      unpack8(xv[i], f);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float v = f[j] * ga + be;
        f[j] = act ? gelu_f(v, act) : v;
      }
      yv[i] = pack8(f);
    }
  } else {
    for (long long i = threadIdx.x; i < hw; i += NT) {
      float v = __bfloat162float(xp[i]) * ga + be;
      yp[i] = __float2bfloat16(act ? gelu_f(v, act) : v);
    }
  }
}

// phase control: ext 0: both phases; 1: phase 1 only (write sums); 2: phase 2 only (read merged sums)
template <bool VEC>
__global__ void __launch_bounds__(NT) inorm_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy,
                                                       __nv_bfloat16* __restrict__ dx, const float* __restrict__ w,
                                                       const float* __restrict__ b, const float* __restrict__ stats,
                                                       float* __restrict__ dw, float* __restrict__ db, float* __restrict__ sums_io,
                                                       int C, long long hw, float inv_count, int act, int ext) {
  const int plane = blockIdx.x;
  const int c = plane % C;
  const float mean = stats[2 * plane], rstd = stats[2 * plane + 1];
  const float wc = w ? w[c] : 1.f, bc = b ? b[c] : 0.f;
  const __nv_bfloat16* xp = x + static_cast<long long>(plane) * hw;
  const __nv_bfloat16* gp = dy + static_cast<long long>(plane) * hw;
  float s1 = 0.f, s2 = 0.f;
  if (ext != 2) {
    if (VEC) {
      const uint4* xv = reinterpret_cast<const uint4*>(xp);
      const uint4* gv = reinterpret_cast<const uint4*>(gp);
      const long long nv = hw >> 3;
      for (long long i = threadIdx.x; i < nv; i += NT) {
        float f[8], g[8];
        unpack8(xv[i], f);
        unpack8(gv[i], g);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xh = (f[j] - mean) * rstd;
          float gg = g[j];
          if (act) gg *= dgelu_f(xh * wc + bc, act);
          s1 += gg;
          s2 += gg * xh;
        }
      }
    } else {
      for (long long i = threadIdx.x; i < hw; i += NT) {
        const float xh = (__bfloat162float(xp[i]) - mean) * rstd;
        float gg = __bfloat162float(gp[i]);
        if (act) gg *= dgelu_f(xh * wc + bc, act);
        s1 += gg;
        s2 += gg * xh;
      }
    }
    block_sum2(s1, s2);
    if (threadIdx.x == 0) {
      if (dw) atomicAdd(dw + c, s2);
      if (db) atomicAdd(db + c, s1);
      if (sums_io) {
        sums_io[2 * plane] = s1;
        sums_io[2 * plane + 1] = s2;
      }
    }
    if (ext == 1) return;
  } else {
    s1 = sums_io[2 * plane];
    s2 = sums_io[2 * plane + 1];
  }
  const float m1 = s1 * inv_count, m2 = s2 * inv_count;
  const float sc = rstd * wc;
  __nv_bfloat16* op = dx + static_cast<long long>(plane) * hw;
  if (VEC) {
    const uint4* xv = reinterpret_cast<const uint4*>(xp);
    const uint4* gv = reinterpret_cast<const uint4*>(gp);
    uint4* ov = reinterpret_cast<uint4*>(op);
    const long long nv = hw >> 3;
    for (long long i = threadIdx.x; i < nv; i += NT) {
      float f[8], g[8];
      unpack8(xv[i], f);
      unpack8(gv[i], g);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float xh = (f[j] - mean) * rstd;
        float gg = g[j];
        if (act) gg *= dgelu_f(xh * wc + bc, act);
        f[j] = sc * (gg - m1 - xh * m2);
      }
      ov[i] = pack8(f);
    }
  } else {
    for (long long i = threadIdx.x; i < hw; i += NT) {
      const float xh = (__bfloat162float(xp[i]) - mean) * rstd;
      float gg = __bfloat162float(gp[i]);
      if (act) gg *= dgelu_f(xh * wc + bc, act);
      op[i] = __float2bfloat16(sc * (gg - m1 - xh * m2));
    }
  }
}

// ------------------------------------------------------------------------------------------ instance norm, channels-last
// x: [B, T, C] with C contiguous (C % 8 == 0, C <= 1024).  Thread (v, r) = (tid % V, tid / V), V = C / CH, owns CH
// channels of every row it meets, so per-channel constants stay in registers.

template <int MODE>
using ClSums = std::conditional_t<MODE == 0, ClForwardSums, ClBackwardSums>;
template <int MODE>
using ClApply = std::conditional_t<MODE == 0, ClForwardApply, ClBackwardApply>;
template <int CH>
using ClWord = std::conditional_t<CH == 8, uint4, uint2>;      // the channels of a thread

// mode 0: sums of (x, x^2).  mode 1: sums of (g, g * xhat) with g = dy * act'(xhat * w + b) for the backward pass.
__device__ __forceinline__ unsigned int xch_ld_acquire(const unsigned int* ptr) {
  unsigned int v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(ptr) : "memory");
  return v;
}
// bounded wait (2 s) of one thread on the peers' flags; false + error word on expiry
__device__ bool xch_wait(const StatExchange& xc, int code) {
  const unsigned int need = *xc.wait_exp + static_cast<unsigned int>(xc.wait_off);
  for (int peer = 0; peer < xc.npeers; ++peer) {
    unsigned long long t0 = 0;
    for (unsigned int it = 0;; ++it) {
      if (static_cast<int>(xch_ld_acquire(xc.wait + peer) - need) >= 0) break;
      if ((it & 255u) == 255u) {
        const unsigned long long now = global_ns();
        if (t0 == 0) t0 = now;
        else if (now - t0 > 2000000000ull) {
          atomicExch(xc.err, code);
          return false;
        }
      }
    }
  }
  return true;
}
__device__ void xch_signal(const StatExchange& xc) {
  *xc.done_ctr = 0;
  if (*reinterpret_cast<volatile int*>(xc.err) != 0) return;   // nothing is published after an expired wait
  atomicAdd(xc.bump, 1u);
  __threadfence_system();
  for (int peer = 0; peer < xc.npeers; ++peer)
    if (xc.sig[peer]) atomicAdd_system(xc.sig[peer], 1u);
}

// The rows of one image travel through a ring in shared memory: the last warp of the CTA fetches stages of whole, consecutive rows (of one
// tensor, or of two in the backward pass) by bulk copies, the others work on them: thread (v, r) on column v of the rows r, r + R, ... of a
// stage, handed to `use(t, x, dy)` (V columns of ClWord, the channels of a thread).  The copies never wait for the arithmetic (GELU' of
// every element) and no registers hold rows on their way.  With the rows in registers, loaded four at a time, load and arithmetic took turns;
// copied by every thread for itself (cp.async), 721 x 1440 tokens took 5 % longer than that, and with the stages of a CTA following one
// another (here they are dealt out over the CTAs: all read one window of some MB that moves through the tensor) 8 %.
__device__ __forceinline__ bool cl_wait(uint32_t bar, uint32_t parity, int* err) {
  if (mbar_wait(bar, parity)) return true;
  if (err) atomicExch(err, 58);
  return false;
}
__device__ __forceinline__ void cl_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
template <typename P>
__device__ __forceinline__ void cl_init(uint4* smem) {      // (by all threads, once; a barrier of the CTA before cl_rows)
  if (threadIdx.x == 0) {
    const uint32_t bars = smem_u32(smem);
    for (int i = 0; i < P::DEPTH; ++i) {
      mbar_init(bars + 16 * i, 1u);
      mbar_init(bars + 16 * i + 8, blockDim.x / 32 - 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
}
template <typename P, bool BACK, typename Use>
__device__ __forceinline__ void cl_rows(uint4* smem, int offset, const __nv_bfloat16* x, const __nv_bfloat16* dy, int V, int r, int R, long long T,
                                        int* err, Use&& use) {
  using Word = ClWord<P::CH>;
  static_assert(P::DEPTH * 16 <= CL_BARRIERS, "two barriers a stage");
  const uint32_t bars = smem_u32(smem);
  const Word* const ring = reinterpret_cast<const Word*>(smem + offset / 16);
  const int rows = P::LAPS * R, half = rows * V;      // rows and words of one tensor in a stage
  const long long hop = static_cast<long long>(gridDim.x) * rows;
  const long long stages = (T + rows - 1) / rows;
  const int count = blockIdx.x < stages ? static_cast<int>((stages - 1 - blockIdx.x) / gridDim.x) + 1 : 0;
  long long t = static_cast<long long>(blockIdx.x + (BACK ? (count - 1LL) * gridDim.x : 0)) * rows;
  int s = 0;
  uint32_t ph = 0;
  auto next = [&]() {
    t += BACK ? -hop : hop;
    if (++s == P::DEPTH) {
      s = 0;
      ph ^= 1u;
    }
  };
  if (threadIdx.x / 32 == blockDim.x / 32 - 1) {
    if ((threadIdx.x & 31) == 0) {
      const uint32_t dst = bars + offset, row = V * sizeof(Word);
      for (int k = 0; k < count; ++k, next()) {
        if (!cl_wait(bars + 16 * s + 8, ph ^ 1u, err)) break;
        const uint32_t bytes = static_cast<uint32_t>(min(static_cast<long long>(rows), T - t)) * row;
        const uint32_t at = dst + s * P::TENSORS * rows * row;
        mbar_expect_tx(bars + 16 * s, P::TENSORS * bytes);
        cl_copy(at, reinterpret_cast<const char*>(x) + t * row, bytes, bars + 16 * s);
        if (P::TENSORS == 2) cl_copy(at + rows * row, reinterpret_cast<const char*>(dy) + t * row, bytes, bars + 16 * s);
      }
    }
    return;
  }
  for (int k = 0; k < count; ++k, next()) {
    if (!cl_wait(bars + 16 * s, ph, err)) break;
    const Word* at = ring + s * P::TENSORS * half + threadIdx.x;
    if (r < R) {
      if (t + rows <= T) {
#pragma unroll
        for (int u = 0; u < P::LAPS; ++u) use(t + u * R + r, at[u * R * V], at[u * R * V + (P::TENSORS == 1 ? 0 : half)]);
      } else {
#pragma unroll 1
        for (int i = r; i < T - t; i += R, at += R * V) use(t + i, at[0], at[P::TENSORS == 1 ? 0 : half]);
      }
    }
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(bars + 16 * s + 8);
  }
}
// bf16 channels of a thread as pairs of fp32
__device__ __forceinline__ void cl_unpack(const uint4& w, f32x2 (&f)[4]) { f2_unpack8(w, f); }
__device__ __forceinline__ void cl_unpack(const uint2& w, f32x2 (&f)[2]) {
  f[0] = f2_pack(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u));
  f[1] = f2_pack(__uint_as_float(w.y << 16), __uint_as_float(w.y & 0xffff0000u));
}

template <int MODE>
__global__ void __launch_bounds__(ClSums<MODE>::THREADS + 32, 1) inorm_cl_sums_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy,
                                                                   const float* __restrict__ w, const float* __restrict__ b,
                                                                   const float* __restrict__ stats, float* __restrict__ sums,
                                                                   float* __restrict__ dw, float* __restrict__ db, int C, long long T,
                                                                   int R, int act, int shifted, const StatExchange xc) {
  extern __shared__ __align__(16) uint4 cl_ring[];
  GeluBwdPairs gc;
  if constexpr (MODE == 1) gc = gelu_bwd_pairs(coef_of(act));
  using P = ClSums<MODE>;
  using Word = ClWord<P::CH>;
  constexpr int PAIRS = P::CH / 2;
  static_assert(cl_sums_fit<P>(), "the partial sums take the ring's place");
  const int V = C / P::CH;
  // (no less; from the parameter alone it is kept in uniform registers: 17.0 us instead of 16.3 at 240 x 480 x 384)
  R = min(R, (static_cast<int>(blockDim.x) - 32) / V);
  const int v = threadIdx.x % V, r = threadIdx.x / V;
  const int bidx = blockIdx.y;
  cl_init<P>(cl_ring);
  chain_begin(xc.npeers == 0, x, dy, w, b, stats);
  __syncthreads();
  constexpr int RING = cl_ring_offset(0, false);
  // partial sums of the rows of threads, in the ring's place: those of row r from C r on, sums before products
  f32x2* const part = reinterpret_cast<f32x2*>(cl_ring + RING / 16);
  f32x2 a0[PAIRS], a1[PAIRS];
  {
    // Pairs of channels in packed fp32 arithmetic: a packed instruction takes two cycles of a scheduler's fp32 pipe, three where it reads three
    // different register pairs, but one issue slot (GELU' with the polynomials by single instructions, whose coefficients need no
    // registers: sums 330 us instead of 305).  With L2 flushed, us, rows in registers -> through the ring: 721 x 1440 x 384 with GELU forward
    // 417 -> 388, backward 775 -> 656 (without GELU 421 -> 383, 660 -> 608); 240 x 480: 90 -> 66, 153 -> 108; 97 x 192: 48 -> 30, 70 -> 40.
    // Both passes of the first looped without a pause, under the power cap: 1210 -> 1088.
    // Backward: pre = x ka + kb with ka = w rstd, kb = b - mean ka is the value the forward pass activated, and
    // sum g xhat = rstd sum g (x - mean).
    f32x2 nmean[PAIRS], ka[PAIRS], kb[PAIRS];
#pragma unroll
    for (int j = 0; j < PAIRS; ++j) {
      a0[j] = a1[j] = f2_pack(0.f, 0.f);
      if (MODE == 1) {
        const int c = v * P::CH + 2 * j;
        const float4 st = *reinterpret_cast<const float4*>(stats + (static_cast<long long>(bidx) * C + c) * 2);
        const float a = (w ? w[c] : 1.f) * st.y, d = (w ? w[c + 1] : 1.f) * st.w;
        nmean[j] = f2_pack(-st.x, -st.z);
        ka[j] = f2_pack(a, d);
        kb[j] = f2_pack((b ? b[c] : 0.f) - st.x * a, (b ? b[c + 1] : 0.f) - st.z * d);
      }
    }
    const __nv_bfloat16* const xb = x + static_cast<long long>(bidx) * T * C;
    const __nv_bfloat16* const gb = MODE == 1 ? dy + static_cast<long long>(bidx) * T * C : nullptr;
    // Shifted sums: sum (x - s) and sum (x - s)^2 with s = the sample's first token, so that the one-pass variance
    // E[(x-s)^2] - E[x-s]^2 does not cancel when |mean| >> std.  (Only when the statistics are local to this device:
    // sums that are merged across ranks need one common shift and stay unshifted.)
    f32x2 nsft[PAIRS];
#pragma unroll
    for (int j = 0; j < PAIRS; ++j) nsft[j] = f2_pack(0.f, 0.f);
    if (MODE == 0 && shifted) {
      cl_unpack(reinterpret_cast<const Word*>(xb)[v], nsft);
#pragma unroll
      for (int j = 0; j < PAIRS; ++j) nsft[j] = f2_mul(nsft[j], f2_pack(-1.f, -1.f));
    }
    auto accum = [&](const Word& xr, const Word& gr) {
      f32x2 f[PAIRS];
      cl_unpack(xr, f);
      if constexpr (MODE == 0) {
#pragma unroll
        for (int j = 0; j < PAIRS; ++j) {
          const f32x2 d = f2_add(f[j], nsft[j]);
          a0[j] = f2_add(a0[j], d);
          a1[j] = f2_fma(d, d, a1[j]);
        }
      } else {
        f32x2 g[PAIRS];
        cl_unpack(gr, g);
#pragma unroll
        for (int j = 0; j < PAIRS; ++j) {
          f32x2 gg = g[j];
          if (act) gg = f2_mul(gg, gelu_bwd2(f2_fma(f[j], ka[j], kb[j]), gc));
          a0[j] = f2_add(a0[j], gg);
          a1[j] = f2_fma(gg, f2_add(f[j], nmean[j]), a1[j]);
        }
      }
    };
    cl_rows<P, false>(cl_ring, RING, xb, gb, V, r, R, T, xc.err, [&](long long, const Word& xr, const Word& gr) { accum(xr, gr); });
    if (MODE == 1) {
#pragma unroll
      for (int j = 0; j < PAIRS; ++j) {
        const int c = v * P::CH + 2 * j;
        const float4 st = *reinterpret_cast<const float4*>(stats + (static_cast<long long>(bidx) * C + c) * 2);
        a1[j] = f2_mul(a1[j], f2_pack(st.y, st.w));
      }
    }
  }
  // Added up without atomics: those on fp32 in shared memory are loops of compare and swap, and with R threads on each word the end of a CTA
  // took some 14 us.
  __syncthreads();
  const int words = C / 2;      // pairs of channels
  if (r < R) {
#pragma unroll
    for (int j = 0; j < PAIRS; ++j) {
      part[r * C + j * V + v] = a0[j];
      part[r * C + words + j * V + v] = a1[j];
    }
  }
  __syncthreads();
  // in two steps where many rows of threads meet: S parts of the rows, then these
  const int S = min(min(R, 32), static_cast<int>(blockDim.x) / words);
  if (S > 1) {
    const int g = threadIdx.x / words, at = threadIdx.x - g * words;
    f32x2 s = f2_pack(0.f, 0.f), q = s;
    if (g < S) {
      for (int k = g; k < R; k += S) {
        s = f2_add(s, part[k * C + at]);
        q = f2_add(q, part[k * C + words + at]);
      }
    }
    __syncthreads();
    if (g < S) {
      part[g * C + at] = s;
      part[g * C + words + at] = q;
    }
    __syncthreads();
  }
  const int left = S > 1 ? S : R;
  for (int i = threadIdx.x; i < words; i += blockDim.x) {
    const int j = i / V, vv = i - j * V;
    f32x2 s = f2_pack(0.f, 0.f), q = s;
    for (int k = 0; k < left; ++k) {
      s = f2_add(s, part[k * C + i]);
      q = f2_add(q, part[k * C + words + i]);
    }
    float s0, s1, q0, q1;
    f2_unpack(s, s0, s1);
    f2_unpack(q, q0, q1);
    const int c = vv * P::CH + 2 * j;
    // one 16-byte vector atomic per two channels (C is a multiple of 8, the buffer is 16-byte aligned)
    atomicAdd(reinterpret_cast<float4*>(sums + (static_cast<long long>(bidx) * C + c) * 2), make_float4(s0, q0, s1, q1));
    if (MODE == 1) {
      if (db) {
        atomicAdd(db + c, s0);
        atomicAdd(db + c + 1, s1);
      }
      if (dw) {
        atomicAdd(dw + c, q0);
        atomicAdd(dw + c + 1, q1);
      }
    }
  }
  if (xc.npeers > 0) {
    // the last CTA of the grid hands this rank's sums to every peer
    __shared__ int last_s;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      const unsigned int prev = atomicAdd(xc.done_ctr, 1u);
      int last = (prev == gridDim.x * gridDim.y - 1) ? 1 : 0;
      if (last && !xch_wait(xc, 56)) last = 2;     // peers still read the previous statistics: give up (error word set)
      last_s = last;
    }
    __syncthreads();
    if (last_s == 1) {
      __threadfence();
      const int n = static_cast<int>(gridDim.y) * 2 * C;
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const float val = __ldcg(sums + i);
        for (int q = 0; q < xc.ndst; ++q) xc.dst[q][i] = val;
      }
      __threadfence_system();
      __syncthreads();
      if (threadIdx.x == 0) xch_signal(xc);
    } else if (last_s == 2 && threadIdx.x == 0) {
      *xc.done_ctr = 0;
    }
  }
}

// mode 0: y = act(xhat * w + b), statistics derived from `sums` (and stored to `stats`).
// mode 1: dx = rstd * w * (g - s1/T - xhat * s2/T) with (s1, s2) in `sums`, (mean, rstd) in `stats`.
template <int MODE>
__global__ void __launch_bounds__(ClApply<MODE>::THREADS + 32, 1) inorm_cl_apply_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy,
                                                                    __nv_bfloat16* __restrict__ out, const float* __restrict__ w,
                                                                    const float* __restrict__ b, const float* __restrict__ sums,
                                                                    float* __restrict__ stats, int C, long long T, int R, float inv_count,
                                                                    float eps, int act, int shifted, const StatExchange xc) {
  using P = ClApply<MODE>;
  const int V = C >> 3;
  const int v = threadIdx.x % V, r = threadIdx.x / V;
  const int bidx = blockIdx.y;
  extern __shared__ __align__(16) uint4 cl_ring[];
  // [C][2] merged sums of this sample (exchange mode only), in front of the ring
  float* const sh_sum = reinterpret_cast<float*>(cl_ring + CL_BARRIERS / 16);
  const int ring = cl_ring_offset(C, xc.npeers > 0);
  cl_init<P>(cl_ring);
  chain_begin(xc.npeers == 0, x, dy, w, b, sums, stats);
  if (xc.npeers > 0) {
    // every peer's sums must have arrived in the local buffer
    __shared__ int ok_s;
    if (threadIdx.x == 0) ok_s = xch_wait(xc, 57) ? 1 : 0;
    __syncthreads();
    if (!ok_s) return;
    // merge the segments once per CTA (coalesced, L1 bypassed: the buffer is rewritten by peers between launches);
    // fixed order, so every rank computes bit-identical statistics
    for (int i = threadIdx.x; i < 2 * C; i += blockDim.x) {
      float acc = 0.f;
      for (int q = 0; q < xc.nsrc; ++q) acc += __ldcg(xc.src + q * xc.src_stride + static_cast<long long>(bidx) * 2 * C + i);
      sh_sum[i] = acc;
    }
    __syncthreads();
  }
  __syncthreads();
  std::conditional_t<MODE == 0, GeluPairs, GeluBwdPairs> gc;
  if constexpr (MODE == 0) gc = gelu_pairs(coef_of(act));
  else gc = gelu_bwd_pairs(coef_of(act));
  // per-channel constants, two channels each.  Forward: y = act(x ka + kb).  Backward: dx = ka (g + k1 + (x - mean) k2)
  f32x2 ka[4], kb[4], nmean[4], k1[4], k2[4];
  float sft[8];                                      // shift of the statistics pass (the sample's first token) or 0
#pragma unroll
  for (int j = 0; j < 8; ++j) sft[j] = 0.f;
  if (MODE == 0 && shifted) unpack8((reinterpret_cast<const uint4*>(x + static_cast<long long>(bidx) * T * C) + v)[0], sft);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float va[2], vb[2], vm[2], v1[2], v2[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c = v * 8 + 2 * j + h;
      const long long sc = (static_cast<long long>(bidx) * C + c) * 2;
      const float wc = w ? w[c] : 1.f, bc = b ? b[c] : 0.f;
      float s0, s1;
      if (xc.npeers > 0) {
        s0 = sh_sum[2 * c];
        s1 = sh_sum[2 * c + 1];
      } else {
        s0 = sums[sc];
        s1 = sums[sc + 1];
      }
      if (MODE == 0) {
        const float dm = s0 * inv_count;                 // mean of (x - shift)
        const float mean = sft[2 * j + h] + dm;
        const float var = fmaxf(s1 * inv_count - dm * dm, 0.f);
        const float rstd = rsqrtf(var + eps);
        va[h] = wc * rstd;
        vb[h] = bc - mean * va[h];
        if (stats && blockIdx.x == 0 && r == 0) {
          stats[sc] = mean;
          stats[sc + 1] = rstd;
        }
      } else {
        const float mean = stats[sc], rstd = stats[sc + 1];
        va[h] = wc * rstd;
        vb[h] = bc - mean * va[h];
        vm[h] = -mean;
        v1[h] = -(s0 * inv_count);
        v2[h] = -(s1 * inv_count) * rstd;
      }
    }
    ka[j] = f2_pack(va[0], va[1]);
    kb[j] = f2_pack(vb[0], vb[1]);
    if (MODE == 1) {
      nmean[j] = f2_pack(vm[0], vm[1]);
      k1[j] = f2_pack(v1[0], v1[1]);
      k2[j] = f2_pack(v2[0], v2[1]);
    }
  }
  const long long base = static_cast<long long>(bidx) * T * C;
  uint4* ov = reinterpret_cast<uint4*>(out + base) + v;
  auto transform = [&](const uint4& xr, const uint4& gr) -> uint4 {
    f32x2 f[4];
    f2_unpack8(xr, f);
    if constexpr (MODE == 0) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        f[j] = f2_fma(f[j], ka[j], kb[j]);
        if (act) f[j] = gelu_fwd2(f[j], gc);
      }
    } else {
      f32x2 g[4];
      f2_unpack8(gr, g);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        f32x2 gg = g[j];
        if (act) gg = f2_mul(gg, gelu_bwd2(f2_fma(f[j], ka[j], kb[j]), gc));
        f[j] = f2_mul(ka[j], f2_fma(f2_add(f[j], nmean[j]), k2[j], f2_add(gg, k1[j])));
      }
    }
    return f2_bf16x8(f);
  };
  // From the end: the last rows that the sums' pass has read are still in L2
  cl_rows<P, true>(cl_ring, ring, x + base, MODE == 1 ? dy + base : nullptr, V, r, R, T, xc.err,
                   [&](long long t, const uint4& xr, const uint4& gr) { ov[t * V] = transform(xr, gr); });
  if (xc.npeers > 0) {
    // the last CTA tells the peers that this rank is done with their sums
    __syncthreads();
    if (threadIdx.x == 0) {
      const unsigned int prev = atomicAdd(xc.done_ctr, 1u);
      if (prev == gridDim.x * gridDim.y - 1) xch_signal(xc);
    }
  }
}

// ------------------------------------------------------------------------------------------ column sums

// out[g, c] = sum_r x_g[r, c] for bf16 rows of C columns (a multiple of 8): the bias gradients.  Row r of group g sits at
// g * gstride + (r / inner) * ostride + (r % inner) * C elements (plain rows: inner = 0).  One read of x; thread (v, r)
// owns eight columns and every R-th row of its slab with eight 16-byte loads in flight, so the HBM latency is covered at
// two CTAs per SM.  Every sum is taken in one fixed order, inside a CTA and over the slabs, so a call repeats itself bit for bit:
// the CTAs leave their sums in `part` ([groups][slabs][C]) and a second launch adds the slabs (one slab: straight to out).
// 16200 tokens: 3072 columns 20 us, 768 columns 9.5 us; 1038240 tokens of 384 columns 122 us (6.6 TB/s); 2048 x 16: 3.6 us.  Atomics
// into a cleared buffer took 18, 11.7, 119 and 4.0 us, each time with other bits, 3.6e-7 off 64 bits where this is 1e-7 off.
constexpr int CS_THREADS = 256;
__global__ void __launch_bounds__(CS_THREADS) colsum_kernel(const uint4* __restrict__ x, float* __restrict__ part, long long rows,
                                                            int V, int vb, int slab, int inner, long long ostride_v,
                                                            long long gstride_v) {
  __shared__ __align__(16) float sh[CS_THREADS * 8];
  chain_begin(true, x);
  const int v0 = blockIdx.x * vb;
  const int nv = min(vb, V - v0);          // 16-byte columns of this CTA
  const int R = CS_THREADS / vb;
  const int v = threadIdx.x % vb, r = threadIdx.x / vb;
  const bool fold = vb < 32 && (vb & (vb - 1)) == 0;      // lanes with the same columns: shuffles, then one lane per warp
  if (r < R && v < nv) {
    float a[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = 0.f;
    const long long t0 = static_cast<long long>(blockIdx.y) * slab;
    const long long t1 = min(t0 + slab, rows);
    const uint4* xv = x + blockIdx.z * gstride_v + v0 + v;
    const bool plain = inner == 0;
    auto row = [&](long long t) -> const uint4* {
      if (plain) return xv + t * V;
      const unsigned hi = static_cast<unsigned>(t) / static_cast<unsigned>(inner);
      return xv + hi * ostride_v + (t - static_cast<long long>(hi) * inner) * V;
    };
    auto add = [&](const uint4& q) {
      float f[8];
      unpack8(q, f);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] += f[j];
    };
    long long t = t0 + r;
    for (; t + 7LL * R < t1; t += 8LL * R) {
      uint4 q[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) q[u] = __ldg(row(t + u * R));
#pragma unroll
      for (int u = 0; u < 8; ++u) add(q[u]);
    }
    for (; t < t1; t += R) add(__ldg(row(t)));
    if (fold) {
      for (int o = 16; o >= vb; o >>= 1) {
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] += __shfl_xor_sync(0xffffffffu, a[j], o);
      }
    }
    if (!fold || (threadIdx.x & 31) < vb) {
      // row `r` of sums, or the warp's: vb * 8 floats each
      float4* const q = reinterpret_cast<float4*>(sh + ((fold ? threadIdx.x >> 5 : r) * vb + v) * 8);
      q[0] = make_float4(a[0], a[1], a[2], a[3]);
      q[1] = make_float4(a[4], a[5], a[6], a[7]);
    }
  }
  __syncthreads();
  const int n = fold ? CS_THREADS / 32 : R;
  float* const dst = part + ((static_cast<long long>(blockIdx.z) * gridDim.y + blockIdx.y) * V + v0) * 8;
  for (int i = threadIdx.x; i < nv * 8; i += CS_THREADS) {
    float t = 0.f;
    for (int k = 0; k < n; ++k) t += sh[k * vb * 8 + i];
    dst[i] = t;
  }
}

// out[g, c] = sum over the slabs (some hundreds of them, 4096 at most); 32 columns by 32 slabs at a time per CTA.  grid (ceil(C / 32), groups)
__global__ void __launch_bounds__(1024) colsum_slabs_kernel(const RowSlabs first, const RowSlabs second) {
  __shared__ float sh[32][33];
  RowSlabs j = blockIdx.z == 0 ? first : second;
  chain_begin(true, j.part);
  const float* const part = j.part;
  float* const out = j.out;
  const int slabs = j.slabs, C = j.C;
  if (blockIdx.x * 32 >= C || static_cast<int>(blockIdx.y) >= j.groups) return;
  const int c = blockIdx.x * 32 + threadIdx.x;
  float a = 0.f;
  if (c < C) {
    const float* p = part + static_cast<long long>(blockIdx.y) * slabs * C + c;
#pragma unroll 8
    for (int k = threadIdx.y; k < slabs; k += 32) a += p[static_cast<long long>(k) * C];
  }
  sh[threadIdx.y][threadIdx.x] = a;
  __syncthreads();
  // warp w adds up column w
  a = sh[threadIdx.x][threadIdx.y];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  const int cw = blockIdx.x * 32 + threadIdx.y;
  if (threadIdx.x == 0 && cw < C) out[static_cast<long long>(blockIdx.y) * C + cw] = a;
}

// ------------------------------------------------------------------------------------------ Lp norms

constexpr int LP_CHUNK = 1 << 16;   // elements of one plane handled by one CTA

template <typename T>
__device__ __forceinline__ float ldf(const T* p, long long i);
template <>
__device__ __forceinline__ float ldf<float>(const float* p, long long i) { return p[i]; }
template <>
__device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16* p, long long i) { return __bfloat162float(p[i]); }


// 16-byte vector access for the loss kernels: VW elements of one latitude row per load (W is a multiple of VW there)
template <typename T>
struct LpVec;
template <>
struct LpVec<float> {
  static constexpr int VW = 4;
  static __device__ __forceinline__ void load(const float* p, long long i, float (&v)[4]) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p + i));
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  }
  static __device__ __forceinline__ void store(float* p, long long i, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p + i) = make_float4(v[0], v[1], v[2], v[3]);
  }
};
template <>
struct LpVec<__nv_bfloat16> {
  static constexpr int VW = 8;
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, long long i, float (&v)[8]) {
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(p + i));
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&a);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __bfloat1622float2(h[j]);
      v[2 * j] = f.x;
      v[2 * j + 1] = f.y;
    }
  }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, long long i, const float (&v)[8]) {
    uint4 a;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&a);
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
    *reinterpret_cast<uint4*>(p + i) = a;
  }
};

template <typename T, int P, bool VEC>
__global__ void __launch_bounds__(NT) lp_norms_kernel(const T* __restrict__ pred, const T* __restrict__ tgt,
                                                      const float* __restrict__ qlat, float* __restrict__ out,
                                                      float* __restrict__ partial, int* __restrict__ counters, int W,
                                                      long long hw, int chunks) {
  const int plane = blockIdx.y, chunk = blockIdx.x;
  const T* pp = pred + static_cast<long long>(plane) * hw;
  const T* tp = tgt + static_cast<long long>(plane) * hw;
  const long long beg = static_cast<long long>(chunk) * LP_CHUNK;
  long long end = beg + LP_CHUNK;
  if (end > hw) end = hw;
  float sd = 0.f, st = 0.f;
  if (VEC) {
    constexpr int VW = LpVec<T>::VW;
#pragma unroll 4
    for (long long i = beg + static_cast<long long>(threadIdx.x) * VW; i < end; i += static_cast<long long>(NT) * VW) {
      const float q = qlat[static_cast<unsigned>(i) / static_cast<unsigned>(W)];
      float p[VW], t[VW];
      LpVec<T>::load(pp, i, p);
      LpVec<T>::load(tp, i, t);
      float ad = 0.f, at = 0.f;
#pragma unroll
      for (int j = 0; j < VW; ++j) {
        const float d = p[j] - t[j];
        if (P == 2) {
          ad = fmaf(d, d, ad);
          at = fmaf(t[j], t[j], at);
        } else {
          ad += fabsf(d);
          at += fabsf(t[j]);
        }
      }
      sd = fmaf(q, ad, sd);
      st = fmaf(q, at, st);
    }
  } else {
    for (long long i = beg + threadIdx.x; i < end; i += NT) {
      const float q = qlat[i / W];
      const float p = ldf<T>(pp, i), t = ldf<T>(tp, i);
      const float d = p - t;
      if (P == 2) {
        sd += q * d * d;
        st += q * t * t;
      } else {
        sd += q * fabsf(d);
        st += q * fabsf(t);
      }
    }
  }
  block_sum2(sd, st);
  __shared__ int last;
  if (threadIdx.x == 0) {
    float* pr = partial + (static_cast<long long>(plane) * chunks + chunk) * 2;
    pr[0] = sd;
    pr[1] = st;
    __threadfence();
    const int done = atomicAdd(counters + plane, 1);
    last = (done == chunks - 1);
  }
  __syncthreads();
  if (last) {
    // fixed-order final sum -> deterministic result
    __threadfence();
    float a = 0.f, b = 0.f;
    const volatile float* pr = partial + static_cast<long long>(plane) * chunks * 2;
    for (int i = threadIdx.x; i < chunks; i += NT) {
      a += pr[2 * i];
      b += pr[2 * i + 1];
    }
    block_sum2(a, b);
    if (threadIdx.x == 0) {
      out[2 * plane] = a;
      out[2 * plane + 1] = b;
      counters[plane] = 0;
    }
  }
}

template <typename T>
__device__ __forceinline__ void stf(T* p, long long i, float v);
template <>
__device__ __forceinline__ void stf<float>(float* p, long long i, float v) { p[i] = v; }
template <>
__device__ __forceinline__ void stf<__nv_bfloat16>(__nv_bfloat16* p, long long i, float v) { p[i] = __float2bfloat16(v); }

template <typename T, int P, bool VEC>
__global__ void __launch_bounds__(NT) lp_bwd_kernel(const T* __restrict__ pred, const T* __restrict__ tgt,
                                                    const float* __restrict__ qlat, const float* __restrict__ coef,
                                                    T* __restrict__ grad, int W, long long hw) {
  const int plane = blockIdx.y;
  const float cf = coef[plane];
  const long long base = static_cast<long long>(plane) * hw;
  const long long beg = static_cast<long long>(blockIdx.x) * LP_CHUNK;
  long long end = beg + LP_CHUNK;
  if (end > hw) end = hw;
  if (VEC) {
    constexpr int VW = LpVec<T>::VW;
#pragma unroll 4
    for (long long i = beg + static_cast<long long>(threadIdx.x) * VW; i < end; i += static_cast<long long>(NT) * VW) {
      const float cq = cf * qlat[static_cast<unsigned>(i) / static_cast<unsigned>(W)];
      float p[VW], t[VW];
      LpVec<T>::load(pred, base + i, p);
      LpVec<T>::load(tgt, base + i, t);
#pragma unroll
      for (int j = 0; j < VW; ++j) {
        const float d = p[j] - t[j];
        const float g = (P == 2) ? 2.f * d : ((d > 0.f) ? 1.f : ((d < 0.f) ? -1.f : 0.f));
        p[j] = cq * g;
      }
      LpVec<T>::store(grad, base + i, p);
    }
  } else {
    for (long long i = beg + threadIdx.x; i < end; i += NT) {
      const float q = qlat[i / W];
      const float d = ldf<T>(pred, base + i) - ldf<T>(tgt, base + i);
      float g;
      if (P == 2) g = 2.f * d;
      else g = (d > 0.f) ? 1.f : ((d < 0.f) ? -1.f : 0.f);
      stf<T>(grad, base + i, cf * q * g);
    }
  }
}

// ------------------------------------------------------------------------------------------ AdamW

__global__ void __launch_bounds__(256) adamw_kernel(const AdamEntry* __restrict__ table, const int* __restrict__ chunk_tensor,
                                                    const long long* __restrict__ chunk_off, long long chunk,
                                                    const float* __restrict__ hyper, const int* __restrict__ err) {
  // A bounded wait that ran out earlier in this step (a lost peer in the gradient all-reduce, a handshake that timed
  // out) leaves gradients that are incomplete: the update is skipped, so that the replicas stay identical until the
  // host reads the error word and raises.
  if (err != nullptr && *reinterpret_cast<const volatile int*>(err) != 0) return;
  const AdamEntry e = table[chunk_tensor[blockIdx.x]];
  const long long off = chunk_off[blockIdx.x];
  long long n = e.n - off;
  if (n > chunk) n = chunk;
  const float lr = hyper[0], b1 = hyper[1], b2 = hyper[2], eps = hyper[3], wd = hyper[4] * e.wd_scale, step = hyper[5],
              gs = hyper[6];
  const bool decoupled = hyper[7] != 0.f;
  const float bc1 = 1.f - powf(b1, step), bc2 = 1.f - powf(b2, step);
  const float step_size = lr / bc1;
  const float inv_sqrt_bc2 = rsqrtf(bc2);
  float* p = e.p + off;
  const float* g = e.g + off;
  float* m = e.m + off;
  float* v = e.v + off;
  __nv_bfloat16* sh = e.shadow ? e.shadow + off : nullptr;
  // chunk and off are multiples of 4, so float4 access is aligned whenever the tensor base is
  const bool vec = ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(m) |
                     reinterpret_cast<uintptr_t>(v)) & 15) == 0;
  const long long n4 = vec ? (n >> 2) : 0;
  for (long long i = threadIdx.x; i < n4; i += blockDim.x) {
    float4 pp = reinterpret_cast<float4*>(p)[i];
    const float4 gg4 = reinterpret_cast<const float4*>(g)[i];
    float4 mm = reinterpret_cast<float4*>(m)[i];
    float4 vv = reinterpret_cast<float4*>(v)[i];
    float P[4] = {pp.x, pp.y, pp.z, pp.w}, G[4] = {gg4.x * gs, gg4.y * gs, gg4.z * gs, gg4.w * gs};
    float M[4] = {mm.x, mm.y, mm.z, mm.w}, V[4] = {vv.x, vv.y, vv.z, vv.w};
    float G2[4];
    if (e.pair_mode) {
      G2[0] = G2[1] = G[0] * G[0] + G[1] * G[1];
      G2[2] = G2[3] = G[2] * G[2] + G[3] * G[3];
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) G2[j] = G[j] * G[j];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float gj = G[j];
      if (decoupled) P[j] *= (1.f - lr * wd);
      else gj += wd * P[j];
      M[j] = b1 * M[j] + (1.f - b1) * gj;
      V[j] = b2 * V[j] + (1.f - b2) * (decoupled ? G2[j] : (e.pair_mode ? G2[j] : gj * gj));
      const float denom = sqrtf(V[j]) * inv_sqrt_bc2 + eps;
      P[j] -= step_size * M[j] / denom;
    }
    reinterpret_cast<float4*>(p)[i] = make_float4(P[0], P[1], P[2], P[3]);
    reinterpret_cast<float4*>(m)[i] = make_float4(M[0], M[1], M[2], M[3]);
    reinterpret_cast<float4*>(v)[i] = make_float4(V[0], V[1], V[2], V[3]);
    if (sh) {
      sh[4 * i] = __float2bfloat16(P[0]);
      sh[4 * i + 1] = __float2bfloat16(P[1]);
      sh[4 * i + 2] = __float2bfloat16(P[2]);
      sh[4 * i + 3] = __float2bfloat16(P[3]);
    }
  }
  for (long long i = (n4 << 2) + threadIdx.x; i < n; i += blockDim.x) {
    float gj = g[i] * gs;
    float g2 = gj * gj;
    if (e.pair_mode) {
      const float go = g[i ^ 1] * gs;   // partner of the (re, im) pair; off is even
      g2 += go * go;
    }
    float pj = p[i];
    if (decoupled) pj *= (1.f - lr * wd);
    else gj += wd * pj;
    const float mj = b1 * m[i] + (1.f - b1) * gj;
    const float vj = b2 * v[i] + (1.f - b2) * ((decoupled || e.pair_mode) ? g2 : gj * gj);
    pj -= step_size * mj / (sqrtf(vj) * inv_sqrt_bc2 + eps);
    p[i] = pj;
    m[i] = mj;
    v[i] = vj;
    if (sh) sh[i] = __float2bfloat16(pj);
  }
}

// ------------------------------------------------------------------------------------------ AFNO block weights

// Complex block weights [2][nb][in][out] (fp32, real and imaginary planes) -> the real form the block GEMMs read, bf16
// [nb][2 out][2 in] with rows (ri', o), columns (ri, i): [[wr^T, -wi^T], [wi^T, wr^T]]; biases [2][nb][out] -> [nb][2 out]
// fp32.  Both layers in one launch: the tensors are small, what counted was some twenty launches of transposes, negations
// and concatenations per pass.  grid (ceil(max in / 32), ceil(max out / 32), 2 nb), block 32 x 8
__global__ void __launch_bounds__(256) afno_pack_kernel(const AfnoLayer a, const AfnoLayer b, int nb) {
  __shared__ float re[32][33], im[32][33];
  AfnoLayer L = blockIdx.z < static_cast<unsigned>(nb) ? a : b;
  chain_begin(true, L.w, L.b);
  const int blk = blockIdx.z % nb, i0 = blockIdx.x * 32, o0 = blockIdx.y * 32;
  if (i0 >= L.nin || o0 >= L.nout) return;
  const long long plane = static_cast<long long>(nb) * L.nin * L.nout;
  const float* w = L.w + static_cast<long long>(blk) * L.nin * L.nout;
  for (int j = threadIdx.y; j < 32; j += 8) {
    const int i = i0 + j, o = o0 + threadIdx.x;
    const bool in = i < L.nin && o < L.nout;
    re[j][threadIdx.x] = in ? w[static_cast<long long>(i) * L.nout + o] : 0.f;
    im[j][threadIdx.x] = in ? w[plane + static_cast<long long>(i) * L.nout + o] : 0.f;
  }
  __syncthreads();
  __nv_bfloat16* const wx = L.wx + static_cast<long long>(blk) * 4 * L.nin * L.nout;
  for (int j = threadIdx.y; j < 32; j += 8) {
    const int o = o0 + j, i = i0 + threadIdx.x;
    if (o < L.nout && i < L.nin) {
      const float r = re[threadIdx.x][j], m = im[threadIdx.x][j];
      __nv_bfloat16* top = wx + static_cast<long long>(o) * 2 * L.nin + i;
      __nv_bfloat16* bot = top + static_cast<long long>(L.nout) * 2 * L.nin;
      top[0] = __float2bfloat16(r);
      top[L.nin] = __float2bfloat16(-m);
      bot[0] = __float2bfloat16(m);
      bot[L.nin] = __float2bfloat16(r);
    }
  }
  if (L.b && blockIdx.x == 0 && threadIdx.y < 2) {
    const int o = o0 + threadIdx.x;
    if (o < L.nout)
      L.bx[(static_cast<long long>(blk) * 2 + threadIdx.y) * L.nout + o] =
          L.b[(static_cast<long long>(threadIdx.y) * nb + blk) * L.nout + o];
  }
}

// The way back for the gradients: dwx fp32 [nb][2 out][2 in] -> dw [2][nb][in][out] with dwr = (d00 + d11)^T, dwi = (d10 - d01)^T,
// and dbx [nb][2 out] -> db [2][nb][out].  Same grid.
__global__ void __launch_bounds__(256) afno_fold_kernel(const AfnoGrad a, const AfnoGrad b, int nb) {
  __shared__ float re[32][33], im[32][33];
  AfnoGrad L = blockIdx.z < static_cast<unsigned>(nb) ? a : b;
  chain_begin(true, L.dwx, L.dbx);
  const int blk = blockIdx.z % nb, i0 = blockIdx.x * 32, o0 = blockIdx.y * 32;
  if (i0 >= L.nin || o0 >= L.nout) return;
  const float* const wx = L.dwx + static_cast<long long>(blk) * 4 * L.nin * L.nout;
  for (int j = threadIdx.y; j < 32; j += 8) {
    const int o = o0 + j, i = i0 + threadIdx.x;
    const bool in = o < L.nout && i < L.nin;
    const float* top = wx + static_cast<long long>(o) * 2 * L.nin + i;
    const float* bot = top + static_cast<long long>(L.nout) * 2 * L.nin;
    re[j][threadIdx.x] = in ? top[0] + bot[L.nin] : 0.f;
    im[j][threadIdx.x] = in ? bot[0] - top[L.nin] : 0.f;
  }
  __syncthreads();
  const long long plane = static_cast<long long>(nb) * L.nin * L.nout;
  float* w = L.dw + static_cast<long long>(blk) * L.nin * L.nout;
  for (int j = threadIdx.y; j < 32; j += 8) {
    const int i = i0 + j, o = o0 + threadIdx.x;
    if (i < L.nin && o < L.nout) {
      w[static_cast<long long>(i) * L.nout + o] = re[threadIdx.x][j];
      w[plane + static_cast<long long>(i) * L.nout + o] = im[threadIdx.x][j];
    }
  }
  if (L.db && blockIdx.x == 0 && threadIdx.y < 2) {
    const int o = o0 + threadIdx.x;
    if (o < L.nout)
      L.db[(static_cast<long long>(threadIdx.y) * nb + blk) * L.nout + o] =
          L.dbx[(static_cast<long long>(blk) * 2 + threadIdx.y) * L.nout + o];
  }
}

// ------------------------------------------------------------------------------------------ spectral weights

// grid: (Cin/32, Cout, ceil(L/32)); block 32x8
__global__ void spectral_expand_kernel(const float2* __restrict__ w, __nv_bfloat16* __restrict__ wx, int Cin, int Cout, int L,
                                       int planar) {
  __shared__ float2 tile[32][33];
  const int c0 = blockIdx.x * 32, o = blockIdx.y, l0 = blockIdx.z * 32;
  for (int j = threadIdx.y; j < 32; j += 8) {
    const int c = c0 + j, l = l0 + threadIdx.x;
    float2 v = make_float2(0.f, 0.f);
    if (c < Cin && l < L) v = w[(static_cast<long long>(c) * Cout + o) * L + l];
    tile[j][threadIdx.x] = v;
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += 8) {
    const int l = l0 + j, c = c0 + threadIdx.x;
    if (l < L && c < Cin) {
      const float2 v = tile[threadIdx.x][j];
      if (planar) {
        __nv_bfloat16* q = wx + (static_cast<long long>(l) * 2 * Cout + o) * Cin + c;
        q[0] = __float2bfloat16(v.x);
        q[static_cast<long long>(Cout) * Cin] = __float2bfloat16(v.y);
        continue;
      }
      // 2x2-block form: rows (ri', o), columns (ri, c):  [[Wr, -Wi], [Wi, Wr]]
      __nv_bfloat16* base = wx + static_cast<long long>(l) * 4 * Cout * Cin;
      const long long r0 = static_cast<long long>(o) * 2 * Cin, r1 = static_cast<long long>(Cout + o) * 2 * Cin;
      base[r0 + c] = __float2bfloat16(v.x);
      base[r0 + Cin + c] = __float2bfloat16(-v.y);
      base[r1 + c] = __float2bfloat16(v.y);
      base[r1 + Cin + c] = __float2bfloat16(v.x);
    }
  }
}

// The same re-layout with 16-byte accesses on both sides, for an even number of degrees and Cin a multiple of 8: a 64-channel
// by 32-degree tile, so that the writes are 128-byte segments (the kernel above: 64 bytes, one element per lane and
// store) and every thread has four 16-byte loads in flight.  384 x 384 x 240: 149 -> 95 us, 6.0 TB/s over reads and writes.
// grid: (ceil(Cin / 64), Cout, ceil(L / 32)); 256 threads
constexpr int SX_PITCH = 64 + 8;      // bf16 per tile row (16-byte aligned rows)
__global__ void __launch_bounds__(256) spectral_expand_vec_kernel(const float2* __restrict__ w, __nv_bfloat16* __restrict__ wx,
                                                                  int Cin, int Cout, int L, int planar) {
  __shared__ __align__(16) __nv_bfloat16 re[32 * SX_PITCH], im[32 * SX_PITCH];
  const int c0 = blockIdx.x * 64, o = blockIdx.y, l0 = blockIdx.z * 32;
  const int lp = (threadIdx.x & 15) * 2, cp = (threadIdx.x >> 4) * 2;     // two degrees, two channels (then + 32)
  float4 v[2][2];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int c = c0 + h * 32 + cp + k;
      v[h][k] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < Cin && l0 + lp < L)
        v[h][k] = __ldcs(reinterpret_cast<const float4*>(w + (static_cast<long long>(c) * Cout + o) * L + l0 + lp));
    }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int at = lp * SX_PITCH + h * 32 + cp;
    *reinterpret_cast<__nv_bfloat162*>(re + at) = __floats2bfloat162_rn(v[h][0].x, v[h][1].x);
    *reinterpret_cast<__nv_bfloat162*>(im + at) = __floats2bfloat162_rn(v[h][0].y, v[h][1].y);
    *reinterpret_cast<__nv_bfloat162*>(re + at + SX_PITCH) = __floats2bfloat162_rn(v[h][0].z, v[h][1].z);
    *reinterpret_cast<__nv_bfloat162*>(im + at + SX_PITCH) = __floats2bfloat162_rn(v[h][0].w, v[h][1].w);
  }
  __syncthreads();
  const int cv = (threadIdx.x & 7) * 8, l = threadIdx.x >> 3;            // eight channels of one degree
  if (l0 + l < L && c0 + cv < Cin) {
    const uint4 r = *reinterpret_cast<const uint4*>(re + l * SX_PITCH + cv);
    const uint4 i = *reinterpret_cast<const uint4*>(im + l * SX_PITCH + cv);
    if (planar) {
      __nv_bfloat16* q = wx + (static_cast<long long>(l0 + l) * 2 * Cout + o) * Cin + c0 + cv;
      *reinterpret_cast<uint4*>(q) = r;
      *reinterpret_cast<uint4*>(q + static_cast<long long>(Cout) * Cin) = i;
      return;
    }
    const uint4 n = make_uint4(i.x ^ 0x80008000u, i.y ^ 0x80008000u, i.z ^ 0x80008000u, i.w ^ 0x80008000u);
    __nv_bfloat16* base = wx + static_cast<long long>(l0 + l) * 4 * Cout * Cin + c0 + cv;
    const long long r0 = static_cast<long long>(o) * 2 * Cin, r1 = static_cast<long long>(Cout + o) * 2 * Cin;
    *reinterpret_cast<uint4*>(base + r0) = r;
    *reinterpret_cast<uint4*>(base + r0 + Cin) = n;
    *reinterpret_cast<uint4*>(base + r1) = i;
    *reinterpret_cast<uint4*>(base + r1 + Cin) = r;
  }
}

// two_block == 0: dwx is the full real 2x2-block gradient [L, 2Cout, 2Cin];  two_block == 1: dwx is [2][L][Cout][Cin]
// holding (dWr, dWi) already.  assign != 0 overwrites dw instead of accumulating into it.
__global__ void spectral_fold_kernel(const float* __restrict__ dwx, float2* __restrict__ dw, int Cin, int Cout, int L,
                                     int two_block, int assign) {
  __shared__ float2 tile[32][33];
  const int c0 = blockIdx.x * 32, o = blockIdx.y, l0 = blockIdx.z * 32;
  for (int j = threadIdx.y; j < 32; j += 8) {
    const int l = l0 + j, c = c0 + threadIdx.x;
    float2 v = make_float2(0.f, 0.f);
    if (l < L && c < Cin) {
      if (two_block) {
        const long long e = (static_cast<long long>(l) * Cout + o) * Cin + c;
        v.x = dwx[e];
        v.y = dwx[e + static_cast<long long>(L) * Cout * Cin];
      } else {
        const float* base = dwx + static_cast<long long>(l) * 4 * Cout * Cin;
        const long long r0 = static_cast<long long>(o) * 2 * Cin, r1 = static_cast<long long>(Cout + o) * 2 * Cin;
        v.x = base[r0 + c] + base[r1 + Cin + c];   // dWr
        v.y = base[r1 + c] - base[r0 + Cin + c];   // dWi
      }
    }
    tile[j][threadIdx.x] = v;
  }
  __syncthreads();
  for (int j = threadIdx.y; j < 32; j += 8) {
    const int c = c0 + j, l = l0 + threadIdx.x;
    if (c < Cin && l < L) {
      float2* d = dw + (static_cast<long long>(c) * Cout + o) * L + l;
      const float2 v = tile[threadIdx.x][j];
      if (assign) {
        *d = v;
      } else {
        float2 cur = *d;
        cur.x += v.x;
        cur.y += v.y;
        *d = cur;
      }
    }
  }
}

// dw = (dWr, dWi) with 16-byte accesses on both sides: [2][L][Cout][Cin] -> complex [Cin, Cout, L], even L, Cin a multiple
// of 4; a 64-channel by 32-degree tile, 256-byte segments in both directions.  384 x 384 x 240: 142 -> 99 us, 5.7 TB/s.
// grid: (ceil(Cin / 64), Cout, ceil(L / 32))
__global__ void __launch_bounds__(256) spectral_fold_vec_kernel(const float* __restrict__ dwx, float2* __restrict__ dw, int Cin,
                                                                int Cout, int L) {
  __shared__ float sh[2][64][33];
  const int c0 = blockIdx.x * 64, o = blockIdx.y, l0 = blockIdx.z * 32;
  const int cv = (threadIdx.x & 15) * 4, lr = threadIdx.x >> 4;          // four channels of degrees lr, lr + 16
  const long long plane = static_cast<long long>(L) * Cout * Cin;
  float4 v[2][2];
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int l = l0 + lr + h * 16;
      v[p][h] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (l < L && c0 + cv < Cin)
        v[p][h] = __ldcs(reinterpret_cast<const float4*>(dwx + p * plane + (static_cast<long long>(l) * Cout + o) * Cin + c0 + cv));
    }
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int l = lr + h * 16;
      sh[p][cv][l] = v[p][h].x;
      sh[p][cv + 1][l] = v[p][h].y;
      sh[p][cv + 2][l] = v[p][h].z;
      sh[p][cv + 3][l] = v[p][h].w;
    }
  __syncthreads();
  const int lp = (threadIdx.x & 15) * 2, cr = threadIdx.x >> 4;          // two degrees of channels cr, cr + 16, ...
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int c = cr + k * 16;
    if (c0 + c < Cin && l0 + lp < L)
      *reinterpret_cast<float4*>(dw + (static_cast<long long>(c0 + c) * Cout + o) * L + l0 + lp) =
          make_float4(sh[0][c][lp], sh[1][c][lp], sh[0][c][lp + 1], sh[1][c][lp + 1]);
  }
}

// rows of (re[C], im[C]) bf16 -> (im[C], -re[C]); C a multiple of 8 (16-byte vectors, sign flip on the bit pattern)
__global__ void swap_ri_kernel(const uint4* __restrict__ in, uint4* __restrict__ out, long long rows, int cv) {
  const long long total = rows * 2 * cv;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long row = i / (2 * cv);
    const int j = static_cast<int>(i - row * 2 * cv);
    if (j < cv) {
      out[i] = in[row * 2 * cv + cv + j];
    } else {
      uint4 v = in[row * 2 * cv + (j - cv)];
      v.x ^= 0x80008000u;
      v.y ^= 0x80008000u;
      v.z ^= 0x80008000u;
      v.w ^= 0x80008000u;
      out[i] = v;
    }
  }
}

// fp32 [rows, cols] -> bf16 [rows, pitch], the columns from cols on zero: the weight operands of one or two pointwise layers in one launch
// (a fill, a cast and a strided copy each before); one 16-byte vector per thread
__global__ void __launch_bounds__(256) cast_pad_kernel(CastPad a, CastPad b) {
  chain_begin(true, a.x, b.x);
  long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  const long long na = a.rows * (a.pitch / 8);
  const bool second = i >= na;
  if (second) i -= na;
  const CastPad& m = second ? b : a;
  const int pitch_v = m.pitch / 8;
  if (i >= m.rows * pitch_v) return;
  const long long r = i / pitch_v;
  const int c = static_cast<int>(i - r * pitch_v) * 8;
  const float* p = m.x + r * m.cols + c;
  float f[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) f[j] = c + j < m.cols ? p[j] : 0.f;
  reinterpret_cast<uint4*>(m.y)[i] = pack8(f);
}

__global__ void __launch_bounds__(256) clear_kernel(float* a, long long na, float* b, long long nb) {
  chain_begin(true);
  const long long va = na / 4, vb = nb / 4, step = static_cast<long long>(gridDim.x) * blockDim.x;
  const long long first = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  for (long long i = first; i < va + vb; i += step)
    reinterpret_cast<float4*>(i < va ? a : b)[i < va ? i : i - va] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (first < na - va * 4) a[va * 4 + first] = 0.f;
  if (first < nb - vb * 4) b[vb * 4 + first] = 0.f;
}

__global__ void cast_kernel(const float* __restrict__ x, __nv_bfloat16* __restrict__ y, long long n) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x)
    y[i] = __float2bfloat16(x[i]);
}

__device__ __forceinline__ uint64_t splitmix(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// counter-based N(0,1): two 64-bit hashes -> Box-Muller; deterministic in (seed, index)
__global__ void fill_normal_kernel(__nv_bfloat16* __restrict__ y, long long n, uint64_t seed) {
  const long long pairs = (n + 1) >> 1;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < pairs;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const uint64_t h = splitmix(seed ^ splitmix(static_cast<uint64_t>(i)));
    const float u1 = (static_cast<float>(h >> 40) + 0.5f) * (1.0f / 16777216.0f);
    const float u2 = (static_cast<float>((h >> 16) & 0xFFFFFF) + 0.5f) * (1.0f / 16777216.0f);
    const float r = sqrtf(-2.f * __logf(u1));
    float sn, cs;
    __sincosf(6.283185307179586f * u2, &sn, &cs);
    y[2 * i] = __float2bfloat16(r * cs);
    if (2 * i + 1 < n) y[2 * i + 1] = __float2bfloat16(r * sn);
  }
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

cudaError_t inorm_fwd(const __nv_bfloat16* x, __nv_bfloat16* y, const float* w, const float* b, float* stats, int planes,
                      int C, long long hw, float eps, int act, int ext_stats, cudaStream_t s) {
  if (act) act = gelu_tanh() ? 2 : 1;
  if (planes <= 0) return cudaSuccess;
  const bool vec = (hw % 8 == 0) && aligned16(x) && aligned16(y);
  const int mode = ext_stats ? 2 : 0;
  if (vec) inorm_fwd_kernel<true><<<planes, NT, 0, s>>>(x, y, w, b, stats, C, hw, eps, act, mode);
  else inorm_fwd_kernel<false><<<planes, NT, 0, s>>>(x, y, w, b, stats, C, hw, eps, act, mode);
  return cudaGetLastError();
}

cudaError_t inorm_partial_stats(const __nv_bfloat16* x, float* sums, int planes, long long hw, cudaStream_t s) {
  if (planes <= 0) return cudaSuccess;
  const bool vec = (hw % 8 == 0) && aligned16(x);
  if (vec) inorm_fwd_kernel<true><<<planes, NT, 0, s>>>(x, nullptr, nullptr, nullptr, sums, 1, hw, 0.f, 0, 1);
  else inorm_fwd_kernel<false><<<planes, NT, 0, s>>>(x, nullptr, nullptr, nullptr, sums, 1, hw, 0.f, 0, 1);
  return cudaGetLastError();
}

cudaError_t inorm_bwd(const __nv_bfloat16* x, const __nv_bfloat16* dy, __nv_bfloat16* dx, const float* w, const float* b,
                      const float* stats, float* dw, float* db, float* sums_io, int planes, int C, long long hw,
                      double count, int act, int ext_sums, cudaStream_t s) {
  if (act) act = gelu_tanh() ? 2 : 1;
  if (planes <= 0) return cudaSuccess;
  const bool vec = (hw % 8 == 0) && aligned16(x) && aligned16(dy) && (dx == nullptr || aligned16(dx));
  const float inv = static_cast<float>(1.0 / count);
  if (vec) inorm_bwd_kernel<true><<<planes, NT, 0, s>>>(x, dy, dx, w, b, stats, dw, db, sums_io, C, hw, inv, act, ext_sums);
  else inorm_bwd_kernel<false><<<planes, NT, 0, s>>>(x, dy, dx, w, b, stats, dw, db, sums_io, C, hw, inv, act, ext_sums);
  return cudaGetLastError();
}

static inline bool cl_ok(int C) { return C % 8 == 0 && C >= 8 && C <= CL_CHANNELS; }
namespace {
template <typename P, typename Kernel>
cudaError_t cl_allow(Kernel* kernel) {
  static std::atomic<uint64_t> devices;      // (each of the kernels has parameters of its own)
  return allow_shared_memory(devices, reinterpret_cast<const void*>(kernel), cl_most_bytes<P>());
}
}  // namespace

cudaError_t inorm_cl_sums(const __nv_bfloat16* x, const __nv_bfloat16* dy, const float* w, const float* b, const float* stats,
                          float* sums, float* dw, float* db, int B, int C, long long T, int act, int mode, int* err, cudaStream_t s,
                          const StatExchange* xch) {
  if (act) act = gelu_tanh() ? 2 : 1;
  // mode: bit 0 = backward pass, bit 1 = forward statistics shifted by the first token (local statistics only)
  const int shifted = ((mode >> 1) & 1) && (!xch || xch->npeers == 0);
  mode &= 1;
  if (!cl_ok(C) || !aligned16(x) || !aligned16(dy)) return cudaErrorInvalidValue;      // (16-byte loads)
  StatExchange xc;
  memset(&xc, 0, sizeof(xc));
  xc.err = err;
  if (xch) xc = *xch;
  auto launch = [&](auto* kernel, auto params) {
    using P = decltype(params);
    const cudaError_t allowed = cl_allow<P>(kernel);
    if (allowed != cudaSuccess) return allowed;
    const ClGeometry g = cl_geometry<P>(C, T, B, sm_count(), false, xc.npeers == 0);
    return launch_chained(kernel, dim3(g.ctas, B), dim3(g.threads), g.bytes, s, 1, xc.npeers == 0, x, dy, w, b, stats, sums, dw, db, C, T, g.rows, act,
                          shifted, xc);
  };
  return mode == 0 ? launch(inorm_cl_sums_kernel<0>, ClSums<0>()) : launch(inorm_cl_sums_kernel<1>, ClSums<1>());
}

cudaError_t inorm_cl_apply(const __nv_bfloat16* x, const __nv_bfloat16* dy, __nv_bfloat16* out, const float* w, const float* b,
                           const float* sums, float* stats, int B, int C, long long T, double count, float eps, int act, int mode, int* err,
                           cudaStream_t s, const StatExchange* xch) {
  if (act) act = gelu_tanh() ? 2 : 1;
  // mode: bit 0 = backward pass, bit 1 = forward statistics shifted by the first token (local statistics only)
  const int shifted = ((mode >> 1) & 1) && (!xch || xch->npeers == 0);
  mode &= 1;
  if (!cl_ok(C) || !aligned16(x) || !aligned16(dy) || !aligned16(out)) return cudaErrorInvalidValue;
  StatExchange xc;
  memset(&xc, 0, sizeof(xc));
  xc.err = err;
  if (xch) xc = *xch;
  const float inv = static_cast<float>(1.0 / count);
  auto launch = [&](auto* kernel, auto params) {
    using P = decltype(params);
    const cudaError_t allowed = cl_allow<P>(kernel);
    if (allowed != cudaSuccess) return allowed;
    const ClGeometry g = cl_geometry<P>(C, T, B, sm_count(), xc.npeers > 0, xc.npeers == 0);
    return launch_chained(kernel, dim3(g.ctas, B), dim3(g.threads), g.bytes, s, 1, xc.npeers == 0, x, dy, out, w, b, sums, stats, C, T, g.rows, inv, eps,
                          act, shifted, xc);
  };
  return mode == 0 ? launch(inorm_cl_apply_kernel<0>, ClApply<0>()) : launch(inorm_cl_apply_kernel<1>, ClApply<1>());
}

namespace {
struct ColsumPlan {
  int V, parts, vb;         // 16-byte columns, CTAs along them, columns of one CTA
  long long slab, slabs;    // rows of one CTA, CTAs along the rows
};
ColsumPlan colsum_plan(long long rows, int C, int groups) {
  ColsumPlan p;
  p.V = C / 8;
  p.parts = (p.V + CS_THREADS - 1) / CS_THREADS;
  p.vb = (p.V + p.parts - 1) / p.parts;
  const int R = CS_THREADS / p.vb;
  // about four CTAs per SM, each with at least one full step of eight rows per thread
  p.slab = (rows * p.parts * groups + 4LL * sm_count() - 1) / (4LL * sm_count());
  if (p.slab < 8LL * R) p.slab = 8LL * R;
  p.slabs = (rows + p.slab - 1) / p.slab;
  return p;
}
}  // namespace

long long colsum_scratch(long long rows, int C, int groups) {
  if (rows <= 0 || C <= 0 || (C & 7) || groups <= 0) return 0;
  const ColsumPlan p = colsum_plan(rows, C, groups);
  return p.slabs > 1 ? p.slabs * groups * C : 0;
}

cudaError_t colsum(const __nv_bfloat16* x, float* out, float* scratch, long long rows, int C, cudaStream_t s, int groups,
                   long long gstride, int inner, long long ostride) {
  if (C <= 0 || groups <= 0) return cudaSuccess;
  if (rows <= 0) return cudaMemsetAsync(out, 0, sizeof(float) * static_cast<size_t>(C) * groups, s);
  if ((C & 7) || (gstride & 7) || (ostride & 7) || groups > 65535 || (inner > 0 && rows >= (1ll << 31)) || !aligned16(x) ||
      !aligned16(out) || (scratch == nullptr && colsum_scratch(rows, C, groups) > 0))
    return cudaErrorInvalidValue;
  const ColsumPlan p = colsum_plan(rows, C, groups);
  float* const part = p.slabs > 1 ? scratch : out;
  // Begun early its CTAs, four to an SM where eight have room, crowd on the SMs that are free.  Behind a product of 24 tiles, us, chained / in the
  // ordinary way: 1038240 x 384 160 / 127, 115200 x 768 42 / 35, 16200 x 3072 26 / 23, 4096 x 384 5.7 / 5.8, 2048 x 16 3.6 / 3.2.
  const cudaError_t e = launch_chained(colsum_kernel, dim3(p.parts, static_cast<unsigned>(p.slabs), groups), dim3(CS_THREADS), 0, s, 1, false,
                                       reinterpret_cast<const uint4*>(x), part, rows, p.V, p.vb, static_cast<int>(p.slab), inner, ostride / 8,
                                       gstride / 8);
  if (e == cudaSuccess && p.slabs > 1) return colsum_add_slabs(RowSlabs{part, out, static_cast<int>(p.slabs), C, groups}, s);
  return e;
}

cudaError_t colsum_add_slabs(const RowSlabs& a, const RowSlabs& b, cudaStream_t s) {
  const dim3 grid((std::max(a.C, b.C) + 31) / 32, std::max(a.groups, b.groups), b.C > 0 ? 2 : 1);
  // Two CTAs and more, begun early, share one SM.  Behind the gradient of weights with row sums, a pass in us, in the ordinary way / chained: 104 x 8 over 12
  // samples of 2080 tokens 15.4 / 17.9, 88 x 16 over 65872 15.0 / 16.8, 64 x 96 over 55328 14.9 / 15.7; one CTA: 32 x 32 over 17472 12.1 / 11.5.
  return launch_chained(colsum_slabs_kernel, grid, dim3(32, 32), 0, s, 1, grid.x * grid.y * grid.z == 1, a, b);
}
cudaError_t colsum_add_slabs(const RowSlabs& a, cudaStream_t s) { return colsum_add_slabs(a, RowSlabs(), s); }

template <typename L>
static dim3 afno_grid(const L& a, const L& b, int nb) {
  const int in = a.nin > b.nin ? a.nin : b.nin, out = a.nout > b.nout ? a.nout : b.nout;
  return dim3((in + 31) / 32, (out + 31) / 32, 2 * nb);
}

cudaError_t afno_pack(const AfnoLayer& a, const AfnoLayer& b, int nb, cudaStream_t s) {
  if (nb <= 0) return cudaSuccess;
  return launch_chained(afno_pack_kernel, afno_grid(a, b, nb), dim3(32, 8), 0, s, 1, true, a, b, nb);
}

cudaError_t afno_fold(const AfnoGrad& a, const AfnoGrad& b, int nb, cudaStream_t s) {
  if (nb <= 0) return cudaSuccess;
  return launch_chained(afno_fold_kernel, afno_grid(a, b, nb), dim3(32, 8), 0, s, 1, true, a, b, nb);
}

// The 16-byte path of the loss kernels needs every row to hold a whole number of vectors, 16-byte aligned planes and
// element indices that fit 32 bits (the row index is a 32-bit division there).
static bool lp_vec_ok(const void* a, const void* b, const void* c, int is_f32, int W, long long hw) {
  const int vw = is_f32 ? 4 : 8;
  const uintptr_t bits = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c);
  return (W % vw) == 0 && (bits & 15) == 0 && hw < (1ll << 31);
}

int lp_norms_chunks(long long hw) { return static_cast<int>((hw + LP_CHUNK - 1) / LP_CHUNK); }

cudaError_t lp_norms(const void* pred, const void* tgt, int is_f32, const float* qlat, float* out, float* scratch,
                     int planes, int H, int W, int P, cudaStream_t s) {
  if (planes <= 0) return cudaSuccess;
  const long long hw = static_cast<long long>(H) * W;
  const int chunks = lp_norms_chunks(hw);
  float* partial = scratch;
  int* counters = reinterpret_cast<int*>(scratch + static_cast<long long>(planes) * chunks * 2);
  // The counters' position depends on (planes, chunks): a scratch buffer that served another shape holds partial sums
  // there.  They are cleared on the stream before every launch (a memset node under graph capture).
  cudaError_t me = cudaMemsetAsync(counters, 0, sizeof(int) * static_cast<size_t>(planes), s);
  if (me != cudaSuccess) return me;
  dim3 grid(chunks, planes);
  const bool vec = lp_vec_ok(pred, tgt, nullptr, is_f32, W, hw);
#define MK_LP_NORMS(T, PP, V) \
  lp_norms_kernel<T, PP, V><<<grid, NT, 0, s>>>((const T*)pred, (const T*)tgt, qlat, out, partial, counters, W, hw, chunks)
#define MK_LP_NORMS_T(T)                        \
  do {                                          \
    if (P == 2) {                               \
      if (vec) MK_LP_NORMS(T, 2, true);         \
      else MK_LP_NORMS(T, 2, false);            \
    } else {                                    \
      if (vec) MK_LP_NORMS(T, 1, true);         \
      else MK_LP_NORMS(T, 1, false);            \
    }                                           \
  } while (0)
  if (is_f32) MK_LP_NORMS_T(float);
  else MK_LP_NORMS_T(__nv_bfloat16);
#undef MK_LP_NORMS_T
#undef MK_LP_NORMS
  return cudaGetLastError();
}

cudaError_t lp_norms_bwd(const void* pred, const void* tgt, int is_f32, const float* qlat, const float* coef, void* grad,
                         int planes, int H, int W, int P, cudaStream_t s) {
  if (planes <= 0) return cudaSuccess;
  const long long hw = static_cast<long long>(H) * W;
  dim3 grid(lp_norms_chunks(hw), planes);
  const bool vec = lp_vec_ok(pred, tgt, grad, is_f32, W, hw);
#define MK_LP_BWD(T, PP, V) \
  lp_bwd_kernel<T, PP, V><<<grid, NT, 0, s>>>((const T*)pred, (const T*)tgt, qlat, coef, (T*)grad, W, hw)
#define MK_LP_BWD_T(T)                        \
  do {                                        \
    if (P == 2) {                             \
      if (vec) MK_LP_BWD(T, 2, true);         \
      else MK_LP_BWD(T, 2, false);            \
    } else {                                  \
      if (vec) MK_LP_BWD(T, 1, true);         \
      else MK_LP_BWD(T, 1, false);            \
    }                                         \
  } while (0)
  if (is_f32) MK_LP_BWD_T(float);
  else MK_LP_BWD_T(__nv_bfloat16);
#undef MK_LP_BWD_T
#undef MK_LP_BWD
  return cudaGetLastError();
}

cudaError_t adamw_step(const AdamEntry* table, const int* chunk_tensor, const long long* chunk_off, int nchunks,
                       long long chunk, const float* hyper, const int* err, cudaStream_t s) {
  if (nchunks <= 0) return cudaSuccess;
  adamw_kernel<<<nchunks, 256, 0, s>>>(table, chunk_tensor, chunk_off, chunk, hyper, err);
  return cudaGetLastError();
}

cudaError_t spectral_expand(const float* w, __nv_bfloat16* wx, int Cin, int Cout, int L, cudaStream_t s, int planar) {
  if ((L & 1) == 0 && (Cin & 7) == 0 && aligned16(w) && aligned16(wx)) {
    spectral_expand_vec_kernel<<<dim3((Cin + 63) / 64, Cout, (L + 31) / 32), 256, 0, s>>>(reinterpret_cast<const float2*>(w), wx,
                                                                                          Cin, Cout, L, planar);
    return cudaGetLastError();
  }
  dim3 grid((Cin + 31) / 32, Cout, (L + 31) / 32), block(32, 8);
  spectral_expand_kernel<<<grid, block, 0, s>>>(reinterpret_cast<const float2*>(w), wx, Cin, Cout, L, planar);
  return cudaGetLastError();
}

cudaError_t spectral_fold(const float* dwx, float* dw, int Cin, int Cout, int L, cudaStream_t s, int two_block, int assign) {
  if (two_block && assign && (L & 1) == 0 && (Cin & 3) == 0 && aligned16(dwx) && aligned16(dw)) {
    spectral_fold_vec_kernel<<<dim3((Cin + 63) / 64, Cout, (L + 31) / 32), 256, 0, s>>>(dwx, reinterpret_cast<float2*>(dw), Cin,
                                                                                        Cout, L);
    return cudaGetLastError();
  }
  dim3 grid((Cin + 31) / 32, Cout, (L + 31) / 32), block(32, 8);
  spectral_fold_kernel<<<grid, block, 0, s>>>(dwx, reinterpret_cast<float2*>(dw), Cin, Cout, L, two_block, assign);
  return cudaGetLastError();
}

cudaError_t swap_ri_bf16(const __nv_bfloat16* in, __nv_bfloat16* out, long long rows, int C, cudaStream_t s) {
  if (rows <= 0) return cudaSuccess;
  if (C <= 0 || (C & 7) || (reinterpret_cast<uintptr_t>(in) & 15) || (reinterpret_cast<uintptr_t>(out) & 15))
    return cudaErrorInvalidValue;
  const long long total = rows * 2 * (C / 8);
  long long blocks = (total + 255) / 256;
  if (blocks > sm_count() * 8) blocks = sm_count() * 8;
  swap_ri_kernel<<<static_cast<unsigned>(blocks), 256, 0, s>>>(reinterpret_cast<const uint4*>(in), reinterpret_cast<uint4*>(out),
                                                               rows, C / 8);
  return cudaGetLastError();
}

cudaError_t cast_f32_bf16(const float* x, __nv_bfloat16* y, long long n, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  long long blocks = (n + 255) / 256;
  if (blocks > sm_count() * 16) blocks = sm_count() * 16;
  cast_kernel<<<static_cast<unsigned>(blocks), 256, 0, s>>>(x, y, n);
  return cudaGetLastError();
}

cudaError_t cast_pad_bf16(const CastPad& a, const CastPad& b, cudaStream_t s) {
  long long total = 0;
  for (const CastPad* m : {&a, &b}) {
    if (m->rows <= 0 || m->cols <= 0) continue;
    if ((m->pitch & 7) || m->pitch < m->cols || !aligned16(m->y)) return cudaErrorInvalidValue;
    total += m->rows * (m->pitch / 8);
  }
  if (total == 0) return cudaSuccess;
  if ((total + 255) / 256 > 0x7fffffffll) return cudaErrorInvalidValue;
  const CastPad none = {nullptr, nullptr, 0, 0, 8};
  return launch_chained(cast_pad_kernel, dim3(static_cast<unsigned>((total + 255) / 256)), dim3(256), 0, s, 1, true, a.rows > 0 && a.cols > 0 ? a : none,
                        b.rows > 0 && b.cols > 0 ? b : none);
}
cudaError_t cast_pad_bf16(const CastPad& a, cudaStream_t s) { return cast_pad_bf16(a, CastPad{nullptr, nullptr, 0, 0, 8}, s); }

cudaError_t clear_f32(float* a, long long na, float* b, long long nb, cudaStream_t s) {
  if (!a) na = 0;
  if (!b) nb = 0;
  if (na + nb <= 0) return cudaSuccess;
  if (!aligned16(a) || !aligned16(b)) return cudaErrorInvalidValue;
  // Up to some 10 MB blocks for four per SM at most; above, four vectors of a thread, however many waves: few blocks that begin early crowd on the
  // SMs that are free.  Behind a product of 24 tiles, us, as up to four per SM / as four vectors: 18.9 MB 4.9 / 3.9, 134 MB 31 / 20, 283 MB 67 / 40 (a
  // fill of torch 4.5, 20, 40); 2.4 MB the same, but the products behind it take the SMs in another order: the decoder's training pass 2000 / 2016.
  const long long vectors = na / 4 + nb / 4, blocks = std::max(std::min((vectors + 255) / 256 + 1, 4LL * sm_count()), (vectors + 1023) / 1024 + 1);
  if (blocks > 0x7fffffffll) return cudaErrorInvalidValue;
  return launch_chained(clear_kernel, dim3(static_cast<unsigned>(blocks)), dim3(256), 0, s, 1, true, a, na, b, nb);
}

cudaError_t fill_normal_bf16(__nv_bfloat16* y, long long n, uint64_t seed, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  long long blocks = ((n + 1) / 2 + 255) / 256;
  if (blocks > sm_count() * 16) blocks = sm_count() * 16;
  fill_normal_kernel<<<static_cast<unsigned>(blocks), 256, 0, s>>>(y, n, seed);
  return cudaGetLastError();
}

}  // namespace mk
