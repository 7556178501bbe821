// Gradient of the weights of a spherical convolution, straight into their own layout:
//
//   dW[c, o, l] = sum_{m <= l} dT[l, m, o] conj(T[l, m, c])         complex fp32, l innermost
//
// The engine's complex product writes real and imaginary planes [l, o, c], of which a second launch makes complex numbers in the order of the
// weights: 0.28 GB written, read and written again for 384 x 384 weights of 240 degrees.  Here a CTA takes four degrees of a tile of 128
// outputs by 64 inputs: eight accumulators of 64 columns fill its tensor memory, and a thread that holds an output's row of all eight writes the
// 32 bytes of four degrees at once, a whole sector.  The degrees of one tile follow one another in the grid, so that the sectors of a
// line meet in L2.  Both planes of both operands are loaded once per 64 orders and serve four products each: 48 KB where the planes took 96.
// 384 x 384 x 240 over 241 orders, L2 flushed, 184 -> 133 us; in a training pass of the convolution (240 x 480) 808 -> 718.  What bounds it is the
// scattered output (590 MB of DRAM traffic at 4.4 TB/s for 280 MB of it): accumulators in two buffers, so that the next tile's products
// run beside the stores, took 150, and eight storing warps 137.
//
// Roles: warps 0 and 18 load the operands of T' and T, warp 1 issues the MMAs, warps 2..17 store (TMEM lanes 32 (w % 4), inputs 16 ((w - 2) / 4)).
// Every wait is bounded; on expiry the kernel records a code in *err and drains.
#include <cuda_bf16.h>

#include "fused_ops.cuh"
#include "launch.cuh"
#include "tcgen05.cuh"

namespace mk {

namespace {

constexpr int TILE_O = 128, TILE_C = 64, DEGREES = 4, BK = 64;
constexpr int BOX = 64 * 128;                           // 64 channels by 64 orders
constexpr int A_PLANE = 2 * BOX, B_PLANE = BOX;
constexpr int STAGE = 2 * (A_PLANE + B_PLANE), STAGES = 4;
constexpr int EPI_WARPS = 16, B_WARP = 2 + EPI_WARPS, THREADS = 32 * (3 + EPI_WARPS);
constexpr uint32_t TMEM_COLS = 512;
constexpr int SMEM = STAGES * STAGE + 8 * (2 * STAGES + 2) + 16 + 1024;
static_assert(SMEM <= SMEM_LIMIT && 2 * DEGREES * TILE_C == TMEM_COLS, "one tile fills the SM");

struct WgradParams {
  int co, ci, L, M;
  int groups, o_tiles;      // groups of DEGREES degrees, tiles of outputs
  uint32_t tiles;
  float2* dw;
  int* err;
};

__global__ void __launch_bounds__(THREADS, 1)
spectral_wgrad_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const WgradParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t pad = (1024u - (raw_addr & 1023u)) & 1023u;
  const uint32_t base = raw_addr + pad, bars = base + STAGES * STAGE;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
  const uint32_t tfull = bars + 8u * (2 * STAGES), tempty = tfull + 8u;
  volatile uint32_t* const tmem_slot = reinterpret_cast<volatile uint32_t*>(smem_raw + pad + STAGES * STAGE + 8 * (2 * STAGES + 2));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 2);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(tfull, 1);
    mbar_init(tempty, EPI_WARPS);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(const_cast<uint32_t*>(tmem_slot))),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  chain_begin(true);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // tile t: outputs from o0, inputs from c0, degrees from l0
  auto tile = [&](uint32_t t, int& o0, int& c0, int& l0) {
    const int xy = static_cast<int>(t) / p.groups;
    l0 = ((xy + 1) * p.groups - 1 - static_cast<int>(t)) * DEGREES;      // (long ones first: the last wave has the short ones)
    c0 = xy / p.o_tiles * TILE_C;
    o0 = xy % p.o_tiles * TILE_O;
  };

  if (warp == 0 || warp == B_WARP) {
    // ------------------------------------------------------------------ operands: 64 orders of both planes
    if (elect_one()) {
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (uint32_t t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
        int o0, c0, l0;
        tile(t, o0, c0, l0);
        for (int l = l0; l < l0 + DEGREES && ok; ++l) {
          for (int k = 0; k < min(l + 1, p.M); k += BK) {
            if (!mbar_wait(empty_bar(s), ph ^ 1u)) {
              atomicExch(p.err, 70);
              ok = false;
              break;
            }
            const uint32_t at = base + s * STAGE;
            if (warp == 0) {
              mbar_expect_tx(full_bar(s), 2 * A_PLANE);
#pragma unroll
              for (int i = 0; i < 4; ++i) tma_load_4d(at + i * BOX, &map_a, full_bar(s), o0 + (i & 1) * 64, k, i >> 1, l);
            } else {
              mbar_expect_tx(full_bar(s), 2 * B_PLANE);
#pragma unroll
              for (int i = 0; i < 2; ++i) tma_load_4d(at + 2 * A_PLANE + i * BOX, &map_b, full_bar(s), c0, k, i, l);
            }
            if (++s == STAGES) {
              s = 0;
              ph ^= 1u;
            }
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      // fp32 accumulators, bf16 operands, both with their rows contiguous; NEG: minus the second one
      constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((TILE_C >> 3) << 17) | ((TILE_O >> 4) << 24);
      constexpr uint32_t NEG = 1u << 14, STEP = (16 * 128) >> 4;
      const uint32_t hi = desc_hi(1024);
      const uint32_t a_lo = desc_lo(base, BOX), b_lo = desc_lo(base + 2 * A_PLANE, BOX);
      int s = 0;
      uint32_t ph = 0, it = 0;
      bool ok = true;
      for (uint32_t t = blockIdx.x; t < p.tiles && ok; t += gridDim.x, ++it) {
        int o0, c0, l0;
        tile(t, o0, c0, l0);
        if (!mbar_wait(tempty, (it & 1u) ^ 1u)) {
          atomicExch(p.err, 71);
          break;
        }
        tc_fence_after();
        for (int l = l0; l < l0 + DEGREES && ok; ++l) {
          const uint32_t re = tmem + (l - l0) * (2 * TILE_C), im = re + TILE_C;
          const int K = min(l + 1, p.M);
          for (int k = 0; k < K; k += BK) {
            if (!mbar_wait(full_bar(s), ph)) {
              atomicExch(p.err, 72);
              ok = false;
              break;
            }
            tc_fence_after();
            const int steps = (min(K - k, BK) + 15) >> 4;      // (orders above the degree are zero)
            const uint32_t off = static_cast<uint32_t>(s) * (STAGE >> 4);
            const uint32_t ar = a_lo + off, ai = ar + (A_PLANE >> 4), br = b_lo + off, bi = br + (B_PLANE >> 4);
            for (int i = 0; i < steps; ++i) {
              const uint32_t d = i * STEP, more = k > 0 || i > 0 ? 1u : 0u;
              tc_mma<2, 1>(re, ar + d, hi, br + d, hi, IDESC, more);
              tc_mma<2, 1>(im, ai + d, hi, br + d, hi, IDESC, more);
              tc_mma<2, 1>(re, ai + d, hi, bi + d, hi, IDESC, 1u);
              tc_mma<2, 1>(im, ar + d, hi, bi + d, hi, IDESC | NEG, 1u);
            }
            tc_commit(empty_bar(s));
            if (++s == STAGES) {
              s = 0;
              ph ^= 1u;
            }
          }
        }
        if (ok) tc_commit(tfull);
      }
    }
  } else {
    // ------------------------------------------------------------------ stores
    const int q = warp & 3, quarter = (warp - 2) >> 2;
    const uint32_t taddr = tmem + (static_cast<uint32_t>(q * 32) << 16) + quarter * 16;
    uint32_t it = 0;
    bool ok = true;
    for (uint32_t t = blockIdx.x; t < p.tiles && ok; t += gridDim.x, ++it) {
      int o0, c0, l0;
      tile(t, o0, c0, l0);
      ok = __all_sync(0xffffffffu, mbar_wait(tfull, it & 1u));
      if (!ok) {
        if (lane == 0) atomicExch(p.err, 73);
        break;
      }
      tc_fence_after();
      const int o = o0 + q * 32 + lane, c = c0 + quarter * 16;
#pragma unroll 1
      for (int g = 0; g < 4; ++g) {
        uint32_t v[2 * DEGREES][4];
#pragma unroll
        for (int i = 0; i < 2 * DEGREES; ++i) tmem_req4(taddr + i * TILE_C + g * 4, v[i]);
#pragma unroll
        for (int i = 0; i < 2 * DEGREES; ++i) tmem_wait4(v[i]);
        if (o < p.co && c + g * 4 < p.ci) {
          float2* const at = p.dw + (static_cast<long long>(c + g * 4) * p.co + o) * p.L + l0;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(at + static_cast<long long>(j) * p.co * p.L), "r"(v[0][j]),
                         "r"(v[1][j]), "r"(v[2][j]), "r"(v[3][j]), "r"(v[4][j]), "r"(v[5][j]), "r"(v[6][j]), "r"(v[7][j])
                         : "memory");
        }
      }
      tc_fence_before();
      __syncwarp();
      if (elect_one()) mbar_arrive(tempty);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

}  // namespace

// Where it takes the place of planes and their re-layout: one sample (a second one would have to add to scattered 32 bytes: 426 us instead of 381
// for two of 384 x 384 x 240), whole sectors, and tiles for half of the SMs.  One degree short of that alignment 8-byte stores made
// 88 us of 68 (200 x 328 x 121).  us, planes / here: 384 x 384 x 128 92 / 59, 256 x 256 x 96 (192 tiles) 35 / 33, 256 x 256 x 64
// (128) 25 / 21, 128 x 64 x 132 (33) 17 / 20, 64 x 64 x 64 (16) 12 / 14.
bool spectral_wgrad_pays(int co, int ci, int L, int samples) {
  const long long tiles = static_cast<long long>((co + TILE_O - 1) / TILE_O) * ((ci + TILE_C - 1) / TILE_C) * (L / DEGREES);
  return samples == 1 && L % DEGREES == 0 && (co & 7) == 0 && (ci & 7) == 0 && 2 * tiles >= sm_count();
}

cudaError_t spectral_wgrad(const __nv_bfloat16* dt, const __nv_bfloat16* t2, float* dw, int co, int ci, int L, int M, int* err_flag,
                           cudaStream_t stream) {
  const long long tiles = static_cast<long long>((co + TILE_O - 1) / TILE_O) * ((ci + TILE_C - 1) / TILE_C) * (L / DEGREES);
  if (co <= 0 || ci <= 0 || L <= 0 || M <= 0 || (co & 7) || (ci & 7) || L % DEGREES != 0 || tiles >= (1ll << 30) ||
      (reinterpret_cast<uintptr_t>(dw) & 31))
    return cudaErrorInvalidValue;
  bind_context(stream);
  static std::atomic<uint64_t> devices;
  const cudaError_t allowed = allow_shared_memory(devices, reinterpret_cast<const void*>(&spectral_wgrad_kernel), SMEM);
  if (allowed != cudaSuccess) return allowed;
  auto operand = [&](const __nv_bfloat16* t, int c) {
    GemmOperand op;
    op.ptr = t;
    op.rows = c;
    op.mn_major = 1;
    op.ld = 2ll * c;
    op.zs_lo = c;                    // real and imaginary plane
    op.zs_hi = 2ll * c * M;
    return op;
  };
  CUtensorMap ma, mb;
  if (!make_map(&ma, operand(dt, co), M, 2, 2, L, 64) || !make_map(&mb, operand(t2, ci), M, 2, 2, L, 64)) return cudaErrorInvalidValue;
  WgradParams p;
  p.co = co;
  p.ci = ci;
  p.L = L;
  p.M = M;
  p.groups = L / DEGREES;
  p.o_tiles = (co + TILE_O - 1) / TILE_O;
  p.tiles = static_cast<uint32_t>(tiles);
  p.dw = reinterpret_cast<float2*>(dw);
  p.err = err_flag;
  const long long sms = sm_count();
  return launch_chained(spectral_wgrad_kernel, dim3(static_cast<unsigned>(tiles < sms ? tiles : sms)), dim3(THREADS), SMEM, stream, 1, true, ma, mb, p);
}

}  // namespace mk
