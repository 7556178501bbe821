// Persistent warp-specialised GEMM for sm_100a: TMA -> shared memory (128B swizzle) -> tcgen05.mma with
// accumulators in tensor memory -> tcgen05.ld epilogue with fused bias / GELU / residual / scatter.
//
// Roles per CTA (one CTA per SM; EW epilogue warps: one per 64-column box and lane quarter of the tile, see epi_warps):
//   warps 0, EW+2  : TMA producers (one elected lane each), which fill every second stage of the ring
//   warp 1         : TMEM allocator + MMA issuer (one elected lane)
//   warps 2..EW+1  : epilogue; warp w reads TMEM lanes [32*(w%4), 32*(w%4)+32) and the 64-column box (w-2)/4 (generic
//                    epilogue: alternating 32-column chunks)
//   warp EW+3      : only in launches whose epilogue operand (residual, saved pre-activation) is prefetched by TMA: its
//                    producer, so that waiting for a free operand buffer never delays A and B
//   warps EW+3..   : only in launches that also sum the rows of A (bias gradients): eight warps that add up the stages of their tile's
//                    turn before these are freed; the producer releases the others in their name
// Two accumulator buffers in TMEM let the epilogue of tile i overlap the main loop of tile i+1.
// Every mbarrier wait is bounded; on expiry the kernel records a code in *err and drains.
//
// CTA pairs (template parameter CG = 2, single-GPU launches only): two CTAs of a thread-block cluster share one
// 256-row tile.  Each CTA loads its own 128 rows of A and HALF of the B tile (plain TMA loads, no multicast, whose
// completion is counted on the leader CTA's barrier); the leader issues tcgen05.mma.cta_group::2, which reads both
// CTAs' shared memory and writes 128 accumulator rows into each CTA's TMEM; tcgen05.commit multicasts the
// "stage free" and "accumulator full" signals to both CTAs.  Per tensor-core cycle every SM then takes a third less
// data from L2 (two thirds with 128-wide tiles).
//
// Complex products (p.cplx = 1, 2, 3): real and imaginary planes of the operands are multiplied without ever forming the real 2x2-block
// matrix.  The column tiles come in two halves (real, imaginary part of the result) and the k loop in two segments that
// select the planes; the one negative product of the four uses the negation bit of the MMA's instruction descriptor.
//   1: D(h) = sum_s A[.., s Kh + k] B(plane h ^ s),  minus at h = 0, s = 1      (product with W)
//   2: the same, minus at h = 1, s = 0                                          (product with the conjugate of W)
//   3: D(h) = sum_s A(plane s ^ h) B(plane s),       minus at h = 1, s = 1      (weight gradient)
// 384 x 384 weights of 240 degrees: the operand takes 69 us to make instead of 95 (half the bytes), the products 87 - 94 us instead
// of 105 - 114, the weight gradient one launch of 90 us instead of two of 78 and a swapped copy of 31.
//
// Folded transforms (p.cplx = 4, 5): a Fourier matrix has rows r and R - r that differ in nothing but the sign of one half of their
// columns, so one product of half the rows serves both.  The two halves are two segments of the k loop with accumulators of their
// own, and the epilogue stores their sum at row r and their difference at row R - r, both from fp32:
//   4: rows are longitudes (synthesis): the halves are the cosine and the sine terms, i.e. the real and imaginary planes of B
//   5: rows are (order, re / im) pairs of all orders up to half the points (analysis): the halves are the even and the odd
//      points; the pairs keep their order, and the imaginary difference changes its sign
//
// Multi-GPU use (one process per GPU, buffers mapped through CUDA IPC):
//   * the k axis of the B operand may be cut into up to 8 segments with their own base pointers and tensor maps
//     (the per-rank segments of a gathered buffer in this device's own memory);
//   * the bf16 output may be replicated into up to 7 more buffers with the layout of D (the same segment of every
//     peer's copy), by plain 16-byte stores or TMA stores over NVLink: no load ever targets peer memory;
//   * producer / consumer ordering across devices uses monotonic counters (PeerSync) checked by the first thread of
//     every CTA before any work and advanced by the last CTA of the grid.
#include "gemm_tcgen05.cuh"
#include "gelu.cuh"
#include "fused_ops.cuh"
#include "launch.cuh"
#include "tcgen05.cuh"

#include <cuda.h>
#include <cuda_bf16.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>

namespace mk {

namespace {

constexpr int BM = 128;
constexpr int A_STAGE_BYTES = BM * 128;
// Epilogue warps of an instance.  The specialised epilogues give every 64-column box of every lane quarter a warp of its
// own: 8 / 12 / 16 warps for 128- / 192- / 256-column tiles.  With eight warps for any width a warp of a wide tile worked
// through its boxes one after the other, two warps per scheduler, at 50 % issue utilisation; the generic epilogue (fp32
// outputs, atomics) needs its registers and stays at eight.
__host__ __device__ constexpr int epi_warps(int bn, int epi) { return epi == 0 ? 8 : bn / 16; }
// Register bound, given as a thread count: the warps of one scheduler's register bank (5, 4 or 3 of them) leave room for one
// 64-register warp of the gradient all-reduce, which overlaps with these GEMMs in data-parallel training.
__host__ __device__ constexpr int bound_threads(int bn, int epi) {
  if (epi == 5) return 32 * (epi_warps(bn, 5) + 12);      // with the row sums: 19, 23 or 27 warps of at most 64 registers
  return epi == 0 || bn == 128 ? 384 : (bn == 192 ? 576 : 736);
}
constexpr int MAX_STAGES = 6;
constexpr int SUM_WARPS = 8;
constexpr int MAX_SEG = 8;

// Handshake of a kernel that consumes buffers its peers have filled and/or fills a buffer that its peers consume.
//   wait[i]   : local flag array (one slot per peer) that must reach *wait_exp[i] + wait_off[i] before the first load
//   bump[i]   : local counter incremented by one when the whole grid has finished
//   sig[i][p] : flag slot in peer p's memory incremented by one when the whole grid has finished
struct PeerSync {
  int np_wait[2], np_sig[2];      // number of peers of the group each wait / signal list refers to
  int nwait, nsig;
  const unsigned int* wait[2];
  const unsigned int* wait_exp[2];
  int wait_off[2];
  unsigned int* bump[2];
  unsigned int* sig[2][MAX_SEG];
  unsigned int* done_ctr;
};

struct BMaps {
  CUtensorMap m[MAX_SEG];
};
// tensor maps of the additional destinations (the same output written into peers' memory)
struct DMaps {
  CUtensorMap m[MAX_SEG - 1];
};

// Division of a 31-bit index by an invariant: q = (umulhi(n, mul) + n) >> shift (Granlund and Montgomery 1994).  Every
// warp of a CTA decodes every tile; with 64-bit divisions that was a third of an epilogue warp's instructions.
struct FastDiv {
  uint32_t d, mul, shift;
};
__device__ __forceinline__ uint32_t fast_div(uint32_t n, const FastDiv& f) { return (__umulhi(n, f.mul) + n) >> f.shift; }

struct KParams {
  int M, N, K;
  int zlo_n, zhi_n;
  int splits, k_per_split;
  int a_mn, b_mn;
  int a_zlo, a_zhi, b_zlo, b_zhi;
  int rmin_a, rmin_b, rmax_a, rmax_b, kmin_a, kmin_b, kmax_a, kmax_b;
  long long d_zlo, d_zhi;
  int rdiv; long long rs_hi, rs_lo;
  int ndiv; long long ns_hi;
  float alpha;
  const float* bias;
  long long bias_zs;              // elements between the bias vectors of consecutive z_lo batches (0: one shared vector)
  int bias_mode, act, save_deriv;
  GeluCoef gelu;
  float act_param;
  const void* resid;
  void* preact;
  void* D;
  int out_f32, accumulate, vec_ok;
  int m_tiles, n_tiles;
  FastDiv dv_n, dv_m, dv_split, dv_zlo;
  uint32_t total_tiles;           // below 2^31
  int a_part;                     // k coordinate of the second part of a K-major A (complex and folded products)
  int n_full;                     // columns in whole 16-byte vectors of the output
  int mirror, fold_rows;          // folded products: rows r < M and mirror - r, which are the rows M to fold_rows
  int cplx, nth, neg_half, neg_seg;   // complex product: mode, column tiles per half, the negative (half, segment)
  int stages, e_tma;
  int d_zlo_on, d_zhi_on;         // fp32 output through TMA: 0 where all batches of that index add into one output
  int rd_shift;                   // log2 of rdiv where the output leaves through TMA (0: rows have one stride)
  float* rowsum;                  // partial sums of the rows of A over k, [group][slab][row] (null: none)
  int producers;                  // TMA producer warps at work
  int rs_groups, rs_slabs;        // groups: z_lo batches with outputs of their own; slabs of one group
  int n_fast;                     // tile order: 1 = n-tile index fastest, 0 = m-tile index fastest
  int* err;
  // ---- B operand gathered from several devices: segment s of the k axis was written by rank s into the local buffer
  int nseg;                       // 1: ordinary single-map operand
  int seg_len[MAX_SEG];           // local k extent of each segment
  int seg_apos[MAX_SEG];          // k coordinate of the segment start in the A operand (padded layout)
  int seg_gstart[MAX_SEG];        // global k index of the segment start (for the kmin/kmax structure)
  // ---- output replicated into peers' memory: ndx additional destinations with the layout of D
  int ndx;
  void* Dx[MAX_SEG - 1];
  // ---- cross-device handshakes (all counters are monotonic and live in device memory)
  PeerSync sync;
};

__device__ __forceinline__ uint4 pack_bf16x8(const float (&x)[8]) {
  f32x2 f[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) f[j] = f2_pack(x[2 * j], x[2 * j + 1]);
  return f2_bf16x8(f);
}

template <int V>
struct IntC {
  static constexpr int value = V;
};

struct TileCoord {
  int zhi, zlo, split, mt, nt;
  int half;             // complex products: real (0) or imaginary (1) part; nt counts the column tiles inside the half
  int k_begin, k_end;   // element range, k_begin multiple of BK
  bool skip;
};

// CG = 2: `t` counts 256-row pair tiles (p.m_tiles is then the number of pair tiles) and `half` (0 / 1) selects this
// CTA's 128 rows; skip decisions are taken for the pair as a whole because the MMA is issued once for both CTAs.
template <int BK, int CG = 1>
__device__ __forceinline__ TileCoord decode_tile(const KParams& p, uint32_t t, int half = 0) {
  TileCoord c;
  // The index that varies fastest walks over the tiles that share the larger operand, so that the CTAs of one wave
  // fetch that operand's tile from DRAM once and hit L2 for the rest (token-major convolutions: many m-tiles of
  // activations against two to six n-tiles of weights -> n fastest).
  auto take = [&](const FastDiv& f) {
    const uint32_t qt = fast_div(t, f);
    const int rem = static_cast<int>(t - qt * f.d);
    t = qt;
    return rem;
  };
  if (p.n_fast) {
    c.nt = take(p.dv_n);
    c.mt = take(p.dv_m);
  } else {
    c.mt = take(p.dv_m);
    c.nt = take(p.dv_n);
  }
  c.half = p.cplx != 0 && c.nt >= p.nth ? 1 : 0;
  c.nt -= c.half * p.nth;
  c.split = take(p.dv_split);
  c.zlo = take(p.dv_zlo);
  c.zhi = static_cast<int>(t);
  const int rmin = p.rmin_a * c.zhi + p.rmin_b;
  const int rmax = p.rmax_a * c.zhi + p.rmax_b;
  int kmin = p.kmin_a * c.zhi + p.kmin_b;
  int kmax = p.kmax_a * c.zhi + p.kmax_b;
  if (kmin < 0) kmin = 0;
  if (kmax > p.K) kmax = p.K;
  int kb = c.split * p.k_per_split;
  int ke = kb + p.k_per_split;
  if (ke > p.K) ke = p.K;
  const int kmin_al = (kmin / BK) * BK;
  if (kb < kmin_al) kb = kmin_al;
  if (ke > kmax) ke = kmax;
  c.k_begin = kb;
  c.k_end = ke;
  const int r0 = c.mt * (BM * CG);
  c.skip = (r0 + BM * CG <= rmin) || (r0 >= rmax) || (p.nseg == 1 && kb >= ke);
  if constexpr (CG == 2) c.mt = c.mt * 2 + half;   // from here on: this CTA's own 128-row block
  return c;
}

// Specialised epilogues leave through TMA stores of 32-row x 128-byte boxes, one per epilogue warp and output.  Without an
// epilogue operand (1, 2) the boxes are staged in a buffer of their own; with one (3, 4) the warp overwrites the operand's
// box in place, element by element, and the store reads from there: no staging, so 192-column tiles fit.
__host__ __device__ constexpr int stg_warp_bytes(int epi) { return epi == 2 || epi == 6 ? 2 * 32 * 128 : (epi == 1 || epi == 5 ? 32 * 128 : 0); }
__host__ __device__ constexpr int stg_bytes(int bn, int epi) { return epi_warps(bn, epi) * stg_warp_bytes(epi); }

// EPI selects a compile-time specialised epilogue (bf16 output but for 5):
//   0 generic (all options decided at run time)      1 plain store
//   2 GELU + saved pre-activation                     3 + residual (TMA-prefetched)      4 * GELU'(aux) (TMA-prefetched)
//   5 fp32 output, stored or added (split-k, summed batches): weight gradients
//   6 sum and difference of two accumulators, stored at row r and its mirror row (folded transforms)
// RAGGED (1 to 4): widths that are no multiple of 8.  A TMA store writes whole 16-byte vectors, also over the edge of its tensor map, and
// what lies behind the last column in a wider matrix is not this launch's: the columns of a last, partial vector leave one by one.
// Instances of their own (128 columns, single CTAs), as the others have no registers to spare.  384 -> 764 over 115200 tokens with a
// column bias, us: 107 (GELU 128), through the generic epilogue 242 (418); 768 columns 72 (88).
// rows of B per stage: whole MN-major boxes of 64 (a pair's half of a 192-wide tile is one and a half of them)
__host__ __device__ constexpr int b_stage_rows(int bn, int cg) { return (bn / cg + 63) / 64 * 64; }

// local k range [lb, le) of segment `sg` for tile `c` (multi-device B operand)
template <int BK>
__device__ __forceinline__ void seg_range(const KParams& p, const TileCoord& c, int sg, int& lb, int& le) {
  int kmin = p.kmin_a * c.zhi + p.kmin_b - p.seg_gstart[sg];
  int kmax = p.kmax_a * c.zhi + p.kmax_b - p.seg_gstart[sg];
  lb = kmin > 0 ? (kmin / BK) * BK : 0;
  le = kmax < p.seg_len[sg] ? kmax : p.seg_len[sg];
}

__device__ __forceinline__ unsigned int ld_acquire_sys_u32(const unsigned int* ptr) {
  unsigned int v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(ptr) : "memory");
  return v;
}

template <int BN, int EB, int EPI, int CG, bool RAGGED>
__global__ void __launch_bounds__(bound_threads(BN, EPI), 1)
gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ BMaps maps_b,
            const __grid_constant__ CUtensorMap map_e, const __grid_constant__ CUtensorMap map_d,
            const __grid_constant__ CUtensorMap map_p, const __grid_constant__ DMaps maps_dx, const KParams p) {
  const CUtensorMap& map_b = maps_b.m[0];
  constexpr int BK = 128 / EB;            // elements per 128-byte k-slab
  constexpr int UMMA_K = 32 / EB;         // elements per tcgen05.mma
  constexpr int BNL = BN / CG;            // rows of the B tile this CTA contributes (a pair splits the tile)
  constexpr int B_STAGE_BYTES = b_stage_rows(BN, CG) * 128;
  constexpr int EW = epi_warps(BN, EPI);
  constexpr int PRODUCER_2 = 2 + EW;      // second TMA producer
  constexpr int E_WARP = 3 + EW;
  constexpr int SUM_WARP = 3 + EW;        // (no instance has both)
  constexpr int STAGE_BYTES = A_STAGE_BYTES + B_STAGE_BYTES;
  constexpr int MN_BOX = 128 / EB;        // extent of an MN-major box along the contiguous dimension
  constexpr int ACC_COLS = EPI == 6 ? 2 * BN : BN;        // columns of one accumulator buffer
  constexpr uint32_t TMEM_COLS = ACC_COLS == 128 ? 256 : 512;   // two of them, rounded up to a power of two
  constexpr uint32_t E_BYTES = BM * BN * 2;    // bf16 epilogue-operand tile
  const int STAGES = p.stages;

  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  const uint32_t pad = (1024u - (raw_addr & 1023u)) & 1023u;
  uint8_t* smem = smem_raw + pad;
  const uint32_t smem_base = raw_addr + pad;

  // layout: [stages][E tile x2 (optional)][staging][barriers]
  const uint32_t e_off = STAGES * STAGE_BYTES;
  const uint32_t stg_off = e_off + (p.e_tma ? 2 * E_BYTES : 0);
  const uint32_t bar_off = stg_off + stg_bytes(BN, EPI);
  uint8_t* bar_ptr = smem + bar_off;
  const uint32_t bar_base = smem_base + bar_off;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (MAX_STAGES + s); };
  auto tfull_bar = [&](int b) { return bar_base + 8u * (2 * MAX_STAGES + b); };
  auto tempty_bar = [&](int b) { return bar_base + 8u * (2 * MAX_STAGES + 2 + b); };
  auto efull_bar = [&](int b) { return bar_base + 8u * (2 * MAX_STAGES + 4 + b); };
  auto eempty_bar = [&](int b) { return bar_base + 8u * (2 * MAX_STAGES + 6 + b); };
  auto sum_bar = [&](int st) { return bar_base + 8u * (2 * MAX_STAGES + 8 + st); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bar_ptr + 8 * (3 * MAX_STAGES + 8));

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // pair geometry: `crank` = rank inside the cluster (the leader is rank 0), tiles are dealt out per cluster
  const int crank = (CG == 2) ? static_cast<int>(cluster_ctarank()) : 0;
  const uint32_t tile0 = (CG == 2) ? (blockIdx.x >> 1) : blockIdx.x;
  const uint32_t tile_step = (CG == 2) ? (gridDim.x >> 1) : gridDim.x;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), EPI == 5 && p.rowsum != nullptr ? 1 + SUM_WARPS : 1);
      if constexpr (EPI == 5) mbar_init(sum_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(tfull_bar(b), 1);
      mbar_init(tempty_bar(b), EW * CG);
      mbar_init(efull_bar(b), 1);
      mbar_init(eempty_bar(b), EW);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    if constexpr (CG == 2) {
      // the same warp of both CTAs allocates, with the same destination offset
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                       smem_u32(const_cast<uint32_t*>(tmem_slot))),
                   "r"(TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                       smem_u32(const_cast<uint32_t*>(tmem_slot))),
                   "r"(TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  chain_begin(p.sync.nwait == 0);
  if (threadIdx.x == 0) {
    // segments written by the peers (and the peers' copies this kernel overwrites) must be ready: bounded wait on local flags.
    // The whole CTA waits (not only the producer) so that no epilogue store of an all-zero tile can run early.
    bool ok = true;
    for (int w = 0; w < p.sync.nwait && ok; ++w) {
      const unsigned int need = *p.sync.wait_exp[w] + static_cast<unsigned int>(p.sync.wait_off[w]);
      for (int peer = 0; peer < p.sync.np_wait[w] && ok; ++peer) {
        uint64_t t0 = 0;
        for (uint32_t it = 0;; ++it) {
          if (static_cast<int>(ld_acquire_sys_u32(p.sync.wait[w] + peer) - need) >= 0) break;
          if ((it & 255u) == 255u) {
            const uint64_t now = global_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > WAIT_LIMIT_NS) {
              atomicExch(p.err, 32 + w);
              ok = false;
              break;
            }
          }
        }
      }
    }
    tmem_slot[1] = ok ? 1u : 0u;
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (CG == 2) cluster_sync_all();   // the partner's barriers are initialised before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const bool peers_ready = tmem_slot[1] != 0u;

  if (warp == 0 || warp == PRODUCER_2) {
    // ------------------------------------------------------------------ TMA producers
    // Two warps take the k slabs of this CTA in turn.  One slab costs a producer its wait, its byte count and two to six TMA
    // instructions one after the other, some 450 - 700 cycles; a slab's MMAs take 256 - 512, and with a single producer it was
    // this thread that most launches waited for, with the loads in flight far from filling the ring.  Back to back, under the power
    // cap: 768 -> 384 over 721 x 1440 tokens 699 -> 649 us, its gradient 707 -> 650, 384 -> 768 with GELU and GELU' 928 -> 882.
    //
    // With an odd number of stages both fill every stage, in turn.  Neither mistakes one lap for another: stages are freed in the
    // order of their MMAs, so that having met the release of slab g - 2 - STAGES a producer that waits for slab g - STAGES knows
    // slab g - 2 STAGES free.  Where the row sums' warps hold stages too there is no such order, and one producer fills them all
    // (p.producers).
    if (elect_one() && (warp == 0 || p.producers == 2)) {
      const int step = p.producers;
      const uint32_t me = warp == 0 ? 0u : 1u;
      int s = static_cast<int>(me);
      uint32_t ph = 0, slab = 0;      // slab: slabs of the CTA so far; this producer fills those of its parity
      bool ok = peers_ready;
      if (p.sync.nwait > 0) asm volatile("fence.proxy.async;" ::: "memory");   // flags acquired in the prologue order the TMA loads below
      // pair: every load of both CTAs is counted on the leader's "full" barrier.  The leader announces the bytes of both; the
      // partner's loads may land first (the barrier's byte count goes negative for a moment, its phase cannot complete
      // before the leader's arrival)
      const uint32_t leader_full0 = (CG == 2) ? mapa_u32(full_bar(0), 0) : 0u;
      const uint32_t load_bytes = A_STAGE_BYTES + (p.b_mn ? B_STAGE_BYTES : BNL * 128);
      const bool a_mn = p.a_mn != 0, b_mn = p.b_mn != 0;
      // this producer's next stage: waits until it is free and loads the k slabs of A at ka, rows m0, and of B at kb, rows nb
      auto stage = [&](const CUtensorMap* mb, int ka, int m0, int azl, int azh, int kb, int nb, int bzl, int bzh, bool pass) {
        if (!mbar_wait(empty_bar(s), ph ^ 1u)) {
          atomicExch(p.err, 1);
          return false;
        }
        if constexpr (EPI == 5) {
          if (pass) mbar_arrive_n(empty_bar(s), SUM_WARPS);
        }
        const uint32_t sa = smem_base + s * STAGE_BYTES;
        const uint32_t sb = sa + A_STAGE_BYTES;
        if constexpr (CG == 2) {
          if (crank == 0) mbar_expect_tx(full_bar(s), 2 * load_bytes);
          const uint32_t bar = leader_full0 + 8u * s;
          if (!a_mn) {
            tma_load_4d_pair(sa, &map_a, bar, ka, m0, azl, azh);
          } else {
#pragma unroll
            for (int j = 0; j < BM / MN_BOX; ++j) tma_load_4d_pair(sa + j * (BK * 128), &map_a, bar, m0 + j * MN_BOX, ka, azl, azh);
          }
          if (!b_mn) {
            tma_load_4d_pair(sb, mb, bar, kb, nb, bzl, bzh);
          } else {
#pragma unroll
            for (int j = 0; j < B_STAGE_BYTES / (BK * 128); ++j)
              tma_load_4d_pair(sb + j * (BK * 128), mb, bar, nb + j * MN_BOX, kb, bzl, bzh);
          }
        } else {
          const uint32_t bar = full_bar(s);
          mbar_expect_tx(bar, load_bytes);
          if (!a_mn) {
            tma_load_4d(sa, &map_a, bar, ka, m0, azl, azh);
          } else {
#pragma unroll
            for (int j = 0; j < BM / MN_BOX; ++j) tma_load_4d(sa + j * (BK * 128), &map_a, bar, m0 + j * MN_BOX, ka, azl, azh);
          }
          if (!b_mn) {
            tma_load_4d(sb, mb, bar, kb, nb, bzl, bzh);
          } else {
#pragma unroll
            for (int j = 0; j < BN / MN_BOX; ++j) tma_load_4d(sb + j * (BK * 128), mb, bar, nb + j * MN_BOX, kb, bzl, bzh);
          }
        }
        s += step;
        if (s >= STAGES) {
          s -= STAGES;
          ph ^= 1u;
        }
        return true;
      };
      const bool simple = p.nseg <= 1 && p.cplx == 0;
      for (uint32_t t = tile0; t < p.total_tiles && ok; t += tile_step) {
        const TileCoord c = decode_tile<BK, CG>(p, t, crank);
        if (c.skip) continue;
        const int m0 = c.mt * BM, nb = c.nt * BN + (CG == 2 ? crank * BNL : 0);
        int azl = p.a_zlo ? c.zlo : 0, bzl = p.b_zlo ? c.zlo : 0;
        const int azh = p.a_zhi ? c.zhi : 0, bzh = p.b_zhi ? c.zhi : 0;
        const int nsg = simple ? 1 : (p.cplx ? 2 : p.nseg);
        for (int sg = 0; sg < nsg && ok; ++sg) {
          int lb = c.k_begin, le = c.k_end, apos = 0;
          const CUtensorMap* mb = &map_b;
          if (!simple) {
            if (p.nseg > 1) {
              seg_range<BK>(p, c, sg, lb, le);
              apos = p.seg_apos[sg];
              mb = &maps_b.m[sg];
            } else {
              // segment and half select the planes, which take the place of the lower batch index
              bzl = p.cplx == 3 ? sg : (sg ^ c.half);
              if (p.cplx == 3) azl = sg ^ c.half;
              else apos = sg * p.a_part;
            }
          }
          const int k0 = lb + static_cast<int>((slab ^ me) & (step - 1)) * BK;
          if constexpr (EPI == 5) {
            if (p.rowsum) {
              int turn = k0 > lb ? 1 : 0;      // slab modulo the column tiles
              for (int k = k0; k < le && ok; k += step * BK) {
                while (turn >= p.n_tiles) turn -= p.n_tiles;
                // another tile's turn: the row sums' warps pass this slab by (the stage is this producer's until it is loaded,
                // so the arrival counts for its next release)
                ok = stage(mb, apos + k, m0, azl, azh, k, nb, bzl, bzh, turn != c.nt);
                turn += step;
              }
              slab += static_cast<uint32_t>(le - lb + BK - 1) / BK;
              continue;
            }
          }
          for (int k = k0; k < le && ok; k += step * BK) ok = stage(mb, apos + k, m0, azl, azh, k, nb, bzl, bzh, false);
          if (le > lb) slab += static_cast<uint32_t>(le - lb + BK - 1) / BK;
        }
      }
    }
  } else if (EPI == 5 && warp >= SUM_WARP) {
    // ------------------------------------------------------------------ sums of the rows of A (bias gradients)
    // The gradient of a bias is the sum over the tokens of the matrix that the weight gradient has in shared memory anyway:
    // read from there, it costs no pass over memory (0.8 or 1.6 GB and two launches at 721 x 1440 tokens).  A is MN-major: a stage
    // holds 64 tokens as rows of 64 channels, twice.  Warp w adds up 16 tokens of one half, a lane 8 channels of every fourth
    // token, in fp32; the column tiles of one row block, which load the same slabs, take the slabs in turn, and for the others
    // the producer frees the stage in the name of these warps.  Every warp writes a partial sum per tile, and a second launch adds
    // them in a fixed order: as exact as the pass of their own that they replace (errors against 64 bits 3.5e-8 one-signed, 1e-7
    // zero-mean, 721 x 1440 tokens, both).  Gradient and sums, a pass of their own / from here, us, 721 x 1440 tokens: 384 x 768
    // 746 / 642, 768 x 384 766 / 736, 384 x 384 451 / 353; 240 x 480: 104 / 91, 111 / 98, 69 / 55; 2048 tokens: 32 / 24.
    if constexpr (EPI == 5) {
      const int w = warp - SUM_WARP, bx = w >> 2;
      const uint32_t cgroup = lane & 7;
      const int k0 = (w & 3) * 16 + (lane >> 3);
      const uint8_t* const col = smem + bx * (BK * 128) + k0 * 128;
      const uint32_t at0 = (cgroup ^ (k0 & 7)) << 4, at1 = (cgroup ^ ((k0 + 4) & 7)) << 4;
      // The thread that issues the MMAs passes every slab in order and announces those of this tile's turn; waiting for the loads'
      // own barrier, these warps could meet the parity of another lap, since they skip slabs.  In a pair that barrier lives in the
      // leader; there the announcement is a commit, which reaches both CTAs when the slab's MMAs are done (told by one thread to
      // another, at cluster scope, 768 x 384 over 721 x 1440 tokens took 950 us).
      uint32_t seen = 0;               // parity of each stage's announcements
      uint32_t first = 0;              // stage of the tile's first slab
      bool ok = peers_ready;
      for (uint32_t t = tile0; t < p.total_tiles; t += tile_step) {
        const TileCoord c = decode_tile<BK, CG>(p, t, crank);
        f32x2 acc[4] = {0ull, 0ull, 0ull, 0ull};
        const int nblocks = c.skip ? 0 : (c.k_end - c.k_begin + BK - 1) / BK;
        uint32_t s = (first + c.nt) % STAGES;
        for (int kb = c.nt; kb < nblocks && ok; kb += p.n_tiles) {
          const uint32_t want = (seen >> s) & 1u;
          ok = __all_sync(0xffffffffu, mbar_wait(sum_bar(s), want));
          if (!ok) {
            if (lane == 0) atomicExch(p.err, 7);
            break;
          }
          seen ^= 1u << s;
          const uint8_t* const st = col + s * STAGE_BYTES;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            f32x2 v[4];
            f2_unpack8(*reinterpret_cast<const uint4*>(st + i * (4 * 128) + (i & 1 ? at1 : at0)), v);
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[j] = f2_add(acc[j], v[j]);
          }
          __syncwarp();
          if (elect_one()) mbar_arrive(empty_bar(s));
          s = (s + p.n_tiles) % STAGES;
        }
        first = (first + nblocks) % STAGES;
        // lanes l, l + 8, l + 16, l + 24 hold the same channels
        const int group = p.rs_groups > 1 ? c.zlo : 0;
        const int z = p.rs_groups > 1 ? c.zhi : c.zhi * p.zlo_n + c.zlo;
        const long long slab = ((static_cast<long long>(z) * p.splits + c.split) * p.n_tiles + c.nt) * 4 + (w & 3);
        const int r0 = c.mt * BM + bx * 64 + static_cast<int>(cgroup) * 8;
        float* const out = p.rowsum + (static_cast<long long>(group) * p.rs_slabs + slab) * p.M + r0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float a, b;
          f2_unpack(acc[j], a, b);
#pragma unroll
          for (int o = 8; o < 32; o <<= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
          }
          if (lane < 8) {
            if (r0 + 2 * j < p.M) out[2 * j] = a;
            if (r0 + 2 * j + 1 < p.M) out[2 * j + 1] = b;
          }
        }
      }
    }
  } else if (warp == E_WARP) {
    // ------------------------------------------------------------------ producer of the epilogue operand
    // A warp of its own: the tile of the residual / saved pre-activation for tile t+2 can only be requested when the
    // epilogue of tile t has released its buffer.  Issued from the operand producer's loop, that wait held back the
    // A and B loads of the tiles in between; issued from another lane of the producer warp, its polling held up that
    // warp's TMA issue.
    if (elect_one() && p.e_tma && peers_ready) {
      if (p.sync.nwait > 0) asm volatile("fence.proxy.async;" ::: "memory");
      uint32_t epi_it = 0;
      for (uint32_t t = tile0; t < p.total_tiles; t += tile_step) {
        const TileCoord c = decode_tile<BK, CG>(p, t, crank);
        if (c.skip && p.accumulate) continue;
        const int eb = epi_it & 1;
        if (!mbar_wait(eempty_bar(eb), ((epi_it >> 1) & 1u) ^ 1u)) {
          atomicExch(p.err, 5);
          break;
        }
        mbar_expect_tx(efull_bar(eb), E_BYTES);
#pragma unroll
        for (int j = 0; j < BN / 64; ++j)
          tma_load_tile(smem_base + e_off + eb * E_BYTES + j * (BM * 128), &map_e, efull_bar(eb), c.nt * BN + j * 64, c.half,
                        (c.mt * BM) >> p.rd_shift, c.zlo, c.zhi);
        ++epi_it;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one() && crank == 0) {
      // instruction descriptor: fp32 accumulate, operand format, majors, N, M (256 rows for a CTA pair)
      const uint32_t fmt = (EB == 2) ? 1u : 2u;   // BF16 : TF32
      const uint32_t idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | (static_cast<uint32_t>(p.a_mn) << 15) |
                             (static_cast<uint32_t>(p.b_mn) << 16) | (static_cast<uint32_t>(BN >> 3) << 17) |
                             (static_cast<uint32_t>((BM * CG) >> 4) << 24);
      const uint32_t a_lbo = p.a_mn ? BK * 128 : 16, a_sbo = 1024;
      const uint32_t b_lbo = p.b_mn ? BK * 128 : 16, b_sbo = 1024;
      const uint32_t a_kstep = (p.a_mn ? UMMA_K * 128 : 32) >> 4;
      const uint32_t b_kstep = (p.b_mn ? UMMA_K * 128 : 32) >> 4;
      const uint32_t a_hi = desc_hi(a_sbo), b_hi = desc_hi(b_sbo);
      const uint32_t a_lo0 = desc_lo(smem_base, a_lbo), b_lo0 = desc_lo(smem_base + A_STAGE_BYTES, b_lbo);
      int s = 0;
      uint32_t ph = 0, acc_it = 0;
      bool ok = peers_ready;
      for (uint32_t t = tile0; t < p.total_tiles && ok; t += tile_step) {
        const TileCoord c = decode_tile<BK, CG>(p, t, crank);
        if (c.skip) continue;
        const int buf = acc_it & 1;
        if (!mbar_wait(tempty_bar(buf), ((acc_it >> 1) & 1u) ^ 1u)) {
          atomicExch(p.err, 2);
          break;
        }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + buf * ACC_COLS;
        uint32_t accum = 0;
        int nblocks = 0;
        if (p.nseg > 1) {
          for (int sg = 0; sg < p.nseg; ++sg) {
            int lb, le;
            seg_range<BK>(p, c, sg, lb, le);
            if (le > lb) nblocks += (le - lb + BK - 1) / BK;
          }
        } else {
          nblocks = (c.k_end - c.k_begin + BK - 1) / BK;
          if (p.cplx) nblocks *= 2;
        }
        // the negative product of a complex one: bit 14 of the instruction descriptor negates B in one half of the k loop
        const uint32_t neg = p.cplx != 0 && c.half == p.neg_half ? 1u << 14 : 0u;
        int turn = 0;
        const int kneg = p.neg_seg ? nblocks >> 1 : 0, kpos = p.neg_seg ? nblocks : nblocks >> 1;
        const int khalf = nblocks >> 1;
        for (int kb = 0; kb < nblocks; ++kb) {
          if (!mbar_wait(full_bar(s), ph)) {
            atomicExch(p.err, 3);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t off = static_cast<uint32_t>(s) * (STAGE_BYTES >> 4);
          const uint32_t id = idesc | (kb >= kneg && kb < kpos ? neg : 0u);
          uint32_t acc_d = tmem_d;
          if constexpr (EPI == 6) {      // the second half of the columns has an accumulator of its own
            if (kb >= khalf) acc_d = tmem_d + BN;
            if (kb == khalf) accum = 0;
          }
#pragma unroll
          for (int kk = 0; kk < BK / UMMA_K; ++kk) {
            tc_mma<EB, CG>(acc_d, a_lo0 + off + kk * a_kstep, a_hi, b_lo0 + off + kk * b_kstep, b_hi, id, accum);
            accum = 1;
          }
          // frees the smem stage (in both CTAs of a pair) once these MMAs have read it
          if constexpr (CG == 2) tc_commit_pair(empty_bar(s));
          else tc_commit(empty_bar(s));
          if constexpr (EPI == 5) {
            if (p.rowsum) {      // announces the slabs that this tile sums up
              if (turn == c.nt) {
                if constexpr (CG == 2) tc_commit_pair(sum_bar(s));
                else mbar_arrive(sum_bar(s));
              }
              if (++turn == p.n_tiles) turn = 0;
            }
          }
          if (++s == STAGES) {
            s = 0;
            ph ^= 1u;
          }
        }
        if constexpr (CG == 2) tc_commit_pair(tfull_bar(buf));   // accumulator complete (both halves)
        else tc_commit(tfull_bar(buf));
        ++acc_it;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue warps
    // Warp w serves TMEM lanes [32*(w%4), +32), one accumulator row per thread.  Specialised epilogues: the 64-column box
    // (w-2)/4.  Generic epilogue: the 32-column chunks with (chunk % 2) == (w-2)/4.
    const int q = warp & 3;
    const int half = (warp - 2) >> 2;
    uint32_t acc_it = 0, epi_it = 0;
    bool ok = peers_ready;
    // the "accumulator drained" barrier of a pair lives in the leader and counts the warps of both CTAs
    const uint32_t leader_tempty0 = (CG == 2) ? mapa_u32(tempty_bar(0), 0) : 0u;
    const f32x2 alpha2 = f2_keep(p.alpha);
    GeluPairs gelu2;
    if constexpr (EPI == 1 || EPI == 2) gelu2 = gelu_pairs(p.gelu);
    for (uint32_t t = tile0; t < p.total_tiles; t += tile_step) {
      const TileCoord c = decode_tile<BK, CG>(p, t, crank);
      if (c.skip && p.accumulate) continue;
      const int rt = q * 32 + lane;                 // row inside the tile
      const int r = c.mt * BM + rt;
      const int n0 = c.nt * BN;
      const bool row_ok = r < p.M;
      const long long row_off = static_cast<long long>(c.zhi) * p.d_zhi + static_cast<long long>(c.zlo) * p.d_zlo +
                                static_cast<long long>(r / p.rdiv) * p.rs_hi + static_cast<long long>(r % p.rdiv) * p.rs_lo;
      const float* const bias_z = p.bias + static_cast<long long>(c.zlo) * p.bias_zs;
      float rbias = 0.f;
      if (p.bias_mode == 1 && row_ok) rbias = __ldg(bias_z + r);
      int buf = 0, ebuf = 0;
      if (!c.skip) {
        buf = acc_it & 1;
        if (ok && !mbar_wait(tfull_bar(buf), (acc_it >> 1) & 1u)) {
          atomicExch(p.err, 4);
          ok = false;
        }
        tc_fence_after();
      }
      const uint8_t* esm = nullptr;
      if (p.e_tma) {
        ebuf = epi_it & 1;
        if (ok && !mbar_wait(efull_bar(ebuf), (epi_it >> 1) & 1u)) {
          atomicExch(p.err, 6);
          ok = false;
        }
        esm = smem + e_off + ebuf * E_BYTES;
      }
      if constexpr (EPI == 5) {
        // ---------------- fp32: the 64 columns of a box in two halves of 32 (128 bytes), staged, then stored or added as full
        // lines.  The generic epilogue's 16-byte accesses, one row per lane, touched 32 lines per instruction (weight
        // gradients of the AFNO filter: 28.6 -> 13.8 us and 22.9 -> 13.1 us).
        const int bx = half;
        const uint32_t box_off = stg_off + (warp - 2) * stg_warp_bytes(5);
        uint8_t* const box = smem + box_off + lane * 128;
        const int r0 = c.mt * BM + q * 32;
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          const int nb = n0 + bx * 64 + h * 32;
          if (nb >= p.N) break;       // uniform across the warp
          tma_store_wait_read<0>();
          __syncwarp();
#pragma unroll
          for (int it = 0; it < 2; ++it) {
            uint32_t v[16];
            if (!c.skip) {
              tmem_ld16(tmem_base + buf * ACC_COLS + bx * 64 + h * 32 + it * 16 + (static_cast<uint32_t>(q * 32) << 16), v);
            } else {
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] = 0u;
            }
#pragma unroll
            for (int g = 0; g < 4; ++g)
              *reinterpret_cast<float4*>(box + (((it * 4 + g) ^ (lane & 7)) << 4)) =
                  make_float4(__uint_as_float(v[4 * g]) * p.alpha, __uint_as_float(v[4 * g + 1]) * p.alpha,
                              __uint_as_float(v[4 * g + 2]) * p.alpha, __uint_as_float(v[4 * g + 3]) * p.alpha);
          }
          fence_async_smem();
          __syncwarp();
          if (elect_one() && r0 < p.M) {
            const int zl = p.d_zlo_on ? c.zlo : 0, zh = p.d_zhi_on ? c.zhi : 0;
            if (p.accumulate) tma_add_tile(&map_d, smem_base + box_off, nb, c.half, r0 >> p.rd_shift, zl, zh);
            else tma_store_tile(&map_d, smem_base + box_off, nb, c.half, r0 >> p.rd_shift, zl, zh);
            tma_store_commit();
          }
        }
        if (!c.skip) {
          tc_fence_before();
          __syncwarp();
          if (elect_one()) {
            if constexpr (CG == 2) mbar_arrive_cluster(leader_tempty0 + 8u * buf);
            else mbar_arrive(tempty_bar(buf));
          }
          ++acc_it;
        }
        continue;
      } else if constexpr (EPI == 6) {
        // ---------------- sum and difference: two boxes of 32 rows, the second in the order of the mirror rows
        const int nb = n0 + half * 64;
        const uint32_t box_off = stg_off + (warp - 2) * stg_warp_bytes(6);
        const int r0 = c.mt * BM + q * 32;
        const bool any = nb < p.N && r0 < p.M;      // uniform across the warp
        const bool pairs = p.cplx == 5;
        if (any) {
          const uint32_t taddr = tmem_base + buf * ACC_COLS + half * 64 + (static_cast<uint32_t>(q * 32) << 16);
          tma_store_wait_read<0>();
          __syncwarp();
          const int ml = pairs ? 30 - lane + 2 * (lane & 1) : 31 - lane;
          uint8_t* const sum_row = smem + box_off + lane * 128;
          uint8_t* const dif_row = smem + box_off + 32 * 128 + ml * 128;
          const uint32_t l7 = static_cast<uint32_t>(lane & 7) << 4, m7 = static_cast<uint32_t>(ml & 7) << 4;
          const f32x2 minus = f2_keep(-1.f);
          const f32x2 sign = f2_keep(pairs && (lane & 1) ? -1.f : 1.f);
#pragma unroll 1
          for (int it = 0; it < 4; ++it) {
            uint32_t u[16], v[16];
            tmem_ld16(taddr + it * 16, u);
            tmem_ld16(taddr + BN + it * 16, v);
#pragma unroll
            for (int gg = 0; gg < 2; ++gg) {
              const uint32_t g = static_cast<uint32_t>((it * 2 + gg) << 4);
              f32x2 a[4], d[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const f32x2 x = f2_pack(__uint_as_float(u[gg * 8 + 2 * j]), __uint_as_float(u[gg * 8 + 2 * j + 1]));
                const f32x2 y = f2_pack(__uint_as_float(v[gg * 8 + 2 * j]), __uint_as_float(v[gg * 8 + 2 * j + 1]));
                a[j] = f2_add(x, y);
                d[j] = f2_mul(f2_fma(y, minus, x), sign);
              }
              *reinterpret_cast<uint4*>(sum_row + (g ^ l7)) = f2_bf16x8(a);
              *reinterpret_cast<uint4*>(dif_row + (g ^ m7)) = f2_bf16x8(d);
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (elect_one()) {
          if constexpr (CG == 2) mbar_arrive_cluster(leader_tempty0 + 8u * buf);
          else mbar_arrive(tempty_bar(buf));
        }
        ++acc_it;
        if (any) {
          fence_async_smem();
          __syncwarp();
          // Every row leaves once: sums up to row M (clipped by their tensor map), differences from there on.  Row 0 has its mirror
          // past the end where that is no row (clipped).  The last box of differences may begin before row M, which no tensor map
          // clips: one box of the W / 64 takes the ordinary path.
          const int m0 = p.mirror - r0 - (pairs ? 30 : 31);
          if (elect_one()) {
            tma_store_tile(&map_d, smem_base + box_off, nb, 0, r0, c.zlo, c.zhi);
            if (m0 >= p.M && m0 < p.fold_rows) tma_store_tile(&map_p, smem_base + box_off + 32 * 128, nb, 0, m0, c.zlo, c.zhi);
            tma_store_commit();
          }
          if (m0 < p.M) {
            __nv_bfloat16* const out = static_cast<__nv_bfloat16*>(p.D) + c.zhi * p.d_zhi;
            for (int i = lane; i < 32 * 8; i += 32) {
              const int j = i >> 3, row = m0 + j, col = nb + (i & 7) * 8;
              if (row < p.M || row >= p.fold_rows || col >= p.N) continue;
              *reinterpret_cast<uint4*>(out + row * p.rs_lo + col) =
                  *reinterpret_cast<const uint4*>(smem + box_off + (32 + j) * 128 + (((i ^ j) & 7) << 4));
            }
          }
        }
        continue;
      } else if constexpr (EPI != 0) {
        // ---------------- specialised bf16 epilogues: registers -> swizzled smem box -> TMA store (full lines, clipped
        // at the matrix edge by the tensor map)
        constexpr bool IN_PLACE = (EPI == 3 || EPI == 4);
        const int bx = half;
        const int nb = n0 + bx * 64;
        // the box this warp's output is written to: staging (1, 2) or the operand's own box (3, 4)
        const uint32_t box_off = IN_PLACE ? e_off + ebuf * E_BYTES + bx * (BM * 128) + q * (32 * 128)
                                          : stg_off + (warp - 2) * stg_warp_bytes(EPI) + (EPI == 2 ? 32 * 128 : 0);
        if (nb < p.N) {     // uniform across the warp
          const uint32_t taddr = tmem_base + buf * ACC_COLS + bx * 64 + (static_cast<uint32_t>(q * 32) << 16);
          // the previous store of this warp must have read its box (the operand box was released after that already)
          if constexpr (!IN_PLACE) {
            tma_store_wait_read<0>();
            __syncwarp();
          }
          const f32x2 rbias2 = f2_pack(rbias, rbias);
          // The 64 columns of a box go through a ROLLED loop of four 16-column steps.  Unrolled, the body of one box ran
          // to tens of KB of straight-line code per epilogue flavour, the epilogue warps (each at another place
          // in it) missed the instruction caches on most fetches, and "no instruction" was their top stall reason.
          // Arithmetic is on pairs of columns (fma / mul on f32x2): same roundings, half the instructions.
          // What is uniform over the launch (column bias, activation) selects one of several copies of the loop, not a branch
          // inside it: every branch that rejoins with the accumulators in registers copied them (12.6 instructions per
          // output element of a plain store, half of them moves).  384 -> 768 with GELU, 721 x 1440 tokens: 831 -> 626 us without the
          // second output, 961 -> 928 us with it; 384 -> 768 over 240 x 480 tokens without: 103 -> 84 us.
          uint8_t* const sw_d = smem + box_off + lane * 128;
          const uint32_t l7 = static_cast<uint32_t>(lane & 7) << 4;
          auto columns = [&](auto bias_c, auto act_c) {
            constexpr int COL_BIAS = decltype(bias_c)::value;
            constexpr int ACT = decltype(act_c)::value;
#pragma unroll 1
            for (int it = 0; it < 4; ++it) {
              uint32_t v[16];
              tmem_ld16(taddr + it * 16, v);
#pragma unroll
              for (int gg = 0; gg < 2; ++gg) {
                const uint32_t sw = static_cast<uint32_t>((it * 2 + gg) << 4) ^ l7;
                f32x2 f[4];
                if constexpr (COL_BIAS == 1) {      // rides on the scaling fma (columns past N are clipped by the store)
                  const int n = min(nb + it * 16 + gg * 8, p.N - 8);
                  const ulonglong2 b0 = __ldg(reinterpret_cast<const ulonglong2*>(bias_z + n));
                  const ulonglong2 b1 = __ldg(reinterpret_cast<const ulonglong2*>(bias_z + n) + 1);
                  f[0] = b0.x; f[1] = b0.y; f[2] = b1.x; f[3] = b1.y;
                } else if constexpr (COL_BIAS == 2) {      // (RAGGED)
                  const int n = nb + it * 16 + gg * 8;
#pragma unroll
                  for (int j = 0; j < 4; ++j) f[j] = f2_pack(__ldg(bias_z + min(n + 2 * j, p.N - 1)), __ldg(bias_z + min(n + 2 * j + 1, p.N - 1)));
                } else {
#pragma unroll
                  for (int j = 0; j < 4; ++j) f[j] = rbias2;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j)
                  f[j] = f2_fma(f2_pack(__uint_as_float(v[gg * 8 + 2 * j]), __uint_as_float(v[gg * 8 + 2 * j + 1])), alpha2, f[j]);
                if constexpr (EPI == 1 && ACT == 1) {
#pragma unroll
                  for (int j = 0; j < 4; ++j) f[j] = gelu_fwd2(f[j], gelu2);
                } else if constexpr (EPI == 1 && ACT != 0) {      // ReLU / soft shrinkage
#pragma unroll
                  for (int j = 0; j < 4; ++j) {
                    float x, y;
                    f2_unpack(f[j], x, y);
                    f[j] = f2_pack(act_fwd(x, ACT, p.act_param, p.gelu), act_fwd(y, ACT, p.act_param, p.gelu));
                  }
                }
                if constexpr (EPI == 2) {      // second output: GELU' of the pre-activation, or the pre-activation itself
                  f32x2 s2[4];
#pragma unroll
                  for (int j = 0; j < 4; ++j) {
                    if constexpr (ACT == 1) {
                      gelu_fwd_bwd2(f[j], gelu2, f[j], s2[j]);
                    } else {
                      s2[j] = f[j];
                      f[j] = gelu_fwd2(f[j], gelu2);
                    }
                  }
                  *reinterpret_cast<uint4*>(sw_d - 32 * 128 + sw) = f2_bf16x8(s2);
                }
                if constexpr (IN_PLACE) {
                  f32x2 e[4];
                  f2_unpack8(*reinterpret_cast<const uint4*>(sw_d + sw), e);
#pragma unroll
                  for (int j = 0; j < 4; ++j) {
                    if constexpr (EPI == 3) f[j] = f2_add(f[j], e[j]);
                    else if constexpr (ACT == 8) f[j] = f2_mul(f[j], e[j]);      // the operand is the saved derivative
                    else {
                      float e0, e1;
                      f2_unpack(e[j], e0, e1);
                      f[j] = f2_mul(f[j], f2_pack(act_bwd(e0, ACT, p.gelu), act_bwd(e1, ACT, p.gelu)));
                    }
                  }
                }
                *reinterpret_cast<uint4*>(sw_d + sw) = f2_bf16x8(f);
              }
            }
          };
          auto with_act = [&](auto bias_c) {
            if constexpr (EPI == 1) {
              if (p.act == 0) columns(bias_c, IntC<0>{});
              else if (p.act == 1) columns(bias_c, IntC<1>{});
              else if (p.act == 3) columns(bias_c, IntC<3>{});
              else columns(bias_c, IntC<5>{});
            } else if constexpr (EPI == 2) {
              if (p.save_deriv) columns(bias_c, IntC<1>{});
              else columns(bias_c, IntC<0>{});
            } else if constexpr (EPI == 3) {
              columns(bias_c, IntC<0>{});
            } else {
              // a copy for each activation: with the code asked for at run time a product times the derivative of GELU (ReLU, shrinkage)
              // took 200 (161, 130) us, 384 -> 768 over 115200 tokens; now 102 (93, 93), times a saved one 93
              if (p.act == 8) columns(bias_c, IntC<8>{});
              else if (p.act == 2) columns(bias_c, IntC<2>{});
              else if (p.act == 4) columns(bias_c, IntC<4>{});
              else columns(bias_c, IntC<6>{});
            }
          };
          if (c.skip) {
            // no product reaches this tile (triangular structure): the epilogue of zeros
#pragma unroll 1
            for (int g = 0; g < 8; ++g) {
              const uint32_t sw = static_cast<uint32_t>(g << 4) ^ l7;
              float x[8];
#pragma unroll
              for (int j = 0; j < 8; ++j)
                x[j] = p.bias_mode != 2 ? rbias : __ldg(bias_z + (RAGGED ? min(nb + g * 8 + j, p.N - 1) : min(nb + g * 8, p.N - 8) + j));
              if constexpr (EPI == 2) {
                float d[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) d[j] = p.save_deriv ? gelu_bwd(x[j], p.gelu) : x[j];
                *reinterpret_cast<uint4*>(sw_d - 32 * 128 + sw) = pack_bf16x8(d);
              }
              if constexpr (EPI == 1 || EPI == 2) {
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = act_fwd(x[j], p.act, p.act_param, p.gelu);
              }
              if constexpr (IN_PLACE) {
                const uint4 ev = *reinterpret_cast<const uint4*>(sw_d + sw);
                const uint32_t ew[4] = {ev.x, ev.y, ev.z, ev.w};
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  const float e = __uint_as_float(j & 1 ? ew[j / 2] & 0xffff0000u : ew[j / 2] << 16);
                  x[j] = EPI == 3 ? x[j] + e : x[j] * act_bwd(e, p.act, p.gelu);
                }
              }
              *reinterpret_cast<uint4*>(sw_d + sw) = pack_bf16x8(x);
            }
          } else if (p.bias_mode == 2) {
            with_act(IntC<RAGGED ? 2 : 1>{});
          } else {
            with_act(IntC<0>{});
          }
        }
        if (!c.skip) {     // the accumulator has been read: the next tile but one may overwrite it
          tc_fence_before();
          __syncwarp();
          if (elect_one()) {
            if constexpr (CG == 2) mbar_arrive_cluster(leader_tempty0 + 8u * buf);
            else mbar_arrive(tempty_bar(buf));
          }
          ++acc_it;
        }
        if (nb < p.N) {
          fence_async_smem();
          __syncwarp();
          const int r0 = c.mt * BM + q * 32;
          if (elect_one() && r0 < p.M && (!RAGGED || nb < p.n_full)) {
            const int rs = r0 >> p.rd_shift;
            if constexpr (EPI == 2) tma_store_tile(&map_p, smem_base + box_off - 32 * 128, nb, 0, rs, c.zlo, c.zhi);
            tma_store_tile(&map_d, smem_base + box_off, nb, c.half, rs, c.zlo, c.zhi);
            if constexpr (EPI == 1) {
              for (int dq = 0; dq < p.ndx; ++dq)   // the same box goes to every peer's copy (plain stores over NVLink)
                tma_store_tile(&maps_dx.m[dq], smem_base + box_off, nb, 0, rs, c.zlo, c.zhi);
            }
            tma_store_commit();
            if constexpr (IN_PLACE) tma_store_wait_read<0>();   // the operand buffer is free once the store has read it
          }
          if constexpr (RAGGED) {
            if (nb + 64 > p.n_full && row_ok) {
              const long long at = row_off + p.n_full;
              const uint8_t* const box = smem + box_off + lane * 128 + (((p.n_full - nb) << 1) ^ ((lane & 7) << 4));
              auto tail = [&](const uint8_t* from, void* to) {
                const uint4 v = *reinterpret_cast<const uint4*>(from);
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
                uint16_t* const o = static_cast<uint16_t*>(to) + at;
#pragma unroll
                for (int j = 0; j < 7; ++j)
                  if (p.n_full + j < p.N) o[j] = static_cast<uint16_t>(w[j / 2] >> (16 * (j & 1)));
              };
              tail(box, p.D);
              if constexpr (EPI == 2) tail(box - 32 * 128, p.preact);
            }
          }
        }
        if constexpr (IN_PLACE) {
          __syncwarp();
          if (elect_one()) mbar_arrive(eempty_bar(ebuf));
          ++epi_it;
        }
        continue;
      } else
#pragma unroll 1
      for (int cc = half; cc < BN / 32; cc += 2) {
        const int nc = n0 + cc * 32;
        if (nc >= p.N) break;       // uniform across the warp
        const uint32_t taddr = tmem_base + buf * ACC_COLS + cc * 32 + (static_cast<uint32_t>(q * 32) << 16);
        // rolled: one copy of the (large, many-layout) body serves the four 8-column groups, which keeps the
        // epilogue within the instruction cache
#pragma unroll 1
        for (int g = 0; g < 4; ++g) {
          const int n = nc + g * 8;
          if (n >= p.N) break;      // uniform across the warp
          uint32_t v[8];
          if (!c.skip) {
            tmem_ld8(taddr + g * 8, v);
          } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = 0u;
          }
          if (!row_ok) continue;
          float f[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(v[j]) * p.alpha;
          if (p.bias_mode == 1) {
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] += rbias;
          } else if (p.bias_mode == 2) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (n + j < p.N) f[j] += __ldg(bias_z + n + j);
          }
          const bool full = (n + 8 <= p.N);
          const long long off = row_off + static_cast<long long>(n / p.ndiv) * p.ns_hi + (n % p.ndiv);
          // epilogue operand for these 8 columns (bf16 tile prefetched by TMA, 128-byte swizzle: the 16-byte chunk
          // index inside each 128-byte row segment is XORed with (row % 8))
          float e8[8];
          if (p.e_tma) {
            const int col = cc * 32 + g * 8;                     // column inside the tile
            const int box = col >> 6, chunk = (col & 63) >> 3;
            const uint4 ev = *reinterpret_cast<const uint4*>(esm + box * (BM * 128) + rt * 128 + ((chunk ^ (rt & 7)) << 4));
            const __nv_bfloat162* eh = reinterpret_cast<const __nv_bfloat162*>(&ev);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 x = __bfloat1622float2(eh[j]);
              e8[2 * j] = x.x;
              e8[2 * j + 1] = x.y;
            }
          }
          if (full && p.vec_ok && !p.accumulate) {
            // ---- vector path: 8 consecutive columns
            if (p.preact) {
              float s8[8];     // second output: the pre-activation, or GELU' of it
#pragma unroll
              for (int j = 0; j < 8; ++j) s8[j] = p.save_deriv ? gelu_bwd(f[j], p.gelu) : f[j];
              if (p.out_f32) {
                float4* o = reinterpret_cast<float4*>(static_cast<float*>(p.preact) + off);
                o[0] = make_float4(s8[0], s8[1], s8[2], s8[3]);
                o[1] = make_float4(s8[4], s8[5], s8[6], s8[7]);
              } else {
                __nv_bfloat162 h[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(s8[2 * j], s8[2 * j + 1]);
                *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.preact) + off) = *reinterpret_cast<uint4*>(h);
              }
            }
            if (p.act & 1) {
#pragma unroll
              for (int j = 0; j < 8; ++j) f[j] = act_fwd(f[j], p.act, p.act_param, p.gelu);
            }
            if (p.resid) {
              if (!p.e_tma) {
                if (p.out_f32) {
                  const float4* ri = reinterpret_cast<const float4*>(static_cast<const float*>(p.resid) + off);
                  const float4 a = ri[0], b = ri[1];
                  e8[0] = a.x; e8[1] = a.y; e8[2] = a.z; e8[3] = a.w;
                  e8[4] = b.x; e8[5] = b.y; e8[6] = b.z; e8[7] = b.w;
                } else {
                  const uint4 rv = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p.resid) + off);
                  const __nv_bfloat162* rh = reinterpret_cast<const __nv_bfloat162*>(&rv);
#pragma unroll
                  for (int j = 0; j < 4; ++j) {
                    const float2 x = __bfloat1622float2(rh[j]);
                    e8[2 * j] = x.x;
                    e8[2 * j + 1] = x.y;
                  }
                }
              }
#pragma unroll
              for (int j = 0; j < 8; ++j) f[j] = (p.act != 0 && !(p.act & 1)) ? f[j] * act_bwd(e8[j], p.act, p.gelu) : f[j] + e8[j];
            }
            if (p.out_f32) {
              float4* o = reinterpret_cast<float4*>(static_cast<float*>(p.D) + off);
              o[0] = make_float4(f[0], f[1], f[2], f[3]);
              o[1] = make_float4(f[4], f[5], f[6], f[7]);
            } else {
              __nv_bfloat162 h[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(f[2 * j], f[2 * j + 1]);
              *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.D) + off) = *reinterpret_cast<uint4*>(h);
              for (int dq = 0; dq < p.ndx; ++dq)
                *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(p.Dx[dq]) + off) = *reinterpret_cast<uint4*>(h);
            }
          } else if (full && p.vec_ok && p.accumulate && p.out_f32 && !p.preact && p.act == 0) {
            // ---- split-k / batch accumulation in fp32: two 16-byte vector atomics instead of eight scalar ones
            float4* o = reinterpret_cast<float4*>(static_cast<float*>(p.D) + off);
            atomicAdd(o, make_float4(f[0], f[1], f[2], f[3]));
            atomicAdd(o + 1, make_float4(f[4], f[5], f[6], f[7]));
          } else {
            // ---- scalar path (ragged edge, unaligned layouts, atomic accumulation)
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int nj = n + j;
              if (nj >= p.N) break;
              const long long o = row_off + static_cast<long long>(nj / p.ndiv) * p.ns_hi + (nj % p.ndiv);
              float x = f[j];
              if (p.preact) {
                const float sx = p.save_deriv ? gelu_bwd(x, p.gelu) : x;
                if (p.out_f32) static_cast<float*>(p.preact)[o] = sx;
                else static_cast<__nv_bfloat16*>(p.preact)[o] = __float2bfloat16(sx);
              }
              if (p.act & 1) x = act_fwd(x, p.act, p.act_param, p.gelu);
              if (p.accumulate) {
                atomicAdd(static_cast<float*>(p.D) + o, x);
              } else {
                if (p.resid) {
                  float rr;
                  if (p.e_tma) rr = e8[j];
                  else rr = p.out_f32 ? static_cast<const float*>(p.resid)[o]
                                      : __bfloat162float(static_cast<const __nv_bfloat16*>(p.resid)[o]);
                  x = (p.act != 0 && !(p.act & 1)) ? x * act_bwd(rr, p.act, p.gelu) : x + rr;
                }
                if (p.out_f32) static_cast<float*>(p.D)[o] = x;
                else {
                  static_cast<__nv_bfloat16*>(p.D)[o] = __float2bfloat16(x);
                  for (int dq = 0; dq < p.ndx; ++dq) static_cast<__nv_bfloat16*>(p.Dx[dq])[o] = __float2bfloat16(x);
                }
              }
            }
          }
        }
      }
      if (!c.skip) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if constexpr (CG == 2) mbar_arrive_cluster(leader_tempty0 + 8u * buf);
          else mbar_arrive(tempty_bar(buf));
        }
        ++acc_it;
      }
      if (p.e_tma) {
        __syncwarp();
        if (lane == 0) mbar_arrive(eempty_bar(ebuf));
        ++epi_it;
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  if constexpr (EPI != 0) {
    if (warp >= 2 && warp < PRODUCER_2) {      // (bulk groups belong to the lane that committed them)
      tma_store_wait_all();
      asm volatile("fence.proxy.async;" ::: "memory");   // order the bulk stores before the generic-proxy signalling below
    }
  }
  tc_fence_before();
  __syncthreads();
  if (p.sync.done_ctr != nullptr && threadIdx.x == 0) {
    // last CTA of the grid: everything this kernel wrote (here and into the peers' copies) is complete and everything it
    // consumed may be overwritten
    __threadfence_system();
    const unsigned int prev = atomicAdd(p.sync.done_ctr, 1u);
    if (prev == gridDim.x - 1) {
      *p.sync.done_ctr = 0;
      // after an expired wait nothing is published: the counters keep describing the last complete generation
      if (*reinterpret_cast<volatile int*>(p.err) == 0) {
        for (int i = 0; i < p.sync.nwait; ++i)
          if (p.sync.bump[i]) atomicAdd(p.sync.bump[i], 1u);
        __threadfence_system();
        for (int i = 0; i < p.sync.nsig; ++i)
          for (int peer = 0; peer < p.sync.np_sig[i]; ++peer)
            if (p.sync.sig[i][peer]) atomicAdd_system(p.sync.sig[i][peer], 1u);
      }
    }
  }
  if constexpr (CG == 2) cluster_sync_all();   // neither CTA leaves (or frees TMEM) while its partner may still touch it
  if (warp == 1) {
    tc_fence_after();
    if constexpr (CG == 2)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// ---------------------------------------------------------------------------------------------- host side

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

char g_err[512] = {0};

EncodeTiledFn get_encode() {
  static EncodeTiledFn fn = nullptr;
  if (fn) return fn;
  void* sym = nullptr;
  cudaDriverEntryPointQueryResult qres;
  cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres);
  if (e != cudaSuccess || qres != cudaDriverEntryPointSuccess || sym == nullptr) return nullptr;
  fn = reinterpret_cast<EncodeTiledFn>(sym);
  return fn;
}

}  // namespace

bool make_map(CUtensorMap* map, const GemmOperand& op, int K, int eb, int zlo_n, int zhi_n, int box_rows_kmajor) {
  EncodeTiledFn enc = get_encode();
  if (!enc) {
    snprintf(g_err, sizeof(g_err), "cuTensorMapEncodeTiled entry point not available");
    return false;
  }
  const int bk = 128 / eb;
  cuuint64_t dims[4];
  cuuint64_t strides[3];
  cuuint32_t box[4];
  cuuint32_t estr[4] = {1, 1, 1, 1};
  const bool use_lo = (op.zs_lo != 0) && zlo_n > 1;
  const bool use_hi = (op.zs_hi != 0) && zhi_n > 1;
  if (!op.mn_major) {
    dims[0] = static_cast<cuuint64_t>(K);
    dims[1] = static_cast<cuuint64_t>(op.rows);
    box[0] = bk;
    box[1] = box_rows_kmajor;
  } else {
    dims[0] = static_cast<cuuint64_t>(op.rows);
    dims[1] = static_cast<cuuint64_t>(K);
    box[0] = 128 / eb;
    box[1] = bk;
  }
  dims[2] = use_lo ? zlo_n : 1;
  dims[3] = use_hi ? zhi_n : 1;
  box[2] = 1;
  box[3] = 1;
  strides[0] = static_cast<cuuint64_t>(op.ld) * eb;
  strides[1] = use_lo ? static_cast<cuuint64_t>(op.zs_lo) * eb : strides[0];
  strides[2] = use_hi ? static_cast<cuuint64_t>(op.zs_hi) * eb : strides[0];
  if ((reinterpret_cast<uintptr_t>(op.ptr) & 15) || (strides[0] & 15) || (strides[1] & 15) || (strides[2] & 15)) {
    snprintf(g_err, sizeof(g_err), "gemm operand not 16-byte aligned (ptr %p ld %lld zs %lld %lld)", op.ptr, op.ld,
             op.zs_lo, op.zs_hi);
    return false;
  }
  CUresult r = enc(map, eb == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4,
                   const_cast<void*>(op.ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    snprintf(g_err, sizeof(g_err),
             "cuTensorMapEncodeTiled failed (%d): dims %llu %llu %llu %llu strides %llu %llu %llu box %u %u", (int)r,
             (unsigned long long)dims[0], (unsigned long long)dims[1], (unsigned long long)dims[2],
             (unsigned long long)dims[3], (unsigned long long)strides[0], (unsigned long long)strides[1],
             (unsigned long long)strides[2], box[0], box[1]);
    return false;
  }
  return true;
}

// CTA pairs that can be resident at once.  Every instance fills an SM with its shared memory, so one answers for all.
static int max_pairs() {
  static const int n = [] {
    cudaLaunchConfig_t qc;
    memset(&qc, 0, sizeof(qc));
    cudaLaunchAttribute qa[1];
    qa[0].id = cudaLaunchAttributeClusterDimension;
    qa[0].val.clusterDim.x = 2;
    qa[0].val.clusterDim.y = 1;
    qa[0].val.clusterDim.z = 1;
    qc.gridDim = dim3(2 * (sm_count() / 2), 1, 1);
    qc.blockDim = dim3(32 * (4 + epi_warps(256, 0)), 1, 1);
    qc.dynamicSmemBytes = SMEM_LIMIT;
    qc.attrs = qa;
    qc.numAttrs = 1;
    int got = 0;
    cudaError_t e = cudaFuncSetAttribute(gemm_kernel<256, 2, 0, 2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&got, gemm_kernel<256, 2, 0, 2, false>, &qc);
    if (e != cudaSuccess || got < 1) {
      (void)cudaGetLastError();
      got = sm_count() / 2;
    }
    return got;
  }();
  return n;
}

// Without the context bound (threads that only inherited the device index, e.g. autograd workers, until their first runtime call) the
// encoding fails.  Once per host thread: the call is not allowed while a stream is capturing, and threads are reused.
void bind_context(cudaStream_t stream) {
  static thread_local bool bound = false;
  if (bound) return;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone) {
    cudaFree(nullptr);
    bound = true;
  }
}

namespace {
// Grid of a product with tiles of few rows or columns.  CTA c walks the tiles c, c + grid, ...: where the tiles of one batch and the grid have
// a factor in common, a CTA meets the same few of them in every batch, and if those are the narrow ones it runs ahead of its
// neighbours.  It idles at the end, and on the way what two tiles share (the halves of 128-byte lines of a folded product's output, the rows of
// activations of a plain one) is met so far apart in time that it leaves L2 in between.  A grid without a common factor mixes
// them.  Synthesis of 1440 points, 64 orders, 136 channels 150 -> 88, 200 channels 187 -> 108; of 256 points, 129 orders, 384 channels
// 35 -> 30 us.  Where a batch has many row tiles, all alike, the column tiles of one row take the place of a batch, and
// at most one wave in sixteen may be added: what the rows cost twice is more than the waves (64 -> 264 channels over 720 x 1440 tokens, 110 waves of pairs
// become 111, 259 -> 149 us; 128 -> 264 over 721 x 1440, 110 and 112, 187 -> 163; 384 -> 264 327 -> 291; 240 x 480 tokens, no wave more, 26.2 -> 26.1).
long long mixed_grid(long long grid, const KParams& kp, int bm, int bn) {
  const bool columns = static_cast<long long>(kp.m_tiles) * kp.n_tiles > 256;
  if (columns && !kp.n_fast) return grid;
  const int tiles = columns ? kp.n_tiles : kp.m_tiles * kp.n_tiles;
  if (tiles <= 1 || tiles > 256 || kp.total_tiles <= static_cast<uint32_t>(grid)) return grid;
  auto gcd = [](long long a, long long b) {
    while (b) {
      const long long t = a % b;
      a = b;
      b = t;
    }
    return a;
  };
  const int classes = static_cast<int>(gcd(grid, tiles));
  long long least = 0, most = 0;
  for (int c = 0; c < classes; ++c) {
    long long area = 0;
    for (int i = c; i < tiles; i += classes) {
      const int mt = columns ? 0 : (kp.n_fast ? i / kp.n_tiles : i % kp.m_tiles), nt = kp.n_fast ? i % kp.n_tiles : i / kp.m_tiles;
      area += static_cast<long long>(std::min(bm, kp.M - mt * bm)) * std::min(bn, kp.N - nt * bn);
    }
    least = c == 0 ? area : std::min(least, area);
    most = std::max(most, area);
  }
  if (most * 4 <= least * 5) return grid;
  const long long total = kp.total_tiles;
  for (long long g = grid - 1; g > grid - 8 && g > 0; --g)
    if (gcd(g, tiles) == 1) return columns && (total + g - 1) / g > (total + grid - 1) / grid + total / (16 * grid) ? grid : g;
  return grid;
}

// Most k slabs of a CTA (or pair) in a launch that begins while the one before it ends.  Its CTAs take the SMs in the order in which these
// become free, and where CTAs that share operands land on different halves of the chip these are fetched twice: long launches lose more
// than the gap they save.  384 -> 384 channels over 721 x 1440 tokens (660 slabs) 342 us in the ordinary way, 354 chained; the decoder's training
// pass, with the gradients of its weights (330 slabs and more) chained 1984, without 1969.  The products of 115200 tokens or 16200 x 768
// -> 3072 have 110 to 150: 596 -> 582 and 518 -> 503 chained.
// Products of several samples that add into one output lose more, from some 64 slabs on (a pass of 4 samples in the ordinary way / chained, us: 304 x 544
// over 37888 tokens each, 144 slabs, 78 / 85; 272 x 888 over 22848, 116 slabs, 92 / 99; 264 x 848 over 17728, 90 slabs, 61 / 67; 296 x 208 over
// 29184, 37 slabs, 39 / 39); of one sample they are even or gain (768 x 384 over 115200, 146 slabs, 73 / 71).
constexpr long long CHAINED_SLABS = 256, CHAINED_SLABS_OF_SAMPLES = 64;

template <int BN, int EB, int EPI, int CG, bool RAGGED = false>
cudaError_t launch_t(const CUtensorMap& ma, const BMaps& mb, const CUtensorMap& me, const CUtensorMap& md,
                     const CUtensorMap& mp, const DMaps& mdx, KParams& kp, cudaStream_t stream) {
  constexpr int STAGE = A_STAGE_BYTES + b_stage_rows(BN, CG) * 128;
  constexpr int FIXED = stg_bytes(BN, EPI) + 8 * (3 * MAX_STAGES + 8) + 16 + 1024;
  const int e_bytes = kp.e_tma ? 2 * BM * BN * 2 : 0;
  int stages = (SMEM_LIMIT - FIXED - e_bytes) / STAGE;
  if (stages > MAX_STAGES) stages = MAX_STAGES;
  if (stages < 2) {
    snprintf(g_err, sizeof(g_err), "not enough shared memory for the requested tile configuration");
    return cudaErrorInvalidValue;
  }
  // (see the producers: with row sums, an even number of stages for two of them)
  kp.producers = 2;
  if (kp.rowsum && stages % 2 != 0) {
    if (stages > 3) --stages;
    else kp.producers = 1;
  }
  kp.stages = stages;
  const int smem = stages * STAGE + e_bytes + FIXED;
  const int threads = 32 * (3 + epi_warps(BN, EPI) + (kp.rowsum ? SUM_WARPS : (kp.e_tma ? 1 : 0)));
  static std::atomic<uint64_t> devices;
  const cudaError_t allowed = allow_shared_memory(devices, reinterpret_cast<const void*>(&gemm_kernel<BN, EB, EPI, CG, RAGGED>), SMEM_LIMIT);
  if (allowed != cudaSuccess) return allowed;
  const int num_sms = sm_count();
  const long long slabs = static_cast<long long>(kp.k_per_split) * (kp.cplx ? 2 : 1) * EB / 128;
  const bool samples = kp.accumulate && ((kp.zlo_n > 1 && kp.d_zlo == 0) || (kp.zhi_n > 1 && kp.d_zhi == 0));
  const long long chained_slabs = samples ? CHAINED_SLABS_OF_SAMPLES : CHAINED_SLABS;
  // tile order (MAKANI_B200_TILE_ORDER=m|n forces one order for A/B timing)
  static const int forced_order = [] {
    const char* e = getenv("MAKANI_B200_TILE_ORDER");
    return (e && e[0] == 'm') ? 0 : ((e && e[0] == 'n') ? 1 : -1);
  }();
  kp.n_fast = forced_order >= 0 ? forced_order : (kp.m_tiles > kp.n_tiles ? 1 : 0);
  if (CG == 2) {
    const int most = max_pairs();
    long long clusters = kp.total_tiles < static_cast<uint32_t>(most) ? kp.total_tiles : most;
    if (clusters < 1) clusters = 1;
    if constexpr (EPI != 0 && EPI != 5) clusters = mixed_grid(clusters, kp, 2 * BM, BN);
    return launch_chained(gemm_kernel<BN, EB, EPI, CG, RAGGED>, dim3(static_cast<unsigned>(2 * clusters)), dim3(threads), smem, stream, 2,
                          kp.total_tiles * slabs <= chained_slabs * clusters, ma, mb,
                          me, md, mp, mdx, kp);
  }
  long long grid = kp.total_tiles < static_cast<uint32_t>(num_sms) ? kp.total_tiles : num_sms;
  if (grid < 1) grid = 1;
  if constexpr (EPI != 0 && EPI != 5) grid = mixed_grid(grid, kp, BM, BN);
  const bool alone = kp.total_tiles * slabs <= chained_slabs * grid && kp.nseg <= 1 && kp.ndx == 0 && kp.sync.nwait == 0 && kp.sync.nsig == 0 && kp.sync.done_ctr == nullptr;
  return launch_chained(gemm_kernel<BN, EB, EPI, CG, RAGGED>, dim3(static_cast<unsigned>(grid)), dim3(threads), smem, stream, 1, alone, ma, mb, me, md,
                        mp, mdx, kp);
}

}  // namespace

// Tensor map of an output or epilogue operand: [M rows][N contiguous] with two batch dimensions, 128-byte swizzle.  Rows
// may be split, r = hi * rd + lo with rd a power of two that divides M and 32: a box is then 32 (or 128) / rd by rd rows.
// With `halves` the second dimension is not part of the rows: two results `halves` elements apart (complex products).
static bool make_map_e(CUtensorMap* map, const void* ptr, int M, int N, int rd, long long rs_hi, long long rs_lo, long long zs_lo,
                       long long zs_hi, int zlo_n, int zhi_n, int box_rows = 128, int ob = 2, long long halves = 0) {
  EncodeTiledFn enc = get_encode();
  if (!enc) return false;
  const long long row_stride = rd > 1 ? rs_hi : rs_lo;
  cuuint64_t dims[5] = {static_cast<cuuint64_t>(N), static_cast<cuuint64_t>(rd), static_cast<cuuint64_t>(M / rd),
                        static_cast<cuuint64_t>(zlo_n), static_cast<cuuint64_t>(zhi_n)};
  cuuint64_t strides[4] = {static_cast<cuuint64_t>(rs_lo) * ob, static_cast<cuuint64_t>(row_stride) * ob,
                           static_cast<cuuint64_t>(zlo_n > 1 ? zs_lo : row_stride) * ob,
                           static_cast<cuuint64_t>(zhi_n > 1 ? zs_hi : row_stride) * ob};
  // one 128-byte swizzle row: 64 bf16 or 32 fp32
  cuuint32_t box[5] = {static_cast<cuuint32_t>(128 / ob), static_cast<cuuint32_t>(rd), static_cast<cuuint32_t>(box_rows / rd), 1, 1};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  if (halves > 0) {
    dims[1] = 2;
    strides[0] = static_cast<cuuint64_t>(halves) * ob;
  }
  if ((reinterpret_cast<uintptr_t>(ptr) & 15) || (strides[0] & 15) || (strides[1] & 15) || (strides[2] & 15) || (strides[3] & 15))
    return false;
  CUresult r = enc(map, ob == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 5, const_cast<void*>(ptr), dims,
                   strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

const char* gemm_last_error() { return g_err; }

namespace {
// Copies `rows` rows of `row_bytes` (multiple of 16) from local memory into the same place of up to 8 destination
// buffers (this device's and its peers'), with the producer handshake folded in: every block waits until all
// peers have consumed the previous contents, the last block to finish publishes the new generation.
__global__ void __launch_bounds__(256) peer_publish_kernel(const uint4* __restrict__ src, long long rows, int row_vec,
                                                           long long src_stride_vec, long long dst_stride_vec, int ndst,
                                                           const PeerSync sy, int* err) {
  struct Dst {
    uint4* p[MAX_SEG];
  };
  __shared__ int ok_s;
  if (threadIdx.x == 0) {
    bool ok = true;
    for (int w = 0; w < sy.nwait && ok; ++w) {
      const unsigned int need = *sy.wait_exp[w] + static_cast<unsigned int>(sy.wait_off[w]);
      for (int peer = 0; peer < sy.np_wait[w] && ok; ++peer) {
        uint64_t t0 = 0;
        for (uint32_t it = 0;; ++it) {
          if (static_cast<int>(ld_acquire_sys_u32(sy.wait[w] + peer) - need) >= 0) break;
          if ((it & 255u) == 255u) {
            const uint64_t now = global_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > WAIT_LIMIT_NS) {
              atomicExch(err, 40 + w);
              ok = false;
              break;
            }
          }
        }
      }
    }
    ok_s = ok ? 1 : 0;
  }
  __syncthreads();
  if (ok_s) {
    const long long total = rows * row_vec;
    for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
      const long long r = i / row_vec;
      const int c = static_cast<int>(i - r * row_vec);
      const uint4 v = src[r * src_stride_vec + c];
      for (int q = 0; q < ndst; ++q) reinterpret_cast<uint4*>(sy.sig[1][q])[r * dst_stride_vec + c] = v;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && sy.done_ctr != nullptr) {
    __threadfence_system();
    const unsigned int prev = atomicAdd(sy.done_ctr, 1u);
    if (prev == gridDim.x - 1) {
      *sy.done_ctr = 0;
      if (*reinterpret_cast<volatile int*>(err) == 0) {   // nothing is published after an expired wait
        for (int i = 0; i < sy.nwait; ++i)
          if (sy.bump[i]) atomicAdd(sy.bump[i], 1u);
        __threadfence_system();
        for (int peer = 0; peer < sy.np_sig[0]; ++peer)
          if (sy.sig[0][peer]) atomicAdd_system(sy.sig[0][peer], 1u);
      }
    }
  }
}

// out = sum over `nsrc` local segments (+ per-channel bias), 8 bf16 per thread step, with the consumer side of the
// handshake folded in: every block waits until all peers have delivered their segment, the last block to finish tells
// the peers that the buffer may be overwritten.  The second signal list carries the segment base pointers.
__global__ void __launch_bounds__(256) peer_sum_kernel(uint4* __restrict__ out, long long nvec, int nsrc,
                                                       const float* __restrict__ bias, int C, const PeerSync sy, int* err) {
  __shared__ int ok_s;
  if (threadIdx.x == 0) {
    bool ok = true;
    for (int w = 0; w < sy.nwait && ok; ++w) {
      const unsigned int need = *sy.wait_exp[w] + static_cast<unsigned int>(sy.wait_off[w]);
      for (int peer = 0; peer < sy.np_wait[w] && ok; ++peer) {
        uint64_t t0 = 0;
        for (uint32_t it = 0;; ++it) {
          if (static_cast<int>(ld_acquire_sys_u32(sy.wait[w] + peer) - need) >= 0) break;
          if ((it & 255u) == 255u) {
            const uint64_t now = global_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > WAIT_LIMIT_NS) {
              atomicExch(err, 44 + w);
              ok = false;
              break;
            }
          }
        }
      }
    }
    ok_s = ok ? 1 : 0;
  }
  __syncthreads();
  if (ok_s) {
    for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < nvec;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
      float acc[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = 0.f;
      if (bias) {
        const int c0 = static_cast<int>((i * 8) % C);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = __ldg(bias + c0 + j);
      }
      for (int q = 0; q < nsrc; ++q) {
        // L1 is bypassed: peers rewrite these buffers between launches
        const uint4 v = __ldcg(reinterpret_cast<const uint4*>(sy.sig[1][q]) + i);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = __bfloat1622float2(h[j]);
          acc[2 * j] += f.x;
          acc[2 * j + 1] += f.y;
        }
      }
      __nv_bfloat162 o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] = __floats2bfloat162_rn(acc[2 * j], acc[2 * j + 1]);
      out[i] = *reinterpret_cast<uint4*>(o);
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && sy.done_ctr != nullptr) {
    __threadfence_system();
    const unsigned int prev = atomicAdd(sy.done_ctr, 1u);
    if (prev == gridDim.x - 1) {
      *sy.done_ctr = 0;
      if (*reinterpret_cast<volatile int*>(err) == 0) {   // nothing is published after an expired wait
        for (int i = 0; i < sy.nwait; ++i)
          if (sy.bump[i]) atomicAdd(sy.bump[i], 1u);
        __threadfence_system();
        for (int peer = 0; peer < sy.np_sig[0]; ++peer)
          if (sy.sig[0][peer]) atomicAdd_system(sy.sig[0][peer], 1u);
      }
    }
  }
}

void fill_sync(PeerSync& sy, const GemmPeer* g) {
  memset(&sy, 0, sizeof(sy));
  if (!g) return;
  for (int i = 0; i < 2; ++i) {
    sy.np_wait[i] = g->np_wait[i];
    sy.np_sig[i] = g->np_sig[i];
  }
  sy.nwait = g->nwait;
  sy.nsig = g->nsig;
  for (int i = 0; i < 2; ++i) {
    sy.wait[i] = g->wait[i];
    sy.wait_exp[i] = g->wait_exp[i];
    sy.wait_off[i] = g->wait_off[i];
    sy.bump[i] = g->bump[i];
    for (int q = 0; q < MAX_SEG; ++q) sy.sig[i][q] = g->sig[i][q];
  }
  sy.done_ctr = g->done_ctr;
}
}  // namespace

cudaError_t peer_publish_launch(const void* src, long long rows, long long row_bytes, long long src_stride_bytes,
                                long long dst_stride_bytes, void* const* dsts, int ndst, const GemmPeer& g, int* err_flag,
                                cudaStream_t stream) {
  if (rows <= 0 || row_bytes <= 0) return cudaSuccess;
  if ((row_bytes & 15) || (src_stride_bytes & 15) || (dst_stride_bytes & 15) || (reinterpret_cast<uintptr_t>(src) & 15) ||
      ndst < 1 || ndst > MAX_SEG || g.nsig > 1)
    return cudaErrorInvalidValue;
  PeerSync sy;
  fill_sync(sy, &g);
  // the second signal list carries the destination base pointers (the protocol itself needs one list only)
  for (int q = 0; q < MAX_SEG; ++q) sy.sig[1][q] = q < ndst ? static_cast<unsigned int*>(dsts[q]) : nullptr;
  for (int q = 0; q < ndst; ++q)
    if (reinterpret_cast<uintptr_t>(dsts[q]) & 15) return cudaErrorInvalidValue;
  const long long total = rows * (row_bytes / 16);
  long long blocks = (total + 255) / 256;
  if (blocks > sm_count() * 4LL) blocks = sm_count() * 4LL;
  peer_publish_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(
      static_cast<const uint4*>(src), rows, static_cast<int>(row_bytes / 16), src_stride_bytes / 16, dst_stride_bytes / 16,
      ndst, sy, err_flag);
  return cudaGetLastError();
}

cudaError_t peer_sum_launch(void* out, long long n_elems, const void* const* srcs, int nsrc, const float* bias, int C,
                            const GemmPeer& g, int* err_flag, cudaStream_t stream) {
  if (n_elems <= 0) return cudaSuccess;
  if ((n_elems & 7) || nsrc < 1 || nsrc > MAX_SEG || g.nsig > 1 || (reinterpret_cast<uintptr_t>(out) & 15) ||
      (bias && (C <= 0 || (C & 7))))
    return cudaErrorInvalidValue;
  PeerSync sy;
  fill_sync(sy, &g);
  for (int q = 0; q < MAX_SEG; ++q) {
    if (q < nsrc && (reinterpret_cast<uintptr_t>(srcs[q]) & 15)) return cudaErrorInvalidValue;
    sy.sig[1][q] = q < nsrc ? static_cast<unsigned int*>(const_cast<void*>(srcs[q])) : nullptr;
  }
  const long long nvec = n_elems / 8;
  long long blocks = (nvec + 255) / 256;
  if (blocks > sm_count() * 4LL) blocks = sm_count() * 4LL;
  peer_sum_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(static_cast<uint4*>(out), nvec, nsrc, bias, C, sy, err_flag);
  return cudaGetLastError();
}

namespace {
FastDiv make_div(int d) {
  FastDiv f;
  f.d = static_cast<uint32_t>(d);
  f.shift = 0;
  while ((1ull << f.shift) < f.d) ++f.shift;
  f.mul = static_cast<uint32_t>(((((1ull << f.shift) - f.d) << 32) / f.d) + 1);
  return f;
}

// Tile width: the fewest padded columns, a tile costing some 32 columns of its own, 64 in the plain store, which waits for the
// activations (every tile of a row fetches them once more) rather than for its epilogue.  Measured, us in 256 / 192 / 128 columns:
//   plain, 115200 rows, K = 384: 384 outputs 44 / 43 / -; 520: 59 / 58 / -; 640: 63 / 68 / 69; 776: 82 / 85 / 93;
//   K = 96: 384: 32 / 28 / -; 640: 42 / 50 / 49;  16200 rows, K = 768: 384: 16 / 14 / -; 640: 20 / 22 / 23
//   GELU with two outputs, 115200 rows, K = 96: 384: 59 / 48 / -; 640: 78 / - / 84; 776: 145 / 108 / -
//   fp32 gradients of 320 rows over 115200 tokens: 384: 47 / 38 / 39; 640: 63 / 60 / 59; 776: 89 / 86 / 88
//   times an operand (no 256): K = 96, 384: - / 39 / 41; 576: - / 54 / 61;  K = 384, 384: - / 54 / 50; 576: - / 70 / 74
int pick_bn(int N, int epi, int e_tma) {
  if (epi == 0 && e_tma) return 128;
  int best = 128;
  long long cost = -1;
  const int widths[3] = {256, 192, 128}, own = epi == 1 ? 64 : 32;
  for (int i = (epi == 3 || epi == 4 ? 1 : 0); i < 3; ++i) {
    const long long c = static_cast<long long>((N + widths[i] - 1) / widths[i]) * (widths[i] + own);
    if (cost < 0 || c < cost) {
      cost = c;
      best = widths[i];
    }
  }
  return best;
}

// Split-k factor of an accumulating launch: whole waves of `slots` CTAs (or pairs), every split costing its tile one
// epilogue of atomics, worth some 16 k-blocks, and no fewer partial sums than `least`.
//
// `least` is twice the SMs over the 128 x 256 tiles.  The tensor core truncates its running sum at every 16 products, so that an
// accumulation over k of them is off by up to k / 16 * 2^-23 (one-signed operands; zero-mean ones a fifth of it).  By time alone a
// 384 x 768 gradient over 721 x 1440 tokens ran in 16 chains with an error of 7.5e-5 against 64 bits (one-signed 3.9e-4); 49 chains,
// again whole waves, give 2.4e-5 (1.1e-4) in 576 us, 16 took 573.  Twice the tiles without whole waves: 33 chains, 3.6e-5, 757 us.
int pick_splits(long long base, int kblocks, int slots, int least) {
  int best = least < kblocks ? least : (kblocks > 0 ? kblocks : 1);
  double cost = 1e300;
  const long long most = least + 4ll * slots / (base > 0 ? base : 1);
  for (int s = best; s <= most && s <= kblocks; ++s) {
    const double waves = static_cast<double>((base * s + slots - 1) / slots);
    const double c = waves * ((kblocks + s - 1) / s + 16.0);
    if (c < cost * 0.999) {
      cost = c;
      best = s;
    }
  }
  return best;
}
}  // namespace

int gemm_plain_columns(int n) { return pick_bn(n, 1, 0); }

cudaError_t gemm_launch(const GemmProblem& p, const GemmOperand& A, const GemmOperand& B, const GemmEpilogue& e,
                        int* err_flag, cudaStream_t stream, const GemmPeer* peer, GemmRowSums* rows) {
  g_err[0] = 0;
  if (rows) rows->done = 0;
  if (p.M <= 0 || p.N <= 0 || p.zlo_n <= 0 || p.zhi_n <= 0) return cudaSuccess;
  bind_context(stream);
  const int eb = p.elem_bytes;
  if (eb != 2 && eb != 4) {
    snprintf(g_err, sizeof(g_err), "elem_bytes must be 2 or 4");
    return cudaErrorInvalidValue;
  }
  int bn = p.bn;
  if (bn != 0 && bn != 128 && bn != 192 && bn != 256) {
    snprintf(g_err, sizeof(g_err), "bn must be 128, 192 or 256");
    return cudaErrorInvalidValue;
  }
  if (eb == 4 && (A.mn_major || B.mn_major)) {
    snprintf(g_err, sizeof(g_err), "tf32 operands must be k-major (row-contiguous tf32 operands are not supported)");
    return cudaErrorInvalidValue;
  }
  if (p.splits > 1 && !e.accumulate) {
    snprintf(g_err, sizeof(g_err), "split-k needs accumulate");
    return cudaErrorInvalidValue;
  }
  if (e.accumulate && (!e.out_f32 || e.resid || e.preact)) {
    snprintf(g_err, sizeof(g_err), "accumulate needs fp32 output without residual/preact");
    return cudaErrorInvalidValue;
  }
  const int bk = 128 / eb;
  KParams kp;
  memset(&kp, 0, sizeof(kp));
  kp.M = p.M; kp.N = p.N; kp.K = p.K;
  kp.zlo_n = p.zlo_n; kp.zhi_n = p.zhi_n;
  kp.splits = p.splits < 1 ? 1 : p.splits;
  const int kblocks = (p.K + bk - 1) / bk;
  kp.a_mn = A.mn_major; kp.b_mn = B.mn_major;
  kp.a_zlo = (A.zs_lo != 0 && p.zlo_n > 1); kp.a_zhi = (A.zs_hi != 0 && p.zhi_n > 1);
  kp.b_zlo = (B.zs_lo != 0 && p.zlo_n > 1); kp.b_zhi = (B.zs_hi != 0 && p.zhi_n > 1);
  kp.rmin_a = p.rmin_a; kp.rmin_b = p.rmin_b; kp.rmax_a = p.rmax_a; kp.rmax_b = p.rmax_b;
  kp.kmin_a = p.kmin_a; kp.kmin_b = p.kmin_b; kp.kmax_a = p.kmax_a; kp.kmax_b = p.kmax_b;
  kp.d_zlo = e.d_zlo; kp.d_zhi = e.d_zhi;
  kp.rdiv = e.rdiv > 0 ? e.rdiv : 1 << 30; kp.rs_hi = e.rs_hi; kp.rs_lo = e.rs_lo;
  kp.ndiv = e.ndiv > 0 ? e.ndiv : 1 << 30; kp.ns_hi = e.ns_hi;
  kp.alpha = e.alpha; kp.bias = e.bias; kp.bias_zs = e.bias ? e.bias_zs : 0; kp.bias_mode = e.bias ? e.bias_mode : 0; kp.act = e.act; kp.save_deriv = (e.save_deriv && e.act == 1 && e.preact) ? 1 : 0; kp.gelu = gelu_coef(gelu_tanh()); kp.act_param = e.act_param;
  kp.resid = e.resid; kp.preact = e.preact; kp.D = e.D;
  kp.out_f32 = e.out_f32; kp.accumulate = e.accumulate;
  // 16-byte vector accesses need every stride (and the bases) aligned
  const int va = e.out_f32 ? 4 : 8;
  auto al = [&](long long s) { return (s % va) == 0; };
  const uintptr_t amask = 15;
  bool vec = al(e.d_zlo) && al(e.d_zhi) && al(e.rs_hi) && al(e.rs_lo) && al(e.ns_hi) && (kp.ndiv % 8 == 0) &&
             ((reinterpret_cast<uintptr_t>(e.D) & amask) == 0);
  if (e.resid) vec = vec && ((reinterpret_cast<uintptr_t>(e.resid) & amask) == 0);
  if (e.preact) vec = vec && ((reinterpret_cast<uintptr_t>(e.preact) & amask) == 0);
  kp.vec_ok = vec ? 1 : 0;
  kp.err = err_flag;
  kp.nseg = 1;
  kp.ndx = 0;
  fill_sync(kp.sync, peer);
  if (peer && peer->ndx > 0) {
    if (peer->ndx > MAX_SEG - 1 || e.out_f32 || e.accumulate || kp.splits != 1 || e.preact) {
      snprintf(g_err, sizeof(g_err), "replicated output: bf16 plain stores only, at most %d extra destinations", MAX_SEG - 1);
      return cudaErrorInvalidValue;
    }
    kp.ndx = peer->ndx;
    for (int q = 0; q < peer->ndx; ++q) kp.Dx[q] = peer->Dx[q];
  }
  if (peer && peer->nseg > 1) {
    if (kp.splits != 1 || peer->nseg > MAX_SEG) {
      snprintf(g_err, sizeof(g_err), "multi-device operand: split-k not supported, at most %d segments", MAX_SEG);
      return cudaErrorInvalidValue;
    }
    kp.nseg = peer->nseg;
    for (int q = 0; q < peer->nseg; ++q) {
      kp.seg_len[q] = peer->seg_len[q];
      kp.seg_apos[q] = peer->seg_apos[q];
      kp.seg_gstart[q] = peer->seg_gstart[q];
    }
  }

  CUtensorMap ma, mb, me;
  memset(&me, 0, sizeof(me));
  // Epilogue operand through TMA when it is bf16 and the destination layout is a plain row-major matrix batch.
  kp.e_tma = 0;
  // Rows split by a power of two (the (mode, re / im) rows of the DFT stages) are one more dimension of the tensor map: the AFNO
  // stages at 90 x 180 tokens take 14 - 21 us each, 22 - 44 us through the generic epilogue.
  const bool one_stride = e.rdiv <= 0 || e.rdiv >= (1 << 30);
  // (rdiv = 1 puts every row at rs_hi: the map's row stride would be rs_lo)
  const bool split_ok = !one_stride && e.rdiv > 1 && e.rdiv <= 32 && (e.rdiv & (e.rdiv - 1)) == 0 && p.M % e.rdiv == 0 && e.rs_hi > 0 &&
                        e.rs_lo > 0;
  const bool plain = (one_stride || split_ok) && (e.ndiv <= 0 || e.ndiv >= (1 << 30));
  const int rd = one_stride ? 1 : e.rdiv;
  const bool folded = p.cplx == 4 || p.cplx == 5;
  auto tile_map = [&](CUtensorMap* m, const void* ptr, int box_rows, int rows_of, int cols_of) {
    return make_map_e(m, ptr, rows_of, cols_of, rd, e.rs_hi, e.rs_lo, e.d_zlo, e.d_zhi, p.zlo_n, p.zhi_n, box_rows, 2, e.d_half);
  };
  kp.rd_shift = 0;
  while (plain && (1 << kp.rd_shift) < rd) ++kp.rd_shift;
  if (e.resid && !e.out_f32 && plain && kp.vec_ok && e.d_zlo >= 0 && e.d_zhi >= 0) {
    if (tile_map(&me, e.resid, BM, p.M, p.N)) kp.e_tma = 1;
  }
  // A specialised epilogue (TMA stores of bf16 tiles) when the launch fits one.
  int epi = 0;
  CUtensorMap md, mp;
  DMaps mdx;
  memset(&md, 0, sizeof(md));
  memset(&mp, 0, sizeof(mp));
  memset(&mdx, 0, sizeof(mdx));
  kp.n_full = p.N / 8 * 8;
  const bool columns_ok = kp.n_full == p.N || p.cplx != 0 || (kp.n_full > 0 && kp.ndx == 0);
  if (eb == 2 && !e.out_f32 && kp.vec_ok && !e.accumulate && plain && e.d_zlo >= 0 && e.d_zhi >= 0 && columns_ok &&
      (kp.bias_mode != 2 || ((reinterpret_cast<uintptr_t>(e.bias) & 15) == 0 && (kp.bias_zs % 4) == 0))) {
    if (folded) epi = !e.resid && !e.preact && e.act == 0 && !e.bias && e.alpha == 1.f && kp.ndx == 0 ? 6 : 0;
    else if (!e.resid && !e.preact && (e.act == 0 || e.act == 1 || e.act == 3 || e.act == 5)) epi = 1;
    else if (!e.resid && e.preact && e.act == 1) epi = 2;
    else if (e.resid && kp.e_tma && !e.preact && e.act == 0) epi = 3;
    else if (e.resid && kp.e_tma && !e.preact && (e.act == 2 || e.act == 4 || e.act == 6 || e.act == 8)) epi = 4;
    if (epi != 0) {
      const int cols = p.cplx ? p.N : kp.n_full;
      bool ok = tile_map(&md, e.D, 32, p.M, cols);
      if (ok && epi == 2) ok = tile_map(&mp, e.preact, 32, p.M, cols);
      if (ok && epi == 6) ok = tile_map(&mp, e.D, 32, p.rows, cols);      // the mirror rows
      if (ok && kp.ndx > 0) {
        if (epi != 1) ok = false;   // replicated output goes through the plain-store epilogue or the generic one
        for (int q = 0; ok && q < kp.ndx; ++q)
          ok = tile_map(&mdx.m[q], kp.Dx[q], 32, p.M, cols);
      }
      if (!ok) epi = 0;
    }
  }
  // fp32 results with nothing but a scale: a dimension whose batches all add into one output is left out of the map
  // (a partial last vector may be added to, what lies behind it by zero, but not stored)
  if (eb == 2 && e.out_f32 && kp.vec_ok && plain && !e.resid && !e.preact && e.act == 0 && kp.bias_mode == 0 && kp.ndx == 0 &&
      (e.accumulate || p.N % 4 == 0) &&
      e.d_zlo >= 0 && e.d_zhi >= 0 && (e.accumulate || ((e.d_zlo > 0 || p.zlo_n == 1) && (e.d_zhi > 0 || p.zhi_n == 1)))) {
    kp.d_zlo_on = e.d_zlo > 0;
    kp.d_zhi_on = e.d_zhi > 0;
    if (make_map_e(&md, e.D, p.M, p.N, rd, e.rs_hi, e.rs_lo, e.d_zlo, e.d_zhi, kp.d_zlo_on ? p.zlo_n : 1, kp.d_zhi_on ? p.zhi_n : 1, 32, 4,
                   e.d_half))
      epi = 5;
  }
  // CTA pairs (256-row tiles, each CTA loads half of the B tile): single-device bf16 launches with at least two row blocks and no
  // row-triangular structure, unless one pair covers all rows: the half that single CTAs would skip for half of the batches costs
  // less than their loads (Legendre analysis of 240 degrees, 241 orders, 384 channels, 240 latitudes 53 -> 46 us, 721 latitudes 102 -> 88; 256
  // channels and 180 degrees the same).  MAKANI_B200_CTA_PAIRS=0 / 1 forces none / all eligible launches.  Measured, time on
  // single CTAs over time on pairs (plain store, product with an operand, GELU with two outputs):
  //   K = 768, 115200 rows: 1.07 - 1.30.  From K = 512 on the long k loop pays for the pair's longer start.
  //   K = 256 - 448: 1024 - 8192 rows 0.89 - 0.96 (768 outputs at 8192 rows 0.91 - 1.09); 16200 rows, 384 outputs 0.92 - 0.99, 768
  //   outputs 0.98 - 1.13; 115200 rows, 384 and 768 outputs 1.03 - 1.23.  A pair has half as many tiles in flight: it pays from
  //   two waves of tiles on.
  //   K = 200, 232, 504 (rows of no whole 64 bytes: loads touch one more sector, and a pair loads half of B): 1024 - 8192 rows
  //   0.95 - 1.06 (504, 768 outputs: 1.11 - 1.23), 16200 rows 1.01 - 1.16, 32768 rows 1.03 - 1.19.
  //   K < 200, 65536 rows and more: 16, 80, 136, 184: 1.02 - 1.50; 64, 96, 128, 160, 192: 0.92 - 1.15, but for 384 outputs times an
  //   operand over 518400 rows at 160 and 192 (0.81 - 0.88).
  // Outputs whose rows pairs would pad stay on single CTAs (384 of 512 rows of a weight gradient: 327 us on pairs, 290 us).
  static const int pairs_mode = [] {
    const char* e = getenv("MAKANI_B200_CTA_PAIRS");
    return (e && e[0] == '0') ? 0 : ((e && e[0] == '1') ? 1 : 2);
  }();
  const bool no_peer = (peer == nullptr) || (peer->nseg <= 1 && peer->ndx == 0 && peer->nwait == 0 && peer->nsig == 0 &&
                                              peer->done_ctr == nullptr);
  const bool ragged = epi >= 1 && epi <= 4 && kp.n_full != p.N && p.cplx == 0;
  const bool triangle = (p.rmin_a != 0 || p.rmax_a != 0) && (p.cplx != 0 || p.M > 2 * BM);
  const bool eligible = eb == 2 && no_peer && !ragged && p.M > BM && !triangle && (p.cplx == 0 || p.cplx >= 3);
  const int pad1 = (p.M + BM - 1) / BM * BM, pad2 = (p.M + 2 * BM - 1) / (2 * BM) * (2 * BM);
  const long long z_all = static_cast<long long>(p.zlo_n) * p.zhi_n;
  const bool waves = pad1 / BM * ((p.N + 255) / 256) * z_all >= 2 * sm_count();
  const bool pays = (p.K >= 512 || p.M >= 65536 || (p.K >= 200 && (waves || p.K % 32 != 0))) && pad2 * 8 <= pad1 * 9;
  const int cg = (eligible && (pairs_mode == 1 || (pairs_mode == 2 && pays))) ? 2 : 1;
  if (bn == 0) bn = pick_bn(p.N, epi, kp.e_tma);
  if ((eb == 4 && bn == 192) || ((epi == 3 || epi == 4 || kp.e_tma) && bn == 256)) bn = 128;
  if ((epi == 0 && kp.e_tma) || epi == 6 || ragged) bn = 128;
  kp.m_tiles = (p.M + BM * cg - 1) / (BM * cg);
  kp.n_tiles = (p.N + bn - 1) / bn;
  kp.cplx = p.cplx;
  kp.nth = kp.n_tiles;
  kp.neg_half = p.cplx == 1 ? 0 : 1;
  kp.neg_seg = p.cplx == 2 ? 0 : 1;
  kp.a_part = p.K;
  if (folded) {
    // (from 64 rows on the mirror rows' boxes start at or after row 0, and the last box of sums ends inside the table; the computed
    // rows and their mirrors make up all rows, or some would stay unwritten)
    if (epi != 6 || kp.splits != 1 || p.splits == 0 || kp.nseg != 1 || rd != 1 || A.mn_major || p.mirror < 64 || (p.a_plane % 8) != 0 ||
        (p.N % 8) != 0 ||
        p.M != (p.cplx == 5 ? 2 * (p.mirror / 4 + 1) : p.mirror / 2 + 1) || p.rows < p.mirror / 2 + 32 ||
        p.rows > p.mirror + (p.cplx == 5 ? 2 : 0) || p.zlo_n != 1) {
      snprintf(g_err, sizeof(g_err), "folded product: bf16, K-major tables, plain aligned rows, at least 64 of them, each computed or a mirror");
      return cudaErrorInvalidValue;
    }
    kp.a_part = static_cast<int>(p.a_plane);
    kp.mirror = p.mirror;
    kp.fold_rows = p.rows;
  } else if (p.cplx) {
    if (eb != 2 || (epi != 1 && epi != 3 && epi != 5) || kp.splits != 1 || p.splits == 0 || kp.nseg != 1 || rd != 1) {
      snprintf(g_err, sizeof(g_err), "complex product: bf16 operands, plain rows, aligned output with or without residual");
      return cudaErrorInvalidValue;
    }
    // the second part of a K-major A starts at k = K, a coordinate of the contiguous dimension: a whole number of 16-byte vectors
    if (p.cplx != 3 && !A.mn_major && (p.K % (16 / eb)) != 0) {
      snprintf(g_err, sizeof(g_err), "complex product: the parts of A must be multiples of %d elements", 16 / eb);
      return cudaErrorInvalidValue;
    }
    kp.n_tiles *= 2;
  }
  const int slots = cg == 2 ? max_pairs() : sm_count();
  // (a bias or an activation is applied once per partial sum, and a segmented k axis is walked by one CTA: one split there)
  const bool choose = p.splits == 0 && e.accumulate && kp.bias_mode == 0 && e.act == 0 && kp.nseg == 1;
  const long long base_tiles = static_cast<long long>(kp.m_tiles) * kp.n_tiles * p.zlo_n * p.zhi_n;
  if (choose) {
    const long long wide = static_cast<long long>((p.M + BM - 1) / BM) * ((p.N + 255) / 256) * p.zlo_n * p.zhi_n;
    kp.splits = pick_splits(base_tiles, kblocks, slots, static_cast<int>((2 * sm_count() + wide - 1) / wide));
  }
  kp.k_per_split = ((kblocks + kp.splits - 1) / kp.splits) * bk;
  if (kp.k_per_split < bk) kp.k_per_split = bk;
  if (base_tiles * kp.splits >= (1ll << 31)) {
    snprintf(g_err, sizeof(g_err), "too many tiles");
    return cudaErrorInvalidValue;
  }
  kp.total_tiles = static_cast<uint32_t>(base_tiles * kp.splits);
  // Sums of the rows of A: only where the launch has A's tokens in shared memory as rows, all of them and each once, and where adding up
  // the partial sums stays short.  Every batch, split and column tile leaves four of them per row; gradient and sums beside it over
  // gradient and a pass of its own, by partial sums: 258 0.75, 512 0.70, 2048 0.73, 3072 0.90, 4096 1.03, 11648 1.06, 12288 0.96 - 1.09,
  // 32768 1.65, 262144 2.1 - 2.5 (67 MB of them for 64 rows).
  if (rows && epi == 5 && A.mn_major && p.cplx == 0 && kp.nseg == 1 && p.rmin_a == 0 && p.rmin_b <= 0 && p.rmax_a == 0 && p.rmax_b >= p.M &&
      p.kmin_a == 0 && p.kmin_b <= 0 && p.kmax_a == 0 && p.kmax_b >= p.K && (p.zlo_n == 1 || A.zs_lo != 0) && (p.zhi_n == 1 || A.zs_hi != 0) &&
      (p.zhi_n == 1 || e.d_zhi == 0)) {
    kp.rs_groups = p.zlo_n > 1 && e.d_zlo != 0 ? p.zlo_n : 1;
    const long long slabs = z_all / kp.rs_groups * kp.splits * kp.n_tiles * 4;
    if (slabs <= 4096 && kp.rs_groups < 65536) {
      kp.rs_slabs = static_cast<int>(slabs);
      kp.rowsum = rows->scratch(rows->ctx, slabs * kp.rs_groups * p.M);      // (null: no memory for them, the caller's pass needs less)
    }
  }
  kp.dv_n = make_div(kp.n_tiles);
  kp.dv_m = make_div(kp.m_tiles);
  kp.dv_split = make_div(kp.splits);
  kp.dv_zlo = make_div(p.zlo_n);
  // planes take the place of the lower batch index
  GemmOperand Am = A, Bm = B;
  if (p.cplx) Bm.zs_lo = p.b_plane;
  if (p.cplx == 3) Am.zs_lo = p.a_plane;
  const int ka = folded ? kp.a_part + p.K : (p.cplx && p.cplx != 3 ? 2 * p.K : p.K);
  if (!make_map(&ma, Am, ka, eb, p.cplx == 3 ? 2 : p.zlo_n, p.zhi_n, BM)) return cudaErrorInvalidValue;
  const int bn_box = bn / cg;     // rows of a K-major B one CTA loads per stage
  BMaps mbs;
  if (kp.nseg > 1) {
    for (int q = 0; q < kp.nseg; ++q) {
      GemmOperand Bq = B;
      Bq.ptr = peer->seg_ptr[q];
      if (!make_map(&mbs.m[q], Bq, peer->seg_len[q], eb, p.zlo_n, p.zhi_n, bn_box)) return cudaErrorInvalidValue;
    }
    for (int q = kp.nseg; q < MAX_SEG; ++q) mbs.m[q] = mbs.m[0];
  } else {
    if (!make_map(&mb, Bm, p.K, eb, p.cplx ? 2 : p.zlo_n, p.zhi_n, bn_box)) return cudaErrorInvalidValue;
    for (int q = 0; q < MAX_SEG; ++q) mbs.m[q] = mb;
  }
  if (!kp.e_tma) me = ma;   // unused, but must be a valid descriptor

  if (epi == 0) md = ma;       // unused maps must be valid descriptors all the same
  if (epi != 2 && epi != 6) mp = ma;
  for (int q = (epi == 1 ? kp.ndx : 0); q < MAX_SEG - 1; ++q) mdx.m[q] = ma;
  if (epi == 6)
    return cg == 2 ? launch_t<128, 2, 6, 2>(ma, mbs, me, md, mp, mdx, kp, stream) : launch_t<128, 2, 6, 1>(ma, mbs, me, md, mp, mdx, kp, stream);
  if (eb == 4) {
    if (bn == 256) return launch_t<256, 4, 0, 1>(ma, mbs, me, md, mp, mdx, kp, stream);
    return launch_t<128, 4, 0, 1>(ma, mbs, me, md, mp, mdx, kp, stream);
  }
  // (epilogues with an operand in shared memory: at most 192 columns, see above)
#define MK_DISPATCH(EPI_)                                                                              \
  if constexpr (EPI_ >= 1 && EPI_ <= 4) {                                                              \
    if (ragged) return launch_t<128, 2, EPI_, 1, true>(ma, mbs, me, md, mp, mdx, kp, stream);          \
  }                                                                                                    \
  if constexpr (EPI_ != 3 && EPI_ != 4) {                                                              \
    if (bn == 256 && cg == 2) return launch_t<256, 2, EPI_, 2>(ma, mbs, me, md, mp, mdx, kp, stream);  \
    if (bn == 256) return launch_t<256, 2, EPI_, 1>(ma, mbs, me, md, mp, mdx, kp, stream);             \
  }                                                                                                    \
  if (cg == 2) {                                                                                       \
    if (bn == 192) return launch_t<192, 2, EPI_, 2>(ma, mbs, me, md, mp, mdx, kp, stream);             \
    return launch_t<128, 2, EPI_, 2>(ma, mbs, me, md, mp, mdx, kp, stream);                            \
  }                                                                                                    \
  if (bn == 192) return launch_t<192, 2, EPI_, 1>(ma, mbs, me, md, mp, mdx, kp, stream);               \
  return launch_t<128, 2, EPI_, 1>(ma, mbs, me, md, mp, mdx, kp, stream);
  auto run = [&]() -> cudaError_t {
    switch (epi) {
      case 1: { MK_DISPATCH(1) }
      case 2: { MK_DISPATCH(2) }
      case 3: { MK_DISPATCH(3) }
      case 4: { MK_DISPATCH(4) }
      case 5: { MK_DISPATCH(5) }
      default: { MK_DISPATCH(0) }
    }
  };
  const cudaError_t launched = run();
  if (launched != cudaSuccess || !kp.rowsum) return launched;
  rows->done = 1;
  rows->slabs = {kp.rowsum, rows->out, kp.rs_slabs, p.M, kp.rs_groups};
  return rows->later ? cudaSuccess : colsum_add_slabs(rows->slabs, stream);
#undef MK_DISPATCH
}

}  // namespace mk
