// Launch geometry of the channels-last instance norm (fused_ops.cu): plain host code, one place for what the launcher asks for and the kernels
// address, so that it can be checked for all sizes without a GPU.
#pragma once
#include <algorithm>

#ifdef __CUDACC__
#define MK_HOST_DEVICE __host__ __device__
#else
#define MK_HOST_DEVICE
#endif

namespace mk {

// The four kernels: channels of a thread, most threads that work on rows (whole rows of them are used, one more warp loads), rows per thread in
// a stage of the ring and stages.  One CTA per SM.  721 x 1440 x 384 with GELU, each launch by itself with L2 flushed, us, by (rows, stages): forward
// sums (1, 8) 147, (2, 5) 139; forward output (1, 8) 274, (2, 5) 285, (2, 3) 258; gradient (1, 8) 428, (2, 4) 387, (4, 2) 367, by four channels
// and 992 threads (4, 3) 389.  The backward sums (303) wait for the fp32 pipe and the issue slots, not for rows: whole stages have no test per row,
// and four channels of a thread are as fast as eight here, 51 us instead of 61 at 240 x 480.
// START: stages that take as long as the start and the end of a CTA.  NARROW: most threads where a row is 64 bytes at most.
struct ClForwardSums { static constexpr int CH = 8, THREADS = 992, LAPS = 2, DEPTH = 5, TENSORS = 1, START = 8, NARROW = 480; };
struct ClForwardApply { static constexpr int CH = 8, THREADS = 992, LAPS = 2, DEPTH = 3, TENSORS = 1, START = 4, NARROW = 480; };
struct ClBackwardSums { static constexpr int CH = 4, THREADS = 992, LAPS = 4, DEPTH = 3, TENSORS = 2, START = 3, NARROW = 480; };
struct ClBackwardApply { static constexpr int CH = 8, THREADS = 608, LAPS = 4, DEPTH = 2, TENSORS = 2, START = 4, NARROW = 608; };

constexpr int CL_CHANNELS = 1024;     // most channels
constexpr int CL_BARRIERS = 128;      // bytes in front of all else
// Bytes of which an SM has no second share, for CTAs of up to 512 threads (of more, two find no registers).  Where a launch of one CTA per SM begins while the
// launch before it ends, these would crowd on the SMs that are free first.  Forward with GELU behind a product, us, without / with: 384 channels, 2048
// tokens 24.3 / 20.9; 256, 4 images of 1024 24.2 / 19.7; 64, 4 of 4096 16.7 / 15.3; 64, 512 tokens 12.6 / 13.0.
constexpr int CL_ALONE = 116 * 1024;
constexpr int CL_FEWEST = 128;        // threads (2048 x 16, both passes: 28 us, from CTAs of full size 40, with rows in registers 34)

// Shared memory: barriers, the merged sums of one image ([C][2] fp32, where the statistics cross devices), the ring.  The ring comes last: what
// stands in front of it does not depend on the rows of threads.
MK_HOST_DEVICE constexpr int cl_ring_offset(int C, bool merged) { return CL_BARRIERS + (merged ? 8 * C : 0); }
template <typename P>
MK_HOST_DEVICE constexpr int cl_ring_bytes(int threads) { return P::DEPTH * P::LAPS * P::TENSORS * 2 * P::CH * threads; }
// the partial sums of all rows of threads (16 bytes for two channels) take the ring's place
template <typename P>
MK_HOST_DEVICE constexpr bool cl_sums_fit() { return P::DEPTH * P::LAPS * P::TENSORS * 2 >= 8; }

// most bytes of a launch
template <typename P>
constexpr int cl_most_bytes() { return std::max(CL_ALONE, cl_ring_offset(CL_CHANNELS, true) + cl_ring_bytes<P>(P::THREADS)); }

// Rows of threads (R: the kernels are told, they cannot derive it from a block of whole warps), threads of a CTA, CTAs per image, bytes of
// shared memory
struct ClGeometry {
  int rows, threads, ctas, bytes;
};
// CTAs of an image.  One CTA per SM; all of them at once, and no more than there are stages, unless that leaves SMs idle (75 images, or
// 149): further waves of smaller shares are taken where stages and starts together come out a tenth shorter.
template <typename P>
int cl_ctas(long long stages, int B, int sms) {
  const int most = std::max(1, sms / B);
  int best = static_cast<int>(std::min<long long>(most, stages));
  if (10ll * most * B >= 9ll * sms && B <= sms) return best;
  auto cost = [&](long long n) { return (B * n + sms - 1) / sms * ((stages + n - 1) / n + P::START); };
  long long least = cost(best) * 9 / 10;
  for (int n = best + 1; n <= std::min<long long>(stages, most + 16); ++n)
    if (cost(n) < least) {
      best = n;
      least = cost(n);
    }
  return best;
}
// Small fields spread over the SMs by smaller CTAs.  With more images than SMs CTAs have half the size, so that one begins while the other ends.  Both
// passes with GELU, us, one CTA of full size per image or more while they fit at once / now: 90 x 180 x 384, 75 images 2058 / 1378;
// 149 4301 / 2523; 32 x 64 x 64, 149 images 137 / 123, 300 205 / 185; 50 images of 90 x 180 x 384 1077 / 934.
// Up to 32 channels over up to eight stages a CTA, smaller CTAs as well: one stage of a thousand rows keeps the CTA waiting for all of it, and its sums
// are as many.  Forward with GELU, us, before the ring / full size / here: 8 channels, 12 images of 24840 12.3 / 13.6 / 11.1; 259200 tokens
// 10.2 / 11.8 / 9.9; 16 channels, 2 of 76752 12.1 / 13.6 / 10.8; 32 channels, 4 of 16000 10.3 / 11.0 / 9.4; but 32 channels over 1038240 tokens
// 36.7 at full size, 38.4 smaller.
template <typename P>
ClGeometry cl_geometry(int C, long long T, int B, int sms, bool merged, bool chained) {
  const int V = C / P::CH;
  const long long most = std::max(1, sms / B);
  const long long share = (T + P::LAPS * most - 1) / (P::LAPS * most);      // rows of threads that would give every CTA one stage
  const bool narrow = C <= 32 && T <= 8 * most * (P::THREADS / V * P::LAPS);
  const int threads = B > sms ? (P::THREADS + 32) / 2 - 32 : narrow ? P::NARROW : P::THREADS;
  const int R = static_cast<int>(std::min<long long>(threads / V, std::max<long long>(share, (CL_FEWEST + V - 1) / V)));
  const long long stages = (T + P::LAPS * R - 1) / (P::LAPS * R);
  const int block = (V * R + 31) / 32 * 32 + 32, ctas = cl_ctas<P>(stages, B, sms), bytes = cl_ring_offset(C, merged) + cl_ring_bytes<P>(V * R);
  const bool alone = chained && block <= 512 && static_cast<long long>(ctas) * B <= sms;
  return {R, block, ctas, alone ? std::max(bytes, CL_ALONE) : bytes};
}

}  // namespace mk
