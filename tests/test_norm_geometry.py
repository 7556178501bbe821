"""Launch geometry of the channels-last instance norm (csrc/norm_ring.h), without a GPU: every byte that the kernels address lies in the shared
memory that their launch asks for, over all channel counts, field sizes and batches, alone and with statistics that cross devices; and the CTAs of a launch share its work out evenly."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "makani_b200", "csrc")

# The kernels' addressing, written out: stage s holds LAPS * R rows of one tensor, then those of the other; thread (v, r), v < V, r < R, reads its
# channels of the rows r, r + R, ...; sums of a pair of channels (8 bytes) of row r of threads sit R * C of them behind the ring's start at most.
PROGRAM = r"""
#include <cstdio>
#include "norm_ring.h"
using namespace mk;
static long long checked = 0, failed = 0;
template <typename P>
void check(const char* name, int C, long long T, int B, int sms, bool merged, bool sums, bool chained) {
  const ClGeometry g = cl_geometry<P>(C, T, B, sms, merged, chained);
  const long long V = C / P::CH, R = g.rows, rows = P::LAPS * R, row = 2ll * C;
  const long long ring = 128 + (merged ? 8ll * C : 0), stages = (T + rows - 1) / rows;
  long long end = ring;
  for (int s = 0; s < P::DEPTH; ++s)
    for (int t = 0; t < P::TENSORS; ++t) {
      const long long at = ring + (s * P::TENSORS + t) * rows * row;
      end = std::max(end, at + ((P::LAPS - 1) * R + R - 1) * row + (V - 1) * 2 * P::CH + 2 * P::CH);
    }
  if (sums) end = std::max(end, ring + 8 * ((R - 1) * C + C));
  const bool ok = R >= 1 && V * R <= g.threads - 32 && g.threads <= P::THREADS + 32 && g.threads % 32 == 0 && end <= g.bytes && g.bytes <= 232448 &&
                  ring % 16 == 0 && g.bytes <= cl_most_bytes<P>() && g.ctas >= 1 && g.ctas <= stages &&
                  16 * P::DEPTH <= 128 &&
                  // a chained launch of one wave: 228 KB of an SM, 1 KB of each block, or its 65536 registers (57 and more a thread) have no room for two
                  (!chained || 1ll * g.ctas * B > sms || 2ll * g.threads * 64 > 65536 || 2 * (g.bytes + 1024) > 228 * 1024);
  ++checked;
  if (!ok && ++failed <= 10)
    std::printf("%s C %d T %lld B %d SMs %d merged %d: R %lld, %d threads, %d CTAs, %lld of %d bytes\n", name, C, T, B, sms, merged, R, g.threads, g.ctas,
                end, g.bytes);
}
// Fields of many stages, any batch: the stages of the SMs that work longest, against an even share
template <typename P>
void balance(const char* name, int C, long long T, int B, int sms) {
  const ClGeometry g = cl_geometry<P>(C, T, B, sms, false, true);
  const long long stages = (T + P::LAPS * g.rows - 1) / (P::LAPS * g.rows), waves = (1ll * g.ctas * B + sms - 1) / sms;
  const double over = static_cast<double>(waves * ((stages + g.ctas - 1) / g.ctas)) * sms / (static_cast<double>(B) * stages);
  ++checked;
  if (over > 1.25 && ++failed <= 10) std::printf("%s C %d T %lld B %d SMs %d: %d CTAs, %.2f of an even share\n", name, C, T, B, sms, g.ctas, over);
}
int main() {
  for (int B = 1; B <= 600; ++B) {
    balance<ClForwardSums>("forward sums", 384, 64800, B, 148);
    balance<ClForwardApply>("forward output", 384, 64800, B, 148);
    balance<ClBackwardSums>("backward sums", 384, 64800, B, 148);
    balance<ClBackwardApply>("backward output", 384, 64800, B, 148);
  }
  const long long fields[] = {1, 2, 3, 7, 31, 50, 64, 100, 255, 300, 719, 720, 1024, 1800, 2048, 2049, 3601, 5000, 6720, 8191, 16200, 18624, 20000, 32400, 57600, 64800, 115200, 259920, 1038240, 4147200, 50000000000};
  const int batches[] = {1, 2, 3, 4, 5, 7, 8, 16, 37, 50, 74, 75, 147, 148, 149, 300, 4096}, sm[] = {148, 132, 16};
  for (int sms : sm)
    for (int B : batches)
      for (int C = 8; C <= 1024; C += 8)
        for (long long T : fields) {
          check<ClForwardSums>("forward sums", C, T, B, sms, false, true, true);
          check<ClForwardSums>("forward sums", C, T, B, sms, false, true, false);
          check<ClBackwardSums>("backward sums", C, T, B, sms, false, true, true);
          check<ClBackwardSums>("backward sums", C, T, B, sms, false, true, false);
          for (int merged = 0; merged < 2; ++merged) {
            check<ClForwardApply>("forward output", C, T, B, sms, merged, false, !merged);
            check<ClBackwardApply>("backward output", C, T, B, sms, merged, false, !merged);
          }
        }
  for (long long T = 1; T <= 12000; ++T)
    for (int C : {8, 16, 24, 48, 64, 72, 96, 104, 128, 192, 232, 384}) {
      check<ClForwardApply>("forward output", C, T, 1, 148, true, false, false);
      check<ClBackwardApply>("backward output", C, T, 2, 148, true, false, false);
    }
  std::printf("%lld checked, %lld failed\n", checked, failed);
  return failed != 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_launches_of_the_instance_norm(tmp_path):
    src, exe = tmp_path / "geometry.cpp", tmp_path / "geometry"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert run.returncode == 0, run.stdout
