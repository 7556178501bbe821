// What the translation units that see torch share: launching one GEMM of the engine from tensors and strides.
#pragma once
#include <torch/extension.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>

#include <cstdint>
#include <utility>
#include <vector>

#include "gemm_tcgen05.cuh"

#define MK_CHECK(cond, ...) TORCH_CHECK(cond, "makani_b200: ", __VA_ARGS__)

namespace mkh {

using torch::Tensor;
constexpr int64_t BIG = 1ll << 30;

// The fields of `Operand`, `Output`, `Tri` and `gemm` in ops/gemm.py
struct Operand {
  const Tensor* t = nullptr;
  int64_t ld = 0;
  bool mn_major = false;
  int64_t offset = 0, zs_lo = 0, zs_hi = 0;
};
struct Output {
  Tensor* t = nullptr;
  int64_t rs_lo = 0, offset = 0, rdiv = BIG, rs_hi = 0, ndiv = BIG, ns_hi = 0, d_zlo = 0, d_zhi = 0;
};
struct Tri {
  int64_t rmin_a = 0, rmin_b = 0, rmax_a = 0, rmax_b = BIG, kmin_a = 0, kmin_b = 0, kmax_a = 0, kmax_b = BIG;
};
enum { ACT_NONE = 0, ACT_GELU = 1, ACT_RELU = 3, ACT_DRELU = 4, ACT_SHRINK = 5, ACT_DSHRINK = 6, ACT_MULAUX = 8 };
enum { BIAS_NONE = 0, BIAS_ROW = 1, BIAS_COL = 2 };
// Partial row sums of a launch, held until they are added up
struct SumsLater {
  Tensor part;
  mk::RowSlabs slabs;
};
struct Gemm {
  int64_t M = 0, N = 0, K = 0;
  Operand A, B;
  Output D;
  int64_t zlo_n = 1, zhi_n = 1, splits = 1, bn = 0;
  Tri tri;
  double alpha = 1.0;
  const Tensor* bias = nullptr;      // (undefined tensors count as none)
  int bias_mode = BIAS_NONE;
  int64_t bias_zs = 0;
  int act = ACT_NONE;
  float act_param = 0.f;
  const Tensor* resid = nullptr;
  int64_t resid_offset = 0;
  Tensor* preact = nullptr;
  int64_t preact_offset = 0;
  bool preact_deriv = false, accumulate = false;
  Tensor* row_sums = nullptr;        // see mk::GemmRowSums
  SumsLater* sums_later = nullptr;   // the partial sums are added up with another launch's
};

// Validates, launches on the current stream and raises; whether the row sums were taken.
bool run(const Gemm& g, const mk::GemmPeer* peer = nullptr);
// Integer parameters as in ops/gemm.py
void complex_product(const Tensor& a, const Tensor& b, Tensor& d, const Tensor* resid, const std::vector<int64_t>& ip);
void folded_product(const Tensor& a, const Tensor& b, Tensor& d, const std::vector<int64_t>& ip);

void check(cudaError_t e, const char* what);
// the device error word that kernels with bounded waits report to
int* error_word(const Tensor& like);
inline cudaStream_t stream() { return at::cuda::getCurrentCUDAStream().stream(); }

// kernel launches of this thread's layer passes
int64_t& launches();

void bind_layers(pybind11::module_& m);

}  // namespace mkh
