// y[rows, N] = f(x)[rows, K] . w[N, K]^T for up to eight rows, where f is the identity or the add + norm that a decoder
// stack puts in front of its projections. Launched with programmatic dependent launch, like the GEMM of stream_gemm.h.
#pragma once
#include "stream_gemm.h"

namespace omni {

enum NormKind : int {
  kNormStack = 1,  // v = sum + res, norm over v as it is, out = v * r * gain (`qwen3_add_norm`)
  kNormLm = 2,     // v = bf16(sum + res), out = v * (gain * r) (`lm_add_norm`)
  kAddLm = 3,      // v = bf16(sum + res), out = v (`lm_add`)
};

// The add + norm in front of a projection. Every CTA makes the rows for itself; the residual goes to another buffer,
// because CTAs that start late still read the old one.
struct FewNorm {
  int kind = 0;
  Summands sum;
  const bf16* res_in = nullptr;
  bf16* res_out = nullptr;
  const bf16* gain = nullptr;
  float eps = 0.f;
};

struct FewPlan {
  CUtensorMap wmap;
  int N = 0, K = 0, rows = 0, R = 16, splits = 1, slots = 1, out = kStreamBf16, xk = 0;
  const bf16* x = nullptr;
  bf16* y = nullptr;
  float* part = nullptr;
  int ldy = 0;
  Epilogue epi;
  size_t smem = 0;
  size_t partial_floats() const { return (size_t)splits * rows * N; }
  Summands summands() const {
    Summands s;
    s.part = part, s.splits = splits, s.split_stride = (int64_t)rows * N, s.ld = N;
    return s;
  }
};

constexpr int kFewRows = 8;  // one tile of m16n8k16; beyond, the tcgen05 kernel of stream_gemm.h is the faster one

void few_configure();
// Whether the norm of `rows` rows of K elements can be made by every CTA of the projection.
bool few_norm_fits(int K, int rows);
// Nonzero where the shape is not one of this kernel's, or (any_shape: taken all the same) is left to stream_gemm.h. x == nullptr:
// the rows come from a FewNorm.
int few_plan(FewPlan* plan, const bf16* w, int N, int K, const bf16* x, int rows, int out, bf16* y, int ldy, float* part,
             Epilogue epi, int sm_count, bool any_shape = false);
cudaError_t few_launch(const FewPlan& plan, const FewNorm& norm, uint32_t* err, cudaStream_t stream, const sm100::Ahead& ahead = {});

}  // namespace omni
