// y[rows, N] = x[rows, K] . w[N, K]^T for prompt-sized row counts: tcgen05 tiles of 256 rows by up to 256 columns on pairs
// of SMs, launched with programmatic dependent launch like the other GEMMs of a chain.
#pragma once
#include "stream_gemm.h"

namespace omni {

struct WidePlan {
  CUtensorMap xmap, wmap;
  int N = 0, K = 0, rows = 0, tn = 256, granule = 0, out = kStreamBf16, ctas = 2;
  bf16* y = nullptr;
  int ldy = 0;
  Epilogue epi;
};

void wide_configure();
// Whether gate|up rows in groups of `granule` fall into whole tiles, so that SwiGLU can be part of the GEMM.
bool wide_fuses(int N, int K, int granule);
// Nonzero where the shape is not one of this kernel's (out: kStreamBf16 or kStreamSwiglu).
int wide_plan(WidePlan* plan, const bf16* w, int N, int K, const bf16* x, int rows, int out, bf16* y, int ldy, Epilogue epi,
              int sm_count, int granule = 0);
cudaError_t wide_launch(const WidePlan& plan, uint32_t* err, cudaStream_t stream);

}  // namespace omni
