// y[rows, N] = x[rows, K] . w[N, K]^T for decode-sized row counts (1..256), built to be chained: launched with
// programmatic dependent launch, it fetches its weights while the kernels before it still run.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "gemm.h"
#include "util.cuh"

namespace omni {

// A matrix that its consumer still has to sum: `splits` f32 partial sums [split][row][n], added in split order from
// zero and rounded to bf16 once, or (splits == 0) finished bf16 rows.
struct Summands {
  const float* part = nullptr;
  const bf16* done = nullptr;
  int splits = 0;
  int64_t split_stride = 0;  // floats
  int ld = 0;                // elements per row
};

// Eight columns of row n from column c on: the bf16 values, widened. At most MAX splits.
template <int MAX = 8>
__device__ __forceinline__ void load_sum8(const Summands& x, int n, int c, float (&v)[8]) {
  if (x.splits == 0) {
    unpack8v(__ldcg(reinterpret_cast<const uint4*>(x.done + (int64_t)n * x.ld + c)), v);
    return;
  }
  const float* p = x.part + (int64_t)n * x.ld + c;
  float4 f[MAX][2];
#pragma unroll
  for (int s = 0; s < MAX; ++s)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      f[s][h] = s < x.splits ? __ldcg(reinterpret_cast<const float4*>(p + s * x.split_stride) + h) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = 0.f;
#pragma unroll
  for (int s = 0; s < MAX; ++s) {  // adding 0 for a missing split leaves the sum unchanged
    v[0] += f[s][0].x, v[1] += f[s][0].y, v[2] += f[s][0].z, v[3] += f[s][0].w;
    v[4] += f[s][1].x, v[5] += f[s][1].y, v[6] += f[s][1].z, v[7] += f[s][1].w;
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = bf16_round(v[k]);
}

enum StreamOut : int { kStreamBf16 = 0, kStreamPartials = 1, kStreamSwiglu = 2 };

struct StreamGemmPlan {
  CUtensorMap wmap, xmap;
  int N = 0, K = 0, rows = 0, M = 64, bn = 8, tn = 16, splits = 1, kbs = 1, stages = 1, slots = 2, issuers = 1, acc_cols = 32;
  int out = kStreamBf16;
  bf16* y = nullptr;     // kStreamBf16: [rows, ldy]; kStreamSwiglu: activations [rows, ldy = N / 2]
  float* part = nullptr; // kStreamPartials
  int ldy = 0;
  Epilogue epi;
  int ctas() const { return ((N + tn - 1) / tn) * splits * ((rows + 127) / 128); }
  size_t partial_floats() const { return (size_t)splits * rows * N; }
  Summands summands() const {
    Summands s;
    s.part = part, s.splits = splits, s.split_stride = (int64_t)rows * N, s.ld = N;
    return s;
  }
};

void stream_configure();
bool stream_supports(int N, int K, int rows);
// Channels per group of the gate|up weight layout the fused SwiGLU wants ([g gate rows; their g up rows; next group ...],
// the last group may be smaller): one tile per SM where the matrix is narrow enough.
int stream_granule(int inter, int sm_count);
int stream_plan(StreamGemmPlan* plan, const bf16* w, int N, int K, const bf16* x, int rows, int out, bf16* y, int ldy,
                float* part, Epilogue epi, int sm_count, int granule = 0, int force_splits = 0);
cudaError_t stream_launch(const StreamGemmPlan& plan, uint32_t* err, cudaStream_t stream);

}  // namespace omni
