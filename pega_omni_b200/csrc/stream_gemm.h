// y[rows, N] = x[rows, K] . w[N, K]^T for decode-sized row counts (1..256), built to be chained: launched with
// programmatic dependent launch, it fetches its weights while the kernels before it still run.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

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

// Eight columns of row n from column c on, of S summands (0: bf16 rows): the bf16 values, widened.
template <int S>
__device__ __forceinline__ void load_sum8(const Summands& x, int n, int c, float (&v)[8]) {
  if constexpr (S == 0) {
    unpack8v(__ldcg(reinterpret_cast<const uint4*>(x.done + (int64_t)n * x.ld + c)), v);
  } else {
    const float* p = x.part + (int64_t)n * x.ld + c;
    float4 f[S][2];
#pragma unroll
    for (int s = 0; s < S; ++s)
#pragma unroll
      for (int h = 0; h < 2; ++h) f[s][h] = __ldcg(reinterpret_cast<const float4*>(p + s * x.split_stride) + h);
#pragma unroll
    for (int s = 1; s < S; ++s) {
      f[0][0].x += f[s][0].x, f[0][0].y += f[s][0].y, f[0][0].z += f[s][0].z, f[0][0].w += f[s][0].w;
      f[0][1].x += f[s][1].x, f[0][1].y += f[s][1].y, f[0][1].z += f[s][1].z, f[0][1].w += f[s][1].w;
    }
    v[0] = bf16_round(f[0][0].x), v[1] = bf16_round(f[0][0].y), v[2] = bf16_round(f[0][0].z), v[3] = bf16_round(f[0][0].w);
    v[4] = bf16_round(f[0][1].x), v[5] = bf16_round(f[0][1].y), v[6] = bf16_round(f[0][1].z), v[7] = bf16_round(f[0][1].w);
  }
}

// go(std::integral_constant<int, S>) for the summand counts that the plans make.
template <typename F>
cudaError_t with_summands(int splits, F&& go) {
  switch (splits) {
    case 0: return go(std::integral_constant<int, 0>());
    case 1: return go(std::integral_constant<int, 1>());
    case 2: return go(std::integral_constant<int, 2>());
    case 4: return go(std::integral_constant<int, 4>());
    case 8: return go(std::integral_constant<int, 8>());
    default: return cudaErrorInvalidValue;
  }
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
// Channels per group of the gate|up weight layout the fused SwiGLU wants ([8 gate rows; their 8 up rows; next group ...]): a
// tile of any multiple of sixteen rows holds whole channels, and an epilogue's piece of eight columns is one group's gates.
// Groups as wide as half a tile would fix the tile for every row count: at one row 12,288 x 2,048 then kept one ring slot a
// warp, and a talker step took 2,176 us instead of 2,091.
constexpr int kGateGroup = 8;
int stream_plan(StreamGemmPlan* plan, const bf16* w, int N, int K, const bf16* x, int rows, int out, bf16* y, int ldy,
                float* part, Epilogue epi, int sm_count, int force_splits = 0);
cudaError_t stream_launch(const StreamGemmPlan& plan, uint32_t* err, cudaStream_t stream);

}  // namespace omni
