// y[rows, N] = x[rows, K] . w[N, K]^T for decode-sized row counts (1..256), built to be chained: launched with
// programmatic dependent launch, it fetches its weights while the kernels before it still run.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "gemm.h"
#include "sm100.cuh"
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

// E columns (2, 4 or 8) of row n from column c on, of S summands (0: bf16 rows): the bf16 values, widened.
template <int S, int E>
__device__ __forceinline__ void load_sum(const Summands& x, int n, int c, float (&v)[E]) {
  if constexpr (S == 0) {
    Run<E>::ldcg(x.done + (int64_t)n * x.ld + c, v);
  } else {
    using Word = std::conditional_t<E == 2, float2, float4>;
    constexpr int H = E == 8 ? 2 : 1;
    const float* p = x.part + (int64_t)n * x.ld + c;
    Word f[S][H];
#pragma unroll
    for (int s = 0; s < S; ++s)
#pragma unroll
      for (int h = 0; h < H; ++h) f[s][h] = __ldcg(reinterpret_cast<const Word*>(p + s * x.split_stride) + h);
#pragma unroll
    for (int k = 0; k < E; ++k) {
      float sum = reinterpret_cast<const float*>(f[0])[k];
#pragma unroll
      for (int s = 1; s < S; ++s) sum += reinterpret_cast<const float*>(f[s])[k];
      v[k] = bf16_round(sum);
    }
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

// go(std::integral_constant<int, E>): columns a thread of the add + norm of `rows` rows of `dim` elements. What is behind its
// wait runs once, so few columns a thread and up to 1,024 threads. Eight columns and this, one pass, us: a talker step of 8
// sessions (1,024 and 2,048 wide) 2,653 and 2,586, of 64 3,714 and 3,613, of 128 5,004 and 4,910, a duplex tick of 64 (4,096)
// 5,713 and 5,652, a Higgs step of 32 (2,560) 3,010 and 2,980. Prompts are many rows whose bytes count.
template <typename F>
cudaError_t with_columns(int dim, int rows, F&& go) {
  if (rows <= 256 && dim <= 2048) return go(std::integral_constant<int, 2>());
  if (rows <= 256 && dim <= 4096) return go(std::integral_constant<int, 4>());
  return go(std::integral_constant<int, 8>());
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
cudaError_t stream_launch(const StreamGemmPlan& plan, uint32_t* err, cudaStream_t stream, bool whole_smem = false, const sm100::Ahead& ahead = {});

}  // namespace omni
