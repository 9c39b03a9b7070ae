// A pass of up to 256 rows of a Qwen3-style decoder stack as a chain of kernels under programmatic dependent launch: per layer
// seven kernels - q|k|v GEMM, rope + KV write + attention, o GEMM, add + norm, gate|up GEMM with SwiGLU, down GEMM,
// add + norm - of which every GEMM has its first weights in shared memory by the time its input rows are there.
// Op order and rounding points of `Stack::forward` (crates/omni-qwen3/src/stack.rs:152-203).
#pragma once
#include <map>
#include <tuple>
#include <vector>

#include "kernels.h"
#include "stream_gemm.h"

namespace omni {

struct Chain {
  cudaStream_t stream = nullptr;
  uint32_t* err = nullptr;
  int sm_count = 148;
  float* partials = nullptr;
  size_t partial_floats = 0;
  int* launches = nullptr;
  std::map<std::tuple<const void*, const void*, const void*, int, int>, StreamGemmPlan>* plans = nullptr;

  // y (bf16 rows, SwiGLU activations) or, for kStreamPartials, *sum
  cudaError_t gemm(const bf16* w, int N, int K, const bf16* x, int rows, int out, bf16* y, int ldy, Summands* sum = nullptr,
                   int granule = 0, Epilogue epi = {}) const {
    const auto key = std::make_tuple((const void*)w, (const void*)x, (const void*)y, rows, out);
    auto it = plans->find(key);
    if (it == plans->end()) {
      StreamGemmPlan plan;
      if (stream_plan(&plan, w, N, K, x, rows, out, y, ldy, partials, epi, sm_count, granule) != 0) return cudaErrorInvalidValue;
      if (out == kStreamPartials && plan.partial_floats() > partial_floats) return cudaErrorInvalidValue;
      it = plans->emplace(key, plan).first;
    }
    if (sum) *sum = it->second.summands();
    ++*launches;
    return stream_launch(it->second, err, stream);
  }
};

#define OMNI_CHAIN(expr)                        \
  do {                                          \
    const cudaError_t e_ = (expr);              \
    if (e_ != cudaSuccess) return e_;           \
  } while (0)

struct ChainBuffers {
  bf16 *x, *res, *qkv, *attn, *act;  // x, res: the normalised rows and the residual stream the pass starts from
};

// Whether a stack of this shape can run as a chain (the rest is up to the row count).
inline bool chain_supports(int hidden, int inter, int q_width, int head_dim) {
  return hidden % 64 == 0 && hidden / 8 <= 1024 && inter % 64 == 0 && q_width % 64 == 0 && (head_dim == 64 || head_dim == 128);
}

constexpr int kChainRows = 256;  // beyond this the GEMMs are contractions, not streams of weights

// gate_up(l) and down(l) pick a layer's MLP; `inter` is its width, its gate|up rows lie in groups of `granule`.
template <typename Layer, typename GateUp, typename Down>
cudaError_t chain_pass(const Chain& c, const std::vector<Layer>& layers, const GateUp& gate_up, const Down& down, int hidden,
                       int inter, int granule, const AttnShape& a, const ChainBuffers& b, int rows, const RowMap& map,
                       const std::vector<bf16*>& kv, int kv_pages, const bf16* final_gain, bf16* keep_out, int every,
                       int which, const QkvTable& lookup = {}, bool prompt = false) {
  const int qd = a.q_heads * a.head_dim, qw = (a.q_heads + 2 * a.kv_heads) * a.head_dim;
  for (size_t i = 0; i < layers.size(); ++i) {
    const Layer& L = layers[i];
    const QkvTable& from = i == 0 ? lookup : QkvTable{};
    Summands sum;
    if (!from.table) OMNI_CHAIN(c.gemm(L.qkv, qw, hidden, b.x, rows, kStreamBf16, b.qkv, qw));
    if (prompt) {  // rows of one sequence attend to one another: every key is written before the first is read
      *c.launches += 2;
      OMNI_CHAIN(launch_rope_kv(b.qkv, L.q_norm, L.k_norm, kv[i], map, rows, a, kv_pages, c.err, c.stream));
      OMNI_CHAIN(launch_attend(b.qkv, kv[i], b.attn, map, rows, a, c.err, c.stream));
    } else {
      ++*c.launches;
      OMNI_CHAIN(launch_rope_attend(b.qkv, from, L.q_norm, L.k_norm, kv[i], b.attn, map, rows, a, kv_pages, c.err, c.stream));
    }
    OMNI_CHAIN(c.gemm(L.o, hidden, qd, b.attn, rows, kStreamPartials, nullptr, hidden, &sum));
    ++*c.launches;
    OMNI_CHAIN(launch_add_norm_sum(sum, b.res, L.ln2, b.x, rows, hidden, a.rms_eps, 1, 0, c.stream));
    OMNI_CHAIN(c.gemm(gate_up(L), 2 * inter, hidden, b.x, rows, kStreamSwiglu, b.act, inter, nullptr, granule));
    OMNI_CHAIN(c.gemm(down(L), hidden, inter, b.act, rows, kStreamPartials, nullptr, hidden, &sum));
    ++*c.launches;
    if (i + 1 < layers.size())
      OMNI_CHAIN(launch_add_norm_sum(sum, b.res, layers[i + 1].ln1, b.x, rows, hidden, a.rms_eps, 1, 0, c.stream));
    else
      OMNI_CHAIN(launch_add_norm_sum(sum, b.res, final_gain, keep_out, rows, hidden, a.rms_eps, every, which, c.stream));
  }
  return cudaSuccess;
}

}  // namespace omni
