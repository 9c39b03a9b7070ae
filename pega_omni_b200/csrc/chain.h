// A pass of up to 256 rows of a Qwen3-style decoder stack as a chain of kernels under programmatic dependent launch: per layer
// seven kernels - q|k|v GEMM, rope + KV write + attention, o GEMM, add + norm, gate|up GEMM with SwiGLU, down GEMM,
// add + norm - of which every GEMM has its first weights in shared memory by the time its input rows are there. For a few
// rows the add + norm is part of the GEMM behind it: five kernels.
// Op order and rounding points of `Stack::forward` (crates/omni-qwen3/src/stack.rs:152-203).
#pragma once
#include <algorithm>
#include <map>
#include <tuple>
#include <vector>

#include "few_rows.h"
#include "kernels.h"
#include "stream_gemm.h"
#include "wide_gemm.h"

namespace omni {

// A GEMM of a chain is planned once per everything its plan holds - operands, shape, output, epilogue - and kept by the model.
struct ChainPlan {
  bool few = false;
  FewPlan f;
  StreamGemmPlan s;
};
using ChainKey = std::tuple<const void*, const void*, const void*, const void*, int, int, int, int, int, int>;
using ChainPlans = std::map<ChainKey, ChainPlan>;

// Stands behind every kernel of a traced program: a stamp of the device's clock, and the kernel's name and shape.
struct ChainTrace {
  struct Line {
    const char* what;
    int N, K, rows;
  };
  unsigned long long* stamps = nullptr;  // device, one per line
  size_t capacity = 0;
  std::vector<Line>* lines = nullptr;    // those of the program being enqueued
  cudaError_t mark(const char* what, int N, int K, int rows, cudaStream_t stream) const {
    if (!lines || lines->size() >= capacity) return cudaSuccess;
    lines->push_back(Line{what, N, K, rows});
    return launch_stamp(stamps + lines->size() - 1, stream);
  }
};

constexpr size_t kAheadBytes = 8 << 20;
constexpr int kChainRows = 256;  // beyond this the GEMMs are contractions, not streams of weights: wide_gemm.h

struct Chain {
  cudaStream_t stream = nullptr;
  uint32_t* err = nullptr;
  int sm_count = 148;
  float* partials = nullptr;
  size_t partial_floats = 0;
  int* launches = nullptr;
  ChainPlans* plans = nullptr;
  const ChainTrace* trace = nullptr;
  // The pass's attention keeps its rows in shared memory (frame_attend_kernel): beside a tcgen05 GEMM under the default carve-out
  // its CTAs find no room before the GEMM ends. One pass, default and whole, us: a talker step of 64 sessions 3,605 and 3,453,
  // of 128 4,906 and 4,836. The talker's own passes want the L1 that this takes away: their attention holds its pages under
  // way in registers, 4,836 and 5,170.
  bool whole_smem = false;

  // What the next GEMM asks into L2 on its way: the first of the weights of the GEMM after it, whose own requests start one
  // kernel before they are needed. For passes that leave DRAM idle, as measured; in brackets the share of the copy rate that the
  // call moves without it. One pass without and with 8 MB, us: a talker step of 1 session (0.25) 1,875 and 1,831, of 8 (0.2) 2,548
  // and 2,514, of 64 (0.2) 3,456 and 3,394, a start of one prompt (0.2) 2,697 and 2,650, a duplex tick of 64 with the depformer's
  // (its passes below 0.2) 5,174 and 5,129 (32 MB: 1,865, 2,560, 3,449, 2,662, 5,279). Where a call moves more, the requests
  // compete with the GEMMs' own: a Higgs step of 3 (0.5) 1,913 and 1,938, a duplex tick of 1 (0.7) 3,174 and 3,198: none there.
  // A pass's last GEMM asks for nothing.
  size_t ahead_cap = 0;
  sm100::Ahead ahead;
  void next(const bf16* w, int N, int K) {
    ahead.at = reinterpret_cast<const char*>(w);
    ahead.bytes = w ? (uint32_t)std::min((size_t)N * K * sizeof(bf16), ahead_cap) : 0u;
  }

  // Behind every launch: counted, and stamped where the program is traced.
  cudaError_t done(cudaError_t launched, const char* what, int N, int K, int rows) const {
    ++*launches;
    return launched == cudaSuccess && trace ? trace->mark(what, N, K, rows, stream) : launched;
  }

  // y (bf16 rows, SwiGLU activations) or, for kStreamPartials, *sum
  cudaError_t gemm(const bf16* w, int N, int K, const bf16* x, int rows, int out, bf16* y, int ldy, Summands* sum = nullptr,
                   int granule = kGateGroup, Epilogue epi = {}) const {
    if (rows > kChainRows) {  // prompts: any row count, so the plan (two tensor maps) is made for the call
      WidePlan wide;
      if (wide_plan(&wide, w, N, K, x, rows, out, y, ldy, epi, sm_count, granule) != 0) return cudaErrorInvalidValue;
      return done(wide_launch(wide, err, stream), out == kStreamSwiglu ? "gemm_swiglu" : "gemm", N, K, rows);
    }
    ChainPlan* p = plan(w, N, K, x, rows, out, y, ldy, epi);
    return p ? launch(*p, {}, sum) : cudaErrorInvalidValue;
  }

  // The same behind the add + norm of `norm.sum` into the residual rows `*res` (then exchanged with `*spare`): in one
  // kernel where few_rows.h takes the shape, otherwise by `apart`, which updates *res in place and writes x.
  template <typename Apart>
  cudaError_t norm_gemm(FewNorm norm, bf16** res, bf16** spare, const Apart& apart, const bf16* w, int N, int K, const bf16* x,
                        int rows, int out, bf16* y, int ldy) const {
    if (few_norm_fits(K, rows) && norm.sum.splits >= 1 && norm.sum.splits <= 4) {
      if (ChainPlan* p = plan(w, N, K, nullptr, rows, out, y, ldy, {})) {
        norm.res_in = *res, norm.res_out = *spare;
        std::swap(*res, *spare);
        return launch(*p, norm, nullptr);
      }
    }
    const cudaError_t e = done(apart(norm.sum, *res), "add_norm", 0, K, rows);
    return e != cudaSuccess ? e : gemm(w, N, K, x, rows, out, y, ldy);
  }

 private:
  ChainPlan* plan(const bf16* w, int N, int K, const bf16* x, int rows, int out, bf16* y, int ldy, Epilogue epi) const {
    const ChainKey key(w, x, y, epi.bias, N, K, rows, out, ldy, epi.kind);
    auto it = plans->find(key);
    if (it != plans->end()) return &it->second;
    ChainPlan p;
    p.few = few_plan(&p.f, w, N, K, x, rows, out, y, ldy, partials, epi, sm_count) == 0;
    if (!p.few) {  // what the tcgen05 kernel cannot take (stores, columns or sums of its own) stays with the other one
      const bool streams = x && stream_plan(&p.s, w, N, K, x, rows, out, y, ldy, partials, epi, sm_count) == 0 &&
                           (out != kStreamPartials || p.s.partial_floats() <= partial_floats);
      p.few = !streams && few_plan(&p.f, w, N, K, x, rows, out, y, ldy, partials, epi, sm_count, true) == 0;
      if (!streams && !p.few) return nullptr;
    }
    if (out == kStreamPartials && (p.few ? p.f.partial_floats() : p.s.partial_floats()) > partial_floats) return nullptr;
    return &plans->emplace(key, p).first->second;
  }
  cudaError_t launch(const ChainPlan& p, const FewNorm& norm, Summands* sum) const {
    if (sum) *sum = p.few ? p.f.summands() : p.s.summands();
    const int out = p.few ? p.f.out : p.s.out;
    const char* what = norm.kind ? (out == kStreamSwiglu ? "norm_gemm_swiglu" : "norm_gemm") : out == kStreamSwiglu ? "gemm_swiglu" : "gemm";
    return p.few ? done(few_launch(p.f, norm, err, stream, ahead), what, p.f.N, p.f.K, p.f.rows)
                 : done(stream_launch(p.s, err, stream, whole_smem, ahead), what, p.s.N, p.s.K, p.s.rows);
  }
};

#define OMNI_CHAIN(expr)                        \
  do {                                          \
    const cudaError_t e_ = (expr);              \
    if (e_ != cudaSuccess) return e_;           \
  } while (0)

struct ChainBuffers {
  bf16 *x, *res, *spare, *qkv, *attn, *act;  // x, res: the normalised rows and the residual stream the pass starts from
};

// Whether a stack of this shape can run as a chain (the rest is up to the row count).
inline bool chain_supports(int hidden, int inter, int q_width, int head_dim) {
  return hidden % 64 == 0 && hidden / 8 <= 1024 && inter % 64 == 0 && q_width % 64 == 0 && (head_dim == 64 || head_dim == 128);
}


// gate_up(l) and down(l) pick a layer's MLP; `inter` is its width, its gate|up rows lie in groups of kGateGroup.
template <typename Layer, typename GateUp, typename Down>
cudaError_t chain_pass(Chain c, const std::vector<Layer>& layers, const GateUp& gate_up, const Down& down, int hidden,
                       int inter, const AttnShape& a, ChainBuffers b, int rows, const RowMap& map,
                       const std::vector<bf16*>& kv, int kv_pages, const bf16* final_gain, bf16* keep_out, int every,
                       int which, const QkvTable& lookup = {}, bool prompt = false) {
  c.whole_smem = !map.pages;
  const int qd = a.q_heads * a.head_dim, qw = (a.q_heads + 2 * a.kv_heads) * a.head_dim;
  Summands sum;
  FewNorm norm;
  norm.kind = kNormStack, norm.eps = a.rms_eps;
  // the add + norm of `sum` by layer gain `gain`, and the GEMM of the rows it makes
  auto norm_gemm = [&](const bf16* gain, const bf16* w, int N, int out, bf16* y, int ldy) {
    norm.sum = sum, norm.gain = gain;
    return c.norm_gemm(norm, &b.res, &b.spare,
                       [&](const Summands& from, bf16* res) {
                         return launch_add_norm_sum(from, res, gain, b.x, rows, hidden, a.rms_eps, 1, 0, c.stream);
                       },
                       w, N, hidden, b.x, rows, out, y, ldy);
  };
  for (size_t i = 0; i < layers.size(); ++i) {
    const Layer& L = layers[i];
    const QkvTable& from = i == 0 ? lookup : QkvTable{};
    if (!from.table) c.next(gate_up(L), 2 * inter, hidden);
    if (i > 0) OMNI_CHAIN(norm_gemm(L.ln1, L.qkv, qw, kStreamBf16, b.qkv, qw));
    else if (!from.table) OMNI_CHAIN(c.gemm(L.qkv, qw, hidden, b.x, rows, kStreamBf16, b.qkv, qw));
    if (prompt) {  // rows of one sequence attend to one another: every key is written before the first is read
      OMNI_CHAIN(c.done(launch_rope_kv(b.qkv, L.q_norm, L.k_norm, kv[i], map, rows, a, kv_pages, c.err, c.stream), "rope_kv", 0, 0, rows));
      OMNI_CHAIN(c.done(launch_attend(b.qkv, kv[i], b.attn, map, rows, a, c.err, c.stream), "attend", 0, 0, rows));
    } else {
      OMNI_CHAIN(c.done(launch_rope_attend(b.qkv, from, L.q_norm, L.k_norm, kv[i], b.attn, map, rows, a, kv_pages, c.sm_count, c.err,
                                       c.stream),
                        "rope_attend", 0, 0, rows));
    }
    c.next(down(L), inter, hidden);
    OMNI_CHAIN(c.gemm(L.o, hidden, qd, b.attn, rows, kStreamPartials, nullptr, hidden, &sum));
    c.next(i + 1 < layers.size() ? layers[i + 1].qkv : nullptr, qw, hidden);
    OMNI_CHAIN(norm_gemm(L.ln2, gate_up(L), 2 * inter, kStreamSwiglu, b.act, inter));
    c.next(i + 1 < layers.size() ? layers[i + 1].o : nullptr, qd, hidden);
    OMNI_CHAIN(c.gemm(down(L), hidden, inter, b.act, rows, kStreamPartials, nullptr, hidden, &sum));
  }
  return c.done(launch_add_norm_sum(sum, b.res, final_gain, keep_out, rows, hidden, a.rms_eps, every, which, c.stream), "add_norm",
                0, hidden, rows);
}

}  // namespace omni
