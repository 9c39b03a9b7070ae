// Talker / code-predictor glue: embedding gathers, the frame embedding, the
// predictor's first input and the fused sampler. Value semantics follow
// crates/omni-qwen3-tts/kernels/talker.cu; ids outside their tables raise the
// device error word instead of reading out of bounds.
#include "kernels.h"
#include "sampler.cuh"
#include "pdl.cuh"
#include "sm100.cuh"

namespace omni {

constexpr int kGroups = 16;

__global__ void gather_kernel(const int32_t* ids, int stride, const bf16* table, int table_rows, bf16* __restrict__ out, int dim, uint32_t* err) {
  grid_trigger();
  grid_wait();
  const int c = threadIdx.x * 8;
  int64_t id = __ldcg(ids + (int64_t)blockIdx.x * stride);  // ids and table may be an earlier kernel's output
  if (id < 0 || id >= table_rows) {
    if (threadIdx.x == 0) raise(err, kErrBadIndex);
    id = 0;
  }
  *reinterpret_cast<uint4*>(out + (int64_t)blockIdx.x * dim + c) =
      __ldcg(reinterpret_cast<const uint4*>(table + id * dim + c));
}

// `talker_prompt_codec` (talker.cu:55-71): x + bias (+ codec embedding), one rounding.
__global__ void prompt_codec_kernel(bf16* x, const bf16* __restrict__ bias,
                                    const bf16* __restrict__ table, int table_rows, const int32_t* __restrict__ ids,
                                    int dim, uint32_t* err) {
  grid_trigger();
  grid_wait();
  const int c = threadIdx.x * 8;
  bf16* row = x + (int64_t)blockIdx.x * dim + c;
  int id = ids[blockIdx.x];
  if (id >= table_rows) {
    if (threadIdx.x == 0) raise(err, kErrBadIndex);
    id = -1;
  }
  float v[8], b[8], e[8];
  ld8cg(row, v);
  ld8(bias + c, b);
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] += b[k];
  if (id >= 0) {
    ld8(table + (int64_t)id * dim + c, e);
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] += e[k];
  }
  st8(row, v);
}

__device__ __forceinline__ int32_t* slot_of(const SlotState& st, int s) {
  return reinterpret_cast<int32_t*>(static_cast<char*>(st.state) + (int64_t)st.lines[s] * st.stride);
}

// `talker_frame_embed` (talker.cu:76-96): f32 sum in the order pad, codebook 0,
// codebooks 1.., one rounding.
__device__ __forceinline__ void frame_embed_row(const SlotState& st, const bf16* pad, const bf16* codec_emb, int vocab,
                                                const bf16* p_emb, int p_vocab, int groups, int dim, uint32_t* err,
                                                float (&acc)[8]) {
  const int s = blockIdx.x, c = threadIdx.x * 8;
  const int32_t* codes = slot_of(st, s);
  float e[8];
  ld8(pad + c, acc);
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] = 0.f + acc[k];
  int c0 = codes[0];
  if (c0 < 0 || c0 >= vocab) {
    if (threadIdx.x == 0) raise(err, kErrBadIndex);
    c0 = 0;
  }
  ld8(codec_emb + (int64_t)c0 * dim + c, e);
#pragma unroll
  for (int k = 0; k < 8; ++k) acc[k] += e[k];
#pragma unroll 5
  for (int g = 1; g < groups; ++g) {
    int cg = codes[g];
    if (cg < 0 || cg >= p_vocab) {
      if (threadIdx.x == 0) raise(err, kErrBadIndex);
      cg = 0;
    }
    ld8(p_emb + ((int64_t)(g - 1) * p_vocab + cg) * dim + c, e);
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[k] += e[k];
  }
}

__global__ void frame_embed_kernel(SlotState st, const bf16* __restrict__ pad, const bf16* __restrict__ codec_emb,
                                   int vocab, const bf16* __restrict__ p_emb, int p_vocab, int groups,
                                   bf16* __restrict__ out, int dim, uint32_t* err) {
  grid_trigger();
  grid_wait();
  float acc[8];
  frame_embed_row(st, pad, codec_emb, vocab, p_emb, p_vocab, groups, dim, err, acc);
  st8(out + (int64_t)blockIdx.x * dim + threadIdx.x * 8, acc);
}

__global__ void frame_embed_norm_kernel(SlotState st, const bf16* __restrict__ pad, const bf16* __restrict__ codec_emb,
                                        int vocab, const bf16* __restrict__ p_emb, int p_vocab, int groups,
                                        const bf16* __restrict__ gain, bf16* __restrict__ res, bf16* __restrict__ x, int dim,
                                        float eps, uint32_t* err) {
  grid_trigger();
  __shared__ float scratch[32];
  const int64_t at = (int64_t)blockIdx.x * dim + threadIdx.x * 8;
  const bool on = threadIdx.x * 8 < dim;
  float v[8] = {}, g[8], ss = 0.f;
  if (on) ld8(gain + threadIdx.x * 8, g);
  grid_wait();
  if (on) frame_embed_row(st, pad, codec_emb, vocab, p_emb, p_vocab, groups, dim, err, v);
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = bf16_round(v[k]), ss += v[k] * v[k];
  const float r = rsqrtf(block_add(ss, scratch) / dim + eps);
  if (!on) return;
  st8(res + at, v);
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = v[k] * r * g[k];
  st8(x + at, v);
}

// `talker_pred_input` (talker.cu:100-106).
__global__ void pred_input_kernel(const bf16* hidden, const bf16* codec_emb, int vocab, const int32_t* codes,
                                  bf16* __restrict__ out, int dim, uint32_t* err) {
  grid_trigger();
  grid_wait();
  const int s = blockIdx.x, c = threadIdx.x * 8;
  const bf16* src;
  if (blockIdx.y == 0) {
    src = hidden + (int64_t)s * dim;
  } else {
    int id = __ldcg(codes + s * kGroups);
    if (id < 0 || id >= vocab) {
      if (threadIdx.x == 0) raise(err, kErrBadIndex);
      id = 0;
    }
    src = codec_emb + (int64_t)id * dim;
  }
  *reinterpret_cast<uint4*>(out + ((int64_t)2 * s + blockIdx.y) * dim + c) = __ldcg(reinterpret_cast<const uint4*>(src + c));
}

__global__ void stamp_kernel(unsigned long long* at) {
  grid_trigger();
  grid_wait();
  *at = sm100::global_timer_ns();
}

cudaError_t launch_stamp(unsigned long long* at, cudaStream_t s) {
  return launch_pdl(stamp_kernel, dim3(1), dim3(1), 0, s, at);
}

cudaError_t launch_gather(const int32_t* ids, int stride, const bf16* table, int table_rows, bf16* out, int rows,
                          int dim, uint32_t* err, cudaStream_t s) {
  return launch_pdl(gather_kernel, dim3(rows), dim3(dim / 8), 0, s, ids, stride, table, table_rows, out, dim, err);
}

cudaError_t launch_prompt_codec(bf16* x, const bf16* bias, const bf16* table, int table_rows, const int32_t* ids,
                                int rows, int dim, uint32_t* err, cudaStream_t s) {
  return launch_pdl(prompt_codec_kernel, dim3(rows), dim3(dim / 8), 0, s, x, bias, table, table_rows, ids, dim, err);
}

cudaError_t launch_frame_embed(SlotState st, const bf16* pad, const bf16* codec_emb, int vocab, const bf16* p_emb,
                               int p_vocab, int groups, bf16* out, int rows, int dim, uint32_t* err, cudaStream_t s) {
  return launch_pdl(frame_embed_kernel, dim3(rows), dim3(dim / 8), 0, s, st, pad, codec_emb, vocab, p_emb, p_vocab, groups, out, dim, err);
}

cudaError_t launch_frame_embed_norm(SlotState st, const bf16* pad, const bf16* codec_emb, int vocab, const bf16* p_emb,
                                    int p_vocab, int groups, const bf16* gain, bf16* res, bf16* x, int rows, int dim,
                                    float eps, uint32_t* err, cudaStream_t s) {
  return launch_pdl(frame_embed_norm_kernel, dim3(rows), dim3(row_threads(dim)), 0, s, st, pad, codec_emb, vocab, p_emb, p_vocab, groups,
                    gain, res, x, dim, eps, err);
}

cudaError_t launch_pred_input(const bf16* hidden, const bf16* codec_emb, int vocab, const int32_t* codes, bf16* out,
                              int rows, int dim, uint32_t* err, cudaStream_t s) {
  return launch_pdl(pred_input_kernel, dim3(rows, 2), dim3(dim / 8), 0, s, hidden, codec_emb, vocab, codes, out, dim, err);
}

// ---- token selection ----------------------------------------------------------
// One 512-thread block per row; the algorithm lives in sampler.cuh. A draw is a chain of block barriers with little between
// them, so what counts is how many there are and how few instructions: half the logits a thread where the vocabulary ends
// at 2,048 (the predictor's heads), sixteen-bit keys where no penalty has touched the row. 9.7 us a draw with full-width
// keys and 4,096 logits (17 us with the nucleus filter).

template <int THREADS, int VOCAB>
__global__ void __launch_bounds__(THREADS)
    sample_kernel(const bf16* logits, sampler::Params prm, const int32_t* __restrict__ frames,
                  const float* __restrict__ uniforms, const int32_t* __restrict__ force, SlotState st,
                  int32_t* __restrict__ codes, NextRow next) {
  using Team = sampler::Team<THREADS, sampler::CtaSync, VOCAB>;
  grid_trigger();
  __shared__ sampler::Shared sh;
  const int s = blockIdx.x, tid = threadIdx.x;
  const bf16* l = logits + (int64_t)s * prm.vocab;
  int32_t* slot = slot_of(st, s);
  const int frame = frames[s], forced = force[s * kGroups + prm.group];
  const float uniform = uniforms[s * kGroups + prm.group];
  grid_wait();
  float mine[Team::PER];
  if (prm.vocab % Team::PER == 0 && (reinterpret_cast<uintptr_t>(logits) & 7) == 0) {
    if (tid * Team::PER < prm.vocab) {
#pragma unroll
      for (int j = 0; j < Team::PER; j += 4) {
        const uint2 u = __ldcg(reinterpret_cast<const uint2*>(l + tid * Team::PER + j));
        mine[j] = __uint_as_float(u.x << 16), mine[j + 1] = __uint_as_float(u.x & 0xffff0000u);
        mine[j + 2] = __uint_as_float(u.y << 16), mine[j + 3] = __uint_as_float(u.y & 0xffff0000u);
      }
    }
  } else {
    for (int j = 0; j < Team::PER; ++j)
      mine[j] = tid * Team::PER + j < prm.vocab ? __bfloat162float(__ldcg(l + tid * Team::PER + j)) : 0.f;
  }
  const int token = Team::sample_row([&](int, int j) { return mine[j]; }, prm, frame, uniform, forced, slot,
                                     Team::seen_word(slot, prm, tid), codes + s * kGroups + prm.group, tid, sh);
  if (!next.table) return;
  const int c = tid * 8;
  float v[8], g[8], ss = 0.f;
  const bool on = c < next.dim;
  if (on) {
    ld8(next.table + (int64_t)token * next.dim + c, v);
    ld8(next.gain + c, g);
#pragma unroll
    for (int k = 0; k < 8; ++k) ss += v[k] * v[k];
  }
  ss = warp_add(ss);
  if ((tid & 31) == 0) sh.red[tid >> 5] = ss;
  __syncthreads();
  const float r = rsqrtf(warp_add((tid & 31) < THREADS / 32 ? sh.red[tid & 31] : 0.f) / next.dim + next.eps);
  if (on) {
    st8(next.res + (int64_t)s * next.dim + c, v);
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = v[k] * r * g[k];
    st8(next.x + (int64_t)s * next.dim + c, v);
  }
}

cudaError_t launch_sample_next(const bf16* logits, const SampleParams& p, const int32_t* frames, const float* uniforms,
                               const int32_t* force, SlotState st, int32_t* codes, const NextRow& next, int rows,
                               cudaStream_t s) {
  if (p.vocab > sampler::kVocabMax || p.vocab < 1) return cudaErrorInvalidValue;
  // the nucleus filter ranks at most kMaxNucleus survivors of the top-k cut: without a cut that small it would
  // silently drop candidates in arrival order
  if (p.top_p < 1.f && (p.top_k <= 0 || p.top_k > sampler::kMaxNucleus)) return cudaErrorInvalidValue;
  sampler::Params prm{p.vocab,  p.temperature, p.top_k,    p.top_p, p.penalty, p.suppress_lo, p.suppress_hi,
                      p.exempt, p.min_frames,  p.penalize, p.group, p.philox,  p.seen_words};
  if (next.table && next.dim > kNextRowMax) return cudaErrorInvalidValue;
  auto go = [&](auto kernel) {
    return launch_pdl(kernel, dim3(rows), dim3(512), 0, s, logits, prm, frames, uniforms, force, st, codes, next);
  };
  return p.vocab <= 2048 ? go(sample_kernel<512, 2048>) : go(sample_kernel<512, 4096>);
}

cudaError_t launch_sample(const bf16* logits, const SampleParams& p, const int32_t* frames, const float* uniforms,
                          const int32_t* force, SlotState st, int32_t* codes, int rows, cudaStream_t s) {
  return launch_sample_next(logits, p, frames, uniforms, force, st, codes, NextRow{}, rows, s);
}

}  // namespace omni
