// Operator-level C ABI (include/omni_b200_ops.h): each kernel as a plain call
// over caller-owned device buffers.
#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <string>

#include "../../include/omni_b200.h"
#include "../../include/omni_b200_ops.h"
#include "chain.h"
#include "codec.h"
#include "gemm.h"
#include "duplex.h"
#include "kernels.h"

using namespace omni;

struct omni_ops {
  int device = 0, sm_count = 148;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev[2] = {nullptr, nullptr};
  GemmScratch scratch;
  uint32_t* err = nullptr;
  std::string error;
  int fail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    error = buf;
    return code;
  }
};

// Nothing of the next launch starts before everything in front of it in the stream has ended. Attention kernels ask for their
// pages, GEMMs for their weights and biases before they wait for the kernel in front of them, because no other kernel of a
// model's call writes those; calls made one by one here may.
__global__ void order_kernel() {}
static cudaError_t order(cudaStream_t s) {
  order_kernel<<<1, 1, 0, s>>>();
  return cudaGetLastError();
}

// go(qkv, out) on 16-byte aligned rows, which the attention kernels' vector accesses need: the caller's own where they are,
// otherwise copies (out is written back; so are the rows of qkv, which may be rotated in place).
template <typename Go>
static cudaError_t on_aligned_rows(void* qkv, size_t qkv_bytes, void* out, size_t out_bytes, cudaStream_t s, Go&& go) {
  if (((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(out)) & 15) == 0) return go(qkv, out);
  const size_t at = (qkv_bytes + 255) & ~(size_t)255;
  char* tmp = nullptr;
  cudaError_t e = cudaMalloc((void**)&tmp, at + out_bytes);
  if (e != cudaSuccess) return e;
  e = cudaMemcpyAsync(tmp, qkv, qkv_bytes, cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess) e = go(tmp, tmp + at);
  if (e == cudaSuccess) e = cudaMemcpyAsync(qkv, tmp, qkv_bytes, cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(out, tmp + at, out_bytes, cudaMemcpyDeviceToDevice, s);
  const cudaError_t done = cudaStreamSynchronize(s);
  cudaFree(tmp);
  return e != cudaSuccess ? e : done;
}

#define OPS_CUDA(ctx, expr)                                                                       \
  do {                                                                                            \
    cudaError_t e_ = (expr);                                                                      \
    if (e_ != cudaSuccess) return (ctx)->fail(OMNI_ERR_CUDA, "%s: %s", #expr, cudaGetErrorString(e_)); \
  } while (0)

extern "C" {

int32_t omni_ops_create(int32_t device, omni_ops** out) {
  if (!out) return OMNI_ERR_INVALID;
  omni_ops* c = new omni_ops();
  *out = c;
  c->device = device;
  OPS_CUDA(c, cudaSetDevice(device));
  cudaDeviceProp prop;
  OPS_CUDA(c, cudaGetDeviceProperties(&prop, device));
  if (prop.major != 10) return c->fail(OMNI_ERR_UNSUPPORTED, "device is sm_%d%d; this library is sm_100a only", prop.major, prop.minor);
  c->sm_count = prop.multiProcessorCount;
  OPS_CUDA(c, cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
  OPS_CUDA(c, cudaEventCreate(&c->ev[0]));
  OPS_CUDA(c, cudaEventCreate(&c->ev[1]));
  if (tc_init() != 0) return c->fail(OMNI_ERR_CUDA, "cuTensorMapEncodeTiled entry point not found");
  tc_configure();
  stream_configure();
  c->scratch.partial_floats = (size_t)64 << 20;  // 256 MB of f32 partials: any test shape
  c->scratch.counter_slots = 1 << 16;
  OPS_CUDA(c, cudaMalloc((void**)&c->scratch.partials, c->scratch.partial_floats * 4));
  OPS_CUDA(c, cudaMalloc((void**)&c->scratch.counters, (size_t)c->scratch.counter_slots * 4));
  OPS_CUDA(c, cudaMemset(c->scratch.counters, 0, (size_t)c->scratch.counter_slots * 4));
  OPS_CUDA(c, cudaMalloc((void**)&c->err, 256));
  OPS_CUDA(c, cudaMemset(c->err, 0, 256));
  return OMNI_OK;
}

void omni_ops_destroy(omni_ops* c) {
  if (!c) return;
  cudaSetDevice(c->device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  cudaFree(c->scratch.partials);
  cudaFree(c->scratch.counters);
  cudaFree(c->err);
  if (c->ev[0]) cudaEventDestroy(c->ev[0]);
  if (c->ev[1]) cudaEventDestroy(c->ev[1]);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
}

const char* omni_ops_last_error(const omni_ops* c) { return c ? c->error.c_str() : "null context"; }

int32_t omni_ops_sync(omni_ops* c, uint32_t* word) {
  if (!c) return OMNI_ERR_INVALID;
  OPS_CUDA(c, cudaStreamSynchronize(c->stream));
  uint32_t w = 0;
  OPS_CUDA(c, cudaMemcpy(&w, c->err, 4, cudaMemcpyDeviceToHost));
  if (word) *word = w;
  if (w != 0) {
    cudaMemset(c->err, 0, 4);
    return c->fail(OMNI_ERR_DEVICE, "device error word 0x%x", w);
  }
  return OMNI_OK;
}

int32_t omni_ops_mark(omni_ops* c, int32_t which) {
  if (!c || which < 0 || which > 1) return OMNI_ERR_INVALID;
  OPS_CUDA(c, cudaEventRecord(c->ev[which], c->stream));
  return OMNI_OK;
}

int32_t omni_ops_elapsed_ms(omni_ops* c, float* ms) {
  if (!c || !ms) return OMNI_ERR_INVALID;
  OPS_CUDA(c, cudaEventSynchronize(c->ev[1]));
  OPS_CUDA(c, cudaEventElapsedTime(ms, c->ev[0], c->ev[1]));
  return OMNI_OK;
}

int32_t omni_op_gemm(omni_ops* c, const void* w, int32_t N, int32_t K, const void* x, int32_t rows, void* y,
                     int32_t ldy, int32_t path, int32_t splits, const void* bias, int32_t epilogue) {
  if (!c || !w || !x || !y || N < 1 || K < 8 || rows < 1) return OMNI_ERR_INVALID;
  if (epilogue != OMNI_EPI_NONE && !bias) return c->fail(OMNI_ERR_INVALID, "epilogue %d needs a bias", epilogue);
  Epilogue epi;
  epi.bias = static_cast<const bf16*>(bias);
  epi.kind = epilogue;
  if (path == OMNI_GEMM_TENSOR_ROWS) {
    if (!rm_supports(N, K, rows)) return c->fail(OMNI_ERR_UNSUPPORTED, "rows-on-M path needs rows <= 128, K %% 64 == 0, K <= 4096");
    RmGemmPlan plan;
    const int rc = rm_plan(&plan, (const bf16*)w, N, K, (const bf16*)x, rows, (bf16*)y, ldy, epi, c->sm_count);
    if (rc != 0) return c->fail(OMNI_ERR_CUDA, "tensor-map encode failed (%d)", rc);
    OPS_CUDA(c, rm_launch(plan, c->err, c->stream));
    return OMNI_OK;
  }
  const bool tensor = path == OMNI_GEMM_TENSOR || (path == OMNI_GEMM_AUTO && rows > 8 && tc_supports(N, K, rows));
  if (!tensor) {
    OPS_CUDA(c, gemv_launch((const bf16*)w, N, K, (const bf16*)x, rows, (bf16*)y, ldy, epi, c->sm_count, c->stream));
    return OMNI_OK;
  }
  if (!tc_supports(N, K, rows)) return c->fail(OMNI_ERR_UNSUPPORTED, "tensor path needs K %% 64 == 0");
  TcGemmPlan plan;
  const int rc = tc_plan(&plan, (const bf16*)w, N, K, (const bf16*)x, rows, (bf16*)y, ldy, epi, c->sm_count, splits);
  if (rc != 0) return c->fail(OMNI_ERR_CUDA, "tensor-map encode failed (%d)", rc);
  OPS_CUDA(c, tc_launch(plan, c->scratch, c->err, c->stream));
  return OMNI_OK;
}

int32_t omni_op_norm_copy(omni_ops* c, const void* x, const void* w, void* out, void* res, int32_t rows, int32_t dim,
                          float eps) {
  if (!c) return OMNI_ERR_INVALID;
  OPS_CUDA(c, launch_norm_copy((const bf16*)x, (const bf16*)w, (bf16*)out, (bf16*)res, rows, dim, eps, c->stream));
  return OMNI_OK;
}

int32_t omni_op_add_norm(omni_ops* c, const void* x, void* res, const void* w, void* out, int32_t rows, int32_t dim,
                         float eps, int32_t every, int32_t which) {
  if (!c || every < 1 || which < 0 || which >= every) return OMNI_ERR_INVALID;
  OPS_CUDA(c, launch_add_norm((const bf16*)x, (bf16*)res, (const bf16*)w, (bf16*)out, rows, dim, eps, every, which,
                              c->stream));
  return OMNI_OK;
}

int32_t omni_op_silu_mul(omni_ops* c, const void* gate_up, void* act, int32_t rows, int32_t inter) {
  if (!c || inter % 8) return OMNI_ERR_INVALID;
  OPS_CUDA(c, launch_silu_mul((const bf16*)gate_up, (bf16*)act, rows, inter, 0, c->stream));
  return OMNI_OK;
}

int32_t omni_op_rope_attend(omni_ops* c, void* qkv, const void* q_norm, const void* k_norm, void* kv,
                            int32_t kv_pages, const int32_t* pos, const int32_t* slot, const int32_t* seq,
                            const int32_t* indptr, const int32_t* pages, int32_t rows, int32_t q_heads,
                            int32_t kv_heads, int32_t head_dim, float eps, float theta, void* out) {
  if (!c || !pos || !slot || !indptr || !pages) return OMNI_ERR_INVALID;
  RowMap map;
  map.pos = pos;
  map.slot = slot;
  map.seq = seq;
  map.indptr = indptr;
  map.pages = pages;
  const AttnShape a{q_heads, kv_heads, head_dim, eps, theta};
  const size_t head = (size_t)rows * head_dim * sizeof(bf16);
  OPS_CUDA(c, on_aligned_rows(qkv, head * (q_heads + 2 * kv_heads), out, head * q_heads, c->stream, [&](void* x, void* y) {
    const cudaError_t e = launch_rope_kv((bf16*)x, (const bf16*)q_norm, (const bf16*)k_norm, (bf16*)kv, map, rows, a, kv_pages,
                                         c->err, c->stream);
    return e != cudaSuccess ? e : launch_attend((const bf16*)x, (const bf16*)kv, (bf16*)y, map, rows, a, c->err, c->stream);
  }));
  return OMNI_OK;
}

int32_t omni_op_decode_attend(omni_ops* c, const void* qkv, const void* q_norm, const void* k_norm, void* kv,
                              int32_t kv_pages, const int32_t* pos, const int32_t* slot, const int32_t* indptr,
                              const int32_t* pages, int32_t rows, int32_t q_heads, int32_t kv_heads, int32_t head_dim,
                              float eps, float theta, void* out) {
  if (!c || !pos || !slot || !indptr || !pages || rows < 1) return OMNI_ERR_INVALID;
  RowMap map;
  map.pos = pos, map.slot = slot, map.indptr = indptr, map.pages = pages;
  const AttnShape a{q_heads, kv_heads, head_dim, eps, theta};
  OPS_CUDA(c, order(c->stream));
  const size_t head = (size_t)rows * head_dim * sizeof(bf16);
  OPS_CUDA(c, on_aligned_rows(const_cast<void*>(qkv), head * (q_heads + 2 * kv_heads), out, head * q_heads, c->stream, [&](void* x, void* y) {
    return launch_rope_attend((const bf16*)x, {}, (const bf16*)q_norm, (const bf16*)k_norm, (bf16*)kv, (bf16*)y, map, rows, a,
                              kv_pages, c->sm_count, c->err, c->stream);
  }));
  return OMNI_OK;
}

int32_t omni_op_chain_gemm(omni_ops* c, const void* w, int32_t N, int32_t K, const void* x, int32_t rows, void* y,
                           int32_t ldy, const void* bias, int32_t epilogue, int32_t swiglu) {
  if (!c || !w || !x || !y || N < 1 || rows < 1 || !stream_supports(N, K, rows)) return OMNI_ERR_INVALID;
  if (epilogue != OMNI_EPI_NONE && (!bias || swiglu)) return c->fail(OMNI_ERR_INVALID, "epilogue %d needs a bias and no swiglu", epilogue);
  int launches = 0;
  ChainPlans plans;
  const Chain chain{c->stream, c->err, c->sm_count, c->scratch.partials, c->scratch.partial_floats, &launches, &plans};
  if (!swiglu) {
    Epilogue epi;
    epi.bias = static_cast<const bf16*>(bias), epi.kind = epilogue;
    OPS_CUDA(c, order(c->stream));
    OPS_CUDA(c, chain.gemm((const bf16*)w, N, K, (const bf16*)x, rows, kStreamBf16, (bf16*)y, ldy, nullptr, 0, epi));
    return OMNI_OK;
  }
  if (!wide_fuses(N, K, kGateGroup)) return c->fail(OMNI_ERR_UNSUPPORTED, "gate and up rows are no groups of %d", kGateGroup);
  bf16* grouped = nullptr;
  OPS_CUDA(c, cudaMalloc((void**)&grouped, (size_t)N * K * sizeof(bf16)));
  cudaError_t e = launch_interleave_gate_up((const bf16*)w, grouped, N / 2, K, kGateGroup, c->stream);
  if (e == cudaSuccess) e = order(c->stream);  // the GEMM asks for its weights before it waits
  if (e == cudaSuccess) e = chain.gemm(grouped, N, K, (const bf16*)x, rows, kStreamSwiglu, (bf16*)y, ldy);
  const cudaError_t done = cudaStreamSynchronize(c->stream);
  cudaFree(grouped);
  OPS_CUDA(c, e);
  OPS_CUDA(c, done);
  return OMNI_OK;
}

int32_t omni_op_chain_norm_gemm(omni_ops* c, const void* w1, int32_t D, int32_t K, const void* x, int32_t rows,
                                void* res, const void* gain, float eps, const void* w2, int32_t N, void* y) {
  if (!c || !w1 || !x || !res || !gain || !w2 || !y || rows < 1 || rows > kChainRows || !stream_supports(D, K, rows) || D % 64)
    return OMNI_ERR_INVALID;
  int launches = 0;
  ChainPlans plans;
  const Chain chain{c->stream, c->err, c->sm_count, c->scratch.partials, c->scratch.partial_floats, &launches, &plans};
  OPS_CUDA(c, order(c->stream));
  bf16* tmp = nullptr;  // the rows of a norm of its own, the other residual of a folded one
  const size_t row_bytes = (size_t)rows * D * sizeof(bf16);
  OPS_CUDA(c, cudaMalloc((void**)&tmp, 2 * row_bytes));
  bf16 *in = (bf16*)res, *spare = tmp + (size_t)rows * D;
  Summands sum;
  FewNorm norm;
  cudaError_t e = chain.gemm((const bf16*)w1, D, K, (const bf16*)x, rows, kStreamPartials, nullptr, D, &sum);
  norm.kind = kNormStack, norm.sum = sum, norm.gain = (const bf16*)gain, norm.eps = eps;
  if (e == cudaSuccess)
    e = chain.norm_gemm(norm, &in, &spare,
                        [&](const Summands& from, bf16* r) {
                          return launch_add_norm_sum(from, r, (const bf16*)gain, tmp, rows, D, eps, 1, 0, c->stream);
                        },
                        (const bf16*)w2, N, D, tmp, rows, kStreamBf16, (bf16*)y, N);
  if (e == cudaSuccess && in != (bf16*)res) e = cudaMemcpyAsync(res, in, row_bytes, cudaMemcpyDeviceToDevice, c->stream);
  const cudaError_t done = cudaStreamSynchronize(c->stream);
  cudaFree(tmp);
  OPS_CUDA(c, e);
  OPS_CUDA(c, done);
  return OMNI_OK;
}

int32_t omni_op_add_norm_sum(omni_ops* c, const float* part, int32_t splits, void* res, const void* gain, void* out,
                             int32_t rows, int32_t dim, float eps, int32_t lm) {
  if (!c || !part || !res || !gain || !out || splits < 1 || rows < 1 || dim < 1) return OMNI_ERR_INVALID;
  const uintptr_t at = reinterpret_cast<uintptr_t>(part) | reinterpret_cast<uintptr_t>(res) | reinterpret_cast<uintptr_t>(gain) |
                       reinterpret_cast<uintptr_t>(out);
  if (at & 15) return c->fail(OMNI_ERR_INVALID, "rows that are not at 16-byte addresses");
  Summands sum;
  sum.part = part, sum.splits = splits, sum.split_stride = (int64_t)rows * dim, sum.ld = dim;
  OPS_CUDA(c, order(c->stream));  // the gain is read early
  if (lm) OPS_CUDA(c, launch_lm_add_norm_sum(sum, (bf16*)res, (const bf16*)gain, (bf16*)out, rows, dim, eps, c->stream));
  else OPS_CUDA(c, launch_add_norm_sum(sum, (bf16*)res, (const bf16*)gain, (bf16*)out, rows, dim, eps, 1, 0, c->stream));
  return OMNI_OK;
}

int32_t omni_op_sample(omni_ops* c, const void* logits, int32_t vocab, float temperature, int32_t top_k, float top_p,
                       float penalty, int32_t suppress_lo, int32_t suppress_hi, int32_t exempt, int32_t min_frames,
                       const int32_t* frames, const float* uniforms, const int32_t* force, void* state,
                       const int32_t* lines, int64_t stride, int32_t penalize, int32_t philox, int32_t* codes,
                       int32_t group, int32_t rows) {
  if (!c || group < 0 || group >= OMNI_GROUPS) return OMNI_ERR_INVALID;
  SampleParams p{};
  p.vocab = vocab;
  p.temperature = temperature;
  p.top_k = top_k;
  p.top_p = top_p;
  p.penalty = penalty;
  p.suppress_lo = suppress_lo;
  p.suppress_hi = suppress_hi;
  p.exempt = exempt;
  p.min_frames = min_frames;
  p.penalize = penalize;
  p.group = group;
  p.philox = philox;
  p.seen_words = (vocab + 31) / 32;
  if (top_p < 1.f && (top_k <= 0 || top_k > 1024))
    return c->fail(OMNI_ERR_UNSUPPORTED, "top_p < 1 needs 0 < top_k <= 1024 (the nucleus filter ranks the survivors of the top-k cut)");
  OPS_CUDA(c, launch_sample((const bf16*)logits, p, frames, uniforms, force, SlotState{state, lines, stride}, codes,
                            rows, c->stream));
  return OMNI_OK;
}

int32_t omni_op_lm_norm(omni_ops* c, const void* y, void* x, const void* alpha, void* out, int32_t rows, int32_t dim,
                        float eps) {
  if (!c || !x) return OMNI_ERR_INVALID;
  if (y)
    OPS_CUDA(c, launch_lm_add_norm((const bf16*)y, (bf16*)x, (const bf16*)alpha, (bf16*)out, rows, dim, eps, c->stream));
  else
    OPS_CUDA(c, launch_lm_norm((const bf16*)x, (const bf16*)alpha, (bf16*)out, rows, dim, eps, c->stream));
  return OMNI_OK;
}

int32_t omni_op_lm_tp_add_norm(omni_ops* c, const void* mine, const void* peer, void* x, const void* alpha, void* out,
                               int32_t rows, int32_t dim, float eps, void* words) {
  if (!c || !mine || !peer || !x || !words) return OMNI_ERR_INVALID;
  TpLink link;
  uint32_t* w = static_cast<uint32_t*>(words);
  link.my_flag = w, link.peer_flag = w + 16, link.counter = w + 32, link.finished = w + 48;
  OPS_CUDA(c, launch_lm_tp_add_norm((const bf16*)mine, (const bf16*)peer, (bf16*)x, (const bf16*)alpha, (bf16*)out, rows,
                                    dim, eps, link, c->err, c->stream));
  return OMNI_OK;
}

int32_t omni_op_lm_embed(omni_ops* c, const int32_t* ids, const void* text_emb, int32_t text_rows,
                         const void* audio_emb, int32_t card_rows, void* out, int32_t rows, int32_t dim) {
  if (!c || !ids || !out) return OMNI_ERR_INVALID;
  const DuplexTables t{(const bf16*)text_emb, (const bf16*)audio_emb, text_rows, card_rows};
  OPS_CUDA(c, launch_lm_embed_ids(ids, nullptr, nullptr, 0, t, (bf16*)out, rows, dim, c->err, c->stream));
  return OMNI_OK;
}

int32_t omni_op_lm_rope_attend(omni_ops* c, void* qkv, void* kv, int32_t kv_pages, const int32_t* pos,
                               const int32_t* slot, const int32_t* seq, const int32_t* indptr, const int32_t* pages,
                               int32_t rows, int32_t heads, float coef, float scale, int32_t context, void* out) {
  if (!c || !qkv || !kv || !pos || !slot || !indptr || !pages || !out) return OMNI_ERR_INVALID;
  OPS_CUDA(c, launch_lm_rope_kv((bf16*)qkv, pos, slot, kv, rows, heads, coef, kv_pages, c->err, c->stream));
  OPS_CUDA(c, launch_lm_attend((const bf16*)qkv, kv, pos, seq, indptr, pages, (bf16*)out, rows, heads, scale, context,
                               kv_pages, c->err, c->stream));
  return OMNI_OK;
}

int32_t omni_op_lm_decode_attend(omni_ops* c, const void* qkv, void* kv, int32_t kv_pages, const int32_t* pos,
                                 const int32_t* slot, const int32_t* indptr, const int32_t* pages, int32_t rows,
                                 int32_t heads, float coef, float scale, int32_t context, void* out) {
  if (!c || !qkv || !kv || !pos || !slot || !indptr || !pages || !out || rows < 1) return OMNI_ERR_INVALID;
  OPS_CUDA(c, order(c->stream));
  OPS_CUDA(c, launch_lm_rope_attend((const bf16*)qkv, kv, pos, slot, indptr, pages, (bf16*)out, rows, heads, coef, scale, context,
                                    kv_pages, c->sm_count, c->err, c->stream));
  return OMNI_OK;
}

int32_t omni_op_lm_dep_embed_norm(omni_ops* c, const void* projected, int32_t k, const void* table, int32_t table_rows,
                                  const int32_t* drawn, const void* alpha, void* x, void* xn, int32_t rows, int32_t dim,
                                  float eps) {
  if (!c || k < 0 || k >= kDepSteps) return OMNI_ERR_INVALID;
  OPS_CUDA(c, launch_lm_dep_embed_norm((const bf16*)projected, k, (const bf16*)table, table_rows, drawn,
                                       (const bf16*)alpha, (bf16*)x, (bf16*)xn, rows, dim, eps, c->err, c->stream));
  return OMNI_OK;
}

int32_t omni_op_lm_dep_kv_attend(omni_ops* c, const void* qkv, void* ws, int32_t step, void* out, int32_t rows,
                                 int32_t heads, float scale) {
  if (!c) return OMNI_ERR_INVALID;
  OPS_CUDA(c, launch_lm_dep_kv_attend((const bf16*)qkv, (bf16*)ws, step, (bf16*)out, rows, heads, scale, c->stream));
  return OMNI_OK;
}

int32_t omni_op_lm_sample(omni_ops* c, const void* logits, int32_t vocab, int64_t ld, float temperature, int32_t top_k,
                          const int32_t* force, const int32_t* seeds, int32_t col, int32_t* drawn, int32_t rows) {
  if (!c || !logits || !force || !seeds || !drawn) return OMNI_ERR_INVALID;
  OPS_CUDA(c, launch_lm_sample((const bf16*)logits, vocab, ld, temperature, top_k, force, seeds, col, drawn, rows,
                               c->stream));
  return OMNI_OK;
}

int32_t omni_op_lm_advance(omni_ops* c, void* state, const int32_t* lines, int64_t stride, const int32_t* init,
                           const int32_t* drawn, const int32_t* caller, const int32_t* force_caller, int32_t* emitted,
                           int32_t rows) {
  if (!c || !state || !lines) return OMNI_ERR_INVALID;
  if (init) OPS_CUDA(c, launch_lm_init(state, lines, stride, init, rows, c->stream));
  if (drawn) {
    if (!caller || !force_caller || !emitted) return OMNI_ERR_INVALID;
    OPS_CUDA(c, launch_lm_advance(state, lines, stride, drawn, caller, force_caller, emitted, rows, c->stream));
  }
  return OMNI_OK;
}

int32_t omni_op_higgs_frame_embed(omni_ops* c, void* state, const int32_t* lines, int64_t stride, const void* table,
                                  void* out, int32_t rows, int32_t dim, int32_t vocab) {
  if (!c || !state || !lines || !table || !out) return OMNI_ERR_INVALID;
  OPS_CUDA(c, launch_higgs_frame_embed(SlotState{state, lines, stride}, (const bf16*)table, (bf16*)out, rows, dim, vocab,
                                       c->err, c->stream));
  return OMNI_OK;
}

int32_t omni_op_higgs_sample(omni_ops* c, const void* logits, int32_t vocab, float temperature, int32_t top_k,
                             const float* uniforms, const int32_t* force, void* state, const int32_t* lines,
                             int64_t stride, int32_t* codes, int32_t rows) {
  if (!c || !logits || !uniforms || !force || !state || !lines || !codes) return OMNI_ERR_INVALID;
  OPS_CUDA(c, launch_higgs_sample((const bf16*)logits, vocab, temperature, top_k, uniforms, force,
                                  SlotState{state, lines, stride}, codes, rows, c->stream));
  return OMNI_OK;
}

int32_t omni_higgs_delay_forced_from(const omni_higgs_delay* d) {
  return d ? std::min(d->steps + 1, OMNI_HIGGS_BOOKS) : OMNI_ERR_INVALID;
}

int32_t omni_higgs_delay_advance(omni_higgs_delay* d, int32_t first) {
  if (!d) return OMNI_ERR_INVALID;
  if (d->done) return 1;
  if (d->steps < OMNI_HIGGS_BOOKS) {  // the ramp: an end drawn here is not one
    d->steps += 1;
  } else if (d->countdown > 0) {
    d->countdown -= 1;
    d->done = d->countdown <= 1;
    if (d->done) d->countdown = 0;
  } else if (first == OMNI_HIGGS_EOC) {
    d->countdown = OMNI_HIGGS_BOOKS - 2 + 1;  // books - 2 more steps; stored + 1 so that 0 means "not running"
  }
  return d->done;
}

int32_t omni_higgs_undelay(const int32_t* rows, int32_t n_rows, int32_t* frames) {
  if (n_rows < 0 || (n_rows > 0 && (!rows || !frames))) return OMNI_ERR_INVALID;
  const int n = std::max(n_rows - (OMNI_HIGGS_BOOKS - 1), 0);
  for (int t = 0; t < n; ++t)
    for (int b = 0; b < OMNI_HIGGS_BOOKS; ++b) frames[t * OMNI_HIGGS_BOOKS + b] = rows[(t + b) * OMNI_HIGGS_BOOKS + b];
  return n;
}

// ---- streaming codec decoder ---------------------------------------------------------------------------------------

int32_t omni_op_codec_rvq(omni_ops* c, const int32_t* codes, const void* books, void* out, int32_t n, int32_t half,
                          int32_t book_rows) {
  if (!c || !codes || !books || !out || half % 8) return OMNI_ERR_INVALID;
  OPS_CUDA(c, launch_codec_rvq(codes, (const bf16*)books, (bf16*)out, n, half, book_rows, c->stream));
  return OMNI_OK;
}

int32_t omni_op_codec_add_norm(omni_ops* c, const void* add, int64_t add_stride, void* res, const void* w, void* out,
                               int32_t rows, int32_t dim, float eps) {
  if (!c || !add || !res || !w || !out || dim % 256 || dim > 1024) return OMNI_ERR_INVALID;
  OPS_CUDA(c, launch_codec_add_norm((const bf16*)add, add_stride, (bf16*)res, (const bf16*)w, (bf16*)out, rows, dim, eps,
                                    c->stream));
  return OMNI_OK;
}

int32_t omni_op_codec_window_attend(omni_ops* c, const void* qkv, void* state, const int32_t* lines, const int32_t* pos,
                                    int64_t stride, int64_t ring_offset, void* out, int32_t n, int32_t heads, float theta) {
  if (!c || !qkv || !state || !lines || !pos || !out) return OMNI_ERR_INVALID;
  OPS_CUDA(c, order(c->stream));
  OPS_CUDA(c, launch_codec_window_attend((const bf16*)qkv, CodecStateRef{(char*)state, lines, pos, stride}, ring_offset,
                                         (bf16*)out, n, heads, theta, c->stream));
  return OMNI_OK;
}

int32_t omni_op_codec_bias_gelu(omni_ops* c, void* x, const void* bias, int64_t rows, int32_t cols) {
  if (!c || !x || !bias || cols % 8) return OMNI_ERR_INVALID;
  OPS_CUDA(c, launch_codec_bias_gelu((bf16*)x, (const bf16*)bias, rows, cols, c->stream));
  return OMNI_OK;
}

int32_t omni_op_codec_bias_snake(omni_ops* c, const void* x, const void* bias, const float* alpha, const float* inv_b,
                                 void* out, int64_t rows, int32_t cols) {
  if (!c || !x || !bias || !alpha || !inv_b || !out || cols % 8) return OMNI_ERR_INVALID;
  OPS_CUDA(c, launch_codec_bias_snake((const bf16*)x, (const bf16*)bias, alpha, inv_b, (bf16*)out, rows, cols, c->stream));
  return OMNI_OK;
}

int32_t omni_op_codec_stage(omni_ops* c, const void* x, const void* bias, const float* alpha, const float* inv_b,
                            void* state, const int32_t* lines, const int32_t* pos, int64_t stride, int64_t hist_offset,
                            void* padded, int32_t n, int32_t T, int32_t C, int32_t H) {
  if (!c || !x || !bias || !state || !lines || !pos || !padded || C % 8 || (alpha != nullptr) != (inv_b != nullptr))
    return OMNI_ERR_INVALID;
  OPS_CUDA(c, launch_codec_stage((const bf16*)x, (const bf16*)bias, alpha, inv_b, CodecStateRef{(char*)state, lines, pos, stride},
                                 hist_offset, (bf16*)padded, n, T, C, H, c->stream));
  return OMNI_OK;
}

int32_t omni_op_codec_gather_taps(omni_ops* c, const void* padded, void* col, int32_t n, int32_t T, int32_t C,
                                  int32_t taps, int32_t dil) {
  if (!c || !padded || !col || C % 8) return OMNI_ERR_INVALID;
  OPS_CUDA(c, launch_codec_gather_taps((const bf16*)padded, (bf16*)col, n, T, C, taps, dil, c->stream));
  return OMNI_OK;
}

int32_t omni_op_codec_conv(omni_ops* c, const void* w, int32_t N, int32_t C, int32_t taps, int32_t dil, const void* padded,
                           int32_t T, int32_t n_streams, void* y, int32_t epilogue, const void* bias, const float* alpha,
                           const float* inv_b) {
  if (!c || !w || !padded || !y || epilogue < 0 || epilogue > 2) return OMNI_ERR_INVALID;
  if (epilogue == kConvBiasSnake && (!bias || !alpha || !inv_b)) return OMNI_ERR_INVALID;
  conv_configure();
  ConvGemmPlan plan;
  const int rc = conv_plan(&plan, (const bf16*)w, N, C, taps, dil, (const bf16*)padded, T, n_streams, (bf16*)y, epilogue,
                           (const bf16*)bias, alpha, inv_b, c->sm_count);
  if (rc != 0) return c->fail(OMNI_ERR_UNSUPPORTED, "conv plan refused (%d): N=%d C=%d taps=%d T=%d", rc, N, C, taps, T);
  OPS_CUDA(c, order(c->stream));
  OPS_CUDA(c, conv_launch(plan, c->err, c->stream));
  return OMNI_OK;
}

int32_t omni_op_codec_overlap_add(omni_ops* c, const void* z, const void* bias, void* state, const int32_t* lines,
                                  const int32_t* pos, int64_t stride, int64_t prev_offset, void* out, int32_t n, int32_t L,
                                  int32_t r, int32_t C) {
  if (!c || !z || !bias || !state || !lines || !out || C % 8) return OMNI_ERR_INVALID;
  OPS_CUDA(c, launch_codec_overlap_add((const bf16*)z, (const bf16*)bias, CodecStateRef{(char*)state, lines, pos, stride},
                                       prev_offset, (bf16*)out, n, L, r, C, c->stream));
  return OMNI_OK;
}

int32_t omni_op_codec_dwconv_ln(omni_ops* c, const void* z, const void* zb, const void* w, const void* b, const void* ln_w,
                                const void* ln_b, void* state, const int32_t* lines, const int32_t* pos, int64_t stride,
                                int64_t hist_offset, void* xin, void* out, int32_t n, int32_t T, int32_t r, int32_t C,
                                float eps) {
  if (!c || !z || !zb || !w || !b || !ln_w || !ln_b || !state || !lines || !pos || !xin || !out || C % 8 || C > 8192)
    return OMNI_ERR_INVALID;
  OPS_CUDA(c, launch_codec_dwconv_ln((const bf16*)z, (const bf16*)zb, (const bf16*)w, (const bf16*)b, (const bf16*)ln_w,
                                     (const bf16*)ln_b, CodecStateRef{(char*)state, lines, pos, stride}, hist_offset,
                                     (bf16*)xin, (bf16*)out, n, T, r, C, eps, c->stream));
  return OMNI_OK;
}

int32_t omni_op_codec_out_conv(omni_ops* c, const void* x, const void* bias, const float* alpha, const float* inv_b,
                               const void* w, const void* wb, void* state, const int32_t* lines, const int32_t* pos,
                               int64_t stride, int64_t hist_offset, float* wav, int32_t n, int32_t T, int32_t C) {
  if (!c || !x || !bias || !alpha || !inv_b || !w || !wb || !state || !lines || !pos || !wav || T % 64 || C % 32 || C > 128)
    return OMNI_ERR_INVALID;
  OPS_CUDA(c, launch_codec_out_conv((const bf16*)x, (const bf16*)bias, alpha, inv_b, (const bf16*)w, (const bf16*)wb,
                                    CodecStateRef{(char*)state, lines, pos, stride}, hist_offset, wav, n, T, C, c->stream));
  return OMNI_OK;
}

}  // extern "C"
