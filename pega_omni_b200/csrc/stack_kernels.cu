// Decoder-stack kernels that are not GEMMs: RMSNorm with the residual stream,
// SwiGLU, per-head q/k norm + rotary embedding + KV write, and decode attention
// over the paged KV. Rounding points follow the reference's kernels
// (crates/omni-qwen3/kernels/qwen3.cu, crates/omni-kern/kernels/common.cuh):
// every tensor that crosses HBM is bf16, arithmetic is f32.
#include <type_traits>

#include "attend.cuh"
#include "decode_attend.cuh"
#include "kernels.h"
#include "pdl.cuh"
#include "prompt_attend.cuh"
#include "rope.cuh"
#include "sampler.cuh"

namespace omni {

// ---- RMSNorm + residual ------------------------------------------------------

// One block per row, eight elements a thread. Semantics of `qwen3_norm_copy`
// (qwen3.cu:18-31).
__global__ void norm_copy_kernel(const bf16* x, const bf16* __restrict__ w, bf16* __restrict__ out,
                                 bf16* __restrict__ res, int dim, float eps) {
  grid_trigger();
  grid_wait();
  __shared__ float scratch[32];
  const int64_t at = (int64_t)blockIdx.x * dim + threadIdx.x * 8;
  const bool on = threadIdx.x * 8 < dim;
  float v[8] = {}, g[8];
  if (on) ld8cg(x + at, v);
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) ss += v[k] * v[k];
  const float r = rsqrtf(block_add(ss, scratch) / dim + eps);
  if (!on) return;
  st8(res + at, v);
  ld8(w + threadIdx.x * 8, g);
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = v[k] * r * g[k];
  st8(out + at, v);
}

// Semantics of `qwen3_add_norm` (qwen3.cu:37-57): the residual is stored
// rounded, the norm is taken over the unrounded sum.
__global__ void add_norm_kernel(const bf16* x, bf16* res, const bf16* __restrict__ w, bf16* out, int dim, float eps, int every, int which) {
  grid_trigger();
  grid_wait();
  __shared__ float scratch[32];
  const int n = blockIdx.x;
  const int64_t at = (int64_t)n * dim + threadIdx.x * 8;
  const bool on = threadIdx.x * 8 < dim;
  float v[8] = {}, rv[8] = {}, g[8];
  if (on) {
    ld8cg(x + at, v);  // (out may be x)
    ld8cg(res + at, rv);
  }
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    v[k] += rv[k];
    ss += v[k] * v[k];
  }
  const float r = rsqrtf(block_add(ss, scratch) / dim + eps);
  if (!on) return;
  st8(res + at, v);
  if (n % every != which) return;
  ld8(w + threadIdx.x * 8, g);
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = v[k] * r * g[k];
  st8(out + (int64_t)(n / every) * dim + threadIdx.x * 8, v);
}

// `silu_mul` (common.cuh:66-76). With `interleaved` = g > 0, the fused row alternates g gate channels and the matching
// g up channels (the weight layout the tensor-core SwiGLU epilogue wants) instead of [all gate | all up].
__global__ void silu_mul_kernel(const bf16* gate_up, bf16* __restrict__ act, int inter, int total,
                                int interleaved) {
  grid_trigger();
  grid_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int64_t n = i / (inter / 8), c = i % (inter / 8) * 8;
  float g[8], u[8];
  const int64_t g_at = interleaved ? (c / interleaved) * 2 * interleaved + c % interleaved : c;
  const int64_t u_at = interleaved ? g_at + min((int64_t)interleaved, inter - c / interleaved * interleaved) : inter + c;
  ld8cg(gate_up + n * 2 * inter + g_at, g);
  ld8cg(gate_up + n * 2 * inter + u_at, u);
#pragma unroll
  for (int k = 0; k < 8; ++k) g[k] = bf16_round(g[k] / (1.f + __expf(-g[k]))) * u[k];
  st8(act + (int64_t)i * 8, g);
}

// add_norm over a GEMM's S summands: a thread owns E columns, and its loads - the partial sums, the residual, the
// gain - are under way together, so the kernel is one L2 round trip and one block reduction long (eight sums of four or eight
// columns are more than the 32 and 46 registers that the compiler gives them: it loads those in batches, a round trip each).
// What is left is the number of instructions, executed once: the counts of summands and columns are template arguments.
template <int S, int E>
__global__ void add_norm_sum_kernel(const Summands x, bf16* __restrict__ res, const bf16* __restrict__ w,
                                    bf16* __restrict__ out, int dim, float eps, int every, int which) {
  grid_trigger();
  __shared__ float scratch[32];
  const int n = blockIdx.x, c = threadIdx.x * E, lane = threadIdx.x & 31;
  const bool on = c < dim;  // the block is a whole number of warps
  float g[E], v[E], rv[E], ss = 0.f;
  if (on) Run<E>::ld(w + c, g);
  grid_wait();
  if (on) {
    Run<E>::ldcg(res + (int64_t)n * dim + c, rv);
    load_sum<S, E>(x, n, c, v);
#pragma unroll
    for (int k = 0; k < E; ++k) {
      v[k] += rv[k];
      ss += v[k] * v[k];
    }
    Run<E>::st(res + (int64_t)n * dim + c, v);
  }
  ss = warp_add(ss);
  if (lane == 0) scratch[threadIdx.x >> 5] = ss;
  if (n % every != which) return;
  __syncthreads();
  const float r = rsqrtf(warp_add(lane < (int)blockDim.x >> 5 ? scratch[lane] : 0.f) / dim + eps);
  if (!on) return;
#pragma unroll
  for (int k = 0; k < E; ++k) v[k] = v[k] * r * g[k];
  Run<E>::st(out + (int64_t)(n / every) * dim + c, v);
}

cudaError_t launch_add_norm_sum(const Summands& x, bf16* res, const bf16* w, bf16* out, int rows, int dim, float eps,
                                int every, int which, cudaStream_t s) {
  if (dim % 8 || dim / 8 > 1024) return cudaErrorInvalidValue;
  return with_summands(x.splits, [&](auto sums) {
    return with_columns(dim, rows, [&](auto columns) {
      constexpr int E = decltype(columns)::value;
      return launch_pdl(add_norm_sum_kernel<decltype(sums)::value, E>, dim3(rows), dim3((dim + E * 32 - 1) / (E * 32) * 32), 0, s, x, res, w, out, dim, eps,
                        every, which);
    });
  });
}

__global__ void interleave_gate_up_kernel(const bf16* __restrict__ src, bf16* __restrict__ dst, int inter, int k,
                                          int granule) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;  // one 16-byte piece
  const int64_t per_row = k / 8, total = (int64_t)2 * inter * per_row;
  if (i >= total) return;
  const int64_t row = i / per_row, piece = i % per_row;
  const bool up = row >= inter;
  const int c = (int)(up ? row - inter : row), group = c / granule;
  const int64_t out_row = (int64_t)group * 2 * granule + (up ? min(granule, inter - group * granule) : 0) + c % granule;
  *reinterpret_cast<uint4*>(dst + out_row * k + piece * 8) = *reinterpret_cast<const uint4*>(src + row * k + piece * 8);
}

cudaError_t launch_interleave_gate_up(const bf16* src, bf16* dst, int inter, int k, int granule, cudaStream_t s) {
  if (k % 8 || granule < 1) return cudaErrorInvalidValue;
  const int64_t pieces = (int64_t)2 * inter * (k / 8);
  interleave_gate_up_kernel<<<(unsigned)((pieces + 255) / 256), 256, 0, s>>>(src, dst, inter, k, granule);
  return cudaGetLastError();
}

cudaError_t launch_norm_copy(const bf16* x, const bf16* w, bf16* out, bf16* res, int rows, int dim, float eps,
                             cudaStream_t s) {
  if (dim % 8 || dim / 8 > 1024) return cudaErrorInvalidValue;
  return launch_pdl(norm_copy_kernel, dim3(rows), dim3(row_threads(dim)), 0, s, x, w, out, res, dim, eps);
}

cudaError_t launch_add_norm(const bf16* x, bf16* res, const bf16* w, bf16* out, int rows, int dim, float eps,
                            int every, int which, cudaStream_t s) {
  if (dim % 8 || dim / 8 > 1024) return cudaErrorInvalidValue;
  return launch_pdl(add_norm_kernel, dim3(rows), dim3(row_threads(dim)), 0, s, x, res, w, out, dim, eps, every, which);
}

cudaError_t launch_silu_mul(const bf16* gate_up, bf16* act, int rows, int inter, int interleaved, cudaStream_t s) {
  const int total = rows * (inter / 8);
  if (interleaved && (inter % 8 || interleaved % 8)) return cudaErrorInvalidValue;
  return launch_pdl(silu_mul_kernel, dim3((total + 255) / 256), dim3(256), 0, s, gate_up, act, inter, total, interleaved);
}

// ---- row -> (sequence, position, page) -----------------------------------------

struct RowAt {
  int seq, pos;
  int64_t slot;            // page * 16 + pos % 16 of the row's own token
  const int32_t* pages;    // the sequence's page list, or nullptr when dense
};

__device__ __forceinline__ RowAt locate(const RowMap& m, int n) {
  RowAt r;
  if (m.pages) {
    r.seq = m.seq ? m.seq[n] : n;
    r.pos = m.pos[n];
    r.slot = m.slot ? m.slot[n] : 0;
    r.pages = m.pages + m.indptr[r.seq];
  } else {
    r.seq = n / m.per;
    r.pos = m.base + n % m.per;
    r.slot = (int64_t)r.seq * 16 + r.pos;
    r.pages = nullptr;
  }
  return r;
}

// A lane's E elements of each half of a head, E = D / 64.
template <int D>
__device__ __forceinline__ void st_half(bf16* dst, int lane, const float (&lo)[D / 64], const float (&hi)[D / 64]) {
  if constexpr (D == 128) {
    reinterpret_cast<__nv_bfloat162*>(dst)[lane] = __floats2bfloat162_rn(lo[0], lo[1]);
    reinterpret_cast<__nv_bfloat162*>(dst)[32 + lane] = __floats2bfloat162_rn(hi[0], hi[1]);
  } else {
    dst[lane] = __float2bfloat16(lo[0]), dst[32 + lane] = __float2bfloat16(hi[0]);
  }
}

// ---- q/k norm + RoPE + KV write -------------------------------------------------

// A CTA per row, a warp per head at a time: a lane's rotation angles depend on the row alone, so they are computed once
// and serve all the heads the warp takes (a powf and a sincosf per head cost four times the memory traffic:
// 87 us a layer at 8,700 rows of 32 heads; 57 us with one head's loads at a time). Semantics of `rope_kv` (qwen3.cu:66-107): RMSNorm over the head, the
// normalised value rounded to bf16 before the gain, half-rotation rotary embedding with inv_freq = theta^(-2i/D); q stays
// in place, k and v go to the row's slot.
template <int D>
__global__ void __launch_bounds__(256) rope_kv_kernel(bf16* __restrict__ qkv, const bf16* __restrict__ q_norm,
                                                      const bf16* __restrict__ k_norm, bf16* __restrict__ kv,
                                                      RowMap map, int hq, int hk, float eps, float theta,
                                                      int kv_pages, uint32_t* err) {
  constexpr int E = D / 64;  // elements of each half a lane owns
  grid_trigger();
  const int n = blockIdx.x, lane = threadIdx.x & 31;
  const RowAt at = locate(map, n);
  float cs[E], sn[E], qlo[E], qhi[E], klo[E], khi[E];
  rope_angles<D>(lane, at.pos, theta, cs, sn);
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int i = lane * E + e;
    qlo[e] = __bfloat162float(q_norm[i]), qhi[e] = __bfloat162float(q_norm[D / 2 + i]);
    klo[e] = __bfloat162float(k_norm[i]), khi[e] = __bfloat162float(k_norm[D / 2 + i]);
  }
  grid_wait();
  const int64_t page = at.slot >> 4;
  const int tok = (int)(at.slot & 15);
  if (page < 0 || page >= kv_pages) {
    if (threadIdx.x == 0) raise(err, kErrBadIndex);
    return;
  }
  // four heads of a warp at a time: their loads are all under way before the first is used
  constexpr int B = 4;
  const int heads = hq + 2 * hk, warps = blockDim.x >> 5;
  bf16* const row = qkv + (int64_t)n * heads * D;
  using Half = std::conditional_t<E == 2, uint32_t, uint16_t>;  // a lane's elements of half a head
  for (int h0 = threadIdx.x >> 5; h0 < heads; h0 += B * warps) {
    Half raw[B][2];
#pragma unroll
    for (int b = 0; b < B; ++b) {
      const int head = h0 + b * warps;
      if (head < heads) {
        const Half* src = reinterpret_cast<const Half*>(row + head * D);
        raw[b][0] = __ldcg(src + lane), raw[b][1] = __ldcg(src + 32 + lane);
      }
    }
#pragma unroll
    for (int b = 0; b < B; ++b) {
      const int head = h0 + b * warps;
      if (head >= heads) break;
      float lo[E], hi[E];
      lo[0] = __uint_as_float((uint32_t)raw[b][0] << 16), hi[0] = __uint_as_float((uint32_t)raw[b][1] << 16);
      if constexpr (E == 2) lo[1] = __uint_as_float(raw[b][0] & 0xffff0000u), hi[1] = __uint_as_float(raw[b][1] & 0xffff0000u);
      if (head < hq) rope_head<D>(lo, hi, qlo, qhi, cs, sn, eps);
      else if (head < hq + hk) rope_head<D>(lo, hi, klo, khi, cs, sn, eps);
      bf16* dst = head < hq ? row + head * D : kv + kv_offset<D>(page, hk, (head - hq) % hk, head >= hq + hk, tok);
      st_half<D>(dst, lane, lo, hi);
    }
  }
}

cudaError_t launch_rope_kv(bf16* qkv, const bf16* q_norm, const bf16* k_norm, bf16* kv, const RowMap& map, int rows,
                           const AttnShape& a, int kv_pages, uint32_t* err, cudaStream_t s) {
  auto go = [&](auto kernel) {
    return launch_pdl(kernel, dim3(rows), dim3(256), 0, s, qkv, q_norm, k_norm, kv, map, a.q_heads, a.kv_heads, a.rms_eps,
                      a.rope_theta, kv_pages, err);
  };
  if (a.head_dim == 128) return go(rope_kv_kernel<128>);
  if (a.head_dim == 64) return go(rope_kv_kernel<64>);
  return cudaErrorInvalidValue;
}

// ---- decode attention -------------------------------------------------------------
// The page loop lives in attend.cuh; here one CTA of four warps handles one (row, kv head). Every warp owns
// kAttnSlots staging slots in dynamic shared memory: its K|V blocks arrive through bulk copies, kAttnSlots of them
// ahead of the block it is working on.

constexpr int kAttnSlots = 1;

template <int D, int G>
__global__ void __launch_bounds__(kAttnWarps * 32) attend_kernel(const bf16* qkv, const bf16* kv, bf16* __restrict__ out,
                                                                 RowMap map, int hq, int hk, float scale, uint32_t* err) {
  grid_trigger();
  grid_wait();
  extern __shared__ __align__(128) unsigned char attend_slots[];
  __shared__ AttnShared<D, G> sh;
  __shared__ __align__(8) uint64_t bars[kAttnWarps * kAttnSlots];
  const int n = blockIdx.x, kh = blockIdx.y;
  const RowAt at = locate(map, n);
  const bf16* q = qkv + ((int64_t)n * (hq + 2 * hk) + kh * G) * D;
  if (threadIdx.x < kAttnWarps * kAttnSlots) sm100::mbar_init(sm100::smem_addr(&bars[threadIdx.x]), 1);
  if (threadIdx.x == 0) sm100::mbar_init_fence();
  for (int i = threadIdx.x; i < G * D; i += blockDim.x) sh.qs[i / D][i % D] = __bfloat162float(__ldcg(q + i));
  __syncthreads();
  const int warp = threadIdx.x >> 5;
  sm100::fence_async_global();  // keys and values written by ordinary stores, read by bulk copies
  PageStage<kAttnSlots> stage{attend_slots + (size_t)warp * kAttnSlots * kv_block_bytes<D>(), bars + warp * kAttnSlots, 0u, err};
  attend_pages<D, G, kAttnWarps>(sh, kv, at.pages, at.seq, at.pos + 1, hk, kh, scale, out + ((int64_t)n * hq + kh * G) * D,
                                 threadIdx.x, sampler::CtaSync(), &stage);
}

template <int D, int G>
static cudaError_t launch_attend_dg(const bf16* qkv, const bf16* kv, bf16* out, const RowMap& map, int rows, int hq, int hk,
                                    uint32_t* err, cudaStream_t s) {
  if (map.seq && map.pages) {  // rows of prompts: sequences with several rows each
    constexpr int bytes = pattn::kStages * pattn::stage_bytes<D>();
    const cudaError_t e = cudaFuncSetAttribute(pattn::prompt_attend_kernel<D, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    return launch_pdl(pattn::prompt_attend_kernel<D, G>, dim3((rows + pattn::kRows - 1) / pattn::kRows, hk), dim3(pattn::kRows * G * 2),
                      bytes, s, qkv, kv, out, map, rows, hq, hk, 1.f / sqrtf((float)D));
  }
  constexpr size_t smem = (size_t)kAttnWarps * kAttnSlots * kv_block_bytes<D>();
  if (smem + sizeof(AttnShared<D, G>) > 40 * 1024) {  // per device and instantiation: above the default limit of dynamic shared memory
    static bool raised[64] = {};
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return cudaErrorInvalidDevice;
    if (!raised[device]) {
      const cudaError_t e = cudaFuncSetAttribute(attend_kernel<D, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
      raised[device] = true;
    }
  }
  return launch_pdl(attend_kernel<D, G>, dim3(rows, hk), dim3(kAttnWarps * 32), smem, s, qkv, kv, out, map, hq, hk,
                    1.f / sqrtf((float)D), err);
}

template <int D>
static cudaError_t launch_attend_d(const bf16* qkv, const bf16* kv, bf16* out, const RowMap& map, int rows,
                                   const AttnShape& a, uint32_t* err, cudaStream_t s) {
  const int hq = a.q_heads, hk = a.kv_heads;
  switch (hq / hk) {
    case 1: return launch_attend_dg<D, 1>(qkv, kv, out, map, rows, hq, hk, err, s);
    case 2: return launch_attend_dg<D, 2>(qkv, kv, out, map, rows, hq, hk, err, s);
    case 4: return launch_attend_dg<D, 4>(qkv, kv, out, map, rows, hq, hk, err, s);
    case 5: return launch_attend_dg<D, 5>(qkv, kv, out, map, rows, hq, hk, err, s);
    case 8: return launch_attend_dg<D, 8>(qkv, kv, out, map, rows, hq, hk, err, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_attend(const bf16* qkv, const bf16* kv, bf16* out, const RowMap& map, int rows, const AttnShape& a,
                          uint32_t* err, cudaStream_t s) {
  if (a.q_heads % a.kv_heads) return cudaErrorInvalidValue;
  if (a.head_dim == 128) return launch_attend_d<128>(qkv, kv, out, map, rows, a, err, s);
  if (a.head_dim == 64) return launch_attend_d<64>(qkv, kv, out, map, rows, a, err, s);
  return cudaErrorInvalidValue;
}

// ---- decode: q/k norm + RoPE + KV write + attention in one kernel ------------------------------------------------
// A CTA of W warps per (sequence, kv head) of paged rows. The G query heads, the key and the value of a row are dealt to the
// warps; q, k and v go to shared memory (k and v also to the row's slot), and the CTA attends to them with the page step
// of decode_attend.cuh, each warp on its own pages. A page is 16 loads of 16 bytes a lane, straight into registers.
// A warp's first page is asked for before grid_wait() - what earlier calls wrote does not depend on the
// projection this kernel waits for - and the row's own token is patched in from shared memory. The page after the one that is
// on its way to registers is on its way to L2: one pass without and with that, us: a talker step of 1 session 1,895 and 1,881,
// of 8 2,564 and 2,551, of 64 3,448 and 3,430, of 128 4,813 and 4,748 (two pages ahead 4,782, four 4,831).

template <int D>
struct RopeShared {
  alignas(16) bf16 q[8][D];
  alignas(16) bf16 k[D];
  alignas(16) bf16 v[D];
};
template <int D, int G, int W>
struct MergeShared {
  float m[W][8], l[W][8];
  float o[W][G][D];
};

// Resident CTAs an SM: registers for one page in a lane's hands and the next on its way.
constexpr int rope_attend_ctas(int W) { return W == 8 ? 1 : 12 / W; }

// A lane's elements of both halves of a head, as they lie in memory.
template <int D>
__device__ __forceinline__ void ld_halves(const bf16* src, int lane, uint32_t (&raw)[2]) {
  using Half = std::conditional_t<D == 128, uint32_t, uint16_t>;
  raw[0] = __ldcg(reinterpret_cast<const Half*>(src) + lane), raw[1] = __ldcg(reinterpret_cast<const Half*>(src + D / 2) + lane);
}
template <int D>
__device__ __forceinline__ void widen_halves(const uint32_t (&raw)[2], float (&lo)[D / 64], float (&hi)[D / 64]) {
  lo[0] = __uint_as_float(raw[0] << 16), hi[0] = __uint_as_float(raw[1] << 16);
  if constexpr (D == 128) lo[1] = __uint_as_float(raw[0] & 0xffff0000u), hi[1] = __uint_as_float(raw[1] & 0xffff0000u);
}

template <int D, int G, int W>
__global__ void __launch_bounds__(W * 32, rope_attend_ctas(W))
    rope_attend_kernel(const bf16* qkv, const bf16* __restrict__ q_norm, const bf16* __restrict__ k_norm, bf16* kv,
                       bf16* __restrict__ out, RowMap map, int hq, int hk, float eps, float theta, float scale, int kv_pages,
                       uint32_t* err) {
  constexpr int E = D / 64;
  grid_trigger();
  __shared__ RopeShared<D> sh;
  __shared__ MergeShared<D, G, W> merge;
  const int lane = threadIdx.x & 31, warp = warp_index();
  const int at = blockIdx.x / hk, n = map.order ? map.order[at] : at, kh = blockIdx.x % hk;
  float qwl[E], qwh[E], kwl[E], kwh[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    qwl[e] = __bfloat162float(q_norm[lane * E + e]), qwh[e] = __bfloat162float(q_norm[D / 2 + lane * E + e]);
    kwl[e] = __bfloat162float(k_norm[lane * E + e]), kwh[e] = __bfloat162float(k_norm[D / 2 + lane * E + e]);
  }
  for (int i = warp * 32 + lane; i < (8 - G) * D / 8; i += W * 32)  // heads past G: zero rows
    *reinterpret_cast<uint4*>(&sh.q[G][0] + i * 8) = make_uint4(0u, 0u, 0u, 0u);
  const int32_t* pages = map.pages + map.indptr[n];
  dattn::Page<D> pg;
  dattn::State<D> st;
  const int pos = map.pos[n], npages = (pos + 16) >> 4, last = npages - 1;
  float cs[E], sn[E];
  rope_angles<D>(lane, pos, theta, cs, sn);
  const int64_t slot = map.slot[n];
  int64_t own = slot >> 4;
  const int tok = (int)(slot & 15);
  const bool owned = own >= 0 && own < kv_pages;  // otherwise the row stores nothing: page 0 is somebody's
  if (!owned) {
    if (warp == 0 && lane == 0) raise(err, kErrBadIndex);
    own = 0;
  }
  auto block = [&](int pi) {
    int64_t page = pi == last ? own : pages[pi];
    if (page < 0 || page >= kv_pages) {
      if (lane == 0) raise(err, kErrBadIndex);
      page = 0;
    }
    return kv + kv_offset<D>(page, hk, kh, 0, 0);
  };
  auto ask = [&](int pi) {
    if (lane == 0 && pi < npages) sm100::prefetch_l2(block(pi), kv_block_bytes<D>());
  };
  if (warp < npages) pg.load(block(warp), lane);
  ask(warp + W);
  grid_wait();
  const bf16* row = qkv + (int64_t)n * ((hq + 2 * hk) * D);
  constexpr int JOBS = (G + 2 + W - 1) / W;
  uint32_t raw[JOBS][2];
#pragma unroll
  for (int jj = 0; jj < JOBS; ++jj) {  // every head of this warp's share is asked for before the first is used
    const int job = warp + jj * W;
    if (job < G + 2) ld_halves<D>(row + (job < G ? kh * G + job : job == G ? hq + kh : hq + hk + kh) * D, lane, raw[jj]);
  }
#pragma unroll
  for (int jj = 0; jj < JOBS; ++jj) {
    const int job = warp + jj * W;
    if (job >= G + 2) continue;
    float lo[E], hi[E];
    widen_halves<D>(raw[jj], lo, hi);
    if (job < G) rope_head<D>(lo, hi, qwl, qwh, cs, sn, eps);
    else if (job == G) rope_head<D>(lo, hi, kwl, kwh, cs, sn, eps);
    st_half<D>(job < G ? sh.q[job] : job == G ? sh.k : sh.v, lane, lo, hi);
    if (job >= G && owned) st_half<D>(kv + kv_offset<D>(own, hk, kh, job - G, tok), lane, lo, hi);
  }
  __syncthreads();
  uint4 q[D / 32];
#pragma unroll
  for (int j = 0; j < D / 32; ++j) q[j] = *reinterpret_cast<const uint4*>(sh.q[lane >> 2] + 8 * (lane & 3) + 32 * j);
  st.reset();
  for (int pi = warp; pi < npages; pi += W) {
    if (pi == last) pg.patch(tok, sh.k, sh.v, lane);
    ask(pi + 2 * W);
    st.step(pg, q, min(16, pos + 1 - pi * 16), scale, lane, pi + W < npages ? block(pi + W) : nullptr);
  }
  st.finish();
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int h = 0; h < 2; ++h)
    if (2 * t + h < G) {
      if (g == 0) merge.m[warp][2 * t + h] = st.m[h], merge.l[warp][2 * t + h] = st.l[h];
#pragma unroll
      for (int i = 0; i < D / 64; ++i) {
        float v[8];
        st.dims8(i, h, v);
        float4* dst = reinterpret_cast<float4*>(&merge.o[warp][2 * t + h][64 * i + 8 * g]);
        dst[0] = make_float4(v[0], v[1], v[2], v[3]), dst[1] = make_float4(v[4], v[5], v[6], v[7]);
      }
    }
  __syncthreads();
  // a warp per head and 64 dims at a time; lane w has the weight of warp w's state (0 where it held no page)
  for (int i = warp; i < G * (D / 64); i += W) {
    const int h = i / (D / 64), d = i % (D / 64) * 64 + 2 * lane;
    const float mw = lane < W ? merge.m[lane][h] : -INFINITY;
    const float e = __expf(mw - warp_fmax(mw));
    const float den = warp_add(lane < W ? e * merge.l[lane][h] : 0.f);
    float o0 = 0.f, o1 = 0.f;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      const float ew = __shfl_sync(0xffffffffu, e, w);
      const float2 o = *reinterpret_cast<const float2*>(&merge.o[w][h][d]);
      o0 += ew * o.x, o1 += ew * o.y;
    }
    const float inv = 1.f / den;
    *reinterpret_cast<__nv_bfloat162*>(out + ((int64_t)n * hq + kh * G + h) * D + d) = __floats2bfloat162_rn(o0 * inv, o1 * inv);
  }
}

// The same for dense frames (the predictor: one page a sequence, one row or the first two of it at once). What is behind the
// wait runs once, at five to six cycles an instruction, so four warps share a (row, kv head): each makes some of the q, k and v
// heads and brings a quarter of the page, all weigh the keys, each sums a quarter of the values' dims. The queries are the M of
// m16n8k16 (rows past G are zero), keys and then dims the N: a lane has one head's scores, and its probabilities are
// the next product's operand as they are. Shared-memory rows are 16 bytes apart modulo 128, so no ldmatrix has a bank conflict.
template <int D, int G>
__global__ void __launch_bounds__(128)
    frame_attend_kernel(const bf16* qkv, const QkvTable lookup, const bf16* __restrict__ q_norm, const bf16* __restrict__ k_norm,
                        bf16* kv, bf16* __restrict__ out, int base, int hq, int hk, float eps, float theta, float scale,
                        int kv_pages, uint32_t* err) {
  constexpr int E = D / 64, W = 4, P = D + 8;
  grid_trigger();
  extern __shared__ __align__(16) bf16 frame_rows[];  // rows of P: zeros, the G queries, the keys 0..pos, their values
  static_assert(P * 2 % 16 == 0);
  const int lane = threadIdx.x & 31, warp = warp_index();
  const int seq = blockIdx.x / hk, kh = blockIdx.x % hk, r = blockIdx.y, per = gridDim.y;
  const int n = seq * per + r, pos = base + r;
  bf16* const qs = frame_rows + P;
  bf16* const kvs[2] = {qs + G * P, qs + (G + 1 + pos) * P};
  float cs[E], sn[E], cs0[E], sn0[E], qwl[E], qwh[E], kwl[E], kwh[E];
  rope_angles<D>(lane, pos, theta, cs, sn);
  if (r > 0) rope_angles<D>(lane, pos - 1, theta, cs0, sn0);  // the row before is this CTA's key, too
#pragma unroll
  for (int e = 0; e < E; ++e) {
    qwl[e] = __bfloat162float(q_norm[lane * E + e]), qwh[e] = __bfloat162float(q_norm[D / 2 + lane * E + e]);
    kwl[e] = __bfloat162float(k_norm[lane * E + e]), kwh[e] = __bfloat162float(k_norm[D / 2 + lane * E + e]);
  }
  if (threadIdx.x < P / 8) *reinterpret_cast<uint4*>(frame_rows + threadIdx.x * 8) = make_uint4(0u, 0u, 0u, 0u);
  const bool owned = seq < kv_pages;  // otherwise the row stores nothing: page 0 is somebody's
  if (!owned && threadIdx.x == 0) raise(err, kErrBadIndex);
  bf16* const page = kv + kv_offset<D>(owned ? seq : 0, hk, kh, 0, 0);
  grid_wait();

  constexpr int JOBS = (G + 4 + W - 1) / W;
  const int jobs = G + 2 + 2 * r, width = (hq + 2 * hk) * D;
  uint32_t raw[JOBS][2];
#pragma unroll
  for (int jj = 0; jj < JOBS; ++jj) {
    const int job = warp + jj * W, m = job < G + 2 ? n : n - 1, part = job < G + 2 ? job : job - 2;
    if (job >= jobs) continue;
    const bf16* row = lookup.table ? lookup.table + (int64_t)__ldcg(lookup.codes + m * 16 + lookup.group) * width : qkv + (int64_t)m * width;
    ld_halves<D>(row + (part < G ? kh * G + part : part == G ? hq + kh : hq + hk + kh) * D, lane, raw[jj]);
  }
  // the tokens that earlier passes wrote
  for (int i = threadIdx.x; i < 2 * base * (D / 8); i += W * 32) {
    const int half = i >= base * (D / 8), at = i - half * base * (D / 8), tok = at / (D / 8), c = at % (D / 8) * 8;
    pattn::cp16(sm100::smem_addr(kvs[half] + tok * P + c), page + (half * 16 + tok) * D + c, true);
  }
#pragma unroll
  for (int jj = 0; jj < JOBS; ++jj) {
    const int job = warp + jj * W;
    if (job >= jobs) continue;
    const bool before = job >= G + 2;
    const int part = before ? job - 2 : job, tok = before ? pos - 1 : pos;
    float lo[E], hi[E];
    widen_halves<D>(raw[jj], lo, hi);
    if (part < G) rope_head<D>(lo, hi, qwl, qwh, cs, sn, eps);
    else if (part == G && !before) rope_head<D>(lo, hi, kwl, kwh, cs, sn, eps);
    else if (part == G) rope_head<D>(lo, hi, kwl, kwh, cs0, sn0, eps);
    st_half<D>(part < G ? qs + part * P : kvs[part - G] + tok * P, lane, lo, hi);
    if (part >= G && !before && owned) st_half<D>(page + ((part - G) * 16 + tok) * D, lane, lo, hi);
  }
  pattn::cp_commit(), pattn::cp_wait<0>();
  __syncthreads();

  // S[heads, keys] = q . K^T: two accumulators for each eight keys
  const int g = lane >> 2, t = lane & 3;
  // ldmatrix rows of this lane: heads past G and tokens to come are the row of zeros (no value may meet a zero weight as Inf)
  const int head = lane & 7, k_tok = (lane & 7) + (lane >> 4) * 8, v_tok = lane & 15;
  const uint32_t q_at = sm100::smem_addr((head < G ? qs + head * P : frame_rows) + (lane >> 3) * 8);
  const uint32_t k_at = sm100::smem_addr((k_tok <= pos ? kvs[0] + k_tok * P : frame_rows) + ((lane >> 3) & 1) * 8);
  float s[2][2][4] = {};
#pragma unroll
  for (int j = 0; j < D / 32; ++j) {
    uint32_t a[4];
    sm100::ldsm4(q_at + j * 64, a);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint32_t b[4];
      sm100::ldsm4(k_at + j * 64 + h * 32, b);
      sm100::mma_16816(s[0][h], a[2 * h], 0u, a[2 * h + 1], 0u, b[0], b[1]);
      sm100::mma_16816(s[1][h], a[2 * h], 0u, a[2 * h + 1], 0u, b[2], b[3]);
    }
  }
  float p[4], mx = -INFINITY, l = 0.f;  // head g, keys 2 t, 2 t + 1, 2 t + 8, 2 t + 9
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int key = 2 * t + (k & 1) + 8 * (k >> 1);
    p[k] = key <= pos ? (s[k >> 1][0][k & 1] + s[k >> 1][1][k & 1]) * scale : -INFINITY;
    mx = fmaxf(mx, p[k]);
  }
  mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1)), mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
#pragma unroll
  for (int k = 0; k < 4; ++k) p[k] = __expf(p[k] - mx), l += p[k];
  l += __shfl_xor_sync(0xffffffffu, l, 1), l += __shfl_xor_sync(0xffffffffu, l, 2);
  uint32_t a0[3], a2[3];
  split3(p[0], p[1], a0), split3(p[2], p[3], a2);
  const float inv = 1.f / l;

  // O[heads, dims] = P . V, this warp's quarter of the dims
  const uint32_t v_at = sm100::smem_addr((v_tok <= pos ? kvs[1] + v_tok * P : frame_rows) + warp * (D / 4) + (lane >> 4) * 8);
  bf16* const dst = out + ((int64_t)n * hq + kh * G + g) * D + warp * (D / 4) + 2 * t;
#pragma unroll
  for (int i = 0; i < D / 64; ++i) {
    uint32_t b[4];
    sm100::ldsm4t(v_at + i * 32, b);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int x = 2; x >= 0; --x) sm100::mma_16816(o, a0[x], 0u, a2[x], 0u, b[2 * h], b[2 * h + 1]);
      if (g < G) *reinterpret_cast<__nv_bfloat162*>(dst + i * 16 + h * 8) = __floats2bfloat162_rn(o[0] * inv, o[1] * inv);
    }
  }
}

template <int D, int G>
static cudaError_t launch_rope_attend_dg(const bf16* qkv, const QkvTable& lookup, const bf16* q_norm, const bf16* k_norm,
                                         bf16* kv, bf16* out, RowMap map, int rows, const AttnShape& a,
                                         int kv_pages, int sm_count, uint32_t* err, cudaStream_t s) {
  const float scale = 1.f / sqrtf((float)D);
  if (!map.pages) {
    if (map.per < 1 || map.per > 2 || map.base < 0 || map.base + map.per > 16) return cudaErrorInvalidValue;
    return launch_pdl(frame_attend_kernel<D, G>, dim3(rows / map.per * a.kv_heads, map.per), dim3(128),
                      (size_t)(1 + G + 2 * (map.base + map.per)) * (D + 8) * sizeof(bf16), s, qkv, lookup, q_norm, k_norm, kv, out, map.base,
                      a.q_heads, a.kv_heads, a.rms_eps, a.rope_theta, scale, kv_pages, err);
  }
  if (map.seq || lookup.table) return cudaErrorInvalidValue;  // one row per sequence
  const int items = rows * a.kv_heads;
  auto go = [&](auto kernel, int warps) {
    return launch_pdl(kernel, dim3(items), dim3(warps * 32), 0, s, qkv, q_norm, k_norm, kv, out, map, a.q_heads,
                      a.kv_heads, a.rms_eps, a.rope_theta, scale, kv_pages, err);
  };
  // items that leave SMs idle: eight warps each, so that 128 keys are one round (sixteen would have to spill: 2,282 against
  // 2,242 us a step of one session, 2,133 against 2,042 us for Higgs at three); up to three CTAs an SM, four warps; beyond, three
  // warps and four CTAs an SM, one wave of 512 items instead of two (64 sessions: 3,416 against 3,513 us a step), and there the
  // longest rows first, which counts from the second wave (592 items) on. Prompts of 32 to 512 tokens, four warps as the rows come
  // and this: 80 sessions 4,418 and 4,256 us, 128 4,747 and 4,697 (four warps in order 4,757, two 4,707).
  if (items > 3 * sm_count) return go(rope_attend_kernel<D, G, 3>, 3);
  map.order = nullptr;
  return items <= sm_count ? go(rope_attend_kernel<D, G, 8>, 8) : go(rope_attend_kernel<D, G, 4>, 4);
}

template <int D>
static cudaError_t launch_rope_attend_d(const bf16* qkv, const QkvTable& lookup, const bf16* q_norm, const bf16* k_norm,
                                        bf16* kv, bf16* out, const RowMap& map, int rows, const AttnShape& a,
                                        int kv_pages, int sm_count, uint32_t* err, cudaStream_t s) {
  switch (a.q_heads / a.kv_heads) {
    case 1: return launch_rope_attend_dg<D, 1>(qkv, lookup, q_norm, k_norm, kv, out, map, rows, a, kv_pages, sm_count, err, s);
    case 2: return launch_rope_attend_dg<D, 2>(qkv, lookup, q_norm, k_norm, kv, out, map, rows, a, kv_pages, sm_count, err, s);
    case 4: return launch_rope_attend_dg<D, 4>(qkv, lookup, q_norm, k_norm, kv, out, map, rows, a, kv_pages, sm_count, err, s);
    case 5: return launch_rope_attend_dg<D, 5>(qkv, lookup, q_norm, k_norm, kv, out, map, rows, a, kv_pages, sm_count, err, s);
    case 8: return launch_rope_attend_dg<D, 8>(qkv, lookup, q_norm, k_norm, kv, out, map, rows, a, kv_pages, sm_count, err, s);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_rope_attend(const bf16* qkv, const QkvTable& lookup, const bf16* q_norm, const bf16* k_norm, bf16* kv,
                               bf16* out, const RowMap& map, int rows, const AttnShape& a, int kv_pages, int sm_count,
                               uint32_t* err, cudaStream_t s) {
  if (a.q_heads % a.kv_heads) return cudaErrorInvalidValue;
  if (a.head_dim == 128) return launch_rope_attend_d<128>(qkv, lookup, q_norm, k_norm, kv, out, map, rows, a, kv_pages, sm_count, err, s);
  if (a.head_dim == 64) return launch_rope_attend_d<64>(qkv, lookup, q_norm, k_norm, kv, out, map, rows, a, kv_pages, sm_count, err, s);
  return cudaErrorInvalidValue;
}

}  // namespace omni
