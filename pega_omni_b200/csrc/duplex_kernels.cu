// Non-GEMM kernels of the duplex (PersonaPlex) token loop. Value semantics follow
// crates/omni-personaplex/kernels/lm.cu (line ranges at each kernel); ids, pages and slots outside their tables
// raise the device error word instead of reading out of bounds.
#include <cuda_fp8.h>

#include "duplex.h"

#include "sm100.cuh"
#include "pdl.cuh"

namespace omni {
namespace {


__device__ __forceinline__ const int32_t* state_row(const void* state, const int32_t* lines, int s, int64_t stride) {
  return reinterpret_cast<const int32_t*>(static_cast<const char*>(state) + (int64_t)lines[s] * stride);
}

// Σ audio_emb[k][ids[1 + k]] over the 16 audio streams, then + text_emb[ids[0]]; every add rounded to bf16; an id
// of -1 contributes nothing (lm.cu:25-43).
__device__ __forceinline__ void embed_row(const int32_t* ids, const DuplexTables& t, bf16* out, int dim, uint32_t* err) {
  const int c = threadIdx.x * 8;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int k = 0; k < kDuplexStreams; ++k) {
    const int stream = k < kDuplexStreams - 1 ? k + 1 : 0;
    const int id = ids[stream];
    if (id < 0) continue;
    if (id >= (stream == 0 ? t.text_rows : t.card_rows)) {
      if (threadIdx.x == 0) raise(err, kErrBadIndex);
      continue;
    }
    const bf16* row = stream == 0 ? t.text_emb + (int64_t)id * dim : t.audio_emb + ((int64_t)k * t.card_rows + id) * dim;
    float e[8];
    ld8(row + c, e);
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = bf16_round(acc[j] + e[j]);
  }
  st8(out + c, acc);
}

// `lm_embed_prompt` (lm.cu:47-59)
__global__ void lm_embed_ids_kernel(const int32_t* __restrict__ ids, const int32_t* __restrict__ voice,
                                    const bf16* __restrict__ voices, int voice_rows, DuplexTables t,
                                    bf16* __restrict__ out, int dim, uint32_t* err) {
  grid_trigger();
  grid_wait();
  const int64_t r = blockIdx.x;
  if (voice && voice[r] >= 0) {
    int v = voice[r];
    if (v >= voice_rows) {
      if (threadIdx.x == 0) raise(err, kErrBadIndex);
      v = 0;
    }
    const int c = threadIdx.x * 8;
    *reinterpret_cast<uint4*>(out + r * dim + c) = *reinterpret_cast<const uint4*>(voices + (int64_t)v * dim + c);
    return;
  }
  embed_row(ids + r * kDuplexStreams, t, out + r * dim, dim, err);
}

// `lm_embed_state` (lm.cu:62-70)
__global__ void lm_embed_state_kernel(const void* state, const int32_t* __restrict__ lines, int64_t stride,
                                      DuplexTables t, bf16* __restrict__ out, int32_t* __restrict__ rows_out, int dim,
                                      uint32_t* err) {
  grid_trigger();
  grid_wait();
  const int s = blockIdx.x;
  const int32_t* row = state_row(state, lines, s, stride);
  if (threadIdx.x < kDuplexStreams) rows_out[s * kDuplexStreams + threadIdx.x] = row[threadIdx.x];
  embed_row(row, t, out + (int64_t)s * dim, dim, err);
}

// y = x * (alpha * rsqrt(eps + mean(x^2))) (lm.cu:74-84); v is 0 in threads past the row
__device__ __forceinline__ void norm_row(const float* v, const bf16* alpha, bf16* out, int dim, float eps, float* scratch) {
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) ss += v[k] * v[k];
  const float r = rsqrtf(block_add(ss, scratch) / dim + eps);
  if (threadIdx.x * 8 >= dim) return;
  float a[8], y[8];
  ld8(alpha + threadIdx.x * 8, a);
#pragma unroll
  for (int k = 0; k < 8; ++k) y[k] = v[k] * (a[k] * r);
  st8(out + threadIdx.x * 8, y);
}

__global__ void lm_norm_kernel(const bf16* x, const bf16* __restrict__ alpha, bf16* __restrict__ out,
                               int dim, float eps) {
  grid_trigger();
  grid_wait();
  __shared__ float scratch[32];
  const int64_t at = (int64_t)blockIdx.x * dim;
  float v[8] = {};
  if (threadIdx.x * 8 < dim) ld8cg(x + at + threadIdx.x * 8, v);
  norm_row(v, alpha, out + at, dim, eps, scratch);
}

// x = bf16(x + y), out = norm(x) over the rounded sum (lm.cu:95-106; out == nullptr: `lm_add`, lm.cu:109-120)
__global__ void lm_add_norm_kernel(const bf16* y, bf16* x, const bf16* __restrict__ alpha,
                                   bf16* __restrict__ out, int dim, float eps) {
  grid_trigger();
  grid_wait();
  __shared__ float scratch[32];
  const int64_t at = (int64_t)blockIdx.x * dim + threadIdx.x * 8;
  float v[8] = {}, u[8];
  if (threadIdx.x * 8 < dim) {
    ld8cg(x + at, v);
    ld8cg(y + at, u);
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = bf16_round(v[k] + u[k]);
    st8(x + at, v);
  }
  if (out) norm_row(v, alpha, out + (int64_t)blockIdx.x * dim, dim, eps, scratch);
}

// The same over a GEMM's summands: every load of a thread's E columns is under way at once.
template <int S, int E>
__global__ void lm_add_norm_sum_kernel(const Summands y, bf16* __restrict__ x, const bf16* __restrict__ alpha,
                                       bf16* __restrict__ out, int dim, float eps) {
  grid_trigger();
  __shared__ float scratch[32];
  const int c = threadIdx.x * E, lane = threadIdx.x & 31;
  const int64_t at = (int64_t)blockIdx.x * dim + c;
  const bool on = c < dim;  // the block is a whole number of warps
  float v[E], u[E], a[E], ss = 0.f;
  if (out && on) Run<E>::ld(alpha + c, a);
  grid_wait();
  if (on) {
    Run<E>::ldcg(x + at, v);
    load_sum<S, E>(y, blockIdx.x, c, u);
#pragma unroll
    for (int k = 0; k < E; ++k) {
      v[k] = bf16_round(v[k] + u[k]);
      ss += v[k] * v[k];
    }
    Run<E>::st(x + at, v);
  }
  if (!out) return;
  ss = warp_add(ss);
  if (lane == 0) scratch[threadIdx.x >> 5] = ss;
  __syncthreads();
  const float r = rsqrtf(warp_add(lane < (int)blockDim.x >> 5 ? scratch[lane] : 0.f) / dim + eps);
  if (!on) return;
#pragma unroll
  for (int k = 0; k < E; ++k) v[k] = v[k] * (a[k] * r);
  Run<E>::st(out + at, v);
}

// ---- tensor-parallel pair: all-reduce of a projection's partial rows, fused with the add + norm that follows -----
// Two ranks (two GPUs, one process each) hold half of the attention heads and half of the MLP channels; after the o
// and down projections each has a partial row block y_r [rows, dim]. This kernel makes y = bf16(y_0 + y_1) on both
// ranks and goes on as lm_add_norm does (x = bf16(x + y), out = norm(x)). The exchange is plain peer-memory traffic:
//   - `mine` sits in this rank's exchange buffer (written by the GEMM launched before this kernel), `peer` is the same
//     buffer of the other rank, mapped into this process;
//   - one thread stores this exchange's number into the PEER's flag word (release, system scope), so each rank polls
//     a word in its own memory; thread 0 of every CTA waits (acquire, system scope, at most kTpWaitNs) until its own
//     flag has reached the number, then the CTA reads the peer's rows with system-scope loads that bypass L1;
//   - exchanges are numbered by a device-resident counter that the last CTA to finish advances, so a captured graph
//     replays the same launch with new numbers; two buffers alternate (o, down), and a rank can only overwrite a
//     buffer two exchanges later, after it has seen the peer's next flag, which the peer raises only when its
//     previous exchange kernel (the reader of that buffer) has completed.
// f32 addition commutes, so both ranks round the same sum: their rows stay bit-identical.
// A wait that runs out raises the error word, takes the peer's rows as zero and lets the kernel finish.
constexpr uint64_t kTpWaitNs = 2000ull * 1000 * 1000;

__global__ void lm_tp_add_norm_kernel(const bf16* __restrict__ mine, const bf16* peer, bf16* __restrict__ x,
                                      const bf16* __restrict__ alpha, bf16* __restrict__ out, int dim, float eps,
                                      uint32_t* my_flag, uint32_t* peer_flag, uint32_t* counter, uint32_t* finished,
                                      uint32_t* err) {
  __shared__ float scratch[32];
  __shared__ int peer_ready;
  const uint32_t number = *reinterpret_cast<volatile uint32_t*>(counter) + 1u;
  if (threadIdx.x == 0) {
    if (blockIdx.x == 0) {
      __threadfence_system();
      asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(peer_flag), "r"(number) : "memory");
    }
    int ok = 1;
    if (*reinterpret_cast<volatile uint32_t*>(err) != 0) {
      ok = 0;  // an earlier kernel gave up: do not wait for a peer that may have given up as well
    } else {
      const uint64_t start = sm100::global_timer_ns();
      for (uint32_t spins = 0;; ++spins) {
        uint32_t seen;
        asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(seen) : "l"(my_flag) : "memory");
        if ((int32_t)(seen - number) >= 0) break;
        if ((spins & 63u) == 63u && sm100::global_timer_ns() - start > kTpWaitNs) {
          raise(err, kErrBarrierTimeout);
          ok = 0;
          break;
        }
      }
    }
    peer_ready = ok;
  }
  __syncthreads();
  const int64_t at = (int64_t)blockIdx.x * dim + threadIdx.x * 8;
  float v[8] = {}, a[8], b[8] = {};
  if (threadIdx.x * 8 < dim) {
    ld8(x + at, v);
    ld8(mine + at, a);
    if (peer_ready) {
      Pack8 raw;
      uint32_t* w = reinterpret_cast<uint32_t*>(&raw);
      asm volatile("ld.relaxed.sys.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                   : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
                   : "l"(peer + at)
                   : "memory");
      unpack8(raw, b);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = bf16_round(v[k] + bf16_round(a[k] + b[k]));
    st8(x + at, v);
  }
  if (out) norm_row(v, alpha, out + (int64_t)blockIdx.x * dim, dim, eps, scratch);
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(finished, 1u) == gridDim.x - 1) {  // every CTA has read the counter: advance it for the next launch
      *finished = 0;
      *reinterpret_cast<volatile uint32_t*>(counter) = number;
      __threadfence();
    }
  }
}

__device__ __forceinline__ uint8_t* page_head(void* kv, int64_t page, int heads, int h) {
  return static_cast<uint8_t*>(kv) + (page * heads + h) * (int64_t)kDuplexPageHeadBytes;
}

__device__ __forceinline__ float e4m3_scale(float amax) { return fmaxf(amax * (1.f / 448.f), 1e-12f); }

// Interleaved rotary embedding + FP8 KV write of one row (value semantics of `lm_rope`, lm.cu:129-184). kRopeParts
// CTAs per row: the 64 rotation angles depend on the row's position alone, so a CTA computes them once into shared
// memory (freq_i = expf(i * coef), sincosf(freq_i * pos)) for all the heads it rotates; its eight warps then walk
// its share of the 3 * heads heads, a lane owning four consecutive elements of the head (two rotation pairs): one
// 8-byte load, and for k / v one 4-byte FP8 store. k and v are quantised per head to E4M3 with the scale
// max(amax / 448, 1e-12), kept as f32 beside the page's values.
constexpr int kRopeWarps = 8, kRopeParts = 4;

__global__ void __launch_bounds__(kRopeWarps * 32)
    lm_rope_kv_kernel(bf16* qkv, const int32_t* __restrict__ pos, const int32_t* __restrict__ slots, void* kv,
                      int heads, float coef, int kv_pages, uint32_t* err) {
  grid_trigger();
  grid_wait();
  __shared__ float cs[kHeliumHeadDim / 2], sn[kHeliumHeadDim / 2];
  const int n = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < kHeliumHeadDim / 2) {
    const float freq = expf((float)threadIdx.x * coef);
    sincosf(freq * (float)pos[n], &sn[threadIdx.x], &cs[threadIdx.x]);
  }
  const int64_t slot = slots[n];
  if (slot < 0 || (slot >> 4) >= kv_pages) {  // nothing is stored: page 0 is some session's
    if (threadIdx.x == 0) raise(err, kErrBadIndex);
    return;
  }
  const int tok = (int)(slot & 15);
  __syncthreads();
  for (int head = blockIdx.y * kRopeWarps + warp; head < 3 * heads; head += kRopeWarps * kRopeParts) {
    bf16* src = qkv + ((int64_t)n * 3 * heads + head) * kHeliumHeadDim + lane * 4;
    const uint2 raw = __ldcg(reinterpret_cast<const uint2*>(src));
    const float2 p0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 p1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    float v[4] = {p0.x, p0.y, p1.x, p1.y};
    if (head < 2 * heads) {  // q and k: pairs (2i, 2i + 1) rotated by angle i
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float c = cs[2 * lane + k], sv = sn[2 * lane + k];
        const float r = v[2 * k], im = v[2 * k + 1];
        v[2 * k] = r * c - im * sv;
        v[2 * k + 1] = r * sv + im * c;
      }
    }
    if (head < heads) {  // q: rounded to bf16 in place
      uint2 o;
      *reinterpret_cast<__nv_bfloat162*>(&o.x) = __floats2bfloat162_rn(v[0], v[1]);
      *reinterpret_cast<__nv_bfloat162*>(&o.y) = __floats2bfloat162_rn(v[2], v[3]);
      *reinterpret_cast<uint2*>(src) = o;
      continue;
    }
    const bool is_v = head >= 2 * heads;
    const int h = head - (is_v ? 2 : 1) * heads;
    const float amax = warp_fmax(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))));
    const float sc = e4m3_scale(amax), inv = 1.f / sc;
    uint8_t* block = page_head(kv, slot >> 4, heads, h);
    const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[0] * inv, v[1] * inv), __NV_SATFINITE, __NV_E4M3);
    const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[2] * inv, v[3] * inv), __NV_SATFINITE, __NV_E4M3);
    *reinterpret_cast<uint32_t*>(block + ((is_v ? 16 : 0) + tok) * kHeliumHeadDim + lane * 4) = lo | hi << 16;
    if (lane == 0) reinterpret_cast<float*>(block + 2 * 16 * kHeliumHeadDim + (is_v ? 64 : 0))[tok] = sc;
  }
}

__device__ __forceinline__ float4 e4m3x4(uint32_t raw) {
  return static_cast<float4>(*reinterpret_cast<const __nv_fp8x4_e4m3*>(&raw));
}

// Decode attention over the FP8 ring (value semantics of `lm_attend` / `attend_row_fp8`, lm.cu:197-290: f32 scores,
// score * (k_scale * scale), __expf, p * v_scale, bf16 out). One CTA per (row, head), four warps. A (page, head) block
// is 4,224 contiguous bytes (16 keys, 16 values, their scales), so a warp stages whole pages into its own two
// shared-memory slots with one bulk copy each (cp.async.bulk, completion on an mbarrier) and has the next page under
// way while it works on the current one. Inside a page a lane scores half a key (64 of the 128 FP8 dims; lanes t and
// t + 16 share key t), the online softmax advances one page (16 keys) at a time, then every lane adds its four output
// dims of the 16 values. The warps' states are merged at the end. Waits are bounded (the error word, then out).
constexpr int kAttendWarps = 4;
constexpr int kAttendSlotBytes = ((kDuplexPageHeadBytes + 127) / 128) * 128;

// One page of one warp: lane = (key `tok`, half of its dims), the online softmax over 16 keys, then four output dims a lane.
__device__ __forceinline__ void page_step(const unsigned char* blk, const float* q, int ntok, float scale, int tok, int half,
                                          int lane, float& m, float& l, float (&acc)[4]) {
  float dot = 0.f;
  {
    const uint4* krow = reinterpret_cast<const uint4*>(blk + tok * kHeliumHeadDim + half * 64);
    const float* qh = q + half * 64;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const uint4 raw = krow[c];
      const float4 k0 = e4m3x4(raw.x), k1 = e4m3x4(raw.y), k2 = e4m3x4(raw.z), k3 = e4m3x4(raw.w);
      const float* qc = qh + c * 16;
      dot += qc[0] * k0.x + qc[1] * k0.y + qc[2] * k0.z + qc[3] * k0.w + qc[4] * k1.x + qc[5] * k1.y + qc[6] * k1.z +
             qc[7] * k1.w;
      dot += qc[8] * k2.x + qc[9] * k2.y + qc[10] * k2.z + qc[11] * k2.w + qc[12] * k3.x + qc[13] * k3.y +
             qc[14] * k3.z + qc[15] * k3.w;
    }
  }
  dot += __shfl_xor_sync(0xffffffffu, dot, 16);  // both halves of key `tok`
  const float ks = reinterpret_cast<const float*>(blk + 2 * 16 * kHeliumHeadDim)[tok];
  const float vs = reinterpret_cast<const float*>(blk + 2 * 16 * kHeliumHeadDim + 64)[tok];
  const float sv = tok < ntok ? dot * (ks * scale) : -INFINITY;
  const float m2 = fmaxf(m, warp_fmax(sv));
  const float corr = __expf(m - m2);
  const float p = __expf(sv - m2);
  float psum = p;  // over the 16 keys (both half-warps hold the same values)
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) psum += __shfl_xor_sync(0xffffffffu, psum, o);
  l = l * corr + psum;
#pragma unroll
  for (int d = 0; d < 4; ++d) acc[d] *= corr;
  m = m2;
  const float pv = p * vs;  // 0 for keys past the row's length
  const uint32_t* vrows = reinterpret_cast<const uint32_t*>(blk + 16 * kHeliumHeadDim) + lane;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const float pj = __shfl_sync(0xffffffffu, pv, j);
    const float4 vf = e4m3x4(vrows[j * (kHeliumHeadDim / 4)]);
    acc[0] += pj * vf.x, acc[1] += pj * vf.y, acc[2] += pj * vf.z, acc[3] += pj * vf.w;
  }
}

struct AttendShared {
  float q[kHeliumHeadDim];
  float ms[kAttendWarps], ls[kAttendWarps];
  float os[kAttendWarps][kHeliumHeadDim];
  uint64_t bar[kAttendWarps][2];
};

__global__ void __launch_bounds__(kAttendWarps * 32)
    lm_attend_kernel(const bf16* qkv, const void* kv, const int32_t* __restrict__ pos,
                     const int32_t* __restrict__ seq, const int32_t* __restrict__ indptr,
                     const int32_t* __restrict__ pages, bf16* __restrict__ out, int heads, float scale, int context,
                     int kv_pages, uint32_t* err) {
  grid_trigger();
  grid_wait();
  extern __shared__ __align__(128) unsigned char attend_smem[];
  AttendShared& sh = *reinterpret_cast<AttendShared*>(attend_smem);
  unsigned char* slots = attend_smem + ((sizeof(AttendShared) + 127) & ~(size_t)127);
  const int n = blockIdx.x, h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int s = seq ? seq[n] : n;
  const int len = min(pos[n] + 1, context), npages = (len + 15) >> 4;
  const int32_t* my_pages = pages + indptr[s];
  if (threadIdx.x < kHeliumHeadDim)
    sh.q[threadIdx.x] = __bfloat162float(__ldcg(qkv + ((int64_t)n * 3 * heads + h) * kHeliumHeadDim + threadIdx.x));
  if (lane == 0) {
    sm100::mbar_init(sm100::smem_addr(&sh.bar[warp][0]), 1);
    sm100::mbar_init(sm100::smem_addr(&sh.bar[warp][1]), 1);
  }
  sm100::mbar_init_fence();
  __syncthreads();

  unsigned char* mine = slots + (size_t)warp * 2 * kAttendSlotBytes;
  sm100::fence_async_global();  // keys and values written by ordinary stores, read by bulk copies
  auto fetch = [&](int pi, int slot) {  // lane 0: one bulk copy of page pi's block for this head
    int64_t page = my_pages[pi];
    if (page < 0 || page >= kv_pages) {
      raise(err, kErrBadIndex);
      page = 0;
    }
    const uint32_t bar = sm100::smem_addr(&sh.bar[warp][slot]);
    sm100::mbar_expect_tx(bar, kDuplexPageHeadBytes);
    sm100::bulk_load(sm100::smem_addr(mine + (size_t)slot * kAttendSlotBytes),
                     page_head(const_cast<void*>(kv), page, heads, h), kDuplexPageHeadBytes, bar);
  };
  float m = -INFINITY, l = 0.f, acc[4] = {0.f, 0.f, 0.f, 0.f};
  const int tok = lane & 15, half = lane >> 4;
  if (warp < npages && lane == 0) fetch(warp, 0);
  uint32_t parity[2] = {0, 0};
  int slot = 0;
  for (int pi = warp; pi < npages; pi += kAttendWarps, slot ^= 1) {
    if (pi + kAttendWarps < npages && lane == 0) fetch(pi + kAttendWarps, slot ^ 1);  // (that slot was read a round ago)
    if (!sm100::mbar_wait(sm100::smem_addr(&sh.bar[warp][slot]), parity[slot], err)) {
      if (pi + kAttendWarps < npages) sm100::mbar_wait(sm100::smem_addr(&sh.bar[warp][slot ^ 1]), parity[slot ^ 1], err);  // nothing may land later
      break;
    }
    parity[slot] ^= 1u;
    const unsigned char* blk = mine + (size_t)slot * kAttendSlotBytes;
    const int ntok = min(16, len - pi * 16);
    page_step(blk, sh.q, ntok, scale, tok, half, lane, m, l, acc);
    __syncwarp();  // every lane is done with this slot before lane 0 refills it in the next round
  }
  if (lane == 0) {
    sh.ms[warp] = m;
    sh.ls[warp] = l;
  }
#pragma unroll
  for (int d = 0; d < 4; ++d) sh.os[warp][lane * 4 + d] = acc[d];
  __syncthreads();
  if (threadIdx.x < kHeliumHeadDim) {
    const int d = threadIdx.x;
    float top = -INFINITY;
#pragma unroll
    for (int w = 0; w < kAttendWarps; ++w) top = fmaxf(top, sh.ms[w]);
    float num = 0.f, den = 0.f;
#pragma unroll
    for (int w = 0; w < kAttendWarps; ++w) {
      const float e = sh.ms[w] == -INFINITY ? 0.f : __expf(sh.ms[w] - top);
      num += sh.os[w][d] * e;
      den += sh.ls[w] * e;
    }
    out[((int64_t)n * heads + h) * kHeliumHeadDim + d] = __float2bfloat16(num / den);
  }
}

// Decode: rotary embedding, FP8 KV write and ring attention of one row per session in one kernel, W warps per (session, head),
// each on its own pages, which come straight into registers: a page's keys while the values before them are summed, the page
// behind on its way to L2. FP8 is exact in f16, so a page's products run on m16n8k16:
//   S[16 keys] = K[16, 128] . q      A = K (one conversion for two values), B = q. Step c of eight has its share of q in column c
//                                    and zeros elsewhere, so no sum runs through two instructions; the columns are added in f32.
//   O[dims] += V^T[dims, 16] . p     A = pairs of value rows, B = p in columns 0, 1, 2: three f16 whose sum is all of an f32,
//                                    scaled by powers of two that keep them clear of f16's range.
// q is bf16 already; scaled by a power of two so that its largest element is near the top of f16, what it loses is below
// 2^-38 of that. The lane 4 g + t that a q element belongs to as an operand also rotates it. Every page's products start from
// zero; maxima, sums and the running output are f32, as in the reference.
// Two conversions of a word are one asm block: the header's intrinsic gives two 16-bit halves, whose packing cost 110 instructions
// a page (41.0 us). Calls one behind the other, 64 rows of 32 heads, f32 arithmetic on staged pages and this: 252 keys
// 43.1 and 30.8 us, 500 keys 74.1 and 51.8, that is 21 us for each further 138 MB (6.6 TB/s); 16 rows of 252 16.5 and 16.2.
struct RingPage {
  uint4 k[2][2], v[4];  // keys g, g + 8: 16 values from 64 j + 16 t on; values of keys 2 t, 2 t + 1, 2 t + 8, 2 t + 9 from 16 g on
  float ks[2], vs[2];   // scales of keys g and g + 8
  __device__ __forceinline__ void load_k(const uint8_t* blk, int g, int t) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int j = 0; j < 2; ++j) k[h][j] = __ldcg(reinterpret_cast<const uint4*>(blk + (g + 8 * h) * kHeliumHeadDim + 64 * j + 16 * t));
      ks[h] = __ldcg(reinterpret_cast<const float*>(blk + 2 * 16 * kHeliumHeadDim) + g + 8 * h);
    }
  }
  __device__ __forceinline__ void load_v(const uint8_t* blk, int g, int t) {
#pragma unroll
    for (int r = 0; r < 4; ++r) v[r] = __ldcg(reinterpret_cast<const uint4*>(blk + (16 + 2 * t + (r & 1) + 8 * (r >> 1)) * kHeliumHeadDim + 16 * g));
#pragma unroll
    for (int h = 0; h < 2; ++h) vs[h] = __ldcg(reinterpret_cast<const float*>(blk + 2 * 16 * kHeliumHeadDim + 64) + g + 8 * h);
  }
};

__device__ __forceinline__ uint32_t ring_word(const uint4& u, int i) { return i == 0 ? u.x : i == 1 ? u.y : i == 2 ? u.z : u.w; }
// Four e4m3 (a word) as f16: bytes 0, 1 in lo, bytes 2, 3 in hi.
__device__ __forceinline__ void e4m3_to_f16(uint32_t four, uint32_t& lo, uint32_t& hi) {
  asm("{\n.reg .b16 l, h;\nmov.b32 {l, h}, %2;\ncvt.rn.f16x2.e4m3x2 %0, l;\ncvt.rn.f16x2.e4m3x2 %1, h;\n}" : "=r"(lo), "=r"(hi) : "r"(four));
}
__device__ __forceinline__ uint32_t half_pair(float lo, float hi) {
  const __half2 h = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}

template <int W>
__global__ void __launch_bounds__(W < 4 ? 128 : W * 32, W < 4 ? 4 : 16 / W)
    lm_rope_attend_kernel(const bf16* qkv, void* kv, const int32_t* __restrict__ pos,
                          const int32_t* __restrict__ slots, const int32_t* __restrict__ indptr,
                          const int32_t* __restrict__ pages, bf16* __restrict__ out, int items, int heads, float coef, float scale,
                          int context, int kv_pages, uint32_t* err) {
  constexpr int TEAMS = W < 4 ? 4 / W : 1, WARPS = TEAMS * W, D = kHeliumHeadDim;
  grid_trigger();
  __shared__ alignas(16) uint8_t own_s[TEAMS][2][D];  // the row's own key and value
  __shared__ float own_scale_s[TEAMS][2];
  __shared__ float ms[WARPS], ls[WARPS];
  __shared__ alignas(16) float os[W == 1 ? 1 : WARPS][D];
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, warp = warp_index() % W, team = warp_index() / W;
  const int item = blockIdx.x * TEAMS + team;
  const bool live = item < items;
  const int n = live ? item / heads : 0, h = live ? item % heads : 0;
  const int at = pos[n], len = min(at + 1, context), npages = live ? (len + 15) >> 4 : 0, own = (at % context) >> 4;
  const int32_t* my_pages = pages + indptr[n];
  int64_t slot_id = slots[n];
  const bool owned = slot_id >= 0 && (slot_id >> 4) < kv_pages;  // otherwise the row stores nothing: page 0 is some session's
  if (!owned) {
    if (live && warp == 0 && lane == 0) raise(err, kErrBadIndex);
    slot_id = 0;
  }
  auto block = [&](int pi) -> const uint8_t* {
    int64_t page = pi == own ? slot_id >> 4 : my_pages[pi];
    if (page < 0 || page >= kv_pages) {
      if (lane == 0) raise(err, kErrBadIndex);
      page = 0;
    }
    return page_head(kv, page, heads, h);
  };
  auto ask = [&](int pi) {
    if (lane == 0 && pi < npages) sm100::prefetch_l2(block(pi), kDuplexPageHeadBytes);
  };
  RingPage pg;
  if (warp < npages) {
    const uint8_t* first = block(warp);
    pg.load_k(first, g, t), pg.load_v(first, g, t);
  }
  ask(warp + W);
  const int d0 = 64 * (g >> 2) + 16 * t + 4 * (g & 3);  // the four elements of a row this lane takes: step g's
  float cs[2], sn[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) sincosf(expf((float)(d0 / 2 + k) * coef) * (float)at, &sn[k], &cs[k]);
  grid_wait();

  const bool mine = live && own % W == warp;  // the own page is this warp's: so are the row's key and value
  auto row4 = [&](int part) { return __ldcg(reinterpret_cast<const uint2*>(qkv + ((int64_t)n * 3 * heads + part * heads + h) * D + d0)); };
  auto widen = [](const uint2& raw, float (&v)[4]) {
    const float2 p0 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 p1 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    v[0] = p0.x, v[1] = p0.y, v[2] = p1.x, v[3] = p1.y;
  };
  auto rotate = [&](float (&v)[4]) {  // pairs (2i, 2i + 1) by angle i
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const float r = v[2 * k], im = v[2 * k + 1];
      v[2 * k] = r * cs[k] - im * sn[k];
      v[2 * k + 1] = r * sn[k] + im * cs[k];
    }
  };
  const uint2 raw_q = row4(0);
  if (mine) {
    uint2 raw[2] = {row4(1), row4(2)};
#pragma unroll
    for (int is_v = 0; is_v < 2; ++is_v) {
      float v[4];
      widen(raw[is_v], v);
      if (!is_v) rotate(v);
      const float amax = warp_fmax(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))));
      const float sc = e4m3_scale(amax), inv = 1.f / sc;
      const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(v[0] * inv, v[1] * inv), __NV_SATFINITE, __NV_E4M3);
      const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(v[2] * inv, v[3] * inv), __NV_SATFINITE, __NV_E4M3);
      const uint32_t four = lo | hi << 16;
      *reinterpret_cast<uint32_t*>(&own_s[team][is_v][d0]) = four;
      if (lane == 0) own_scale_s[team][is_v] = sc;
      if (owned) {
        uint8_t* blk = page_head(kv, slot_id >> 4, heads, h);
        const int tok = (int)(slot_id & 15);
        *reinterpret_cast<uint32_t*>(blk + (is_v * 16 + tok) * D + d0) = four;
        if (lane == 0) reinterpret_cast<float*>(blk + 2 * 16 * D + is_v * 64)[tok] = sc;
      }
    }
    __syncwarp();
  }
  // the query as the B operand: this lane's four elements are column g of step g
  uint32_t q0, q1;
  float q_scale = scale;
  {
    float v[4];
    widen(raw_q, v);
    rotate(v);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = bf16_round(v[k]);
    const float top = sm100::redux_max(fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3]))));
    // times 2^(14 - the largest element's exponent); below 2^-112 the factor stays 2^126, where f16 holds every bf16, and
    // infinities and NaN stay what they are
    const uint32_t e = max(15u, min(254u, __float_as_uint(top) >> 23));
    const float up = __uint_as_float((268u - e) << 23);
    q_scale *= __uint_as_float((e - 14u) << 23);
    q0 = half_pair(v[0] * up, v[1] * up), q1 = half_pair(v[2] * up, v[3] * up);
  }

  const float w0 = t == 0 ? 1.f : t == 1 ? 0x1p-22f : 0.f, w1 = t == 0 ? 0x1p-11f : 0.f;  // of columns 2 t and 2 t + 1
  float m = -INFINITY, l = 0.f, acc[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) acc[i] = 0.f;
  for (int pi = warp; pi < npages; pi += W) {
    ask(pi + 2 * W);
    const int ntok = min(16, len - pi * 16);
    if (pi == own) {
      const int tok = (int)(slot_id & 15);
#pragma unroll
      for (int x = 0; x < 2; ++x)
        if (g + 8 * x == tok) {
          pg.k[x][0] = *reinterpret_cast<const uint4*>(&own_s[team][0][16 * t]), pg.k[x][1] = *reinterpret_cast<const uint4*>(&own_s[team][0][64 + 16 * t]);
          pg.ks[x] = own_scale_s[team][0], pg.vs[x] = own_scale_s[team][1];
        }
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (2 * t + (r & 1) + 8 * (r >> 1) == tok) pg.v[r] = *reinterpret_cast<const uint4*>(&own_s[team][1][16 * g]);
    }
    if (ntok < 16) {  // tokens past the end: whatever lies there must not meet a zero weight as NaN
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (2 * t + (r & 1) + 8 * (r >> 1) >= ntok) pg.v[r] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int x = 0; x < 2; ++x)
        if (g + 8 * x >= ntok) pg.vs[x] = 0.f;
    }
    float s[2][4] = {};
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      uint32_t a0, a1, a2, a3;
      e4m3_to_f16(ring_word(pg.k[0][c >> 2], c & 3), a0, a2), e4m3_to_f16(ring_word(pg.k[1][c >> 2], c & 3), a1, a3);
      sm100::mma_16816_f16(s[c & 1], a0, a1, a2, a3, g == c ? q0 : 0u, g == c ? q1 : 0u);
    }
    float sv[2], p[2];
#pragma unroll
    for (int x = 0; x < 2; ++x) {  // key g + 8 x
      float dot = (s[0][2 * x] + s[0][2 * x + 1]) + (s[1][2 * x] + s[1][2 * x + 1]);
      dot += __shfl_xor_sync(0xffffffffu, dot, 1);
      dot += __shfl_xor_sync(0xffffffffu, dot, 2);
      sv[x] = g + 8 * x < ntok ? dot * (pg.ks[x] * q_scale) : -INFINITY;
    }
    const bool more = pi + W < npages;
    const uint8_t* next = more ? block(pi + W) : nullptr;
    if (more) pg.load_k(next, g, t);
    const float m2 = fmaxf(m, sm100::redux_max(fmaxf(sv[0], sv[1]))), corr = __expf(m - m2);
    p[0] = __expf(sv[0] - m2), p[1] = __expf(sv[1] - m2);
    l = l * corr + (p[0] + p[1]);
    m = m2;
    // weights p * v_scale, times 2^(14 - the largest scale's exponent)
    const uint32_t ve = max(15u, min(254u, __float_as_uint(sm100::redux_max(fmaxf(pg.vs[0], pg.vs[1]))) >> 23));
    const float up = __uint_as_float((268u - ve) << 23), down = __uint_as_float((ve - 14u) << 23);
    const float pv[2] = {p[0] * pg.vs[0] * up, p[1] * pg.vs[1] * up};
    float x[4];  // of keys 2 t, 2 t + 1, 2 t + 8, 2 t + 9
#pragma unroll
    for (int r = 0; r < 4; ++r) x[r] = __shfl_sync(0xffffffffu, pv[r >> 1], 4 * (2 * t + (r & 1)));
    uint32_t b[2];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      float y0 = x[2 * half], y1 = x[2 * half + 1];
      uint32_t piece = 0u;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const uint32_t two = half_pair(y0, y1);
        if (g == i) piece = two;
        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&two));
        y0 = (y0 - f.x) * 2048.f, y1 = (y1 - f.y) * 2048.f;
      }
      b[half] = piece;
    }
    const float f0 = w0 * down, f1 = w1 * down;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const uint32_t u0 = ring_word(pg.v[0], w), u1 = ring_word(pg.v[1], w), u2 = ring_word(pg.v[2], w), u3 = ring_word(pg.v[3], w);
#pragma unroll
      for (int half = 0; half < 2; ++half) {  // dims 4 w + 2 half and the next are rows g and g + 8
        uint32_t a0, a1, a2, a3;
        e4m3_to_f16(__byte_perm(u0, u1, half ? 0x7362 : 0x5140), a0, a1), e4m3_to_f16(__byte_perm(u2, u3, half ? 0x7362 : 0x5140), a2, a3);
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
        sm100::mma_16816_f16(sum, a0, a1, a2, a3, b[0], b[1]);
#pragma unroll
        for (int d = 0; d < 2; ++d)
          acc[4 * w + 2 * half + d] = fmaf(acc[4 * w + 2 * half + d], corr, fmaf(sum[2 * d + 1], f1, sum[2 * d] * f0));
      }
    }
    if (more) pg.load_v(next, g, t);
  }
  // the three columns are lanes t = 0 and 1: each adds the other's and takes eight of the sixteen dims
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
  float o[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float theirs = __shfl_xor_sync(0xffffffffu, t & 1 ? acc[k] : acc[8 + k], 1);
    o[k] = (t & 1 ? acc[8 + k] : acc[k]) + theirs;
  }
  bf16* const dst = out + ((int64_t)n * heads + h) * D;
  if constexpr (W == 1) {
    if (!live || t > 1) return;
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] /= l;
    st8(dst + 16 * g + 8 * t, o);
  } else {
    const int w = team * W + warp;
    if (t < 2) {
      float4* to = reinterpret_cast<float4*>(&os[w][16 * g + 8 * t]);
      to[0] = make_float4(o[0], o[1], o[2], o[3]), to[1] = make_float4(o[4], o[5], o[6], o[7]);
    }
    if (lane == 0) ms[w] = m, ls[w] = l;
    __syncthreads();
    if (!live) return;
    for (int d = warp * 32 + lane; d < D; d += W * 32) {
      float top = -INFINITY;
#pragma unroll
      for (int x = 0; x < W; ++x) top = fmaxf(top, ms[team * W + x]);
      float num = 0.f, den = 0.f;
#pragma unroll
      for (int x = 0; x < W; ++x) {
        const float e = ms[team * W + x] == -INFINITY ? 0.f : __expf(ms[team * W + x] - top);
        num += os[team * W + x][d] * e;
        den += ls[team * W + x] * e;
      }
      dst[d] = __float2bfloat16(num / den);
    }
  }
}

// `lm_dep_embed_norm` (lm.cu:301-313)
__global__ void lm_dep_embed_norm_kernel(const bf16* projected, int k, const bf16* __restrict__ table, int table_rows,
                                         const int32_t* drawn,
                                         const bf16* __restrict__ alpha, bf16* __restrict__ x, bf16* __restrict__ xn,
                                         int dim, float eps, uint32_t* err) {
  grid_trigger();
  grid_wait();
  __shared__ float scratch[32];
  const int s = blockIdx.x, c = threadIdx.x * 8;
  int64_t id = __ldcg(drawn + s * kDuplexDrawn + k);
  if (id < 0 || id >= table_rows) {
    if (threadIdx.x == 0) raise(err, kErrBadIndex);
    id = 0;
  }
  float v[8] = {}, e[8];
  if (c < dim) {
    ld8cg(projected + ((int64_t)s * kDepSteps + k) * dim + c, v);
    ld8(table + id * dim + c, e);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = bf16_round(v[j] + e[j]);
    st8(x + (int64_t)s * dim + c, v);
  }
  norm_row(v, alpha, xn + (int64_t)s * dim, dim, eps, scratch);
}

// `lm_dep_kv_attend` (lm.cu:319-366): a warp per (session, head), a lane owns two of the 64 dims; the step's own K
// and V stay in registers.
__global__ void lm_dep_kv_attend_kernel(const bf16* qkv, bf16* ws, int step,
                                        bf16* __restrict__ out, int heads, float scale) {
  grid_trigger();
  grid_wait();
  const int s = blockIdx.x, h = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (h >= heads) return;
  const int width = heads * kDepHeadDim;
  const bf16* row = qkv + (int64_t)s * 3 * width;
  const int at = h * kDepHeadDim + lane * 2;
  const __nv_bfloat162 q2 = __ldcg(reinterpret_cast<const __nv_bfloat162*>(row + at));
  const __nv_bfloat162 k2 = __ldcg(reinterpret_cast<const __nv_bfloat162*>(row + width + at));
  const __nv_bfloat162 v2 = __ldcg(reinterpret_cast<const __nv_bfloat162*>(row + 2 * width + at));
  bf16* base = ws + (int64_t)s * kDepSteps * 2 * width;
  *reinterpret_cast<__nv_bfloat162*>(base + (int64_t)step * 2 * width + at) = k2;
  *reinterpret_cast<__nv_bfloat162*>(base + (int64_t)step * 2 * width + width + at) = v2;
  const float q0 = __bfloat162float(q2.x), q1 = __bfloat162float(q2.y);
  float m = -INFINITY, l = 0.f, a0 = 0.f, a1 = 0.f;
  for (int t = 0; t <= step; ++t) {
    __nv_bfloat162 kt = k2, vt = v2;
    if (t < step) {
      kt = __ldcg(reinterpret_cast<const __nv_bfloat162*>(base + (int64_t)t * 2 * width + at));
      vt = __ldcg(reinterpret_cast<const __nv_bfloat162*>(base + (int64_t)t * 2 * width + width + at));
    }
    const float sc = warp_add(q0 * __bfloat162float(kt.x) + q1 * __bfloat162float(kt.y)) * scale;
    const float m2 = fmaxf(m, sc);
    const float corr = __expf(m - m2);
    const float p = __expf(sc - m2);
    l = l * corr + p;
    a0 = a0 * corr + p * __bfloat162float(vt.x);
    a1 = a1 * corr + p * __bfloat162float(vt.y);
    m = m2;
  }
  const float inv_l = 1.f / l;
  *reinterpret_cast<__nv_bfloat162*>(out + (int64_t)s * width + at) = __floats2bfloat162_rn(a0 * inv_l, a1 * inv_l);
}

// ---- Gumbel-max draw over the top-k (value semantics of `lm_sample`, lm.cu:368-537) ----------------------------
// Every element's score depends only on (logit, seed, index): key = 16-bit order key of the bf16 logit, the cut is
// the k-th largest key (ties kept), score = logit / T - log(-log u) with u = ((mix(seed ^ mix(index)) >> 8) + 0.5) /
// 2^24, winner = largest (order_key(score), lowest index).
//
// One CTA per row. The row is read from global memory ONCE: a thread keeps R packed pairs of keys (256 threads x 4 for a
// codebook of 2,048, 1,024 x 16 or x 32 for a text vocabulary up to 65,536), in registers as far as 64 a thread go: -Xptxas -v
// shows 96 bytes of spill stores at R = 16 and 288 at R = 32, none for a codebook. The cut is then found by bisection on
// the key's 16 bits, two at a time from the top: the counts of keys >= three candidates take one warp reduction each and
// one block barrier a round (the per-warp counts are double-buffered in shared memory). The survivors' scores are
// computed from the same registers and the winner is reduced by shuffles and one pass over the warps' results.

__device__ __forceinline__ uint32_t order_key32(float v) {
  const uint32_t u = __float_as_uint(v);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ uint32_t order_key16(uint32_t bits) {  // bits: a bf16 in the low half
  return (bits & 0x8000u) ? (~bits & 0xffffu) : (bits | 0x8000u);
}
__device__ __forceinline__ float logit_of(uint32_t key) {  // the inverse of order_key16
  const uint32_t bits = (key & 0x8000u) ? (key & 0x7fffu) : (~key & 0xffffu);
  return __uint_as_float(bits << 16);
}
__device__ __forceinline__ uint32_t mix32(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}

template <int THREADS, int R>
__global__ void __launch_bounds__(THREADS)
    lm_sample_kernel(const bf16* logits, int vocab, int64_t ld, float temperature, int top_k,
                     const int32_t* __restrict__ force, const int32_t* __restrict__ seeds, int col,
                     int32_t* __restrict__ drawn) {
  constexpr int WARPS = THREADS / 32;
  grid_trigger();
  const int s = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  __shared__ uint32_t counts[2][3][WARPS];
  __shared__ unsigned long long best[WARPS];
  const int forced = force[s * kDuplexDrawn + col];
  const uint32_t seed = mix32((uint32_t)seeds[2 * s] ^ mix32((uint32_t)seeds[2 * s + 1] + 0x9e3779b9u * (col + 1)));
  grid_wait();
  if (forced >= 0) {
    if (tid == 0) drawn[s * kDuplexDrawn + col] = forced;
    return;
  }
  // element 2 * (r * THREADS + tid) + {0, 1} lives in the low / high half of reg[r]; 0 past the vocabulary (the smallest
  // key there is: -NaN with every mantissa bit set orders lowest, and no count ever includes index >= vocab)
  const uint16_t* row = reinterpret_cast<const uint16_t*>(logits + (int64_t)s * ld);
  const bool pairs = (reinterpret_cast<uintptr_t>(row) & 3) == 0;
  uint32_t reg[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = 2 * (r * THREADS + tid);
    uint32_t two = 0u;
    if (pairs && i + 1 < vocab) {
      two = __ldcg(reinterpret_cast<const uint32_t*>(row + i));
    } else {
      if (i < vocab) two = __ldcg(row + i);
      if (i + 1 < vocab) two |= (uint32_t)__ldcg(row + i + 1) << 16;
    }
    reg[r] = two;
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = 2 * (r * THREADS + tid);
    const uint32_t k0 = i < vocab ? order_key16(reg[r] & 0xffffu) : 0u, k1 = i + 1 < vocab ? order_key16(reg[r] >> 16) : 0u;
    reg[r] = k0 | k1 << 16;
  }
  const float inv_t = temperature > 0.f ? 1.f / temperature : 1.f;
  const int keep = top_k > 0 && top_k < vocab ? top_k : vocab;
  uint32_t cut = 0;
  if (temperature > 0.f && keep < vocab) {
#pragma unroll 1
    for (int bit = 14; bit >= 0; bit -= 2) {
      uint32_t c[3] = {0u, 0u, 0u};
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const uint32_t k0 = reg[r] & 0xffffu, k1 = reg[r] >> 16;
#pragma unroll
        for (int q = 0; q < 3; ++q) {  // candidates >= 1: the padding keys (0) never count
          const uint32_t cand = cut | (uint32_t)(q + 1) << bit;
          c[q] += (k0 >= cand) + (k1 >= cand);
        }
      }
      const int buf = (bit >> 1) & 1;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        c[q] = __reduce_add_sync(0xffffffffu, c[q]);
        if (lane == 0) counts[buf][q][warp] = c[q];
      }
      __syncthreads();
      uint32_t digit = 0;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const uint32_t total = __reduce_add_sync(0xffffffffu, lane < WARPS ? counts[buf][q][lane] : 0u);
        if (total >= (uint32_t)keep) digit = q + 1;
      }
      cut |= digit << bit;
    }
  }
  unsigned long long mine = 0ull;
#pragma unroll
  for (int r = 0; r < R; ++r) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int i = 2 * (r * THREADS + tid) + e;
      const uint32_t key = e ? reg[r] >> 16 : reg[r] & 0xffffu;
      if (i >= vocab || key < cut) continue;
      float score = logit_of(key) * inv_t;
      if (temperature > 0.f) {
        const float u = ((mix32(seed ^ mix32((uint32_t)i)) >> 8) + 0.5f) * (1.f / 16777216.f);
        score -= __logf(-__logf(u));
      }
      const unsigned long long packed = (unsigned long long)order_key32(score) << 32 | (uint32_t)(0xffffffffu - i);
      mine = packed > mine ? packed : mine;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, mine, o);
    mine = other > mine ? other : mine;
  }
  if (lane == 0) best[warp] = mine;
  __syncthreads();
  if (warp == 0) {
    mine = lane < WARPS ? best[lane] : 0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long other = __shfl_xor_sync(0xffffffffu, mine, o);
      mine = other > mine ? other : mine;
    }
    if (lane == 0) drawn[s * kDuplexDrawn + col] = (int32_t)(0xffffffffu - (uint32_t)(mine & 0xffffffffull));
  }
}

// `lm_advance` (lm.cu:546-573): one thread per session.
__global__ void lm_advance_kernel(void* state, const int32_t* __restrict__ lines, int64_t stride,
                                  const int32_t* drawn, const int32_t* __restrict__ caller,
                                  const int32_t* __restrict__ force_caller, int32_t* __restrict__ emitted, int seqs) {
  grid_trigger();
  grid_wait();
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= seqs) return;
  int32_t* row = const_cast<int32_t*>(state_row(state, lines, s, stride));
  int32_t* pending = row + kDuplexStreams;
  int32_t d[kDuplexDrawn], heard[kDuplexBooks];
#pragma unroll
  for (int k = 0; k < kDuplexDrawn; ++k) d[k] = __ldcg(drawn + s * kDuplexDrawn + k);
#pragma unroll
  for (int k = 0; k < kDuplexBooks; ++k) {
    const int f = force_caller[s * kDuplexBooks + k];
    heard[k] = f >= 0 ? f : caller[s * kDuplexBooks + k];
  }
  emitted[s * kDuplexDrawn] = row[0];
  emitted[s * kDuplexDrawn + 1] = row[1];
#pragma unroll
  for (int k = 1; k < kDuplexBooks; ++k) emitted[s * kDuplexDrawn + 1 + k] = d[1 + k];
#pragma unroll
  for (int k = 0; k < kDuplexDrawn; ++k) row[k] = d[k];
  row[kDuplexDrawn] = heard[0];
#pragma unroll
  for (int k = 0; k < kDuplexBooks - 1; ++k) {
    row[kDuplexDrawn + 1 + k] = pending[k];
    pending[k] = heard[1 + k];
  }
}

// `lm_init` (lm.cu:576-581)
__global__ void lm_init_kernel(void* state, const int32_t* __restrict__ lines, int64_t stride,
                               const int32_t* __restrict__ init) {
  grid_trigger();
  grid_wait();
  const int s = blockIdx.x;
  int32_t* own = const_cast<int32_t*>(state_row(state, lines, s, stride));
  if (threadIdx.x < kDuplexStateWords) own[threadIdx.x] = init[s * kDuplexStateWords + threadIdx.x];
}

// `lm_copy_kv` (lm.cu:584-593) for this library's layout: a warp per (token, head) moves the 128-byte key row, the
// 128-byte value row and the two scales.
__global__ void lm_copy_kv_kernel(void* kv, const int32_t* __restrict__ src_slot, const int32_t* __restrict__ dst_slot,
                                  int heads, int kv_pages, uint32_t* err) {
  grid_trigger();
  grid_wait();
  const int r = blockIdx.x, h = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (h >= heads) return;
  int64_t src = src_slot[r], dst = dst_slot[r];
  if (src < 0 || dst < 0 || (src >> 4) >= kv_pages || (dst >> 4) >= kv_pages) {
    if (lane == 0) raise(err, kErrBadIndex);
    return;
  }
  const uint8_t* from = page_head(kv, src >> 4, heads, h);
  uint8_t* to = page_head(kv, dst >> 4, heads, h);
  const int st = (int)(src & 15), dt = (int)(dst & 15);
  reinterpret_cast<uint32_t*>(to + dt * kHeliumHeadDim)[lane] = reinterpret_cast<const uint32_t*>(from + st * kHeliumHeadDim)[lane];
  reinterpret_cast<uint32_t*>(to + (16 + dt) * kHeliumHeadDim)[lane] =
      reinterpret_cast<const uint32_t*>(from + (16 + st) * kHeliumHeadDim)[lane];
  if (lane < 2)
    reinterpret_cast<float*>(to + 2 * 16 * kHeliumHeadDim + 64 * lane)[dt] =
        reinterpret_cast<const float*>(from + 2 * 16 * kHeliumHeadDim + 64 * lane)[st];
}

// Rows are read eight bytes at a time, pages by bulk copies.
bool ring_aligned(const void* qkv, const void* kv) {
  return (reinterpret_cast<uintptr_t>(qkv) & 7) == 0 && (reinterpret_cast<uintptr_t>(kv) & 15) == 0;
}

bool row_dim_ok(int dim) { return dim % 8 == 0 && dim / 8 <= 1024 && dim / 8 >= 32; }

}  // namespace

cudaError_t launch_lm_embed_ids(const int32_t* ids, const int32_t* voice, const bf16* voices, int voice_rows,
                                DuplexTables t, bf16* out, int rows, int dim, uint32_t* err, cudaStream_t s) {
  if (!row_dim_ok(dim)) return cudaErrorInvalidValue;
  return launch_pdl(lm_embed_ids_kernel, dim3(rows), dim3(dim / 8), 0, s, ids, voice, voices, voice_rows, t, out, dim, err);
}

cudaError_t launch_lm_embed_state(const void* state, const int32_t* lines, int64_t stride, DuplexTables t, bf16* out,
                                  int32_t* rows_out, int rows, int dim, uint32_t* err, cudaStream_t s) {
  if (!row_dim_ok(dim)) return cudaErrorInvalidValue;
  return launch_pdl(lm_embed_state_kernel, dim3(rows), dim3(dim / 8), 0, s, state, lines, stride, t, out, rows_out, dim, err);
}

cudaError_t launch_lm_norm(const bf16* x, const bf16* alpha, bf16* out, int rows, int dim, float eps, cudaStream_t s) {
  if (!row_dim_ok(dim)) return cudaErrorInvalidValue;
  return launch_pdl(lm_norm_kernel, dim3(rows), dim3(row_threads(dim)), 0, s, x, alpha, out, dim, eps);
}

cudaError_t launch_lm_add_norm(const bf16* y, bf16* x, const bf16* alpha, bf16* out, int rows, int dim, float eps,
                               cudaStream_t s) {
  if (!row_dim_ok(dim)) return cudaErrorInvalidValue;
  return launch_pdl(lm_add_norm_kernel, dim3(rows), dim3(row_threads(dim)), 0, s, y, x, alpha, out, dim, eps);
}

cudaError_t launch_lm_add_norm_sum(const Summands& y, bf16* x, const bf16* alpha, bf16* out, int rows, int dim, float eps,
                                   cudaStream_t s) {
  if (!row_dim_ok(dim)) return cudaErrorInvalidValue;
  return with_summands(y.splits, [&](auto sums) {
    return with_columns(dim, rows, [&](auto columns) {
      constexpr int E = decltype(columns)::value;
      return launch_pdl(lm_add_norm_sum_kernel<decltype(sums)::value, E>, dim3(rows), dim3((dim + E * 32 - 1) / (E * 32) * 32), 0, s, y, x, alpha, out, dim, eps);
    });
  });
}

cudaError_t launch_lm_tp_add_norm(const bf16* mine, const bf16* peer, bf16* x, const bf16* alpha, bf16* out, int rows,
                                  int dim, float eps, const TpLink& link, uint32_t* err, cudaStream_t s) {
  if (!row_dim_ok(dim) || !peer || !link.my_flag || !link.peer_flag) return cudaErrorInvalidValue;
  lm_tp_add_norm_kernel<<<rows, row_threads(dim), 0, s>>>(mine, peer, x, alpha, out, dim, eps, link.my_flag, link.peer_flag,
                                                 link.counter, link.finished, err);
  return cudaGetLastError();
}

cudaError_t launch_lm_rope_kv(bf16* qkv, const int32_t* pos, const int32_t* slots, void* kv, int rows, int heads,
                              float coef, int kv_pages, uint32_t* err, cudaStream_t s) {
  if (!ring_aligned(qkv, kv)) return cudaErrorInvalidValue;
  return launch_pdl(lm_rope_kv_kernel, dim3(rows, kRopeParts), dim3(kRopeWarps * 32), 0, s, qkv, pos, slots, kv, heads, coef, kv_pages, err);
}

cudaError_t launch_lm_attend(const bf16* qkv, const void* kv, const int32_t* pos, const int32_t* seq,
                             const int32_t* indptr, const int32_t* pages, bf16* out, int rows, int heads, float scale,
                             int context, int kv_pages, uint32_t* err, cudaStream_t s) {
  const size_t smem = ((sizeof(AttendShared) + 127) & ~(size_t)127) + (size_t)kAttendWarps * 2 * kAttendSlotBytes;
  static bool raised[64] = {};  // per device: 70 KB of staging slots is above the default 48 KB of dynamic shared memory
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return cudaErrorInvalidDevice;
  if (!raised[device]) {
    const cudaError_t e = cudaFuncSetAttribute(lm_attend_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    raised[device] = true;
  }
  return launch_pdl(lm_attend_kernel, dim3(rows, heads), dim3(kAttendWarps * 32), smem, s, qkv, kv, pos, seq, indptr, pages, out, heads, scale, context, kv_pages, err);
}

cudaError_t launch_lm_rope_attend(const bf16* qkv, void* kv, const int32_t* pos, const int32_t* slots,
                                  const int32_t* indptr, const int32_t* pages, bf16* out, int rows, int heads, float coef,
                                  float scale, int context, int kv_pages, int sm_count, uint32_t* err, cudaStream_t s) {
  if (!ring_aligned(qkv, kv)) return cudaErrorInvalidValue;
  const int items = rows * heads;
  auto go = [&](auto kernel, int warps) {
    const int teams = warps < 4 ? 4 / warps : 1;
    return launch_pdl(kernel, dim3((items + teams - 1) / teams), dim3(teams * warps * 32), 0, s, qkv, kv, pos, slots, indptr, pages, out,
                      items, heads, coef, scale, context, kv_pages, err);
  };
  // As many warps an item as run at once, sixteen an SM: 64 rows of 252 keys 30.8 us with one warp an item, 34.6 with two, 36.9
  // with four (a merge through shared memory and fewer pages a warp). One warp stores 16 bytes a lane, so rows at addresses that
  // do not take them have two.
  const int64_t room = (int64_t)16 * sm_count;
  if (items * 16 <= room) return go(lm_rope_attend_kernel<16>, 16);
  if (items * 8 <= room) return go(lm_rope_attend_kernel<8>, 8);
  if (items * 4 <= room) return go(lm_rope_attend_kernel<4>, 4);
  return items * 2 <= room || (reinterpret_cast<uintptr_t>(out) & 15) ? go(lm_rope_attend_kernel<2>, 2) : go(lm_rope_attend_kernel<1>, 1);
}

cudaError_t launch_lm_dep_embed_norm(const bf16* projected, int k, const bf16* table, int table_rows,
                                     const int32_t* drawn, const bf16* alpha, bf16* x, bf16* xn, int rows, int dim,
                                     float eps, uint32_t* err, cudaStream_t s) {
  if (!row_dim_ok(dim)) return cudaErrorInvalidValue;
  return launch_pdl(lm_dep_embed_norm_kernel, dim3(rows), dim3(row_threads(dim)), 0, s, projected, k, table, table_rows, drawn, alpha, x, xn, dim, eps, err);
}

cudaError_t launch_lm_dep_kv_attend(const bf16* qkv, bf16* ws, int step, bf16* out, int rows, int heads, float scale,
                                    cudaStream_t s) {
  if (step < 0 || step >= kDepSteps) return cudaErrorInvalidValue;
  return launch_pdl(lm_dep_kv_attend_kernel, dim3(rows, (heads + 3) / 4), dim3(128), 0, s, qkv, ws, step, out, heads, scale);
}

cudaError_t launch_lm_sample(const bf16* logits, int vocab, int64_t ld, float temperature, int top_k,
                             const int32_t* force, const int32_t* seeds, int col, int32_t* drawn, int rows,
                             cudaStream_t s) {
  if (vocab < 1 || col < 0 || col >= kDuplexDrawn) return cudaErrorInvalidValue;
  auto go = [&](auto kernel, int threads) {
    return launch_pdl(kernel, dim3(rows), dim3(threads), 0, s, logits, vocab, ld, temperature, top_k, force, seeds, col, drawn);
  };
  if (vocab <= 2048) return go(lm_sample_kernel<256, 4>, 256);
  if (vocab <= 32768) return go(lm_sample_kernel<1024, 16>, 1024);
  if (vocab <= 65536) return go(lm_sample_kernel<1024, 32>, 1024);
  return cudaErrorInvalidValue;
}

cudaError_t launch_lm_advance(void* state, const int32_t* lines, int64_t stride, const int32_t* drawn,
                              const int32_t* caller, const int32_t* force_caller, int32_t* emitted, int rows,
                              cudaStream_t s) {
  return launch_pdl(lm_advance_kernel, dim3((rows + 127) / 128), dim3(128), 0, s, state, lines, stride, drawn, caller, force_caller, emitted, rows);
}

cudaError_t launch_lm_copy_kv(void* kv, const int32_t* src_slot, const int32_t* dst_slot, int tokens, int heads,
                              int kv_pages, uint32_t* err, cudaStream_t s) {
  if (tokens < 1) return cudaSuccess;
  return launch_pdl(lm_copy_kv_kernel, dim3(tokens, (heads + 3) / 4), dim3(128), 0, s, kv, src_slot, dst_slot, heads, kv_pages, err);
}

cudaError_t launch_lm_init(void* state, const int32_t* lines, int64_t stride, const int32_t* init, int rows,
                           cudaStream_t s) {
  return launch_pdl(lm_init_kernel, dim3(rows), dim3(32), 0, s, state, lines, stride, init);
}

}  // namespace omni
