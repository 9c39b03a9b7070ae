// Decode attention of one (row, kv head) on the warp-level tensor instructions. The G query heads that share a kv head
// are the N = 8 dimension of m16n8k16, the 16 keys (then 16 dims of the values) are M, so a page of 16 keys costs
// D / 16 + D / 8 instructions instead of a few hundred multiply-adds and shuffles:
//   S^T[16 keys, heads] = K[16, D] . q^T        A = K rows as they lie in the page, B = q
//   O^T[16 dims, heads] += V^T[16, 16 keys] . P^T   A = pairs of value rows, B = P
// Queries and keys are bf16 values already and the sums are f32, as in the reference (qwen3.cu:123-207); a probability
// goes in as the sum of three bf16, which is all of it. A matrix instruction cuts off what does not fit its accumulator
// instead of rounding it, so no sum runs through many of them: two accumulators a score, one a page of values, added in f32.
// Share of outputs that are not the bf16 nearest to float64's, 12 to 1,100 keys: 0.01 to 0.04 % (scalar kernel of
// attend.cuh 0.01 to 0.05 %; two bf16 a probability and one accumulator throughout 0.05 to 0.23 %, and a talker step of 64
// sessions 47 us shorter).
// The K dimension of an MMA may be permuted as long as both operands agree: a lane takes 16 consecutive bytes of a key
// (or query) row, which serve as its share of two consecutive steps, so every load is one 16-byte access.
#pragma once
#include "sm100.cuh"
#include "util.cuh"

namespace omni {
namespace dattn {

__device__ __forceinline__ uint32_t word(const uint4& u, int i) { return i == 0 ? u.x : i == 1 ? u.y : i == 2 ? u.z : u.w; }

// A page's K|V block ([K | V][16][D] bf16, contiguous) in a warp's registers. lane = 4 g + t: keys g and g + 8 (dims
// 8 t + 32 j ..), values of keys 2 t, 2 t + 1, 2 t + 8, 2 t + 9 (dims 8 g + 64 i ..).
template <int D>
struct Page {
  uint4 k[2][D / 32];
  uint4 v[4][D / 64];
  __device__ __forceinline__ void load(const bf16* block, int lane) {
    load_k(block, lane);
    load_v(block, lane);
  }
  __device__ __forceinline__ void load_k(const bf16* block, int lane) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int j = 0; j < D / 32; ++j) k[h][j] = __ldcg(reinterpret_cast<const uint4*>(block + (g + 8 * h) * D + 8 * t + 32 * j));
  }
  __device__ __forceinline__ void load_v(const bf16* block, int lane) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int i = 0; i < D / 64; ++i)
        v[r][i] = __ldcg(reinterpret_cast<const uint4*>(block + 16 * D + (2 * t + (r & 1) + 8 * (r >> 1)) * D + 8 * g + 64 * i));
  }
  // Token `tok`'s key and value rows replaced by those at kr / vr (shared memory).
  __device__ __forceinline__ void patch(int tok, const bf16* kr, const bf16* vr, int lane) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (g + 8 * h == tok) {
#pragma unroll
        for (int j = 0; j < D / 32; ++j) k[h][j] = *reinterpret_cast<const uint4*>(kr + 8 * t + 32 * j);
      }
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if (2 * t + (r & 1) + 8 * (r >> 1) == tok) {
#pragma unroll
        for (int i = 0; i < D / 64; ++i) v[r][i] = *reinterpret_cast<const uint4*>(vr + 8 * g + 64 * i);
      }
  }
};

// The running state of a warp: maxima and sums of heads 2 t and 2 t + 1 (the sums are this lane's keys' share until
// finish()), and the weighted values: acc[4 i + e][2 * which dim + which head] of dims 64 i + 8 g + 2 e + {0, 1}.
template <int D>
struct State {
  float m[2], l[2], acc[D / 16][4];
  __device__ __forceinline__ void reset() {
    m[0] = m[1] = -INFINITY, l[0] = l[1] = 0.f;
#pragma unroll
    for (int i = 0; i < D / 16; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  }
  // q: row g of [8][D] (heads past G are zero rows), 16 bytes per 32 dims. `next`: the block whose keys are asked for as
  // soon as this page's have been used, and whose values follow at the end (nullptr: none).
  __device__ __forceinline__ void step(Page<D>& pg, const uint4 (&q)[D / 32], int ntok, float scale, int lane,
                                       const bf16* next = nullptr) {
    const int g = lane >> 2, t = lane & 3;
    float s[4] = {0.f, 0.f, 0.f, 0.f}, s2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < D / 32; ++j) {
      sm100::mma_16816(s, pg.k[0][j].x, pg.k[1][j].x, pg.k[0][j].y, pg.k[1][j].y, q[j].x, q[j].y);
      sm100::mma_16816(s2, pg.k[0][j].z, pg.k[1][j].z, pg.k[0][j].w, pg.k[1][j].w, q[j].z, q[j].w);
    }
    if (next) pg.load_k(next, lane);
#pragma unroll
    for (int k = 0; k < 4; ++k) s[k] += s2[k];
    // s[0], s[1]: key g, heads 2t, 2t + 1; s[2], s[3]: key g + 8
#pragma unroll
    for (int k = 0; k < 4; ++k) s[k] = (g + (k >> 1) * 8) < ntok ? s[k] * scale : -INFINITY;
    float p[4], corr[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float mx = fmaxf(s[h], s[2 + h]);
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      const float m2 = fmaxf(m[h], mx);
      corr[h] = __expf(m[h] - m2);
      p[h] = __expf(s[h] - m2), p[2 + h] = __expf(s[2 + h] - m2);
      l[h] = l[h] * corr[h] + (p[h] + p[2 + h]);
      m[h] = m2;
    }
    // P^T as the B operand: this lane needs head g's probabilities of keys 2t, 2t + 1, 2t + 8, 2t + 9; key k's sit in
    // lane 4 (k & 7) + g / 2, element (k >> 3) * 2 + (g & 1)
    float w[4];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int src = 4 * (2 * t + r) + (g >> 1);
      const float lo0 = __shfl_sync(0xffffffffu, p[0], src), lo1 = __shfl_sync(0xffffffffu, p[1], src);
      const float hi0 = __shfl_sync(0xffffffffu, p[2], src), hi1 = __shfl_sync(0xffffffffu, p[3], src);
      w[r] = (g & 1) ? lo1 : lo0, w[2 + r] = (g & 1) ? hi1 : hi0;
    }
    uint32_t b0[3], b1[3];
    split3(w[0], w[1], b0), split3(w[2], w[3], b1);
    if (ntok < 16) {  // rows past the end hold whatever an earlier sequence left: they must not meet a zero weight as Inf
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (2 * t + (r & 1) + 8 * (r >> 1) >= ntok) {
#pragma unroll
          for (int i = 0; i < D / 64; ++i) pg.v[r][i] = make_uint4(0u, 0u, 0u, 0u);
        }
    }
#pragma unroll
    for (int i = 0; i < D / 64; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t v0 = word(pg.v[0][i], e), v1 = word(pg.v[1][i], e), v2 = word(pg.v[2][i], e), v3 = word(pg.v[3][i], e);
        const uint32_t a0 = __byte_perm(v0, v1, 0x5410), a1 = __byte_perm(v0, v1, 0x7632);
        const uint32_t a2 = __byte_perm(v2, v3, 0x5410), a3 = __byte_perm(v2, v3, 0x7632);
        float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int x = 2; x >= 0; --x) sm100::mma_16816(sum, a0, a1, a2, a3, b0[x], b1[x]);
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[4 * i + e][k] = fmaf(acc[4 * i + e][k], corr[k & 1], sum[k]);
      }
    if (next) pg.load_v(next, lane);
  }
  // Sums of the lanes' shares: every lane then holds its two heads' sums over all keys of the warp.
  __device__ __forceinline__ void finish() {
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) l[h] += __shfl_xor_sync(0xffffffffu, l[h], o);
  }
  // Eight consecutive dims (64 i + 8 g ..) of head 2 t + h.
  __device__ __forceinline__ void dims8(int i, int h, float (&v)[8]) const {
#pragma unroll
    for (int e = 0; e < 4; ++e) v[2 * e] = acc[4 * i + e][h], v[2 * e + 1] = acc[4 * i + e][2 + h];
  }
};

}  // namespace dattn
}  // namespace omni
