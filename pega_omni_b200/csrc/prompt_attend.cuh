// Attention of prompt rows: many rows of a sequence attend to the same keys, so the products are contractions and run on
// m16n8k16. A CTA takes 32 rows and one kv head: its G query heads of those rows are 32 * G rows of M, sixteen to a warp;
// keys and values come two pages (32 keys) at a time into shared memory by cp.async, three stages deep, where every warp
// reads them with ldmatrix. Rows may belong to several sequences: the CTA goes through the runs of rows of one sequence in
// turn, and rows outside the run (or keys past a row's position) are masked. Value semantics of `attend`
// (crates/omni-qwen3/kernels/qwen3.cu:123-207): f32 scores, online softmax in f32; a probability enters the second product
// as the sum of three bf16, which is all of it, and sums are kept out of long chains of matrix instructions (decode_attend.cuh):
// 0.01 to 0.02 % of the outputs of prompts of 77 to 512 rows are not the bf16 nearest to float64's (scalar kernel 0.01 to
// 0.02 %, two bf16 a probability 0.17 to 0.22 %).
// Measured alone with cold caches at 7,604 rows of 28 ragged prompts, D = 128, G = 2: 144 us a layer (109 us with two bf16 a
// probability; scalar multiply-adds, each row reading its keys for itself: 1,184 us at 8,700 rows). Three CTAs an SM with
// fewer registers are no faster. Bound by the matrix instructions' issue and shared-memory reads alike: 128 instructions a
// warp and 64 x 32 tile at G = 2, and every warp reads the 16 KB of a stage for its sixteen rows (about 512 cycles each).
// -Xptxas -v: 48 bytes of spill stores at <128, 2>, 12 at <128, 5>, 172 at <128, 8>.
#pragma once
#include "attend.cuh"
#include "pdl.cuh"
#include "sm100.cuh"

namespace omni {
namespace pattn {

constexpr int kRows = 32, kKeys = 32, kStages = 3;

template <int D>
__host__ __device__ constexpr int stage_bytes() { return kKeys * 2 * D * 2; }  // K and V of 32 tokens

__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool fetch) {  // zeros where !fetch
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(fetch ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <int D, int G>
__global__ void __launch_bounds__(kRows * G * 2, G >= 4 ? 1 : 2)
    prompt_attend_kernel(const bf16* qkv, const bf16* kv, bf16* __restrict__ out, RowMap map,
                         int rows, int hq, int hk, float scale) {
  constexpr int kThreads = kRows * G * 2, C = D / 8;  // C: 16-byte chunks of a row
  extern __shared__ __align__(128) unsigned char prompt_smem[];
  __shared__ int seq_s[kRows], pos_s[kRows];
  grid_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * kRows, kh = blockIdx.y, count = min(kRows, rows - n0);
  if (threadIdx.x < kRows) {
    const bool there = (int)threadIdx.x < count;
    seq_s[threadIdx.x] = there ? map.seq[n0 + threadIdx.x] : -1;
    pos_s[threadIdx.x] = there ? map.pos[n0 + threadIdx.x] : -1;
  }
  __syncthreads();
  const uint32_t ring = sm100::smem_addr(prompt_smem);

  // this lane's two rows of M: (row, head of the group)
  int row[2], head[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int m = warp * 16 + g + 8 * h;
    row[h] = m / G, head[h] = m % G;
  }
  uint32_t q[D / 16][4];  // their queries as A fragments
  const int warp_r0 = warp * 16 / G, warp_r1 = (warp * 16 + 15) / G;  // rows this warp holds heads of

  for (int r0 = 0; r0 < count;) {
    // the run of rows of one sequence from r0 on, and its last key
    const int seq = seq_s[r0];
    const uint32_t same = __ballot_sync(0xffffffffu, seq_s[lane] == seq) >> r0;
    const int len = same == 0xffffffffu ? 32 : __ffs(~same) - 1, r1 = r0 + len;
    const int my_pos = lane >= r0 && lane < r1 ? pos_s[lane] : -1;
    const int last = __reduce_max_sync(0xffffffffu, my_pos);
    const bool mine = lane >= warp_r0 && lane <= warp_r1;
    const int warp_last = __reduce_max_sync(0xffffffffu, mine ? my_pos : -1);
    const int warp_least = __reduce_min_sync(0xffffffffu, mine ? my_pos : 0x7fffffff);  // keys every row of the warp sees
    int limit[2];  // keys 0 .. limit count for this lane's rows
#pragma unroll
    for (int h = 0; h < 2; ++h) limit[h] = row[h] >= r0 && row[h] < r1 ? pos_s[row[h]] : -1;
    const int32_t* pages = map.pages + map.indptr[seq];
    const int tiles = (last + kKeys) / kKeys;
    // the two pages of the next tile to fetch, read a tile ahead
    int page[2];
    auto look = [&](int tile) {
#pragma unroll
      for (int p = 0; p < 2; ++p) page[p] = tile * kKeys + p * 16 <= last ? pages[tile * 2 + p] : 0;
    };
    auto fetch = [&](int tile) {
      if (tile < tiles) {
        const uint32_t dst = ring + (uint32_t)(tile % kStages) * stage_bytes<D>();
        const bf16* base[2] = {kv + kv_offset<D>(page[0], hk, kh, 0, 0), kv + kv_offset<D>(page[1], hk, kh, 0, 0)};
#pragma unroll
        for (int u = 0; u < (kKeys * 2 * C + kThreads - 1) / kThreads; ++u) {
          const int i = threadIdx.x + u * kThreads;
          if (kKeys * 2 * C % kThreads && i >= kKeys * 2 * C) break;
          const int c = i % C, tok = i / C % 16, which = i / (C * 16) & 1, pg = i / (C * 32);
          // a stage: K of 32 tokens, V of 32 tokens; chunk c of a token sits at c ^ (token & 7)
          cp16(dst + (uint32_t)((which * kKeys + pg * 16 + tok) * C + (c ^ (tok & 7))) * 16u, base[pg] + (which * 16 + tok) * D + c * 8,
               tile * kKeys + pg * 16 + tok <= last);
        }
        look(tile + 1);
      }
      cp_commit();
    };
    look(0);
    if (r0 == 0) grid_wait();
    for (int s = 0; s < kStages - 1; ++s) fetch(s);
    // every run starts from nothing and stores its own rows: what it leaves in the other rows' sums (0 times another
    // sequence's values, which is no 0 where those are infinite) is never used
    float mx[2] = {-INFINITY, -INFINITY}, sum[2] = {0.f, 0.f}, acc[D / 8][4] = {};
    if (r0 == 0) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const bf16* src = qkv + ((int64_t)(n0 + min(row[h], count - 1)) * (hq + 2 * hk) + kh * G + head[h]) * D + 2 * t;
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          q[k][h] = __ldcg(reinterpret_cast<const uint32_t*>(src + k * 16));
          q[k][2 + h] = __ldcg(reinterpret_cast<const uint32_t*>(src + k * 16 + 8));
        }
      }
    }
    for (int tile = 0; tile < tiles; ++tile) {
      cp_wait<kStages - 2>();
      __syncthreads();  // the tile is there for everyone, and everyone is done with the one before
      fetch(tile + kStages - 1);
      if (tile * kKeys > warp_last) continue;
      const uint32_t kb = ring + (uint32_t)(tile % kStages) * stage_bytes<D>(), vb = kb + kKeys * D * 2;
      float s[4][4] = {}, s2[4][4] = {};
#pragma unroll
      for (int k = 0; k < D / 16; ++k) {
#pragma unroll
        for (int jj = 0; jj < 2; ++jj) {  // 16 keys: matrices (keys 0-7, k 0-7), (keys 0-7, k 8-15), (keys 8-15, ...)
          const int tok = jj * 16 + (lane & 7) + ((lane >> 4) << 3);
          uint32_t b[4];
          sm100::ldsm4(kb + (uint32_t)(tok * C + ((k * 2 + ((lane >> 3) & 1)) ^ (tok & 7))) * 16u, b);
          sm100::mma_16816(k & 1 ? s2[jj * 2] : s[jj * 2], q[k], b[0], b[1]);
          sm100::mma_16816(k & 1 ? s2[jj * 2 + 1] : s[jj * 2 + 1], q[k], b[2], b[3]);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[j][e] += s2[j][e];
      float corr[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float top = -INFINITY;
        if (tile * kKeys + kKeys - 1 <= warp_least) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) s[j][2 * h + e] *= scale, top = fmaxf(top, s[j][2 * h + e]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int key = tile * kKeys + j * 8 + 2 * t + e;
              float& x = s[j][2 * h + e];
              x = key <= limit[h] ? x * scale : -INFINITY;
              top = fmaxf(top, x);
            }
        }
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
        const float m2 = fmaxf(mx[h], top), ref = m2 == -INFINITY ? 0.f : m2;
        corr[h] = __expf(mx[h] - ref);
        mx[h] = m2;
        float part = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float& x = s[j][2 * h + e];
            x = __expf(x - ref);
            part += x;
          }
        sum[h] = sum[h] * corr[h] + part;  // this lane's keys; the other lanes' are added at the end
      }
      uint32_t p[2][3][4];  // 16 keys each
#pragma unroll
      for (int kk = 0; kk < 2; ++kk)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          uint32_t part[3];
          split3(s[kk * 2 + (x >> 1)][(x & 1) * 2], s[kk * 2 + (x >> 1)][(x & 1) * 2 + 1], part);
          p[kk][0][x] = part[0], p[kk][1][x] = part[1], p[kk][2][x] = part[2];
        }
#pragma unroll
      for (int i = 0; i < D / 16; ++i) {  // 16 dims
        float o[2][4] = {};
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
          const int tok = kk * 16 + (lane & 15);
          uint32_t b[4];
          sm100::ldsm4t(vb + (uint32_t)(tok * C + ((i * 2 + (lane >> 4)) ^ (tok & 7))) * 16u, b);
#pragma unroll
          for (int x = 2; x >= 0; --x) {
            sm100::mma_16816(o[0], p[kk][x], b[0], b[1]);
            sm100::mma_16816(o[1], p[kk][x], b[2], b[3]);
          }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[2 * i + u][e] = fmaf(acc[2 * i + u][e], corr[e >> 1], o[u][e]);
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 1);
      sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 2);
      if (limit[h] < 0) continue;  // not a row of this run
      const float inv = 1.f / sum[h];
      bf16* dst = out + ((int64_t)(n0 + row[h]) * hq + kh * G + head[h]) * D + 2 * t;
#pragma unroll
      for (int i = 0; i < D / 8; ++i)
        *reinterpret_cast<__nv_bfloat162*>(dst + i * 8) = __floats2bfloat162_rn(acc[i][2 * h] * inv, acc[i][2 * h + 1] * inv);
    }
    cp_wait<0>();
    __syncthreads();  // the ring is free for the next run
    r0 = r1;
  }
}

}  // namespace pattn
}  // namespace omni
