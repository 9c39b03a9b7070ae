// The GEMM of the kernel chains for up to eight rows (see few_rows.h).
//
// A decode node of a few rows is latency: its weights were asked for before its inputs existed, so what counts is the
// path from the inputs' arrival to the outputs' stores. tcgen05 puts four hand-overs on it (rows to shared memory by TMA,
// MMA issue, commit, TMEM load); here the weights are M of m16n8k16 and the rows its N, and a warp keeps everything it
// needs to itself: its eighth of K, its own ring of weight blocks, its rows of x, so that only the final sum over the
// eight warps crosses a barrier. One m16n8k16 takes 2 cycles of the SM's pipe, which is ten times the rate at which DRAM
// delivers weights, and up to eight rows there is nothing for a larger tile to reuse. Two 8-row tiles of x a warp double the
// rows' arrival and the shared memory they take from the rings: at 16 rows a talker step took 3,526 us against 3,361 with the
// tcgen05 kernel, a Higgs step 2,375 against 2,326, a duplex tick 4,604 against 4,548.
// The add + norm before a projection is made by every CTA from the summands (L2 broadcast reads, 16 KB to 100 KB) while
// one or two pieces a lane suffice (few_norm_fits); a kernel of its own takes 2.7 us and beyond that is faster. Measured as nodes of a
// traced chain (omni_talker_trace, whose stamp adds half a microsecond) at one row: 1,024 x 3,072 2.8 us, 6,144 x 1,024 with
// norm and SwiGLU 4.1 us, 4,096 x 1,024 with norm 3.6 us (4.5 to 5.3 us and 2.7 us for the norm with the tcgen05 kernel of
// stream_gemm.cu).
#include "few_rows.h"

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "few_share.h"
#include "pdl.cuh"
#include "sm100.cuh"

namespace omni {
namespace {

constexpr int kWarps = kFewWarps, kKb = kFewKb, kFewSlots = 8;
constexpr int kNormChunks = 2;  // 8-element pieces of the rows that a lane holds across the norm's sum

struct FewArgs {
  const bf16* x;
  bf16* y;
  float* part;
  const bf16* bias;
  uint32_t* err;
  FewNorm norm;
  sm100::Ahead ahead;
  float inv_k;
  int N, K, rows, R, slots, ldy, kind, nkb, span, per, xk, lanes_log2, rounds;
};

__device__ __forceinline__ void st_shared16(uint32_t addr, const uint4& v) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// Where a lane's pieces of the rows lie (few_share.h), and where they go.
struct Share : FewShare {
  int warp;
  int64_t at;   // the lane's first piece (few_at)
  uint32_t xs;  // row n's share in shared memory
};

// The add + norm's rows, RD pieces a lane, from S partial sums; `keep`: this CTA stores the residual.
template <int NORM, int S, int RD>
__device__ __forceinline__ void norm_rows(const FewArgs& a, const Share& h, bool keep, float (*ss_s)[kWarps], const uint4* gain) {
  const int64_t at = h.at;
  const float* part = a.norm.sum.part + at;
  constexpr int B = S >= 4 ? 2 : RD < 4 ? RD : RD == 4 && S == 1 ? 4 : 2;  // pieces under way at a time
  float v[RD][8], ss = 0.f;
#pragma unroll
  for (int j0 = 0; j0 < RD; j0 += B) {
    uint4 r[B];
    float4 f[B][S][2];
#pragma unroll
    for (int j = 0; j < B; ++j) {
      const int o = few_step(h, j0 + j);
      r[j] = __ldcg(reinterpret_cast<const uint4*>(a.norm.res_in + at + o));
#pragma unroll
      for (int s = 0; s < S; ++s) {
        const float4* q = reinterpret_cast<const float4*>(part + s * a.norm.sum.split_stride + o);
        f[j][s][0] = __ldcg(q), f[j][s][1] = __ldcg(q + 1);
      }
    }
#pragma unroll
    for (int j = 0; j < B; ++j) {
      float u[8], mine = 0.f;
      unpack8v(r[j], u);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        float t = reinterpret_cast<const float*>(&f[j][0][0])[k];
#pragma unroll
        for (int s = 1; s < S; ++s) t += reinterpret_cast<const float*>(&f[j][s][0])[k];
        t = bf16_round(t) + u[k];
        if constexpr (NORM != kNormStack) t = bf16_round(t);
        v[j0 + j][k] = t;
        mine += t * t;
      }
      ss += h.first + (j0 + j) * h.lanes < h.pieces ? mine : 0.f;
    }
    if (j0 + B < RD) asm volatile("" ::: "memory");
  }
  float scale = 1.f;
  if constexpr (NORM != kAddLm) {
    for (int o = h.lanes >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (h.live && h.first == 0) ss_s[h.n][h.warp] = ss;
    __syncthreads();
    const float4 s0 = *reinterpret_cast<const float4*>(&ss_s[h.n & 7][0]), s1 = *reinterpret_cast<const float4*>(&ss_s[h.n & 7][4]);
    scale = rsqrtf((((s0.x + s0.y) + (s0.z + s0.w)) + ((s1.x + s1.y) + (s1.z + s1.w))) * a.inv_k + a.norm.eps);
  }
#pragma unroll
  for (int j = 0; j < RD; ++j) {
    if (!h.live || h.first + j * h.lanes >= h.pieces) break;
    if (keep) st8(a.norm.res_out + at + j * h.lanes * 8, v[j]);
    if constexpr (NORM != kAddLm) {
      float g[8];
      unpack8v(gain[j], g);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[j][k] = NORM == kNormLm ? v[j][k] * (g[k] * scale) : v[j][k] * scale * g[k];
    }
    st_shared16(h.xs + (uint32_t)(h.first + j * h.lanes) * 16u, pack8v(v[j]));
  }
}

template <int RD>
__device__ __forceinline__ void plain_rows(const FewArgs& a, const Share& h) {
  const uint4* src = reinterpret_cast<const uint4*>(a.x + (int64_t)(h.live ? h.n : 0) * a.K + h.c0) + h.first;
  for (int j0 = 0; h.first + j0 * h.lanes < h.pieces; j0 += RD) {
    uint4 v[RD];
#pragma unroll
    for (int j = 0; j < RD; ++j) v[j] = __ldcg(src + (h.first + (j0 + j) * h.lanes < h.pieces ? (j0 + j) * h.lanes : 0));
#pragma unroll
    for (int j = 0; j < RD; ++j)
      if (h.live && h.first + (j0 + j) * h.lanes < h.pieces) st_shared16(h.xs + (uint32_t)(h.first + (j0 + j) * h.lanes) * 16u, v[j]);
  }
}

// MT: 16-row tiles of weights per CTA (10: up to ten).
// Every instruction behind grid_wait() is on the chain's critical path and is executed once: what costs is how many a
// warp goes through (about 5 cycles each, more when its line has to come from L2), hence the index arithmetic in front of
// the wait, loops that run as often as there is work and bodies chosen by the number of pieces and sums.
template <int MT, int NORM, int OUT>
__global__ void __launch_bounds__(kWarps * 32, 2) few_rows_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ FewArgs a) {
  using namespace sm100;
  extern __shared__ unsigned char few_smem_raw[];
  __shared__ __align__(8) uint64_t bars_s[kWarps * kFewSlots];
  __shared__ __align__(16) float ss_s[8][kWarps];
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int tile = blockIdx.x, split = blockIdx.y;
  // k-blocks: `span` per split, `per` per warp, the last of each fewer
  const int kb0 = few_first(warp, split, a.span, a.per), nk = few_count(warp, split, a.span, a.per, a.nkb);
  const uint32_t slot_bytes = (uint32_t)a.R * 128u;
  const uint32_t ring0 = (smem_addr(few_smem_raw) + 1023u) & ~1023u;
  const uint32_t ring = ring0 + (uint32_t)(warp * a.slots) * slot_bytes;
  // this warp's rows of x: [rows][xk] bf16 (xk = 64 * per, + 8 against bank conflicts)
  const uint32_t xs = ring0 + (uint32_t)(kWarps * a.slots) * slot_bytes + (uint32_t)(warp * a.rows * a.xk) * 2u;
  const uint32_t bars = smem_addr(bars_s) + 8u * (uint32_t)(warp * kFewSlots);
  auto load_w = [&](int i, int slot) {
    mbar_expect_tx(bars + 8u * slot, slot_bytes);
    tma_load_3d(ring + (uint32_t)slot * slot_bytes, &wmap, bars + 8u * slot, 0, tile * a.R, kb0 + i, kEvictFirst);
  };
  const int ahead = min(a.slots, nk);
  if (lane == 0) {
    prefetch_tensormap(&wmap);
    for (int s = 0; s < a.slots; ++s) mbar_init(bars + 8u * s, 1);
    mbar_init_fence();
    for (int i = 0; i < ahead; ++i) load_w(i, i);
  }
  grid_trigger();
  if (warp == kWarps - 1 && lane == 0) ask_ahead(a.ahead, blockIdx.y * gridDim.x + blockIdx.x, gridDim.x * gridDim.y);
  __syncwarp();

  // ---- everything that does not depend on the rows comes before grid_wait(), the first weights' arrival included ----
  Share h;
  static_cast<FewShare&>(h) = few_share(lane, kb0, nk, a.lanes_log2, a.rows);
  h.warp = warp, h.at = few_at(h, a.K), h.xs = xs + (uint32_t)(h.n * a.xk) * 2u;
  const int mts = MT <= 4 ? MT : a.R >> 4;
  // ldmatrix rows of this lane: weights [0, 8) k 0..7, [8, 16) k 0..7, [0, 8) k 8..15, [8, 16) k 8..15; x rows past the
  // last read row 0 (their columns of the result are not stored)
  uint32_t x_lane = xs + (uint32_t)(((lane & 7) < a.rows ? lane & 7 : 0) * a.xk + (lane >> 3) * 8) * 2u, w_lane[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) w_lane[k] = ring + (uint32_t)(lane & 15) * 128u + (uint32_t)(((k * 2 + (lane >> 4)) ^ (lane & 7)) << 4);
  const int stride = a.R + 4, warp_floats = a.slots * a.R * 32;
  float* const red0 = reinterpret_cast<float*>(few_smem_raw + (ring0 - smem_addr(few_smem_raw)));
  float* const red = red0 + warp * warp_floats + (lane & 3) * 2 * stride + (lane >> 2);
  const int rounds = (h.pieces + h.lanes - 1) >> a.lanes_log2;
  uint4 g[kNormChunks];
  if constexpr (NORM == kNormStack || NORM == kNormLm) {
#pragma unroll
    for (int j = 0; j < kNormChunks; ++j)
      if (h.first + j * h.lanes < h.pieces) g[j] = __ldg(reinterpret_cast<const uint4*>(a.norm.gain + h.c0) + h.first + j * h.lanes);
  }
  bool fine = true;
  for (int i = 0; i < ahead; ++i) fine = mbar_wait(bars + 8u * i, 0, a.err) && fine;
  grid_wait();

  // ---- the rows ----
  if constexpr (NORM == 0) {
    if (rounds <= 1) plain_rows<1>(a, h);
    else if (((rounds + 3) >> 2) & 1) plain_rows<4>(a, h);
    else plain_rows<8>(a, h);  // a whole number of eights: half the round trips (a duplex tick of 8 4,535 -> 4,485 us)
  } else {
    const bool keep = tile == (int)gridDim.x - 1;
    auto with = [&](auto sums) {
      constexpr int S = decltype(sums)::value;
      if (a.rounds <= 1) norm_rows<NORM, S, 1>(a, h, keep, ss_s, g);
      else norm_rows<NORM, S, kNormChunks>(a, h, keep, ss_s, g);
    };
    if (a.norm.sum.splits == 1) with(std::integral_constant<int, 1>());
    else if (a.norm.sum.splits == 2) with(std::integral_constant<int, 2>());
    else with(std::integral_constant<int, 4>());
  }
  __syncwarp();

  // ---- w . x^T ----
  float acc[MT][4];
#pragma unroll
  for (int m = 0; m < MT; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;
  uint32_t turn = 0, off = 0;  // of the ring; off: bytes to the slot
#pragma unroll 1
  for (int i = 0, slot = 0; i < nk; ++i) {
    if (i >= ahead) fine = mbar_wait(bars + 8u * slot, turn, a.err);
    if (!fine) {  // nothing may land once the CTA has left
      for (int j = max(i + 1, ahead); j < min(nk, i + a.slots); ++j) mbar_wait(bars + 8u * (j % a.slots), (uint32_t)(j / a.slots) & 1u, a.err);
      break;
    }
    uint32_t b[2][4];
    ldsm4(x_lane, b[0]), ldsm4(x_lane + 64, b[1]);
    x_lane += 128u;
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      if (MT <= 4 || m < mts) {
        uint32_t w[4][4];
#pragma unroll
        for (int k = 0; k < 4; ++k) ldsm4(w_lane[k] + off + m * 2048, w[k]);
#pragma unroll
        for (int k = 0; k < 4; ++k) mma_16816(acc[m], w[k], b[k >> 1][(k & 1) * 2], b[k >> 1][(k & 1) * 2 + 1]);
      }
    }
    if (ahead < nk) {  // a ring that does not hold the warp's whole share
      __syncwarp();
      if (lane == 0 && i + a.slots < nk) load_w(i + a.slots, slot);
    }
    off += slot_bytes;
    if (++slot == a.slots) slot = 0, off = 0, turn ^= 1u;
  }

  // ---- sum over the warps, through each warp's own (spent) ring: [row of x][weight row]; SwiGLU, whose 16-row tiles are
  // eight gates and their ups, all gates then all ups ----
  __syncwarp();
#pragma unroll
  for (int m = 0; m < MT; ++m)
    if (MT <= 4 || m < mts) {
      float* at = red + m * (OUT == kStreamSwiglu ? 8 : 16);
      float* at2 = OUT == kStreamSwiglu ? at + (a.R >> 1) : at + 8;
      at[0] = acc[m][0], at[stride] = acc[m][1];
      at2[0] = acc[m][2], at2[stride] = acc[m][3];
    }
  __syncthreads();
  auto total = [&](int at) {
    float f[kWarps];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) f[w] = red0[w * warp_floats + at];
    return ((f[0] + f[1]) + (f[2] + f[3])) + ((f[4] + f[5]) + (f[6] + f[7]));
  };
  const int halves = OUT == kStreamSwiglu ? 1 : 0, cols = min(a.R, a.N - tile * a.R) >> halves, c0 = (tile * a.R) >> halves;
#pragma unroll 1
  for (int n = warp; n < a.rows; n += kWarps) {  // a row per warp, a column per lane
#pragma unroll 1
    for (int c = lane; c < cols; c += 32) {
      const float v = total(n * stride + c);
      if constexpr (OUT == kStreamSwiglu) {
        const float u = bf16_round(total(n * stride + (a.R >> 1) + c)), gate = bf16_round(v);
        a.y[(int64_t)n * a.ldy + c0 + c] = __float2bfloat16(silu_bf16(gate) * u);
      } else if constexpr (OUT == kStreamPartials) {
        a.part[((int64_t)split * a.rows + n) * a.N + c0 + c] = v;
      } else {
        float o = bf16_round(v);
        if (a.kind != kEpiNone) {
          o = bf16_round(o + __bfloat162float(a.bias[c0 + c]));
          if (a.kind == kEpiBiasSilu) o = o / (1.f + __expf(-o));
        }
        a.y[(int64_t)n * a.ldy + c0 + c] = __float2bfloat16(o);
      }
    }
  }
}

// More than a third of an SM's shared memory each, so that an SM takes one CTA of this kernel and one of the next, whose
// weights are then on their way, but not two of the same while another SM is idle; rings stop at half of it.
constexpr int kFewMinSmem = 76 * 1024, kFewHalf = 112 * 1024, kFewMaxSmem = 148 * 1024;

template <int MT, typename F>
cudaError_t few_dispatch_tile(int norm, int out, F&& go) {
  const bool bf = out == kStreamBf16, swi = out == kStreamSwiglu;
  if (norm == 0) return bf ? go(few_rows_kernel<MT, 0, kStreamBf16>) : swi ? go(few_rows_kernel<MT, 0, kStreamSwiglu>) : go(few_rows_kernel<MT, 0, kStreamPartials>);
  if (norm == kNormStack && out != kStreamPartials) return bf ? go(few_rows_kernel<MT, kNormStack, kStreamBf16>) : go(few_rows_kernel<MT, kNormStack, kStreamSwiglu>);
  if (norm == kNormLm && out != kStreamPartials) return bf ? go(few_rows_kernel<MT, kNormLm, kStreamBf16>) : go(few_rows_kernel<MT, kNormLm, kStreamSwiglu>);
  if (norm == kAddLm && bf) return go(few_rows_kernel<MT, kAddLm, kStreamBf16>);
  return cudaErrorInvalidValue;
}

template <typename F>
cudaError_t few_dispatch(int mts, int norm, int out, F&& go) {
  if (mts == 1) return few_dispatch_tile<1>(norm, out, go);
  if (mts == 2) return few_dispatch_tile<2>(norm, out, go);
  if (mts == 3) return few_dispatch_tile<3>(norm, out, go);
  if (mts == 4) return few_dispatch_tile<4>(norm, out, go);
  return few_dispatch_tile<10>(norm, out, go);
}

}  // namespace

void few_configure() {
  auto set = [](auto kernel) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFewMaxSmem + 1024); };
  for (int mts : {1, 2, 3, 4, 10})
    for (int norm : {0, (int)kNormStack, (int)kNormLm, (int)kAddLm})
      for (int out : {kStreamBf16, kStreamPartials, kStreamSwiglu}) few_dispatch(mts, norm, out, set);
}

static int few_rounds(int nkb, int splits, int rows) {
  const int lanes = 1 << few_lanes_log2(rows);
  return (few_per(nkb, splits) * 8 + lanes - 1) / lanes;
}

// Two pieces a lane only for rows of up to 2,048: longer ones (one row, that is) are in front of products long enough to hide
// the norm's own kernel, a Higgs step of one (2,560) 1,716 us folded and 1,598 apart, a duplex tick (4,096) 3,261 and 3,230;
// four rows of 1,024 the other way round, a talker step of four 2,431 us and 2,540.
bool few_norm_fits(int K, int rows) {
  return rows <= kFewRows && K % kKb == 0 && few_rounds(K / kKb, 1, rows) <= (K <= 2048 ? kNormChunks : 1);
}

// R weight rows a CTA, K in `splits`: what fits into shared memory and what it would cost (us behind the rows' arrival).
struct FewShape {
  int R, splits, slots;
  size_t smem;
  double cost, even;  // even: by the busiest SM's weights and rows alone
  bool early;         // most of every warp's share is under way before the rows are there
};

// Fitted to a sweep of R and the splits over nine shapes from 2,048 x 2,048 to 4,096 x 11,264 at one to eight rows. The
// terms: DRAM, less what the rings hold before the rows are there and more where CTAs are fewer than SMs; an SM's copies at
// 0.1 us each; a warp's chain of blocks, a round trip each unless the ring is deeper (one slot also adds to DRAM, as
// nothing is under way while a warp works); the rows' bytes. Against the most even load alone: 12,288 x 4,096 19.7 ->
// 14.7 us, 4,096 x 4,096 9.1 -> 6.8, 2,560 x 9,728 10.4 -> 8.4.
static FewShape few_shape(int N, int K, int rows, int R, int splits, int sm_count) {
  FewShape f{R, splits, 0, 0, 1e30, 1e30, false};
  const int nkb = K / kKb, per = few_per(nkb, splits), level = kWarps * R * kKb * 2;
  const int x_bytes = kWarps * rows * (per * kKb + 8) * 2;
  if (x_bytes > 72 * 1024) return f;
  f.slots = std::min(per, kFewSlots);
  if (1024 + x_bytes + f.slots * level > kFewMaxSmem) f.slots = std::max(1, (kFewHalf - 1024 - x_bytes) / level);
  if (1024 + x_bytes + f.slots * level > kFewMaxSmem) return f;
  f.smem = std::max<size_t>(kFewMinSmem, 1024 + (size_t)x_bytes + (size_t)f.slots * level);
  const double ctas = (N + R - 1) / R * splits, sms = sm_count, resident = f.smem <= kFewHalf ? 2 : 1;
  const double dram = 2.0 * N * K / 6.8e6 * std::max(1.0, sms / ctas) * (per <= f.slots ? 0.5 : 1.0);
  const double copies = ctas * kWarps * per / sms * 0.1;
  const double chain = per <= f.slots ? 0.2 * per : per * (0.55 + 0.0088 * R) / f.slots;
  const double x = rows * 2.0 * K / splits / 31e3 * std::ceil(std::min(ctas, resident * sms) / sms);
  // where the norm behind the product is folded into the next one, all of its CTAs read every sum
  const double sums = 0.15 * splits + (splits > 1 && few_norm_fits(N, rows) ? 4.0 * splits * rows * N / 150e3 : 0.0);
  f.cost = std::max({dram, copies, chain}) + (f.slots == 1 && per > 1 ? 0.35 * std::min(dram, chain) : 0.0);
  f.cost = f.cost * (ctas > resident * sms ? 1.1 : 1.0) + x + sums + 0.02 * copies;
  f.even = std::ceil(ctas / sms) * (R * 2.0 * K / splits / 44e3 + rows * 2.0 * K / splits / 31e3) + sums;
  f.early = 2 * per <= 3 * f.slots;
  return f;
}

int few_plan(FewPlan* plan, const bf16* w, int N, int K, const bf16* x, int rows, int out, bf16* y, int ldy, float* part,
             Epilogue epi, int sm_count, bool any_shape) {
  if (rows < 1 || rows > kFewRows || K % kKb || N < 1) return -2;
  if (!x && !few_norm_fits(K, rows)) return -2;
  if (out == kStreamSwiglu && N % (2 * kGateGroup)) return -2;
  if ((reinterpret_cast<uintptr_t>(w) & 15) || (reinterpret_cast<uintptr_t>(x) & 15)) return -3;
  FewPlan& p = *plan;
  p.N = N, p.K = K, p.rows = rows, p.out = out, p.x = x, p.y = y, p.ldy = ldy, p.part = part, p.epi = epi;
  FewShape best{};
  best.cost = 1e30;
  // The most even load of weights and rows, whose tiles are narrow and leave little to do behind the wait, where it has
  // most of every warp's share in its ring by then; otherwise by cost.
  FewShape even = best;
  even.even = 1e30;
  for (int R = 16; R <= 160; R += 16)
    for (int S : {1, 2, 4}) {
      if (S > 1 && (out != kStreamPartials || S * kWarps > K / kKb)) break;
      const FewShape shape = few_shape(N, K, rows, R, S, sm_count);
      if (shape.cost < best.cost) best = shape;
      if (shape.even < even.even) even = shape;
    }
  if (even.early) best = even;
  if (best.cost > 1e29) return -2;
  // Left to the tcgen05 kernel: rows that take so much of an SM's shared memory that the rings hold too little of the weights
  // (the line lies between the 40 and 48 KB of the nearest measured shapes), and from three rows on weights beyond the 126 MB of
  // L2, which no ring holds much of. As nodes of a tick or step, us for all of them, this kernel and that one, the rows' share in
  // brackets: 8 rows of 12,288 x 4,096 (32 layers, 64 KB) -103, 22,528 x 4,096 (64) -314, 4,096 x 11,264 (48) -109, but
  // 2,560 x 9,728 (36 layers, 40) +129, 19,456 x 2,560 (40) -6; 4 rows (32 KB) of 22,528 x 4,096, 185 MB, -108, but 12,288 x 4,096,
  // 101 MB, +111; 1 row of 22,528 x 4,096 +97.
  const size_t x_share = (size_t)few_per(K / kKb, best.splits) * kKb * kWarps * rows * 2;
  if (x && !any_shape && (x_share > 42 * 1024 || (rows > 2 && (int64_t)N * K > 64 << 20))) return -2;
  p.R = best.R, p.splits = best.splits, p.slots = best.slots, p.smem = best.smem;
  p.xk = few_per(K / kKb, p.splits) * kKb + 8;
  const int nkb = K / kKb;
  const uint64_t wd[3] = {kKb, (uint64_t)N, (uint64_t)nkb}, ws[2] = {(uint64_t)K * 2, kKb * 2};
  const uint32_t wb[3] = {kKb, (uint32_t)p.R, 1};
  return tc_encode_bf16(&p.wmap, w, 3, wd, ws, wb) == 0 ? 0 : -4;
}

cudaError_t few_launch(const FewPlan& p, const FewNorm& norm, uint32_t* err, cudaStream_t stream, const sm100::Ahead& ahead) {
  const int sums = norm.sum.splits;
  if (norm.kind && sums != 1 && sums != 2 && sums != 4) return cudaErrorInvalidValue;
  FewArgs a;
  a.x = p.x, a.y = p.y, a.part = p.part, a.bias = p.epi.bias, a.err = err, a.norm = norm, a.kind = p.epi.kind;
  a.inv_k = 1.f / (float)p.K, a.ahead = ahead;
  a.N = p.N, a.K = p.K, a.rows = p.rows, a.R = p.R, a.slots = p.slots, a.ldy = p.ldy;
  a.nkb = p.K / kKb, a.span = few_span(a.nkb, p.splits), a.per = few_per(a.nkb, p.splits), a.xk = p.xk;
  a.lanes_log2 = few_lanes_log2(p.rows), a.rounds = few_rounds(a.nkb, p.splits, p.rows);
  const dim3 grid((p.N + p.R - 1) / p.R, p.splits);
  return few_dispatch(p.R / 16, norm.kind, p.out, [&](auto kernel) {
    return launch_pdl(kernel, grid, dim3(kWarps * 32), p.smem, stream, p.wmap, a);
  });
}

}  // namespace omni
