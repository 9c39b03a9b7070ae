// The decode-sized GEMM of the kernel chains (see stream_gemm.h).
//
// Bound by its weights' bytes where they are many, by the path from the rows' arrival to the stores where they are few:
// rows to shared memory by TMA, the MMAs' issue, commit, TMEM to registers, stores. Hence the rows on M (64 or 128 TMEM
// lanes, a tile of weights as narrow as fills the chip once on N), weights asked for before the rows exist, four issuing
// threads and split K without a reduction of its own. Measured as nodes of a chain at 64 rows, from the rows' being there to the
// CTAs' end: 12,288 x 2,048 with SwiGLU 9.9 us (its weights alone take 7.7 us from DRAM), 12,288 x 4,096 18.1 us (15.4),
// 22,528 x 4,096 with SwiGLU 33.5 us (28.3), 4,096 x 1,024 3.0 us; a phase of the persistent tick kernel took 7 us at least.
#include "stream_gemm.h"

#include <algorithm>

#include "few_rows.h"
#include "pdl.cuh"
#include "sm100.cuh"
#include "wide_gemm.h"

namespace omni {
namespace {

constexpr int kKb = 64;  // K elements per k-block: one 128-byte swizzle row
constexpr int kMaxSlots = 8, kIssuers = 4;
constexpr int kThreads = 256;  // W producer, X producer, four MMA issuers, two more: all eight are the epilogue

struct StreamArgs {
  bf16* y;
  float* part;
  const bf16* bias;
  uint32_t* err;
  sm100::Ahead ahead;
  int N, rows, M, bn, tn, splits, kbs, stages, slots, issuers, ldy, kind, vec;
  uint32_t acc_cols, tmem_cols;
};

// P pieces of eight columns of 16 accumulator rows, `step` columns apart, the accumulators summed in issuer order: rows
// lane / 4 (v[p][0], v[p][1]) and lane / 4 + 8, columns 2 (lane % 4) and the next. Every load is under way before the wait.
template <int P>
__device__ __forceinline__ void acc_pieces(uint32_t addr, int step, int pieces, const StreamArgs& a, float (&v)[P][4]) {
  uint32_t r[kIssuers * P][4];
#pragma unroll
  for (int i = 0; i < kIssuers; ++i)
#pragma unroll
    for (int p = 0; p < P; ++p) {
      if (i < a.issuers && p < pieces) sm100::tmem_ld_16x8_issue(addr + (uint32_t)i * a.acc_cols + (uint32_t)(p * step), r[i * P + p]);
      else r[i * P + p][0] = r[i * P + p][1] = r[i * P + p][2] = r[i * P + p][3] = 0u;
    }
  sm100::tmem_ld_16x8_fence<kIssuers * P>(r);
#pragma unroll
  for (int p = 0; p < P; ++p)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      auto f = [&](int i) { return __uint_as_float(r[i * P + p][k]); };
      v[p][k] = (f(0) + f(1)) + (f(2) + f(3));
    }
}

template <int OUT>
__global__ void __launch_bounds__(kThreads, 1)
    stream_gemm_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap xmap,
                       const StreamArgs a) {
  using namespace sm100;
  extern __shared__ unsigned char stream_smem_raw[];
  __shared__ __align__(8) uint64_t bars_s[3 * kMaxSlots + 1];
  __shared__ uint32_t tmem_slot_s;
  __shared__ float bias_s[OUT == kStreamBf16 ? 256 : 1];
  const uint32_t base = (smem_addr(stream_smem_raw) + 1023u) & ~1023u;
  const uint32_t bars = smem_addr(bars_s);
  auto full_w = [&](int s) { return bars + 8u * s; };
  auto full_x = [&](int s) { return bars + 8u * (kMaxSlots + s); };
  auto empty = [&](int s) { return bars + 8u * (2 * kMaxSlots + s); };
  const uint32_t acc_bar = bars + 8u * (3 * kMaxSlots);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int tile = blockIdx.x, split = blockIdx.y, m0 = blockIdx.z * 128;
  const int st0 = (int)((int64_t)a.stages * split / a.splits), st1 = (int)((int64_t)a.stages * (split + 1) / a.splits);
  const int n_st = st1 - st0;
  const uint32_t x_slice = (uint32_t)a.bn * 128u, w_slice = (uint32_t)a.tn * 128u;
  const uint32_t x_bytes = x_slice * (uint32_t)a.kbs, w_bytes = w_slice * (uint32_t)a.kbs, slot_bytes = x_bytes + w_bytes;

  auto load_w = [&](int i, int slot) {  // stage st0 + i's weights
    mbar_expect_tx(full_w(slot), w_bytes);
    tma_load_3d(base + (uint32_t)slot * slot_bytes + x_bytes, &wmap, full_w(slot), 0, tile * a.tn, (st0 + i) * a.kbs, kEvictFirst);
  };

  if (threadIdx.x == 0) {
    prefetch_tensormap(&wmap);
    for (int s = 0; s < a.slots; ++s) mbar_init(full_w(s), 1), mbar_init(full_x(s), 1), mbar_init(empty(s), 1);
    mbar_init(acc_bar, a.issuers);
    mbar_init_fence();
    for (int i = 0; i < min(a.slots, n_st); ++i) load_w(i, i);
    prefetch_tensormap(&xmap);
  }
  if (warp == 2) tmem_alloc(smem_addr(&tmem_slot_s), a.tmem_cols);
  if constexpr (OUT == kStreamBf16) {
    if (a.kind != kEpiNone && (int)threadIdx.x < min(a.tn, a.N - tile * a.tn)) bias_s[threadIdx.x] = __bfloat162float(a.bias[tile * a.tn + threadIdx.x]);
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tmem_slot_s);
  // only now: were the next kernel let in before this CTA has its TMEM columns, it could take them and then wait for
  // this kernel to complete
  grid_trigger();

  if (warp == 0) {
    if (lane == 0) {
      int slot = 0;
      uint32_t phase = 0;
      for (int i = a.slots; i < n_st; ++i) {
        if (!mbar_wait(empty(slot), phase, a.err)) {
          drain_ring(full_w(0), a.slots, i, a.err);
          break;
        }
        load_w(i, slot);
        if (++slot == a.slots) slot = 0, phase ^= 1u;
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      grid_wait();
      fence_async_global();  // rows written by ordinary stores, read by TMA
      int slot = 0;
      uint32_t phase = 0;
      for (int i = 0; i < n_st; ++i) {
        if (i >= a.slots && !mbar_wait(empty(slot), phase ^ 1u, a.err)) {
          drain_ring(full_x(0), a.slots, i, a.err);
          break;
        }
        mbar_expect_tx(full_x(slot), x_bytes);
        tma_load_3d(base + (uint32_t)slot * slot_bytes, &xmap, full_x(slot), 0, m0, (st0 + i) * a.kbs, kEvictLast);
        if (++slot == a.slots) slot = 0, phase ^= 1u;
      }
    }
  } else if (warp < 2 + kIssuers) {
    // issuer `me` takes stages me, me + issuers, ... into its own accumulator: one thread issues an MMA only every
    // 80 cycles or so, half of what the tensor pipe takes at these shapes
    const int me = warp - 2;
    if (me < a.issuers) {
      const uint32_t idesc = idesc_bf16_f32(a.M, a.tn), acc = tmem + (uint32_t)me * a.acc_cols;
      bool alive = true;
      int slot = me % a.slots;
      uint32_t phase = (uint32_t)(me / a.slots) & 1u;
      for (int i = me; i < n_st; i += a.issuers) {
        alive = mbar_wait(full_w(slot), phase, a.err) && mbar_wait(full_x(slot), phase, a.err);
        if (!alive) break;
        tc_fence_after_sync();
        const uint64_t adesc = kmajor_sw128_desc(base + (uint32_t)slot * slot_bytes);
        const uint64_t bdesc = kmajor_sw128_desc(base + (uint32_t)slot * slot_bytes + x_bytes);
        if (elect_one()) {
          for (int j = 0; j < a.kbs; ++j) {
            const uint64_t ad = adesc + (uint64_t)((uint32_t)j * (x_slice >> 4)), bd = bdesc + (uint64_t)((uint32_t)j * (w_slice >> 4));
#pragma unroll
            for (int k = 0; k < kKb / 16; ++k)
              mma_bf16(acc, ad + (uint64_t)(k * 2), bd + (uint64_t)(k * 2), idesc, (i > me || j > 0 || k > 0) ? 1u : 0u);
          }
          mma_commit(empty(slot));
        }
        __syncwarp();
        slot += a.issuers;
        while (slot >= a.slots) slot -= a.slots, phase ^= 1u;
      }
      if (alive && elect_one()) mma_commit(acc_bar);
      __syncwarp();
    }
  }
  else if (warp == 7 && elect_one()) ask_ahead(a.ahead, (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x, gridDim.x * gridDim.y * gridDim.z);
  __syncwarp();

  // ---- epilogue: two warps a TMEM quadrant, sixteen rows at a time as m16n8 fragments, so that every lane has work where
  // M = 64 leaves half of a quadrant's lanes empty. M = 64: the quadrant's rows are 16 q .. 16 q + 15, and its warps share
  // the columns; M = 128: 32 q .. 32 q + 31, sixteen a warp. From the last product to the CTA's end at 64 rows, before
  // (four warps, a row a lane, eight columns at a time) and now: 48 columns with SwiGLU 1.9 and 1.0 us, 176 columns 4.9 and
  // 2.6, 96 columns of bf16 4.5 and 1.9, 32 columns 2.0 and 1.1, 64 columns of partial sums 1.4 and 0.9.
  const int quad = warp & 3, half = warp >> 2, g = lane >> 2, t2 = (lane & 3) * 2;
  const int r0 = a.M == 128 ? quad * 32 + half * 16 : quad * 16;
  const uint32_t lane_addr = tmem + ((uint32_t)(quad * 32 + (a.M == 128 ? half * 16 : 0)) << 16);
  const int m_lo = m0 + r0 + g, m_hi = m_lo + 8;
  const bool lo = m_lo < a.rows, hi = m_hi < a.rows;
  // units of this warp: groups of gates and their ups, or pieces of eight columns
  const int n0 = tile * a.tn, width = min(a.tn, a.N - n0), unit = OUT == kStreamSwiglu ? 2 * kGateGroup : 8;
  const int units = (width + unit - 1) / unit, share = a.M == 128 ? units : (units + 1) >> 1;
  const int u0 = a.M == 128 ? 0 : half * share, u1 = min(units, u0 + share);
  grid_wait();
  const bool ok = mbar_wait(acc_bar, 0, a.err);
  tc_fence_after_sync();
  if (ok && m0 + r0 < a.rows) {
    if constexpr (OUT == kStreamSwiglu) {
      constexpr int P = 2;
      bf16* const y = a.y + (size_t)m_lo * a.ldy + (n0 >> 1) + t2;
      for (int u = u0; u < u1; u += P) {
        float v[2 * P][4];
        acc_pieces<2 * P>(lane_addr + (uint32_t)(u * 16), 8, 2 * (u1 - u), a, v);
#pragma unroll
        for (int p = 0; p < P; ++p) {
          float o[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) o[k] = silu_bf16(bf16_round(v[2 * p][k])) * bf16_round(v[2 * p + 1][k]);
          if (u + p < u1) {
            if (lo) *reinterpret_cast<__nv_bfloat162*>(y + (u + p) * kGateGroup) = __floats2bfloat162_rn(o[0], o[1]);
            if (hi) *reinterpret_cast<__nv_bfloat162*>(y + (size_t)8 * a.ldy + (u + p) * kGateGroup) = __floats2bfloat162_rn(o[2], o[3]);
          }
        }
      }
    } else {
      constexpr int P = 4;
      for (int u = u0; u < u1; u += P) {
        float v[P][4];
        acc_pieces<P>(lane_addr + (uint32_t)(u * 8), 8, u1 - u, a, v);
#pragma unroll
        for (int p = 0; p < P; ++p) {
          if (u + p >= u1) break;
          const int c = (u + p) * 8 + t2, n = n0 + c;
          if constexpr (OUT == kStreamPartials) {
            float* dst = a.part + ((size_t)split * a.rows + m_lo) * a.N + n;
            if (lo) *reinterpret_cast<float2*>(dst) = make_float2(v[p][0], v[p][1]);
            if (hi) *reinterpret_cast<float2*>(dst + (size_t)8 * a.N) = make_float2(v[p][2], v[p][3]);
          } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              v[p][k] = bf16_round(v[p][k]);
              if (a.kind != kEpiNone) {  // (past the row's end: a sum that is not stored)
                v[p][k] = bf16_round(v[p][k] + bias_s[c + (k & 1)]);
                if (a.kind == kEpiBiasSilu) v[p][k] = v[p][k] / (1.f + __expf(-v[p][k]));
              }
            }
            bf16* dst = a.y + (size_t)m_lo * a.ldy + n;
            bf16* dst8 = dst + (size_t)8 * a.ldy;
            if (a.vec) {
              if (lo) *reinterpret_cast<__nv_bfloat162*>(dst) = __floats2bfloat162_rn(v[p][0], v[p][1]);
              if (hi) *reinterpret_cast<__nv_bfloat162*>(dst8) = __floats2bfloat162_rn(v[p][2], v[p][3]);
            } else {
#pragma unroll
              for (int k = 0; k < 2; ++k) {
                if (lo && n + k < a.N) dst[k] = __float2bfloat16(v[p][k]);
                if (hi && n + k < a.N) dst8[k] = __float2bfloat16(v[p][2 + k]);
              }
            }
          }
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 2) tmem_dealloc(tmem, a.tmem_cols);
}

// More than half of an SM's shared memory whatever the ring needs: kernels of a chain start on whichever SM has room, so
// CTAs small enough to share an SM would pile up on the first ones free and leave the rest of the chip idle.
constexpr int kMinSmem = 116 * 1024, kMaxSmem = 200 * 1024;

}  // namespace

void stream_configure() {
  few_configure();
  wide_configure();
  cudaFuncSetAttribute(stream_gemm_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
  cudaFuncSetAttribute(stream_gemm_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
  cudaFuncSetAttribute(stream_gemm_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
}

bool stream_supports(int N, int K, int rows) { return K % kKb == 0 && K >= kKb && N >= 1 && rows >= 1; }

// Weight rows per tile (tn) and K splits: the shape with the shortest estimated time after the inputs are there. A CTA
// pulls its tile's rows at about 120 GB/s whatever the number of CTAs (they all read the same rows, while the weights of later
// GEMMs are on their way). That is a fit: with 170, as its weights, a talker step of 64 sessions took 3,375 us instead of 3,351,
// of 128 4,629 and 4,596; with 90 3,335, 4,596, but a duplex tick of 64 5,175 instead of 5,135. The tensor pipe
// takes (M + tn) / 4 cycles per 16 elements of K, stores leave an SM at 57 GB/s, and weights only count where a shape
// loads some SMs more than others, since they were asked for before the inputs were there.
static double stream_cost(int N, int K, int rows, int M, int bn, int tn, int S, int out, int sms, int row_tiles) {
  const int ctas = (N + tn - 1) / tn * S * row_tiles;
  const double per_sm = (ctas + sms - 1) / sms, kc = (double)K / S;
  const double t_x = kc * 2 * bn * per_sm / 120e3;
  const double t_w = kc * 2 * tn * per_sm / std::min(170e3, 6.5e6 / std::min(ctas, sms));
  const double t_mma = kc / 16 * std::max(0.25 * (M + tn), tn > 128 ? 40.0 : 20.0) * per_sm / 1900;
  const double t_out = std::min(rows, 128) * tn * (out == kStreamPartials ? 4.0 : out == kStreamSwiglu ? 1.0 : 2.0) * per_sm / 57e3;
  return std::max({t_x + 0.3 * t_mma, t_mma, 0.5 * t_x + t_w}) + t_out + 0.1 * S;
}

int stream_plan(StreamGemmPlan* plan, const bf16* w, int N, int K, const bf16* x, int rows, int out, bf16* y, int ldy,
                float* part, Epilogue epi, int sm_count, int force_splits) {
  if (!stream_supports(N, K, rows)) return -2;
  if (out == kStreamPartials && N % 8) return -2;
  if (out == kStreamSwiglu && (N % (2 * kGateGroup) || ldy % 8)) return -2;
  if ((reinterpret_cast<uintptr_t>(w) & 15) || (reinterpret_cast<uintptr_t>(x) & 15)) return -3;
  if (out == kStreamSwiglu && (reinterpret_cast<uintptr_t>(y) & 15)) return -3;
  StreamGemmPlan& p = *plan;
  p.N = N, p.K = K, p.rows = rows, p.out = out, p.y = y, p.ldy = ldy, p.part = part, p.epi = epi;
  p.M = rows <= 64 ? 64 : 128;
  p.bn = std::min(128, (rows + 7) / 8 * 8);
  const int nkb = K / kKb, row_tiles = (rows + 127) / 128;
  double best = 1e30;
  for (int tn = 16; tn <= 256; tn += 16)
    for (int S : {1, 2, 4, 8}) {
      if (S > 1 && (out != kStreamPartials || S * 2 > nkb)) break;
      if (force_splits > 0 && S != force_splits) continue;
      const double cost = stream_cost(N, K, rows, p.M, p.bn, tn, S, out, sm_count, row_tiles);
      if (cost < best - 1e-9) best = cost, p.tn = tn, p.splits = S;
    }
  if (best > 1e29) return -2;
  // k-blocks per stage: as many (up to four) as leave three stages in the ring; a copy costs its thread about 0.16 us
  const int kb_bytes = (p.bn + p.tn) * 128, room = kMaxSmem - 1024 - (p.M - p.bn) * 128;
  p.kbs = 1;
  for (int k : {4, 2})
    if (k * 2 <= nkb / p.splits && room / (k * kb_bytes) >= 3) {
      p.kbs = k;
      break;
    }
  p.stages = (nkb + p.kbs - 1) / p.kbs;
  const int per = (p.stages + p.splits - 1) / p.splits;
  p.slots = std::min({kMaxSlots, per, room / (p.kbs * kb_bytes)});
  if (p.slots < 1 || p.stages < p.splits) return -2;
  p.acc_cols = p.tn <= 32 ? 32 : p.tn <= 64 ? 64 : p.tn <= 128 ? 128 : 256;
  // a slot belongs to one issuer for good (slots is a multiple of issuers): a wait on a barrier parity means "this phase"
  // only to a thread that has seen every phase of the barrier. Every split has a stage for each issuer.
  p.issuers = std::min({kIssuers, p.stages / p.splits, 512 / p.acc_cols, p.slots});
  p.slots -= p.slots % p.issuers;
  const uint64_t wd[3] = {kKb, (uint64_t)N, (uint64_t)nkb}, ws[2] = {(uint64_t)K * 2, kKb * 2};
  const uint32_t wb[3] = {kKb, (uint32_t)p.tn, (uint32_t)p.kbs};
  if (tc_encode_bf16(&p.wmap, w, 3, wd, ws, wb) != 0) return -4;
  const uint64_t xd[3] = {kKb, (uint64_t)rows, (uint64_t)nkb}, xs[2] = {(uint64_t)K * 2, kKb * 2};
  const uint32_t xb[3] = {kKb, (uint32_t)p.bn, (uint32_t)p.kbs};
  if (tc_encode_bf16(&p.xmap, x, 3, xd, xs, xb) != 0) return -4;
  return 0;
}

cudaError_t stream_launch(const StreamGemmPlan& p, uint32_t* err, cudaStream_t stream, bool whole_smem, const sm100::Ahead& ahead) {
  StreamArgs a;
  a.ahead = ahead;
  a.y = p.y, a.part = p.part, a.bias = p.epi.bias, a.err = err, a.kind = p.epi.kind;
  a.N = p.N, a.rows = p.rows, a.M = p.M, a.bn = p.bn, a.tn = p.tn, a.splits = p.splits, a.kbs = p.kbs;
  a.stages = p.stages, a.slots = p.slots, a.issuers = p.issuers, a.ldy = p.ldy;
  a.vec = p.ldy % 8 == 0 && p.N % 8 == 0 && (reinterpret_cast<uintptr_t>(p.y) & 15) == 0;
  a.acc_cols = (uint32_t)p.acc_cols;
  a.tmem_cols = 32;
  while (a.tmem_cols < a.acc_cols * (uint32_t)p.issuers) a.tmem_cols *= 2;
  const size_t smem = std::max<size_t>(kMinSmem, 1024 + (size_t)p.slots * p.kbs * (p.bn + p.tn) * 128 + (size_t)(p.M - p.bn) * 128);
  const dim3 grid((p.N + p.tn - 1) / p.tn, p.splits, (p.rows + 127) / 128);
  switch (p.out) {
    case kStreamBf16: return launch_pdl_smem(whole_smem, stream_gemm_kernel<0>, grid, dim3(kThreads), smem, stream, p.wmap, p.xmap, a);
    case kStreamPartials: return launch_pdl_smem(whole_smem, stream_gemm_kernel<1>, grid, dim3(kThreads), smem, stream, p.wmap, p.xmap, a);
    default: return launch_pdl_smem(whole_smem, stream_gemm_kernel<2>, grid, dim3(kThreads), smem, stream, p.wmap, p.xmap, a);
  }
}

}  // namespace omni
