// The codec decoder's causal conv as an implicit GEMM on tcgen05 (declared in codec.h).
//
// The reference materialises every conv's dilated im2col matrix [rows, taps * C] and hands it to a library GEMM
// (crates/omni-qwen3-tts/src/codec.rs:60-93, kernels/codec.cu:291-318). Here the im2col matrix never exists: the
// activation is kept once, padded with its history, as [stream][H + T][C], and the K loop walks (tap, channel block);
// for tap j the activation tile of 128 output rows is the same rank-3/4 TMA box shifted down by j * dil rows. The rows
// of a tile are SB streams x TB consecutive frame rows (TB * SB = 128), so a tile never reads across a stream's padding.
//
//   warp 0: weight producer, a ring of {activation tile x kbs, weight tile tn x 64 x kbs}; the first loads of a launch go
//           out before the kernels in front have finished (the weights, 0.2 GB, do not stay in L2 from frame to frame);
//   warp 1: activation producer;
//   warps 2, 3: MMA issuers (M = 128 rows, N = tn output channels). One thread issues an MMA every 80 to 100 cycles and
//           spends 200 on a stage's wait and commit, twice what narrow tiles' MMAs take, so two issuers take the
//           stages in turn (four gain nothing more: 13.4 and 13.0 us for 768 x 5,376 at one stream, 17.0 us with one), each with its own accumulator; a stage of the ring belongs to one issuer for good;
//   twelve warps: epilogue, three per TMEM lane quadrant, 32 channels of 32 rows per step. The epilogue (SnakeBeta over
//           every value of a tile, or a read-modify-write of the residual stream) is hidden behind the next tile's K
//           loop by a second set of accumulators where a CTA has more than one tile.
//
// Channel counts that are not multiples of 64 (96 in the last decoder block) take the "ragged" loads: the activation
// box past channel C is zero-filled by TMA, so whatever weight columns of the next tap the weight box then covers
// multiply zeros.
#include <algorithm>

#include "codec.h"
#include "gemm.h"
#include "sm100.cuh"
#include "pdl.cuh"

namespace omni {

namespace {

constexpr int kConvK = 64;        // channels per k-block: one 128-byte swizzle row
constexpr int kConvRows = 128;    // output rows per tile
constexpr int kConvRing = 168 * 1024;
constexpr int kConvMaxStages = 8, kConvIssuers = 2;
constexpr int kConvEpilogueWarps = 12;  // three per TMEM lane quadrant, each taking every third 32-channel step
constexpr int kConvThreads = 32 * (2 + kConvIssuers + kConvEpilogueWarps);
constexpr int kStagePitch = 36;   // floats per row of an epilogue warp's 32 x 32 staging block (16-byte aligned, conflict-free)
constexpr size_t kConvSmem = (size_t)kConvRing + 1024 + kConvEpilogueWarps * 32 * kStagePitch * sizeof(float);
static_assert(kConvSmem <= 232448 - 512, "shared memory of a CTA");

struct ConvArgs {
  bf16* y;
  const bf16* bias;
  const float* alpha;
  const float* inv_b;
  uint32_t* err;
  int N, C, taps, dil, T, seqs, TB, SB, tb_log2, tn, kbs, cpb, ragged, stages, kind, t_tiles, n_tiles, tiles, box_rows, issuers, bufs;
  uint32_t acc_cols, tmem_cols;  // TMEM columns per accumulator (a power of two >= tn) and in all
};

// The walk over a launch's tiles without a division per tile: tile = n + n_tiles * (t + t_tiles * s).
struct TileWalk {
  int n, t, s, dn, dt, ds;
  __device__ __forceinline__ explicit TileWalk(const ConvArgs& a) {
    auto split = [&](int v, int& n_, int& t_, int& s_) {
      n_ = v % a.n_tiles;
      const int r = v / a.n_tiles;
      t_ = r % a.t_tiles, s_ = r / a.t_tiles;
    };
    split((int)blockIdx.x, n, t, s);
    split((int)gridDim.x, dn, dt, ds);
  }
  __device__ __forceinline__ void next(const ConvArgs& a) {
    n += dn, t += dt, s += ds;
    if (n >= a.n_tiles) n -= a.n_tiles, ++t;
    if (t >= a.t_tiles) t -= a.t_tiles, ++s;
  }
};

// Persistent: a CTA walks tiles blockIdx.x, blockIdx.x + gridDim.x, ... (output-channel tile fastest, so CTAs that run
// together share activation rows in L2). The ring never drains between tiles.
__global__ void __launch_bounds__(kConvThreads, 1)
    conv_gemm_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                     const __grid_constant__ ConvArgs a) {
  using namespace sm100;
  extern __shared__ unsigned char conv_smem_raw[];
  __shared__ __align__(8) uint64_t bars_s[2 * kConvMaxStages + 4];
  __shared__ uint32_t tmem_slot_s;
  __shared__ int gave_up_s, issued_s[2];  // a wait ran out; stages the producers had filled by then (-1: all)
  const uint32_t raw = smem_addr(conv_smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* base_ptr = conv_smem_raw + (base - raw);
  const uint32_t x_slice = (uint32_t)a.box_rows * kConvK * 2, x_bytes = (uint32_t)a.kbs * x_slice;
  const uint32_t w_slice = (uint32_t)a.tn * kConvK * 2, w_bytes = (uint32_t)a.kbs * w_slice, stage_bytes = x_bytes + w_bytes;
  const uint32_t bars = smem_addr(bars_s);
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (kConvMaxStages + s); };
  auto acc_full = [&](int b) { return bars + 8u * (2 * kConvMaxStages + b); };
  auto acc_empty = [&](int b) { return bars + 8u * (2 * kConvMaxStages + 2 + b); };
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int steps = a.taps * a.cpb / a.kbs;
  // weights first in a stage, then the activation box (whose MMA reads may run past the stage)
  auto load_w = [&](int n0, int tap, int cb, int stage) {
    mbar_expect_tx(full_bar(stage), w_bytes);
    if (a.ragged) tma_load_2d(base + stage * stage_bytes, &wmap, full_bar(stage), tap * a.C + cb * kConvK, n0, kEvictLast);
    else tma_load_3d(base + stage * stage_bytes, &wmap, full_bar(stage), 0, n0, tap * a.cpb + cb, kEvictLast);
  };

  if (threadIdx.x == 0) {
    gave_up_s = 0, issued_s[0] = issued_s[1] = -1;
    prefetch_tensormap(&wmap);
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(full_bar(s), 2);  // the two producers
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full(b), a.issuers);
      mbar_init(acc_empty(b), kConvEpilogueWarps);  // one arrival per epilogue warp
    }
    mbar_init_fence();
    for (int i = 0, tap = 0, cb = 0; i < min(a.stages, steps); ++i) {
      load_w(((int)blockIdx.x % a.n_tiles) * a.tn, tap, cb, i);
      cb += a.kbs;
      if (cb >= a.cpb) cb = 0, ++tap;
    }
    prefetch_tensormap(&xmap);
  }
  if (warp == 2) tmem_alloc(smem_addr(&tmem_slot_s), a.tmem_cols);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&tmem_slot_s);
  grid_trigger();  // not before this CTA holds its TMEM columns: the next kernel could take them and wait for this one
  if (warp != 0) grid_wait();

  if (warp < 2) {
    if (lane == 0) {
      const bool is_w = warp == 0;
      if (!is_w) fence_async_global();  // rows written by ordinary stores, read by TMA
      int stage = 0, done = 0;
      uint32_t phase = 0;
      bool alive = true;
      TileWalk at(a);
      for (int tile = blockIdx.x; tile < a.tiles && alive; tile += gridDim.x, at.next(a)) {
        const int n0 = at.n * a.tn, t0 = at.t * a.TB, s0 = at.s * a.SB;
        int tap = 0, cb = 0;
        for (int i = 0; i < steps; ++i, ++done) {
          if (done >= a.stages) {
            alive = mbar_wait(empty_bar(stage), phase ^ 1u, a.err);
            if (!alive) break;
          }
          if (is_w) {
            if (done >= min(a.stages, steps)) load_w(n0, tap, cb, stage);  // the first ones are under way already
          } else {
            const uint32_t dst = base + stage * stage_bytes + w_bytes;
            mbar_expect_tx(full_bar(stage), x_bytes);
            if (a.ragged) tma_load_3d(dst, &xmap, full_bar(stage), cb * kConvK, t0 + tap * a.dil, s0, kEvictNormal);
            else tma_load_4d(dst, &xmap, full_bar(stage), 0, t0 + tap * a.dil, s0, cb, kEvictNormal);
          }
          cb += a.kbs;
          if (cb >= a.cpb) cb = 0, ++tap;
          if (++stage == a.stages) stage = 0, phase ^= 1u;
        }
      }
      if (!alive) gave_up_s = 1, issued_s[warp] = done;
    }
    __syncwarp();
  } else if (warp < 2 + kConvIssuers) {
    const int me = warp - 2;
    if (me < a.issuers) {
      const uint32_t idesc = idesc_bf16_f32(kConvRows, a.tn);
      const int ragged_k = a.ragged ? (a.C - (a.cpb - 1) * kConvK + 15) / 16 : kConvK / 16;  // 16-channel steps of a tap's last block
      int use = 0, count = me;  // count: this issuer's next stage, counted over the launch
      int stage = me % a.stages;
      uint32_t phase = (uint32_t)(me / a.stages) & 1u;
      bool alive = true;
      int tile_first = 0;
      for (int tile = blockIdx.x; tile < a.tiles && alive; tile += gridDim.x, ++use, tile_first += steps) {
        const int buf = a.bufs == 2 ? use & 1 : 0, turn = a.bufs == 2 ? use >> 1 : use;
        // the epilogue of this accumulator's previous tile must have read it out (a fresh barrier passes at once)
        alive = mbar_wait(acc_empty(buf), ((uint32_t)turn & 1u) ^ 1u, a.err);
        if (!alive) break;
        tc_fence_after_sync();
        const uint32_t acc = tmem_base + (uint32_t)(buf * a.issuers + me) * a.acc_cols;
        bool more = false;
        for (; count < tile_first + steps; count += a.issuers) {
          alive = mbar_wait(full_bar(stage), phase, a.err);
          if (!alive) break;
          tc_fence_after_sync();
          if (elect_one()) {
            const uint64_t bdesc = kmajor_sw128_desc(base + stage * stage_bytes), adesc = kmajor_sw128_desc(base + stage * stage_bytes + w_bytes);
            const int ks = a.ragged && (count - tile_first) % a.cpb == a.cpb - 1 ? ragged_k : kConvK / 16;
            for (int j = 0; j < a.kbs; ++j) {
              const uint64_t ad = adesc + (uint64_t)((uint32_t)j * (x_slice >> 4)), bd = bdesc + (uint64_t)((uint32_t)j * (w_slice >> 4));
#pragma unroll
              for (int k = 0; k < kConvK / 16; ++k)
                if (k < ks) mma_bf16(acc, ad + (uint64_t)(k * 2), bd + (uint64_t)(k * 2), idesc, (more || j > 0 || k > 0) ? 1u : 0u);
            }
            mma_commit(empty_bar(stage));
          }
          __syncwarp();
          more = true;
          stage += a.issuers;
          while (stage >= a.stages) stage -= a.stages, phase ^= 1u;
        }
        if (alive && elect_one()) mma_commit(acc_full(buf));
        __syncwarp();
      }
      if (!alive && lane == 0) gave_up_s = 1;
    }
  } else {
    // Epilogue. A warp reaches the 32 TMEM lanes of quadrant warp % 4, one output row per thread, and takes the tile 32
    // channels at a time. A thread's row is 2 * N bytes away from its neighbour's, so storing from that layout would
    // cost one memory transaction per thread and 16 bytes; instead the 32 x 32 f32 block goes through shared memory
    // and comes back with four lanes per row (8 channels each), so that a warp instruction covers 8 rows x 64 bytes.
    // The old values of an accumulating GEMM, the bias and the SnakeBeta parameters are read in that layout too.
    const int quad = warp & 3, turn = (warp - 2 - kConvIssuers) >> 2;  // this warp takes steps turn, turn + 3, ... of 32 channels
    float* stg = reinterpret_cast<float*>(base_ptr + kConvRing) + (warp - 2 - kConvIssuers) * (32 * kStagePitch);
    const int sub_row = lane >> 2, chunk = lane & 3;
    // the four rows this lane stores in every step, relative to the tile's first
    int stream_of[4];
    uint32_t row_at[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int m = quad * 32 + 8 * i + sub_row;
      stream_of[i] = m < a.box_rows ? m >> a.tb_log2 : a.seqs;  // never live past the box
      row_at[i] = (uint32_t)((stream_of[i] * a.T + (m & (a.TB - 1))) * a.N);
    }
    int use = 0;
    bool alive = true;
    TileWalk at(a);
    for (int tile = blockIdx.x; tile < a.tiles && alive; tile += gridDim.x, ++use, at.next(a)) {
      const int buf = a.bufs == 2 ? use & 1 : 0, round = a.bufs == 2 ? use >> 1 : use;
      const int n0 = at.n * a.tn, live_streams = a.seqs - at.s * a.SB;
      bf16* const tile_y = a.y + ((int64_t)at.s * a.SB * a.T + at.t * a.TB) * a.N;
      const uint32_t lane_addr = tmem_base + (uint32_t)(buf * a.issuers) * a.acc_cols + ((uint32_t)(quad * 32) << 16);
      const bool warp_live = __any_sync(0xffffffffu, stream_of[0] < live_streams);
      // the residual's old values of this warp's first step are asked for before the accumulator is there
      uint4 old[4] = {};
      auto load_old = [&](int c0) {
        const int nn = n0 + c0 + 8 * chunk;
        if (a.kind == kConvAccumulate && c0 + 8 * chunk < a.tn && nn + 8 <= a.N) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (stream_of[i] < live_streams) old[i] = __ldcg(reinterpret_cast<const uint4*>(tile_y + row_at[i] + nn));
        }
      };
      load_old(32 * turn);
      alive = mbar_wait(acc_full(buf), (uint32_t)round & 1u, a.err);
      if (!alive) break;
      tc_fence_after_sync();
#pragma unroll 1
      for (int c0 = warp_live ? 32 * turn : a.tn; c0 < a.tn; c0 += 32 * (kConvEpilogueWarps / 4)) {
        uint32_t r0[16], r1[16];
        const bool second = c0 + 16 < a.tn;  // tn is a multiple of 16: the last step may hold one half only
        tmem_ld16_issue(lane_addr + c0, r0);  // warp-wide: every lane takes part whether or not its row is live
        if (second) {
          tmem_ld16_issue(lane_addr + c0 + 16, r1);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) r1[j] = 0u;
        }
        const int nn = n0 + c0 + 8 * chunk;
        const bool cols_live = c0 + 8 * chunk < a.tn && nn + 8 <= a.N;
        if (c0 != 32 * turn) load_old(c0);
        tmem_ld_fence(r0, r1);
        for (int q = 1; q < a.issuers; ++q) {  // the other issuers' sums, in their order
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (h == 1 && !second) break;
            float o[16];
            tmem_ld16(lane_addr + (uint32_t)q * a.acc_cols + c0 + 16 * h, o);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              uint32_t& r = h == 0 ? r0[j] : r1[j];
              r = __float_as_uint(__uint_as_float(r) + o[j]);
            }
          }
        }
        uint4* mine = reinterpret_cast<uint4*>(stg + lane * kStagePitch);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          mine[q] = make_uint4(r0[4 * q], r0[4 * q + 1], r0[4 * q + 2], r0[4 * q + 3]);
          mine[4 + q] = make_uint4(r1[4 * q], r1[4 * q + 1], r1[4 * q + 2], r1[4 * q + 3]);
        }
        __syncwarp();
        if (cols_live) {
          float b[8], al[8], ib[8];
          if (a.kind == kConvBiasSnake) {
            ld8v(a.bias + nn, b);
            const float4 a0 = *reinterpret_cast<const float4*>(a.alpha + nn), a1 = *reinterpret_cast<const float4*>(a.alpha + nn + 4);
            const float4 i0 = *reinterpret_cast<const float4*>(a.inv_b + nn), i1 = *reinterpret_cast<const float4*>(a.inv_b + nn + 4);
            al[0] = a0.x, al[1] = a0.y, al[2] = a0.z, al[3] = a0.w, al[4] = a1.x, al[5] = a1.y, al[6] = a1.z, al[7] = a1.w;
            ib[0] = i0.x, ib[1] = i0.y, ib[2] = i0.z, ib[3] = i0.w, ib[4] = i1.x, ib[5] = i1.y, ib[6] = i1.z, ib[7] = i1.w;
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (stream_of[i] >= live_streams) continue;
            const float4* src = reinterpret_cast<const float4*>(stg + (8 * i + sub_row) * kStagePitch + 8 * chunk);
            const float4 lo = src[0], hi = src[1];
            float o[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            if (a.kind == kConvAccumulate) {
              float prev[8];
              unpack8v(old[i], prev);
#pragma unroll
              for (int j = 0; j < 8; ++j) o[j] += prev[j];
            } else if (a.kind == kConvBiasSnake) {
#pragma unroll
              for (int j = 0; j < 8; ++j) o[j] = snake_beta(bf16_round(o[j]) + b[j], al[j], ib[j]);
            }
            st8v(tile_y + row_at[i] + nn, o);
          }
        }
        __syncwarp();  // the block is read out before the next step overwrites it
      }
      // this warp's part of the accumulator has been read (a warp without a step of its own arrives all the same)
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty(buf));
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (gave_up_s && threadIdx.x == 0) {
    // no copy may land once the CTA has left: a stage that only one producer filled gets the other's arrival from here,
    // so that its barrier, too, tells when the copy is there
    const int all = ((a.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x) * steps;
    const int w = issued_s[0] < 0 ? all : issued_s[0], x = issued_s[1] < 0 ? all : issued_s[1];
    for (int i = min(w, x); i < max(w, x); ++i) mbar_arrive(full_bar(i % a.stages));
    drain_ring(full_bar(0), a.stages, max(w, x), a.err);
  }
  if (warp == 2) tmem_dealloc(tmem_base, a.tmem_cols);
}

// How a launch of `tn` output channels a tile is run: k-blocks per stage and copy, stages, issuers, sets of accumulators.
struct ConvShape {
  int kbs, stages, issuers, bufs, acc_cols;
  double cycles;
};

ConvShape conv_shape(const ConvGemmPlan& p, int tn, int sm_count) {
  const int tiles = (p.N + tn - 1) / tn * p.row_tiles, waves = (tiles + sm_count - 1) / sm_count, kb = p.taps * p.cpb;
  ConvShape best{};
  best.cycles = 1e30;
  for (int kbs : {4, 3, 2, 1}) {
    if (kbs > 1 && (p.ragged || p.cpb % kbs)) continue;
    ConvShape s{};
    const int bytes = (p.box_rows + tn) * kConvK * 2, steps = kb / kbs;
    s.kbs = kbs, s.bufs = waves > 1 ? 2 : 1, s.acc_cols = tn <= 32 ? 32 : tn <= 64 ? 64 : tn <= 128 ? 128 : 256;
    // an MMA reads 128 rows from where the box starts: the last one must end inside the ring
    s.stages = std::min(kConvMaxStages, (kConvRing - (kConvRows - p.box_rows) * kConvK * 2) / (kbs * bytes));
    if (s.stages < 2) continue;
    const int most = std::min({kConvIssuers, 512 / (s.bufs * s.acc_cols), steps});
    for (s.issuers = 1; s.issuers <= most; ++s.issuers) {
      // cycles per k-block, fitted to a sweep over the decoder's shapes: the tensor pipe (math, operand fetch), the issuers,
      // a producer's copies, what L2 delivers to an SM (62 bytes a cycle), a copy's latency against what the ring holds
      const int stages = s.stages - s.stages % s.issuers;
      double per = std::max({2.0 * tn, 128.0 + tn, (4 * 100 + 200.0 / kbs) / s.issuers, 550.0 / kbs, bytes / 62.0, 1100.0 / ((stages - 1) * kbs)});
      if (stages < 2 * s.issuers) per *= 1.1;  // an issuer's only stage is refilled while it waits
      const double tile = kb * per, epilogue = 7.0 * tn * (s.issuers > 1 ? 1.3 : 1.0) + 800;
      s.cycles = waves * std::max(tile, s.bufs == 2 ? epilogue : 0.0) + epilogue + 1500;
      if (s.cycles < best.cycles) best = s, best.stages = stages;
    }
  }
  return best;
}

}  // namespace

void conv_configure() {
  cudaFuncSetAttribute(conv_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kConvSmem);
}

int conv_plan(ConvGemmPlan* plan, const bf16* w, int N, int C, int taps, int dil, const bf16* x, int T, int seqs, bf16* y,
              int kind, const bf16* bias, const float* alpha, const float* inv_b, int sm_count) {
  if (N < 8 || N % 8 || C < 8 || C % 8 || taps < 1 || T < 1 || seqs < 1) return -2;
  if ((reinterpret_cast<uintptr_t>(w) & 15) || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(y) & 15))
    return -3;
  ConvGemmPlan& p = *plan;
  p.N = N, p.C = C, p.taps = taps, p.dil = dil, p.T = T, p.seqs = seqs, p.y = y;
  p.kind = kind, p.bias = bias, p.alpha = alpha, p.inv_b = inv_b;
  p.TB = 1;
  while (p.TB < kConvRows && T % (p.TB * 2) == 0) p.TB *= 2;
  p.SB = kConvRows / p.TB;
  p.row_tiles = (T / p.TB) * ((seqs + p.SB - 1) / p.SB);
  // a tile's box: no more streams than there are, but whole groups of eight rows (the swizzle's period)
  int boxes = p.SB;
  while (boxes / 2 >= seqs && p.TB * (boxes / 2) >= 8) boxes /= 2;
  p.box_rows = p.TB * boxes;
  p.cpb = (C + kConvK - 1) / kConvK;
  p.ragged = C % kConvK != 0;
  ConvShape best{};
  best.cycles = 1e30;
  for (int tn = 16; tn <= 256; tn += 16) {
    if (tn > (N + 15) / 16 * 16) break;
    const ConvShape shape = conv_shape(p, tn, sm_count);
    if (shape.cycles < best.cycles) best = shape, p.tn = tn;
  }
  if (best.cycles > 1e29) return -2;
  p.kbs = best.kbs, p.stages = best.stages, p.issuers = best.issuers, p.bufs = best.bufs, p.acc_cols = best.acc_cols;
  p.n_tiles = (N + p.tn - 1) / p.tn;
  p.ctas = std::min(p.n_tiles * p.row_tiles, sm_count);
  const int P = (taps - 1) * dil + T, Ktot = taps * C;
  if (p.ragged) {
    const uint64_t xd[3] = {(uint64_t)C, (uint64_t)P, (uint64_t)seqs};
    const uint64_t xs[2] = {(uint64_t)C * 2, (uint64_t)P * C * 2};
    const uint32_t xb[3] = {kConvK, (uint32_t)p.TB, (uint32_t)boxes};
    if (tc_encode_bf16(&p.xmap, x, 3, xd, xs, xb) != 0) return -4;
    const uint64_t wd[2] = {(uint64_t)Ktot, (uint64_t)N};
    const uint64_t ws[1] = {(uint64_t)Ktot * 2};
    const uint32_t wb[2] = {kConvK, (uint32_t)p.tn};
    if (tc_encode_bf16(&p.wmap, w, 2, wd, ws, wb) != 0) return -4;
  } else {
    const uint64_t xd[4] = {kConvK, (uint64_t)P, (uint64_t)seqs, (uint64_t)p.cpb};
    const uint64_t xs[3] = {(uint64_t)C * 2, (uint64_t)P * C * 2, kConvK * 2};
    const uint32_t xb[4] = {kConvK, (uint32_t)p.TB, (uint32_t)boxes, (uint32_t)p.kbs};
    if (tc_encode_bf16(&p.xmap, x, 4, xd, xs, xb) != 0) return -4;
    const uint64_t wd[3] = {kConvK, (uint64_t)N, (uint64_t)(Ktot / kConvK)};
    const uint64_t ws[2] = {(uint64_t)Ktot * 2, kConvK * 2};
    const uint32_t wb[3] = {kConvK, (uint32_t)p.tn, (uint32_t)p.kbs};
    if (tc_encode_bf16(&p.wmap, w, 3, wd, ws, wb) != 0) return -4;
  }
  return 0;
}

cudaError_t conv_launch(const ConvGemmPlan& p, uint32_t* err, cudaStream_t stream) {
  ConvArgs a{};
  a.y = p.y, a.bias = p.bias, a.alpha = p.alpha, a.inv_b = p.inv_b, a.err = err;
  a.N = p.N, a.C = p.C, a.taps = p.taps, a.dil = p.dil, a.T = p.T, a.seqs = p.seqs, a.TB = p.TB, a.SB = p.SB;
  while ((1 << a.tb_log2) < p.TB) ++a.tb_log2;
  a.tn = p.tn, a.kbs = p.kbs, a.cpb = p.cpb, a.ragged = p.ragged, a.stages = p.stages, a.kind = p.kind;
  a.t_tiles = p.T / p.TB, a.n_tiles = p.n_tiles, a.tiles = p.n_tiles * p.row_tiles;
  a.box_rows = p.box_rows, a.issuers = p.issuers, a.bufs = p.bufs, a.acc_cols = (uint32_t)p.acc_cols;
  a.tmem_cols = 32;
  while (a.tmem_cols < a.acc_cols * (uint32_t)(p.issuers * p.bufs)) a.tmem_cols *= 2;
  return launch_pdl(conv_gemm_kernel, dim3(p.ctas), dim3(kConvThreads), kConvSmem, stream, p.xmap, p.wmap, a);
}

}  // namespace omni
