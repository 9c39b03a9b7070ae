// The prompt-sized GEMM (see wide_gemm.h).
//
// Bound by the tensor pipe. A pair of CTAs (one cluster, the two SMs of a TPC) works on one tile of 256 rows of x by tn
// rows of w with cta_group::2 MMAs: each CTA holds half of either operand, so a k-block of 64 costs an SM 32 KB of shared
// memory fill per 512 tensor cycles where a 128 x 256 tile of its own would cost 48 KB, more than L2 delivers to all SMs at
// once. Persistent: the accumulator is double-buffered in TMEM (2 x 256 columns), so four warps store a tile while the
// next one is multiplied, and the ring of operands never drains between tiles. Tiles are walked in bands of eight row
// tiles, so that the tiles under way share their operands in L2. Measured at 8,700 rows: 12,288 x 2,048 286 us
// (1,529 TFLOP/s; the split-K tiles of gemm.cu 696 us), 2,048 x 6,144 154 us (1,419; 215 us), 2,048 x 2,048 53 us
// (1,379; 114 us); at 257 rows 4,096 x 2,048 12.6 us (33.7 us).
#include "wide_gemm.h"

#include <algorithm>

#include "pdl.cuh"
#include "sm100.cuh"

namespace omni {
namespace {

constexpr int kWideKb = 64, kWideRows = 256, kWideThreads = 192, kBand = 8, kWideMaxSlots = 6;
constexpr int kPer = 2;        // k-blocks per ring slot and copy
constexpr int kAccCols = 256;  // TMEM columns of one accumulator
constexpr int kWideSmem = 225 * 1024;

struct WideArgs {
  bf16* y;
  const bf16* bias;
  uint32_t* err;
  int N, rows, nkb, tn, slots, ldy, kind, granule, m_tiles, n_tiles, vec;
};

__device__ __forceinline__ uint32_t cta_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// `addr` of this CTA as CTA `rank` of the cluster has it.
__device__ __forceinline__ uint32_t map_shared(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void store_remote(uint32_t cluster_addr, uint32_t v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}
// `bytes` that will not arrive count as arrived on a barrier of this CTA.
__device__ __forceinline__ void forgo_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// A box of this CTA's own copy of an operand; the bytes are counted on `bar`, a barrier of either CTA of the pair.
__device__ __forceinline__ void pair_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z, uint64_t hint) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2.L2::cache_hint"
      " [%0], [%1, {%3, %4, %5}], [%2], %6;"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(z), "l"(hint)
      : "memory");
}
__device__ __forceinline__ void pair_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrives on `bar` of both CTAs when every MMA issued so far by this thread has finished.
__device__ __forceinline__ void pair_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"((uint16_t)3)
               : "memory");
}
template <int OUT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kWideThreads, 1)
    wide_gemm_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap, const WideArgs a) {
  using namespace sm100;
  extern __shared__ unsigned char wide_smem_raw[];
  __shared__ __align__(8) uint64_t bars_s[2 * kWideMaxSlots + 4];
  __shared__ uint32_t tmem_slot_s;
  __shared__ int gave_up_s, issued_s[2];  // a wait of the pair ran out; stages its producers had filled by then (-1: all; the leader's)
  const uint32_t base = (smem_addr(wide_smem_raw) + 1023u) & ~1023u, bars = smem_addr(bars_s);
  auto full = [&](int s) { return bars + 8u * s; };  // the leader's counts the bytes of both CTAs
  auto empty = [&](int s) { return bars + 8u * (kWideMaxSlots + s); };
  auto acc_full = [&](int s) { return bars + 8u * (2 * kWideMaxSlots + s); };
  auto acc_empty = [&](int s) { return bars + 8u * (2 * kWideMaxSlots + 2 + s); };  // the leader's: both CTAs' epilogue warps
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cta_rank();
  const int tiles = a.m_tiles * a.n_tiles, first = blockIdx.x >> 1, stride = gridDim.x >> 1;
  const uint32_t x_bytes = kPer * 128 * 128, w_slice = (uint32_t)(a.tn >> 1) * 128u, slot_bytes = x_bytes + kPer * w_slice;
  // tile -> (row tile, column tile): bands of kBand row tiles, column by column
  auto place = [&](int tile, int& m, int& n) {
    const int band = tile / (kBand * a.n_tiles), in = tile % (kBand * a.n_tiles), height = min(kBand, a.m_tiles - band * kBand);
    m = band * kBand + in % height, n = in / height;
  };
  auto give_up = [&]() {  // known to both CTAs
    store_remote(map_shared(smem_addr(&gave_up_s), 0), 1u);
    store_remote(map_shared(smem_addr(&gave_up_s), 1), 1u);
  };
  if (threadIdx.x == 0) {
    gave_up_s = 0, issued_s[0] = issued_s[1] = -1;
    prefetch_tensormap(&xmap);
    prefetch_tensormap(&wmap);
    for (int s = 0; s < a.slots; ++s) mbar_init(full(s), 1), mbar_init(empty(s), 1);
    for (int s = 0; s < 2; ++s) mbar_init(acc_full(s), 1), mbar_init(acc_empty(s), 8);
    mbar_init_fence();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_slot_s)), "r"(2 * kAccCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync();  // the peer's barriers exist before anything arrives on them
  tc_fence_after_sync();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tmem_slot_s);
  grid_trigger();  // not before this CTA holds its TMEM columns: the next kernel could take them and wait for this one
  grid_wait();

  if (warp == 0) {
    if (lane == 0) {
      fence_async_global();  // rows written by ordinary stores, read by TMA
      int slot = 0, done = 0;
      uint32_t phase = 1;
      bool alive = true;
      for (int tile = first; tile < tiles && alive; tile += stride) {
        int m, n;
        place(tile, m, n);
        const int x_row = m * kWideRows + (int)rank * 128, w_row = n * a.tn + (int)rank * (a.tn >> 1);
        for (int kb = 0; kb < a.nkb; kb += kPer) {  // past the last k-block the copies bring zeros
          alive = mbar_wait(empty(slot), phase, a.err);
          if (!alive) break;
          if (rank == 0) mbar_expect_tx(full(slot), 2 * slot_bytes);
          const uint32_t dst = base + (uint32_t)slot * slot_bytes, bar = map_shared(full(slot), 0);
          pair_load_3d(dst, &xmap, bar, 0, x_row, kb, kEvictNormal);
          pair_load_3d(dst + x_bytes, &wmap, bar, 0, w_row, kb, kEvictNormal);
          ++done;
          if (++slot == a.slots) slot = 0, phase ^= 1u;
        }
      }
      if (!alive) {
        store_remote(map_shared(smem_addr(&issued_s[rank]), 0), (uint32_t)done);
        give_up();
      }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      // one thread issues an MMA every 80 cycles and spends about 200 on a slot's wait and commit: two k-blocks a slot
      // keep that below the 1,024 cycles which their MMAs take at 256 columns
      const uint32_t idesc = idesc_bf16_f32(kWideRows, a.tn);
      int slot = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 1;
      bool alive = true;
      for (int tile = first; tile < tiles && alive; tile += stride) {
        alive = mbar_wait(acc_empty(acc), acc_phase, a.err);
        tc_fence_after_sync();
        const uint32_t d = tmem + (uint32_t)(acc * kAccCols);
        for (int kb = 0; kb < a.nkb && alive; kb += kPer) {
          alive = mbar_wait(full(slot), phase, a.err);
          if (!alive) break;
          tc_fence_after_sync();
          if (elect_one()) {
            const uint64_t ad = kmajor_sw128_desc(base + (uint32_t)slot * slot_bytes);
            const uint64_t bd = kmajor_sw128_desc(base + (uint32_t)slot * slot_bytes + x_bytes);
            const int some = min(kPer, a.nkb - kb);
#pragma unroll
            for (int j = 0; j < kPer; ++j)
              if (j < some) {
#pragma unroll
                for (int k = 0; k < kWideKb / 16; ++k)
                  pair_mma(d, ad + (uint64_t)(j * (128 * 128 >> 4) + k * 2), bd + (uint64_t)(j * (int)(w_slice >> 4) + k * 2), idesc, (kb > 0 || j > 0 || k > 0) ? 1u : 0u);
              }
            pair_commit(empty(slot));
          }
          __syncwarp();
          if (++slot == a.slots) slot = 0, phase ^= 1u;
        }
        if (alive && elect_one()) pair_commit(acc_full(acc));
        __syncwarp();
        if (++acc == 2) acc = 0, acc_phase ^= 1u;
      }
      if (!alive && lane == 0) give_up();
    }
  } else {
    const int quad = warp & 3;
    int acc = 0;
    uint32_t phase = 0;
    for (int tile = first; tile < tiles; tile += stride) {
      int m, n;
      place(tile, m, n);
      if (!mbar_wait(acc_full(acc), phase, a.err)) break;
      tc_fence_after_sync();
      const uint32_t lane_addr = tmem + (uint32_t)(acc * kAccCols) + ((uint32_t)(quad * 32) << 16);
      const int row = m * kWideRows + (int)rank * 128 + quad * 32 + lane;
      const bool live = row < a.rows, warp_live = m * kWideRows + (int)rank * 128 + quad * 32 < a.rows;
      if (warp_live) {
        if constexpr (OUT == kStreamSwiglu) {
          // the tile's columns are groups of `granule` gates and their ups (the matrix's last group may hold fewer)
          const int groups = a.tn / (2 * a.granule), inter = a.N >> 1;
          for (int gr = 0; gr < groups; ++gr) {
            const int ch0 = (n * groups + gr) * a.granule, half = min(a.granule, inter - ch0), at = gr * 2 * a.granule;
            for (int c = 0; c < half; c += 8) {
              uint32_t r[2][8];
              tmem_ld8_issue(lane_addr + at + c, r[0]);
              tmem_ld8_issue(lane_addr + at + half + c, r[1]);
              tmem_ld8_fence<2>(r);
              float o[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                o[j] = silu_bf16(bf16_round(__uint_as_float(r[0][j]))) * bf16_round(__uint_as_float(r[1][j]));
              }
              if (live) st8(a.y + (size_t)row * a.ldy + ch0 + c, o);
            }
          }
        } else {
          const int n0 = n * a.tn, cols = min(a.tn, a.N - n0);
          for (int c = 0; c < cols; c += 32) {  // tn is a multiple of 32
            uint32_t r[4][8];
#pragma unroll
            for (int i = 0; i < 4; ++i) tmem_ld8_issue(lane_addr + c + i * 8, r[i]);
            tmem_ld8_fence<4>(r);
            if (!live) continue;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int col = n0 + c + i * 8;
              float v[8];
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                v[j] = bf16_round(__uint_as_float(r[i][j]));
                if (a.kind != kEpiNone && col + j < a.N) {
                  v[j] = bf16_round(v[j] + __bfloat162float(a.bias[col + j]));
                  if (a.kind == kEpiBiasSilu) v[j] = v[j] / (1.f + __expf(-v[j]));
                }
              }
              bf16* dst = a.y + (size_t)row * a.ldy + col;
              if (a.vec) {
                if (col < a.N) st8(dst, v);
              } else {
                for (int j = 0; j < 8 && col + j < a.N; ++j) dst[j] = __float2bfloat16(v[j]);
              }
            }
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) arrive_remote(map_shared(acc_empty(acc), 0));
      if (++acc == 2) acc = 0, phase ^= 1u;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync();  // no CTA leaves while the other may still arrive on its barriers or read its operands
  if (*reinterpret_cast<volatile int*>(&gave_up_s)) {
    // ... nor while copies are under way, which count on the leader's barriers: a stage that only one CTA filled is
    // completed from here for the other, so that its barrier, too, tells when the copy is there
    if (rank == 0 && threadIdx.x == 0) {
      const int per = (a.nkb + kPer - 1) / kPer, all = (tiles - first + stride - 1) / stride * per;
      const int mine = issued_s[0] < 0 ? all : issued_s[0], peer = issued_s[1] < 0 ? all : issued_s[1];
      for (int i = peer; i < mine; ++i) forgo_tx(full(i % a.slots), slot_bytes);
      for (int i = mine; i < peer; ++i) mbar_expect_tx(full(i % a.slots), slot_bytes);
      drain_ring(full(0), a.slots, max(mine, peer), a.err);
    }
    __syncthreads();
    cluster_sync();
  }
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kAccCols) : "memory");
}

}  // namespace

void wide_configure() {
  cudaFuncSetAttribute(wide_gemm_kernel<kStreamBf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWideSmem);
  cudaFuncSetAttribute(wide_gemm_kernel<kStreamSwiglu>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWideSmem);
}

// A tile holds whole groups and is a multiple of 32 columns.
static bool tile_fits(int tn, int granule) { return tn % 32 == 0 && tn <= 256 && (granule == 0 || tn % (2 * granule) == 0); }

bool wide_fuses(int N, int K, int granule) {
  if (granule < 8 || granule % 8 || N % 16 || K % kWideKb) return false;
  for (int tn = 32; tn <= 256; tn += 32)
    if (tile_fits(tn, granule)) return true;
  return false;
}

int wide_plan(WidePlan* plan, const bf16* w, int N, int K, const bf16* x, int rows, int out, bf16* y, int ldy, Epilogue epi,
              int sm_count, int granule) {
  if (rows < 1 || N < 1 || K < kWideKb || K % kWideKb || out == kStreamPartials) return -2;
  if ((reinterpret_cast<uintptr_t>(w) & 15) || (reinterpret_cast<uintptr_t>(x) & 15)) return -3;
  if (out == kStreamSwiglu && (reinterpret_cast<uintptr_t>(y) & 15)) return -3;
  WidePlan& p = *plan;
  p.N = N, p.K = K, p.rows = rows, p.out = out, p.y = y, p.ldy = ldy, p.epi = epi, p.granule = granule;
  const int pairs = std::max(1, sm_count / 2), m_tiles = (rows + kWideRows - 1) / kWideRows;
  if (out != kStreamSwiglu) granule = 0;
  else if (!wide_fuses(N, K, granule) || ldy % 8) return -2;
  // measured: a k-block of a tile takes 0.05 us + 1.34 ns a column (32 columns 0.135 us, 256 columns 0.39 us), a tile's
  // stores 12 ns a column, of which only the last tile's are not hidden
  double best = 1e30;
  for (int tn = 32; tn <= 256; tn += 32) {
    if (!tile_fits(tn, granule)) continue;
    const int waves = (m_tiles * ((N + tn - 1) / tn) + pairs - 1) / pairs;
    const double cost = waves * (K / kWideKb) * (0.05 + 0.00134 * tn) + 0.012 * tn;
    if (cost < best) best = cost, p.tn = tn;
  }
  p.ctas = 2 * std::min(pairs, m_tiles * ((N + p.tn - 1) / p.tn));
  const uint64_t nkb = K / kWideKb, st[2] = {(uint64_t)K * 2, kWideKb * 2};
  const uint64_t xd[3] = {kWideKb, (uint64_t)rows, nkb}, wd[3] = {kWideKb, (uint64_t)N, nkb};
  const uint32_t xb[3] = {kWideKb, 128, kPer}, wb[3] = {kWideKb, (uint32_t)p.tn / 2, kPer};
  if (tc_encode_bf16(&p.xmap, x, 3, xd, st, xb) != 0 || tc_encode_bf16(&p.wmap, w, 3, wd, st, wb) != 0) return -4;
  return 0;
}

cudaError_t wide_launch(const WidePlan& p, uint32_t* err, cudaStream_t stream) {
  WideArgs a;
  a.y = p.y, a.bias = p.epi.bias, a.err = err, a.kind = p.epi.kind;
  a.N = p.N, a.rows = p.rows, a.nkb = p.K / kWideKb, a.tn = p.tn, a.ldy = p.ldy, a.granule = p.granule;
  a.m_tiles = (p.rows + kWideRows - 1) / kWideRows, a.n_tiles = (p.N + p.tn - 1) / p.tn;
  a.vec = p.ldy % 8 == 0 && p.N % 8 == 0 && (reinterpret_cast<uintptr_t>(p.y) & 15) == 0;
  a.slots = std::min(kWideMaxSlots, (kWideSmem - 1024) / (kPer * (128 + p.tn / 2) * 128));
  if (p.out == kStreamSwiglu) return launch_pdl(wide_gemm_kernel<kStreamSwiglu>, dim3(p.ctas), dim3(kWideThreads), kWideSmem, stream, p.xmap, p.wmap, a);
  return launch_pdl(wide_gemm_kernel<kStreamBf16>, dim3(p.ctas), dim3(kWideThreads), kWideSmem, stream, p.xmap, p.wmap, a);
}

}  // namespace omni
