// Device helpers shared by every kernel of the library: bf16 packing, warp and
// block reductions, the device error word.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

namespace omni {

// threadIdx.x / 32 as a value that is the same in every lane, which the compiler cannot see by itself: what follows from it -
// roles, ring slots, descriptors, addresses - stays in uniform registers. Every thread of the warp calls it. One pass, us: a
// talker step of one session 2,076 -> 1,958 (few_rows.cu and rope_attend_kernel), of 64 3,815 -> 3,719 (stream_gemm.cu), a codec
// frame of 64 streams 1,177 -> 1,150 (codec_gemm.cu). Not in wide_gemm.cu and prompt_attend.cuh, which were 1 and 2 % slower.
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0); }


typedef __nv_bfloat16 bf16;

// Device error word: kernels OR a code into it instead of trapping, the host
// reads it after the call. Kernels that wait on hardware barriers return early
// once it is non-zero so one failure cannot stall a whole graph.
enum DeviceError : uint32_t {
  kErrNone = 0,
  kErrBarrierTimeout = 1u << 0,  // a bounded mbarrier wait ran out
  kErrBadIndex = 1u << 1,        // an id / page / slot outside its table
  kErrBadShape = 1u << 2,
};

__device__ __forceinline__ void raise(uint32_t* err, uint32_t code) { atomicOr(err, code); }

__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16(x)); }

// bf16(g / (1 + exp(-g))) of a bf16 gate. The exponential is taken of -|g|, so the divisor lies in (1, 2], where the fast
// division is good. Of the 65,280 finite gates one (-2^-8, next to a tie) does not give the bf16 nearest to float64's; the
// full division by 1 + exp(-g) misses 17, which it returns as 0, and takes a duplex tick of 64 sessions 180 us longer.
__device__ __forceinline__ float silu_bf16(float g) {
  const float e = __expf(-fabsf(g));
  return bf16_round(__fdividef(g < 0.f ? g * e : g, 1.f + e));
}

struct alignas(16) Pack8 {
  __nv_bfloat162 h[4];
};

// Eight bf16 (one 16-byte access) widened to f32.
__device__ __forceinline__ void unpack8(const Pack8& p, float* v) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(p.h[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}

__device__ __forceinline__ Pack8 pack8(const float* v) {
  Pack8 p;
#pragma unroll
  for (int i = 0; i < 4; ++i) p.h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
  return p;
}


// The same eight values moved as one 16-byte word: an access through uint4 is a single vector instruction wherever the
// struct copy above might be split into four.
__device__ __forceinline__ void unpack8v(const uint4& u, float* v) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(h[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}

__device__ __forceinline__ uint4 pack8v(const float* v) {
  uint4 u;
  __nv_bfloat162 t;
  t = __floats2bfloat162_rn(v[0], v[1]);
  u.x = *reinterpret_cast<const uint32_t*>(&t);
  t = __floats2bfloat162_rn(v[2], v[3]);
  u.y = *reinterpret_cast<const uint32_t*>(&t);
  t = __floats2bfloat162_rn(v[4], v[5]);
  u.z = *reinterpret_cast<const uint32_t*>(&t);
  t = __floats2bfloat162_rn(v[6], v[7]);
  u.w = *reinterpret_cast<const uint32_t*>(&t);
  return u;
}

__device__ __forceinline__ void ld8v(const bf16* src, float* v) { unpack8v(*reinterpret_cast<const uint4*>(src), v); }
__device__ __forceinline__ void st8v(bf16* dst, const float* v) { *reinterpret_cast<uint4*>(dst) = pack8v(v); }
// Eight bf16 at a 16-byte aligned address.
__device__ __forceinline__ void ld8(const bf16* src, float* v) { ld8v(src, v); }
__device__ __forceinline__ void st8(bf16* dst, const float* v) { st8v(dst, v); }

// The same past L1, for rows that another SM wrote while this kernel had already started.
__device__ __forceinline__ void ld8cg(const bf16* src, float* v) { unpack8v(__ldcg(reinterpret_cast<const uint4*>(src)), v); }

// E = 2, 4 or 8 bf16 as one access, widened to f32.
template <int E>
struct Run {
  using Word = std::conditional_t<E == 8, uint4, std::conditional_t<E == 4, uint2, uint32_t>>;
  static __device__ __forceinline__ void widen(const Word& u, float* v) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < E / 2; ++i) {
      const float2 f = __bfloat1622float2(h[i]);
      v[2 * i] = f.x, v[2 * i + 1] = f.y;
    }
  }
  static __device__ __forceinline__ void ld(const bf16* src, float* v) { widen(__ldg(reinterpret_cast<const Word*>(src)), v); }
  static __device__ __forceinline__ void ldcg(const bf16* src, float* v) { widen(__ldcg(reinterpret_cast<const Word*>(src)), v); }
  static __device__ __forceinline__ void st(bf16* dst, const float* v) {
    Word u;
#pragma unroll
    for (int i = 0; i < E / 2; ++i) reinterpret_cast<__nv_bfloat162*>(&u)[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    *reinterpret_cast<Word*>(dst) = u;
  }
};

// Two f32 values as the sum of three bf16 each (value, rest of it, rest of that), packed: 24 bits of a value, its whole
// mantissa. A matrix instruction on bf16 then multiplies it as f32 would.
__device__ __forceinline__ void split3(float a, float b, uint32_t (&part)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
    part[i] = *reinterpret_cast<const uint32_t*>(&t);
    const float2 f = __bfloat1622float2(t);
    a -= f.x, b -= f.y;
  }
}

__device__ __forceinline__ float warp_add(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float warp_fmax(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sum over the block, a whole number of warps; `scratch` is 32 floats of shared memory. Ends with a
// barrier so `scratch` can be reused at once.
__device__ __forceinline__ float block_add(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  v = warp_add(v);
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  v = lane < nwarps ? scratch[lane] : 0.f;
  v = warp_add(v);
  __syncthreads();
  return v;
}

// Threads of a block that works on a row of `dim` elements, eight a thread: whole warps, since in a part of one block_add
// would add up as many warps as it has lanes.
inline int row_threads(int dim) { return (dim + 255) / 256 * 32; }

}  // namespace omni
