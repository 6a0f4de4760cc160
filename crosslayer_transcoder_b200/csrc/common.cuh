// Shared declarations of the CUDA side: error reporting, device status words,
// small device helpers.  sm_100a only.
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <stdio.h>

namespace clt {

// ---- host-side error string (one per thread) ---------------------------------
void set_error(const char* fmt, ...);
const char* last_error();

#define CLT_CHECK_ARG(cond, ...)                 \
  do {                                           \
    if (!(cond)) {                               \
      ::clt::set_error(__VA_ARGS__);             \
      return 1;                                  \
    }                                            \
  } while (0)

#define CLT_CHECK_CUDA(expr)                                                        \
  do {                                                                              \
    cudaError_t _e = (expr);                                                        \
    if (_e != cudaSuccess) {                                                        \
      ::clt::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e),      \
                       __FILE__, __LINE__);                                         \
      return 2;                                                                     \
    }                                                                               \
  } while (0)

// ---- device status word --------------------------------------------------------
// Kernels never trap.  A kernel that gives up on a wait or meets an index out of
// range writes one of these codes (first writer wins) and returns; the host
// reads the word at its next synchronisation point.
enum DeviceStatus : int {
  kOk = 0,
  kTimeoutFull = 0x10,       // MMA warp gave up waiting for a TMA stage
  kTimeoutEmpty = 0x11,      // TMA warp gave up waiting for a free stage
  kTimeoutTmemFull = 0x12,   // epilogue gave up waiting for the accumulator
  kTimeoutTmemEmpty = 0x13,  // MMA warp gave up waiting for the epilogue
  kBadIndex = 0x20,          // an index read from memory was out of range
  kOverflow = 0x21,          // a fixed-capacity list overflowed
};

__device__ __forceinline__ void report_status(int* status, int code) {
  if (status != nullptr) atomicCAS(status, 0, code);
}

// ---- small device helpers -----------------------------------------------------
__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

template <class T>
struct ToFloat;
template <>
struct ToFloat<float> {
  __device__ static __forceinline__ float get(float v) { return v; }
};
template <>
struct ToFloat<__nv_bfloat16> {
  __device__ static __forceinline__ float get(__nv_bfloat16 v) { return __bfloat162float(v); }
};

// 8 consecutive fp32 values of a lane as one 32-byte store (p a multiple of 32 bytes).  Two 16-byte stores at a lane
// distance of 32 bytes touch every sector of the warp's kilobyte twice, half of it each time: encoder gradients
// of the sparse steps 489 -> 383, 1000 -> 865 and 310 -> 248 us.  (The decoder pass with the optimizer, whose three
// streams are read as well, is 3 % slower with 32-byte accesses and keeps 16.)
__device__ __forceinline__ void st_f32x8(float* p, const float4& a, const float4& b) {
  asm volatile("st.global.cs.v8.f32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};" ::"f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w),
               "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w), "l"(p)
               : "memory");
}
__host__ __device__ __forceinline__ bool aligned32(const void* p) { return ((uintptr_t)p & 31) == 0; }
// streaming store of 8 values to a 16-byte aligned address, in one access where it is a multiple of 32
__device__ __forceinline__ void st_cs8(float* p, const float4& a, const float4& b) {
  if (aligned32(p)) {
    st_f32x8(p, a, b);
  } else {
    __stcs(reinterpret_cast<float4*>(p), a);
    __stcs(reinterpret_cast<float4*>(p) + 1, b);
  }
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum of `v` (uniform over a warp) of the warps before this one, and of all; 1024 threads.
__device__ __forceinline__ int block1024_offset(int v, int& all) {
  __shared__ int warp_values[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) warp_values[w] = v;
  __syncthreads();
  int x = warp_values[lane];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  all = __shfl_sync(0xffffffffu, x, 31);
  const int before = __shfl_sync(0xffffffffu, x, w) - v;
  __syncthreads();  // the array may be written again
  return before;
}

// Column sums over the 32 rows held by one warp.  Each lane holds 32 values
// (one row, 32 consecutive columns); on return lane j holds the sum over all
// lanes of column j.  Recursive halving: 31 shuffles for 32 columns.
__device__ __forceinline__ float warp_colsum32(float (&v)[32]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) {
    const bool upper = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < off; ++i) {
      float send = upper ? v[i] : v[i + off];
      float keep = upper ? v[i + off] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  return v[0];
}

}  // namespace clt
