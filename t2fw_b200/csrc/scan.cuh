// Pieces of the shape- and dtype-general scan kernels (lfw_scan.cuh, dfw_scan.cu): staging of a few steps'
// vectors in shared memory, and sums over a warp for several values at once.
//
// A scan step is a few dozen instructions on a state held in registers; read straight from global memory its
// vectors cost a memory latency per step (0.7 us per step measured, 95 us for 129 steps).  So a CTA, whose
// warps all work on one batch row, fetches the vectors of a group of steps asynchronously while the group
// before is being computed.
#pragma once

#include "common.cuh"

namespace t2fw {
namespace scan {

// Asynchronous copy of n elements (contiguous in global and in shared memory) by the whole CTA.  Copies need
// 4-byte alignment; a 16-bit array at an odd element offset is copied through registers instead (and is then
// in place after the next barrier like everything else).  dst is 16-byte aligned.
template <typename T>
__device__ __forceinline__ void stage(T *dst, const T *src, int n, int tid, int nthreads) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int bytes = n * (int)sizeof(T);
  const uintptr_t a = reinterpret_cast<uintptr_t>(src);
  if ((a & 15u) == 0) {
    const int n16 = bytes >> 4;
    for (int i = tid; i < n16; i += nthreads)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16 * i), "l"(reinterpret_cast<const char *>(src) + 16 * i) : "memory");
    for (int i = (n16 << 4) / (int)sizeof(T) + tid; i < n; i += nthreads) dst[i] = src[i];
  } else if (sizeof(T) >= 4 || (a & 3u) == 0) {
    const int n4 = bytes >> 2;
    for (int i = tid; i < n4; i += nthreads)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d + 4 * i), "l"(reinterpret_cast<const char *>(src) + 4 * i) : "memory");
    for (int i = (n4 << 2) / (int)sizeof(T) + tid; i < n; i += nthreads) dst[i] = src[i];
  } else {
#pragma unroll 8
    for (int i = tid; i < n; i += nthreads) dst[i] = src[i];
  }
}
// n rows of w elements that lie ld elements apart in global memory
template <typename T>
__device__ __forceinline__ void stage_rows(T *dst, const T *src, int n, int w, int ld, int tid, int nthreads) {
  for (int i = tid; i < n * w; i += nthreads) {
    const int r = i / w, c = i - r * w;
    if constexpr (sizeof(T) >= 4)
      asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + i)),
                   "l"(src + (size_t)r * ld + c), "n"(sizeof(T) >= 4 ? sizeof(T) : 4) : "memory");
    else
      dst[i] = src[(size_t)r * ld + c];
  }
}
// The same with loops that are not unrolled, for the decay rule's backward, whose fetch is part of a long loop body
// (48 x 300, 100 x 100, fp16: 1012 us unrolled by four, 896 rolled; fp32, 16 x 129, 96 x 48: 72 and 69.5).
template <typename T>
__device__ __forceinline__ void stage_rolled(T *dst, const T *src, int n, int tid, int nthreads) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const int bytes = n * (int)sizeof(T);
  const uintptr_t a = reinterpret_cast<uintptr_t>(src);
  if ((a & 15u) == 0) {
    const int n16 = bytes >> 4;
#pragma unroll 1
    for (int i = tid; i < n16; i += nthreads)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16 * i), "l"(reinterpret_cast<const char *>(src) + 16 * i) : "memory");
#pragma unroll 1
    for (int i = (n16 << 4) / (int)sizeof(T) + tid; i < n; i += nthreads) dst[i] = src[i];
  } else if (sizeof(T) >= 4 || (a & 3u) == 0) {
    const int n4 = bytes >> 2;
#pragma unroll 1
    for (int i = tid; i < n4; i += nthreads)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d + 4 * i), "l"(reinterpret_cast<const char *>(src) + 4 * i) : "memory");
#pragma unroll 1
    for (int i = (n4 << 2) / (int)sizeof(T) + tid; i < n; i += nthreads) dst[i] = src[i];
  } else {
#pragma unroll 4
    for (int i = tid; i < n; i += nthreads) dst[i] = src[i];
  }
}
template <typename T>
__device__ __forceinline__ void stage_rows_rolled(T *dst, const T *src, int n, int w, int ld, int tid, int nthreads) {
#pragma unroll 1
  for (int i = tid; i < n * w; i += nthreads) {
    const int r = i / w, c = i - r * w;
    if constexpr (sizeof(T) >= 4)
      asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + i)),
                   "l"(src + (size_t)r * ld + c), "n"(sizeof(T) >= 4 ? sizeof(T) : 4) : "memory");
    else
      dst[i] = src[(size_t)r * ld + c];
  }
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Sums of R values (R a power of two) over the L lanes of an aligned group, lane = number within it: at each distance
// a lane keeps half of its values and hands over the partner's half, so R <= L sums cost about R + log2(L / R)
// shuffles instead of R log2(L).  On return v[0] is the total of value *which; the lanes for which the function
// returns true cover each value once.
template <int R, int L = 32, typename A>
__device__ __forceinline__ bool lane_sums(A *v, int lane, int *which) {
  static_assert(R <= L, "one value per lane at most");
  int idx = 0, live = R;
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) {
    if (live > 1) {
      const bool up = (lane & o) != 0;
      live >>= 1;
#pragma unroll
      for (int i = 0; i < live; ++i) {
        const A send = up ? v[i] : v[i + live], keep = up ? v[i + live] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
      idx += up ? live : 0;
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
  *which = idx;
  return (lane & (L / R - 1)) == 0;
}

}  // namespace scan
}  // namespace t2fw
