// Arithmetic of one recurrent step on eight state columns of one row, shared by the kernels that walk a
// sequence step by step (steps.cu, lfw_decode_bulk.cu) so that they agree bit for bit: packed pairs of
// fp32 (one instruction per two elements), the row sum as even + odd partial sums and then a butterfly
// over the lanes of the row, widest distance first.
#pragma once

#include "common.cuh"

namespace t2fw {
namespace steps {

using f2 = unsigned long long;      // two fp32 values in one 64-bit register

__device__ __forceinline__ f2 pack2(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(f2 v, float &lo, float &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// eight consecutive 16-bit values <-> four fp32 pairs
template <typename T> struct Oct;
template <> struct Oct<__half> {
  static __device__ __forceinline__ void unpack(const uint4 &u, f2 (&v)[4]) {
    const __half2 *h = reinterpret_cast<const __half2 *>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 p = __half22float2(h[i]);
      v[i] = pack2(p.x, p.y);
    }
  }
  static __device__ __forceinline__ uint4 pack(const f2 (&v)[4]) {
    uint4 u;
    __half2 *h = reinterpret_cast<__half2 *>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float a, b;
      unpack2(v[i], a, b);
      h[i] = __floats2half2_rn(a, b);
    }
    return u;
  }
};
template <> struct Oct<__nv_bfloat16> {
  static __device__ __forceinline__ void unpack(const uint4 &u, f2 (&v)[4]) {
    const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 p = __bfloat1622float2(h[i]);
      v[i] = pack2(p.x, p.y);
    }
  }
  static __device__ __forceinline__ uint4 pack(const f2 (&v)[4]) {
    uint4 u;
    __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float a, b;
      unpack2(v[i], a, b);
      h[i] = __floats2bfloat162_rn(a, b);
    }
    return u;
  }
};

// S' = (a g) S + x k on eight columns (x2, a2: the row's value and gate in both halves); returns this thread's share of S' q
__device__ __forceinline__ float decay_step8(f2 (&s)[4], const f2 (&g)[4], const f2 (&k)[4], const f2 (&q)[4], f2 x2,
                                             f2 a2) {
  f2 acc = 0ull;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    s[e] = fma2(s[e], mul2(a2, g[e]), mul2(x2, k[e]));
    acc = fma2(s[e], q[e], acc);
  }
  float lo, hi;
  unpack2(acc, lo, hi);
  return lo + hi;
}

// Row sums of R rows over KT lanes.  At each distance a lane keeps half of its rows and hands the partner's
// half over, so R rows cost about R shuffles instead of R log2(KT); the additions are the butterfly's.
// On return v[0] is the total of row *row (an index below R) in every lane for which the function says so.
template <int KT, int R>
__device__ __forceinline__ bool row_sums(float (&v)[R], int kc, int *row) {
  static_assert(R <= KT, "at most one row per lane");
  int idx = 0;
  constexpr int kLevels = KT == 2 ? 1 : KT == 4 ? 2 : KT == 8 ? 3 : KT == 16 ? 4 : 5;
#pragma unroll
  for (int l = 0; l < kLevels; ++l) {
    const int o = KT >> (l + 1), live = (R >> l) > 1 ? (R >> l) : 1;
    if (live > 1) {
      const bool up = (kc & o) != 0;
#pragma unroll
      for (int i = 0; i < (live >> 1); ++i) {
        const float send = up ? v[i] : v[i + (live >> 1)], keep = up ? v[i + (live >> 1)] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
      idx += up ? (live >> 1) : 0;
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
  *row = idx;
  return (kc & (KT / R - 1)) == 0;
}

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

}  // namespace steps
}  // namespace t2fw
