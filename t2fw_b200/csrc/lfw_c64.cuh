// Building blocks of the 64-step chunk kernels of the decay rule (D = K = 64, 16-bit storage):
// lfw_c64_fwd.cu (outputs of a chunk) and lfw_c64_bwd.cu (the five sequence gradients).
//
// Algebra.  A chunk is 64 steps t = 0..63 with gates a_t (d side, `forget`) and g_t (k side,
// `f_key`).  With cumulative products A_t = a_0..a_t, G_t = g_0..g_t and the anchor REF = 31 in
// the middle of the chunk, the in-chunk decay between two steps factors into ratios to the anchor
//     pm_g[t] = G_t / G_REF        (t > REF: product of g_{REF+1..t};  t <= REF: 1 / product of g_{t+1..REF})
// so that no product over more than 32 steps is ever formed or inverted, and only one-sided.
// "mid" operands carry these ratios (q * pm_g, k / pm_g, dO * pm_a, x / pm_a); their pair products
// P = tril((q pm_g)(k / pm_g)^T), Z = tril((dO pm_a)(x / pm_a)^T) are the exact in-chunk decays.
// The same operands serve the terms through the state at the chunk start and through the state
// gradient at the chunk end: the 64 x 64 state block carries the anchor product of the side that is
// contracted away, and the result is scaled by that of its own side.  (The chunk-local kernel alone
// anchors its operands at the chunk's end or start, lfw_c64_local.cu.)
// A batch row whose one-sided 32-step products leave [2^-100, 2^100], or that holds a NaN or an infinity, is flagged and
// recomputed by the sequential scan kernels.  A call looks at every input on the way to its flags: the chunk-local kernel at the
// gates and the two value tensors that it contracts, the carry at the states that it walks, the output kernel at the query, the
// gradient kernel at x, k and the start states.
// The fused layer has no gate products out of range and no scan behind it: its kernels round so that a NaN stays one.
//
// Operand tiles are 64 x 64 fp32 (TF32-rounded) in the K-major 128-byte-swizzle layout of the
// tcgen05 shared-memory descriptor: two column blocks of 32 floats; inside a block row r is 128
// bytes at r * 128 and its eight 16-byte chunks are XOR-ed with (r % 8).  A tile [rows][cols] is
// the A or B operand of a product that contracts over `cols`.  Every wait is bounded.
#pragma once

#include "async_copy.cuh"
#include "common.cuh"
#include "umma.cuh"

namespace t2fw {
namespace c64 {

constexpr int kC = 64;                 // chunk length = checkpoint interval
constexpr int kDim = 64;               // D = K = 64
constexpr int kTile = 64 * 64 * 4;     // bytes of one operand tile
constexpr int kColBlock = 64 * 128;    // bytes of one 32-column block of a tile
constexpr int kRawBytes = kC * kDim * 2;
constexpr float kTinyState = 9.094947e-13f;     // 2^-40: smallest gate magnitude used in products
// Below this gate magnitude the pair terms of the gate gradient are summed directly.  The factored
// form divides a cancelled sum by the gate; measured against the step-by-step result its error is
// 7e-4 of the largest gradient for gates of 2^-13, 3e-3 at 2^-14.5, 5e-3 at 2^-16.5 and 4e-2 at
// 2^-18.5 (tolerance 2e-2).  Every entry costs a chunk of the pass a few hundred cycles, and N(0,1)
// gates fall below 2^-10 three times per chunk, below 2^-13 0.4 times.
constexpr float kTinyGate = 1.220703125e-4f;    // 2^-13
constexpr float kRangeLo = 7.888609e-31f;       // 2^-100
constexpr float kRangeHi = 1.267651e+30f;       // 2^100

// Round to TF32 (10 mantissa bits), nearest with ties away from zero - what cvt.rna.tf32.f32 does -
// as integer instructions: the conversion instruction runs on the quarter-rate pipe and there
// are hundreds of them per thread and chunk.  For a value that is ONLY stored as a tensor-core operand the
// mask can be left out: the tensor core ignores the low 13 bits of an fp32 operand (shared memory and tensor
// memory alike; tests/test_umma_gpu.py checks it), so adding half a unit of the last kept place is enough.
// The integer addition makes a zero of the NaN that arithmetic gives (0x7fffffff): without kNaN the row is one that
// is flagged.  kNaN: the half unit is added in floating point, one instruction more (everywhere: 96 x 1024 training
// 174 -> 183 us), with the same result for every other value.
template <bool kNaN = false>
__device__ __forceinline__ float bias_tf32(float v) {
  if (kNaN) return fmaf(__uint_as_float(__float_as_uint(v) & 0xff800000u), 0x1p-11f, v);
  return __uint_as_float(__float_as_uint(v) + 0x1000u);
}
template <bool kNaN = false>
__device__ __forceinline__ float rna_tf32(float v) {
  return __uint_as_float(__float_as_uint(bias_tf32<kNaN>(v)) & 0xffffe000u);
}

// The largest magnitude of three values, NaN if one of them is none (fmaxf would drop it): the range tests take the values
// along with the products, for no more instructions than without
__device__ __forceinline__ float max3_abs(float a, float b, float c) {
  float r;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float min3_abs(float a, float b, float c) {      // (drops a NaN)
  float r;
  asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
// whether all n values are finite numbers
template <int n>
__device__ __forceinline__ bool all_finite(const float (&v)[n]) {
  float m = 0.f;
#pragma unroll
  for (int j = 0; j < n; j += 2) m = max3_abs(m, v[j], v[j + 1]);
  return m <= 3.4028235e38f;
}

// 1 / v as the hardware's approximation (about 1 ulp; denormals count as zero, which every caller has excluded)
__device__ __forceinline__ float rcp_fast(float v) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}

__device__ __forceinline__ float sanitize_gate(float g) {
  return fabsf(g) < kTinyState ? copysignf(kTinyState, g) : g;
}

// shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

constexpr uint32_t kIdesc64 = umma::make_idesc_tf32(64, 64, false, false);
// descriptor offset of k-step ks (eight contraction columns) of a tile
__device__ __forceinline__ uint64_t kstep(int ks) { return (uint64_t)(((ks >> 2) * kColBlock + (ks & 3) * 32) >> 4); }

// D[tmem] (+)= A[tmem] * B[smem]^T: the A operand is read from tensor memory (row r of an M = 64
// operand in lane 32 * (r / 16) + r % 16 of a lane set, one 32-bit column per contraction index).
__device__ __forceinline__ void mma_tf32_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t desc_b, uint32_t idesc,
                                            bool accumulate) {
  const uint32_t acc = accumulate ? 1u : 0u, zero = 0u;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n"
      "}\n" ::"r"(d_tmem),
      "r"(a_tmem), "l"(desc_b), "r"(idesc), "r"(acc), "r"(zero)
      : "memory");
}

// 16-byte asynchronous copy global -> shared (no register, no scoreboard)
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(umma::smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// One lane of a converged warp.  The MMA-issuing code runs with the whole warp converged on
// warp-uniform values (so the descriptors live in uniform registers) and only the instruction
// itself is predicated on the elected lane.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile(
      "{\n"
      ".reg .pred P;\n"
      "elect.sync _|P, 0xffffffff;\n"
      "selp.u32 %0, 1, 0, P;\n"
      "}\n"
      : "=r"(pred));
  return pred != 0;
}
// warp index as a value the compiler knows to be the same in all lanes
__device__ __forceinline__ int uniform_warp_idx() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

// The work items of a persistent CTA: chunks first, first + stride, .. of the rows (problem rows; batch items when the
// state is a grid of blocks), and for each of them its nsub blocks in order - one CTA walks all blocks of a chunk, so
// that a thread meets its own results again when it sums over them.  Stepped without divisions.
struct ItemWalk {
  int row, c, sub;       // row, chunk, block
  int64_t unit;          // row * nc + c
  int step_row, step_c, nc, nsub;
  uint32_t stride;
  __device__ __forceinline__ ItemWalk(uint32_t first, uint32_t stride_, int64_t nc_, int nsub_) {
    nc = (int)nc_;
    nsub = nsub_;
    stride = stride_;
    unit = first;
    sub = 0;
    row = (int)(first / (uint32_t)nc);
    c = (int)first - row * nc;
    step_row = (int)(stride / (uint32_t)nc);
    step_c = (int)stride - step_row * nc;
  }
  __device__ __forceinline__ void step() {
    if (++sub < nsub) return;
    sub = 0;
    unit += stride;
    row += step_row;
    c += step_c;
    if (c >= nc) {
      c -= nc;
      ++row;
    }
  }
  // problem row, and the batch item and head (or block) that the tensors' windows are named by
  __device__ __forceinline__ int bh() const { return nsub == 1 ? row : row * nsub + sub; }
  __device__ __forceinline__ void item(int heads, int *b, int *h) const {
    if (nsub != 1 || heads == 1) {
      *b = row;
      *h = sub;
      return;
    }
    *b = (int)((uint32_t)row / (uint32_t)heads);
    *h = row - *b * heads;
  }
};

__device__ __forceinline__ void sync_all() {
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
}

}  // namespace c64
}  // namespace t2fw
