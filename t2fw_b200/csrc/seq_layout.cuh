// Where the [64 steps][64 features] blocks of the sequence tensors lie, and how they are fetched.
//
// Every sequence tensor of a call is a 2-D array of 16-bit elements, rows = batch item x time,
// described to the copy engine by a tensor map (cuTensorMapEncodeTiled); a chunk's block of one
// tensor is ONE tiled bulk copy (cp.async.bulk.tensor.2d) of a 64 x 64 box that lands as a dense
// row-major [64][64] block in shared memory.  The plain operators pass [B*T, 64] arrays; the fused
// layer entry points pass the projection output [B*T, 4*H*64] (query | key | value | gate, heads
// inside a row) and read the heads in place, so no folded copies of the tensors are ever made.
// Rows of a box that fall outside the array arrive as zeros; rows that belong to the next batch
// item (a partial last chunk) are overwritten with identity steps by the kernels.
#pragma once

#include <cuda.h>

#include "async_copy.cuh"
#include "common.cuh"

namespace t2fw {
namespace seq {

constexpr int kMaxTensors = 6;

enum : int {
  kFusedLayer = 1,     // the d-side gate is the constant 1 (nothing is read for it), the k-side gate tensor holds
                       //   pre-activations, gate = max(sigmoid(g), 1/8), and the query is scaled
  kContiguous = 2,     // every tensor is a dense [rows][64] array: a chunk's block is one linear 8 KB copy
};
constexpr float kGateFloor = 0.125f;   // with gates >= 1/8 no 32-step product leaves the safe range

struct Maps {
  CUtensorMap m[kMaxTensors];    // one per input tensor of the kernel
  CUtensorMap out;               // fused layer, backward: the gradient of the projection output
  const void *base[kMaxTensors]; // the arrays themselves (used for the linear copies of dense [rows][64] arrays)
  int col[kMaxTensors];          // column of sub-item 0 in a row of that tensor (elements)
  int hdiv[kMaxTensors];         // sub-item h of a batch item reads the 64-column window number
  int hmod[kMaxTensors];         //   (h / hdiv) % hmod of that tensor
  int heads;                     // sub-items per batch item: problem row bh = b * heads + h.  Heads of a
                                 // layer: hdiv = 1, hmod = heads.  A D x K state cut into 64 x 64 blocks:
                                 // h = i * (K/64) + j, d-side tensors hdiv = K/64, hmod = D/64, k-side 1, K/64
  int nsub, nk;                  // state cut into a grid of 64 x 64 blocks: nsub blocks per batch item (1: no grid), block
                                 // i * nk + j; results are summed over the blocks of the other axis
  int64_t state_item;            // elements of one state of a batch item (or problem row without a grid), and the
  int state_ld;                  //   stride of its rows
  int flags;
  float q_scale;                 // fused layer: factor on the query tensor
};

// element offset of the 64 x 64 block of sub-item `sub` of item `b` (problem row without a grid), state number c of S
__device__ __forceinline__ size_t state_off(const Maps &mp, int b, int sub, int64_t c, int64_t S) {
  const int i = mp.nsub == 1 ? 0 : sub / mp.nk, j = mp.nsub == 1 ? 0 : sub - i * mp.nk;
  return ((size_t)b * S + c) * mp.state_item + (size_t)i * 64 * mp.state_ld + j * 64;
}

// an output tensor: element (row of the 2-D array, feature) at p[row * ld + col + 64 * h + feature]
template <typename T>
struct Out {
  T *p;
  int64_t ld;
  int col;
};

// box (64 features x 64 rows) with its first row `row` and first column `col` -> dst (8 KB, 128-byte aligned)
__device__ __forceinline__ void load_block(void *dst, const CUtensorMap *map, int col, int row, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          acp::smem_u32(dst)),
      "l"(map), "r"(col), "r"(row), "r"(acp::smem_u32(bar))
      : "memory");
}

// dense [64][64] block in shared memory -> box whose first row is `row` and first column `col` (neither negative); the
// caller commits the group
__device__ __forceinline__ void store_block(const CUtensorMap *map, int col, int row, const void *src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(map), "r"(col), "r"(row),
               "r"(acp::smem_u32(src))
               : "memory");
}

// ---- activations of the fused layer: gate = max(sigmoid(g), 1/8), rounded to the storage type (what a separate
//      elementwise pass followed by the plain operator would have fed the kernels) ------------------------
template <typename T>
__device__ __forceinline__ float round_to(float v) {
  const T r = (T)v;
  return Elem<T>::ld(&r);
}
// e^-g and 1 / v as single hardware approximations (about 2 ulp; the library forms add range handling that these
// arguments do not need: an overflow gives gate 0, which the floor lifts, and denormals count as zero)
__device__ __forceinline__ float exp_neg(float g) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(g * -1.4426950408889634f));
  return r;
}
__device__ __forceinline__ float rcp1p(float e) {      // 1 / (1 + e)
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.f + e));
  return r;
}
__device__ __forceinline__ float floored(float s) {      // NaN stays NaN (fmaxf would give the floor)
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(s), "f"(kGateFloor));
  return r;
}
template <typename T>
__device__ __forceinline__ float sigmoid_gate(float g) {
  return round_to<T>(floored(rcp1p(exp_neg(g))));
}
// The block of tensor i for the chunk whose first row is `row` (nv valid rows), sub-item h.
// Dense [rows][64] arrays: one linear bulk copy of the valid rows; otherwise the tiled copy of the
// whole box.  Returns the bytes that will arrive on the barrier.
template <typename T>
__device__ __forceinline__ uint32_t fetch_block(const Maps &mp, int i, void *dst, int row, int h, int nv, uint64_t *bar) {
  if (mp.flags & kContiguous) {
    const uint32_t bytes = (uint32_t)nv * 64u * sizeof(T);
    acp::bulk_g2s(dst, static_cast<const T *>(mp.base[i]) + (size_t)row * 64, bytes, bar);
    return bytes;
  }
  load_block(dst, &mp.m[i], mp.col[i] + ((h / mp.hdiv[i]) % mp.hmod[i]) * 64, row, bar);
  return 64u * 64u * sizeof(T);
}

// host: tensor map of a [rows][cols] array of 16-bit elements with `ld` elements between rows
int make_map(CUtensorMap *out, const void *base, uint64_t rows, uint64_t cols, uint64_t ld);

}  // namespace seq
}  // namespace t2fw
