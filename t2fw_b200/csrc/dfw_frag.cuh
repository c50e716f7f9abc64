// Warp-level tensor-core fragments of the chunked delta rule (dfw_fwd.cu, dfw_bwd.cu): 64 x 64 matrices, TF32
// (m16n8k8) and 16-bit (m16n8k16) products with fp32 accumulation.
//
// Fragment image.  A 64 x 64 fp32 matrix X[r][c] as 1024 float4: element (rb, cb, lane) at (rb * 8 + cb) * 32 + lane
// holds, with g = lane / 4 and t = lane % 4,
//     x, y = X[16 rb + g][8 cb + 2t], [.. + 1]        z, w = X[16 rb + g + 8][8 cb + 2t], [.. + 1]
// which is how a warp's accumulators of rows 16 rb .. lie in its registers.  The sum over the contraction index
// does not depend on its order, so with logical index t read as column 2t and t + 4 as column 2t + 1 the same
// float4 is, without any exchange between lanes,
//   * the A operand of rows 16 rb .. , contraction columns 8 cb ..:  (x, z, y, w)
//   * the B operand of two 8-column tiles n = 16 rb + g and n = 16 rb + 8 + g, contraction columns 8 cb ..: (x, y), (z, w)
// A result therefore feeds the next product from registers, and travels through memory in 512-byte warp accesses.
//
// Raw 16-bit blocks [64][64] lie in shared memory as 128-byte rows whose eight 16-byte pieces are XOR-ed with
// (row % 8): ldmatrix reads them, straight or transposed, without bank conflicts, and its registers hold two
// consecutive contraction values, i.e. the operands of a 16-bit product as they are and, widened (every 16-bit
// value is exact in TF32), those of a TF32 product in the order above.
#pragma once

#include "async_copy.cuh"
#include "common.cuh"

namespace t2fw {
namespace frag {

constexpr int kC = 64;                       // chunk length
constexpr int kDim = 64;                     // D = M = 64
constexpr int kImg = kC * kDim;              // floats of an image
constexpr int kRaw = kC * kDim * 2;          // bytes of a raw block
constexpr int kThreads = 128;                // four warps
constexpr int kLdL = 68;                     // row stride (floats) of matrices that are read along columns (conflict-free)

// ---- products ------------------------------------------------------------------------------------
__device__ __forceinline__ void mma_tf32(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <typename T>
__device__ __forceinline__ void mma_16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1);
template <>
__device__ __forceinline__ void mma_16<__half>(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma_16<__nv_bfloat16>(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ---- operand values --------------------------------------------------------------------------------
// TF32 rounding (nearest, ties away) of a value that only feeds products: the tensor core drops the low 13 bits, so half a
// unit of the last kept place is added.  rnd: in floating point, for a NaN to stay one.  op: one integer addition, which makes
// a zero of the NaN that arithmetic gives (0x7fffffff), where another operand brings the NaN along as well.
__device__ __forceinline__ float rnd(float v) { return fmaf(__uint_as_float(__float_as_uint(v) & 0xff800000u), 0x1p-11f, v); }
__device__ __forceinline__ uint32_t op(float v) { return __float_as_uint(v) + 0x1000u; }
// v = hi + lo with both parts TF32 operands: together 22 bits (of a NaN, lo is one)
__device__ __forceinline__ void split(float v, uint32_t &hi, uint32_t &lo) {
  hi = op(v) & 0xffffe000u;
  lo = __float_as_uint(v - __uint_as_float(hi));
}
// the two 16-bit values of a register as TF32 operands (exact)
template <typename T> __device__ __forceinline__ uint32_t lo16(uint32_t u);
template <typename T> __device__ __forceinline__ uint32_t hi16(uint32_t u);
template <> __device__ __forceinline__ uint32_t lo16<__half>(uint32_t u) {
  return __float_as_uint(__low2float(*reinterpret_cast<const __half2 *>(&u)));
}
template <> __device__ __forceinline__ uint32_t hi16<__half>(uint32_t u) {
  return __float_as_uint(__high2float(*reinterpret_cast<const __half2 *>(&u)));
}
template <> __device__ __forceinline__ uint32_t lo16<__nv_bfloat16>(uint32_t u) { return u << 16; }
template <> __device__ __forceinline__ uint32_t hi16<__nv_bfloat16>(uint32_t u) { return u & 0xffff0000u; }
template <typename T> __device__ __forceinline__ uint32_t pack16(float a, float b);
template <> __device__ __forceinline__ uint32_t pack16<__half>(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&h);
}
template <> __device__ __forceinline__ uint32_t pack16<__nv_bfloat16>(float a, float b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&h);
}

// ---- raw 16-bit blocks in shared memory -------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ int raw_off(int row, int piece) { return row * 128 + ((piece ^ (row & 7)) << 4); }
__device__ __forceinline__ void ldsm(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// A operand, rows r0 .. r0+15 of the block, contraction columns 16 kk ..
__device__ __forceinline__ void raw_a(uint32_t (&r)[4], uint32_t base, int r0, int kk, int lane) {
  ldsm(r, base + raw_off(r0 + (lane & 15), 2 * kk + (lane >> 4)));
}
// A operand, rows = block columns m0 .. m0+15, contraction = block rows k0 .. k0+15
__device__ __forceinline__ void raw_at(uint32_t (&r)[4], uint32_t base, int m0, int k0, int lane) {
  ldsm_t(r, base + raw_off(k0 + (lane & 7) + ((lane >> 4) & 1) * 8, (m0 >> 3) + ((lane >> 3) & 1)));
}
// B operands of two 8-column tiles, columns = block rows n0 .. n0+15, contraction columns 16 kk ..:
// tile 0: r[0], r[1], tile 1: r[2], r[3] (first and second eight contraction values)
__device__ __forceinline__ void raw_b(uint32_t (&r)[4], uint32_t base, int n0, int kk, int lane) {
  ldsm(r, base + raw_off(n0 + (lane & 7) + ((lane >> 4) & 1) * 8, 2 * kk + ((lane >> 3) & 1)));
}
// the same with columns = block columns n0 .. n0+15, contraction = block rows k0 .. k0+15
__device__ __forceinline__ void raw_bt(uint32_t (&r)[4], uint32_t base, int k0, int n0, int lane) {
  ldsm_t(r, base + raw_off(k0 + (lane & 15), (n0 >> 3) + (lane >> 4)));
}
// TF32 product of 16 contraction values with both operands from raw registers / A from raw registers
template <typename T>
__device__ __forceinline__ void mma_raw_a(float (&c)[4], const uint32_t (&a)[4], int s, uint32_t b0, uint32_t b1) {
  mma_tf32(c, lo16<T>(a[2 * s]), lo16<T>(a[2 * s + 1]), hi16<T>(a[2 * s]), hi16<T>(a[2 * s + 1]), b0, b1);
}
// A operand from accumulators (rows of the warp, contraction columns = the eight columns of the tile)
__device__ __forceinline__ void mma_acc_a(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  mma_tf32(c, a[0], a[2], a[1], a[3], b0, b1);
}

// Block [64][64] of a dense [rows][64] array into shared memory, asynchronously; rows beyond nvalid become zeros.
template <typename T, int kN = kThreads>
__device__ __forceinline__ void load_raw(unsigned char *dst, const T *src, int nvalid, int tid) {
#pragma unroll
  for (int j = 0; j < 512 / kN; ++j) {
    const int i = tid + kN * j, r = i >> 3, p = i & 7;
    unsigned char *d = dst + raw_off(r, p);
    if (r < nvalid)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(d)), "l"(src + (size_t)r * kDim + p * 8) : "memory");
    else
      *reinterpret_cast<uint4 *>(d) = make_uint4(0u, 0u, 0u, 0u);
  }
}
// this warp's rows 16 w .. of a raw-format block in shared memory to a dense [rows][64] array, in whole rows
template <typename T>
__device__ __forceinline__ void rows_out(T *dst, const unsigned char *src, int w, int nvalid, int lane) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = 16 * w + 4 * i + (lane >> 3), p = lane & 7;
    if (r < nvalid) *reinterpret_cast<uint4 *>(dst + (size_t)r * kDim + 8 * p) = *reinterpret_cast<const uint4 *>(src + raw_off(r, p));
  }
}
// an image (or any 16 KB) into shared memory, asynchronously
template <int kN = kThreads>
__device__ __forceinline__ void load_image(float *dst, const float *src, int tid) {
#pragma unroll
  for (int j = 0; j < 1024 / kN; ++j) {
    const int i = tid + kN * j;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst + 4 * i)), "l"(src + 4 * i) : "memory");
  }
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void zero(float (&c)[8][4]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) c[i][0] = c[i][1] = c[i][2] = c[i][3] = 0.f;
}
// a warp's rows of an image: accumulators -> memory (optionally rounded and negated), memory -> registers
template <bool kRound>
__device__ __forceinline__ void store_rows(float *img, const float (&c)[8][4], int w, int lane, float sign = 1.f) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float4 v = make_float4(sign * c[i][0], sign * c[i][1], sign * c[i][2], sign * c[i][3]);
    if (kRound) v = make_float4(rnd(v.x), rnd(v.y), rnd(v.z), rnd(v.w));
    reinterpret_cast<float4 *>(img)[(w * 8 + i) * 32 + lane] = v;
  }
}
__device__ __forceinline__ float4 image_at(const float *img, int rb, int cb, int lane) {
  return reinterpret_cast<const float4 *>(img)[(rb * 8 + cb) * 32 + lane];
}
__device__ __forceinline__ uint32_t bits(float v) { return __float_as_uint(v); }

// c[n tiles] += A B^T over 64 contraction values, A = a warp's rows as accumulator registers (already operands),
// B = image in shared memory (rows = result columns)
__device__ __forceinline__ void mma_image(float (&c)[8][4], const uint32_t (&a)[8][4], const float *img, int lane) {
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int np = 0; np < 4; ++np) {
      const float4 b = image_at(img, np, j, lane);
      mma_acc_a(c[2 * np], a[j], bits(b.x), bits(b.y));
      mma_acc_a(c[2 * np + 1], a[j], bits(b.z), bits(b.w));
    }
}

// K^T B with the raw block K [t][m] and B [t][n] in shared memory (row stride kLdL): this warp's 32 x 32 part of the
// result, rows 32 (w / 2) .., columns 32 (w % 2) .. (a square part halves the reads of B, which cost most), to an image
template <typename T, bool kRoundB, bool kRoundOut>
__device__ __forceinline__ void mma_kt_b(float *img, uint32_t k, const float *B, float sign, int w, int lane) {
  const int g = lane >> 2, t = lane & 3, rb = 2 * (w >> 1), cb = 4 * (w & 1);
  float c[2][4][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int n = 0; n < 4; ++n) c[i][n][0] = c[i][n][1] = c[i][n][2] = c[i][n][3] = 0.f;
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) {
    uint32_t a[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) raw_at(a[i], k, 16 * (rb + i), 16 * kk, lane);
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const float *p = B + (16 * kk + 8 * s + 2 * t) * kLdL + 8 * (cb + n) + g;
        const uint32_t b0 = kRoundB ? op(p[0]) : bits(p[0]), b1 = kRoundB ? op(p[kLdL]) : bits(p[kLdL]);
#pragma unroll
        for (int i = 0; i < 2; ++i) mma_raw_a<T>(c[i][n], a[i], s, b0, b1);
      }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      float4 v = make_float4(sign * c[i][n][0], sign * c[i][n][1], sign * c[i][n][2], sign * c[i][n][3]);
      if (kRoundOut) v = make_float4(rnd(v.x), rnd(v.y), rnd(v.z), rnd(v.w));
      reinterpret_cast<float4 *>(img)[((rb + i) * 8 + cb + n) * 32 + lane] = v;
    }
}

// ---- (I + L)^-1 of a strictly lower triangular 64 x 64 matrix, fp32 -----------------------------------
// L in Ls [64][kLdL], the inverse to Ts [64][kLd] (diagonal blocks with their zeros; the blocks above the diagonal are
// neither written nor meant to be read).  Warp w owns block row w: it inverts its 16 x 16 diagonal block by
// substitution, one column per lane, and, once all of those are there, its blocks left of it from right to left,
//     T_ij = -( sum_{j<k<=i} T_ik L_kj ) T_jj ,
// which needs nothing from the other block rows of T.  The products are three TF32 products each (operands split in
// two), i.e. fp32-like.  Called by all four warps; ends without a barrier.
constexpr int kLdT = 72;      // stride of T where it is read along rows (8-byte reads, conflict-free)
// kLd: row stride of Ts
__device__ __forceinline__ void mma_split(float (&c)[4], const uint32_t (&ah)[4], const uint32_t (&al)[4], float b0, float b1) {
  uint32_t bh0, bl0, bh1, bl1;
  split(b0, bh0, bl0);
  split(b1, bh1, bl1);
  mma_acc_a(c, ah, bh0, bh1);
  mma_acc_a(c, al, bh0, bh1);
  mma_acc_a(c, ah, bl0, bl1);
}
template <int kLd>
__device__ __forceinline__ void unit_lower_inverse(const float *Ls, float *Ts, int w, int lane) {
  const int g = lane >> 2, t = lane & 3;
  if (lane < 16) {
    const float *Lb = Ls + (16 * w) * kLdL + 16 * w;
    float x[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      float a = r == lane ? 1.f : 0.f;
#pragma unroll
      for (int k4 = 0; k4 < r; k4 += 4) {
        const float4 l = *reinterpret_cast<const float4 *>(Lb + r * kLdL + k4);
        a = fmaf(-l.x, x[k4], a);
        if (k4 + 1 < r) a = fmaf(-l.y, x[k4 + 1], a);
        if (k4 + 2 < r) a = fmaf(-l.z, x[k4 + 2], a);
        if (k4 + 3 < r) a = fmaf(-l.w, x[k4 + 3], a);
      }
      x[r] = a;
      Ts[(16 * w + r) * kLd + 16 * w + lane] = a;
    }
  }
  __syncthreads();
  uint32_t th[4][2][4], tl[4][2][4];      // T_{w, w-r}, as A operands (hi, lo), r = 0 the diagonal block
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const float2 u = *reinterpret_cast<const float2 *>(Ts + (16 * w + g) * kLd + 16 * w + 8 * s + 2 * t);
    const float2 v = *reinterpret_cast<const float2 *>(Ts + (16 * w + g + 8) * kLd + 16 * w + 8 * s + 2 * t);
    split(u.x, th[0][s][0], tl[0][s][0]);
    split(u.y, th[0][s][1], tl[0][s][1]);
    split(v.x, th[0][s][2], tl[0][s][2]);
    split(v.y, th[0][s][3], tl[0][s][3]);
  }
#pragma unroll
  for (int jj = 0; jj < 3; ++jj) {
    const int j = w - 1 - jj;
    if (j < 0) break;
    float m[2][4] = {};
#pragma unroll
    for (int r = 0; r <= jj; ++r) {
      const float *L = Ls + (16 * (w - r)) * kLdL + 16 * j;
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int n = 0; n < 2; ++n)
          mma_split(m[n], th[r][s], tl[r][s], L[(8 * s + 2 * t) * kLdL + 8 * n + g], L[(8 * s + 2 * t + 1) * kLdL + 8 * n + g]);
    }
    uint32_t mh[2][4], ml[2][4];
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) split(-m[n][e], mh[n][e], ml[n][e]);
    const float *D = Ts + (16 * j) * kLd + 16 * j;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      float c[4] = {};
#pragma unroll
      for (int s = 0; s < 2; ++s)
        mma_split(c, mh[s], ml[s], D[(8 * s + 2 * t) * kLd + 8 * n + g], D[(8 * s + 2 * t + 1) * kLd + 8 * n + g]);
      *reinterpret_cast<float2 *>(Ts + (16 * w + g) * kLd + 16 * j + 8 * n + 2 * t) = make_float2(c[0], c[1]);
      *reinterpret_cast<float2 *>(Ts + (16 * w + g + 8) * kLd + 16 * j + 8 * n + 2 * t) = make_float2(c[2], c[3]);
#pragma unroll
      for (int e = 0; e < 4; ++e) split(c[e], th[jj + 1][n][e], tl[jj + 1][n][e]);
    }
  }
}

// strictly lower triangle of X Y^T (both raw blocks), rows 16 w .. of this warp, into Ls [64][kLdL]: exact products
template <typename T>
__device__ __forceinline__ void gram_lower(float *Ls, uint32_t x, uint32_t y, int w, int lane) {
  const int g = lane >> 2, t = lane & 3;
  uint32_t a[4][4];
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) raw_a(a[kk], x, 16 * w, kk, lane);
#pragma unroll
  for (int np = 0; np < 4; ++np) {
    if (np > w) break;
    float c[2][4] = {};
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      uint32_t b[4];
      raw_b(b, y, 16 * np, kk, lane);
      mma_16<T>(c[0], a[kk], b[0], b[1]);
      mma_16<T>(c[1], a[kk], b[2], b[3]);
    }
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int col = 16 * np + 8 * n + 2 * t, r0 = 16 * w + g, r1 = r0 + 8;
      *reinterpret_cast<float2 *>(Ls + r0 * kLdL + col) = make_float2(col < r0 ? c[n][0] : 0.f, col + 1 < r0 ? c[n][1] : 0.f);
      *reinterpret_cast<float2 *>(Ls + r1 * kLdL + col) = make_float2(col < r1 ? c[n][2] : 0.f, col + 1 < r1 ? c[n][3] : 0.f);
    }
  }
}

// ---- the carries: 16 rows of a state per warp or pair of warps, a ring of stages filled by bulk copies ------------------------------------------------
template <int kStages>
__device__ __forceinline__ void init_ring(uint64_t *full, int tid) {
  if (tid == 0) {
    for (int i = 0; i < kStages; ++i) acp::mbar_init(&full[i], 1);
    acp::mbar_fence_init();
  }
  __syncthreads();
}
// A chain that gave up at step i of n, with the stages up to i + kStages - 2 requested: they land (a bounded wait each) before
// the block leaves its shared memory to the next one.
template <int kStages>
__device__ __forceinline__ void drain_ring(uint64_t *full, int i, int n) {
  for (int j = i; j < n && j < i + kStages - 1; ++j) acp::mbar_wait(&full[j % kStages], (uint32_t)(j / kStages) & 1u);
}
// A state row with a NaN or an infinity in one column has them in all columns after the next step.  The rows that the carries
// start from and add are made so at once: then the products of the chain need not round with care (op), and one element tells
// of its row.  c: rows g and g + 8 of a warp's 16, the four lanes of a row hold its columns.  z0, z1: 0, or NaN.
template <int kN>
__device__ __forceinline__ void row_nonfinite(const float (&c)[kN][4], float &z0, float &z1) {
#pragma unroll
  for (int n = 0; n < kN; ++n) {
    z0 = fmaf(c[n][0], 0.f, fmaf(c[n][1], 0.f, z0));
    z1 = fmaf(c[n][2], 0.f, fmaf(c[n][3], 0.f, z1));
  }
#pragma unroll
  for (int o = 1; o < 4; o <<= 1) {
    z0 += __shfl_xor_sync(0xffffffffu, z0, o);
    z1 += __shfl_xor_sync(0xffffffffu, z1, o);
  }
}
template <int kN>
__device__ __forceinline__ void spread_nonfinite(float (&c)[kN][4], float z0, float z1) {
  if (z0 == 0.f && z1 == 0.f) return;
#pragma unroll
  for (int n = 0; n < kN; ++n) {
    c[n][0] += z0; c[n][1] += z0;
    c[n][2] += z1; c[n][3] += z1;
  }
}
// the carries' start: with kH = 2 a row's other columns are the partner warp's (x: [kW][2][2][8] floats)
template <int kH>
__device__ __forceinline__ void spread_start(float (&c)[8 / kH][4], float *x, int wl, int ch, int lane) {
  float z0 = 0.f, z1 = 0.f;
  row_nonfinite(c, z0, z1);
  if (kH == 2) {
    float *own = x + ((wl * 2 + ch) * 2) * 8 + (lane >> 2), *oth = x + ((wl * 2 + (ch ^ 1)) * 2) * 8 + (lane >> 2);
    if ((lane & 3) == 0) {
      own[0] = z0;
      own[8] = z1;
    }
    __syncthreads();
    z0 += oth[0];
    z1 += oth[8];
    __syncthreads();      // x is used again
  }
  spread_nonfinite(c, z0, z1);
}
// operands as a part of an image, with their rows' 0 or NaN
__device__ __forceinline__ float4 with_rows(const uint32_t (&a)[4], float z0, float z1) {
  return make_float4(__uint_as_float(a[0]) + z0, __uint_as_float(a[1]) + z0, __uint_as_float(a[2]) + z1, __uint_as_float(a[3]) + z1);
}
// One step's product for a warp of 16 rows and 1 / kH of the columns (part ch) of X += A B^T: A = all 64 columns of X as
// operands, the own ones first (own), then the partner's (oth, kH = 2); B in registers, which take the next step's B as they
// are used: its loads run under this product.
template <int kH>
__device__ __forceinline__ int carry_col(int jj, int ch) { return kH == 1 ? jj : (jj & 3) + 4 * (jj < 4 ? ch : ch ^ 1); }
template <int kH>
__device__ __forceinline__ void carry_load_b(float4 (&bq)[8][4 / kH], const float *img, int ch, int lane) {
#pragma unroll
  for (int jj = 0; jj < 8; ++jj)
#pragma unroll
    for (int np = 0; np < 4 / kH; ++np) bq[jj][np] = image_at(img, 4 / kH * ch + np, carry_col<kH>(jj, ch), lane);
}
template <int kH>
__device__ __forceinline__ void carry_product(float (&c)[8 / kH][4], const uint32_t (&own)[8 / kH][4], const uint32_t (&oth)[4][4],
                                              float4 (&bq)[8][4 / kH], const float *next, int ch, int lane) {
#pragma unroll
  for (int jj = 0; jj < 8; ++jj)
#pragma unroll
    for (int np = 0; np < 4 / kH; ++np) {
      const float4 b = bq[jj][np];
      mma_acc_a(c[2 * np], jj < 8 / kH ? own[jj % (8 / kH)] : oth[jj & 3], bits(b.x), bits(b.y));
      mma_acc_a(c[2 * np + 1], jj < 8 / kH ? own[jj % (8 / kH)] : oth[jj & 3], bits(b.z), bits(b.w));
      bq[jj][np] = image_at(next, 4 / kH * ch + np, carry_col<kH>(jj, ch), lane);
    }
}
// How B rows are spread: one or two of a row's four blocks per CTA with a pair of warps each, while that leaves a CTA an SM of
// its own (every CTA fetches the whole transition matrix of a chunk); else a row per CTA with a warp per block, the ring as deep as
// shared memory allows as long as an SM holds one CTA.  Training calls, fp16, a warp per block in one CTA with three stages that
// all threads copy -> now: 1 row x 4096 steps 161 -> 117 us, 8 x 4096 212 -> 162, 32 x 4096 418 -> 346, 48 x 1333 186 -> 167,
// 74 x 1333 257 -> 244, 96 x 1024 242 -> 236, 200 x 512 253 -> 244, 384 x 341 347 -> 342; pairs of warps instead at 96 and 200
// rows: 240, 250.
enum CarryPlan { kSpread1, kSpread2, kDeep, kDense };
inline CarryPlan carry_plan(int64_t B, int n_sm) { return 4 * B <= n_sm ? kSpread1 : 2 * B <= n_sm ? kSpread2 : B <= n_sm ? kDeep : kDense; }
// shared memory of a carry besides its ring of stages: barriers, and the halves' exchange
template <int kW, int kH, int kStages> constexpr int kCarryStatic = kStages * 8 + (kH == 2 ? 2 * kW * 8 * 32 * 16 : 16);
constexpr int kSharedLimit = 227 * 1024;

}  // namespace frag
int lfw_chunk_status_ptr(int **out);      // lfw_c64_local.cu
int lfw_chunk_sm_count(int *out);
}  // namespace t2fw
