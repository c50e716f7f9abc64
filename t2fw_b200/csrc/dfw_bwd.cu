// Delta rule, chunked backward (D = M = 64, 16-bit storage, chunks of 64 steps).  Replaces
// t2fw/csrc/dfw_kernel.cu:198-384 for these shapes.
//
// With L = strict_lower(K K^T), T = (I + L)^-1 of a chunk, S0 / S_end its start / end state, R the state gradient at
// its end, and Dl the forward's deltas:
//     E = d_value = Ub + Wb R^T         Wb = T^T K ,  Ub = T^T strict_upper(K Q^T) dO
//     R_start = R + dO^T Q - E^T K = R + R Qb + Nb     with  Qb = -Wb^T K ,  Nb = dO^T Q - Ub^T K
//     S0 = S_end - Dl^T K                              (the state is walked back from final_state)
//     d_query = dO S0 + strict_lower(dO Dl^T) K
//     d_key   = Dl R + strict_upper(Dl dO^T) Q - Y K - E S0 ,   Y = strict_upper(Dl E^T) + strict_lower(E Dl^T)
// As in the forward one 64 x 64 x 64 product per chunk is sequential (R); the walk back of the state is a sum.
//
//   dfw_prep_bwd_kernel   (row, chunk)   Wb, Ub, Qb^T, Nb, (Dl^T K)^T
//   dfw_carry_bwd_kernel  row            chunks in reverse: R_end and S0^T of every chunk; d_state
//   dfw_grad_kernel       (row, chunk)   E = d_value, d_query, d_key
// Fragment images and operand precision as in dfw_fwd.cu: products among K, Q and dO are exact, Wb and Ub come from T
// (and the right-hand side) split in two, everything else is TF32 with fp32 accumulation.
//
// What bounds it is latency at few warps, no pipe.  B*H = 96, T = 1024, fp16, cold caches: prep 60 us, tensor pipe 50 %,
// issue slots 35 %, 11 warps per SM; carry 28 us, 4 warps on each of 96 SMs, tensor 18 %; gradients 78 us, tensor 40 %,
// issue slots 30 %, 15 warps per SM that wait most for the other group at the five meetings, then for global memory
// (252 bytes of spills per thread among it).  Whole backward 188 -> 165 us.
#include "dfw_frag.cuh"

namespace t2fw {

using namespace frag;

namespace {

// ---- prep: grid = B * nc, four warps -----------------------------------------------------------------
constexpr int oK = 0, oQ = kRaw, oG = 2 * kRaw, oT = 3 * kRaw, oL = oT + kC * kLdL * 4;
constexpr int kSmemPrep = oL + kC * kLdL * 4;

template <typename T>
__global__ void __launch_bounds__(kThreads, 3)
dfw_prep_bwd_kernel(const T *__restrict__ go, const T *__restrict__ q, const T *__restrict__ k, const float *__restrict__ delta,
                    float *__restrict__ Wimg, float *__restrict__ Ub, float *__restrict__ Qimg, float *__restrict__ Nimg,
                    float *__restrict__ Gimg, int64_t T_, int nc) {
  extern __shared__ __align__(128) unsigned char sm[];
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  float *Ts = reinterpret_cast<float *>(sm + oT), *Ls = reinterpret_cast<float *>(sm + oL);
  const uint32_t aK = smem_u32(sm + oK), aQ = smem_u32(sm + oQ), aG = smem_u32(sm + oG);
  const int64_t b = blockIdx.x / (uint32_t)nc, t0 = (int64_t)(blockIdx.x - (uint32_t)b * nc) * kC;
  const int nvalid = (int)(T_ - t0 < kC ? T_ - t0 : kC);
  const size_t base = ((size_t)b * T_ + t0) * kDim, img = (size_t)blockIdx.x * kImg;
  dependency_wait();
  load_raw(sm + oK, k + base, nvalid, tid);
  load_raw(sm + oQ, q + base, nvalid, tid);
  load_raw(sm + oG, go + base, nvalid, tid);
  commit();
  wait<0>();
  __syncthreads();
  gram_lower<T>(Ls, aK, aK, w, lane);
  __syncwarp();
  unit_lower_inverse<kLdL>(Ls, Ts, w, lane);
  // C = strict_upper(K Q^T), rows t = 16 w ..: the warps with the least to do in the inverse have the most blocks here
  float *Cs = Ls;
  {
    float c[4][2][4] = {};
    uint32_t a[4][4];
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) raw_a(a[kk], aK, 16 * w, kk, lane);
#pragma unroll
    for (int np = 0; np < 4; ++np) {
      if (np < w) continue;
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        uint32_t r[4];
        raw_b(r, aQ, 16 * np, kk, lane);
        mma_16<T>(c[np][0], a[kk], r[0], r[1]);
        mma_16<T>(c[np][1], a[kk], r[2], r[3]);
      }
    }
    __syncthreads();             // L is no longer read: C over it, as an image
#pragma unroll
    for (int np = 0; np < 4; ++np) {
      if (np < w) continue;
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const int col = 16 * np + 8 * n + 2 * t, r0 = 16 * w + g, r1 = r0 + 8;
        reinterpret_cast<float4 *>(Cs)[(w * 8 + 2 * np + n) * 32 + lane] =
            make_float4(col > r0 ? rnd(c[np][n][0]) : 0.f, col + 1 > r0 ? rnd(c[np][n][1]) : 0.f, col > r1 ? rnd(c[np][n][2]) : 0.f,
                        col + 1 > r1 ? rnd(c[np][n][3]) : 0.f);
      }
    }
  }
  __syncthreads();
  float u[8][4];      // Ub^T, rows d = 16 w .., columns t
  {
    float r[8][4];      // right-hand side transposed: rhs^T[d][t] = sum_{s>t} dO[s][d] C[t][s]
    zero(r);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      uint32_t a[4];
      raw_at(a, aG, 16 * w, 16 * kk, lane);
#pragma unroll
      for (int np = 0; np <= kk; ++np)
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const float4 c4 = image_at(Cs, np, 2 * kk + s, lane);
          mma_raw_a<T>(r[2 * np], a, s, bits(c4.x), bits(c4.y));
          mma_raw_a<T>(r[2 * np + 1], a, s, bits(c4.z), bits(c4.w));
        }
    }
    zero(u);      // Ub^T[d][t] = sum_{s>=t} rhs^T[d][s] T[s][t]
#pragma unroll
    for (int j = 0; j < 8; ++j) {      // s = 8 j ..
      uint32_t ah[4], al[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) split(r[j][e], ah[e], al[e]);
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        if (n > (j | 1)) continue;      // blocks of T above the diagonal
        const float *p = Ts + (8 * j + 2 * t) * kLdL + 8 * n + g;
        mma_split(u[n], ah, al, p[0], p[kLdL]);
      }
    }
    float *up = Ub + img + 16 * w + g;      // [t][d]: eight lanes = 32 contiguous bytes of a step
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int s = 8 * n + 2 * t;
      up[s * kDim] = u[n][0];
      up[(s + 1) * kDim] = u[n][1];
      up[s * kDim + 8] = u[n][2];
      up[(s + 1) * kDim + 8] = u[n][3];
    }
  }
  {   // Nb = dO^T Q - Ub^T K, rows d = 16 w ..
    float c[8][4];
    zero(c);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      uint32_t a[4], ua[2][4];
      raw_at(a, aG, 16 * w, 16 * kk, lane);
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int e = 0; e < 4; ++e) ua[s][e] = op(-u[2 * kk + s][e]);
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        uint32_t r[4], x[4];
        raw_bt(r, aQ, 16 * kk, 16 * np, lane);
        raw_bt(x, aK, 16 * kk, 16 * np, lane);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          mma_16<T>(c[2 * np + n], a, r[2 * n], r[2 * n + 1]);
#pragma unroll
          for (int s = 0; s < 2; ++s) mma_acc_a(c[2 * np + n], ua[s], lo16<T>(x[2 * n + s]), hi16<T>(x[2 * n + s]));
        }
      }
    }
    float z0 = 0.f, z1 = 0.f;      // a NaN in Ub^T (which op has dropped) or in a column of c
    row_nonfinite(u, z0, z1);
    row_nonfinite(c, z0, z1);
    spread_nonfinite(c, z0, z1);
    store_rows<false>(Nimg + img, c, w, lane);
  }
  float wb[8][4];      // Wb = T^T K, rows t = 16 w ..
  {
    zero(wb);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      if (kk < w) continue;
      uint32_t ah[2][4], al[2][4];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const float *p = Ts + (16 * kk + 8 * s + 2 * t) * kLdL + 16 * w + g;
        split(p[0], ah[s][0], al[s][0]);
        split(p[kLdL], ah[s][1], al[s][1]);
        split(p[8], ah[s][2], al[s][2]);
        split(p[kLdL + 8], ah[s][3], al[s][3]);
      }
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        uint32_t r[4];
        raw_bt(r, aK, 16 * kk, 16 * np, lane);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            const uint32_t b0 = lo16<T>(r[2 * n + s]), b1 = hi16<T>(r[2 * n + s]);
            mma_acc_a(wb[2 * np + n], ah[s], b0, b1);
            mma_acc_a(wb[2 * np + n], al[s], b0, b1);
          }
      }
    }
    store_rows<true>(Wimg + img, wb, w, lane);
  }
  __syncthreads();             // T and C are no longer read
  float *Ws = Ls, *Ds = Ts;    // Wb [64][kLdL] over C; Dl [64][kLdL] over T
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int i = tid + kThreads * j, r = i >> 4, p = i & 15;
    float *d = Ds + r * kLdL + 4 * p;
    if (r < nvalid)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(d)), "l"(delta + base + (size_t)r * kDim + 4 * p) : "memory");
    else
      *reinterpret_cast<float4 *>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  commit();
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    *reinterpret_cast<float2 *>(Ws + (16 * w + g) * kLdL + 8 * n + 2 * t) = make_float2(rnd(wb[n][0]), rnd(wb[n][1]));
    *reinterpret_cast<float2 *>(Ws + (16 * w + g + 8) * kLdL + 8 * n + 2 * t) = make_float2(rnd(wb[n][2]), rnd(wb[n][3]));
  }
  __syncthreads();
  mma_kt_b<T, false, true>(Qimg + img, aK, Ws, -1.f, w, lane);      // Qb^T = -K^T Wb
  wait<0>();
  __syncthreads();
  mma_kt_b<T, true, false>(Gimg + img, aK, Ds, 1.f, w, lane);       // (Dl^T K)^T = K^T Dl
}

// ---- carry, chunks in reverse: blocks of 16 rows of R [d][m] and of S^T [m][d], spread over CTAs and warps as in the forward ----
// Qb^T and the CTA's parts of Nb and (Dl^T K)^T of a chunk arrive together by bulk copies; R_end (row-major) replaces Nb and
// S0^T (an image) replaces (Dl^T K)^T.
template <typename T, int kW, int kH, int kStages>
__global__ void __launch_bounds__(32 * kH * kW)
dfw_carry_bwd_kernel(const T *__restrict__ gs, const T *__restrict__ final_state, const float *__restrict__ Qimg,
                     float *__restrict__ NR, float *__restrict__ GS, T *__restrict__ ds, int nc, int *__restrict__ status) {
  extern __shared__ __align__(128) unsigned char sm[];
  __shared__ __align__(8) uint64_t full[kStages];
  __shared__ uint4 xs[kH == 2 ? 2 : 1][kH == 2 ? kW : 1][kH == 2 ? 8 : 1][kH == 2 ? 32 : 1];      // operands of the block's rows, by step parity
  constexpr int kN = 8 / kH;                                            // 8-column tiles of a warp
  constexpr int kPart = kW * kImg / 4, kStage = kImg + 2 * kPart;      // floats
  float *ring = reinterpret_cast<float *>(sm);
  const int tid = threadIdx.x, wl = tid / (32 * kH), ch = kH == 1 ? 0 : (tid >> 5) & 1, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int64_t b = blockIdx.x / (4 / kW);
  const int w0 = (int)(blockIdx.x % (4 / kW)) * kW, w = w0 + wl;
  const size_t img0 = (size_t)b * nc * kImg;
  init_ring<kStages>(full, tid);
  dependency_wait();
  auto fetch = [&](int i) {      // i-th chunk from the end; one thread
    if (i >= nc) return;
    const size_t o = img0 + (size_t)(nc - 1 - i) * kImg;
    uint64_t *bar = &full[i % kStages];
    float *dst = ring + (i % kStages) * kStage;
    acp::mbar_expect_tx(bar, (uint32_t)(kStage * sizeof(float)));
    acp::bulk_g2s(dst, Qimg + o, kImg * (uint32_t)sizeof(float), bar);
    acp::bulk_g2s(dst + kImg, NR + o + w0 * (kImg / 4), kPart * (uint32_t)sizeof(float), bar);
    acp::bulk_g2s(dst + kImg + kPart, GS + o + w0 * (kImg / 4), kPart * (uint32_t)sizeof(float), bar);
  };
  if (tid == 0) {
    for (int i = 0; i < kStages - 1; ++i) fetch(i);
  }
  float R[kN][4], S[kN][4];
  {
    const T *rp = gs + ((size_t)b * kDim + 16 * w + g) * kDim + 32 * ch + 2 * t;
    const T *sp = final_state + (size_t)b * kDim * kDim + (32 * ch + 2 * t) * kDim + 16 * w + g;      // S^T[m = 16 w + g][d]
#pragma unroll
    for (int n = 0; n < kN; ++n) {
      const uint32_t u = *reinterpret_cast<const uint32_t *>(rp + 8 * n), x = *reinterpret_cast<const uint32_t *>(rp + 8 * kDim + 8 * n);
      R[n][0] = __uint_as_float(lo16<T>(u)); R[n][1] = __uint_as_float(hi16<T>(u));
      R[n][2] = __uint_as_float(lo16<T>(x)); R[n][3] = __uint_as_float(hi16<T>(x));
      S[n][0] = Elem<T>::ld(sp + 8 * n * kDim); S[n][1] = Elem<T>::ld(sp + (8 * n + 1) * kDim);
      S[n][2] = Elem<T>::ld(sp + 8 * n * kDim + 8); S[n][3] = Elem<T>::ld(sp + (8 * n + 1) * kDim + 8);
    }
  }
  spread_start<kH>(R, reinterpret_cast<float *>(&xs[0][0][0][0]), wl, ch, lane);
  int fail = acp::mbar_wait(&full[0], 0) ? 0 : 1;
  float4 bq[8][4 / kH];
  carry_load_b<kH>(bq, ring, ch, lane);
  int i = 0;
  for (; i < nc; ++i) {
    uint32_t own[kN][4], oth[4][4];
#pragma unroll
    for (int n = 0; n < kN; ++n) {
#pragma unroll
      for (int e = 0; e < 4; ++e) own[n][e] = op(R[n][e]);
      if (kH == 2) xs[i & 1][wl][4 * ch + n][lane] = make_uint4(own[n][0], own[n][1], own[n][2], own[n][3]);
    }
    const int in = i + 1 < nc ? i + 1 : i;      // (the last chunk's matrix once more: nobody uses it)
    if (!acp::mbar_wait(&full[in % kStages], (uint32_t)(in / kStages) & 1u)) fail = 1;
    if (__syncthreads_or(fail)) break;      // the halves are exchanged; the buffer refilled next is no longer read
    if (tid == 0) fetch(i + kStages - 1);
    const float *buf = ring + (i % kStages) * kStage;
    const size_t o = img0 + (size_t)(nc - 1 - i) * kImg;
    float *rp = NR + o + (16 * w + g) * kDim + 32 * ch + 2 * t;
    float4 *const img = reinterpret_cast<float4 *>(GS + o) + (w * 8 + 4 * ch) * 32 + lane;
    const float z0 = R[0][0] * 0.f, z1 = R[0][2] * 0.f;
#pragma unroll
    for (int n = 0; n < kN; ++n) {
      if (kH == 2) {
        const uint4 u = xs[i & 1][wl][4 * (ch ^ 1) + (n & 3)][lane];
        oth[n & 3][0] = u.x; oth[n & 3][1] = u.y; oth[n & 3][2] = u.z; oth[n & 3][3] = u.w;
      }
      const float4 gx = image_at(buf + kImg + kPart, wl, 4 * ch + n, lane), nx = image_at(buf + kImg, wl, 4 * ch + n, lane);
      S[n][0] -= gx.x; S[n][1] -= gx.y; S[n][2] -= gx.z; S[n][3] -= gx.w;
      img[n * 32] = make_float4(rnd(S[n][0]), rnd(S[n][1]), rnd(S[n][2]), rnd(S[n][3]));
      const float4 r4 = with_rows(own[n], z0, z1);
      *reinterpret_cast<float2 *>(rp + 8 * n) = make_float2(r4.x, r4.y);
      *reinterpret_cast<float2 *>(rp + 8 * kDim + 8 * n) = make_float2(r4.z, r4.w);
      R[n][0] += nx.x; R[n][1] += nx.y; R[n][2] += nx.z; R[n][3] += nx.w;
    }
    carry_product<kH>(R, own, oth, bq, ring + (in % kStages) * kStage, ch, lane);
  }
  if (fail) atomicExch(status, 1);
  if (i < nc && tid == 0) drain_ring<kStages>(full, i, nc);
  T *dp = ds + ((size_t)b * kDim + 16 * w + g) * kDim + 32 * ch + 2 * t;
#pragma unroll
  for (int n = 0; n < kN; ++n) {
    *reinterpret_cast<uint32_t *>(dp + 8 * n) = pack16<T>(R[n][0], R[n][1]);
    *reinterpret_cast<uint32_t *>(dp + 8 * kDim + 8 * n) = pack16<T>(R[n][2], R[n][3]);
  }
}

template <typename T, int kW, int kH, int kStages>
int launch_carry_bwd(const void *gs, const void *final_state, const float *Qb, float *NR, float *GS, void *ds, int64_t B, int nc,
                     int *status, cudaStream_t st) {
  constexpr int kSmem = kStages * (kImg + 2 * kW * kImg / 4) * 4;
  static_assert(kSmem + kCarryStatic<kW, kH, kStages> <= kSharedLimit, "shared memory limit");
  auto *const carry = &dfw_carry_bwd_kernel<T, kW, kH, kStages>;
  T2FW_ALLOW_SMEM(carry, kSmem);
  T2FW_CHECK_CUDA(launch_dependent(carry, dim3((unsigned)(B * (4 / kW))), dim3(32 * kH * kW), kSmem, st, (const T *)gs,
                                   (const T *)final_state, Qb, NR, GS, (T *)ds, nc, status));
  return T2FW_OK;
}

// ---- gradients: grid = B * nc, eight warps ---------------------------------------------------------------------
// Two groups of four warps, warp w of a group = steps 16 w ..: group 0 forms E and everything that contracts with
// strictly lower blocks (d_query, part of d_key), group 1 the rest of d_key; equal numbers of products, and half
// the registers of one group doing both.  The groups meet at a named barrier: each of the five meetings is in both
// branches, where __syncthreads() would be undefined.
constexpr int kThreadsG = 256;
__device__ __forceinline__ void meet() { asm volatile("bar.sync 1, %0;" ::"n"(kThreadsG) : "memory"); }
constexpr int kLdD = 72;      // row stride of Dl: 8-byte reads along its rows are free of bank conflicts
constexpr int oKg = 0, oQg = kRaw, oGg = 2 * kRaw, oDg = 3 * kRaw, oRg = oDg + kC * kLdD * 4;      // R, then E image
constexpr int oSg = oRg + kImg * 4;                                                               // S0^T image, then group 0's d_key
constexpr int oEg = oSg + kImg * 4, kSmemGrad = oEg + kRaw;                                       // d_value on its way out
// R is read along rows (8 bytes of eight consecutive rows at a time) and along columns (4 bytes of every other row): its
// 16-byte pieces are XOR-ed with twice a number that differs between any four rows a wavefront of either kind touches.
__device__ __forceinline__ int r_off(int d, int m) {
  return d * kDim + ((((m >> 2) ^ (2 * ((d & 3) ^ ((d >> 2) & 1)))) << 2) | (m & 3));
}

template <typename T>
__global__ void __launch_bounds__(kThreadsG, 2)
dfw_grad_kernel(const T *__restrict__ go, const T *__restrict__ q, const T *__restrict__ k, const float *__restrict__ delta,
                const float *__restrict__ Wimg, const float *__restrict__ Ub, const float *__restrict__ Rrow,
                const float *__restrict__ STimg, T *__restrict__ dq, T *__restrict__ dk, T *__restrict__ dv, int64_t T_, int nc) {
  extern __shared__ __align__(128) unsigned char sm[];
  const int tid = threadIdx.x, w = (tid >> 5) & 3, group = tid >> 7, lane = tid & 31, g = lane >> 2, t = lane & 3;
  float *Ds = reinterpret_cast<float *>(sm + oDg), *Rs = reinterpret_cast<float *>(sm + oRg), *Es = Rs;
  float *Ss = reinterpret_cast<float *>(sm + oSg);
  const uint32_t aK = smem_u32(sm + oKg), aQ = smem_u32(sm + oQg), aG = smem_u32(sm + oGg);
  const uint32_t blk = gridDim.x - 1 - blockIdx.x;      // last first: what prep wrote last is still in L2
  const int64_t b = blk / (uint32_t)nc, t0 = (int64_t)(blk - (uint32_t)b * nc) * kC;
  const int nvalid = (int)(T_ - t0 < kC ? T_ - t0 : kC);
  const size_t base = ((size_t)b * T_ + t0) * kDim, img = (size_t)blk * kImg;
  dependency_wait();
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int i = tid + kThreadsG * j, r = i >> 4, p = i & 15;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(Rs + r_off(r, 4 * p))), "l"(Rrow + img + r * kDim + 4 * p) : "memory");
    float *d = Ds + r * kLdD + 4 * p;
    if (r < nvalid)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(d)), "l"(delta + base + (size_t)r * kDim + 4 * p) : "memory");
    else
      *reinterpret_cast<float4 *>(d) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  commit();
  load_raw<T, kThreadsG>(sm + oGg, go + base, nvalid, tid);
  load_raw<T, kThreadsG>(sm + oKg, k + base, nvalid, tid);
  load_raw<T, kThreadsG>(sm + oQg, q + base, nvalid, tid);
  load_image<kThreadsG>(Ss, STimg + img, tid);
  commit();
  const int r0 = 16 * w + g, r1 = r0 + 8;
  uint32_t ea[8][4];      // -E as an operand, own rows
  float ck[8][4];         // d_key
  zero(ck);

  if (group == 0) {
    float e[8][4];      // E = Ub + Wb R^T
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const float4 w4 = image_at(Wimg + img, w, n, lane);
      ea[n][0] = bits(w4.x); ea[n][1] = bits(w4.y); ea[n][2] = bits(w4.z); ea[n][3] = bits(w4.w);
      const float2 u0 = *reinterpret_cast<const float2 *>(Ub + img + r0 * kDim + 8 * n + 2 * t);
      const float2 u1 = *reinterpret_cast<const float2 *>(Ub + img + r1 * kDim + 8 * n + 2 * t);
      e[n][0] = u0.x; e[n][1] = u0.y; e[n][2] = u1.x; e[n][3] = u1.y;
    }
    wait<1>();
    meet();             // R and Dl are there
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        const float2 r2 = *reinterpret_cast<const float2 *>(Rs + r_off(8 * n + g, 8 * j + 2 * t));
        mma_acc_a(e[n], ea[j], bits(r2.x), bits(r2.y));
      }
    wait<0>();
    meet();             // R has been read by both groups; raw blocks and S0^T are there
#pragma unroll
    for (int n = 0; n < 8; ++n) {
#pragma unroll
      for (int x = 0; x < 4; ++x) ea[n][x] = bits(rnd(-e[n][x]));
      reinterpret_cast<uint4 *>(Es)[(w * 8 + n) * 32 + lane] = make_uint4(ea[n][0], ea[n][1], ea[n][2], ea[n][3]);
      *reinterpret_cast<uint32_t *>(sm + oEg + raw_off(r0, n) + 4 * t) = pack16<T>(e[n][0], e[n][1]);
      *reinterpret_cast<uint32_t *>(sm + oEg + raw_off(r1, n) + 4 * t) = pack16<T>(e[n][2], e[n][3]);
    }
    meet();             // (-E) image complete
    rows_out<T>(dv + base, sm + oEg, w, nvalid, lane);
    uint32_t ga[4][4];      // dO, own rows
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) raw_a(ga[kk], aG, 16 * w, kk, lane);
    float cq[8][4];         // d_query = dO S0 ..
    zero(cq);
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        const float4 s4 = image_at(Ss, np, j, lane);
        mma_raw_a<T>(cq[2 * np], ga[j >> 1], j & 1, bits(s4.x), bits(s4.y));
        mma_raw_a<T>(cq[2 * np + 1], ga[j >> 1], j & 1, bits(s4.z), bits(s4.w));
      }
#pragma unroll 1
    for (int ip = 0; ip <= w; ++ip) {      // .. + strict_lower(dO Dl^T) K;  d_key: strict_lower(-E Dl^T) K; 16 steps at a time
      const int s0 = 16 * ip;
      float x[2][4] = {}, y[2][4] = {};
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const float2 d2 = *reinterpret_cast<const float2 *>(Ds + (s0 + 8 * n + g) * kLdD + 8 * j + 2 * t);
          const uint32_t b0 = op(d2.x), b1 = op(d2.y);
          mma_raw_a<T>(x[n], ga[j >> 1], j & 1, b0, b1);
          mma_acc_a(y[n], ea[j], b0, b1);
        }
      uint32_t xa[2][4], ya[2][4];
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const bool in = s0 + 8 * n + 2 * t + (i & 1) < (i < 2 ? r0 : r1);
          xa[n][i] = in ? op(x[n][i]) : 0u;
          ya[n][i] = in ? op(y[n][i]) : 0u;
        }
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        uint32_t r[4];
        raw_bt(r, aK, s0, 16 * np, lane);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            const uint32_t b0 = lo16<T>(r[2 * n + s]), b1 = hi16<T>(r[2 * n + s]);
            mma_acc_a(cq[2 * np + n], xa[s], b0, b1);
            mma_acc_a(ck[2 * np + n], ya[s], b0, b1);
          }
      }
    }
    meet();             // S0^T, Q and K have been read
    store_rows<false>(Ss, ck, w, lane);
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      *reinterpret_cast<uint32_t *>(sm + oQg + raw_off(r0, n) + 4 * t) = pack16<T>(cq[n][0], cq[n][1]);
      *reinterpret_cast<uint32_t *>(sm + oQg + raw_off(r1, n) + 4 * t) = pack16<T>(cq[n][2], cq[n][3]);
    }
    meet();             // group 0's part of d_key is there
  } else {
    wait<1>();
    meet();
    uint32_t da[8][4];      // Dl, own rows
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float2 x = *reinterpret_cast<const float2 *>(Ds + r0 * kLdD + 8 * j + 2 * t);
      const float2 y = *reinterpret_cast<const float2 *>(Ds + r1 * kLdD + 8 * j + 2 * t);
      da[j][0] = op(x.x); da[j][1] = op(x.y); da[j][2] = op(y.x); da[j][3] = op(y.y);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)      // Dl R
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        mma_acc_a(ck[n], da[j], bits(Rs[r_off(8 * j + 2 * t, 8 * n + g)]), bits(Rs[r_off(8 * j + 2 * t + 1, 8 * n + g)]));
      }
    wait<0>();
    meet();
    meet();             // (-E) image complete
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float4 e4 = image_at(Es, w, j, lane);
      ea[j][0] = bits(e4.x); ea[j][1] = bits(e4.y); ea[j][2] = bits(e4.z); ea[j][3] = bits(e4.w);
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)      // -E S0
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        const float4 s4 = image_at(Ss, np, j, lane);
        mma_acc_a(ck[2 * np], ea[j], bits(s4.x), bits(s4.y));
        mma_acc_a(ck[2 * np + 1], ea[j], bits(s4.z), bits(s4.w));
      }
#pragma unroll 1
    for (int ip = w; ip < 4; ++ip) {      // strict_upper(Dl dO^T) Q and strict_upper(-Dl E^T) K
      const int s0 = 16 * ip;
      float x[2][4] = {}, y[2][4] = {};
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        uint32_t r[4];
        raw_b(r, aG, s0, kk, lane);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int s = 0; s < 2; ++s)
            mma_acc_a(x[n], da[2 * kk + s], lo16<T>(r[2 * n + s]), hi16<T>(r[2 * n + s]));
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 e4 = image_at(Es, ip, j, lane);
        mma_acc_a(y[0], da[j], bits(e4.x), bits(e4.y));
        mma_acc_a(y[1], da[j], bits(e4.z), bits(e4.w));
      }
      uint32_t xa[2][4], ya[2][4];
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const bool in = s0 + 8 * n + 2 * t + (i & 1) > (i < 2 ? r0 : r1);
          xa[n][i] = in ? op(x[n][i]) : 0u;
          ya[n][i] = in ? op(y[n][i]) : 0u;
        }
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        uint32_t r[4], x2[4];
        raw_bt(r, aQ, s0, 16 * np, lane);
        raw_bt(x2, aK, s0, 16 * np, lane);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            mma_acc_a(ck[2 * np + n], xa[s], lo16<T>(r[2 * n + s]), hi16<T>(r[2 * n + s]));
            mma_acc_a(ck[2 * np + n], ya[s], lo16<T>(x2[2 * n + s]), hi16<T>(x2[2 * n + s]));
          }
      }
    }
    meet();
    meet();
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const float4 c4 = image_at(Ss, w, n, lane);
      *reinterpret_cast<uint32_t *>(sm + oKg + raw_off(r0, n) + 4 * t) = pack16<T>(ck[n][0] + c4.x, ck[n][1] + c4.y);
      *reinterpret_cast<uint32_t *>(sm + oKg + raw_off(r1, n) + 4 * t) = pack16<T>(ck[n][2] + c4.z, ck[n][3] + c4.w);
    }
  }
  __syncwarp();
  // this warp's own rows of Q (group 0: d_query) or K (group 1: d_key), now results
  rows_out<T>((group ? dk : dq) + base, sm + (group ? oKg : oQg), w, nvalid, lane);
}

template <typename T>
int backward_typed(const void *go, const void *gs, const void *q, const void *k, const void *delta, const void *final_state, void *dq,
                   void *dk, void *dv, void *ds, int64_t B, int64_t T_, void *scratch, cudaStream_t st) {
  const int64_t nc = ceil_div64(T_, kC), n = B * nc;
  if (n >= (1ll << 31)) {
    set_error("chunked delta rule: %lld chunks exceed a grid", (long long)n);
    return T2FW_ERR_UNSUPPORTED;
  }
  float *W = static_cast<float *>(scratch), *U = W + n * kImg, *Qb = U + n * kImg, *NR = Qb + n * kImg, *GS = NR + n * kImg;
  auto *const prep = &dfw_prep_bwd_kernel<T>;
  T2FW_ALLOW_SMEM(prep, kSmemPrep);
  T2FW_CHECK_CUDA(launch_dependent(prep, dim3((unsigned)n), dim3(kThreads), kSmemPrep, st, (const T *)go, (const T *)q, (const T *)k,
                                   (const float *)delta, W, U, Qb, NR, GS, T_, (int)nc));
  int *status = nullptr;
  int rc = lfw_chunk_status_ptr(&status);
  if (rc != T2FW_OK) return rc;
  int n_sm = 0;
  rc = lfw_chunk_sm_count(&n_sm);
  if (rc != T2FW_OK) return rc;
  const CarryPlan plan = carry_plan(B, n_sm);
  rc = plan == kSpread1   ? launch_carry_bwd<T, 1, 2, 9>(gs, final_state, Qb, NR, GS, ds, B, (int)nc, status, st)
       : plan == kSpread2 ? launch_carry_bwd<T, 2, 2, 6>(gs, final_state, Qb, NR, GS, ds, B, (int)nc, status, st)
                          : launch_carry_bwd<T, 4, 1, 4>(gs, final_state, Qb, NR, GS, ds, B, (int)nc, status, st);
  if (rc != T2FW_OK) return rc;
  auto *const grad = &dfw_grad_kernel<T>;
  T2FW_ALLOW_SMEM(grad, kSmemGrad);
  T2FW_CHECK_CUDA(launch_dependent(grad, dim3((unsigned)n), dim3(kThreadsG), kSmemGrad, st, (const T *)go, (const T *)q, (const T *)k,
                                   (const float *)delta, (const float *)W, (const float *)U, (const float *)NR, (const float *)GS, (T *)dq,
                                   (T *)dk, (T *)dv, T_, (int)nc));
  T2FW_CHECK_LAUNCH(3);
  return T2FW_OK;
}

}  // namespace

int dfw_chunk_backward(const void *go, const void *gs, const void *q, const void *k, const void *delta, const void *final_state,
                       void *dq, void *dk, void *dv, void *ds, int64_t B, int64_t T_, int dtype, void *scratch, cudaStream_t st) {
  if (dtype == T2FW_F16) return backward_typed<__half>(go, gs, q, k, delta, final_state, dq, dk, dv, ds, B, T_, scratch, st);
  return backward_typed<__nv_bfloat16>(go, gs, q, k, delta, final_state, dq, dk, dv, ds, B, T_, scratch, st);
}

}  // namespace t2fw
