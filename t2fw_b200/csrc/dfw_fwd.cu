// Delta rule, chunked forward (D = M = 64, 16-bit storage, chunks of 64 steps).  Replaces
// t2fw/csrc/dfw_kernel.cu:105-196 for these shapes.
//
// With L = strict_lower(K K^T), T = (I + L)^-1, W = T K, U = T V of a chunk and S its start state:
//     Dl = U - W S^T        O = Q S^T + strict_lower(Q K^T) Dl
//     S_next = S + Dl^T K = S + S Qc + N      with  Qc = -W^T K,  N = U^T K
// Qc and N do not depend on the state, so what is sequential over the chunks is ONE 64 x 64 x 64 product per chunk;
// everything else is parallel over (row, chunk).  The identity part of the transition stays exact in fp32
// accumulators, as if Dl^T K were added to the state.
//
//   dfw_prep_fwd_kernel   (row, chunk)   T; W, U^T, Qc^T, N as fragment images (16 KB each)
//   dfw_carry_fwd_kernel  row            the chain over the chunks; the start state of every chunk as an image
//   dfw_out_fwd_kernel    (row, chunk)   Dl and the outputs
// All three work on fragment images (dfw_frag.cuh): operands go from accumulators to operands without passing
// through tiles, 16-bit operands are used as they lie in memory (products of Q, K and V among themselves are
// exact), everything else is TF32 with fp32 accumulation, W and U from T split in two (22 bits).
//
// Why mma.sync: with operands in fragment order a warp needs no barrier, no tile conversion and no round trip
// through tensor memory between products, and small CTAs overlap one another's latencies; the tcgen05 form of this
// path converted every operand to tiles and walked the whole chunk sequentially per row, 7.2 k cycles each on at
// most one SM per row.  What bounds it now is latency at few warps, no pipe: with
// cold caches (B*H = 96, T = 1024, fp16) prep 39 us, tensor pipe 52 %, issue slots 39 %, 14 warps per SM that wait for
// fixed latencies, the tensor pipe and barriers; carry 20 us, 4 warps on each of 96 SMs, tensor 29 %, waiting for its own
// chain; out 33 us, tensor 32 %, DRAM 42 %, waiting for the images.  Whole forward 108 -> 91 us;
// 48 rows of 1333 steps, bf16, the whole call 110 -> 61 us.
#include "dfw_frag.cuh"

namespace t2fw {

using namespace frag;

namespace {

// ---- prep: grid = B * nc, four warps -----------------------------------------------------------------
constexpr int oK = 0, oV = kRaw, oT = 2 * kRaw, oL = oT + kC * kLdT * 4, kSmemPrep = oL + kC * kLdL * 4;

template <typename T>
__global__ void __launch_bounds__(kThreads, 4)
dfw_prep_fwd_kernel(const T *__restrict__ k, const T *__restrict__ v, float *__restrict__ Wimg, float *__restrict__ UTimg,
                    float *__restrict__ Qimg, float *__restrict__ Nimg, int64_t T_, int nc) {
  extern __shared__ __align__(128) unsigned char sm[];
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  float *Ts = reinterpret_cast<float *>(sm + oT), *Ls = reinterpret_cast<float *>(sm + oL);
  const uint32_t aK = smem_u32(sm + oK), aV = smem_u32(sm + oV);
  const int64_t b = blockIdx.x / (uint32_t)nc, t0 = (int64_t)(blockIdx.x - (uint32_t)b * nc) * kC;
  const int nvalid = (int)(T_ - t0 < kC ? T_ - t0 : kC);
  const size_t base = ((size_t)b * T_ + t0) * kDim, img = (size_t)blockIdx.x * kImg;
  dependency_wait();
  load_raw(sm + oK, k + base, nvalid, tid);
  load_raw(sm + oV, v + base, nvalid, tid);
  commit();
  wait<0>();
  __syncthreads();
  gram_lower<T>(Ls, aK, aK, w, lane);
  __syncwarp();
  unit_lower_inverse<kLdT>(Ls, Ts, w, lane);
  __syncthreads();

  {   // W = T K, rows 16 w ..: to memory and, rounded, over L for the product below
    float c[8][4];
    zero(c);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      if (kk > w) break;
      uint32_t ah[2][4], al[2][4];
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const float2 u = *reinterpret_cast<const float2 *>(Ts + (16 * w + g) * kLdT + 16 * kk + 8 * s + 2 * t);
        const float2 x = *reinterpret_cast<const float2 *>(Ts + (16 * w + g + 8) * kLdT + 16 * kk + 8 * s + 2 * t);
        split(u.x, ah[s][0], al[s][0]);
        split(u.y, ah[s][1], al[s][1]);
        split(x.x, ah[s][2], al[s][2]);
        split(x.y, ah[s][3], al[s][3]);
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
            mma_acc_a(c[2 * np + n], ah[s], b0, b1);
            mma_acc_a(c[2 * np + n], al[s], b0, b1);
          }
      }
    }
    store_rows<true>(Wimg + img, c, w, lane);
    float *Ws = Ls;      // L is no longer needed by anyone
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      *reinterpret_cast<float2 *>(Ws + (16 * w + g) * kLdL + 8 * n + 2 * t) = make_float2(rnd(c[n][0]), rnd(c[n][1]));
      *reinterpret_cast<float2 *>(Ws + (16 * w + g + 8) * kLdL + 8 * n + 2 * t) = make_float2(rnd(c[n][2]), rnd(c[n][3]));
    }
  }
  {   // U^T = V^T T^T, rows d = 16 w ..; then N = U^T K
    float c[8][4];
    zero(c);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      uint32_t a[4];
      raw_at(a, aV, 16 * w, 16 * kk, lane);
#pragma unroll
      for (int n = 2 * kk; n < 8; ++n)
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const float2 u = *reinterpret_cast<const float2 *>(Ts + (8 * n + g) * kLdT + 16 * kk + 8 * s + 2 * t);
          uint32_t h0, l0, h1, l1;
          split(u.x, h0, l0);
          split(u.y, h1, l1);
          mma_raw_a<T>(c[n], a, s, h0, h1);
          mma_raw_a<T>(c[n], a, s, l0, l1);
        }
    }
    store_rows<false>(UTimg + img, c, w, lane);
    float d[8][4];
    zero(d);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      uint32_t a[2][4];
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int e = 0; e < 4; ++e) a[s][e] = bits(rnd(c[2 * kk + s][e]));
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        uint32_t r[4];
        raw_bt(r, aK, 16 * kk, 16 * np, lane);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
          for (int s = 0; s < 2; ++s) mma_acc_a(d[2 * np + n], a[s], lo16<T>(r[2 * n + s]), hi16<T>(r[2 * n + s]));
      }
    }
    store_rows<false>(Nimg + img, d, w, lane);
  }
  __syncthreads();
  mma_kt_b<T, false, true>(Qimg + img, aK, Ls, -1.f, w, lane);      // Qc^T = -K^T W
}

// ---- carry: the 16-row blocks of a state never meet, so a row's four may be spread over 4 / kW CTAs; kH warps per block, each
// 1 / kH of the columns ----
// Qc^T and the CTA's part of N of a chunk arrive together by bulk copies.  Start states replace N: a chunk's N is in shared
// memory before its start state is written.  A step is a chain: operands, exchange of the halves (kH = 2), products (a warp's 64 take
// about 1 k cycles, hence the halves where SMs are free), next operands.
template <typename T, int kW, int kH, int kStages>
__global__ void __launch_bounds__(32 * kH * kW)
dfw_carry_fwd_kernel(const T *__restrict__ state, const float *__restrict__ Qimg, float *__restrict__ NSimg,
                     T *__restrict__ final_state, int nc, int *__restrict__ status) {
  extern __shared__ __align__(128) unsigned char sm[];
  __shared__ __align__(8) uint64_t full[kStages];
  __shared__ uint4 xs[kH == 2 ? 2 : 1][kH == 2 ? kW : 1][kH == 2 ? 8 : 1][kH == 2 ? 32 : 1];      // operands of the block's rows, by step parity
  constexpr int kN = 8 / kH;                                            // 8-column tiles of a warp
  constexpr int kPart = kW * kImg / 4, kStage = kImg + kPart;      // floats
  float *ring = reinterpret_cast<float *>(sm);
  const int tid = threadIdx.x, wl = tid / (32 * kH), ch = kH == 1 ? 0 : (tid >> 5) & 1, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int64_t b = blockIdx.x / (4 / kW);
  const int w0 = (int)(blockIdx.x % (4 / kW)) * kW, w = w0 + wl;
  const size_t img0 = (size_t)b * nc * kImg;
  init_ring<kStages>(full, tid);
  dependency_wait();
  auto fetch = [&](int c) {      // one thread
    if (c >= nc) return;
    float *dst = ring + (c % kStages) * kStage;
    acp::mbar_expect_tx(&full[c % kStages], (uint32_t)(kStage * sizeof(float)));
    acp::bulk_g2s(dst, Qimg + img0 + (size_t)c * kImg, kImg * (uint32_t)sizeof(float), &full[c % kStages]);
    acp::bulk_g2s(dst + kImg, NSimg + img0 + (size_t)c * kImg + w0 * (kImg / 4), kPart * (uint32_t)sizeof(float), &full[c % kStages]);
  };
  if (tid == 0) {
    for (int c = 0; c < kStages - 1; ++c) fetch(c);
  }
  float S[kN][4];
  const T *sp = state + ((size_t)b * kDim + 16 * w + g) * kDim + 32 * ch + 2 * t;
#pragma unroll
  for (int n = 0; n < kN; ++n) {
    const uint32_t u = *reinterpret_cast<const uint32_t *>(sp + 8 * n), x = *reinterpret_cast<const uint32_t *>(sp + 8 * kDim + 8 * n);
    S[n][0] = __uint_as_float(lo16<T>(u)); S[n][1] = __uint_as_float(hi16<T>(u));
    S[n][2] = __uint_as_float(lo16<T>(x)); S[n][3] = __uint_as_float(hi16<T>(x));
  }
  spread_start<kH>(S, reinterpret_cast<float *>(&xs[0][0][0][0]), wl, ch, lane);
  int fail = acp::mbar_wait(&full[0], 0) ? 0 : 1;
  float4 bq[8][4 / kH];
  carry_load_b<kH>(bq, ring, ch, lane);
  int c = 0;
  for (; c < nc; ++c) {
    uint32_t own[kN][4], oth[4][4];
#pragma unroll
    for (int n = 0; n < kN; ++n) {
#pragma unroll
      for (int e = 0; e < 4; ++e) own[n][e] = op(S[n][e]);
      if (kH == 2) xs[c & 1][wl][4 * ch + n][lane] = make_uint4(own[n][0], own[n][1], own[n][2], own[n][3]);
    }
    const int cn = c + 1 < nc ? c + 1 : c;      // (the last chunk's matrix once more: nobody uses it)
    if (!acp::mbar_wait(&full[cn % kStages], (uint32_t)(cn / kStages) & 1u)) fail = 1;
    if (__syncthreads_or(fail)) break;      // the halves are exchanged; the buffer refilled next is no longer read
    if (tid == 0) fetch(c + kStages - 1);
    const float *buf = ring + (c % kStages) * kStage;
    float4 *const img = reinterpret_cast<float4 *>(NSimg + img0 + (size_t)c * kImg) + (w * 8 + 4 * ch) * 32 + lane;
    const float z0 = S[0][0] * 0.f, z1 = S[0][2] * 0.f;
#pragma unroll
    for (int n = 0; n < kN; ++n) {
      if (kH == 2) {
        const uint4 u = xs[c & 1][wl][4 * (ch ^ 1) + (n & 3)][lane];
        oth[n & 3][0] = u.x; oth[n & 3][1] = u.y; oth[n & 3][2] = u.z; oth[n & 3][3] = u.w;
      }
      img[n * 32] = with_rows(own[n], z0, z1);
      const float4 nx = image_at(buf + kImg, wl, 4 * ch + n, lane);
      S[n][0] += nx.x; S[n][1] += nx.y; S[n][2] += nx.z; S[n][3] += nx.w;
    }
    carry_product<kH>(S, own, oth, bq, ring + (cn % kStages) * kStage, ch, lane);
  }
  if (fail) atomicExch(status, 1);
  if (c < nc && tid == 0) drain_ring<kStages>(full, c, nc);
  T *fp = final_state + ((size_t)b * kDim + 16 * w + g) * kDim + 32 * ch + 2 * t;
#pragma unroll
  for (int n = 0; n < kN; ++n) {
    *reinterpret_cast<uint32_t *>(fp + 8 * n) = pack16<T>(S[n][0], S[n][1]);
    *reinterpret_cast<uint32_t *>(fp + 8 * kDim + 8 * n) = pack16<T>(S[n][2], S[n][3]);
  }
}

template <typename T, int kW, int kH, int kStages>
int launch_carry_fwd(const void *state, const float *Qc, float *NS, void *final_state, int64_t B, int nc, int *status, cudaStream_t st) {
  constexpr int kSmem = kStages * (kImg + kW * kImg / 4) * 4;
  static_assert(kSmem + kCarryStatic<kW, kH, kStages> <= kSharedLimit, "shared memory limit");
  auto *const carry = &dfw_carry_fwd_kernel<T, kW, kH, kStages>;
  T2FW_ALLOW_SMEM(carry, kSmem);
  T2FW_CHECK_CUDA(launch_dependent(carry, dim3((unsigned)(B * (4 / kW))), dim3(32 * kH * kW), kSmem, st, (const T *)state, Qc, NS,
                                   (T *)final_state, nc, status));
  return T2FW_OK;
}

// ---- outputs: grid = B * nc, four warps ------------------------------------------------------------------
constexpr int oQo = 0, oKo = kRaw, oSo = 2 * kRaw, oWo = oSo + kImg * 4, kSmemOut = oWo + kImg * 4;      // W, then Dl^T

template <typename T>
__global__ void __launch_bounds__(kThreads, 4)
dfw_out_fwd_kernel(const T *__restrict__ q, const T *__restrict__ k, const float *__restrict__ Wimg,
                   const float *__restrict__ UTimg, const float *__restrict__ Simg, T *__restrict__ out,
                   float *__restrict__ delta, int64_t T_, int nc) {
  extern __shared__ __align__(128) unsigned char sm[];
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  float *Ss = reinterpret_cast<float *>(sm + oSo), *Ws = reinterpret_cast<float *>(sm + oWo);
  const uint32_t aQ = smem_u32(sm + oQo), aK = smem_u32(sm + oKo);
  const int64_t b = blockIdx.x / (uint32_t)nc, t0 = (int64_t)(blockIdx.x - (uint32_t)b * nc) * kC;
  const int nvalid = (int)(T_ - t0 < kC ? T_ - t0 : kC);
  const size_t base = ((size_t)b * T_ + t0) * kDim, img = (size_t)blockIdx.x * kImg;
  dependency_wait();
  load_image(Ws, Wimg + img, tid);
  load_image(Ss, Simg + img, tid);
  commit();
  load_raw(sm + oQo, q + base, nvalid, tid);
  load_raw(sm + oKo, k + base, nvalid, tid);
  commit();
  float4 u[8];
#pragma unroll
  for (int n = 0; n < 8; ++n) u[n] = image_at(UTimg + img, w, n, lane);
  wait<1>();
  __syncthreads();

  float c[8][4];
  {   // Dl^T = U^T - S W^T, rows d = 16 w .., columns t
    uint32_t a[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float4 s4 = image_at(Ss, w, j, lane);
      a[j][0] = bits(s4.x) ^ 0x80000000u; a[j][1] = bits(s4.y) ^ 0x80000000u;
      a[j][2] = bits(s4.z) ^ 0x80000000u; a[j][3] = bits(s4.w) ^ 0x80000000u;
    }
#pragma unroll
    for (int n = 0; n < 8; ++n) { c[n][0] = u[n].x; c[n][1] = u[n].y; c[n][2] = u[n].z; c[n][3] = u[n].w; }
    mma_image(c, a, Ws, lane);
    float *dp = delta + base + 16 * w + g;      // eight lanes = 32 contiguous bytes of a step
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int s = 8 * n + 2 * t;
      if (s < nvalid) {
        dp[(size_t)s * kDim] = c[n][0];
        dp[(size_t)s * kDim + 8] = c[n][2];
      }
      if (s + 1 < nvalid) {
        dp[(size_t)(s + 1) * kDim] = c[n][1];
        dp[(size_t)(s + 1) * kDim + 8] = c[n][3];
      }
    }
  }
  wait<0>();
  __syncthreads();             // every warp has read W; Q and K are there
#pragma unroll
  for (int n = 0; n < 8; ++n)
    reinterpret_cast<float4 *>(Ws)[(w * 8 + n) * 32 + lane] =
        make_float4(rnd(c[n][0]), rnd(c[n][1]), rnd(c[n][2]), rnd(c[n][3]));
  __syncthreads();

  uint32_t qa[4][4];
#pragma unroll
  for (int kk = 0; kk < 4; ++kk) raw_a(qa[kk], aQ, 16 * w, kk, lane);
  zero(c);
#pragma unroll
  for (int j = 0; j < 8; ++j)      // Q S^T, rows t = 16 w .., columns d
#pragma unroll
    for (int np = 0; np < 4; ++np) {
      const float4 s4 = image_at(Ss, np, j, lane);
      mma_raw_a<T>(c[2 * np], qa[j >> 1], j & 1, bits(s4.x), bits(s4.y));
      mma_raw_a<T>(c[2 * np + 1], qa[j >> 1], j & 1, bits(s4.z), bits(s4.w));
    }
#pragma unroll
  for (int ip = 0; ip < 4; ++ip) {      // + strict_lower(Q K^T) Dl, 16 steps i at a time
    if (ip > w) break;
    float p[2][4] = {};
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      uint32_t r[4];
      raw_b(r, aK, 16 * ip, kk, lane);
      mma_16<T>(p[0], qa[kk], r[0], r[1]);
      mma_16<T>(p[1], qa[kk], r[2], r[3]);
    }
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      uint32_t a[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int col = 16 * ip + 8 * s + 2 * t + (e & 1), row = 16 * w + g + 8 * (e >> 1);
        a[e] = col < row ? op(p[s][e]) : 0u;
      }
#pragma unroll
      for (int np = 0; np < 4; ++np) {
        const float4 d4 = image_at(Ws, np, 2 * ip + s, lane);
        mma_acc_a(c[2 * np], a, bits(d4.x), bits(d4.y));
        mma_acc_a(c[2 * np + 1], a, bits(d4.z), bits(d4.w));
      }
    }
  }
  // through this warp's own rows of Q (read by nobody else), then out in whole rows
  __syncwarp();
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    *reinterpret_cast<uint32_t *>(sm + oQo + raw_off(16 * w + g, n) + 4 * t) = pack16<T>(c[n][0], c[n][1]);
    *reinterpret_cast<uint32_t *>(sm + oQo + raw_off(16 * w + g + 8, n) + 4 * t) = pack16<T>(c[n][2], c[n][3]);
  }
  __syncwarp();
  rows_out<T>(out + base, sm + oQo, w, nvalid, lane);
}

template <typename T>
int forward_typed(const void *q, const void *k, const void *v, const void *state, void *out, void *final_state, void *delta,
                  int64_t B, int64_t T_, void *scratch, cudaStream_t st) {
  const int64_t nc = ceil_div64(T_, kC), n = B * nc;
  if (n >= (1ll << 31)) {
    set_error("chunked delta rule: %lld chunks exceed a grid", (long long)n);
    return T2FW_ERR_UNSUPPORTED;
  }
  float *W = static_cast<float *>(scratch), *U = W + n * kImg, *Qc = U + n * kImg, *NS = Qc + n * kImg;
  auto *const prep = &dfw_prep_fwd_kernel<T>;
  T2FW_ALLOW_SMEM(prep, kSmemPrep);
  T2FW_CHECK_CUDA(launch_dependent(prep, dim3((unsigned)n), dim3(kThreads), kSmemPrep, st, (const T *)k, (const T *)v, W, U, Qc, NS, T_, (int)nc));
  int *status = nullptr;
  int rc = lfw_chunk_status_ptr(&status);
  if (rc != T2FW_OK) return rc;
  int n_sm = 0;
  rc = lfw_chunk_sm_count(&n_sm);
  if (rc != T2FW_OK) return rc;
  const CarryPlan plan = carry_plan(B, n_sm);
  rc = plan == kSpread1   ? launch_carry_fwd<T, 1, 2, 10>(state, Qc, NS, final_state, B, (int)nc, status, st)
       : plan == kSpread2 ? launch_carry_fwd<T, 2, 2, 8>(state, Qc, NS, final_state, B, (int)nc, status, st)
       : plan == kDeep    ? launch_carry_fwd<T, 4, 1, 7>(state, Qc, NS, final_state, B, (int)nc, status, st)
                          : launch_carry_fwd<T, 4, 1, 3>(state, Qc, NS, final_state, B, (int)nc, status, st);
  if (rc != T2FW_OK) return rc;
  auto *const outk = &dfw_out_fwd_kernel<T>;
  T2FW_ALLOW_SMEM(outk, kSmemOut);
  T2FW_CHECK_CUDA(launch_dependent(outk, dim3((unsigned)n), dim3(kThreads), kSmemOut, st, (const T *)q, (const T *)k, (const float *)W,
                                   (const float *)U, (const float *)NS, (T *)out, (float *)delta, T_, (int)nc));
  T2FW_CHECK_LAUNCH(3);
  return T2FW_OK;
}

}  // namespace

bool dfw_chunk_supported(int64_t D, int64_t M, int dtype) {
  return D == kDim && M == kDim && (dtype == T2FW_F16 || dtype == T2FW_BF16);
}

// fp32 images per chunk: W, U^T, Qc^T, N (then the start state); backward: Wb, Ub, Qb^T, Nb (then R_end), (Dl^T K)^T
// (then S0^T)
size_t dfw_chunk_scratch_bytes(int64_t B, int64_t T_, bool backward) {
  return align_up((size_t)B * ceil_div64(T_, kC) * (backward ? 5 : 4) * kImg * sizeof(float), 256);
}

int dfw_chunk_forward(const void *q, const void *k, const void *v, const void *state, void *out, void *final_state, void *delta,
                      int64_t B, int64_t T_, int dtype, void *scratch, cudaStream_t st) {
  if (dtype == T2FW_F16) return forward_typed<__half>(q, k, v, state, out, final_state, delta, B, T_, scratch, st);
  return forward_typed<__nv_bfloat16>(q, k, v, state, out, final_state, delta, B, T_, scratch, st);
}

}  // namespace t2fw
