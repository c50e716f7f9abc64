// Outputs of the chunked decay-rule forward for states of up to 128 x 128 (D, K = 64 or 128, one of them 128; 16-bit storage,
// chunks of 64 steps): the third phase, as lfw_c64_fwd.cu is for 64 x 64 states (notation there).
//
// As a grid of 64 x 64 blocks every block would scale its windows' operands again, and blocks that share a window would form
// the same in-chunk decays and sum their outputs through memory.  Here a chunk is one problem:
//     P   = tril( (q pm_g) (k / pm_g)^T )      [t][s]       over all K features
//     O1  = (G_REF .* S0) (q pm_g)^T           [d][t]       all d features in the 128 lanes of tensor memory
//     O2  = (x / pm_a)^T P^T                   [d][t]
//     o_t = pm_a[t] .* (A_REF O1 + O2)_t
// Thread (feature, 16-step quarter) walks the k-side and the d-side gates of the feature with its number, as in the 64 x 64
// kernel; a side with 64 features leaves the upper half of the threads without work there.
//
// 16 rows x 16384 steps, 128 x 128 (4096 chunks): 433 us as a grid of blocks -> 180 us.
#include "lfw_c64.cuh"
#include "seq_layout.cuh"

namespace t2fw {

using namespace c64;

int lfw_chunk_status_ptr(int **out);   // lfw_c64_local.cu
int lfw_chunk_sm_count(int *out);

namespace {

constexpr int kThreadsW = 512;
constexpr int kWide = 128;                         // features of a side, the upper half possibly unused
constexpr int kS0LdW = 272;                        // row stride (bytes) of the start-state landing zone
// shared-memory map (bytes from the 1024-byte aligned base)
constexpr int oTw = 0;                             // [q, k][window] tiles [step][feature]; P over the first k tile
constexpr int oS0w = oTw + 4 * kTile;              // start state, [128][kS0LdW] 16-bit
constexpr int oQtw = oS0w + kWide * kS0LdW;        // [k, d][4][128] products of the quarters
constexpr int oRawW = oQtw + 2 * 4 * kWide * 4;    // [x, f, q, k, fk][window]
constexpr int kSmemW = oRawW + 10 * kRawBytes + 1024;
static_assert(oRawW % 128 == 0 && oS0w % 16 == 0, "copy destination alignment");
static_assert(kSmemW + 256 <= 227 * 1024, "shared memory limit");

// tensor-memory columns
constexpr int cS2w = 0, cXw = 128, cPw = 192, cO1w = 256, cO2w = 320;
constexpr int kTmemColsW = 512;
constexpr uint32_t kIdesc128 = umma::make_idesc_tf32(128, 64, false, false);

template <typename T>
__global__ void __launch_bounds__(kThreadsW, 1)
lfw_wide_fwd_kernel(const __grid_constant__ seq::Maps mp, const T *__restrict__ state, const T *__restrict__ ckpt,
                    T *__restrict__ out, int *__restrict__ rowflag, int *__restrict__ status, int64_t T_, int64_t nc,
                    int64_t total, int D, int K) {
  extern __shared__ __align__(1024) unsigned char sm_raw[];
  unsigned char *sm = sm_raw + ((1024u - (umma::smem_u32(sm_raw) & 1023u)) & 1023u);
  __shared__ __align__(8) uint64_t barG, barV, barP, barO;
  __shared__ uint32_t tmem_slot;
  __shared__ int s_fail, s_bad2[2];

  const int tid = threadIdx.x, warp = uniform_warp_idx(), lane = tid & 31;
  const int q4 = warp & 3, tq = warp >> 2, t0 = 16 * tq;
  const int feat = 32 * q4 + lane, win = feat >> 6, wf = feat & 63;      // own feature on both sides: window, number in it
  const int nd = D >> 6, nk = K >> 6;
  const bool has_k = feat < K, has_d = feat < D;
  float *qtot = reinterpret_cast<float *>(sm + oQtw);

  // tensors: 0 x, 1 f, 2 q, 3 k, 4 fk.  Gate blocks and value blocks on barriers of their own, as in the 64 x 64 kernel.
  auto issue_raw = [&](const ItemWalk &w, bool gates) {     // thread 0 only
    uint64_t *bar = gates ? &barG : &barV;
    const int row = (int)(w.row * T_ + w.c * kC);
    acp::mbar_expect_tx(bar, (uint32_t)(gates ? nd + nk : nd + 2 * nk) * kRawBytes);
#pragma unroll 1
    for (int i = 0; i < 5; ++i) {
      if ((i == 1 || i == 4) != gates) continue;
      for (int j = 0; j < (i < 2 ? nd : nk); ++j) seq::load_block(sm + oRawW + (2 * i + j) * kRawBytes, &mp.m[i], 64 * j, row, bar);
    }
  };
  auto issue_state = [&](const ItemWalk &w) {   // every thread: 16-byte pieces, in whole rows
    const T *s0p = (w.c == 0) ? state + (size_t)w.row * D * K : ckpt + ((size_t)w.row * nc + w.c - 1) * D * K;
    const int pieces = K >> 3;
    for (int i = tid; i < D * pieces; i += kThreadsW) {
      const int r = nk == 2 ? i >> 4 : i >> 3, p = i & (pieces - 1);
      cp_async16(sm + oS0w + r * kS0LdW + p * 16, s0p + (size_t)i * 8);
    }
    cp_async_commit();
  };

  if (tid == 0) {
    umma::mbar_init(&barG, 1);
    umma::mbar_init(&barV, 1);
    umma::mbar_init(&barP, 1);
    umma::mbar_init(&barO, 2);       // O1, O2
    umma::mbar_fence_init();
    s_fail = 0;
    s_bad2[0] = s_bad2[1] = 0;
  }
  if (warp == 0) umma::tmem_alloc(&tmem_slot, kTmemColsW);
  sync_all();
  dependency_wait();
  const uint32_t tb = __shfl_sync(0xffffffffu, tmem_slot, 0);
  const uint32_t tl = umma::tmem_addr(tb, 32 * q4, 0);
  ItemWalk wn(blockIdx.x, gridDim.x, nc, 1);
  uint32_t n_issued[2] = {0u, 0u}, n_landed[2] = {0u, 0u};      // thread 0: rounds of gates and of values
  if (wn.unit < total) {
    if (tid == 0) {
      issue_raw(wn, true);
      issue_raw(wn, false);
      n_issued[0] = n_issued[1] = 1u;
    }
    issue_state(wn);
  }
  const uint32_t aT = umma::smem_u32(sm + oTw);
  unsigned char *const tq_col = sm + oTw + win * kTile + (wf >> 5) * kColBlock + ((wf & 3) << 2) + t0 * 128;
  const int tswz = ((wf >> 2) & 7) << 4;
  // P tile: row 16 q4 + lane (the lower half warps hold it), columns t0 ..
  const int p_row = 16 * q4 + (lane & 15);
  unsigned char *const prow = sm + oTw + 2 * kTile + (t0 >> 5) * kColBlock + p_row * 128;
  const int psw = (((t0 >> 2) & 7) ^ (p_row & 7)) << 4;
  const T *raw = reinterpret_cast<const T *>(sm + oRawW + win * kRawBytes) + t0 * kDim + wf;
  auto rawv = [&](int blk, int j) { return Elem<T>::ld(raw + 2 * blk * kC * kDim + j * kDim); };

  uint32_t it = 0;
  for (; wn.unit < total; ++it) {
    const ItemWalk w = wn;
    wn.step();
    const int64_t left = T_ - (int64_t)w.c * kC;
    const int nvalid = (int)(left < kC ? left : kC);
    const bool partial = nvalid < kC;      // steps beyond the valid ones become identity steps
    int &s_bad = s_bad2[it & 1];

    cp_async_wait_all();       // this thread's share of the start state (requested one chunk ahead)
    if (acp::mbar_wait(&barG, it & 1u)) ++n_landed[0];
    else s_fail = 1;

    // ---- gates of the own feature and quarter on both sides, products of the quarters ----
    float gk[16], gd[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      gk[j] = has_k && t0 + j < nvalid ? rawv(4, j) : 1.f;
      gd[j] = has_d && t0 + j < nvalid ? rawv(1, j) : 1.f;
    }
    float mn = kRangeHi;
#pragma unroll
    for (int j = 0; j < 16; ++j) mn = min3_abs(mn, gk[j], gd[j]);
    if (!(mn >= kTinyState)) {      // rare: some gate needs the clamp
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        gk[j] = sanitize_gate(gk[j]);
        gd[j] = sanitize_gate(gd[j]);
      }
    }
    float pk = gk[0], pd = gd[0];
#pragma unroll
    for (int j = 1; j < 16; ++j) { pk *= gk[j]; pd *= gd[j]; }
    qtot[tq * kWide + feat] = pk;
    qtot[(4 + tq) * kWide + feat] = pd;
    __syncthreads();           // also: the start state has landed
    if (s_fail) break;
    if (tid == 0 && wn.unit < total) {
      issue_raw(wn, true);
      ++n_issued[0];
    }
    if (acp::mbar_wait(&barV, it & 1u)) ++n_landed[1];
    else s_fail = 1;

    // ---- operands ----
    float lo = kRangeHi, hi = 0.f;
    if (has_k) {   // (uniform in a warp) k side: q pm_g and k / pm_g as [step][feature] tiles
      float s = tq == 0 ? qtot[kWide + feat] : tq == 3 ? qtot[2 * kWide + feat] : 1.f;
      float mw[16], vw[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        mw[j] = rawv(2, j);
        vw[j] = rawv(3, j);
      }
      if (partial) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          mw[j] = t0 + j < nvalid ? mw[j] : 0.f;
          vw[j] = t0 + j < nvalid ? vw[j] : 0.f;
        }
      }
      lo = hi = fabsf(s);
      if (tq < 2) {
#pragma unroll
        for (int j = 15; j >= 0; --j) {
          const float e = mw[j];
          mw[j] = bias_tf32(e * rcp_fast(s));
          vw[j] = bias_tf32(vw[j] * s);
          s *= gk[j];
          lo = fminf(lo, fabsf(s));
          hi = max3_abs(hi, s, e);      // the query's values too
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          s *= gk[j];
          lo = fminf(lo, fabsf(s));
          hi = max3_abs(hi, s, mw[j]);
          mw[j] = bias_tf32(mw[j] * s);
          vw[j] = bias_tf32(vw[j] * rcp_fast(s));
        }
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        unsigned char *p = tq_col + (tswz ^ ((j & 7) << 4)) + j * 128;
        *reinterpret_cast<float *>(p) = mw[j];
        *reinterpret_cast<float *>(p + 2 * kTile) = vw[j];
      }
    }
    float up;                  // A_REF of the own feature; gd[j] becomes pm_a[j]
    {   // d side: x / pm_a into tensor memory
      const float q0 = qtot[4 * kWide + feat], q1 = qtot[5 * kWide + feat];
      up = q0 * q1;
      float s = tq == 0 ? q1 : tq == 3 ? qtot[6 * kWide + feat] : 1.f;
      float vw[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) vw[j] = has_d && t0 + j < nvalid ? rawv(0, j) : 0.f;
      lo = fminf(lo, fabsf(s));
      hi = max3_abs(hi, s, s);
      if (tq < 2) {
#pragma unroll
        for (int j = 15; j >= 0; --j) {
          const float a = gd[j];
          gd[j] = rcp_fast(s);
          vw[j] = bias_tf32(vw[j] * s);
          s *= a;
          lo = fminf(lo, fabsf(s));
          hi = max3_abs(hi, s, s);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          s *= gd[j];
          lo = fminf(lo, fabsf(s));
          hi = max3_abs(hi, s, s);
          gd[j] = s;
          vw[j] = bias_tf32(vw[j] * rcp_fast(s));
        }
      }
      umma::tmem_st16(tl + cXw + t0, vw);
    }
    if (!(lo >= kRangeLo && hi <= kRangeHi)) s_bad = 1;
    for (int c = 0; c < nk; ++c) {   // state: row d = own feature, a quarter of the columns k, scaled by G_REF
      const int k0 = nk * t0 + 16 * c;
      float sv[16];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        uint4 u = make_uint4(0u, 0u, 0u, 0u);
        if (has_d) u = *reinterpret_cast<const uint4 *>(sm + oS0w + feat * kS0LdW + k0 * 2 + 16 * i);
        const T *e = reinterpret_cast<const T *>(&u);
#pragma unroll
        for (int j = 0; j < 8; ++j) sv[8 * i + j] = Elem<T>::ld(e + j);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 a = *reinterpret_cast<const float4 *>(qtot + k0 + 4 * i);
        const float4 b = *reinterpret_cast<const float4 *>(qtot + kWide + k0 + 4 * i);
        sv[4 * i] = bias_tf32(sv[4 * i] * (a.x * b.x));
        sv[4 * i + 1] = bias_tf32(sv[4 * i + 1] * (a.y * b.y));
        sv[4 * i + 2] = bias_tf32(sv[4 * i + 2] * (a.z * b.z));
        sv[4 * i + 3] = bias_tf32(sv[4 * i + 3] * (a.w * b.w));
      }
      umma::tmem_st16(tl + cS2w + k0, sv);
    }
    umma::tmem_st_wait();
    umma::fence_async_smem();
    sync_all();       // operands complete, raw blocks and start state consumed

    if (warp == 0) {      // P, on its own barrier
      const uint64_t dq = desc_sw128(aT), dk = desc_sw128(aT + 2 * kTile);
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) umma::mma_tf32(tb + cPw, dq + kstep(ks), dk + kstep(ks), kIdesc64, ks > 0);
        if (nk == 2) {
          const uint64_t dq1 = desc_sw128(aT + kTile), dk1 = desc_sw128(aT + 3 * kTile);
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) umma::mma_tf32(tb + cPw, dq1 + kstep(ks), dk1 + kstep(ks), kIdesc64, true);
        }
        umma::mma_commit(&barP);
      }
      __syncwarp();
    } else if (warp == 2) {      // O1
      const uint64_t dq = desc_sw128(aT);
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) mma_tf32_ts(tb + cO1w, tb + cS2w + 8 * ks, dq + kstep(ks), kIdesc128, ks > 0);
        if (nk == 2) {
          const uint64_t dq1 = desc_sw128(aT + kTile);
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) mma_tf32_ts(tb + cO1w, tb + cS2w + 64 + 8 * ks, dq1 + kstep(ks), kIdesc128, true);
        }
        umma::mma_commit(&barO);
      }
      __syncwarp();
    }
    if (wn.unit < total) {
      if (tid == 0) {
        issue_raw(wn, false);
        ++n_issued[1];
      }
      issue_state(wn);
    }
    if (tid == 0) {
      if (s_bad) atomicExch(rowflag + w.row, 1);      // the scan kernel redoes this row
      s_bad2[(it & 1) ^ 1] = 0;
    }

    // ---- P: mask, round, store as the [t][s] operand (over k / pm_g, which only the P product reads) ----
    if (!umma::mbar_wait(&barP, it & 1u)) s_fail = 1;
    umma::fence_after_sync();
    {
      // a warp holds 16 x 16 values: on the diagonal it masks, below it nothing is masked, above it all is zero
      float v[16];
      if (tq <= q4) {
        umma::tmem_ld16(tl + cPw + t0, v);
        umma::tmem_ld_wait();
        if (tq == q4) {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = j <= lane ? bias_tf32(v[j]) : 0.f;
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = bias_tf32(v[j]);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = 0.f;
      }
      if (lane < 16) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          *reinterpret_cast<float4 *>(prow + (psw ^ (j << 4))) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
      }
    }
    umma::fence_async_smem();
    sync_all();
    if (s_fail) break;
    if (warp == 4) {      // O2
      const uint64_t dp = desc_sw128(aT + 2 * kTile);
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) mma_tf32_ts(tb + cO2w, tb + cXw + 8 * ks, dp + kstep(ks), kIdesc128, ks > 0);
        umma::mma_commit(&barO);
      }
      __syncwarp();
    }
    if (!umma::mbar_wait(&barO, it & 1u)) s_fail = 1;
    umma::fence_after_sync();
    float o1[16], o2[16];
    umma::tmem_ld16(tl + cO1w + t0, o1);
    umma::tmem_ld16(tl + cO2w + t0, o2);
    umma::tmem_ld_wait();
    if (has_d) {      // 32 features of a step are 64 contiguous bytes
      T *po = out + ((size_t)w.row * T_ + (size_t)w.c * kC + t0) * D + feat;
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (!partial || t0 + j < nvalid) po[(size_t)j * D] = (T)(gd[j] * fmaf(up, o1[j], o2[j]));
    }
    __syncwarp();
    // No barrier here: what the next chunk writes before its first barrier (products of the quarters) nobody still
    // reads, and its tiles and tensor-memory operands are written after that barrier.
    umma::fence_before_sync();
  }
  cp_async_wait_all();
  __syncthreads();      // s_fail of the last chunk is visible
  if (tid == 0 && s_fail) {
    atomicExch(status, 1);
    // bounded: let copies that are still in flight land before the CTA leaves
    if (n_issued[0] > n_landed[0]) acp::mbar_wait(&barG, n_landed[0] & 1u);
    if (n_issued[1] > n_landed[1]) acp::mbar_wait(&barV, n_landed[1] & 1u);
  }
  sync_all();
  if (warp == 0) umma::tmem_dealloc(tb, kTmemColsW);
}

}  // namespace

// mp: tensor maps of x, f, q, k, fk (dense [items * T][D or K] arrays); state / ckpt [items][.][D][K]; rowflag per item
int lfw_wide_forward_out(const seq::Maps &mp, const void *state, const void *ckpt, void *out, int *rowflag, int64_t items,
                         int64_t T_, int64_t D, int64_t K, int dtype, cudaStream_t st) {
  int *status = nullptr;
  int rc = lfw_chunk_status_ptr(&status);
  if (rc != T2FW_OK) return rc;
  int n_sm = 0;
  rc = lfw_chunk_sm_count(&n_sm);
  if (rc != T2FW_OK) return rc;
  const int64_t nc = ceil_div64(T_, kC), total = items * nc;
  const unsigned grid = (unsigned)(total < n_sm ? total : n_sm);
#define T2FW_LAUNCH(TT)                                                                                          \
  do {                                                                                                           \
    auto *const kern1 = &lfw_wide_fwd_kernel<TT>;                                                                \
    T2FW_ALLOW_SMEM(kern1, kSmemW);                                                                              \
    T2FW_CHECK_CUDA(launch_dependent(lfw_wide_fwd_kernel<TT>, dim3(grid), dim3(kThreadsW), kSmemW, st, mp,       \
                                     (const TT *)state, (const TT *)ckpt, (TT *)out, rowflag, status, T_, nc,    \
                                     total, (int)D, (int)K));                                                    \
  } while (0)
  if (dtype == T2FW_F16) T2FW_LAUNCH(__half); else T2FW_LAUNCH(__nv_bfloat16);
#undef T2FW_LAUNCH
  T2FW_CHECK_LAUNCH(1);
  return T2FW_OK;
}

}  // namespace t2fw
