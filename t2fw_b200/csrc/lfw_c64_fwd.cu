// Outputs of the chunked decay-rule forward on the tcgen05 tensor core (D = K = 64, 16-bit
// storage, chunks of 64 steps): the third phase after the chunk-local states and the carry over
// chunks.  Replaces the reference's materialised states and output einsum
// (t2fw/csrc/lfw_kernel.cu:43-57, t2fw/csrc/lfw.cpp:45).
//
// Per chunk, with S0 the state at the chunk start (the caller's state or the 16-bit checkpoint the
// carry wrote; notation of lfw_c64.cuh):
//     P   = tril( (q pm_g) (k / pm_g)^T )      [t][s]  in-chunk decays, k side
//     O1  = (G_REF .* S0) (q pm_g)^T           [d][t]  to be scaled by A_REF
//     O2  = (x / pm_a)^T P^T                   [d][t]
//     o_t = pm_a[t] .* (A_REF O1 + O2)_t
// i.e. three 64 x 64 x 64 contractions.  The state carries the k side's anchor product only and the d
// side's scales the result, so the mid-anchored query tile serves P and O1 (no operand is scaled by two
// 32-step products).
//
// A CTA works on TWO chunks at a time.  An M = 64 accumulator takes 16 lanes of every 32-lane quarter of
// tensor memory; chunk 0 of the pair uses one lane set and chunk 1 the other, so a thread's lane decides its
// chunk and every operand and every result exists once.  Thread (chunk, feature, 16-step quarter) walks the
// k-side gates of its feature (operand tiles [step][feature] in shared memory), then the d-side gates
// (operand x / pm_a straight into tensor memory, row = feature), and reads the outputs of its own feature
// and steps back, so that the ratios never leave its registers.  Odd chunk lanes are rotated by 16 features
// so that the half warps touch different banks.
//
// What bounds it: the latency of its phases at one CTA of 16 warps per SM (issue slots 39 % busy, tensor pipe 14 %, DRAM
// 25 %; a warp waits for loads, instructions, fixed latencies and shared memory about equally); against the one-chunk version with ratio tables in shared memory, config B*H = 96,
// T = 1024 (1536 chunks): 12.7 k -> 8.6 k warp instructions per chunk, 57 -> 39 us per launch with cold caches.
//
// One persistent CTA of 16 warps per SM.  The raw 8 KB input blocks of the next pair are requested as soon as
// this pair's operands are built.  Every wait is bounded.
#include "lfw_c64.cuh"
#include "seq_layout.cuh"

namespace t2fw {

using namespace c64;

int lfw_chunk_status_ptr(int **out);   // lfw_c64_local.cu
int lfw_chunk_sm_count(int *out);

namespace {

constexpr int kThreadsF = 512;
constexpr int kS0Ld = 144;                         // row stride (bytes) of the start-state landing zone
// shared-memory map (bytes from the 1024-byte aligned base), everything once per chunk of the pair
constexpr int oT = 0;                              // [chunk][2] tiles [step][feature]: q pm_g, k / pm_g -> P
constexpr int oS0L = oT + 4 * kTile;               // [chunk] start state, [64][kS0Ld] 16-bit
constexpr int oQt = oS0L + 2 * kDim * kS0Ld;       // [chunk][side][4][64] products of the quarters
constexpr int oRaw = oQt + 2 * 2 * 4 * kDim * 4;   // [chunk] x, f, q, k, fk
constexpr int kSmemF = oRaw + 2 * 5 * kRawBytes + 1024;   // + slack for the 1024-byte alignment
static_assert(oRaw % 128 == 0 && oS0L % 16 == 0, "copy destination alignment");
static_assert(kSmemF + 256 <= 227 * 1024, "shared memory limit");

// tensor-memory columns, one lane set per chunk
constexpr int cS2 = 0, cX = 64, cP = 128, cO1 = 192, cO2 = 256;
constexpr int kTmemColsF = 512;

// kMode: 0 the plain operator, 1 the fused layer (forget gate 1, k-side gates from pre-activations), 2 a grid of blocks (outputs summed over the blocks of a row)
template <typename T, int kMode>
__global__ void __launch_bounds__(kThreadsF, 1)
lfw_c64_fwd_kernel(const __grid_constant__ seq::Maps mp, const T *__restrict__ state, const T *__restrict__ ckpt,
                   const seq::Out<T> out, int *__restrict__ rowflag, int *__restrict__ status, int64_t T_,
                   int64_t nc, int64_t total) {
  constexpr bool kFused = kMode == 1, kGrid = kMode == 2;
  extern __shared__ __align__(1024) unsigned char sm_raw[];
  unsigned char *sm = sm_raw + ((1024u - (umma::smem_u32(sm_raw) & 1023u)) & 1023u);   // swizzle atoms are 1024-byte aligned
  __shared__ __align__(8) uint64_t barG, barV, barP, barO;
  __shared__ uint32_t tmem_slot;
  __shared__ int s_fail, s_bad2[2][2];

  const int tid = threadIdx.x, warp = uniform_warp_idx(), lane = tid & 31;
  // lane quarter of tensor memory, 16-step quarter of the chunk, chunk of the pair, row in the quarter
  const int q4 = warp & 3, tq = warp >> 2, h = lane >> 4, fl = lane & 15;
  const int feat = 16 * ((q4 + h) & 3) + fl;       // own feature, both sides
  const int t0 = 16 * tq;
  float *qtot = reinterpret_cast<float *>(sm + oQt) + h * 2 * 4 * kDim;      // of the own chunk

  // tensors: 0 x, 1 f, 2 q, 3 k, 4 fk
  const float q_scale = kFused ? mp.q_scale : 1.f;
  auto valid_steps = [&](const ItemWalk &w) {
    if (w.unit >= total) return 0;
    const int64_t left = T_ - (int64_t)w.c * kC;
    return (int)(left < kC ? left : kC);
  };
  // Two groups with a barrier each: the gate blocks (f, fk) are free again after the products of the quarters, the value
  // blocks (x, q, k) only once the operands are built, so the next pair's gates are requested that much earlier.
  auto issue_raw = [&](const ItemWalk *w, bool gates) {     // thread 0 only: one copy per tensor and chunk
    const uint32_t n = gates ? (kFused ? 1u : 2u) : 3u;
    uint64_t *bar = gates ? &barG : &barV;
    uint32_t bytes = 0;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int nv = valid_steps(w[e]);
      if (nv > 0) bytes += n * ((mp.flags & seq::kContiguous) ? (uint32_t)nv * kDim * sizeof(T) : (uint32_t)kRawBytes);
    }
    acp::mbar_expect_tx(bar, bytes);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int nv = valid_steps(w[e]);
      if (nv <= 0) continue;
      int b, hc;
      w[e].item(mp.heads, &b, &hc);
      const int row = (int)(b * T_ + w[e].c * kC);
#pragma unroll
      for (int i = 0; i < 5; ++i)
        if ((i == 1 || i == 4) == gates && !(i == 1 && kFused))
          seq::fetch_block<T>(mp, i, sm + oRaw + (e * 5 + i) * kRawBytes, row, hc, nv, bar);
    }
  };
  // start states of the pair (the caller's state for the first chunk of a row, else the checkpoint written
  // by the carry): one 16-byte asynchronous copy per thread and chunk into the padded landing zones
  auto issue_state = [&](const ItemWalk *w) {   // every thread
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      if (w[e].unit >= total) continue;
      const T *s0p = (w[e].c == 0) ? state + seq::state_off(mp, w[e].row, w[e].sub, 0, 1)
                                   : ckpt + seq::state_off(mp, w[e].row, w[e].sub, w[e].c - 1, nc);
      cp_async16(sm + oS0L + e * kDim * kS0Ld + (tid >> 3) * kS0Ld + (tid & 7) * 16, s0p + (size_t)(tid >> 3) * mp.state_ld + (tid & 7) * 8);
    }
    cp_async_commit();
  };

  if (tid == 0) {
    umma::mbar_init(&barG, 1);
    umma::mbar_init(&barV, 1);
    umma::mbar_init(&barP, 2);       // one commit per chunk
    umma::mbar_init(&barO, 4);       // O1 and O2 of both chunks
    umma::mbar_fence_init();
    s_fail = 0;
    s_bad2[0][0] = s_bad2[0][1] = s_bad2[1][0] = s_bad2[1][1] = 0;
  }
  if (warp == 0) umma::tmem_alloc(&tmem_slot, kTmemColsF);
  sync_all();
  dependency_wait();
  const uint32_t tb = __shfl_sync(0xffffffffu, tmem_slot, 0);
  const uint32_t tl = umma::tmem_addr(tb, 32 * q4, 0);
  const int nsub = kGrid ? mp.nsub : 1;
  ItemWalk wn[2] = {ItemWalk(2 * blockIdx.x, 2 * gridDim.x, nc, nsub), ItemWalk(2 * blockIdx.x + 1, 2 * gridDim.x, nc, nsub)};
  uint32_t n_issued[2] = {0u, 0u}, n_landed[2] = {0u, 0u};      // thread 0: bulk-copy rounds of the gates and of the values
  if (2 * (int64_t)blockIdx.x < total) {
    if (tid == 0) {
      issue_raw(wn, true);
      issue_raw(wn, false);
      n_issued[0] = n_issued[1] = 1u;
    }
    issue_state(wn);
  }
  const uint32_t aT = umma::smem_u32(sm + oT);
  // tile column offset of the own feature: row r of the swizzled tile adds r * 128 and XORs r % 8 into bits 4-6
  unsigned char *const tq_col = sm + oT + h * 2 * kTile + (feat >> 5) * kColBlock + ((feat & 3) << 2) + t0 * 128;
  const int tswz = ((feat >> 2) & 7) << 4;
  // P tile: row 16 q4 + fl, columns t0 ..
  const int p_row = 16 * q4 + fl;
  unsigned char *const prow = sm + oT + (h * 2 + 1) * kTile + (t0 >> 5) * kColBlock + p_row * 128;
  const int psw = (((t0 >> 2) & 7) ^ (p_row & 7)) << 4;
  const T *raw = reinterpret_cast<const T *>(sm + oRaw + h * 5 * kRawBytes) + t0 * kDim + feat;
  auto rawv = [&](int blk, int j) { return Elem<T>::ld(raw + blk * kC * kDim + j * kDim); };

  uint32_t it = 0;
  for (; wn[0].unit < total; ++it) {
    const ItemWalk w0 = wn[0], w1 = wn[1];
    wn[0].step();
    wn[1].step();
    const int nv0 = valid_steps(w0), nv1 = valid_steps(w1);
    const int nvalid = h ? nv1 : nv0;
    const bool partial = nv0 < kC || nv1 < kC;      // steps beyond the valid ones become identity steps
    int *s_bad = s_bad2[it & 1];

    cp_async_wait_all();       // this thread's share of the start states (requested one pair ahead)
    if (acp::mbar_wait(&barG, it & 1u)) ++n_landed[0];
    else s_fail = 1;

    // ---- gates of the own feature and quarter on both sides, products of the quarters ----
    float gk[16], gd[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      gk[j] = rawv(4, j);
      if (kFused) gk[j] = seq::sigmoid_gate<T>(gk[j]);
      gd[j] = kFused ? 1.f : rawv(1, j);
    }
    if (partial) {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        gk[j] = t0 + j < nvalid ? gk[j] : 1.f;
        gd[j] = t0 + j < nvalid ? gd[j] : 1.f;
      }
    }
    float mn = kRangeHi;      // (the fused layer's gates are at least 1/8)
    if (!kFused) {
#pragma unroll
      for (int j = 0; j < 16; ++j) mn = min3_abs(mn, gk[j], gd[j]);
    }
    if (!kFused && !(mn >= kTinyState)) {      // rare: some gate needs the clamp
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        gk[j] = sanitize_gate(gk[j]);
        gd[j] = sanitize_gate(gd[j]);
      }
    }
    float pk = gk[0], pd = gd[0];
#pragma unroll
    for (int j = 1; j < 16; ++j) { pk *= gk[j]; pd *= gd[j]; }
    qtot[tq * kDim + feat] = pk;
    qtot[(4 + tq) * kDim + feat] = pd;
    __syncthreads();           // also: the start states of both chunks have landed
    if (s_fail) break;
    if (tid == 0 && wn[0].unit < total) {
      issue_raw(wn, true);
      ++n_issued[0];
    }
    if (acp::mbar_wait(&barV, it & 1u)) ++n_landed[1];
    else s_fail = 1;

    // ---- operands ----
    float lo, hi;
    {   // k side: q pm_g and k / pm_g as [step][feature] tiles
      float s = tq == 0 ? qtot[kDim + feat] : tq == 3 ? qtot[2 * kDim + feat] : 1.f;
      float mw[16], vw[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        mw[j] = rawv(2, j);
        vw[j] = rawv(3, j);
      }
      if (kFused) {
#pragma unroll
        for (int j = 0; j < 16; ++j) mw[j] = seq::round_to<T>(mw[j] * q_scale);
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
          mw[j] = bias_tf32<kFused>(e * rcp_fast(s));
          vw[j] = bias_tf32<kFused>(vw[j] * s);
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
          mw[j] = bias_tf32<kFused>(mw[j] * s);
          vw[j] = bias_tf32<kFused>(vw[j] * rcp_fast(s));
        }
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        unsigned char *p = tq_col + (tswz ^ ((j & 7) << 4)) + j * 128;
        *reinterpret_cast<float *>(p) = mw[j];
        *reinterpret_cast<float *>(p + kTile) = vw[j];
      }
    }
    float up;                  // A_REF of the own feature; gd[j] becomes pm_a[j]
    {   // d side: x / pm_a into tensor memory
      const float q0 = qtot[4 * kDim + feat], q1 = qtot[5 * kDim + feat];
      up = kFused ? 1.f : q0 * q1;
      float s = tq == 0 ? q1 : tq == 3 ? qtot[6 * kDim + feat] : 1.f;
      float vw[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) vw[j] = rawv(0, j);
      if (partial) {
#pragma unroll
        for (int j = 0; j < 16; ++j) vw[j] = t0 + j < nvalid ? vw[j] : 0.f;
      }
      if (!kFused) {
        lo = fminf(lo, fabsf(s));
        hi = max3_abs(hi, s, s);
      }
      if (kFused) {
        // gates 1: the values as they are (exact in TF32)
      } else if (tq < 2) {
#pragma unroll
        for (int j = 15; j >= 0; --j) {
          const float a = gd[j];
          gd[j] = rcp_fast(s);
          vw[j] = bias_tf32<kFused>(vw[j] * s);
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
          vw[j] = bias_tf32<kFused>(vw[j] * rcp_fast(s));
        }
      }
      umma::tmem_st16(tl + cX + t0, vw);
    }
    if (!(lo >= kRangeLo && hi <= kRangeHi)) s_bad[h] = 1;
    {   // state: row d = own feature, columns k = t0 .. t0 + 15, scaled by G_REF
      float sv[16];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const uint4 u = *reinterpret_cast<const uint4 *>(sm + oS0L + h * kDim * kS0Ld + feat * kS0Ld + t0 * 2 + 16 * i);
        const T *e = reinterpret_cast<const T *>(&u);
#pragma unroll
        for (int j = 0; j < 8; ++j) sv[8 * i + j] = Elem<T>::ld(e + j);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 a = *reinterpret_cast<const float4 *>(qtot + t0 + 4 * i);
        const float4 b = *reinterpret_cast<const float4 *>(qtot + kDim + t0 + 4 * i);
        sv[4 * i] = bias_tf32<kFused>(sv[4 * i] * (a.x * b.x));
        sv[4 * i + 1] = bias_tf32<kFused>(sv[4 * i + 1] * (a.y * b.y));
        sv[4 * i + 2] = bias_tf32<kFused>(sv[4 * i + 2] * (a.z * b.z));
        sv[4 * i + 3] = bias_tf32<kFused>(sv[4 * i + 3] * (a.w * b.w));
      }
      umma::tmem_st16(tl + cS2 + t0, sv);
    }
    umma::tmem_st_wait();
    umma::fence_async_smem();
    sync_all();       // operands complete, raw blocks and start states consumed

    // P of both chunks first and on their own barrier (warps 0, 1), then O1 (warps 2, 3): chains of eight dependent
    // instructions from several warps interleave in the tensor core
    if (warp < 4) {
      const int e = warp & 1;
      const uint32_t ls = umma::tmem_addr(tb, 16 * e, 0);
      const uint64_t dq = desc_sw128(aT + e * 2 * kTile), dk = desc_sw128(aT + (e * 2 + 1) * kTile);
      if (elect_one()) {
        if (warp < 2) {
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) umma::mma_tf32(ls + cP, dq + kstep(ks), dk + kstep(ks), kIdesc64, ks > 0);
          umma::mma_commit(&barP);
        } else {
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) mma_tf32_ts(ls + cO1, ls + cS2 + 8 * ks, dq + kstep(ks), kIdesc64, ks > 0);
          umma::mma_commit(&barO);
        }
      }
      __syncwarp();
    }
    if (wn[0].unit < total) {
      if (tid == 0) {
        issue_raw(wn, false);
        ++n_issued[1];
      }
      issue_state(wn);
    }
    if (tid == 0) {
      if (s_bad[0]) atomicExch(rowflag + w0.row, 1);      // the scan kernel redoes these rows
      if (s_bad[1] && nv1 > 0) atomicExch(rowflag + w1.row, 1);
      s_bad2[(it & 1) ^ 1][0] = s_bad2[(it & 1) ^ 1][1] = 0;
    }

    // ---- P: mask, round, store as the [t][s] operand (over k / pm_g, which only the P product reads) ----
    if (!umma::mbar_wait(&barP, it & 1u)) s_fail = 1;
    umma::fence_after_sync();
    {
      // a warp holds 16 x 16 values: on the diagonal it masks, below it nothing is masked, above it all is zero
      float v[16];
      if (tq <= q4) {
        umma::tmem_ld16(tl + cP + t0, v);
        umma::tmem_ld_wait();
        if (tq == q4) {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = j <= fl ? bias_tf32<kFused>(v[j]) : 0.f;
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = bias_tf32<kFused>(v[j]);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = 0.f;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *reinterpret_cast<float4 *>(prow + (psw ^ (j << 4))) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    }
    umma::fence_async_smem();
    sync_all();
    if (s_fail) break;
    if (warp == 4 || warp == 5) {      // O2
      const int e = warp & 1;
      const uint32_t ls = umma::tmem_addr(tb, 16 * e, 0);
      const uint64_t dp = desc_sw128(aT + (e * 2 + 1) * kTile);
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) mma_tf32_ts(ls + cO2, ls + cX + 8 * ks, dp + kstep(ks), kIdesc64, ks > 0);
        umma::mma_commit(&barO);
      }
      __syncwarp();
    }
    // first row and column window of the own chunk in the output array; 16 features of one step are 32 contiguous bytes
    int b, hcol;
    (h ? w1 : w0).item(mp.heads, &b, &hcol);
    const bool add = kGrid && hcol % mp.nk != 0;      // not the first block of its row of blocks
    hcol = (kGrid ? hcol / mp.nk : hcol) * kDim;
    T *po = out.p + ((size_t)b * T_ + (size_t)(h ? w1.c : w0.c) * kC + t0) * out.ld + out.col + hcol + feat;
    if (!umma::mbar_wait(&barO, it & 1u)) s_fail = 1;
    umma::fence_after_sync();
    float o1[16], o2[16];
    umma::tmem_ld16(tl + cO1 + t0, o1);
    umma::tmem_ld16(tl + cO2 + t0, o2);
    umma::tmem_ld_wait();
    const int64_t ld = kMode ? out.ld : kDim;
    if (kGrid && add) {      // this thread's own sum over the blocks before
      T old[16] = {};
      if (t0 < nvalid) {
#pragma unroll
        for (int j = 0; j < 16; ++j) old[j] = po[(t0 + j < nvalid ? j : 0) * ld];
      }
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (t0 + j < nvalid) po[j * ld] = (T)fmaf(gd[j], fmaf(up, o1[j], o2[j]), Elem<T>::ld(&old[j]));
    } else if (!partial) {
#pragma unroll
      for (int j = 0; j < 16; ++j) po[j * ld] = (T)(gd[j] * fmaf(up, o1[j], o2[j]));
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (t0 + j < nvalid) po[j * ld] = (T)(gd[j] * fmaf(up, o1[j], o2[j]));
    }
    __syncwarp();
    // No barrier here: what the next pair writes before its first barrier (products of the quarters) nobody still
    // reads, and its tiles and tensor-memory operands are written after that barrier.
    umma::fence_before_sync();
  }
  cp_async_wait_all();
  __syncthreads();      // s_fail of the last pair is visible
  if (tid == 0 && s_fail) {
    atomicExch(status, 1);
    // bounded: let copies that are still in flight land before the CTA leaves
    if (n_issued[0] > n_landed[0]) acp::mbar_wait(&barG, n_landed[0] & 1u);
    if (n_issued[1] > n_landed[1]) acp::mbar_wait(&barV, n_landed[1] & 1u);
  }
  sync_all();
  if (warp == 0) umma::tmem_dealloc(tb, kTmemColsF);
}

}  // namespace

// mp: tensor maps of x, f, q, k, fk; state / ckpt [BH][.][64][64]; the outputs go to out.
int lfw_c64_forward_out(const seq::Maps &mp, const void *state, const void *ckpt, void *out, int64_t out_ld,
                        int out_col, int *rowflag, int64_t BH, int64_t T_, int dtype, cudaStream_t st) {
  int *status = nullptr;
  int rc = lfw_chunk_status_ptr(&status);
  if (rc != T2FW_OK) return rc;
  int n_sm = 0;
  rc = lfw_chunk_sm_count(&n_sm);
  if (rc != T2FW_OK) return rc;
  const int64_t nc = ceil_div64(T_, kC), total = BH / mp.nsub * nc;
  const int64_t pairs = (total + 1) / 2;
  const unsigned grid = (unsigned)(pairs < n_sm ? pairs : n_sm);
#define T2FW_LAUNCH(TT, FF)                                                                              \
  do {                                                                                               \
    auto *const kern1 = &lfw_c64_fwd_kernel<TT, FF>; \
    T2FW_ALLOW_SMEM(kern1, kSmemF);      \
    T2FW_CHECK_CUDA(launch_dependent(lfw_c64_fwd_kernel<TT, FF>, dim3(grid), dim3(kThreadsF), kSmemF, st, mp,       \
                                     (const TT *)state, (const TT *)ckpt, seq::Out<TT>{(TT *)out, out_ld, out_col}, \
                                     rowflag, status, T_, nc, total));                               \
  } while (0)
  const bool fused = (mp.flags & seq::kFusedLayer) != 0;
#define T2FW_MODES(TT)                                                                              \
  do {                                                                                              \
    if (mp.nsub > 1) T2FW_LAUNCH(TT, 2); else if (fused) T2FW_LAUNCH(TT, 1); else T2FW_LAUNCH(TT, 0); \
  } while (0)
  if (dtype == T2FW_F16) T2FW_MODES(__half); else T2FW_MODES(__nv_bfloat16);
#undef T2FW_MODES
#undef T2FW_LAUNCH
  T2FW_CHECK_LAUNCH(1);
  return T2FW_OK;
}

}  // namespace t2fw
