// Sequence gradients of the chunked decay-rule backward on the tcgen05 tensor core (D = K = 64,
// 16-bit storage, chunks of 64 steps): d_x, d_f, d_q, d_k, d_f_key of one chunk from its inputs,
// the state at the chunk start (checkpoint) and the state gradient at the chunk end (carried over
// the chunks by the carry kernel).  Replaces the reference's reverse scan, its
// materialised state gradients, five einsums and two in-place multiplies
// (t2fw/csrc/lfw_kernel.cu:61-102, t2fw/csrc/lfw.cpp:84-93).
//
// The k side (d_q, d_k, d_f_key) and the d side (d_x, d_f) are mirror images: "own" is the side whose
// gradients are formed, "other" the side that is contracted away.  For own = k, other = d (notation of
// lfw_c64.cuh; S0 = start state, R = end state gradient, both viewed [own][other]):
//     Z    = tril( (dO pm_a) (x / pm_a)^T )            [t][s], in-chunk decays of the other side
//     TQ1  = (A_REF .* S0) (dO pm_a)^T                 [k][t]   to be scaled by G_REF
//     TQ2  = (k / pm_g) Z^T                            [k][t]
//     T2   = (q pm_g) Z                                [k][s]
//     T7   = (A_63/A_REF .* R) (x / pm_a)^T            [k][s]   to be scaled by G_63/G_REF
//     d_q  = pm_g .* (G_REF TQ1 + TQ2)     d_k = (T2 + G_63/G_REF T7) ./ pm_g
//     g_t d_g_t = sum_{s>=t} [(q pm_g) .* (G_REF TQ1 + TQ2) - (k / pm_g) .* T2]_s
//                 + sum_{i<t} [(k / pm_g) .* G_63/G_REF T7]_i + G_63 .* sum_d A_63 S0 R   (d_f_key = that / g_t)
// The suffix sum cancels the pair terms (i, s >= t) of its two parts; both parts come from the same
// TF32-rounded Z and operands, so the cancellation is exact up to fp32 accumulation.  Where a gate
// is below 2^-13 even that is not enough (the result is divided by the gate), and the pair terms
// i < t <= s are summed directly for that (t, feature).
// The state blocks carry the anchor products of the OTHER side, so the mid-anchored tiles serve both
// the in-chunk and the state products, and the own side's anchor products scale the results: no operand
// is scaled by two 32-step products, and four tiles are built instead of eight.
//
// Both sides run at the same time.  An M = 64 accumulator takes 16 lanes of every 32-lane quarter of
// tensor memory, so the k side's results fill one lane set (lanes 0-15 of the quarters) and the d side's
// the other: a thread's lane decides its side, a thread (side, feature, 16-step quarter of the chunk) forms
// the ratios and the scaled operands of its own feature from one walk over its steps, puts them into
// tensor memory (A operand of its own side, row = feature) and into the [step][feature] tile (B operand of
// the other side), and later reads its own results back: one feature over 16 consecutive steps, so the
// sums over time are register-local plus one exchange between the four threads of a feature.  The d side's
// rows are rotated by 16 features against the k side's so that the two half warps touch different banks.
//
// What bounds it: the latency of its phases at one CTA of 16 warps per SM.  Issue slots are 45 % busy (25.5 k warp
// instructions per chunk; 53 k in the version that ran the two sides one after the other), the tensor pipe 18 %, DRAM 18 %; a
// warp waits for barriers, fixed latencies, shared memory and instructions about equally.  B*H = 96, T = 1024 (1536 chunks):
// 151 -> 99 us per launch with cold caches.
//
// One persistent CTA of 16 warps per SM; six raw 8 KB input blocks per chunk by bulk asynchronous copy (the
// next chunk's are requested once this chunk's operands are built); operand tiles in shared memory (TF32,
// 128-byte swizzle), accumulators in tensor memory.  Every wait is bounded.
#include "lfw_c64.cuh"
#include "seq_layout.cuh"

namespace t2fw {

using namespace c64;

int lfw_chunk_status_ptr(int **out);   // lfw_c64_local.cu
int lfw_chunk_sm_count(int *out);


namespace {

constexpr int kThreadsB = 512;
constexpr int kFixCap = 128;           // tiny-gate entries per chunk
constexpr int kFixRows = 16;           // features with tiny gates per chunk whose operand rows are kept
constexpr int kS0Ld = 144;             // row stride (bytes) of the start-state landing zone (64 x 16-bit + pad)
constexpr int kRLd = 272;              // row stride (bytes) of the end-gradient landing zone (64 x fp32 + pad)
// shared-memory map (bytes from the 1024-byte aligned base); side 0 = k, 1 = d
constexpr int oT = 0;                               // [side][2] tiles [step][feature]: Mm (q pm | dO pm), Vm (k / pm | x / pm)
constexpr int oZ = oT + 4 * kTile;                  // [own side][2] tiles: Z [t][s], Z^T [s][t]
constexpr int oS0L = oZ + 4 * kTile;                // start state of the chunk, [64][kS0Ld]
constexpr int oRL = oS0L + kDim * kS0Ld;            // end state gradient of the chunk, [64][kRLd]
constexpr int oQt = oRL + kDim * kRLd;              // quarter products [side][4][64]
constexpr int oPrd = oQt + 2 * 4 * kDim * 4;        // [side][2][64]: product up to the anchor, after the anchor
constexpr int oXc = oPrd + 2 * 2 * kDim * 4;        // partial sums [3][4 quarters][side][64]
constexpr int oBnd = oXc + 3 * 4 * 2 * kDim * 4;    // boundary-term partials [side][4][64]
constexpr int oFixCode = oBnd + 2 * 4 * kDim * 4;   // [kFixCap] int: step << 8 | side << 6 | feature
constexpr int oFixVal = oFixCode + kFixCap * 4;     // [kFixCap] float
constexpr int oFixMask = oFixVal + kFixCap * 4;     // [side][64] one bit per step
constexpr int oFixSlot = oFixMask + 2 * kDim * 8;   // [side][64] int: row slot of a feature, -1 = none
constexpr int oFixRow = oFixSlot + 2 * kDim * 4;    // [kFixRows][2][64] floats: operand rows Mw, Vw
constexpr int oRaw = oFixRow + kFixRows * 2 * kDim * 4;   // x, f (fused layer: gate pre-activations), q, k, fk, dO
constexpr int kSmemB = oRaw + 6 * kRawBytes + 1024; // + slack for the 1024-byte alignment
static_assert(oRaw % 128 == 0 && oFixMask % 8 == 0 && oS0L % 16 == 0 && oRL % 16 == 0, "alignment");
static_assert(kSmemB + 256 <= 227 * 1024, "shared memory limit");

// tensor-memory columns, both lane sets: four A operands, then the accumulators.  T2 takes Z's columns over
// once Z has been read out.
constexpr int cS2 = 0, cR2 = 64, cVw = 128, cMw = 192;
constexpr int cZ = 256, cT2 = 256, cTQ1 = 320, cTQ2 = 384, cT7 = 448;
constexpr int kTmemCols = 512;

// kMode: 0 the plain operator, 1 the fused layer, 2 a grid of blocks (gradients summed over the blocks of the other axis)
template <typename T, int kMode>
__global__ void __launch_bounds__(kThreadsB, 1)
lfw_c64_bwd_kernel(const __grid_constant__ seq::Maps mp, const T *__restrict__ state, const T *__restrict__ ckpt,
                   const float *__restrict__ Rend, const seq::Out<T> dx, const seq::Out<T> df, const seq::Out<T> dq,
                   const seq::Out<T> dk, const seq::Out<T> dfk, int *__restrict__ rowflag, int *__restrict__ status,
                   int64_t T_, int64_t nc, int64_t total) {
  constexpr bool kFused = kMode == 1, kGrid = kMode == 2;
  extern __shared__ __align__(1024) unsigned char sm_raw[];
  unsigned char *sm = sm_raw + ((1024u - (umma::smem_u32(sm_raw) & 1023u)) & 1023u);
  __shared__ __align__(8) uint64_t barRaw, barG, barZ, barM1, barM2;
  __shared__ uint32_t tmem_slot;
  __shared__ int s_fail, s_bad2[2], fix_n2[2], fix_rows_n;

  const int tid = threadIdx.x, warp = uniform_warp_idx(), lane = tid & 31;
  // lane quarter of tensor memory, 16-step quarter of the chunk, side (0 k, 1 d), row in the quarter
  const int q4 = warp & 3, tq = warp >> 2, h = lane >> 4, fl = lane & 15;
  const int feat = 16 * ((q4 + h) & 3) + fl;          // own feature (tensor-memory row 16 q4 + fl of lane set h)
  const int t0 = 16 * tq;                             // first own step; also the first own column of the state blocks

  float *qtot = reinterpret_cast<float *>(sm + oQt);
  float *prd = reinterpret_cast<float *>(sm + oPrd);
  float *xc = reinterpret_cast<float *>(sm + oXc);
  float *bndp = reinterpret_cast<float *>(sm + oBnd);
  int *fix_code = reinterpret_cast<int *>(sm + oFixCode);
  float *fix_val = reinterpret_cast<float *>(sm + oFixVal);
  unsigned long long *fix_mask = reinterpret_cast<unsigned long long *>(sm + oFixMask);
  int *fix_slot = reinterpret_cast<int *>(sm + oFixSlot);
  float *fix_rows = reinterpret_cast<float *>(sm + oFixRow);
  T *raw = reinterpret_cast<T *>(sm + oRaw);     // [6][64][64]: x, f, q, k, fk, dO

  // tensors: 0 x, 1 f, 2 q, 3 k, 4 fk, 5 dO
  const bool unit_forget = kFused && (mp.flags & seq::kUnitForget) != 0;
  const bool sigmoid_gate = kFused && (mp.flags & seq::kSigmoidGate) != 0;
  const float q_scale = kFused ? mp.q_scale : 1.f;
  auto issue_raw = [&](const ItemWalk &w) {     // thread 0 only: one copy per tensor
    int b, hc;
    w.item(mp.heads, &b, &hc);
    const int row = (int)(b * T_ + w.c * kC);
    const int nv = (int)((T_ - (int64_t)w.c * kC < kC) ? T_ - (int64_t)w.c * kC : kC);
    const uint32_t per = (mp.flags & seq::kContiguous) ? (uint32_t)nv * kDim * sizeof(T) : (uint32_t)kRawBytes;
    acp::mbar_expect_tx(&barRaw, (unit_forget ? 5u : 6u) * per);
#pragma unroll
    for (int i = 0; i < 6; ++i)
      if (!(i == 1 && unit_forget)) seq::fetch_block<T>(mp, i, sm + oRaw + i * kRawBytes, row, hc, nv, &barRaw);
  };
  // fused layer: the gate pre-activations once more, into the block that the constant forget gate leaves free.
  // The epilogue reads them, after the raw blocks have been handed to the next chunk.
  auto issue_preact = [&](const ItemWalk &w) {
    int b, hc;
    w.item(mp.heads, &b, &hc);
    const int nv = (int)((T_ - (int64_t)w.c * kC < kC) ? T_ - (int64_t)w.c * kC : kC);
    acp::mbar_expect_tx(&barG, (mp.flags & seq::kContiguous) ? (uint32_t)nv * kDim * sizeof(T) : (uint32_t)kRawBytes);
    seq::fetch_block<T>(mp, 4, sm + oRaw + kRawBytes, (int)(b * T_ + w.c * kC), hc, nv, &barG);
  };
  // start state (16-bit, 8 KB) and end state gradient (fp32, 16 KB) of a chunk into the padded
  // landing zones: three 16-byte asynchronous copies per thread
  auto issue_state = [&](const ItemWalk &w) {   // every thread
    const T *s0p = (w.c == 0) ? state + seq::state_off(mp, w.row, w.sub, 0, 1) : ckpt + seq::state_off(mp, w.row, w.sub, w.c - 1, nc);
    const float *rp = Rend + ((size_t)w.bh() * nc + w.c) * kDim * kDim;
    cp_async16(sm + oS0L + (tid >> 3) * kS0Ld + (tid & 7) * 16, s0p + (size_t)(tid >> 3) * mp.state_ld + (tid & 7) * 8);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c16 = tid + i * kThreadsB;
      cp_async16(sm + oRL + (c16 >> 4) * kRLd + (c16 & 15) * 16, rp + (c16 >> 4) * kDim + (c16 & 15) * 4);
    }
    cp_async_commit();
  };

  if (tid == 0) {
    umma::mbar_init(&barRaw, 1);
    umma::mbar_init(&barG, 1);
    umma::mbar_init(&barZ, 2);       // one commit per side
    umma::mbar_init(&barM1, 4);      // TQ1 and T7 of both sides
    umma::mbar_init(&barM2, 4);      // TQ2 and T2 of both sides
    umma::mbar_fence_init();
    s_fail = 0;
    s_bad2[0] = s_bad2[1] = fix_n2[0] = fix_n2[1] = fix_rows_n = 0;
  }
  if (tid < 2 * kDim) fix_mask[tid] = 0ull;
  for (int i = tid; i < 4 * kTile / 16; i += kThreadsB)      // the blocks above the diagonal of Z are never written again
    *reinterpret_cast<float4 *>(sm + oZ + 16 * i) = make_float4(0.f, 0.f, 0.f, 0.f);
  if (warp == 0) umma::tmem_alloc(&tmem_slot, kTmemCols);
  sync_all();
  dependency_wait();
  const uint32_t tb = __shfl_sync(0xffffffffu, tmem_slot, 0);
  const uint32_t tl = umma::tmem_addr(tb, 32 * q4, 0);
  bool raw_pending = false, pre_pending = false;      // thread 0
  ItemWalk wi(blockIdx.x, gridDim.x, nc, kGrid ? mp.nsub : 1), wn = wi;           // this chunk and the next one
  if (wi.unit < total) {
    if (tid == 0) {
      issue_raw(wi);
      raw_pending = true;
    }
    issue_state(wi);
  }
  const uint32_t aT = umma::smem_u32(sm);
  // tile column offset of the own feature: row r of the swizzled tile adds r * 128 and XORs r % 8 into bits 4-6
  const int tcol = (feat >> 5) * kColBlock + ((feat & 3) << 2), tswz = ((feat >> 2) & 7) << 4;
  // Z tiles of the own side: row 16 q4 + fl, columns t0 .. (16-byte pieces XOR-ed with the row); and column
  // 16 q4 + fl of the transposed tile, rows t0 .., the second half warp four rows on
  const int zt_row = 16 * q4 + fl;
  unsigned char *const zrow = sm + oZ + h * 2 * kTile + (t0 >> 5) * kColBlock + zt_row * 128;
  const int zsw = (((t0 >> 2) & 7) ^ (zt_row & 7)) << 4;
  unsigned char *const zt_lo = sm + oZ + (h * 2 + 1) * kTile + (zt_row >> 5) * kColBlock + t0 * 128 + ((zt_row & 3) << 2) + 512 * h;
  unsigned char *const zt_hi = zt_lo - 1024 * h;
  const int ztsw = (((zt_row >> 2) & 7) ^ (4 * h)) << 4;
  const T *gcol = raw + (h ? 1 : 4) * kC * kDim + t0 * kDim + feat;
  const T *mcol = raw + (h ? 5 : 2) * kC * kDim + t0 * kDim + feat;
  const T *vcol = raw + (h ? 0 : 3) * kC * kDim + t0 * kDim + feat;

  uint32_t it = 0;
  for (; wn.unit < total; ++it) {
    wi = wn;
    wn.step();
    const int64_t t0c = (int64_t)wi.c * kC;
    const int nvalid = (int)((T_ - t0c < kC) ? T_ - t0c : kC);
    // first row and column windows of the chunk in the output arrays
    int ob, oh;
    wi.item(mp.heads, &ob, &oh);
    const int64_t row0 = (int64_t)ob * T_ + t0c;
    // grid: block (i, j) holds d-side window i and k-side window j; `add`: not the first block of the sum over the other axis
    const int gi = kGrid ? oh / mp.nk : 0, gj = kGrid ? oh - gi * mp.nk : 0;
    const int hcol = (kGrid ? (h ? gi : gj) : oh) * kDim;
    const bool add = kGrid && (h ? gj : gi) != 0;
    int &fix_n = fix_n2[it & 1], &s_bad = s_bad2[it & 1];

    if (!acp::mbar_wait(&barRaw, it & 1u)) s_fail = 1;
    if (tid == 0) raw_pending = false;

    // ---- gates of the own feature and quarter, product of the quarter ----
    float g[16];
    float g_min = kRangeHi;
#pragma unroll
    for (int j = 0; j < 16; ++j) g[j] = Elem<T>::ld(gcol + j * kDim);
    if (kFused) {
      if (sigmoid_gate && h == 0) {
#pragma unroll
        for (int j = 0; j < 16; ++j) g[j] = seq::sigmoid_gate<T>(g[j]);
      }
      if (unit_forget && h == 1) {
#pragma unroll
        for (int j = 0; j < 16; ++j) g[j] = 1.f;
      }
    }
    if (nvalid < kC) {      // partial chunk: identity steps beyond the valid ones
#pragma unroll
      for (int j = 0; j < 16; ++j) g[j] = t0 + j < nvalid ? g[j] : 1.f;
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) g_min = fminf(g_min, fabsf(g[j]));
    if (!(g_min >= kTinyState)) {      // rare (also NaN): some gate needs the clamp
#pragma unroll
      for (int j = 0; j < 16; ++j) g[j] = sanitize_gate(g[j]);
    }
    {
      float p0 = g[0], p1 = g[1];      // two chains
#pragma unroll
      for (int j = 2; j < 16; j += 2) { p0 *= g[j]; p1 *= g[j + 1]; }
      qtot[(h * 4 + tq) * kDim + feat] = p0 * p1;
    }
    umma::named_barrier(1 + q4, 128);      // the four warps that hold the quarters of the same features
    float pm[16], up, after, pm_prev;      // ratios to the anchor; products up to and after it; ratio of the step before
    {
      const float *qt = qtot + h * 4 * kDim + feat;
      const float q0 = qt[0], q1 = qt[kDim], q2 = qt[2 * kDim], q3 = qt[3 * kDim];
      up = q0 * q1;
      after = q2 * q3;
      pm_prev = tq == 0 ? rcp_fast(up) : tq == 1 ? rcp_fast(q1) : tq == 2 ? 1.f : q2;
      if (tq == 1) {
        prd[(h * 2) * kDim + feat] = up;
        prd[(h * 2 + 1) * kDim + feat] = after;
      }
      const float carry = tq == 0 ? q1 : tq == 3 ? q2 : 1.f;
      float mw[16], vw[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        mw[j] = Elem<T>::ld(mcol + j * kDim);
        vw[j] = Elem<T>::ld(vcol + j * kDim);
      }
      if (kFused && q_scale != 1.f && h == 0) {
#pragma unroll
        for (int j = 0; j < 16; ++j) mw[j] = seq::round_to<T>(mw[j] * q_scale);
      }
      if (nvalid < kC) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          mw[j] = t0 + j < nvalid ? mw[j] : 0.f;
          vw[j] = t0 + j < nvalid ? vw[j] : 0.f;
        }
      }
      // the walk away from the anchor: downwards for the first two quarters (s = 1 / pm), upwards for the others
      float s = carry, lo = fabsf(carry), hi = lo;
      if (tq < 2) {
#pragma unroll
        for (int j = 15; j >= 0; --j) {
          pm[j] = rcp_fast(s);
          mw[j] = rna_tf32(mw[j] * pm[j]);
          vw[j] = rna_tf32(vw[j] * s);
          s *= g[j];
          lo = fminf(lo, fabsf(s));
          hi = fmaxf(hi, fabsf(s));
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          s *= g[j];
          lo = fminf(lo, fabsf(s));
          hi = fmaxf(hi, fabsf(s));
          pm[j] = s;
          mw[j] = rna_tf32(mw[j] * s);
          vw[j] = rna_tf32(vw[j] * rcp_fast(s));
        }
      }
      if (!(lo >= kRangeLo && hi <= kRangeHi)) s_bad = 1;      // also NaN
      umma::tmem_st16(tl + cMw + t0, mw);
      umma::tmem_st16(tl + cVw + t0, vw);
      unsigned char *tp = sm + oT + h * 2 * kTile + tcol + t0 * 128;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        unsigned char *p = tp + (tswz ^ ((j & 7) << 4)) + j * 128;
        *reinterpret_cast<float *>(p) = mw[j];
        *reinterpret_cast<float *>(p + kTile) = vw[j];
      }
      if (g_min < kTinyGate) {      // rare: some gate of this quarter is tiny; exact pair sums for those later
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (fabsf(g[j]) < kTinyGate && t0 + j < nvalid) {
            const int slot = atomicAdd(&fix_n, 1);
            if (slot < kFixCap) {
              fix_code[slot] = ((t0 + j) << 8) | (h << 6) | feat;
              if (atomicOr(&fix_mask[h * kDim + feat], 1ull << (t0 + j)) == 0ull) {      // first entry of this feature
                const int rs = atomicAdd(&fix_rows_n, 1);
                fix_slot[h * kDim + feat] = rs < kFixRows ? rs : -1;
                if (rs >= kFixRows) s_bad = 1;
              }
            } else {
              s_bad = 1;
            }
          }
        }
      }
    }
    cp_async_wait_all();       // this thread's share of the start state and end gradient
    umma::fence_async_smem();
    sync_all();                // tiles, anchor products and state blocks of all threads
    if (s_fail) break;

    // ---- Z of both sides: each a chain of eight dependent instructions, issued by lanes of two warps so that
    //      the chains interleave in the tensor core, which executes in issue order ----
    if (warp < 2) {
      const uint32_t d = umma::tmem_addr(tb, 16 * warp, cZ);
      const uint32_t other = aT + oT + (warp ^ 1) * 2 * kTile;
      const uint64_t da = desc_sw128(other), db = desc_sw128(other + kTile);
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) umma::mma_tf32(d, da + kstep(ks), db + kstep(ks), kIdesc64, ks > 0);
        umma::mma_commit(&barZ);
      }
      __syncwarp();
    }
    if (kFused && sigmoid_gate && tid == 0) {      // every thread is past the epilogue of the chunk before
      issue_preact(wi);
      pre_pending = true;
    }
    if (fix_n > 0 && fix_mask[h * kDim + feat] != 0ull) {      // rare: the direct pair sums of this feature read its operand rows
      const int rs = fix_slot[h * kDim + feat];
      if (rs >= 0) {
        float *row = fix_rows + rs * 2 * kDim + t0;
        float a[16], b[16];
        // (a divergent tensor-memory load is not possible: the values come back from the tile)
        const unsigned char *tp = sm + oT + h * 2 * kTile + tcol + t0 * 128;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const unsigned char *p = tp + (tswz ^ ((j & 7) << 4)) + j * 128;
          a[j] = *reinterpret_cast<const float *>(p);
          b[j] = *reinterpret_cast<const float *>(p + kTile);
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          row[j] = a[j];
          row[kDim + j] = b[j];
        }
      }
    }

    // ---- state blocks as A operands: row = own feature, columns t0 .. t0 + 15 of the other side, scaled by the
    //      other side's anchor products; their elementwise product is the boundary term ----
    {
      const float *oref = prd + (h ^ 1) * 2 * kDim + t0;
      float sv[16], rv[16];
      if (h == 0) {         // S(own = k, other = d = t0 + j): a column of the stored blocks
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          sv[j] = Elem<T>::ld(reinterpret_cast<const T *>(sm + oS0L + (t0 + j) * kS0Ld) + feat);
          rv[j] = *(reinterpret_cast<const float *>(sm + oRL + (t0 + j) * kRLd) + feat);
        }
      } else {              // S(own = d, other = k = t0 + j): a row segment
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint4 u = *reinterpret_cast<const uint4 *>(sm + oS0L + feat * kS0Ld + t0 * 2 + 16 * i);
          const T *e = reinterpret_cast<const T *>(&u);
#pragma unroll
          for (int j = 0; j < 8; ++j) sv[8 * i + j] = Elem<T>::ld(e + j);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 r4 = *reinterpret_cast<const float4 *>(sm + oRL + feat * kRLd + t0 * 4 + 16 * i);
          rv[4 * i] = r4.x; rv[4 * i + 1] = r4.y; rv[4 * i + 2] = r4.z; rv[4 * i + 3] = r4.w;
        }
      }
      __syncwarp();
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 a = *reinterpret_cast<const float4 *>(oref + 4 * i), b = *reinterpret_cast<const float4 *>(oref + kDim + 4 * i);
        const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float s2 = sv[4 * i + j] * av[j], r2 = rv[4 * i + j] * bv[j];
          acc = fmaf(s2, r2, acc);
          sv[4 * i + j] = bias_tf32(s2);
          rv[4 * i + j] = bias_tf32(r2);
        }
      }
      umma::tmem_st16(tl + cS2 + t0, sv);
      umma::tmem_st16(tl + cR2 + t0, rv);
      bndp[(h * 4 + tq) * kDim + feat] = acc;
    }
    umma::tmem_st_wait();
    sync_all();       // all operands in place; raw blocks and landing zones are consumed

    if (warp >= 2 && warp < 6) {      // TQ1 (warps 2, 3) and T7 (warps 4, 5) of side warp & 1
      const int side = warp & 1, is7 = (warp - 2) >> 1;
      const uint32_t ls = umma::tmem_addr(tb, 16 * side, 0);
      const uint32_t d = ls + (is7 ? cT7 : cTQ1), a = ls + (is7 ? cR2 : cS2);
      const uint64_t db = desc_sw128(aT + oT + ((side ^ 1) * 2 + is7) * kTile);
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) mma_tf32_ts(d, a + 8 * ks, db + kstep(ks), kIdesc64, ks > 0);
        umma::mma_commit(&barM1);
      }
      __syncwarp();
    }
    if (wn.unit < total) {      // the next chunk's inputs and state blocks
      if (tid == 0) {
        issue_raw(wn);
        raw_pending = true;
      }
      issue_state(wn);
    }
    if (tid == 0) {
      if (s_bad) atomicExch(rowflag + wi.row, 1);      // the scan kernels redo this row
      s_bad2[(it & 1) ^ 1] = 0;
      fix_n2[(it & 1) ^ 1] = 0;
    }

    // ---- Z: mask, round, store as [t][s] and [s][t].  A warp holds rows 16 q4 .. + 15 and columns t0 .. t0 + 15: on
    //      the diagonal it masks, below it nothing is masked, above it the blocks stay zero ----
    if (!umma::mbar_wait(&barZ, it & 1u)) s_fail = 1;
    umma::fence_after_sync();
    if (tq <= q4) {
      float v[16];
      umma::tmem_ld16(tl + cZ + t0, v);
      umma::tmem_ld_wait();
      if (tq == q4) {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = j <= fl ? bias_tf32(v[j]) : 0.f;
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = bias_tf32(v[j]);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *reinterpret_cast<float4 *>(zrow + (zsw ^ (j << 4))) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
      // transposed: the half warps take rows four apart, which lie in different halves of the swizzle
#pragma unroll
      for (int j = 0; j < 16; ++j)
        *reinterpret_cast<float *>(((j & 4) ? zt_hi : zt_lo) + j * 128 + (ztsw ^ ((j & 7) << 4))) = h ? v[j ^ 4] : v[j];
    }
    umma::fence_async_smem();
    sync_all();
    if (s_fail) break;

    if (warp >= 2 && warp < 6) {      // TQ2 = Vw Z^T (warps 2, 3), T2 = Mw Z (warps 4, 5)
      const int side = warp & 1, is2 = (warp - 2) >> 1;
      const uint32_t ls = umma::tmem_addr(tb, 16 * side, 0);
      const uint32_t d = ls + (is2 ? cT2 : cTQ2), a = ls + (is2 ? cMw : cVw);
      const uint64_t db = desc_sw128(aT + oZ + (side * 2 + is2) * kTile);
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) mma_tf32_ts(d, a + 8 * ks, db + kstep(ks), kIdesc64, ks > 0);
        umma::mma_commit(&barM2);
      }
      __syncwarp();
    }
    // ---- tiny gates: pair terms i < t <= s summed directly (runs under the MMAs), one warp per
    //      entry, from the feature's operand rows ----
    const int n_fix = fix_n < kFixCap ? fix_n : kFixCap;
    if (n_fix > 0) {
      // the tile holds Z with the rounding increment but unmasked: the value the tensor core uses
      auto zval = [](const unsigned char *p) {
        return __uint_as_float(*reinterpret_cast<const uint32_t *>(p) & 0xffffe000u);
      };
      for (int e = warp - 8; e >= 0 && e < n_fix; e += 8) {
        const int code = fix_code[e], t = code >> 8, sf = code & 127, rs = fix_slot[sf];
        if (rs < 0) continue;      // no row slot: the batch row is flagged
        const unsigned char *zt = sm + oZ + (sf >> 6) * 2 * kTile;
        const float *row = fix_rows + rs * 2 * kDim;
        // sum_{s >= t} Mw[s] sum_{i < t} Z[s][i] Vw[i]: lanes over i, independent loads over s
        float acc = 0.f;
        for (int i = lane; i < t; i += 32) {
          const unsigned char *zcol = zt + (i >> 5) * kColBlock + ((i & 3) << 2);      // tile offset of (s, i) without the s terms
          const int ic = (i >> 2) & 7;
          float a0 = 0.f, a1 = 0.f;      // two chains: the sums are latency-bound
          int s = t;
          if ((kC - t) & 1) {
            a0 = row[s] * zval(zcol + s * 128 + ((ic ^ (s & 7)) << 4));
            ++s;
          }
#pragma unroll 4
          for (; s < kC; s += 2) {
            a0 = fmaf(row[s], zval(zcol + s * 128 + ((ic ^ (s & 7)) << 4)), a0);
            a1 = fmaf(row[s + 1], zval(zcol + (s + 1) * 128 + ((ic ^ ((s + 1) & 7)) << 4)), a1);
          }
          acc = fmaf(a0 + a1, row[kDim + i], acc);
        }
        acc = warp_sum(acc);
        if (lane == 0) fix_val[e] = acc;
      }
      __syncthreads();      // the direct sums are visible (fix_n is final since the operand stage)
    }

    // ---- epilogue: own feature, steps t0 .. t0 + 15 ----
    // state terms first, while the in-chunk products run: H = inclusive suffix of Mw TQ1 + exclusive prefix of Vw T7
    float H[16], tot_a, tot_p;
    if (!umma::mbar_wait(&barM1, it & 1u)) s_fail = 1;
    umma::fence_after_sync();
    {
      float a[16], b[16];
      umma::tmem_ld16(tl + cT7 + t0, a);
      umma::tmem_ld16(tl + cVw + t0, b);
      umma::tmem_ld_wait();
      float run = 0.f;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        H[j] = run;
        run = fmaf(a[j], b[j], run);
      }
      tot_p = run * after;
      umma::tmem_ld16(tl + cTQ1 + t0, a);
      umma::tmem_ld16(tl + cMw + t0, b);
      umma::tmem_ld_wait();
      run = 0.f;
#pragma unroll
      for (int j = 15; j >= 0; --j) {
        run = fmaf(a[j], b[j], run);
        H[j] = fmaf(H[j], after, run * up);
      }
      tot_a = run * up;
    }
    // element pointers of step t0; one row pitch further per step.  The plain operator writes
    // dense [rows][64] arrays.
    const seq::Out<T> &o_dv = h ? dx : dk, &o_gt = h ? df : dfk;
    const int64_t ld_mu = kMode ? dq.ld : kDim, ld_dv = kMode ? o_dv.ld : kDim, ld_gt = kMode ? o_gt.ld : kDim;
    T *p_mu = dq.p + (size_t)(row0 + t0) * dq.ld + dq.col + hcol + feat;
    T *p_dv = o_dv.p + (size_t)(row0 + t0) * o_dv.ld + o_dv.col + hcol + feat;
    const int n_own = nvalid - t0;      // valid own steps (may be negative)
    const bool full = n_own >= 16;

    if (!umma::mbar_wait(&barM2, it & 1u)) s_fail = 1;
    umma::fence_after_sync();
    float sb[16], run_b = 0.f;
#pragma unroll
    for (int half = 1; half >= 0; --half) {
      float tq2[8], t2[8];
      {
        float mw[8], vw[8];
        umma::tmem_ld8(tl + cTQ2 + t0 + 8 * half, tq2);
        umma::tmem_ld8(tl + cT2 + t0 + 8 * half, t2);
        umma::tmem_ld8(tl + cMw + t0 + 8 * half, mw);
        umma::tmem_ld8(tl + cVw + t0 + 8 * half, vw);
        umma::tmem_ld_wait();
#pragma unroll
        for (int j = 7; j >= 0; --j) {
          run_b += mw[j] * tq2[j] - vw[j] * t2[j];
          sb[8 * half + j] = run_b;
        }
      }
      // grid: this thread's own sums over the blocks before, as stored.  All loads of a batch before the first use or
      // store, none behind a branch of its own: each would be a round trip to L2.
      T old_mu[8] = {}, old_dv[8] = {};
      if (kGrid && add && n_own > 0) {
        const T *pm_old = h == 0 ? p_mu : p_dv;      // (the d side has no such result: any valid address)
        const int64_t ld_old = h == 0 ? ld_mu : ld_dv;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int jj = 8 * half + j < n_own ? 8 * half + j : 0;
          old_mu[j] = pm_old[jj * ld_old];
          old_dv[j] = p_dv[jj * ld_dv];
        }
      }
      float tq1[8], t7[8];
      umma::tmem_ld8(tl + cTQ1 + t0 + 8 * half, tq1);
      umma::tmem_ld8(tl + cT7 + t0 + 8 * half, t7);
      umma::tmem_ld_wait();
#pragma unroll
      for (int j = 7; j >= 0; --j) {
        const int jj = 8 * half + j;
        const float ip = rcp_fast(pm[jj]);
        const float dmu = pm[jj] * fmaf(up, tq1[j], tq2[j]), ddv = ip * fmaf(after, t7[j], t2[j]);
        pm[jj] = (jj > 0 ? pm[jj > 0 ? jj - 1 : 0] : pm_prev) * ip;      // from here on: 1 / gate of the step
        if (full || jj < n_own) {
          if (h == 0) p_mu[jj * ld_mu] = (T)(kFused ? dmu * q_scale : kGrid ? dmu + Elem<T>::ld(&old_mu[j]) : dmu);
          p_dv[jj * ld_dv] = (T)(kGrid ? ddv + Elem<T>::ld(&old_dv[j]) : ddv);
        }
      }
    }
    T *p_gt = o_gt.p == nullptr ? nullptr : o_gt.p + (size_t)(row0 + t0) * o_gt.ld + o_gt.col + hcol + feat;
    T old_gt[16] = {};
    if (kGrid && add && n_own > 0) {
#pragma unroll
      for (int j = 0; j < 16; ++j) old_gt[j] = p_gt[(j < n_own ? j : 0) * ld_gt];
    }
    {
      const int o = h * kDim + feat;
      xc[(0 * 4 + tq) * 2 * kDim + o] = tot_a;
      xc[(1 * 4 + tq) * 2 * kDim + o] = run_b;
      xc[(2 * 4 + tq) * 2 * kDim + o] = tot_p;
      umma::named_barrier(1 + q4, 128);       // the four quarters of the same features
      float base = 0.f, add_b = 0.f;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        base += bndp[(h * 4 + r) * kDim + feat];
      }
      base *= up * after;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (r > tq) {        // later steps
          base += xc[(0 * 4 + r) * 2 * kDim + o];
          add_b += xc[(1 * 4 + r) * 2 * kDim + o];
        }
        if (r < tq) base += xc[(2 * 4 + r) * 2 * kDim + o];      // earlier steps
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) sb[j] += add_b;
      if (n_fix > 0) {      // (uniform) tiny gates in this chunk: their pair terms were summed directly
        for (int e = 0; e < n_fix; ++e) {
          const int code = fix_code[e], jj = (code >> 8) - t0;
          if ((code & 127) == o && (unsigned)jj < 16u) {
            const float v = fix_val[e];
#pragma unroll
            for (int j = 0; j < 16; ++j) sb[j] = (jj == j) ? v : sb[j];
          }
        }
        __syncthreads();      // everybody has read the entries: clear them for the next chunk
        if (tid < 2 * kDim) fix_mask[tid] = 0ull;
        if (tid == 0) fix_rows_n = 0;
        __syncthreads();
      }
      if (kFused && sigmoid_gate) {
        if (!acp::mbar_wait(&barG, it & 1u)) s_fail = 1;
        if (tid == 0) pre_pending = false;
      }
      if (o_gt.p != nullptr) {
        const T *pre = raw + kC * kDim + t0 * kDim + feat;     // fused layer: pre-activations
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          float dg = (H[j] + base + sb[j]) * pm[j];
          if (kFused && sigmoid_gate && h == 0) {      // d gate / d pre-activation, from the pre-activation itself in fp32
            const float e = seq::exp_neg(Elem<T>::ld(pre + j * kDim)), sg = seq::rcp1p(e);
            dg *= sg > seq::kGateFloor ? sg * sg * e : 0.f;      // s (1 - s) = s^2 e^{-g}
          }
          if (full || j < n_own) p_gt[j * ld_gt] = (T)(kGrid ? dg + Elem<T>::ld(&old_gt[j]) : dg);
        }
      }
      __syncwarp();
    }
    umma::fence_before_sync();      // this chunk's accumulator reads are ordered before the next barrier
  }
  cp_async_wait_all();
  __syncthreads();      // s_fail of the last chunk is visible
  if (tid == 0 && s_fail) {
    atomicExch(status, 1);
    if (raw_pending) acp::mbar_wait(&barRaw, it & 1u);   // bounded: let the copies in flight land
    if (pre_pending) acp::mbar_wait(&barG, it & 1u);
  }
  sync_all();
  if (warp == 0) umma::tmem_dealloc(tb, kTmemCols);
}

}  // namespace

// mp: tensor maps of x, f, q, k, fk, dO; outs: dx, df, dq, dk, dfk (pointer, row pitch, column) - df may be null.
int lfw_c64_backward_main(const seq::Maps &mp, const void *state, const void *ckpt, const float *Rend,
                          void *const outs[5], const int64_t out_ld[5], const int out_col[5], int *rowflag,
                          int64_t BH, int64_t T_, int dtype, cudaStream_t st) {
  int *status = nullptr;
  int rc = lfw_chunk_status_ptr(&status);
  if (rc != T2FW_OK) return rc;
  int n_sm = 0;
  rc = lfw_chunk_sm_count(&n_sm);
  if (rc != T2FW_OK) return rc;
  const int64_t nc = ceil_div64(T_, kC), total = BH / mp.nsub * nc;
  const unsigned grid = (unsigned)(total < n_sm ? total : n_sm);
#define T2FW_OUT(TT, i) seq::Out<TT>{(TT *)outs[i], out_ld[i], out_col[i]}
#define T2FW_LAUNCH(TT, FF)                                                                           \
  do {                                                                                                \
    auto *const kern1 = &lfw_c64_bwd_kernel<TT, FF>; \
    T2FW_ALLOW_SMEM(kern1, kSmemB);       \
    T2FW_CHECK_CUDA(launch_dependent(lfw_c64_bwd_kernel<TT, FF>, dim3(grid), dim3(kThreadsB), kSmemB, st, mp,   \
                                     (const TT *)state, (const TT *)ckpt, Rend, T2FW_OUT(TT, 0), T2FW_OUT(TT, 1), \
                                     T2FW_OUT(TT, 2), T2FW_OUT(TT, 3), T2FW_OUT(TT, 4), rowflag, status, T_, nc,  \
                                     total));                                                         \
  } while (0)
  const bool fused = (mp.flags & (seq::kUnitForget | seq::kSigmoidGate)) != 0 || mp.q_scale != 1.f;
#define T2FW_MODES(TT)                                                                              \
  do {                                                                                              \
    if (mp.nsub > 1) T2FW_LAUNCH(TT, 2); else if (fused) T2FW_LAUNCH(TT, 1); else T2FW_LAUNCH(TT, 0); \
  } while (0)
  if (dtype == T2FW_F16) T2FW_MODES(__half); else T2FW_MODES(__nv_bfloat16);
#undef T2FW_MODES
#undef T2FW_LAUNCH
#undef T2FW_OUT
  T2FW_CHECK_LAUNCH(1);
  return T2FW_OK;
}

}  // namespace t2fw

