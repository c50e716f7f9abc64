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
// One persistent CTA per SM: 16 warps that compute and four that only issue (products, the next chunk's inputs, the finished
// chunk's results).  What runs once per chunk or rarely is kept in rolled loops: a launch starts with cold instruction caches,
// and the first chunk waits for every line of the code (156 KB, unrolled throughout: 31 k cycles; a chunk afterwards 12 k).
// A computing warp reports "my part is in place" on an mbarrier and goes on; whoever needs all parts waits
// for the barrier.  With the issuing done by computing warps, those fell behind by up to 3 k cycles per chunk and the others
// waited for them at the next step.  Inputs arrive and results leave by bulk copies; the results are staged over the operand
// tiles.  (A bulk copy costs its issuing warp about 70 cycles whatever its size.)
//
// What bounds it: the phases of the computing warps (gates and operands 3.1 k cycles, state operands 2.0 k, Z 1.2 k, sums and
// results 4.5 k of 11 k per chunk), in which all warps want the same unit at the same time; products and copies run under them.
// Issue slots 58 % busy (28.2 k warp instructions per chunk, polling included), tensor pipe 21 %, DRAM 21 %; B*H = 96, T = 1024
// (1536 chunks): 99 us per launch with cold caches before the issuing warps, 79 to 81 with them.
// Whole training step, without issuing warps -> with them: 96 rows x 1024 steps 200 -> 175 to 181 us from box to box (N(0,1)
// gates, of which 0.4 per chunk are tiny: their listing and sums took 6 k cycles, now 0.5 k), fused layer 8 x 12 heads x 1024
// 258 -> 197 us.
#include "lfw_c64.cuh"
#include "seq_layout.cuh"

namespace t2fw {

using namespace c64;

int lfw_chunk_status_ptr(int **out);   // lfw_c64_local.cu
int lfw_chunk_sm_count(int *out);


namespace {

constexpr int kThreadsB = 512;         // computing threads
constexpr int kWarpsB = kThreadsB / 32;
constexpr int kThreadsAll = kThreadsB + 128;
// Registers per thread after the split; the block is launched with 96 for each (the largest multiple of eight of which 640
// threads get one), and 512 * 112 + 128 * 24 is less than 640 * 96.
constexpr int kRegsCompute = 112, kRegsIssue = 24;
static_assert(kThreadsB * kRegsCompute + 128 * kRegsIssue <= kThreadsAll * 96, "register split");
constexpr int kFixCap = 128;           // tiny-gate entries per chunk
constexpr int kFixParts = 512;         // partial sums of all entries together
constexpr int kS0Ld = 144;             // row stride (bytes) of the start-state landing zone (64 x 16-bit + pad)
constexpr int kRLd = 256;              // row stride (bytes) of the end-gradient landing zone (64 x fp32)
// shared-memory map (bytes from the 1024-byte aligned base); side 0 = k, 1 = d
// Two buffers of four tiles that change places with every chunk: operands [side][2] tiles [step][feature]: Mm (q pm | dO pm),
// Vm (k / pm | x / pm), over which the results are staged once TQ1 and T7 have read them; and Z [own side][2] tiles: Z [t][s],
// Z^T [s][t].  So the next chunk's operands never meet results that are still on their way out.
constexpr int kTiles = 4 * kTile;
constexpr int oS0L = 2 * kTiles;                    // start state of the chunk, [64][kS0Ld]
constexpr int oRL = oS0L + kDim * kS0Ld;            // end state gradient of the chunk, [64][kRLd]
constexpr int oQt = oRL + kDim * kRLd;              // quarter products [side][4][64]
constexpr int oXc = oQt + 2 * 4 * kDim * 4;         // partial sums [3][4 quarters][side][64]
constexpr int oBnd = oXc + 3 * 4 * 2 * kDim * 4;    // boundary-term partials [side][4][64]
constexpr int oFixCode = oBnd + 2 * 4 * kDim * 4;   // [kFixCap] int: step << 8 | side << 6 | feature
constexpr int oFixPart = oFixCode + kFixCap * 4;    // [kFixParts] float
constexpr int oDer0 = oFixPart + kFixParts * 4;     // fused layer: derivatives of the gates, [32 steps][64] floats; the other
constexpr int oRaw = oDer0 + kRawBytes;             //   32 steps where the forget gates, which it does not have, would arrive
constexpr int oDer1 = oRaw + kRawBytes;             // raw blocks: x, f, q, k, fk, dO
constexpr int kSmemB = oRaw + 6 * kRawBytes + 1024; // + slack for the 1024-byte alignment
static_assert(oRaw % 128 == 0 && oS0L % 16 == 0 && oRL % 16 == 0, "alignment");
static_assert(kFixCap * 4 <= kFixParts, "at least four parts per entry");
static_assert(kSmemB + 256 <= 227 * 1024, "shared memory limit");

// tensor-memory columns, both lane sets: four A operands, then the accumulators.  T2 takes Z's columns over
// once Z has been read out.
constexpr int cS2 = 0, cR2 = 64, cVw = 128, cMw = 192;
constexpr int cZ = 256, cT2 = 256, cTQ1 = 320, cTQ2 = 384, cT7 = 448;
constexpr int kTmemCols = 512;

// kMode: 0 the plain operator, 1 the fused layer (forget gate 1, k-side gates from pre-activations), 2 a grid of blocks
// (gradients summed over the blocks of the other axis)
template <typename T, int kMode>
__global__ void __launch_bounds__(kThreadsAll, 1)
lfw_c64_bwd_kernel(const __grid_constant__ seq::Maps mp, const T *__restrict__ state, const T *__restrict__ ckpt,
                   const float *__restrict__ Rend, const seq::Out<T> dx, const seq::Out<T> df, const seq::Out<T> dq,
                   const seq::Out<T> dk, const seq::Out<T> dfk, int *__restrict__ rowflag, int *__restrict__ status,
                   int64_t T_, int64_t nc, int64_t total) {
  constexpr bool kFused = kMode == 1, kGrid = kMode == 2;
  extern __shared__ __align__(1024) unsigned char sm_raw[];
  unsigned char *sm = sm_raw + ((1024u - (umma::smem_u32(sm_raw) & 1023u)) & 1023u);
  __shared__ __align__(8) uint64_t barRaw, barState, barT, barA, barZs, barZ, barM1, barM2, barOut;
  __shared__ uint32_t tmem_slot;
  __shared__ int s_bad2[2], fix_n2[2];

  const int tid = threadIdx.x, warp = uniform_warp_idx(), lane = tid & 31;
  // lane quarter of tensor memory, 16-step quarter of the chunk, side (0 k, 1 d), row in the quarter
  const int q4 = warp & 3, tq = warp >> 2, h = lane >> 4, fl = lane & 15;
  const int feat = 16 * ((q4 + h) & 3) + fl;          // own feature (tensor-memory row 16 q4 + fl of lane set h)
  const int t0 = 16 * tq;                             // first own step; also the first own column of the state blocks

  float *qtot = reinterpret_cast<float *>(sm + oQt);
  float *xc = reinterpret_cast<float *>(sm + oXc);
  float *bndp = reinterpret_cast<float *>(sm + oBnd);
  int *fix_code = reinterpret_cast<int *>(sm + oFixCode);
  T *raw = reinterpret_cast<T *>(sm + oRaw);     // [6][64][64]: x, f, q, k, fk, dO

  // tensors: 0 x, 1 f, 2 q, 3 k, 4 fk, 5 dO
  const float q_scale = kFused ? mp.q_scale : 1.f;
  auto valid_steps = [&](const ItemWalk &w) {
    const int64_t left = T_ - (int64_t)w.c * kC;
    return (int)(left < kC ? left : kC);
  };
  auto issue_raw = [&](const ItemWalk &w) {     // one thread: one copy per tensor
    int b, hc;
    w.item(mp.heads, &b, &hc);
    const int row = (int)(b * T_ + w.c * kC), nv = valid_steps(w);
    const uint32_t per = (mp.flags & seq::kContiguous) ? (uint32_t)nv * kDim * sizeof(T) : (uint32_t)kRawBytes;
    acp::mbar_expect_tx(&barRaw, (kFused ? 5u : 6u) * per);
#pragma unroll 1
    for (int i = 0; i < 6; ++i)
      if (!(i == 1 && kFused)) seq::fetch_block<T>(mp, i, sm + oRaw + i * kRawBytes, row, hc, nv, &barRaw);
  };
  // one warp: start state of a chunk (16-bit, 8 KB; row by row into the padded landing zone) and end state gradient (fp32,
  // 16 KB, pieces XOR-ed by row as the carry left them)
  auto issue_state = [&](const ItemWalk &w) {
    const T *s0p = (w.c == 0) ? state + seq::state_off(mp, w.row, w.sub, 0, 1) : ckpt + seq::state_off(mp, w.row, w.sub, w.c - 1, nc);
    if (lane == 0) {
      acp::mbar_expect_tx(&barState, kDim * kDim * (uint32_t)(sizeof(float) + sizeof(T)));
      acp::bulk_g2s(sm + oRL, Rend + ((size_t)w.bh() * nc + w.c) * kDim * kDim, kDim * kDim * (uint32_t)sizeof(float), &barState);
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < kDim; r += 32)
      acp::bulk_g2s(sm + oS0L + (lane + r) * kS0Ld, s0p + (size_t)(lane + r) * mp.state_ld, kDim * (uint32_t)sizeof(T), &barState);
  };
  // this warp's writes are complete: tiles (for the tensor core) and tensor memory
  auto report = [&](uint64_t *bar) {
    umma::fence_async_smem();
    umma::fence_before_sync();
    __syncwarp();
    if (lane == 0) acp::mbar_arrive(bar);
  };

  if (tid == 0) {
    umma::mbar_init(&barRaw, 1);
    umma::mbar_init(&barState, 1);
    umma::mbar_init(&barT, kWarpsB + 1);  // operand tiles, and the results before have left the other buffer
    umma::mbar_init(&barA, kWarpsB);      // state operands
    umma::mbar_init(&barZs, kWarpsB);     // Z tiles
    umma::mbar_init(&barZ, 1);
    umma::mbar_init(&barM1, 1);           // TQ1 and T7 of both sides
    umma::mbar_init(&barM2, 1);           // TQ2 and T2 of both sides
    umma::mbar_init(&barOut, kWarpsB);    // results staged
    umma::mbar_fence_init();
    s_bad2[0] = s_bad2[1] = fix_n2[0] = fix_n2[1] = 0;
  }
  if (warp == 0) umma::tmem_alloc(&tmem_slot, kTmemCols);
  sync_all();
  dependency_wait();
  const uint32_t tb = __shfl_sync(0xffffffffu, tmem_slot, 0);
  ItemWalk wn(blockIdx.x, gridDim.x, nc, kGrid ? mp.nsub : 1);
  uint32_t it = 0;
  int fail = 0;
  if (warp >= kWarpsB) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsIssue));
    if (warp == kWarpsB) {      // ---- products ----
      const uint32_t aSm = umma::smem_u32(sm);
      for (; wn.unit < total && !fail; ++it, wn.step()) {
        const uint32_t ph = it & 1u;
        const uint32_t aT = aSm + ph * kTiles, aZ = aSm + (ph ^ 1u) * kTiles;
        const uint32_t ls = tb, ls1 = umma::tmem_addr(tb, 16, 0);      // lane sets of the k side and the d side
        // The chains of dependent instructions of the two sides and of the two results take turns: the tensor core
        // executes in issue order.
        if (!umma::mbar_wait(&barT, ph)) fail = 1;
        umma::fence_after_sync();
        if (elect_one()) {      // Z of either side from the other side's tiles
          const uint64_t k0 = desc_sw128(aT), k1 = desc_sw128(aT + kTile), d0 = desc_sw128(aT + 2 * kTile), d1 = desc_sw128(aT + 3 * kTile);
#pragma unroll 1
          for (int ks = 0; ks < 8; ++ks) {
            umma::mma_tf32(ls + cZ, d0 + kstep(ks), d1 + kstep(ks), kIdesc64, ks > 0);
            umma::mma_tf32(ls1 + cZ, k0 + kstep(ks), k1 + kstep(ks), kIdesc64, ks > 0);
          }
          umma::mma_commit(&barZ);
        }
        __syncwarp();
        if (!umma::mbar_wait(&barA, ph)) fail = 1;
        umma::fence_after_sync();
        if (elect_one()) {
          const uint64_t k0 = desc_sw128(aT), k1 = desc_sw128(aT + kTile), d0 = desc_sw128(aT + 2 * kTile), d1 = desc_sw128(aT + 3 * kTile);
#pragma unroll 1
          for (int ks = 0; ks < 8; ++ks) {
            mma_tf32_ts(ls + cTQ1, ls + cS2 + 8 * ks, d0 + kstep(ks), kIdesc64, ks > 0);
            mma_tf32_ts(ls1 + cTQ1, ls1 + cS2 + 8 * ks, k0 + kstep(ks), kIdesc64, ks > 0);
            mma_tf32_ts(ls + cT7, ls + cR2 + 8 * ks, d1 + kstep(ks), kIdesc64, ks > 0);
            mma_tf32_ts(ls1 + cT7, ls1 + cR2 + 8 * ks, k1 + kstep(ks), kIdesc64, ks > 0);
          }
          umma::mma_commit(&barM1);
        }
        __syncwarp();
        if (!umma::mbar_wait(&barZs, ph)) fail = 1;
        umma::fence_after_sync();
        if (elect_one()) {      // TQ2 = Vw Z^T, T2 = Mw Z
          const uint64_t k0 = desc_sw128(aZ), k1 = desc_sw128(aZ + kTile), d0 = desc_sw128(aZ + 2 * kTile), d1 = desc_sw128(aZ + 3 * kTile);
#pragma unroll 1
          for (int ks = 0; ks < 8; ++ks) {
            mma_tf32_ts(ls + cTQ2, ls + cVw + 8 * ks, k0 + kstep(ks), kIdesc64, ks > 0);
            mma_tf32_ts(ls1 + cTQ2, ls1 + cVw + 8 * ks, d0 + kstep(ks), kIdesc64, ks > 0);
            mma_tf32_ts(ls + cT2, ls + cMw + 8 * ks, k1 + kstep(ks), kIdesc64, ks > 0);
            mma_tf32_ts(ls1 + cT2, ls1 + cMw + 8 * ks, d1 + kstep(ks), kIdesc64, ks > 0);
          }
          umma::mma_commit(&barM2);
        }
        __syncwarp();
      }
    } else if (warp == kWarpsB + 1) {      // ---- raw blocks ----
      int item = 0;
      for (;; ++it, wn.step()) {
        if (it > 0) {
          if (!umma::mbar_wait(&barT, (it - 1) & 1u)) fail = 1;      // every warp has read its raw values
          if (lane == 0 && s_bad2[(it - 1) & 1u]) atomicExch(rowflag + item, 1);      // the scan kernels redo this row
        }
        if (wn.unit >= total || fail) break;
        item = wn.row;
        if (lane == 0) issue_raw(wn);
      }
      // after a wait that gave up, copies may still be on their way into this CTA: bounded, let them land
      if (it > 0) acp::mbar_wait(&barRaw, (it - 1) & 1u);
    } else if (warp == kWarpsB + 2) {      // ---- state blocks ----
      for (;; ++it, wn.step()) {
        if (it > 0 && !umma::mbar_wait(&barA, (it - 1) & 1u)) fail = 1;      // the landing zones have been read
        if (wn.unit >= total || fail) break;
        issue_state(wn);
      }
      if (it > 0) acp::mbar_wait(&barState, (it - 1) & 1u);
    } else {      // ---- results ----
      if (lane == 0) acp::mbar_arrive(&barT);
      for (; wn.unit < total && !fail; ++it, wn.step()) {
        if (!umma::mbar_wait(&barOut, it & 1u)) fail = 1;
        if (lane == 0 && !fail) {
          const unsigned char *const uT = sm + (it & 1u) * kTiles;
          int ob, oh;
          wn.item(mp.heads, &ob, &oh);
          const int64_t row0 = (int64_t)ob * T_ + (int64_t)wn.c * kC;
          const int nvalid = valid_steps(wn);
          if (kMode == 0) {      // dense [rows][64] arrays: one linear copy per tensor
            const uint32_t bytes = (uint32_t)nvalid * kDim * sizeof(T);
            acp::bulk_s2g(dq.p + row0 * kDim, uT, bytes);
            acp::bulk_s2g(dk.p + row0 * kDim, uT + kRawBytes, bytes);
            acp::bulk_s2g(dfk.p + row0 * kDim, uT + 2 * kRawBytes, bytes);
            acp::bulk_s2g(dx.p + row0 * kDim, uT + 3 * kRawBytes, bytes);
            acp::bulk_s2g(df.p + row0 * kDim, uT + 4 * kRawBytes, bytes);
          } else if (kFused && nvalid == kC) {      // boxes of the gradient of the projection output
            seq::store_block(&mp.out, dq.col + oh * kDim, (int)row0, uT);
            seq::store_block(&mp.out, dk.col + oh * kDim, (int)row0, uT + kRawBytes);
            seq::store_block(&mp.out, dfk.col + oh * kDim, (int)row0, uT + 2 * kRawBytes);
            seq::store_block(&mp.out, dx.col + oh * kDim, (int)row0, uT + 3 * kRawBytes);
          }
          acp::bulk_commit();
          acp::bulk_wait_read<0>();
          acp::mbar_arrive(&barT);      // the buffer is free for the next chunk's Z
        }
      }
      if (lane == 0) acp::bulk_wait_all();
    }
    if (fail) atomicExch(status, 1);
  } else {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsCompute));
  const uint32_t tl = umma::tmem_addr(tb, 32 * q4, 0);
  // tile column offset of the own feature: row r of the swizzled tile adds r * 128 and XORs r % 8 into bits 4-6
  const int tcol = (feat >> 5) * kColBlock + ((feat & 3) << 2), tswz = ((feat >> 2) & 7) << 4;
  // Z tiles of the own side: row 16 q4 + fl, columns t0 .. (16-byte pieces XOR-ed with the row); and column
  // 16 q4 + fl of the transposed tile, rows t0 .., the second half warp four rows on
  const int zt_row = 16 * q4 + fl;
  const int zrow = h * 2 * kTile + (t0 >> 5) * kColBlock + zt_row * 128;
  const int zsw = (((t0 >> 2) & 7) ^ (zt_row & 7)) << 4;
  const int zt_lo = (h * 2 + 1) * kTile + (zt_row >> 5) * kColBlock + t0 * 128 + ((zt_row & 3) << 2) + 512 * h;
  const int zt_hi = zt_lo - 1024 * h;
  const int ztsw = (((zt_row >> 2) & 7) ^ (4 * h)) << 4;
  // column of the end gradient: as in a tile, a row's pieces are XOR-ed with (row % 8)
  const int rcol = ((feat >> 5) << 7) + ((feat & 3) << 2), rswz = tswz;
  const T *gcol = raw + (h ? 1 : 4) * kC * kDim + t0 * kDim + feat;
  const T *mcol = raw + (h ? 5 : 2) * kC * kDim + t0 * kDim + feat;
  const T *vcol = raw + (h ? 0 : 3) * kC * kDim + t0 * kDim + feat;
  // fused layer: the gates' derivatives of the quarter, steps 0 .. 31 and 32 .. 63 in different places
  float *const der = reinterpret_cast<float *>(sm + (tq < 2 ? oDer0 : oDer1)) + (t0 & 31) * kDim + 16 * q4 + fl;

  for (; wn.unit < total; ++it) {
    const ItemWalk wi = wn;
    wn.step();
    const uint32_t ph = it & 1u;
    const int nvalid = valid_steps(wi);
    // first row and column windows of the chunk in the output arrays
    int ob, oh;
    wi.item(mp.heads, &ob, &oh);
    const int64_t row0 = (int64_t)ob * T_ + (int64_t)wi.c * kC;
    // grid: block (i, j) holds d-side window i and k-side window j; `add`: not the first block of the sum over the other axis
    const int gi = kGrid ? oh / mp.nk : 0, gj = kGrid ? oh - gi * mp.nk : 0;
    const bool add = kGrid && (h ? gj : gi) != 0;
    int &fix_n = fix_n2[ph], &s_bad = s_bad2[ph];
    // this chunk's operand tiles (then its results) and its Z tiles
    unsigned char *const uT = sm + ph * kTiles, *const uZ = sm + (ph ^ 1u) * kTiles;

    if (!acp::mbar_wait(&barRaw, ph)) fail = 1;

    // ---- gates of the own feature and quarter, product of the quarter ----
    float g[16];
    float g_min = kRangeHi;
    if (kFused) {      // the two half warps share the activations of the k side's feature; the d side's gates are 1
      float a[8];
      const T *p = raw + 4 * kC * kDim + (t0 + 8 * h) * kDim + 16 * q4 + fl;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float e = seq::exp_neg(Elem<T>::ld(p + j * kDim)), sg = seq::rcp1p(e);
        a[j] = seq::round_to<T>(seq::floored(sg));
        // d gate / d pre-activation in fp32: s (1 - s) = s^2 e^-g
        der[(8 * h + j) * kDim] = sg > seq::kGateFloor ? sg * sg * e : 0.f;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float o = __shfl_xor_sync(0xffffffffu, a[j], 16);
        g[j] = h ? 1.f : a[j];
        g[8 + j] = h ? 1.f : o;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) g[j] = Elem<T>::ld(gcol + j * kDim);
    }
    if (nvalid < kC) {      // partial chunk: identity steps beyond the valid ones
#pragma unroll
      for (int j = 0; j < 16; ++j) g[j] = t0 + j < nvalid ? g[j] : 1.f;
    }
    if (!kFused) {          // (the fused layer's gates are at least 1/8)
#pragma unroll
      for (int j = 0; j < 16; j += 2) g_min = min3_abs(g_min, g[j], g[j + 1]);
      if (!(g_min >= kTinyState)) {      // rare: some gate needs the clamp
#pragma unroll
        for (int j = 0; j < 16; ++j) g[j] = sanitize_gate(g[j]);
      }
    }
    {
      float p0 = g[0], p1 = g[1];      // two chains
#pragma unroll
      for (int j = 2; j < 16; j += 2) { p0 *= g[j]; p1 *= g[j + 1]; }
      qtot[(h * 4 + tq) * kDim + feat] = p0 * p1;
    }
    float mw[16], vw[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      mw[j] = Elem<T>::ld(mcol + j * kDim);
      vw[j] = Elem<T>::ld(vcol + j * kDim);
    }
    if (umma::named_barrier_or(5, kThreadsB, fail)) break;      // (the whole group leaves together)
    unsigned tiny = 0;                     // steps of the quarter with tiny gates
    float pm[16], up, after, pm_prev;      // ratios to the anchor; products up to and after it; ratio of the step before
    {
      const float *qt = qtot + h * 4 * kDim + feat;
      const float q0 = qt[0], q1 = qt[kDim], q2 = qt[2 * kDim], q3 = qt[3 * kDim];
      up = q0 * q1;
      after = q2 * q3;
      pm_prev = tq == 0 ? rcp_fast(up) : tq == 1 ? rcp_fast(q1) : tq == 2 ? 1.f : q2;
      const float carry = tq == 0 ? q1 : tq == 3 ? q2 : 1.f;
      if (kFused) {
#pragma unroll
        for (int j = 0; j < 16; ++j) mw[j] = h ? mw[j] : seq::round_to<T>(mw[j] * q_scale);
      }
      if (nvalid < kC) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          mw[j] = t0 + j < nvalid ? mw[j] : 0.f;
          vw[j] = t0 + j < nvalid ? vw[j] : 0.f;
        }
      }
      // The walk away from the anchor: downwards for the first two quarters (s = 1 / pm), upwards for the others; and back
      // with the reciprocal of the product at the far end, which the gates on the way turn into that of every step.
      float s = carry, lo = fabsf(carry), hi = lo, r;
      if (tq < 2) {
#pragma unroll
        for (int j = 15; j >= 0; --j) {
          const float e = vw[j];
          vw[j] = rna_tf32<kFused>(e * s);
          if (j == 0) r = rcp_fast(s);
          s *= g[j];
          lo = fminf(lo, fabsf(s));
          hi = max3_abs(hi, s, e);      // x and k too
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (j > 0) r *= g[j];
          pm[j] = r;
          mw[j] = rna_tf32<kFused>(mw[j] * r);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          s *= g[j];
          lo = fminf(lo, fabsf(s));
          hi = max3_abs(hi, s, vw[j]);
          pm[j] = s;
          mw[j] = rna_tf32<kFused>(mw[j] * s);
        }
        r = rcp_fast(s);
#pragma unroll
        for (int j = 15; j >= 0; --j) {
          vw[j] = rna_tf32<kFused>(vw[j] * r);
          r *= g[j];
        }
      }
      if (!(lo >= kRangeLo && hi <= kRangeHi)) s_bad = 1;
      umma::tmem_st16(tl + cMw + t0, mw);
      umma::tmem_st16(tl + cVw + t0, vw);
      unsigned char *tp = uT + h * 2 * kTile + tcol + t0 * 128;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        unsigned char *p = tp + (tswz ^ ((j & 7) << 4)) + j * 128;
        *reinterpret_cast<float *>(p) = mw[j];
        *reinterpret_cast<float *>(p + kTile) = vw[j];
      }
      if (!kFused && g_min < kTinyGate) {      // rare: exact pair sums for these steps, listed further down
#pragma unroll
        for (int j = 0; j < 16; ++j) tiny |= (fabsf(g[j]) < kTinyGate && t0 + j < nvalid ? 1u : 0u) << j;
      }
    }
    umma::tmem_st_wait();
    report(&barT);

    if (tid == 0) {      // (the other chunk's; read by nobody any more, written behind the next barrier)
      s_bad2[ph ^ 1u] = 0;
      fix_n2[ph ^ 1u] = 0;
    }

    // ---- state blocks as A operands: row = own feature, columns t0 .. t0 + 15 of the other side, scaled by the
    //      other side's anchor products; their elementwise product is the boundary term ----
    if (!acp::mbar_wait(&barState, ph)) fail = 1;
    {
      const float *oq = qtot + (h ^ 1) * 4 * kDim + t0;
      float sv[16], rv[16];
      if (h == 0) {         // S(own = k, other = d = t0 + j): a column of the stored blocks
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          sv[j] = Elem<T>::ld(reinterpret_cast<const T *>(sm + oS0L + (t0 + j) * kS0Ld) + feat);
          rv[j] = *reinterpret_cast<const float *>(sm + oRL + (t0 + j) * kRLd + rcol + (rswz ^ ((j & 7) << 4)));
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
          const float4 r4 = *reinterpret_cast<const float4 *>(sm + oRL + feat * kRLd + (((4 * tq + i) ^ (feat & 7)) << 4));
          rv[4 * i] = r4.x; rv[4 * i + 1] = r4.y; rv[4 * i + 2] = r4.z; rv[4 * i + 3] = r4.w;
        }
      }
      __syncwarp();
      float acc = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 q0 = *reinterpret_cast<const float4 *>(oq + 4 * i), q1 = *reinterpret_cast<const float4 *>(oq + kDim + 4 * i);
        const float4 q2 = *reinterpret_cast<const float4 *>(oq + 2 * kDim + 4 * i), q3 = *reinterpret_cast<const float4 *>(oq + 3 * kDim + 4 * i);
        const float av[4] = {q0.x * q1.x, q0.y * q1.y, q0.z * q1.z, q0.w * q1.w};
        const float bv[4] = {q2.x * q3.x, q2.y * q3.y, q2.z * q3.z, q2.w * q3.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float s2 = sv[4 * i + j] * av[j], r2 = rv[4 * i + j] * bv[j];
          acc = fmaf(s2, r2, acc);
          sv[4 * i + j] = bias_tf32<kFused>(s2);
          rv[4 * i + j] = bias_tf32<kFused>(r2);
        }
      }
      umma::tmem_st16(tl + cS2 + t0, sv);
      umma::tmem_st16(tl + cR2 + t0, rv);
      bndp[(h * 4 + tq) * kDim + feat] = acc;
      if (!kFused && !(fabsf(acc) <= 3.4028235e38f)) atomicExch(rowflag + wi.row, 1);      // no finite number in a state
    }
    umma::tmem_st_wait();
    report(&barA);
    if (!kFused) {
      for (; tiny != 0; tiny &= tiny - 1) {
        const int slot = atomicAdd(&fix_n, 1);
        if (slot < kFixCap) fix_code[slot] = ((t0 + __ffs(tiny) - 1) << 8) | (h << 6) | feat;
        else atomicExch(rowflag + wi.row, 1);      // the scan kernels redo this row
      }
      __syncwarp();
    }

    // ---- Z: mask, round, store as [t][s] and [s][t].  A warp holds rows 16 q4 .. + 15 and columns t0 .. t0 + 15: on
    //      the diagonal it masks, below it nothing is masked, above it all is zero ----
    if (!umma::mbar_wait(&barZ, ph)) fail = 1;
    umma::fence_after_sync();
    {
      float v[16];
      if (tq <= q4) {
        umma::tmem_ld16(tl + cZ + t0, v);
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
        *reinterpret_cast<float4 *>(uZ + zrow + (zsw ^ (j << 4))) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
      // transposed: the half warps take rows four apart, which lie in different halves of the swizzle
#pragma unroll
      for (int j = 0; j < 16; ++j)
        *reinterpret_cast<float *>(uZ + ((j & 4) ? zt_hi : zt_lo) + j * 128 + (ztsw ^ ((j & 7) << 4))) = h ? v[j ^ 4] : v[j];
    }
    report(&barZs);

    // ---- epilogue: own feature, steps t0 .. t0 + 15 ----
    // state terms first, while the in-chunk products run: H = inclusive suffix of Mw TQ1 + exclusive prefix of Vw T7
    float H[16], tot_a, tot_p;
    if (!umma::mbar_wait(&barM1, ph)) fail = 1;
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

    // ---- tiny gates: pair terms i < t <= s summed directly (runs under the MMAs) from the tiles, an entry's sum over s by
    //      several warps ----
    if (!kFused && !umma::mbar_wait(&barZs, ph)) fail = 1;      // the entries and Z tiles of all warps
    const int n_fix = kFused ? 0 : fix_n < kFixCap ? fix_n : kFixCap;
    const int parts_log = n_fix <= kFixParts / 16 ? 4 : n_fix <= kFixParts / 8 ? 3 : 2, n_parts = 1 << parts_log;
    float *const fix_part = reinterpret_cast<float *>(sm + oFixPart);      // [entry][n_parts]
    if (n_fix > 0) {
#pragma unroll 1
      for (int task = warp; task < n_fix * n_parts; task += kWarpsB) {
        const int code = fix_code[task >> parts_log], t = code >> 8, sf = code & 127, f = sf & 63;
        const unsigned char *const mt = uT + (sf >> 6) * 2 * kTile + (f >> 5) * kColBlock + ((f & 3) << 2);      // column of Mw
        const unsigned char *const zt = uZ + (sf >> 6) * 2 * kTile + ((lane & 3) << 2);
        auto at = [](const unsigned char *p, int r, int piece) {      // row r of a tile's column; as the tensor core reads it
          return __uint_as_float(*reinterpret_cast<const uint32_t *>(p + r * 128 + ((piece ^ (r & 7)) << 4)) & 0xffffe000u);
        };
        // sum_{s >= t} Mw[s] sum_{i < t} Z[s][i] Vw[i]: lanes over i and i + 32, this part's s
        float a0 = 0.f, a1 = 0.f;
#pragma unroll 2
        for (int r = t + (task & (n_parts - 1)); r < kC; r += n_parts) {
          const float m = at(mt, r, (f >> 2) & 7);
          a0 = fmaf(m, at(zt, r, lane >> 2), a0);
          a1 = fmaf(m, at(zt + kColBlock, r, lane >> 2), a1);
        }
        float acc = lane < t ? a0 * at(mt + kTile, lane, (f >> 2) & 7) : 0.f;
        if (lane + 32 < t) acc = fmaf(a1, at(mt + kTile, lane + 32, (f >> 2) & 7), acc);
        acc = warp_sum(acc);
        if (lane == 0) fix_part[task] = acc;
      }
      umma::named_barrier(5, kThreadsB);      // the direct sums are visible, the tiles are free
    }

    if (!umma::mbar_wait(&barM2, ph)) fail = 1;
    umma::fence_after_sync();
    // Every warp is past its last read of the operand tiles: the results are staged there as [5][64 steps][64 features]
    // blocks (d_q, d_k, d_f_key, d_x, d_f) and leave in whole rows.
    T *const stage = reinterpret_cast<T *>(uT) + t0 * kDim + feat;
    T *const s_dv = stage + (h ? 3 : 1) * kC * kDim, *const s_gt = stage + (h ? 4 : 2) * kC * kDim;
    const int rr = tid >> 3, rp = tid & 7;      // row and 16-byte piece of this thread where rows leave by plain stores
    auto place = [&](const seq::Out<T> &o, int col) { return o.p + (size_t)(row0 + rr) * o.ld + o.col + col + rp * 8; };
    if (kGrid && (gi | gj) != 0) {      // this thread's own sums over the blocks before
      uint4 old[5];
      if (rr < nvalid) {
        const seq::Out<T> *const o[5] = {&dq, &dk, &dfk, &dx, &df};
#pragma unroll
        for (int i = 0; i < 5; ++i)
          if ((i < 3 ? gi : gj) != 0) old[i] = *reinterpret_cast<const uint4 *>(place(*o[i], (i < 3 ? gj : gi) * kDim));
#pragma unroll
        for (int i = 0; i < 5; ++i)
          if ((i < 3 ? gi : gj) != 0) reinterpret_cast<uint4 *>(uT)[i * 512 + tid] = old[i];
      }
      umma::named_barrier(5, kThreadsB);
    }
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
        if (h == 0) stage[jj * kDim] = (T)(kFused ? dmu * q_scale : kGrid && add ? dmu + Elem<T>::ld(stage + jj * kDim) : dmu);
        s_dv[jj * kDim] = (T)(kGrid && add ? ddv + Elem<T>::ld(s_dv + jj * kDim) : ddv);
      }
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
            float v = 0.f;
            for (int i = 0; i < n_parts; ++i) v += fix_part[e * n_parts + i];
#pragma unroll
            for (int j = 0; j < 16; ++j) sb[j] = (jj == j) ? v : sb[j];
          }
        }
      }
      if (!(kFused && h == 1)) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          float dg = (H[j] + base + sb[j]) * pm[j];
          if (kFused) dg *= der[j * kDim];
          s_gt[j * kDim] = (T)(kGrid && add ? dg + Elem<T>::ld(s_gt + j * kDim) : dg);
        }
      }
      __syncwarp();
    }
    // ---- own part of the results staged ----
    if (kGrid || (kFused && nvalid < kC)) {      // rows that no bulk copy can take: 16 bytes per thread
      const int kcol = (kGrid ? gj : oh) * kDim, dcol = (kGrid ? gi : oh) * kDim;
      umma::named_barrier(5, kThreadsB);
      if (rr < nvalid) {
        const uint4 *v = reinterpret_cast<const uint4 *>(uT) + tid;
        *reinterpret_cast<uint4 *>(place(dq, kcol)) = v[0];
        *reinterpret_cast<uint4 *>(place(dk, kcol)) = v[512];
        *reinterpret_cast<uint4 *>(place(dfk, kcol)) = v[2 * 512];
        *reinterpret_cast<uint4 *>(place(dx, dcol)) = v[3 * 512];
        if (!kFused) *reinterpret_cast<uint4 *>(place(df, dcol)) = v[4 * 512];
      }
    }
    report(&barOut);
  }
  if (fail) atomicExch(status, 1);
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
    T2FW_CHECK_CUDA(launch_dependent(lfw_c64_bwd_kernel<TT, FF>, dim3(grid), dim3(kThreadsAll), kSmemB, st, mp,   \
                                     (const TT *)state, (const TT *)ckpt, Rend, T2FW_OUT(TT, 0), T2FW_OUT(TT, 1), \
                                     T2FW_OUT(TT, 2), T2FW_OUT(TT, 3), T2FW_OUT(TT, 4), rowflag, status, T_, nc,  \
                                     total));                                                         \
  } while (0)
  const bool fused = (mp.flags & seq::kFusedLayer) != 0;
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

