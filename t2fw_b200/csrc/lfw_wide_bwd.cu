// Sequence gradients of the chunked decay-rule backward for states of up to 128 x 128 (D, K = 64 or 128, one of them 128;
// 16-bit storage, chunks of 64 steps): what lfw_c64_bwd.cu is for 64 x 64 states (notation and identities there).
//
// As a grid of 64 x 64 blocks every block would scale its windows' operands again, form the same in-chunk decays as the other
// blocks of its row or column, and add its gradients to theirs through memory.  Here a chunk is one problem: the operands of
// all windows are built once, Z of either side is one contraction over all features of the other side, and the gradients of a
// side's 128 features fill the lanes of tensor memory.  The sides take turns:
//     build      tiles [step][feature] of both sides; Z of both sides
//     k side     TQ1, T7 over the windows of the d side; TQ2, T2; sums over time; d_q, d_k, d_f_key
//     d side     the same with the roles exchanged; d_x, d_f
// Thread (feature, 16-step quarter) serves the feature with its number on either side; a side with 64 features leaves the upper
// half of the threads without work there.  The side loop is rolled (one copy of its code; see lfw_c64_bwd.cu on cold
// instruction caches).
//
// Tensor memory: A operands and accumulators of the side at work; TQ2 and T2 take the state operands' columns over, and the
// d side's ratios wait there for its turn.  Shared memory: raw values land where tiles will be (a thread takes its values into
// registers before the barrier that precedes the tiles' first write), Z tiles and staged results share one area.
//
// Issue slots 50 % busy (70 k warp instructions per chunk of four blocks), tensor pipe 12 %, DRAM 17 % (16 rows x 2048 steps).
// 16 rows x 16384 steps, 128 x 128 (4096 chunks): 1052 us as a grid of blocks -> 515 us (557 with the end gradients
// loaded by the threads that use them: the d side's rows are 256 bytes apart, 9 k of 37 k cycles per chunk).  Bound by the latency of
// its phases, as the 64 x 64 kernel was before its issuing warps: block barriers, and state blocks that are loaded when they are needed.
#include "lfw_c64.cuh"
#include "seq_layout.cuh"

namespace t2fw {

using namespace c64;

int lfw_chunk_status_ptr(int **out);   // lfw_c64_local.cu
int lfw_chunk_sm_count(int *out);

namespace {

constexpr int kThreadsW = 512;
constexpr int kWarpsW = kThreadsW / 32;
constexpr int kWide = 128;             // features of a side, the upper half possibly unused
constexpr int kFixCap = 128;           // tiny-gate entries per chunk
constexpr int kFixParts = 512;         // partial sums of all entries of a chunk together
// shared-memory map (bytes from the 1024-byte aligned base); side 0 = k, 1 = d
constexpr int kSideTiles = 4 * kTile;               // of a side: [Mm, Vm][window] tiles [step][feature]
constexpr int oTw = 0;                              // [side]; raw values of the next chunk over Mm: q, k / dO, x [window]
constexpr int oXw = oTw + 2 * kSideTiles;           // end gradients, Z [t][s], Z^T [s][t] of the side at work; then its results
constexpr int oGw = oXw + 3 * kTile;                // raw gates: f, fk [window]
constexpr int oQtw = oGw + 4 * kRawBytes;           // [side][4][128] products of the quarters
constexpr int oXcw = oQtw + 2 * 4 * kWide * 4;      // partial sums [3][4 quarters][128]
constexpr int oBndw = oXcw + 3 * 4 * kWide * 4;     // boundary-term partials [4][128]
constexpr int oFixCodeW = oBndw + 4 * kWide * 4;    // [kFixCap] int: step << 8 | side << 7 | feature
constexpr int oFixPartW = oFixCodeW + kFixCap * 4;  // [kFixParts] float
constexpr int kSmemWB = oFixPartW + kFixParts * 4 + 1024;
static_assert(oGw % 128 == 0 && oXw % 1024 == 0, "alignment");
static_assert(kSmemWB + 256 <= 227 * 1024, "shared memory limit");
static_assert(kFixCap * 4 <= kFixParts, "at least four parts per entry");

// tensor-memory columns
constexpr int cMw = 0, cVw = 64, cS2 = 128, cR2 = 192, cTQ2 = 128, cT2 = 192, cTQ1 = 256, cT7 = 320, cZ = 384, cPm = 448;
constexpr int kTmemColsW = 512;
constexpr uint32_t kIdesc128 = umma::make_idesc_tf32(128, 64, false, false);

template <typename T> struct GradsW {
  T *dx, *df, *dq, *dk, *dfk;
};

template <typename T>
__global__ void __launch_bounds__(kThreadsW, 1)
lfw_wide_bwd_kernel(const __grid_constant__ seq::Maps mp, const T *__restrict__ state, const T *__restrict__ ckpt,
                    const float *__restrict__ Rend, const GradsW<T> gr, int *__restrict__ rowflag, int *__restrict__ status,
                    int64_t T_, int64_t nc, int64_t total, int D, int K) {
  extern __shared__ __align__(1024) unsigned char sm_raw[];
  unsigned char *sm = sm_raw + ((1024u - (umma::smem_u32(sm_raw) & 1023u)) & 1023u);
  __shared__ __align__(8) uint64_t barG, barV, barR, barZ, barM1, barM2;
  __shared__ uint32_t tmem_slot;
  __shared__ int s_bad2[2], fix_n2[2];

  const int tid = threadIdx.x, warp = uniform_warp_idx(), lane = tid & 31;
  const int q4 = warp & 3, tq = warp >> 2, t0 = 16 * tq;
  const int feat = 32 * q4 + lane, win = feat >> 6, wf = feat & 63;      // own feature on both sides: window, number in it
  const int nd = D >> 6, nk = K >> 6;
  float *qtot = reinterpret_cast<float *>(sm + oQtw);
  float *xc = reinterpret_cast<float *>(sm + oXcw);
  float *bndp = reinterpret_cast<float *>(sm + oBndw);
  int *fix_code = reinterpret_cast<int *>(sm + oFixCodeW);
  float *fix_part = reinterpret_cast<float *>(sm + oFixPartW);

  // tensors: 0 x, 1 f, 2 q, 3 k, 4 fk, 5 dO
  auto issue_gates = [&](const ItemWalk &w) {     // thread 0 only
    const int row = (int)(w.row * T_ + w.c * kC);
    acp::mbar_expect_tx(&barG, (uint32_t)(nd + nk) * kRawBytes);
#pragma unroll 1
    for (int i = 0; i < nd + nk; ++i) {
      const int j = i < nd ? i : i - nd;
      seq::load_block(sm + oGw + ((i < nd ? 0 : 2) + j) * kRawBytes, i < nd ? &mp.m[1] : &mp.m[4], 64 * j, row, &barG);
    }
  };
  auto issue_values = [&](const ItemWalk &w) {     // thread 0 only
    const int row = (int)(w.row * T_ + w.c * kC);
    acp::mbar_expect_tx(&barV, (uint32_t)(2 * (nd + nk)) * kRawBytes);
#pragma unroll 1
    for (int j = 0; j < nk; ++j) {
      seq::load_block(sm + oTw + j * kRawBytes, &mp.m[2], 64 * j, row, &barV);
      seq::load_block(sm + oTw + (2 + j) * kRawBytes, &mp.m[3], 64 * j, row, &barV);
    }
#pragma unroll 1
    for (int j = 0; j < nd; ++j) {
      seq::load_block(sm + oTw + kSideTiles + j * kRawBytes, &mp.m[5], 64 * j, row, &barV);
      seq::load_block(sm + oTw + kSideTiles + (2 + j) * kRawBytes, &mp.m[0], 64 * j, row, &barV);
    }
  };

  if (tid == 0) {
    umma::mbar_init(&barG, 1);
    umma::mbar_init(&barV, 1);
    umma::mbar_init(&barR, 1);
    umma::mbar_init(&barZ, 2);       // one commit per side
    umma::mbar_init(&barM1, 2);      // TQ1, T7 of one window
    umma::mbar_init(&barM2, 2);      // TQ2, T2
    umma::mbar_fence_init();
    s_bad2[0] = s_bad2[1] = fix_n2[0] = fix_n2[1] = 0;
  }
  if (warp == 0) umma::tmem_alloc(&tmem_slot, kTmemColsW);
  sync_all();
  dependency_wait();
  const uint32_t tb = __shfl_sync(0xffffffffu, tmem_slot, 0);
  const uint32_t tl = umma::tmem_addr(tb, 32 * q4, 0);
  ItemWalk wn(blockIdx.x, gridDim.x, nc, 1);
  bool gates_pending = false, values_pending = false;      // thread 0
  if (wn.unit < total && tid == 0) {
    issue_gates(wn);
    issue_values(wn);
    gates_pending = values_pending = true;
  }
  const uint32_t aT = umma::smem_u32(sm + oTw), aX = umma::smem_u32(sm + oXw);
  // own column of a side's tiles: row r of the swizzled tile adds r * 128 and XORs r % 8 into bits 4-6
  const int tcol = win * kTile + (wf >> 5) * kColBlock + ((wf & 3) << 2) + t0 * 128, tswz = ((wf >> 2) & 7) << 4;
  const T *const rawg = reinterpret_cast<const T *>(sm + oGw + win * kRawBytes) + t0 * kDim + wf;      // f; fk two blocks on
  const T *const rawm = reinterpret_cast<const T *>(sm + oTw + win * kRawBytes) + t0 * kDim + wf;      // q; k two blocks on
  // Z tiles: row 16 q4 + lane % 16 (the half warp of the side), columns t0 ..; the same as a column of the transposed tile
  const int zt_row = 16 * q4 + (lane & 15);
  unsigned char *const zrow = sm + oXw + (t0 >> 5) * kColBlock + zt_row * 128;
  const int zsw = (((t0 >> 2) & 7) ^ (zt_row & 7)) << 4;
  unsigned char *const ztc = sm + oXw + kTile + (zt_row >> 5) * kColBlock + t0 * 128 + ((zt_row & 3) << 2);
  const int ztsw = ((zt_row >> 2) & 7) << 4;

  int fail = 0;                         // a wait of this thread gave up
  uint32_t it = 0, n1 = 0, n2 = 0;      // chunks; rounds of TQ1 / T7 and of TQ2 / T2
  uint32_t nr = 0, nr_issued = 0;       // rounds of end gradients, (thread 0) requested
  // thread 0: end gradients of window v of the other side and all windows of this one, blocks of 16 KB at r0, nc chunks apart
  auto issue_r = [&](const float *r0, int side, int v) {
    const int n = side ? nd : nk;
    acp::mbar_expect_tx(&barR, (uint32_t)n * kTile);
    for (int o = 0; o < n; ++o)
      acp::bulk_g2s(sm + oXw + o * kTile, r0 + (size_t)(side ? o * nk + v : v * nk + o) * nc * kDim * kDim, kTile, &barR);
    ++nr_issued;
  };
  for (; wn.unit < total; ++it) {
    const ItemWalk w = wn;
    wn.step();
    const int64_t left = T_ - (int64_t)w.c * kC;
    const int nvalid = (int)(left < kC ? left : kC);
    int &s_bad = s_bad2[it & 1], &fix_n = fix_n2[it & 1];

    // ---- gates of the own feature and quarter on both sides, products of the quarters; raw values of the k side ----
    if (acp::mbar_wait(&barG, it & 1u)) gates_pending = false;
    else fail = 1;
    float g[2][16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      g[0][j] = feat < K && t0 + j < nvalid ? Elem<T>::ld(rawg + 2 * kC * kDim + j * kDim) : 1.f;
      g[1][j] = feat < D && t0 + j < nvalid ? Elem<T>::ld(rawg + j * kDim) : 1.f;
    }
    float g_min = kRangeHi;
#pragma unroll
    for (int j = 0; j < 16; ++j) g_min = min3_abs(g_min, g[0][j], g[1][j]);
    unsigned tiny = 0;      // steps of the quarter with tiny gates, k side in the low half
    if (g_min < kTinyGate) {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        tiny |= (fabsf(g[0][j]) < kTinyGate ? 1u : 0u) << j;
        tiny |= (fabsf(g[1][j]) < kTinyGate ? 0x10000u : 0u) << j;
      }
    }
    if (!(g_min >= kTinyState)) {      // rare: some gate needs the clamp
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        g[0][j] = sanitize_gate(g[0][j]);
        g[1][j] = sanitize_gate(g[1][j]);
      }
    }
#pragma unroll
    for (int sd = 0; sd < 2; ++sd) {
      float p0 = g[sd][0], p1 = g[sd][1];
#pragma unroll
      for (int j = 2; j < 16; j += 2) { p0 *= g[sd][j]; p1 *= g[sd][j + 1]; }
      qtot[(sd * 4 + tq) * kWide + feat] = p0 * p1;
    }
    if (acp::mbar_wait(&barV, it & 1u)) values_pending = false;
    else fail = 1;
    float mw[16], vw[16], pm[16];
    auto values = [&](int sd, bool has) {
      const T *p = rawm + sd * (kSideTiles / 2);
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        mw[j] = has && t0 + j < nvalid ? Elem<T>::ld(p + j * kDim) : 0.f;
        vw[j] = has && t0 + j < nvalid ? Elem<T>::ld(p + 2 * kC * kDim + j * kDim) : 0.f;
      }
    };
    values(0, feat < K);
    umma::fence_async_smem();
    if (__syncthreads_or(fail)) break;      // products complete; the k side's values are in registers
    const float *const r0 = Rend + ((size_t)w.row * nd * nk * nc + w.c) * kDim * kDim;      // block 0; nc chunks per block
    if (tid == 0) {
      issue_r(r0, 0, 0);      // the results before have left
      if (wn.unit < total) {
        issue_gates(wn);
        gates_pending = true;
      }
    }
    // The walk away from the anchor: downwards for the first two quarters (s = 1 / pm), upwards for the others; and back with
    // the reciprocal of the product at the far end, which the gates on the way turn into that of every step.
    auto walk = [&](int sd, const float (&gg)[16]) {
      const float *qt = qtot + sd * 4 * kWide + feat;
      float s = tq == 0 ? qt[kWide] : tq == 3 ? qt[2 * kWide] : 1.f, lo = fabsf(s), hi = lo, r;
      if (tq < 2) {
#pragma unroll
        for (int j = 15; j >= 0; --j) {
          const float e = vw[j];
          vw[j] = rna_tf32(e * s);
          if (j == 0) r = rcp_fast(s);
          s *= gg[j];
          lo = fminf(lo, fabsf(s));
          hi = max3_abs(hi, s, e);      // x and k too
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          if (j > 0) r *= gg[j];
          pm[j] = r;
          mw[j] = rna_tf32(mw[j] * r);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          s *= gg[j];
          lo = fminf(lo, fabsf(s));
          hi = max3_abs(hi, s, vw[j]);
          pm[j] = s;
          mw[j] = rna_tf32(mw[j] * s);
        }
        r = rcp_fast(s);
#pragma unroll
        for (int j = 15; j >= 0; --j) {
          vw[j] = rna_tf32(vw[j] * r);
          r *= gg[j];
        }
      }
      if (!(lo >= kRangeLo && hi <= kRangeHi)) s_bad = 1;
      unsigned char *tp = sm + oTw + sd * kSideTiles + tcol;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        unsigned char *p = tp + (tswz ^ ((j & 7) << 4)) + j * 128;
        *reinterpret_cast<float *>(p) = mw[j];
        *reinterpret_cast<float *>(p + 2 * kTile) = vw[j];
      }
    };
    // d side last would leave its ratios in registers, but the k side's turn comes first: build the k side, put its operands
    // into tensor memory, keep its ratios, and let the d side's wait in tensor memory.
    walk(0, g[0]);
    umma::tmem_st16(tl + cMw + t0, mw);
    umma::tmem_st16(tl + cVw + t0, vw);
    float pm_k[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) pm_k[j] = pm[j];
    values(1, feat < D);
    __syncthreads();      // the d side's values are in registers
    walk(1, g[1]);
    umma::tmem_st16(tl + cPm + t0, pm);
#pragma unroll
    for (int j = 0; j < 16; ++j) pm[j] = pm_k[j];
    for (; tiny != 0; tiny &= tiny - 1) {      // rare: exact pair sums for these steps
      const int b = __ffs(tiny) - 1, slot = atomicAdd(&fix_n, 1);
      if (slot < kFixCap) fix_code[slot] = ((t0 + (b & 15)) << 8) | ((b >> 4) << 7) | feat;
      else s_bad = 1;
    }
    __syncwarp();
    umma::tmem_st_wait();
    umma::fence_async_smem();
    sync_all();           // tiles of both sides
    if (warp < 2) {       // Z of side `warp` from the other side's tiles, in the lane set of that number
      const uint32_t dz = umma::tmem_addr(tb, 16 * warp, cZ), ot = aT + (warp ^ 1) * kSideTiles;
      const int n = warp ? nk : nd;
      if (elect_one()) {
#pragma unroll 1
        for (int v = 0; v < n; ++v) {
          const uint64_t da = desc_sw128(ot + v * kTile), db = desc_sw128(ot + (2 + v) * kTile);
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) umma::mma_tf32(dz, da + kstep(ks), db + kstep(ks), kIdesc64, v + ks > 0);
        }
        umma::mma_commit(&barZ);
      }
      __syncwarp();
    }
    if (tid == 0) {
      if (s_bad) atomicExch(rowflag + w.row, 1);      // the scan kernels redo this row
      s_bad2[(it & 1) ^ 1] = 0;
      fix_n2[(it & 1) ^ 1] = 0;
    }
    const int n_fix = fix_n < kFixCap ? fix_n : kFixCap;
    const int parts_log = n_fix <= kFixParts / 16 ? 4 : n_fix <= kFixParts / 8 ? 3 : 2, n_parts = 1 << parts_log;
    const T *const s0 = (w.c == 0) ? state + (size_t)w.row * D * K : ckpt + ((size_t)w.row * nc + w.c - 1) * D * K;

#pragma unroll 1
    for (int side = 0; side < 2; ++side) {
      const bool has = feat < (side ? D : K);
      const int n_oth = side ? nk : nd;
      float up, after, pm_prev;      // products up to the anchor and after it; ratio of the step before the quarter
      {
        const float *qt = qtot + side * 4 * kWide + feat;
        const float q0 = qt[0], q1 = qt[kWide], q2 = qt[2 * kWide], q3 = qt[3 * kWide];
        up = q0 * q1;
        after = q2 * q3;
        pm_prev = tq == 0 ? rcp_fast(up) : tq == 1 ? rcp_fast(q1) : tq == 2 ? 1.f : q2;
      }
      if (side == 1) {      // the d side's own operands from its tiles, its ratios from where they wait
        if (tid == 0) {
          acp::bulk_wait_read<0>();      // the k side's results have left
          issue_r(r0, 1, 0);
        }
        const unsigned char *tp = sm + oTw + kSideTiles + tcol;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const unsigned char *p = tp + (tswz ^ ((j & 7) << 4)) + j * 128;
          mw[j] = *reinterpret_cast<const float *>(p);
          vw[j] = *reinterpret_cast<const float *>(p + 2 * kTile);
        }
        umma::tmem_st16(tl + cMw + t0, mw);
        umma::tmem_st16(tl + cVw + t0, vw);
        umma::tmem_ld16(tl + cPm + t0, pm);
        umma::tmem_ld_wait();
      }

      // ---- state blocks as A operands, one window of the other side after the other: row = own feature, columns t0 ..
      //      t0 + 15, scaled by the other side's anchor products; their elementwise product is the boundary term ----
      float acc = 0.f;
#pragma unroll 1
      for (int v = 0; v < n_oth; ++v) {
        float sv[16], rv[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) sv[j] = rv[j] = 0.f;
        if (has) {
          if (side == 0) {         // a column of the stored state, own = k
            const T *sp = s0 + (size_t)(64 * v + t0) * K + feat;
#pragma unroll
            for (int j = 0; j < 16; ++j) sv[j] = Elem<T>::ld(sp + (size_t)j * K);
          } else {                 // a row segment, own = d
            const T *sp = s0 + (size_t)feat * K + 64 * v + t0;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const uint4 u = *reinterpret_cast<const uint4 *>(sp + 8 * i);
              const T *e = reinterpret_cast<const T *>(&u);
#pragma unroll
              for (int j = 0; j < 8; ++j) sv[8 * i + j] = Elem<T>::ld(e + j);
            }
          }
        }
        // end gradients: rows d of a block, 16-byte pieces of a row XOR-ed with (row % 8)
        if (!acp::mbar_wait(&barR, nr++ & 1u)) fail = 1;
        if (has) {
          const unsigned char *rb = sm + oXw + win * kTile;
          if (side == 0) {
            rb += t0 * 256 + ((wf >> 5) << 7) + ((wf & 3) << 2);
#pragma unroll
            for (int j = 0; j < 16; ++j) rv[j] = *reinterpret_cast<const float *>(rb + j * 256 + (tswz ^ ((j & 7) << 4)));
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float4 r4 = *reinterpret_cast<const float4 *>(rb + wf * 256 + (((4 * tq + i) ^ (wf & 7)) << 4));
              rv[4 * i] = r4.x; rv[4 * i + 1] = r4.y; rv[4 * i + 2] = r4.z; rv[4 * i + 3] = r4.w;
            }
          }
        }
        __syncwarp();
        const float *oq = qtot + (side ^ 1) * 4 * kWide + 64 * v + t0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 q0 = *reinterpret_cast<const float4 *>(oq + 4 * i), q1 = *reinterpret_cast<const float4 *>(oq + kWide + 4 * i);
          const float4 q2 = *reinterpret_cast<const float4 *>(oq + 2 * kWide + 4 * i), q3 = *reinterpret_cast<const float4 *>(oq + 3 * kWide + 4 * i);
          const float av[4] = {q0.x * q1.x, q0.y * q1.y, q0.z * q1.z, q0.w * q1.w};
          const float bv[4] = {q2.x * q3.x, q2.y * q3.y, q2.z * q3.z, q2.w * q3.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float s2 = sv[4 * i + j] * av[j], r2 = rv[4 * i + j] * bv[j];
            acc = fmaf(s2, r2, acc);
            sv[4 * i + j] = bias_tf32(s2);
            rv[4 * i + j] = bias_tf32(r2);
          }
        }
        if (v > 0) {      // the window before has been read
          if (!umma::mbar_wait(&barM1, n1++ & 1u)) fail = 1;
          umma::fence_after_sync();
        }
        umma::tmem_st16(tl + cS2 + t0, sv);
        umma::tmem_st16(tl + cR2 + t0, rv);
        umma::tmem_st_wait();
        umma::fence_async_smem();
        sync_all();      // also: the end gradients have been read
        if (tid == 0 && v + 1 < n_oth) issue_r(r0, side, v + 1);
        if (warp == 2 || warp == 4) {      // TQ1 from Mm, T7 from Vm of the other side
          const int is7 = warp >> 2;
          const uint64_t db = desc_sw128(aT + (side ^ 1) * kSideTiles + (2 * is7 + v) * kTile);
          const uint32_t d = tb + (is7 ? cT7 : cTQ1), a = tb + (is7 ? cR2 : cS2);
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) mma_tf32_ts(d, a + 8 * ks, db + kstep(ks), kIdesc128, v + ks > 0);
            umma::mma_commit(&barM1);
          }
          __syncwarp();
        }
      }
      bndp[tq * kWide + feat] = acc;
      if (!(fabsf(acc) <= 3.4028235e38f)) atomicExch(rowflag + w.row, 1);      // no finite number in a state

      // ---- Z: mask, round, store as [t][s] and [s][t].  A warp holds rows 16 q4 .. + 15 and columns t0 .. t0 + 15: on the
      //      diagonal it masks, below it nothing is masked, above it all is zero ----
      if (side == 0 && !umma::mbar_wait(&barZ, it & 1u)) fail = 1;
      umma::fence_after_sync();
      {
        float z[16];
        if (tq <= q4) {
          umma::tmem_ld16(tl + cZ + t0, z);
          umma::tmem_ld_wait();
          if (tq == q4) {
#pragma unroll
            for (int j = 0; j < 16; ++j) z[j] = j <= (lane & 15) ? bias_tf32(z[j]) : 0.f;
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) z[j] = bias_tf32(z[j]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) z[j] = 0.f;
        }
        if (lane >> 4 == side) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            *reinterpret_cast<float4 *>(zrow + (zsw ^ (j << 4))) = make_float4(z[4 * j], z[4 * j + 1], z[4 * j + 2], z[4 * j + 3]);
#pragma unroll
          for (int j = 0; j < 16; ++j) *reinterpret_cast<float *>(ztc + j * 128 + (ztsw ^ ((j & 7) << 4))) = z[j];
        }
      }
      // TQ2 and T2 take the state operands' columns: those must have been read
      if (!umma::mbar_wait(&barM1, n1++ & 1u)) fail = 1;
      umma::fence_after_sync();
      umma::fence_async_smem();
      sync_all();
      if (warp == 1 || warp == 3) {      // TQ2 = Vw Z^T, T2 = Mw Z
        const int is2 = warp >> 1;
        const uint64_t db = desc_sw128(aX + is2 * kTile);
        const uint32_t d = tb + (is2 ? cT2 : cTQ2), a = tb + (is2 ? cMw : cVw);
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) mma_tf32_ts(d, a + 8 * ks, db + kstep(ks), kIdesc128, ks > 0);
          umma::mma_commit(&barM2);
        }
        __syncwarp();
      }
      // ---- tiny gates: pair terms i < t <= s summed directly (runs under the MMAs) from the tiles, an entry's sum over s by
      //      several warps ----
      if (n_fix > 0) {
#pragma unroll 1
        for (int task = warp; task < n_fix * n_parts; task += kWarpsW) {
          const int code = fix_code[task >> parts_log], t = code >> 8, f = code & 127;
          if (((code >> 7) & 1) != side) continue;
          const unsigned char *const mt = sm + oTw + side * kSideTiles + (f >> 6) * kTile + ((f >> 5) & 1) * kColBlock + ((f & 3) << 2);
          const unsigned char *const zt = sm + oXw + ((lane & 3) << 2);
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
          float sum = lane < t ? a0 * at(mt + 2 * kTile, lane, (f >> 2) & 7) : 0.f;
          if (lane + 32 < t) sum = fmaf(a1, at(mt + 2 * kTile, lane + 32, (f >> 2) & 7), sum);
          sum = warp_sum(sum);
          if (lane == 0) fix_part[task] = sum;
        }
        umma::fence_async_smem();
        __syncthreads();      // the direct sums are visible, the tiles are free
      }
      if (side == 1 && tid == 0 && wn.unit < total) {      // nobody reads tiles of this chunk any more
        issue_values(wn);
        values_pending = true;
      }

      // ---- sums over time and results: own feature, steps t0 .. t0 + 15 ----
      // state terms first, while the in-chunk products run: H = inclusive suffix of Mw TQ1 + exclusive prefix of Vw T7
      float H[16], tot_a, tot_p;
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
      if (!umma::mbar_wait(&barM2, n2++ & 1u)) fail = 1;
      umma::fence_after_sync();
      // staged over Z as dense [64][K] or [64][D] blocks: d_q, d_k, d_f_key / d_x, d_f
      const int ext = side ? D : K;
      T *const stage = reinterpret_cast<T *>(sm + oXw) + t0 * ext + feat;
      T *const s_mu = stage + 2 * kC * ext, *const s_gt = stage + kC * ext;      // (k side only: d_q); gate gradient
      float sb[16], run_b = 0.f;
#pragma unroll
      for (int half = 1; half >= 0; --half) {
        float tq2[8], t2[8];
        {
          float m8[8], v8[8];
          umma::tmem_ld8(tl + cTQ2 + t0 + 8 * half, tq2);
          umma::tmem_ld8(tl + cT2 + t0 + 8 * half, t2);
          umma::tmem_ld8(tl + cMw + t0 + 8 * half, m8);
          umma::tmem_ld8(tl + cVw + t0 + 8 * half, v8);
          umma::tmem_ld_wait();
#pragma unroll
          for (int j = 7; j >= 0; --j) {
            run_b += m8[j] * tq2[j] - v8[j] * t2[j];
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
          if (has) {
            if (side == 0) s_mu[jj * ext] = (T)dmu;
            stage[jj * ext] = (T)ddv;
          }
        }
      }
      {
        xc[(0 * 4 + tq) * kWide + feat] = tot_a;
        xc[(1 * 4 + tq) * kWide + feat] = run_b;
        xc[(2 * 4 + tq) * kWide + feat] = tot_p;
        umma::named_barrier(1 + q4, 128);       // the four quarters of the same features
        float base = 0.f, add_b = 0.f;
#pragma unroll
        for (int r = 0; r < 4; ++r) base += bndp[r * kWide + feat];
        base *= up * after;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          if (r > tq) {        // later steps
            base += xc[(0 * 4 + r) * kWide + feat];
            add_b += xc[(1 * 4 + r) * kWide + feat];
          }
          if (r < tq) base += xc[(2 * 4 + r) * kWide + feat];      // earlier steps
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) sb[j] += add_b;
        for (int e = 0; e < n_fix; ++e) {      // tiny gates in this chunk: their pair terms were summed directly
          const int code = fix_code[e], jj = (code >> 8) - t0;
          if ((code & 255) == (side << 7 | feat) && (unsigned)jj < 16u) {
            float sum = 0.f;
            for (int i = 0; i < n_parts; ++i) sum += fix_part[e * n_parts + i];
#pragma unroll
            for (int j = 0; j < 16; ++j) sb[j] = (jj == j) ? sum : sb[j];
          }
        }
        if (has) {
#pragma unroll
          for (int j = 0; j < 16; ++j) s_gt[j * ext] = (T)((H[j] + base + sb[j]) * pm[j]);
        }
        __syncwarp();
      }
      umma::fence_async_smem();
      sync_all();      // results staged
      if (tid == 0) {
        const size_t at = ((size_t)w.row * T_ + (size_t)w.c * kC) * ext;
        const uint32_t bytes = (uint32_t)(nvalid * ext) * (uint32_t)sizeof(T);
        const T *const st = reinterpret_cast<const T *>(sm + oXw);
        acp::bulk_s2g((side ? gr.dx : gr.dk) + at, st, bytes);
        acp::bulk_s2g((side ? gr.df : gr.dfk) + at, st + kC * ext, bytes);
        if (side == 0) acp::bulk_s2g(gr.dq + at, st + 2 * kC * ext, bytes);
        acp::bulk_commit();
        if (side == 1) acp::bulk_wait_read<0>();      // the next chunk's first barrier stands before Z's next write
      }
    }
  }
  if (tid == 0) acp::bulk_wait_all();
  if (fail) atomicExch(status, 1);
  if (tid == 0) {      // after a wait that gave up, copies may still be on their way into this CTA: bounded, let them land
    if (gates_pending) acp::mbar_wait(&barG, it & 1u);
    if (values_pending) acp::mbar_wait(&barV, it & 1u);
    if (nr_issued > 0) acp::mbar_wait(&barR, (nr_issued - 1) & 1u);
  }
  sync_all();
  if (warp == 0) umma::tmem_dealloc(tb, kTmemColsW);
}

}  // namespace

// mp: tensor maps of x, f, q, k, fk, dO (dense [items * T][D or K] arrays); outs: dx, df, dq, dk, dfk; rowflag per item
int lfw_wide_backward_main(const seq::Maps &mp, const void *state, const void *ckpt, const float *Rend, void *const outs[5],
                           int *rowflag, int64_t items, int64_t T_, int64_t D, int64_t K, int dtype, cudaStream_t st) {
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
    auto *const kern1 = &lfw_wide_bwd_kernel<TT>;                                                                \
    T2FW_ALLOW_SMEM(kern1, kSmemWB);                                                                             \
    const GradsW<TT> g{(TT *)outs[0], (TT *)outs[1], (TT *)outs[2], (TT *)outs[3], (TT *)outs[4]};               \
    T2FW_CHECK_CUDA(launch_dependent(lfw_wide_bwd_kernel<TT>, dim3(grid), dim3(kThreadsW), kSmemWB, st, mp,      \
                                     (const TT *)state, (const TT *)ckpt, Rend, g, rowflag, status, T_, nc,      \
                                     total, (int)D, (int)K));                                                    \
  } while (0)
  if (dtype == T2FW_F16) T2FW_LAUNCH(__half); else T2FW_LAUNCH(__nv_bfloat16);
#undef T2FW_LAUNCH
  T2FW_CHECK_LAUNCH(1);
  return T2FW_OK;
}

}  // namespace t2fw
