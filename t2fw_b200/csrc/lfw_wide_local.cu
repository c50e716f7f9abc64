// Chunk-local state contributions of the decay rule for states of up to 128 x 128 (D, K = 64 or 128, one of them 128; 16-bit
// storage, chunks of 64 steps): the first phase of the chunked forward and backward, what lfw_c64_local.cu is for 64 x 64
// states (formulas there).
//
// As a grid of 64 x 64 blocks every block would read and scale its two windows again.  Here a chunk's operands are built once
// and one chain of products forms all its blocks: d features in the 128 lanes of tensor memory, k features in its columns.
// Results and decay vectors leave in the layout of the blocks, which the carry goes through as before.
//
// Persistent CTAs of 16 warps, two per SM; thread (feature, 16-step quarter) serves the feature with its number on both sides.
// 16 rows x 16384 steps, 128 x 128 (4096 chunks): 162 us as a grid of blocks -> 136 us; the results alone are 268 MB.  The range
// test's look at the values costs 2 (142 -> 144, in turn on one box).
#include "lfw_c64.cuh"
#include "seq_layout.cuh"

namespace t2fw {

using namespace c64;

int lfw_chunk_status_ptr(int **out);   // lfw_c64_local.cu
int lfw_chunk_sm_count(int *out);

namespace {

constexpr int kThreadsW = 512;
constexpr int kCtasPerSmW = 2;
constexpr int kWide = 128;                         // features of a side, the upper half possibly unused
constexpr int kColBlockW = kWide * 128;            // bytes of one 32-column block of the k-side tile
// shared-memory map (bytes from the 1024-byte aligned base)
constexpr int oTkW = 0;                            // k-side tile [k][t]; then results on their way out
constexpr int oQtW = oTkW + 2 * kColBlockW;        // [d, k][4][128] products of the quarters
constexpr int oRawLW = oQtW + 2 * 4 * kWide * 4;   // [val_d, gate_d, val_k, gate_k][window]
constexpr int kSmemLW = oRawLW + 8 * kRawBytes + 1024;
static_assert(oRawLW % 128 == 0, "copy destination alignment");
static_assert(kCtasPerSmW * (kSmemLW + 1024) <= 227 * 1024, "two CTAs per SM");
constexpr int cAw = 0, cDw = 64;                   // tensor-memory columns
constexpr int kTmemColsLW = 256;

// kSuffix = true : value * (product of the gates AFTER the step, to the chunk end)   [forward]
// kSuffix = false: value * (product of the gates up to and including the step)       [backward]
template <typename T, bool kSuffix>
__global__ void __launch_bounds__(kThreadsW, kCtasPerSmW)
lfw_wide_local_kernel(const __grid_constant__ seq::Maps mp, float *__restrict__ M, float *__restrict__ Ac, float *__restrict__ Gc,
                      int *__restrict__ flags, int *__restrict__ rowflag, int items, int *__restrict__ status, int64_t T_,
                      int64_t nc, int64_t total, int nd, int nk) {
  extern __shared__ __align__(1024) unsigned char sm_raw[];
  unsigned char *sm = sm_raw + ((1024u - (umma::smem_u32(sm_raw) & 1023u)) & 1023u);
  __shared__ __align__(8) uint64_t barRaw, barM;
  __shared__ uint32_t tmem_slot;
  __shared__ int s_bad2[2];

  const int tid = threadIdx.x, warp = uniform_warp_idx(), lane = tid & 31;
  const int q4 = warp & 3, tq = warp >> 2, t0 = 16 * tq;
  const int feat = 32 * q4 + lane, win = feat >> 6, wf = feat & 63;      // own feature on both sides: window, number in it
  const bool has_d = win < nd, has_k = win < nk;
  float *qtot = reinterpret_cast<float *>(sm + oQtW) + feat;
  auto issue_raw = [&](const ItemWalk &w) {     // thread 0 only
    const int row = (int)(w.row * T_ + w.c * kC);
    acp::mbar_expect_tx(&barRaw, (uint32_t)(2 * (nd + nk)) * kRawBytes);
#pragma unroll 1
    for (int i = 0; i < 4; ++i)
      for (int j = 0; j < (i < 2 ? nd : nk); ++j) seq::load_block(sm + oRawLW + (2 * i + j) * kRawBytes, &mp.m[i], 64 * j, row, &barRaw);
  };

  if (tid == 0) {
    umma::mbar_init(&barRaw, 1);
    umma::mbar_init(&barM, 1);
    umma::mbar_fence_init();
    s_bad2[0] = s_bad2[1] = 0;
  }
  if (warp == 0) umma::tmem_alloc(&tmem_slot, kTmemColsLW);
  sync_all();
  dependency_wait();
  // row flags of the call (null: they are kept), set by the kernels behind this one
  if (rowflag != nullptr)
    for (int i = (int)(blockIdx.x * kThreadsW) + tid; i < items; i += (int)(gridDim.x * kThreadsW)) rowflag[i] = 0;
  const uint32_t tb = __shfl_sync(0xffffffffu, tmem_slot, 0);
  const uint32_t tl = umma::tmem_addr(tb, 32 * q4, 0);
  const uint32_t idesc = umma::make_idesc_tf32(128, 64 * nk, false, false);
  ItemWalk wn(blockIdx.x, gridDim.x, nc, 1);
  bool raw_pending = false;      // thread 0
  if (wn.unit < total && tid == 0) {
    issue_raw(wn);
    raw_pending = true;
  }
  const T *raw = reinterpret_cast<const T *>(sm + oRawLW + win * kRawBytes) + t0 * kDim + wf;
  // k-side tile: row = own feature, 16-byte pieces of steps t0 ..
  unsigned char *const krow = sm + oTkW + (t0 >> 5) * kColBlockW + feat * 128;
  const int ksw = (((t0 >> 2) & 7) ^ (feat & 7)) << 4;

  int fail = 0;                  // a wait of this thread gave up
  uint32_t it = 0;
  for (; wn.unit < total; ++it) {
    const ItemWalk w = wn;
    wn.step();
    const int64_t left = T_ - (int64_t)w.c * kC;
    const int nvalid = (int)(left < kC ? left : kC);      // steps beyond the valid ones become identity steps
    int &s_bad = s_bad2[it & 1];

    if (acp::mbar_wait(&barRaw, it & 1u)) raw_pending = false;
    else fail = 1;

    auto gates = [&](int blk, bool has, float (&g)[16]) {
      const T *p = raw + 2 * blk * kC * kDim;
      float mn = kRangeHi;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        g[j] = has && t0 + j < nvalid ? Elem<T>::ld(p + j * kDim) : 1.f;
        if (j & 1) mn = min3_abs(mn, g[j - 1], g[j]);
      }
      if (!(mn >= kTinyState)) {      // rare: some gate needs the clamp
#pragma unroll
        for (int j = 0; j < 16; ++j) g[j] = sanitize_gate(g[j]);
      }
      float p0 = g[0], p1 = g[1];
#pragma unroll
      for (int j = 2; j < 16; j += 2) { p0 *= g[j]; p1 *= g[j + 1]; }
      return p0 * p1;
    };
    // values of one side times the running product from the anchoring end, and the chunk's total
    auto walk = [&](int blk, bool has, const float (&g)[16], const float *qt, float (&v)[16]) {
      const T *p = raw + 2 * blk * kC * kDim;
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = has && t0 + j < nvalid ? Elem<T>::ld(p + j * kDim) : 0.f;
      float s = 1.f, hi = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (kSuffix ? i > tq : i < tq) s *= qt[i * kWide];
      if (kSuffix) {
#pragma unroll
        for (int j = 15; j >= 0; --j) {
          const float e = v[j];
          v[j] = bias_tf32(e * s);
          s *= g[j];
          hi = max3_abs(hi, s, e);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          s *= g[j];
          hi = max3_abs(hi, s, v[j]);
          v[j] = bias_tf32(v[j] * s);
        }
      }
      if (!(hi <= kRangeHi)) s_bad = 1;     // a product out of range, a gate or a value that is no finite number
      return s;
    };
    const bool edge = tq == (kSuffix ? 0 : 3);      // this quarter ends with the chunk's total
    const size_t block0 = (size_t)w.row * nd * nk;  // problem row of block (0, 0); block (i, j) is i * nk + j further on
    {
      float gk[16], gd[16];
      qtot[(4 + tq) * kWide] = gates(3, has_k, gk);
      qtot[tq * kWide] = gates(1, has_d, gd);
      umma::named_barrier(1 + q4, 128);      // the four warps that hold the quarters of the same features
      float v[16];
      float s = walk(2, has_k, gk, qtot + 4 * kWide, v);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *reinterpret_cast<float4 *>(krow + (ksw ^ (j << 4))) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
      if (edge && has_k)
        for (int i = 0; i < nd; ++i) Gc[((block0 + i * nk + win) * nc + w.c) * kDim + wf] = s;
      s = walk(0, has_d, gd, qtot, v);
      if (edge && has_d)
        for (int j = 0; j < nk; ++j) Ac[((block0 + win * nk + j) * nc + w.c) * kDim + wf] = s;
      __syncwarp();
      umma::tmem_st16(tl + cAw + t0, v);
    }
    umma::tmem_st_wait();
    umma::fence_async_smem();
    umma::fence_before_sync();
    const bool stop = __syncthreads_or(fail) != 0;      // operands complete, raw blocks consumed
    umma::fence_after_sync();
    if (stop) break;

    if (warp == 0) {
      const uint64_t dk = desc_sw128(umma::smem_u32(sm + oTkW));
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
          mma_tf32_ts(tb + cDw, tb + cAw + 8 * ks, dk + (uint64_t)(((ks >> 2) * kColBlockW + (ks & 3) * 32) >> 4), idesc, ks > 0);
        umma::mma_commit(&barM);
      }
      __syncwarp();
    }
    if (tid == 0) {
      if (wn.unit < total) {
        issue_raw(wn);
        raw_pending = true;
      }
      for (int i = 0; i < nd * nk; ++i) flags[(block0 + i) * nc + w.c] = s_bad;
      s_bad2[(it & 1) ^ 1] = 0;
    }
    if (!umma::mbar_wait(&barM, it & 1u)) {
      fail = 1;
      flags[block0 * nc + w.c] = 1;      // results unusable: let the scan kernels redo the row
    }
    umma::fence_after_sync();
    for (int j = 0; j < nk; ++j) {
      // Row d = own feature, columns k = 64 j + t0 .. + 15.  The rows of a quarter pass through the k-side tile (consumed), their
      // 16-byte pieces XOR-ed with (row % 8), and leave as whole rows just so: the readers expect them in that order.
      float v[16];
      umma::tmem_ld16(tl + cDw + 64 * j + t0, v);
      umma::tmem_ld_wait();
      unsigned char *stg = sm + oTkW + feat * 256;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4 *>(stg + (((4 * tq + i) ^ (feat & 7)) << 4)) = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
      umma::named_barrier(1 + q4, 128);
#pragma unroll
      for (int i = 0; i < 4; ++i) {      // two rows per instruction
        const int r = 32 * q4 + 8 * tq + 2 * i + (lane >> 4), p = lane & 15;
        if (r < 64 * nd)
          *reinterpret_cast<float4 *>(M + (((block0 + (r >> 6) * nk + j) * nc + w.c) * kDim + (r & 63)) * kDim + 4 * p) =
              *reinterpret_cast<const float4 *>(sm + oTkW + r * 256 + (p << 4));
      }
      umma::named_barrier(1 + q4, 128);
    }
    // A full barrier: the next chunk's tile rows are 128 bytes, these results' 256, so that a quarter's operands go where
    // another quarter's results may still be on their way out.
    umma::fence_before_sync();
    __syncthreads();
  }
  if (fail) atomicExch(status, 1);
  if (tid == 0 && raw_pending) acp::mbar_wait(&barRaw, it & 1u);      // bounded: let copies that are still in flight land
  sync_all();
  if (warp == 0) umma::tmem_dealloc(tb, kTmemColsLW);
}

}  // namespace

// Forward flavour: M = L_c from (x, f) and (k, fk).  Backward flavour: M = G_c from (dO, f), (q, fk).  mp describes the four
// tensors in that order (dense [items * T][D or K] arrays).
int lfw_wide_local(bool backward, const seq::Maps &mp, float *M, float *Ac, float *Gc, int *flags, int *rowflag, int64_t items,
                   int64_t T_, int64_t D, int64_t K, int dtype, cudaStream_t st) {
  const int64_t nc = ceil_div64(T_, kC), total = items * nc;
  int *status = nullptr;
  int rc = lfw_chunk_status_ptr(&status);
  if (rc != T2FW_OK) return rc;
  int sms = 0;
  rc = lfw_chunk_sm_count(&sms);
  if (rc != T2FW_OK) return rc;
  const int64_t max_ctas = (int64_t)sms * kCtasPerSmW;
  const unsigned grid = (unsigned)(total < max_ctas ? total : max_ctas);
#define T2FW_LAUNCH(TT, SUF)                                                                                        \
  do {                                                                                                              \
    auto *const kern1 = &lfw_wide_local_kernel<TT, SUF>;                                                            \
    T2FW_ALLOW_SMEM(kern1, kSmemLW);                                                                                \
    T2FW_CHECK_CUDA(launch_dependent(lfw_wide_local_kernel<TT, SUF>, dim3(grid), dim3(kThreadsW), kSmemLW, st, mp, M, Ac, Gc, \
                                     flags, rowflag, (int)items, status, T_, nc, total, (int)(D / kDim), (int)(K / kDim)));   \
  } while (0)
  if (dtype == T2FW_F16) {
    if (backward) T2FW_LAUNCH(__half, false); else T2FW_LAUNCH(__half, true);
  } else {
    if (backward) T2FW_LAUNCH(__nv_bfloat16, false); else T2FW_LAUNCH(__nv_bfloat16, true);
  }
#undef T2FW_LAUNCH
  T2FW_CHECK_LAUNCH(1);
  return T2FW_OK;
}

}  // namespace t2fw
