// Chunk-local state contributions of the decay rule on the tcgen05 tensor core (D = K = 64,
// 16-bit storage, chunks of 64 steps): the first phase of the chunked forward and backward, before
// the carry over the chunks.  Together with the carry it replaces the reference's sequential scans
// (t2fw/csrc/lfw_kernel.cu:18-59 and :61-102).
//
// Forward:  L_c[d][k] = sum_t (x_t[d] * prod_{j>t} f_j[d]) * (k_t[k] * prod_{j>t} fk_j[k])
//           the chunk's own contribution to the state at the chunk end (products run to the end
//           of the chunk: nothing is divided, and no factor exceeds the inputs for gates <= 1)
// Backward: G_c[d][k] = sum_s (dO_s[d] * prod_{j<=s} f_j[d]) * (q_s[k] * prod_{j<=s} fk_j[k])
//           the chunk's own contribution to the state gradient at the chunk start
// Both are one 64 x 64 x 64 contraction over the chunk's steps, plus the chunk's total decay
// vectors.  A chunk whose products exceed 2^100 is flagged (its batch row is redone by the scan
// kernels); products that underflow lose nothing.
//
// Persistent CTAs of 16 warps, two per SM, each on TWO chunks at a time: chunk 0 of the pair in one lane
// set of tensor memory, chunk 1 in the other (an M = 64 operand or accumulator takes half of the lanes), so
// nothing is stored twice.  Thread (chunk, feature, 16-step quarter) walks the gates of its feature on both
// sides with a running product that starts from the quarters between it and the anchoring end of the chunk:
// the d-side values become the A operand in tensor memory (row = feature), the k-side values a feature-major
// shared-memory tile; eight MMAs per chunk; the fp32 result leaves with 16-byte stores.
//
// What bounds it: the latency of its phases (issue slots 50 % busy, DRAM 28 %; two CTAs per SM hide part of it), loads most.
// Config B*H = 96, T = 1024 (1536 chunks): 30 -> 22.5 us per launch with cold caches against the version
// with one chunk per iteration (5.6 k warp instructions per chunk).
#include <mutex>

#include "lfw_c64.cuh"
#include "seq_layout.cuh"

namespace t2fw {

using namespace c64;


namespace {

constexpr int kThreadsL = 512;
constexpr int kCtasPerSmL = 2;
// shared-memory map (bytes from the 1024-byte aligned base), everything once per chunk of the pair
constexpr int oTk = 0;                             // [chunk] k-side tile [k][t]
constexpr int oQtL = oTk + 2 * kTile;              // [chunk][side][4][64] products of the quarters
constexpr int oRawL = oQtL + 2 * 2 * 4 * kDim * 4; // [chunk] val_d, gate_d, val_k, gate_k
constexpr int kSmemL = oRawL + 2 * 4 * kRawBytes + 1024;
static_assert(oRawL % 128 == 0, "bulk-copy destination alignment");
static_assert(kCtasPerSmL * (kSmemL + 1024) <= 227 * 1024, "two CTAs per SM");

constexpr int cA = 0, cD = 64;                     // tensor-memory columns, one lane set per chunk
constexpr int kTmemColsL = 128;

// kSuffix = true : value * (product of the gates AFTER the step, to the chunk end)   [forward]
// kSuffix = false: value * (product of the gates up to and including the step)       [backward]
template <typename T, bool kSuffix, bool kFused>
__global__ void __launch_bounds__(kThreadsL, kCtasPerSmL)
lfw_c64_local_kernel(const __grid_constant__ seq::Maps mp, float *__restrict__ M, float *__restrict__ Ac,
                     float *__restrict__ Gc, int *__restrict__ flags, int *__restrict__ rowflag, int items,
                     int *__restrict__ status, int64_t T_, int64_t nc, int64_t total) {
  extern __shared__ __align__(1024) unsigned char sm_raw[];
  unsigned char *sm = sm_raw + ((1024u - (umma::smem_u32(sm_raw) & 1023u)) & 1023u);
  __shared__ __align__(8) uint64_t barRaw, barM;
  __shared__ uint32_t tmem_slot;
  __shared__ int s_fail, s_bad2[2][2];

  const int tid = threadIdx.x, warp = uniform_warp_idx(), lane = tid & 31;
  // lane quarter of tensor memory, 16-step quarter of the chunk, chunk of the pair, row in the quarter
  const int q4 = warp & 3, tq = warp >> 2, h = lane >> 4, fl = lane & 15;
  const int feat = 16 * ((q4 + h) & 3) + fl;       // own feature, both sides
  const int t0 = 16 * tq;
  float *qtot = reinterpret_cast<float *>(sm + oQtL) + h * 2 * 4 * kDim + feat;      // own chunk and feature

  // tensors: 0 val_d, 1 gate_d, 2 val_k, 3 gate_k
  const float k_scale = kFused ? mp.q_scale : 1.f;
  auto valid_steps = [&](const ItemWalk &w, int64_t ci) {
    if (ci >= total) return 0;
    const int64_t left = T_ - (int64_t)w.c * kC;
    return (int)(left < kC ? left : kC);
  };
  auto issue_raw = [&](const ItemWalk *w, int64_t ci) {     // thread 0 only: one copy per tensor and chunk
    uint32_t bytes = 0;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int nv = valid_steps(w[e], ci + e);
      if (nv > 0) bytes += (kFused ? 3u : 4u) * ((mp.flags & seq::kContiguous) ? (uint32_t)nv * kDim * sizeof(T) : (uint32_t)kRawBytes);
    }
    acp::mbar_expect_tx(&barRaw, bytes);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int nv = valid_steps(w[e], ci + e);
      if (nv <= 0) continue;
      int b, hc;
      w[e].item(mp.heads, &b, &hc);
      const int row = (int)(b * T_ + w[e].c * kC);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (!(i == 1 && kFused)) seq::fetch_block<T>(mp, i, sm + oRawL + (e * 4 + i) * kRawBytes, row, hc, nv, &barRaw);
    }
  };

  if (tid == 0) {
    umma::mbar_init(&barRaw, 1);
    umma::mbar_init(&barM, 2);       // one commit per chunk
    umma::mbar_fence_init();
    s_fail = 0;
    s_bad2[0][0] = s_bad2[0][1] = s_bad2[1][0] = s_bad2[1][1] = 0;
  }
  if (warp == 0) umma::tmem_alloc(&tmem_slot, kTmemColsL);
  sync_all();
  dependency_wait();
  // row flags of the call (null: they are kept), set by the kernels behind this one
  if (rowflag != nullptr)
    for (int i = (int)(blockIdx.x * kThreadsL) + tid; i < items; i += (int)(gridDim.x * kThreadsL)) rowflag[i] = 0;
  const uint32_t tb = __shfl_sync(0xffffffffu, tmem_slot, 0);
  const uint32_t tl = umma::tmem_addr(tb, 32 * q4, 0);
  // (the blocks of a grid are problem rows of their own here)
  ItemWalk wn[2] = {ItemWalk(2 * blockIdx.x, 2 * gridDim.x, nc, 1), ItemWalk(2 * blockIdx.x + 1, 2 * gridDim.x, nc, 1)};
  bool raw_pending = false;      // thread 0
  if (2 * (int64_t)blockIdx.x < total && tid == 0) {
    issue_raw(wn, 2 * (int64_t)blockIdx.x);
    raw_pending = true;
  }
  const T *raw = reinterpret_cast<const T *>(sm + oRawL + h * 4 * kRawBytes) + t0 * kDim + feat;
  auto rawv = [&](int blk, int j) { return Elem<T>::ld(raw + blk * kC * kDim + j * kDim); };
  // k-side tile: row = own feature, 16-byte pieces of steps t0 ..
  unsigned char *const krow = sm + oTk + h * kTile + (t0 >> 5) * kColBlock + feat * 128;
  const int ksw = (((t0 >> 2) & 7) ^ (feat & 7)) << 4;

  uint32_t it = 0;
  for (int64_t ci = 2 * (int64_t)blockIdx.x; ci < total; ci += 2 * (int64_t)gridDim.x, ++it) {
    const int nv0 = valid_steps(wn[0], ci), nv1 = valid_steps(wn[1], ci + 1);
    wn[0].step();
    wn[1].step();
    const int nvalid = h ? nv1 : nv0;
    const bool partial = nv0 < kC || nv1 < kC;      // steps beyond the valid ones become identity steps
    int *s_bad = s_bad2[it & 1];

    if (acp::mbar_wait(&barRaw, it & 1u)) raw_pending = false;
    else s_fail = 1;

    // gates of one side, own feature and quarter
    auto gates = [&](int blk, bool kside, float (&g)[16]) {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        if (kFused && !kside) g[j] = 1.f;
        else g[j] = rawv(blk, j);
        if (kFused && kside) g[j] = seq::sigmoid_gate<T>(g[j]);
      }
      if (partial) {
#pragma unroll
        for (int j = 0; j < 16; ++j) g[j] = t0 + j < nvalid ? g[j] : 1.f;
      }
      if (kFused) return;             // (at least 1/8)
      float mn = kRangeHi;
#pragma unroll
      for (int j = 0; j < 16; j += 2) mn = min3_abs(mn, g[j], g[j + 1]);
      if (!(mn >= kTinyState)) {      // rare: some gate needs the clamp
#pragma unroll
        for (int j = 0; j < 16; ++j) g[j] = sanitize_gate(g[j]);
      }
    };
    auto product = [](const float (&g)[16]) {
      float p0 = g[0], p1 = g[1];
#pragma unroll
      for (int j = 2; j < 16; j += 2) { p0 *= g[j]; p1 *= g[j + 1]; }
      return p0 * p1;
    };
    // values of one side times the running product from the anchoring end; the chunk's total goes to `tot`
    auto walk = [&](int blk, bool kside, const float (&g)[16], const float *qt, float *tot, float (&w)[16]) {
#pragma unroll
      for (int j = 0; j < 16; ++j) w[j] = rawv(blk, j);
      if (kFused && kside) {
#pragma unroll
        for (int j = 0; j < 16; ++j) w[j] = seq::round_to<T>(w[j] * k_scale);
      }
      if (partial) {
#pragma unroll
        for (int j = 0; j < 16; ++j) w[j] = t0 + j < nvalid ? w[j] : 0.f;
      }
      if (kFused && !kside) {         // gates 1: the values as they are (exact in TF32)
        if (tq == (kSuffix ? 0 : 3) && nvalid > 0) tot[(size_t)(ci + h) * kDim + feat] = 1.f;
        return;
      }
      float s = 1.f, hi = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (kSuffix ? i > tq : i < tq) s *= qt[i * kDim];
      if (kSuffix) {
#pragma unroll
        for (int j = 15; j >= 0; --j) {
          const float e = w[j];
          w[j] = bias_tf32<kFused>(e * s);
          s *= g[j];
          hi = max3_abs(hi, s, e);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          s *= g[j];
          hi = max3_abs(hi, s, w[j]);
          w[j] = bias_tf32<kFused>(w[j] * s);
        }
      }
      if (!(hi <= kRangeHi)) s_bad[h] = 1;     // a product out of range, a gate or a value that is no finite number
      if (tq == (kSuffix ? 0 : 3) && nvalid > 0) tot[(size_t)(ci + h) * kDim + feat] = s;
    };

    float gk[16], gd[16];
    gates(3, true, gk);
    qtot[(4 + tq) * kDim] = product(gk);
    if (!kFused) {
      gates(1, false, gd);
      qtot[tq * kDim] = product(gd);
    }
    umma::named_barrier(1 + q4, 128);      // the four warps that hold the quarters of the same features
    {
      float w[16];
      walk(2, true, gk, qtot + 4 * kDim, Gc, w);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *reinterpret_cast<float4 *>(krow + (ksw ^ (j << 4))) = make_float4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
      walk(0, false, gd, qtot, Ac, w);
      umma::tmem_st16(tl + cA + t0, w);
    }
    umma::tmem_st_wait();
    umma::fence_async_smem();
    sync_all();       // operands complete, raw blocks consumed
    if (s_fail) break;

    if (warp < 2) {
      const uint32_t ls = umma::tmem_addr(tb, 16 * warp, 0);
      const uint64_t dk = desc_sw128(umma::smem_u32(sm + oTk) + warp * kTile);
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) mma_tf32_ts(ls + cD, ls + cA + 8 * ks, dk + kstep(ks), kIdesc64, ks > 0);
        umma::mma_commit(&barM);
      }
      __syncwarp();
    }
    if (tid == 0) {
      if (ci + 2 * (int64_t)gridDim.x < total) {
        issue_raw(wn, ci + 2 * (int64_t)gridDim.x);
        raw_pending = true;
      }
      flags[ci] = s_bad[0];
      if (nv1 > 0) flags[ci + 1] = s_bad[1];
      s_bad2[(it & 1) ^ 1][0] = s_bad2[(it & 1) ^ 1][1] = 0;
    }
    if (!umma::mbar_wait(&barM, it & 1u)) {
      s_fail = 1;
      if (nvalid > 0) flags[ci + h] = 1;      // results unusable: let the scan kernels redo the row
    }
    umma::fence_after_sync();
    {
      // Row d = own feature, columns k = t0 .. t0 + 15.  Stored straight from here, the lanes of a warp would write 32
      // different lines with every instruction; so the rows of a quarter pass through the k-side tile (consumed), its
      // 16-byte pieces XOR-ed with the row, and leave as whole rows, in memory with their pieces XOR-ed with (row % 8) too
      // (the gradient kernel reads them along rows and along columns).
      float v[16];
      umma::tmem_ld16(tl + cD + t0, v);
      umma::tmem_ld_wait();
      unsigned char *stg = sm + oTk + h * kTile + feat * 256;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *reinterpret_cast<float4 *>(stg + (((4 * tq + j) ^ (feat & 7)) << 4)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
      umma::named_barrier(1 + q4, 128);
#pragma unroll
      for (int i = 0; i < 4; ++i) {      // two rows per instruction: rows 8 (tq & 1) .. of this quarter's 16 in chunk tq >> 1
        const int e = tq >> 1, r = 16 * ((q4 + e) & 3) + 8 * (tq & 1) + 2 * i + h;
        const float4 o = *reinterpret_cast<const float4 *>(sm + oTk + e * kTile + r * 256 + ((fl ^ (r & 7)) << 4));
        if (e == 0 || nv1 > 0) *reinterpret_cast<float4 *>(M + ((size_t)(ci + e) * kDim + r) * kDim + 4 * (fl ^ (r & 7))) = o;
      }
    }
    // No full barrier here: before the next one the next pair writes only products of quarters, which nobody reads any
    // more, and, after the quarter's own barrier, the operand rows of its features, which only this quarter's warps used.
    umma::fence_before_sync();
  }
  __syncthreads();      // s_fail of the last pair is visible
  if (tid == 0 && s_fail) {
    atomicExch(status, 1);
    if (raw_pending) acp::mbar_wait(&barRaw, it & 1u);      // bounded: let copies that are still in flight land
  }
  sync_all();
  if (warp == 0) umma::tmem_dealloc(tb, kTmemColsL);
}

}  // namespace

__device__ int g_umma_status = 0;

namespace {
int *g_umma_status_addr[64] = {};
int g_sm_count[64] = {};
std::mutex g_status_mutex;
}

// device address of the status word kernels set when a bounded wait expires
int lfw_chunk_status_ptr(int **out) {
  int dev = 0;
  T2FW_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) {
    set_error("device index %d out of range", dev);
    return T2FW_ERR_UNSUPPORTED;
  }
  std::lock_guard<std::mutex> lock(g_status_mutex);
  if (g_umma_status_addr[dev] == nullptr) {
    int n = 0;
    T2FW_CHECK_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    void *p = nullptr;
    T2FW_CHECK_CUDA(cudaGetSymbolAddress(&p, g_umma_status));
    g_sm_count[dev] = n;                               // filled before the address is published
    g_umma_status_addr[dev] = static_cast<int *>(p);
  }
  *out = g_umma_status_addr[dev];
  return T2FW_OK;
}

// number of SMs of the current device (cached with the status address)
int lfw_chunk_sm_count(int *out) {
  int *unused = nullptr;
  const int rc = lfw_chunk_status_ptr(&unused);
  if (rc != T2FW_OK) return rc;
  int dev = 0;
  T2FW_CHECK_CUDA(cudaGetDevice(&dev));
  *out = g_sm_count[dev];
  return T2FW_OK;
}

int lfw_chunk_umma_status() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_umma_status, sizeof(int)) != cudaSuccess) return -1;
  return v;
}

// Forward flavour: M = L_c from (x, f) and (k, fk).  Backward flavour: M = G_c from (dO, f), (q, fk).
// mp describes the four tensors in that order (mp.q_scale applies to the third one).
int lfw_chunk_local_umma(bool backward, const seq::Maps &mp, float *M, float *Ac, float *Gc, int *flags, int *rowflag,
                         int64_t BH, int64_t T_, int dtype, cudaStream_t st) {
  const int64_t nc = ceil_div64(T_, kC), total = BH * nc;
  int *status = nullptr;
  int rc = lfw_chunk_status_ptr(&status);
  if (rc != T2FW_OK) return rc;
  int sms = 0;
  rc = lfw_chunk_sm_count(&sms);
  if (rc != T2FW_OK) return rc;
  const int64_t max_ctas = (int64_t)sms * kCtasPerSmL;
  const int64_t pairs = (total + 1) / 2;
  const unsigned grid = (unsigned)(pairs < max_ctas ? pairs : max_ctas);
#define T2FW_LAUNCH(TT, SUF, FF)                                                                          \
  do {                                                                                                \
    auto *const kern1 = &lfw_c64_local_kernel<TT, SUF, FF>; \
    T2FW_ALLOW_SMEM(kern1, kSmemL);       \
    T2FW_CHECK_CUDA(launch_dependent(lfw_c64_local_kernel<TT, SUF, FF>, dim3(grid), dim3(kThreadsL), kSmemL, st, mp, M, \
                                     Ac, Gc, flags, rowflag, (int)(BH / mp.nsub), status, T_, nc, total));                         \
  } while (0)
  const bool fused = (mp.flags & seq::kFusedLayer) != 0;
#define T2FW_FUSED(TT, SUF)                                                   \
  do {                                                                        \
    if (fused) T2FW_LAUNCH(TT, SUF, true); else T2FW_LAUNCH(TT, SUF, false);  \
  } while (0)
  if (dtype == T2FW_F16) {
    if (backward) T2FW_FUSED(__half, false); else T2FW_FUSED(__half, true);
  } else {
    if (backward) T2FW_FUSED(__nv_bfloat16, false); else T2FW_FUSED(__nv_bfloat16, true);
  }
#undef T2FW_FUSED
#undef T2FW_LAUNCH
  T2FW_CHECK_LAUNCH(1);
  return T2FW_OK;
}

}  // namespace t2fw

