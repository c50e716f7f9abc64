// Chunked decay rule for D = K = 64, 16-bit storage, checkpoint interval 64: the carry over the
// chunks and the launch sequences of the forward and the backward call.
//
// Forward (replaces t2fw/csrc/lfw_kernel.cu:18-59 and the output einsum t2fw/csrc/lfw.cpp:45):
//   1. lfw_c64_local_kernel<.., true>   per (row, chunk): L_c, the chunk's own contribution to the
//      state at its end, and the chunk's total decay vectors
//   2. lfw_c64_carry_kernel<.., true>   elementwise over chunks: S_{c+1} = (Ac Gc^T) .* S_c + L_c, written
//      as the 16-bit checkpoints (slot c = state after chunk c; the last slot is the next state)
//   3. lfw_c64_fwd_kernel               per (row, chunk): the outputs from the chunk's start state
// Backward (replaces t2fw/csrc/lfw_kernel.cu:61-102 and t2fw/csrc/lfw.cpp:84-93):
//   1. lfw_c64_local_kernel<.., false>  G_c, the chunk's own contribution to the state gradient at its start
//   2. lfw_c64_carry_kernel<.., false>  from the last chunk down: R_end(c-1) = (Ac Gc^T) .* R_end(c) + G_c,
//      stored in place of G_c (fp32); what is left after chunk 0 is d_state
//   3. lfw_c64_bwd_kernel               per (row, chunk): d_x, d_f, d_q, d_k, d_f_key
// Scratch (floats): M[B][nc][64][64], 16-byte pieces of a row XOR-ed with (row % 8) | Ac[B][nc][64] | Gc[B][nc][64] |
// flags[B][nc] (int) | rowflag[B] (int).  A flagged row (gate products outside the range of the factored form, values that are no
// finite numbers) is recomputed by the scan kernels afterwards.
// States of up to 128 x 128 (D, K = 64 or 128) have kernels of their own for 1. and 3. (lfw_wide_*.cu) and share the carry, whose
// rows are their 64 x 64 blocks.
// Larger ones (D, K multiples of 64): the recurrence never mixes state rows or columns, so a D x K state
// is a (D/64) x (K/64) grid of independent blocks, problem rows of their own for the kernels (B above counts them);
// block (i, j) reads the d-side vectors' window i and the k-side vectors' window j in place, states and checkpoints are
// read and written in place too, and what leaves the state is summed over the other axis' blocks by the output and
// gradient kernels, whose CTAs walk all blocks of a chunk: a thread adds to what it wrote itself.  Flags are then per batch
// item.
#include "lfw_c64.cuh"
#include "seq_layout.cuh"

namespace t2fw {

using namespace c64;

int lfw_chunk_local_umma(bool backward, const seq::Maps &mp, float *M, float *Ac, float *Gc, int *flags, int *rowflag,
                         int64_t BH, int64_t T_, int dtype, cudaStream_t st);
int lfw_c64_forward_out(const seq::Maps &mp, const void *state, const void *ckpt, void *out, int64_t out_ld,
                        int out_col, int *rowflag, int64_t BH, int64_t T_, int dtype, cudaStream_t st);
int lfw_c64_backward_main(const seq::Maps &mp, const void *state, const void *ckpt, const float *Rend,
                          void *const outs[5], const int64_t out_ld[5], const int out_col[5], int *rowflag,
                          int64_t BH, int64_t T_, int dtype, cudaStream_t st);
int lfw_chunk_sm_count(int *out);   // lfw_c64_local.cu
int lfw_wide_forward_out(const seq::Maps &mp, const void *state, const void *ckpt, void *out, int *rowflag, int64_t items,
                         int64_t T_, int64_t D, int64_t K, int dtype, cudaStream_t st);      // lfw_wide_fwd.cu
int lfw_wide_local(bool backward, const seq::Maps &mp, float *M, float *Ac, float *Gc, int *flags, int *rowflag, int64_t items,
                   int64_t T_, int64_t D, int64_t K, int dtype, cudaStream_t st);
int lfw_wide_backward_main(const seq::Maps &mp, const void *state, const void *ckpt, const float *Rend, void *const outs[5],
                           int *rowflag, int64_t items, int64_t T_, int64_t D, int64_t K, int dtype, cudaStream_t st);

namespace {

struct Scratch {
  float *M, *Ac, *Gc;
  int *flags, *rowflag;
  void *ck_all;      // 16-bit states after every chunk [B][nc][64][64]; only for checkpoint intervals > 64
};

inline size_t scratch_floats(int64_t B, int64_t nc) {
  return (size_t)B * nc * kDim * kDim + 2 * (size_t)B * nc * kDim + (size_t)B * nc + (size_t)B;
}

inline size_t scratch_bytes(int64_t B, int64_t nc, int64_t ckpt_every) {
  size_t n = align_up(scratch_floats(B, nc) * sizeof(float), 256);
  if (ckpt_every != kC) n += align_up((size_t)B * nc * kDim * kDim * 2, 256);
  return n;
}

inline Scratch carve(void *scratch, int64_t B, int64_t nc) {
  Scratch s;
  s.M = static_cast<float *>(scratch);
  s.Ac = s.M + (size_t)B * nc * kDim * kDim;
  s.Gc = s.Ac + (size_t)B * nc * kDim;
  s.flags = reinterpret_cast<int *>(s.Gc + (size_t)B * nc * kDim);
  s.rowflag = s.flags + (size_t)B * nc;
  s.ck_all = static_cast<unsigned char *>(scratch) + align_up(scratch_floats(B, nc) * sizeof(float), 256);
  return s;
}

constexpr int kCarryThreads = 256;

// kCols consecutive values of a row: fp32 scratch and 16-bit states
template <int kCols> struct Piece;
template <> struct Piece<4> { using F = float4; using H = uint2; };
template <> struct Piece<2> { using F = float2; using H = uint32_t; };
__device__ __forceinline__ float2 widen(__half2 v) { return __half22float2(v); }
__device__ __forceinline__ float2 widen(__nv_bfloat162 v) { return __bfloat1622float2(v); }
__device__ __forceinline__ void narrow(__half2 *p, float a, float b) { *p = __floats2half2_rn(a, b); }
__device__ __forceinline__ void narrow(__nv_bfloat162 *p, float a, float b) { *p = __floats2bfloat162_rn(a, b); }
template <typename T> struct Two;
template <> struct Two<__half> { using type = __half2; };
template <> struct Two<__nv_bfloat16> { using type = __nv_bfloat162; };
template <typename T, int kCols>
__device__ __forceinline__ void load16(float (&v)[kCols], const T *p) {
  const typename Piece<kCols>::H u = *reinterpret_cast<const typename Piece<kCols>::H *>(p);
#pragma unroll
  for (int i = 0; i < kCols / 2; ++i) {
    const float2 w = widen(reinterpret_cast<const typename Two<T>::type *>(&u)[i]);
    v[2 * i] = w.x;
    v[2 * i + 1] = w.y;
  }
}
template <typename T, int kCols>
__device__ __forceinline__ void store16(T *p, const float (&v)[kCols]) {
  typename Piece<kCols>::H u;
#pragma unroll
  for (int i = 0; i < kCols / 2; ++i) narrow(reinterpret_cast<typename Two<T>::type *>(&u) + i, v[2 * i], v[2 * i + 1]);
  *reinterpret_cast<typename Piece<kCols>::H *>(p) = u;
}

// States of the call: one 64 x 64 block per problem row (nsub = 1), or a grid of nsub blocks per item
struct Grid2D {
  int nsub, nk;
  int item, ld;          // elements of a state, row stride
};

// One thread per (row, d, kCols consecutive k); a block covers 4 kCols state rows of one batch row.  The
// recurrence over the chunks is a dependent chain, so the loads of up to 16 chunks are all issued
// before the chain starts (one round of memory latency per 16 chunks); the decay vectors of those
// chunks are shared by the block and go through shared memory.
//   kFwd:  S_{c+1} = (Ac Gc^T) S_c + L_c from the caller's state; checkpoint slot c = S_{c+1}
//   !kFwd: R_end(c-1) = (Ac Gc^T) R_end(c) + G_c from grad_state, last chunk first; G_c is
//          overwritten with R_end(c); the value left after chunk 0 is d_state
template <typename T, bool kFwd, int kCols>
__global__ void __launch_bounds__(kCarryThreads, kCols == 4 ? 3 : 5)
lfw_c64_carry_kernel(const T *__restrict__ init, float *__restrict__ M, const float *__restrict__ Ac,
                     const float *__restrict__ Gc, const int *__restrict__ flags, int *__restrict__ rowflag,
                     T *__restrict__ out, const Grid2D gr, int64_t nc) {
  using F = typename Piece<kCols>::F;
  constexpr int kBatch = 16;                                 // chunks whose loads are in flight together
  constexpr int kCarryRows = kCarryThreads / (kDim / kCols);         // state rows of the block
  __shared__ float a_s[kBatch][kCarryRows];
  __shared__ __align__(16) float g_s[kBatch][kDim];
  const int tid = threadIdx.x;
  dependency_wait();
  const int64_t b = blockIdx.x / (kDim / kCarryRows);
  const int d0 = (int)(blockIdx.x % (kDim / kCarryRows)) * kCarryRows;
  // (M's rows lie with their 16-byte pieces XOR-ed with (row % 8): a thread's piece of M holds columns k0 ..)
  const int dl = tid / (kDim / kCols), d = d0 + dl, kp = tid % (kDim / kCols) * kCols, k0 = kp ^ ((d & 7) << 2);
  // where this block of the states lies: item, offset inside one state, row stride
  const int item = gr.nsub == 1 ? (int)b : (int)b / gr.nsub, sub = (int)b - item * gr.nsub;
  const int in_state = (sub / gr.nk * kDim + d) * gr.ld + sub % gr.nk * kDim + k0, whole = gr.item;
  // init may be null: the carry then starts from zero (the summary of a sequence segment)
  alignas(16) float S[kCols] = {};
  if (init != nullptr) load16<T, kCols>(S, init + (size_t)item * whole + in_state);
  int any = 0;
  const int n = (int)nc;
  T *op = out + (size_t)item * (kFwd ? nc : 1) * whole + in_state;      // forward: the block's next checkpoint
  // this thread's values of the first chunk of the walk; one chunk further along it per step
  float *mp = M + (((size_t)b * nc + (kFwd ? 0 : nc - 1)) * kDim + d) * kDim + kp;
  constexpr int kNext = (kFwd ? 1 : -1) * kDim * kDim;
  const float *ac = Ac + (size_t)b * nc * kDim + d0, *gc = Gc + (size_t)b * nc * kDim;
  for (int c0 = 0; c0 < n; c0 += kBatch) {
    F l[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j)
      l[j] = *reinterpret_cast<const F *>(mp + (c0 + j < n ? j : 0) * kNext);
    __syncthreads();      // the previous batch's decay vectors are no longer read
    for (int i = tid; i < kBatch * (kCarryRows + kDim); i += kCarryThreads) {
      const int j = i / (kCarryRows + kDim), r = i % (kCarryRows + kDim);
      int c = c0 + j < n ? c0 + j : n - 1;
      if (!kFwd) c = n - 1 - c;
      if (r < kCarryRows) a_s[j][r] = ac[c * kDim + r];
      else g_s[j][r - kCarryRows] = gc[c * kDim + r - kCarryRows];
    }
    if (d0 == 0 && tid < kBatch && c0 + tid < n) any |= flags[(size_t)b * nc + c0 + tid];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      if (c0 + j < n) {
        if (!kFwd) *reinterpret_cast<F *>(mp) = *reinterpret_cast<const F *>(S);
        const float a = a_s[j][dl];
        const F g = *reinterpret_cast<const F *>(&g_s[j][k0]);
#pragma unroll
        for (int i = 0; i < kCols; ++i) S[i] = a * reinterpret_cast<const float *>(&g)[i] * S[i] + reinterpret_cast<const float *>(&l[j])[i];
        if (kFwd) {
          store16<T, kCols>(op, S);
          op += whole;
        }
        mp += kNext;
      }
    }
  }
  if (!kFwd) store16<T, kCols>(op, S);
  if (any || !all_finite(S)) atomicExch(rowflag + item, 1);      // (a NaN or an infinity that has got into a state stays in it)
}

// The carry of BH problem rows.  Two values per thread make twice as many blocks (five of them share an SM, of the others three),
// so that one block's loads run under another's chain; where one round of loads holds all chunks, or the rows alone fill the
// chip, their smaller accesses cost more than that gives, and with few rounds so does a second wave of blocks that four values do
// not need.  The kernel with two / four values, us: 64 rows x 256 chunks 141 / 164, 96 x 16 11.3 / 10.3.  Training calls, 64 x 64, fp16: rows x chunks
//     16 x 64   148.8 / 151.0     64 x 20  155.8 / 156.6     96 x 20  212.5 / 205.8     128 x 20  271.1 / 272.6
//     64 x 64   418.9 / 426.8     96 x 32  310.4 / 311.0    128 x 64  789.3 / 817.1     192 x 64 1156.4 / 1151.4
// (148 SMs: rows 93 to 111 have the second wave; beyond 128 rows neither is ahead by more than 2 %).
template <typename T, bool kFwd>
cudaError_t launch_carry(const T *init, float *M, const float *Ac, const float *Gc, const int *flags, int *rowflag, T *out,
                         const Grid2D &gr, int64_t BH, int64_t nc, cudaStream_t st) {
  int n_sm = 0;
  if (lfw_chunk_sm_count(&n_sm) != T2FW_OK) return cudaErrorUnknown;
  const bool second_wave = BH * 8 > 5 * n_sm && BH * 4 <= 3 * n_sm;      // with two values only
  if (nc > 16 && BH <= 128 && !(second_wave && nc < 32))
    return launch_dependent(lfw_c64_carry_kernel<T, kFwd, 2>, dim3((unsigned)(BH * 8)), dim3(kCarryThreads), 0, st, init, M, Ac,
                            Gc, flags, rowflag, out, gr, nc);
  return launch_dependent(lfw_c64_carry_kernel<T, kFwd, 4>, dim3((unsigned)(BH * 4)), dim3(kCarryThreads), 0, st, init, M, Ac, Gc,
                          flags, rowflag, out, gr, nc);
}

// Checkpoint interval of m chunks: slot j of the caller's checkpoints = state after chunk
// min((j + 1) m, nc) - 1 of the per-chunk states.
template <typename T>
__global__ void __launch_bounds__(256)
lfw_c64_pick_ckpt_kernel(const T *__restrict__ all, T *__restrict__ ckpt, int64_t B, int64_t nc, int64_t m,
                         int64_t slots, int64_t kVec) {      // kVec: 16-byte pieces of one state
  const int64_t n = B * slots * kVec;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t v = i % kVec, j = (i / kVec) % slots, b = i / (kVec * slots);
    const int64_t c = ((j + 1) * m < nc ? (j + 1) * m : nc) - 1;
    reinterpret_cast<uint4 *>(ckpt)[(b * slots + j) * kVec + v] =
        reinterpret_cast<const uint4 *>(all)[(b * nc + c) * kVec + v];
  }
}

// One sequence tensor of a call: base pointer, width of a row (elements), column of sub-item 0,
// and which 64-column window sub-item h reads: (h / hdiv) % hmod (0, 0 = head h of `heads`).
struct Tensor2D {
  const void *p;
  int64_t width;
  int col;
  int hdiv = 0, hmod = 0;
};

// Tensor maps for a kernel whose inputs are `ts` (in the kernel's order); rows = batch items x T.
int build_maps(seq::Maps &mp, const Tensor2D *ts, int n, int64_t rows, int heads, int flags, float q_scale) {
  if (rows >= (1ll << 31) || rows * heads / kC + rows * heads >= (1ll << 31)) {
    set_error("chunked decay rule: batch x time = %lld rows exceed the copy engine's 31-bit coordinates", (long long)rows);
    return T2FW_ERR_UNSUPPORTED;
  }
  bool dense = heads == 1;
  for (int i = 0; i < n; ++i) dense = dense && (ts[i].p == nullptr || (ts[i].width == kDim && ts[i].col == 0));
  if (dense) flags |= seq::kContiguous;               // [rows][64] arrays: linear copies, no tensor maps needed
  for (int i = 0; i < n; ++i) {
    mp.col[i] = ts[i].col;
    mp.base[i] = ts[i].p;
    mp.hdiv[i] = ts[i].hdiv > 0 ? ts[i].hdiv : 1;
    mp.hmod[i] = ts[i].hmod > 0 ? ts[i].hmod : heads;
    if (ts[i].p == nullptr || dense) continue;        // constant tensor (unit forget gate) / no map needed
    bool shared = false;
    for (int j = 0; j < i && !shared; ++j)
      if (ts[j].p == ts[i].p && ts[j].width == ts[i].width) {
        mp.m[i] = mp.m[j];                            // several tensors inside one array
        shared = true;
      }
    if (!shared) {
      const int rc = seq::make_map(&mp.m[i], ts[i].p, (uint64_t)rows, (uint64_t)ts[i].width, (uint64_t)ts[i].width);
      if (rc != T2FW_OK) return rc;
    }
  }
  mp.heads = heads;
  mp.flags = flags;
  mp.q_scale = q_scale;
  return T2FW_OK;
}

// The tensors of a call, plain or fused: x, f, q, k, fk, dO in that order (f.p null = constant 1).
struct Call {
  Tensor2D x, f, q, k, fk, go;
  int64_t B, T_;        // batch items, steps;  problem rows BH = B * heads
  int heads, flags;
  float q_scale;
  Grid2D grid{1, 1, kDim * kDim, kDim};
};
// States of up to 128 x 128 have kernels of their own that take a chunk of all blocks as one problem (lfw_wide_*.cu).
// 16 x 16384, 128 x 128: chunk-local 136 us against 162 as a grid of blocks, outputs 180 against 433,
// gradients 515 against 1052.  Rectangles, whole training call, against the grid: 128 x 64, 16 x 16384 1038 / 1097, 96 x 1024
// 379 / 388; 64 x 128 1077 / 1102, 394 / 397; 3 x 777 and 24 x 160 as fast; forward alone, 12 x 1500, 40.0 / 41.8, 41.6 / 42.5.
bool wide(const Grid2D &g) { return g.nsub > 1 && g.nk <= 2 && g.nsub / g.nk <= 2; }
void set_grid(seq::Maps &mp, const Grid2D &g) {
  mp.nsub = g.nsub; mp.nk = g.nk; mp.state_item = g.item; mp.state_ld = (int)g.ld;
}

// The states after every chunk (16-bit) from the caller's state: local kernel + carry.
template <typename T>
int chunk_states(const Call &c, const Scratch &s, const void *state, T *ck_all, int dtype, cudaStream_t st) {
  const int64_t BH = c.B * c.heads, nc = ceil_div64(c.T_, kC), rows = c.B * c.T_;
  seq::Maps mp;
  const Tensor2D loc[4] = {c.x, c.f, c.k, c.fk};
  int rc = build_maps(mp, loc, 4, rows, c.heads, c.flags, 1.f);
  if (rc != T2FW_OK) return rc;
  set_grid(mp, c.grid);
  rc = wide(c.grid) ? lfw_wide_local(false, mp, s.M, s.Ac, s.Gc, s.flags, s.rowflag, c.B, c.T_, c.x.width, c.k.width, dtype, st)
                    : lfw_chunk_local_umma(false, mp, s.M, s.Ac, s.Gc, s.flags, s.rowflag, BH, c.T_, dtype, st);
  if (rc != T2FW_OK) return rc;
  T2FW_CHECK_CUDA((launch_carry<T, true>((const T *)state, s.M, s.Ac, s.Gc, s.flags, s.rowflag, ck_all, c.grid, BH, nc, st)));
  T2FW_CHECK_LAUNCH(1);
  return T2FW_OK;
}

// ckpt_every = m * 64.  m = 1: the carry writes the caller's checkpoints directly.  m > 1: the
// per-chunk states go to scratch and every m-th one (and the last) is copied out.
template <typename T>
int forward_typed(const Call &c, const void *state, void *out, int64_t out_ld, int out_col, void *ckpt, int dtype,
                  int64_t ckpt_every, void *scratch, cudaStream_t st) {
  const int64_t BH = c.B * c.heads, nc = ceil_div64(c.T_, kC), rows = c.B * c.T_, m = ckpt_every / kC;
  Scratch s = carve(scratch, BH, nc);
  T *ck_all = m == 1 ? (T *)ckpt : (T *)s.ck_all;
  int rc = chunk_states<T>(c, s, state, ck_all, dtype, st);
  if (rc != T2FW_OK) return rc;
  seq::Maps mp;
  const Tensor2D all[5] = {c.x, c.f, c.q, c.k, c.fk};
  rc = build_maps(mp, all, 5, rows, c.heads, c.flags, c.q_scale);
  if (rc != T2FW_OK) return rc;
  set_grid(mp, c.grid);
  rc = wide(c.grid) ? lfw_wide_forward_out(mp, state, ck_all, out, s.rowflag, c.B, c.T_, out_ld, c.grid.ld, dtype, st)
                    : lfw_c64_forward_out(mp, state, ck_all, out, out_ld, out_col, s.rowflag, BH, c.T_, dtype, st);
  if (rc != T2FW_OK || m == 1) return rc;
  const int64_t items = BH / c.grid.nsub, slots = ceil_div64(c.T_, ckpt_every), n = items * slots * (c.grid.item / 8);
  const int64_t blocks = ceil_div64(n, 256);
  lfw_c64_pick_ckpt_kernel<T><<<(unsigned)(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, st>>>(
      ck_all, (T *)ckpt, items, nc, m, slots, c.grid.item / 8);
  T2FW_CHECK_LAUNCH(1);
  return T2FW_OK;
}

// ckpt_every > 64: the states at the chunk starts that the caller's checkpoints do not hold are
// rebuilt from the caller's state first, exactly as the forward call built them.
template <typename T>
int backward_typed(const Call &c, const void *gs, const void *state, const void *ckpt, void *const outs[5],
                   const int64_t out_ld[5], const int out_col[5], void *ds, int dtype, int64_t ckpt_every,
                   void *scratch, cudaStream_t st) {
  const int64_t BH = c.B * c.heads, nc = ceil_div64(c.T_, kC), rows = c.B * c.T_, m = ckpt_every / kC;
  Scratch s = carve(scratch, BH, nc);
  if (m > 1) {
    const int rc0 = chunk_states<T>(c, s, state, (T *)s.ck_all, dtype, st);
    if (rc0 != T2FW_OK) return rc0;
    ckpt = s.ck_all;
  }
  seq::Maps mp;
  const Tensor2D loc[4] = {c.go, c.f, c.q, c.fk};
  int rc = build_maps(mp, loc, 4, rows, c.heads, c.flags, c.q_scale);
  if (rc != T2FW_OK) return rc;
  set_grid(mp, c.grid);
  int *const flag0 = m > 1 ? nullptr : s.rowflag;
  rc = wide(c.grid) ? lfw_wide_local(true, mp, s.M, s.Ac, s.Gc, s.flags, flag0, c.B, c.T_, c.x.width, c.k.width, dtype, st)
                    : lfw_chunk_local_umma(true, mp, s.M, s.Ac, s.Gc, s.flags, flag0, BH, c.T_, dtype, st);
  if (rc != T2FW_OK) return rc;
  T2FW_CHECK_CUDA((launch_carry<T, false>((const T *)gs, s.M, s.Ac, s.Gc, s.flags, s.rowflag, (T *)ds, c.grid, BH, nc, st)));
  T2FW_CHECK_LAUNCH(1);
  const Tensor2D all[6] = {c.x, c.f, c.q, c.k, c.fk, c.go};
  rc = build_maps(mp, all, 6, rows, c.heads, c.flags, c.q_scale);
  if (rc != T2FW_OK) return rc;
  set_grid(mp, c.grid);
  if (c.f.p == nullptr) {      // fused layer: the four gradients are column windows of one array
    rc = seq::make_map(&mp.out, outs[0], (uint64_t)rows, (uint64_t)out_ld[0], (uint64_t)out_ld[0]);
    if (rc != T2FW_OK) return rc;
  }
  if (wide(c.grid))
    return lfw_wide_backward_main(mp, state, ckpt, s.M, outs, s.rowflag, c.B, c.T_, out_ld[0], out_ld[2], dtype, st);
  return lfw_c64_backward_main(mp, state, ckpt, s.M, outs, out_ld, out_col, s.rowflag, BH, c.T_, dtype, st);
}

Call plain_call(const void *x, const void *f, const void *q, const void *k, const void *fk, const void *go, int64_t B,
                int64_t T_) {
  Call c;
  c.x = {x, kDim, 0}; c.f = {f, kDim, 0}; c.q = {q, kDim, 0}; c.k = {k, kDim, 0}; c.fk = {fk, kDim, 0};
  c.go = {go, kDim, 0};
  c.B = B; c.T_ = T_; c.heads = 1; c.flags = 0; c.q_scale = 1.f;
  return c;
}

// A D x K state cut into (D/64) x (K/64) blocks: sub-item h = i * nk + j of a batch item is block (i, j); the d-side
// tensors [B*T][D] are read at window i, the k-side tensors [B*T][K] at window j.
Call grid_call(const void *x, const void *f, const void *q, const void *k, const void *fk, const void *go, int64_t B,
               int64_t T_, int nd, int nk) {
  const int64_t D = (int64_t)nd * kDim, K = (int64_t)nk * kDim;
  Call c;
  c.x = {x, D, 0, nk, nd}; c.f = {f, D, 0, nk, nd}; c.go = {go, D, 0, nk, nd};
  c.q = {q, K, 0, 1, nk}; c.k = {k, K, 0, 1, nk}; c.fk = {fk, K, 0, 1, nk};
  c.B = B; c.T_ = T_; c.heads = nd * nk; c.flags = 0; c.q_scale = 1.f;
  c.grid = {nd * nk, nk, (int)(D * K), (int)K};
  return c;
}

// fused layer: qkvg [B][T][4 * H * 64] = query | key | value | gate pre-activation, heads inside a row
Call fused_call(const void *qkvg, const void *go, int64_t B, int64_t T_, int H) {
  const int64_t C = (int64_t)H * kDim;
  Call c;
  c.q = {qkvg, 4 * C, 0}; c.k = {qkvg, 4 * C, (int)C}; c.x = {qkvg, 4 * C, (int)(2 * C)};
  c.fk = {qkvg, 4 * C, (int)(3 * C)};
  c.f = {nullptr, 0, 0};
  c.go = {go, C, 0};
  c.B = B; c.T_ = T_; c.heads = H; c.flags = seq::kFusedLayer; c.q_scale = 0.125f;   // 1 / sqrt(64)
  return c;
}

}  // namespace

bool lfw_chunk_supported(int64_t D, int64_t K, int dtype, int64_t ckpt_every) {
  return D == kDim && K == kDim && ckpt_every >= kC && ckpt_every % kC == 0 &&
         (dtype == T2FW_F16 || dtype == T2FW_BF16);
}

size_t lfw_chunk_forward_scratch_bytes(int64_t B, int64_t T_, int64_t ckpt_every) {
  return scratch_bytes(B, ceil_div64(T_, kC), ckpt_every);
}

size_t lfw_chunk_backward_scratch_bytes(int64_t B, int64_t T_, int64_t ckpt_every) {
  return scratch_bytes(B, ceil_div64(T_, kC), ckpt_every);
}

// Both calls need every pointer 16-byte aligned (the C ABI routes other callers to the scan
// kernels).
int lfw_chunk_forward(const void *x, const void *f, const void *q, const void *k, const void *fk,
                      const void *state, void *out, void *ckpt, int64_t B, int64_t T_, int dtype,
                      int64_t ckpt_every, void *scratch, cudaStream_t st, const int **rowflag_out) {
  if (rowflag_out) *rowflag_out = carve(scratch, B, ceil_div64(T_, kC)).rowflag;
  const Call c = plain_call(x, f, q, k, fk, nullptr, B, T_);
  if (dtype == T2FW_F16) return forward_typed<__half>(c, state, out, kDim, 0, ckpt, dtype, ckpt_every, scratch, st);
  return forward_typed<__nv_bfloat16>(c, state, out, kDim, 0, ckpt, dtype, ckpt_every, scratch, st);
}

int lfw_chunk_backward(const void *go, const void *gs, const void *x, const void *f, const void *q,
                       const void *k, const void *fk, const void *state, const void *ckpt, void *dx,
                       void *df, void *dq, void *dk, void *dfk, void *ds, int64_t B, int64_t T_,
                       int dtype, int64_t ckpt_every, void *scratch, cudaStream_t st, const int **rowflag_out) {
  if (rowflag_out) *rowflag_out = carve(scratch, B, ceil_div64(T_, kC)).rowflag;
  const Call c = plain_call(x, f, q, k, fk, go, B, T_);
  void *const outs[5] = {dx, df, dq, dk, dfk};
  const int64_t ld[5] = {kDim, kDim, kDim, kDim, kDim};
  const int col[5] = {0, 0, 0, 0, 0};
  if (dtype == T2FW_F16)
    return backward_typed<__half>(c, gs, state, ckpt, outs, ld, col, ds, dtype, ckpt_every, scratch, st);
  return backward_typed<__nv_bfloat16>(c, gs, state, ckpt, outs, ld, col, ds, dtype, ckpt_every, scratch, st);
}

// ---- states that are grids of 64 x 64 blocks; all arrays dense, rowflag per batch item ----------------
bool lfw_grid_supported(int64_t D, int64_t K, int dtype, int64_t ckpt_every) {
  return (dtype == T2FW_F16 || dtype == T2FW_BF16) && ckpt_every >= kC && ckpt_every % kC == 0 && D % kDim == 0 && K % kDim == 0 &&
         D <= 256 && K <= 256 && (D > kDim || K > kDim);
}

size_t lfw_grid_scratch_bytes(int64_t B, int64_t T_, int64_t D, int64_t K, int64_t ckpt_every) {
  return scratch_bytes(B * (D / kDim) * (K / kDim), ceil_div64(T_, kC), ckpt_every);
}

int lfw_grid_forward(const void *x, const void *f, const void *q, const void *k, const void *fk, const void *state, void *out,
                     void *ckpt, int64_t B, int64_t T_, int64_t D, int64_t K, int dtype, int64_t ckpt_every, void *scratch,
                     cudaStream_t st, const int **rowflag_out) {
  const int nd = (int)(D / kDim), nk = (int)(K / kDim);
  *rowflag_out = carve(scratch, B * nd * nk, ceil_div64(T_, kC)).rowflag;
  const Call c = grid_call(x, f, q, k, fk, nullptr, B, T_, nd, nk);
  if (dtype == T2FW_F16) return forward_typed<__half>(c, state, out, D, 0, ckpt, dtype, ckpt_every, scratch, st);
  return forward_typed<__nv_bfloat16>(c, state, out, D, 0, ckpt, dtype, ckpt_every, scratch, st);
}

int lfw_grid_backward(const void *go, const void *gs, const void *x, const void *f, const void *q, const void *k, const void *fk,
                      const void *state, const void *ckpt, void *dx, void *df, void *dq, void *dk, void *dfk, void *ds, int64_t B,
                      int64_t T_, int64_t D, int64_t K, int dtype, int64_t ckpt_every, void *scratch, cudaStream_t st,
                      const int **rowflag_out) {
  const int nd = (int)(D / kDim), nk = (int)(K / kDim);
  *rowflag_out = carve(scratch, B * nd * nk, ceil_div64(T_, kC)).rowflag;
  const Call c = grid_call(x, f, q, k, fk, go, B, T_, nd, nk);
  void *const outs[5] = {dx, df, dq, dk, dfk};
  const int64_t ld[5] = {D, D, K, K, K};
  const int col[5] = {0, 0, 0, 0, 0};
  if (dtype == T2FW_F16) return backward_typed<__half>(c, gs, state, ckpt, outs, ld, col, ds, dtype, ckpt_every, scratch, st);
  return backward_typed<__nv_bfloat16>(c, gs, state, ckpt, outs, ld, col, ds, dtype, ckpt_every, scratch, st);
}

// ---- summary of a sequence segment (for splitting the time axis over devices) ------------------
// Total decay of a segment per feature: the product of the chunks' decay vectors.  A row with a
// flagged chunk (gate products beyond 2^100) gets NaN decays, so that whatever is built on the
// summary shows the problem instead of hiding it.
__global__ void __launch_bounds__(128)
lfw_c64_decay_totals_kernel(const float *__restrict__ Ac, const float *__restrict__ Gc, const int *__restrict__ rowflag,
                            float *__restrict__ A_out, float *__restrict__ G_out, int64_t B, int64_t nc) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= B * 2 * kDim) return;
  const int64_t b = i / (2 * kDim);
  const int side = (int)((i / kDim) & 1), feat = (int)(i % kDim);
  const float *src = side ? Gc : Ac;
  float p = 1.f;
  for (int64_t c = 0; c < nc; ++c) p *= src[((size_t)b * nc + c) * kDim + feat];
  if (rowflag[b] != 0) p = __int_as_float(0x7fc00000);
  (side ? G_out : A_out)[b * kDim + feat] = p;
}

template <typename T>
int summary_typed(bool backward, const void *val_d, const void *gate_d, const void *val_k, const void *gate_k,
                  void *end_state, float *A_out, float *G_out, int64_t B, int64_t T_, int dtype, void *scratch,
                  cudaStream_t st) {
  const int64_t nc = ceil_div64(T_, kC), rows = B * T_;
  Scratch s = carve(scratch, B, nc);
  seq::Maps mp;
  const Tensor2D loc[4] = {{val_d, kDim, 0}, {gate_d, kDim, 0}, {val_k, kDim, 0}, {gate_k, kDim, 0}};
  int rc = build_maps(mp, loc, 4, rows, 1, 0, 1.f);
  if (rc != T2FW_OK) return rc;
  const Grid2D one{1, 1, kDim * kDim, kDim};
  set_grid(mp, one);
  rc = lfw_chunk_local_umma(backward, mp, s.M, s.Ac, s.Gc, s.flags, s.rowflag, B, T_, dtype, st);
  if (rc != T2FW_OK) return rc;
  if (backward) {      // the state gradient at the segment start that the segment's own output gradients cause
    T2FW_CHECK_CUDA((launch_carry<T, false>(nullptr, s.M, s.Ac, s.Gc, s.flags, s.rowflag, (T *)end_state, one, B, nc, st)));
  } else {             // the state at the segment end that the segment's own inputs cause
    T2FW_CHECK_CUDA((launch_carry<T, true>(nullptr, s.M, s.Ac, s.Gc, s.flags, s.rowflag, (T *)s.ck_all, one, B, nc, st)));
    lfw_c64_pick_ckpt_kernel<T><<<(unsigned)ceil_div64(B * (kDim * kDim / 8), 256), 256, 0, st>>>(
        (const T *)s.ck_all, (T *)end_state, B, nc, nc, 1, (int64_t)(kDim * kDim / 8));
  }
  lfw_c64_decay_totals_kernel<<<(unsigned)ceil_div64(B * 2 * kDim, 128), 128, 0, st>>>(s.Ac, s.Gc, s.rowflag, A_out,
                                                                                     G_out, B, nc);
  T2FW_CHECK_LAUNCH(backward ? 2 : 3);
  return T2FW_OK;
}

size_t lfw_segment_summary_scratch_bytes(int64_t B, int64_t T_) { return scratch_bytes(B, ceil_div64(T_, kC), 2 * kC); }

// forward flavour: (val_d, gate_d, val_k, gate_k) = (x, f, k, f_key), end_state = the state a zero state becomes over
// the segment; backward flavour: (dO, f, q, f_key), end_state = the state gradient at the segment start for a zero
// gradient at its end.  A_out, G_out [B][64] fp32: the segment's total decays.
int lfw_segment_summary(bool backward, const void *val_d, const void *gate_d, const void *val_k, const void *gate_k,
                        void *end_state, float *A_out, float *G_out, int64_t B, int64_t T_, int dtype, void *scratch,
                        cudaStream_t st) {
  if (dtype == T2FW_F16)
    return summary_typed<__half>(backward, val_d, gate_d, val_k, gate_k, end_state, A_out, G_out, B, T_, dtype, scratch, st);
  return summary_typed<__nv_bfloat16>(backward, val_d, gate_d, val_k, gate_k, end_state, A_out, G_out, B, T_, dtype,
                                      scratch, st);
}

// ---- fused layer entry points (heads read in place from the projection output) ----------------
size_t lfw_fused_scratch_bytes(int64_t B, int64_t T_, int H) { return lfw_chunk_forward_scratch_bytes(B * H, T_, kC); }

int lfw_fused_forward(const void *qkvg, const void *state, void *out, void *ckpt, int64_t B, int64_t T_, int H,
                      int dtype, void *scratch, cudaStream_t st) {
  const Call c = fused_call(qkvg, nullptr, B, T_, H);
  const int64_t C = (int64_t)H * kDim;
  if (dtype == T2FW_F16) return forward_typed<__half>(c, state, out, C, 0, ckpt, dtype, kC, scratch, st);
  return forward_typed<__nv_bfloat16>(c, state, out, C, 0, ckpt, dtype, kC, scratch, st);
}

int lfw_fused_backward(const void *go, const void *gs, const void *qkvg, const void *state, const void *ckpt,
                       void *d_qkvg, void *ds, int64_t B, int64_t T_, int H, int dtype, void *scratch,
                       cudaStream_t st) {
  const Call c = fused_call(qkvg, go, B, T_, H);
  const int64_t C = (int64_t)H * kDim;
  // gradients land in d_qkvg [B][T][4C]: query | key | value | gate; there is no forget tensor
  void *const outs[5] = {d_qkvg, nullptr, d_qkvg, d_qkvg, d_qkvg};
  const int64_t ld[5] = {4 * C, 0, 4 * C, 4 * C, 4 * C};
  const int col[5] = {(int)(2 * C), 0, 0, (int)C, (int)(3 * C)};
  if (dtype == T2FW_F16) return backward_typed<__half>(c, gs, state, ckpt, outs, ld, col, ds, dtype, kC, scratch, st);
  return backward_typed<__nv_bfloat16>(c, gs, state, ckpt, outs, ld, col, ds, dtype, kC, scratch, st);
}

}  // namespace t2fw
