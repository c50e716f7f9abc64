// Decay-rule ("LFW") scan kernels: the shape- and dtype-general path.
//
//   S_t = (f_t fk_t^T) .* S_{t-1} + x_t k_t^T ,  o_t = S_t q_t
//
// A group of lanes owns a line of the D x K state (a row in the "row" orientation, a column in the
// "column" orientation), the lanes spread along the other axis, and time is walked
// sequentially with the state in registers in the accumulation type (float, or double for
// double storage).  Every output of the reference's forward (scan kernel + einsum,
// t2fw/csrc/lfw_kernel.cu:18-59, t2fw/csrc/lfw.cpp:45) and backward (reverse scan + five
// einsums + two in-place multiplies, t2fw/csrc/lfw_kernel.cu:61-102, t2fw/csrc/lfw.cpp:84-93)
// is produced inside the kernels; no [B,T,D,K] tensor exists.  Only every C-th state is
// stored; the backward pass recomputes the others from those checkpoints.
//
// The backward runs the same code twice with the two axes exchanged, side by side:
//   row orientation    (own = d, lanes = k): d_x = R k, d_f = (R.*S_prev) fk, d_state
//   column orientation (own = k, lanes = d): d_k = R^T x, d_f_key = (R.*S_prev)^T f, d_q = S^T dO
// so every reduction is a warp reduction and the result is deterministic.
//
// A chain of T steps bounds these kernels.  The steps' vectors come from shared memory, fetched a group ahead
// (scan.cuh); the sums of a step share their shuffles; the two orientations run side by side; the backward
// walks a checkpoint's steps forward once to leave the state at each segment start and then segment by segment
// (128 forward steps per 64 instead of 160).  Eight, 16 or 32 lanes own a line (lanes_for), and eight sums are formed
// together: seven exchanges for four lines where a line per warp took 40.
//
// The two orientations of the backward are one launch: kernels of their own would run one after the other (16 x 129, 96 x 48,
// fp32: 107 us against 69.5), or the second would read its inputs on the word of the first that they are there, for which
// there is no rule.
//
// These kernels also redo the batch rows that the chunk kernels flagged (gate products outside the range of
// the factored form): CTAs walk over all work items and skip the rows without a flag, and the launch is a
// dependent one.  An all-clear costs 4.9 us forward and 5.7 us backward with cold caches (96 x 1024, one flag per row).
//
// The kernels are templates; lfw_scan_{f16,bf16,f32,f64}.cu instantiate them for one storage type each (compiled side
// by side), lfw_scan.cu picks the type.
#pragma once

#include <initializer_list>

#include "scan.cuh"

namespace t2fw {
namespace lfw_scan {

// one storage type's calls, defined below and instantiated in that type's file
template <typename T>
int fwd_typed(const void *x, const void *f, const void *q, const void *k, const void *fk, const void *state, void *out,
              void *ckpt, int64_t B, int64_t T_, int64_t D, int64_t K, int64_t C, cudaStream_t st, const int *rowflag);
template <typename T>
int bwd_typed(const void *go, const void *gs, const void *x, const void *f, const void *q, const void *k, const void *fk,
              const void *state, const void *ckpt, void *dx, void *df, void *dq, void *dk, void *dfk, void *ds, int64_t B,
              int64_t T_, int64_t D, int64_t K, int64_t C, cudaStream_t st, const int *rowflag);

#ifdef T2FW_LFW_SCAN_DEFINE

namespace {

constexpr int kWarpsPerCta = 4;
constexpr int kThreads = kWarpsPerCta * 32;
constexpr size_t kSmemMost = 224 * 1024;      // backward: dynamic shared memory of a CTA

template <typename T>
struct FwdArgs {
  const T *x, *f, *q, *k, *fk, *state;
  T *out, *ckpt;
  int64_t B, T_;
  int D, K;
  int64_t C, nslots;
  int G;                  // steps per group
  int64_t items;          // work items: (batch row, block of state rows)
  const int *rowflag;     // if not null, only batch rows with a non-zero flag are processed
};

// One buffer: fk, k, q [G][K], x, f [G][lines of the CTA], each part 16-byte aligned
template <typename T>
__host__ __device__ inline int fwd_part(int G, int n) { return (int)((((size_t)G * n * sizeof(T)) + 15) / 16 * 16); }

// Element c of a state row lies in lane c % L of the L lanes that own OWN rows; the first SAFE elements of a lane
// exist for every row length that takes this NL.
template <typename T, int L, int NL, int SAFE, int OWN>
__global__ void __launch_bounds__(kThreads, sizeof(T) == 8 ? 1 : 4) lfw_scan_fwd_kernel(const FwdArgs<T> a) {
  using A = typename Elem<T>::acc;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int RC = kThreads / L * OWN;      // state rows of the CTA
  constexpr int U = 8 / OWN;                  // steps whose sums are formed together
  const int tid = threadIdx.x, l = tid % L, rl = tid / L * OWN;
  const int kp = fwd_part<T>(a.G, a.K), dp = fwd_part<T>(a.G, RC), buf_bytes = 3 * kp + 2 * dp;
  const int blocks_d = (a.D + RC - 1) / RC;
  dependency_wait();
  for (int64_t item = blockIdx.x; item < a.items; item += gridDim.x) {
    const int64_t b = item / blocks_d;
    if (a.rowflag != nullptr && a.rowflag[b] == 0) continue;      // the same for the whole CTA
    const int rb = (int)(item - b * blocks_d) * RC, nrows = a.D - rb < RC ? a.D - rb : RC;

    auto fetch = [&](int64_t t0, int which) {
      const int n = (int)(a.T_ - t0 < a.G ? a.T_ - t0 : a.G);
      unsigned char *p = smem_raw + which * buf_bytes;
      const int64_t ko = (b * a.T_ + t0) * a.K, od = (b * a.T_ + t0) * a.D + rb;
      scan::stage(reinterpret_cast<T *>(p), a.fk + ko, n * a.K, tid, kThreads);
      scan::stage(reinterpret_cast<T *>(p + kp), a.k + ko, n * a.K, tid, kThreads);
      scan::stage(reinterpret_cast<T *>(p + 2 * kp), a.q + ko, n * a.K, tid, kThreads);
      scan::stage_rows(reinterpret_cast<T *>(p + 3 * kp), a.x + od, n, nrows, a.D, tid, kThreads);
      scan::stage_rows(reinterpret_cast<T *>(p + 3 * kp + dp), a.f + od, n, nrows, a.D, tid, kThreads);
      scan::commit();
    };
    fetch(0, 0);

    A S[OWN][NL];
#pragma unroll
    for (int o = 0; o < OWN; ++o)
#pragma unroll
      for (int j = 0; j < NL; ++j)
        S[o][j] = rl + o < nrows && l + L * j < a.K ? Elem<T>::ld(a.state + (b * a.D + rb + rl + o) * a.K + l + L * j) : A(0);

    int which = 0;
    int64_t ck_next = a.C < a.T_ ? a.C : a.T_, slot = 0;      // step count at the next checkpoint
    for (int64_t t0 = 0; t0 < a.T_; t0 += a.G, which ^= 1) {
      if (t0 + a.G < a.T_) fetch(t0 + a.G, which ^ 1);
      else scan::commit();
      scan::wait<1>();
      __syncthreads();
      const int n = (int)(a.T_ - t0 < a.G ? a.T_ - t0 : a.G);
      const unsigned char *p = smem_raw + which * buf_bytes;
      const T *sg = reinterpret_cast<const T *>(p) + l, *sk = reinterpret_cast<const T *>(p + kp) + l;
      const T *sq = reinterpret_cast<const T *>(p + 2 * kp) + l;
      const T *sx = reinterpret_cast<const T *>(p + 3 * kp) + rl, *sf = reinterpret_cast<const T *>(p + 3 * kp + dp) + rl;
      auto step = [&](int t, A *acc) {
        A xo[OWN], ao[OWN];
#pragma unroll
        for (int o = 0; o < OWN; ++o) {
          const bool in = rl + o < nrows;
          xo[o] = in ? Elem<T>::ld(sx + t * nrows + o) : A(0);
          ao[o] = in ? Elem<T>::ld(sf + t * nrows + o) : A(0);
          acc[o] = A(0);
        }
#pragma unroll
        for (int j = 0; j < NL; ++j) {
          const bool in = j < SAFE || l + L * j < a.K;
          const A g = in ? Elem<T>::ld(sg + t * a.K + L * j) : A(0), k = in ? Elem<T>::ld(sk + t * a.K + L * j) : A(0);
          const A q = in ? Elem<T>::ld(sq + t * a.K + L * j) : A(0);
#pragma unroll
          for (int o = 0; o < OWN; ++o) {
            S[o][j] = S[o][j] * (ao[o] * g) + xo[o] * k;
            acc[o] += S[o][j] * q;
          }
        }
      };
      T *out = a.out + (b * a.T_ + t0) * a.D + rb + rl;
      for (int t = 0; t < n;) {
        const int te = ck_next - t0 < n ? (int)(ck_next - t0) : n;      // up to the next checkpoint
        for (; t + U <= te; t += U) {
          A acc[8];
#pragma unroll
          for (int u = 0; u < U; ++u) step(t + u, acc + u * OWN);
          int i;
          if (scan::lane_sums<8, L>(acc, l, &i) && rl + i % OWN < nrows)
            Elem<T>::st(out + (int64_t)(t + i / OWN) * a.D + i % OWN, acc[0]);
        }
        for (; t < te; ++t) {
          A acc[OWN];
          step(t, acc);
          int i;
          if (scan::lane_sums<OWN, L>(acc, l, &i) && rl + i < nrows) Elem<T>::st(out + (int64_t)t * a.D + i, acc[0]);
        }
        if (t0 + te == ck_next) {
#pragma unroll
          for (int o = 0; o < OWN; ++o)
#pragma unroll
            for (int j = 0; j < NL; ++j)
              if (rl + o < nrows && l + L * j < a.K)
                Elem<T>::st(a.ckpt + ((b * a.nslots + slot) * a.D + rb + rl + o) * a.K + l + L * j, S[o][j]);
          ++slot;
          ck_next = ck_next + a.C < a.T_ ? ck_next + a.C : a.T_;
        }
      }
      __syncthreads();
    }
  }
}

// Arguments of one orientation of the backward.  "own" is the axis whose lines a warp owns, "lane" the axis
// the lanes spread over.
template <typename T>
struct LineArgs {
  const T *xo, *go, *po;  // own-axis vectors  [B,T,NO]: (x, f, dO) or (k, fk, q)
  const T *xl, *gl, *pl;  // lane-axis vectors [B,T,NLn]: (k, fk, q) or (x, f, dO)
  T *d_xo;                // sum over lanes of R * xl             -> d_x  or d_k
  T *d_go;                // sum over lanes of R * S_prev * gl    -> d_f  or d_f_key
  T *d_po;                // sum over lanes of S_t * pl           -> d_q  (column orientation only)
  T *d_state;             // row orientation only
  int NO, NLn;            // own extent, lane extent
  int64_t so, sl;         // strides of the own / lane axis inside one [D,K] state
  int64_t items;          // work items: (batch row, block of own lines); 0: not in this launch
  int seg, mids;          // steps per segment; segment starts whose states are kept besides the chunk's
};

template <typename T>
struct BwdArgs {
  LineArgs<T> col, row;
  const T *state0, *ckpt, *grad_state;
  int64_t B, T_, C, nslots;
  const int *rowflag;
};

// Which segment a warp is at.  A checkpoint interval of ns segments is first walked forward over all but the last
// (target -1), leaving the state at every ms-th segment start; then segments are taken from the last to the
// first, each reached from the nearest start that was kept (ms = 1 unless the interval is very long).
struct SegWalk {
  int64_t c;              // checkpoint interval
  int ns, ms, cur, target;
  int64_t T_, C;
  int seg, mids;
  __device__ __forceinline__ void open() {      // interval c
    const int64_t n = T_ - c * C < C ? T_ - c * C : C;
    ns = (int)((n + seg - 1) / seg);
    ms = (ns + mids) / (mids + 1);
    cur = 0;
    target = ns > 1 ? -1 : 0;
  }
  __device__ __forceinline__ void step() {
    if (target < 0) {
      if (cur < ns - 2) { ++cur; return; }
      target = ns - 1;
      cur = target / ms * ms;
    } else if (cur < target) {
      ++cur;
    } else if (--target >= 0) {
      cur = target / ms * ms;
    } else if (--c >= 0) {
      open();
    }
  }
  __device__ __forceinline__ int64_t first() const { return c * C + (int64_t)cur * seg; }
  __device__ __forceinline__ int count() const {
    const int64_t end = (c + 1) * C < T_ ? (c + 1) * C : T_, left = end - first();
    return (int)(left < seg ? left : seg);
  }
};

// shared memory: two buffers of xl, gl, pl [seg][NLn] and xo, go, po [seg][RC] (storage type), then per warp the
// states of a segment's steps and the kept segment starts (accumulation type)
template <typename T>
__host__ __device__ inline int bwd_part(int seg, int n) { return (int)((((size_t)seg * n * sizeof(T)) + 15) / 16 * 16); }

// One block of own lines of batch row b
template <typename T, int L, int NL, int SAFE, bool WITH_SP>
__device__ __forceinline__ void line_bwd(const BwdArgs<T> &a, const LineArgs<T> &ln, int64_t b, int block, unsigned char *smem) {
  using A = typename Elem<T>::acc;
  constexpr int RC = kThreads / L;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, l = tid % L, rl = tid / L;
  const int lp = bwd_part<T>(ln.seg, ln.NLn), op = bwd_part<T>(ln.seg, RC), buf_bytes = 3 * lp + 3 * op;
  A *hist = reinterpret_cast<A *>(smem + 2 * buf_bytes) + (size_t)warp * (ln.seg + ln.mids) * NL * 32;
  A *mid = hist + (size_t)ln.seg * NL * 32;

  const int ob = block * RC, nown = ln.NO - ob < RC ? ln.NO - ob : RC;
  const int o0 = ob + rl;
  const bool mine = o0 < ln.NO;
  const int64_t DK = (int64_t)ln.NO * ln.NLn;

  auto state_off = [&](int j) { return o0 * ln.so + (int64_t)(l + L * j) * ln.sl; };
  auto valid = [&](int j) { return mine && (l + L * j) < ln.NLn; };

  SegWalk w;
  w.T_ = a.T_; w.C = a.C; w.seg = ln.seg; w.mids = ln.mids;
  w.c = (a.T_ + a.C - 1) / a.C - 1;
  w.open();
  auto fetch = [&](const SegWalk &s, int which) {
    const int n = s.count();
    const int64_t lo = (b * a.T_ + s.first()) * ln.NLn, oo = (b * a.T_ + s.first()) * ln.NO + ob;
    unsigned char *p = smem + which * buf_bytes;
    scan::stage_rolled(reinterpret_cast<T *>(p), ln.xl + lo, n * ln.NLn, tid, kThreads);
    scan::stage_rolled(reinterpret_cast<T *>(p + lp), ln.gl + lo, n * ln.NLn, tid, kThreads);
    scan::stage_rows_rolled(reinterpret_cast<T *>(p + 3 * lp), ln.xo + oo, n, nown, ln.NO, tid, kThreads);
    scan::stage_rows_rolled(reinterpret_cast<T *>(p + 3 * lp + op), ln.go + oo, n, nown, ln.NO, tid, kThreads);
    if (s.cur == s.target) {      // upstream vectors: only where the gradients are formed
      scan::stage_rolled(reinterpret_cast<T *>(p + 2 * lp), ln.pl + lo, n * ln.NLn, tid, kThreads);
      scan::stage_rows_rolled(reinterpret_cast<T *>(p + 3 * lp + 2 * op), ln.po + oo, n, nown, ln.NO, tid, kThreads);
    }
    scan::commit();
  };
  A R[NL], S[NL];
#pragma unroll
  for (int j = 0; j < NL; ++j)
    R[j] = valid(j) ? Elem<T>::ld(a.grad_state + b * DK + state_off(j)) : A(0);

  SegWalk nx = w;
  int which = 1;
#pragma unroll 1
  for (bool first = true; first || w.c >= 0; first = false) {      // the first trip only fetches
    if (nx.c >= 0) fetch(nx, which ^ 1);
    else scan::commit();
    if (first) {
      nx.step();
      which = 0;
      continue;
    }

    if (w.cur == 0) {      // the interval's own checkpoint
      const T *src = (w.c == 0) ? a.state0 + b * DK : a.ckpt + (b * a.nslots + (w.c - 1)) * DK;
#pragma unroll
      for (int j = 0; j < NL; ++j) S[j] = valid(j) ? Elem<T>::ld(src + state_off(j)) : A(0);
    } else if (w.target >= 0 && w.cur % w.ms == 0) {      // a kept segment start
      const A *m = mid + (size_t)(w.cur / w.ms - 1) * NL * 32;
#pragma unroll
      for (int j = 0; j < NL; ++j) S[j] = m[j * 32 + lane];
    }
    scan::wait<1>();
    __syncthreads();

    const int n = w.count();
    const unsigned char *p = smem + which * buf_bytes;
    const T *s_xl = reinterpret_cast<const T *>(p) + l, *s_gl = reinterpret_cast<const T *>(p + lp) + l;
    const T *s_pl = reinterpret_cast<const T *>(p + 2 * lp) + l;
    const T *s_xo = reinterpret_cast<const T *>(p + 3 * lp) + rl, *s_go = reinterpret_cast<const T *>(p + 3 * lp + op) + rl;
    const T *s_po = reinterpret_cast<const T *>(p + 3 * lp + 2 * op) + rl;
    const bool last = w.cur == w.target;
    auto vec = [&](const T *v, int t, int j) {
      return (j < SAFE || l + L * j < ln.NLn) ? Elem<T>::ld(v + t * ln.NLn + L * j) : A(0);
    };
    auto own = [&](const T *v, int t) { return mine ? Elem<T>::ld(v + t * nown) : A(0); };

#pragma unroll(NL <= 8 ? 2 : 1)
    for (int t = 0; t < n; ++t) {      // forward over the segment
      const A xo = own(s_xo, t), go = own(s_go, t);
#pragma unroll
      for (int j = 0; j < NL; ++j) {
        const A g = vec(s_gl, t, j), x = vec(s_xl, t, j);
        if (last) hist[(t * NL + j) * 32 + lane] = S[j];
        S[j] = S[j] * (go * g) + xo * x;
      }
    }
    if (w.target < 0 && (w.cur + 1) % w.ms == 0) {
      A *m = mid + (size_t)((w.cur + 1) / w.ms - 1) * NL * 32;
#pragma unroll
      for (int j = 0; j < NL; ++j) m[j * 32 + lane] = S[j];
    }
    if (last) {
      const int64_t ob_t = (b * a.T_ + w.first()) * ln.NO + o0;
      constexpr int kSums = WITH_SP ? 4 : 2, U = 8 / kSums;      // U steps' sums are formed together
      auto step = [&](int t, A *v) {      // S is the state after step t
        const A go = own(s_go, t), po = own(s_po, t);
#pragma unroll
        for (int i = 0; i < kSums; ++i) v[i] = A(0);
#pragma unroll
        for (int j = 0; j < NL; ++j) {
          const A g = vec(s_gl, t, j), x = vec(s_xl, t, j), p = vec(s_pl, t, j);
          const A sp = hist[(t * NL + j) * 32 + lane];
          const A r = R[j] + po * p;    // gradient w.r.t. S_t
          v[0] += r * x;
          v[1] += (r * sp) * g;
          if (WITH_SP) v[2] += S[j] * p;
          R[j] = r * (go * g);          // what flows on to S_{t-1}
          S[j] = sp;
        }
      };
      auto put = [&](int t, int i, A v) {      // sum i of the steps t, t - 1, ..
        const int kind = i % kSums;
        if (kind < 3 && mine) {
          T *dst = kind == 0 ? ln.d_xo : kind == 1 ? ln.d_go : ln.d_po;
          Elem<T>::st(dst + ob_t + (int64_t)(t - i / kSums) * ln.NO, v);
        }
      };
      int t = n - 1, i;
      for (; t + 1 >= U; t -= U) {
        A v[8];
#pragma unroll
        for (int u = 0; u < U; ++u) step(t - u, v + u * kSums);
        if (scan::lane_sums<8, L>(v, l, &i)) put(t, i, v[0]);
      }
      for (; t >= 0; --t) {
        A v[kSums];
        step(t, v);
        if (scan::lane_sums<kSums, L>(v, l, &i)) put(t, i, v[0]);
      }
    }
    __syncthreads();
    w = nx;
    nx.step();
    which ^= 1;
  }
  if (!WITH_SP) {
#pragma unroll
    for (int j = 0; j < NL; ++j)
      if (valid(j)) Elem<T>::st(ln.d_state + b * DK + state_off(j), R[j]);
  }
}

// Both orientations side by side, the columns' items first.  LC, NC, SC: lanes, elements per lane (NL) and elements that
// exist for every line (SAFE) of the columns; LR, NR, SR: of the rows.
template <typename T, int LC, int NC, int SC, int LR, int NR, int SR>
__global__ void __launch_bounds__(kThreads) lfw_line_bwd_kernel(const BwdArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  dependency_wait();
  for (int64_t item = blockIdx.x; item < a.col.items + a.row.items; item += gridDim.x) {
    const bool col = item < a.col.items;
    const int64_t i = col ? item : item - a.col.items;
    const int blocks = col ? (a.col.NO + kThreads / LC - 1) / (kThreads / LC) : (a.row.NO + kThreads / LR - 1) / (kThreads / LR);
    const int64_t b = i / blocks;
    if (a.rowflag != nullptr && a.rowflag[b] == 0) continue;      // the same for the whole CTA
    if (col) line_bwd<T, LC, NC, SC, true>(a, a.col, b, (int)(i - b * blocks), smem_raw);
    else line_bwd<T, LR, NR, SR, false>(a, a.row, b, (int)(i - b * blocks), smem_raw);
  }
}

// Lanes per line for lines of up to 128 elements (backward: by the mean of the two orientations' lines).  Eight cost the
// fewest instructions, where they still give every scheduler a warp and a half; with fewer lines a step's length is what
// counts, and the lines are spread over 16 lanes while that fills half of the schedulers, over a warp below.  Rows of 150
// steps, fp32, us at 8 / 16 / 32 lanes.  64 x 64, forward: 192 lines 23.7 / 18.9 / 17.1, 576 24.1 / 19.0 / 17.3, 896
// 24.1 / 19.2 / 19.8, 2688 32.1 / 32.4 / 41.9, 3584 32.3 / 32.6 / 45.6, 6400 41.6 / 50.7 / 69.8; backward: 192 75 / 59 / 51, 896
// 79 / 77 / 77, 2688 165 / 137 / 180, 3584 177 / 186 / 238, 6400 269 / 275 / 382.  100 x 100 turns earlier (2400 lines, forward
// 41.7 / 49.0 / 49.6, backward 296 / 312 / 301).
int lanes_for(int64_t lines) { return lines >= 148 * 24 ? 8 : lines >= 148 * 4 ? 16 : 32; }

// CTAs of a launch: one per work item; the walk over flagged rows only is cut to a few waves
unsigned grid_for(int64_t items, const int *rowflag) {
  const int64_t most = rowflag != nullptr ? 148 * 4 : (int64_t)1 << 30;
  return (unsigned)(items < most ? items : most);
}

template <typename T, int L, int NL, int SAFE, int OWN>
int launch_fwd(FwdArgs<T> a, cudaStream_t st) {
  constexpr int RC = kThreads / L * OWN;
  a.items = a.B * ((a.D + RC - 1) / RC);
  auto bytes = [&](int G) { return 2 * (size_t)(3 * fwd_part<T>(G, a.K) + 2 * fwd_part<T>(G, RC)); };
  for (a.G = 32; a.G > 1 && (a.G / 2 >= a.T_ || bytes(a.G) > 48 * 1024);) a.G /= 2;
  const size_t smem = bytes(a.G);
  T2FW_CHECK_CUDA(launch_dependent(&lfw_scan_fwd_kernel<T, L, NL, SAFE, OWN>, dim3(grid_for(a.items, a.rowflag)),
                                   dim3(kThreads), smem, st, a));
  T2FW_CHECK_LAUNCH(1);
  return T2FW_OK;
}

// Rows per group of lanes: MORE share the key-side loads; one while MORE would leave the chip with less than four
// warps per SM (the chain of steps is then what counts, and more CTAs shorten each step).
template <typename T, int L, int NL, int SAFE, int MORE>
int launch_fwd_rows(const FwdArgs<T> &a, cudaStream_t st) {
  if (a.B * a.D * L / (32 * MORE) >= 148 * 4 || a.rowflag != nullptr) return launch_fwd<T, L, NL, SAFE, MORE>(a, st);
  return launch_fwd<T, L, NL, SAFE, 1>(a, st);
}

}  // namespace

template <typename T>
int fwd_typed(const void *x, const void *f, const void *q, const void *k, const void *fk,
              const void *state, void *out, void *ckpt, int64_t B, int64_t T_, int64_t D,
              int64_t K, int64_t C, cudaStream_t st, const int *rowflag) {
  FwdArgs<T> a{};
  a.x = (const T *)x; a.f = (const T *)f; a.q = (const T *)q; a.k = (const T *)k; a.fk = (const T *)fk;
  a.state = (const T *)state; a.out = (T *)out; a.ckpt = (T *)ckpt;
  a.B = B; a.T_ = T_; a.D = (int)D; a.K = (int)K; a.C = C; a.nslots = ceil_div64(T_, C); a.rowflag = rowflag;
  // elements per lane: the smallest that holds the row (double: in four sizes)
  if constexpr (sizeof(T) == 8) {
    if (K <= 64) return launch_fwd<T, 32, 2, 0, 1>(a, st);
    if (K <= 128) return launch_fwd<T, 32, 4, 0, 1>(a, st);
    if (K <= 256) return launch_fwd<T, 32, 8, 0, 1>(a, st);
    if (K <= 512) return launch_fwd<T, 32, 16, 0, 1>(a, st);
  } else {
    const int lanes = rowflag != nullptr ? 8 : lanes_for(B * D);
    if (K <= 128 && lanes == 32) {
      if (K <= 32) return launch_fwd<T, 32, 1, 0, 1>(a, st);
      if (K <= 64) return launch_fwd<T, 32, 2, 1, 1>(a, st);
      if (K <= 96) return launch_fwd<T, 32, 3, 2, 1>(a, st);
      return launch_fwd<T, 32, 4, 3, 1>(a, st);
    }
    if (K <= 128 && lanes == 16) {
      if (K <= 32) return launch_fwd<T, 16, 2, 0, 1>(a, st);
      if (K <= 48) return launch_fwd<T, 16, 3, 2, 1>(a, st);
      if (K <= 64) return launch_fwd<T, 16, 4, 3, 1>(a, st);
      if (K <= 96) return launch_fwd<T, 16, 6, 4, 1>(a, st);
      return launch_fwd<T, 16, 8, 6, 1>(a, st);
    }
    if (K <= 16) return launch_fwd_rows<T, 8, 2, 0, 2>(a, st);
    if (K <= 32) return launch_fwd_rows<T, 8, 4, 2, 2>(a, st);
    if (K <= 48) return launch_fwd_rows<T, 8, 6, 4, 2>(a, st);
    if (K <= 64) return launch_fwd_rows<T, 8, 8, 6, 2>(a, st);
    if (K <= 80) return launch_fwd_rows<T, 8, 10, 8, 2>(a, st);
    if (K <= 104) return launch_fwd_rows<T, 8, 13, 10, 2>(a, st);
    if (K <= 128) return launch_fwd_rows<T, 8, 16, 13, 2>(a, st);
    if (K <= 256) return launch_fwd_rows<T, 32, 8, 4, 4>(a, st);
    if (K <= 512) return launch_fwd_rows<T, 32, 16, 8, 4>(a, st);
  }
  set_error("lfw forward: K=%lld exceeds the supported maximum of 512", (long long)K);
  return T2FW_ERR_UNSUPPORTED;
}

namespace {

template <typename T, int LC, int NC, int SC, int LR, int NR, int SR>
int launch_lines(BwdArgs<T> a, cudaStream_t st) {
  using A = typename Elem<T>::acc;
  if (a.col.items) a.col.items = a.B * ceil_div64(a.col.NO, kThreads / LC);
  if (a.row.items) a.row.items = a.B * ceil_div64(a.row.NO, kThreads / LR);
  const int64_t items = a.col.items + a.row.items;
  // Segments of 16 steps and as many kept starts as an interval of 64 steps has, where that leaves room for two CTAs per
  // SM (a launch that does not fill the chip once may take the SM); else less history.
  const size_t most = items <= 148 && a.rowflag == nullptr ? kSmemMost : 112 * 1024;
  size_t smem = 0;
  for (int which = 0; which < 2; ++which) {
    LineArgs<T> &ln = which ? a.row : a.col;
    auto bytes = [&](int seg, int mids) {
      return 2 * (size_t)(3 * bwd_part<T>(seg, ln.NLn) + 3 * bwd_part<T>(seg, kThreads / (which ? LR : LC))) +
             (size_t)kWarpsPerCta * (seg + mids) * (which ? NR : NC) * 32 * sizeof(A);
    };
    int seg = 16, mids = 3;
    while (seg > 4 && bytes(seg, mids) > most) seg /= 2;
    while (bytes(seg, mids) > kSmemMost && (seg > 1 || mids > 1)) {
      if (mids > seg) mids /= 2;
      else seg /= 2;
    }
    while (mids < 7 && bytes(seg, mids + 4) <= most) mids += 4;
    ln.seg = seg;
    ln.mids = mids;
    if (ln.items && bytes(seg, mids) > smem) smem = bytes(seg, mids);
  }
  if (smem > kSmemMost) {
    set_error("lfw backward: %zu bytes of shared memory needed", smem);
    return T2FW_ERR_UNSUPPORTED;
  }
  auto *const kernel = &lfw_line_bwd_kernel<T, LC, NC, SC, LR, NR, SR>;
  T2FW_ALLOW_SMEM(kernel, (int)kSmemMost);
  T2FW_CHECK_CUDA(launch_dependent(kernel, dim3(grid_for(items, a.rowflag)), dim3(kThreads), smem, st, a));
  T2FW_CHECK_LAUNCH(1);
  return T2FW_OK;
}

// A rung serves the longer orientation's lines; `m` is the length of the other's.  Nearly as long: the same rung, without
// conditions on the elements that exist.  Up to half as long: half of the lanes with the same elements per lane (of eight
// lanes half of the elements).  Between: the same rung with conditions, or kInTurn where those would be ten and more per lane,
// which no registers keep: the lines are many there and two launches cost less.  fp32, 16 x 129, 96 x 48: 69.5 us (with
// conditions 80); 48 x 300, 100 x 50: 473 (728); 16 x 129, 96 x 64: 123.  In turn: 48 x 200, 60 x 90 303 (414 with conditions),
// 48 x 300, 100 x 60 725 (723), fp16 783 (860).
constexpr int kInTurn = -1;      // not a status
template <typename T, int L, int NL, int SAFE>
int launch_rung(const BwdArgs<T> &a, int m, cudaStream_t st) {
  if constexpr (SAFE > 0) {
    constexpr int LH = L > 8 ? L / 2 : 8, NH = L > 8 ? NL : (NL + 1) / 2;
    if (m > L * SAFE) return launch_lines<T, L, NL, SAFE, L, NL, SAFE>(a, st);
    if (m <= LH * NH)
      return a.col.NLn > a.row.NLn ? launch_lines<T, L, NL, SAFE, LH, NH, 0>(a, st) : launch_lines<T, LH, NH, 0, L, NL, SAFE>(a, st);
  }
  if constexpr (L == 8 && NL > 8) return kInTurn;
  else return launch_lines<T, L, NL, 0, L, NL, 0>(a, st);
}

// The orientations asked for, in one launch wherever a kernel has their pair of lengths.  Rungs: the smallest that holds the
// lines, for the number of lanes.
template <typename T>
int launch_bwd(BwdArgs<T> a, bool columns, bool rows, cudaStream_t st) {
  a.col.items = columns;
  a.row.items = rows;
  const int nc = columns ? a.col.NLn : a.row.NLn, nr = rows ? a.row.NLn : a.col.NLn;
  const int n = nc > nr ? nc : nr, m = nc < nr ? nc : nr;
  if constexpr (sizeof(T) == 8) {
    if (n <= 64) return launch_rung<T, 32, 2, 0>(a, m, st);
    if (n <= 128) return launch_rung<T, 32, 4, 0>(a, m, st);
    return n <= 256 ? launch_rung<T, 32, 8, 0>(a, m, st) : launch_rung<T, 32, 16, 0>(a, m, st);
  } else {
    if (n > 256) return launch_rung<T, 32, 16, 8>(a, m, st);
    if (n > 128) return launch_rung<T, 32, 8, 4>(a, m, st);
    const int lanes = a.rowflag != nullptr ? 8 : lanes_for(a.B * ((columns ? a.col.NO : a.row.NO) + (rows ? a.row.NO : a.col.NO)) / 2);
    if (lanes == 32)
      return n <= 32 ? launch_rung<T, 32, 1, 0>(a, m, st) : n <= 64 ? launch_rung<T, 32, 2, 1>(a, m, st)
             : n <= 96 ? launch_rung<T, 32, 3, 2>(a, m, st) : launch_rung<T, 32, 4, 3>(a, m, st);
    if (lanes >= 16) {
      if (n <= 32) return launch_rung<T, 16, 2, 0>(a, m, st);
      if (n <= 48) return launch_rung<T, 16, 3, 2>(a, m, st);
      if (n <= 64) return launch_rung<T, 16, 4, 3>(a, m, st);
      return n <= 96 ? launch_rung<T, 16, 6, 4>(a, m, st) : launch_rung<T, 16, 8, 6>(a, m, st);
    }
    if (n <= 16) return launch_rung<T, 8, 2, 0>(a, m, st);
    if (n <= 32) return launch_rung<T, 8, 4, 2>(a, m, st);
    if (n <= 64) return launch_rung<T, 8, 8, 4>(a, m, st);
    const int rc = n <= 80 ? launch_rung<T, 8, 10, 8>(a, m, st) : n <= 104 ? launch_rung<T, 8, 13, 10>(a, m, st)
                   : launch_rung<T, 8, 16, 13>(a, m, st);
    if (rc != kInTurn) return rc;
    const int first = launch_bwd<T>(a, true, false, st);      // lines of one length: their own rung
    return first != T2FW_OK ? first : launch_bwd<T>(a, false, true, st);
  }
}

}  // namespace

template <typename T>
int bwd_typed(const void *go, const void *gs, const void *x, const void *f, const void *q,
              const void *k, const void *fk, const void *state, const void *ckpt, void *dx,
              void *df, void *dq, void *dk, void *dfk, void *ds, int64_t B, int64_t T_, int64_t D,
              int64_t K, int64_t C, cudaStream_t st, const int *rowflag) {
  BwdArgs<T> a{};
  a.state0 = (const T *)state; a.ckpt = (const T *)ckpt; a.grad_state = (const T *)gs;
  a.B = B; a.T_ = T_; a.C = C < T_ ? C : T_; a.nslots = ceil_div64(T_, C); a.rowflag = rowflag;
  LineArgs<T> &row = a.row, &col = a.col;
  row.xo = (const T *)x; row.go = (const T *)f; row.po = (const T *)go;
  row.xl = (const T *)k; row.gl = (const T *)fk; row.pl = (const T *)q;
  row.d_xo = (T *)dx; row.d_go = (T *)df; row.d_po = nullptr; row.d_state = (T *)ds;
  row.NO = (int)D; row.NLn = (int)K; row.so = K; row.sl = 1;
  col.xo = (const T *)k; col.go = (const T *)fk; col.po = (const T *)q;
  col.xl = (const T *)x; col.gl = (const T *)f; col.pl = (const T *)go;
  col.d_xo = (T *)dk; col.d_go = (T *)dfk; col.d_po = (T *)dq; col.d_state = nullptr;
  col.NO = (int)K; col.NLn = (int)D; col.so = 1; col.sl = K;
  // Arrays that do not start on 16 bytes (views into larger buffers, a rare call) keep a launch per orientation, one after
  // the other.
  uintptr_t at = 0;
  for (const void *p : {go, gs, x, f, q, k, fk, state, ckpt}) at |= reinterpret_cast<uintptr_t>(p);
  if (rowflag != nullptr || at % 16 == 0) return launch_bwd<T>(a, true, true, st);
  const int rc = launch_bwd<T>(a, true, false, st);
  return rc != T2FW_OK ? rc : launch_bwd<T>(a, false, true, st);
}

#define T2FW_LFW_SCAN_TYPE(T)                                                                                             \
  template int fwd_typed<T>(const void *, const void *, const void *, const void *, const void *, const void *, void *,  \
                            void *, int64_t, int64_t, int64_t, int64_t, int64_t, cudaStream_t, const int *);             \
  template int bwd_typed<T>(const void *, const void *, const void *, const void *, const void *, const void *,          \
                            const void *, const void *, const void *, void *, void *, void *, void *, void *, void *,     \
                            int64_t, int64_t, int64_t, int64_t, int64_t, cudaStream_t, const int *);

#endif  // T2FW_LFW_SCAN_DEFINE

}  // namespace lfw_scan
}  // namespace t2fw
