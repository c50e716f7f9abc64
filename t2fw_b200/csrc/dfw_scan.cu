// Delta-rule ("DFW") scan kernels: every shape and type.
//
//   o_t = S_{t-1} q_t ,  delta_t = v_t - S_{t-1} k_t ,  S_t = S_{t-1} + delta_t k_t^T
//
// A line of the D x M state lies in the registers (accumulation type) of L lanes of a warp, element c in lane
// c % L; time is sequential and every reduction is a reduction over those lanes (deterministic).
//
//   forward  (own = d rows)    : outputs, delta, final state
//                                (reference kernel: t2fw/csrc/dfw_kernel.cu:105-196)
//   backward rows (own = d)    : d_value_t = G_t k_t, the G recurrence, d_state
//                                (reference kernel: t2fw/csrc/dfw_kernel.cu:198-283)
//   backward cols (own = m)    : d_query, d_key; walks the state column backwards from the
//                                final state, S_{t-1} = S_t - delta_t k_t^T
//                                (reference kernel: t2fw/csrc/dfw_kernel.cu:285-384)
//
// A chain of T steps bounds these kernels: in a step the products of a line are summed, the sum goes round the
// lanes and the line is updated with it.  L = 8 up to 128 elements (four lines per warp): three exchanges per sum
// instead of five, each of them for four lines, against eight to sixteen products per lane in two chains; longer
// lines take all 32 lanes.  Sixteen lanes would gain an eighth for few lines and lose half for many, and are left out (64 x 64,
// 150 steps, fp32, us at 8 / 16 / 32 lanes; forward: 192 lines 28.0 / 24.6 / 24.8, 1792 28.2 / 28.4 / 48.8, 3584
// 35.8 / 53.6 / 64.4; backward: 192 61 / 54 / 57, 1792 62 / 66 / 76, 4480 78 / 123 / 140).  The steps' vectors come from shared memory, fetched a group of steps ahead (scan.cuh).
// Whole call, fp32: 16 rows of 129 steps 96 x 48, forward and backward 278 -> 92 us; 48 rows of 300 steps 100 x 100
// 876 -> 480; forward alone, 40 rows of 200 steps 64 x 64, 139 -> 47.
#include "scan.cuh"

namespace t2fw {

namespace {

constexpr int kWarpsPerCta = 4;
constexpr int kThreads = kWarpsPerCta * 32;
constexpr int kSmemMost = 48 * 1024;
constexpr int lines_per_cta(int L) { return kWarpsPerCta * 32 / L; }

// n elements of one step's vectors, padded so that the next part of a buffer is 16-byte aligned
template <typename T>
__host__ __device__ inline int part(int G, int n) { return (int)((((size_t)G * n * sizeof(T)) + 15) / 16 * 16); }

template <int L, typename A>
__device__ __forceinline__ A line_sum(A v) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Elements l, l + L, .. of a row of n; the first SAFE are known to exist for every row that takes this NL
template <int L, int NL, int SAFE, typename T>
__device__ __forceinline__ void load_row(const T *row, int l, int n, typename Elem<T>::acc (&o)[NL]) {
#pragma unroll
  for (int j = 0; j < NL; ++j)
    o[j] = (j < SAFE || l + L * j < n) ? Elem<T>::ld(row + l + L * j) : typename Elem<T>::acc(0);
}

template <int NL, typename A>
__device__ __forceinline__ A dot(const A (&a)[NL], const A (&b)[NL]) {
  A s0 = A(0), s1 = A(0);      // two chains
#pragma unroll
  for (int j = 0; j < NL; j += 2) {
    s0 += a[j] * b[j];
    if (j + 1 < NL) s1 += a[j + 1] * b[j + 1];
  }
  return s0 + s1;
}

template <typename T>
struct FwdArgs {
  const T *q, *k, *v, *state;
  T *out, *fin;
  typename Elem<T>::acc *delta;
  int64_t T_;
  int D, M, G, blocks;      // steps per group, CTAs per batch row
};

// One buffer: k, q [G][M], v [G][lines of the CTA]
template <typename T, int L, int NL, int SAFE>
__global__ void __launch_bounds__(kThreads, sizeof(T) == 8 ? 2 : 4) dfw_fwd_kernel(const FwdArgs<T> a) {
  using A = typename Elem<T>::acc;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int RC = lines_per_cta(L);
  const int tid = threadIdx.x, l = tid % L, line = tid / L;
  const int64_t b = blockIdx.x / (unsigned)a.blocks;
  const int rb = (int)(blockIdx.x - b * a.blocks) * RC, nrows = a.D - rb < RC ? a.D - rb : RC;
  const bool in = line < nrows;
  const int mp = part<T>(a.G, a.M), buf_bytes = 2 * mp + part<T>(a.G, RC);
  dependency_wait();

  auto fetch = [&](int64_t t0, int which) {
    const int n = (int)(a.T_ - t0 < a.G ? a.T_ - t0 : a.G);
    unsigned char *p = smem_raw + which * buf_bytes;
    const int64_t mo = (b * a.T_ + t0) * a.M;
    scan::stage(reinterpret_cast<T *>(p), a.k + mo, n * a.M, tid, kThreads);
    scan::stage(reinterpret_cast<T *>(p + mp), a.q + mo, n * a.M, tid, kThreads);
    scan::stage_rows(reinterpret_cast<T *>(p + 2 * mp), a.v + (b * a.T_ + t0) * a.D + rb, n, nrows, a.D, tid, kThreads);
    scan::commit();
  };
  fetch(0, 0);

  const int64_t so = (b * a.D + rb + line) * a.M;
  A S[NL];
#pragma unroll
  for (int j = 0; j < NL; ++j) S[j] = in && l + L * j < a.M ? Elem<T>::ld(a.state + so + l + L * j) : A(0);

  int which = 0;
  for (int64_t t0 = 0; t0 < a.T_; t0 += a.G, which ^= 1) {
    if (t0 + a.G < a.T_) fetch(t0 + a.G, which ^ 1);
    else scan::commit();
    scan::wait<1>();
    __syncthreads();
    const int n = (int)(a.T_ - t0 < a.G ? a.T_ - t0 : a.G);
    const unsigned char *p = smem_raw + which * buf_bytes;
    const T *sk = reinterpret_cast<const T *>(p), *sq = reinterpret_cast<const T *>(p + mp);
    const T *sv = reinterpret_cast<const T *>(p + 2 * mp);
    const int64_t od = (b * a.T_ + t0) * a.D + rb + line;
    A kl[NL], ql[NL];
    load_row<L, NL, SAFE>(sk, l, a.M, kl);
    load_row<L, NL, SAFE>(sq, l, a.M, ql);
    A vt = in ? Elem<T>::ld(sv + line) : A(0);
    for (int t = 0; t < n; ++t) {
      const int tn = t + 1 < n ? t + 1 : t;      // the next step's vectors, ahead of this step's chain
      A kn[NL], qn[NL];
      load_row<L, NL, SAFE>(sk + tn * a.M, l, a.M, kn);
      load_row<L, NL, SAFE>(sq + tn * a.M, l, a.M, qn);
      const A vn = in ? Elem<T>::ld(sv + tn * nrows + line) : A(0);
      const A dl = vt - line_sum<L>(dot(S, kl));
      const A so_t = line_sum<L>(dot(S, ql));
#pragma unroll
      for (int j = 0; j < NL; ++j) S[j] += dl * kl[j];
      if (l == 0 && in) {
        Elem<T>::st(a.out + od + (int64_t)t * a.D, so_t);
        a.delta[od + (int64_t)t * a.D] = dl;
      }
#pragma unroll
      for (int j = 0; j < NL; ++j) { kl[j] = kn[j]; ql[j] = qn[j]; }
      vt = vn;
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < NL; ++j)
    if (in && l + L * j < a.M) Elem<T>::st(a.fin + so + l + L * j, S[j]);
}

template <typename T>
struct BwdArgs {
  const T *go, *gs, *q, *k, *fin;
  const typename Elem<T>::acc *delta;
  typename Elem<T>::acc *dv_acc;      // d_value in the accumulation type: written by the rows, read by the columns
  T *dq, *dk, *dv, *ds;
  int64_t T_;
  int D, M, G, blocks;
};

// rows: the recurrence of G_t, d_value, d_state.  One buffer: k, q [G][M], dO [G][lines of the CTA]
template <typename T, int L, int NL, int SAFE>
__global__ void __launch_bounds__(kThreads, sizeof(T) == 8 ? 2 : 4) dfw_bwd_rows_kernel(const BwdArgs<T> a) {
  using A = typename Elem<T>::acc;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int RC = lines_per_cta(L);
  const int tid = threadIdx.x, l = tid % L, line = tid / L;
  const int64_t b = blockIdx.x / (unsigned)a.blocks;
  const int rb = (int)(blockIdx.x - b * a.blocks) * RC, nrows = a.D - rb < RC ? a.D - rb : RC;
  const bool in = line < nrows;
  const bool two = static_cast<const void *>(a.dv) != static_cast<const void *>(a.dv_acc);
  const int mp = part<T>(a.G, a.M), buf_bytes = 2 * mp + part<T>(a.G, RC);
  dependency_wait();

  auto fetch = [&](int64_t t0, int which) {
    const int n = (int)(a.T_ - t0 < a.G ? a.T_ - t0 : a.G);
    unsigned char *p = smem_raw + which * buf_bytes;
    const int64_t mo = (b * a.T_ + t0) * a.M;
    scan::stage(reinterpret_cast<T *>(p), a.k + mo, n * a.M, tid, kThreads);
    scan::stage(reinterpret_cast<T *>(p + mp), a.q + mo, n * a.M, tid, kThreads);
    scan::stage_rows(reinterpret_cast<T *>(p + 2 * mp), a.go + (b * a.T_ + t0) * a.D + rb, n, nrows, a.D, tid, kThreads);
    scan::commit();
  };
  int64_t t0 = (a.T_ - 1) / a.G * a.G;
  fetch(t0, 0);

  const int64_t so = (b * a.D + rb + line) * a.M;
  A G[NL];
#pragma unroll
  for (int j = 0; j < NL; ++j) G[j] = in && l + L * j < a.M ? Elem<T>::ld(a.gs + so + l + L * j) : A(0);

  int which = 0;
  for (; t0 >= 0; t0 -= a.G, which ^= 1) {
    if (t0 > 0) fetch(t0 - a.G, which ^ 1);
    else scan::commit();
    scan::wait<1>();
    __syncthreads();
    const int n = (int)(a.T_ - t0 < a.G ? a.T_ - t0 : a.G);
    const unsigned char *p = smem_raw + which * buf_bytes;
    const T *sk = reinterpret_cast<const T *>(p), *sq = reinterpret_cast<const T *>(p + mp);
    const T *sg = reinterpret_cast<const T *>(p + 2 * mp);
    const int64_t od = (b * a.T_ + t0) * a.D + rb + line;
    A kl[NL], ql[NL];
    load_row<L, NL, SAFE>(sk + (n - 1) * a.M, l, a.M, kl);
    load_row<L, NL, SAFE>(sq + (n - 1) * a.M, l, a.M, ql);
    A gt = in ? Elem<T>::ld(sg + (n - 1) * nrows + line) : A(0);
    for (int t = n - 1; t >= 0; --t) {
      const int tn = t > 0 ? t - 1 : 0;      // the next step's vectors, ahead of this step's chain
      A kn[NL], qn[NL];
      load_row<L, NL, SAFE>(sk + tn * a.M, l, a.M, kn);
      load_row<L, NL, SAFE>(sq + tn * a.M, l, a.M, qn);
      const A gn = in ? Elem<T>::ld(sg + tn * nrows + line) : A(0);
      const A s = line_sum<L>(dot(G, kl));
#pragma unroll
      for (int j = 0; j < NL; ++j) G[j] = (G[j] + gt * ql[j]) - s * kl[j];
      if (l == 0 && in) {
        Elem<T>::st(a.dv + od + (int64_t)t * a.D, s);
        if (two) a.dv_acc[od + (int64_t)t * a.D] = s;
      }
#pragma unroll
      for (int j = 0; j < NL; ++j) { kl[j] = kn[j]; ql[j] = qn[j]; }
      gt = gn;
    }
    __syncthreads();
  }
#pragma unroll
  for (int j = 0; j < NL; ++j)
    if (in && l + L * j < a.M) Elem<T>::st(a.ds + so + l + L * j, G[j]);
}

// columns: d_query, d_key (own = m, lanes over d).  One buffer: delta, d_value, dO [G][D], k, q [G][lines of the CTA]
template <typename T, int L, int NL, int SAFE>
__global__ void __launch_bounds__(kThreads, sizeof(T) == 8 ? 2 : 4) dfw_bwd_cols_kernel(const BwdArgs<T> a) {
  using A = typename Elem<T>::acc;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int RC = lines_per_cta(L);
  const int tid = threadIdx.x, l = tid % L, line = tid / L;
  const int64_t b = blockIdx.x / (unsigned)a.blocks;
  const int mb = (int)(blockIdx.x - b * a.blocks) * RC, ncols = a.M - mb < RC ? a.M - mb : RC;
  const bool in = line < ncols;
  const int ap = part<A>(a.G, a.D), dp = part<T>(a.G, a.D), op = part<T>(a.G, RC), buf_bytes = 2 * ap + dp + 2 * op;
  dependency_wait();

  auto fetch = [&](int64_t t0, int which) {
    const int n = (int)(a.T_ - t0 < a.G ? a.T_ - t0 : a.G);
    unsigned char *p = smem_raw + which * buf_bytes;
    const int64_t od = (b * a.T_ + t0) * a.D, om = (b * a.T_ + t0) * a.M + mb;
    scan::stage(reinterpret_cast<A *>(p), a.delta + od, n * a.D, tid, kThreads);
    scan::stage(reinterpret_cast<A *>(p + ap), static_cast<const A *>(a.dv_acc) + od, n * a.D, tid, kThreads);
    scan::stage(reinterpret_cast<T *>(p + 2 * ap), a.go + od, n * a.D, tid, kThreads);
    scan::stage_rows(reinterpret_cast<T *>(p + 2 * ap + dp), a.k + om, n, ncols, a.M, tid, kThreads);
    scan::stage_rows(reinterpret_cast<T *>(p + 2 * ap + dp + op), a.q + om, n, ncols, a.M, tid, kThreads);
    scan::commit();
  };
  int64_t t0 = (a.T_ - 1) / a.G * a.G;
  fetch(t0, 0);

  A G[NL], S[NL];
#pragma unroll
  for (int j = 0; j < NL; ++j) {
    const int64_t o = (b * a.D + l + L * j) * a.M + mb + line;
    const bool ok = in && l + L * j < a.D;
    G[j] = ok ? Elem<T>::ld(a.gs + o) : A(0);
    S[j] = ok ? Elem<T>::ld(a.fin + o) : A(0);
  }

  int which = 0;
  for (; t0 >= 0; t0 -= a.G, which ^= 1) {
    if (t0 > 0) fetch(t0 - a.G, which ^ 1);
    else scan::commit();
    scan::wait<1>();
    __syncthreads();
    const int n = (int)(a.T_ - t0 < a.G ? a.T_ - t0 : a.G);
    const unsigned char *p = smem_raw + which * buf_bytes;
    const A *sd = reinterpret_cast<const A *>(p), *se = reinterpret_cast<const A *>(p + ap);
    const T *sg = reinterpret_cast<const T *>(p + 2 * ap);
    const T *sk = reinterpret_cast<const T *>(p + 2 * ap + dp), *sq = reinterpret_cast<const T *>(p + 2 * ap + dp + op);
    const int64_t om = (b * a.T_ + t0) * a.M + mb + line;
#pragma unroll 2
    for (int t = n - 1; t >= 0; --t) {
      A dl[NL], el[NL], gl[NL];
      load_row<L, NL, SAFE>(sg + t * a.D, l, a.D, gl);
#pragma unroll
      for (int j = 0; j < NL; ++j) {
        const bool ok = j < SAFE || l + L * j < a.D;
        dl[j] = ok ? sd[t * a.D + l + L * j] : A(0);
        el[j] = ok ? se[t * a.D + l + L * j] : A(0);
      }
      const A km = in ? Elem<T>::ld(sk + t * ncols + line) : A(0);
      const A qm = in ? Elem<T>::ld(sq + t * ncols + line) : A(0);
      A aq = A(0), ak = A(0);
#pragma unroll
      for (int j = 0; j < NL; ++j) {
        const A sp = S[j] - dl[j] * km;      // S_{t-1}
        aq += gl[j] * sp;
        ak += dl[j] * G[j] - el[j] * sp;
        G[j] += gl[j] * qm - el[j] * km;
        S[j] = sp;
      }
      // half of the lanes go on with one sum, half with the other
      const bool up = (l & (L / 2)) != 0;
      const A send = up ? aq : ak, keep = up ? ak : aq;
      const A sum = line_sum<L / 2>(keep + __shfl_xor_sync(0xffffffffu, send, L / 2));
      if (l % (L / 2) == 0 && in) Elem<T>::st((up ? a.dk : a.dq) + om + (int64_t)t * a.M, sum);
    }
    __syncthreads();
  }
}

// Steps per group: as many as two buffers hold in 48 KB (several CTAs per SM), at most 32
template <typename F>
int group_steps(int64_t T_, F bytes) {
  int G = 32;
  while (G > 1 && (G / 2 >= T_ || 2 * bytes(G) > (size_t)kSmemMost)) G /= 2;
  return G;
}

template <typename T, int L, int NL, int SAFE>
int launch_fwd(FwdArgs<T> a, int64_t B, cudaStream_t st) {
  constexpr int RC = lines_per_cta(L);
  auto bytes = [&](int G) { return (size_t)(2 * part<T>(G, a.M) + part<T>(G, RC)); };
  a.G = group_steps(a.T_, bytes);
  a.blocks = (a.D + RC - 1) / RC;
  T2FW_CHECK_CUDA(launch_dependent(&dfw_fwd_kernel<T, L, NL, SAFE>, dim3((unsigned)(B * a.blocks)), dim3(kThreads),
                                   2 * bytes(a.G), st, a));
  T2FW_CHECK_LAUNCH(1);
  return T2FW_OK;
}

template <typename T, int L, int NL, int SAFE>
int launch_rows(BwdArgs<T> a, int64_t B, cudaStream_t st) {
  constexpr int RC = lines_per_cta(L);
  auto bytes = [&](int G) { return (size_t)(2 * part<T>(G, a.M) + part<T>(G, RC)); };
  a.G = group_steps(a.T_, bytes);
  a.blocks = (a.D + RC - 1) / RC;
  T2FW_CHECK_CUDA(launch_dependent(&dfw_bwd_rows_kernel<T, L, NL, SAFE>, dim3((unsigned)(B * a.blocks)), dim3(kThreads),
                                   2 * bytes(a.G), st, a));
  T2FW_CHECK_LAUNCH(1);
  return T2FW_OK;
}

template <typename T, int L, int NL, int SAFE>
int launch_cols(BwdArgs<T> a, int64_t B, cudaStream_t st) {
  using A = typename Elem<T>::acc;
  constexpr int RC = lines_per_cta(L);
  auto bytes = [&](int G) { return (size_t)(2 * part<A>(G, a.D) + part<T>(G, a.D) + 2 * part<T>(G, RC)); };
  a.G = group_steps(a.T_, bytes);
  a.blocks = (a.M + RC - 1) / RC;
  T2FW_CHECK_CUDA(launch_dependent(&dfw_bwd_cols_kernel<T, L, NL, SAFE>, dim3((unsigned)(B * a.blocks)), dim3(kThreads),
                                   2 * bytes(a.G), st, a));
  T2FW_CHECK_LAUNCH(1);
  return T2FW_OK;
}

// Lanes per line and elements per lane for lines of n elements: the smallest that holds them.
#define T2FW_DFW_LINES(n, call)                       \
  do {                                                \
    const int64_t _n = (n);                           \
    if (_n <= 16) return call(8, 2, 0);               \
    if (_n <= 32) return call(8, 4, 2);               \
    if (_n <= 48) return call(8, 6, 4);               \
    if (_n <= 64) return call(8, 8, 6);               \
    if (_n <= 80) return call(8, 10, 8);              \
    if (_n <= 104) return call(8, 13, 10);            \
    if (_n <= 128) return call(8, 16, 13);            \
    if (_n <= 256) return call(32, 8, 4);             \
    if (_n <= 512) return call(32, 16, 8);            \
  } while (0)

template <typename T>
int fwd_typed(const void *q, const void *k, const void *v, const void *state, void *out,
              void *fin, void *delta, int64_t B, int64_t T_, int64_t D, int64_t M,
              cudaStream_t st) {
  FwdArgs<T> a{};
  a.q = (const T *)q; a.k = (const T *)k; a.v = (const T *)v; a.state = (const T *)state;
  a.out = (T *)out; a.fin = (T *)fin; a.delta = (typename Elem<T>::acc *)delta;
  a.T_ = T_; a.D = (int)D; a.M = (int)M;
#define T2FW_CALL(L, NL, SAFE) launch_fwd<T, L, NL, SAFE>(a, B, st)
  T2FW_DFW_LINES(M, T2FW_CALL);
#undef T2FW_CALL
  set_error("dfw forward: M=%lld exceeds the supported maximum of 512", (long long)M);
  return T2FW_ERR_UNSUPPORTED;
}

template <typename T>
int rows_typed(const BwdArgs<T> &a, int64_t B, cudaStream_t st) {
#define T2FW_CALL(L, NL, SAFE) launch_rows<T, L, NL, SAFE>(a, B, st)
  T2FW_DFW_LINES(a.M, T2FW_CALL);
#undef T2FW_CALL
  return T2FW_ERR_UNSUPPORTED;
}

template <typename T>
int cols_typed(const BwdArgs<T> &a, int64_t B, cudaStream_t st) {
#define T2FW_CALL(L, NL, SAFE) launch_cols<T, L, NL, SAFE>(a, B, st)
  T2FW_DFW_LINES(a.D, T2FW_CALL);
#undef T2FW_CALL
  return T2FW_ERR_UNSUPPORTED;
}
#undef T2FW_DFW_LINES

template <typename T>
int bwd_typed(const void *go, const void *gs, const void *q, const void *k, const void *delta,
              const void *fin, void *dq, void *dk, void *dv, void *ds, void *dv_acc, int64_t B,
              int64_t T_, int64_t D, int64_t M, cudaStream_t st) {
  using A = typename Elem<T>::acc;
  if (D > 512 || M > 512) {
    set_error("dfw backward: D=%lld, M=%lld exceed the supported maximum of 512", (long long)D,
              (long long)M);
    return T2FW_ERR_UNSUPPORTED;
  }
  BwdArgs<T> a{};
  a.go = (const T *)go; a.gs = (const T *)gs; a.q = (const T *)q; a.k = (const T *)k; a.fin = (const T *)fin;
  a.delta = (const A *)delta; a.dv_acc = (A *)dv_acc;
  a.dq = (T *)dq; a.dk = (T *)dk; a.dv = (T *)dv; a.ds = (T *)ds;
  a.T_ = T_; a.D = (int)D; a.M = (int)M;
  const int rc = rows_typed<T>(a, B, st);
  return rc != T2FW_OK ? rc : cols_typed<T>(a, B, st);
}

}  // namespace

int dfw_scan_forward(const void *q, const void *k, const void *v, const void *state, void *out,
                     void *fin, void *delta, int64_t B, int64_t T_, int64_t D, int64_t M,
                     int dtype, cudaStream_t st) {
  switch (dtype) {
    case T2FW_F16: return fwd_typed<__half>(q, k, v, state, out, fin, delta, B, T_, D, M, st);
    case T2FW_BF16: return fwd_typed<__nv_bfloat16>(q, k, v, state, out, fin, delta, B, T_, D, M, st);
    case T2FW_F32: return fwd_typed<float>(q, k, v, state, out, fin, delta, B, T_, D, M, st);
    case T2FW_F64: return fwd_typed<double>(q, k, v, state, out, fin, delta, B, T_, D, M, st);
  }
  set_error("unknown dtype %d", dtype);
  return T2FW_ERR_BAD_ARG;
}

int dfw_scan_backward(const void *go, const void *gs, const void *q, const void *k,
                      const void *delta, const void *fin, void *dq, void *dk, void *dv, void *ds,
                      void *dv_acc, int64_t B, int64_t T_, int64_t D, int64_t M, int dtype,
                      cudaStream_t st) {
  switch (dtype) {
    case T2FW_F16:
      return bwd_typed<__half>(go, gs, q, k, delta, fin, dq, dk, dv, ds, dv_acc, B, T_, D, M, st);
    case T2FW_BF16:
      return bwd_typed<__nv_bfloat16>(go, gs, q, k, delta, fin, dq, dk, dv, ds, dv_acc, B, T_, D, M, st);
    case T2FW_F32:
      return bwd_typed<float>(go, gs, q, k, delta, fin, dq, dk, dv, ds, dv_acc, B, T_, D, M, st);
    case T2FW_F64:
      return bwd_typed<double>(go, gs, q, k, delta, fin, dq, dk, dv, ds, dv_acc, B, T_, D, M, st);
  }
  set_error("unknown dtype %d", dtype);
  return T2FW_ERR_BAD_ARG;
}

}  // namespace t2fw
