// Short sequences walked step by step with the state in registers: the decay rule over n steps (a ring of
// decode steps, or a whole T < 64 forward call) and the delta rule over a few steps, 16-bit storage.
//
// Why a kernel of its own: a chain of n decode launches moves the whole state through memory n times and
// pays a launch each time (512 rows: 3.6 us per step); a chunked call on a short sequence pays three
// dependent launches and the padding to 64 steps.  Here the state is read once, kept in fp32 registers and
// written once, and the steps' vectors (640 bytes per step at D = K = 64) arrive in shared memory in
// double-buffered groups of eight steps.  Few rows: bound by launch and the latency of a step (0.15 us);
// many rows: by shared-memory reads of the key-side vectors (three 16-byte reads per thread for R rows) and
// about 16 packed instructions per eight columns and step, 1 us per 1000 row-steps.  Keeping the vectors in
// shared memory as fp32 saves the conversions but doubles those reads and was slower (96 rows x 48 steps:
// 19.3 us against 14.5).  Forward call at D = K = 64, fp16, chunked -> here: 96 rows x 2 steps 23.3 -> 2.2 us,
// 96 x 48 19.8 -> 14.5, 2048 x 48 205 -> 105; delta rule 96 x 1 16.2 -> 1.9, 2048 x 48 164 -> 93.
//
// A CTA of 128 threads owns R * 1024 / K rows of one batch item's state: thread (rr, kc) the eight columns
// 8 kc .. of R rows.  Rows are independent of one another given the key-side vectors, so a small batch is
// spread over more CTAs by giving each thread fewer rows (R = 4, 2, 1).
// Replaces t2fw/csrc/lfw_kernel.cu:18-59 with the einsum of t2fw/csrc/lfw.cpp:45, and
// t2fw/csrc/dfw_kernel.cu:105-196, for these sizes.
#include "seq_layout.cuh"
#include "steps.cuh"

namespace t2fw {

using namespace steps;

namespace {

constexpr int kThreadsS = 128;
constexpr int kGroup = 8;      // steps whose vectors are fetched together

template <typename T>
struct StepArgs {
  const T *x, *f, *q, *k, *fk, *state;      // delta rule: x = value, f and fk unused
  T *out, *next;
  float *delta;                             // delta rule only
  int64_t row_d, step_d, row_k, step_k;     // element strides of a batch item and of a step
  int64_t step_o;                           // fused layer: stride of a step in the outputs
  int n, D, slabs;
  int heads;                                // rows of the grid per batch item: row b h reads 64-column window h
  float q_scale;                            // fused layer
};

// kRing: the state is rounded to the storage type after every step, as a chain of single-step calls through
// memory does it; in the other modes it stays fp32 to the end, as in a T > 1 call.
// kFused: decay-rule layer on a projection output, query | key | value | gate of all heads in one row: the
// query scale and the gate activation are applied to the fetched vectors (rounded to the storage type, as a
// separate pass followed by the plain operator would have left them) and the forget gate is 1.
enum class Mode { kDecay, kRing, kFused, kDelta };

template <typename T, int KT, int R, Mode kMode>
__global__ void __launch_bounds__(kThreadsS)
steps_kernel(const StepArgs<T> a) {
  constexpr bool kDelta = kMode == Mode::kDelta, kFused = kMode == Mode::kFused;
  constexpr int K = 8 * KT, RP = kThreadsS / KT, SL = R * RP;      // rows of this CTA
  constexpr int kKvecs = kDelta ? 2 : 3, kDvecs = kDelta || kFused ? 1 : 2;
  constexpr int kStep = kKvecs * K + kDvecs * SL;                  // elements per step in shared memory
  __shared__ __align__(16) T buf[2][kGroup * kStep];
  const int tid = threadIdx.x, kc = tid % KT, rr = tid / KT;
  dependency_wait();
  const int64_t b = blockIdx.x / a.slabs;
  const int d0 = (int)(blockIdx.x % a.slabs) * SL;
  const int rows = a.D - d0 < SL ? a.D - d0 : SL;
  // sequence vectors of this row: batch item and 64-column window (one window for the plain operators)
  const int64_t item = kFused ? b / a.heads : b;
  const int64_t off_d = item * a.row_d + (kFused ? (b % a.heads) * 64 : 0) + d0;
  const int64_t off_k = item * a.row_k + (kFused ? (b % a.heads) * 64 : 0);
  // outputs (and deltas) are [B][T][D] with all heads in a row
  const int64_t off_o = kFused ? item * a.n * a.step_o + (b % a.heads) * 64 + d0 : off_d;
  const int64_t step_o = kFused ? a.step_o : a.step_d;

  // 16-byte pieces of a step: fk | k | q | x | f   (delta rule: k | q | v)
  const T *const kv0 = kDelta ? a.k : a.fk, *const kv1 = kDelta ? a.q : a.k;
  auto fetch = [&](int t0, int which) {
    constexpr int kP = kKvecs * KT, dP = SL / 8, per = kP + kDvecs * dP;
    for (int i = tid; i < kGroup * per; i += kThreadsS) {
      const int t = i / per, p = i % per;
      if (t0 + t >= a.n) break;
      T *dst = &buf[which][t * kStep];
      if (p < kP) {
        const int v = p / KT, o = (p % KT) * 8;
        cp_async16(dst + v * K + o,
                   (v == 0 ? kv0 : v == 1 ? kv1 : a.q) + off_k + (int64_t)(t0 + t) * a.step_k + o);
      } else {
        const int v = (p - kP) / dP, o = ((p - kP) % dP) * 8;
        if (o < rows)
          cp_async16(dst + kKvecs * K + v * SL + o,
                     (v == 0 ? a.x : a.f) + off_d + (int64_t)(t0 + t) * a.step_d + o);
      }
    }
    cp_async_commit();
  };
  fetch(0, 0);

  f2 S[R][4];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int row = r * RP + rr;
    const uint4 u = row < rows ? *reinterpret_cast<const uint4 *>(a.state + ((b * a.D + d0 + row) * K + 8 * kc))
                               : make_uint4(0, 0, 0, 0);
    Oct<T>::unpack(u, S[r]);
  }

  for (int t0 = 0, which = 0; t0 < a.n; t0 += kGroup, which ^= 1) {
    if (t0 + kGroup < a.n) fetch(t0 + kGroup, which ^ 1);
    else cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    const int nt = a.n - t0 < kGroup ? a.n - t0 : kGroup;
    if constexpr (kFused) {
      for (int i = tid; i < nt * K; i += kThreadsS) {
        T *g = &buf[which][(i / K) * kStep + i % K], *q = g + 2 * K;
        Elem<T>::st(g, seq::sigmoid_gate<T>(Elem<T>::ld(g)));      // the backward's gate, bit for bit
        *q = (T)(Elem<T>::ld(q) * a.q_scale);
      }
      __syncthreads();
    }
#pragma unroll 2
    for (int t = 0; t < nt; ++t) {
      const T *p = &buf[which][t * kStep];
      const T *pd = p + kKvecs * K + rr;
      auto column = [&](int v, f2 (&o)[4]) { Oct<T>::unpack(reinterpret_cast<const uint4 *>(p + v * K)[kc], o); };
      auto both = [](const T *v) { const float w = Elem<T>::ld(v); return pack2(w, w); };
      float acc[R];
      if constexpr (!kDelta) {
        f2 g[4], k[4], q[4];
        column(0, g);
        column(1, k);
        column(2, q);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          acc[r] = decay_step8(S[r], g, k, q, both(pd + r * RP), kFused ? pack2(1.f, 1.f) : both(pd + SL + r * RP));
          if (kMode == Mode::kRing) {
            const uint4 u = Oct<T>::pack(S[r]);
            Oct<T>::unpack(u, S[r]);
          }
        }
      } else {
        f2 k[4], q[4];
        column(0, k);
        column(1, q);
        float sk[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {      // outputs and deltas come from the state before the update
          f2 ao = 0ull, ak = 0ull;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            ao = fma2(S[r][e], q[e], ao);
            ak = fma2(S[r][e], k[e], ak);
          }
          float lo, hi;
          unpack2(ao, lo, hi);
          acc[r] = lo + hi;
          unpack2(ak, lo, hi);
          sk[r] = lo + hi;
        }
#pragma unroll
        for (int o = KT >> 1; o > 0; o >>= 1)
#pragma unroll
          for (int r = 0; r < R; ++r) sk[r] += __shfl_xor_sync(0xffffffffu, sk[r], o);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float dl = Elem<T>::ld(pd + r * RP) - sk[r];
          const f2 d2 = pack2(dl, dl);
#pragma unroll
          for (int e = 0; e < 4; ++e) S[r][e] = fma2(d2, k[e], S[r][e]);
          const int row = r * RP + rr;
          if (kc == 0 && row < rows) a.delta[off_o + (int64_t)(t0 + t) * step_o + row] = dl;
        }
      }
      int r;
      if (row_sums<KT, R>(acc, kc, &r)) {
        const int row = r * RP + rr;
        if (row < rows) Elem<T>::st(a.out + off_o + (int64_t)(t0 + t) * step_o + row, acc[0]);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int row = r * RP + rr;
    if (row < rows) *reinterpret_cast<uint4 *>(a.next + ((b * a.D + d0 + row) * K + 8 * kc)) = Oct<T>::pack(S[r]);
  }
}

template <typename T, int KT, int R, Mode kMode>
int launch(StepArgs<T> a, int64_t B, cudaStream_t st) {
  constexpr int SL = R * (kThreadsS / KT);
  a.slabs = (a.D + SL - 1) / SL;
  T2FW_CHECK_CUDA(launch_dependent(steps_kernel<T, KT, R, kMode>, dim3((unsigned)(B * a.slabs)), dim3(kThreadsS), 0,
                                   st, a));
  T2FW_CHECK_LAUNCH(1);
  return T2FW_OK;
}

// Rows per thread: four amortise the loads of the key-side vectors best; fewer while the grid would leave
// SMs without a CTA (148 SMs, two CTAs each).
template <typename T, int KT, Mode kMode>
int by_rows(const StepArgs<T> &a, int64_t B, cudaStream_t st) {
  constexpr int RP = kThreadsS / KT;
  auto ctas = [&](int r) { return B * ((a.D + r * RP - 1) / (r * RP)); };
  if (a.D > 2 * RP && ctas(4) >= 2 * 148) return launch<T, KT, 4, kMode>(a, B, st);
  if (a.D > RP && ctas(2) >= 2 * 148) return launch<T, KT, 2, kMode>(a, B, st);
  return launch<T, KT, 1, kMode>(a, B, st);
}

template <typename T, Mode kMode>
int by_k(const StepArgs<T> &a, int64_t B, int64_t K, cudaStream_t st) {
  switch (K) {
    case 32: return by_rows<T, 4, kMode>(a, B, st);
    case 64: return by_rows<T, 8, kMode>(a, B, st);
    case 128: return by_rows<T, 16, kMode>(a, B, st);
  }
  set_error("step kernel: K=%lld is not covered", (long long)K);
  return T2FW_ERR_UNSUPPORTED;
}

template <typename T>
StepArgs<T> step_args(const void *x, const void *f, const void *q, const void *k, const void *fk, const void *state,
                      void *out, void *next, void *delta, int64_t n, int64_t D, int64_t row_d, int64_t step_d,
                      int64_t row_k, int64_t step_k) {
  StepArgs<T> a{};
  a.x = (const T *)x; a.f = (const T *)f; a.q = (const T *)q; a.k = (const T *)k; a.fk = (const T *)fk;
  a.state = (const T *)state; a.out = (T *)out; a.next = (T *)next; a.delta = (float *)delta;
  a.row_d = row_d; a.step_d = step_d; a.row_k = row_k; a.step_k = step_k;
  a.n = (int)n; a.D = (int)D;
  return a;
}

}  // namespace

bool steps_supported(int64_t B, int64_t D, int64_t K, int dtype) {
  return (dtype == T2FW_F16 || dtype == T2FW_BF16) && (K == 32 || K == 64 || K == 128) && D % 8 == 0 && D <= 512 &&
         B * 64 < (1ll << 31);
}

// n decay-rule steps on x, f [n][B][D] and q, k, fk [n][B][K], the state rounded after every step
int lfw_steps_ring(const void *x, const void *f, const void *q, const void *k, const void *fk, const void *state,
                   void *out, void *next, int64_t n, int64_t B, int64_t D, int64_t K, int dtype, cudaStream_t st) {
  if (dtype == T2FW_F16)
    return by_k<__half, Mode::kRing>(step_args<__half>(x, f, q, k, fk, state, out, next, nullptr, n, D, D, B * D, K, B * K), B, K, st);
  return by_k<__nv_bfloat16, Mode::kRing>(step_args<__nv_bfloat16>(x, f, q, k, fk, state, out, next, nullptr, n, D, D, B * D, K, B * K), B, K, st);
}

// a forward call of T steps on [B][T][D] / [B][T][K] arrays with one checkpoint slot (the next state)
int lfw_steps_forward(const void *x, const void *f, const void *q, const void *k, const void *fk, const void *state,
                      void *out, void *next, int64_t B, int64_t T_, int64_t D, int64_t K, int dtype, cudaStream_t st) {
  if (dtype == T2FW_F16)
    return by_k<__half, Mode::kDecay>(step_args<__half>(x, f, q, k, fk, state, out, next, nullptr, T_, D, T_ * D, D, T_ * K, K), B, K, st);
  return by_k<__nv_bfloat16, Mode::kDecay>(step_args<__nv_bfloat16>(x, f, q, k, fk, state, out, next, nullptr, T_, D, T_ * D, D, T_ * K, K), B, K, st);
}

// the fused layer on qkvg [B][T][4 H 64] = query | key | value | gate, outputs [B][T][H 64]
int lfw_steps_fused(const void *qkvg, const void *state, void *out, void *next, int64_t B, int64_t T_, int H, int dtype,
                    cudaStream_t st) {
  const int64_t C = (int64_t)H * 64;
#define T2FW_FUSED(TT)                                                                                                   \
  do {                                                                                                                   \
    const TT *p = (const TT *)qkvg;                                                                                      \
    StepArgs<TT> a = step_args<TT>(p + 2 * C, nullptr, p, p + C, p + 3 * C, state, out, next, nullptr, T_, 64, T_ * 4 * C, \
                                   4 * C, T_ * 4 * C, 4 * C);                                                            \
    a.heads = H;                                                                                                         \
    a.q_scale = 0.125f; /* 1 / sqrt(64) */                                                                               \
    a.step_o = C;                                                                                                        \
    return by_rows<TT, 8, Mode::kFused>(a, B * H, st);                                                                   \
  } while (0)
  if (dtype == T2FW_F16) T2FW_FUSED(__half);
  T2FW_FUSED(__nv_bfloat16);
#undef T2FW_FUSED
}

int dfw_steps_forward(const void *q, const void *k, const void *v, const void *state, void *out, void *fin, void *delta,
                      int64_t B, int64_t T_, int64_t D, int64_t M, int dtype, cudaStream_t st) {
  if (dtype == T2FW_F16)
    return by_k<__half, Mode::kDelta>(step_args<__half>(v, nullptr, q, k, nullptr, state, out, fin, delta, T_, D, T_ * D, D, T_ * M, M), B, M, st);
  return by_k<__nv_bfloat16, Mode::kDelta>(step_args<__nv_bfloat16>(v, nullptr, q, k, nullptr, state, out, fin, delta, T_, D, T_ * D, D, T_ * M, M), B, M, st);
}

}  // namespace t2fw
