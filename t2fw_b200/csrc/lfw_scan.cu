// Decay-rule scan kernels: choice of the storage type.  The kernels are in lfw_scan.cuh.
#include "lfw_scan.cuh"

namespace t2fw {

using namespace lfw_scan;

int lfw_scan_forward(const void *x, const void *f, const void *q, const void *k, const void *fk,
                     const void *state, void *out, void *ckpt, int64_t B, int64_t T_, int64_t D,
                     int64_t K, int dtype, int64_t C, cudaStream_t st, const int *rowflag) {
  switch (dtype) {
    case T2FW_F16: return fwd_typed<__half>(x, f, q, k, fk, state, out, ckpt, B, T_, D, K, C, st, rowflag);
    case T2FW_BF16: return fwd_typed<__nv_bfloat16>(x, f, q, k, fk, state, out, ckpt, B, T_, D, K, C, st, rowflag);
    case T2FW_F32: return fwd_typed<float>(x, f, q, k, fk, state, out, ckpt, B, T_, D, K, C, st, rowflag);
    case T2FW_F64: return fwd_typed<double>(x, f, q, k, fk, state, out, ckpt, B, T_, D, K, C, st, rowflag);
  }
  set_error("unknown dtype %d", dtype);
  return T2FW_ERR_BAD_ARG;
}

int lfw_scan_backward(const void *go, const void *gs, const void *x, const void *f, const void *q,
                      const void *k, const void *fk, const void *state, const void *ckpt,
                      void *dx, void *df, void *dq, void *dk, void *dfk, void *ds, int64_t B,
                      int64_t T_, int64_t D, int64_t K, int dtype, int64_t C, cudaStream_t st,
                      const int *rowflag) {
  if (D > 512 || K > 512) {
    set_error("lfw backward: D=%lld, K=%lld exceed the supported maximum of 512", (long long)D,
              (long long)K);
    return T2FW_ERR_UNSUPPORTED;
  }
  switch (dtype) {
    case T2FW_F16:
      return bwd_typed<__half>(go, gs, x, f, q, k, fk, state, ckpt, dx, df, dq, dk, dfk, ds, B, T_, D, K, C, st, rowflag);
    case T2FW_BF16:
      return bwd_typed<__nv_bfloat16>(go, gs, x, f, q, k, fk, state, ckpt, dx, df, dq, dk, dfk, ds, B, T_, D, K, C, st, rowflag);
    case T2FW_F32:
      return bwd_typed<float>(go, gs, x, f, q, k, fk, state, ckpt, dx, df, dq, dk, dfk, ds, B, T_, D, K, C, st, rowflag);
    case T2FW_F64:
      return bwd_typed<double>(go, gs, x, f, q, k, fk, state, ckpt, dx, df, dq, dk, dfk, ds, B, T_, D, K, C, st, rowflag);
  }
  set_error("unknown dtype %d", dtype);
  return T2FW_ERR_BAD_ARG;
}

}  // namespace t2fw
