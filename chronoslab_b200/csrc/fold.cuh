// Apply kernel of folded levels (fold.cu): the two-matrix row product.
#pragma once

#include "hier.h"
#include "spmv.cuh"

namespace chronos {

// out = Q b + E e on a folded level, L lanes per row (and out . dw).
template <typename T, typename BT, typename OT, int L, bool DOT, bool QI16, bool EI16>
__global__ void __launch_bounds__(kApplyThreads)
k_fold_apply(int n, const int *__restrict__ qrp, const int *__restrict__ qci,
             const int *__restrict__ qbase, const uint16_t *__restrict__ q16,
             const T *__restrict__ qv, const int *__restrict__ erp, const int *__restrict__ eci,
             const int *__restrict__ ebase, const uint16_t *__restrict__ e16,
             const T *__restrict__ ev, const BT *__restrict__ b, const T *__restrict__ e,
             OT *__restrict__ out, const double *__restrict__ dw, double *part, unsigned *ticket,
             double *dot_out) {
  pdl_begin();
  constexpr int R = 32 / L;
  const int lane = threadIdx.x & 31, g = lane / L, gl = lane & (L - 1);
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  double dacc = 0.0;
  for (int base = warp * R; base < n; base += nwarps * R) {     // warp-uniform trip count
    const int row = base + g;
    T a = T(0);
    if (row < n) {
      const int qs = __ldg(qrp + row), qe = __ldg(qrp + row + 1);
      const int es = __ldg(erp + row), ee = __ldg(erp + row + 1);
      const int qb = QI16 ? __ldg(qbase + row) : 0, eb = EI16 ? __ldg(ebase + row) : 0;
      a = csr_row_dot<T, T, T, L, EI16>(es + gl, ee, eb, eci, e16, ev, e);
      a += csr_row_dot<T, T, BT, L, QI16>(qs + gl, qe, qb, qci, q16, qv, b);
    }
    a = group_sum<L>(a);
    if (row < n && gl == 0) {
      const OT o = (OT)a;
      out[row] = o;
      if (DOT) dacc += (double)o * dw[row];
    }
  }
  if (DOT) {
    grid_dot(dacc, part, ticket, dot_out);
  }
}

template <typename T, typename BT, typename OT, bool DOT>
void fold_apply(cudaStream_t st, int lanes, const DMat &Q, const DMat &E, const BT *b,
                       const T *e, OT *out, const double *dw, double *part, unsigned *tick,
                       double *dot_out) {
  const int n = Q.nrows;
  const int grid = std::min<int>(ceil_div((int64_t)n * lanes, kApplyThreads), num_sms() * 8);
  auto launch = [&](auto kern) {
    launch_pdl(kern, grid, kApplyThreads, st, n, (const int *)Q.rp.get(), (const int *)Q.ci.get(),
               (const int *)Q.cbase.get(), (const uint16_t *)Q.c16.get(), vals<T>(Q),
               (const int *)E.rp.get(), (const int *)E.ci.get(), (const int *)E.cbase.get(),
               (const uint16_t *)E.c16.get(), vals<T>(E), b, e, out, dw, part, tick, dot_out);
  };
#define CHRONOS_FOLD_CASE(LL)                                                              \
  case LL:                                                                                 \
    if (Q.idx16 && E.idx16) launch(k_fold_apply<T, BT, OT, LL, DOT, true, true>);          \
    else if (E.idx16) launch(k_fold_apply<T, BT, OT, LL, DOT, false, true>);               \
    else if (Q.idx16) launch(k_fold_apply<T, BT, OT, LL, DOT, true, false>);               \
    else launch(k_fold_apply<T, BT, OT, LL, DOT, false, false>);                           \
    break;
  switch (lanes) {
    CHRONOS_FOLD_CASE(1)
    CHRONOS_FOLD_CASE(2)
    CHRONOS_FOLD_CASE(4)
    CHRONOS_FOLD_CASE(8)
    CHRONOS_FOLD_CASE(16)
    CHRONOS_FOLD_CASE(32)
    default: throw Error(CHRONOS_EINVAL, "fold_apply: bad lane count");
  }
#undef CHRONOS_FOLD_CASE
}

}  // namespace chronos
