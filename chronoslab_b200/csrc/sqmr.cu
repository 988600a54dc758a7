// SQMR (LinearSolver/SQMR.m:1-108) with the V-cycle as left preconditioner.
//
// The recurrence and its scalars stay on the device, one iteration as the body
// of a conditional while node, as in PCG_CJ's loop: the operator with q'(A q),
// the residual update with ||r||^2, the V-cycle with r'u, ||u||^2 and the step's
// scalars, and the update of d, x and q.  Six vector kernels and five host
// synchronisations an iteration took 6.6 ms for 37 iterations on elasticity
// 17^3 (16,524 rows, FP64 hierarchy), 5.2 ms of them with the folded V-cycle;
// 1.54 ms with the loop on the device, 1.42 ms with three of its four dots added
// by the kernels that use them (sum_partials) instead of finished where they form.
#include <algorithm>
#include <cmath>

#include "hier.h"
#include "spmv.cuh"

namespace chronos {

namespace {

// Device scalars of the recurrence.
enum SqmrScalar {
  SQ_BB = 0, SQ_RHO0, SQ_RHO1, SQ_VV, SQ_ALPHA, SQ_TAU, SQ_THETA0, SQ_CD, SQ_CQ,
  SQ_BETA, SQ_ITER, SQ_ITMAX, SQ_TOL, SQ_INFO, SQ_EXIT, SQ_TRUE, SQ_COUNT = 20
};

__global__ void __launch_bounds__(256)
k_sq_dot(int n, const double *__restrict__ a, const double *__restrict__ b, double *part,
         unsigned *ticket, double *out) {
  pdl_begin();
  double s = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    s += a[i] * b[i];
  double t[1] = {s};
  grid_reduce<1>(t, part, ticket, StoreScalar{out});
}

// State before the loop: tau = ||q||, theta0 = 0 (SQMR.m:24-36).
__global__ void k_sq_init(double *sc, double itmax, double tol) {
  pdl_begin();
  sc[SQ_TAU] = sqrt(sc[SQ_VV]);
  sc[SQ_RHO0] = sc[SQ_RHO1];
  sc[SQ_THETA0] = 0.0;
  sc[SQ_ITER] = 0.0;
  sc[SQ_ITMAX] = itmax;
  sc[SQ_TOL] = tol;
  sc[SQ_INFO] = 0.0;
  sc[SQ_EXIT] = 0.0;
}

// r -= alpha v with alpha = rho0 / sigma, and the partials of ||r||^2; sigma from
// the operator's partials; a vanishing one (info 10) leaves r as it is.
__global__ void __launch_bounds__(256)
k_sq_residual(int n, const double *__restrict__ v, double *__restrict__ r,
              const double *__restrict__ sigma_part, int slots, double *rr_part, double *sc) {
  pdl_begin();
  const double rho0 = sc[SQ_RHO0];
  double t[1];
  sum_partials<1>(sigma_part, slots, t);
  const double sigma = t[0];
  const bool broke = fabs(sigma) < 1e-20 * rho0;
  const double alpha = rho0 / sigma;
  double s = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double x = broke ? r[i] : -alpha * v[i] + r[i];
    r[i] = x;
    s += x * x;
  }
  t[0] = s;
  block_partials<1>(t, rr_part);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    sc[SQ_ALPHA] = alpha;
    if (broke) sc[SQ_INFO] = 10.0;
  }
}

// ||u||^2 and the step's scalars: theta, gamma, tau, the coefficients of d, the
// stop test and beta (SQMR.m:60-96).
struct FinSqStep {
  double *sc;
  cudaGraphConditionalHandle handle;
  int use_cond;
  double bb, tau, theta0, alpha, rr, rho0, rho1, it, itmax, tol, info0;
  __device__ void load() {
    bb = sc[SQ_BB]; tau = sc[SQ_TAU]; theta0 = sc[SQ_THETA0]; alpha = sc[SQ_ALPHA];
    rho0 = sc[SQ_RHO0]; it = sc[SQ_ITER];
    itmax = sc[SQ_ITMAX]; tol = sc[SQ_TOL]; info0 = sc[SQ_INFO];
  }
  __device__ void operator()(const double *t) const {
    const double now = it + 1.0;
    sc[SQ_ITER] = now;
    if (info0 != 0.0) {                                  // sigma vanished: x stays
      sc[SQ_CD] = 1.0;
      if (use_cond) cudaGraphSetConditional(handle, 0u);
      return;
    }
    const double theta1 = sqrt(t[0]) / tau;
    const double gamma = 1.0 / sqrt(1.0 + theta1 * theta1);
    sc[SQ_TAU] = tau * theta1 * gamma;
    sc[SQ_CD] = gamma * gamma * theta0 * theta0;
    sc[SQ_CQ] = gamma * gamma * alpha;
    sc[SQ_THETA0] = theta1;
    const bool met = sqrt(rr) / sqrt(bb) < tol;
    const bool broke = !met && fabs(rho0) < 1e-20 * rho1;
    const bool go = !met && !broke;
    sc[SQ_EXIT] = met ? 1.0 : 0.0;
    if (broke) sc[SQ_INFO] = 20.0;
    if (go) {
      sc[SQ_BETA] = rho1 / rho0;
      sc[SQ_RHO0] = rho1;
    }
    if (use_cond) cudaGraphSetConditional(handle, go && now < itmax ? 1u : 0u);
  }
};
__global__ void __launch_bounds__(256)
k_sq_step(int n, const double *__restrict__ u, const double *__restrict__ rr_part,
          const double *__restrict__ rho_part, int slots, double *part, unsigned *ticket,
          double *sc, cudaGraphConditionalHandle handle, int use_cond) {
  pdl_begin();
  FinSqStep fin{sc, handle, use_cond};
  fin.load();
  double rr[1], rho1[1];
  sum_partials<1>(rr_part, slots, rr);
  __syncthreads();                             // the sums share their staging
  sum_partials<1>(rho_part, slots, rho1);
  fin.rr = rr[0];
  fin.rho1 = rho1[0];
  double s = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    s += u[i] * u[i];
  double t[1] = {s};
  grid_reduce<1>(t, part, ticket, fin);
}

// d = cd d + cq q, x += d, q = u + beta q.
__global__ void __launch_bounds__(256)
k_sq_update(int n, const double *__restrict__ u, double *__restrict__ d, double *__restrict__ q,
            double *__restrict__ x, const double *__restrict__ sc) {
  pdl_begin();
  if (sc[SQ_INFO] == 10.0) return;
  const double cd = sc[SQ_CD], cq = sc[SQ_CQ], beta = sc[SQ_BETA];
  const bool go = sc[SQ_EXIT] == 0.0 && sc[SQ_INFO] == 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double qi = q[i];
    const double di = cq * qi + cd * d[i];
    d[i] = di;
    x[i] += di;
    if (go) q[i] = u[i] + beta * qi;
  }
}

// y = A x or z - A x (FP64), with the dot y'w when w is given.
template <int MODE, bool DOT>
void operator_apply(cudaStream_t st, const DMat &A, const double *x, const double *z, double *y,
                    const double *w, double *part, unsigned *tick, double *out) {
  if (A.nb > 0)
    sell3_apply<double, double, double, double, MODE, DOT>(st, A.sell_T, A.nb, A.nchunk, A.choff,
                                                           A.chw, A.sci, A.bv64.get(), A.nslots, x,
                                                           z, y, 1.0, w, part, tick, out);
  else
    mat_apply<double, double, double, double, MODE, DOT>(st, A, A.v64.get(), x, z, y, 1.0, w, part,
                                                         tick, out);
}

}  // namespace

// Vectors, scalars and the loop's graph.  For the handle's own operator they are
// parked between calls (IdleStates), up to kSqmrParkBytes: making the graph anew takes
// 0.33 ms, a quarter of a call at 17^3 (1.26 and 1.60 ms), 7 % of one at 32^3
// (104,544 rows: 4.18 and 4.48 ms).
constexpr size_t kSqmrParkBytes = (size_t)32 << 20;
struct SqmrState {
  int n = 0;
  DBuf<double> vec, sc, part;
  DBuf<unsigned> tickets;
  double *b = nullptr, *x = nullptr, *r = nullptr, *q = nullptr, *d = nullptr, *v = nullptr;
  LoopGraph loop;
  explicit SqmrState(int rows) : n(rows), vec(6 * (size_t)rows), sc(SQ_COUNT), part(5 * 2048),
                                 tickets(4) {
    b = vec.get();
    x = b + n; r = x + n; q = r + n; d = q + n; v = d + n;
  }
};

static void capture_sqmr(Hier &h, SqmrState &s, const DMat &A, cudaGraphConditionalHandle handle,
                         int use_cond) {
  cudaStream_t st = h.st;
  const int n = s.n, nb = std::max(1, std::min(num_sms() * 8, (int)ceil_div(n, 256)));
  double *sc = s.sc.get(), *part = s.part.get();
  unsigned *tk = s.tickets.get();
  // (three of the four dots stay partials, added by the kernels that use them)
  double *sigma_part = part + 3 * 2048, *rr_part = part + 4 * 2048;
  const int slots = num_sms() * 8;               // no producer's grid is larger
  operator_apply<MODE_PLAIN, true>(st, A, s.q, nullptr, s.v, s.q, sigma_part, tk, nullptr);
  launch_pdl(k_sq_residual, nb, 256, st, n, (const double *)s.v, s.r, (const double *)sigma_part,
             slots, rr_part, sc);
  h.vcycle(s.r, s.v, s.r, nullptr);
  launch_pdl(k_sq_step, nb, 256, st, n, (const double *)s.v, (const double *)rr_part,
             vcycle_dot_partials(h), slots, part, tk, sc, handle, use_cond);
  launch_pdl(k_sq_update, nb, 256, st, n, (const double *)s.v, s.d, s.q, s.x,
             (const double *)sc);
}

void sqmr_solve(Hier &h, const DMat *op, const double *b_h, double *x_h, int itmax, double tol,
                int *iters, double *relres, int *info) {
  cudaStream_t st = h.st;
  const int n = h.levels[0].n;
  ensure_reduction_state(h);                    // the V-cycle's dot
  const DMat &A = op ? *op : h.levels[0].A;
  auto state = op ? nullptr : std::static_pointer_cast<SqmrState>(idle_states().take(&h));
  if (!state) state = std::make_shared<SqmrState>(n);
  SqmrState &s = *state;
  const int nb = std::max(1, std::min(num_sms() * 8, (int)ceil_div(n, 256)));
  double *sc = s.sc.get(), *part = s.part.get();
  unsigned *tk = s.tickets.get();
  s.tickets.zero(st);
  // partials past the producers' grids are zero
  s.part.zero(st);
  zero_vcycle_partials(h);
  CHRONOS_CUDA(cudaMemcpyAsync(s.b, b_h, sizeof(double) * n, cudaMemcpyHostToDevice, st));
  CHRONOS_CUDA(cudaMemcpyAsync(s.x, x_h, sizeof(double) * n, cudaMemcpyHostToDevice, st));
  CHRONOS_CUDA(cudaMemsetAsync(s.d, 0, sizeof(double) * n, st));
  // SQMR.m:24-36
  launch_pdl(k_sq_dot, nb, 256, st, n, (const double *)s.b, (const double *)s.b, part, tk,
             sc + SQ_BB);
  operator_apply<MODE_RESID, false>(st, A, s.x, s.b, s.r, nullptr, nullptr, nullptr, nullptr);
  h.vcycle(s.r, s.q, s.r, sc + SQ_RHO1);
  launch_pdl(k_sq_dot, nb, 256, st, n, (const double *)s.q, (const double *)s.q, part, tk,
             sc + SQ_VV);
  launch_pdl(k_sq_init, 1, 1, st, sc, (double)itmax, tol);
  double got[SQ_COUNT] = {};
  if (itmax > 0) {
    if (!s.loop.ready())
      s.loop.build(st, h.prm.use_graph, [&](cudaGraphConditionalHandle handle) {
        capture_sqmr(h, s, A, handle, h.prm.use_graph ? 1 : 0);
      });
    if (h.prm.use_graph) {
      s.loop.launch(st);
    } else {
      for (int k = 0; k < itmax; ++k) {
        s.loop.launch(st);
        CHRONOS_CUDA(cudaMemcpyAsync(got, sc, sizeof(got), cudaMemcpyDeviceToHost, st));
        CHRONOS_CUDA(cudaStreamSynchronize(st));
        if (got[SQ_EXIT] != 0.0 || got[SQ_INFO] != 0.0) break;
      }
    }
  }
  // the true residual
  operator_apply<MODE_RESID, false>(st, A, s.x, s.b, s.v, nullptr, nullptr, nullptr, nullptr);
  launch_pdl(k_sq_dot, nb, 256, st, n, (const double *)s.v, (const double *)s.v, part, tk,
             sc + SQ_TRUE);
  CHRONOS_CUDA(cudaMemcpyAsync(got, sc, sizeof(got), cudaMemcpyDeviceToHost, st));
  CHRONOS_CUDA(cudaMemcpyAsync(x_h, s.x, sizeof(double) * n, cudaMemcpyDeviceToHost, st));
  CHRONOS_CUDA(cudaStreamSynchronize(st));
  *iters = (int)(got[SQ_ITER] + 0.5);
  *info = *iters >= itmax ? 1 : (int)(got[SQ_INFO] + 0.5);
  *relres = std::sqrt(got[SQ_TRUE]) / std::sqrt(got[SQ_BB]);
  if (!op && sizeof(double) * s.vec.size() <= kSqmrParkBytes)
    idle_states().park(&h, std::move(state));
}

}  // namespace chronos
