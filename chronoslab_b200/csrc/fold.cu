// Folded levels of the V-cycle (hier.h, struct Fold).  A level's V(1,1) part is
// linear in its right-hand side b and the coarse correction e:
//   x1 = S b,              S = omega G'G
//   b_c = P'(b - A x1)     = R b,        R = P'(I - A S)
//   x2 = x1 + P e
//   out = x2 + S (b - A x2) = Q b + E e,  Q = S (2I - A S),  E = (I - S A) P
// Applied operator by operator that is eight kernels (G, G', A, P' on the way
// down, P, A, G, G' on the way up), and on all but the largest levels each of
// them is mostly a launch and one row's chain of dependent loads.  The products
// are formed once, in FP64, by the setup's sparse product kernels, as far as
// they pay (the limits stand with the measurements below):
//   FOLD_SMOOTH  S                six kernels
//   FOLD_DOWN    S and R          four: R b; S b + P e; the residual; x2 + S r
//   FOLD_ALL     R, Q, E          two: R b; Q b + E e
//   FOLD_DENSE   D = Q + E B R, B the level below's dense operator (the coarsest
//                level's inverse, or its D): one matrix-vector product is the
//                whole tail of the cycle
#include <algorithm>

#include "hier.h"
#include "spmv.cuh"

namespace chronos {

namespace {

// v *= w
__global__ void k_scale_values(int64_t n, double w, double *__restrict__ v) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
       k += (int64_t)gridDim.x * blockDim.x)
    v[k] *= w;
}

// M = add I + sign M (a warp per row); *missing set where a row stores no
// diagonal entry.
__global__ void __launch_bounds__(256)
k_add_identity(int n, const int *__restrict__ rp, const int *__restrict__ ci,
               double *__restrict__ v, double sign, double add, int *missing) {
  const int lane = threadIdx.x & 31;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += nw) {
    bool diag = false;
    for (int k = rp[i] + lane; k < rp[i + 1]; k += 32) {
      const bool d = ci[k] == i;
      diag |= d;
      v[k] = d ? add + sign * v[k] : sign * v[k];
    }
    if (!__any_sync(0xffffffffu, diag) && lane == 0) *missing = 1;
  }
}

// Y = E B: row r of Y (m wide) from E's row and the dense rows of B.
__global__ void __launch_bounds__(256)
k_sparse_dense(int m, const int *__restrict__ rp, const int *__restrict__ ci,
               const double *__restrict__ v, const double *__restrict__ B,
               double *__restrict__ Y) {
  const int r = blockIdx.x, s = rp[r], e = rp[r + 1];
  for (int j = threadIdx.x; j < m; j += blockDim.x) {
    double t = 0.0;
    for (int k = s; k < e; ++k) t = fma(v[k], B[(size_t)ci[k] * m + j], t);
    Y[(size_t)r * m + j] = t;
  }
}

// D = Y R + Q, row r: Y's row in shared memory against the columns of R (the
// rows of R'), then Q's entries on top.
__global__ void __launch_bounds__(256)
k_dense_tail(int n, int m, const double *__restrict__ Y, const int *__restrict__ trp,
             const int *__restrict__ tci, const double *__restrict__ tv,
             const int *__restrict__ qrp, const int *__restrict__ qci,
             const double *__restrict__ qv, double *__restrict__ D) {
  extern __shared__ double y[];
  const int r = blockIdx.x;
  for (int c = threadIdx.x; c < m; c += blockDim.x) y[c] = Y[(size_t)r * m + c];
  __syncthreads();
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    double t = 0.0;
    for (int k = trp[j]; k < trp[j + 1]; ++k) t = fma(y[tci[k]], tv[k], t);
    D[(size_t)r * n + j] = t;
  }
  __syncthreads();
  for (int k = qrp[r] + threadIdx.x; k < qrp[r + 1]; k += blockDim.x)
    D[(size_t)r * n + qci[k]] += qv[k];
}

// A sparse product on the device.
struct Prod {
  int rows = 0, cols = 0;
  int64_t nnz = 0;
  DBuf<int> rp, ci;
  DBuf<double> v;
};

// p = x y; false, and p empty, where that is more work than a fold is worth.
template <typename X, typename Y>
bool multiply(int m, int ncols, const X &x, const Y &y, Prod &p, cudaStream_t st,
              int64_t max_products) {
  p = Prod();
  p.rows = m;
  p.cols = ncols;
  return spgemm_device(m, ncols, x.rp, x.ci, x.v, y.rp, y.ci, y.v, p.rp, p.ci, p.v, &p.nnz, st,
                       max_products);
}

struct View {
  const int *rp, *ci;
  const double *v;
  explicit View(const DMat &d) : rp(d.rp.get()), ci(d.ci.get()), v(d.v64.get()) {}
};

bool add_identity(Prod &p, double sign, double add, cudaStream_t st) {
  DBuf<int> missing(1);
  missing.zero(st);
  k_add_identity<<<std::max(1, std::min<int>(ceil_div(p.rows, 8), num_sms() * 16)), 256, 0, st>>>(
      p.rows, p.rp.get(), p.ci.get(), p.v.get(), sign, add, missing.get());
  CHRONOS_CHECK_LAUNCH();
  int h = 0;
  CHRONOS_CUDA(cudaMemcpyAsync(&h, missing.get(), sizeof(int), cudaMemcpyDeviceToHost, st));
  CHRONOS_CUDA(cudaStreamSynchronize(st));
  return h == 0;
}

// R replaces three kernels by one and Q, E three by one; each may read up to
// this many entries (about 4 us of gathers) for that.  us per PCG iteration of
// no folding / SMOOTH / DOWN / ALL on level 1: poisson 20^3 FP64 (R 0.12M, Q + E
// 0.65M entries) 53 / 49 / 43 / 35; poisson 48^3 FP32 (1.8M, 9.5M) 81 / 73 / 66 /
// 101; poisson 64^3 FP32 (4.2M, 23M) 109 / 98 / 105 / 185.
constexpr int64_t kFoldEntries = 2 << 20;
// Products of two entries that any of the folds' sparse products may take: twice what
// the largest kept one does (diffusion 64^3, level 2, S U: 15M; A S 9M at most), some
// 6 ms.
constexpr int64_t kFoldProducts = 16 * kFoldEntries;
// Longest row of a factor of the products: a row that long is a chain of its entries
// in one warp.  39,305 rows of which one couples to all others (a constraint) spent
// 148 ms on the products and 98 on the rest of the setup, for 0.23 of 0.58 ms an
// iteration; where the smoother's row is as long, A S fills as well.
// Also the longest row of the two-matrix apply (32 lanes: 16 batches of four entries),
// which has no other path for long rows, as the one-matrix applies do.
constexpr int kFoldLongest = 2048;
// A dense tail has at most kFoldDenseRows rows (FP64: 34 MB a product), where
// the level's operator is dense enough (n^2 <= kFoldDenseRatio entries of A)
// for the folded rows to be nearly full anyway.  Elasticity 17^3, FP64, 1629
// rows of 200 entries: 48 us per iteration with the tail, 58 without; poisson
// 64^3, 1544 rows of 15: 94 and 91.
constexpr int kFoldDenseRows = 2048;
constexpr int64_t kFoldDenseRatio = 32;

// Upper bound of the entries of G'G.
int64_t smoother_bound(const DMat &G) {
  int64_t t = 0;
  for (int i = 0; i < G.nrows; ++i) {
    const int64_t k = G.rp_h[i + 1] - G.rp_h[i];
    t += k * k;
  }
  return t;
}

// Lanes per row of a two-matrix apply: one batch of four entries a lane covers
// an average row, and as many more lanes, up to one an entry, as the GPU has
// threads idle (the longest rows' batches are then shorter chains); a longest row far
// above the average takes eight batches a lane at most.
int fold_lanes(int64_t entries, int rows, int longest) {
  const double avg = (double)entries / std::max(rows, 1);
  const int64_t resident = (int64_t)num_sms() * 2048;
  int L = 1;
  while (L < 32 && (4 * L < avg || (L < avg && (int64_t)rows * 2 * L <= resident / 4) ||
                    longest > 32 * L))
    L *= 2;
  return L;
}

int longest_row(const DMat &M) {
  int t = 0;
  for (int i = 0; i < M.nrows; ++i) t = std::max(t, M.rp_h[i + 1] - M.rp_h[i]);
  return t;
}

void adopt(Prod &p, DMat &d, bool fp32, cudaStream_t st) {
  adopt_csr(p.rows, p.cols, p.nnz, p.rp, p.ci, p.v, d, fp32, st);
}

}  // namespace

std::unique_ptr<Fold> fold_operators(const DMat &A, const DMat &G, const DMat &Gt, const DMat &P,
                                     const DMat &Pt, double omega, const double *B, bool fp32,
                                     cudaStream_t st) {
  const int n = A.nrows, nc = P.ncols;
  auto f = std::make_unique<Fold>();
  const bool dense = B && n <= kFoldDenseRows && (int64_t)n * n <= kFoldDenseRatio * A.nnz;
  // S replaces G and G' in both smoothing steps and spares a vector between
  // them; a factor with long rows fills up when it is squared
  const int64_t worth = 2 * G.nnz + 2 * (int64_t)n + kFoldEntries / 2;
  // (a bound of 2^31 could also be a product that the row pointers cannot hold)
  const int64_t most = std::min<int64_t>(4 * worth, INT32_MAX - 1);
  if ((!dense && smoother_bound(G) > most) || longest_row(Gt) > kFoldLongest) return nullptr;
  Prod S, U, R, Q, E, X;
  if (!multiply(n, n, View(Gt), View(G), S, st, most)) return nullptr;
  if (!dense && S.nnz > worth) return nullptr;
  k_scale_values<<<std::max<int>(1, std::min<int64_t>(ceil_div(S.nnz, 256), num_sms() * 8)), 256,
                   0, st>>>(S.nnz, omega, S.v.get());
  CHRONOS_CHECK_LAUNCH();
  auto smooth_only = [&]() -> std::unique_ptr<Fold> {
    if (S.nnz > worth) return nullptr;
    adopt(S, f->S, fp32, st);
    f->form = FOLD_SMOOTH;
    return std::move(f);
  };
  // R has at least about as many entries as A, Q and E four times R's
  // (twice and more where its rows are short): no product that would be dropped
  if (!dense && (A.nnz < (int64_t)16 * n ? 2 : 1) * A.nnz > kFoldEntries) return smooth_only();
  if (std::max(longest_row(A), longest_row(Pt)) > kFoldLongest) return smooth_only();
  if (!multiply(n, n, View(A), S, U, st, kFoldProducts) || !add_identity(U, -1.0, 1.0, st) ||
      !multiply(nc, n, View(Pt), U, R, st, kFoldProducts) ||        // U = I - A S
      (!dense && R.nnz > kFoldEntries))
    return smooth_only();
  const bool all =
      (dense || (3 * A.nnz <= kFoldEntries && 4 * R.nnz <= kFoldEntries)) &&
      add_identity(U, 1.0, 1.0, st) &&                              // I + U
      multiply(n, n, S, U, Q, st, kFoldProducts) && (dense || Q.nnz <= kFoldEntries) &&
      multiply(n, n, S, View(A), X, st, kFoldProducts) &&
      add_identity(X, -1.0, 1.0, st) &&                             // I - S A
      multiply(n, nc, X, View(P), E, st, kFoldProducts) &&
      (dense || Q.nnz + E.nnz <= kFoldEntries);
  U = Prod();
  X = Prod();
  if (all && !dense) {
    adopt(Q, f->Q, fp32, st);
    adopt(E, f->E, fp32, st);
    const int longest = std::max(longest_row(f->Q), longest_row(f->E));
    if (longest <= kFoldLongest) {
      adopt(S, f->S, fp32, st);
      adopt(R, f->R, fp32, st);
      f->lanes = fold_lanes(f->Q.nnz, n, longest);
      f->R.wide = wide_rows(f->R, kWideTake);
      f->form = FOLD_ALL;
      return f;
    }
    f->Q = DMat();
    f->E = DMat();
  }
  if (!all || !dense) {
    if (S.nnz > worth || R.nnz > kFoldEntries) return smooth_only();
    adopt(S, f->S, fp32, st);
    const int longest = std::max(longest_row(f->S), longest_row(P));
    f->form = FOLD_SMOOTH;
    if (longest <= kFoldLongest) {
      adopt(R, f->R, fp32, st);
      f->lanes = fold_lanes(f->S.nnz + P.nnz, n, longest);
      f->form = FOLD_DOWN;
    }
    return f;
  }
  f->D.alloc((size_t)n * n);
  DBuf<double> Y((size_t)n * nc), tv;
  DBuf<int> trp, tci;
  csr_transpose_device(nc, n, R.nnz, R.rp, R.ci, R.v, trp, tci, tv, st);
  k_sparse_dense<<<n, 256, 0, st>>>(nc, E.rp.get(), E.ci.get(), E.v.get(), B,
                                    Y.get());
  CHRONOS_CHECK_LAUNCH();
  k_dense_tail<<<n, 256, sizeof(double) * nc, st>>>(n, nc, Y.get(), trp.get(), tci.get(),
                                                    tv.get(), Q.rp.get(), Q.ci.get(),
                                                    Q.v.get(), f->D.get());
  CHRONOS_CHECK_LAUNCH();
  CHRONOS_CUDA(cudaStreamSynchronize(st));
  f->form = FOLD_DENSE;
  return f;
}

void tune_fold(Fold &F, bool fp32, cudaStream_t st) {
  if (F.form == FOLD_SMOOTH || F.form == FOLD_DOWN) autotune_lanes(F.S, fp32, st);
  if (F.form == FOLD_DOWN) autotune_lanes(F.R, fp32, st);
}

void build_folds(Hier &h) {
  for (auto &L : h.levels) L.fold.reset();
  // the algebra above is one pre- and one postsmoothing step; a caller who
  // chose the storage of the operators (spmv_format) gets them applied so
  if (h.prm.nupre > 1 || h.prm.nupost != 1 || h.prm.spmv_format != 0) return;
  for (int l = (int)h.levels.size() - 2; l >= 0; --l) {
    Level &L = h.levels[l];
    const Level &C = h.levels[l + 1];
    // level 1 keeps its fused dot and conversions: no dense form
    const double *B = nullptr;
    if (l > 0 && C.coarsest) B = C.W.get();
    else if (l > 0 && C.fold && C.fold->form == FOLD_DENSE) B = C.fold->D.get();
    L.fold = fold_operators(L.A, L.G, L.Gt, L.P, L.Pt, L.omega, B, h.precision == CHRONOS_FP32,
                            h.st);
  }
}

}  // namespace chronos
