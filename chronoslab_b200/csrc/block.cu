// Block of K right-hand sides solved together: SpMM V-cycles and K independent
// PCG_CJ recurrences (PCG_CJ.m:34-66 per column) in one CUDA graph.
//
// Vectors are row-major n x K (X[i*K + j]).  In the SpMM kernel K/VEC
// consecutive lanes own one row, each lane VEC columns: every stored value and
// column index is fetched once (a broadcast) and reused K times, and the
// gathers X[c*K + 0..K-1] are K-wide coalesced loads.  Each column keeps its
// own scalars, iteration count and stopping test; a converged column is frozen
// (its x, res and p no longer change), so every column takes the steps of its own
// PCG_CJ, to rounding: a block cycle folds fewer levels, and sums its rows in
// another order, than a single vector's.  The block dot products are K-wide
// deterministic grid reductions.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "hier.h"
#include "spmv.cuh"

namespace chronos {

template <int K> struct StoreK {
  double *dst;
  __device__ bool operator()(int j, const double *t) const {
    dst[j] = t[j];
    return false;
  }
  __device__ void done(bool) const {}
};

// VEC consecutive elements as one 8- or 16-byte access (aligned: K is a
// multiple of VEC and every block starts on a 256-byte boundary).
template <typename T, int VEC> struct Vec;
template <> struct Vec<float, 4> {
  __device__ static void ld(const float *p, float (&o)[4]) {
    const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
    o[0] = t.x; o[1] = t.y; o[2] = t.z; o[3] = t.w;
  }
  __device__ static void st(float *p, const float (&o)[4]) {
    *reinterpret_cast<float4 *>(p) = make_float4(o[0], o[1], o[2], o[3]);
  }
};
template <> struct Vec<float, 2> {
  __device__ static void ld(const float *p, float (&o)[2]) {
    const float2 t = __ldg(reinterpret_cast<const float2 *>(p));
    o[0] = t.x; o[1] = t.y;
  }
  __device__ static void st(float *p, const float (&o)[2]) {
    *reinterpret_cast<float2 *>(p) = make_float2(o[0], o[1]);
  }
};
template <> struct Vec<double, 2> {
  __device__ static void ld(const double *p, double (&o)[2]) {
    const double2 t = __ldg(reinterpret_cast<const double2 *>(p));
    o[0] = t.x; o[1] = t.y;
  }
  __device__ static void st(double *p, const double (&o)[2]) {
    *reinterpret_cast<double2 *>(p) = make_double2(o[0], o[1]);
  }
};

// Lanes own VEC consecutive right-hand-side columns of one row: K/VEC lanes
// per row; each stored value and column index is fetched once per row group
// and applied to K columns.  split (a power of two, K/VEC*split <= 32) lane
// sets share a row's entries, set s taking entries s, s+split, ...: a coarse
// level has too few rows to fill the GPU and its time is one row's chain of
// loads (spmm_split).
template <typename VT, typename XT, typename ZT, typename YT, int K, int VEC, int MODE, bool DOT,
          bool SPLIT>
__global__ void __launch_bounds__(kApplyThreads)
k_csr_spmm(int n, int split_arg, const int *__restrict__ rp, const int *__restrict__ ci,
           const VT *__restrict__ v, const XT *__restrict__ X, const ZT *Z, YT *Y, VT alpha,
           const double *__restrict__ DW, double *part, unsigned *ticket, double *dot_out) {
  pdl_begin();
  constexpr int LPR = K / VEC;
  const int split = SPLIT ? split_arg : 1;
  const int per_row = LPR * split, R = 32 / per_row;
  const int lane = threadIdx.x & 31, g = lane / per_row, j0 = (lane % LPR) * VEC;
  const int part_of = (lane / LPR) & (split - 1);
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  double dacc[VEC];
#pragma unroll
  for (int e = 0; e < VEC; ++e) dacc[e] = 0.0;
  for (int base = warp * R; base < n; base += nwarps * R) {     // warp-uniform trip count
    const int row = base + g;
    VT s[VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) s[e] = VT(0);
    if (row < n) {
      const int e1 = __ldg(rp + row + 1);
      int k = __ldg(rp + row) + part_of;
      for (; k + 3 * split < e1; k += 4 * split) {   // four entries' loads in flight
        int c[4];
        VT a[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          c[u] = __ldg(ci + k + u * split);
          a[u] = __ldg(v + k + u * split);
        }
        XT xv[4][VEC];
#pragma unroll
        for (int u = 0; u < 4; ++u) Vec<XT, VEC>::ld(X + (size_t)c[u] * K + j0, xv[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int e = 0; e < VEC; ++e) s[e] += a[u] * (VT)xv[u][e];
      }
      if (k < e1) {        // the last 1..3 entries: loads clamped to the first, sums selected
        int c[3];
        VT a[3];
#pragma unroll
        for (int u = 0; u < 3; ++u) {
          const int ku = k + u * split < e1 ? k + u * split : k;
          c[u] = __ldg(ci + ku);
          a[u] = __ldg(v + ku);
        }
        XT xv[3][VEC];
#pragma unroll
        for (int u = 0; u < 3; ++u) Vec<XT, VEC>::ld(X + (size_t)c[u] * K + j0, xv[u]);
#pragma unroll
        for (int u = 0; u < 3; ++u)
#pragma unroll
          for (int e = 0; e < VEC; ++e) {
            const VT t = s[e] + a[u] * (VT)xv[u][e];
            s[e] = k + u * split < e1 ? t : s[e];
          }
      }
    }
    for (int o = LPR; o < per_row; o <<= 1)
#pragma unroll
      for (int e = 0; e < VEC; ++e) s[e] += __shfl_xor_sync(0xffffffffu, s[e], o);
    if (row < n && part_of == 0) {
      const size_t o = (size_t)row * K + j0;
      ZT zv[VEC];
      if (MODE == MODE_RESID || MODE == MODE_AXPY) Vec<ZT, VEC>::ld(Z + o, zv);
      YT out[VEC];
#pragma unroll
      for (int e = 0; e < VEC; ++e) {
        VT r;
        if (MODE == MODE_PLAIN) r = s[e];
        else if (MODE == MODE_SCALE) r = alpha * s[e];
        else if (MODE == MODE_RESID) r = (VT)zv[e] - s[e];
        else r = (VT)zv[e] + alpha * s[e];
        out[e] = (YT)r;
        if (DOT) dacc[e] += (double)out[e] * DW[o + e];
      }
      Vec<YT, VEC>::st(Y + o, out);
    }
  }
  if (DOT) {
    double vals[1][VEC];
#pragma unroll
    for (int e = 0; e < VEC; ++e) vals[0][e] = dacc[e];
    grid_reduce_cols<K, VEC, 1>(vals, part, ticket, StoreK<K>{dot_out});
  }
}

// 16-byte accesses when every operand is FP32 (VEC 4), else VEC 2.
template <typename XT, typename ZT, typename YT, int K>
struct SpmmVec {
  static constexpr int v4 = (sizeof(XT) == 4 && sizeof(YT) == 4 && sizeof(ZT) == 4) ? 4 : 2;
  static constexpr int value = v4 > K ? K : v4;
};

// Lane sets sharing a row: doubled while the rows with twice the lanes still
// fit the GPU's resident threads and every set keeps at least four entries
// (one batch of loads in flight).  Diffusion 64^3, 16 columns, residual on the
// levels of 97,128 / 21,463 / 4,851 rows (11-13 entries a row): 6.9 / 6.5 / 5.5 us
// unsplit, 5.9 / 4.6 / 4.1 us; on the finest level (262,144 rows of 7 entries)
// the split form's runtime strides cost more than they give (35 against 22 us).
inline int spmm_split(const DMat &M, int lanes_per_row) {
  const int64_t resident = (int64_t)num_sms() * 2048;
  int s = 1;
  while (2 * s * lanes_per_row <= 32 && (int64_t)M.nrows * lanes_per_row * 2 * s <= resident &&
         M.nnz >= (int64_t)M.nrows * 4 * s)
    s *= 2;
  return s;
}

template <typename VT, typename XT, typename ZT, typename YT, int K, int MODE, bool DOT>
static void spmm(cudaStream_t st, const DMat &M, const VT *vals, const XT *X, const ZT *Z, YT *Y,
                 VT alpha, const double *DW = nullptr, double *part = nullptr,
                 unsigned *tick = nullptr, double *dot_out = nullptr) {
  constexpr int VEC = SpmmVec<XT, ZT, YT, K>::value;
  const int n = M.nrows;
  if (n <= 0) return;
  const int split = spmm_split(M, K / VEC);
  const int rows_per_block = kApplyThreads * VEC / (K * split);
  int blocks = (int)ceil_div(n, rows_per_block);
  blocks = std::min(blocks, num_sms() * 8);
  launch_pdl(split > 1 ? k_csr_spmm<VT, XT, ZT, YT, K, VEC, MODE, DOT, true>
                       : k_csr_spmm<VT, XT, ZT, YT, K, VEC, MODE, DOT, false>,
             blocks, kApplyThreads, st, n, split, M.rp.get(), M.ci.get(), vals, X, Z, Y, alpha, DW,
             part, tick, dot_out);
  CHRONOS_CHECK_LAUNCH();
}

// Y = W B on the coarsest level (W FP64 n x n row-major, B n x K row-major).
template <typename TI, typename TO, int K>
__global__ void k_dense_matmat(int n, const double *__restrict__ W,
                               const TI *__restrict__ B, TO *__restrict__ Y) {
  pdl_begin();
  const int row = blockIdx.x, j = threadIdx.x % K, g = threadIdx.x / K, G = blockDim.x / K;
  __shared__ double red[256];
  double s = 0.0;
  for (int c = g; c < n; c += G) s += W[(size_t)row * n + c] * (double)B[(size_t)c * K + j];
  red[threadIdx.x] = s;
  __syncthreads();
  if (g == 0) {
    double t = 0.0;
    for (int q = 0; q < G; ++q) t += red[q * K + j];
    Y[(size_t)row * K + j] = (TO)t;
  }
}

// ---------------------------------------------------------------------------

struct BlockState {
  int K = 0, n = 0;
  std::vector<DBuf<float>> b32, x32, r32, t32;
  std::vector<DBuf<double>> b64, x64, r64, t64;
  DBuf<double> x, res, p, axp, pres;
  DBuf<double> norms;           // ||b||^2 and ||r0||^2 per column
  DBuf<double> sc;              // per-column scalars, see BS_* below
  DBuf<double> part;
  DBuf<unsigned> tickets;
  LoopGraph loop;
};

// per-column scalar arrays (each K wide) inside sc
enum { BS_BNORM = 0, BS_PTAP, BS_ALPHA, BS_PRES_AXP, BS_RESITER, BS_ITER, BS_ACTIVE, BS_FLAG,
       BS_COUNT };
// after the K-wide arrays: tol, itmax
__host__ __device__ constexpr int bs_off(int which, int K) { return which * K; }

// dst[j] = A(:,j)'B(:,j)
template <int K>
__global__ void __launch_bounds__(256)
k_bdot(int n, const double *__restrict__ A, const double *__restrict__ B, double *part,
       unsigned *ticket, double *dst) {
  pdl_begin();
  double s = 0.0;
  const size_t total = (size_t)n * K;
  for (size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x; o < total;
       o += (size_t)gridDim.x * blockDim.x)
    s += A[o] * B[o];
  double vals[1][1] = {{s}};
  grid_reduce_cols<K, 1, 1>(vals, part, ticket, StoreK<K>{dst});
}

template <typename T, typename BT, typename OT, int K>
static void vcycle_block(Hier &h, BlockState &s, int l, const BT *b, OT *out, const double *dw,
                         double *dot_out);

template <typename T> static T *blk(std::vector<DBuf<float>> &f, std::vector<DBuf<double>> &d, int l);
template <> float *blk<float>(std::vector<DBuf<float>> &f, std::vector<DBuf<double>> &, int l) { return f[l].get(); }
template <> double *blk<double>(std::vector<DBuf<float>> &, std::vector<DBuf<double>> &d, int l) { return d[l].get(); }

template <typename T, typename BT, typename OT, int K>
static void vcycle_block(Hier &h, BlockState &s, int l, const BT *b, OT *out, const double *dw,
                         double *dot_out) {
  Level &L = h.levels[l];
  cudaStream_t st = h.st;
  const int n = L.n;
  double *part = s.part.get();
  unsigned *tick = s.tickets.get();
  if (L.coarsest) {
    launch_pdl(k_dense_matmat<BT, OT, K>, n, 256, st, n, (const double *)L.W.get(), b, out);
    CHRONOS_CHECK_LAUNCH();
    if constexpr (std::is_same_v<OT, double>)
      if (dw)                                   // a single-level hierarchy
        launch_pdl(k_bdot<K>, std::min(num_sms() * 4, (int)ceil_div((int64_t)n * K, 256)), 256,
                   st, n, (const double *)out, dw, part, tick, dot_out);
    return;
  }
  T *x = blk<T>(s.x32, s.x64, l), *r = blk<T>(s.r32, s.r64, l), *t = blk<T>(s.t32, s.t64, l);
  const T w = (T)L.omega;
  if (L.fold && L.fold->form == FOLD_DENSE) {
    launch_pdl(k_dense_matmat<BT, OT, K>, n, 256, st, n,
               (const double *)L.fold->D.get(), b, out);
    CHRONOS_CHECK_LAUNCH();
    return;
  }
  if (L.fold) {
    // the smoother folded, and the restriction (fold.cu) where its longer rows
    // gather at most 16 MB (some 4 us, two launches) more over the K columns; Q
    // and E would gather several times as much.  Diffusion 64^3 x 16 FP32: 366 us
    // per iteration unfolded, 349 with R on every folded level, 342 so; 45^3 x 5
    // FP64: 187, 191 and 172.
    const Fold &F = *L.fold;
    const bool down = F.form != FOLD_SMOOTH &&
                      (double)(F.R.nnz - L.A.nnz - L.Pt.nnz) * K * sizeof(T) <= 16e6;
    T *bc = blk<T>(s.b32, s.b64, l + 1), *xc = blk<T>(s.x32, s.x64, l + 1);
    spmm<T, BT, T, T, K, MODE_PLAIN, false>(st, F.S, vals<T>(F.S), b, (const T *)nullptr, x, T(1));
    if (!down) {
      spmm<T, T, BT, T, K, MODE_RESID, false>(st, L.A, vals<T>(L.A), x, b, r, T(1));
      spmm<T, T, T, T, K, MODE_PLAIN, false>(st, L.Pt, vals<T>(L.Pt), r, (const T *)nullptr, bc,
                                             T(1));
    } else {
      spmm<T, BT, T, T, K, MODE_PLAIN, false>(st, F.R, vals<T>(F.R), b, (const T *)nullptr, bc,
                                              T(1));
    }
    vcycle_block<T, T, T, K>(h, s, l + 1, bc, xc, nullptr, nullptr);
    spmm<T, T, T, T, K, MODE_AXPY, false>(st, L.P, vals<T>(L.P), xc, x, x, T(1));
    spmm<T, T, BT, T, K, MODE_RESID, false>(st, L.A, vals<T>(L.A), x, b, r, T(1));
    if (dw)
      spmm<T, T, T, OT, K, MODE_AXPY, true>(st, F.S, vals<T>(F.S), r, x, out, T(1), dw, part, tick,
                                            dot_out);
    else
      spmm<T, T, T, OT, K, MODE_AXPY, false>(st, F.S, vals<T>(F.S), r, x, out, T(1));
    return;
  }
  spmm<T, BT, T, T, K, MODE_PLAIN, false>(st, L.G, vals<T>(L.G), b, (const T *)nullptr, t, T(1));
  spmm<T, T, T, T, K, MODE_SCALE, false>(st, L.Gt, vals<T>(L.Gt), t, (const T *)nullptr, x, w);
  for (int k = 1; k < h.prm.nupre; ++k) {
    spmm<T, T, BT, T, K, MODE_RESID, false>(st, L.A, vals<T>(L.A), x, b, r, T(1));
    spmm<T, T, T, T, K, MODE_PLAIN, false>(st, L.G, vals<T>(L.G), r, (const T *)nullptr, t, T(1));
    spmm<T, T, T, T, K, MODE_AXPY, false>(st, L.Gt, vals<T>(L.Gt), t, x, x, w);
  }
  spmm<T, T, BT, T, K, MODE_RESID, false>(st, L.A, vals<T>(L.A), x, b, r, T(1));
  T *bc = blk<T>(s.b32, s.b64, l + 1), *xc = blk<T>(s.x32, s.x64, l + 1);
  spmm<T, T, T, T, K, MODE_PLAIN, false>(st, L.Pt, vals<T>(L.Pt), r, (const T *)nullptr, bc, T(1));
  vcycle_block<T, T, T, K>(h, s, l + 1, bc, xc, nullptr, nullptr);
  spmm<T, T, T, T, K, MODE_AXPY, false>(st, L.P, vals<T>(L.P), xc, x, x, T(1));
  const int npost = h.prm.nupost;
  for (int k = 0; k < npost; ++k) {
    spmm<T, T, BT, T, K, MODE_RESID, false>(st, L.A, vals<T>(L.A), x, b, r, T(1));
    spmm<T, T, T, T, K, MODE_PLAIN, false>(st, L.G, vals<T>(L.G), r, (const T *)nullptr, t, T(1));
    if (k + 1 < npost)
      spmm<T, T, T, T, K, MODE_AXPY, false>(st, L.Gt, vals<T>(L.Gt), t, x, x, w);
    else if (dw)
      spmm<T, T, T, OT, K, MODE_AXPY, true>(st, L.Gt, vals<T>(L.Gt), t, x, out, w, dw, part, tick,
                                            dot_out);
    else
      spmm<T, T, T, OT, K, MODE_AXPY, false>(st, L.Gt, vals<T>(L.Gt), t, x, out, w);
  }
  if (npost == 0) {
    if (dw)
      spmm<T, T, T, OT, K, MODE_AXPY, true>(st, L.Gt, vals<T>(L.Gt), t, x, out, T(0), dw, part,
                                            tick, dot_out);
    else
      spmm<T, T, T, OT, K, MODE_AXPY, false>(st, L.Gt, vals<T>(L.Gt), t, x, out, T(0));
  }
}

// ---- block PCG kernels ------------------------------------------------------

template <int K>
__global__ void k_bpcg_p_update(int n, const double *__restrict__ pres, double *__restrict__ p,
                                const double *__restrict__ sc) {
  pdl_begin();
  const double *ptap = sc + bs_off(BS_PTAP, K), *pa = sc + bs_off(BS_PRES_AXP, K);
  const double *it = sc + bs_off(BS_ITER, K), *act = sc + bs_off(BS_ACTIVE, K);
  const size_t total = (size_t)n * K;
  for (size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x; o < total;
       o += (size_t)gridDim.x * blockDim.x) {
    const int j = (int)(o % K);
    if (act[j] == 0.0) continue;
    if (it[j] < 0.5) p[o] = pres[o];
    else p[o] = pres[o] + (-pa[j] / ptap[j]) * p[o];
  }
}

template <int K> struct FinAlphaBlock {
  double *sc;
  __device__ bool operator()(int j, const double *t) const {
    if (sc[bs_off(BS_ACTIVE, K) + j] == 0.0) return false;
    const double ptap = t[j], pr = t[K + j];
    sc[bs_off(BS_PTAP, K) + j] = ptap;
    if (!(ptap > 0.0) || !isfinite(pr)) {
      sc[bs_off(BS_ALPHA, K) + j] = 0.0;
      sc[bs_off(BS_FLAG, K) + j] = 2.0;          // breakdown
    } else {
      sc[bs_off(BS_ALPHA, K) + j] = pr / ptap;
    }
    return false;
  }
  __device__ void done(bool) const {}
};

// axp = A p (FP64, block) with p'axp and p'res per column.  262,144 rows x 16
// columns: 83 us with a one-level reduction finished by one thread, 52 us (its
// vectors and the operator are 122 MB, 19 us; the gathers of p move 235 MB
// from L2).
template <int K>
__global__ void __launch_bounds__(kApplyThreads)
k_bpcg_spmm(int n, const int *__restrict__ rp, const int *__restrict__ ci,
            const double *__restrict__ v, const double *__restrict__ p,
            const double *__restrict__ res, double *__restrict__ axp, double *part,
            unsigned *ticket, double *sc) {
  pdl_begin();
  constexpr int LPR = K / 2;                      // two columns per lane (double2)
  constexpr int R = 32 / LPR;
  const int lane = threadIdx.x & 31, g = lane / LPR, j0 = (lane % LPR) * 2;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  double d0[2] = {0.0, 0.0}, d1[2] = {0.0, 0.0};
  for (int base = warp * R; base < n; base += nwarps * R) {
    const int row = base + g;
    if (row < n) {
      double s[2] = {0.0, 0.0};
      const int e1 = __ldg(rp + row + 1);
      int k = __ldg(rp + row);
      for (; k + 3 < e1; k += 4) {            // four entries' loads in flight
        int c[4];
        double a[4], pv[4][2];
#pragma unroll
        for (int u = 0; u < 4; ++u) { c[u] = __ldg(ci + k + u); a[u] = __ldg(v + k + u); }
#pragma unroll
        for (int u = 0; u < 4; ++u) Vec<double, 2>::ld(p + (size_t)c[u] * K + j0, pv[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          s[0] += a[u] * pv[u][0];
          s[1] += a[u] * pv[u][1];
        }
      }
      if (k < e1) {        // the last 1..3 entries: loads clamped to the first, sums selected
        int c[3];
        double a[3], pv[3][2];
#pragma unroll
        for (int u = 0; u < 3; ++u) {
          const int ku = k + u < e1 ? k + u : k;
          c[u] = __ldg(ci + ku);
          a[u] = __ldg(v + ku);
        }
#pragma unroll
        for (int u = 0; u < 3; ++u) Vec<double, 2>::ld(p + (size_t)c[u] * K + j0, pv[u]);
#pragma unroll
        for (int u = 0; u < 3; ++u)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const double t = s[e] + a[u] * pv[u][e];
            s[e] = k + u < e1 ? t : s[e];
          }
      }
      const size_t o = (size_t)row * K + j0;
      Vec<double, 2>::st(axp + o, s);
      double po[2], ro[2];
      Vec<double, 2>::ld(p + o, po);
      Vec<double, 2>::ld(res + o, ro);
      for (int e = 0; e < 2; ++e) {
        d0[e] += po[e] * s[e];
        d1[e] += po[e] * ro[e];
      }
    }
  }
  double vals[2][2] = {{d0[0], d0[1]}, {d1[0], d1[1]}};
  grid_reduce_cols<K, 2, 2>(vals, part, ticket, FinAlphaBlock<K>{sc});
}

template <int K> struct FinResidualBlock {
  double *sc;
  cudaGraphConditionalHandle handle;
  int use_cond;
  // one column's stop test; true while it goes on
  __device__ bool operator()(int j, const double *t) const {
    if (sc[bs_off(BS_ACTIVE, K) + j] == 0.0) return false;
    const double tol = sc[BS_COUNT * K], itmax = sc[BS_COUNT * K + 1];
    const double it = sc[bs_off(BS_ITER, K) + j] + 1.0;
    const double r = sqrt(t[j]) / sc[bs_off(BS_BNORM, K) + j];
    const bool stop = r < tol || it >= itmax || sc[bs_off(BS_FLAG, K) + j] != 0.0 || !isfinite(r);
    sc[bs_off(BS_ITER, K) + j] = it;
    sc[bs_off(BS_RESITER, K) + j] = r;
    if (stop) sc[bs_off(BS_ACTIVE, K) + j] = 0.0;
    return !stop;
  }
  __device__ void done(bool any) const {
    sc[BS_COUNT * K + 2] = any ? 1.0 : 0.0;
    if (use_cond) cudaGraphSetConditional(handle, any ? 1u : 0u);
  }
};

template <int K>
__global__ void __launch_bounds__(256)
k_bpcg_xr_update(int n, double *__restrict__ x, double *__restrict__ res,
                 const double *__restrict__ p, const double *__restrict__ axp, double *part,
                 unsigned *ticket, double *sc, cudaGraphConditionalHandle handle, int use_cond) {
  pdl_begin();
  // K threads of a group of K walk the K columns of consecutive rows
  const int j = threadIdx.x % K;
  const bool act = sc[bs_off(BS_ACTIVE, K) + j] != 0.0;
  const double alpha = sc[bs_off(BS_ALPHA, K) + j];
  double rr = 0.0;
  const size_t total = (size_t)n * K;
  for (size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x; o < total;
       o += (size_t)gridDim.x * blockDim.x) {
    double ri = res[o];
    if (act) {
      x[o] += alpha * p[o];
      ri -= alpha * axp[o];
      res[o] = ri;
    }
    rr += ri * ri;
  }
  double vals[1][1] = {{rr}};
  grid_reduce_cols<K, 1, 1>(vals, part, ticket, FinResidualBlock<K>{sc, handle, use_cond});
}

// ||B(:,j)||^2 and ||R(:,j)||^2 into sc (BNORM, RESITER hold squares until init)
template <int K>
__global__ void k_bpcg_init(double *sc, const double *b2, const double *r2, double tol,
                            double itmax) {
  pdl_begin();
  const int j = threadIdx.x;                      // one block of K threads
  const double bn = sqrt(b2[j]);
  sc[bs_off(BS_BNORM, K) + j] = bn;
  sc[bs_off(BS_RESITER, K) + j] = bn > 0.0 ? sqrt(r2[j]) / bn : 0.0;
  sc[bs_off(BS_ITER, K) + j] = 0.0;
  sc[bs_off(BS_FLAG, K) + j] = 0.0;
  sc[bs_off(BS_ACTIVE, K) + j] = (bn > 0.0 && itmax > 0.0) ? 1.0 : 0.0;
  if (j == 0) {
    sc[BS_COUNT * K] = tol;
    sc[BS_COUNT * K + 1] = itmax;
  }
}

// Between the callers' layouts (element (i, j) at i*ri + j*cj of the n x m
// staged block) and the solve's row-major n x K block (columns m..K-1 zero
// going in, dropped coming out): tiles of 32 rows through shared memory, so
// both sides are read and written along their contiguous dimension.
template <int K, bool IN>
__global__ void __launch_bounds__(256)
k_block_layout(int n, int m, int64_t ri, int64_t cj, double *__restrict__ staged,
               double *__restrict__ rows) {
  __shared__ double tile[32][K + 1];
  const bool col_major = ri == 1;
  for (int i0 = blockIdx.x * 32; i0 < n; i0 += gridDim.x * 32) {
    for (int q = threadIdx.x; q < 32 * K; q += blockDim.x) {
      const int i = IN && col_major ? q % 32 : q / K, j = IN && col_major ? q / 32 : q % K;
      if (i0 + i < n)
        tile[i][j] = !IN ? rows[(size_t)(i0 + i) * K + j]
                     : j < m ? staged[(i0 + i) * ri + j * cj] : 0.0;
    }
    __syncthreads();
    for (int q = threadIdx.x; q < 32 * K; q += blockDim.x) {
      const int i = !IN && col_major ? q % 32 : q / K, j = !IN && col_major ? q / 32 : q % K;
      if (i0 + i < n) {
        if (IN) rows[(size_t)(i0 + i) * K + j] = tile[i][j];
        else if (j < m) staged[(i0 + i) * ri + j * cj] = tile[i][j];
      }
    }
    __syncthreads();
  }
}

// zero columns with b = 0 (PCG_CJ.m:12-16)
template <int K>
__global__ void k_zero_null_columns(int n, double *x, const double *sc) {
  const size_t total = (size_t)n * K;
  for (size_t o = blockIdx.x * (size_t)blockDim.x + threadIdx.x; o < total;
       o += (size_t)gridDim.x * blockDim.x)
    if (sc[bs_off(BS_BNORM, K) + (int)(o % K)] == 0.0) x[o] = 0.0;
}

template <int K>
static void capture_block_iteration(Hier &h, BlockState &s, cudaGraphConditionalHandle handle,
                                    int use_cond) {
  cudaStream_t st = h.st;
  const int n = s.n;
  double *sc = s.sc.get();
  unsigned *tk = s.tickets.get();
  const int nb = std::max(1, std::min(num_sms() * 8, (int)ceil_div((int64_t)n * K, 256)));
  if (h.precision == CHRONOS_FP32)
    vcycle_block<float, double, double, K>(h, s, 0, s.res.get(), s.pres.get(), s.axp.get(),
                                           sc + bs_off(BS_PRES_AXP, K));
  else
    vcycle_block<double, double, double, K>(h, s, 0, s.res.get(), s.pres.get(), s.axp.get(),
                                            sc + bs_off(BS_PRES_AXP, K));
  launch_pdl(k_bpcg_p_update<K>, nb, 256, st, n, (const double *)s.pres.get(), s.p.get(),
             (const double *)sc);
  CHRONOS_CHECK_LAUNCH();
  const DMat &A = h.levels[0].A;
  const int blocks = std::min(num_sms() * 8, (int)ceil_div(n, kApplyThreads * 2 / K));
  launch_pdl(k_bpcg_spmm<K>, blocks, kApplyThreads, st, n, (const int *)A.rp.get(),
             (const int *)A.ci.get(), (const double *)A.v64.get(), (const double *)s.p.get(),
             (const double *)s.res.get(), s.axp.get(), s.part.get() + 2 * K * 2048,
             tk + kReduceTickets, sc);
  CHRONOS_CHECK_LAUNCH();
  launch_pdl(k_bpcg_xr_update<K>, nb, 256, st, n, s.x.get(), s.res.get(),
             (const double *)s.p.get(), (const double *)s.axp.get(),
             s.part.get() + 4 * K * 2048, tk + 2 * kReduceTickets, sc, handle, use_cond);
  CHRONOS_CHECK_LAUNCH();
}

template <int K>
static void block_solve(Hier &h, int m, const BlockIn &B, const double *X0_h, double *X_h,
                        int itmax, double tol, int *iters, int *flags, double *seconds) {
  cudaStream_t st = h.st;
  auto &sp = h.block;
  if (!sp || sp->K != K) {
    sp.reset();
    auto made = std::make_shared<BlockState>();    // the handle's once it is complete
    BlockState &s = *made;
    s.K = K;
    s.n = h.levels[0].n;
    const bool fp32 = h.precision == CHRONOS_FP32;
    const int nl = (int)h.levels.size();
    s.b32.resize(nl); s.x32.resize(nl); s.r32.resize(nl); s.t32.resize(nl);
    s.b64.resize(nl); s.x64.resize(nl); s.r64.resize(nl); s.t64.resize(nl);
    for (int l = 0; l < nl; ++l) {
      const size_t m = (size_t)std::max(h.levels[l].n, 1) * K;
      if (fp32) { s.b32[l].alloc(m); s.x32[l].alloc(m); s.r32[l].alloc(m); s.t32[l].alloc(m); }
      else { s.b64[l].alloc(m); s.x64[l].alloc(m); s.r64[l].alloc(m); s.t64[l].alloc(m); }
    }
    const size_t m0 = (size_t)s.n * K;
    s.x.alloc(m0); s.res.alloc(m0); s.p.alloc(m0); s.axp.alloc(m0); s.pres.alloc(m0);
    s.norms.alloc(2 * K);
    s.p.zero(st);
    s.axp.zero(st);
    s.sc.alloc((size_t)BS_COUNT * K + 8);
    s.part.alloc((size_t)6 * K * 2048);
    s.tickets.alloc(4 * kReduceTickets);
    s.tickets.zero(st);
    sp = std::move(made);
  }
  BlockState &s = *sp;
  const int n = s.n;
  // (A p is not formed yet when the host blocks come in, nor needed when x goes out;
  // b has served once res is formed, before the first M^-1 res)
  double *staged = s.axp.get(), *b = s.pres.get(), *b2 = s.norms.get(), *r2 = s.norms.get() + K;
  // host blocks -> row-major device blocks; a row-major host block of exactly
  // K columns is already in the solve's layout
  const int lb = std::max(1, std::min(num_sms() * 8, (int)ceil_div(n, 32)));
  auto pack = [&](const BlockIn &src, double *dst) {
    if (src.ld > 0) {                              // row-major, rows ld apart
      double *to = m == K ? dst : staged;
      if (src.ld == m)                             // one copy: row by row is far slower
        CHRONOS_CUDA(cudaMemcpyAsync(to, src.p, sizeof(double) * n * m, cudaMemcpyHostToDevice,
                                     st));
      else
        CHRONOS_CUDA(cudaMemcpy2DAsync(to, sizeof(double) * m, src.p, sizeof(double) * src.ld,
                                       sizeof(double) * m, n, cudaMemcpyHostToDevice, st));
      if (m == K) return;
      k_block_layout<K, true><<<lb, 256, 0, st>>>(n, m, m, 1, staged, dst);
    } else {
      CHRONOS_CUDA(cudaMemcpyAsync(staged, src.p, sizeof(double) * n * m,
                                   cudaMemcpyHostToDevice, st));
      k_block_layout<K, true><<<lb, 256, 0, st>>>(n, m, 1, n, staged, dst);
    }
    CHRONOS_CHECK_LAUNCH();
  };
  pack(B, b);
  if (X0_h) pack(BlockIn{X0_h, 0}, s.x.get());
  else s.x.zero(st);
  cudaEvent_t e0, e1;
  CHRONOS_CUDA(cudaEventCreate(&e0));
  CHRONOS_CUDA(cudaEventCreate(&e1));
  CHRONOS_CUDA(cudaEventRecord(e0, st));
  const DMat &A = h.levels[0].A;
  spmm<double, double, double, double, K, MODE_RESID, false>(st, A, A.v64.get(), s.x.get(), b,
                                                             s.res.get(), 1.0);
  const int nb = std::max(1, std::min(num_sms() * 8, (int)ceil_div((int64_t)n * K, 256)));
  launch_pdl(k_bdot<K>, nb, 256, st, n, (const double *)b, (const double *)b, s.part.get(),
             s.tickets.get() + 3 * kReduceTickets, b2);
  launch_pdl(k_bdot<K>, nb, 256, st, n, (const double *)s.res.get(), (const double *)s.res.get(),
             s.part.get(),
             s.tickets.get() + 3 * kReduceTickets, r2);
  launch_pdl(k_bpcg_init<K>, 1, K, st, s.sc.get(), (const double *)b2, (const double *)r2, tol,
             (double)itmax);
  if (itmax > 0 && !h.prm.use_graph) {
    // one iteration per graph launch from a host loop (profilers cannot see
    // the kernel nodes of a graph holding a conditional node); same kernels
    if (!s.loop.ready())
      s.loop.build(st, false,
                   [&](cudaGraphConditionalHandle) { capture_block_iteration<K>(h, s, 0, 0); });
    double act_h[K];
    for (int k = 0; k < itmax; ++k) {
      CHRONOS_CUDA(cudaMemcpyAsync(act_h, s.sc.get() + bs_off(BS_ACTIVE, K), sizeof(act_h),
                                   cudaMemcpyDeviceToHost, st));
      CHRONOS_CUDA(cudaStreamSynchronize(st));
      bool any = false;
      for (int j = 0; j < K; ++j) any |= act_h[j] != 0.0;
      if (!any) break;
      s.loop.launch(st);
    }
  } else if (itmax > 0) {
    if (!s.loop.ready())
      s.loop.build(st, true, [&](cudaGraphConditionalHandle handle) {
        capture_block_iteration<K>(h, s, handle, 1);
      });
    // the while loop runs its body once before testing: skip it when no
    // column is active (all b = 0)
    double act_h[K];
    CHRONOS_CUDA(cudaMemcpyAsync(act_h, s.sc.get() + bs_off(BS_ACTIVE, K), sizeof(act_h),
                                 cudaMemcpyDeviceToHost, st));
    CHRONOS_CUDA(cudaStreamSynchronize(st));
    bool any = false;
    for (int j = 0; j < K; ++j) any |= act_h[j] != 0.0;
    if (any) s.loop.launch(st);
  }
  k_zero_null_columns<K><<<nb, 256, 0, st>>>(n, s.x.get(), s.sc.get());
  CHRONOS_CHECK_LAUNCH();
  CHRONOS_CUDA(cudaEventRecord(e1, st));
  k_block_layout<K, false><<<lb, 256, 0, st>>>(n, m, 1, n, staged, s.x.get());
  CHRONOS_CHECK_LAUNCH();
  std::vector<double> sc_h((size_t)BS_COUNT * K + 8);
  s.sc.download(sc_h.data(), sc_h.size(), st);
  s.axp.download(X_h, (size_t)n * m, st);
  CHRONOS_CUDA(cudaStreamSynchronize(st));
  float ms = 0.f;
  CHRONOS_CUDA(cudaEventElapsedTime(&ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (seconds) *seconds = ms * 1e-3;
  for (int j = 0; j < m; ++j) {
    iters[j] = (int)(sc_h[bs_off(BS_ITER, K) + j] + 0.5);
    const double r = sc_h[bs_off(BS_RESITER, K) + j];
    flags[j] = (sc_h[bs_off(BS_BNORM, K) + j] == 0.0) ? 0
               : (r > tol || !std::isfinite(r) || sc_h[bs_off(BS_FLAG, K) + j] != 0.0) ? 1 : 0;
  }
}

void Hier::pcg_block(int nrhs, const BlockIn &B, const double *X0_h, double *X_h, int itmax,
                     double tol, int *iters, int *flags, double *seconds) {
  CHRONOS_REQUIRE(nrhs >= 1 && nrhs <= 16, CHRONOS_EINVAL, "block solve: 1 <= nrhs <= 16");
  int K = 2;                     // padded with zero right-hand sides (they stay at x = 0)
  while (K < nrhs) K <<= 1;
  switch (K) {
    case 2: block_solve<2>(*this, nrhs, B, X0_h, X_h, itmax, tol, iters, flags, seconds); break;
    case 4: block_solve<4>(*this, nrhs, B, X0_h, X_h, itmax, tol, iters, flags, seconds); break;
    case 8: block_solve<8>(*this, nrhs, B, X0_h, X_h, itmax, tol, iters, flags, seconds); break;
    default: block_solve<16>(*this, nrhs, B, X0_h, X_h, itmax, tol, iters, flags, seconds); break;
  }
}

}  // namespace chronos
