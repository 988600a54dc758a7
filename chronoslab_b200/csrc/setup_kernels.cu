// Setup-phase kernels of the solve path (sm_100a):
//  * FSAI numeric phase: a group of lanes per row gathers the local SPD system
//    A[P,P], -A[P,i] of its pattern, factors it in FP64 (LDL' in registers up
//    to 32 unknowns, Cholesky in shared memory up to 64), solves, and scales
//    the row by 1/sqrt(a_ii - A_iP A_PP^-1 A_Pi) (cpt_afsai_coef.cpp:440-541).
//    Rows are bucketed by local size so each bucket runs with the lane group
//    or shared-memory tile that fits it.
//  * Galerkin product P'*(A*P) (cpt_aspAMG.m:277) as two row-wise sparse
//    products with per-row hash tables: symbolic count, then numeric
//    accumulation in Gustavson order (each output entry summed in the order
//    of the left factor's row, products and sums rounded separately), exact
//    zeros dropped, rows sorted.
//  * Coarsest level: dense FP64 Cholesky, inverse from the factor, dense
//    matvec apply (AMG_Vcycle.m:9-10).
#include <cub/cub.cuh>
#include <thrust/iterator/transform_iterator.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <numeric>
#include <string>

#include "internal.h"

namespace chronos {

// =============================================================================
// FSAI numeric
// =============================================================================

// Position of column c in the sorted row [k, ke) of aci, or -1.
__device__ __forceinline__ int find_col(const int *aci, int k, int ke, int c) {
  int lo = k, hi = ke - 1;
  while (lo <= hi) {
    int mid = (lo + hi) >> 1;
    int v = aci[mid];
    if (v == c) return mid;
    if (v < c) lo = mid + 1; else hi = mid - 1;
  }
  return -1;
}

// Row i of G by one warp (cpt_afsai_coef.cpp:440-541): gathers A[P,P] and
// -A[P,i] into the warp's shared-memory tile M (MMAX x MMAX, row-major lower,
// then rhs and y), factors and solves, and writes the scaled row.  Sets bit 0
// of *flags for a non-SPD local block or a non-positive Schur complement.
template <int MMAX>
__device__ __forceinline__ void fsai_row(int i, const int *__restrict__ arp,
                                         const int *__restrict__ aci, const double *__restrict__ av,
                                         const int *__restrict__ grp, const int *__restrict__ gci,
                                         double *__restrict__ gval, int *flags, double *M,
                                         int lane) {
  double *rhs = M + MMAX * MMAX;                // -A[i,P] (kept for the Schur term)
  double *y = rhs + MMAX;                       // solution
  const int gs = grp[i], ge = grp[i + 1];
  const int m = ge - gs - 1;                    // strictly-lower entries
  const int *P = gci + gs;
  const int ai = arp[i], aie = arp[i + 1];
  // Gather: column c (owned by lane c mod 32) from row P[c], entries P[j], j >= c.
  for (int c = lane; c < m; c += 32) {
    const int r = P[c];
    int k = arp[r];
    const int ke = arp[r + 1];
    // first entry with column >= r (binary search)
    int lo = k, hi = ke;
    while (lo < hi) { int mid = (lo + hi) >> 1; if (aci[mid] < r) lo = mid + 1; else hi = mid; }
    k = lo;
    for (int j = c; j < m; ++j) {
      const int pj = P[j];
      while (k < ke && aci[k] < pj) ++k;
      M[j * MMAX + c] = (k < ke && aci[k] == pj) ? av[k] : 0.0;
    }
    const int pos = find_col(aci, ai, aie, r);
    rhs[c] = pos >= 0 ? -av[pos] : 0.0;
  }
  double aii = 0.0;
  bool have_diag = false;
  {
    const int pos = find_col(aci, ai, aie, i);
    if (pos >= 0) { aii = av[pos]; have_diag = true; }
  }
  __syncwarp();
  bool spd = true;
  // Right-looking Cholesky; lane j owns rows j, j+32.
  for (int k = 0; k < m; ++k) {
    double d = M[k * MMAX + k];
    if (!(d > 0.0)) { spd = false; break; }     // warp-uniform (all lanes read the same d)
    d = sqrt(d);
    __syncwarp();
    for (int j = k + 1 + lane; j < m; j += 32) M[j * MMAX + k] /= d;
    if (lane == 0) M[k * MMAX + k] = d;
    __syncwarp();
    for (int j = k + 1 + lane; j < m; j += 32) {
      const double ljk = M[j * MMAX + k];
      for (int l = k + 1; l <= j; ++l) M[j * MMAX + l] -= ljk * M[l * MMAX + k];
    }
    __syncwarp();
  }
  double scal = 0.0;
  if (spd) {
    for (int j = lane; j < m; j += 32) y[j] = rhs[j];
    __syncwarp();
    for (int k = 0; k < m; ++k) {               // L z = rhs
      const double zk = y[k] / M[k * MMAX + k];
      __syncwarp();
      if (lane == 0) y[k] = zk;
      for (int j = k + 1 + lane; j < m; j += 32) y[j] -= M[j * MMAX + k] * zk;
      __syncwarp();
    }
    for (int k = m - 1; k >= 0; --k) {          // L^T y = z
      const double yk = y[k] / M[k * MMAX + k];
      __syncwarp();
      if (lane == 0) y[k] = yk;
      for (int j = lane; j < k; j += 32) y[j] -= M[k * MMAX + j] * yk;
      __syncwarp();
    }
    double part = 0.0;
    for (int j = lane; j < m; j += 32) part += rhs[j] * y[j];
    part = warp_sum(part);
    scal = aii - part;
  }
  bool ok = spd && have_diag && scal > 0.0;
  if (!ok) {
    if (lane == 0) atomicOr(flags, 1);
    scal = 1.0;
    if (!spd)                                    // keep a defined row: diagonal scaling only
      for (int j = lane; j < m; j += 32) y[j] = 0.0;
    __syncwarp();
  }
  const double s = 1.0 / sqrt(scal);
  for (int j = lane; j < m; j += 32) gval[gs + j] = s * y[j];
  if (lane == 0) gval[gs + m] = s;
}

// Positions of the columns col[u] in the sorted rows [lo[u], hi[u]) of aci, or
// -1: U binary searches step together, so their dependent loads overlap.  A
// step's interval shrinks by the same amount whichever side is taken: one
// compare and one add a search.
template <int U>
__device__ __forceinline__ void find_cols(const int *__restrict__ aci, int (&lo)[U],
                                          const int (&hi)[U], const int (&col)[U]) {
  int n[U], longest = 0;
#pragma unroll
  for (int u = 0; u < U; ++u) {
    n[u] = hi[u] - lo[u];
    longest = max(longest, n[u]);
  }
  for (; longest > 1; longest -= longest >> 1) {
    int c[U];
#pragma unroll
    for (int u = 0; u < U; ++u) c[u] = n[u] > 1 ? __ldg(aci + lo[u] + (n[u] >> 1) - 1) : 0x7fffffff;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (c[u] < col[u]) lo[u] += n[u] >> 1;
      n[u] -= n[u] >> 1;
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u)
    if (n[u] <= 0 || __ldg(aci + lo[u]) != col[u]) lo[u] = -1;
}

// Row i of G by T lanes (32/T rows per warp; i < 0: an idle group), local
// systems of up to MMAX <= T unknowns.  Lane j holds row j of the lower
// triangle in registers, R[0..j], and takes LDL' steps: at step k the pivot is
// broadcast, every lane scales its own entry by the pivot's reciprocal and
// leaves it in the group's shared-memory tile, column by column, from where
// the update reads the whole column two entries at a time (one 16-byte
// broadcast) and the backward substitution its row of L'.  The forward
// substitution rides along.  Registers past the diagonal collect products
// that nothing reads.  Unknowns beyond m are identity rows, so a row's
// operations do not depend on the T it runs with.
// One reciprocal per step and no division or square root: with a warp per
// row, the factor in shared memory and a lane per column walking A's rows
// this took 1419 us for 227k rows of mostly 15 unknowns (61^3 diffusion),
// bound by those and by the serial walk; with the column sent round by
// shuffles 351 us, with the column from shared memory 297 us, with the shorter
// search and blocks of four warps for eight 266 us, still bound by issue (71 %
// of the slots).  Two unknowns a lane, which halves a row's shuffles, reciprocals
// and column reads, took as long: its 96 registers leave 20 warps an SM for 32.
// The entries A[P,P] are found by T lanes taking the pairs (c, c+s mod m) of
// each distance s, four searches in flight.
template <int T, int MMAX>
__device__ __forceinline__ void fsai_row_reg(int i, const int *__restrict__ arp,
                                             const int *__restrict__ aci,
                                             const double *__restrict__ av,
                                             const int *__restrict__ grp,
                                             const int *__restrict__ gci,
                                             double *__restrict__ gval, int *flags, double *S) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int LD = MMAX + 2;                  // columns start on 16 bytes
  const int j = threadIdx.x & (T - 1);          // lane of the group
  int gs = 0, m = 0, ib = 0, ie = 0;
  if (i >= 0) {
    gs = __ldg(grp + i);
    m = __ldg(grp + i + 1) - gs - 1;            // strictly-lower entries
    ib = __ldg(arp + i);
    ie = __ldg(arp + i + 1);
  }
  const int mw = __reduce_max_sync(FULL, m);    // of the warp's rows
  const bool live = j < m;
  int pj = 0, rb = 0, re = 0;
  if (live) {
    pj = __ldg(gci + gs + j);
    rb = __ldg(arp + pj);
    re = __ldg(arp + pj + 1);
  }
  // -A[i, P[j]] and a_ii
  double y = 0.0, aii = 0.0;
  bool have_diag = false;
  {
    int lo[2] = {ib, ib};
    const int hi[2] = {live ? ie : ib, ie}, col[2] = {pj, i};
    find_cols<2>(aci, lo, hi, col);
    if (lo[0] >= 0) y = -__ldg(av + lo[0]);
    if (lo[1] >= 0) {
      aii = __ldg(av + lo[1]);
      have_diag = true;
    }
  }
  const double rhs = y;
  // A[P[a], P[b]], a <= b, into S[b][a]
  for (int s0 = 0; 2 * s0 <= mw; s0 += 4) {
    int lo[4], hi[4], col[4], at[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int s = s0 + u;
      const bool on = live && 2 * s <= m;
      int b = j + s;
      if (b >= m) b -= m;
      if (!on) b = j;
      const int pb = __shfl_sync(FULL, pj, b, T), rbb = __shfl_sync(FULL, rb, b, T),
                reb = __shfl_sync(FULL, re, b, T);
      const bool up = j <= b;                   // row P[j], column P[b]
      lo[u] = on ? (up ? rb : rbb) : 0;
      hi[u] = on ? (up ? re : reb) : 0;
      col[u] = up ? pb : pj;
      at[u] = on ? (up ? b * LD + j : j * LD + b) : -1;
    }
    find_cols<4>(aci, lo, hi, col);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (at[u] >= 0) S[at[u]] = lo[u] >= 0 ? __ldg(av + lo[u]) : 0.0;
  }
  __syncwarp();
  double R[MMAX];
#pragma unroll
  for (int l = 0; l < MMAX; ++l) R[l] = (live && l <= j) ? S[j * LD + l] : (l == j ? 1.0 : 0.0);
  __syncwarp();                                 // S becomes the columns of L
  bool spd = true;
  double dinv = 1.0;                            // 1 / pivot of this lane's step
#pragma unroll
  for (int k = 0; k < MMAX; ++k) {
    if (k < mw) {                               // warp-uniform
      const double d = __shfl_sync(FULL, R[k], k, T);
      if (k < m && !(d > 0.0)) spd = false;
      const double inv = 1.0 / d;
      const double mine = R[k];                 // before scaling
      const double l_jk = mine * inv;
      const double zk = __shfl_sync(FULL, y, k, T);
      if (j > k) y = fma(-l_jk, zk, y);
      if (j == k) dinv = inv;
      if (j < MMAX) S[k * LD + j] = l_jk;
      __syncwarp();
#pragma unroll
      for (int l = (k + 1) & ~1; l < MMAX; l += 2) {
        const double2 v = *reinterpret_cast<const double2 *>(S + k * LD + l);
        if (l > k) R[l] = fma(-mine, v.x, R[l]);
        R[l + 1] = fma(-mine, v.y, R[l + 1]);
      }
    }
  }
  y *= dinv;
#pragma unroll
  for (int k = MMAX - 1; k > 0; --k) {          // L' y = D^-1 z
    if (k < mw) {
      const double yk = __shfl_sync(FULL, y, k, T);
      if (j < k && k < m) y = fma(-S[j * LD + k], yk, y);
    }
  }
  double part = live ? rhs * y : 0.0;
#pragma unroll
  for (int o = T / 2; o > 0; o >>= 1) part += __shfl_xor_sync(FULL, part, o, T);
  double scal = aii - part;
  const bool ok = spd && have_diag && scal > 0.0;
  if (i < 0) return;
  if (!ok) {
    if (j == 0) atomicOr(flags, 1);
    scal = 1.0;
    if (!spd) y = 0.0;                          // keep a defined row: diagonal scaling only
  }
  const double s = 1.0 / sqrt(scal);
  if (live) gval[gs + j] = s * y;
  if (j == 0) gval[gs + m] = s;
}

// Lanes per row of a tile of MMAX unknowns (0: a warp per row with the
// shared-memory factor of fsai_row), warps per block, and shared memory of
// the block.
__host__ __device__ constexpr int fsai_lanes(int mmax) {
  return mmax <= 4 ? 4 : mmax <= 8 ? 8 : mmax <= 16 ? 16 : mmax <= 32 ? 32 : 0;
}
__host__ __device__ constexpr int fsai_warps(int mmax) { return mmax <= 32 ? 4 : 2; }
__host__ __device__ constexpr int fsai_group_doubles(int mmax) {
  return mmax <= 32 ? mmax * (mmax + 2) : mmax * mmax + 3 * mmax;
}
__host__ __device__ constexpr int fsai_rows_per_block(int mmax) {
  return fsai_lanes(mmax) ? fsai_warps(mmax) * 32 / fsai_lanes(mmax) : fsai_warps(mmax);
}
constexpr size_t fsai_smem(int mmax) {
  return (size_t)fsai_rows_per_block(mmax) * fsai_group_doubles(mmax) * sizeof(double);
}

template <int MMAX>
__device__ __forceinline__ void fsai_block_row(int i, const int *arp, const int *aci,
                                               const double *av, const int *grp, const int *gci,
                                               double *gval, int *flags, double *smem) {
  constexpr int T = fsai_lanes(MMAX);
  if constexpr (T > 0)
    fsai_row_reg<T, MMAX>(i, arp, aci, av, grp, gci, gval, flags,
                          smem + (threadIdx.x / T) * fsai_group_doubles(MMAX));
  else if (i >= 0)
    fsai_row<MMAX>(i, arp, aci, av, grp, gci, gval, flags,
                   smem + (threadIdx.x >> 5) * fsai_group_doubles(MMAX), threadIdx.x & 31);
}

// Entry of the list that a thread's group works on, or -1 past its end.
template <int MMAX> __device__ __forceinline__ int fsai_list_entry(int nb) {
  constexpr int T = fsai_lanes(MMAX) ? fsai_lanes(MMAX) : 32;
  const int64_t q = blockIdx.x * (int64_t)fsai_rows_per_block(MMAX) + threadIdx.x / T;
  return q < nb ? (int)q : -1;
}

template <int MMAX>
__global__ void __launch_bounds__(fsai_warps(MMAX) * 32)
k_fsai_numeric(int nb, const int *__restrict__ rows, const int *__restrict__ arp,
               const int *__restrict__ aci, const double *__restrict__ av,
               const int *__restrict__ grp, const int *__restrict__ gci,
               double *__restrict__ gval, int *flags) {
  extern __shared__ __align__(16) double smem[];
  const int q = fsai_list_entry<MMAX>(nb);
  fsai_block_row<MMAX>(q >= 0 ? rows[q] : -1, arp, aci, av, grp, gci, gval, flags, smem);
}

template <int MMAX>
static void launch_fsai(int cnt, const int *rows, const int *arp, const int *aci, const double *av,
                        const int *grp, const int *gci, double *gval, int *flags,
                        cudaStream_t st) {
  if (cnt <= 0) return;
  CHRONOS_CUDA(cudaFuncSetAttribute(k_fsai_numeric<MMAX>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)fsai_smem(MMAX)));
  k_fsai_numeric<MMAX><<<ceil_div(cnt, fsai_rows_per_block(MMAX)), fsai_warps(MMAX) * 32,
                         fsai_smem(MMAX), st>>>(cnt, rows, arp, aci, av, grp, gci, gval, flags);
  CHRONOS_CHECK_LAUNCH();
}

// The buckets of fsai_numeric_device and fsai_numeric_noalloc: local systems
// of at most 4, 8, 16, 32 and 64 unknowns.
constexpr int kFsaiBuckets = 5;
__host__ __device__ constexpr int fsai_bucket(int m) {
  return m <= 4 ? 0 : m <= 8 ? 1 : m <= 16 ? 2 : m <= 32 ? 3 : 4;
}
static void launch_fsai_bucket(int b, int cnt, const int *rows, const int *arp, const int *aci,
                               const double *av, const int *grp, const int *gci, double *gval,
                               int *flags, cudaStream_t st) {
  switch (b) {
    case 0: launch_fsai<4>(cnt, rows, arp, aci, av, grp, gci, gval, flags, st); break;
    case 1: launch_fsai<8>(cnt, rows, arp, aci, av, grp, gci, gval, flags, st); break;
    case 2: launch_fsai<16>(cnt, rows, arp, aci, av, grp, gci, gval, flags, st); break;
    case 3: launch_fsai<32>(cnt, rows, arp, aci, av, grp, gci, gval, flags, st); break;
    default: launch_fsai<64>(cnt, rows, arp, aci, av, grp, gci, gval, flags, st); break;
  }
}

// One problem of a batched FSAI numeric launch (device pointers).
struct FsaiProblemDev {
  const int *arp, *aci;
  const double *av;
  const int *grp, *gci;
  double *gval;
};

// The rows of many problems in one launch: item k = (problem, row); flags
// per problem.
template <int MMAX>
__global__ void __launch_bounds__(fsai_warps(MMAX) * 32)
k_fsai_numeric_batched(int nb, const int2 *__restrict__ items,
                       const FsaiProblemDev *__restrict__ tab, int *flags) {
  extern __shared__ __align__(16) double smem[];
  const int q = fsai_list_entry<MMAX>(nb);
  const int2 it = q >= 0 ? items[q] : make_int2(0, -1);
  const FsaiProblemDev pr = tab[it.x];
  fsai_block_row<MMAX>(it.y, pr.arp, pr.aci, pr.av, pr.grp, pr.gci, pr.gval, flags + it.x, smem);
}

int fsai_numeric_device(int n, const int *arp, const int *aci, const double *av, const int *grp,
                        const int *gci, double *gval, const std::vector<int> &rowlen_h,
                        cudaStream_t st) {
  // Bucket rows by local system size m = rowlen - 1.
  std::vector<int> rows[kFsaiBuckets];
  for (int i = 0; i < n; ++i) {
    const int m = rowlen_h[i] - 1;
    CHRONOS_REQUIRE(m <= 64, CHRONOS_ENOTSUP, "FSAI local system larger than 64 (nstep*step_size)");
    rows[fsai_bucket(m)].push_back(i);
  }
  DBuf<int> flags(1);
  flags.zero(st);
  DBuf<int> drows[kFsaiBuckets];
  for (int b = 0; b < kFsaiBuckets; ++b) {
    drows[b].upload(rows[b], st);
    launch_fsai_bucket(b, (int)rows[b].size(), drows[b].get(), arp, aci, av, grp, gci, gval,
                       flags.get(), st);
  }
  int fl = 0;
  CHRONOS_CUDA(cudaMemcpyAsync(&fl, flags.get(), sizeof(int), cudaMemcpyDeviceToHost, st));
  CHRONOS_CUDA(cudaStreamSynchronize(st));
  return fl;
}

// -----------------------------------------------------------------------------
// FSAI numeric phase of many problems at once (a batch's level): every row of
// every problem goes to the smallest tile (MMAX: lanes and registers up to 32
// unknowns, shared memory above) that holds its local system, and each tile size is
// one launch over all problems' rows.
// Which tile sizes exist -- the bucket edges -- is chosen per batch shape by
// timing the candidate sets below on the batch's own rows (CUDA events); a
// row's arithmetic does not depend on its tile, so every set gives the same
// values bit for bit and the timed runs may overwrite one another.
// -----------------------------------------------------------------------------

namespace {

const std::vector<std::vector<int>> &fsai_bucket_sets() {
  static const std::vector<std::vector<int>> sets = {
      {16, 32, 64}, {8, 16, 32, 64}, {16, 24, 32, 48, 64}, {8, 16, 24, 32, 48, 64}};
  return sets;
}

template <int MMAX>
void launch_fsai_batched(int cnt, const int2 *items, const FsaiProblemDev *tab, int *flags,
                         cudaStream_t st) {
  if (cnt == 0) return;
  CHRONOS_CUDA(cudaFuncSetAttribute(k_fsai_numeric_batched<MMAX>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)fsai_smem(MMAX)));
  k_fsai_numeric_batched<MMAX><<<ceil_div(cnt, fsai_rows_per_block(MMAX)), fsai_warps(MMAX) * 32,
                                 fsai_smem(MMAX), st>>>(cnt, items, tab, flags);
  CHRONOS_CHECK_LAUNCH();
}

void launch_fsai_tile(int mmax, int cnt, const int2 *items, const FsaiProblemDev *tab, int *flags,
                      cudaStream_t st) {
  switch (mmax) {
    case 8: launch_fsai_batched<8>(cnt, items, tab, flags, st); break;
    case 16: launch_fsai_batched<16>(cnt, items, tab, flags, st); break;
    case 24: launch_fsai_batched<24>(cnt, items, tab, flags, st); break;
    case 32: launch_fsai_batched<32>(cnt, items, tab, flags, st); break;
    case 48: launch_fsai_batched<48>(cnt, items, tab, flags, st); break;
    case 64: launch_fsai_batched<64>(cnt, items, tab, flags, st); break;
    default: throw Error(CHRONOS_EINVAL, "no FSAI tile of this size");
  }
}

std::mutex g_fsai_tune_mu;
std::map<std::string, int> g_fsai_tune;       // batch shape -> index of the chosen set

}  // namespace

int fsai_bucket_set_count() { return (int)fsai_bucket_sets().size(); }

std::vector<int> fsai_numeric_batched(const std::vector<FsaiJob> &jobs, cudaStream_t st,
                                      int *chosen_set, int force_set) {
  CHRONOS_REQUIRE(force_set < (int)fsai_bucket_sets().size(), CHRONOS_EINVAL,
                  "no such FSAI tile set");
  const int nj = (int)jobs.size();
  std::vector<int> out(nj, 0);
  if (nj == 0) return out;
  // local sizes: histogram (the batch's shape) and the largest
  std::vector<int64_t> hist(65, 0);
  for (const auto &j : jobs)
    for (int i = 0; i < j.n; ++i) {
      const int m = (*j.rowlen)[i] - 1;
      CHRONOS_REQUIRE(m >= 0 && m <= 64, m > 64 ? CHRONOS_ENOTSUP : CHRONOS_EINVAL,
                      "FSAI local system larger than 64 (nstep*step_size) or an empty row");
      hist[m]++;
    }
  std::vector<FsaiProblemDev> tab_h(nj);
  for (int p = 0; p < nj; ++p)
    tab_h[p] = {jobs[p].arp, jobs[p].aci, jobs[p].av, jobs[p].grp, jobs[p].gci, jobs[p].gval};
  DBuf<FsaiProblemDev> tab;
  tab.upload(tab_h, st);
  DBuf<int> flags(nj);
  // items of one bucket set, bucket by bucket: (problem, row)
  const auto &sets = fsai_bucket_sets();
  auto build_items = [&](const std::vector<int> &set, std::vector<int2> &items,
                         std::vector<int> &start) {
    const int nb = (int)set.size();
    std::vector<int> bucket_of(65);
    for (int m = 0; m <= 64; ++m) {
      int b = 0;
      while (set[b] < m) ++b;
      bucket_of[m] = b;
    }
    start.assign(nb + 1, 0);
    for (int m = 0; m <= 64; ++m) start[bucket_of[m] + 1] += (int)hist[m];
    for (int b = 0; b < nb; ++b) start[b + 1] += start[b];
    items.resize(start[nb]);
    std::vector<int> cur(start.begin(), start.end() - 1);
    for (int p = 0; p < nj; ++p)
      for (int i = 0; i < jobs[p].n; ++i) items[cur[bucket_of[(*jobs[p].rowlen)[i] - 1]]++] = {p, i};
  };
  auto run = [&](const std::vector<int> &set, const DBuf<int2> &items, const std::vector<int> &start) {
    flags.zero(st);
    for (size_t b = 0; b < set.size(); ++b)
      launch_fsai_tile(set[b], start[b + 1] - start[b], items.get() + start[b], tab.get(),
                       flags.get(), st);
  };
  std::string key;
  for (int m = 0; m <= 64; ++m)
    if (hist[m]) key += std::to_string(m) + ":" + std::to_string(hist[m]) + ",";
  int choice = force_set >= 0 ? force_set : -1;
  if (choice < 0) {
    std::lock_guard<std::mutex> lk(g_fsai_tune_mu);
    auto it = g_fsai_tune.find(key);
    if (it != g_fsai_tune.end()) choice = it->second;
  }
  const int64_t rows = std::accumulate(hist.begin(), hist.end(), (int64_t)0);
  if (choice < 0 && rows < 20000) choice = 0;            // small batch: launch-bound either way
  std::vector<int2> items_h;
  std::vector<int> start;
  DBuf<int2> items;
  if (choice < 0) {
    const bool verbose = std::getenv("CHRONOS_TUNE_VERBOSE") != nullptr;
    cudaEvent_t e0, e1;
    CHRONOS_CUDA(cudaEventCreate(&e0));
    CHRONOS_CUDA(cudaEventCreate(&e1));
    float best = 1e30f;
    for (int s = 0; s < (int)sets.size(); ++s) {
      build_items(sets[s], items_h, start);
      items.upload(items_h, st);
      run(sets[s], items, start);                         // warm-up (the attributes, caches)
      CHRONOS_CUDA(cudaEventRecord(e0, st));
      run(sets[s], items, start);
      CHRONOS_CUDA(cudaEventRecord(e1, st));
      CHRONOS_CUDA(cudaEventSynchronize(e1));
      float ms = 0.f;
      CHRONOS_CUDA(cudaEventElapsedTime(&ms, e0, e1));
      if (verbose) {
        std::string edges;
        for (int m : sets[s]) edges += std::to_string(m) + " ";
        std::fprintf(stderr, "chronos tune: fsai batch %lld rows, tiles %s %.4f ms\n",
                     (long long)rows, edges.c_str(), ms);
      }
      if (ms < best) { best = ms; choice = s; }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    std::lock_guard<std::mutex> lk(g_fsai_tune_mu);
    g_fsai_tune[key] = choice;
  }
  build_items(sets[choice], items_h, start);
  items.upload(items_h, st);
  run(sets[choice], items, start);
  flags.download(out.data(), nj, st);
  CHRONOS_CUDA(cudaStreamSynchronize(st));
  if (chosen_set) *chosen_set = choice;
  return out;
}

// =============================================================================
// Sparse product C = X * Y with per-row hash tables in global memory
// =============================================================================

// prod[i]: the products of row i; their sum added to *sum.
__global__ void __launch_bounds__(256)
k_spgemm_products(int m, const int *xrp, const int *xci, const int *yrp, int64_t *prod, int64_t *sum) {
  __shared__ int64_t warp[8];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  int64_t s = 0;
  if (i < m) {
    for (int k = xrp[i]; k < xrp[i + 1]; ++k) {
      const int j = xci[k];
      s += yrp[j + 1] - yrp[j];
    }
    prod[i] = s;
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) warp[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    s = 0;
    for (int w = 0; w < 8; ++w) s += warp[w];
    atomicAdd(reinterpret_cast<unsigned long long *>(sum), (unsigned long long)s);
  }
}

__device__ __forceinline__ unsigned hash_slot(int key, unsigned mask) {
  return ((unsigned)key * 2654435761u) & mask;
}

// Inserts key into the open-addressing table (keys initialised to -1);
// returns the slot and whether this call created it.
__device__ __forceinline__ unsigned hash_insert(int *keys, unsigned mask, int key, bool *fresh) {
  unsigned s = hash_slot(key, mask);
  while (true) {
    int cur = keys[s];
    if (cur == key) { *fresh = false; return s; }
    if (cur == -1) {
      int prev = atomicCAS(keys + s, -1, key);
      if (prev == -1) { *fresh = true; return s; }
      if (prev == key) { *fresh = false; return s; }
    }
    s = (s + 1) & mask;
  }
}

// Symbolic: unique columns per row (warp per row, rows [r0, r1)).
__global__ void k_spgemm_symbolic(int r0, int r1, const int *rows, const int *xrp, const int *xci,
                                  const int *yrp, const int *yci, const int64_t *toff,
                                  const unsigned *tcap, int *keys, int *cnt) {
  const int lane = threadIdx.x & 31;
  const int t = r0 + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (t >= r1) return;
  const int i = rows[t];
  int *tk = keys + toff[t - r0];
  const unsigned cap = tcap[t - r0], mask = cap - 1;
  for (unsigned s = lane; s < cap; s += 32) tk[s] = -1;
  __syncwarp();
  int mine = 0;
  for (int k = xrp[i]; k < xrp[i + 1]; ++k) {
    const int j = xci[k];
    for (int kk = yrp[j] + lane; kk < yrp[j + 1]; kk += 32) {
      bool fresh;
      hash_insert(tk, mask, yci[kk], &fresh);
      mine += fresh;
    }
  }
  mine = warp_sum(mine);
  if (lane == 0) cnt[i] = mine;
}

// Numeric: accumulate in the order of row i of X (products rounded, then
// added), emit the nonzero entries unsorted into [crp_sym[i], ...); cnt_out[i]
// = number emitted.
__global__ void k_spgemm_numeric(int r0, int r1, const int *rows, const int *xrp, const int *xci,
                                 const double *xv, const int *yrp, const int *yci,
                                 const double *yv, const int64_t *toff, const unsigned *tcap,
                                 int *keys, double *vals, const int64_t *crp_sym, int *cci,
                                 double *cv, int *cnt_out) {
  const int lane = threadIdx.x & 31;
  const int t = r0 + (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (t >= r1) return;
  const int i = rows[t];
  int *tk = keys + toff[t - r0];
  double *tv = vals + toff[t - r0];
  const unsigned cap = tcap[t - r0], mask = cap - 1;
  for (unsigned s = lane; s < cap; s += 32) { tk[s] = -1; tv[s] = 0.0; }
  __syncwarp();
  for (int k = xrp[i]; k < xrp[i + 1]; ++k) {
    const int j = xci[k];
    const double a = xv[k];
    for (int kk = yrp[j] + lane; kk < yrp[j + 1]; kk += 32) {
      bool fresh;
      const unsigned s = hash_insert(tk, mask, yci[kk], &fresh);
      tv[s] = __dadd_rn(tv[s], __dmul_rn(a, yv[kk]));
    }
    __syncwarp();
  }
  __syncwarp();
  int64_t base = crp_sym[i];
  int emitted = 0;
  for (unsigned s0 = 0; s0 < cap; s0 += 32) {
    const unsigned s = s0 + lane;
    bool keep = false;
    int key = -1;
    double val = 0.0;
    if (s < cap) {
      key = tk[s];
      val = tv[s];
      keep = key != -1 && val != 0.0;
    }
    const unsigned bal = __ballot_sync(0xffffffffu, keep);
    if (keep) {
      const int off = __popc(bal & ((1u << lane) - 1u));
      cci[base + emitted + off] = key;
      cv[base + emitted + off] = val;
    }
    emitted += __popc(bal);
  }
  if (lane == 0) cnt_out[i] = emitted;
}

// Shared-memory variants for rows whose distinct columns fill at most half of
// a warp's table (kSpgemmSmSlots at the largest; rows beyond go to the global
// tables above).  The products of a row are taken 32 at a time across the
// entries of X's row -- Y's rows (a prolongation's) are often far shorter than
// a warp -- and the lanes that hold the same column add theirs in lane order,
// which is X's row order: every output entry is the same sum, rounded at the
// same places, as a row-wise Gustavson product's.  A row's table is as large as
// its class needs, so that short rows fill the SM with warps; the numeric
// kernel sorts its row in the table before it leaves.  A*P and P'*(A*P) of
// elasticity 26^3 (57k rows, 81 entries times 4 to 5): an entry of X at a time
// in 4096-slot tables (4 warps per SM) 6.6 ms, then 1.7 ms in the segmented
// sort; now 1.5 ms together.
constexpr int kSpgemmSmSlots = 4096;

// One class of rows, of at most SLOTS / 2 distinct columns: warps per block.
template <int SLOTS> struct SpgemmClass {
  static constexpr int warps = SLOTS <= 1024 ? 8 : 4;
};

// Entries [k0, k0 + 32) of row X: lane l holds entry k0 + l's value, the offset
// of Y's row minus the products before it, and the running product count.
struct SpgemmChunk {
  double a = 0.0;
  int base = 0, inc = 0, total = 0;
  __device__ __forceinline__ void load(int k, int ke, const int *__restrict__ xci,
                                       const double *__restrict__ xv,
                                       const int *__restrict__ yrp) {
    const int lane = threadIdx.x & 31;
    int ys = 0, len = 0;
    a = 0.0;
    if (k < ke) {
      const int j = __ldg(xci + k);
      if (xv) a = __ldg(xv + k);
      ys = __ldg(yrp + j);
      len = __ldg(yrp + j + 1) - ys;
    }
    inc = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    total = __shfl_sync(0xffffffffu, inc, 31);
    base = ys - (inc - len);
  }
  // lane holding product t's entry of X
  __device__ __forceinline__ int owner(int t) const {
    int lo = 0;
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
      if (__shfl_sync(0xffffffffu, inc, lo + step - 1) <= t) lo += step;
    return lo;
  }
};

// Symbolic: cnt[i] = distinct columns of the rows whose bound (products, at
// most ncols) is in (lo, SLOTS/2], or for the largest class everything above
// lo: -1 (and *nbig) when they outgrow half the table.
template <int SLOTS>
__global__ void __launch_bounds__(32 * SpgemmClass<SLOTS>::warps)
k_spgemm_symbolic_sm(int m, int ncols, int lo, const int *__restrict__ xrp,
                     const int *__restrict__ xci, const int *__restrict__ yrp,
                     const int *__restrict__ yci, const int64_t *__restrict__ prod,
                     int *__restrict__ cnt, int *nbig, const int64_t *__restrict__ sum,
                     int64_t max_products) {
  if (*sum > max_products) return;            // more than the caller wants formed
  constexpr int W = SpgemmClass<SLOTS>::warps;
  constexpr bool TOP = SLOTS == kSpgemmSmSlots;
  extern __shared__ int spg_keys[];
  const int lane = threadIdx.x & 31;
  int *tk = spg_keys + (threadIdx.x >> 5) * SLOTS;
  const int nw = gridDim.x * W;
  for (int i = blockIdx.x * W + (threadIdx.x >> 5); i < m; i += nw) {
    const int64_t p = __ldg(prod + i);
    const int bound = (int)(p < ncols ? p : ncols);
    if (bound <= lo || (!TOP && bound > SLOTS / 2)) continue;
    unsigned tsz = 32;
    while (tsz < SLOTS && tsz < 2u * bound) tsz <<= 1;
    for (unsigned s = lane; s < tsz; s += 32) tk[s] = -1;
    __syncwarp();
    int count = 0;
    bool over = false;
    const int xs = __ldg(xrp + i), xe = __ldg(xrp + i + 1);
    for (int k0 = xs; k0 < xe && !over; k0 += 32) {
      SpgemmChunk c;
      c.load(k0 + lane, xe, xci, nullptr, yrp);
      for (int t0 = 0; t0 < c.total && !over; t0 += 32) {
        const int t = t0 + lane, o = c.owner(t);
        const int base = __shfl_sync(0xffffffffu, c.base, o);
        bool fresh = false;
        if (t < c.total) hash_insert(tk, tsz - 1, __ldg(yci + base + t), &fresh);
        count += __popc(__ballot_sync(0xffffffffu, fresh));
        over = TOP && 2 * count > SLOTS;               // the same for every lane
      }
    }
    if (lane == 0) {
      cnt[i] = over ? -1 : count;
      if (over) atomicAdd(nbig, 1);
    }
    __syncwarp();
  }
}

// Numeric for the rows with cnt in (lo, SLOTS/2]: the nonzero entries, columns
// ascending, at cci/cv[crp_sym[i]..]; cnt_out[i] = number emitted.
template <int SLOTS>
__global__ void __launch_bounds__(32 * SpgemmClass<SLOTS>::warps)
k_spgemm_numeric_sm(int m, int lo, const int *__restrict__ xrp, const int *__restrict__ xci,
                    const double *__restrict__ xv, const int *__restrict__ yrp,
                    const int *__restrict__ yci, const double *__restrict__ yv,
                    const int *__restrict__ cnt, const int64_t *__restrict__ crp_sym,
                    int *__restrict__ cci, double *__restrict__ cv, int *__restrict__ cnt_out) {
  constexpr int W = SpgemmClass<SLOTS>::warps;
  constexpr unsigned FULL = 0xffffffffu;
  extern __shared__ double spg_vals[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  double *tv = spg_vals + (size_t)wib * SLOTS;
  int *tk = reinterpret_cast<int *>(spg_vals + (size_t)W * SLOTS) + wib * SLOTS;
  const int nw = gridDim.x * W;
  for (int i = blockIdx.x * W + wib; i < m; i += nw) {
    const int n = __ldg(cnt + i);
    if (n <= lo || n > SLOTS / 2) continue;
    unsigned tsz = 32;
    while (tsz < 2u * n) tsz <<= 1;
    for (unsigned s = lane; s < tsz; s += 32) { tk[s] = -1; tv[s] = 0.0; }
    __syncwarp();
    const int xs = __ldg(xrp + i), xe = __ldg(xrp + i + 1);
    for (int k0 = xs; k0 < xe; k0 += 32) {
      SpgemmChunk c;
      c.load(k0 + lane, xe, xci, xv, yrp);
      for (int t0 = 0; t0 < c.total; t0 += 32) {
        const int t = t0 + lane, o = c.owner(t);
        const int base = __shfl_sync(FULL, c.base, o);
        const double a = __shfl_sync(FULL, c.a, o);
        const bool on = t < c.total;
        int col = -1 - lane;                           // idle lanes: alone
        double prod = 0.0;
        if (on) {
          col = __ldg(yci + base + t);
          prod = __dmul_rn(a, __ldg(yv + base + t));
        }
        unsigned same = __match_any_sync(FULL, col);
        const bool lead = on && (same & ((1u << lane) - 1u)) == 0;
        unsigned s = 0;
        double acc = 0.0;
        if (lead) {
          bool fresh;
          s = hash_insert(tk, tsz - 1, col, &fresh);
          acc = tv[s];
        }
        // the column's lanes in ascending order, one a round
        const int rounds = __reduce_max_sync(FULL, lead ? __popc(same) : 0);
        for (int q = 0; q < rounds; ++q) {
          const double v = __shfl_sync(FULL, prod, same ? __ffs(same) - 1 : lane);
          if (same) {
            acc = __dadd_rn(acc, v);
            same &= same - 1;
          }
        }
        if (lead) tv[s] = acc;
        __syncwarp();
      }
    }
    // the kept entries to the table's front (writes never pass the reads) ...
    int kept = 0;
    for (unsigned s0 = 0; s0 < tsz; s0 += 32) {
      const int key = tk[s0 + lane];
      const double val = tv[s0 + lane];
      const bool keep = key != -1 && val != 0.0;
      const unsigned bal = __ballot_sync(FULL, keep);
      if (keep) {
        const int at = kept + __popc(bal & ((1u << lane) - 1u));
        tk[at] = key;
        tv[at] = val;
      }
      kept += __popc(bal);
      __syncwarp();
    }
    // ... sorted by column (bitonic over the next power of two)
    int N = 2;
    while (N < kept) N <<= 1;
    for (int t = kept + lane; t < N; t += 32) tk[t] = 0x7fffffff;
    __syncwarp();
    for (int k = 2; k <= N; k <<= 1)
      for (int j = k >> 1; j > 0; j >>= 1) {
        for (int t = lane; t < N / 2; t += 32) {
          const int p = 2 * t - (t & (j - 1)), q = p + j;
          const int kp = tk[p], kq = tk[q];
          if ((kp > kq) == ((p & k) == 0)) {
            const double vp = tv[p], vq = tv[q];
            tk[p] = kq; tk[q] = kp;
            tv[p] = vq; tv[q] = vp;
          }
        }
        __syncwarp();
      }
    const int64_t out = __ldg(crp_sym + i);
    for (int t = lane; t < kept; t += 32) {
      cci[out + t] = tk[t];
      cv[out + t] = tv[t];
    }
    if (lane == 0) cnt_out[i] = kept;
    __syncwarp();
  }
}

template <int SLOTS>
static void spgemm_symbolic(int m, int ncols, int lo, const int *xrp, const int *xci,
                            const int *yrp, const int *yci, const int64_t *prod, int *cnt,
                            int *nbig, const int64_t *sum, int64_t max_products,
                            cudaStream_t st) {
  using C = SpgemmClass<SLOTS>;
  const int grid = std::max(1, std::min<int>(ceil_div(m, C::warps), num_sms() * 16));
  const size_t smem = (size_t)C::warps * SLOTS * sizeof(int);
  CHRONOS_CUDA(cudaFuncSetAttribute(k_spgemm_symbolic_sm<SLOTS>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  k_spgemm_symbolic_sm<SLOTS><<<grid, 32 * C::warps, smem, st>>>(m, ncols, lo, xrp, xci, yrp, yci,
                                                                 prod, cnt, nbig, sum,
                                                                 max_products);
  CHRONOS_CHECK_LAUNCH();
}

template <int SLOTS>
static void spgemm_numeric(int m, int lo, const int *xrp, const int *xci, const double *xv,
                           const int *yrp, const int *yci, const double *yv, const int *cnt,
                           const int64_t *crp_sym, int *cci, double *cv, int *cnt_out,
                           cudaStream_t st) {
  using C = SpgemmClass<SLOTS>;
  const size_t smem = (size_t)C::warps * SLOTS * (sizeof(int) + sizeof(double));
  CHRONOS_CUDA(cudaFuncSetAttribute(k_spgemm_numeric_sm<SLOTS>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int grid = std::max(1, std::min<int>(ceil_div(m, C::warps), num_sms() * 16));
  k_spgemm_numeric_sm<SLOTS><<<grid, 32 * C::warps, smem, st>>>(
      m, lo, xrp, xci, xv, yrp, yci, yv, cnt, crp_sym, cci, cv, cnt_out);
  CHRONOS_CHECK_LAUNCH();
}

// Rows from their places in the symbolic layout to the final one (a warp per
// row); rows computed in global tables (sym_cnt beyond the largest class) come
// from the second pair of arrays.
__global__ void __launch_bounds__(256)
k_compact_rows(int m, const int64_t *__restrict__ src_rp, const int *__restrict__ sym_cnt,
               const int *__restrict__ crp, const int *__restrict__ sci,
               const double *__restrict__ sv, const int *__restrict__ bci,
               const double *__restrict__ bv, int *__restrict__ dci, double *__restrict__ dv) {
  const int lane = threadIdx.x & 31;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < m; i += nw) {
    const int64_t s = src_rp[i];
    const int d = crp[i], c = crp[i + 1] - d;
    const bool big = sym_cnt[i] > kSpgemmSmSlots / 2;
    const int *ci = big ? bci : sci;
    const double *v = big ? bv : sv;
    for (int k = lane; k < c; k += 32) {
      dci[d + k] = ci[s + k];
      dv[d + k] = v[s + k];
    }
  }
}

__global__ void k_narrow(int n, const int64_t *__restrict__ a, int *__restrict__ b) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    b[i] = (int)a[i];
}

// Exclusive sums of the n + 1 counts (the last one 0) into offs, 64-bit; the
// negative marks of rows still to be counted add nothing.
struct NonNegative {
  __host__ __device__ int64_t operator()(int c) const { return c > 0 ? c : 0; }
};
static void scan_counts(int n, const int *cnt, int64_t *offs, DBuf<unsigned char> &tmp,
                        cudaStream_t st) {
  thrust::transform_iterator<NonNegative, const int *> in(cnt, NonNegative{});
  size_t bytes = 0;
  CHRONOS_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, bytes, in, offs, n + 1, st));
  if (tmp.size() < bytes) tmp.alloc(std::max<size_t>(bytes, 1));
  CHRONOS_CUDA(cub::DeviceScan::ExclusiveSum(tmp.get(), bytes, in, offs, n + 1, st));
}

static unsigned next_pow2(uint64_t v) {
  uint64_t p = 32;
  while (p < v) p <<= 1;
  return (unsigned)p;
}

bool spgemm_device(int m, int ncols, const int *xrp, const int *xci, const double *xv,
                   const int *yrp, const int *yci, const double *yv, DBuf<int> &crp,
                   DBuf<int> &cci, DBuf<double> &cv, int64_t *nnz_c, cudaStream_t st,
                   int64_t max_products) {
  crp.alloc((size_t)m + 1);
  if (m == 0) {
    crp.zero(st);
    *nnz_c = 0;
    return true;
  }
  const int64_t most = max_products > 0 ? max_products : INT64_MAX;
  // behind the row offsets: the products' sum and the rows beyond the tables, read
  // with the offsets' last in one copy
  DBuf<int64_t> dprod((size_t)m + 1), drps((size_t)m + 3);
  int64_t *sum = drps.get() + m + 1;
  int *dnbig = reinterpret_cast<int *>(sum + 1);
  CHRONOS_CUDA(cudaMemsetAsync(sum, 0, 2 * sizeof(int64_t), st));
  DBuf<unsigned char> tmp;
  k_spgemm_products<<<ceil_div(m, 256), 256, 0, st>>>(m, xrp, xci, yrp, dprod.get(), sum);
  CHRONOS_CHECK_LAUNCH();
  // symbolic: in each warp's shared table; rows whose distinct columns outgrow
  // the largest (cnt = -1) again in global tables sized from their products.
  // counts: cnt (m + 1), emitted (m + 1)
  DBuf<int> counts(2 * ((size_t)m + 1));
  int *cnt = counts.get(), *cnt2 = cnt + m + 1;
  counts.zero(st);
  spgemm_symbolic<256>(m, ncols, 0, xrp, xci, yrp, yci, dprod.get(), cnt, dnbig, sum,
                       most, st);
  spgemm_symbolic<1024>(m, ncols, 128, xrp, xci, yrp, yci, dprod.get(), cnt, dnbig, sum,
                        most, st);
  spgemm_symbolic<kSpgemmSmSlots>(m, ncols, 512, xrp, xci, yrp, yci, dprod.get(), cnt, dnbig, sum,
                                  most, st);
  scan_counts(m, cnt, drps.get(), tmp, st);
  int64_t heads[3] = {};
  CHRONOS_CUDA(cudaMemcpyAsync(heads, drps.get() + m, sizeof(heads), cudaMemcpyDeviceToHost, st));
  CHRONOS_CUDA(cudaStreamSynchronize(st));
  int64_t total = heads[0];
  const int nbig = (int)heads[2];
  if (heads[1] > most) return false;
  std::vector<int> cnt_h;
  if (nbig > 0) {
    cnt_h.resize(m);
    CHRONOS_CUDA(cudaMemcpyAsync(cnt_h.data(), cnt, sizeof(int) * m, cudaMemcpyDeviceToHost, st));
    CHRONOS_CUDA(cudaStreamSynchronize(st));
  }
  std::vector<int> big;                                // rows for the global tables
  for (int i = 0; i < m && nbig > 0; ++i)
    if (cnt_h[i] < 0) big.push_back(i);
  DBuf<int> dbig;
  std::vector<int> bounds{0};
  DBuf<int> keys;
  DBuf<double> vals;
  DBuf<int64_t> toff;
  DBuf<unsigned> tcap;
  if (nbig > 0) {
    std::vector<int64_t> prod(m);
    dprod.download(prod.data(), m, st);
    CHRONOS_CUDA(cudaStreamSynchronize(st));
    std::vector<unsigned> cap(nbig);
    const uint64_t colcap = (uint64_t)2 * (uint64_t)std::max(ncols, 1);
    for (int t = 0; t < nbig; ++t)
      cap[t] = next_pow2(std::min<uint64_t>(2 * (uint64_t)prod[big[t]] + 1, colcap));
    // chunks of rows whose tables fit the slot budget
    const uint64_t budget = (uint64_t)1 << 24;     // 16M slots (192 MB with values)
    uint64_t acc = 0;
    for (int t = 0; t < nbig; ++t) {
      if (acc + cap[t] > budget && t > bounds.back()) { bounds.push_back(t); acc = 0; }
      acc += cap[t];
    }
    bounds.push_back(nbig);
    uint64_t maxchunk = 0;
    std::vector<int64_t> toff_h(nbig);
    for (size_t c = 0; c + 1 < bounds.size(); ++c) {
      int64_t a = 0;
      for (int t = bounds[c]; t < bounds[c + 1]; ++t) { toff_h[t] = a; a += cap[t]; }
      maxchunk = std::max<uint64_t>(maxchunk, (uint64_t)a);
    }
    keys.alloc(maxchunk);
    vals.alloc(maxchunk);
    toff.upload(toff_h, st);
    tcap.upload(cap.data(), nbig, st);
    dbig.upload(big, st);
    for (size_t c = 0; c + 1 < bounds.size(); ++c) {
      const int t0 = bounds[c], t1 = bounds[c + 1];
      k_spgemm_symbolic<<<ceil_div((int64_t)(t1 - t0) * 32, 256), 256, 0, st>>>(
          t0, t1, dbig.get(), xrp, xci, yrp, yci, toff.get() + t0, tcap.get() + t0, keys.get(),
          cnt);
      CHRONOS_CHECK_LAUNCH();
    }
    scan_counts(m, cnt, drps.get(), tmp, st);
    CHRONOS_CUDA(cudaMemcpyAsync(&total, drps.get() + m, sizeof(total), cudaMemcpyDeviceToHost,
                                 st));
    CHRONOS_CUDA(cudaStreamSynchronize(st));
  }
  DBuf<int> sci(std::max<int64_t>(total, 1)), sci2;
  DBuf<double> sv(std::max<int64_t>(total, 1)), sv2;
  spgemm_numeric<128>(m, 0, xrp, xci, xv, yrp, yci, yv, cnt, drps.get(), sci.get(), sv.get(), cnt2,
                      st);
  spgemm_numeric<512>(m, 64, xrp, xci, xv, yrp, yci, yv, cnt, drps.get(), sci.get(), sv.get(),
                      cnt2, st);
  spgemm_numeric<2048>(m, 256, xrp, xci, xv, yrp, yci, yv, cnt, drps.get(), sci.get(), sv.get(),
                       cnt2, st);
  spgemm_numeric<kSpgemmSmSlots>(m, 1024, xrp, xci, xv, yrp, yci, yv, cnt, drps.get(), sci.get(),
                                 sv.get(), cnt2, st);
  if (nbig > 0) {
    for (size_t c = 0; c + 1 < bounds.size(); ++c) {
      const int t0 = bounds[c], t1 = bounds[c + 1];
      k_spgemm_numeric<<<ceil_div((int64_t)(t1 - t0) * 32, 256), 256, 0, st>>>(
          t0, t1, dbig.get(), xrp, xci, xv, yrp, yci, yv, toff.get() + t0, tcap.get() + t0,
          keys.get(), vals.get(), drps.get(), sci.get(), sv.get(), cnt2);
      CHRONOS_CHECK_LAUNCH();
    }
    // their segments sorted by column into the second pair of arrays
    std::vector<int64_t> rps((size_t)m + 1), sb(nbig), se(nbig);
    std::vector<int> got(m);
    drps.download(rps.data(), (size_t)m + 1, st);
    CHRONOS_CUDA(cudaMemcpyAsync(got.data(), cnt2, sizeof(int) * m, cudaMemcpyDeviceToHost, st));
    CHRONOS_CUDA(cudaStreamSynchronize(st));
    for (int t = 0; t < nbig; ++t) {
      sb[t] = rps[big[t]];
      se[t] = sb[t] + got[big[t]];
    }
    DBuf<int64_t> dsb, dse;
    dsb.upload(sb, st);
    dse.upload(se, st);
    sci2.alloc(total);
    sv2.alloc(total);
    size_t bytes = 0;
    CHRONOS_CUDA(cub::DeviceSegmentedSort::SortPairs(nullptr, bytes, sci.get(), sci2.get(),
                                                     sv.get(), sv2.get(), total, nbig, dsb.get(),
                                                     dse.get(), st));
    if (tmp.size() < bytes) tmp.alloc(std::max<size_t>(bytes, 1));
    CHRONOS_CUDA(cub::DeviceSegmentedSort::SortPairs(tmp.get(), bytes, sci.get(), sci2.get(),
                                                     sv.get(), sv2.get(), total, nbig, dsb.get(),
                                                     dse.get(), st));
    CHRONOS_CUDA(cudaStreamSynchronize(st));   // dsb, dse leave this scope
  }
  scan_counts(m, cnt2, dprod.get(), tmp, st);    // the product counts have served
  int64_t nnz = 0;
  CHRONOS_CUDA(cudaMemcpyAsync(&nnz, dprod.get() + m, sizeof(nnz), cudaMemcpyDeviceToHost, st));
  CHRONOS_CUDA(cudaStreamSynchronize(st));
  CHRONOS_REQUIRE(nnz < INT32_MAX, CHRONOS_ENOTSUP, "sparse product exceeds 2^31 entries");
  k_narrow<<<std::min<int>(ceil_div(m + 1, 256), num_sms() * 8), 256, 0, st>>>(m + 1, dprod.get(),
                                                                               crp.get());
  CHRONOS_CHECK_LAUNCH();
  if (nnz == total && nbig == 0) {             // nothing dropped: the rows lie where they belong
    cci = std::move(sci);
    cv = std::move(sv);
  } else {
    cci.alloc(std::max<int64_t>(nnz, 1));
    cv.alloc(std::max<int64_t>(nnz, 1));
    k_compact_rows<<<std::min<int>(ceil_div(m, 8), num_sms() * 16), 256, 0, st>>>(
        m, drps.get(), cnt, crp.get(), sci.get(), sv.get(), nbig ? sci2.get() : sci.get(),
        nbig ? sv2.get() : sv.get(), cci.get(), cv.get());
    CHRONOS_CHECK_LAUNCH();
  }
  CHRONOS_CUDA(cudaStreamSynchronize(st));
  *nnz_c = nnz;
  return true;
}

// =============================================================================
// Dense coarse level
// =============================================================================

// Blocked right-looking Cholesky, 32-column panels: k_chol_panel factors the
// diagonal block (every block of the grid for itself, in one warp's registers)
// and solves its 64 rows of the panel against it, k_chol_update subtracts the
// panel's outer product from the trailing lower tiles.  The inverse of the
// factor is put together from its 32 x 32 diagonal blocks' by doubling, and
// A^-1 = X'X, all on 64 x 64 FP64 tiles.  One thread block for the whole
// factorisation and a block per column for the inverse, a barrier per column,
// took 53 ms for the coarsest level of diffusion 36^3 (about 950 rows), its assembly
// and upload included; now 4.7 ms.
constexpr int kCholNb = 32;

// c += op(A) op(B) over k in [k0, k1): rows i0 + tx + 16 r, columns
// j0 + ty + 16 q of a 64 x 64 tile; la(i, k) and lb(k, j) give 0 outside.
// KA / KB: the operand is contiguous along k.
template <bool KA, bool KB, typename LA, typename LB>
__device__ __forceinline__ void tile_gemm(int i0, int j0, int k0, int k1, LA la, LB lb,
                                          double (&c)[4][4]) {
  __shared__ double As[16][65], Bs[16][65];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  for (int k = k0; k < k1; k += 16) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = tid + 256 * u;
      const int ia = KA ? e >> 4 : e & 63, ka = KA ? e & 15 : e >> 6;
      const int jb = KB ? e >> 4 : e & 63, kb = KB ? e & 15 : e >> 6;
      As[ka][ia] = k + ka < k1 ? la(i0 + ia, k + ka) : 0.0;
      Bs[kb][jb] = k + kb < k1 ? lb(k + kb, j0 + jb) : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < 16; ++kk) {
      double av[4], bv[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        av[r] = As[kk][tx + 16 * r];
        bv[r] = Bs[kk][ty + 16 * r];
      }
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) c[r][q] = fma(av[r], bv[q], c[r][q]);
    }
    __syncthreads();
  }
}

// Panel [k0, k0 + nb): D receives the diagonal block's factor (32 x 32, column
// by column; the other blocks of the grid still read A's), A the rows below it.
// info[0]: what the panels before it found; info[1], read by later launches only:
// that, or the 1-based index of this panel's first non-positive pivot.
__global__ void __launch_bounds__(256)
k_chol_panel(int n, int k0, int nb, double *A, double *D, int *info) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ double Ls[kCholNb][kCholNb + 1], Xs[kCholNb][65];
  __shared__ int bad;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (*info) {
    if (blockIdx.x == 0 && tid == 0) info[1] = *info;
    return;
  }
  const int r0 = k0 + nb + blockIdx.x * 64;
  for (int e = tid; e < nb * 64; e += 256) {
    const int i = e & 63, j = e >> 6;
    Xs[j][i] = r0 + i < n ? A[(size_t)(k0 + j) * n + r0 + i] : 0.0;
  }
  if (wid == 0) {
    double R[kCholNb];
#pragma unroll
    for (int c = 0; c < kCholNb; ++c)
      R[c] = (lane < nb && c <= lane) ? A[(size_t)(k0 + c) * n + k0 + lane]
                                      : (c == lane ? 1.0 : 0.0);
    int first = 0;
#pragma unroll
    for (int k = 0; k < kCholNb; ++k) {
      const double d = __shfl_sync(FULL, R[k], k);
      if (!(d > 0.0) && first == 0) first = k0 + k + 1;
      const double s = sqrt(d), l = R[k] / s;
      R[k] = lane == k ? s : l;
#pragma unroll
      for (int c = k + 1; c < kCholNb; ++c) {
        const double v = __shfl_sync(FULL, l, c);
        if (lane >= c) R[c] = fma(-l, v, R[c]);
      }
    }
    if (lane == 0) bad = first;
#pragma unroll
    for (int c = 0; c < kCholNb; ++c) Ls[lane][c] = c <= lane ? R[c] : 0.0;
  }
  __syncthreads();
  if (blockIdx.x == 0) {
    for (int e = tid; e < kCholNb * kCholNb; e += 256) D[e] = Ls[e & 31][e >> 5];
    if (tid == 0) info[1] = bad;
  }
  if (bad) return;
  // row x of the panel: x L' = a, lane j its entry j; a warp's eight rows together
  double L[kCholNb];
#pragma unroll
  for (int c = 0; c < kCholNb; ++c) L[c] = Ls[lane][c];
  const double inv = 1.0 / Ls[lane][lane];
  double x[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) x[q] = lane < nb ? Xs[lane][wid * 8 + q] : 0.0;
#pragma unroll
  for (int k = 0; k < kCholNb; ++k) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const double xk = __shfl_sync(FULL, x[q] * inv, k);
      x[q] = lane == k ? xk : lane > k ? fma(-L[k], xk, x[q]) : x[q];
    }
  }
  if (lane < nb)
#pragma unroll
    for (int q = 0; q < 8; ++q) Xs[lane][wid * 8 + q] = x[q];
  __syncthreads();
  for (int e = tid; e < nb * 64; e += 256) {
    const int i = e & 63, j = e >> 6;
    if (r0 + i < n) A[(size_t)(k0 + j) * n + r0 + i] = Xs[j][i];
  }
}

// Lower tiles of the trailing matrix [t0, n)^2 minus the panel's X X'.
__global__ void __launch_bounds__(256)
k_chol_update(int n, int k0, int t0, double *A, const int *info) {
  if (*info || blockIdx.y < blockIdx.x) return;
  const int i0 = t0 + blockIdx.y * 64, j0 = t0 + blockIdx.x * 64;
  double c[4][4] = {};
  tile_gemm<false, false>(
      i0, j0, k0, t0, [&](int i, int k) { return i < n ? A[(size_t)k * n + i] : 0.0; },
      [&](int k, int j) { return j < n ? A[(size_t)k * n + j] : 0.0; }, c);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = i0 + tx + 16 * r, j = j0 + ty + 16 * q;
      if (i < n && j < n) A[(size_t)j * n + i] -= c[r][q];
    }
}

// The diagonal blocks' factors into place, the strict upper triangle zero.
__global__ void __launch_bounds__(256)
k_chol_finish(int n, double *A, const double *__restrict__ D) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < (int64_t)n * n;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(e % n), j = (int)(e / n), b = j / kCholNb;
    if (i < j) A[e] = 0.0;
    else if (i / kCholNb == b)
      A[e] = D[(size_t)b * kCholNb * kCholNb + (j % kCholNb) * kCholNb + i % kCholNb];
  }
}

int dense_cholesky_device(int n, double *A, cudaStream_t st) {
  if (n <= 0) return 0;
  const int np = ceil_div(n, kCholNb);
  DBuf<double> D((size_t)np * kCholNb * kCholNb);
  DBuf<int> info((size_t)np + 1);               // before each panel, and after the last
  info.zero(st);
  for (int p = 0; p < np; ++p) {
    const int k0 = p * kCholNb, nb = std::min(kCholNb, n - k0), rest = n - k0 - nb;
    k_chol_panel<<<std::max(1u, ceil_div(rest, 64)), 256, 0, st>>>(
        n, k0, nb, A, D.get() + (size_t)p * kCholNb * kCholNb, info.get() + p);
    CHRONOS_CHECK_LAUNCH();
    if (rest > 0) {
      const unsigned t = ceil_div(rest, 64);
      k_chol_update<<<dim3(t, t), 256, 0, st>>>(n, k0, k0 + nb, A, info.get() + p + 1);
      CHRONOS_CHECK_LAUNCH();
    }
  }
  k_chol_finish<<<std::min<int64_t>(ceil_div((int64_t)n * n, 256), (int64_t)num_sms() * 8), 256, 0,
                  st>>>(n, A, D.get());
  CHRONOS_CHECK_LAUNCH();
  int h = 0;
  CHRONOS_CUDA(cudaMemcpyAsync(&h, info.get() + np, sizeof(int), cudaMemcpyDeviceToHost, st));
  CHRONOS_CUDA(cudaStreamSynchronize(st));
  return h;
}

// Inverses of L's 32 x 32 diagonal blocks (a warp each, lane j column j).
__global__ void __launch_bounds__(32)
k_tri_inverse_diag(int n, const double *__restrict__ L, double *__restrict__ X) {
  __shared__ double Ls[kCholNb][kCholNb + 1];
  const int k0 = blockIdx.x * kCholNb, nb = min(kCholNb, n - k0), lane = threadIdx.x;
  for (int j = 0; j < kCholNb; ++j)
    Ls[lane][j] = (lane < nb && j < nb && j <= lane) ? L[(size_t)(k0 + j) * n + k0 + lane]
                                                     : (lane == j ? 1.0 : 0.0);
  __syncwarp();
  double x[kCholNb];
#pragma unroll
  for (int i = 0; i < kCholNb; ++i) {
    double t = i == lane ? 1.0 : 0.0;
#pragma unroll
    for (int k = 0; k < i; ++k) t = fma(-Ls[i][k], x[k], t);
    x[i] = t / Ls[i][i];
  }
  if (lane < nb)
#pragma unroll
    for (int i = 0; i < kCholNb; ++i)
      if (i < nb) X[(size_t)(k0 + lane) * n + k0 + i] = x[i];
}

// One doubling of the inverse: with the s x s diagonal blocks of X done, the
// blocks below them, X21 = -X22 (L21 X11); FIRST computes T = L21 X11.
template <bool FIRST>
__global__ void __launch_bounds__(256)
k_tri_inverse_merge(int n, int s, const double *__restrict__ L, double *X, double *T) {
  const int c0 = blockIdx.z * 2 * s, b0 = c0 + s, b1 = min(n, b0 + s);
  const int i0 = b0 + blockIdx.y * 64, j0 = c0 + blockIdx.x * 64;
  if (i0 >= b1) return;
  double c[4][4] = {};
  if (FIRST)
    tile_gemm<false, true>(
        i0, j0, j0, b0, [&](int i, int k) { return i < b1 ? L[(size_t)k * n + i] : 0.0; },
        [&](int k, int j) { return j < b0 ? X[(size_t)j * n + k] : 0.0; }, c);
  else
    tile_gemm<false, true>(
        i0, j0, b0, min(b1, i0 + 64), [&](int i, int k) { return i < b1 ? X[(size_t)k * n + i] : 0.0; },
        [&](int k, int j) { return j < b0 ? T[(size_t)j * n + k] : 0.0; }, c);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = i0 + tx + 16 * r, j = j0 + ty + 16 * q;
      if (i < b1 && j < b0) (FIRST ? T : X)[(size_t)j * n + i] = FIRST ? c[r][q] : -c[r][q];
    }
}

// W = X'X with X lower triangular, every tile from its first nonzero row on.
__global__ void __launch_bounds__(256)
k_gram(int n, const double *__restrict__ X, double *__restrict__ W) {
  const int i0 = blockIdx.y * 64, j0 = blockIdx.x * 64;
  double c[4][4] = {};
  tile_gemm<true, true>(
      i0, j0, max(i0, j0), n, [&](int i, int k) { return i < n ? X[(size_t)i * n + k] : 0.0; },
      [&](int k, int j) { return j < n ? X[(size_t)j * n + k] : 0.0; }, c);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = i0 + tx + 16 * r, j = j0 + ty + 16 * q;
      if (i < n && j < n) W[(size_t)j * n + i] = c[r][q];
    }
}

void dense_inverse_from_chol(int n, const double *L, double *W, cudaStream_t st) {
  // (beyond 25,600 rows an array of the dense solve takes 5.2 GB)
  CHRONOS_REQUIRE(n <= 25600, CHRONOS_ENOTSUP, "coarsest level too large for the dense solve");
  DBuf<double> X((size_t)n * n);
  X.zero(st);
  k_tri_inverse_diag<<<ceil_div(n, kCholNb), 32, 0, st>>>(n, L, X.get());
  CHRONOS_CHECK_LAUNCH();
  for (int s = kCholNb; s < n; s *= 2) {       // T in W, which is written last
    const unsigned t = ceil_div(s, 64), pairs = ceil_div(n - s, 2 * s);
    k_tri_inverse_merge<true><<<dim3(t, t, pairs), 256, 0, st>>>(n, s, L, X.get(), W);
    CHRONOS_CHECK_LAUNCH();
    k_tri_inverse_merge<false><<<dim3(t, t, pairs), 256, 0, st>>>(n, s, L, X.get(), W);
    CHRONOS_CHECK_LAUNCH();
  }
  const unsigned t = ceil_div(n, 64);
  k_gram<<<dim3(t, t), 256, 0, st>>>(n, X.get(), W);
  CHRONOS_CHECK_LAUNCH();
  CHRONOS_CUDA(cudaStreamSynchronize(st));
}

// x = W b: NT threads a row, each with eight loads of W in flight: the whole row up
// to 2048 columns, longer rows (a single level or one that stopped coarsening) in
// rounds of 2048.  With a warp a row and four in flight the product was a
// chain of batches on 8 warps an SM: 1212 rows of the folded tail of elasticity
// 45^3 (11.8 MB, from L2) 11.5 us, now 6.1; 208 rows 3.6 and 2.5 us.  (Rows of many
// small systems at once, k_group_dense, fill the GPU with a warp each.)
template <int NT, typename TI, typename TO>
__global__ void __launch_bounds__(NT < 128 ? 128 : NT)
k_dense_matvec(int n, const double *__restrict__ W, const TI *__restrict__ b,
               TO *__restrict__ x) {
  pdl_begin();
  __shared__ double red[8];
  const int t = threadIdx.x & (NT - 1);
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) / NT;
  if (row >= n) return;                          // whole groups: a block is one row where NT > 32
  const double *w = W + (size_t)row * n;
  double s = 0.0;
  for (int j0 = t; j0 < n; j0 += 8 * NT) {
    double wv[8], bv[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int j = j0 + u * NT;
      wv[u] = j < n ? __ldg(w + j) : 0.0;
      bv[u] = j < n ? (double)__ldg(b + j) : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (j0 + u * NT < n) s = fma(wv[u], bv[u], s);
  }
  s = warp_sum(s);
  if (NT > 32) {
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (t == 0) {
#pragma unroll
      for (int k = 1; k < NT / 32; ++k) s += red[k];
    }
  }
  if (t == 0) x[row] = (TO)s;
}

template <typename TI, typename TO>
void dense_matvec(int n, const double *W, const TI *b, TO *x, cudaStream_t st) {
  if (n <= 256)
    launch_pdl(k_dense_matvec<32, TI, TO>, ceil_div(n, 4), 128, st, n, W, b, x);
  else if (n <= 1024)
    launch_pdl(k_dense_matvec<128, TI, TO>, n, 128, st, n, W, b, x);
  else
    launch_pdl(k_dense_matvec<256, TI, TO>, n, 256, st, n, W, b, x);
  CHRONOS_CHECK_LAUNCH();
}
template void dense_matvec<float, float>(int, const double *, const float *, float *, cudaStream_t);
template void dense_matvec<double, double>(int, const double *, const double *, double *, cudaStream_t);

// =============================================================================
// Vector helpers
// =============================================================================

__global__ void k_f64_to_f32(int64_t n, const double *s, float *d) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < n;
       k += (int64_t)gridDim.x * blockDim.x)
    d[k] = (float)s[k];
}

void convert_f64_to_f32(int64_t n, const double *src, float *dst, cudaStream_t st) {
  if (n <= 0) return;
  k_f64_to_f32<<<std::min<int64_t>(ceil_div(n, 256), 4096), 256, 0, st>>>(n, src, dst);
  CHRONOS_CHECK_LAUNCH();
}

// =============================================================================
// CSR layouts on the device: transpose, 16-bit column offsets
// =============================================================================

__global__ void k_row_ids(int n, const int *__restrict__ rp, int *__restrict__ rid) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    for (int k = rp[i]; k < rp[i + 1]; ++k) rid[k] = i;
}

__global__ void k_col_count(int nnz, const int *__restrict__ ci, int *__restrict__ cnt) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nnz; k += gridDim.x * blockDim.x)
    atomicAdd(cnt + ci[k], 1);
}

__global__ void k_iota(int n, int *__restrict__ a) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) a[k] = k;
}

__global__ void k_transpose_fill(int nnz, const int *__restrict__ perm, const int *__restrict__ rid,
                                 const double *__restrict__ v, int *__restrict__ tci,
                                 double *__restrict__ tv) {
  for (int d = blockIdx.x * blockDim.x + threadIdx.x; d < nnz; d += gridDim.x * blockDim.x) {
    const int k = perm[d];
    tci[d] = rid[k];
    tv[d] = v[k];
  }
}

// Entry k of row i lands in row ci[k] of the transpose; a stable radix sort
// of the row-major entries by column keeps each transposed row in ascending
// order of i (then of k), which is the order the host transpose fills.
void csr_transpose_device(int nrows, int ncols, int64_t nnz64, const int *rp, const int *ci,
                          const double *v, DBuf<int> &trp, DBuf<int> &tci, DBuf<double> &tv,
                          cudaStream_t st) {
  CHRONOS_REQUIRE(nnz64 < INT32_MAX, CHRONOS_ENOTSUP, "matrix with 2^31 or more entries");
  const int nnz = (int)nnz64;
  trp.alloc((size_t)ncols + 1);
  tci.alloc(std::max(nnz, 1));
  tv.alloc(std::max(nnz, 1));
  DBuf<int> cnt((size_t)ncols + 1);
  cnt.zero(st);
  const int grid = std::max(1, std::min<int>(ceil_div(std::max(nnz, 1), 256), num_sms() * 16));
  if (nnz > 0) {
    k_col_count<<<grid, 256, 0, st>>>(nnz, ci, cnt.get());
    CHRONOS_CHECK_LAUNCH();
  }
  size_t bytes = 0;
  CHRONOS_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, bytes, cnt.get(), trp.get(), ncols + 1, st));
  {
    DBuf<unsigned char> tmp(std::max<size_t>(bytes, 1));
    CHRONOS_CUDA(cub::DeviceScan::ExclusiveSum(tmp.get(), bytes, cnt.get(), trp.get(), ncols + 1,
                                               st));
    CHRONOS_CUDA(cudaStreamSynchronize(st));
  }
  if (nnz == 0) return;
  DBuf<int> rid(nnz), idx(nnz), perm(nnz), keys(nnz);
  k_row_ids<<<std::max(1, std::min<int>(ceil_div(std::max(nrows, 1), 256), num_sms() * 16)), 256,
              0, st>>>(nrows, rp, rid.get());
  CHRONOS_CHECK_LAUNCH();
  k_iota<<<grid, 256, 0, st>>>(nnz, idx.get());
  CHRONOS_CHECK_LAUNCH();
  int end_bit = 1;
  while (end_bit < 31 && (1LL << end_bit) < (long long)ncols) ++end_bit;
  bytes = 0;
  CHRONOS_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, bytes, ci, keys.get(), idx.get(),
                                               perm.get(), nnz, 0, end_bit, st));
  {
    DBuf<unsigned char> tmp(std::max<size_t>(bytes, 1));
    CHRONOS_CUDA(cub::DeviceRadixSort::SortPairs(tmp.get(), bytes, ci, keys.get(), idx.get(),
                                                 perm.get(), nnz, 0, end_bit, st));
    k_transpose_fill<<<grid, 256, 0, st>>>(nnz, perm.get(), rid.get(), v, tci.get(), tv.get());
    CHRONOS_CHECK_LAUNCH();
    CHRONOS_CUDA(cudaStreamSynchronize(st));
  }
}

// A warp per row, coalesced along the columns.
__global__ void __launch_bounds__(256)
k_csr_check(int n, int ncols, const int *__restrict__ rp, const int *__restrict__ ci, int *bad) {
  const int lane = threadIdx.x & 31;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  int f = 0;
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += nw) {
    const int s = rp[i], e = rp[i + 1];
    for (int k = s + lane; k < e; k += 32) {
      const int c = ci[k];
      if (c < 0 || c >= ncols) f |= 1;
      if (k > s && ci[k - 1] >= c) f |= 2;
    }
  }
  if (f) atomicOr(bad, f);
}

int csr_check_device(int nrows, int ncols, const int *rp, const int *ci, cudaStream_t st) {
  DBuf<int> bad(1);
  bad.zero(st);
  k_csr_check<<<std::max(1, std::min<int>(ceil_div(nrows, 8), num_sms() * 16)), 256, 0, st>>>(
      nrows, ncols, rp, ci, bad.get());
  CHRONOS_CHECK_LAUNCH();
  int h = 0;
  CHRONOS_CUDA(cudaMemcpyAsync(&h, bad.get(), sizeof(int), cudaMemcpyDeviceToHost, st));
  CHRONOS_CUDA(cudaStreamSynchronize(st));
  return h;
}

__global__ void k_row_span(int n, const int *__restrict__ rp, const int *__restrict__ ci,
                           int *__restrict__ base, int *__restrict__ wide) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int s = rp[i], e = rp[i + 1];
    int lo = 0;
    if (e > s) {
      lo = ci[s];
      int hi = lo;
      for (int k = s + 1; k < e; ++k) {
        lo = min(lo, ci[k]);
        hi = max(hi, ci[k]);
      }
      if (hi - lo > 0xffff) atomicOr(wide, 1);
    }
    base[i] = lo;
  }
}

__global__ void k_col_offsets16(int n, const int *__restrict__ rp, const int *__restrict__ ci,
                                const int *__restrict__ base, uint16_t *__restrict__ off) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    for (int k = rp[i]; k < rp[i + 1]; ++k) off[k] = (uint16_t)(ci[k] - base[i]);
}

bool csr_offsets16_device(int nrows, int64_t nnz, const int *rp, const int *ci, DBuf<int> &base,
                          DBuf<uint16_t> &off, cudaStream_t st) {
  if (nrows <= 0) return false;
  base.alloc(nrows);
  DBuf<int> wide(1);
  wide.zero(st);
  const int grid = std::max(1, std::min<int>(ceil_div(nrows, 256), num_sms() * 16));
  k_row_span<<<grid, 256, 0, st>>>(nrows, rp, ci, base.get(), wide.get());
  CHRONOS_CHECK_LAUNCH();
  int w = 0;
  CHRONOS_CUDA(cudaMemcpyAsync(&w, wide.get(), sizeof(int), cudaMemcpyDeviceToHost, st));
  CHRONOS_CUDA(cudaStreamSynchronize(st));
  if (w) {
    base.release();
    return false;
  }
  off.alloc(std::max<int64_t>(nnz, 1));
  k_col_offsets16<<<grid, 256, 0, st>>>(nrows, rp, ci, base.get(), off.get());
  CHRONOS_CHECK_LAUNCH();
  return true;
}

__global__ void k_dot_partial(int n, const double *a, const double *b, double *part) {
  __shared__ double red[32];
  double s = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    s += a[i] * b[i];
  s = block_sum(s, red);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

double device_dot(int n, const double *a, const double *b, double *scratch, cudaStream_t st) {
  const int blocks = 256;
  k_dot_partial<<<blocks, 256, 0, st>>>(n, a, b, scratch);
  CHRONOS_CHECK_LAUNCH();
  double h[256];
  CHRONOS_CUDA(cudaMemcpyAsync(h, scratch, sizeof(h), cudaMemcpyDeviceToHost, st));
  CHRONOS_CUDA(cudaStreamSynchronize(st));
  double s = 0.0;
  for (int i = 0; i < blocks; ++i) s += h[i];
  return s;
}

__global__ void k_axpby(int n, double a, const double *x, double b, double *y) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    y[i] = a * x[i] + b * y[i];
}

void device_axpby(int n, double a, const double *x, double b, double *y, cudaStream_t st) {
  k_axpby<<<std::min<int64_t>(ceil_div(n, 256), 4096), 256, 0, st>>>(n, a, x, b, y);
  CHRONOS_CHECK_LAUNCH();
}

__global__ void k_scale_copy(int n, double a, const double *x, double *y) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    y[i] = a * x[i];
}

void device_scale_copy(int n, double a, const double *x, double *y, cudaStream_t st) {
  k_scale_copy<<<std::min<int64_t>(ceil_div(n, 256), 4096), 256, 0, st>>>(n, a, x, y);
  CHRONOS_CHECK_LAUNCH();
}

__global__ void k_diag_mul(int n, const double *d, const double *x, double *y) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    y[i] = d[i] * x[i];
}

void device_diag_mul(int n, const double *d, const double *x, double *y, cudaStream_t st) {
  k_diag_mul<<<std::min<int64_t>(ceil_div(n, 256), 4096), 256, 0, st>>>(n, d, x, y);
  CHRONOS_CHECK_LAUNCH();
}

// One warp per row: grad[k] = -lambda_i * u_{col(k)} over the row's entries.
__global__ void k_adjoint_scatter(int n, const int *rp, const int *ci, const double *lam,
                                  const double *u, double *grad) {
  const int lane = threadIdx.x & 31;
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (row >= n) return;
  const double li = -lam[row];
  for (int k = rp[row] + lane; k < rp[row + 1]; k += 32) grad[k] = li * u[ci[k]];
}

void adjoint_scatter(int n, const int *rp, const int *ci, const double *lambda, const double *u,
                     double *grad, cudaStream_t st) {
  if (n <= 0) return;
  k_adjoint_scatter<<<ceil_div((int64_t)n * 32, 256), 256, 0, st>>>(n, rp, ci, lambda, u, grad);
  CHRONOS_CHECK_LAUNCH();
}

// =============================================================================
// FSAI numeric phase without allocation (chronos_fsai_numeric_noalloc)
// =============================================================================
//
// Same kernels as fsai_numeric_device, but the scratch they need -- the
// row-bucket lists and the flag word -- lives in one file-scope device array
// instead of cudaMalloc'd buffers.  The array is a fixed 12 MiB + 256 B per
// device that loads the library, held until the process exits.  Every call
// shares it: calls that overlap on the GPU (two streams, two host threads)
// race on it and must be serialised by the caller.

constexpr int kNoAllocMaxRows = 1 << 20;
constexpr int kNoAllocHeader = 64;            // ints: [0..4] bucket counts, [5] flags
static __device__ __align__(256) int g_fsai_noalloc_scratch[kNoAllocHeader + 3 * kNoAllocMaxRows];

// In host code g_fsai_noalloc_scratch names a host-side stand-in, not a device
// address: the device address is looked up once per device with
// cudaGetSymbolAddress (with that device current) and cached here.
static int *g_noalloc_addr[64] = {nullptr};
static std::mutex g_noalloc_mu;

static int *noalloc_scratch_address() {
  int dev = 0;
  CHRONOS_CUDA(cudaGetDevice(&dev));
  CHRONOS_REQUIRE(dev >= 0 && dev < 64, CHRONOS_EINVAL, "device ordinal out of range");
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_addr[dev]) {
    void *p = nullptr;
    CHRONOS_CUDA(cudaGetSymbolAddress(&p, g_fsai_noalloc_scratch));
    g_noalloc_addr[dev] = static_cast<int *>(p);
  }
  return g_noalloc_addr[dev];
}

// Place of entry pos of bucket b: three lists of kNoAllocMaxRows ints; buckets
// 3 and 4 fill the first two from their ends (the buckets hold n <=
// kNoAllocMaxRows rows together, so they never meet).
__host__ __device__ constexpr int noalloc_slot(int b, int pos) {
  return kNoAllocHeader + (b < 3 ? b * kNoAllocMaxRows + pos
                                 : (b - 2) * kNoAllocMaxRows - 1 - pos);
}

// Checks row i of both patterns and sorts it into the buckets of
// fsai_numeric_device.  The numeric kernel indexes A's rows by G's columns and
// writes G's row at gval[grp[i] .. grp[i+1]-1] with the diagonal last, so a
// malformed row sets flag bit 2 (and is not bucketed): a G row without
// entries, a last column other than i, strictly-lower columns not ascending
// or outside [0, i); an A row whose pointers decrease or whose columns are not
// ascending inside [0, n); row pointers of either that do not start at 0.
// A row longer than 64 strictly-lower entries sets flag bit 1.
// A warp's rows of one bucket take their places with one atomic: an atomic
// per row on five counters was the whole time of this kernel (227k rows:
// 155 us).
__global__ void __launch_bounds__(256)
k_fsai_bucket_rows(int n, const int *__restrict__ arp, const int *__restrict__ aci,
                   const int *__restrict__ grp, const int *__restrict__ gci, int *scratch) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  int b = -1, flag = 0;
  if (i < n) {
    const int gs = grp[i], ge = grp[i + 1];
    bool bad = ge <= gs || (i == 0 && (gs != 0 || arp[0] != 0));
    if (!bad) {
      bad = gci[ge - 1] != i;
      for (int k = gs, prev = -1; !bad && k < ge - 1; ++k) {
        const int c = gci[k];
        bad = c <= prev || c >= i;
        prev = c;
      }
    }
    const int as = arp[i], ae = arp[i + 1];
    bad = bad || ae < as;
    for (int k = as, prev = -1; !bad && k < ae; ++k) {
      const int c = aci[k];
      bad = c <= prev || c >= n;
      prev = c;
    }
    const int m = ge - gs - 1;
    if (bad) flag = 4;
    else if (m > 64) flag = 2;
    else b = fsai_bucket(m);
  }
  if (flag) atomicOr(scratch + kFsaiBuckets, flag);
#pragma unroll
  for (int q = 0; q < kFsaiBuckets; ++q) {
    const unsigned in = __ballot_sync(0xffffffffu, b == q);
    if (!in) continue;
    int base = 0;
    if (lane == __ffs(in) - 1) base = atomicAdd(scratch + q, __popc(in));
    base = __shfl_sync(0xffffffffu, base, __ffs(in) - 1);
    if (b == q) scratch[noalloc_slot(q, base + __popc(in & ((1u << lane) - 1u)))] = i;
  }
}

int fsai_numeric_noalloc(int n, const int *arp, const int *aci, const double *av, const int *grp,
                         const int *gci, double *gval, cudaStream_t st) {
  CHRONOS_REQUIRE(n > 0 && n <= kNoAllocMaxRows, CHRONOS_EINVAL,
                  "chronos_fsai_numeric_noalloc: n must be in [1, 1048576] (its static scratch "
                  "holds 1048576 rows)");
  int *scr = noalloc_scratch_address();
  // the previous call's contents remain: clear the counts and the flag word
  CHRONOS_CUDA(cudaMemsetAsync(scr, 0, kNoAllocHeader * sizeof(int), st));
  k_fsai_bucket_rows<<<ceil_div(n, 256), 256, 0, st>>>(n, arp, aci, grp, gci, scr);
  CHRONOS_CHECK_LAUNCH();
  int hdr[kFsaiBuckets + 1] = {};
  CHRONOS_CUDA(cudaMemcpyAsync(hdr, scr, sizeof(hdr), cudaMemcpyDeviceToHost, st));
  CHRONOS_CUDA(cudaStreamSynchronize(st));
  // no numeric kernel runs on a malformed pattern: it would read A and write
  // G's values outside the rows the caller's buffers hold
  CHRONOS_REQUIRE(!(hdr[kFsaiBuckets] & 4), CHRONOS_EINVAL,
                  "malformed CSR: a G row is empty, does not end with its diagonal or has "
                  "strictly-lower columns not ascending in [0, i); or A's row pointers / "
                  "columns are not a sorted 0-based CSR");
  CHRONOS_REQUIRE(!(hdr[kFsaiBuckets] & 2), CHRONOS_ENOTSUP,
                  "FSAI local system larger than 64 (nstep*step_size)");
  for (int b = 0; b < kFsaiBuckets; ++b)       // a list from the end: its lowest address
    launch_fsai_bucket(b, hdr[b], scr + (b < 3 ? noalloc_slot(b, 0) : noalloc_slot(b, hdr[b] - 1)),
                       arp, aci, av, grp, gci, gval, scr + kFsaiBuckets, st);
  int fl = 0;
  CHRONOS_CUDA(cudaMemcpyAsync(&fl, scr + kFsaiBuckets, sizeof(int), cudaMemcpyDeviceToHost, st));
  CHRONOS_CUDA(cudaStreamSynchronize(st));
  return fl;
}

}  // namespace chronos

extern "C" int chronos_fsai_numeric_noalloc(int n, const int *iat_A_d, const int *ja_A_d,
                                            const double *val_A_d, const int *iat_G_d,
                                            const int *ja_G_d, double *val_G_d, int *is_posdef,
                                            void *stream) {
  try {
    CHRONOS_REQUIRE(iat_A_d && ja_A_d && val_A_d && iat_G_d && ja_G_d && val_G_d && is_posdef,
                    CHRONOS_EINVAL, "null argument");
    const int fl = chronos::fsai_numeric_noalloc(n, iat_A_d, ja_A_d, val_A_d, iat_G_d, ja_G_d,
                                                 val_G_d, static_cast<cudaStream_t>(stream));
    *is_posdef = (fl & 1) ? 0 : 1;
    return CHRONOS_OK;
  } catch (const chronos::Error &e) {
    chronos::set_last_error(e.what());
    return e.code;
  } catch (const std::exception &e) {
    chronos::set_last_error(e.what());
    return CHRONOS_EINVAL;
  }
}
