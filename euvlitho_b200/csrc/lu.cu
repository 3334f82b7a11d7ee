// Batched complex FP64 LU with partial pivoting and triangular solves.
//
// Replaces matinv (header.h:1468-1557: Eigen colPivHouseholderQr for N<=5000,
// cuSOLVER Xgetrf/Xgetrs with host round trips above).  The reference only ever
// applies an inverse to a matrix, so the library factors once and solves with
// the right-hand sides it needs.
//
// Blocked right-looking LU, panel width LU_NB:
//   panel  : columns [j0, j0+nb) of rows [j0, n) (pivot = first max of
//            |re|+|im| as LAPACK izamax, row swap, scale, rank-1 update), the
//            rows in the registers of a cluster of up to 16 CTAs per matrix;
//   laswp  : the panel's row swaps applied to the other columns;
//   trsm   : U12 = L11^-1 A12 (unit lower, L11 staged in shared memory);
//   update : A22 -= L21 U12 with the batched DMMA zgemm;
//   look-ahead: the next panel is factored on a high-priority side stream while
//            the rest of the update runs (the panel alone fills only `batch` SMs).
// Solve: the row swaps on B, then one launch that keeps 8 or 12 columns of X in
// shared memory per CTA through both substitutions, or blocks of 32 rows (two
// launches each) where fewer columns fit.
#include <cooperative_groups.h>

#include "common.cuh"

namespace euv {

namespace cg = cooperative_groups;

int zgemm_sub(int m, int n, int k, const double2* a, long long lda, long long sa,
              const double2* b, long long ldb, long long sb, double2* c, long long ldc,
              long long sc, int batch, cudaStream_t stream, const Slots& slots = Slots{});
int zgemm(int m, int n, int k, cplx alpha, const double* scale, const double2* a, long long lda,
          long long sa, const double2* b, long long ldb, long long sb, cplx beta, double2* c,
          long long ldc, long long sc, cplx diag, int batch, const int* steps, int step,
          cudaStream_t stream, const GemmTerms& terms = GemmTerms{});

constexpr int LU_NB = 32;
constexpr int LU_PANEL_THREADS = 512;

__device__ __forceinline__ cplx ld2(const double2* p) {
  double2 v = *p;
  return mk(v.x, v.y);
}
__device__ __forceinline__ void st2(double2* p, cplx v) { *p = make_double2(v.x, v.y); }

__global__ void __launch_bounds__(LU_PANEL_THREADS) lu_panel_kernel(int n, int j0, int jb,
                                                                    double2* A, long long lda,
                                                                    long long sa, int* ipiv,
                                                                    int* info) {
  A += (long long)blockIdx.x * sa;
  ipiv += (long long)blockIdx.x * n;
  __shared__ double red_v[LU_PANEL_THREADS / 32];
  __shared__ int red_i[LU_PANEL_THREADS / 32];
  __shared__ int s_piv;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nthr = blockDim.x;
  for (int jj = j0; jj < j0 + jb; ++jj) {
    // pivot search: first index of max |re|+|im| in rows jj..n-1
    double best = -1.0;
    int bidx = n;
    for (int r = jj + tid; r < n; r += nthr) {
      double v = cabs1(ld2(&A[r + (long long)jj * lda]));
      if (v > best) {
        best = v;
        bidx = r;
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      double ov = __shfl_down_sync(0xffffffffu, best, off);
      int oi = __shfl_down_sync(0xffffffffu, bidx, off);
      if (ov > best || (ov == best && oi < bidx)) {
        best = ov;
        bidx = oi;
      }
    }
    if (lane == 0) {
      red_v[warp] = best;
      red_i[warp] = bidx;
    }
    __syncthreads();
    if (tid == 0) {
      double bv = red_v[0];
      int bi = red_i[0];
      for (int w = 1; w < nthr / 32; ++w) {
        if (red_v[w] > bv || (red_v[w] == bv && red_i[w] < bi)) {
          bv = red_v[w];
          bi = red_i[w];
        }
      }
      if (bi >= n) bi = jj;
      s_piv = bi;
      ipiv[jj] = bi;
    }
    __syncthreads();
    const int piv = s_piv;
    if (piv != jj) {
      for (int c = j0 + tid; c < j0 + jb; c += nthr) {
        double2 t = A[jj + (long long)c * lda];
        A[jj + (long long)c * lda] = A[piv + (long long)c * lda];
        A[piv + (long long)c * lda] = t;
      }
    }
    __syncthreads();
    const cplx d = ld2(&A[jj + (long long)jj * lda]);
    if (d.x == 0.0 && d.y == 0.0) {
      if (tid == 0 && info[blockIdx.x] == 0) info[blockIdx.x] = jj + 1;
      __syncthreads();
      continue;
    }
    const cplx inv = cdiv(mk(1.0, 0.0), d);
    for (int r = jj + 1 + tid; r < n; r += nthr) {
      double2* p = &A[r + (long long)jj * lda];
      st2(p, ld2(p) * inv);
    }
    __syncthreads();
    const int rows = n - jj - 1;
    const int cols = j0 + jb - jj - 1;
    if (rows > 0 && cols > 0) {
      for (int idx = tid; idx < rows * cols; idx += nthr) {
        int r = jj + 1 + idx % rows;
        int c = jj + 1 + idx / rows;
        double2* p = &A[r + (long long)c * lda];
        st2(p, ld2(p) - ld2(&A[r + (long long)jj * lda]) * ld2(&A[jj + (long long)c * lda]));
      }
    }
    __syncthreads();
  }
}

// Panel factorisation by a cluster of LC CTAs per matrix with the panel rows
// in registers (n - j0 <= LC * LC_THREADS rows): thread t of cluster rank q
// holds row j0 + q*LC_THREADS + t.  Columns are taken in blocks of LC_BLK
// with the block's columns at compile-time register indices v[0..LC_BLK); the
// register row is rotated by LC_BLK after each block (one block's code for the
// whole panel, no runtime register indexing).  One cluster barrier per column
// jj (a block barrier for one CTA): before it, every CTA finds its candidate (first
// max of |re|+|im| in its rows >= jj, a NaN as zero; every warp reduces the warp maxima
// itself) and sends
// the candidate's value, index and row to every CTA through distributed shared
// memory, one column per lane of the warp that holds the row, and rank 0 sends
// row jj the same way; after it, every thread reduces the LC candidates in
// rank order (same pivot in every CTA), takes the pivot row from the winner's
// slot, swaps, scales and applies the rank-1 update to its own row.  The swap
// at column jj exchanges only the columns from jj on (the part of the two rows
// the remaining columns use), so every column c of the panel holds the swaps of
// pivots ..c and lacks exactly those of pivots c+1..: the laswp launch after the
// panel applies them (sub = 1).  Slots alternate by column parity: a slot is
// rewritten two barriers after it was read.  A block's columns are stored when
// it ends, pivots and the singular flag when the panel ends.  Every thread
// executes every barrier the same number of times whatever the data (a zero
// pivot skips only the arithmetic).
constexpr int LC_THREADS = 256;
constexpr int LC_WARPS = LC_THREADS / 32;
constexpr int LC_BLK = 4;
static_assert(LU_NB == 32, "one panel column per lane");
static_assert(LU_NB % LC_BLK == 0, "whole blocks");

// A panel column costs about 1.5 us at 256 rows (1.8 before the three reductions in
// hardware, the reciprocal with one division and the search under the update); what
// is left is a chain of two barriers, the reductions, the division and 31 updates of
// a row by every thread.
// Candidates compare as the bits of |re|+|im| (order of non-negative doubles), ties
// to the smallest row: three warp reductions in hardware.  A NaN compares as zero, so
// that it is no pivot beside a number, as in lu_panel_kernel.  Lanes without a row hold
// key 0 and row n.
struct Cand {
  unsigned long long key;
  int row;
};
__device__ __forceinline__ Cand warp_argmax(unsigned long long key, int row) {
  const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
  const int r = __reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? row : 0x7fffffff);
  return Cand{((unsigned long long)mh << 32) | ml, r};
}
__device__ __forceinline__ unsigned long long abs_key(cplx v) {
  const double a = cabs1(v);
  return __double2hiint(a) > 0x7ff00000 ? 0ull : (unsigned long long)__double_as_longlong(a);
}

// 1 / d: one real division, d scaled by a power of two so that |d|^2 neither
// over- nor underflows (the exponents at the ends of the range divide as cdiv)
__device__ __forceinline__ cplx crecip(cplx d) {
  const double m = fmax(fabs(d.x), fabs(d.y));
  const int e = (__double2hiint(m) >> 20) & 0x7ff;
  if (e < 2 || e > 2044) return cdiv(mk(1.0, 0.0), d);
  const double s = __hiloint2double((2046 - e) << 20, 0);
  const double x = d.x * s, y = d.y * s;
  const double r = s / (x * x + y * y);
  return mk(x * r, -y * r);
}

template <int LC>
__global__ void __launch_bounds__(LC_THREADS, 1)
    lu_panel_cluster_kernel(int n, int j0, int jb, double2* A, long long lda, long long sa,
                            int* ipiv, int* info) {
  dependent_begin();
  cg::cluster_group cluster = cg::this_cluster();
  const int q = LC == 1 ? 0 : (int)cluster.block_rank();
  const int mat = blockIdx.x / LC;
  A += (long long)mat * sa;
  ipiv += (long long)mat * n;
  __shared__ unsigned long long s_wk[LU_NB][LC_WARPS];
  __shared__ int s_wi[LU_NB][LC_WARPS];
  __shared__ unsigned long long s_ck[LU_NB][LC];
  __shared__ int s_ci[LU_NB][LC];
  __shared__ double2 s_crow[2][LC][LU_NB];  // candidate rows, by rank
  __shared__ double2 s_rjj[2][LU_NB];       // row jj
  __shared__ int s_piv[LU_NB];
  int zero_col = 0;  // first zero pivot + 1
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r = j0 + q * LC_THREADS + tid;
  const bool own = r < n;
  cplx v[LU_NB];
#pragma unroll
  for (int k = 0; k < LU_NB; ++k)
    v[k] = (own && k < jb) ? ld2(&A[r + (long long)(j0 + k) * lda]) : mk(0.0, 0.0);
  // this warp's candidate of the first column; later ones are found as soon as
  // their column is updated, under the rest of the rank-1 update
  Cand w = warp_argmax(own ? abs_key(v[0]) : 0ull, own ? r : n);
#pragma unroll 1
  for (int c0 = 0; c0 < jb; c0 += LC_BLK) {  // jb is the same for every thread
#pragma unroll
    for (int i = 0; i < LC_BLK; ++i) {
      const int c = c0 + i;
      if (c >= jb) break;
      const int jj = j0 + c, buf = c & 1;
      if (lane == 0) {
        s_wk[c][warp] = w.key;
        s_wi[c][warp] = w.row;
      }
      __syncthreads();
      {
        const Cand b = warp_argmax(lane < LC_WARPS ? s_wk[c][lane] : 0ull,
                                   lane < LC_WARPS ? s_wi[c][lane] : n);
        const int bi = b.row;
        if (bi < n && (bi - j0 - q * LC_THREADS) >> 5 == warp) {
          if (r == bi)
#pragma unroll
            for (int k = i; k < LU_NB; ++k) s_crow[buf][q][k] = make_double2(v[k].x, v[k].y);
          __syncwarp();
          if (LC > 1 && lane >= i) {
            const double2 x = s_crow[buf][q][lane];
#pragma unroll
            for (int t = 0; t < LC; ++t)
              if (t != q) *cluster.map_shared_rank(&s_crow[buf][q][lane], t) = x;
          }
        }
        if (warp == 0 && lane < LC) {
          if (LC == 1) {
            s_ck[c][0] = b.key;
            s_ci[c][0] = bi;
          } else {
            *cluster.map_shared_rank(&s_ck[c][q], lane) = b.key;
            *cluster.map_shared_rank(&s_ci[c][q], lane) = bi;
          }
        }
      }
      if (q == 0 && warp == 0) {
        if (lane == c)
#pragma unroll
          for (int k = i; k < LU_NB; ++k) s_rjj[buf][k] = make_double2(v[k].x, v[k].y);
        __syncwarp();
        if (LC > 1 && lane >= i) {
          const double2 x = s_rjj[buf][lane];
#pragma unroll
          for (int t = 1; t < LC; ++t) *cluster.map_shared_rank(&s_rjj[buf][lane], t) = x;
        }
      }
      if (LC == 1)
        __syncthreads();
      else
        cluster.sync();
      unsigned long long bk = s_ck[c][0];
      int bi = s_ci[c][0], qw = 0;
#pragma unroll
      for (int t = 1; t < LC; ++t) {
        const unsigned long long ok = s_ck[c][t];
        const int oi = s_ci[c][t];
        if (ok > bk || (ok == bk && oi < bi)) {
          bk = ok;
          bi = oi;
          qw = t;
        }
      }
      const int piv = (bi < jj || bi >= n) ? jj : bi;
      if (tid == 0) s_piv[c] = piv;
      const double2* prow = piv == jj ? s_rjj[buf] : s_crow[buf][qw];
      if (own && piv != jj && (r == jj || r == piv)) {
        const double2* src = r == jj ? prow : s_rjj[buf];
#pragma unroll
        for (int k = i; k < LU_NB; ++k) v[k] = mk(src[k].x, src[k].y);
      }
      const double2 dd = prow[i];
      const bool zero = dd.x == 0.0 && dd.y == 0.0;
      if (zero && zero_col == 0) zero_col = jj + 1;
      const bool below = own && r > jj;
      cplx l = mk(0.0, 0.0);
      if (!zero && below) {
        l = v[i] * crecip(mk(dd.x, dd.y));
        v[i] = l;
      }
      // column c + 1 first: its candidates are sought while the others are updated
      if (i + 1 < LU_NB) {
        if (!zero && below) v[i + 1] = v[i + 1] - l * mk(prow[i + 1].x, prow[i + 1].y);
        w = warp_argmax(below ? abs_key(v[i + 1]) : 0ull, below ? r : n);
      }
      if (!zero && below) {
        // columns c+2 .. jb-1 are v[i+2 .. jb-1-c0]; blocks of 8 past them are skipped
#pragma unroll
        for (int k0 = 0; k0 < LU_NB; k0 += 8) {
          if (k0 + 8 > i + 2 && k0 < jb - c0) {
#pragma unroll
            for (int k = k0; k < k0 + 8; ++k)
              if (k > i + 1) v[k] = v[k] - l * mk(prow[k].x, prow[k].y);
          }
        }
      }
    }
    if (own)
#pragma unroll
      for (int i = 0; i < LC_BLK; ++i)
        if (c0 + i < jb) st2(&A[r + (long long)(j0 + c0 + i) * lda], v[i]);
#pragma unroll
    for (int k = 0; k < LU_NB; ++k) v[k] = k + LC_BLK < LU_NB ? v[k + LC_BLK] : mk(0.0, 0.0);
  }
  __syncthreads();
  if (q == 0) {
    if (tid < jb) ipiv[j0 + tid] = s_piv[tid];
    if (tid == 0 && zero_col != 0 && info[mat] == 0) info[mat] = zero_col;
  }
}

// behind: a launch like launch_dependent's
template <int LC>
static void panel_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, int batch,
                         cudaStream_t st, bool behind = false) {
  cfg = {};
  cfg.gridDim = dim3(LC * batch);
  cfg.blockDim = dim3(LC_THREADS);
  cfg.stream = st;
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = behind ? 1 : 0;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = LC;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = LC > 1 ? 2 : 1;
}

template <int LC>
static int launch_panel(int n, int j0, int jb, double2* A, long long lda, long long sa, int* ipiv,
                        int* info, int batch, cudaStream_t st, bool behind) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute at[2];
  panel_config<LC>(cfg, at, batch, st, behind);
  EUV_CUDA_TRY(cudaLaunchKernelEx(&cfg, lu_panel_cluster_kernel<LC>, n, j0, jb, A, lda, sa, ipiv,
                                  info));
  EUV_LAUNCH_CHECK();
  return EUV_OK;
}

// Whether this device runs clusters of 16 (beyond the portable size), asked once.
static bool panel16() {
  static int state[64];  // 0 unknown, 1 yes, 2 no
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  int st = __atomic_load_n(&state[dev], __ATOMIC_ACQUIRE);
  if (st == 0) {
    int clusters = 0;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[2];
    panel_config<16>(cfg, at, 1, nullptr);
    const bool ok = cudaFuncSetAttribute(lu_panel_cluster_kernel<16>,
                                         cudaFuncAttributeNonPortableClusterSizeAllowed,
                                         1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&clusters, lu_panel_cluster_kernel<16>, &cfg) ==
                        cudaSuccess &&
                    clusters > 0;
    if (!ok) (void)cudaGetLastError();
    st = ok ? 1 : 2;
    __atomic_store_n(&state[dev], st, __ATOMIC_RELEASE);
  }
  return st == 1;
}

// Row swaps ipiv[j0..j0+jb) applied to every column outside [skip0, skip1).
// Columns in [skip0, skip1) (the panel's own) are skipped when sub == 0; with
// sub > 0 the panel was factored sub columns at a time and already applied to
// each of its columns the swaps up to the end of that column's sub-panel, so
// only the later ones remain.
__global__ void lu_laswp_kernel(int n, int ncols, int j0, int jb, int skip0, int skip1,
                                double2* A, long long lda, long long sa, const int* ipiv,
                                long long ipiv_stride, int sub) {
  dependent_begin();
  const int b = blockIdx.y;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncols) return;
  int first = j0;
  if (c >= skip0 && c < skip1) {
    if (sub <= 0) return;
    first = skip0 + ((c - skip0) / sub + 1) * sub;
  }
  A += (long long)b * sa;
  ipiv += (long long)b * ipiv_stride;
  for (int jj = first; jj < j0 + jb; ++jj) {
    int p = ipiv[jj];
    if (p != jj) {
      double2 t = A[jj + (long long)c * lda];
      A[jj + (long long)c * lda] = A[p + (long long)c * lda];
      A[p + (long long)c * lda] = t;
    }
  }
}

// X = T^-1 X for a jb x jb triangular block T of the factor (unit lower when
// lower != 0, non-unit upper otherwise) and the jb-row slab X of `ncols` columns,
// one warp per column, T staged in shared memory: lane r holds row r of X; step q
// broadcasts the finished x_q by shuffle and every later (lower) or earlier
// (upper) lane subtracts its term, so a column takes jb short steps instead of
// one thread's chain of jb^2/2 dependent products.  8 columns per CTA.
constexpr int LU_TRSM_WARPS = 8;
__global__ void __launch_bounds__(32 * LU_TRSM_WARPS)
    lu_trsm_warp_kernel(int jb, int ncols, int lower, const double2* T, long long ldt,
                        long long st, double2* X, long long ldx, long long sx, Slots slots) {
  dependent_begin();
  __shared__ double2 Ts[LU_NB][LU_NB + 1];
  const int b = blockIdx.y;
  const int lane = threadIdx.x & 31;
  const int col = blockIdx.x * LU_TRSM_WARPS + (threadIdx.x >> 5);
  const bool live = col < ncols && !slots.empty(b, col);  // warp-uniform
  T += (long long)b * st;
  X += (long long)b * sx;
  for (int idx = threadIdx.x; idx < jb * jb; idx += blockDim.x) {
    const int r = idx % jb, c = idx / jb;
    Ts[r][c] = T[r + (long long)c * ldt];
  }
  __syncthreads();
  if (!live) return;  // whole warps (the flag's load is under the staging's)
  double2* Xc = X + (long long)col * ldx;
  cplx x = lane < jb ? ld2(&Xc[lane]) : mk(0.0, 0.0);
  if (lower) {
    for (int q = 0; q < jb; ++q) {
      const cplx xq = mk(__shfl_sync(0xffffffffu, x.x, q), __shfl_sync(0xffffffffu, x.y, q));
      if (lane > q && lane < jb) x = x - mk(Ts[lane][q].x, Ts[lane][q].y) * xq;
    }
  } else {
    // each lane's reciprocal pivot, off the serial chain
    const cplx rinv = lane < jb ? crecip(mk(Ts[lane][lane].x, Ts[lane][lane].y)) : mk(0.0, 0.0);
    for (int q = jb - 1; q >= 0; --q) {
      if (lane == q) x = x * rinv;
      const cplx xq = mk(__shfl_sync(0xffffffffu, x.x, q), __shfl_sync(0xffffffffu, x.y, q));
      if (lane < q) x = x - mk(Ts[lane][q].x, Ts[lane][q].y) * xq;
    }
  }
  if (lane < jb) st2(&Xc[lane], x);
}

static inline dim3 trsm_grid(int ncols, int batch) {
  return dim3((ncols + LU_TRSM_WARPS - 1) / LU_TRSM_WARPS, batch);
}

__global__ void zero_int_kernel(int* p, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = 0;
}

// Side stream (highest priority) and fork/join events of the look-ahead, one
// set per host thread and device, created by the first call (which therefore
// has to come before any stream capture).
struct LuSide {
  cudaStream_t hi = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
};
static cudaError_t lu_side(LuSide** out) {
  static thread_local LuSide per_dev[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  LuSide& s = per_dev[dev];
  if (s.hi == nullptr) {
    int lo = 0, hi = 0;
    if ((e = cudaDeviceGetStreamPriorityRange(&lo, &hi)) != cudaSuccess) return e;
    if ((e = cudaStreamCreateWithPriority(&s.hi, cudaStreamNonBlocking, hi)) != cudaSuccess) return e;
    if ((e = cudaEventCreateWithFlags(&s.fork, cudaEventDisableTiming)) != cudaSuccess) return e;
    if ((e = cudaEventCreateWithFlags(&s.join, cudaEventDisableTiming)) != cudaSuccess) return e;
  }
  *out = &s;
  return cudaSuccess;
}

// Row-swap granularity the laswp after panel j0 applies to the panel's own
// columns: 1 after the cluster kernel (column c lacks the swaps of pivots
// c+1..), 0 after lu_panel_kernel (the panel's columns are complete).
static int panel_sub(int n, int j0) {
  return n - j0 <= 8 * LC_THREADS || (n - j0 <= 16 * LC_THREADS && panel16()) ? 1 : 0;
}

// CTAs of a trailing update up to which it runs before the next panel, on the same
// stream: one wave of four per SM.  Such an update is over by the time the look-ahead's
// events and its separate update of the panel's columns take (two units of N = 361
// 2.11 -> 2.06 ms per call, four of N = 121 0.52 -> 0.51); at twice as many the update's
// time shows (two units of N = 545 5.69 -> 5.74 ms).
constexpr int LU_ONE_WAVE = 4 * 148;
static int lu_panel(int n, int j0, int jb, double2* A, long long lda, long long sa, int* ipiv,
                    int* info, int batch, cudaStream_t st, bool behind) {
  const int rows = n - j0;
  // the tuning table may spread a panel's rows over more CTAs than they need
  const int lc_min = tune_lookup(EUV_KNOB_LU_CLUSTER, n, batch);
  if (rows <= LC_THREADS && lc_min <= 1)
    return launch_panel<1>(n, j0, jb, A, lda, sa, ipiv, info, batch, st, behind);
  if (rows <= 2 * LC_THREADS && lc_min <= 2)
    return launch_panel<2>(n, j0, jb, A, lda, sa, ipiv, info, batch, st, behind);
  if (rows <= 4 * LC_THREADS && lc_min <= 4)
    return launch_panel<4>(n, j0, jb, A, lda, sa, ipiv, info, batch, st, behind);
  if (rows <= 8 * LC_THREADS) return launch_panel<8>(n, j0, jb, A, lda, sa, ipiv, info, batch, st, behind);
  if (rows <= 16 * LC_THREADS && panel16())
    return launch_panel<16>(n, j0, jb, A, lda, sa, ipiv, info, batch, st, behind);
  lu_panel_kernel<<<batch, LU_PANEL_THREADS, 0, st>>>(n, j0, jb, A, lda, sa, ipiv, info);
  EUV_LAUNCH_CHECK();
  return EUV_OK;
}

// U12 = L11^-1 A12 and A22 -= L21 U12 of panel [j0, j0+jb) for the columns
// [c0, c0+nc) (rows j0.. of the factor).
static int lu_update(int n, int j0, int jb, int c0, int nc, double2* A, long long lda,
                     long long sa, int batch, cudaStream_t st, const Slots& slots) {
  if (nc <= 0) return EUV_OK;
  EUV_CUDA_TRY(launch_dependent(lu_trsm_warp_kernel, trsm_grid(nc, batch), dim3(32 * LU_TRSM_WARPS),
                                0, st, jb, nc, 1, A + j0 + (long long)j0 * lda, lda, sa,
                                A + j0 + (long long)c0 * lda, lda, sa, slots.from(c0)));
  EUV_LAUNCH_CHECK();
  const int rest = n - j0 - jb;
  if (rest <= 0) return EUV_OK;
  // (below 256 rows the look at the slots takes as long as the tiles that it saves)
  return zgemm_sub(rest, nc, jb, A + (j0 + jb) + (long long)j0 * lda, lda, sa,
                   A + j0 + (long long)c0 * lda, lda, sa, A + (j0 + jb) + (long long)c0 * lda,
                   lda, sa, batch, st, rest > 256 ? slots.from(c0) : Slots{});
}

// Right-looking LU with one panel of look-ahead: after panel j, its update of
// the next panel's columns runs first; then the next panel is factored on the
// high-priority side stream (its batch CTAs take SMs as soon as any frees up)
// while the update of the remaining columns runs on the caller's stream.  The
// column sets are disjoint; the laswp of the next panel waits for both.
// extra: columns n .. n + extra - 1 of A are right-hand sides, which every step
// swaps and updates with the trailing columns: they end as L^-1 P B (lu_back
// finishes them).  The forward substitution so rides in launches that are there
// anyway, most of it under the panel chain (B200, image calls, with the blocked
// backward pass above N = 1562: 2048 nm, eight slices, 61.7 -> 53.4 ms; M3D at N =
// 2121 44.0 -> 38.1 ms; 24 units of N = 625 6.50 -> 6.23 ms).  order: the source slots that
// those columns are; CTAs of empty ones only return (12 of 200 slots filled: four units of N
// = 1681 10.70 -> 10.36 ms, six of 961 5.05 -> 4.98).
int lu_factor(int n, double2* A, long long lda, long long sa, int* ipiv, int* info, int batch,
              cudaStream_t stream, int extra, const int* order, long long ostride) {
  if (n <= 0 || batch <= 0) return EUV_OK;
  const Slots slots{order, ostride, n};
  LuSide* side = nullptr;
  EUV_CUDA_TRY(lu_side(&side));
  zero_int_kernel<<<(batch + 255) / 256, 256, 0, stream>>>(info, batch);
  EUV_LAUNCH_CHECK();
  int j0 = 0, jb = n < LU_NB ? n : LU_NB;
  int rc = lu_panel(n, j0, jb, A, lda, sa, ipiv, info, batch, stream, true);
  if (rc) return rc;
  bool behind = true;  // the last panel ran on this stream
  for (;;) {
    dim3 gs((n + extra + 127) / 128, batch);
    if (behind) {
      EUV_CUDA_TRY(launch_dependent(lu_laswp_kernel, gs, dim3(128), 0, stream, n, n + extra, j0, jb,
                                    j0, j0 + jb, A, lda, sa, ipiv, n, panel_sub(n, j0)));
    } else {
      lu_laswp_kernel<<<gs, 128, 0, stream>>>(n, n + extra, j0, jb, j0, j0 + jb, A, lda, sa, ipiv, n,
                                              panel_sub(n, j0));
    }
    EUV_LAUNCH_CHECK();
    const int rest = n - j0 - jb;
    if (rest <= 0) {
      if ((rc = lu_update(n, j0, jb, n, extra, A, lda, sa, batch, stream, slots))) return rc;
      break;
    }
    const int j1 = j0 + jb, nb2 = rest < LU_NB ? rest : LU_NB, rem = rest - nb2 + extra;
    const long long ctas = (long long)((rest + 31) / 32) * ((nb2 + rem + 63) / 64) * batch;
    behind = rem <= 0 || ctas <= LU_ONE_WAVE;
    if (behind) {
      if ((rc = lu_update(n, j0, jb, j1, nb2 + rem, A, lda, sa, batch, stream, slots))) return rc;
      if ((rc = lu_panel(n, j1, nb2, A, lda, sa, ipiv, info, batch, stream, true))) return rc;
    } else {
      if ((rc = lu_update(n, j0, jb, j1, nb2, A, lda, sa, batch, stream, slots))) return rc;
      EUV_CUDA_TRY(cudaEventRecord(side->fork, stream));
      EUV_CUDA_TRY(cudaStreamWaitEvent(side->hi, side->fork, 0));
      if ((rc = lu_panel(n, j1, nb2, A, lda, sa, ipiv, info, batch, side->hi, false))) return rc;
      if ((rc = lu_update(n, j0, jb, j1 + nb2, rem, A, lda, sa, batch, stream, slots))) return rc;
      EUV_CUDA_TRY(cudaEventRecord(side->join, side->hi));
      EUV_CUDA_TRY(cudaStreamWaitEvent(stream, side->join, 0));
    }
    j0 = j1;
    jb = nb2;
  }
  return EUV_OK;
}

// Forward (unit lower L) and backward (upper U) substitution of RC right-hand
// sides per CTA with X resident in shared memory (xs[c*n + r]) for the whole
// solve; L and U are streamed once per CTA in blocks of LS_BLK rows/columns:
//   diagonal block : staged in shared memory (its loads issued during the
//                    previous block's update); warp c solves column c, lane i
//                    = block row i, each solved entry broadcast by shuffle;
//   off-diagonal   : x(r) -= T(r, block) x(block) for the rows below (forward)
//                    or above (backward).  RC = 8 runs it on the FP64 tensor
//                    path: 8-row tiles x 8 right-hand sides x K = 4 DMMAs, four
//                    per complex step, two tiles' loads in flight per warp;
//                    RC = 12 (two column tiles, the second half used) when the
//                    launch then takes fewer waves (24 units x 67 columns: 144
//                    CTAs instead of 216 on 148 SMs).
// Replaces 2*ceil(n/32) trsm launches + as many K=32 GEMMs per solve.
constexpr int LS_THREADS = 512;
constexpr int LS_WARPS = LS_THREADS / 32;
constexpr int LS_BLK = 32;
constexpr size_t LS_SMEM_MAX = 200 * 1024;

__device__ __forceinline__ void dmma884(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// Two elements per thread of the diagonal block at (j0, j0), zero outside jb.
struct DiagPrefetch {
  double2 v[2];
  __device__ __forceinline__ void load(const double2* LU, long long lda, int j0, int jb, int tid) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int i = tid + k * LS_THREADS, r = i % LS_BLK, q = i / LS_BLK;
      v[k] = (r < jb && q < jb) ? LU[j0 + r + (long long)(j0 + q) * lda] : make_double2(0.0, 0.0);
    }
  }
  __device__ __forceinline__ void store(double2 (*ds)[LS_BLK + 1], int tid) const {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int i = tid + k * LS_THREADS;
      ds[i % LS_BLK][i / LS_BLK] = v[k];
    }
  }
};
static_assert(2 * LS_THREADS == LS_BLK * LS_BLK, "DiagPrefetch covers the block");

// xs[c*n + r] -= sum_{q<jb} T(r, j0+q) xs[c*n + j0+q], r in [r_lo, r_hi), c < RC
template <int RC>
__device__ __forceinline__ void update_rows(double2* xs, int n, const double2* LU, long long lda,
                                            int j0, int jb, int r_lo, int r_hi, int tid) {
  if constexpr (RC == 8 || RC == 12) {
    // NT column tiles of 8 right-hand sides (RC = 12: the second tile half
    // used); each row tile's L fragment serves all of them.  UT row tiles'
    // loads in flight per warp (one at RC = 12, for the registers).
    constexpr int NT = (RC + 7) / 8, UT = RC == 8 ? 2 : 1;
    const int lane = tid & 31, warp = tid >> 5, kq = lane & 3, g = lane >> 2;
    double br[NT][8], bi[NT][8];  // B fragments: x(j0 + 4ks + kq) of right-hand side 8nt + g
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        const int q = 4 * ks + kq, c = 8 * nt + g;
        const double2 v = (q < jb && c < RC) ? xs[c * n + j0 + q] : make_double2(0.0, 0.0);
        br[nt][ks] = v.x;
        bi[nt][ks] = v.y;
      }
    const int ntiles = (r_hi - r_lo + 7) / 8;
    for (int t = warp; t < ntiles; t += UT * LS_WARPS) {
      double2 a[UT][8];
#pragma unroll
      for (int u = 0; u < UT; ++u) {
        const int tt = t + u * LS_WARPS, r = r_lo + tt * 8 + g;
        const bool rok = tt < ntiles && r < r_hi;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          const int q = 4 * ks + kq;
          a[u][ks] = (rok && q < jb) ? LU[r + (long long)(j0 + q) * lda] : make_double2(0.0, 0.0);
        }
      }
#pragma unroll
      for (int u = 0; u < UT; ++u) {
        const int tt = t + u * LS_WARPS;
        if (tt >= ntiles) break;  // warp-uniform
        const int r = r_lo + tt * 8 + g;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          double cr0 = 0.0, cr1 = 0.0, ci0 = 0.0, ci1 = 0.0;
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) {
            dmma884(cr0, cr1, a[u][ks].x, br[nt][ks]);
            dmma884(cr0, cr1, -a[u][ks].y, bi[nt][ks]);
            dmma884(ci0, ci1, a[u][ks].x, bi[nt][ks]);
            dmma884(ci0, ci1, a[u][ks].y, br[nt][ks]);
          }
          const int c0 = 8 * nt + 2 * kq;
          if (r < r_hi && c0 < RC) {
            double2* p0 = &xs[c0 * n + r];
            double2* p1 = &xs[(c0 + 1) * n + r];
            const double2 o0 = *p0, o1 = *p1;
            *p0 = make_double2(o0.x - cr0, o0.y - ci0);
            *p1 = make_double2(o1.x - cr1, o1.y - ci1);
          }
        }
      }
    }
  } else {
    for (int r = r_lo + tid; r < r_hi; r += LS_THREADS) {
      cplx acc[RC];
#pragma unroll
      for (int c = 0; c < RC; ++c) acc[c] = mk(0.0, 0.0);
      // eight loads in flight, then their products in order (left to the compiler, the
      // loads of one right-hand side waited for each other: six matrices of N = 961 1090 or
      // 1177 us by its version of the loop, 838 so; four of 1681, eight columns, 4.12 -> 3.83 ms)
      const double2* lp = LU + r + (long long)j0 * lda;
      int q = 0;
      for (; q + 8 <= jb; q += 8) {
        double2 lv[8];
#pragma unroll
        for (int e = 0; e < 8; ++e, lp += lda) lv[e] = *lp;
#pragma unroll
        for (int e = 0; e < 8; ++e)
#pragma unroll
          for (int c = 0; c < RC; ++c)
            acc[c] = acc[c] + mk(lv[e].x, lv[e].y) * ld2(&xs[c * n + j0 + q + e]);
      }
      for (; q < jb; ++q, lp += lda) {
        const cplx l1 = ld2(lp);
#pragma unroll
        for (int c = 0; c < RC; ++c) acc[c] = acc[c] + l1 * ld2(&xs[c * n + j0 + q]);
      }
#pragma unroll
      for (int c = 0; c < RC; ++c) st2(&xs[c * n + r], ld2(&xs[c * n + r]) - acc[c]);
    }
  }
}

// BACK: the forward half is done (lu_factor's extra columns), U x = y only.
template <int RC, bool BACK>
__global__ void __launch_bounds__(LS_THREADS) lu_subst_kernel(int n, int nrhs, const double2* LU,
                                                              long long lda, long long sa,
                                                              double2* B, long long ldb,
                                                              long long sb, const int* order,
                                                              long long ostride) {
  dependent_begin();
  extern __shared__ double2 xs[];
  __shared__ double2 ds[LS_BLK][LS_BLK + 1];
  const int b = blockIdx.y, c0 = blockIdx.x * RC;
  const int nc = (nrhs - c0) < RC ? (nrhs - c0) : RC;
  if (order != nullptr) {
    // every column of this CTA is an empty source slot (order < 0): its
    // right-hand sides are zero and so is the solution, already in place
    bool any = false;
    for (int c = 0; c < nc; ++c) any |= order[(long long)b * ostride + c0 + c] >= 0;
    if (!any) return;  // the same for every thread of the CTA
  }
  LU += (long long)b * sa;
  B += (long long)b * sb;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  DiagPrefetch pf;
  const int jl = ((n - 1) / LS_BLK) * LS_BLK;  // last diagonal block
  pf.load(LU, lda, BACK ? jl : 0, BACK ? n - jl : (n < LS_BLK ? n : LS_BLK), tid);
  for (int i = tid; i < RC * n; i += LS_THREADS) {
    const int c = i / n, r = i - c * n;
    xs[i] = c < nc ? B[r + (long long)(c0 + c) * ldb] : make_double2(0.0, 0.0);
  }
  pf.store(ds, tid);
  __syncthreads();
  // ---- forward: L y = b
  for (int j0 = 0; !BACK && j0 < n; j0 += LS_BLK) {
    const int jb = (n - j0) < LS_BLK ? (n - j0) : LS_BLK;
    if (warp < nc) {
      double2* xc = xs + (long long)warp * n + j0;
      cplx x = lane < jb ? ld2(&xc[lane]) : mk(0.0, 0.0);
#pragma unroll
      for (int q = 0; q < LS_BLK; ++q) {
        const cplx xq = mk(__shfl_sync(0xffffffffu, x.x, q), __shfl_sync(0xffffffffu, x.y, q));
        if (lane > q && lane < jb) x = x - ld2(&ds[lane][q]) * xq;
      }
      if (lane < jb) st2(&xc[lane], x);
    }
    __syncthreads();
    // next diagonal block: the forward pass's successor, or the backward pass's first
    const int jn = j0 + LS_BLK < n ? j0 + LS_BLK : jl;
    pf.load(LU, lda, jn, (n - jn) < LS_BLK ? (n - jn) : LS_BLK, tid);
    update_rows<RC>(xs, n, LU, lda, j0, jb, j0 + jb, n, tid);
    pf.store(ds, tid);
    __syncthreads();
  }
  // ---- backward: U x = y
  for (int j0 = jl; j0 >= 0; j0 -= LS_BLK) {
    const int jb = (n - j0) < LS_BLK ? (n - j0) : LS_BLK;
    if (warp < nc) {
      double2* xc = xs + (long long)warp * n + j0;
      cplx x = lane < jb ? ld2(&xc[lane]) : mk(0.0, 0.0);
      // each lane's reciprocal pivot, off the serial chain below
      const cplx rinv = lane < jb ? crecip(ld2(&ds[lane][lane])) : mk(0.0, 0.0);
#pragma unroll
      for (int q = LS_BLK - 1; q >= 0; --q) {
        if (q < jb) {  // warp-uniform
          if (lane == q) x = x * rinv;
          const cplx xq = mk(__shfl_sync(0xffffffffu, x.x, q), __shfl_sync(0xffffffffu, x.y, q));
          if (lane < q) x = x - ld2(&ds[lane][q]) * xq;
        }
      }
      if (lane < jb) st2(&xc[lane], x);
    }
    __syncthreads();
    if (j0 > 0) pf.load(LU, lda, j0 - LS_BLK, LS_BLK, tid);
    update_rows<RC>(xs, n, LU, lda, j0, jb, 0, j0, tid);
    if (j0 > 0) pf.store(ds, tid);
    __syncthreads();
  }
  for (int i = tid; i < RC * n; i += LS_THREADS) {
    const int c = i / n, r = i - c * n;
    if (c < nc) B[r + (long long)(c0 + c) * ldb] = xs[i];
  }
}

template <int RC, bool BACK>
static int launch_subst(int n, int nrhs, const double2* LU, long long lda, long long sa,
                        double2* B, long long ldb, long long sb, int batch, const int* order,
                        long long ostride, cudaStream_t stream) {
  static int smem_done[64];
  const int smem = (int)((size_t)RC * n * sizeof(double2));
  EUV_CUDA_TRY(ensure_smem(lu_subst_kernel<RC, BACK>, smem, smem_done));
  dim3 grid((nrhs + RC - 1) / RC, batch);
  EUV_CUDA_TRY(launch_dependent(lu_subst_kernel<RC, BACK>, grid, dim3(LS_THREADS), smem, stream, n,
                                nrhs, LU, lda, sa, B, ldb, sb, order, ostride));
  EUV_LAUNCH_CHECK();
  return EUV_OK;
}

// Right-hand sides per CTA of the one-launch solve, 0 where one column of X does
// not fit shared memory (or the batch the grid).  12 instead of 8 where that takes
// fewer waves (one CTA per SM either way: the resident columns fill its shared
// memory), or where the tuning table says so.
static int subst_columns(int n, int nrhs, int batch, bool slots, int* rc) {
  *rc = 0;
  if (batch > 65535) return EUV_OK;
  const size_t col = (size_t)n * sizeof(double2);
  if (12 * col <= LS_SMEM_MAX && nrhs >= 12) {
    const int tuned = tune_lookup(EUV_KNOB_LU_SUBST_COLS, n, batch);
    bool twelve = tuned == 12;
    if (tuned == 0) {
      int sms = 0, dev = 0;
      EUV_CUDA_TRY(cudaGetDevice(&dev));
      EUV_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
      const long long w8 = ((long long)((nrhs + 7) / 8) * batch + sms - 1) / sms;
      const long long w12 = ((long long)((nrhs + 11) / 12) * batch + sms - 1) / sms;
      // with empty source slots skipped the launch holds fewer live CTAs than
      // its grid, so a tie in waves goes to 12 (measured: 24 units of N = 961,
      // 96 slots for families of 96, 92 and 12 sources, step 25.35 -> 24.97 ms)
      twelve = sms > 0 && (w12 < w8 || (slots && w12 == w8));
    }
    if (twelve) {
      *rc = 12;
      return EUV_OK;
    }
  }
  for (int r = 8; r >= 1; r >>= 1)
    if (r * col <= LS_SMEM_MAX && nrhs >= r) {
      *rc = r;
      return EUV_OK;
    }
  return EUV_OK;
}

// The one-launch solve needs eight columns per CTA to run on the FP64 tensor path;
// above N = 1562 fewer fit, and every CTA streams the factor for four or two columns
// (B200, four units of N = 1681, 380 columns: 10.5 -> 3.8 ms).  A handful of
// columns takes one launch anyway.
static bool subst_pays(int cols, int nrhs) { return cols >= 8 || (cols > 0 && nrhs <= 8); }

template <bool BACK>
static int subst(int rc, int n, int nrhs, const double2* LU, long long lda, long long sa, double2* B,
                 long long ldb, long long sb, int batch, const int* order, long long ostride,
                 cudaStream_t stream) {
  switch (rc) {
    case 12: return launch_subst<12, BACK>(n, nrhs, LU, lda, sa, B, ldb, sb, batch, order, ostride, stream);
    case 8: return launch_subst<8, BACK>(n, nrhs, LU, lda, sa, B, ldb, sb, batch, order, ostride, stream);
    case 4: return launch_subst<4, BACK>(n, nrhs, LU, lda, sa, B, ldb, sb, batch, order, ostride, stream);
    case 2: return launch_subst<2, BACK>(n, nrhs, LU, lda, sa, B, ldb, sb, batch, order, ostride, stream);
    default: return launch_subst<1, BACK>(n, nrhs, LU, lda, sa, B, ldb, sb, batch, order, ostride, stream);
  }
}

// U X = Y or (lower) L Y = B by blocks of LU_NB rows, two launches each.
static int blocked_solve(bool lower, int n, int nrhs, const double2* LU, long long lda, long long sa,
                         double2* B, long long ldb, long long sb, int batch, cudaStream_t stream,
                         const Slots& slots) {
  const int nblk = (n + LU_NB - 1) / LU_NB;
  for (int k = 0; k < nblk; ++k) {
    const int j0 = (lower ? k : nblk - 1 - k) * LU_NB, jb = (n - j0) < LU_NB ? (n - j0) : LU_NB;
    EUV_CUDA_TRY(launch_dependent(lu_trsm_warp_kernel, trsm_grid(nrhs, batch),
                                  dim3(32 * LU_TRSM_WARPS), 0, stream, jb, nrhs, lower ? 1 : 0,
                                  LU + j0 + (long long)j0 * lda, lda, sa, B + j0, ldb, sb, slots));
    EUV_LAUNCH_CHECK();
    const int r0 = lower ? j0 + jb : 0, rows = lower ? n - r0 : j0;
    if (rows > 0) {
      const int rc = zgemm_sub(rows, nrhs, jb, LU + r0 + (long long)j0 * lda, lda, sa, B + j0, ldb, sb,
                               B + r0, ldb, sb, batch, stream, slots);
      if (rc != EUV_OK) return rc;
    }
  }
  return EUV_OK;
}

int lu_solve(int n, int nrhs, const double2* LU, long long lda, long long sa, const int* ipiv,
             double2* B, long long ldb, long long sb, int batch, cudaStream_t stream,
             const int* order, long long ostride) {
  if (n <= 0 || nrhs <= 0 || batch <= 0) return EUV_OK;
  const Slots slots{order, ostride, 0};
  dim3 gs((nrhs + 127) / 128, batch);
  lu_laswp_kernel<<<gs, 128, 0, stream>>>(n, nrhs, 0, n, 0, 0, B, ldb, sb, ipiv, n, 0);
  EUV_LAUNCH_CHECK();
  int cols = 0;
  int rc = subst_columns(n, nrhs, batch, order != nullptr, &cols);
  if (rc) return rc;
  if (subst_pays(cols, nrhs))
    return subst<false>(cols, n, nrhs, LU, lda, sa, B, ldb, sb, batch, order, ostride, stream);
  if ((rc = blocked_solve(true, n, nrhs, LU, lda, sa, B, ldb, sb, batch, stream, slots))) return rc;
  return blocked_solve(false, n, nrhs, LU, lda, sa, B, ldb, sb, batch, stream, slots);
}

// U X = Y for columns that lu_factor carried along.
int lu_back(int n, int nrhs, const double2* LU, long long lda, long long sa, double2* B,
            long long ldb, long long sb, int batch, cudaStream_t stream, const int* order,
            long long ostride) {
  if (n <= 0 || nrhs <= 0 || batch <= 0) return EUV_OK;
  int cols = 0;
  const int rc = subst_columns(n, nrhs, batch, order != nullptr, &cols);
  if (rc) return rc;
  if (subst_pays(cols, nrhs))
    return subst<true>(cols, n, nrhs, LU, lda, sa, B, ldb, sb, batch, order, ostride, stream);
  return blocked_solve(false, n, nrhs, LU, lda, sa, B, ldb, sb, batch, stream, Slots{order, ostride, 0});
}

}  // namespace euv

extern "C" size_t euv_lu_workspace_bytes(int n, int batch) {
  (void)n;
  (void)batch;
  return 0;
}

extern "C" int euv_lu_factor(int n, euv_c64* d_a, int lda, long long stride_a, int* d_ipiv,
                             int* d_info, int batch, void* stream) {
  if (n < 0 || lda < (n > 0 ? n : 1) || batch < 0 || (n > 0 && batch > 0 && (!d_a || !d_ipiv || !d_info))) {
    euv_set_error("euv_lu_factor: bad arguments (n=%d lda=%d batch=%d)", n, lda, batch);
    return EUV_ERR_BAD_ARG;
  }
  return euv::lu_factor(n, reinterpret_cast<double2*>(d_a), lda, stride_a, d_ipiv, d_info, batch,
                        (cudaStream_t)stream, 0, nullptr, 0);
}

extern "C" int euv_lu_solve(int n, int nrhs, const euv_c64* d_lu, int lda, long long stride_a,
                            const int* d_ipiv, euv_c64* d_b, int ldb, long long stride_b,
                            int batch, void* stream) {
  if (n < 0 || nrhs < 0 || lda < (n > 0 ? n : 1) || ldb < (n > 0 ? n : 1) || batch < 0) {
    euv_set_error("euv_lu_solve: bad arguments (n=%d nrhs=%d lda=%d ldb=%d)", n, nrhs, lda, ldb);
    return EUV_ERR_BAD_ARG;
  }
  return euv::lu_solve(n, nrhs, reinterpret_cast<const double2*>(d_lu), lda, stride_a, d_ipiv,
                       reinterpret_cast<double2*>(d_b), ldb, stride_b, batch,
                       (cudaStream_t)stream, nullptr, 0);
}
