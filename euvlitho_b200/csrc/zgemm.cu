// Batched complex FP64 GEMM on the B200 FP64 tensor path (DMMA).
//
// Replaces matproduct (header.h:1559-1619: Eigen product for N<=5000, cuBLAS
// Zgemm with host round trips above).  FP64 has no tcgen05 kind on sm_100a, so
// the FP64 form uses mma.sync.m8n8k4.f64 (the FP64 tensor instruction).
//
// Products (zgemm_kernel): CTA tile (32 MI) x 32 complex, K tile 16, 4 warps (2x2),
// warp tile (16 MI) x 16 as MI x 2 blocks of mma.m16n8k4.f64.  Three CTAs per SM
// and small tiles keep the FP64 pipe busy where a matrix is a few tiles plus an
// edge (N = 961 = 15 x 64 + 1): blocks of 16 x 8 past the edge are not multiplied
// and the waves are short.  Rank-k updates C -= A B of the LU (zgemm_upd_kernel):
// 32 x 64 or 64 x 64 tiles on m8n8k4, C preloaded into the accumulators.
// Operands are staged global->shared with 16-byte cp.async (one complex element
// per copy) in a 2- or 3-stage pipeline; copies and fragment loads (one 128-bit
// load = re+im) are bank-conflict free: A k-major with a 2-element pad, B by
// columns with odd columns swizzled (with B k-major too, the copies of 16
// consecutive k met 4-fold conflicts: six units of N = 961, N x 2N, 2.47 ms and
// 73 % of the DMMA pipe, now 2.32 ms and 78 %).
//
// THREE: the complex product from three real ones, P1 = Ar Br, P2 = Ai Bi, P3 =
// (Ar + Ai)(Br + Bi); Re = P1 - P2, Im = P3 - P1 - P2 (Knuth; Higham, "Stability
// of a method for multiplying complex matrices with three real matrix
// multiplications", 1992: as accurate as four in the norm, the imaginary part
// alone may lose the digits by which it is smaller than the real one).  The slab's
// N^3 products take it: they are bound by the FP64 pipe (37 TF/s measured for
// every DMMA shape) and their errors enter as norms.  euv_zgemm keeps four.
// B200, whole calls: N = 961, 6 units 27.2 -> 20.8 ms (the products 21.5 -> 15.2);
// M3D at N = 2121 53.5 -> 44.3 ms; N = 121, 4 units 0.90 -> 0.69 ms.
#include "common.cuh"

namespace euv {

constexpr int GBM = 64;
constexpr int GBN = 64;
constexpr int GBK = 16;
constexpr int GSTAGES = 3;
constexpr int GTHREADS = 128;

struct GemmArgs {
  int m, n, k;
  double2 alpha, beta, diag;
  const double* scale;
  const double2* a;
  long long lda, sa;
  const double2* b;
  long long ldb, sb;
  double2* c;
  GemmTerms t;
  long long ldc, sc;
  const int* steps;
  int step;
  Slots slots;  // of B's and C's columns (zgemm_upd_kernel)
};

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool pred) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  int sz = pred ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(sz));
}
__device__ __forceinline__ void cp_async16_all(void* smem, const void* gmem) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// element (k, column j) of a B tile: columns 16 apart, k of odd columns with bit 2
// flipped, so that the copies (16 consecutive k) and the fragment loads (4 k of 8
// columns) both hit distinct banks
__device__ __forceinline__ int b_at(int k, int j) { return j * GBK + (k ^ ((j & 1) << 2)); }
// C -= A B (alpha, beta, scale, diag ignored).  The accumulators start from C,
// whose loads are issued right after the first operand copies, and the A
// fragments are negated: no read of C after the products.
// MI: 8-row blocks per warp (tile BM = 16 MI rows x 64 columns); ST: cp.async stages.
template <int MI, int ST>
__global__ void __launch_bounds__(GTHREADS, MI == 2 ? 4 : 2) zgemm_upd_kernel(GemmArgs p) {
  dependent_begin();
  constexpr int BM = 16 * MI;
  constexpr int AP = BM + 2;
  extern __shared__ double2 smem[];
  double2* As = smem;
  double2* Bs = smem + ST * GBK * AP;
  const int bz = blockIdx.z;
  const int m0 = blockIdx.x * BM;
  const int n0 = blockIdx.y * GBN;
  const double2* A = p.a + (long long)bz * p.sa;
  const double2* B = p.b + (long long)bz * p.sb;
  double2* C = p.c + (long long)bz * p.sc;
  const int tid = threadIdx.x;
  if (p.slots.order != nullptr && n0 >= p.slots.first) {  // nothing but empty slots
    const int col = n0 + tid;
    const bool live = tid < GBN && col < p.n && !p.slots.empty(bz, col);
    if (!__syncthreads_or(live)) return;
  }

  const int warp = tid >> 5, lane = tid & 31;
  const int wm = (warp & 1) * (8 * MI), wn = (warp >> 1) * 32;
  double accr[MI][4][2], acci[MI][4][2];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      accr[i][j][0] = accr[i][j][1] = 0.0;
      acci[i][j][0] = acci[i][j][1] = 0.0;
    }

  const int ktiles = (p.k + GBK - 1) / GBK;
  auto load_tile = [&](int stage, int kt) {
    const int k0 = kt * GBK;
    double2* as = As + stage * GBK * AP;
    double2* bs = Bs + stage * GBK * GBN;
#pragma unroll
    for (int r = 0; r < (BM * GBK) / GTHREADS; ++r) {
      int idx = tid + r * GTHREADS;
      int i = idx % BM, kk = idx / BM;
      int gi = m0 + i, gk = k0 + kk;
      bool ok = gi < p.m && gk < p.k;
      const double2* src = ok ? A + gi + (long long)gk * p.lda : A;
      cp_async16(&as[kk * AP + i], src, ok);
    }
#pragma unroll
    for (int r = 0; r < (GBN * GBK) / GTHREADS; ++r) {
      int idx = tid + r * GTHREADS;
      int kk = idx % GBK, j = idx / GBK;
      int gk = k0 + kk, gj = n0 + j;
      bool ok = gk < p.k && gj < p.n;
      const double2* src = ok ? B + gk + (long long)gj * p.ldb : B;
      cp_async16(&bs[b_at(kk, j)], src, ok);
    }
  };

#pragma unroll
  for (int s = 0; s < ST - 1; ++s) {
    if (s < ktiles) load_tile(s, s);
    cp_async_commit();
  }
  {
#pragma unroll
    for (int mi = 0; mi < MI; ++mi) {
      const int row = m0 + wm + mi * 8 + (lane >> 2);
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int col = n0 + wn + ni * 8 + (lane & 3) * 2 + e;
          const double2 v = (row < p.m && col < p.n) ? C[row + (long long)col * p.ldc]
                                                     : make_double2(0.0, 0.0);
          accr[mi][ni][e] = v.x;
          acci[mi][ni][e] = v.y;
        }
    }
  }
  for (int kt = 0; kt < ktiles; ++kt) {
    cp_async_wait<ST - 2>();
    __syncthreads();
    {
      int nk = kt + ST - 1;
      if (nk < ktiles) load_tile(nk % ST, nk);
      cp_async_commit();
    }
    const double2* as = As + (kt % ST) * GBK * AP;
    const double2* bs = Bs + (kt % ST) * GBK * GBN;
#pragma unroll
    for (int ks = 0; ks < GBK; ks += 4) {
      const int kk = ks + (lane & 3);
      double ar[MI], ai[MI], an[MI], br[4], bi[4];
#pragma unroll
      for (int mi = 0; mi < MI; ++mi) {
        double2 v = as[kk * AP + wm + mi * 8 + (lane >> 2)];
        v.x = -v.x;
        v.y = -v.y;
        ar[mi] = v.x;
        ai[mi] = v.y;
        an[mi] = -v.y;
      }
#pragma unroll
      for (int ni = 0; ni < 4; ++ni) {
        double2 v = bs[b_at(kk, wn + ni * 8 + (lane >> 2))];
        br[ni] = v.x;
        bi[ni] = v.y;
      }
#pragma unroll
      for (int mi = 0; mi < MI; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
          dmma(accr[mi][ni][0], accr[mi][ni][1], ar[mi], br[ni]);
          dmma(accr[mi][ni][0], accr[mi][ni][1], an[mi], bi[ni]);
          dmma(acci[mi][ni][0], acci[mi][ni][1], ar[mi], bi[ni]);
          dmma(acci[mi][ni][0], acci[mi][ni][1], ai[mi], br[ni]);
        }
    }
  }
  cp_async_wait<0>();

#pragma unroll
  for (int mi = 0; mi < MI; ++mi) {
    const int row = m0 + wm + mi * 8 + (lane >> 2);
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int col = n0 + wn + ni * 8 + (lane & 3) * 2 + e;
        if (row < p.m && col < p.n)
          C[row + (long long)col * p.ldc] = make_double2(accr[mi][ni][e], acci[mi][ni][e]);
      }
  }
}

// C = alpha A B + beta Cin + beta2 Cin2 + diag I
constexpr int PBN = 32;
template <int MI>
constexpr size_t prod_smem() {
  return (size_t)GSTAGES * GBK * (32 * MI + 2 + PBN) * sizeof(double2);
}

__device__ __forceinline__ void dmma16(double (&d)[4], double a0, double a1, double b) {
  asm volatile(
      "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
      "{%0,%1,%2,%3};\n"
      : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
      : "d"(a0), "d"(a1), "d"(b));
}

template <bool V>
struct Flag {
  static constexpr bool value = V;
};

template <bool THREE, int MI>
__global__ void __launch_bounds__(GTHREADS, 3) zgemm_kernel(GemmArgs p) {
  dependent_begin();
  constexpr int BM = 32 * MI, AP = BM + 2, NACC = THREE ? 3 : 2;
  extern __shared__ double2 smem[];
  double2* As = smem;
  double2* Bs = smem + GSTAGES * GBK * AP;
  const int bz = blockIdx.z;
  const int m0 = blockIdx.x * BM;
  const int n0 = blockIdx.y * PBN;
  const double2* A = p.a + (long long)bz * p.sa;
  const double2* B = p.b + (long long)bz * p.sb;
  double2* C = p.c + (long long)bz * p.sc;
  const int tid = threadIdx.x;

  if (p.t.need != nullptr && p.t.need[bz] <= p.t.need_above) return;
  if (p.steps != nullptr && p.step >= p.steps[bz]) {
    if (!step_copies(p.t.paired, p.steps[bz], p.step)) return;
    // inactive double-angle step for this batch entry: C = A
    // eight loads in flight per thread before their stores
    constexpr int U = 8;
    for (int base = 0; base < BM * PBN; base += GTHREADS * U) {
      double2 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int idx = base + tid + u * GTHREADS;
        const int gi = m0 + idx % BM, gj = n0 + idx / BM;
        v[u] = (idx < BM * PBN && gi < p.m && gj < p.n) ? A[gi + (long long)gj * p.lda]
                                                         : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int idx = base + tid + u * GTHREADS;
        const int gi = m0 + idx % BM, gj = n0 + idx / BM;
        if (idx < BM * PBN && gi < p.m && gj < p.n) C[gi + (long long)gj * p.ldc] = v[u];
      }
    }
    return;
  }

  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int wm = (warp & 1) * (16 * MI), wn = (warp >> 1) * 16;
  // blocks of 16 rows / 8 columns of this warp that hold part of C (warp-uniform)
  const int mb = min(MI, max(0, (p.m - m0 - wm + 15) / 16));
  const int nb = mb > 0 ? min(2, max(0, (p.n - n0 - wn + 7) / 8)) : 0;
  double acc[NACC][MI][2][4];
#pragma unroll
  for (int x = 0; x < NACC; ++x)
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[x][i][j][e] = 0.0;

  // a thread's elements of a tile: rows ia + 0, k = ka + r (128 / BM) of A and
  // columns jb + 8 r, k = kb of B; source addresses advance by 16 k per tile, and
  // only the last tile of a K that is not a multiple of 16 checks k
  constexpr int KA = GTHREADS / BM, RA = GBK / KA, RB = PBN * GBK / GTHREADS;
  const int ktiles = (p.k + GBK - 1) / GBK;
  const int ia = tid % BM, ka = tid / BM, kb = tid % GBK, jb = tid / GBK;
  const bool arow = m0 + ia < p.m;
  const long long astep = (long long)KA * p.lda, atile = (long long)GBK * p.lda;
  // a tile inside both matrices: byte offsets of 32 bits from the two bases and no
  // tests (the address arithmetic of the checked form costs more issue slots
  // than the products)
  const bool inside = m0 + BM <= p.m && n0 + PBN <= p.n &&
                      (unsigned long long)p.lda * p.k < (1ull << 28) &&
                      (unsigned long long)p.ldb * p.n < (1ull << 28);
  const unsigned oa = 16u * (unsigned)(m0 + ia + ka * p.lda);
  const unsigned ob = 16u * (unsigned)(kb + (long long)(n0 + jb) * p.ldb);
  const unsigned sa_ = 16u * (unsigned)astep, sb_ = 128u * (unsigned)p.ldb;
  auto load_tile = [&](int stage, int kt) {
    double2* as = As + stage * GBK * AP + ka * AP + ia;
    double2* bs = Bs + stage * GBK * PBN + b_at(kb, jb);  // 8 columns further: + 8 GBK
    const int left = p.k - kt * GBK;  // k of this tile inside the sum
    if (inside && left >= GBK) {
      const unsigned a0 = oa + (unsigned)kt * (16u * (unsigned)atile);
      const unsigned b0 = ob + (unsigned)kt * (16u * GBK);
#pragma unroll
      for (int r = 0; r < RA; ++r)
        cp_async16_all(&as[r * KA * AP], reinterpret_cast<const char*>(A) + (a0 + r * sa_));
#pragma unroll
      for (int r = 0; r < RB; ++r)
        cp_async16_all(&bs[8 * GBK * r], reinterpret_cast<const char*>(B) + (b0 + r * sb_));
      return;
    }
    const double2* a = A + (arow ? m0 + ia : 0) + (long long)(ka + kt * GBK) * p.lda;
    const double2* b = B + kb + kt * GBK;
#pragma unroll
    for (int r = 0; r < RA; ++r) {
      const bool ok = arow && ka + r * KA < left;
      cp_async16(&as[r * KA * AP], ok ? a + r * astep : A, ok);
    }
#pragma unroll
    for (int r = 0; r < RB; ++r) {
      const int j = n0 + jb + 8 * r;
      const bool ok = j < p.n && kb < left;
      cp_async16(&bs[8 * GBK * r], ok ? b + (long long)j * p.ldb : B, ok);
    }
  };
#pragma unroll
  for (int s = 0; s < GSTAGES - 1; ++s) {
    if (s < ktiles) load_tile(s, s);
    cp_async_commit();
  }
  // the k loop, without the block tests where the warp's whole tile lies inside C
  // (branches between the products keep their operand loads from moving ahead)
  auto k_loop = [&](auto whole) {
    int st = 0, ld = GSTAGES - 1;  // stage of this tile and of the one to load
    for (int kt = 0; kt < ktiles; ++kt) {
      cp_async_wait<GSTAGES - 2>();
      __syncthreads();
      if (kt + GSTAGES - 1 < ktiles) load_tile(ld, kt + GSTAGES - 1);
      cp_async_commit();
      const double2* as = As + st * GBK * AP + t * AP + wm + g;
      const double2* bs = Bs + st * GBK * PBN + (wn + g) * GBK;
      if (++st == GSTAGES) st = 0;
      if (++ld == GSTAGES) ld = 0;
      if (!whole.value && nb == 0) continue;
#pragma unroll
      for (int ks = 0; ks < GBK; ks += 4) {
        double2 a[MI][2], b[2];
        double sa[MI][2], sb[2];
#pragma unroll
        for (int mi = 0; mi < MI; ++mi)
#pragma unroll
          for (int h = 0; h < 2; ++h) a[mi][h] = as[ks * AP + mi * 16 + 8 * h];
#pragma unroll
        for (int ni = 0; ni < 2; ++ni) b[ni] = bs[ni * 8 * GBK + ((ks + t) ^ ((g & 1) << 2))];
        // THREE: the sums of the third product, else -Im A
#pragma unroll
        for (int mi = 0; mi < MI; ++mi)
#pragma unroll
          for (int h = 0; h < 2; ++h) sa[mi][h] = THREE ? a[mi][h].x + a[mi][h].y : -a[mi][h].y;
#pragma unroll
        for (int ni = 0; ni < 2; ++ni) sb[ni] = THREE ? b[ni].x + b[ni].y : 0.0;
#pragma unroll
        for (int mi = 0; mi < MI; ++mi) {
          if (!whole.value && mi >= mb) break;
#pragma unroll
          for (int ni = 0; ni < 2; ++ni) {
            if (!whole.value && ni >= nb) break;
            dmma16(acc[0][mi][ni], a[mi][0].x, a[mi][1].x, b[ni].x);
            if (THREE) {
              dmma16(acc[1][mi][ni], a[mi][0].y, a[mi][1].y, b[ni].y);
              dmma16(acc[NACC - 1][mi][ni], sa[mi][0], sa[mi][1], sb[ni]);
            } else {
              dmma16(acc[1][mi][ni], a[mi][0].x, a[mi][1].x, b[ni].y);
              dmma16(acc[0][mi][ni], sa[mi][0], sa[mi][1], b[ni].y);
              dmma16(acc[1][mi][ni], a[mi][0].y, a[mi][1].y, b[ni].x);
            }
          }
        }
      }
    }
  };
  if (mb == MI && nb == 2)
    k_loop(Flag<true>{});
  else
    k_loop(Flag<false>{});
  cp_async_wait<0>();

  const double sc = p.scale ? p.scale[bz] : 1.0;
  const cplx alpha = mk(p.alpha.x * sc, p.alpha.y * sc);
  cplx beta = mk(p.beta.x, p.beta.y);
  if (p.t.beta_b) beta = beta * mk(p.t.beta_b[bz].x, p.t.beta_b[bz].y);
  const bool use_beta = (p.beta.x != 0.0 || p.beta.y != 0.0);
  const double2* Cin = p.t.cin ? p.t.cin + (long long)bz * p.t.scin : C;
  const bool use_2 = p.t.cin2 != nullptr;
  const double2* Cin2 = use_2 ? p.t.cin2 + (long long)bz * p.t.scin2 : C;
  const cplx beta2 = use_2 ? mk(p.t.beta2.x, p.t.beta2.y) * mk(p.t.beta2_b[bz].x, p.t.beta2_b[bz].y)
                           : mk(0.0, 0.0);
  const cplx dg = mk(p.diag.x, p.diag.y);
#pragma unroll
  for (int mi = 0; mi < MI; ++mi) {
    // the reads of this row block's added matrices before its stores (a load
    // after a store through the same pointer type would wait for it)
    cplx old[2][4];
#pragma unroll
    for (int ni = 0; ni < 2; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = m0 + wm + mi * 16 + g + 8 * (e >> 1);
        const int col = n0 + wn + ni * 8 + 2 * t + (e & 1);
        const bool in = row < p.m && col < p.n;
        const long long at = row + (long long)col * p.ldc;
        cplx o = mk(0.0, 0.0);
        if (use_beta && in) o = beta * mk(Cin[at].x, Cin[at].y);
        if (use_2 && in) o = o + beta2 * mk(Cin2[at].x, Cin2[at].y);
        old[ni][e] = o;
      }
#pragma unroll
    for (int ni = 0; ni < 2; ++ni)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int row = m0 + wm + mi * 16 + g + 8 * (e >> 1);
        const int col = n0 + wn + ni * 8 + 2 * t + (e & 1);
        if (row < p.m && col < p.n) {
          const double p1 = acc[0][mi][ni][e], p2 = acc[1][mi][ni][e];
          cplx v = alpha * (THREE ? mk(p1 - p2, acc[NACC - 1][mi][ni][e] - p1 - p2) : mk(p1, p2));
          v = v + old[ni][e];
          if (row == col) v = v + dg;
          C[row + (long long)col * p.ldc] = make_double2(v.x, v.y);
        }
      }
  }
}

template <int MI, int ST>
constexpr size_t zgemm_smem() {
  return (size_t)ST * GBK * (16 * MI + 2 + GBN) * sizeof(double2);
}

template <typename K>
static int zgemm_run(K kernel, int rows, int cols, size_t smem, int* done, const GemmArgs& p,
                     int batch, cudaStream_t stream) {
  dim3 grid((p.m + rows - 1) / rows, (p.n + cols - 1) / cols, batch);
  EUV_CUDA_TRY(ensure_smem(kernel, (int)smem, done));
  EUV_CUDA_TRY(launch_dependent(kernel, grid, dim3(GTHREADS), smem, stream, p));
  EUV_LAUNCH_CHECK();
  return EUV_OK;
}

int zgemm_launch(const GemmArgs& p, int batch, cudaStream_t stream, bool upd = false) {
  if (p.m <= 0 || p.n <= 0 || batch <= 0) return EUV_OK;
  static int done[6][64];
  if (upd && p.k <= 2 * GBK)
    // rank-k update with k <= 32 (the LU's trailing updates): 32 x 64 tiles and
    // two stages (both k tiles in flight at once) for four CTAs per SM
    return zgemm_run(zgemm_upd_kernel<2, 2>, 32, GBN, zgemm_smem<2, 2>(), done[0], p, batch, stream);
  if (upd)
    return zgemm_run(zgemm_upd_kernel<4, GSTAGES>, GBM, GBN, zgemm_smem<4, GSTAGES>(), done[1], p,
                     batch, stream);
  // a grid holds 65535 column tiles: the columns beyond in launches of their own (a copying
  // step or a diagonal there would take an operand of that many rows)
  constexpr int kCols = 65535 * PBN;
  if (p.n > kCols) {
    if (p.steps != nullptr || (p.m > kCols && (p.diag.x != 0.0 || p.diag.y != 0.0))) {
      euv_set_error("zgemm: unsupported shape");
      return EUV_ERR_BAD_ARG;
    }
    GemmArgs q = p;
    for (int c0 = 0; c0 < p.n; c0 += kCols) {
      q.n = p.n - c0 < kCols ? p.n - c0 : kCols;
      const int rc = zgemm_launch(q, batch, stream);
      if (rc || p.n - c0 <= kCols) return rc;
      q.b += (long long)kCols * p.ldb;
      q.c += (long long)kCols * p.ldc;
      if (q.t.cin) q.t.cin += (long long)kCols * p.ldc;
      if (q.t.cin2) q.t.cin2 += (long long)kCols * p.ldc;
      q.diag = make_double2(0.0, 0.0);
    }
  }
  // 64 x 32 tiles; 32 x 32 where those leave SMs without a CTA (or the tuning table says
  // so), and of the four-product form where up to four waves of three CTAs per SM end in one
  // of a single CTA per SM (B200, us, 64 -> 32 rows -> the tiles of 64 x 64 before: N = 961
  // 346 -> 262 -> 303; N = 121, 64 entries, 56 -> 46 -> 49; N = 441, six, 172 -> 138 -> 145;
  // 700 x 40 x 700, 24 entries, 255 -> 202 -> 218)
  const int tuned = tune_lookup(EUV_KNOB_ZGEMM_ROWS, p.m, batch);
  bool small = tuned == 32;
  if (tuned == 0) {
    const long long ctas = (long long)((p.m + 63) / 64) * ((p.n + PBN - 1) / PBN) * batch;
    const int wave = 3 * 148;
    small = ctas < 148 || (!p.t.three && ctas > wave && ctas < 4 * wave && (ctas - 1) % wave < 148);
  }
  if (p.t.three)
    return small ? zgemm_run(zgemm_kernel<true, 1>, 32, PBN, prod_smem<1>(), done[2], p, batch, stream)
                 : zgemm_run(zgemm_kernel<true, 2>, 64, PBN, prod_smem<2>(), done[3], p, batch, stream);
  return small ? zgemm_run(zgemm_kernel<false, 1>, 32, PBN, prod_smem<1>(), done[4], p, batch, stream)
               : zgemm_run(zgemm_kernel<false, 2>, 64, PBN, prod_smem<2>(), done[5], p, batch, stream);
}

// C -= A B (the rank-k updates of the blocked LU and its solves)
int zgemm_sub(int m, int n, int k, const double2* a, long long lda, long long sa,
              const double2* b, long long ldb, long long sb, double2* c, long long ldc,
              long long sc, int batch, cudaStream_t stream, const Slots& slots) {
  GemmArgs p = {};
  p.m = m;
  p.n = n;
  p.k = k;
  p.a = a;
  p.lda = lda;
  p.sa = sa;
  p.b = b;
  p.ldb = ldb;
  p.sb = sb;
  p.c = c;
  p.ldc = ldc;
  p.sc = sc;
  p.slots = slots;
  return zgemm_launch(p, batch, stream, true);
}

int zgemm(int m, int n, int k, cplx alpha, const double* scale, const double2* a, long long lda,
          long long sa, const double2* b, long long ldb, long long sb, cplx beta, double2* c,
          long long ldc, long long sc, cplx diag, int batch, const int* steps, int step,
          cudaStream_t stream, const GemmTerms& terms) {
  GemmArgs p;
  p.m = m;
  p.n = n;
  p.k = k;
  p.alpha = make_double2(alpha.x, alpha.y);
  p.beta = make_double2(beta.x, beta.y);
  p.diag = make_double2(diag.x, diag.y);
  p.scale = scale;
  p.a = a;
  p.lda = lda;
  p.sa = sa;
  p.b = b;
  p.ldb = ldb;
  p.sb = sb;
  p.c = c;
  p.t = terms;
  p.ldc = ldc;
  p.sc = sc;
  p.steps = steps;
  p.step = step;
  p.slots = Slots{};
  return zgemm_launch(p, batch, stream);
}

}  // namespace euv

extern "C" int euv_zgemm(int m, int n, int k, euv_c64 alpha, const double* d_scale,
                         const euv_c64* d_a, int lda, long long stride_a, const euv_c64* d_b,
                         int ldb, long long stride_b, euv_c64 beta, euv_c64* d_c, int ldc,
                         long long stride_c, euv_c64 diag_add, int batch, const int* d_steps,
                         int step, void* stream) {
  if (m < 0 || n < 0 || k < 0 || batch < 0 || lda < (m > 0 ? m : 1) || ldc < (m > 0 ? m : 1) ||
      ldb < (k > 0 ? k : 1) || d_a == nullptr || d_b == nullptr || d_c == nullptr) {
    euv_set_error("euv_zgemm: bad arguments (m=%d n=%d k=%d lda=%d ldb=%d ldc=%d)", m, n, k, lda,
                  ldb, ldc);
    return EUV_ERR_BAD_ARG;
  }
  if (d_steps != nullptr && (m != n || m != k)) {
    euv_set_error("euv_zgemm: step predication needs square operands");
    return EUV_ERR_BAD_ARG;
  }
  return euv::zgemm(m, n, k, euv::fromc(alpha), d_scale, reinterpret_cast<const double2*>(d_a),
                    lda, stride_a, reinterpret_cast<const double2*>(d_b), ldb, stride_b,
                    euv::fromc(beta), reinterpret_cast<double2*>(d_c), ldc, stride_c,
                    euv::fromc(diag_add), batch, d_steps, step, (cudaStream_t)stream, euv::GemmTerms{});
}
