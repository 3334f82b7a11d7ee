// RCWA (Fourier-modal) solve of the absorber on the Mo/Si multilayer, batched
// over units (clip, Bloch family, polarisation).  Replaces ampS and its callees
// in header.h (maskamp 1147-1206, multilayerS 5-363, absorberS0 754-1145,
// absorberS 365-752, the tail of ampS 1355-1465).
//
// Formulation.  For a slice with Toeplitz matrix D (header.h:416-443) the
// reference diagonalises D = W diag(al^2) W^-1 and forms the T-matrix blocks
// T1UL..T1BR from W, al, B1 = i(k W - kp/k Sigma W) and gamma = exp(i al d).
// Writing X = W(U1U+U1B), Y = W al (U1U-U1B) and G = i(k I - diag(kp/k) Sigma),
// those blocks collapse to
//     X1 = c (G1^-1 G2 X2) - i s Y2,   Y1 = -i D s (G1^-1 G2 X2) + c Y2,
// with c = cos(sqrt(D) d) and s = sin(sqrt(D) d)/sqrt(D) -- entire functions
// of D, so no eigenvectors, square-root branches or W^-1 are needed.  At the
// bottom (Ru cap, header.h:1292-1303) G X2 = diag(Bru (URUU+URUB)) t and
// Y2 = diag(alru (URUU-URUB)) t, i.e. the row relation P X2 + Q Y2 = 0 with
// P = -diag(adm) G and Q = I, which the slices' c and s carry to the top; there
// X1 = b + e, Y1 = diag(klm) (e - b) for incident e and reflected b
// (header.h:1355-1391), one N x N system for b = Ax (header.h:1394-1465).
// c and s are polynomials of D about its spectrum (slab polynomials below);
// euv_matfun_cs, which takes any D, expands about 0 (a degree-8 Taylor
// polynomial of A = D h^2 at h = d/2^m, then m double-angle steps s <- 2 s c,
// c <- 2 c^2 - I).  Every step is a GEMM.
#include <stdarg.h>
#include <stdio.h>
#include <string.h>
#include <math.h>

#include <cooperative_groups.h>

#include "common.cuh"

namespace euv {

int zgemm(int m, int n, int k, cplx alpha, const double* scale, const double2* a, long long lda,
          long long sa, const double2* b, long long ldb, long long sb, cplx beta, double2* c,
          long long ldc, long long sc, cplx diag, int batch, const int* steps, int step,
          cudaStream_t stream, const GemmTerms& terms = GemmTerms{});
// extra: right-hand sides in the columns after A's (L^-1 P B on return, for lu_back), order
// as for lu_solve
int lu_factor(int n, double2* A, long long lda, long long sa, int* ipiv, int* info, int batch,
              cudaStream_t stream, int extra = 0, const int* order = nullptr, long long ostride = 0);
int lu_back(int n, int nrhs, const double2* LU, long long lda, long long sa, double2* B,
            long long ldb, long long sb, int batch, cudaStream_t stream, const int* order,
            long long ostride);
// order (optional): per batch entry, ostride ints whose first nrhs mark the
// right-hand sides; a CTA whose columns are all < 0 (zero columns) is skipped
int lu_solve(int n, int nrhs, const double2* LU, long long lda, long long sa, const int* ipiv,
             double2* B, long long ldb, long long sb, int batch, cudaStream_t stream,
             const int* order = nullptr, long long ostride = 0);
int gemm_mixed(int m, int n, int k, cplx alpha, const double* scale, const double2* a,
               long long lda, long long sa, const double2* b, long long ldb, long long sb,
               cplx beta, double2* c, long long ldc, long long sc, cplx diag, int batch,
               const int* steps, int step, void* work, size_t work_bytes, int* status,
               cudaStream_t stream, int reuse, const GemmTerms& terms);
size_t gemm_mixed_workspace_bytes(int m, int n, int k, int batch);

// ||A||_1 bound for the degree-8 Taylor step of cos/sin(sqrt(A)): the dropped
// term is ~theta^9/18!, 1.6e-16 at theta = 1 (FP64) and 2e-8 at theta = 8,
// which the mixed form uses (its split-FP16x3 products carry ~1e-6 relative error,
// and each double-angle step saved also saves its error growth).
constexpr double kThetaFp64 = 1.0;
constexpr double kThetaMixed = 8.0;
inline double theta_for(int precision) {
  return precision == EUV_PREC_MIXED ? kThetaMixed : kThetaFp64;
}
constexpr int kMaxSteps = 40;

// ---------------------------------------------------------------- mask DFT
// Separable DFT of the vacuum indicator V (the mask bits; the absorber's is
// delta - F_V), frequencies l in [-lh, lh], m in [-mh, mh].  V is real, so only
// l >= 0 is summed and F(-l, -m) = conj F(l, m).  Mask row jj carries the pattern
// rows y = meshy (ndivy - 1 - jj + y_offset) + r (header.h:1153-1166; rows outside
// the mask read as absorber, rows past the grid drop out), so both stages run
// over mask pixels:
//   T(l, jj) = sum_ii V(ii, jj) Wx(ii, l),   F(l, m) = sum_jj T(l, jj) Wy(jj, m),
// Wx, Wy the twiddles summed over a pixel's mesh.
// Stage 1 multiplies the bits on the FP64 tensor path: the A fragments of 16 mask
// rows are decoded from the packed bits in registers, the columns are Re and Im of
// the l's.  It is bound by the FP64 pipe; the masked adds it replaces waited on
// shared memory and summed both signs of the frequency (B200, this stage: two 1024
// nm masks, 25 x 25 frequencies, 170 -> 23 us; sixteen 2048 nm masks, 81 x 81, 2.92
// -> 0.74 ms).
constexpr int SP_ROWS = 128, SP_K = 32, SP_CL = 8;

// exp(-2 pi i q / n), 0 <= q < n, n < 2^60: the angle within a quarter turn, so that its
// rounding stays below the result's
__device__ __forceinline__ cplx unit_root(long long q, long long n) {
  const long long k = (8 * q + n) / (2 * n);  // nearest quarter turn
  double s, c;
  sincospi((double)(4 * q - k * n) / (double)(2 * n), &s, &c);
  switch (k & 3) {
    case 0: return mk(c, -s);
    case 1: return mk(-s, -c);
    case 2: return mk(-c, s);
    default: return mk(s, c);
  }
}

// Wx[ii][2 (lh + 1)]: Re, Im of sum_r exp(-2 pi i l (meshx ii + r) / fx).  Unscaled, so
// that l = 0 sums whole numbers exactly; with 1 / (fx fy) here every add of a row rounded
// the same way at sizes that are no powers of two (lines on 672 x 280: 3.7e-15 of the
// spectrum, 1.7e-15 now; eight-slice image there 8e-15, 3e-15 now).
__global__ void spectrum_wx_kernel(int ndivx, int meshx, int fx, int lh, double* W) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ndivx * (lh + 1)) return;
  const int l = t % (lh + 1), ii = t / (lh + 1);
  double re = 0.0, im = 0.0;
  for (int r = 0; r < meshx; ++r) {
    const cplx w = unit_root(((long long)l * (meshx * ii + r)) % fx, fx);
    re += w.x;
    im += w.y;
  }
  W[2 * t] = re;
  W[2 * t + 1] = im;
}
// Wy[m' + mr jj] = sum over the pattern rows of mask row jj of exp(-2 pi i m y / fy)
__global__ void spectrum_wy_kernel(int ndivy, int meshy, int fy, int y_offset, int mh, double2* W) {
  dependent_begin();
  const int t = blockIdx.x * blockDim.x + threadIdx.x, mr = 2 * mh + 1;
  if (t >= ndivy * mr) return;
  const int m = t % mr - mh, jj = t / mr;
  double re = 0.0, im = 0.0;
  for (int r = 0; r < meshy; ++r) {
    const int y = meshy * (ndivy - 1 - jj + y_offset) + r;
    if (y < 0 || y >= fy) continue;
    long long q = ((long long)m * y) % fy;
    if (q < 0) q += fy;
    const cplx w = unit_root(q, fy);
    re += w.x;
    im += w.y;
  }
  W[t] = make_double2(re, im);
}

// The 32 bits from bit `at` on (MSB first, the first bit in bit 31), zero past `end`
__device__ __forceinline__ unsigned bits32(const uint8_t* mask, long long at, long long end) {
  if (at >= end) return 0u;
  const long long b = at >> 3, last = (end + 7) >> 3;
  unsigned long long v = 0;
#pragma unroll
  for (int k = 0; k < 5; ++k) v = (v << 8) | (b + k < last ? mask[b + k] : 0);
  unsigned w = (unsigned)(v >> (8 - (int)(at & 7)));
  if (end - at < 32) w &= ~0u << (32 - (int)(end - at));
  return w;
}

// Stage 1.  A cluster of 8 CTAs takes 128 rows of one mask and one tile of 8 NB
// columns; CTA q sums its eighth of the pixels ii, 8 warps with 16 rows each, W
// staged by 32 pixels; the eight partial sums meet in distributed shared memory.
template <int NB>
__global__ void __cluster_dims__(SP_CL, 1, 1) __launch_bounds__(256)
    spectrum_rows_kernel(const uint8_t* bits, long long mask_bytes, int ndivx, int ndivy, int lh,
                         const double* W, double2* T) {
  dependent_begin();
  namespace cg = cooperative_groups;
  constexpr int ST = NB * 8 + 4;  // doubles per staged pixel: conflict-free fragments
  cg::cluster_group cluster = cg::this_cluster();
  const int q = (int)cluster.block_rank();
  extern __shared__ double2 sm_spec[];
  double* ws = reinterpret_cast<double*>(sm_spec);  // [2][SP_K][ST], then [SP_ROWS][NB * 8]
  const int g = blockIdx.z, row0 = (blockIdx.x / SP_CL) * SP_ROWS, c0 = blockIdx.y * NB * 8;
  const int cols = 2 * (lh + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, fg = lane >> 2, ft = lane & 3;
  const uint8_t* mask = bits + (long long)g * mask_bytes;
  // pixels [xa, xb) of this CTA, whole steps of SP_K
  const int share = ((ndivx + SP_CL - 1) / SP_CL + SP_K - 1) / SP_K * SP_K;
  const int xa = q * share, xb = min(ndivx, xa + share);
  const int steps = xb > xa ? (xb - xa + SP_K - 1) / SP_K : 0;
  auto stage = [&](int k) {
    double* w = ws + (k & 1) * SP_K * ST;
    for (int i = tid; i < SP_K * NB * 4; i += 256) {  // pairs of columns: 16-byte copies
      const int c = 2 * (i % (NB * 4)), x = xa + k * SP_K + i / (NB * 4);
      const bool ok = x < ndivx && c0 + c < cols;
      const double* src = ok ? W + (long long)x * cols + c0 + c : W;
      const unsigned sa = (unsigned)__cvta_generic_to_shared(&w[(i / (NB * 4)) * ST + c]);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(src),
                   "r"(ok ? 16 : 0)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  double acc[NB][4];
#pragma unroll
  for (int j = 0; j < NB; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[j][e] = 0.0;
  const int ra = row0 + warp * 16 + fg, rb = ra + 8;
  if (steps > 0) stage(0);
  for (int k = 0; k < steps; ++k) {
    const int x = xa + k * SP_K;
    const long long at = (long long)ndivx * ra + x, bt = (long long)ndivx * rb + x;
    const unsigned wa = ra < ndivy ? bits32(mask, at, (long long)ndivx * (ra + 1)) : 0u;
    const unsigned wb = rb < ndivy ? bits32(mask, bt, (long long)ndivx * (rb + 1)) : 0u;
    if (k + 1 < steps) {
      stage(k + 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const double* w = ws + (k & 1) * SP_K * ST;
#pragma unroll
    for (int s = 0; s < SP_K / 4; ++s) {
      const int sh = 31 - (4 * s + ft);
      const double a0 = __hiloint2double((int)((wa >> sh) & 1u) * 0x3ff00000, 0);
      const double a1 = __hiloint2double((int)((wb >> sh) & 1u) * 0x3ff00000, 0);
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        const double b = w[(4 * s + ft) * ST + 8 * j + fg];
        asm volatile(
            "mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, "
            "{%0,%1,%2,%3};\n"
            : "+d"(acc[j][0]), "+d"(acc[j][1]), "+d"(acc[j][2]), "+d"(acc[j][3])
            : "d"(a0), "d"(a1), "d"(b));
      }
    }
    __syncthreads();
  }
  double* red = ws;  // [SP_ROWS][NB * 8]
#pragma unroll
  for (int j = 0; j < NB; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e)
      red[(warp * 16 + fg + 8 * (e >> 1)) * (NB * 8) + 8 * j + 2 * ft + (e & 1)] = acc[j][e];
  cluster.sync();
  // rows 16 q .. 16 q + 15: lanes take consecutive rows
  for (int i = tid; i < 16 * NB * 4; i += 256) {
    const int r = 16 * q + i % 16, c = 2 * (i / 16), jj = row0 + r;
    double2 v = make_double2(0.0, 0.0);
#pragma unroll
    for (int t = 0; t < SP_CL; ++t) {
      const double* p = cluster.map_shared_rank(red, t) + r * (NB * 8) + c;
      v.x += p[0];
      v.y += p[1];
    }
    if (jj < ndivy && c0 + c < cols)
      T[((long long)g * (lh + 1) + (c0 + c) / 2) * ndivy + jj] = v;
  }
  cluster.sync();  // a peer may still read this CTA's sums
}
template <int NB>
constexpr size_t spectrum_smem() {
  const size_t a = 2 * (size_t)SP_K * (NB * 8 + 4) * sizeof(double);
  const size_t b = (size_t)SP_ROWS * NB * 8 * sizeof(double);
  return a > b ? a : b;
}

// F(l, m) from the K chunks' partial sums P[part][g][l >= 0][m'] over the grid's cells,
// both signs of l and, unless select_vacuum, the absorber's spectrum delta - F
__global__ void spectrum_reduce_kernel(const double2* part, int parts, int masks, int lh, int mh,
                                       double cells, int select_vacuum, double2* out) {
  dependent_begin();
  const int lr = 2 * lh + 1, mr = 2 * mh + 1;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)masks * lr * mr) return;
  const int l = (int)(t % lr) - lh, m = (int)(t / lr % mr) - mh, g = (int)(t / ((long long)lr * mr));
  const long long total = (long long)masks * (lh + 1) * mr;
  const bool neg = l < 0;
  const double2* p = part + ((long long)g * (lh + 1) + (neg ? -l : l)) * mr + (neg ? mh - m : mh + m);
  double2 s = p[0];
  for (int k = 1; k < parts; ++k) {
    const double2 v = p[k * total];
    s.x += v.x;
    s.y += v.y;
  }
  s.x /= cells;
  s.y /= neg ? -cells : cells;
  if (!select_vacuum) {
    s.x = (l == 0 && m == 0 ? 1.0 : 0.0) - s.x;
    s.y = -s.y;
  }
  out[t] = s;
}

// K chunks of stage 2: ndivy / parts a multiple of 64 where that is possible
static int spectrum_parts(int ndivy) {
  if (ndivy % 64) return 1;
  int parts = ndivy / 64 < 16 ? ndivy / 64 : 16;
  while ((ndivy / 64) % parts) --parts;
  return parts;
}

// ---------------------------------------------------------------- D and G
struct SliceParams {
  double k, dx, dy;
  const double* dxs;  // per-unit periods (NULL: dx, dy for every unit)
  const double* dys;
  int n, lmax, mmax, lr2, mr2, n_slices, slice;
  cplx eps_m1;   // eps_abs - 1
  cplx sig_m1;   // 1/eps_abs - 1
  cplx logeps;   // log(eps_abs)
};

// D gets the slab's normalised matrix (D - a I) / R, a and R of the unit in
// shift (i a) and radius (poly_coef_kernel):
// D(i,j) = k^2 eps[..] - i eta[..] kx_j (X) / - i zeta[..] ky_j (Y), minus kxy2_i
// on the diagonal (header.h:416-443); G(i,j) = i(k delta_ij - kp_i/k sigma[..] kp_j)
// (B1 = G W1, header.h:596-623).  D may be null; want_g = 1:
// G, 2 E with G = i k (I - E), 3 the bottom boundary row -diag(adm) G.
__global__ void build_dg_kernel(SliceParams p, const double2* spectra, const int* spec_of_unit,
                                const int* lidx, const int* midx, const double* kx0,
                                const double* ky0, const int* polar, const double2* adm,
                                const double2* shift, const double* radius, double2* D,
                                long long sd, double2* G, long long sg, int want_g) {
  dependent_begin();
  // grid: x = column j, y = row chunk, z = unit (no 64-bit division per element)
  const int u = blockIdx.z, j = blockIdx.x;
  // the unit's and column's constants once per CTA: no FP64 division per element
  __shared__ double s_c[10];  // 2pi/dx, 2pi/dy, 1/k, kx_j, ky_j, kx0, ky0, a, 1/R
  if (threadIdx.x == 0) {
    const double twopi = 6.283185307179586476925286766559;
    const double dxu = p.dxs ? p.dxs[u] : p.dx, dyu = p.dys ? p.dys[u] : p.dy;
    const double gx = twopi / dxu, gy = twopi / dyu;
    s_c[0] = gx;
    s_c[1] = gy;
    s_c[2] = 1.0 / p.k;
    s_c[3] = kx0[u] + gx * lidx[j];
    s_c[4] = ky0[u] + gy * midx[j];
    s_c[5] = kx0[u];
    s_c[6] = ky0[u];
    if (D != nullptr) {
      s_c[7] = shift[u].y;   // shift holds i a
      s_c[8] = -shift[u].x;
      s_c[9] = 1.0 / radius[u];
    }
  }
  __syncthreads();
  const int i = blockIdx.y * blockDim.x + threadIdx.x;
  if (i >= p.n) return;
  const long long t = (long long)j * p.n + i;
  const int li = lidx[i], mi = midx[i], lj = lidx[j], mj = midx[j];
  const int l = li - lj + 2 * p.lmax, m = mi - mj + 2 * p.mmax;
  const double2* sp = spectra + ((long long)spec_of_unit[u] * p.n_slices + p.slice) * p.lr2 * p.mr2;
  const double2 f2 = sp[l + (long long)p.lr2 * m];
  const cplx F = mk(f2.x, f2.y);
  const bool dc = (l == 2 * p.lmax) && (m == 2 * p.mmax);
  const double gx = s_c[0], gy = s_c[1], ik = s_c[2];
  const double kxi = s_c[5] + gx * li, kyi = s_c[6] + gy * mi;
  const double kxj = s_c[3], kyj = s_c[4];
  const int pol = polar[u];
  if (D != nullptr) {
    cplx eps = p.eps_m1 * F;
    if (dc) eps.x += 1.0;
    cplx leps = p.logeps * F;
    cplx v = (p.k * p.k) * eps;
    if (pol == 0) {
      // -i * eta * kx_j, eta = i 2 pi l / dx * leps  ->  +2 pi l/dx * leps * kx_j
      v = v + (gx * (double)(l - 2 * p.lmax) * kxj) * leps;
    } else {
      v = v + (gy * (double)(m - 2 * p.mmax) * kyj) * leps;
    }
    if (i == j) {
      v.x -= kxi * kxi + kyi * kyi + s_c[7];
      v.y -= s_c[8];
    }
    D[(long long)u * sd + t] = make_double2(s_c[9] * v.x, s_c[9] * v.y);
  }
  if (want_g) {
    cplx sig = p.sig_m1 * F;
    if (dc) sig.x += 1.0;
    const double kpi = pol == 0 ? kxi : kyi, kpj = pol == 0 ? kxj : kyj;
    if (want_g == 2) {
      // E = diag(kp/k) sigma diag(kp/k), with G = i k (I - E)
      cplx v = (kpi * ik * (kpj * ik)) * sig;
      G[(long long)u * sg + t] = make_double2(v.x, v.y);
    } else {
      // G = i (k delta - kp_i/k sig kp_j)
      cplx a = (-kpi * ik * kpj) * sig;
      if (i == j) a.x += p.k;
      cplx v = cmul_i(a);
      if (want_g == 3) {
        const double2 y = adm[(long long)u * p.n + i];
        v = -(mk(y.x, y.y) * v);
      }
      G[(long long)u * sg + t] = make_double2(v.x, v.y);
    }
  }
}

// ---------------------------------------------------------------- multilayer
struct StackParams {
  double k;
  cplx emo, esi, eru, emosi2, erusi, esio2;
  double dmo, dmosi, dsi, dsimo, dsiru, dru;
  int nml;
  double dx, dy;
  const double* dxs;  // per-unit periods (NULL: dx, dy for every unit)
  const double* dys;
  int n;
};

struct Blk {
  cplx ul, ur, bl, br;
};

__device__ __forceinline__ Blk iface(cplx cj, cplx al_out, cplx al_in, double thick) {
  // 1/2 (Cj +- al_out/al_in Cjp) exp(-+ i al_in d) (header.h:68-92 pattern)
  cplx expz = cexp_(cmul_i(al_in) * thick);
  cplx a = cdiv(al_out, al_in);
  cplx pl = 0.5 * (cj + a), mi = 0.5 * (cj - a);
  Blk b;
  b.ul = cdiv(pl, expz);
  b.ur = cdiv(mi, expz);
  b.bl = mi * expz;
  b.br = pl * expz;
  return b;
}
__device__ __forceinline__ void apply_blk(const Blk& b, cplx& uu, cplx& ub) {
  cplx nu = b.ul * uu + b.ur * ub;
  cplx nb = b.bl * uu + b.br * ub;
  uu = nu;
  ub = nb;
}

// Per order: URUU, URUB (header.h:5-363), alru, Bru (header.h:1292-1303), and
// the admittance y2 / gx2 of the bottom boundary, y2 = alru (URUU-URUB) and
// gx2 = Bru (URUU+URUB); klm = sqrt(k^2-kxy2) as a real root (header.h:1283).
__global__ void multilayer_kernel(StackParams p, const int* lidx, const int* midx,
                                  const double* kx0, const double* ky0, const int* polar,
                                  double2* adm, double* klm, int n_units) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= p.n * n_units) return;
  const int u = t / p.n, i = t % p.n;
  const double twopi = 6.283185307179586476925286766559;
  const double kx = kx0[u] + twopi * lidx[i] / (p.dxs ? p.dxs[u] : p.dx);
  const double ky = ky0[u] + twopi * midx[i] / (p.dys ? p.dys[u] : p.dy);
  const double kxy2 = kx * kx + ky * ky;
  const double k = p.k, k2 = k * k;
  const double kp = polar[u] == 0 ? kx : ky;
  auto al = [&](cplx e) { return csqrt_p(mk(k2 * e.x - kxy2, k2 * e.y)); };
  cplx alsio2 = al(p.esio2), almo = al(p.emo), alsi = al(p.esi), almosi2 = al(p.emosi2),
       alru = al(p.eru), alrusi = al(p.erusi);
  auto ratio = [&](cplx enu, cplx eden) {
    cplx a = mk(k, 0.0) - cdiv(mk(kp * kp / k, 0.0), enu);
    cplx b = mk(k, 0.0) - cdiv(mk(kp * kp / k, 0.0), eden);
    return cdiv(a, b);
  };
  Blk TMO = iface(ratio(p.emosi2, p.emo), almosi2, almo, p.dmo);
  Blk TMOSI = iface(ratio(p.emo, p.emosi2), almo, almosi2, p.dmosi);
  Blk TSI = iface(ratio(p.emosi2, p.esi), almosi2, alsi, p.dsi);
  Blk TSIMO = iface(ratio(p.esi, p.emosi2), alsi, almosi2, p.dsimo);
  Blk TSIRU = iface(ratio(p.esi, p.erusi), alsi, alrusi, p.dsiru);
  Blk TRU = iface(ratio(p.erusi, p.eru), alrusi, alru, p.dru);
  Blk TN = iface(ratio(p.esio2, p.emo), alsio2, almo, p.dmo);
  cplx uu = TN.ul, ub = TN.bl;  // substrate (header.h:294-324)
  for (int l = p.nml - 1; l >= 0; --l) {  // header.h:326-359
    if (l < p.nml - 1) apply_blk(TMO, uu, ub);
    apply_blk(TMOSI, uu, ub);
    apply_blk(TSI, uu, ub);
    if (l > 0)
      apply_blk(TSIMO, uu, ub);
    else
      apply_blk(TSIRU, uu, ub);
  }
  apply_blk(TRU, uu, ub);  // URUU, URUB (header.h:361-362)
  const cplx bru = mk(0.0, k) - cmul_i(cdiv(mk(kp * kp / k, 0.0), p.eru));
  const cplx s = uu + ub, d = uu - ub;
  // a node of the total field (gx2 = 0) is the limit of a large admittance
  const cplx gv = bru * s;
  const cplx yv = (gv.x == 0.0 && gv.y == 0.0) ? mk(1e30, 0.0) : cdiv(alru * d, gv);
  adm[t] = make_double2(yv.x, yv.y);
  klm[t] = sqrt(k2 - kxy2);  // NaN for evanescent orders, as the reference
}

// ---------------------------------------------------------------- matrix functions
__global__ void zero_f64_kernel(double* p, int n) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = 0.0;
}

// norm[b] = max_j sum_i (|re|+|im|)(D[b](i,j)): one warp per column.
__global__ void norm1_kernel(int n, const double2* D, double* norm) {
  dependent_begin();
  const int b = blockIdx.y;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= n) return;
  const double2* col = D + (long long)b * n * n + (long long)warp * n;
  double s = 0.0;
  for (int i = lane; i < n; i += 32) s += fabs(col[i].x) + fabs(col[i].y);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
  if (lane == 0) atomicMax(reinterpret_cast<unsigned long long*>(&norm[b]), __double_as_longlong(s));
}

// m = smallest m >= 0 with norm*(d/2^m)^2 <= theta (capped at m_max); h = d/2^m.
__global__ void scale_kernel(int batch, double theta, const double* norm, const double* thick, int m_max,
                             int* steps, double* h, double* h2, double* h4, int* capped) {
  dependent_begin();
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= batch) return;
  double d = thick[b];
  double v = norm[b] * d * d;
  int m = 0;
  while (v > theta && m < kMaxSteps) {
    v *= 0.25;
    ++m;
  }
  if (m > m_max) {
    m = m_max;
    if (capped) atomicOr(capped, EUV_STATUS_STEPS_CLAMPED);
  }
  double hh = ldexp(d, -m);
  steps[b] = m;
  h[b] = hh;
  h2[b] = hh * hh;
  h4[b] = hh * hh * hh * hh;
}

// Taylor coefficients: cos: (-1)^n/(2n)!, sinc: (-1)^n/(2n+1)!, n = 0..8.
__constant__ double c_cos[9] = {1.0, -1.0 / 2.0, 1.0 / 24.0, -1.0 / 720.0, 1.0 / 40320.0,
                                -1.0 / 3628800.0, 1.0 / 479001600.0, -1.0 / 87178291200.0,
                                1.0 / 20922789888000.0};
__constant__ double c_sin[9] = {1.0, -1.0 / 6.0, 1.0 / 120.0, -1.0 / 5040.0, 1.0 / 362880.0,
                                -1.0 / 39916800.0, 1.0 / 6227020800.0, -1.0 / 1307674368000.0,
                                1.0 / 355687428096000.0};

// With A = h^2 D, P2 = A^2, P3 = A^3, P4 = A^4 (scaled):
//   Cc = sum_{n<4} a_n A^n,  Tc = sum_{n<4} a_{n+4} A^n + a_8 A^4
//   Cs = h sum_{n<4} b_n A^n, Ts = h (sum_{n<4} b_{n+4} A^n + b_8 A^4)
// so that cos = Cc + P4 Tc and sin/sqrt = Cs + P4 Ts.
__global__ void taylor_prep_kernel(int n, int batch, const double2* D, const double2* P2,
                                   const double2* P3, const double2* P4, const double* h,
                                   const double* h2, double2* Cc, double2* Tc, double2* Cs,
                                   double2* Ts) {
  dependent_begin();
  const long long nn = (long long)n * n;
  const int b = blockIdx.y;
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nn) return;
  const long long o = (long long)b * nn + t;
  const int i = (int)(t % n), j = (int)(t / n);
  const double e = (i == j) ? 1.0 : 0.0;
  const double hb = h[b], s2 = h2[b];
  const double2 d = D[o], p2 = P2[o], p3 = P3[o], p4 = P4[o];
  const double ax = s2 * d.x, ay = s2 * d.y;
  double ccx = c_cos[0] * e + c_cos[1] * ax + c_cos[2] * p2.x + c_cos[3] * p3.x;
  double ccy = c_cos[1] * ay + c_cos[2] * p2.y + c_cos[3] * p3.y;
  double tcx = c_cos[4] * e + c_cos[5] * ax + c_cos[6] * p2.x + c_cos[7] * p3.x + c_cos[8] * p4.x;
  double tcy = c_cos[5] * ay + c_cos[6] * p2.y + c_cos[7] * p3.y + c_cos[8] * p4.y;
  double csx = c_sin[0] * e + c_sin[1] * ax + c_sin[2] * p2.x + c_sin[3] * p3.x;
  double csy = c_sin[1] * ay + c_sin[2] * p2.y + c_sin[3] * p3.y;
  double tsx = c_sin[4] * e + c_sin[5] * ax + c_sin[6] * p2.x + c_sin[7] * p3.x + c_sin[8] * p4.x;
  double tsy = c_sin[5] * ay + c_sin[6] * p2.y + c_sin[7] * p3.y + c_sin[8] * p4.y;
  Cc[o] = make_double2(ccx, ccy);
  Tc[o] = make_double2(tcx, tcy);
  Cs[o] = make_double2(hb * csx, hb * csy);
  Ts[o] = make_double2(hb * tsx, hb * tsy);
}

// ---------------------------------------------------------------- slab polynomials
// c = cos(sqrt(D) d) and s = sin(sqrt(D) d)/sqrt(D) as polynomials in D about
// its spectrum.  D = k^2 T(eps) - diag(kxy^2) + (small commutator): the finite
// Toeplitz section T(eps) of a two-valued pattern has its field of values on
// the segment from 1 to eps_abs, the diagonal is real, and the log(eps) term is
// a commutator of norm <= w.  So the field of values lies in a flat ellipse
// around a (centre, foci a +- c, sum of semi-axes |c| rho), known from the
// configuration alone, and a Chebyshev expansion on it converges like
// tau^n / n!, tau = d (sum of semi-axes) / (4 |sqrt a|): about 1 for a 60 nm
// slab, where the expansion about 0 needs ||D||_1 d^2 ~ 10^3 halved by 5 to 6
// double-angle steps (two products each, and each doubles the error).
// Evaluated as a polynomial in E = (D - a)/R by blocks of q powers (Paterson-
// Stockmeyer): p = c_0 + B_0 + E^q (B_1 + E^q (...)), B_j = sum_{1..q} c_{qj+i}
// E^i.  The identity part c_0 stays a number per unit: the matrices c - c_0 and
// s - s_0 that enter later products are then small against c_0 and s_0, and so is
// the error the split products make (their FP32 sums lose 2^-24 of the running
// sum at every step; with the identity inside the operands the 2048 nm
// eight-slice image was 1.6e-5 off, 7e-6 for the expansion about 0).  Products:
// q - 1 for the powers and 2 (J - 1) for the two functions; q and J from poly_plan,
// a double-angle step (two products, as many as one more block; it doubles the error
// of its operands) only where degree q * jcap is not enough (orders near grazing) or
// the terms outgrow their sum (kPolyWide).  With the row recursion of euv_amp (no
// G^-1, no product with the solved columns) the call takes 8 N^3 products instead of
// 25 for a 60 nm slab in the mixed form.  B200, whole image calls: four 1024 nm clips
// at N = 625 (24 units, mixed) 11.64 -> 8.15 ms and 1.1e-5 -> 1.5e-6 of the exact
// image; N = 961, 6 units, FP64 46.9 -> 27.2 ms; M3D at N = 2121, FP64 94.1 -> 53.5 ms.
constexpr int PF_K = 30;       // largest degree (one per lane of a warp)
constexpr int PF_Q = 6;        // largest q
constexpr int PF_J = 5;        // largest block count
constexpr int PF_SAMPLES = 64; // points on the ellipse
constexpr double kPolyTolFp64 = 1e-15;  // first dropped term; the ones after it fall factorially
constexpr double kPolyTolMixed = 5e-8;  // the split products carry ~1e-6
// A unit in split-plane products whose poly_growth exceeds kPolyWide (an order box that is
// wide against a period) takes double-angle steps down to kPolyGrowth, and its powers are
// multiplied with the diagonals apart: the powers' terms are there up to e^growth / 2
// larger than their sum, and E is mostly its diagonal, of which the FP32 sums of a power
// lose 2^-24 at every step (GemmTerms::apart).  Image errors, root mean square of eight
// masks, steps by degree alone -> these -> one step without the diagonals apart:
// 1088 x 272 nm, 25 x 25 orders (growth 5.4) 1.2e-5 -> 1.4e-6 -> 5.3e-6; 256 nm, 17 x 17
// (5.2) 5.7e-6 -> 1.0e-6 -> 4.9e-6, 19 x 19 (6.4) 5.4e-6 -> 0.9e-6 (to growth 3.2: 4.7e-6).
// Below the line the error is 0.3 to 3e-6 as it is (296 x 1104 nm, growth 3.9: 2.4e-6),
// up to 6e-6 for strong absorbers near grazing, where the products of the top interface set it.
constexpr double kPolyWide = 4.0;
constexpr double kPolyGrowth = 2.5;

struct PolyRegion {
  cplx a, c;         // centre, focal half-axis (complex)
  double rho, r;     // ellipse a + c (rho e^it + e^-it / rho)/2; scale of E
};

// kxy2 in [lo, hi] over the orders; w: norm bound of the commutator term.
__host__ __device__ inline PolyRegion poly_region(double k, cplx eps_m1, double lo, double hi,
                                                  double w) {
  const cplx u = (0.5 * k * k) * eps_m1, v = mk(0.5 * (hi - lo), 0.0);
  PolyRegion g;
  g.a = mk(k * k + u.x - 0.5 * (hi + lo), u.y);
  w += 1e-9 * k * k;
  // parallelogram with corners +-p, +-q; foci along the principal direction
  const cplx p = u + v, q = u - v;
  const double lp = cabs(p), lq = cabs(q), len = lp > lq ? lp : lq;
  cplx dir = csqrt_p(u * u + v * v);
  const double ld = cabs(dir);
  dir = ld > 0.0 ? (1.0 / ld) * dir : mk(1.0, 0.0);
  double best_sum = 2.0 * len, best_c = 0.0;  // the circle through the far corner
  for (int t = 1; t <= 16 && len > 0.0; ++t) {
    const double cm = len * t / 16.0;
    double rho = 1.0;
    for (int i = 0; i < 2; ++i) {
      const cplx x = cdiv(i ? q : p, cm * dir);
      const double m = cabs(x + csqrt_p(x * x - mk(1.0, 0.0)));
      const double r = m > 1.0 ? m : 1.0 / m;
      if (r > rho) rho = r;
    }
    if (cm * rho < best_sum) {
      best_sum = cm * rho;
      best_c = cm;
    }
  }
  // semi-axes, widened by the disc of radius w
  const double minor2 = best_sum > 0.0 ? best_c * best_c / best_sum : 0.0;  // a - b
  const double sa = 0.5 * (best_sum + minor2) + w, sb = 0.5 * (best_sum - minor2) + w;
  double cm = sqrt((sa - sb) * (sa + sb));
  if (cm < 0.02 * sa) cm = 0.02 * sa;  // near a circle: keep the foci apart
  g.c = cm * dir;
  g.rho = (sa + sb) / cm;
  g.r = sa;
  return g;
}

// Degree that brings the first dropped term of both functions below tol: the
// bound tau^n/n! with the smallest |sqrt z| on the ellipse, or, where the
// ellipse comes near 0, the Taylor bound (h^2 |z|)^n / (2n)!.  PF_K + 1: more.
__host__ __device__ inline int poly_degree(const PolyRegion& g, double h, double tol) {
  const double a = cabs(g.a), sum = g.rho * cabs(g.c);
  const double near = a - g.r;
  const double tau = near > 0.0 ? 0.25 * h * sum / sqrt(near) : 1e300;
  const double z = h * h * (a + g.r);
  double t1 = 2.0, t2 = 2.0;
  for (int n = 1; n <= PF_K + 1; ++n) {
    t1 *= tau / n;
    t2 *= z / ((2.0 * n - 1.0) * (2.0 * n));
    if (t1 <= tol || t2 <= tol) return n > 1 ? n - 1 : 1;
  }
  return PF_K + 1;
}

// ln of the largest term of the functions' powers of E at thickness h: the maximum of
// h |Im sqrt(a + R E)| over |E| = 1.
__host__ __device__ inline double poly_growth(const PolyRegion& g, double h) {
  const double a = cabs(g.a);
  return h * (g.r <= 2.0 * a ? g.r / (2.0 * sqrt(a)) : sqrt(g.r - a));
}

struct PolyPlan {
  int q, jcap, j, m;  // powers, block limit; blocks and double-angle steps launched
  bool apart;         // a unit's powers may need their diagonals apart
};

// q, and the block limit.  deg > 0: an estimate of the degree the launch's units
// need (they share their period), q is the one with the fewest products, then the
// fewest blocks: degree 11-12 (60 nm slabs of 1 um clips, mixed) takes q = 6, J = 2, 7
// products, 19 (the same, FP64) q = 5, J = 4, 10.  deg = 0, clips of several periods
// in one launch: q from the slab alone, so that a unit's arithmetic does not
// depend on the others; tau0 = d k |eps - 1| / 4 is the pattern's part of tau.  Mixed:
// 7.5 nm slices need degree 5-6 (q = 3: 4 products), 20-30 nm 7-8 (q = 4: 5), 60 nm
// 10-12 (q = 5, J = 2..3: 6-8); FP64: 10-12 (q = 5) and 18-20 (q = 6).
__host__ __device__ inline void poly_shape(int precision, double k, cplx eps_m1, double d, int deg,
                                           int* q, int* jcap) {
  *jcap = precision == EUV_PREC_MIXED ? 4 : 5;
  if (deg > 0) {
    int best = 1 << 30;
    for (int c = 3; c <= PF_Q; ++c) {
      const int j = (deg + c - 1) / c, cost = 8 * (c - 1 + 2 * (j - 1)) + j;
      if (j <= *jcap && cost < best) {
        best = cost;
        *q = c;
      }
    }
    if (best < (1 << 30)) return;
    *q = PF_Q;  // beyond every q's reach: the longest blocks
    return;
  }
  const double tau0 = 0.25 * d * k * cabs(eps_m1);
  if (precision == EUV_PREC_MIXED)
    *q = tau0 < 0.16 ? 3 : (tau0 < 0.5 ? 4 : 5);
  else
    *q = tau0 < 0.2 ? 5 : 6;
}

// Blocks and double-angle steps of one unit: the fewest steps with which jcap
// blocks reach the degree, and of a unit beyond `wide` down to kPolyGrowth, at most m_max.
// Returns false when the degree is not reached.
__host__ __device__ inline bool poly_pick(const PolyRegion& g, double d, double tol, double wide,
                                          int q, int jcap, int m_max, int* j, int* m) {
  const double growth = poly_growth(g, d) > wide ? kPolyGrowth : 1e300;
  for (int mm = 0;; ++mm) {
    const double h = ldexp(d, -mm);
    const int deg = poly_degree(g, h, tol);
    const int jj = (deg + q - 1) / q;
    const bool ok = jj <= jcap && deg <= PF_K;
    if ((ok && poly_growth(g, h) <= growth) || mm >= m_max) {
      *j = ok ? jj : jcap;
      *m = mm;
      return ok;
    }
  }
}

struct PolySlices {
  double k, dx, dy;
  const double* dxs;
  const double* dys;
  int n, lmax, mmax, n_slices, n_units;
  double tol, wide;  // wide: kPolyWide in split-plane products, else without limit
  cplx eps_m1[EUV_MAX_SLICES];
  double leps[EUV_MAX_SLICES];  // |log eps|
  double d[EUV_MAX_SLICES];
  // blocks and steps launched and the steps a unit may take
  int q[EUV_MAX_SLICES], jcap[EUV_MAX_SLICES], j[EUV_MAX_SLICES], m[EUV_MAX_SLICES];
  int m_limit[EUV_MAX_SLICES];
  int m_any;  // the steps of a unit whose spectrum is no pattern's (slab_steps_kernel)
  bool apart[EUV_MAX_SLICES];  // some unit may be wide
};

// Coefficients of block b, function f of (unit, slice): PF_Q complex values, the
// factor of E^(i+1) at i.
__host__ __device__ inline long long poly_coef_at(int n_units, int slice, int unit, int f, int b) {
  return ((((long long)slice * n_units + unit) * 2 + f) * PF_J + b) * PF_Q;
}
// Identity parts [unit] of function f of a slice after t double-angle steps.
__host__ __device__ inline long long poly_id_at(int n_units, int slice, int t, int f) {
  return (((long long)slice * (kMaxSteps + 2) + t) * 2 + f) * n_units;
}

// One CTA of 64 threads per (unit, slice): the ellipse from the unit's own
// orders, the two functions at 64 points of it, their Fourier coefficients there
// (= Chebyshev coefficients times rho^n / 2) and from those the block
// coefficients.  Latency of one small launch for all slices; it replaces the
// three norm / scaling launches per slice of the expansion about 0.
__global__ void __launch_bounds__(PF_SAMPLES)
    poly_coef_kernel(PolySlices p, const double2* spectra, const int* spec_of_unit,
                     const int* lidx, const int* midx, const double* kx0, const double* ky0,
                     const int* polar, double2* coef, double2* ident, double2* shift,
                     double* radius, int* steps, int* blocks, int* wide, int* more, int* status) {
  dependent_begin();
  const int u = blockIdx.x, sl = blockIdx.y, tid = threadIdx.x;
  __shared__ double s_lo[2], s_hi[2], s_km[2];
  __shared__ cplx s_f[2][PF_SAMPLES], s_w[PF_SAMPLES], s_a[2][PF_K + 1];
  const double twopi = 6.283185307179586476925286766559;
  const double gx = twopi / (p.dxs ? p.dxs[u] : p.dx), gy = twopi / (p.dys ? p.dys[u] : p.dy);
  const bool pol_x = polar[u] == 0;
  double lo = 1e300, hi = 0.0, km = 0.0;
  for (int i = tid; i < p.n; i += PF_SAMPLES) {
    const double kx = kx0[u] + gx * lidx[i], ky = ky0[u] + gy * midx[i];
    const double v = kx * kx + ky * ky;
    lo = fmin(lo, v);
    hi = fmax(hi, v);
    km = fmax(km, fabs(pol_x ? kx : ky));
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, off));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, off));
    km = fmax(km, __shfl_xor_sync(0xffffffffu, km, off));
  }
  // Is this the spectrum F of a pattern with values in [0, 1]?  Then F is Hermitian, F(0)
  // lies in [0, 1] and sum |F|^2 <= F(0).  B = sum |F| bounds any other's field of values.
  const int W = (4 * p.lmax + 1) * (4 * p.mmax + 1);
  const double2* F = spectra + ((long long)spec_of_unit[u] * p.n_slices + sl) * W;
  double sum = 0.0, sq = 0.0, skew = 0.0;
#pragma unroll 8
  for (int i = tid; i < W; i += PF_SAMPLES) {
    const double2 a = F[i], b = F[W - 1 - i];
    sum += fabs(a.x) + fabs(a.y);
    sq = fma(a.x, a.x, fma(a.y, a.y, sq));
    skew += fabs(a.x - b.x) + fabs(a.y + b.y);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, off);
    sq += __shfl_xor_sync(0xffffffffu, sq, off);
    skew += __shfl_xor_sync(0xffffffffu, skew, off);
  }
  if ((tid & 31) == 0) {
    s_lo[tid >> 5] = lo;
    s_hi[tid >> 5] = hi;
    s_km[tid >> 5] = km;
    s_f[0][tid >> 5] = mk(sum, sq);
    s_f[1][tid >> 5] = mk(skew, 0.0);
  }
  __syncthreads();
  lo = fmin(s_lo[0], s_lo[1]);
  hi = fmax(s_hi[0], s_hi[1]);
  km = fmax(s_km[0], s_km[1]);
  const cplx fs = s_f[0][0] + s_f[0][1];
  const double bound = fs.x, f0 = F[W / 2].x;
  const bool pattern = s_f[1][0].x + s_f[1][1].x <= 1e-6 && f0 >= -1e-9 && f0 <= 1.0 + 1e-9 &&
                       fs.y <= 1.000001 * f0 + 1e-9;
  __syncthreads();  // s_f is written again
  // every thread takes the same decisions from the same numbers
  double w = (pol_x ? gx * p.lmax : gy * p.mmax) * p.leps[sl] * km;
  if (!pattern) w = 2.0 * bound * w + bound * p.k * p.k * cabs(p.eps_m1[sl]);
  // beyond twice any pattern's (sum |re| + |im| <= sqrt(2 W)), infinite or NaN: flagged
  const bool sane = bound <= 2.0 * sqrt(2.0 * W);
  const PolyRegion g = poly_region(p.k, p.eps_m1[sl], lo, hi, sane ? w : 0.0);
  const int q = p.q[sl], jl = p.j[sl];
  int jb, m;
  bool ok = pattern ? poly_pick(g, p.d[sl], p.tol, p.wide, q, p.jcap[sl], p.m_limit[sl], &jb, &m)
                    : poly_pick(g, p.d[sl], p.tol, p.wide, q, jl, sane ? p.m_any : 0, &jb, &m) && sane;
  if (jb > jl) {  // more blocks than launched
    jb = jl;
    ok = poly_degree(g, ldexp(p.d[sl], -m), 100.0 * p.tol) <= q * jb;
  }
  const double h = ldexp(p.d[sl], -m);
  {
    double sn, cs;
    sincospi(2.0 * tid / PF_SAMPLES, &sn, &cs);
    s_w[tid] = mk(cs, -sn);  // e^{-i theta}
    const cplx dz = g.c * mk(0.5 * (g.rho + 1.0 / g.rho) * cs, 0.5 * (g.rho - 1.0 / g.rho) * sn);
    const cplx r = csqrt_p(g.a + dz), ra = csqrt_p(g.a), rs = r + ra;
    // e^{i h sqrt z} as e^{i h sqrt a} e^{i h (sqrt z - sqrt a)}: the difference
    // without cancellation
    const cplx dphi = (rs.x == 0.0 && rs.y == 0.0) ? mk(0.0, 0.0) : h * cdiv(dz, rs);
    const cplx ep = cexp_(cmul_i(h * ra)) * cexp_(cmul_i(dphi));
    const cplx em = cexp_(-cmul_i(h * ra)) * cexp_(-cmul_i(dphi));
    s_f[0][tid] = 0.5 * (ep + em);
    const cplx x2 = (h * h) * (r * r);
    s_f[1][tid] = cabs1(x2) < 1e-4
                      ? h * (mk(1.0, 0.0) - (1.0 / 6.0) * x2 + (1.0 / 120.0) * (x2 * x2))
                      : cdiv(0.5 * (ep - em), cmul_i(r));
  }
  __syncthreads();
  const int deg = q * jb;
  static_assert(2 * (PF_K + 1) <= PF_SAMPLES && PF_K < 32, "one thread per coefficient");
  if (tid < 2 * (PF_K + 1)) {
    const int f = tid / (PF_K + 1), n = tid % (PF_K + 1);
    cplx s = mk(0.0, 0.0);
    for (int t = 0; t < PF_SAMPLES; ++t) s = s + s_f[f][t] * s_w[(n * t) % PF_SAMPLES];
    // a_n of sum a_n T_n: f^_n = a_n rho^n / 2 (n > 0)
    double e = (n ? 2.0 : 1.0) / PF_SAMPLES;
    for (int t = 0; t < n; ++t) e /= g.rho;
    s_a[f][n] = n <= deg ? e * s : mk(0.0, 0.0);
  }
  __syncthreads();
  // monomial coefficients in E = (z - a)/R: lane i of warp f collects the E^i
  // terms of T_n(E R / c) with the three-term recurrence
  const int f = tid >> 5, lane = tid & 31;
  const cplx ratio = cdiv(mk(g.r, 0.0), g.c);
  double tp = 0.0, tc = lane == 0 ? 1.0 : 0.0;  // T_{n-1}, T_n
  cplx acc = mk(0.0, 0.0);
  for (int n = 0; n <= deg; ++n) {
    acc = acc + tc * s_a[f][n];
    double up = __shfl_up_sync(0xffffffffu, tc, 1);
    if (lane == 0) up = 0.0;
    const double tn = n == 0 ? up : 2.0 * up - tp;
    tp = tc;
    tc = tn;
  }
  for (int t = 0; t < lane && t < PF_K; ++t) acc = acc * ratio;
  double2* out = coef + poly_coef_at(p.n_units, sl, u, f, 0);
  for (int b = 0; b < PF_J; ++b) {
    const int i = lane - 1 - q * b;
    if (lane < PF_Q) out[b * PF_Q + lane] = make_double2(0.0, 0.0);
    __syncwarp();
    if (b < jb && i >= 0 && i < q) out[b * PF_Q + i] = make_double2(acc.x, acc.y);
  }
  if (lane == 0) s_a[f][0] = acc;
  __syncthreads();
  if (tid == 0) {
    const long long t = (long long)sl * p.n_units + u;
    const cplx ia = cmul_i(g.a);
    shift[t] = make_double2(ia.x, ia.y);
    radius[t] = g.r;
    steps[t] = m < p.m[sl] ? m : p.m[sl];
    more[t] = m - steps[t];
    blocks[t] = jb;
    wide[t] = poly_growth(g, p.d[sl]) > p.wide;
    cplx c = s_a[0][0], sn = s_a[1][0];
    for (int i = 0; i <= p.m[sl]; ++i) {
      ident[poly_id_at(p.n_units, sl, i, 0) + u] = make_double2(c.x, c.y);
      ident[poly_id_at(p.n_units, sl, i, 1) + u] = make_double2(sn.x, sn.y);
      if (i < steps[t]) {
        sn = 2.0 * (sn * c);
        c = 2.0 * (c * c) - mk(1.0, 0.0);
      }
    }
    if (!ok) atomicOr(status, EUV_STATUS_STEPS_CLAMPED);
  }
}

// Double-angle steps beyond the launched ones, of units whose spectrum is no pattern's (more
// > 0; the others return at once: 1.5 us per slice).  A cluster of 8 CTAs per unit, S <-
// 2 S C + 2 c0 S + 2 s0 C, C <- 2 C C + 4 c0 C between the pairs [C | S] in a and b, the
// result in a, the identity parts in c0, s0.  Plain FP64 tiles: no caller of this library
// takes them, they keep euv_amp right for any spectrum.
constexpr int SX_CL = 8, SX_T = 32, SX_K = 16;
__global__ void __cluster_dims__(SX_CL, 1, 1) __launch_bounds__(256)
    slab_steps_kernel(int n, const int* more, double2* c0, double2* s0, double2* a, double2* b,
                      long long sp) {
  dependent_begin();
  const int u = blockIdx.y;
  const int steps = more[u];
  if (steps <= 0) return;
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ double2 s_l[2][SX_K][SX_T], s_r[SX_T][SX_K + 1];
  const int rank = (int)cluster.block_rank(), tx = threadIdx.x % SX_T, ty = threadIdx.x / SX_T;
  const long long nn = (long long)n * n;
  const int tiles = (n + SX_T - 1) / SX_T;
  cplx c = mk(c0[u].x, c0[u].y), s = mk(s0[u].x, s0[u].y);
  const double2* src = a + u * sp;
  double2* dst = b + u * sp;
  for (int t = 0; t < steps; ++t) {
    for (int tile = rank; tile < tiles * tiles; tile += SX_CL) {
      const int i = tile % tiles * SX_T + tx, j0 = tile / tiles * SX_T;
      cplx acc[2][4] = {};
      for (int k0 = 0; k0 < n; k0 += SX_K) {
        for (int y = ty; y < SX_K; y += 8)
          for (int f = 0; f < 2; ++f)
            s_l[f][y][tx] = i < n && k0 + y < n ? src[f * nn + (long long)(k0 + y) * n + i]
                                                : make_double2(0.0, 0.0);
        for (int t2 = threadIdx.x; t2 < SX_T * SX_K; t2 += 256) {
          const int k = k0 + t2 % SX_K, j = j0 + t2 / SX_K;
          s_r[t2 / SX_K][t2 % SX_K] =
              k < n && j < n ? src[(long long)j * n + k] : make_double2(0.0, 0.0);
        }
        __syncthreads();
        for (int k = 0; k < SX_K; ++k)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const double2 r = s_r[ty + 8 * e][k];
#pragma unroll
            for (int f = 0; f < 2; ++f)
              acc[f][e] = acc[f][e] + mk(s_l[f][k][tx].x, s_l[f][k][tx].y) * mk(r.x, r.y);
          }
        __syncthreads();
      }
      for (int e = 0; e < 4; ++e) {
        const int j = j0 + ty + 8 * e;
        if (i >= n || j >= n) continue;
        const long long at = (long long)j * n + i;
        const cplx C = mk(src[at].x, src[at].y), S = mk(src[nn + at].x, src[nn + at].y);
        const cplx cn = 2.0 * (acc[0][e] + 2.0 * (c * C));
        const cplx sn = 2.0 * (acc[1][e] + c * S + s * C);
        dst[at] = make_double2(cn.x, cn.y);
        dst[nn + at] = make_double2(sn.x, sn.y);
      }
    }
    s = 2.0 * (s * c);
    c = 2.0 * (c * c) - mk(1.0, 0.0);
    cluster.sync();
    const double2* p = src;
    src = dst;
    dst = const_cast<double2*>(p);
  }
  if (src != a + u * sp)
    for (long long t = rank * 256 + threadIdx.x; t < 2 * nn; t += SX_CL * 256) dst[t] = src[t];
  if (rank == 0 && threadIdx.x == 0) {
    c0[u] = make_double2(c.x, c.y);
    s0[u] = make_double2(s.x, s.y);
  }
}

// Blocks B_b of both functions for b = b0 (and b0 - 1 when NB = 2), [c | s] side
// by side per unit, from E..E^q (one unit's powers nn apart, units sp apart).
// HBM-bound: q reads and 2 NB writes of 16 bytes per element.
template <int Q, int NB>
__global__ void __launch_bounds__(256)
    poly_block_kernel(int n, const double2* pw, long long sp, const double2* coef, int n_units,
                      int slice, int b0, double2* top, double2* low, long long so) {
  dependent_begin();
  __shared__ double2 s_c[NB][2][Q];
  const int u = blockIdx.z, j = blockIdx.x;
  if (threadIdx.x < NB * 2 * Q) {
    const int t = threadIdx.x, i = t % Q, f = (t / Q) % 2, b = t / (2 * Q);
    s_c[b][f][i] = coef[poly_coef_at(n_units, slice, u, f, b0 - b) + i];
  }
  __syncthreads();
  const int i = blockIdx.y * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long nn = (long long)n * n, t = (long long)j * n + i;
  double2 x[Q];
#pragma unroll
  for (int e = 0; e < Q; ++e) x[e] = pw[(long long)u * sp + e * nn + t];
#pragma unroll
  for (int b = 0; b < NB; ++b)
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      cplx v = mk(0.0, 0.0);
#pragma unroll
      for (int e = 0; e < Q; ++e) v = v + mk(s_c[b][f][e].x, s_c[b][f][e].y) * mk(x[e].x, x[e].y);
      (b ? low : top)[(long long)u * so + f * nn + t] = make_double2(v.x, v.y);
    }
}

template <int NB>
static int poly_blocks(int q, int n, const double2* pw, long long sp, const double2* coef, int U,
                       int slice, int b0, double2* top, double2* low, long long so,
                       cudaStream_t stream) {
  const dim3 g((unsigned)n, (unsigned)((n + 255) / 256), U);
  const auto kernel = q == 3   ? poly_block_kernel<3, NB>
                      : q == 4 ? poly_block_kernel<4, NB>
                      : q == 5 ? poly_block_kernel<5, NB>
                               : poly_block_kernel<6, NB>;
  EUV_CUDA_TRY(launch_dependent(kernel, g, dim3(256), 0, stream, n, pw, sp, coef, U, slice, b0, top,
                                low, so));
  EUV_LAUNCH_CHECK();
  return EUV_OK;
}

// ---------------------------------------------------------------- elementwise
// Top interface (klm = diag of the vacuum wave numbers, columns scaled).  With
// c = c0 + C, s = s0 + S, D = a + R E the rows c - i s klm and i D s - c klm are
//   diag(v) + V,  V = C - i S klm,                          v = c0 - i s0 klm
//   diag(w) + W,  W = i R E S + i a S + i R s0 E - C klm,    w = i a s0 - c0 klm
// (W holds i R E S on entry), and M takes the diagonal parts' share of
// P (diag(v) + V) + Q (diag(w) + W); Q = I when null, with W's whole share.
// Batch strides: sc (C, S), sw (E, V, W, M), sp (P, Q).
__global__ void top_rows_kernel(int n, const double* klm, const double2* shift,
                                const double* radius, const double2* c0, const double2* s0,
                                const double2* C, const double2* S, long long sc, const double2* E,
                                double2* V, double2* W, double2* M, long long sw, const double2* P,
                                const double2* Q, long long sp) {
  dependent_begin();
  const int b = blockIdx.z, j = blockIdx.x;
  const int i = blockIdx.y * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long t = (long long)j * n + i;
  const double kl = klm[(long long)b * n + j];
  const cplx ia = mk(shift[b].x, shift[b].y), u0 = mk(c0[b].x, c0[b].y), u1 = mk(s0[b].x, s0[b].y);
  const cplx v = u0 - kl * cmul_i(u1), w = ia * u1 - kl * u0;
  const double2 c2 = C[b * sc + t], s2 = S[b * sc + t], e2 = E[b * sw + t], w2 = W[b * sw + t];
  const double2 p2 = P[b * sp + t];
  const cplx c = mk(c2.x, c2.y), s = mk(s2.x, s2.y);
  const cplx vv = c - kl * cmul_i(s);
  const cplx ww = mk(w2.x, w2.y) + ia * s + (radius[b] * cmul_i(u1)) * mk(e2.x, e2.y) - kl * c;
  cplx m = mk(p2.x, p2.y) * v;
  if (Q != nullptr) {
    const double2 q2 = Q[b * sp + t];
    m = m + mk(q2.x, q2.y) * w;
  } else {
    m = m + ww;
    if (i == j) m = m + w;
  }
  V[b * sw + t] = make_double2(vv.x, vv.y);
  W[b * sw + t] = make_double2(ww.x, ww.y);
  M[b * sw + t] = make_double2(m.x, m.y);
}

// The same for the incident wave of the source columns (klm -> -klm), o =
// src_order[s]: V2[:, s], W2[:, s], and the diagonal parts' share of the right-hand
// side -(P (diag + V2) + Q (diag + W2)) in rhs; zero for empty slots.
__global__ void source_rows_kernel(int n, int nsrc, const int* src_order, const double* klm,
                                   const double2* shift, const double2* c0, const double2* s0,
                                   const double2* C, const double2* S, long long sc,
                                   const double2* V, const double2* W, long long sw,
                                   const double2* P, const double2* Q, long long sp, double2* V2,
                                   double2* W2, double2* rhs, long long sr) {
  dependent_begin();
  const int b = blockIdx.z, s = blockIdx.x;
  const int i = blockIdx.y * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int o = src_order[(long long)b * nsrc + s];
  const long long t = ((long long)b * nsrc + s) * n + i;
  double2* r_out = rhs + b * sr + (long long)s * n + i;
  if (o < 0) {
    V2[t] = W2[t] = *r_out = make_double2(0.0, 0.0);
    return;
  }
  const long long e = (long long)o * n + i;
  const double kl = klm[(long long)b * n + o];
  const cplx ia = mk(shift[b].x, shift[b].y), u0 = mk(c0[b].x, c0[b].y), u1 = mk(s0[b].x, s0[b].y);
  const cplx v = u0 + kl * cmul_i(u1), w = ia * u1 + kl * u0;
  const double2 cv = C[b * sc + e], sv = S[b * sc + e], vv = V[b * sw + e], wv = W[b * sw + e];
  const double2 pv = P[b * sp + e];
  const cplx w2 = mk(wv.x + 2.0 * kl * cv.x, wv.y + 2.0 * kl * cv.y);
  cplx r = mk(pv.x, pv.y) * v;
  if (Q != nullptr) {
    const double2 qv = Q[b * sp + e];
    r = r + mk(qv.x, qv.y) * w;
  } else {
    r = r + w2;
    if (i == o) r = r + w;
  }
  V2[t] = make_double2(vv.x - 2.0 * kl * sv.y, vv.y + 2.0 * kl * sv.x);
  W2[t] = make_double2(w2.x, w2.y);
  *r_out = make_double2(-r.x, -r.y);
}

// Bottom of several slices (Q = I): what of P c + i D s and c + i P s is not a
// product of two matrices,
//   R1 = c0 P + i a S + i R s0 E + i a s0,   R2 = C + i s0 P + c0.
__global__ void bottom_rows_kernel(int n, const double2* shift, const double* radius,
                                   const double2* c0, const double2* s0, const double2* C,
                                   const double2* S, long long sc, const double2* E, long long se,
                                   const double2* P, long long sp, double2* R1, double2* R2,
                                   long long sr) {
  dependent_begin();
  const int b = blockIdx.z, j = blockIdx.x;
  const int i = blockIdx.y * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long t = (long long)j * n + i;
  const cplx ia = mk(shift[b].x, shift[b].y), u0 = mk(c0[b].x, c0[b].y), u1 = mk(s0[b].x, s0[b].y);
  const double2 c2 = C[b * sc + t], s2 = S[b * sc + t], e2 = E[b * se + t], p2 = P[b * sp + t];
  const cplx p = mk(p2.x, p2.y);
  cplx r1 = u0 * p + ia * mk(s2.x, s2.y) + (radius[b] * cmul_i(u1)) * mk(e2.x, e2.y);
  cplx r2 = mk(c2.x, c2.y) + cmul_i(u1) * p;
  if (i == j) {
    r1 = r1 + ia * u1;
    r2 = r2 + u0;
  }
  R1[b * sr + t] = make_double2(r1.x, r1.y);
  R2[b * sr + t] = make_double2(r2.x, r2.y);
}

// Ax[b](i,s) = r x + (1 - r) [i == src_order], r = src_2kz / (2 klm): x is the
// reflected amplitude of a unit wave in order src_order, the caller's 2 kz its
// weight (header.h:1394-1465); zero for empty slots.
__global__ void ax_out_kernel(int n, int nsrc, const int* src_order, const double* src_2kz,
                              const double* klm, const double2* x, long long sx, double2* ax) {
  dependent_begin();
  const int b = blockIdx.z, s = blockIdx.x;
  const int i = blockIdx.y * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long bs = (long long)b * nsrc + s;
  const int o = src_order[bs];
  if (o < 0) {
    ax[bs * n + i] = make_double2(0.0, 0.0);
    return;
  }
  const double r = src_2kz[bs] / (2.0 * klm[(long long)b * n + o]);
  double2 v = x[b * sx + (long long)s * n + i];
  v.x = r * v.x + (i == o ? 1.0 - r : 0.0);
  v.y = r * v.y;
  ax[bs * n + i] = v;
}

// ---------------------------------------------------------------- workspace
struct Bump {
  char* base;
  size_t cap, off;
  bool ok;
  template <typename T>
  T* take(size_t count) {
    size_t bytes = ((count * sizeof(T)) + 255) & ~(size_t)255;
    if (off + bytes > cap) ok = false;
    T* p = reinterpret_cast<T*>(base + off);
    off += bytes;
    return (ok && base) ? p : nullptr;
  }
};

inline unsigned grid1(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

// An LU's zero pivots (info != 0) as EUV_STATUS_SINGULAR in the status word.
__global__ void flag_singular_kernel(const int* info, int n, int* status) {
  dependent_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && info[i] != 0) atomicOr(status, EUV_STATUS_SINGULAR);
}

// GEMM dispatch by precision (FP64 DMMA, or split-FP16x3 tcgen05 tensor cores for
// the bulk products of the mixed form; `status` receives EUV_STATUS_TIMEOUT).
// Gemm reuse flags (mixed form only): the previous call through the same Gemm
// split this unchanged operand in the same role and shape, so its fp16 planes
// in the workspace are current.
constexpr int kReuseA = 1;
constexpr int kReuseB = 2;

// Order count up to which the mixed form multiplies in FP64: a product of split
// planes is three launches of which the two splits and the product's prologue and
// epilogue are latency (22 us at N = 121), the FP64 one 7-9 us.  By N alone, so that
// a unit's arithmetic does not depend on the batch: B200, 256 nm clips at N = 121,
// eight slices, 4 units 2.44 -> 1.34 ms, 16 units 2.53 -> 1.66 ms, 64 units 3.79 ->
// 4.69 ms; at N = 169 4 units gain as much and 48 lose a third, so the line is drawn
// below.  Launches of several periods (the served form) are batches by purpose and
// keep the split planes.
constexpr int kMixedFp64Orders = EUV_MIXED_FP64_ORDERS;

struct Gemm {
  int precision;
  void* mwork;
  size_t mbytes;
  cudaStream_t stream;
  int* status = nullptr;
  int operator()(int m, int n, int k, cplx alpha, const double* scale, const double2* a,
                 long long lda, long long sa, const double2* b, long long ldb, long long sb,
                 cplx beta, double2* c, long long ldc, long long sc, cplx diag, int batch,
                 const int* steps = nullptr, int step = 0, int reuse = 0,
                 const GemmTerms& terms = GemmTerms{}) const {
    if (precision == EUV_PREC_MIXED)
      return gemm_mixed(m, n, k, alpha, scale, a, lda, sa, b, ldb, sb, beta, c, ldc, sc, diag,
                        batch, steps, step, mwork, mbytes, status, stream, reuse, terms);
    return zgemm(m, n, k, alpha, scale, a, lda, sa, b, ldb, sb, beta, c, ldc, sc, diag, batch,
                 steps, step, stream, terms);
  }
};

// Matrix functions for a batch: on return *pc, *ps point to cos / sinc (they
// may be swapped with the temporaries t0, t1).
struct MatfunBufs {
  double2 *P2, *P3, *P4, *T1, *T2;
  double *norm, *h, *h2, *h4;
  int* steps;
  int* capped;
};

int matfun(int n, int batch, const double2* D, const double* thick, double2** pc, double2** ps,
           const MatfunBufs& w, int m_max, const Gemm& gemm, cudaStream_t stream) {
  const long long nn = (long long)n * n;
  const int bs = 256;
  dim3 ge(grid1(nn, bs), batch);
  zero_f64_kernel<<<grid1(batch, 256), 256, 0, stream>>>(w.norm, batch);
  EUV_LAUNCH_CHECK();
  dim3 gn(grid1((long long)n * 32, 256), batch);
  EUV_CUDA_TRY(launch_dependent(norm1_kernel, gn, dim3(256), 0, stream, n, D, w.norm));
  EUV_LAUNCH_CHECK();
  EUV_CUDA_TRY(launch_dependent(scale_kernel, dim3(grid1(batch, 128)), dim3(128), 0, stream, batch,
                                theta_for(gemm.precision), w.norm, thick, m_max, w.steps, w.h, w.h2,
                                w.h4, w.capped));
  EUV_LAUNCH_CHECK();
  const cplx one = mk(1.0, 0.0), zero = mk(0.0, 0.0);
  int rc;
  // P2 = h^4 D D, P3 = h^2 P2 D, P4 = P2 P2
  if ((rc = gemm(n, n, n, one, w.h4, D, n, nn, D, n, nn, zero, w.P2, n, nn, zero, batch))) return rc;
  if ((rc = gemm(n, n, n, one, w.h2, w.P2, n, nn, D, n, nn, zero, w.P3, n, nn, zero, batch, nullptr, 0,
                 kReuseB))) return rc;  // D as B again
  if ((rc = gemm(n, n, n, one, nullptr, w.P2, n, nn, w.P2, n, nn, zero, w.P4, n, nn, zero, batch,
                 nullptr, 0, kReuseA))) return rc;  // P2 as A again
  double2* C = *pc;
  double2* S = *ps;
  EUV_CUDA_TRY(launch_dependent(taylor_prep_kernel, ge, dim3(bs), 0, stream, n, batch, D, w.P2,
                                w.P3, w.P4, w.h, w.h2, C, w.T1, S, w.T2));
  EUV_LAUNCH_CHECK();
  if ((rc = gemm(n, n, n, one, nullptr, w.P4, n, nn, w.T1, n, nn, one, C, n, nn, zero, batch))) return rc;
  if ((rc = gemm(n, n, n, one, nullptr, w.P4, n, nn, w.T2, n, nn, one, S, n, nn, zero, batch,
                 nullptr, 0, kReuseA))) return rc;  // P4 as A again
  // double-angle steps; entries with fewer steps copy through (C = A)
  double2* tS = w.P2;
  double2* tC = w.P3;
  for (int step = 0; step < m_max; ++step) {
    if ((rc = gemm(n, n, n, mk(2.0, 0.0), nullptr, S, n, nn, C, n, nn, zero, tS, n, nn, zero,
                   batch, w.steps, step)))
      return rc;
    if ((rc = gemm(n, n, n, mk(2.0, 0.0), nullptr, C, n, nn, C, n, nn, zero, tC, n, nn,
                   mk(-1.0, 0.0), batch, w.steps, step, kReuseB)))  // C as B again
      return rc;
    double2* t = S;
    S = tS;
    tS = t;
    t = C;
    C = tC;
    tC = t;
  }
  *pc = C;
  *ps = S;
  return EUV_OK;
}

// Launch shape of a slice's polynomials: q of the slab, and the blocks and
// double-angle steps of the widest ellipse any unit of the descriptor can have
// (smallest period, incidence up to k0_max on both axes).
static PolyPlan poly_plan(const euv_amp_desc* d, int slice, double tol, double wide) {
  const double twopi = 6.283185307179586476925286766559;
  const double gx = twopi / d->dx, gy = twopi / d->dy;
  const double k0 = d->k0_max > 0 ? d->k0_max : d->k;
  const double kx = k0 + gx * d->lmax, ky = k0 + gy * d->mmax;
  const cplx e = mk(d->eabs[slice].re, d->eabs[slice].im), em1 = e - mk(1.0, 0.0);
  const double leps = hypot(0.5 * log(e.x * e.x + e.y * e.y), atan2(e.y, e.x));
  const double wx = gx * d->lmax * kx, wy = gy * d->mmax * ky;
  const PolyRegion g = poly_region(d->k, em1, 0.0, kx * kx + ky * ky, leps * (wx > wy ? wx : wy));
  const int limit = d->m_max > 0 && d->m_max < kMaxSteps ? d->m_max : kMaxSteps;
  PolyPlan r;
  int deg = 0;
  if (!d->d_dx && !d->d_dy) {
    // degree of a typical unit: incidence along one axis only, and the corners of
    // the order box only if the set holds them
    const double lx = gx * d->lmax, ly = gy * d->mmax;
    const bool box = d->n_orders == (2 * d->lmax + 1) * (2 * d->mmax + 1);
    const double ax = kx * kx + (box ? ly * ly : 0.0), ay = ky * ky + (box ? lx * lx : 0.0);
    const PolyRegion t = poly_region(d->k, em1, 0.0, ax > ay ? ax : ay, leps * (wx > wy ? wx : wy));
    double h = d->dabs[slice];
    if (poly_growth(t, h) > wide)
      for (int m = 0; m < limit && poly_growth(t, h) > kPolyGrowth; ++m) h *= 0.5;
    deg = poly_degree(t, h, tol);
    if (deg > PF_K) deg = 0;
  }
  poly_shape(d->precision, d->k, em1, d->dabs[slice], deg, &r.q, &r.jcap);
  poly_pick(g, d->dabs[slice], tol, wide, r.q, r.jcap, limit, &r.j, &r.m);
  r.apart = poly_growth(g, d->dabs[slice]) > wide;
  if (r.m > 0) r.j = r.jcap;  // a unit that needs fewer steps may need all the blocks
  return r;
}

// Factors of the Euler product for (I - E)^-1, E = diag(kp/k) Sigma diag(kp/k).
// A finite section of the Toeplitz operator of 1/eps(x) has 2-norm at most
// sup |1/eps| = max(1, 1/|eps_abs|), so ||E||_2 <= (max|kp|/k)^2 max(1, 1/|eps|).
// Returns the F with ||E||^(2^F) <= 1e-7, or 0 (use LU) when the bound is weak.
static int euler_factors(const euv_amp_desc* d) {
  const double twopi = 6.283185307179586476925286766559;
  const double k0 = d->k0_max > 0 ? d->k0_max : d->k;
  const double kpx = k0 + twopi * (d->lmax + 1) / d->dx;
  const double kpy = k0 + twopi * (d->mmax + 1) / d->dy;
  const double kp = kpx > kpy ? kpx : kpy;
  double sup = 1.0;
  for (int n = 0; n < d->n_slices; ++n) {
    const double a = sqrt(d->eabs[n].re * d->eabs[n].re + d->eabs[n].im * d->eabs[n].im);
    if (1.0 / a > sup) sup = 1.0 / a;
  }
  const double e = (kp / d->k) * (kp / d->k) * sup;
  if (!(e < 0.5)) return 0;
  // The product serves the mixed form only, whose split-FP16x3 products carry ~1e-6
  // relative error each: a truncation ||E||^(2^F) <= 1e-7 stays below that.
  // the product of F factors is sum_{j < 2^F} E^j: truncation ||E||^(2^F)
  int f = 1;
  double v = e * e;  // ||E||^(2^f)
  while (v > 1e-7 && f < 8) {
    v = v * v;
    ++f;
  }
  return f;
}

// All workspace carving in one place so the size query and the run agree.
struct AmpWork {
  double2 *pw, *pair[3];  // per unit: 6 powers, three pairs of N^2 matrices
  double2 *adm, *V2, *W2, *coef, *ident, *shift;
  double *klm, *radius;
  int *steps, *blocks, *wide, *more, *ipiv, *info, *capped;
  void* mwork;
  size_t mbytes;
};

static bool carve(const euv_amp_desc* d, Bump& bp, AmpWork& w) {
  const long long N = d->n_orders, U = d->n_units, nn = N * N, NS = d->n_slices;
  const long long cols = U * N * (d->n_src > 0 ? d->n_src : 1);
  w.pw = bp.take<double2>(6 * U * nn);
  for (int i = 0; i < 3; ++i) w.pair[i] = bp.take<double2>(2 * U * nn);
  w.adm = bp.take<double2>(U * N);
  w.V2 = bp.take<double2>(cols);
  w.W2 = bp.take<double2>(cols);
  w.coef = bp.take<double2>(NS * U * 2 * PF_J * PF_Q);
  w.ident = bp.take<double2>(NS * U * 2 * (kMaxSteps + 2));
  w.shift = bp.take<double2>(NS * U);
  w.klm = bp.take<double>(U * N);
  w.radius = bp.take<double>(NS * U);
  w.steps = bp.take<int>(NS * U);
  w.blocks = bp.take<int>(NS * U);
  w.wide = bp.take<int>(NS * U);
  w.more = bp.take<int>(NS * U);
  w.ipiv = bp.take<int>(U * N);
  w.info = bp.take<int>(U);
  w.capped = bp.take<int>(1);
  // the mixed products are N x N x N, N x 2N x N for the two functions together,
  // and N x n_src x N for the source columns
  const long long ncol = d->n_src > 2 * N ? d->n_src : 2 * N;
  w.mbytes = d->precision == EUV_PREC_MIXED ? gemm_mixed_workspace_bytes((int)N, (int)ncol, (int)N, (int)U) : 0;
  w.mwork = w.mbytes ? bp.take<char>(w.mbytes) : nullptr;
  return bp.ok;
}

static int check_desc(const euv_amp_desc* d) {
  if (!d) return 0;
  if (d->n_orders <= 0 || d->n_units <= 0 || d->lmax < 0 || d->mmax < 0 || d->n_slices <= 0 ||
      d->n_slices > EUV_MAX_SLICES || d->n_src < 0 || d->k <= 0 || d->dx <= 0 || d->dy <= 0 ||
      !d->d_lindex || !d->d_mindex || !d->d_kx0 || !d->d_ky0 || !d->d_polar || !d->d_spec ||
      (d->n_src > 0 && (!d->d_src_order || !d->d_src_2kz)) ||
      (d->precision != EUV_PREC_FP64 && d->precision != EUV_PREC_MIXED) || d->euler_f < -1 ||
      d->euler_f > 8)
    return 0;
  for (int n = 0; n < d->n_slices; ++n)
    if (!(d->dabs[n] >= 0.0) || (d->eabs[n].re == 0.0 && d->eabs[n].im == 0.0)) return 0;
  return 1;
}

}  // namespace euv

using namespace euv;

extern "C" int euv_amp_euler_factors(const euv_amp_desc* d) {
  if (!d || !check_desc(d)) {
    euv_set_error("euv_amp_euler_factors: invalid descriptor");
    return -2;
  }
  if (d->precision != EUV_PREC_MIXED) return 0;
  if (d->euler_f != 0) return d->euler_f;
  const int f = euler_factors(d);
  return f > 0 ? f : -1;
}

extern "C" size_t euv_amp_workspace_bytes(const euv_amp_desc* d) {
  if (!check_desc(d)) return 0;
  Bump bp{nullptr, (size_t)-1, 0, true};
  AmpWork w;
  carve(d, bp, w);
  return bp.off;
}

static cplx clog_host(euv_c64 e) {
  return mk(0.5 * log(e.re * e.re + e.im * e.im), atan2(e.im, e.re));
}

extern "C" int euv_amp(const euv_amp_desc* d, const euv_c64* d_spectra, euv_c64* d_ax,
                       void* d_work, size_t work_bytes, void* stream_) {
  if (!check_desc(d) || !d_spectra || !d_ax) {
    euv_set_error("euv_amp: invalid descriptor or null buffer");
    return EUV_ERR_BAD_ARG;
  }
  cudaStream_t stream = (cudaStream_t)stream_;
  Bump bp{reinterpret_cast<char*>(d_work), work_bytes, 0, true};
  AmpWork w;
  if (!d_work || !carve(d, bp, w)) {
    euv_set_error("euv_amp: workspace too small (%zu bytes given, %zu needed)", work_bytes,
                  euv_amp_workspace_bytes(d));
    return EUV_ERR_WORKSPACE;
  }
  const int N = d->n_orders, U = d->n_units, NS = d->n_slices;
  const long long nn = (long long)N * N;
  const int bs = 256;
  const dim3 gdg((unsigned)N, (unsigned)((N + bs - 1) / bs), U);  // build_dg: column, rows, unit
  const cplx one = mk(1.0, 0.0), zero = mk(0.0, 0.0);
  // device-detected conditions go to the caller's status word, else to a
  // workspace word nobody reads
  int* status = d->d_status ? d->d_status : w.capped;
  const bool small = N <= kMixedFp64Orders && !d->d_dx && !d->d_dy;
  Gemm gemm{small ? EUV_PREC_FP64 : d->precision, w.mwork, w.mbytes, stream, status};
  int rc;

  if (!d->d_status) EUV_CUDA_TRY(cudaMemsetAsync(w.capped, 0, sizeof(int), stream));
  SliceParams sp;
  sp.k = d->k;
  sp.dx = d->dx;
  sp.dy = d->dy;
  sp.dxs = d->d_dx;
  sp.dys = d->d_dy;
  sp.n = N;
  sp.lmax = d->lmax;
  sp.mmax = d->mmax;
  sp.lr2 = 4 * d->lmax + 1;
  sp.mr2 = 4 * d->mmax + 1;
  sp.n_slices = NS;
  auto slice_params = [&](int n) {
    SliceParams q = sp;
    q.slice = n;
    cplx e = fromc(d->eabs[n]);
    q.eps_m1 = e - mk(1.0, 0.0);
    q.sig_m1 = cdiv(mk(1.0, 0.0), e) - mk(1.0, 0.0);
    q.logeps = clog_host(d->eabs[n]);
    return q;
  };

  StackParams stp;
  stp.k = d->k;
  stp.emo = fromc(d->stack.eps_mo);
  stp.esi = fromc(d->stack.eps_si);
  stp.eru = fromc(d->stack.eps_ru);
  stp.emosi2 = fromc(d->stack.eps_mosi2);
  stp.erusi = fromc(d->stack.eps_rusi);
  stp.esio2 = fromc(d->stack.eps_sio2);
  stp.dmo = d->stack.d_mo;
  stp.dmosi = d->stack.d_mosi;
  stp.dsi = d->stack.d_si;
  stp.dsimo = d->stack.d_simo;
  stp.dsiru = d->stack.d_siru;
  stp.dru = d->stack.d_ru;
  stp.nml = d->stack.nml;
  stp.dx = d->dx;
  stp.dy = d->dy;
  stp.dxs = d->d_dx;
  stp.dys = d->d_dy;
  stp.n = N;
  multilayer_kernel<<<grid1((long long)N * U, 128), 128, 0, stream>>>(
      stp, d->d_lindex, d->d_mindex, d->d_kx0, d->d_ky0, d->d_polar, w.adm, w.klm, U);
  EUV_LAUNCH_CHECK();

  const double2* spec = reinterpret_cast<const double2*>(d_spectra);
  // polynomial shapes of the slices, and the units' coefficients in one launch
  PolySlices ps;
  ps.k = d->k;
  ps.dx = d->dx;
  ps.dy = d->dy;
  ps.dxs = d->d_dx;
  ps.dys = d->d_dy;
  ps.n = N;
  ps.lmax = d->lmax;
  ps.mmax = d->mmax;
  ps.n_slices = NS;
  ps.n_units = U;
  ps.tol = d->precision == EUV_PREC_MIXED ? kPolyTolMixed : kPolyTolFp64;
  ps.m_any = d->m_max > 0 && d->m_max < kMaxSteps ? d->m_max : kMaxSteps;
  ps.wide = gemm.precision == EUV_PREC_MIXED ? kPolyWide : 1e300;
  for (int n = 0; n < NS; ++n) {
    const PolyPlan r = poly_plan(d, n, ps.tol, ps.wide);
    const SliceParams q = slice_params(n);
    ps.eps_m1[n] = q.eps_m1;
    ps.leps[n] = cabs(q.logeps);
    ps.d[n] = d->dabs[n];
    ps.q[n] = r.q;
    ps.jcap[n] = r.jcap;
    ps.j[n] = r.j;
    ps.m[n] = r.m;
    ps.apart[n] = r.apart;
    ps.m_limit[n] = d->m_max > 0 && d->m_max < r.m ? d->m_max : r.m;
  }
  EUV_CUDA_TRY(launch_dependent(poly_coef_kernel, dim3(U, NS), dim3(PF_SAMPLES), 0, stream, ps,
                                spec, d->d_spec, d->d_lindex, d->d_mindex, d->d_kx0, d->d_ky0, d->d_polar, w.coef,
                                w.ident, w.shift, w.radius, w.steps, w.blocks, w.wide,
                                w.more, status));
  EUV_LAUNCH_CHECK();

  // Mixed form: G^-1 by the Euler product (I - E)^-1 = prod_f (I + E^(2^f)),
  // f < euler_f, when the config bound on ||E||_2 makes it converge fast.
  const int euler_f = d->precision != EUV_PREC_MIXED ? 0
                      : d->euler_f > 0                ? d->euler_f
                      : d->euler_f < 0                ? 0
                                                      : euler_factors(d);
  // a batch of N-row matrices: first element and batch stride
  struct Mat {
    double2* p;
    long long s;
  };
  // powers of E side by side per unit; pairs: [c | s], its other buffer, [P | Q]
  Mat pw[6], cs[2] = {{w.pair[0], 2 * nn}, {w.pair[1], 2 * nn}}, pq = {w.pair[2], 2 * nn};
  for (int i = 0; i < 6; ++i) pw[i] = Mat{w.pw + i * nn, 6 * nn};
  auto build = [&](int slice, const Mat* E, const Mat* G, int want_g) -> int {
    EUV_CUDA_TRY(launch_dependent(build_dg_kernel, gdg, bs, 0, stream, slice_params(slice), spec,
                                  d->d_spec, d->d_lindex, d->d_mindex, d->d_kx0, d->d_ky0,
                                  d->d_polar, w.adm, w.shift + (size_t)slice * U,
                                  w.radius + (size_t)slice * U, E ? E->p : nullptr, E ? E->s : 0,
                                  G ? G->p : nullptr, G ? G->s : 0, want_g));
    EUV_LAUNCH_CHECK();
    return EUV_OK;
  };
  // C = alpha scale A B + beta Cin (C itself unless given) + ..., N x n x N
  struct Term {
    const Mat* cin = nullptr;
    const double2* beta_b = nullptr;
    const Mat* cin2 = nullptr;
    const double2* beta2_b = nullptr;
    cplx beta2 = mk(1.0, 0.0);
    const int* need = nullptr;
    int need_above = 0;
    const int* apart = nullptr;
  };
  auto mul = [&](cplx alpha, const double* scale, const Mat& A, const Mat& B, cplx beta,
                 const Mat& C, int reuse, const Term& x = Term{}, int n = 0) -> int {
    GemmTerms t;
    t.cin = x.cin ? x.cin->p : C.p;
    t.scin = x.cin ? x.cin->s : C.s;
    t.beta_b = x.beta_b;
    t.cin2 = x.cin2 ? x.cin2->p : nullptr;
    t.scin2 = x.cin2 ? x.cin2->s : 0;
    t.beta2 = make_double2(x.beta2.x, x.beta2.y);
    t.beta2_b = x.beta2_b;
    t.need = x.need;
    t.need_above = x.need_above;
    t.apart = x.apart;
    t.three = true;
    return gemm(N, n > 0 ? n : N, N, alpha, scale, A.p, N, A.s, B.p, N, B.s, beta, C.p, N, C.s,
                zero, U, nullptr, 0, reuse, t);
  };
  auto swap = [](Mat& a, Mat& b) {
    const Mat t = a;
    a = b;
    b = t;
  };
  // c - c0 and s - s0 of slice n, side by side per unit, in cs[0] on return; E in pw[0]
  auto slab = [&](int n) -> int {
    const int q = ps.q[n], J = ps.j[n], m = ps.m[n];
    int r2;
    // E^2; [E^3 | E^4] = E^2 [E | E^2]; [E^5 | E^6] = E^2 [E^3 | E^4]
    Term apart;
    if (ps.apart[n]) apart.apart = w.wide + (size_t)n * U;
    if ((r2 = mul(one, nullptr, pw[0], pw[0], zero, pw[1], 0, apart))) return r2;
    if ((r2 = mul(one, nullptr, pw[1], pw[0], zero, pw[2], 0, apart, q > 3 ? 2 * N : N)))
      return r2;
    if (q > 4 && (r2 = mul(one, nullptr, pw[1], pw[2], zero, pw[4], kReuseA, apart,
                           q > 5 ? 2 * N : N)))
      return r2;
    const double2* pb = pw[0].p;
    if (J > 1) {
      if ((r2 = poly_blocks<2>(q, N, pb, 6 * nn, w.coef, U, n, J - 1, cs[0].p, cs[1].p, 2 * nn, stream)))
        return r2;
    } else if ((r2 = poly_blocks<1>(q, N, pb, 6 * nn, w.coef, U, n, 0, cs[0].p, nullptr, 2 * nn, stream))) {
      return r2;
    }
    for (int b = J - 2; b >= 0; --b) {
      if (b < J - 2 &&
          (r2 = poly_blocks<1>(q, N, pb, 6 * nn, w.coef, U, n, b, cs[1].p, nullptr, 2 * nn, stream)))
        return r2;
      // units whose ellipse needs no block above b hold B_b already
      Term x;
      x.need = w.blocks + (size_t)n * U;
      x.need_above = b + 1;
      if ((r2 = mul(one, nullptr, pw[q - 1], cs[0], one, cs[1], b < J - 2 ? kReuseA : 0, x, 2 * N)))
        return r2;
      swap(cs[0], cs[1]);
    }
    // double-angle steps s <- 2 s c, c <- 2 c^2 - I on the parts beside the
    // identity: S <- 2 S C + 2 c0 S + 2 s0 C, C <- 2 C C + 4 c0 C; units with
    // fewer steps copy through
    const int* st = w.steps + (size_t)n * U;
    for (int step = 0; step < m; ++step) {
      const double2 *c = cs[0].p, *s = cs[0].p + nn;
      GemmTerms t;
      t.cin = s;
      t.scin = t.scin2 = 2 * nn;
      t.three = true;
      t.paired = (step | 1) < m;  // an odd count ends with a step that all units enter
      t.beta_b = w.ident + poly_id_at(U, n, step, 0);
      t.cin2 = c;
      t.beta2 = make_double2(2.0, 0.0);
      t.beta2_b = w.ident + poly_id_at(U, n, step, 1);
      if ((r2 = gemm(N, N, N, mk(2.0, 0.0), nullptr, s, N, 2 * nn, c, N, 2 * nn, mk(2.0, 0.0),
                     cs[1].p + nn, N, 2 * nn, zero, U, st, step, 0, t)))
        return r2;
      t.cin = c;
      t.cin2 = nullptr;
      if ((r2 = gemm(N, N, N, mk(2.0, 0.0), nullptr, c, N, 2 * nn, c, N, 2 * nn, mk(4.0, 0.0),
                     cs[1].p, N, 2 * nn, zero, U, st, step, kReuseB, t)))  // c as B again
        return r2;
      swap(cs[0], cs[1]);
    }
    EUV_CUDA_TRY(launch_dependent(slab_steps_kernel, dim3(SX_CL, U), dim3(256), 0, stream, N,
                                  w.more + (size_t)n * U, w.ident + poly_id_at(U, n, m, 0),
                                  w.ident + poly_id_at(U, n, m, 1), cs[0].p, cs[1].p, 2 * nn));
    EUV_LAUNCH_CHECK();
    return EUV_OK;
  };
  // The boundary relation P X + Q Y = 0 of the fields at the top of the slices
  // done so far, carried upwards (rows combine, so no interface matrix is
  // inverted): at the cap Y2 = diag(adm) G X2, i.e. P = -diag(adm) G, Q = I;
  // through a slice X2 = c X1 + i s Y1, Y2 = i D s X1 + c Y1, so
  //   P <- P c + i Q D s,   Q <- Q c + i P s,   D = a + R E.
  const cplx pi_ = mk(0.0, 1.0), m1 = mk(-1.0, 0.0);
  for (int n = NS - 1; n >= 0; --n) {
    const bool bottom = (n == NS - 1), top = (n == 0);
    const Mat P = pq, Q{pq.p + nn, 2 * nn};
    if (!bottom && d->refresh_sigma) {
      // the slices' own 1/eps: X of slice n+1 is G_{n+1}^-1 G_n times X of slice
      // n, so P <- P G_{n+1}^-1 G_n
      Mat E = pw[0], En = pw[1], cur = P;
      if (euler_f > 0) {
        // P (I + E)(I + E^2)(I + E^4)... (I - E_n): both G are i k (I - E)
        if ((rc = build(n + 1, nullptr, &E, 2))) return rc;
        for (int f = 0; f < euler_f; ++f) {
          const Mat dst = pw[2 + (f & 1)];
          if ((rc = mul(one, nullptr, cur, E, one, dst, 0, Term{&cur}))) return rc;
          cur = dst;
          if (f + 1 < euler_f) {
            if ((rc = mul(one, nullptr, E, E, zero, En, kReuseB))) return rc;  // E as B again
            swap(E, En);
          }
        }
        if ((rc = build(n, nullptr, &En, 2))) return rc;
        if ((rc = mul(m1, nullptr, cur, En, one, P, 0, Term{&cur}))) return rc;
      } else {
        if ((rc = build(n + 1, nullptr, &E, 1))) return rc;
        if ((rc = build(n, nullptr, &En, 1))) return rc;
        if ((rc = lu_factor(N, E.p, N, E.s, w.ipiv, w.info, U, stream))) return rc;
        EUV_CUDA_TRY(launch_dependent(flag_singular_kernel, dim3(grid1(U, 256)), dim3(256), 0,
                                      stream, w.info, U, status));
        EUV_LAUNCH_CHECK();
        if ((rc = lu_solve(N, N, E.p, N, E.s, w.ipiv, En.p, N, En.s, U, stream))) return rc;
        if ((rc = mul(one, nullptr, P, En, zero, pw[2], 0))) return rc;
        EUV_CUDA_TRY(cudaMemcpy2DAsync(P.p, P.s * sizeof(double2), pw[2].p, pw[2].s * sizeof(double2),
                                       nn * sizeof(double2), U, cudaMemcpyDeviceToDevice, stream));
      }
    }
    // bottom slice sigma is used for every slice unless refresh_sigma (header.h:1327-1353)
    if ((rc = build(n, &pw[0], bottom ? &P : nullptr, bottom ? 3 : 0))) return rc;
    if ((rc = slab(n))) return rc;
    const Mat C = cs[0], S{cs[0].p + nn, 2 * nn}, E = pw[0];
    const double* rad = w.radius + (size_t)n * U;
    const double2* ia = w.shift + (size_t)n * U;
    // c = c0 + C, s = s0 + S, D = a + R E
    const double2* c0 = w.ident + poly_id_at(U, n, ps.m[n], 0);
    const double2* s0 = w.ident + poly_id_at(U, n, ps.m[n], 1);
    if (top) {
      // Top interface: X1 = b + e, Y1 = klm (e - b) for incident e and reflected
      // b (header.h:1355-1465), so M b = rhs e with
      //   M = P (c - i s klm) + Q (i D s - c klm),
      //   rhs = -(P (c + i s klm) + Q (i D s + c klm)).
      const int ns = d->n_src;
      const Mat V = pw[1], W = pw[2], M = pw[3];  // the powers above E are free now
      const long long sn = (long long)N * ns;
      // the right-hand sides stand behind M's columns (in the next two buffers), so
      // that the factorisation carries them along; more than fit are solved apart
      const bool behind = ns <= 2 * N;
      const Mat V2{w.V2, sn}, W2{w.W2, sn};
      const Mat ax = behind ? pw[4] : Mat{reinterpret_cast<double2*>(d_ax), sn};
      const double2* Qp = bottom ? nullptr : Q.p;
      if ((rc = mul(pi_, rad, E, S, zero, W, 0))) return rc;
      EUV_CUDA_TRY(launch_dependent(top_rows_kernel, gdg, dim3(bs), 0, stream, N, w.klm, ia, rad,
                                    c0, s0, C.p, S.p, C.s, E.p, V.p, W.p, M.p, E.s, P.p, Qp, P.s));
      EUV_LAUNCH_CHECK();
      const dim3 gs((unsigned)ns, (unsigned)((N + bs - 1) / bs), U);
      if (ns > 0) {
        EUV_CUDA_TRY(launch_dependent(source_rows_kernel, gs, dim3(bs), 0, stream, N, ns,
                                      d->d_src_order, w.klm, ia, c0, s0, C.p, S.p, C.s, V.p, W.p,
                                      V.s, P.p, Qp, P.s, V2.p, W2.p, ax.p, ax.s));
        EUV_LAUNCH_CHECK();
      }
      if ((rc = mul(one, nullptr, P, V, one, M, 0))) return rc;
      if (ns > 0 && (rc = mul(m1, nullptr, P, V2, one, ax, kReuseA, Term{}, ns))) return rc;
      if (!bottom) {
        if ((rc = mul(one, nullptr, Q, W, one, M, 0))) return rc;
        if (ns > 0 && (rc = mul(m1, nullptr, Q, W2, one, ax, kReuseA, Term{}, ns))) return rc;
      }
      if ((rc = lu_factor(N, M.p, N, M.s, w.ipiv, w.info, U, stream, behind ? ns : 0,
                          behind ? d->d_src_order : nullptr, ns)))
        return rc;
      EUV_CUDA_TRY(launch_dependent(flag_singular_kernel, dim3(grid1(U, 256)), dim3(256), 0, stream,
                                    w.info, U, status));
      EUV_LAUNCH_CHECK();
      if (ns > 0) {
        // CTAs of empty source slots only (order < 0, zero columns) return, as above
        if ((rc = behind ? lu_back(N, ns, M.p, N, M.s, ax.p, N, ax.s, U, stream, d->d_src_order, ns)
                         : lu_solve(N, ns, M.p, N, M.s, w.ipiv, ax.p, N, ax.s, U, stream,
                                    d->d_src_order, ns)))
          return rc;
        EUV_CUDA_TRY(launch_dependent(ax_out_kernel, gs, dim3(bs), 0, stream, N, ns, d->d_src_order,
                                      d->d_src_2kz, w.klm, ax.p, ax.s,
                                      reinterpret_cast<double2*>(d_ax)));
        EUV_LAUNCH_CHECK();
      }
      return EUV_OK;
    }
    const Mat R1 = cs[1], R2{cs[1].p + nn, 2 * nn};
    if (bottom) {
      // Q = I: R1 = P c + i D s, R2 = c + i P s
      EUV_CUDA_TRY(launch_dependent(bottom_rows_kernel, gdg, dim3(bs), 0, stream, N, ia, rad, c0,
                                    s0, C.p, S.p, C.s, E.p, E.s, P.p, P.s, R1.p, R2.p, R1.s));
      EUV_LAUNCH_CHECK();
      if ((rc = mul(pi_, rad, E, S, one, R1, 0))) return rc;
      if ((rc = mul(pi_, nullptr, P, S, one, R2, kReuseB))) return rc;  // S as B again
      if ((rc = mul(one, nullptr, P, C, one, R1, kReuseA))) return rc;  // P as A again
    } else {
      // T = Q s, R2 = Q c + i P s, R1 = P c + i T D
      const Mat T = pw[1];
      if ((rc = mul(one, nullptr, Q, S, one, T, 0, Term{&Q, s0}))) return rc;
      if ((rc = mul(one, nullptr, Q, C, one, R2, kReuseA, Term{&Q, c0, &P, s0, pi_}))) return rc;
      if ((rc = mul(one, nullptr, P, C, one, R1, kReuseB, Term{&P, c0, &T, ia}))) return rc;
      if ((rc = mul(pi_, nullptr, P, S, one, R2, kReuseA))) return rc;  // P as A again
      if ((rc = mul(pi_, rad, T, E, one, R1, 0))) return rc;
    }
    swap(pq, cs[1]);
  }
  return EUV_OK;
}

// ------------------------------------------------------------------ spectrum
extern "C" size_t euv_mask_spectrum_workspace_bytes(int n_masks, int ndivx, int ndivy, int fdivx,
                                                    int fdivy, int lh, int mh) {
  (void)fdivx;
  (void)fdivy;
  const size_t mr = 2 * (size_t)mh + 1, lp = (size_t)lh + 1;
  Bump bp{nullptr, (size_t)-1, 0, true};
  bp.take<double>((size_t)ndivx * 2 * lp);
  bp.take<double2>((size_t)ndivy * mr);
  const size_t nm = n_masks > 1 ? n_masks : 1;
  bp.take<double2>(nm * lp * ndivy);
  bp.take<double2>(nm * (size_t)spectrum_parts(ndivy) * lp * mr);
  bp.take<char>(256);  // the run's alignment slack between the two arrays
  return bp.off;
}

template <int NB>
static int launch_spectrum_rows(const uint8_t* bits, long long mask_bytes, int ndivx, int ndivy,
                                int lh, int tiles, int masks, const double* W, double2* T,
                                cudaStream_t stream) {
  static int done[64];
  constexpr size_t sm = spectrum_smem<NB>();
  EUV_CUDA_TRY(ensure_smem(spectrum_rows_kernel<NB>, (int)sm, done));
  const dim3 g(SP_CL * ((ndivy + SP_ROWS - 1) / SP_ROWS), tiles, masks);
  EUV_CUDA_TRY(launch_dependent(spectrum_rows_kernel<NB>, g, dim3(256), sm, stream, bits,
                                mask_bytes, ndivx, ndivy, lh, W, T));
  EUV_LAUNCH_CHECK();
  return EUV_OK;
}

// Masks are transformed in groups that fit the workspace (all of them when it
// was sized by euv_mask_spectrum_workspace_bytes for n_masks): three launches per
// group after the two twiddle tables.
extern "C" int euv_mask_spectrum(const uint8_t* d_bits, int n_masks, int ndivx, int ndivy,
                                 int fdivx, int fdivy, int lh, int mh, int select_vacuum,
                                 int y_offset, euv_c64* d_out, void* d_work, size_t work_bytes, void* stream_) {
  if (!d_bits || !d_out || n_masks < 0 || ndivx <= 0 || ndivy <= 0 || fdivx <= 0 || fdivy <= 0 ||
      fdivx % ndivx || fdivy % ndivy || lh < 0 || mh < 0 || 2 * lh + 1 > fdivx ||
      2 * mh + 1 > fdivy || ((long long)ndivx * ndivy) % 8) {
    euv_set_error("euv_mask_spectrum: bad arguments");
    return EUV_ERR_BAD_ARG;
  }
  cudaStream_t stream = (cudaStream_t)stream_;
  const int lp = lh + 1, lr = 2 * lh + 1, mr = 2 * mh + 1;
  const int meshx = fdivx / ndivx, meshy = fdivy / ndivy;
  Bump bp{reinterpret_cast<char*>(d_work), work_bytes, 0, true};
  double* Wx = bp.take<double>((size_t)ndivx * 2 * lp);
  double2* Wy = bp.take<double2>((size_t)ndivy * mr);
  const int parts = spectrum_parts(ndivy);
  const size_t t_bytes = (size_t)lp * ndivy * sizeof(double2);
  const size_t p_bytes = (size_t)parts * lp * mr * sizeof(double2);
  const size_t left = bp.ok && work_bytes > bp.off + 256 ? work_bytes - bp.off - 256 : 0;
  long long group = (long long)(left / (t_bytes + p_bytes));
  if (group > 65535) group = 65535;  // grid z limit
  if (!d_work || !bp.ok || group < 1) {
    euv_set_error("euv_mask_spectrum: workspace too small");
    return EUV_ERR_WORKSPACE;
  }
  double2* T = reinterpret_cast<double2*>(reinterpret_cast<char*>(d_work) + bp.off);
  spectrum_wx_kernel<<<grid1((long long)ndivx * lp, 256), 256, 0, stream>>>(
      ndivx, meshx, fdivx, lh, Wx);
  EUV_LAUNCH_CHECK();
  EUV_CUDA_TRY(launch_dependent(spectrum_wy_kernel, dim3(grid1((long long)ndivy * mr, 256)),
                                dim3(256), 0, stream, ndivy, meshy, fdivy, y_offset, mh, Wy));
  EUV_LAUNCH_CHECK();
  const long long mask_bytes = (long long)ndivx * ndivy / 8;
  // column tiles of at most eight blocks of 8, as even as they come
  const int blocks = (2 * lp + 7) / 8, tiles = (blocks + 7) / 8, nb = (blocks + tiles - 1) / tiles;
  for (long long g0 = 0; g0 < n_masks; g0 += group) {
    const int ng = (int)(n_masks - g0 < group ? n_masks - g0 : group);
    const uint8_t* b = d_bits + g0 * mask_bytes;
    int rc = EUV_OK;
#define EUV_SPECTRUM_CASE(NB) \
  case NB: rc = launch_spectrum_rows<NB>(b, mask_bytes, ndivx, ndivy, lh, tiles, ng, Wx, T, stream); break
    switch (nb) {
      EUV_SPECTRUM_CASE(1);
      EUV_SPECTRUM_CASE(2);
      EUV_SPECTRUM_CASE(3);
      EUV_SPECTRUM_CASE(4);
      EUV_SPECTRUM_CASE(5);
      EUV_SPECTRUM_CASE(6);
      EUV_SPECTRUM_CASE(7);
      default: rc = launch_spectrum_rows<8>(b, mask_bytes, ndivx, ndivy, lh, tiles, ng, Wx, T, stream);
    }
#undef EUV_SPECTRUM_CASE
    if (rc) return rc;
    // P (mr x ng lp) = Wy (mr x ndivy) T (ndivy x ng lp), K split in `parts` chunks
    const int kc = ndivy / parts;
    const long long cols = (long long)ng * lp;
    double2* P = reinterpret_cast<double2*>(
        reinterpret_cast<char*>(T) + ((ng * t_bytes + 255) & ~(size_t)255));
    rc = zgemm(mr, (int)cols, kc, mk(1.0, 0.0), nullptr, Wy, mr, (long long)kc * mr, T, ndivy, kc,
               mk(0.0, 0.0), P, mr, (long long)mr * cols, mk(0.0, 0.0), parts, nullptr, 0, stream);
    if (rc) return rc;
    const long long total = (long long)ng * lr * mr;
    EUV_CUDA_TRY(launch_dependent(spectrum_reduce_kernel, dim3(grid1(total, 256)), dim3(256), 0,
                                  stream, P, parts, ng, lh, mh,
                                  (double)fdivx * (double)fdivy, select_vacuum,
                                  reinterpret_cast<double2*>(d_out) + g0 * lr * mr));
    EUV_LAUNCH_CHECK();
  }
  return EUV_OK;
}

// ------------------------------------------------------------------ matfun
extern "C" size_t euv_matfun_workspace_bytes(int n, int batch) {
  Bump bp{nullptr, (size_t)-1, 0, true};
  const long long nn = (long long)n * n;
  for (int i = 0; i < 5; ++i) bp.take<double2>(nn * batch);
  for (int i = 0; i < 4; ++i) bp.take<double>(batch);
  bp.take<int>(batch);
  bp.take<int>(1);
  bp.take<char>(gemm_mixed_workspace_bytes(n, n, n, batch));
  return bp.off;
}

extern "C" int euv_matfun_cs(int n, const euv_c64* d_d, const double* d_thick, euv_c64* d_cos,
                             euv_c64* d_sin, int batch, int m_max, int precision, void* d_work,
                             size_t work_bytes, void* stream_) {
  if (n <= 0 || batch <= 0 || !d_d || !d_thick || !d_cos || !d_sin || m_max < 0 ||
      m_max > kMaxSteps || (precision != EUV_PREC_FP64 && precision != EUV_PREC_MIXED)) {
    euv_set_error("euv_matfun_cs: bad arguments");
    return EUV_ERR_BAD_ARG;
  }
  cudaStream_t stream = (cudaStream_t)stream_;
  const long long nn = (long long)n * n;
  Bump bp{reinterpret_cast<char*>(d_work), work_bytes, 0, true};
  MatfunBufs mb;
  mb.P2 = bp.take<double2>(nn * batch);
  mb.P3 = bp.take<double2>(nn * batch);
  mb.P4 = bp.take<double2>(nn * batch);
  mb.T1 = bp.take<double2>(nn * batch);
  mb.T2 = bp.take<double2>(nn * batch);
  mb.norm = bp.take<double>(batch);
  mb.h = bp.take<double>(batch);
  mb.h2 = bp.take<double>(batch);
  mb.h4 = bp.take<double>(batch);
  mb.steps = bp.take<int>(batch);
  mb.capped = bp.take<int>(1);
  size_t mbytes = gemm_mixed_workspace_bytes(n, n, n, batch);
  void* mw = bp.take<char>(mbytes);
  if (!d_work || !bp.ok) {
    euv_set_error("euv_matfun_cs: workspace too small");
    return EUV_ERR_WORKSPACE;
  }
  Gemm gemm{precision, mw, mbytes, stream};
  double2* C = reinterpret_cast<double2*>(d_cos);
  double2* S = reinterpret_cast<double2*>(d_sin);
  double2* C0 = C;
  double2* S0 = S;
  int rc = matfun(n, batch, reinterpret_cast<const double2*>(d_d), d_thick, &C, &S, mb, m_max,
                  gemm, stream);
  if (rc) return rc;
  if (C != C0) EUV_CUDA_TRY(cudaMemcpyAsync(C0, C, nn * batch * sizeof(double2), cudaMemcpyDeviceToDevice, stream));
  if (S != S0) EUV_CUDA_TRY(cudaMemcpyAsync(S0, S, nn * batch * sizeof(double2), cudaMemcpyDeviceToDevice, stream));
  return EUV_OK;
}

// ------------------------------------------------------------------ matfun, no allocation
// Scratch of euv_matfun_cs_noalloc: a fixed device array in this library, so the
// entry point needs no workspace from the caller and allocates nothing.  It is
// EUV_NOALLOC_SCRATCH_BYTES on every GPU that loads the library, for the life of
// the process.  Every call uses the same array.
static __device__ __align__(256) unsigned char g_matfun_scratch[EUV_NOALLOC_SCRATCH_BYTES];

namespace {
// Device address of g_matfun_scratch per device, looked up on the first call
// made with that device current (cudaGetSymbolAddress is a host-side query).
void* g_scratch_ptr[64];
int g_scratch_ready[64];

int scratch_for_current_device(void** out) {
  int dev = 0;
  EUV_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) {
    euv_set_error("euv_matfun_cs_noalloc: device ordinal %d out of range", dev);
    return EUV_ERR_BAD_ARG;
  }
  if (!__atomic_load_n(&g_scratch_ready[dev], __ATOMIC_ACQUIRE)) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_matfun_scratch);
    if (e != cudaSuccess || p == nullptr) {
      euv_set_error("euv_matfun_cs_noalloc: cudaGetSymbolAddress failed on device %d: %s", dev,
                    cudaGetErrorString(e));
      return EUV_ERR_CUDA;
    }
    g_scratch_ptr[dev] = p;
    __atomic_store_n(&g_scratch_ready[dev], 1, __ATOMIC_RELEASE);
  }
  *out = g_scratch_ptr[dev];
  return EUV_OK;
}
}  // namespace

extern "C" int euv_matfun_cs_noalloc(int n, const euv_c64* d_d, const double* d_thick,
                                     euv_c64* d_cos, euv_c64* d_sin, int batch, int m_max,
                                     void* stream_) {
  if (n <= 0 || batch <= 0 || !d_d || !d_thick || !d_cos || !d_sin || m_max < 0 ||
      m_max > kMaxSteps) {
    euv_set_error("euv_matfun_cs_noalloc: bad arguments");
    return EUV_ERR_BAD_ARG;
  }
  size_t need;
  {
    Bump dry{nullptr, (size_t)-1, 0, true};
    const long long nn0 = (long long)n * n;
    for (int i = 0; i < 5; ++i) dry.take<double2>(nn0 * batch);
    for (int i = 0; i < 4; ++i) dry.take<double>(batch);
    dry.take<int>(batch);
    dry.take<int>(1);
    need = dry.off;
  }
  if (need > (size_t)EUV_NOALLOC_SCRATCH_BYTES) {
    euv_set_error("euv_matfun_cs_noalloc: n=%d batch=%d needs %zu bytes of scratch, above the "
                  "fixed %zu bytes (use euv_matfun_cs with a caller workspace)",
                  n, batch, need, (size_t)EUV_NOALLOC_SCRATCH_BYTES);
    return EUV_ERR_BAD_ARG;
  }
  void* scratch = nullptr;
  int rc = scratch_for_current_device(&scratch);
  if (rc) return rc;
  cudaStream_t stream = (cudaStream_t)stream_;
  const long long nn = (long long)n * n;
  Bump bp{reinterpret_cast<char*>(scratch), (size_t)EUV_NOALLOC_SCRATCH_BYTES, 0, true};
  MatfunBufs mb;
  mb.P2 = bp.take<double2>(nn * batch);
  mb.P3 = bp.take<double2>(nn * batch);
  mb.P4 = bp.take<double2>(nn * batch);
  mb.T1 = bp.take<double2>(nn * batch);
  mb.T2 = bp.take<double2>(nn * batch);
  mb.norm = bp.take<double>(batch);
  mb.h = bp.take<double>(batch);
  mb.h2 = bp.take<double>(batch);
  mb.h4 = bp.take<double>(batch);
  mb.steps = bp.take<int>(batch);
  mb.capped = bp.take<int>(1);
  if (!bp.ok) {
    euv_set_error("euv_matfun_cs_noalloc: scratch layout overflow");
    return EUV_ERR_BAD_ARG;
  }
  // The array keeps the previous call's contents: the only state that must
  // start at zero is the cap flag (the column-norm maxima are cleared by matfun).
  EUV_CUDA_TRY(cudaMemsetAsync(mb.capped, 0, sizeof(int), stream));
  Gemm gemm{EUV_PREC_FP64, nullptr, 0, stream};
  double2* C = reinterpret_cast<double2*>(d_cos);
  double2* S = reinterpret_cast<double2*>(d_sin);
  double2* C0 = C;
  double2* S0 = S;
  rc = matfun(n, batch, reinterpret_cast<const double2*>(d_d), d_thick, &C, &S, mb, m_max, gemm,
              stream);
  if (rc) return rc;
  if (C != C0)
    EUV_CUDA_TRY(cudaMemcpyAsync(C0, C, nn * batch * sizeof(double2), cudaMemcpyDeviceToDevice, stream));
  if (S != S0)
    EUV_CUDA_TRY(cudaMemcpyAsync(S0, S, nn * batch * sizeof(double2), cudaMemcpyDeviceToDevice, stream));
  return EUV_OK;
}
