// Mixed-precision complex GEMM on the 5th-generation tensor cores (tcgen05).
//
// C = alpha*scale[b] * A B + beta C + diag*I for complex FP64 A (MxK), B (KxN),
// C (MxN), column-major and batched (GemmTerms: the beta term may read another
// matrix of C's shape, and a second such term may be added; the operands' diagonals may
// be multiplied apart), computed as split-FP16x3 with power-of-two scaling: every row of
// A and every column of B is scaled by 2^e (e from its largest |re|, |im|, so
// that the scaled values lie below 2^15), each scaled FP64 real is split into
// two fp16 values x = hi + lo (hi = x rounded to fp16, lo = the remainder
// rounded to fp16) and each real product is hi*hi + hi*lo + lo*hi with FP32
// accumulation in tensor memory (kind::f16, twice the TF32 rate); the
// epilogue multiplies by 2^-(e_row + e_col).  fp16 carries the same 11
// significant bits as TF32, so the products keep about 22 bits (the scaling
// only moves the values into fp16's exponent range; entries more than 2^24
// below their row's or column's largest lose relative precision but add at
// most 2^-38 of it to a product).  The complex product uses four real products:
//   Re = ArBr - AiBi,  Im = ArBi + AiBr   (the minus sign through the MMA's
//   negate-A bit): twelve real products per K=16 step, issued as nine
//   tcgen05.mma (the three Ar products as N = 256 against [Br | Bi], writing
//   the adjacent Re and Im accumulators at once).  The FP32 accumulation error
//   grows with the K it spans, so the two halves of K have their own Re/Im
//   accumulators (four in all), summed in FP64 by the epilogue.
// Error per product ~1e-6 relative: the bulk products of the slab matrix
// functions tolerate it (intensity error < 1e-4, see the tests); the interface
// solves stay FP64.
//
// Operands are first rewritten (split_*_kernel: the row or column maxima,
// then the split) as four fp16 planes [batch][Re_hi, Re_lo, Im_hi, Im_lo]
// [rows][Kp] with K contiguous (K-major for both A and B), Kp = K rounded up
// to 32, and the exponents [batch][rows].  The GEMM kernel:
//   warp 0     : TMA producer (3-D tensor maps, 64-byte swizzle, 3 stages of
//                4x(128x32) A + 4x(128x32) B fp16 = 64 KB);
//   warp 1     : TMEM allocation (512 columns: four 128-column accumulators of
//                a 128x128 tile) and the single-thread MMA issue loop;
//   warps 2..9 : epilogue, tcgen05.ld of 32 TMEM lanes (= rows) x 64 columns each,
//                complex FP64 result written column by column (coalesced).
// All waits are bounded (about 2 s); a timeout ORs EUV_STATUS_TIMEOUT into the
// status word, drains the copies and MMAs in flight, frees TMEM and returns.
#include <cuda_fp16.h>

#include "tcgen05.cuh"

namespace euv {

constexpr int MX_BM = 128;
constexpr int MX_BN = 128;
constexpr int MX_BK = 32;  // fp16 elements: 64-byte rows, one 64B swizzle span
constexpr int MX_STAGES = 3;
constexpr int MX_PLANES = 4;
constexpr int MX_A_TILE = MX_BM * MX_BK * 2;  // 8 KB
constexpr int MX_B_TILE = MX_BN * MX_BK * 2;  // 8 KB
constexpr int MX_STAGE_BYTES = MX_PLANES * (MX_A_TILE + MX_B_TILE);  // 64 KB
constexpr int MX_EPI_WARPS = 8;
constexpr int MX_THREADS = 64 + 32 * MX_EPI_WARPS;
constexpr int MX_TMEM_COLS = 512;
constexpr int MX_COL_OFF = MX_STAGES * MX_STAGE_BYTES + 256;  // column factors, after the barriers
constexpr int MX_DIAG_OFF = MX_COL_OFF + MX_BN * (int)sizeof(double);
constexpr size_t MX_SMEM = (size_t)MX_DIAG_OFF + 1024;
// NX = 3 holds B's diagonal too; 2 KB more for the others took L1 from their epilogues (N =
// 169, 48 entries, 59.0 -> 59.9 us)
constexpr size_t MX_SMEM_DIAG = MX_SMEM + MX_BN * sizeof(double2);
constexpr unsigned long long MX_TIMEOUT_NS = 2000000000ull;
// stage slot of each B plane (gmem order Re_hi, Re_lo, Im_hi, Im_lo)
__device__ constexpr int kBSlot[4] = {0, 2, 1, 3};

struct MixedArgs {
  int m, n, kp;
  double2 alpha, beta, diag;
  const double* scale;
  const double2* a;  // original FP64 operands (copy mode, GemmTerms::apart)
  long long lda, sa;
  const double2* b;
  long long ldb, sb;
  double2* c;
  GemmTerms t;
  long long ldc, sc;
  const int* steps;
  int step;
  int* err;
  const int* ea;  // [b][m] power-of-two exponent each row of A was scaled by
  const int* eb;  // [b][n] the same for the columns of B
};

__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                          int* err) {
  return mbar_wait_bounded(bar, parity, abort_flag, err, MX_TIMEOUT_NS);
}
// Instruction descriptor of kind::f16: D f32, A and B f16 (format 0), both K-major.
__host__ __device__ __forceinline__ constexpr uint32_t idesc_f16_mn(bool neg_a, int m, int n) {
  return (1u << 4) | ((neg_a ? 1u : 0u) << 13) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ constexpr uint32_t idesc_f16(bool neg_a) {
  return idesc_f16_mn(neg_a, MX_BM, MX_BN);
}
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Order of a tile's k-blocks.  An FP32 accumulator in TMEM loses up to 2^-24 of
// its running sum at every step, so a large term should enter late: for
// operands with a dominant diagonal (the rows carried through the slices, the
// matrix functions) the large terms of a tile lie in the k-blocks of its own
// rows (a_ii b_ij) and of its own columns (a_ij b_jj).  Those of the columns go
// last in the first accumulator set, those of the rows last in the second; the
// other blocks are dealt half to each set in front of them.  Measured: intensity
// error of the 2048 nm eight-slice step 6.3e-6 -> 2.2e-6, same time.
struct KOrder {
  int a0, na, b0, nb, lo, nlo, hi, nhi, o0, h0;  // h0: blocks of the first set
  __device__ __forceinline__ KOrder(int nkb, int m0, int n0) {
    constexpr int W = MX_BM / MX_BK;
    a0 = m0 / MX_BK;
    na = a0 < nkb ? (nkb - a0 < W ? nkb - a0 : W) : 0;
    b0 = (n0 / MX_BK) % nkb;
    nb = nkb - b0 < W ? nkb - b0 : W;
    if (na > 0 && b0 < a0 + na && b0 + nb > a0) {  // overlap: the columns' blocks beside the rows'
      if (b0 < a0) {
        nb = a0 - b0;
      } else {
        nb = b0 + nb > a0 + na ? b0 + nb - a0 - na : 0;
        b0 = a0 + na;
      }
    }
    if (nkb <= 2 * W) na = nb = 0;  // short sums: ascending
    lo = a0 < b0 ? a0 : b0;
    nlo = a0 < b0 ? na : nb;
    hi = a0 < b0 ? b0 : a0;
    nhi = a0 < b0 ? nb : na;
    const int others = nkb - na - nb;
    o0 = (others + 1) / 2;
    h0 = o0 + nb;
    nkb_ = nkb;
  }
  int nkb_;
  __device__ __forceinline__ int operator()(int i) const {
    if (i >= o0 && i < h0) return b0 + (i - o0);
    if (i >= nkb_ - na) return a0 + (i - (nkb_ - na));
    int r = i < o0 ? i : i - nb;
    if (r >= lo) r += nlo;
    if (r >= hi) r += nhi;
    return r;
  }
};

// NX: matrices the epilogue adds (0: none, 1: the beta term, 2: GemmTerms::cin2 too, 3:
// the diagonals' rows and columns of GemmTerms::apart).
// The epilogue cannot overlap the main loop (the four accumulators fill TMEM, the
// stages shared memory, so an SM holds one CTA) and moves 256 KB per matrix and
// tile: eight warps, the first chunk of the added matrices loaded and the rest
// prefetched into L2 while the main loop runs, each later chunk's loads issued
// one chunk ahead, scale factors as two numbers per element instead of an ldexp.
template <int NX>
__global__ void __launch_bounds__(MX_THREADS, 1)
    gemm_split3_kernel(const __grid_constant__ CUtensorMap tmA,
                       const __grid_constant__ CUtensorMap tmB, MixedArgs p) {
  dependent_begin();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + MX_STAGES * MX_STAGE_BYTES);
  uint64_t* empty = full + MX_STAGES;
  uint64_t* accum = empty + MX_STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.z;
  const int m0 = blockIdx.x * MX_BM, n0 = blockIdx.y * MX_BN;
  double2* C = p.c + (long long)b * p.sc;

  if (p.t.need != nullptr && p.t.need[b] <= p.t.need_above) return;
  if (p.steps != nullptr && p.step >= p.steps[b]) {
    if (!step_copies(p.t.paired, p.steps[b], p.step)) return;
    // inactive double-angle step of this batch entry: C = A on this tile
    // (eight loads in flight per thread before their stores: the CTA holds a
    // whole SM's shared memory, so the copy must not wait on each element)
    const double2* A = p.a + (long long)b * p.sa;
    constexpr int U = 8;
    for (int base = 0; base < MX_BM * MX_BN; base += MX_THREADS * U) {
      double2 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int idx = base + threadIdx.x + u * MX_THREADS;
        const int gi = m0 + idx % MX_BM, gj = n0 + idx / MX_BM;
        v[u] = (idx < MX_BM * MX_BN && gi < p.m && gj < p.n) ? A[gi + (long long)gj * p.lda]
                                                             : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int idx = base + threadIdx.x + u * MX_THREADS;
        const int gi = m0 + idx % MX_BM, gj = n0 + idx / MX_BM;
        if (idx < MX_BM * MX_BN && gi < p.m && gj < p.n) C[gi + (long long)gj * p.ldc] = v[u];
      }
    }
    return;
  }

  auto a_tile = [&](int s, int pl) { return smem + s * MX_STAGE_BYTES + pl * MX_A_TILE; };
  auto b_tile = [&](int s, int pl) {
    return smem + s * MX_STAGE_BYTES + MX_PLANES * MX_A_TILE + pl * MX_B_TILE;
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < MX_STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(accum, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(MX_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const int nkb = p.kp / MX_BK;
  const KOrder order(nkb, m0, n0);

  if (warp == 0) {
    if (lane == 0) {
      int issued = 0;
      for (int kb = 0; kb < nkb; ++kb) {
        const int s = kb % MX_STAGES;
        const uint32_t ph = (uint32_t)((kb / MX_STAGES) & 1);
        if (!mbar_wait(&empty[s], ph ^ 1u, abort_flag, p.err)) break;
        mbar_expect_tx(&full[s], (uint32_t)MX_STAGE_BYTES);
        const int k0 = order(kb) * MX_BK;
        for (int pl = 0; pl < MX_PLANES; ++pl)
          tma_load_3d(a_tile(s, pl), &tmA, k0, m0, b * MX_PLANES + pl, &full[s]);
        // B planes in the stage as Re_hi, Im_hi, Re_lo, Im_lo: [Br | Bi] of a
        // precision level are adjacent, one N = 256 operand
        for (int pl = 0; pl < MX_PLANES; ++pl)
          tma_load_3d(b_tile(s, kBSlot[pl]), &tmB, k0, n0, b * MX_PLANES + pl, &full[s]);
        issued = kb + 1;
      }
      if (*abort_flag) {
        // drain this thread's copies in flight (bounded) before the CTA exits
        for (int kb = (issued > MX_STAGES ? issued - MX_STAGES : 0); kb < issued; ++kb) {
          const unsigned long long t0 = globaltimer();
          while (!mbar_try(&full[kb % MX_STAGES], (uint32_t)((kb / MX_STAGES) & 1)) &&
                 globaltimer() - t0 < MX_TIMEOUT_NS) {
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // Planes: 0 Re_hi 1 Re_lo 2 Im_hi 3 Im_lo.  The FP32 accumulation in
      // TMEM loses precision in proportion to the K it runs over (measured: the
      // error is the same for exactly split operands and grows linearly in K), so
      // the K range is split in two halves with their own Re/Im accumulators,
      // summed in FP64 by the epilogue.
      // Products: Re = +ArBr -AiBi, Im = +ArBi +AiBr, each as hi*hi + hi*lo +
      // lo*hi.  The Ar terms of Re and Im share their A operand: one MMA of
      // N = 256 against [Br | Bi] (adjacent in the stage) writes both
      // accumulators (Re and Im of a K half are adjacent TMEM columns); the Ai
      // terms differ in sign and take two N = 128 MMAs each (Re negated).
      // A planes: 0 Re_hi 1 Re_lo 2 Im_hi 3 Im_lo; B stage slots: kBSlot.
      const int ar_a[3] = {0, 0, 1}, ar_b[3] = {0, 2, 0};  // B slot of [Br|Bi] hi / lo
      const int ai_a[3] = {2, 2, 3};
      const int ai_bi[3] = {1, 3, 1}, ai_br[3] = {0, 2, 0};  // slots of Bi / Br
      const uint32_t id_pos = idesc_f16(false), id_neg = idesc_f16(true);
      const uint32_t id_wide = idesc_f16_mn(false, MX_BM, 2 * MX_BN);
      const int half = order.h0;  // blocks [0, half) -> set 0, [half, nkb) -> set 1
      // Shared-memory descriptors of stage 0, computed once: the tile of stage s
      // lies s * MX_STAGE_BYTES further and a K16 step 32 bytes further, i.e.
      // + s * (MX_STAGE_BYTES >> 4) and + 2 in the 14-bit address field, which
      // cannot carry (shared addresses stay below 2^18).  The issue loop then
      // only adds.
      uint64_t dA[MX_PLANES], dB[MX_PLANES];
#pragma unroll
      for (int pl = 0; pl < MX_PLANES; ++pl) {
        dA[pl] = umma_desc_sw64(a_tile(0, pl));
        dB[pl] = umma_desc_sw64(b_tile(0, pl));
      }
      int s = 0;
      uint32_t ph = 0;
      for (int kb = 0; kb < nkb; ++kb) {
        if (!mbar_wait(&full[s], ph, abort_flag, p.err)) break;
        tc_fence_after();
        const int set = kb < half ? 0 : 1;
        const uint32_t t_re = tmem + (uint32_t)(2 * set * MX_BN);
        const uint32_t t_im = t_re + (uint32_t)MX_BN;
        const int kb0 = set ? half : 0;
        const uint64_t so = (uint64_t)s * (uint64_t)(MX_STAGE_BYTES >> 4);
#pragma unroll
        for (int k16 = 0; k16 < MX_BK / 16; ++k16) {
          const uint32_t first = (kb != kb0 || k16) ? 1u : 0u;
          const uint64_t ko = so + (uint64_t)(2 * k16);
#pragma unroll
          for (int q = 0; q < 3; ++q)
            umma_f16(t_re, dA[ar_a[q]] + ko, dB[ar_b[q]] + ko, id_wide, (first | q) ? 1u : 0u);
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            umma_f16(t_re, dA[ai_a[q]] + ko, dB[ai_bi[q]] + ko, id_neg, 1u);
            umma_f16(t_im, dA[ai_a[q]] + ko, dB[ai_br[q]] + ko, id_pos, 1u);
          }
        }
        umma_commit(&empty[s]);  // frees the stage when these MMAs complete
        if (++s == MX_STAGES) {
          s = 0;
          ph ^= 1u;
        }
      }
      umma_commit(accum);  // always: the epilogue / teardown waits on it
    }
  } else {
    // epilogue: warps 2..9; TMEM lanes (warp % 4) * 32 .. +31 = tile rows, two
    // warps per lane quarter with 64 columns each
    constexpr int EC = 8, NCH = MX_BN / 2 / EC;
    const int q = warp & 3, half = (warp - 2) >> 2;
    const int cb = n0 + half * (MX_BN / 2);
    const int row = m0 + q * 32 + lane;
    const bool rok = row < p.m;
    double* s_cf = reinterpret_cast<double*>(smem + MX_COL_OFF);
    const double2* Cin = p.t.cin ? p.t.cin + (long long)b * p.t.scin : C;
    const double2* Cin2 = NX == 2 ? p.t.cin2 + (long long)b * p.t.scin2 : C;
    // NX = 3: C += diag(A) B + A diag(B) - diag(A) diag(B), B's k x k blocks one by one
    const bool apart = NX == 3 && p.t.apart[b] != 0;
    const double2* Bf = NX == 3 ? p.b + (long long)b * p.sb : C;
    const double2* Af = NX == 3 ? p.a + (long long)b * p.sa : C;
    double2* s_db = reinterpret_cast<double2*>(smem + MX_DIAG_OFF);
    auto block_col = [&](int col) { return col >= p.m ? col - p.m : col; };
    // undo the power-of-two scaling of the operands: 2^-(exponents of row and column)
    if (threadIdx.x - 64 < MX_BN) {
      const int col = n0 + (int)threadIdx.x - 64;
      s_cf[threadIdx.x - 64] = col < p.n ? ldexp(1.0, -p.eb[(long long)b * p.n + col]) : 0.0;
      if (NX == 3)
        s_db[threadIdx.x - 64] = apart && col < p.n ? Bf[block_col(col) + (long long)col * p.ldb]
                                                    : make_double2(0.0, 0.0);
    }
    asm volatile("bar.sync 1, %0;" ::"r"(32 * MX_EPI_WARPS) : "memory");
    const double sc = (p.scale ? p.scale[b] : 1.0) *
                      (rok ? ldexp(1.0, -p.ea[(long long)b * p.m + row]) : 0.0);
    const cplx alpha = mk(p.alpha.x * sc, p.alpha.y * sc);
    cplx beta = mk(p.beta.x, p.beta.y), beta2 = mk(0.0, 0.0);
    if (NX >= 1 && p.t.beta_b) beta = beta * mk(p.t.beta_b[b].x, p.t.beta_b[b].y);
    if (NX == 2) beta2 = mk(p.t.beta2.x, p.t.beta2.y) * mk(p.t.beta2_b[b].x, p.t.beta2_b[b].y);
    const cplx dg = mk(p.diag.x, p.diag.y);
    if (NX == 3) {
      const double2 da = apart && rok ? Af[row + (long long)row * p.lda] : make_double2(0.0, 0.0);
      beta = mk(da.x, da.y);
    }
    if (NX == 1 || NX == 2 || apart) {
      // four lanes per column, one 128-byte line each
#pragma unroll
      for (int c = lane >> 2; c < MX_BN / 2; c += 8) {
        const int r = m0 + q * 32 + (lane & 3) * 8, col = cb + c;
        if (r < p.m && col < p.n) {
          if (NX == 3) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(Bf + r + (long long)col * p.ldb));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(Af + r + (long long)block_col(col) * p.lda));
          } else {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(Cin + r + (long long)col * p.ldc));
            if (NX == 2)
              asm volatile("prefetch.global.L2 [%0];" ::"l"(Cin2 + r + (long long)col * p.ldc));
          }
        }
      }
    }
    // NX >= 2: one buffer (registers), each chunk's reads with its own TMEM loads
    constexpr int NB = NX >= 2 ? 1 : 2;
    double2 o1[NB][EC], o2[NB][EC];
    auto fetch = [&](int ch, double2(&x1)[EC], double2(&x2)[EC]) {
#pragma unroll
      for (int j = 0; j < EC; ++j) {
        const int col = cb + ch * EC + j;
        if (NX == 3) {
          const bool in = apart && rok && col < p.n;
          x1[j] = in ? Bf[row + (long long)col * p.ldb] : make_double2(0.0, 0.0);
          x2[j] = in ? Af[row + (long long)block_col(col) * p.lda] : make_double2(0.0, 0.0);
        } else {
          const bool in = rok && col < p.n;
          const long long at = row + (long long)col * p.ldc;
          if (NX >= 1) x1[j] = in ? Cin[at] : make_double2(0.0, 0.0);
          if (NX == 2) x2[j] = in ? Cin2[at] : make_double2(0.0, 0.0);
        }
      }
    };
    if (NX >= 1) fetch(0, o1[0], o2[0]);
    const bool waited = mbar_wait(accum, 0u, abort_flag, p.err) && !*abort_flag && nkb > 0;
    const bool ok = __all_sync(0xffffffffu, waited);  // tcgen05.ld below is warp-collective
    tc_fence_after();
    if (ok) {
      const uint32_t t0 = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * (MX_BN / 2));
#pragma unroll
      for (int ch = 0; ch < NCH; ++ch) {
        if (cb + ch * EC >= p.n) break;  // warp-uniform
        uint32_t vr[EC], vi[EC], cr[EC], ci[EC];
        tmem_ld8(t0 + (uint32_t)(ch * EC), vr);
        tmem_ld8(t0 + (uint32_t)(MX_BN + ch * EC), vi);
        tmem_ld8(t0 + (uint32_t)(2 * MX_BN + ch * EC), cr);
        tmem_ld8(t0 + (uint32_t)(3 * MX_BN + ch * EC), ci);
        // the next chunk's reads before this chunk's stores: a load after a
        // store through the same pointer type would otherwise wait for it
        if (NX == 1 && ch + 1 < NCH) fetch(ch + 1, o1[(ch + 1) % NB], o2[(ch + 1) % NB]);
        if (NX >= 2 && ch > 0) fetch(ch, o1[0], o2[0]);
        tmem_ld_wait();
        if (rok) {
#pragma unroll
          for (int j = 0; j < EC; ++j) {
            const int col = cb + ch * EC + j;
            if (col < p.n) {
              // K halves: set 0 at columns [0, 2BN), set 1 (empty if nkb == 1) at [2BN, 4BN)
              const double s1r = nkb > 1 ? (double)__uint_as_float(cr[j]) : 0.0;
              const double s1i = nkb > 1 ? (double)__uint_as_float(ci[j]) : 0.0;
              const double f = s_cf[col - n0];
              cplx v = alpha * mk(f * ((double)__uint_as_float(vr[j]) + s1r),
                                  f * ((double)__uint_as_float(vi[j]) + s1i));
              if (NX >= 1) v = v + beta * mk(o1[ch % NB][j].x, o1[ch % NB][j].y);
              if (NX == 3) beta2 = mk(s_db[col - n0].x, s_db[col - n0].y);
              if (NX >= 2) v = v + beta2 * mk(o2[ch % NB][j].x, o2[ch % NB][j].y);
              if (NX == 3 && row == block_col(col)) v = v - beta * beta2;
              if (row == col) v = v + dg;
              C[row + (long long)col * p.ldc] = make_double2(v.x, v.y);
            }
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    if (*abort_flag) {
      // the MMAs in flight must finish before their TMEM is released (bounded)
      const unsigned long long t0 = globaltimer();
      while (!mbar_try(accum, 0u) && globaltimer() - t0 < MX_TIMEOUT_NS) {
      }
    }
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(MX_TMEM_COLS)
                 : "memory");
  }
}

// x (FP64, already scaled by a power of two) -> x = hi + lo, hi = x rounded to
// fp16, lo = the remainder rounded to fp16: hi*hi + hi*lo + lo*hi carries about
// 22 significant bits of each product, as TF32x3 does.
__device__ __forceinline__ void split_f16(double x, __half& hi, __half& lo) {
  hi = __double2half(x);
  lo = __double2half(x - (double)__half2float(hi));
}

// Exponent s with max |x| * 2^s in [2^14, 2^15): fp16 holds the scaled values
// (largest finite 65504) with hi and lo normal down to 2^-14 of that range.
__device__ __forceinline__ int scale_exponent(double mx) {
  if (!(mx > 0.0) || !isfinite(mx)) return 0;
  int e;
  frexp(mx, &e);
  return 15 - e;
}

// A (col-major complex M x K) -> planes [b][4][M][Kp] of fp16, K contiguous,
// each row scaled by 2^ea[b][row] (the row's largest |re|, |im| to [2^14,
// 2^15)).  One CTA per 32 rows: pass 1 finds the row maxima (lanes = rows, one
// coalesced 512-byte column slice per warp load), pass 2 splits 32 x 32 tiles
// transposed through shared memory (the slab is re-read from L2).
__global__ void split_a_kernel(int M, int K, int Kp, const double2* A, long long lda,
                               long long sa, __half* out, int* ea, const int* steps, int step,
                               const int* apart) {
  __shared__ double2 tile[32][33];
  __shared__ double red[8][32];
  __shared__ double s_scale[32];
  const int b = blockIdx.y;
  if (steps != nullptr && step >= steps[b]) return;  // inactive entry: the GEMM copies
  const int m0 = blockIdx.x * 32;
  const bool ap = apart != nullptr && apart[b] != 0;
  A += (long long)b * sa;
  const int tx = threadIdx.x, ty = threadIdx.y;
  {
    double mx = 0.0;
    const int r = m0 + tx;
    if (r < M)
      for (int k = ty; k < K; k += 8) {
        if (ap && k == r) continue;
        const double2 v = A[r + (long long)k * lda];
        mx = fmax(mx, fmax(fabs(v.x), fabs(v.y)));
      }
    red[ty][tx] = mx;
  }
  __syncthreads();
  if (ty == 0) {
    double mx = red[0][tx];
    for (int j = 1; j < 8; ++j) mx = fmax(mx, red[j][tx]);
    const int e = scale_exponent(mx);
    s_scale[tx] = ldexp(1.0, e);
    if (m0 + tx < M) ea[(long long)b * M + m0 + tx] = e;
  }
  __syncthreads();
  const long long plane = (long long)M * Kp;
  __half* o = out + (long long)b * MX_PLANES * plane;
  for (int k0 = 0; k0 < Kp; k0 += 32) {
    for (int j = ty; j < 32; j += 8) {
      const int m = m0 + tx, k = k0 + j;
      tile[j][tx] = (m < M && k < K && !(ap && k == m)) ? A[m + (long long)k * lda]
                                                        : make_double2(0.0, 0.0);
    }
    __syncthreads();
    for (int j = ty; j < 32; j += 8) {
      const int m = m0 + j, k = k0 + tx;
      if (m < M && k < Kp) {
        const double2 v = tile[tx][j];
        const double sc = s_scale[j];
        __half rh, rl, ih, il;
        split_f16(v.x * sc, rh, rl);
        split_f16(v.y * sc, ih, il);
        const long long off = (long long)m * Kp + k;
        o[off] = rh;
        o[plane + off] = rl;
        o[2 * plane + off] = ih;
        o[3 * plane + off] = il;
      }
    }
    __syncthreads();
  }
}

// B (col-major complex K x N) -> planes [b][4][N][Kp] of fp16, K contiguous,
// each column scaled by 2^eb[b][col]; one warp per column (max, then split).
__global__ void split_b_kernel(int K, int N, int Kp, const double2* B, long long ldb,
                               long long sb, __half* out, int* eb, const int* steps, int step,
                               const int* apart) {
  const int b = blockIdx.y;
  if (steps != nullptr && step >= steps[b]) return;
  const bool ap = apart != nullptr && apart[b] != 0;
  const int lane = threadIdx.x & 31;
  const int n = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (n >= N) return;  // warp-uniform
  const double2* col = B + (long long)b * sb + (long long)n * ldb;
  double mx = 0.0;
  for (int k = lane; k < K; k += 32) {
    if (ap && k == n % K) continue;
    const double2 v = col[k];
    mx = fmax(mx, fmax(fabs(v.x), fabs(v.y)));
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  const int e = scale_exponent(mx);
  if (lane == 0) eb[(long long)b * N + n] = e;
  const double sc = ldexp(1.0, e);
  const long long plane = (long long)N * Kp;
  __half* o = out + (long long)b * MX_PLANES * plane + (long long)n * Kp;
  for (int k = lane; k < Kp; k += 32) {
    const double2 v = k < K && !(ap && k == n % K) ? col[k] : make_double2(0.0, 0.0);
    __half rh, rl, ih, il;
    split_f16(v.x * sc, rh, rl);
    split_f16(v.y * sc, ih, il);
    o[k] = rh;
    o[plane + k] = rl;
    o[2 * plane + k] = ih;
    o[3 * plane + k] = il;
  }
}

// The same splits with the operand's slab staged in shared memory, so that HBM
// sees one read and the plane writes (the two-pass kernels above re-read the
// slab, from HBM once the slabs of all resident CTAs exceed L2).  R rows of A
// (or R columns of B) per CTA, R * K * 16 bytes of shared memory; used when
// that fits (split_slab_rows), the two-pass kernels otherwise.
constexpr size_t MX_SLAB_BYTES = 100 * 1024;      // several CTAs per SM
constexpr size_t MX_SLAB_BYTES_ONE = 200 * 1024;  // one row or column per CTA
constexpr int MX_SLAB_THREADS = 256;
// 16-byte asynchronous copy global -> shared (zero-filled when !pred): the
// whole slab of a CTA is in flight at once, not eight loads per thread
__device__ __forceinline__ void slab_cp16(void* smem, const void* gmem, bool pred) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem),
               "r"(pred ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void slab_cp_wait() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// Row stride (elements) of the A slab: K rounded up to 8, plus 8 / R, so that
// the loads' stores (R consecutive rows per run of lanes) and the row-wise
// reads of the split both hit distinct 16-byte bank groups.
template <int R>
__host__ __device__ constexpr int slab_a_stride(int K) {
  return ((K + 7) / 8) * 8 + (R > 1 ? 8 / R : 0);
}

template <int R>
__global__ void __launch_bounds__(MX_SLAB_THREADS)
    split_a_slab_kernel(int M, int K, int Kp, const double2* A, long long lda, long long sa,
                        __half* out, int* ea, const int* steps, int step, const int* apart) {
  dependent_begin();
  extern __shared__ double2 slab[];  // [R][Ks]: element (row r, column k) at r * Ks + k
  const int Ks = slab_a_stride<R>(K);
  __shared__ double s_scale[R];
  const int b = blockIdx.y;
  if (steps != nullptr && step >= steps[b]) return;  // inactive entry: the GEMM copies
  const int m0 = blockIdx.x * R;
  const int rows = M - m0 < R ? M - m0 : R;
  A += (long long)b * sa;
  // consecutive threads take consecutive rows of a column (runs of R * 16
  // bytes); every copy of the slab in flight before the first wait
  for (int t = threadIdx.x; t < K * R; t += MX_SLAB_THREADS) {
    const int k = t / R, r = t % R;
    const bool ok = r < rows;
    slab_cp16(&slab[r * Ks + k], ok ? A + (m0 + r) + (long long)k * lda : A, ok);
  }
  slab_cp_wait();
  __syncthreads();
  if (apart != nullptr && apart[b] != 0) {
    if ((int)threadIdx.x < rows && m0 + (int)threadIdx.x < K)
      slab[threadIdx.x * Ks + m0 + threadIdx.x] = make_double2(0.0, 0.0);
    __syncthreads();
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < R) {
    double mx = 0.0;
    for (int k = lane; k < K; k += 32) {
      const double2 v = slab[warp * Ks + k];
      mx = fmax(mx, fmax(fabs(v.x), fabs(v.y)));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    if (lane == 0) {
      const int e = scale_exponent(mx);
      s_scale[warp] = ldexp(1.0, e);
      if (warp < rows) ea[(long long)b * M + m0 + warp] = e;
    }
  }
  __syncthreads();
  const long long plane = (long long)M * Kp;
  __half* o = out + (long long)b * MX_PLANES * plane;
  // two consecutive k per thread: one 4-byte store per plane (Kp is even)
  const int kh = Kp >> 1;
  for (int t = threadIdx.x; t < rows * kh; t += MX_SLAB_THREADS) {
    const int r = t / kh, k = 2 * (t % kh);
    const double2 v0 = k < K ? slab[r * Ks + k] : make_double2(0.0, 0.0);
    const double2 v1 = k + 1 < K ? slab[r * Ks + k + 1] : make_double2(0.0, 0.0);
    const double sc = s_scale[r];
    __half2 rh, rl, ih, il;
    split_f16(v0.x * sc, rh.x, rl.x);
    split_f16(v0.y * sc, ih.x, il.x);
    split_f16(v1.x * sc, rh.y, rl.y);
    split_f16(v1.y * sc, ih.y, il.y);
    __half2* o2 = reinterpret_cast<__half2*>(o + (long long)(m0 + r) * Kp + k);
    const long long p2 = plane >> 1;
    o2[0] = rh;
    o2[p2] = rl;
    o2[2 * p2] = ih;
    o2[3 * p2] = il;
  }
}

template <int R>
__global__ void __launch_bounds__(MX_SLAB_THREADS)
    split_b_slab_kernel(int K, int N, int Kp, const double2* B, long long ldb, long long sb,
                        __half* out, int* eb, const int* steps, int step, const int* apart) {
  dependent_begin();
  extern __shared__ double2 slab[];  // [R][K]: element (k, column c) at c * K + k
  __shared__ double s_scale[R];
  const int b = blockIdx.y;
  if (steps != nullptr && step >= steps[b]) return;
  const int n0 = blockIdx.x * R;
  const int cols = N - n0 < R ? N - n0 : R;
  B += (long long)b * sb;
  for (int t = threadIdx.x; t < K * R; t += MX_SLAB_THREADS) {
    const int c = t / K, k = t % K;
    const bool ok = c < cols;
    slab_cp16(&slab[t], ok ? B + k + (long long)(n0 + c) * ldb : B, ok);
  }
  slab_cp_wait();
  __syncthreads();
  if (apart != nullptr && apart[b] != 0) {
    if ((int)threadIdx.x < cols)
      slab[threadIdx.x * K + (n0 + threadIdx.x) % K] = make_double2(0.0, 0.0);
    __syncthreads();
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < R) {
    double mx = 0.0;
    for (int k = lane; k < K; k += 32) {
      const double2 v = slab[warp * K + k];
      mx = fmax(mx, fmax(fabs(v.x), fabs(v.y)));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    if (lane == 0) {
      const int e = scale_exponent(mx);
      s_scale[warp] = ldexp(1.0, e);
      if (warp < cols) eb[(long long)b * N + n0 + warp] = e;
    }
  }
  __syncthreads();
  const long long plane = (long long)N * Kp;
  __half* o = out + (long long)b * MX_PLANES * plane;
  const int kh = Kp >> 1;
  for (int t = threadIdx.x; t < cols * kh; t += MX_SLAB_THREADS) {
    const int c = t / kh, k = 2 * (t % kh);
    const double2 v0 = k < K ? slab[c * K + k] : make_double2(0.0, 0.0);
    const double2 v1 = k + 1 < K ? slab[c * K + k + 1] : make_double2(0.0, 0.0);
    const double sc = s_scale[c];
    __half2 rh, rl, ih, il;
    split_f16(v0.x * sc, rh.x, rl.x);
    split_f16(v0.y * sc, ih.x, il.x);
    split_f16(v1.x * sc, rh.y, rl.y);
    split_f16(v1.y * sc, ih.y, il.y);
    __half2* o2 = reinterpret_cast<__half2*>(o + (long long)(n0 + c) * Kp + k);
    const long long p2 = plane >> 1;
    o2[0] = rh;
    o2[p2] = rl;
    o2[2 * p2] = ih;
    o2[3 * p2] = il;
  }
}

// Rows (columns) per CTA of the slab splits: the most of 8, 4, 2 whose slab
// fits MX_SLAB_BYTES (so that several CTAs share an SM and keep enough loads
// in flight), else 1 up to MX_SLAB_BYTES_ONE; 0 beyond (the two-pass kernels).
static int split_slab_rows(int K) {
  const size_t row = (size_t)K * sizeof(double2);
  for (int r = 8; r >= 2; r >>= 1)
    if ((size_t)r * row <= MX_SLAB_BYTES) return r;
  return row <= MX_SLAB_BYTES_ONE ? 1 : 0;
}

template <int R>
static int launch_split_slab(bool a_role, int rows, int K, int Kp, const double2* X, long long ld,
                             long long st, __half* out, int* ex, int batch, const int* steps,
                             int step, const int* apart, cudaStream_t stream) {
  static int done_a[64], done_b[64];
  const int smem = R * (a_role ? slab_a_stride<R>(K) : K) * (int)sizeof(double2);
  dim3 g((unsigned)((rows + R - 1) / R), batch);
  if (a_role) {
    EUV_CUDA_TRY(ensure_smem(split_a_slab_kernel<R>, smem, done_a));
    EUV_CUDA_TRY(launch_dependent(split_a_slab_kernel<R>, g, dim3(MX_SLAB_THREADS), smem, stream,
                                  rows, K, Kp, X, ld, st, out, ex, steps, step, apart));
  } else {
    EUV_CUDA_TRY(ensure_smem(split_b_slab_kernel<R>, smem, done_b));
    EUV_CUDA_TRY(launch_dependent(split_b_slab_kernel<R>, g, dim3(MX_SLAB_THREADS), smem, stream, K,
                                  rows, Kp, X, ld, st, out, ex, steps, step, apart));
  }
  EUV_LAUNCH_CHECK();
  return EUV_OK;
}

// Split of one operand: A role (rows = M) or B role (rows = N, the columns).
static int split_operand(bool a_role, int rows, int K, int Kp, const double2* X, long long ld,
                         long long st, __half* out, int* ex, int batch, const int* steps, int step,
                         const int* apart, cudaStream_t stream) {
  switch (split_slab_rows(K)) {
    case 8: return launch_split_slab<8>(a_role, rows, K, Kp, X, ld, st, out, ex, batch, steps, step, apart, stream);
    case 4: return launch_split_slab<4>(a_role, rows, K, Kp, X, ld, st, out, ex, batch, steps, step, apart, stream);
    case 2: return launch_split_slab<2>(a_role, rows, K, Kp, X, ld, st, out, ex, batch, steps, step, apart, stream);
    case 1: return launch_split_slab<1>(a_role, rows, K, Kp, X, ld, st, out, ex, batch, steps, step, apart, stream);
    default: break;
  }
  if (a_role) {
    dim3 g((rows + 31) / 32, batch), t(32, 8);
    split_a_kernel<<<g, t, 0, stream>>>(rows, K, Kp, X, ld, st, out, ex, steps, step, apart);
  } else {
    dim3 gb((unsigned)((rows + 7) / 8), batch);
    split_b_kernel<<<gb, 256, 0, stream>>>(K, rows, Kp, X, ld, st, out, ex, steps, step, apart);
  }
  EUV_LAUNCH_CHECK();
  return EUV_OK;
}

// ------------------------------------------------------------------ host
// planes tensor [batch*4][rows][kp] fp16 -> 3-D map (kp, rows, batch*4), box (32, box_rows, 1)
static int make_map(CUtensorMap* map, __half* base, int rows, int kp, int nplanes, int box_rows) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) {
    euv_set_error("cuTensorMapEncodeTiled is not available from the driver");
    return EUV_ERR_CUDA;
  }
  const cuuint64_t dims[3] = {(cuuint64_t)kp, (cuuint64_t)rows, (cuuint64_t)nplanes};
  const cuuint64_t strides[2] = {(cuuint64_t)kp * 2, (cuuint64_t)kp * 2 * rows};
  const cuuint32_t box[3] = {(cuuint32_t)MX_BK, (cuuint32_t)box_rows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, base, dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    euv_set_error("cuTensorMapEncodeTiled failed (%d) for the fp16 planes", (int)r);
    return EUV_ERR_CUDA;
  }
  return EUV_OK;
}

static inline int round_up(int x, int a) { return (x + a - 1) / a * a; }

size_t gemm_mixed_workspace_bytes(int m, int n, int k, int batch) {
  const size_t kp = (size_t)round_up(k > 0 ? k : 1, MX_BK);
  size_t a = (size_t)batch * MX_PLANES * (size_t)m * kp * 2;
  size_t b = (size_t)batch * MX_PLANES * (size_t)n * kp * 2;
  const size_t ea = ((size_t)batch * (size_t)m * 4 + 1023) & ~(size_t)1023;
  const size_t eb = ((size_t)batch * (size_t)n * 4 + 1023) & ~(size_t)1023;
  a = (a + 1023) & ~(size_t)1023;
  b = (b + 1023) & ~(size_t)1023;
  return a + ea + b + eb + 1024;
}

int gemm_mixed(int m, int n, int k, cplx alpha, const double* scale, const double2* a,
               long long lda, long long sa, const double2* b, long long ldb, long long sb,
               cplx beta, double2* c, long long ldc, long long sc, cplx diag, int batch,
               const int* steps, int step, void* work, size_t work_bytes, int* status,
               cudaStream_t stream, int reuse, const GemmTerms& terms) {
  if (m <= 0 || n <= 0 || batch <= 0) return EUV_OK;
  if (terms.apart && (m != k || (n != k && n != 2 * k) || alpha.x != 1.0 || alpha.y != 0.0 ||
                      scale || beta.x != 0.0 || beta.y != 0.0 || steps)) {
    euv_set_error("gemm_mixed: diagonals apart are for plain products of square blocks");
    return EUV_ERR_BAD_ARG;
  }
  if (k <= 0 || batch > 65535 || (size_t)batch * MX_PLANES > 0x7fffffff) {
    euv_set_error("gemm_mixed: unsupported shape");
    return EUV_ERR_BAD_ARG;
  }
  const int kp = round_up(k, MX_BK);
  const size_t need = gemm_mixed_workspace_bytes(m, n, k, batch);
  if (work == nullptr || work_bytes < need ||
      (reinterpret_cast<uintptr_t>(work) & 255u) != 0) {
    euv_set_error("gemm_mixed: workspace too small or misaligned (%zu < %zu)", work_bytes, need);
    return EUV_ERR_WORKSPACE;
  }
  // A's planes and exponents come first, so that a call with the same A and
  // another column count n finds them where the last call left them
  char* w = reinterpret_cast<char*>(work);
  __half* pa = reinterpret_cast<__half*>(w);
  size_t abytes = ((size_t)batch * MX_PLANES * (size_t)m * kp * 2 + 1023) & ~(size_t)1023;
  int* ea = reinterpret_cast<int*>(w + abytes);
  abytes += ((size_t)batch * (size_t)m * 4 + 1023) & ~(size_t)1023;
  __half* pb = reinterpret_cast<__half*>(w + abytes);
  size_t bbytes = ((size_t)batch * MX_PLANES * (size_t)n * kp * 2 + 1023) & ~(size_t)1023;
  int* eb = reinterpret_cast<int*>(w + abytes + bbytes);
  size_t ebytes = ((size_t)batch * (size_t)n * 4 + 1023) & ~(size_t)1023;
  // the caller's sticky status word, else a per-call word in the workspace
  int* err = status;
  if (err == nullptr) {
    err = reinterpret_cast<int*>(w + abytes + bbytes + ebytes);
    EUV_CUDA_TRY(cudaMemsetAsync(err, 0, sizeof(int), stream));
  }
  // reuse bit 0 / bit 1: the A / B planes (and scale exponents) in this
  // workspace are already those of the operand (the caller's previous call
  // split the same unchanged matrix in the same role and shape; for A the
  // column count n may differ), so the split is skipped
  // entries the product leaves alone (GemmTerms::need) need no planes of B either
  // (A's are kept whole for a caller that reuses them)
  const int* sk = terms.need ? terms.need : steps;
  const int sk_at = terms.need ? terms.need_above : step;
  int rc;
  if (!(reuse & 1) &&
      (rc = split_operand(true, m, k, kp, a, lda, sa, pa, ea, batch, steps, step, terms.apart,
                          stream)))
    return rc;
  if (!(reuse & 2) &&
      (rc = split_operand(false, n, k, kp, b, ldb, sb, pb, eb, batch, sk, sk_at, terms.apart,
                          stream)))
    return rc;
  CUtensorMap ta, tb;
  rc = make_map(&ta, pa, m, kp, batch * MX_PLANES, MX_BM);
  if (rc) return rc;
  rc = make_map(&tb, pb, n, kp, batch * MX_PLANES, MX_BN);
  if (rc) return rc;
  MixedArgs p;
  p.m = m;
  p.n = n;
  p.kp = kp;
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
  p.err = err;
  p.ea = ea;
  p.eb = eb;
  dim3 grid((m + MX_BM - 1) / MX_BM, (n + MX_BN - 1) / MX_BN, batch);
  const int nx = terms.apart ? 3 : terms.cin2 ? 2 : (beta.x != 0.0 || beta.y != 0.0) ? 1 : 0;
  static int smem_done[4][64];
  auto launch = [&](auto kernel, int* done, size_t smem = MX_SMEM) -> int {
    EUV_CUDA_TRY(ensure_smem(kernel, (int)smem, done));
    EUV_CUDA_TRY(launch_dependent(kernel, grid, dim3(MX_THREADS), smem, stream, ta, tb, p));
    EUV_LAUNCH_CHECK();
    return EUV_OK;
  };
  if (nx == 0) return launch(gemm_split3_kernel<0>, smem_done[0]);
  if (nx == 1) return launch(gemm_split3_kernel<1>, smem_done[1]);
  if (nx == 2) return launch(gemm_split3_kernel<2>, smem_done[2]);
  return launch(gemm_split3_kernel<3>, smem_done[3], MX_SMEM_DIAG);
}

}  // namespace euv

using namespace euv;

extern "C" size_t euv_zgemm_mixed_workspace_bytes(int m, int n, int k, int batch) {
  if (m <= 0 || n <= 0 || k <= 0 || batch <= 0) return 0;
  return gemm_mixed_workspace_bytes(m, n, k, batch);
}

extern "C" int euv_zgemm_mixed(int m, int n, int k, euv_c64 alpha, const double* d_scale,
                                const euv_c64* d_a, int lda, long long stride_a,
                                const euv_c64* d_b, int ldb, long long stride_b, euv_c64 beta,
                                euv_c64* d_c, int ldc, long long stride_c, euv_c64 diag,
                                int batch, const int* d_steps, int step, void* d_work,
                                size_t work_bytes, int* d_status, void* stream) {
  if (m <= 0 || n <= 0 || k <= 0 || batch <= 0 || lda < m || ldc < m || ldb < k || !d_a ||
      !d_b || !d_c || (d_steps != nullptr && (m != n || m != k))) {
    euv_set_error("euv_zgemm_mixed: bad arguments (m=%d n=%d k=%d)", m, n, k);
    return EUV_ERR_BAD_ARG;
  }
  return gemm_mixed(m, n, k, fromc(alpha), d_scale, reinterpret_cast<const double2*>(d_a), lda,
                    stride_a, reinterpret_cast<const double2*>(d_b), ldb, stride_b, fromc(beta),
                    reinterpret_cast<double2*>(d_c), ldc, stride_c, fromc(diag), batch, d_steps,
                    step, d_work, work_bytes, d_status, (cudaStream_t)stream, 0, GemmTerms{});
}
