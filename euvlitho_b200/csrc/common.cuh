// Shared device helpers for the EUV mask-3D library (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>
#include "../../include/euvl_b200.h"

namespace euv {

struct cplx {
  double x, y;
};

__host__ __device__ __forceinline__ cplx mk(double a, double b) { cplx r; r.x = a; r.y = b; return r; }
__host__ __device__ __forceinline__ cplx operator+(cplx a, cplx b) { return mk(a.x + b.x, a.y + b.y); }
__host__ __device__ __forceinline__ cplx operator-(cplx a, cplx b) { return mk(a.x - b.x, a.y - b.y); }
__host__ __device__ __forceinline__ cplx operator-(cplx a) { return mk(-a.x, -a.y); }
__host__ __device__ __forceinline__ cplx operator*(cplx a, cplx b) {
  return mk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__host__ __device__ __forceinline__ cplx operator*(double s, cplx a) { return mk(s * a.x, s * a.y); }
__host__ __device__ __forceinline__ cplx operator*(cplx a, double s) { return mk(s * a.x, s * a.y); }
__host__ __device__ __forceinline__ cplx cmul_i(cplx a) { return mk(-a.y, a.x); }  // i*a
__host__ __device__ __forceinline__ cplx cdiv(cplx a, cplx b) {
  // Smith's algorithm (scaled division, avoids overflow of |b|^2)
  if (fabs(b.x) >= fabs(b.y)) {
    double r = b.y / b.x, d = b.x + b.y * r;
    return mk((a.x + a.y * r) / d, (a.y - a.x * r) / d);
  } else {
    double r = b.x / b.y, d = b.x * r + b.y;
    return mk((a.x * r + a.y) / d, (a.y * r - a.x) / d);
  }
}
__host__ __device__ __forceinline__ double cabs1(cplx a) { return fabs(a.x) + fabs(a.y); }
__host__ __device__ __forceinline__ double cabs(cplx a) { return hypot(a.x, a.y); }

// Principal square root, branch cut on the negative real axis with the sign of
// the imaginary part deciding the side (C99 csqrt semantics), from
// sqrt(z) = sqrt((|z|+x)/2) + i sign(y) sqrt((|z|-x)/2), evaluated without
// cancellation: t = sqrt((|z|+|x|)/2), then the other part is |y|/(2t).
__host__ __device__ __forceinline__ cplx csqrt_p(cplx z) {
  double x = z.x, y = z.y;
  if (x == 0.0 && y == 0.0) return mk(0.0, y);
  double t = sqrt(0.5 * (hypot(x, y) + fabs(x)));
  if (x >= 0.0) return mk(t, y / (2.0 * t));
  return mk(fabs(y) / (2.0 * t), copysign(t, y));
}

// Further terms of a batched GEMM, C = alpha A B + beta Cin + beta2 Cin2 + diag I:
// Cin is C itself unless given, Cin2 is optional, both with C's leading dimension;
// beta_b and beta2_b multiply beta and beta2 per batch entry (beta_b null: 1).
struct GemmTerms {
  const double2* cin = nullptr;
  long long scin = 0;  // batch strides
  const double2* beta_b = nullptr;
  const double2* cin2 = nullptr;
  long long scin2 = 0;
  double2 beta2 = {0.0, 0.0};
  const double2* beta2_b = nullptr;
  // entries with need[b] <= need_above are left as they are (C untouched)
  const int* need = nullptr;
  int need_above = 0;
  // steps come in pairs (0, 1), (2, 3) ... that end in the buffer they began in: an
  // entry inactive in both is left alone, one active in the first only is copied
  // back by the second
  bool paired = false;
  // FP64 form: three real products per complex one (zgemm.cu)
  bool three = false;
  // mixed form, C = A B (m = k, n = k or 2 k): entries with apart[b] != 0 multiply the
  // operands without the diagonals of their k x k blocks and add those rows and columns
  // in FP64 (gemm_mixed.cu)
  const int* apart = nullptr;
};

// Columns of a matrix that are source slots: column c >= first is slot c - first, and one
// with order[b * stride + slot] < 0 is empty (a zero column, which swaps, solves and updates
// leave as it is).
struct Slots {
  const int* order = nullptr;  // null: every column counts
  long long stride = 0;
  int first = 0;
  __device__ __forceinline__ bool empty(int b, int c) const {
    return order != nullptr && c >= first && order[b * stride + (c - first)] < 0;
  }
  // the same columns counted from column c0
  __host__ __device__ Slots from(int c0) const { return Slots{order, stride, first - c0}; }
};

// Whether an inactive entry (step >= steps) of a step-predicated GEMM copies A to C.
__host__ __device__ __forceinline__ bool step_copies(bool paired, int steps, int step) {
  return !paired || ((step & 1) && steps == step);
}

// exp(z) for complex z.
__host__ __device__ __forceinline__ cplx cexp_(cplx z) {
  double e = exp(z.x);
  double s, c;
  sincos(z.y, &s, &c);
  return mk(e * c, e * s);
}

__device__ __forceinline__ cplx ld(const euv_c64* p) {
  double2 v = *reinterpret_cast<const double2*>(p);
  return mk(v.x, v.y);
}
__device__ __forceinline__ void st(euv_c64* p, cplx v) {
  *reinterpret_cast<double2*>(p) = make_double2(v.x, v.y);
}
__host__ __device__ __forceinline__ cplx fromc(euv_c64 a) { return mk(a.re, a.im); }

// First statement of a kernel launched by launch_dependent (no effect otherwise).
__device__ __forceinline__ void dependent_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// The one spin loop of every device wait in the library: polls ready() and,
// every 256 polls, abort() and the %globaltimer clock.  Returns 1 when ready,
// 0 when aborted (another role gave up), -1 after limit_ns nanoseconds.
template <class Ready, class Abort>
__device__ __forceinline__ int bounded_spin(Ready ready, Abort abort, unsigned long long limit_ns) {
  const unsigned long long t0 = globaltimer();
  for (uint32_t it = 0;; ++it) {
    if (ready()) return 1;
    if ((it & 255u) == 255u) {
      if (abort()) return 0;
      if (globaltimer() - t0 > limit_ns) return -1;
    }
  }
}

}  // namespace euv

#define EUV_CUDA_TRY(expr)                                     \
  do {                                                         \
    cudaError_t _e = (expr);                                   \
    if (_e != cudaSuccess) {                                   \
      euv_set_error("%s:%d CUDA error %s (%s)", __FILE__,      \
                    __LINE__, cudaGetErrorString(_e), #expr);  \
      return EUV_ERR_CUDA;                                     \
    }                                                          \
  } while (0)

// Every kernel launch of the library is followed by this check, which also
// counts the launch (euv_kernel_launches()).
#define EUV_LAUNCH_CHECK()        \
  do {                            \
    euv_count_launch();           \
    EUV_CUDA_TRY(cudaGetLastError()); \
  } while (0)

extern "C" void euv_set_error(const char* fmt, ...);
extern "C" void euv_count_launch(void);

namespace euv {
// The tuning table's pick for (knob, k0, k1), 0 when there is none (api.cu).
int tune_lookup(int knob, int k0, int k1);

// A launch that may be set up while its predecessor on the stream still runs: the
// kernel begins with dependent_begin(), which waits for that grid's end and memory.
// For the chains of short launches that the slabs, the LU and the spectra are: N = 121,
// 8 slices 1.70 -> 1.45 ms, ragged clip with refresh_sigma 2.40 -> 2.11, N = 961 a
// hundredth or two.  No kernel lets its successor in before it ends: with
// griddepcontrol.launch_dependents at its start the successor's CTAs take the places of
// CTAs still to come (1.72 and 2.28 ms for the two).  A kernel that follows an event of
// another stream is launched plainly.
template <typename... KA, typename... A>
inline cudaError_t launch_dependent(void (*kernel)(KA...), dim3 grid, dim3 block, size_t smem,
                                    cudaStream_t stream, A... args) {
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, KA(args)...);
}

// Raise a kernel's dynamic shared-memory limit once per device (the first call
// happens outside any stream capture; later calls do nothing).
template <typename K>
inline cudaError_t ensure_smem(K kernel, int bytes, int* done_per_device) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (__atomic_load_n(&done_per_device[dev], __ATOMIC_ACQUIRE) >= bytes) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) __atomic_store_n(&done_per_device[dev], bytes, __ATOMIC_RELEASE);
  return e;
}
}  // namespace euv
