// Shared helpers of the sm_103a kernels behind the C ABI in include/axisym_gb300.h.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <string>

#include "../../include/axisym_gb300.h"

namespace axi {

// Per-thread message of the last failing entry point (read by axi_last_error).
void set_error(const char* fmt, ...);
void clear_error();

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

inline int ceil_div(long long a, long long b) { return static_cast<int>((a + b - 1) / b); }

// Turns a launch error into AXI_ERR_CUDA with a message naming the kernel.
inline int launch_status(const char* what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("%s: CUDA launch failed: %s", what, cudaGetErrorString(e));
    return AXI_ERR_CUDA;
  }
  return AXI_OK;
}

inline int check_grid(const char* what, int nr, int nz, int min_nr = 3, int min_nz = 3) {
  if (nr < min_nr || nz < min_nz) {
    set_error("%s: grid %d x %d is smaller than %d x %d", what, nr, nz, min_nr, min_nz);
    return AXI_ERR_INVALID;
  }
  return AXI_OK;
}

inline int check_ptr(const char* what, const void* p, const char* name) {
  if (p == nullptr) {
    set_error("%s: %s is null", what, name);
    return AXI_ERR_INVALID;
  }
  return AXI_OK;
}

// Every pointer in `ptrs` non-null; `names` names them in the same order.
inline int check_ptrs(const char* what, std::initializer_list<const void*> ptrs,
                      std::initializer_list<const char*> names) {
  const char* const* n = names.begin();
  for (const void* p : ptrs) {
    const char* name = n != names.end() ? *n++ : "pointer";
    if (p == nullptr) {
      set_error("%s: %s is null", what, name);
      return AXI_ERR_INVALID;
    }
  }
  return AXI_OK;
}

// Number of SMs on the current device (cached per device).
int sm_count();

// Launch with programmatic dependent launch (the kernel may start while its
// predecessor on the stream runs; it waits with pdl_wait before it touches
// what that one reads or writes) and, with cluster > 1, thread-block clusters.
template <typename... P, typename... A>
inline int launch_chain(bool pdl, const char* what, void (*kernel)(P...), dim3 grid, dim3 block,
                        size_t smem, cudaStream_t s, int cluster, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  cfg.attrs = at;
  cfg.numAttrs = 0;
  if (pdl) {
    at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    at[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    at[cfg.numAttrs].val.clusterDim.x = cluster;
    at[cfg.numAttrs].val.clusterDim.y = at[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
  if (e != cudaSuccess) {
    set_error("%s: CUDA launch failed: %s", what, cudaGetErrorString(e));
    cudaGetLastError();
    return AXI_ERR_CUDA;
  }
  return AXI_OK;
}
// Waits until the grids this one depends on are complete and their writes visible.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the next grid of a chain start once every block got here.
__device__ __forceinline__ void pdl_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

}  // namespace axi

#define AXI_TRY(expr)            \
  do {                           \
    int _st = (expr);            \
    if (_st != AXI_OK) return _st; \
  } while (0)

// Rounded arithmetic that the compiler may not contract into FMA: used where
// results must match the reference's numpy evaluation bit for bit.
template <typename T> __device__ __forceinline__ T rn_mul(T a, T b);
template <typename T> __device__ __forceinline__ T rn_add(T a, T b);
template <typename T> __device__ __forceinline__ T rn_sub(T a, T b);
template <typename T> __device__ __forceinline__ T rn_div(T a, T b);
template <> __device__ __forceinline__ double rn_mul(double a, double b) { return __dmul_rn(a, b); }
template <> __device__ __forceinline__ double rn_add(double a, double b) { return __dadd_rn(a, b); }
template <> __device__ __forceinline__ double rn_sub(double a, double b) { return __dsub_rn(a, b); }
template <> __device__ __forceinline__ double rn_div(double a, double b) { return __ddiv_rn(a, b); }
template <> __device__ __forceinline__ float rn_mul(float a, float b) { return __fmul_rn(a, b); }
template <> __device__ __forceinline__ float rn_add(float a, float b) { return __fadd_rn(a, b); }
template <> __device__ __forceinline__ float rn_sub(float a, float b) { return __fsub_rn(a, b); }
template <> __device__ __forceinline__ float rn_div(float a, float b) { return __fdiv_rn(a, b); }

// Division by a divisor that serves several quotients: the same correctly
// rounded quotients as the / operator, for 4 FP64 instructions each instead of
// about 20 (FP64 issues at 1/64 of the FP32 rate on GB300, so the FP64 stencils
// are bound by exactly these). With the reciprocal held as y_h + y_l
// (y_h = RN(1 / b), y_l its remainder), q = RN(a y_h + RN(a y_l)) is within one
// unit of the quotient (Brisebarre, Muller and Raina, "Accelerating correctly
// rounded floating-point division when the divisor is known in advance", IEEE
// TC 53, 2004), so r = a - q b is exact and RN(q + r y_h) is correctly rounded
// (Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM JRD 34, 1990). Dividends and divisors outside the exponent
// range where all of it stays normal take the plain division; a zero dividend
// gives its signed zero.
template <typename T>
struct KnownDivisor {
  T b;
  KnownDivisor() = default;
  __host__ __device__ __forceinline__ explicit KnownDivisor(T d) : b(d) {}
  __device__ __forceinline__ T quotient(T a) const { return rn_div(a, b); }
};

template <>
struct KnownDivisor<double> {
  double b, yh, yl;
  int ok;
  KnownDivisor() = default;
  __host__ __device__ __forceinline__ explicit KnownDivisor(double d) : b(d) {
#ifdef __CUDA_ARCH__
    const unsigned int e = ((unsigned int)__double2hiint(d) >> 20) & 0x7ffu;
    yh = __drcp_rn(d);
    yl = __dmul_rn(__fma_rn(-yh, d, 1.0), yh);
#else
    unsigned long long bits;
    memcpy(&bits, &d, sizeof(bits));
    const unsigned int e = (unsigned int)(bits >> 52) & 0x7ffu;
    yh = 1.0 / d;
    yl = std::fma(-yh, d, 1.0) * yh;
#endif
    ok = e - 623u <= 800u;
  }
  __device__ __forceinline__ double quotient(double a) const {
    const unsigned int hi = (unsigned int)__double2hiint(a);
    if (ok) {
      if (((hi >> 20) & 0x7ffu) - 523u <= 1000u) {
        const double q = __fma_rn(a, yh, __dmul_rn(a, yl));
        return __fma_rn(__fma_rn(-q, b, a), yh, q);
      }
      if (((hi << 1) | (unsigned int)__double2loint(a)) == 0) return __dmul_rn(a, yh);
    }
    return __ddiv_rn(a, b);
  }
};

// Bit tests that need no FP64 instruction.
__device__ __forceinline__ bool is_pos_zero(double x) { return __double_as_longlong(x) == 0; }
__device__ __forceinline__ bool is_zero_bits(double x) { return (__double_as_longlong(x) << 1) == 0; }
__device__ __forceinline__ int exponent_bits(double x) {
  return (__double2hiint(x) >> 20) & 0x7ff;
}
// (double)x without the FP64 pipe, which converts at the FP64 rate: a normal
// float is the same number with its exponent rebiased.
static __device__ __noinline__ double widen_plain(float x) { return (double)x; }
__device__ __forceinline__ double widen(float x) {
  const unsigned int b = __float_as_uint(x), e = (b >> 23) & 0xffu;
  if (e - 1u < 254u)
    return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + (896u << 20))),
                            (int)(b << 29));
  return (b << 1) == 0 ? __hiloint2double((int)b, 0) : widen_plain(x);
}
// x with its sign flipped where `flip` (the compiler negates with an FP64 add)
__device__ __forceinline__ double flip_sign(double x, bool flip) {
  return __hiloint2double(__double2hiint(x) ^ (flip ? (int)0x80000000 : 0), __double2loint(x));
}
__device__ __forceinline__ float flip_sign(float x, bool flip) { return flip ? -x : x; }

// Outside its blend band the smoothed Heaviside (kernels/smooth_Heaviside.py:10-14)
// of a finite phi, from a finite old value, is exactly 1 or 0: the blend's
// bracket is finite there and is multiplied by zero. True: `h` holds it (no
// FP64 instruction); false: the caller evaluates the expression. w > 0, normal.
__device__ __forceinline__ bool heaviside_outside(double h_old, double phi, double w, double& h) {
  const long long a = __double_as_longlong(phi) & 0x7fffffffffffffffll;
  if (exponent_bits(h_old) == 0x7ff || a < __double_as_longlong(w) ||
      (int)(a >> 52) - exponent_bits(w) > 1000 || (a >> 52) > 1023 + 900 ||
      (unsigned int)(exponent_bits(w) - 1) >= 0x7feu || __double_as_longlong(w) < 0)
    return false;
  h = __double_as_longlong(phi) >= 0 ? 1.0 : 0.0;
  return true;
}

// Host-side product of two scalars (kept separate so no contraction applies).
template <typename T> inline T rn_host_mul(T a, T b) { return a * b; }

template <typename T> __device__ __forceinline__ T dev_sin(T x);
template <> __device__ __forceinline__ double dev_sin(double x) { return sin(x); }
template <> __device__ __forceinline__ float dev_sin(float x) { return sinf(x); }

template <typename T> struct Pi;
template <> struct Pi<double> { static constexpr double v = 3.141592653589793; };
template <> struct Pi<float> { static constexpr float v = 3.14159265f; };

// Error-free float transformations (Knuth's two-sum; the FMA form of the
// exact product): a + b = s + e and a * b = p + e exactly. Used where float
// values are carried as unevaluated pairs (hi + lo) to keep more than float
// precision in float storage and arithmetic.
namespace axi_eft {
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}
__device__ __forceinline__ void two_prod(float a, float b, float& p, float& e) {
  p = __fmul_rn(a, b);
  e = fmaf(a, b, -p);
}
// (hi, lo) + v as a renormalised pair: hi' is the rounded sum, lo' the
// remainder; hi' + lo' = hi + lo + v up to the rounding of the low part.
__device__ __forceinline__ void pair_add(float& hi, float& lo, float v) {
  float s, e, h2, l2;
  two_sum(hi, v, s, e);
  two_sum(s, __fadd_rn(lo, e), h2, l2);
  hi = h2;
  lo = l2;
}
}  // namespace axi_eft
