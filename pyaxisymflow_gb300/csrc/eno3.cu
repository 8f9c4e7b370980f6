// ENO3 Euler-forward advection on the meridional plane, axis mirror by index
// reflection.
//
// The reference builds (2 nr, nz) buffers whose lower half is the field flipped
// about the axis (with parity +1 or -1), runs four pystencils flux kernels on
// the interior [2:-2, 2:-2] of that buffer and copies the upper half back
// (kernels/advect_vorticity_via_eno3.py:28-42). Only the upper half survives,
// so this kernel evaluates exactly the upper-half cells and reads row -1-k of
// the mirror as parity * row k. Upper-half rows nr-2, nr-1 and columns 0, 1,
// nz-2, nz-1 lie in the pystencils ghost layers: they receive a zero flux.
//
// Each face value is shared by its two cells: the x_back kernel of cell c
// (pyst_kernels/advection_flux.py:61-73) evaluates the same upwind selector
// (u[c] > -u[c-1] is u[c-1] > -u[c]) and the same three products, in the same
// order, as the x_front kernel of cell c-1 (:32-44), so one face routine serves
// both. The flux accumulation keeps the reference's statement order:
// flux = 0; += a F_x_front; -= a F_x_back; += a F_y_front; -= a F_y_back;
// field += flux (pyst_kernels/advection_timestep.py:45-54), a = -dt/dx.
#include "axi_common.cuh"

namespace {

// Upwind selector u0 > -u1 (advection_flux.py:33). Doubles compare as integers
// (sign and magnitude; zeros equal), which spares an FP64 instruction; NaN and
// infinities take the comparison itself, out of line (inlined it would run for
// every cell under a predicate, at full cost).
__device__ __noinline__ bool upwind_plain(double u0, double u1) { return u0 > -u1; }
__device__ __forceinline__ bool upwind(float u0, float u1) { return u0 > -u1; }
__device__ __forceinline__ bool upwind(double u0, double u1) {
  const long long b0 = __double_as_longlong(u0), b1 = __double_as_longlong(u1);
  const long long m0 = b0 & 0x7fffffffffffffffll, m1 = b1 & 0x7fffffffffffffffll;
  if (exponent_bits(u0) == 0x7ff || exponent_bits(u1) == 0x7ff) return upwind_plain(u0, u1);
  return (b0 < 0 ? -m0 : m0) > (b1 < 0 ? m1 : -m1);
}

// Conservative face value of f*u between cells 0 and 1 (advection_flux.py:34-43):
// the operands of the upwind side selected first, then evaluated once.
template <typename T>
__device__ __forceinline__ T face_cons(T fm1, T f0, T f1, T f2, T um1, T u0, T u1, T u2) {
  const T third = T(1) / T(3), five6 = T(5) / T(6), sixth = T(1) / T(6);
  const bool l = upwind(u0, u1);
  const T a = rn_add(rn_mul(rn_mul(third, l ? f1 : f0), l ? u1 : u0),
                     rn_mul(rn_mul(five6, l ? f0 : f1), l ? u0 : u1));
  return rn_sub(a, rn_mul(rn_mul(sixth, l ? fm1 : f2), l ? um1 : u2));
}

// Non-conservative face value of f between cells 0 and 1 (advection_flux.py:193-199).
template <typename T>
__device__ __forceinline__ T face_noncons(T fm1, T f0, T f1, T f2, bool l) {
  const T third = T(1) / T(3), five6 = T(5) / T(6), sixth = T(1) / T(6);
  return rn_sub(rn_add(rn_mul(third, l ? f1 : f0), rn_mul(five6, l ? f0 : f1)),
                rn_mul(sixth, l ? fm1 : f2));
}

// A reference-map cell of a warp (all lanes call it): its new value. Out of
// line, so that none of it runs ahead of the test for an all-zero warp.
template <typename T>
__device__ __noinline__ T noncons_cell(T fm1, T f0, T f1, T f2, T gm2, T gm1, T g1, T g2, T v0, T v1,
                                       T wm1, T w0, T w1, T a, bool inner) {
  const T xf = face_noncons(fm1, f0, f1, f2, upwind(v0, v1));
  const T xb = __shfl_up_sync(0xffffffffu, xf, 1);
  const T yf = face_noncons(gm1, f0, g1, g2, upwind(w0, w1));
  const T yb = face_noncons(gm2, gm1, f0, g1, upwind(wm1, w0));
  T flux = T(0);
  flux = rn_add(flux, rn_mul(rn_mul(a, xf), v0));
  flux = rn_sub(flux, rn_mul(rn_mul(a, xb), v0));
  flux = rn_add(flux, rn_mul(rn_mul(a, yf), w0));
  flux = rn_sub(flux, rn_mul(rn_mul(a, yb), w0));
  return rn_add(f0, inner ? flux : T(0));
}

// 0 for +0 only
__device__ __forceinline__ unsigned int value_bits(float x) { return __float_as_uint(x); }
__device__ __forceinline__ unsigned int value_bits(double x) {
  return (unsigned int)__double2hiint(x) | (unsigned int)__double2loint(x);
}
__device__ __forceinline__ bool finite_bits(float x) {
  return (__float_as_uint(x) & 0x7f800000u) != 0x7f800000u;
}
__device__ __forceinline__ bool finite_bits(double x) { return exponent_bits(x) != 0x7ff; }

// One Euler step for NF fields sharing the velocity (u_z even, u_r odd).
// src[k] holds the pre-step copy of field k, dst[k] (a copy of it on entry)
// receives the new values.
//
// Bound by FP64 issue in the double form. A z face serves its two cells: a
// warp covers 31 cells of a row, lane l holding the face behind its cell and
// passing it to lane l + 1 (lane 0 only forms a face). The conservative form
// also walks up `strip` rows keeping the r face between them: 25 instructions
// per cell where forming all four faces took 56. A warp whose reference-map
// stencils are all +0 (outside the solid and its extrapolation band) leaves
// them without any. Measured at 1024 x 512: omega 60 -> 43 us, both eta fields
// 90 -> 18 us.
constexpr int ENO_WARPS = 8;   // warps per block, one strip of rows each
constexpr int ENO_COLS = 31;   // cells per warp

template <typename T, int NF, bool CONS>
__global__ void __launch_bounds__(32 * ENO_WARPS)
    eno3_step_kernel(T* __restrict__ dst0, T* __restrict__ dst1, const T* __restrict__ src0,
                     const T* __restrict__ src1, bool odd0, bool odd1, const T* __restrict__ uz,
                     const T* __restrict__ ur, int nr, int nz, T a,
                     const double* __restrict__ dt_dev, T dx, int strip) {
  __shared__ T s_a;
  // a device-resident time step (the soft-sphere loop): a = -(dt / dx)
  if (threadIdx.x == 0 && threadIdx.y == 0)
    s_a = dt_dev ? -rn_div(static_cast<T>(dt_dev[0]), dx) : a;
  __syncthreads();
  a = s_a;
  const int lane = threadIdx.x;
  const int j = blockIdx.x * ENO_COLS - 1 + lane;
  const int first = (blockIdx.y * ENO_WARPS + threadIdx.y) * strip;
  const int last = min(first + strip, nr);
  const bool cell = lane > 0 && j < nz;
  const bool inner_j = lane > 0 && j >= 2 && j <= nz - 3;
  // Every load of a row is unconditional (columns and rows clamped into the
  // grid, the clamped values unused), so that all are in flight at once.
  auto col = [nz](int x) { return min(max(x, 0), nz - 1); };
  const int cm2 = col(j - 2), cm1 = col(j - 1), c0 = col(j), c1 = col(j + 1), c2 = col(j + 2);
  // rows i - 2 .. i + 2 at column j; below the axis mirrored
  auto below2 = [=](int i) { return (long long)(i >= 2 ? i - 2 : 1 - i) * nz + c0; };
  auto below1 = [=](int i) { return (long long)(i >= 1 ? i - 1 : -i) * nz + c0; };
  T yb = T(0);  // conservative: r face below row i
  if (CONS && first < last) {
    const long long c = (long long)first * nz + c0, up = (long long)min(first + 1, nr - 1) * nz + c0;
    yb = face_cons(flip_sign(src0[below2(first)], odd0 && first < 2),
                   flip_sign(src0[below1(first)], odd0 && first < 1), src0[c], src0[up],
                   flip_sign(ur[below2(first)], first < 2), flip_sign(ur[below1(first)], first < 1),
                   ur[c], ur[up]);
  }
  for (int i = first; i < last; ++i) {
    const long long row = (long long)i * nz;
    const long long rm2 = below2(i), rm1 = below1(i);
    const long long r1 = (long long)min(i + 1, nr - 1) * nz + c0;
    const long long r2 = (long long)min(i + 2, nr - 1) * nz + c0;
    const bool inner = inner_j && i <= nr - 3;
    const T v0 = uz[row + c0], v1 = uz[row + c1];
    const T w0 = ur[row + c0], w1 = ur[r1];
    const T wm1 = flip_sign(ur[rm1], i < 1);
    T vm1 = T(0), v2 = T(0), w2 = T(0);
    if (CONS) {
      vm1 = uz[row + cm1];
      v2 = uz[row + c2];
      w2 = ur[r2];
    }
    T fm2[NF], fm1[NF], f0[NF], f1[NF], f2[NF], gm2[NF], gm1[NF], g1[NF], g2[NF];
    // every value of the stencils +0 (tested as integers: a comparison with zero
    // would be an FP64 instruction per value)
    unsigned int zero_bits = 0;
#pragma unroll
    for (int k = 0; k < NF; ++k) {
      const T* __restrict__ src = k == 0 ? src0 : src1;
      fm1[k] = src[row + cm1];
      f0[k] = src[row + c0];
      f1[k] = src[row + c1];
      f2[k] = src[row + c2];
      gm1[k] = src[rm1];
      g1[k] = src[r1];
      g2[k] = src[r2];
      if (!CONS) {
        fm2[k] = src[row + cm2];
        gm2[k] = src[rm2];
        zero_bits |= value_bits(fm2[k]) | value_bits(fm1[k]) | value_bits(f0[k]) |
                     value_bits(f1[k]) | value_bits(f2[k]) | value_bits(gm2[k]) |
                     value_bits(gm1[k]) | value_bits(g1[k]) | value_bits(g2[k]);
      }
      const bool odd = k == 0 ? odd0 : odd1;
      gm1[k] = flip_sign(gm1[k], i < 1 && odd);
      if (!CONS) gm2[k] = flip_sign(gm2[k], i < 2 && odd);
    }
    // a warp whose cells are all +0 keeps them (with finite velocities)
    const bool zero = !CONS && i >= 2 && zero_bits == 0 && finite_bits(v0) && finite_bits(w0) &&
                      finite_bits(a);
    if (!CONS && __all_sync(0xffffffffu, zero)) continue;
#pragma unroll
    for (int k = 0; k < NF; ++k) {
      T* __restrict__ dst = k == 0 ? dst0 : dst1;
      T out;
      if constexpr (CONS) {
        const T xf = face_cons(fm1[k], f0[k], f1[k], f2[k], vm1, v0, v1, v2);
        const T xb = __shfl_up_sync(0xffffffffu, xf, 1);
        const T yf = face_cons(gm1[k], f0[k], g1[k], g2[k], wm1, w0, w1, w2);
        T flux = T(0);
        flux = rn_add(flux, rn_mul(a, xf));
        flux = rn_sub(flux, rn_mul(a, xb));
        flux = rn_add(flux, rn_mul(a, yf));
        flux = rn_sub(flux, rn_mul(a, yb));
        yb = yf;
        out = rn_add(f0[k], inner ? flux : T(0));
      } else {
        out = noncons_cell(fm1[k], f0[k], f1[k], f2[k], gm2[k], gm1[k], g1[k], g2[k], v0, v1, wm1,
                           w0, w1, a, inner);
      }
      // ghost cells take a zero flux (which turns -0 into +0)
      if (cell) dst[row + j] = out;
    }
  }
}

template <typename T, int NF, bool CONS>
int eno3_launch(T* f0, T* f1, T par0, T par1, const T* uz, const T* ur, T* scratch, int nr,
                int nz, T dt_by_dx, cudaStream_t s, const char* what,
                const double* dt_dev = nullptr, T dx = T(0)) {
  if (nr < 3 || nz < 5) {
    axi::set_error("%s: grid %d x %d too small for ENO3 (needs nr >= 3, nz >= 5)", what, nr, nz);
    return AXI_ERR_INVALID;
  }
  AXI_TRY(axi::check_ptrs(what, {f0, uz, ur, scratch},
                          {NF == 2 ? "eta1" : "vorticity", "u_z", "u_r", "scratch"}));
  if (NF == 2) AXI_TRY(axi::check_ptr(what, f1, "eta2"));
  const size_t bytes = (size_t)nr * nz * sizeof(T);
  if (cudaMemcpyAsync(scratch, f0, bytes, cudaMemcpyDeviceToDevice, s) != cudaSuccess)
    return axi::launch_status(what);
  T* s1 = nullptr;
  if (NF == 2) {
    s1 = scratch + (size_t)nr * nz;
    if (cudaMemcpyAsync(s1, f1, bytes, cudaMemcpyDeviceToDevice, s) != cudaSuccess)
      return axi::launch_status(what);
  }
  // Strips as long as the GPU stays filled (24 warps per SM): a longer strip
  // spares FP64 instructions but walks its rows one load latency after the
  // other (strips of 8, filling it less: 41 us for omega, but 42 instead of 26
  // for eta, most of which is zeros).
  const int cols = axi::ceil_div(nz, ENO_COLS);
  const long long per = (long long)nr * cols / (24LL * axi::sm_count());
  const int most = CONS ? 4 : 1;
  const int strip = per < 1 ? 1 : per > most ? most : (int)per;
  dim3 grid(cols, axi::ceil_div(nr, ENO_WARPS * strip));
  eno3_step_kernel<T, NF, CONS><<<grid, dim3(32, ENO_WARPS), 0, s>>>(
      f0, f1, scratch, s1, par0 < T(0), par1 < T(0), uz, ur, nr, nz, -dt_by_dx, dt_dev, dx, strip);
  return axi::launch_status(what);
}

}  // namespace

#define AXI_DEFINE_ENO3(SUF, T)                                                                \
  extern "C" int axi_advect_vorticity_eno3_##SUF(T* vort, const T* u_z, const T* u_r,          \
                                                 T* scratch, int nr, int nz, T dt_by_dx,       \
                                                 void* stream) {                               \
    axi::clear_error();                                                                        \
    return eno3_launch<T, 1, true>(vort, nullptr, T(-1), T(0), u_z, u_r, scratch, nr, nz,      \
                                   dt_by_dx, axi::as_stream(stream), "advect_vorticity_eno3"); \
  }                                                                                            \
  extern "C" int axi_advect_vorticity_eno3_periodic_##SUF(T* vort, T* u_z, T* u_r, T* scratch, \
                                                          int nr, int nz, T dt_by_dx,          \
                                                          int ghost, void* stream) {           \
    axi::clear_error();                                                                        \
    AXI_TRY(axi_periodic_ghost_comm_##SUF(u_z, nr, nz, ghost, stream));                        \
    AXI_TRY(axi_periodic_ghost_comm_##SUF(u_r, nr, nz, ghost, stream));                        \
    AXI_TRY(axi_periodic_ghost_comm_##SUF(vort, nr, nz, ghost, stream));                       \
    return eno3_launch<T, 1, true>(vort, nullptr, T(-1), T(0), u_z, u_r, scratch, nr, nz,      \
                                   dt_by_dx, axi::as_stream(stream),                           \
                                   "advect_vorticity_eno3_periodic");                          \
  }                                                                                            \
  extern "C" int axi_advect_refmap_eno3_##SUF(T* eta1, T* eta2, const T* u_z, const T* u_r,    \
                                              T* scratch2, int nr, int nz, T dt_by_dx,         \
                                              void* stream) {                                  \
    axi::clear_error();                                                                        \
    return eno3_launch<T, 2, false>(eta1, eta2, T(1), T(-1), u_z, u_r, scratch2, nr, nz,       \
                                    dt_by_dx, axi::as_stream(stream), "advect_refmap_eno3");   \
  }                                                                                            \
  extern "C" int axi_advect_refmap_eno3_periodic_##SUF(T* eta1, T* eta2, T* u_z, T* u_r,       \
                                                       T* scratch2, int nr, int nz,            \
                                                       T dt_by_dx, int ghost, T z_max, T dx,   \
                                                       void* stream) {                         \
    axi::clear_error();                                                                        \
    AXI_TRY(axi_periodic_ghost_comm_##SUF(u_z, nr, nz, ghost, stream));                        \
    AXI_TRY(axi_periodic_ghost_comm_##SUF(u_r, nr, nz, ghost, stream));                        \
    AXI_TRY(axi_periodic_ghost_comm_eta_##SUF(eta1, nr, nz, ghost, z_max, dx, stream));        \
    AXI_TRY(axi_periodic_ghost_comm_##SUF(eta2, nr, nz, ghost, stream));                       \
    return eno3_launch<T, 2, false>(eta1, eta2, T(1), T(-1), u_z, u_r, scratch2, nr, nz,       \
                                    dt_by_dx, axi::as_stream(stream),                          \
                                    "advect_refmap_eno3_periodic");                            \
  }

AXI_DEFINE_ENO3(f64, double)
AXI_DEFINE_ENO3(f32, float)

// The soft-sphere loop's two advections with the time step read on the device
// (state[AXI_SOFT_DT]): eta (non-conservative, eta1 even and eta2 odd about the
// axis, elasto_kernels/advect_refmap_via_eno3.py:8-44) or omega (conservative,
// odd), the arithmetic of the host-dt entries above.
extern "C" int axi_soft_advect_eno3_f64(double* f0, double* f1, int refmap, const double* u_z,
                                        const double* u_r, double* scratch, int nr, int nz,
                                        double dx, const double* state, void* stream) {
  axi::clear_error();
  AXI_TRY(axi::check_ptrs("soft_advect_eno3", {f0, u_z, u_r, scratch, state},
                          {refmap ? "eta1" : "omega", "u_z", "u_r", "scratch", "state"}));
  if (refmap) {
    AXI_TRY(axi::check_ptr("soft_advect_eno3", f1, "eta2"));
    return eno3_launch<double, 2, false>(f0, f1, 1.0, -1.0, u_z, u_r, scratch, nr, nz, 0.0,
                                         axi::as_stream(stream), "soft_advect_eno3",
                                         state + AXI_SOFT_DT, dx);
  }
  return eno3_launch<double, 1, true>(f0, nullptr, -1.0, 0.0, u_z, u_r, scratch, nr, nz, 0.0,
                                      axi::as_stream(stream), "soft_advect_eno3",
                                      state + AXI_SOFT_DT, dx);
}
