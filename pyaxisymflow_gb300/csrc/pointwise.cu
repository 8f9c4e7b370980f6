// Pointwise and nearest-neighbour grid kernels of the per-timestep hot path.
//
// z (the contiguous axis) on threadIdx.x so every warp reads and writes 32
// consecutive doubles. The double kernels are bound by FP64 issue (one warp
// instruction per scheduler and 64 cycles), so divisions by the grid constants
// and by the row's radius go through KnownDivisor, and cells whose operands
// are all zero (most of the elastic stress field) take no FP64 instruction. Where the reference kernel has no
// transcendental function the arithmetic is issued with the *_rn intrinsics
// in the reference's own evaluation order, so results are bit-identical to the
// numpy evaluation of the reference (no FMA contraction).
#include "axi_common.cuh"

namespace {

constexpr int BX = 32;
constexpr int BY = 8;

inline dim3 grid2d(int nr, int nz) { return dim3(axi::ceil_div(nz, BX), axi::ceil_div(nr, BY)); }

// Blocks of 8 rows whose threads walk along z in steps of gridDim.x * 32, so
// that what depends on the row alone is formed once per block. Enough blocks
// for eight warps per scheduler (4 blocks per SM) and an equal number of steps
// per block.
inline dim3 grid_rows(int nr, int nz) {
  const int gy = axi::ceil_div(nr, BY), steps = axi::ceil_div(nz, BX);
  const int want = axi::ceil_div(4LL * axi::sm_count(), gy);
  const int per = want >= steps ? 1 : steps / want;
  return dim3(axi::ceil_div(steps, per), gy);
}

template <typename T>
__device__ __forceinline__ bool same_bits(T a, T b);
template <>
__device__ __forceinline__ bool same_bits(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}
template <>
__device__ __forceinline__ bool same_bits(float a, float b) {
  return __float_as_int(a) == __float_as_int(b);
}

// Divisors of the block's rows, taken at column 0; a cell whose R differs
// (R is an array of the caller's) uses its own.
template <typename T>
struct RowDivisors {
  KnownDivisor<T>* d;
  __device__ __forceinline__ void fill(const T* __restrict__ R, int nr, int nz) const {
    if (threadIdx.y == 0 && threadIdx.x < BY) {
      const int i = min((int)(blockIdx.y * BY + threadIdx.x), nr - 1);
      d[threadIdx.x] = KnownDivisor<T>(R[(long long)i * nz]);
    }
    __syncthreads();
  }
  __device__ __forceinline__ KnownDivisor<T> get(T r) const {
    const KnownDivisor<T> k = d[threadIdx.y];
    return same_bits(k.b, r) ? k : KnownDivisor<T>(r);
  }
};
// kernels/compute_velocity_from_psi.py:9-17
// One-sided differences at the grid's edges, out of line: inlined, the
// compiler evaluated them for every cell and selected (9 more FP64
// instructions on 18).
template <typename T>
__device__ __noinline__ T edge_difference(const T* __restrict__ p, long long step, bool start) {
  if (start) {
    // -p[2] + 4 p[1] - 3 p[0]
    return rn_sub(rn_add(-p[2 * step], rn_mul(T(4), p[step])), rn_mul(T(3), p[0]));
  }
  // p[-3] - 4 p[-2] + 3 p[-1], p at the last point
  return rn_add(rn_sub(p[-2 * step], rn_mul(T(4), p[-step])), rn_mul(T(3), p[0]));
}

template <typename T>
__global__ void __launch_bounds__(BX * BY)
    velocity_from_psi_kernel(T* __restrict__ u_z, T* __restrict__ u_r, const T* __restrict__ psi,
                             const T* __restrict__ R, int nr, int nz, KnownDivisor<T> two_dx) {
  __shared__ KnownDivisor<T> s_div[BY];
  const RowDivisors<T> rows{s_div};
  rows.fill(R, nr, nz);
  const int i = blockIdx.y * BY + threadIdx.y;
  if (i >= nr) return;
  for (int j = blockIdx.x * BX + threadIdx.x; j < nz; j += gridDim.x * BX) {
    const long long c = (long long)i * nz + j;
    const KnownDivisor<T> r = rows.get(R[c]);
    T dz;
    if (i == 0 || i == nr - 1)
      dz = edge_difference(psi + c, nz, i == 0);
    else
      dz = rn_sub(psi[c + nz], psi[c - nz]);
    u_z[c] = r.quotient(two_dx.quotient(dz));
    T dr;
    if (j == 0 || j == nz - 1)
      dr = edge_difference(psi + c, 1, j == 0);
    else
      dr = rn_sub(psi[c + 1], psi[c - 1]);
    u_r[c] = r.quotient(two_dx.quotient(-dr));
  }
}

// kernels/periodic_boundary_ghost_comm.py:9-13 (shift == 0) and :23-31 (eta):
// field[:, :g] = field[:, -2g:-g] - shift; field[:, -g:] = field[:, g:2g] + shift,
// shift = z_max - 2 g dx (applied in the reference's order: a - z_max + 2 g dx).
template <typename T>
__global__ void ghost_comm_kernel(T* __restrict__ f, int nr, int nz, int g, bool eta, T z_max,
                                  T two_g_dx) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;  // 0 .. 2g-1
  const int i = blockIdx.y;
  if (k >= 2 * g || i >= nr) return;
  T* row = f + (long long)i * nz;
  if (k < g) {
    T v = row[nz - 2 * g + k];
    row[k] = eta ? rn_add(rn_sub(v, z_max), two_g_dx) : v;
  } else {
    const int kk = k - g;
    T v = row[g + kk];
    row[nz - g + kk] = eta ? rn_sub(rn_add(v, z_max), two_g_dx) : v;
  }
}

// kernels/compute_vorticity_from_velocity.py:11-13 on [1:-1, 1:-1]
template <typename T>
__global__ void vorticity_from_velocity_kernel(T* __restrict__ vort, const T* __restrict__ u_z,
                                               const T* __restrict__ u_r, int nr, int nz,
                                               KnownDivisor<T> two_dx) {
  const int j = blockIdx.x * BX + threadIdx.x;
  const int i = blockIdx.y * BY + threadIdx.y;
  if (i < 1 || j < 1 || i >= nr - 1 || j >= nz - 1) return;
  const long long c = (long long)i * nz + j;
  T a = two_dx.quotient(rn_sub(u_r[c + 1], u_r[c - 1]));
  T b = two_dx.quotient(rn_sub(u_z[c + nz], u_z[c - nz]));
  vort[c] = rn_sub(a, b);
}

// kernels/brinkmann_penalize.py:11-16 at one point
template <typename T>
__device__ __forceinline__ void penalise_point(T ldt, T chi, T U_z, T U_r, T vz, T vr, T& pz,
                                               T& pr) {
  const T lc = rn_mul(ldt, chi);
  if constexpr (sizeof(T) == 8) {
    // outside the body lc is +0 and the penalised velocity is the velocity
    // itself ((v + 0 U) / 1; a zero velocity may change its sign)
    if (is_pos_zero(lc) && exponent_bits(U_z) != 0x7ff && exponent_bits(U_r) != 0x7ff &&
        !is_zero_bits(vz) && !is_zero_bits(vr)) {
      pz = vz;
      pr = vr;
      return;
    }
  }
  const KnownDivisor<T> denom(rn_add(T(1), lc));
  pz = denom.quotient(rn_add(vz, rn_mul(lc, U_z)));
  pr = denom.quotient(rn_add(vr, rn_mul(lc, U_r)));
}

template <typename T>
__global__ void brinkman_kernel(T lam, T dt, const T* __restrict__ chi, T U_z, T U_r,
                                const T* __restrict__ gz, const T* __restrict__ gr,
                                T* __restrict__ pz, T* __restrict__ pr, long long n) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  T z, r;
  penalise_point(rn_mul(lam, dt), chi[k], U_z, U_r, gz[k], gr[k], z, r);
  pz[k] = z;
  pr[k] = r;
}

// ---------------------------------------------------------------------------
// The loop body of a rigid sphere between the solve and the advection
// (examples/FlowPastSphere/flow_past_sphere.py:143-175) as three passes. As
// array operations it is 17 launches, two of them reductions by a single block
// (51 and 30 us on 384 x 201 cells), against 10 us for the three.
// ---------------------------------------------------------------------------
// u_z += add; *umax = max(|u_z| + |u_r|), by the order of the bits (the sums are
// not negative, and a NaN sorts last). *umax starts at +0.
__global__ void __launch_bounds__(256) sphere_speed_kernel(double* __restrict__ uz,
                                                           const double* __restrict__ ur,
                                                           double add, long long n,
                                                           unsigned long long* umax) {
  unsigned long long m = 0;
  for (long long k = (long long)blockIdx.x * 256 + threadIdx.x; k < n;
       k += (long long)gridDim.x * 256) {
    const double z = rn_add(uz[k], add);
    uz[k] = z;
    const unsigned long long b =
        (unsigned long long)__double_as_longlong(rn_add(fabs(z), fabs(ur[k])));
    m = (b & 0x7fffffffffffffffull) > m ? (b & 0x7fffffffffffffffull) : m;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_xor_sync(0xffffffffu, m, o);
    m = v > m ? v : m;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(umax, m);
}

// The velocity kept in old_z, old_r and penalised in place for a body at rest;
// partials[block] = the block's sum of r chi u_z (fixed order).
constexpr int SPHERE_CELLS = 1024;  // cells per block
__global__ void __launch_bounds__(256) sphere_penalise_kernel(
    double* __restrict__ uz, double* __restrict__ ur, double* __restrict__ old_z,
    double* __restrict__ old_r, const double* __restrict__ chi, const double* __restrict__ R,
    double lam, double dt, long long n, double* __restrict__ partials) {
  __shared__ double warps[8];
  const double ldt = rn_mul(lam, dt);
  double sum = 0.0;
  bool any = false;
#pragma unroll
  for (int q = 0; q < SPHERE_CELLS / 256; ++q) {
    const long long k = (long long)blockIdx.x * SPHERE_CELLS + q * 256 + threadIdx.x;
    if (k >= n) break;
    const double vz = uz[k], vr = ur[k], c = chi[k];
    double pz, pr;
    penalise_point(ldt, c, 0.0, 0.0, vz, vr, pz, pr);
    old_z[k] = vz;
    old_r[k] = vr;
    uz[k] = pz;
    ur[k] = pr;
    if (!is_zero_bits(c) || exponent_bits(pz) == 0x7ff) {
      sum += rn_mul(rn_mul(R[k], c), pz);
      any = true;
    }
  }
  // most blocks lie outside the body and spend no FP64 instruction here
  if (!__syncthreads_or(any)) {
    if (threadIdx.x == 0) partials[blockIdx.x] = 0.0;
    return;
  }
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x < 32) {
    double x = threadIdx.x < 8 ? warps[threadIdx.x] : 0.0;
    for (int o = 4; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (threadIdx.x == 0) partials[blockIdx.x] = x;
  }
}

// vort = curl(u - old) on the inner cells (kernels/compute_vorticity_from_velocity.py:11-13),
// w += vort everywhere; the first block also adds up the partial sums.
__device__ __forceinline__ bool same_finite(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b) && exponent_bits(a) != 0x7ff;
}
__global__ void sphere_curl_kernel(double* __restrict__ w, double* __restrict__ vort,
                                   const double* __restrict__ uz, const double* __restrict__ ur,
                                   const double* __restrict__ old_z,
                                   const double* __restrict__ old_r, int nr, int nz,
                                   KnownDivisor<double> two_dx,
                                   const double* __restrict__ partials, int n_partials,
                                   double* __restrict__ sum) {
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.y == 0 && threadIdx.x < 32) {
    double x = 0.0;
    for (int q = threadIdx.x; q < n_partials; q += 32)
      if (!is_zero_bits(partials[q])) x += partials[q];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (threadIdx.x == 0) *sum = x;
  }
  const int j = blockIdx.x * BX + threadIdx.x;
  const int i = blockIdx.y * BY + threadIdx.y;
  if (i >= nr || j >= nz) return;
  const long long c = (long long)i * nz + j;
  double v;
  if (i < 1 || j < 1 || i >= nr - 1 || j >= nz - 1) {
    v = vort[c];
  } else {
    const double re = ur[c + 1], rw = ur[c - 1], zn = uz[c + nz], zs = uz[c - nz];
    const double ore = old_r[c + 1], orw = old_r[c - 1], ozn = old_z[c + nz], ozs = old_z[c - nz];
    if (same_finite(re, ore) && same_finite(rw, orw) && same_finite(zn, ozn) &&
        same_finite(zs, ozs)) {
      v = 0.0;  // outside the body: differences of equal values
    } else {
      const double a = two_dx.quotient(rn_sub(rn_sub(re, ore), rn_sub(rw, orw)));
      const double b = two_dx.quotient(rn_sub(rn_sub(zn, ozn), rn_sub(zs, ozs)));
      v = rn_sub(a, b);
    }
    vort[c] = v;
  }
  const double w0 = w[c];
  if (is_pos_zero(v) && !is_zero_bits(w0)) return;  // w + 0
  w[c] = rn_add(w0, v);
}

// kernels/smooth_Heaviside.py:10-14
template <typename T>
__global__ void heaviside_kernel(T* __restrict__ H, const T* __restrict__ phi, T w, long long n) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const T p = phi[k];
  if constexpr (sizeof(T) == 8) {
    double v;
    if (heaviside_outside(H[k], p, w, v)) {
      H[k] = v;
      return;
    }
  }
  T h = rn_mul(T(0), H[k]);
  h = rn_add(h, (p >= w) ? T(1) : T(0));
  // (|phi| < w) * 0.5 * (1 + phi / w + sin(pi * phi / w) / pi), left to right
  const T a = rn_add(T(1), rn_div(p, w));
  const T s = rn_div(dev_sin(rn_div(rn_mul(Pi<T>::v, p), w)), Pi<T>::v);
  const T m05 = (fabs(p) < w) ? T(0.5) : T(0);
  h = rn_add(h, rn_mul(m05, rn_add(a, s)));
  H[k] = h;
}

// kernels/kill_boundary_vorticity_sine.py:9-14: both z strips of width w <= 8
// (2 w <= nz, so they do not overlap). 16 lanes own one row: lanes 0 .. w - 1
// the left strip, 8 .. 8 + w - 1 the right one; the source columns are read
// before any write. One sine per lane: with a thread per row their chain of up
// to 16 took 16 us on any grid.
template <typename T>
__global__ void __launch_bounds__(128)
    kill_z_kernel(T* __restrict__ vort, const T* __restrict__ Z, int nr, int nz, int w,
                  T half_dx, KnownDivisor<T> w1, KnownDivisor<T> dx) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 4;
  const int k = threadIdx.x & 7;
  const bool right = threadIdx.x & 8;
  const bool live = i < nr && k < w;
  T* row = vort + (long long)i * nz;
  const int j = right ? nz - w + k : k;
  T v = T(0);
  if (live) {
    const T z = Z[(long long)i * nz + j];
    const T src = row[right ? nz - w : w - 1];
    const T x = rn_sub(right ? rn_sub(T(1), z) : z, half_dx);
    const T arg = dx.quotient(w1.quotient(rn_mul(rn_mul(Pi<T>::v, x), T(0.5))));
    v = rn_mul(dev_sin(arg), src);
  }
  __syncwarp();
  if (live) row[j] = v;
}

// kernels/kill_boundary_vorticity_sine.py:23-27: outer-r strip, then row 0 = 0.
// Threads (j, k) own row nr - w + k of column j; the source row is read before
// any write.
template <typename T>
__global__ void __launch_bounds__(1024)
    kill_r_kernel(T* __restrict__ vort, const T* __restrict__ R, int nr, int nz, int w,
                  T half_dx, KnownDivisor<T> w1, KnownDivisor<T> dx) {
  const int j = blockIdx.x * 32 + threadIdx.x;
  const T src = j < nz ? vort[(long long)(nr - w) * nz + j] : T(0);
  __syncthreads();
  if (j >= nz) return;
  for (int k = threadIdx.y; k < w; k += blockDim.y) {
    const long long c = (long long)(nr - w + k) * nz + j;
    const T x = rn_sub(rn_sub(T(1), R[c]), half_dx);
    const T arg = dx.quotient(w1.quotient(rn_mul(rn_mul(Pi<T>::v, x), T(0.5))));
    vort[c] = rn_mul(dev_sin(arg), src);
  }
  if (threadIdx.y == 0) vort[j] = T(0);
}

// kernels/diffusion_RK2.py:15-25: the bracketed operator at interior cell c.
// r and inv_r2 = 1 / r^2 depend on the row alone.
template <typename T>
struct DiffusionRow {
  KnownDivisor<T> r;
  T inv_r2;
  DiffusionRow() = default;
  __device__ __forceinline__ explicit DiffusionRow(T x) : r(x), inv_r2(rn_div(T(1), rn_mul(x, x))) {}
};

template <typename T>
__device__ __forceinline__ T rk2_operator(const T* __restrict__ w, const DiffusionRow<T>& row,
                                          long long c, int nz, const KnownDivisor<T>& dx2,
                                          const KnownDivisor<T>& two_dx) {
  const T n = w[c + nz], s = w[c - nz], e = w[c + 1], wst = w[c - 1], ctr = w[c];
  T lap = rn_add(rn_add(rn_add(n, s), e), wst);
  lap = dx2.quotient(rn_sub(lap, rn_mul(T(4), ctr)));
  const T adv = row.r.quotient(two_dx.quotient(rn_sub(n, s)));
  return rn_sub(rn_add(lap, adv), rn_mul(ctr, row.inv_r2));
}

// Stage 1 (diffusion_RK2.py:9-26): out = tmp: tmp = w; tmp[1:-1,1:-1] += 0.5 nu dt L(w)
// Stage 2 (:27-44): out = vort: vort[1:-1,1:-1] += nu dt L(tmp)
// coef: 0.5 nu dt or nu dt; with dt_dev its factor of the device-resident dt.
template <typename T, int STAGE>
__global__ void __launch_bounds__(BX * BY)
    rk2_kernel(T* __restrict__ out, const T* __restrict__ f, const T* __restrict__ R, int nr,
               int nz, T coef, KnownDivisor<T> dx2, KnownDivisor<T> two_dx,
               const double* __restrict__ dt_dev = nullptr) {
  __shared__ DiffusionRow<T> s_row[BY];
  __shared__ T s_coef;
  if (threadIdx.y == 0 && threadIdx.x < BY) {
    const int i = min((int)(blockIdx.y * BY + threadIdx.x), nr - 1);
    s_row[threadIdx.x] = DiffusionRow<T>(R[(long long)i * nz]);
  }
  if (threadIdx.y == 1 && threadIdx.x == 0)
    s_coef = dt_dev ? rn_mul(coef, static_cast<T>(dt_dev[0])) : coef;
  __syncthreads();
  const int i = blockIdx.y * BY + threadIdx.y;
  if (i >= nr) return;
  const T cf = s_coef;
  for (int j = blockIdx.x * BX + threadIdx.x; j < nz; j += gridDim.x * BX) {
    const long long c = (long long)i * nz + j;
    const bool inner = i > 0 && j > 0 && i < nr - 1 && j < nz - 1;
    if (STAGE == 2 && !inner) continue;
    T v = STAGE == 1 ? f[c] : out[c];
    if (inner) {
      const T r = R[c];
      const T op = same_bits(s_row[threadIdx.y].r.b, r)
                       ? rk2_operator(f, s_row[threadIdx.y], c, nz, dx2, two_dx)
                       : rk2_operator(f, DiffusionRow<T>(r), c, nz, dx2, two_dx);
      v = rn_add(v, rn_mul(cf, op));
    }
    out[c] = v;
  }
}

template <typename T>
void launch_rk2_stage1(T* tmp, const T* vort, const T* R, int nr, int nz, T coef, T dx,
                       cudaStream_t s, const double* dt_dev = nullptr) {
  rk2_kernel<T, 1><<<grid_rows(nr, nz), dim3(BX, BY), 0, s>>>(
      tmp, vort, R, nr, nz, coef, KnownDivisor<T>(rn_host_mul(dx, dx)),
      KnownDivisor<T>(rn_host_mul(T(2), dx)), dt_dev);
}
template <typename T>
void launch_rk2_stage2(T* vort, const T* tmp, const T* R, int nr, int nz, T coef, T dx,
                       cudaStream_t s, const double* dt_dev = nullptr) {
  rk2_kernel<T, 2><<<grid_rows(nr, nz), dim3(BX, BY), 0, s>>>(
      vort, tmp, R, nr, nz, coef, KnownDivisor<T>(rn_host_mul(dx, dx)),
      KnownDivisor<T>(rn_host_mul(T(2), dx)), dt_dev);
}

// elasto_kernels/solid_sigma.py:18-29: gradients where the reference writes
// them, then the stress from whatever the gradient arrays hold, times chi where
// it is given (soft_sphere_streaming.py:236-238). Where the eight neighbours
// are +0 (eta outside the solid and its extrapolation band) the gradients are
// +0 and the stress is a zero of known sign.
template <typename T>
__global__ void __launch_bounds__(BX * BY)
    solid_sigma_kernel(T* __restrict__ s11, T* __restrict__ s12, T* __restrict__ s22, T G,
                       KnownDivisor<T> two_dx, const T* __restrict__ e1,
                       const T* __restrict__ e2, T* __restrict__ e1z, T* __restrict__ e1r,
                       T* __restrict__ e2z, T* __restrict__ e2r, int nr, int nz,
                       const T* __restrict__ chi) {
  const int j = blockIdx.x * BX + threadIdx.x;
  const int i = blockIdx.y * BY + threadIdx.y;
  if (i >= nr || j >= nz) return;
  const long long c = (long long)i * nz + j;
  const bool inner = i > 0 && i < nr - 1 && j > 0 && j < nz - 1;
  if constexpr (sizeof(T) == 8) {
    if (inner) {
      const T x = chi ? chi[c] : T(1);
      const bool zero =
          is_pos_zero(e1[c + 1]) && is_pos_zero(e1[c - 1]) && is_pos_zero(e1[c + nz]) &&
          is_pos_zero(e1[c - nz]) && is_pos_zero(e2[c + 1]) && is_pos_zero(e2[c - 1]) &&
          is_pos_zero(e2[c + nz]) && is_pos_zero(e2[c - nz]);
      // positive finite G, dx and non-negative finite chi: only then the signs are known
      if (zero && (unsigned int)(exponent_bits(G) - 1) < 0x7feu && __double2hiint(G) > 0 &&
          two_dx.ok && __double2hiint(two_dx.b) > 0 && __double2hiint(x) >= 0 &&
          exponent_bits(x) != 0x7ff) {
        e1z[c] = e2z[c] = e1r[c] = e2r[c] = T(0);
        s12[c] = -T(0);
        s11[c] = T(0);
        s22[c] = -T(0);
        return;
      }
    }
  }
  T g1z = e1z[c], g2z = e2z[c], g1r = e1r[c], g2r = e2r[c];
  if (j > 0 && j < nz - 1) {
    g1z = two_dx.quotient(rn_sub(e1[c + 1], e1[c - 1]));
    g2z = two_dx.quotient(rn_sub(e2[c + 1], e2[c - 1]));
    e1z[c] = g1z;
    e2z[c] = g2z;
  }
  if (i == 0) {
    g1r = two_dx.quotient(rn_sub(rn_add(-e1[2LL * nz + j], rn_mul(T(4), e1[(long long)nz + j])),
                                 rn_mul(T(3), e1[j])));
    g2r = two_dx.quotient(rn_sub(rn_add(-e2[2LL * nz + j], rn_mul(T(4), e2[(long long)nz + j])),
                                 rn_mul(T(3), e2[j])));
    e1r[c] = g1r;
    e2r[c] = g2r;
  } else if (inner) {
    g1r = two_dx.quotient(rn_sub(e1[c + nz], e1[c - nz]));
    g2r = two_dx.quotient(rn_sub(e2[c + nz], e2[c - nz]));
    e1r[c] = g1r;
    e2r[c] = g2r;
  }
  const T v12 = rn_mul(-G, rn_add(rn_mul(g1z, g1r), rn_mul(g2z, g2r)));
  T t = rn_add(rn_mul(g1r, g1r), rn_mul(g2r, g2r));
  t = rn_sub(rn_sub(t, rn_mul(g1z, g1z)), rn_mul(g2z, g2z));
  const T v11 = rn_mul(rn_mul(T(0.5), G), t);
  if (chi) {
    const T x = chi[c];
    s12[c] = rn_mul(v12, x);
    s11[c] = rn_mul(v11, x);
    s22[c] = rn_mul(-v11, x);
  } else {
    s12[c] = v12;
    s11[c] = v11;
    s22[c] = -v11;
  }
}

// elasto_kernels/div_tau.py:8-28: tau on [1:-1, 1:-1] and row 0 [0, 1:-1].
// Where the stencil holds the zeros that solid_sigma_kernel leaves outside the
// solid (t11 +0, t12 and t22 -0) tau is +0.
template <typename T>
__global__ void __launch_bounds__(BX * BY)
    div_tau_kernel(T* __restrict__ tz, T* __restrict__ tr, const T* __restrict__ t11,
                   const T* __restrict__ t12, const T* __restrict__ t22, const T* __restrict__ R,
                   int nr, int nz, KnownDivisor<T> two_dx) {
  const int j = blockIdx.x * BX + threadIdx.x;
  const int i = blockIdx.y * BY + threadIdx.y;
  if (i >= nr - 1 || j < 1 || j >= nz - 1) return;
  const long long c = (long long)i * nz + j;
  const T r = R[c];
  if constexpr (sizeof(T) == 8) {
    if (i > 0) {
      const long long nzero = 1ll << 63;
      auto neg = [nzero](double x) { return __double_as_longlong(x) == nzero; };
      if (is_pos_zero(t11[c + 1]) && is_pos_zero(t11[c - 1]) && neg(t12[c + nz]) &&
          neg(t12[c - nz]) && neg(t12[c]) && neg(t12[c + 1]) && neg(t12[c - 1]) &&
          neg(t22[c + nz]) && neg(t22[c - nz]) && neg(t22[c]) &&
          (unsigned int)(exponent_bits(r) - 1) < 0x7feu && __double2hiint(r) > 0 && two_dx.ok &&
          __double2hiint(two_dx.b) > 0) {
        tz[c] = T(0);
        tr[c] = T(0);
        return;
      }
    }
  }
  if (i == 0) {
    T a = rn_sub(rn_sub(t11[c + 1], t11[c - 1]), t12[c + 2LL * nz]);
    a = rn_sub(rn_add(a, rn_mul(T(4), t12[c + nz])), rn_mul(T(3), t12[c]));
    const KnownDivisor<T> rd(r);
    tz[c] = rn_add(two_dx.quotient(a), rd.quotient(t12[c]));
    T b = rn_sub(rn_sub(t12[c + 1], t12[c - 1]), t22[c + 2LL * nz]);
    b = rn_sub(rn_add(b, rn_mul(T(4), t22[c + nz])), rn_mul(T(3), t22[c]));
    tr[c] = rn_add(two_dx.quotient(b), rd.quotient(t22[c]));
  } else {
    const KnownDivisor<T> rd(r);
    T a = rn_add(rn_sub(t11[c + 1], t11[c - 1]), t12[c + nz]);
    a = rn_sub(a, t12[c - nz]);
    tz[c] = rn_add(two_dx.quotient(a), rd.quotient(t12[c]));
    T b = rn_add(rn_sub(t12[c + 1], t12[c - 1]), t22[c + nz]);
    b = rn_sub(b, t22[c - nz]);
    tr[c] = rn_add(two_dx.quotient(b), rd.quotient(t22[c]));
  }
}

// elasto_kernels/div_tau.py:30-34: vort[1:-1,1:-1] += dt (dtau_r/dz - dtau_z/dr) / (2 dx)
// (nothing to add where tau is +0 around and vort is not zero).
template <typename T>
__global__ void __launch_bounds__(BX * BY)
    curl_tau_kernel(T* __restrict__ w, const T* __restrict__ tz, const T* __restrict__ tr, int nr,
                    int nz, T dt, KnownDivisor<T> two_dx,
                    const double* __restrict__ dt_dev = nullptr) {
  const int j = blockIdx.x * BX + threadIdx.x;
  const int i = blockIdx.y * BY + threadIdx.y;
  if (i < 1 || j < 1 || i >= nr - 1 || j >= nz - 1) return;
  if (dt_dev) dt = static_cast<T>(dt_dev[0]);
  const long long c = (long long)i * nz + j;
  if constexpr (sizeof(T) == 8) {
    if (is_pos_zero(tr[c + 1]) && is_pos_zero(tr[c - 1]) && is_pos_zero(tz[c + nz]) &&
        is_pos_zero(tz[c - nz]) && exponent_bits(dt) != 0x7ff && two_dx.ok &&
        !is_zero_bits(w[c]))
      return;
  }
  T a = rn_sub(rn_sub(tr[c + 1], tr[c - 1]), tz[c + nz]);
  a = rn_add(a, tz[c - nz]);
  w[c] = rn_add(w[c], two_dx.quotient(rn_mul(dt, a)));
}

template <typename T>
int ghost_comm(T* f, int nr, int nz, int g, bool eta, T z_max, T dx, cudaStream_t s) {
  if (g <= 0 || nz < 4 * g || nr < 1 || nr > 65535) {
    axi::set_error("periodic_ghost_comm: invalid ghost size %d for nz = %d", g, nz);
    return AXI_ERR_INVALID;
  }
  AXI_TRY(axi::check_ptr("periodic_ghost_comm", f, "field"));
  const int threads = 2 * g <= 256 ? 2 * g : 256;
  dim3 grid(axi::ceil_div(2 * g, threads), nr);
  ghost_comm_kernel<T><<<grid, threads, 0, s>>>(f, nr, nz, g, eta, z_max,
                                                 rn_host_mul(T(2 * g), dx));
  return axi::launch_status("periodic_ghost_comm");
}

}  // namespace

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------

#define AXI_DEFINE_VELOCITY(SUF, T)                                                           \
  extern "C" int axi_velocity_from_psi_unb_##SUF(T* u_z, T* u_r, const T* psi, const T* R,    \
                                                 int nr, int nz, T dx, void* stream) {        \
    axi::clear_error();                                                                       \
    AXI_TRY(axi::check_grid("velocity_from_psi", nr, nz));                                    \
    AXI_TRY(axi::check_ptrs("velocity_from_psi", {u_z, u_r, psi, R},                           \
                            {"u_z", "u_r", "psi", "R"}));                                      \
    velocity_from_psi_kernel<T><<<grid_rows(nr, nz), dim3(BX, BY), 0,                         \
                                  axi::as_stream(stream)>>>(                                  \
        u_z, u_r, psi, R, nr, nz, KnownDivisor<T>(rn_host_mul(T(2), dx)));                                                        \
    return axi::launch_status("velocity_from_psi");                                           \
  }                                                                                           \
  extern "C" int axi_velocity_from_psi_periodic_##SUF(T* u_z, T* u_r, T* psi, const T* R,     \
                                                      int nr, int nz, T dx, int ghost,        \
                                                      void* stream) {                         \
    axi::clear_error();                                                                       \
    AXI_TRY(axi::check_grid("velocity_from_psi_periodic", nr, nz));                           \
    AXI_TRY(axi::check_ptrs("velocity_from_psi_periodic", {u_z, u_r, psi, R},                  \
                            {"u_z", "u_r", "psi", "R"}));                                      \
    AXI_TRY(ghost_comm<T>(psi, nr, nz, ghost, false, T(0), dx, axi::as_stream(stream)));      \
    velocity_from_psi_kernel<T><<<grid_rows(nr, nz), dim3(BX, BY), 0,                         \
                                  axi::as_stream(stream)>>>(                                  \
        u_z, u_r, psi, R, nr, nz, KnownDivisor<T>(rn_host_mul(T(2), dx)));                                                        \
    return axi::launch_status("velocity_from_psi_periodic");                                  \
  }

#define AXI_DEFINE_VORTICITY(SUF, T)                                                          \
  extern "C" int axi_vorticity_from_velocity_unb_##SUF(T* vort, const T* u_z, const T* u_r,   \
                                                       int nr, int nz, T dx, void* stream) {  \
    axi::clear_error();                                                                       \
    AXI_TRY(axi::check_grid("vorticity_from_velocity", nr, nz));                              \
    AXI_TRY(axi::check_ptrs("vorticity_from_velocity", {vort, u_z, u_r},                       \
                            {"vort", "u_z", "u_r"}));                                          \
    vorticity_from_velocity_kernel<T>                                                         \
        <<<grid2d(nr, nz), dim3(BX, BY), 0, axi::as_stream(stream)>>>(vort, u_z, u_r, nr, nz,  \
                                                                      KnownDivisor<T>(        \
                                                                          rn_host_mul(T(2), dx))); \
    return axi::launch_status("vorticity_from_velocity");                                     \
  }                                                                                           \
  extern "C" int axi_vorticity_from_velocity_periodic_##SUF(T* vort, T* u_z, T* u_r, int nr,  \
                                                            int nz, T dx, int ghost,          \
                                                            void* stream) {                   \
    axi::clear_error();                                                                       \
    AXI_TRY(axi::check_grid("vorticity_from_velocity_periodic", nr, nz));                     \
    AXI_TRY(axi::check_ptrs("vorticity_from_velocity_periodic", {vort, u_z, u_r},              \
                            {"vort", "u_z", "u_r"}));                                          \
    AXI_TRY(ghost_comm<T>(u_r, nr, nz, ghost, false, T(0), dx, axi::as_stream(stream)));      \
    AXI_TRY(ghost_comm<T>(u_z, nr, nz, ghost, false, T(0), dx, axi::as_stream(stream)));      \
    vorticity_from_velocity_kernel<T>                                                         \
        <<<grid2d(nr, nz), dim3(BX, BY), 0, axi::as_stream(stream)>>>(vort, u_z, u_r, nr, nz,  \
                                                                      KnownDivisor<T>(        \
                                                                          rn_host_mul(T(2), dx))); \
    return axi::launch_status("vorticity_from_velocity_periodic");                            \
  }

#define AXI_DEFINE_POINTWISE(SUF, T)                                                           \
  extern "C" int axi_brinkmann_penalize_##SUF(T lam, T dt, const T* chi, T U_z, T U_r,         \
                                              const T* gz, const T* gr, T* pz, T* pr,          \
                                              int64_t n, void* stream) {                       \
    axi::clear_error();                                                                        \
    if (n < 0) { axi::set_error("brinkmann_penalize: negative size"); return AXI_ERR_INVALID; } \
    if (n == 0) return AXI_OK;                                                                 \
    AXI_TRY(axi::check_ptrs("brinkmann_penalize", {chi, gz, gr, pz, pr},                       \
                            {"char_func", "grid_u_z", "grid_u_r", "penalized_u_z",             \
                             "penalized_u_r"}));                                               \
    brinkman_kernel<T><<<axi::ceil_div(n, 256), 256, 0, axi::as_stream(stream)>>>(            \
        lam, dt, chi, U_z, U_r, gz, gr, pz, pr, n);                                            \
    return axi::launch_status("brinkmann_penalize");                                          \
  }                                                                                            \
  extern "C" int axi_smooth_heaviside_##SUF(T* H, const T* phi, T w, int64_t n, void* stream) { \
    axi::clear_error();                                                                        \
    if (n < 0) { axi::set_error("smooth_heaviside: negative size"); return AXI_ERR_INVALID; }  \
    if (n == 0) return AXI_OK;                                                                 \
    AXI_TRY(axi::check_ptrs("smooth_heaviside", {H, phi}, {"H", "phi"}));                      \
    heaviside_kernel<T><<<axi::ceil_div(n, 256), 256, 0, axi::as_stream(stream)>>>(H, phi, w, n); \
    return axi::launch_status("smooth_heaviside");                                             \
  }                                                                                            \
  extern "C" int axi_kill_boundary_vorticity_sine_z_##SUF(T* vort, const T* Z, int nr, int nz, \
                                                          int width, T dx, void* stream) {     \
    axi::clear_error();                                                                        \
    if (width < 2 || width > 8 || 2 * width > nz || nr < 1) {                                  \
      axi::set_error("kill_boundary_vorticity_sine_z: width %d unsupported for nz = %d", width, nz); \
      return AXI_ERR_INVALID;                                                                  \
    }                                                                                          \
    AXI_TRY(axi::check_ptrs("kill_boundary_vorticity_sine_z", {vort, Z}, {"vorticity", "Z"})); \
    kill_z_kernel<T><<<axi::ceil_div(16LL * nr, 128), 128, 0, axi::as_stream(stream)>>>(        \
        vort, Z, nr, nz, width, rn_host_mul(T(0.5), dx), KnownDivisor<T>(T(width - 1)),        \
        KnownDivisor<T>(dx));                                                                  \
    return axi::launch_status("kill_boundary_vorticity_sine_z");                               \
  }                                                                                            \
  extern "C" int axi_kill_boundary_vorticity_sine_r_##SUF(T* vort, const T* R, int nr, int nz, \
                                                          int width, T dx, void* stream) {     \
    axi::clear_error();                                                                        \
    if (width < 2 || width > nr || nz < 1) {                                                   \
      axi::set_error("kill_boundary_vorticity_sine_r: width %d unsupported for nr = %d", width, nr); \
      return AXI_ERR_INVALID;                                                                  \
    }                                                                                          \
    AXI_TRY(axi::check_ptrs("kill_boundary_vorticity_sine_r", {vort, R}, {"vorticity", "R"})); \
    kill_r_kernel<T><<<axi::ceil_div(nz, 32), dim3(32, width < 32 ? width : 32), 0,            \
                       axi::as_stream(stream)>>>(vort, R, nr, nz, width,                       \
                                                 rn_host_mul(T(0.5), dx),                      \
                                                 KnownDivisor<T>(T(width - 1)),                \
                                                 KnownDivisor<T>(dx));                         \
    return axi::launch_status("kill_boundary_vorticity_sine_r");                               \
  }                                                                                            \
  extern "C" int axi_diffusion_rk2_unb_##SUF(T* vort, T* tmp, const T* R, int nr, int nz, T nu, \
                                             T dt, T dx, void* stream) {                       \
    axi::clear_error();                                                                        \
    AXI_TRY(axi::check_grid("diffusion_rk2", nr, nz));                                         \
    AXI_TRY(axi::check_ptrs("diffusion_rk2", {vort, tmp, R},                                   \
                            {"vorticity", "temp_vorticity", "R"}));                            \
    cudaStream_t s = axi::as_stream(stream);                                                   \
    const T c1 = rn_host_mul(rn_host_mul(T(0.5), nu), dt), c2 = rn_host_mul(nu, dt);           \
    launch_rk2_stage1<T>(tmp, vort, R, nr, nz, c1, dx, s);                                     \
    launch_rk2_stage2<T>(vort, tmp, R, nr, nz, c2, dx, s);                                     \
    return axi::launch_status("diffusion_rk2");                                                \
  }                                                                                            \
  extern "C" int axi_diffusion_rk2_periodic_##SUF(T* vort, T* tmp, const T* R, int nr, int nz, \
                                                  T nu, T dt, T dx, int ghost, void* stream) { \
    axi::clear_error();                                                                        \
    AXI_TRY(axi::check_grid("diffusion_rk2_periodic", nr, nz));                                \
    AXI_TRY(axi::check_ptrs("diffusion_rk2_periodic", {vort, tmp, R},                          \
                            {"vorticity", "temp_vorticity", "R"}));                            \
    cudaStream_t s = axi::as_stream(stream);                                                   \
    const T c1 = rn_host_mul(rn_host_mul(T(0.5), nu), dt), c2 = rn_host_mul(nu, dt);           \
    AXI_TRY(ghost_comm<T>(vort, nr, nz, ghost, false, T(0), dx, s));                           \
    launch_rk2_stage1<T>(tmp, vort, R, nr, nz, c1, dx, s);                                     \
    AXI_TRY(ghost_comm<T>(tmp, nr, nz, ghost, false, T(0), dx, s));                            \
    launch_rk2_stage2<T>(vort, tmp, R, nr, nz, c2, dx, s);                                     \
    return axi::launch_status("diffusion_rk2_periodic");                                       \
  }                                                                                            \
  extern "C" int axi_periodic_ghost_comm_##SUF(T* f, int nr, int nz, int ghost, void* stream) { \
    axi::clear_error();                                                                        \
    return ghost_comm<T>(f, nr, nz, ghost, false, T(0), T(0), axi::as_stream(stream));         \
  }                                                                                            \
  extern "C" int axi_periodic_ghost_comm_eta_##SUF(T* f, int nr, int nz, int ghost, T z_max,   \
                                                   T dx, void* stream) {                       \
    axi::clear_error();                                                                        \
    return ghost_comm<T>(f, nr, nz, ghost, true, z_max, dx, axi::as_stream(stream));           \
  }                                                                                            \
  extern "C" int axi_solid_sigma_##SUF(T* s11, T* s12, T* s22, T G, T dx, const T* e1,        \
                                       const T* e2, T* e1z, T* e1r, T* e2z, T* e2r, int nr,    \
                                       int nz, void* stream) {                                 \
    axi::clear_error();                                                                        \
    AXI_TRY(axi::check_grid("solid_sigma", nr, nz));                                           \
    AXI_TRY(axi::check_ptrs("solid_sigma", {s11, s12, s22, e1, e2, e1z, e1r, e2z, e2r},        \
                            {"sigma_11", "sigma_12", "sigma_22", "eta1", "eta2", "eta1_z",     \
                             "eta1_r", "eta2_z", "eta2_r"}));                                  \
    solid_sigma_kernel<T><<<grid2d(nr, nz), dim3(BX, BY), 0, axi::as_stream(stream)>>>(        \
        s11, s12, s22, G, KnownDivisor<T>(rn_host_mul(T(2), dx)), e1, e2, e1z, e1r, e2z, e2r, nr, nz, \
        static_cast<const T*>(nullptr));                                                       \
    return axi::launch_status("solid_sigma");                                                  \
  }                                                                                            \
  extern "C" int axi_update_vorticity_from_solid_stress_##SUF(                                 \
      T* vort, T* tau_z, T* tau_r, const T* t11, const T* t12, const T* t22, const T* R,       \
      int nr, int nz, T dt, T dx, void* stream) {                                              \
    axi::clear_error();                                                                        \
    AXI_TRY(axi::check_grid("update_vorticity_from_solid_stress", nr, nz));                    \
    AXI_TRY(axi::check_ptrs("update_vorticity_from_solid_stress",                              \
                            {vort, tau_z, tau_r, t11, t12, t22, R},                            \
                            {"vorticity", "tau_z", "tau_r", "sigma_11", "sigma_12",            \
                             "sigma_22", "R"}));                                               \
    cudaStream_t s = axi::as_stream(stream);                                                   \
    const KnownDivisor<T> two_dx(rn_host_mul(T(2), dx));                                       \
    div_tau_kernel<T><<<grid2d(nr, nz), dim3(BX, BY), 0, s>>>(tau_z, tau_r, t11, t12, t22, R,  \
                                                               nr, nz, two_dx);                \
    curl_tau_kernel<T><<<grid2d(nr, nz), dim3(BX, BY), 0, s>>>(vort, tau_z, tau_r, nr, nz, dt, \
                                                                two_dx);                       \
    return axi::launch_status("update_vorticity_from_solid_stress");                           \
  }

AXI_DEFINE_VELOCITY(f64, double)
AXI_DEFINE_VELOCITY(f32, float)
AXI_DEFINE_VORTICITY(f64, double)
AXI_DEFINE_VORTICITY(f32, float)
AXI_DEFINE_POINTWISE(f64, double)
AXI_DEFINE_POINTWISE(f32, float)

// The soft-sphere loop's dt-dependent kernels with the time step read on the
// device (state[AXI_SOFT_DT]); the arithmetic of the host-dt entries above.
extern "C" int axi_soft_update_vorticity_from_solid_stress_f64(
    double* vort, double* tau_z, double* tau_r, const double* t11, const double* t12,
    const double* t22, const double* R, int nr, int nz, double dx, const double* state,
    void* stream) {
  axi::clear_error();
  AXI_TRY(axi::check_grid("soft_update_vorticity_from_solid_stress", nr, nz));
  AXI_TRY(axi::check_ptrs("soft_update_vorticity_from_solid_stress",
                          {vort, tau_z, tau_r, t11, t12, t22, R, state},
                          {"vorticity", "tau_z", "tau_r", "sigma_11", "sigma_12", "sigma_22", "R",
                           "state"}));
  cudaStream_t s = axi::as_stream(stream);
  const KnownDivisor<double> two_dx(rn_host_mul(2.0, dx));
  div_tau_kernel<double><<<grid2d(nr, nz), dim3(BX, BY), 0, s>>>(tau_z, tau_r, t11, t12, t22, R,
                                                                  nr, nz, two_dx);
  curl_tau_kernel<double><<<grid2d(nr, nz), dim3(BX, BY), 0, s>>>(
      vort, tau_z, tau_r, nr, nz, 0.0, two_dx, state + AXI_SOFT_DT);
  return axi::launch_status("soft_update_vorticity_from_solid_stress");
}

extern "C" int axi_soft_diffusion_rk2_f64(double* vort, double* tmp, const double* R, int nr,
                                          int nz, double nu, double dx, const double* state,
                                          void* stream) {
  axi::clear_error();
  AXI_TRY(axi::check_grid("soft_diffusion_rk2", nr, nz));
  AXI_TRY(axi::check_ptrs("soft_diffusion_rk2", {vort, tmp, R, state},
                          {"vorticity", "temp_vorticity", "R", "state"}));
  cudaStream_t s = axi::as_stream(stream);
  launch_rk2_stage1<double>(tmp, vort, R, nr, nz, rn_host_mul(0.5, nu), dx, s, state + AXI_SOFT_DT);
  launch_rk2_stage2<double>(vort, tmp, R, nr, nz, nu, dx, s, state + AXI_SOFT_DT);
  return axi::launch_status("soft_diffusion_rk2");
}

// The soft loop's stress: axi_solid_sigma_f64 followed by sigma *= chi
// (axi_soft_stress_mask_f64) in one pass.
extern "C" int axi_soft_stress_f64(double* s11, double* s12, double* s22, double G, double dx,
                                   const double* e1, const double* e2, double* e1z, double* e1r,
                                   double* e2z, double* e2r, const double* chi, int nr, int nz,
                                   void* stream) {
  axi::clear_error();
  AXI_TRY(axi::check_grid("soft_stress", nr, nz));
  AXI_TRY(axi::check_ptrs("soft_stress", {s11, s12, s22, e1, e2, e1z, e1r, e2z, e2r, chi},
                          {"sigma_11", "sigma_12", "sigma_22", "eta1", "eta2", "eta1_z", "eta1_r",
                           "eta2_z", "eta2_r", "chi"}));
  solid_sigma_kernel<double><<<grid2d(nr, nz), dim3(BX, BY), 0, axi::as_stream(stream)>>>(
      s11, s12, s22, G, KnownDivisor<double>(rn_host_mul(2.0, dx)), e1, e2, e1z, e1r, e2z, e2r, nr,
      nz, chi);
  return axi::launch_status("soft_stress");
}

extern "C" int axi_sphere_speed_f64(double* u_z, const double* u_r, double add, int64_t n,
                                    double* umax, void* stream) {
  axi::clear_error();
  if (n < 1) {
    axi::set_error("sphere_speed: no cells");
    return AXI_ERR_INVALID;
  }
  AXI_TRY(axi::check_ptrs("sphere_speed", {u_z, u_r, umax}, {"u_z", "u_r", "umax"}));
  cudaStream_t s = axi::as_stream(stream);
  if (cudaMemsetAsync(umax, 0, sizeof(double), s) != cudaSuccess)
    return axi::launch_status("sphere_speed");
  const long long blocks = (n + 1023) / 1024, cap = 8LL * axi::sm_count();
  sphere_speed_kernel<<<(unsigned)(blocks < cap ? blocks : cap), 256, 0, s>>>(
      u_z, u_r, add, n, reinterpret_cast<unsigned long long*>(umax));
  return axi::launch_status("sphere_speed");
}

extern "C" int64_t axi_sphere_penalise_partials(int nr, int nz) {
  return ((int64_t)nr * nz + SPHERE_CELLS - 1) / SPHERE_CELLS;
}

extern "C" int axi_sphere_penalise_f64(double* vorticity, double* penal, double* u_z, double* u_r,
                                       double* old_u_z, double* old_u_r, const double* chi,
                                       const double* R, double lam, double dt, int nr, int nz,
                                       double dx, double* partials, double* drag, void* stream) {
  axi::clear_error();
  AXI_TRY(axi::check_grid("sphere_penalise", nr, nz));
  const void* ptrs[] = {vorticity, penal, u_z, u_r, old_u_z, old_u_r, chi, R, partials, drag};
  for (const void* p : ptrs) AXI_TRY(axi::check_ptr("sphere_penalise", p, "field"));
  cudaStream_t s = axi::as_stream(stream);
  const long long n = (long long)nr * nz;
  const int blocks = (int)axi_sphere_penalise_partials(nr, nz);
  sphere_penalise_kernel<<<blocks, 256, 0, s>>>(u_z, u_r, old_u_z, old_u_r, chi, R, lam, dt, n,
                                                partials);
  sphere_curl_kernel<<<grid2d(nr, nz), dim3(BX, BY), 0, s>>>(
      vorticity, penal, u_z, u_r, old_u_z, old_u_r, nr, nz,
      KnownDivisor<double>(rn_host_mul(2.0, dx)), partials, blocks, drag);
  return axi::launch_status("sphere_penalise");
}
