// Least-squares front-marching extrapolation of the reference map (eta).
//
// core/src/extrapolate_using_least_squares.hpp:142-446 restated for the GPU:
//   sweep: every cell with current ^ target set and a known (current == 1)
//   cell among its 8 neighbours is a front cell; it fits c0 + c1 x + c2 y to
//   the known cells of a 3x3 window shifted towards the known side (start
//   codes, core/src/lstsq/ExtrapolationConfig.hpp:131-158), solves the 3x3
//   normal equations with the reference's pivoted elimination
//   (core/src/lstsq/least_squares.hpp:10-59) and evaluates the fit at the
//   cell; afterwards all front cells become known. Sweeps repeat until no
//   front cell is left.
// Within a sweep every front cell reads only known cells (the window mask is
// the pre-sweep flag), so front cells are independent and run in parallel;
// the arithmetic keeps the reference's order (no FMA) and gives the same bits.
//
// Layout: one multi-block pass collects the candidate cells (current ^ target)
// into a list. Eight sweeps over that list are spread over the GPU (one launch
// each on flags that the mirroring pass made, three on the caller's own); one
// block runs any that are still needed, up to the cap. Neighbours outside the array count as unknown; a window that
// leaves the array sets AXI_ERR_RANGE (the reference reads out of bounds).
#include "axi_common.cuh"

namespace {

constexpr int LSQ_THREADS = 1024;

struct LsqHeader {
  int n_candidates;
  int n_front;
  int status;
  int sweeps;
  // multi-block sweeps: front counts (three-launch sweeps: even / odd sweeps;
  // one-launch sweeps: sweep mod 3), the done flag
  int front_count[2];
  int done;
  int fail;  // one-launch sweeps: (sweep + 1) << 8 | status of the first failure
};
static_assert(sizeof(LsqHeader) == 32, "header is the first 32 bytes of the work buffer");

__global__ void lsq_collect_kernel(const int16_t* __restrict__ cf, const int16_t* __restrict__ tf,
                                   long long n, LsqHeader* hdr, int* __restrict__ list) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  if (cf[k] ^ tf[k]) {
    const int slot = atomicAdd(&hdr->n_candidates, 1);
    list[slot] = (int)k;
  }
}

__device__ __forceinline__ int start_code(int positional_sum, int total_sum) {
  // ExtrapolationConfig.hpp:131-138 (code) and :143-148 (start code, grid 3).
  // The reference's float and double expressions of these small integers are
  // exact up to the final truncation, which integer division does as well.
  const int t = positional_sum > 4 ? (positional_sum + 1) / 2 * 2 : positional_sum;
  return (2 * (2 * t / total_sum) - 6) / 2;
}

// The reference's unqualified abs(double) is C's int abs(int).
// With the usual magnitudes the fraction bits are cleared on the integer pipe.
__device__ __forceinline__ double int_abs(double x) {
  const long long b = __double_as_longlong(x) & 0x7fffffffffffffffll;
  const int e = (int)(b >> 52) - 1023;
  if (e < 0) return 0.0;
  if (e < 31) return __longlong_as_double(b & ~(0xfffffffffffffll >> e));
  int i = __double2int_rz(x);
  return (double)(i < 0 ? -i : i);
}
// x > y for non-negative doubles (and no NaN in y) by their bits
__device__ __forceinline__ bool greater_bits(double x, double y) {
  return __double_as_longlong(x) > __double_as_longlong(y);
}

__device__ __forceinline__ void gauss3x2(double A[3][5], double sol[2][3]) {
  KnownDivisor<double> pivot[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    int max_row = i;
    double max_el = int_abs(A[i][i]);
#pragma unroll
    for (int k = i + 1; k < 3; ++k) {
      if (greater_bits(int_abs(A[k][i]), max_el)) {
        max_el = fabs(A[k][i]);
        max_row = k;
      }
    }
#pragma unroll
    for (int k = i + 1; k < 3; ++k) {
      if (max_row != k) continue;
#pragma unroll
      for (int c = i; c < 5; ++c) {
        const double t = A[k][c];
        A[k][c] = A[i][c];
        A[i][c] = t;
      }
    }
    pivot[i] = KnownDivisor<double>(A[i][i]);
#pragma unroll
    for (int k = i + 1; k < 3; ++k) {
      const double c = pivot[i].quotient(-A[k][i]);
      A[k][i] = 0.0;
#pragma unroll
      for (int j = i + 1; j < 5; ++j) A[k][j] = __dadd_rn(A[k][j], __dmul_rn(c, A[i][j]));
    }
  }
#pragma unroll
  for (int comp = 0; comp < 2; ++comp) {
#pragma unroll
    for (int i = 2; i >= 0; --i) {
      sol[comp][i] = pivot[i].quotient(A[i][3 + comp]);
#pragma unroll
      for (int k = i - 1; k >= 0; --k)
        A[k][3 + comp] = __dsub_rn(A[k][3 + comp], __dmul_rn(A[k][i], sol[comp][i]));
    }
  }
}

// The flag of a cell as the sweep at hand sees it: the array itself, ...
struct PlainFlags {
  const int16_t* f;
  __device__ __forceinline__ int operator()(long long g) const { return f[g]; }
};
// ... or, where a sweep stores sweep + 2 into the cells it fills (0: unknown,
// 1: known from the start), whether the cell was known before it.
struct SweepFlags {
  const volatile int16_t* f;
  int sweep;
  __device__ __forceinline__ int operator()(long long g) const {
    const int v = f[g];
    return v >= 1 && v <= sweep + 1;
  }
};

// Front scan of candidate cell k (extrapolate_using_least_squares.hpp:196-253):
// a cell still to be filled (current ^ target) with a known neighbour among
// its 8 is a front cell; f receives its position and start codes.
template <typename Flags>
__device__ __forceinline__ bool front_cell(const Flags cf, const int16_t* __restrict__ tf, int n0,
                                           int n1, int k, int4& f) {
  // Flags only ever go 0 -> 1, so the collected list is a superset of the
  // live candidates; re-test current ^ target against the live flag.
  if ((cf(k) ^ tf[k]) == 0) return false;
  const int j = k / n1, i = k - j * n1;
  int s = 0, sx = 0, sy = 0;
#pragma unroll
  for (int jl = -1; jl <= 1; ++jl) {
    const int jj = j + jl;
#pragma unroll
    for (int il = -1; il <= 1; ++il) {
      const int ii = i + il;
      int v = 0;
      if (jj >= 0 && jj < n0 && ii >= 0 && ii < n1) v = cf((long long)jj * n1 + ii);
      if (jl != 0 || il != 0) s += v;
      sx += v * (il + 1);
      sy += v * (jl + 1);
    }
  }
  if (s == 0) return false;
  f = make_int4(i, j, start_code(sx, s), start_code(sy, s));
  return true;
}

// Product of a flag and a value. A flag of 0 or 1 needs no FP64 instruction
// (0 x is a zero of x's sign, or NaN).
__device__ __forceinline__ double masked(int m, double x) {
  if (m == 1) return x;
  const unsigned int hi = (unsigned int)__double2hiint(x);
  if (m == 0 && ((hi >> 20) & 0x7ffu) != 0x7ffu)
    return __hiloint2double((int)(hi & 0x80000000u), 0);
  return __dmul_rn((double)m, x);
}

// Local least-squares fit of front cell f (extrapolate_using_least_squares.hpp:274-438);
// false (nothing written) when the 3x3 window leaves the grid. The normal
// matrix is symmetric and its first row and column are plain sums of the
// masked values where the flags are 0 or 1 (0 and 1 are their own squares and
// a masked value times its flag is itself), which leaves 7 of the 15 sums with
// products, in the reference's order.
template <typename Flags>
__device__ __forceinline__ bool fit_cell(const Flags cf, double* ex, double* ey,
                                         const double* __restrict__ gx,
                                         const double* __restrict__ gy, int n0, int n1, int4 f) {
  const int i = f.x, j = f.y;
  const int i0 = i + f.z, j0 = j + f.w;
  if (i0 < 0 || j0 < 0 || i0 + 3 > n1 || j0 + 3 > n0) return false;
  double xm[9], ym[9], r0[9], r1[9], m[9];
  bool unit = true;
#pragma unroll
  for (int jl = 0; jl < 3; ++jl) {
    const double y = gy[j0 + jl];
#pragma unroll
    for (int il = 0; il < 3; ++il) {
      const int p = 3 * jl + il;
      const long long g = (long long)(j0 + jl) * n1 + i0 + il;
      const int mk = cf(g);
      unit = unit && (mk == 0 || mk == 1);
      m[p] = mk == 0 ? 0.0 : mk == 1 ? 1.0 : (double)mk;
      xm[p] = masked(mk, gx[i0 + il]);
      ym[p] = masked(mk, y);
      r0[p] = masked(mk, ex[g]);
      r1[p] = masked(mk, ey[g]);
    }
  }
  auto sum = [](const double (&a)[9]) {
    double acc = 0.0;
#pragma unroll
    for (int t = 0; t < 9; ++t) acc = __dadd_rn(acc, a[t]);
    return acc;
  };
  auto dot = [](const double (&a)[9], const double (&b)[9]) {
    double acc = 0.0;
#pragma unroll
    for (int t = 0; t < 9; ++t) acc = __dadd_rn(acc, __dmul_rn(a[t], b[t]));
    return acc;
  };
  double A[3][5];
  if (unit) {
    A[0][0] = sum(m);
    A[0][1] = sum(xm);
    A[0][2] = sum(ym);
    A[0][3] = sum(r0);
    A[0][4] = sum(r1);
  } else {
    A[0][0] = dot(m, m);
    A[0][1] = dot(m, xm);
    A[0][2] = dot(m, ym);
    A[0][3] = dot(m, r0);
    A[0][4] = dot(m, r1);
  }
  A[1][0] = A[0][1];
  A[1][1] = dot(xm, xm);
  A[1][2] = dot(xm, ym);
  A[1][3] = dot(xm, r0);
  A[1][4] = dot(xm, r1);
  A[2][0] = A[0][2];
  A[2][1] = A[1][2];
  A[2][2] = dot(ym, ym);
  A[2][3] = dot(ym, r0);
  A[2][4] = dot(ym, r1);
  double sol[2][3];
  gauss3x2(A, sol);
  const double loc[3] = {1.0, gx[i], gy[j]};
  double e0 = 0.0, e1 = 0.0;
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    e0 = __dadd_rn(e0, __dmul_rn(sol[0][t], loc[t]));
    e1 = __dadd_rn(e1, __dmul_rn(sol[1][t], loc[t]));
  }
  const long long c = (long long)j * n1 + i;
  ex[c] = e0;
  ey[c] = e1;
  return true;
}

// All remaining sweeps in one CTA: scan, fits, flag update, until no front is
// left (or the cap). Continues from the sweep count and status that earlier
// multi-block sweeps left in the header.
__device__ __forceinline__ void finish_sweeps(int16_t* cf, const int16_t* tf, double* ex,
                                              double* ey, const double* gx, const double* gy,
                                              int n0, int n1, int max_sweeps, LsqHeader* hdr,
                                              const int* list, int4* front) {
  __shared__ int s_front;
  __shared__ int s_status;
  const int ncand = hdr->n_candidates;
  if (threadIdx.x == 0) s_status = AXI_OK;
  int sweeps = hdr->sweeps;
  for (;;) {
    if (threadIdx.x == 0) s_front = 0;
    __syncthreads();
    // 1. front scan
    for (int q = threadIdx.x; q < ncand; q += LSQ_THREADS) {
      int4 f;
      if (front_cell(PlainFlags{cf}, tf, n0, n1, list[q], f)) front[atomicAdd(&s_front, 1)] = f;
    }
    __syncthreads();
    const int nfront = s_front;
    if (nfront == 0) break;
    if (++sweeps > max_sweeps) {
      if (threadIdx.x == 0) s_status = AXI_ERR_NOT_CONVERGED;
      break;
    }
    // 2. local fits
    for (int q = threadIdx.x; q < nfront; q += LSQ_THREADS)
      if (!fit_cell(PlainFlags{cf}, ex, ey, gx, gy, n0, n1, front[q])) s_status = AXI_ERR_RANGE;
    __syncthreads();
    // 3. flag update (extrapolate_using_least_squares.hpp:441-444)
    for (int q = threadIdx.x; q < nfront; q += LSQ_THREADS) {
      const int4 f = front[q];
      cf[(long long)f.y * n1 + f.x] = 1;
    }
    __syncthreads();
    if (s_status != AXI_OK) break;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    hdr->status = s_status;
    hdr->sweeps = sweeps;
    hdr->done = 1;
  }
}

__global__ void __launch_bounds__(LSQ_THREADS)
    lsq_sweep_kernel(int16_t* cf, const int16_t* tf, double* ex, double* ey, const double* gx,
                     const double* gy, int n0, int n1, int max_sweeps, LsqHeader* hdr,
                     const int* list, int4* front) {
  if (hdr->status != AXI_OK || hdr->done) return;
  finish_sweeps(cf, tf, ex, ey, gx, gy, n0, n1, max_sweeps, hdr, list, front);
}

// fit_cell by four lanes (flags 0 or 1): lane `part` forms three of the sums,
// the same terms in the same order, and every lane solves the system. All
// lanes of the warp call it; `active` per group of four. False: the window
// leaves the grid.
__device__ __forceinline__ bool fit_cell_quad(const SweepFlags cf, double* ex, double* ey,
                                              const double* __restrict__ gx,
                                              const double* __restrict__ gy, int n0, int n1,
                                              int4 f, bool active) {
  const int lane = threadIdx.x & 31, part = lane & 3, quad = lane & 28;
  const int i = f.x, j = f.y;
  const int i0 = i + f.z, j0 = j + f.w;
  const bool inside = i0 >= 0 && j0 >= 0 && i0 + 3 <= n1 && j0 + 3 <= n0;
  double one[9], xm[9], ym[9], r0[9], r1[9];
  int count = 0;
#pragma unroll
  for (int p = 0; p < 9; ++p) one[p] = xm[p] = ym[p] = r0[p] = r1[p] = 0.0;
  if (active && inside) {
#pragma unroll
    for (int jl = 0; jl < 3; ++jl) {
      const double y = gy[j0 + jl];
#pragma unroll
      for (int il = 0; il < 3; ++il) {
        const int p = 3 * jl + il;
        const long long g = (long long)(j0 + jl) * n1 + i0 + il;
        const int m = cf(g);
        count += m;
        one[p] = m ? 1.0 : 0.0;
        xm[p] = masked(m, gx[i0 + il]);
        ym[p] = masked(m, y);
        r0[p] = masked(m, ex[g]);
        r1[p] = masked(m, ey[g]);
      }
    }
  }
  // sums part + 4 q: 0 (0,1) 1 (0,2) 2 (0,3) 3 (0,4) 4 (1,1) 5 (1,3) 6 (1,4)
  // 7 (1,2) 8 (2,2) 9 (2,3) 10 (2,4), columns 3 and 4 the right-hand sides
  double acc[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    double t = 0.0;
#pragma unroll
    for (int p = 0; p < 9; ++p) {
      const double a = q == 0 ? one[p] : q == 1 ? xm[p] : ym[p];
      const double b = q == 0   ? (part == 0 ? xm[p] : part == 1 ? ym[p] : part == 2 ? r0[p] : r1[p])
                       : q == 1 ? (part == 0 ? xm[p] : part == 1 ? r0[p] : part == 2 ? r1[p] : ym[p])
                                : (part == 0 ? ym[p] : part == 1 ? r0[p] : r1[p]);
      t = __dadd_rn(t, __dmul_rn(a, b));
    }
    acc[q] = t;
  }
  auto from = [&](int q, int p) { return __shfl_sync(0xffffffffu, acc[q], quad + p); };
  double A[3][5];
  A[0][0] = (double)count;
  A[0][1] = A[1][0] = from(0, 0);
  A[0][2] = A[2][0] = from(0, 1);
  A[0][3] = from(0, 2);
  A[0][4] = from(0, 3);
  A[1][1] = from(1, 0);
  A[1][3] = from(1, 1);
  A[1][4] = from(1, 2);
  A[1][2] = A[2][1] = from(1, 3);
  A[2][2] = from(2, 0);
  A[2][3] = from(2, 1);
  A[2][4] = from(2, 2);
  if (!active) A[0][0] = A[1][1] = A[2][2] = 1.0;  // no division by zero beside the others
  double sol[2][3];
  gauss3x2(A, sol);
  if (active && inside && part < 2) {
    double e = __dadd_rn(0.0, part == 0 ? sol[0][0] : sol[1][0]);
    e = __dadd_rn(e, __dmul_rn(part == 0 ? sol[0][1] : sol[1][1], gx[i]));
    e = __dadd_rn(e, __dmul_rn(part == 0 ? sol[0][2] : sol[1][2], gy[j]));
    (part == 0 ? ex : ey)[(long long)j * n1 + i] = e;
  }
  return inside;
}

// Sweep `sweep` of the eta extrapolation (flags 0 or 1) in one launch: four
// lanes scan a candidate and fit it at once if it is a front cell. The cells
// filled are marked sweep + 2, which this sweep reads as unknown and the next
// ones as known (SweepFlags), so neither the front list nor a pass that sets
// the flags is needed; the launch boundary is the barrier between sweeps.
// Bound by the latency of one fit (an FP64 instruction holds a scheduler's
// FP64 unit for 64 cycles whatever the number of active lanes), so blocks are
// single warps spread over the SMs. One lane per candidate (270 FP64
// instructions instead of 150) took 14 us a sweep, 16 lanes per front cell (a
// warp's front cells after each other, since they come in clusters) 18-24 us.
constexpr int FS_THREADS = 32;
__device__ __forceinline__ int* sweep_count(LsqHeader* hdr, int sweep) {
  const int q = sweep % 3;
  return q == 0 ? &hdr->n_front : &hdr->front_count[q - 1];
}

__global__ void __launch_bounds__(FS_THREADS)
    lsq_fused_sweep_kernel(int16_t* cf, const int16_t* __restrict__ tf, double* ex, double* ey,
                           const double* __restrict__ gx, const double* __restrict__ gy, int n0,
                           int n1, int max_sweeps, LsqHeader* hdr, const int* __restrict__ list,
                           int sweep) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *sweep_count(hdr, sweep + 1) = 0;
  const int fail = *reinterpret_cast<volatile int*>(&hdr->fail);
  if (sweep > 0 && (*sweep_count(hdr, sweep - 1) == 0 || (fail != 0 && (fail >> 8) <= sweep)))
    return;
  const SweepFlags flags{cf, sweep};
  const int ncand = hdr->n_candidates;
  const int lane = threadIdx.x, part = lane & 3;
  for (int base = blockIdx.x * 8; base < ncand; base += gridDim.x * 8) {
    const int q = base + (lane >> 2);
    const int k = q < ncand ? list[q] : 0;
    const int j = k / n1, i = k - j * n1;
    const bool live = q < ncand && (flags(k) ^ tf[k]) != 0;
    // neighbour sums (front_cell): lane `part` takes row j + part - 1
    int s = 0, sx = 0, sy = 0;
    const int jj = j + part - 1;
    if (live && part < 3 && jj >= 0 && jj < n0) {
#pragma unroll
      for (int il = -1; il <= 1; ++il) {
        const int ii = i + il;
        const int v = ii >= 0 && ii < n1 ? flags((long long)jj * n1 + ii) : 0;
        if (part != 1 || il != 0) s += v;
        sx += v * (il + 1);
        sy += v * part;
      }
    }
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, o);
      sx += __shfl_xor_sync(0xffffffffu, sx, o);
      sy += __shfl_xor_sync(0xffffffffu, sy, o);
    }
    const bool front = live && s != 0;
    if (!__any_sync(0xffffffffu, front)) continue;
    if (lane == 0) hdr->sweeps = sweep + 1;
    if (sweep + 1 > max_sweeps) {
      // the cap: counted as one more sweep, nothing filled
      if (lane == 0) hdr->fail = (sweep + 1) << 8 | AXI_ERR_NOT_CONVERGED;
      continue;
    }
    if (lane == 0) *sweep_count(hdr, sweep) = 1;  // any front cell: the next sweep runs
    const int4 f = make_int4(i, j, front ? start_code(sx, s) : 0, front ? start_code(sy, s) : 0);
    const bool ok = fit_cell_quad(flags, ex, ey, gx, gy, n0, n1, f, front);
    if (front && part == 0) {
      if (!ok) hdr->fail = (sweep + 1) << 8 | AXI_ERR_RANGE;
      if (cf[k] == 0) cf[k] = (int16_t)(sweep + 2);
    }
  }
}

// After `sweeps` fused sweeps: flags back to 0 / 1, any further sweeps in the
// first block, and (state given: the soft loop) the outcome folded into its state
// block (the status bit of a failure, sticky, and the largest sweep count
// seen) and the filled cells of the upper half copied to eta1 and eta2. A chain
// of three loads a candidate (a step with one block / eight, same GPU: 256 x 128
// 195.0 / 193.9 us, 1024 x 512 437.1 / 433.0).
constexpr int FINISH_BLOCKS = 8;
__global__ void __launch_bounds__(LSQ_THREADS)
    lsq_finish_kernel(int16_t* cf, const int16_t* tf, double* ex, double* ey, const double* gx,
                      const double* gy, int n0, int n1, int max_sweeps, LsqHeader* hdr,
                      const int* list, int4* front, int sweeps, double* state, double* eta1,
                      double* eta2) {
  const int ncand = hdr->n_candidates;
  const int fail = hdr->fail;
  const bool more = fail == 0 && *sweep_count(hdr, sweeps - 1) != 0;
  if (more && blockIdx.x > 0) return;
  const int first = blockIdx.x * LSQ_THREADS + threadIdx.x;
  const int step = more ? LSQ_THREADS : FINISH_BLOCKS * LSQ_THREADS;
  const int half = n0 / 2 * n1;
  auto copy_back = [&](int k) {
    if (!state || k < half) return;
    eta1[k - half] = ex[k];
    eta2[k - half] = ey[k];
  };
  for (int q = first; q < ncand; q += step) {
    const int k = list[q];
    if (cf[k] > 1) cf[k] = 1;
    if (!more) copy_back(k);
  }
  if (more) {
    __syncthreads();
    finish_sweeps(cf, tf, ex, ey, gx, gy, n0, n1, max_sweeps, hdr, list, front);
    __syncthreads();
    for (int q = first; q < ncand; q += step) copy_back(list[q]);
  } else if (first == 0) {
    hdr->status = fail & 0xff;
    hdr->done = 1;
  }
  if (!state || first != 0) return;
  if (hdr->status != AXI_OK)
    atomicOr(reinterpret_cast<unsigned long long*>(state + AXI_SOFT_STATUS),
             1ull << hdr->status);
  if ((double)hdr->sweeps > state[AXI_SOFT_SWEEPS]) state[AXI_SOFT_SWEEPS] = hdr->sweeps;
}

// The same sweep spread over the GPU, three launches per sweep (scan, fits,
// flag update; a launch boundary is the barrier between them). A fixed
// number of these sweeps is issued; once no front is left (or on a failure)
// the remaining launches return at once, and lsq_sweep_kernel finishes
// whatever sweeps are still needed. Front cells of a sweep are independent
// (each reads only the flags before the sweep), so the results are the
// single-CTA kernel's.
__global__ void lsq_scan_mb_kernel(const int16_t* __restrict__ cf,
                                   const int16_t* __restrict__ tf, int n0, int n1,
                                   LsqHeader* hdr, const int* __restrict__ list,
                                   int4* __restrict__ front, int parity) {
  if (hdr->status != AXI_OK || hdr->done) return;
  const int ncand = hdr->n_candidates;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < ncand; q += gridDim.x * blockDim.x) {
    int4 f;
    if (front_cell(PlainFlags{cf}, tf, n0, n1, list[q], f))
      front[atomicAdd(&hdr->front_count[parity], 1)] = f;
  }
}

__global__ void lsq_fit_mb_kernel(const int16_t* __restrict__ cf, double* __restrict__ ex,
                                  double* __restrict__ ey, const double* __restrict__ gx,
                                  const double* __restrict__ gy, int n0, int n1, int max_sweeps,
                                  LsqHeader* hdr, const int4* __restrict__ front, int parity) {
  if (hdr->status != AXI_OK || hdr->done) return;
  const int nfront = hdr->front_count[parity];
  if (nfront == 0) return;
  if (hdr->sweeps + 1 > max_sweeps) {
    // the cap: counted as one more sweep, as the single-CTA loop does
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      hdr->status = AXI_ERR_NOT_CONVERGED;
      hdr->sweeps += 1;
    }
    return;
  }
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nfront; q += gridDim.x * blockDim.x)
    if (!fit_cell(PlainFlags{cf}, ex, ey, gx, gy, n0, n1, front[q]))
      atomicCAS(&hdr->status, AXI_OK, AXI_ERR_RANGE);
}

__global__ void lsq_flag_mb_kernel(int16_t* __restrict__ cf, int n1, LsqHeader* hdr,
                                   const int4* __restrict__ front, int parity) {
  if (hdr->done || hdr->status == AXI_ERR_NOT_CONVERGED) return;
  const int nfront = hdr->front_count[parity];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    hdr->front_count[parity ^ 1] = 0;  // the next sweep's count
    if (nfront == 0)
      hdr->done = 1;
    else
      hdr->sweeps += 1;
  }
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nfront; q += gridDim.x * blockDim.x) {
    const int4 f = front[q];
    cf[(long long)f.y * n1 + f.x] = 1;
  }
}

}  // namespace

extern "C" int64_t axi_lsq_work_bytes(int n0, int n1) {
  const long long n = (long long)n0 * n1;
  return (int64_t)(sizeof(LsqHeader) + 16 + n * (long long)sizeof(int) + 16 +
                   n * (long long)sizeof(int4));
}

namespace {

// Sweeps issued as multi-block launches before the single-CTA kernel takes
// over: front marching needs about extrap_zone / dx sweeps (6 or 7 on the
// soft-sphere grids, plus one that finds no front), so these usually finish
// the extrapolation.
constexpr int MB_SWEEPS = 8;

int sweep_blocks(int per_sm) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return per_sm * (sms > 0 ? sms : 1);
}

// Flags of any value (the drop-in on the caller's own flags): three launches a
// sweep.
void issue_sweeps(int16_t* cf, const int16_t* tf, double* ex, double* ey, const double* gx,
                  const double* gy, int n0, int n1, int max_sweeps, LsqHeader* hdr,
                  const int* list, int4* front, cudaStream_t s) {
  const int blocks = sweep_blocks(2);
  for (int k = 0; k < MB_SWEEPS; ++k) {
    const int parity = k & 1;
    lsq_scan_mb_kernel<<<blocks, 256, 0, s>>>(cf, tf, n0, n1, hdr, list, front, parity);
    lsq_fit_mb_kernel<<<blocks, 128, 0, s>>>(cf, ex, ey, gx, gy, n0, n1, max_sweeps, hdr, front,
                                              parity);
    lsq_flag_mb_kernel<<<blocks, 256, 0, s>>>(cf, n1, hdr, front, parity);
  }
  lsq_sweep_kernel<<<1, LSQ_THREADS, 0, s>>>(cf, tf, ex, ey, gx, gy, n0, n1, max_sweeps, hdr,
                                             list, front);
}

// Flags that lsq_prepare_kernel made (0 or 1): one launch a sweep. On the
// soft-sphere step at 1024 x 512 (about 4000 candidates, 6 sweeps) the whole
// extrapolation took 235 us with three launches a sweep (kernel times summed)
// and takes 121.
void issue_fused_sweeps(int16_t* cf, const int16_t* tf, double* ex, double* ey, const double* gx,
                        const double* gy, int n0, int n1, int max_sweeps, LsqHeader* hdr,
                        const int* list, int4* front, cudaStream_t s, double* state = nullptr,
                        double* eta1 = nullptr, double* eta2 = nullptr) {
  const int blocks = sweep_blocks(4);
  for (int k = 0; k < MB_SWEEPS; ++k)
    lsq_fused_sweep_kernel<<<blocks, FS_THREADS, 0, s>>>(cf, tf, ex, ey, gx, gy, n0, n1,
                                                         max_sweeps, hdr, list, k);
  lsq_finish_kernel<<<FINISH_BLOCKS, LSQ_THREADS, 0, s>>>(cf, tf, ex, ey, gx, gy, n0, n1, max_sweeps, hdr,
                                              list, front, MB_SWEEPS, state, eta1, eta2);
}

struct LsqWork {
  LsqHeader* hdr;
  int* list;
  int4* front;
};

LsqWork lsq_work(void* work, long long n) {
  char* base = static_cast<char*>(work);
  size_t off = 32 + n * sizeof(int);
  off = (off + 15) & ~size_t(15);
  return LsqWork{reinterpret_cast<LsqHeader*>(base), reinterpret_cast<int*>(base + 32),
                 reinterpret_cast<int4*>(base + off)};
}

// Reads the header back (synchronises): the outcome as an AXI status.
int lsq_outcome(const char* what, const LsqHeader* hdr, int n0, int n1, int max_sweeps,
                int* sweeps_out, cudaStream_t s) {
  LsqHeader h;
  if (cudaMemcpyAsync(&h, hdr, sizeof(h), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return axi::launch_status(what);
  if (sweeps_out) *sweeps_out = h.sweeps;
  if (h.status == AXI_ERR_NOT_CONVERGED) {
    axi::set_error("%s: no convergence after %d sweeps", what, max_sweeps);
  } else if (h.status == AXI_ERR_RANGE) {
    axi::set_error("%s: a 3x3 fitting window leaves the %d x %d grid", what, n0, n1);
  }
  return h.status;
}

int lsq_run(int16_t* cf, const int16_t* tf, double* ex, double* ey, const double* gx,
            const double* gy, int n0, int n1, int max_sweeps, void* work, int* sweeps_out,
            cudaStream_t s) {
  const char* what = "extrapolate_lsq_first_order";
  if (n0 < 1 || n1 < 1 || max_sweeps < 0) {
    axi::set_error("%s: invalid size %d x %d", what, n0, n1);
    return AXI_ERR_INVALID;
  }
  AXI_TRY(axi::check_ptrs(what, {cf, tf, ex, ey, gx, gy, work},
                          {"current_flag", "target_flag", "eta_x", "eta_y", "grid_x", "grid_y",
                           "work"}));
  const long long n = (long long)n0 * n1;
  const LsqWork w = lsq_work(work, n);
  if (cudaMemsetAsync(w.hdr, 0, sizeof(LsqHeader), s) != cudaSuccess)
    return axi::launch_status(what);
  lsq_collect_kernel<<<axi::ceil_div(n, 256), 256, 0, s>>>(cf, tf, n, w.hdr, w.list);
  issue_sweeps(cf, tf, ex, ey, gx, gy, n0, n1, max_sweeps, w.hdr, w.list, w.front, s);
  AXI_TRY(axi::launch_status(what));
  return lsq_outcome(what, w.hdr, n0, n1, max_sweeps, sweeps_out, s);
}

// Adds the lanes' cells to the candidate list, one atomic per warp.
__device__ __forceinline__ void add_candidate(bool cand, long long k, LsqHeader* hdr, int* list) {
  const unsigned int mask = __ballot_sync(0xffffffffu, cand);
  if (mask == 0) return;
  const int lane = threadIdx.x & 31;
  int base = 0;
  if (lane == 0) base = atomicAdd(&hdr->n_candidates, __popc(mask));
  base = __shfl_sync(0xffffffffu, base, 0);
  if (cand) list[base + __popc(mask & ((1u << lane) - 1))] = (int)k;
}

// extrapolate_eta_using_least_squares_unb.py:19-24 and
// extrapolate_using_least_squares.py:33-35: doubled (2 nr, nz) buffers, upper
// half = field, lower half = flipped mirror; flags from the doubled level set
// and the list of cells to fill. One thread per cell of the field. KEEP: eta1
// and eta2 are left as they are; else they get what a copy of the upper half
// would give, so that only the filled cells remain to be copied back.
template <bool KEEP>
__global__ void lsq_prepare_kernel(const uint8_t* __restrict__ inside,
                                   const double* __restrict__ phi, double* eta1, double* eta2,
                                   double* __restrict__ phid, double* __restrict__ e1d,
                                   double* __restrict__ e2d, int16_t* __restrict__ cf,
                                   int16_t* __restrict__ tf, double zone, int nr, int nz,
                                   LsqHeader* hdr, int* __restrict__ list) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = blockIdx.y;
  const bool in_grid = j < nz;
  const long long src = (long long)i * nz + j;
  const long long up = (long long)(nr + i) * nz + j, down = (long long)(nr - 1 - i) * nz + j;
  bool cand = false;
  if (in_grid) {
    const int in = inside[src] ? 1 : 0;
    const double p = -phi[src];
    const double m1 = masked(in, eta1[src]);
    const double m2 = masked(in, eta2[src]);
    const int16_t c = p < 0.0 ? 1 : 0, t = p < zone ? 1 : 0;
    cand = c != t;
    phid[up] = p;
    phid[down] = p;
    e1d[up] = m1;
    e1d[down] = m1;
    e2d[up] = m2;
    e2d[down] = -m2;
    cf[up] = c;
    cf[down] = c;
    tf[up] = t;
    tf[down] = t;
    if (!KEEP) {
      eta1[src] = m1;
      eta2[src] = m2;
    }
  }
  add_candidate(cand, up, hdr, list);
  add_candidate(cand, down, hdr, list);
}

__global__ void lsq_copyback_kernel(const double* __restrict__ e1d, const double* __restrict__ e2d,
                                    double* __restrict__ eta1, double* __restrict__ eta2, int nr,
                                    int nz) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = blockIdx.y;
  if (j >= nz || i >= nr) return;
  const long long c = (long long)i * nz + j;
  const long long d = (long long)(nr + i) * nz + j;
  eta1[c] = e1d[d];
  eta2[c] = e2d[d];
}

}  // namespace

extern "C" int axi_extrapolate_lsq_first_order_f64(int16_t* current_flag,
                                                   const int16_t* target_flag, double* eta_x,
                                                   double* eta_y, const double* grid_x,
                                                   const double* grid_y, int n0, int n1,
                                                   int max_sweeps, void* work, int* sweeps_out,
                                                   void* stream) {
  axi::clear_error();
  return lsq_run(current_flag, target_flag, eta_x, eta_y, grid_x, grid_y, n0, n1, max_sweeps,
                 work, sweeps_out, axi::as_stream(stream));
}

extern "C" int axi_extrapolate_eta_with_least_squares_f64(
    const uint8_t* inside_solid, const double* ball_phi, double* eta1, double* eta2,
    double* ball_phi_double, double* eta1_double, double* eta2_double, int16_t* current_flag,
    int16_t* target_flag, double extrap_zone, int nr, int nz, const double* grid_x,
    const double* grid_y, int max_sweeps, void* work, int* sweeps_out, void* stream) {
  axi::clear_error();
  const char* what = "extrapolate_eta_with_least_squares";
  if (nr < 1 || nz < 1 || 2 * nr > 65535) {
    axi::set_error("%s: invalid grid %d x %d", what, nr, nz);
    return AXI_ERR_INVALID;
  }
  AXI_TRY(axi::check_ptrs(what,
                          {inside_solid, ball_phi, eta1, eta2, ball_phi_double, eta1_double,
                           eta2_double, current_flag, target_flag, grid_x, grid_y, work},
                          {"inside_solid", "ball_phi", "eta1", "eta2", "ball_phi_double",
                           "eta1_double", "eta2_double", "current_flag", "target_flag", "grid_x",
                           "grid_y", "work"}));
  cudaStream_t s = axi::as_stream(stream);
  dim3 g1(axi::ceil_div(nz, 128), nr);
  const int n0 = 2 * nr, n1 = nz;
  const LsqWork w = lsq_work(work, (long long)n0 * n1);
  if (max_sweeps < 0) {
    axi::set_error("%s: invalid sweep limit %d", what, max_sweeps);
    return AXI_ERR_INVALID;
  }
  if (cudaMemsetAsync(w.hdr, 0, sizeof(LsqHeader), s) != cudaSuccess)
    return axi::launch_status(what);
  lsq_prepare_kernel<true><<<g1, 128, 0, s>>>(inside_solid, ball_phi, eta1, eta2, ball_phi_double,
                                              eta1_double, eta2_double, current_flag, target_flag,
                                              extrap_zone, nr, nz, w.hdr, w.list);
  issue_fused_sweeps(current_flag, target_flag, eta1_double, eta2_double, grid_x, grid_y, n0, n1,
                     max_sweeps, w.hdr, w.list, w.front, s);
  AXI_TRY(axi::launch_status(what));
  AXI_TRY(lsq_outcome(what, w.hdr, n0, n1, max_sweeps, sweeps_out, s));
  lsq_copyback_kernel<<<g1, 128, 0, s>>>(eta1_double, eta2_double, eta1, eta2, nr, nz);
  return axi::launch_status(what);
}

// The soft loop's extrapolation without a host round trip: the same kernels
// as axi_extrapolate_eta_with_least_squares_f64; the outcome goes to
// state[AXI_SOFT_STATUS] (bit 1 << AXI_ERR_NOT_CONVERGED or AXI_ERR_RANGE) and
// state[AXI_SOFT_SWEEPS] instead of the return value.
extern "C" int axi_soft_extrapolate_eta_f64(
    const uint8_t* inside_solid, const double* ball_phi, double* eta1, double* eta2,
    double* ball_phi_double, double* eta1_double, double* eta2_double, int16_t* current_flag,
    int16_t* target_flag, double extrap_zone, int nr, int nz, const double* grid_x,
    const double* grid_y, int max_sweeps, void* work, double* state, void* stream) {
  axi::clear_error();
  const char* what = "soft_extrapolate_eta";
  if (nr < 1 || nz < 1 || 2 * nr > 65535 || max_sweeps < 0) {
    axi::set_error("%s: invalid grid %d x %d", what, nr, nz);
    return AXI_ERR_INVALID;
  }
  AXI_TRY(axi::check_ptrs(what,
                          {inside_solid, ball_phi, eta1, eta2, ball_phi_double, eta1_double,
                           eta2_double, current_flag, target_flag, grid_x, grid_y, work, state},
                          {"inside_solid", "ball_phi", "eta1", "eta2", "ball_phi_double",
                           "eta1_double", "eta2_double", "current_flag", "target_flag", "grid_x",
                           "grid_y", "work", "state"}));
  cudaStream_t s = axi::as_stream(stream);
  dim3 g1(axi::ceil_div(nz, 128), nr);
  const int n0 = 2 * nr, n1 = nz;
  const LsqWork w = lsq_work(work, (long long)n0 * n1);
  if (cudaMemsetAsync(w.hdr, 0, sizeof(LsqHeader), s) != cudaSuccess)
    return axi::launch_status(what);
  lsq_prepare_kernel<false><<<g1, 128, 0, s>>>(inside_solid, ball_phi, eta1, eta2,
                                               ball_phi_double, eta1_double, eta2_double,
                                               current_flag, target_flag, extrap_zone, nr, nz,
                                               w.hdr, w.list);
  issue_fused_sweeps(current_flag, target_flag, eta1_double, eta2_double, grid_x, grid_y, n0, n1,
                     max_sweeps, w.hdr, w.list, w.front, s, state, eta1, eta2);
  return axi::launch_status(what);
}
