// FP64 products on the tensor cores by integer slicing: kernels, host helpers
// and the C entries of the standalone spectral transform (see sliced_gemm.cuh).
#include <cuda_fp16.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "sliced_gemm.cuh"

namespace axi_sl {
namespace {

using axi_tma::mbar_expect_tx;
using axi_tma::mbar_init;
using axi_tma::mbar_wait;
using axi_tma::smem_u32;

// ---------------------------------------------------------------------------
// Slicing. One block per 8 rows: the largest exponent of each row, then each
// thread turns 8 consecutive K elements of one row into nine 16-byte pieces
// (one per digit plane). Lanes 0 .. 7 of a warp hold the 8 rows of one core
// matrix, so each plane store of a warp is four full 128-byte lines. All
// arithmetic is on integers (FP64 instructions run at 1/64 of their rate).
// ---------------------------------------------------------------------------
constexpr int SL_THREADS = 256;

// sum of 64 * 2^(7 j): makes every digit non-negative
constexpr unsigned long long DIGIT_BIAS = [] {
  unsigned long long b = 0;
  for (int j = 0; j < DIGITS; ++j) b += 64ull << (BITS * j);
  return b;
}();

// x 2^62 / 2^(emax + 1 - bias) as a signed integer plus DIGIT_BIAS; emax: the
// row's largest biased exponent (at least 1).
__device__ __forceinline__ unsigned long long biased_fixed(double x, int emax) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int e = (int)(b >> 52) & 0x7ff;
  unsigned long long m = b & 0xfffffffffffffull;
  if (e) m |= 1ull << 52;
  const int s = emax - (e ? e : 1) - 9;  // right shift; at least -9
  if (s <= 0)
    m <<= -s;
  else
    m = s > 54 ? 0ull : ((m >> (s - 1)) + 1) >> 1;  // rounded to nearest
  return (b >> 63) ? DIGIT_BIAS - m : DIGIT_BIAS + m;
}

template <bool VEC>
__device__ __forceinline__ void load8(const double* p, long long ks, int n, double (&v)[8]) {
  if (VEC && n >= 8) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double2 t = *reinterpret_cast<const double2*>(p + 2 * q);
      v[2 * q] = t.x;
      v[2 * q + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = q < n ? p[q * ks] : 0.0;
  }
}

template <bool VEC>
__device__ __forceinline__ void slice_rows(const SliceJob& j, const double* src, long long rs,
                                           int group, int* s_max) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = lane & 7;
  const int row = group * 8 + r;
  const int K = j.K, nk = (K + BK - 1) / BK;
  const bool live = row < j.rows;
  const double* p = src + (long long)row * rs;
  const long long ks = j.ks;
  // pass 1: largest biased exponent of each row
  int em = 0;
  for (int k = (warp * 4 + (lane >> 3)) * 8; k < K; k += SL_THREADS) {
    double v[8];
    load8<VEC>(p + k * ks, ks, live ? min(8, K - k) : 0, v);
#pragma unroll
    for (int q = 0; q < 8; ++q)
      em = max(em, (int)((unsigned long long)__double_as_longlong(v[q]) >> 52) & 0x7ff);
  }
  if (threadIdx.x < 8) s_max[threadIdx.x] = 1;
  __syncthreads();
  atomicMax(&s_max[r], em);
  __syncthreads();
  em = s_max[r];
  const bool finite = em != 0x7ff;
  if (warp == 0 && lane < 8) j.exps[row] = finite ? em - 1022 : EXP_NONFINITE;
  // pass 2: the digits
  const bool is_a = j.kind == KIND_A;
  const int br = is_a ? BM : BN;                // rows per block of the layout
  const int stage = is_a ? A_STAGE : B_STAGE;   // bytes per (row block, K step)
  // A: planes of [2 K halves][16 row groups], B: [2 K halves][planes][4 row groups]
  const int plane_stride = is_a ? BM * BK * 2 : BN / 8 * 128;
  const int half_stride = is_a ? BM / 8 * 128 : DIGITS * BN / 8 * 128;
  uint8_t* dst = j.planes + (size_t)(row / br) * nk * stage + (row % br) / 8 * 128 + r * 16;
  for (int k = (warp * 4 + (lane >> 3)) * 8; k < nk * BK; k += SL_THREADS) {
    double v[8];
    load8<VEC>(p + k * ks, ks, live && finite ? min(8, K - k) : 0, v);
    unsigned long long f[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) f[q] = biased_fixed(v[q], em);
    uint8_t* d = dst + (size_t)(k / BK) * stage + ((k / 8) & 1) * half_stride;
#pragma unroll
    for (int i = 0; i < DIGITS; ++i) {
      const int sh = BITS * (DIGITS - 1 - i);
      uint32_t w[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t u0 = (uint32_t)(f[2 * q] >> sh), u1 = (uint32_t)(f[2 * q + 1] >> sh);
        if (i > 0) {
          u0 &= 127u;
          u1 &= 127u;
        }
        // half(1024 + u) has the bits 0x6400 + u; subtract 1024 + 64
        const uint32_t h = 0x64006400u + u0 + (u1 << 16);
        const __half2 x = __hsub2(*reinterpret_cast<const __half2*>(&h),
                                  __half2half2(__ushort_as_half(0x6440)));
        w[q] = *reinterpret_cast<const uint32_t*>(&x);
      }
      *reinterpret_cast<uint4*>(d + i * plane_stride) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

__global__ void __launch_bounds__(SL_THREADS)
    slice_kernel(const SliceJob* __restrict__ jobs, const int4* __restrict__ items,
                 const double* src_override, long long rs_override) {
  __shared__ int s_max[8];
  const int4 it = items[blockIdx.x];
  const SliceJob& j = jobs[it.x];
  const double* src = src_override ? src_override : j.src;
  const long long rs = src_override ? rs_override : j.rs;
  // 16-byte loads where every row starts on 16 bytes and K runs contiguously
  const bool vec = j.ks == 1 && (rs & 1) == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0;
  if (vec)
    slice_rows<true>(j, src, rs, it.y, s_max);
  else
    slice_rows<false>(j, src, rs, it.y, s_max);
}

// ---------------------------------------------------------------------------
// Product.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// D (TMEM, FP32) (+)= A (smem, FP16) * B (smem, FP16)
__device__ __forceinline__ void umma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
      : "memory");
}
// bulk copy of contiguous bytes (16-byte aligned, a multiple of 16)
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes,
                                          uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

// Unswizzled K-major operand: core matrices of 8 rows x 16 bytes (128
// contiguous bytes); `lead` bytes between the two K halves of a 16-element
// step, 128 bytes between groups of 8 rows.
__device__ __forceinline__ uint64_t operand_desc(uint32_t saddr, uint32_t lead) {
  return static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4) |
         (static_cast<uint64_t>(lead >> 4) << 16) | (static_cast<uint64_t>(128 >> 4) << 32) |
         (static_cast<uint64_t>(1) << 46);
}
// D = F32, A = B = F16, both K-major, M = 128
__device__ __forceinline__ constexpr uint32_t idesc_f16(int n) {
  return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(BM >> 4) << 24);
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                 "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// The two accumulator sets overlap by two groups of 32 columns (2 x 288 of 512
// columns): set 0 starts at column 0, set 1 at column 224. The columns shared
// are groups 7, 8 of set 0 and groups 0, 1 of set 1.
constexpr int SET1 = 512 - DIGITS * BN;
constexpr int SHARED_GROUPS = (2 * DIGITS * BN - 512) / BN;
static_assert(SHARED_GROUPS == 2 && SET1 % BN == 0, "accumulator sets");

// Sum of the accumulators of one output element as hi 2^28 + lo: groups
// 0 .. 4 go to hi, 5 .. 8 to lo (weights 2^(7 (8 - d)) relative to the last).
template <int G>
__device__ __forceinline__ void add_group(uint32_t bits, long long& hi, long long& lo) {
  const int s = __float2int_rn(__uint_as_float(bits));
  if constexpr (G <= 4)
    hi += (long long)s * (1 << (BITS * (4 - G)));
  else
    lo += (long long)s * (1 << (BITS * (8 - G)));
}

template <int G>
__device__ __forceinline__ void add_groups8(uint32_t (&r)[8], long long* hi, long long* lo) {
#pragma unroll
  for (int q = 0; q < 8; ++q) add_group<G>(r[q], hi[q], lo[q]);
}

// Groups FIRST .. FIRST + COUNT - 1 of this warp's 16 columns into hi, lo.
template <int FIRST, int COUNT>
__device__ __forceinline__ void drain_groups(uint32_t taddr, long long (&hi)[16],
                                             long long (&lo)[16]) {
  if constexpr (COUNT > 0) {
    constexpr int N = COUNT >= 2 ? 2 : COUNT;  // up to 32 registers in flight
    uint32_t r[N][2][8];
#pragma unroll
    for (int g = 0; g < N; ++g)
#pragma unroll
      for (int h = 0; h < 2; ++h) tmem_ld8(taddr + (FIRST + g) * BN + 8 * h, r[g][h]);
    tmem_wait_ld();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      add_groups8<FIRST>(r[0][h], hi + 8 * h, lo + 8 * h);
      if constexpr (N > 1) add_groups8<FIRST + 1>(r[1][h], hi + 8 * h, lo + 8 * h);
    }
    drain_groups<FIRST + N, COUNT - N>(taddr, hi, lo);
  }
}

// (hi 2^28 + lo) 2^e rounded once to FP64, with integer instructions.
__device__ __forceinline__ double assemble(long long hi, long long lo, int e) {
  // 128-bit sum: (w1, w0)
  unsigned long long w0 = (unsigned long long)hi << 28;
  long long w1 = hi >> 36;
  const unsigned long long lo_u = (unsigned long long)lo;
  w0 += lo_u;
  w1 += (lo >> 63) + (w0 < lo_u ? 1 : 0);
  const unsigned long long sign = (unsigned long long)w1 & 0x8000000000000000ull;
  if (w1 < 0) {
    w0 = ~w0 + 1;
    w1 = ~w1 + (w0 == 0 ? 1 : 0);
  }
  if ((w0 | (unsigned long long)w1) == 0) return 0.0;
  // leading 64 bits m (top bit set), value = m 2^p
  int p;
  unsigned long long m, rest;
  if (w1 != 0) {
    const int n = __clzll(w1);
    m = n == 0 ? (unsigned long long)w1
               : ((unsigned long long)w1 << n) | (w0 >> (64 - n));
    rest = n == 0 ? w0 : w0 << n;
    p = 64 - n;
  } else {
    const int n = __clzll((long long)w0);
    m = w0 << n;
    rest = 0;
    p = -n;
  }
  // round to 53 bits, ties to even
  unsigned long long r = m >> 11;
  const uint32_t tail = (uint32_t)m & 0x7ffu;
  r += (tail > 0x400u || (tail == 0x400u && (rest != 0 || (r & 1)))) ? 1 : 0;
  const int be = 1023 + 63 + p + e;  // biased exponent of m's top bit
  if (be >= 1 && be <= 2045)
    return __longlong_as_double((long long)(sign | (((unsigned long long)(be - 1) << 52) + r)));
  const double v = scalbn((double)r, be - 1075);  // overflow, or a subnormal result
  return sign ? -v : v;
}

// Persistent, warp-specialised: warp 0 copies stages, warp 1 issues MMAs,
// warps 2 .. 9 (two per TMEM lane quarter, 16 columns each) drain an
// accumulator set while the MMAs fill the other. A unit of work is one tile
// and up to 512 of its K; the integer sums run on over the units of a tile.
__global__ void __launch_bounds__(THREADS, 1)
    sliced_gemm_kernel(const GemmJob* __restrict__ jobs, const int4* __restrict__ tiles,
                       int n_tiles, int* __restrict__ err, double* c_override, int ldc_override) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) &
                                             ~static_cast<uintptr_t>(127));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + NSTAGE * STAGE_BYTES);
  // full[NSTAGE], empty[NSTAGE], acc_full, acc_shared (drained), quiet
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * NSTAGE + 3);
  int* progress = reinterpret_cast<int*>(tmem_slot + 1);  // [0] loads issued, [1] consumed
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + NSTAGE);
  const uint32_t acc_full = smem_u32(bars + 2 * NSTAGE);
  const uint32_t acc_shared = smem_u32(bars + 2 * NSTAGE + 1);
  const uint32_t quiet = smem_u32(bars + 2 * NSTAGE + 2);

  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_shared, EPI_WARPS);
    mbar_init(quiet, 1);
    progress[0] = 0;
    progress[1] = 0;
    axi_tma::fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int g = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
        const int4 tr = tiles[t];  // job, row block of A, row block of B, K steps
        const GemmJob& job = jobs[tr.x];
        const int nk = tr.w;
        const uint8_t* a = job.a + (size_t)tr.y * nk * A_STAGE;
        const uint8_t* b = job.b + (size_t)tr.z * nk * B_STAGE;
        for (int kb = 0; kb < nk; ++kb, ++g) {
          const int s = g % NSTAGE, use = g / NSTAGE;
          if (use > 0 && !mbar_wait(empty0 + 8 * s, (use - 1) & 1, err, ERR_PRODUCER)) {
            ok = false;
            break;
          }
          const uint32_t st = smem_u32(smem + s * STAGE_BYTES);
          const uint32_t fb = full0 + 8 * s;
          mbar_expect_tx(fb, STAGE_BYTES);
          bulk_load(st, a + (size_t)kb * A_STAGE, A_STAGE, fb);
          bulk_load(st + A_STAGE, b + (size_t)kb * B_STAGE, B_STAGE, fb);
        }
      }
      progress[0] = g;
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      int g = 0, u = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
        const int nk = tiles[t].w;
        for (int k0 = 0; k0 < nk && ok; k0 += CHUNK, ++u) {
          // the set before the last is drained, and of the last the shared columns
          if (u > 0 && !mbar_wait(acc_shared, (u - 1) & 1, err, ERR_MMA)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d = tmem + (u & 1) * SET1;
          const int k1 = min(nk, k0 + CHUNK);
          for (int kb = k0; kb < k1; ++kb, ++g) {
            const int s = g % NSTAGE, use = g / NSTAGE;
            if (!mbar_wait(full0 + 8 * s, use & 1, err, ERR_MMA)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t st = smem_u32(smem + s * STAGE_BYTES);
            const uint64_t a = operand_desc(st, BM / 8 * 128);
            const uint64_t b = operand_desc(st + A_STAGE, DIGITS * BN / 8 * 128);
            // plane 0 of A against all nine planes of B, in two halves (N <= 256):
            // it also starts every accumulator of the set
            constexpr int H = DIGITS * BN / 2;
            const uint32_t first = kb == k0 ? 0u : 1u;
            umma_f16(d, a, b, idesc_f16(H), first);
            umma_f16(d + H, a, b + (H / 8 * 128 >> 4), idesc_f16(H), first);
#pragma unroll
            for (int i = 1; i < DIGITS; ++i)
              umma_f16(d + i * BN, a + (i * BM * BK * 2 >> 4), b, idesc_f16((DIGITS - i) * BN), 1u);
            umma_commit(empty0 + 8 * s);
          }
          if (ok) umma_commit(acc_full);
        }
      }
      progress[1] = g;
      umma_commit(quiet);
      mbar_wait(quiet, 0, err, ERR_MMA);
    }
    __syncwarp();
  } else {
    const int q = warp & 3;          // TMEM lane quarter
    const int half = (warp - 2) >> 2;  // columns 16 half .. 16 half + 15
    const uint32_t lane_base = static_cast<uint32_t>(32 * q) << 16;
    int u = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
      const int4 tr = tiles[t];
      const GemmJob& job = jobs[tr.x];
      const int M = job.M, N = job.N;
      double* const c = c_override ? c_override : job.c;
      const long long ldc = c_override ? ldc_override : job.ldc;
      const double* const scale = job.scale;
      const int row = tr.y * BM + 32 * q + lane;
      const int col0 = tr.z * BN + 16 * half;
      const int ea = job.ea[row];
      const int* eb = job.eb + col0;
      const int nk = tr.w;
      long long hi[16], lo[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) hi[j] = lo[j] = 0;
      for (int k0 = 0; k0 < nk; k0 += CHUNK, ++u) {
        ok = __all_sync(0xffffffffu, mbar_wait(acc_full, u & 1, err, ERR_EPILOGUE));
        if (!ok) break;
        tc_fence_after();
        const uint32_t ta = tmem + lane_base + (u & 1) * SET1 + 16 * half;
        // the columns that the next unit also uses come first
        if (u & 1) {
          drain_groups<0, SHARED_GROUPS>(ta, hi, lo);
        } else {
          drain_groups<DIGITS - SHARED_GROUPS, SHARED_GROUPS>(ta, hi, lo);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acc_shared) : "memory");
        if (u & 1) {
          drain_groups<SHARED_GROUPS, DIGITS - SHARED_GROUPS>(ta, hi, lo);
        } else {
          drain_groups<0, DIGITS - SHARED_GROUPS>(ta, hi, lo);
        }
      }
      if (!ok) break;
      if (row < M) {
        double* const cr = c + row * ldc + col0;
        const double* const sr = scale ? scale + (long long)row * N + col0 : nullptr;
        const int n = min(16, N - col0);
        const bool vec = n == 16 && (reinterpret_cast<uintptr_t>(cr) & 15) == 0;
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          double v[2];
#pragma unroll
          for (int w = 0; w < 2; ++w) {
            const int e = eb[j + w];
            // ea + eb - 12 - 7 * 8; a row or column that is not finite gives NaN
            v[w] = assemble(hi[j + w], lo[j + w], ea + e - 68);
            if (ea == EXP_NONFINITE || e == EXP_NONFINITE)
              v[w] = __longlong_as_double(0x7ff8000000000000ll);
            if (sr && j + w < n) v[w] *= sr[j + w];
          }
          if (vec) {
            *reinterpret_cast<double2*>(cr + j) = make_double2(v[0], v[1]);
          } else {
            if (j < n) cr[j] = v[0];
            if (j + 1 < n) cr[j + 1] = v[1];
          }
        }
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && progress[1] < progress[0]) {
    // a failure left copies in flight: wait for them (bounded) before exiting
    for (int g = progress[1]; g < progress[0]; ++g)
      if (!axi_tma::mbar_wait_drain(full0 + 8 * (g % NSTAGE), (g / NSTAGE) & 1))
        atomicCAS(err, 0, ERR_DRAIN);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem, 512);
}

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

}  // namespace

void append_slice_items(std::vector<int4>& items, int job, int rows, int kind) {
  for (int g = 0; g < slice_items(rows, kind); ++g) items.push_back(make_int4(job, g, 0, 0));
}

void append_gemm_tiles(std::vector<int4>& tiles, int job, int M, int N, int K) {
  for (int m = 0; m < (M + BM - 1) / BM; ++m)
    for (int n = 0; n < (N + BN - 1) / BN; ++n) tiles.push_back(make_int4(job, m, n, k_steps(K)));
}

void order_tiles(std::vector<int4>& tiles) {
  std::stable_sort(tiles.begin(), tiles.end(),
                   [](const int4& a, const int4& b) { return a.w > b.w; });
}

int launch_slice(const SliceJob* jobs_dev, const int4* items_dev, int n_items, cudaStream_t s,
                 const double* src, long long rs) {
  if (n_items <= 0) return AXI_OK;
  slice_kernel<<<n_items, SL_THREADS, 0, s>>>(jobs_dev, items_dev, src, rs);
  return axi::launch_status("slice");
}

int launch_gemm(const GemmJob* jobs_dev, const int4* tiles_dev, int n_tiles, int* err_dev,
                cudaStream_t s, double* c, int ldc) {
  static std::once_flag once;
  static cudaError_t attr_status = cudaSuccess;
  std::call_once(once, [] {
    attr_status = cudaFuncSetAttribute(sliced_gemm_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
  });
  if (attr_status != cudaSuccess) {
    axi::set_error("sliced GEMM: cannot reserve %d bytes of shared memory", SMEM_BYTES);
    return AXI_ERR_CUDA;
  }
  if (n_tiles <= 0) return AXI_OK;
  const int sms = axi::sm_count();
  sliced_gemm_kernel<<<n_tiles < sms ? n_tiles : sms, THREADS, SMEM_BYTES, s>>>(
      jobs_dev, tiles_dev, n_tiles, err_dev, c, ldc);
  return axi::launch_status("sliced_gemm");
}

size_t spectral_slice_bytes(int nr, int nz) {
  return std::max(slice_bytes(nr, nz, KIND_B), slice_bytes(nz, nr, KIND_B));
}

void spectral_jobs(int nr, int nz, const double* in, long long ld_in, double* out, int ld_out,
                   double* work, void* slices, const void* const basis[4], const double* inv_eig,
                   SliceJob sl[4], GemmJob gm[4]) {
  double* x = work;
  double* y = work + (size_t)nr * nz;
  sl[0] = slice_job(in, ld_in, 1, nr, nz, KIND_B, slices);
  sl[1] = slice_job(x, nr, 1, nz, nr, KIND_B, slices);
  sl[2] = slice_job(y, nz, 1, nr, nz, KIND_B, slices);
  sl[3] = slice_job(x, nr, 1, nz, nr, KIND_B, slices);
  double* c[4] = {x, y, x, out};
  const int ldc[4] = {nr, nz, nr, ld_out};
  for (int st = 0; st < 4; ++st) {
    const int M = st % 2 == 0 ? nz : nr, N = st % 2 == 0 ? nr : nz, K = M;
    GemmJob& g = gm[st];
    g.a = static_cast<const uint8_t*>(basis[st]);
    g.ea = reinterpret_cast<const int*>(g.a + plane_bytes(M, K, KIND_A));
    g.b = sl[st].planes;
    g.eb = sl[st].exps;
    g.c = c[st];
    g.scale = st == 1 ? inv_eig : nullptr;
    g.M = M;
    g.N = N;
    g.ldc = ldc[st];
    g.nk = k_steps(K);
  }
}

}  // namespace axi_sl

// ---------------------------------------------------------------------------
// C entries.
// ---------------------------------------------------------------------------
namespace {

using namespace axi_sl;

// Plan of the standalone transform: [SliceJob x 4][GemmJob x 4][slice items x 4]
// [tiles x 4][error word][sliced bases x 4][sliced field][X, Y]
struct TransformLayout {
  size_t sjobs, gjobs, items[4], tiles[4], err, basis[4], slices, work, total;
  int n_items[4], n_tiles[4];
};

TransformLayout transform_layout(int nr, int nz) {
  TransformLayout L;
  size_t o = 0;
  L.sjobs = o; o = align_up(o + 4 * sizeof(SliceJob), 256);
  L.gjobs = o; o = align_up(o + 4 * sizeof(GemmJob), 256);
  for (int st = 0; st < 4; ++st) {
    const int M = st % 2 == 0 ? nz : nr, N = st % 2 == 0 ? nr : nz;
    L.n_items[st] = slice_items(N, KIND_B);
    L.n_tiles[st] = gemm_tiles(M, N);
    L.items[st] = o; o = align_up(o + L.n_items[st] * sizeof(int4), 256);
    L.tiles[st] = o; o = align_up(o + L.n_tiles[st] * sizeof(int4), 256);
  }
  L.err = o; o = align_up(o + 16, 256);
  for (int st = 0; st < 4; ++st) {
    const int M = st % 2 == 0 ? nz : nr;
    L.basis[st] = o; o = align_up(o + slice_bytes(M, M, KIND_A), 256);
  }
  L.slices = o; o = align_up(o + spectral_slice_bytes(nr, nz), 256);
  L.work = o; o = align_up(o + (size_t)2 * nr * nz * sizeof(double), 256);
  L.total = o;
  return L;
}

// Slices one matrix (blocking: the job record is copied from this stack).
int slice_now(const SliceJob& j, cudaStream_t s) {
  std::vector<int4> items;
  append_slice_items(items, 0, j.rows, j.kind);
  const size_t off = align_up(sizeof(SliceJob), 256);
  char* d = nullptr;
  if (cudaMallocAsync(reinterpret_cast<void**>(&d), off + items.size() * sizeof(int4), s) !=
      cudaSuccess)
    return axi::launch_status("slice");
  int st = AXI_OK;
  if (cudaMemcpyAsync(d, &j, sizeof(j), cudaMemcpyHostToDevice, s) != cudaSuccess ||
      cudaMemcpyAsync(d + off, items.data(), items.size() * sizeof(int4), cudaMemcpyHostToDevice,
                      s) != cudaSuccess)
    st = axi::launch_status("slice");
  if (st == AXI_OK)
    st = launch_slice(reinterpret_cast<const SliceJob*>(d), reinterpret_cast<const int4*>(d + off),
                      (int)items.size(), s);
  cudaFreeAsync(d, s);
  if (cudaStreamSynchronize(s) != cudaSuccess && st == AXI_OK) st = axi::launch_status("slice");
  return st;
}

int check_shape(const char* what, int a, int b) {
  if (a <= 0 || b <= 0 || a > (1 << 20) || b > (1 << 20)) {
    axi::set_error("%s: invalid shape %d x %d", what, a, b);
    return AXI_ERR_INVALID;
  }
  return AXI_OK;
}

}  // namespace

extern "C" int64_t axi_sliced_operand_bytes(int rows, int K) {
  if (rows <= 0 || K <= 0) return 0;
  return (int64_t)align_up(slice_bytes(rows, K, KIND_A), 256);
}

extern "C" int axi_slice_operand_f64(void* dst, const double* src, int64_t row_stride,
                                     int64_t k_stride, int rows, int K, void* stream) {
  axi::clear_error();
  const char* what = "slice_operand";
  AXI_TRY(check_shape(what, rows, K));
  AXI_TRY(axi::check_ptrs(what, {dst, src}, {"dst", "src"}));
  return slice_now(slice_job(src, row_stride, k_stride, rows, K, KIND_A, dst),
                   axi::as_stream(stream));
}

extern "C" int64_t axi_sliced_field_bytes(int nr, int nz) {
  if (nr <= 0 || nz <= 0) return 0;
  return (int64_t)align_up(spectral_slice_bytes(nr, nz), 256);
}

extern "C" int64_t axi_sliced_transform_bytes(int nr, int nz) {
  if (nr <= 0 || nz <= 0) return 0;
  return (int64_t)transform_layout(nr, nz).total;
}

extern "C" int axi_sliced_transform_plan(void* plan, const double* Er_inv_w, const double* EzinvT,
                                         const double* inv_eig, const double* Er,
                                         const double* EzT, int nr, int nz, void* stream) {
  axi::clear_error();
  const char* what = "sliced_transform_plan";
  AXI_TRY(check_shape(what, nr, nz));
  AXI_TRY(axi::check_ptrs(what, {plan, Er_inv_w, EzinvT, inv_eig, Er, EzT},
                          {"plan", "Er_inv_w", "EzinvT", "inv_eig", "Er", "EzT"}));
  cudaStream_t s = axi::as_stream(stream);
  const TransformLayout L = transform_layout(nr, nz);
  char* base = static_cast<char*>(plan);
  // A operands: E_z^-1 and E_z are stored transposed
  const double* src[4] = {EzinvT, Er_inv_w, EzT, Er};
  const void* basis[4];
  for (int st = 0; st < 4; ++st) {
    const int M = st % 2 == 0 ? nz : nr;
    basis[st] = base + L.basis[st];
    const bool transposed = st % 2 == 0;
    AXI_TRY(slice_now(slice_job(src[st], transposed ? 1 : M, transposed ? M : 1, M, M, KIND_A,
                                base + L.basis[st]), s));
  }
  SliceJob sl[4];
  GemmJob gm[4];
  spectral_jobs(nr, nz, nullptr, nz, nullptr, nz, reinterpret_cast<double*>(base + L.work),
                base + L.slices, basis, inv_eig, sl, gm);
  std::vector<char> head(L.err + 16, 0);
  memcpy(&head[L.sjobs], sl, sizeof(sl));
  memcpy(&head[L.gjobs], gm, sizeof(gm));
  for (int st = 0; st < 4; ++st) {
    const int M = st % 2 == 0 ? nz : nr, N = st % 2 == 0 ? nr : nz;
    std::vector<int4> items, tiles;
    append_slice_items(items, st, N, KIND_B);
    append_gemm_tiles(tiles, st, M, N, M);
    memcpy(&head[L.items[st]], items.data(), items.size() * sizeof(int4));
    memcpy(&head[L.tiles[st]], tiles.data(), tiles.size() * sizeof(int4));
  }
  if (cudaMemcpyAsync(plan, head.data(), head.size(), cudaMemcpyHostToDevice, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return axi::launch_status(what);
  return AXI_OK;
}

extern "C" int axi_sliced_transform_run(const void* plan, double* out, int ld_out,
                                        const double* in, int ld_in, int nr, int nz,
                                        void* stream) {
  axi::clear_error();
  const char* what = "sliced_transform_run";
  AXI_TRY(check_shape(what, nr, nz));
  AXI_TRY(axi::check_ptrs(what, {plan, out, in}, {"plan", "out", "in"}));
  if (ld_in < nz || ld_out < nz) {
    axi::set_error("%s: row strides %d, %d below nz = %d", what, ld_in, ld_out, nz);
    return AXI_ERR_INVALID;
  }
  cudaStream_t s = axi::as_stream(stream);
  const TransformLayout L = transform_layout(nr, nz);
  char* base = static_cast<char*>(const_cast<void*>(plan));
  const SliceJob* sj = reinterpret_cast<const SliceJob*>(base + L.sjobs);
  const GemmJob* gj = reinterpret_cast<const GemmJob*>(base + L.gjobs);
  int* err = reinterpret_cast<int*>(base + L.err);
  for (int st = 0; st < 4; ++st) {
    AXI_TRY(launch_slice(sj, reinterpret_cast<const int4*>(base + L.items[st]), L.n_items[st], s,
                         st == 0 ? in : nullptr, ld_in));
    AXI_TRY(launch_gemm(gj, reinterpret_cast<const int4*>(base + L.tiles[st]), L.n_tiles[st], err,
                        s, st == 3 ? out : nullptr, ld_out));
  }
  return AXI_OK;
}

extern "C" int axi_sliced_transform_status(const void* plan, int nr, int nz, int* error,
                                           void* stream) {
  axi::clear_error();
  const char* what = "sliced_transform_status";
  AXI_TRY(check_shape(what, nr, nz));
  AXI_TRY(axi::check_ptrs(what, {plan, error}, {"plan", "error"}));
  cudaStream_t s = axi::as_stream(stream);
  const char* base = static_cast<const char*>(plan);
  if (cudaMemcpyAsync(error, base + transform_layout(nr, nz).err, sizeof(int),
                      cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return axi::launch_status(what);
  return AXI_OK;
}

// ---------------------------------------------------------------------------
// C (M, N) = A (M, K) B (N, K)^T .* S, both operands sliced per call.
// ---------------------------------------------------------------------------
namespace {

struct GemmLayout {
  size_t sjobs, gjob, items, tiles, err, a, b, total;
  int n_items, n_tiles;
};

GemmLayout gemm_layout(int M, int N, int K) {
  GemmLayout L;
  size_t o = 0;
  L.sjobs = o; o = align_up(o + 2 * sizeof(SliceJob), 256);
  L.gjob = o; o = align_up(o + sizeof(GemmJob), 256);
  L.n_items = slice_items(M, KIND_A) + slice_items(N, KIND_B);
  L.n_tiles = gemm_tiles(M, N);
  L.items = o; o = align_up(o + L.n_items * sizeof(int4), 256);
  L.tiles = o; o = align_up(o + L.n_tiles * sizeof(int4), 256);
  L.err = o; o = align_up(o + 16, 256);
  L.a = o; o = align_up(o + slice_bytes(M, K, KIND_A), 256);
  L.b = o; o = align_up(o + slice_bytes(N, K, KIND_B), 256);
  L.total = o;
  return L;
}

}  // namespace

extern "C" int64_t axi_sliced_gemm_work_bytes(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  return (int64_t)gemm_layout(M, N, K).total;
}

extern "C" int axi_sliced_gemm_f64(double* C, const double* A, const double* B, const double* S,
                                   int M, int N, int K, void* work, void* stream) {
  axi::clear_error();
  const char* what = "sliced_gemm";
  AXI_TRY(check_shape(what, M, N));
  AXI_TRY(check_shape(what, K, K));
  AXI_TRY(axi::check_ptrs(what, {C, A, B, work}, {"C", "A", "B", "work"}));
  cudaStream_t s = axi::as_stream(stream);
  const GemmLayout L = gemm_layout(M, N, K);
  char* base = static_cast<char*>(work);
  SliceJob sl[2] = {slice_job(A, K, 1, M, K, KIND_A, base + L.a),
                    slice_job(B, K, 1, N, K, KIND_B, base + L.b)};
  GemmJob g;
  g.a = sl[0].planes; g.ea = sl[0].exps; g.b = sl[1].planes; g.eb = sl[1].exps;
  g.c = C; g.scale = S; g.M = M; g.N = N; g.ldc = N; g.nk = k_steps(K);
  std::vector<int4> items, tiles;
  append_slice_items(items, 0, M, KIND_A);
  append_slice_items(items, 1, N, KIND_B);
  append_gemm_tiles(tiles, 0, M, N, K);
  std::vector<char> head(L.err + 16, 0);
  memcpy(&head[L.sjobs], sl, sizeof(sl));
  memcpy(&head[L.gjob], &g, sizeof(g));
  memcpy(&head[L.items], items.data(), items.size() * sizeof(int4));
  memcpy(&head[L.tiles], tiles.data(), tiles.size() * sizeof(int4));
  if (cudaMemcpyAsync(work, head.data(), head.size(), cudaMemcpyHostToDevice, s) != cudaSuccess)
    return axi::launch_status(what);
  AXI_TRY(launch_slice(reinterpret_cast<const SliceJob*>(base + L.sjobs),
                       reinterpret_cast<const int4*>(base + L.items), L.n_items, s));
  int* err = reinterpret_cast<int*>(base + L.err);
  AXI_TRY(launch_gemm(reinterpret_cast<const GemmJob*>(base + L.gjob),
                      reinterpret_cast<const int4*>(base + L.tiles), L.n_tiles, err, s));
  int code = 0;
  if (cudaMemcpyAsync(&code, err, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return axi::launch_status(what);
  if (code) {
    axi::set_error("%s: a wait on the tensor-core pipeline ran out (code %d)", what, code);
    return AXI_ERR_CUDA;
  }
  return AXI_OK;
}
