// FP64 products on the tensor cores by integer slicing: kernels, host helpers
// and the C entries of the standalone spectral transform (see sliced_gemm.cuh).
#include <cuda_fp16.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "sliced_gemm.cuh"

namespace axi_sl {
namespace {

using axi_tma::elect_one;
using axi_tma::mbar_expect_tx;
using axi_tma::mbar_init;
using axi_tma::mbar_wait;
using axi_tma::smem_u32;

// ---------------------------------------------------------------------------
// Slicing. A block takes 8 rows (or a share of their K): the largest exponent of
// each row, then each thread turns 8 consecutive K elements of one row into
// eight 16-byte pieces (one per digit plane). Lanes 0 .. 7 of a warp hold the 8
// rows of one core matrix, so each plane store of a warp is four full 128-byte
// lines. All arithmetic is on integers (FP64 instructions run at 1/64 of their
// rate).
// ---------------------------------------------------------------------------
constexpr int SL_THREADS = 256;

// 128 in every byte: makes every digit non-negative
constexpr unsigned long long DIGIT_BIAS = 0x8080808080808080ull;

// Biased exponent of x, as the row maxima count it: 0 for zeros and subnormal
// numbers, NOT_FINITE for infinities and NaN.
__device__ __forceinline__ int exponent_of(double x) {
  const int e = (int)((unsigned long long)__double_as_longlong(x) >> 52) & 0x7ff;
  return e == 0x7ff ? NOT_FINITE : e;
}

// x 2^shift 2^62 / 2^(emax + 1 - bias) as a signed integer plus DIGIT_BIAS,
// whose bytes are the digits plus 128; emax: the row's largest biased exponent
// (at least 1), shifts included.
__device__ __forceinline__ unsigned long long biased_fixed(double x, int emax, int shift) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int e = (int)(b >> 52) & 0x7ff;
  unsigned long long m = b & 0xfffffffffffffull;
  if (e) m |= 1ull << 52;
  const int s = emax - (e ? e : 1) - shift - 9;  // right shift; at least -9 (m = 0: any)
  if (s <= 0)
    m <<= min(-s, 9);
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

// Powers of two that balance eight neighbouring K elements of a radial product
// (spectral_jobs): the left operand's are multiplied by those of the field's
// columns, the field's own divided by them.
template <int BAL>
__device__ __forceinline__ void load_shifts(const int* col_exps, int k, int K, int (&c)[8]) {
#pragma unroll
  for (int q = 0; q < 8; ++q) c[q] = 0;
  if (BAL == 0 || k >= K) return;
  const int4 a = *reinterpret_cast<const int4*>(col_exps + k);
  const int4 b = *reinterpret_cast<const int4*>(col_exps + k + 4);
  const int e[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int q = 0; q < 8; ++q) c[q] = BAL > 0 ? max(e[q], 1) : BALANCE_BIAS - max(e[q], 1);
}

// BAL: 0 as it is, 1 the left and -1 the right operand of a balanced product.
template <bool VEC, int BAL>
__device__ __forceinline__ void slice_rows(const SliceJob& j, const double* src, long long rs,
                                           int group, int part, int parts, int* s_max) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r = lane & 7;
  const int row = group * 8 + r;
  const int K = j.K, nk = (K + BK - 1) / BK;
  const bool live = row < j.rows;
  const double* p = src + (long long)row * rs;
  const long long ks = j.ks;
  const int k_lane = (warp * 4 + (lane >> 3)) * 8;
  // pass 1: largest biased exponent of each row
  int em = 0;
  if (j.have_exps) {
    em = live ? j.exps[row] : 0;
  } else {
    for (int k = k_lane; k < K; k += SL_THREADS) {
      double v[8];
      int c[8];
      load8<VEC>(p + k * ks, ks, live ? min(8, K - k) : 0, v);
      load_shifts<BAL>(j.col_exps, k, K, c);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int e = exponent_of(v[q]);
        if (BAL == 0)
          em = max(em, e);
        else if ((__double_as_longlong(v[q]) << 1) != 0)
          em = max(em, e == NOT_FINITE ? e : max(e, 1) + c[q]);
      }
    }
    if (threadIdx.x < 8) s_max[threadIdx.x] = 0;
    __syncthreads();
    atomicMax(&s_max[r], em);
    __syncthreads();
    em = s_max[r];
    if (part == 0 && warp == 0 && lane < 8) j.exps[row] = em;
  }
  const bool finite = em != NOT_FINITE;
  em = max(em, 1);
  // pass 2: the digits
  const int br = j.block;                       // rows per block of the layout
  const bool is_a = br == BM;
  const int stage = DIGITS * br * BK * 2;       // bytes per (row block, K step)
  // A: planes of [2 K halves][row groups], B: [2 K halves][planes][row groups]
  const int plane_stride = is_a ? BM * BK * 2 : br / 8 * 128;
  const int half_stride = is_a ? BM / 8 * 128 : DIGITS * br / 8 * 128;
  uint8_t* dst = j.planes + (size_t)(row / br) * nk * stage + (row % br) / 8 * 128 + r * 16;
  for (int k = part * SL_THREADS + k_lane; k < nk * BK; k += parts * SL_THREADS) {
    double v[8];
    load8<VEC>(p + k * ks, ks, live && finite ? min(8, K - k) : 0, v);
    unsigned long long f[8];
    int c[8];
    load_shifts<BAL>(j.col_exps, k, K, c);
#pragma unroll
    for (int q = 0; q < 8; ++q) f[q] = biased_fixed(v[q], em, c[q]);
    uint8_t* d = dst + (size_t)(k / BK) * stage + ((k / 8) & 1) * half_stride;
#pragma unroll
    for (int i = 0; i < DIGITS; ++i) {
      // digit i is byte 7 - i
      uint32_t w[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t w0 = (uint32_t)(f[2 * q] >> (i < 4 ? 32 : 0));
        const uint32_t w1 = (uint32_t)(f[2 * q + 1] >> (i < 4 ? 32 : 0));
        const uint32_t byte = 3 - i % 4;
        // half(1024 + u) has the bits 0x6400 + u; subtract 1024 + 128
        const uint32_t h =
            (__byte_perm(w0, w1, byte | byte << 4 | (byte + 4) << 8 | (byte + 4) << 12) &
             0x00ff00ffu) | 0x64006400u;
        const __half2 x = __hsub2(*reinterpret_cast<const __half2*>(&h),
                                  __half2half2(__ushort_as_half(0x6480)));
        w[q] = *reinterpret_cast<const uint32_t*>(&x);
      }
      *reinterpret_cast<uint4*>(d + i * plane_stride) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

__device__ __forceinline__ int pad_rows_dev(int rows, int block) {
  return (rows + block - 1) / block * block;
}

// One item: a group of 8 rows, and share `part` of `parts` of its K.
__device__ __forceinline__ void slice_item(const SliceJob& j, const double* src, long long rs,
                                           int group, int part, int parts) {
  __shared__ int s_max[8];
  // 16-byte loads where every row starts on 16 bytes and K runs contiguously
  const bool vec = j.ks == 1 && (rs & 1) == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0;
  auto slice = [&](auto bal) {
    if (vec)
      slice_rows<true, bal()>(j, src, rs, group, part, parts, s_max);
    else
      slice_rows<false, bal()>(j, src, rs, group, part, parts, s_max);
  };
  if (j.balance == 0)
    slice(std::integral_constant<int, 0>());
  else if (j.balance > 0)
    slice(std::integral_constant<int, 1>());
  else
    slice(std::integral_constant<int, -1>());
}

// items: job, group of 8 rows, share of K, shares. The tables are written and
// synchronised when the plan is made, long before this launch, so that they may
// be read ahead of its dependencies.
__global__ void __launch_bounds__(SL_THREADS)
    slice_kernel(const SliceJob* __restrict__ jobs, const int4* __restrict__ items,
                 const double* src_override, long long rs_override, int* err_begin) {
  const int4 it = items[blockIdx.x];
  const SliceJob& j = jobs[it.x];
  axi::pdl_trigger();
  axi::pdl_wait();
  // a new run: an earlier one's failure goes to the record beside the word
  if (err_begin && blockIdx.x == 0 && threadIdx.x == 0 && err_begin[0] != 0) {
    err_begin[1] = err_begin[0];
    err_begin[0] = 0;
  }
  // what the next product's epilogue accumulates into starts at zero
  for (int q = (it.y * it.w + it.z) * SL_THREADS + threadIdx.x; q < j.n_clear;
       q += (pad_rows_dev(j.rows, j.block) / 8) * it.w * SL_THREADS)
    j.clear[q] = 0;
  slice_item(j, src_override ? src_override : j.src, src_override ? rs_override : j.rs, it.y, it.z,
             it.w);
}

// One matrix, a group of rows per block, without tables.
__global__ void __launch_bounds__(SL_THREADS) slice_matrix_kernel(const SliceJob j) {
  slice_item(j, j.src, j.rs, blockIdx.x, 0, 1);
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

// Sum of the accumulators of one output element as hi 2^32 + lo: groups
// 0 .. 3 go to hi, 4 .. 7 to lo (weights 2^(8 (7 - d)) relative to the last).
template <int G>
__device__ __forceinline__ void add_group(uint32_t bits, long long& hi, long long& lo) {
  const int s = __float2int_rn(__uint_as_float(bits));
  if constexpr (G <= 3)
    hi += (long long)s * (1 << (8 * (3 - G)));
  else
    lo += (long long)s * (1 << (8 * (7 - G)));
}

template <int G>
__device__ __forceinline__ void add_groups8(uint32_t (&r)[8], long long* hi, long long* lo) {
#pragma unroll
  for (int q = 0; q < 8; ++q) add_group<G>(r[q], hi[q], lo[q]);
}

// Groups FIRST .. FIRST + COUNT - 1 of this warp's BN / 2 columns into hi, lo.
template <int BN, int FIRST, int COUNT>
__device__ __forceinline__ void drain_groups(uint32_t taddr, long long (&hi)[BN / 2],
                                             long long (&lo)[BN / 2]) {
  if constexpr (COUNT > 0) {
    constexpr int H = BN / 16;                   // 8-column pieces
    constexpr int MOST = 4 / H;                  // up to 32 registers in flight
    constexpr int N = COUNT >= MOST ? MOST : COUNT;
    uint32_t r[N][H][8];
#pragma unroll
    for (int g = 0; g < N; ++g)
#pragma unroll
      for (int h = 0; h < H; ++h) tmem_ld8(taddr + (FIRST + g) * BN + 8 * h, r[g][h]);
    tmem_wait_ld();
#pragma unroll
    for (int h = 0; h < H; ++h) {
      add_groups8<FIRST>(r[0][h], hi + 8 * h, lo + 8 * h);
      if constexpr (N > 1) add_groups8<FIRST + 1>(r[1][h], hi + 8 * h, lo + 8 * h);
      if constexpr (N > 2) add_groups8<FIRST + 2>(r[2][h], hi + 8 * h, lo + 8 * h);
      if constexpr (N > 3) add_groups8<FIRST + 3>(r[3][h], hi + 8 * h, lo + 8 * h);
    }
    drain_groups<BN, FIRST + N, COUNT - N>(taddr, hi, lo);
  }
}

// (hi 2^32 + lo) 2^e rounded once to FP64, with integer instructions.
__device__ __forceinline__ double assemble(long long hi, long long lo, int e) {
  // 128-bit sum: (w1, w0)
  unsigned long long w0 = (unsigned long long)hi << 32;
  long long w1 = hi >> 32;
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

constexpr int smem_bytes(int bn) { return NSTAGE * (A_STAGE + b_stage(bn)) + 128 + 256; }

// Persistent, warp-specialised: warp 0 copies stages, warp 1 issues MMAs,
// warps 2 .. 9 (two per TMEM lane quarter, BN / 2 columns each) drain one of
// two accumulator sets while the MMAs fill the other. A unit of work is one
// tile and up to 128 of its K; the integer sums run on over the units of a tile.
//
// Bound by shared memory: an MMA of N columns takes the larger of N / 2 cycles
// (the tensor rate) and 32 + N / 4 (its operands at 128 bytes per cycle), 624 a
// step of 16 K with BN = 32, into which the copies of the next steps write
// another 40 KB. The issuing thread took 844 a step until it ran under
// elect.sync (those of eight cases then went from 418 to 380 us).
//
// A block ends when no asynchronous operation of its own can still reach its
// shared memory: its loads are consumed, its MMAs complete, and the releases of
// its last stages have arrived.
template <int BN>
__global__ void __launch_bounds__(THREADS, 1)
    sliced_gemm_kernel(const GemmJob* __restrict__ jobs, const int4* __restrict__ tiles,
                       int n_tiles, int trigger, int* __restrict__ err, double* c_override,
                       int ldc_override) {
  constexpr int B_STAGE = b_stage(BN);
  constexpr int STAGE_BYTES = A_STAGE + B_STAGE;
  constexpr int COLS = BN / 2;  // columns per epilogue warp
  constexpr int SET = DIGITS * BN;  // TMEM columns of an accumulator set
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) &
                                             ~static_cast<uintptr_t>(127));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + NSTAGE * STAGE_BYTES);
  // full[NSTAGE], empty[NSTAGE], acc_full[2], acc_empty[2], quiet
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * NSTAGE + 5);
  int* progress = reinterpret_cast<int*>(tmem_slot + 1);  // [0] loads issued, [1] consumed
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + NSTAGE);
  const uint32_t acc_full = smem_u32(bars + 2 * NSTAGE);
  const uint32_t acc_empty = smem_u32(bars + 2 * NSTAGE + 2);
  const uint32_t quiet = smem_u32(bars + 2 * NSTAGE + 4);

  // The next kernel of the chain (slicing) may start early only where this one
  // leaves half of the SMs free: its blocks do not fit beside these (registers),
  // and on few free SMs they would pile up (a 1024 x 512 solve: 174 -> 198 us).
  if (trigger) axi::pdl_trigger();
  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full + 8 * b, 1);
      mbar_init(acc_empty + 8 * b, EPI_WARPS);
    }
    mbar_init(quiet, 1);
    progress[0] = 0;
    progress[1] = 0;
    axi_tma::fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 2 * SET);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      int g = 0, s = 0;
      uint32_t lap = 1;  // parity of the phase that frees a stage
      bool ok = true;
      axi::pdl_wait();
      for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
        const int4 tr = tiles[t];  // job, row block of A, row block of B, K steps
        const GemmJob& job = jobs[tr.x];
        const int nk = tr.w;
        const uint8_t* a = job.a + (size_t)tr.y * nk * A_STAGE;
        const uint8_t* b = job.b + (size_t)tr.z * nk * B_STAGE;
        for (int kb = 0; kb < nk; ++kb, ++g) {
          if (g >= NSTAGE && !mbar_wait(empty0 + 8 * s, lap, err, ERR_PRODUCER)) {
            ok = false;
            break;
          }
          const uint32_t st = smem_u32(smem + s * STAGE_BYTES);
          const uint32_t fb = full0 + 8 * s;
          mbar_expect_tx(fb, STAGE_BYTES);
          bulk_load(st, a + (size_t)kb * A_STAGE, A_STAGE, fb);
          bulk_load(st + A_STAGE, b + (size_t)kb * B_STAGE, B_STAGE, fb);
          if (++s == NSTAGE) s = 0, lap ^= 1;
        }
      }
      progress[0] = g;
      // releases of the last stages (commits arrive on their barriers by
      // themselves, also after the block has gone)
      for (int q = 0; q < NSTAGE && ok; ++q) {
        if (g + q >= NSTAGE) ok = mbar_wait(empty0 + 8 * s, lap, err, ERR_PRODUCER);
        if (++s == NSTAGE) s = 0, lap ^= 1;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (elect_one()) {
      const uint64_t a0 = operand_desc(smem_u32(smem), BM / 8 * 128);
      const uint64_t b0 = operand_desc(smem_u32(smem) + A_STAGE, DIGITS * BN / 8 * 128);
      int g = 0, u = 0, s = 0;
      uint32_t lap = 0;
      bool ok = true;
      axi::pdl_wait();  // the time limit of the waits starts once the predecessor is done
      for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
        const int nk = tiles[t].w;
        for (int k0 = 0; k0 < nk && ok; k0 += CHUNK, ++u) {
          const int set = u & 1, use = u >> 1;
          if (use > 0 && !mbar_wait(acc_empty + 8 * set, (use - 1) & 1, err, ERR_MMA)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d = tmem + set * SET;
          const int k1 = min(nk, k0 + CHUNK);
          for (int kb = k0; kb < k1; ++kb, ++g) {
            if (!mbar_wait(full0 + 8 * s, lap, err, ERR_MMA)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint64_t a = a0 + static_cast<uint32_t>(s * (STAGE_BYTES >> 4));
            const uint64_t b = b0 + static_cast<uint32_t>(s * (STAGE_BYTES >> 4));
            // Plane 0 of A against all planes of B also starts every accumulator;
            // the others follow from the narrowest to the widest, so that the
            // MMAs still queued when the commit goes in keep the tensor pipe
            // busy while this thread gets to the next step (797 cycles a step
            // with the narrowest last; products of eight cases 380 -> 362 us).
#pragma unroll
            for (int q = 0; q < DIGITS; ++q) {
              const int i = (DIGITS - q) % DIGITS;
              umma_f16(d + i * BN, a + (i * BM * BK * 2 >> 4), b, idesc_f16((DIGITS - i) * BN),
                       i > 0 || kb > k0 ? 1u : 0u);
            }
            umma_commit(empty0 + 8 * s);
            if (++s == NSTAGE) s = 0, lap ^= 1;
          }
          if (ok) umma_commit(acc_full + 8 * set);
        }
      }
      progress[1] = g;
      umma_commit(quiet);
      // (also after a failure, whose code would end mbar_wait early: MMAs in
      // flight must not outlive the block's shared and tensor memory)
      if (!axi_tma::mbar_wait_drain(quiet, 0)) atomicCAS(err, 0, ERR_MMA);
    }
    __syncwarp();
  } else {
    const int q = warp & 3;            // TMEM lane quarter
    const int half = (warp - 2) >> 2;  // columns COLS half .. COLS half + COLS - 1
    const uint32_t lane_base = static_cast<uint32_t>(32 * q) << 16;
    int u = 0;
    bool ok = true;
    axi::pdl_wait();
    // (a failure ends the waiting, not the loop: the results of this tile and
    // the later ones are written as NaN)
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
      const int4 tr = tiles[t];
      const GemmJob& job = jobs[tr.x];
      const int M = job.M, N = job.N;
      double* const c = c_override ? c_override : job.c;
      const long long ldc = c_override ? ldc_override : job.ldc;
      const double* const scale = job.scale;
      const int row = tr.y * BM + 32 * q + lane;
      const int col0 = tr.z * BN + COLS * half;
      const int ea_raw = job.ea[row];
      const int ea = max(ea_raw, 1) - 1022;
      const int* eb = job.eb + col0;
      const int e_off = 68 + job.exp_bias;  // 12 + 8 * 7 of the digits' weights
      int* const row_exps = job.row_exps;
      int* const col_exps = job.col_exps;
      int e_max = 0, e_col = 0;
      const int nk = tr.w;
      long long hi[COLS], lo[COLS];
#pragma unroll
      for (int j = 0; j < COLS; ++j) hi[j] = lo[j] = 0;
      for (int k0 = 0; k0 < nk && ok; k0 += CHUNK, ++u) {
        const int set = u & 1;
        ok = __all_sync(0xffffffffu,
                        mbar_wait(acc_full + 8 * set, (u >> 1) & 1, err, ERR_EPILOGUE));
        if (!ok) break;
        tc_fence_after();
        drain_groups<BN, 0, DIGITS>(tmem + lane_base + set * SET + COLS * half, hi, lo);
        tc_fence_before();
        __syncwarp();
        if (lane == 0)
          asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acc_empty + 8 * set)
                       : "memory");
      }
      const bool row_in = row < M;
      double* const cr = c + row * ldc + col0;
      const double* const sr = scale ? scale + (long long)row * N + col0 : nullptr;
      const int n = row_in ? min(COLS, N - col0) : 0;
      const bool vec = n == COLS && (reinterpret_cast<uintptr_t>(cr) & 15) == 0;
#pragma unroll
      for (int j = 0; j < COLS; j += 2) {
        double v[2];
#pragma unroll
        for (int w = 0; w < 2; ++w) {
          const int e_raw = eb[j + w];
          const int e = max(e_raw, 1) - 1022;
          // a row or column that is not finite gives NaN, a failure everywhere
          v[w] = assemble(hi[j + w], lo[j + w], ea + e - e_off);
          if (ea_raw == NOT_FINITE || e_raw == NOT_FINITE || !ok)
            v[w] = __longlong_as_double(0x7ff8000000000000ll);
          if (sr && j + w < n) v[w] *= sr[j + w];
          const int ev = j + w < n ? exponent_of(v[w]) : 0;
          e_max = max(e_max, ev);
          if (col_exps) {  // the largest of the column's finite values
            const int most = __reduce_max_sync(0xffffffffu, ev == NOT_FINITE ? 0 : ev);
            if (lane == j + w) e_col = most;
          }
        }
        if (vec) {
          *reinterpret_cast<double2*>(cr + j) = make_double2(v[0], v[1]);
        } else {
          if (j < n) cr[j] = v[0];
          if (j + 1 < n) cr[j + 1] = v[1];
        }
      }
      // what the next slicing needs: row maxima (so that it reads its source
      // once) or column maxima
      if (row_exps && e_max > 0) atomicMax(row_exps + row, e_max);
      if (col_exps && e_col > 0 && col0 + lane < N) atomicMax(col_exps + col0 + lane, e_col);
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
  if (warp == 1) tmem_dealloc(tmem, 2 * SET);
}

size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

}  // namespace

void append_slice_items(std::vector<int4>& items, int job, int rows, int block, int parts) {
  for (int g = 0; g < slice_groups(rows, block); ++g)
    for (int p = 0; p < parts; ++p) items.push_back(make_int4(job, g, p, parts));
}

void append_gemm_tiles(std::vector<int4>& tiles, int job, int M, int N, int K, int form) {
  const int cols = form_cols(form);
  for (int m = 0; m < (M + BM - 1) / BM; ++m)
    for (int n = 0; n < (N + cols - 1) / cols; ++n) tiles.push_back(make_int4(job, m, n, k_steps(K)));
}

void order_tiles(std::vector<int4>& tiles) {
  std::stable_sort(tiles.begin(), tiles.end(),
                   [](const int4& a, const int4& b) { return a.w > b.w; });
}

int launch_slice(const SliceJob* jobs_dev, const int4* items_dev, int n_items, cudaStream_t s,
                 const double* src, long long rs, int* err_begin, bool chained) {
  if (n_items <= 0) return AXI_OK;
  return axi::launch_chain(chained, "slice", slice_kernel, dim3(n_items), dim3(SL_THREADS), 0, s, 1, jobs_dev,
                         items_dev, src, rs, err_begin);
}

template <int BN>
int launch_tiles(const GemmJob* jobs_dev, const int4* tiles_dev, int n_tiles, int* err_dev,
                 cudaStream_t s, double* c, int ldc) {
  static std::once_flag once;
  static cudaError_t attr_status = cudaSuccess;
  std::call_once(once, [] {
    attr_status = cudaFuncSetAttribute(sliced_gemm_kernel<BN>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(BN));
  });
  if (attr_status != cudaSuccess) {
    axi::set_error("sliced GEMM: cannot reserve %d bytes of shared memory", smem_bytes(BN));
    return AXI_ERR_CUDA;
  }
  if (n_tiles <= 0) return AXI_OK;
  const int sms = axi::sm_count();
  const int blocks = n_tiles < sms ? n_tiles : sms;
  return axi::launch_chain(true, "sliced_gemm", sliced_gemm_kernel<BN>, dim3(blocks),
                           dim3(THREADS), smem_bytes(BN), s, 1, jobs_dev, tiles_dev, n_tiles,
                           2 * blocks <= sms ? 1 : 0, err_dev, c, ldc);
}

int launch_gemm(const GemmJob* jobs_dev, const int4* tiles_dev, int n_tiles, int form, int* err_dev,
                cudaStream_t s, double* c, int ldc) {
  return form == FORM_NARROW ? launch_tiles<16>(jobs_dev, tiles_dev, n_tiles, err_dev, s, c, ldc)
                             : launch_tiles<32>(jobs_dev, tiles_dev, n_tiles, err_dev, s, c, ldc);
}

namespace {
// The field's planes, which the four stages use in turn (padding to 32 rows
// covers every form), those of the radial bases, which stages 1 and 3 do, then
// the exponents: of each stage's field rows, of the columns of X (twice) and of
// the radial bases' rows (twice).
size_t spectral_plane_bytes(int nr, int nz) {
  return align_up(std::max(plane_bytes(nr, nz, 32), plane_bytes(nz, nr, 32)), 256);
}
size_t radial_plane_bytes(int nr) { return align_up(plane_bytes(nr, nr, BM), 256); }
}  // namespace

size_t spectral_slice_bytes(int nr, int nz) {
  return spectral_plane_bytes(nr, nz) + radial_plane_bytes(nr) +
         (size_t)2 * (2 * pad_rows(nr, 32) + pad_rows(nz, 32) + pad_rows(nr, BM)) * sizeof(int);
}

void spectral_jobs(int nr, int nz, const int form[4], const double* in, long long ld_in,
                   double* out, int ld_out, double* work, void* slices,
                   const void* const basis[4], const double* const radial[2],
                   const double* inv_eig, SliceJob sl[SLICE_JOBS], GemmJob gm[4]) {
  double* x = work;
  double* y = work + (size_t)nr * nz;
  uint8_t* radial_planes = static_cast<uint8_t*>(slices) + spectral_plane_bytes(nr, nz);
  int* exps = reinterpret_cast<int*>(radial_planes + radial_plane_bytes(nr));
  auto take = [&exps](int n) {
    int* p = exps;
    exps += n;
    return p;
  };
  int *rows[4], *cols[4] = {nullptr, nullptr, nullptr, nullptr};
  for (int st = 0; st < 4; ++st) rows[st] = take(pad_rows(st % 2 == 0 ? nr : nz, 32));
  for (int st = 0; st < 4; st += 2) cols[st] = take(pad_rows(nr, 32));
  const double* src[4] = {in, x, y, x};
  const long long rs[4] = {ld_in, nr, nz, nr};
  double* c[4] = {x, y, x, out};
  const int ldc[4] = {nr, nz, nr, ld_out};
  for (int st = 0; st < 4; ++st) {
    const bool along_r = st % 2 == 1;
    const int M = along_r ? nr : nz, N = along_r ? nz : nr, K = M;
    sl[st] = slice_job(src[st], rs[st], 1, N, K, form_cols(form[st]), slices, rows[st]);
    GemmJob& g = gm[st];
    g.b = sl[st].planes;
    g.eb = sl[st].exps;
    g.c = c[st];
    g.scale = st == 1 ? inv_eig : nullptr;
    g.M = M;
    g.N = N;
    g.ldc = ldc[st];
    g.nk = k_steps(K);
    // X leaves its column maxima for the balanced product, Y its row maxima
    g.col_exps = cols[st];
    g.row_exps = st == 1 ? rows[2] : nullptr;
    sl[st].have_exps = st == 2;
    sl[st].clear = st == 1 ? rows[2] : cols[st];
    sl[st].n_clear = sl[st].clear ? pad_rows(nr, 32) : 0;
    if (along_r) {
      SliceJob& a = sl[4 + st / 2];
      a = slice_job(radial[st / 2], nr, 1, nr, nr, BM, radial_planes, take(pad_rows(nr, BM)));
      a.balance = 1;
      sl[st].balance = -1;
      a.col_exps = sl[st].col_exps = cols[st - 1];
      g.a = a.planes;
      g.ea = a.exps;
      g.exp_bias = BALANCE_BIAS;
    } else {
      g.a = static_cast<const uint8_t*>(basis[st]);
      g.ea = reinterpret_cast<const int*>(g.a + plane_bytes(M, K, BM));
      g.exp_bias = 0;
    }
  }
}

}  // namespace axi_sl

// ---------------------------------------------------------------------------
// C entries.
// ---------------------------------------------------------------------------
namespace {

using namespace axi_sl;

// Plan of the standalone transform: [error word of the run, record of earlier
// runs][SliceJob x 6][GemmJob x 4][slice items x 4][tiles x 4][sliced z bases,
// radial bases][sliced field][X, Y]
// It depends on the grid alone, so that a run finds the plan that was written,
// whatever device is current: the forms and shares are those of a GB300.
constexpr int PLAN_SMS = 152;
struct TransformLayout {
  size_t err, sjobs, gjobs, items[4], tiles[4], basis[4], slices, work, total;
  int n_items[4], n_tiles[4], form[4], parts[4];
};

TransformLayout transform_layout(int nr, int nz) {
  TransformLayout L;
  size_t o = 0;
  L.err = o; o = align_up(o + 16, 256);
  L.sjobs = o; o = align_up(o + SLICE_JOBS * sizeof(SliceJob), 256);
  L.gjobs = o; o = align_up(o + 4 * sizeof(GemmJob), 256);
  for (int st = 0; st < 4; ++st) {
    const int M = st % 2 == 0 ? nz : nr, N = st % 2 == 0 ? nr : nz;
    L.form[st] = choose_form(gemm_tiles(M, N, FORM_NARROW), PLAN_SMS);
    const int groups = stage_groups(nr, nz, st, L.form[st]);
    L.parts[st] = slice_parts(groups, M, PLAN_SMS);
    L.n_items[st] = groups * L.parts[st];
    L.n_tiles[st] = gemm_tiles(M, N, L.form[st]);
    // room for any form, so that the size does not depend on the device
    L.items[st] = o;
    o = align_up(o + (size_t)stage_groups(nr, nz, st, FORM_WIDE) * ((M + 255) / 256) * sizeof(int4),
                 256);
    L.tiles[st] = o; o = align_up(o + gemm_tiles(M, N, FORM_NARROW) * sizeof(int4), 256);
  }
  for (int st = 0; st < 4; ++st) {
    L.basis[st] = o;
    o = align_up(o + (st % 2 == 0 ? slice_bytes(nz, nz, BM) : (size_t)nr * nr * sizeof(double)), 256);
  }
  L.slices = o; o = align_up(o + spectral_slice_bytes(nr, nz), 256);
  L.work = o; o = align_up(o + (size_t)2 * nr * nz * sizeof(double), 256);
  L.total = o;
  return L;
}

// Slices one matrix and waits for it.
int slice_now(const SliceJob& j, cudaStream_t s) {
  slice_matrix_kernel<<<slice_groups(j.rows, j.block), SL_THREADS, 0, s>>>(j);
  AXI_TRY(axi::launch_status("slice"));
  return cudaStreamSynchronize(s) == cudaSuccess ? AXI_OK : axi::launch_status("slice");
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
  return (int64_t)align_up(slice_bytes(rows, K, BM), 256);
}

extern "C" int axi_slice_operand_f64(void* dst, const double* src, int64_t row_stride,
                                     int64_t k_stride, int rows, int K, void* stream) {
  axi::clear_error();
  const char* what = "slice_operand";
  AXI_TRY(check_shape(what, rows, K));
  AXI_TRY(axi::check_ptrs(what, {dst, src}, {"dst", "src"}));
  return slice_now(slice_job(src, row_stride, k_stride, rows, K, BM, dst, exps_of(dst, rows, K, BM)),
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
  // E_z^-1 and E_z, stored transposed, sliced; copies of the radial bases
  const double* src[4] = {EzinvT, Er_inv_w, EzT, Er};
  const void* basis[4];
  for (int st = 0; st < 4; ++st) {
    basis[st] = base + L.basis[st];
    if (st % 2 == 0) {
      AXI_TRY(slice_now(slice_job(src[st], 1, nz, nz, nz, BM, base + L.basis[st],
                                  exps_of(base + L.basis[st], nz, nz, BM)), s));
    } else if (cudaMemcpyAsync(base + L.basis[st], src[st], (size_t)nr * nr * sizeof(double),
                               cudaMemcpyDeviceToDevice, s) != cudaSuccess) {
      return axi::launch_status(what);
    }
  }
  const double* radial[2] = {static_cast<const double*>(basis[1]),
                             static_cast<const double*>(basis[3])};
  SliceJob sl[SLICE_JOBS];
  GemmJob gm[4];
  spectral_jobs(nr, nz, L.form, nullptr, nz, nullptr, nz, reinterpret_cast<double*>(base + L.work),
                base + L.slices, basis, radial, inv_eig, sl, gm);
  std::vector<char> head(L.basis[0], 0);
  memcpy(&head[L.sjobs], sl, sizeof(sl));
  memcpy(&head[L.gjobs], gm, sizeof(gm));
  for (int st = 0; st < 4; ++st) {
    const int M = st % 2 == 0 ? nz : nr, N = st % 2 == 0 ? nr : nz;
    std::vector<int4> items, tiles;
    append_stage_items(items, 0, nr, nz, st, L.form[st], L.parts[st]);
    append_gemm_tiles(tiles, st, M, N, M, L.form[st]);
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
                         st == 0 ? in : nullptr, ld_in, st == 0 ? err : nullptr));
    AXI_TRY(launch_gemm(gj, reinterpret_cast<const int4*>(base + L.tiles[st]), L.n_tiles[st],
                        L.form[st], err, s, st == 3 ? out : nullptr, ld_out));
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
  int words[2];
  if (cudaMemcpyAsync(words, static_cast<const char*>(plan) + transform_layout(nr, nz).err,
                      sizeof(words), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return axi::launch_status(what);
  *error = words[0] ? words[0] : words[1];
  return AXI_OK;
}

// ---------------------------------------------------------------------------
// C (M, N) = A (M, K) B (N, K)^T .* S, both operands sliced per call.
// ---------------------------------------------------------------------------
namespace {

struct GemmLayout {
  size_t sjobs, gjob, items, tiles, err, a, b, total;
  int n_items, n_tiles, form;
};

GemmLayout gemm_layout(int M, int N, int K) {
  GemmLayout L;
  size_t o = 0;
  L.sjobs = o; o = align_up(o + 2 * sizeof(SliceJob), 256);
  L.gjob = o; o = align_up(o + sizeof(GemmJob), 256);
  L.form = choose_form(gemm_tiles(M, N, FORM_NARROW), axi::sm_count());
  L.n_items = slice_groups(M, BM) + slice_groups(N, form_cols(L.form));
  L.n_tiles = gemm_tiles(M, N, L.form);
  L.items = o; o = align_up(o + (size_t)(slice_groups(M, BM) + slice_groups(N, 32)) * sizeof(int4), 256);
  L.tiles = o; o = align_up(o + gemm_tiles(M, N, FORM_NARROW) * sizeof(int4), 256);
  L.err = o; o = align_up(o + 16, 256);
  L.a = o; o = align_up(o + slice_bytes(M, K, BM), 256);
  L.b = o; o = align_up(o + slice_bytes(N, K, 32), 256);
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
  const int cols = form_cols(L.form);
  SliceJob sl[2] = {slice_job(A, K, 1, M, K, BM, base + L.a, exps_of(base + L.a, M, K, BM)),
                    slice_job(B, K, 1, N, K, cols, base + L.b, exps_of(base + L.b, N, K, cols))};
  GemmJob g;
  g.a = sl[0].planes; g.ea = sl[0].exps; g.b = sl[1].planes; g.eb = sl[1].exps;
  g.c = C; g.scale = S; g.row_exps = nullptr; g.col_exps = nullptr; g.exp_bias = 0;
  g.M = M; g.N = N; g.ldc = N; g.nk = k_steps(K);
  std::vector<int4> items, tiles;
  append_slice_items(items, 0, M, BM, 1);
  append_slice_items(items, 1, N, cols, 1);
  append_gemm_tiles(tiles, 0, M, N, K, L.form);
  std::vector<char> head(L.err + 16, 0);
  memcpy(&head[L.sjobs], sl, sizeof(sl));
  memcpy(&head[L.gjob], &g, sizeof(g));
  memcpy(&head[L.items], items.data(), items.size() * sizeof(int4));
  memcpy(&head[L.tiles], tiles.data(), tiles.size() * sizeof(int4));
  if (cudaMemcpyAsync(work, head.data(), head.size(), cudaMemcpyHostToDevice, s) != cudaSuccess)
    return axi::launch_status(what);
  AXI_TRY(launch_slice(reinterpret_cast<const SliceJob*>(base + L.sjobs),
                       reinterpret_cast<const int4*>(base + L.items), L.n_items, s, nullptr, 0,
                       nullptr, false));  // (its tables were copied just now)
  int* err = reinterpret_cast<int*>(base + L.err);
  AXI_TRY(launch_gemm(reinterpret_cast<const GemmJob*>(base + L.gjob),
                      reinterpret_cast<const int4*>(base + L.tiles), L.n_tiles, L.form, err, s));
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
