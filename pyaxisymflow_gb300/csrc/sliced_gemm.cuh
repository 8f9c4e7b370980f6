// FP64 matrix products on the tcgen05 tensor cores, by integer slicing.
//
//   C[M, N] = A[M, K] * B[N, K]^T   (FP64 in and out), optionally .* S[M, N]
//
// The method is the error-free slicing of Ozaki, Ogita, Oishi and Rump
// ("Error-free transformations of matrix multiplication by using fast
// routines of matrix multiplication", Numer. Algorithms 59, 2012): every row
// of an operand is scaled by a power of two to |x| < 1 and written as nine
// signed 7-bit digits,
//
//   x = sum_{i=0..8} d_i 2^(-6 - 7 i),  |d_i| <= 64      (62 bits below the row's
//                                                          power of two)
//
// each digit plane stored as 16-bit floats (small integers, exact). A product
// of two planes is a sum of integers of at most 2^12, so the FP32 accumulators
// of the tensor cores hold it exactly; the planes i, j with i + j = d <= 8
// share accumulator d. Over K = 512 the accumulators 0 .. 7 stay within
// 8 * 512 * 2^12 = 2^24 (exact), accumulator 8 (weight 2^-68) rounds in its
// last bit. The epilogue adds the accumulators as integers (96 bits, exact for
// any K) and rounds to FP64 once.
//
// Error of the four-product spectral solve against long double on the same
// bases, 48 x 96 to 256 x 512 cells, smooth and white right-hand sides:
// psi 0.8-2.0e-16 (FP64 FMA products 1.1-20e-16),
// u_z 3-24e-16 (5-25e-16), u_r 4-53e-16 (8-76e-16), smaller in every case.
// With eight digits psi stayed at 3-9e-16 but u_z and u_r went to 1-6e-14 (psi
// near the axis is a cancelling sum), so nine are used.
//
// Why: GB300 executes FP64 at about 1.2 TFLOP/s and FP16 tensor work at about
// 2 PFLOP/s. 45 plane products cost 45 * 2 M N K FP16 operations, 1/40 of the
// time of the FP64 pipe. Measured, a soft-sphere step on 1024 x 512 cells (four
// products): 4169 us with FP64 FMA products, 1143 us with these; a step of the
// drop-in loop on 384 x 201 cells: 1178 and 488 us; a double engine step of
// eight cases of 256 x 128 to 1024 x 512: 3543 us with FP64 DCTs in z and FMA
// products in r, 837 us with four of these; of one 512 x 256 case 299 us
// (553 with four FMA products) and 193 us.
//
// Operands are laid out by the slicing kernel exactly as shared memory wants
// them: per block of rows and per 16 K-elements one contiguous piece (A: 128
// rows, 36 KB; B: 32 rows, 9 KB) in the tensor core's unswizzled K-major
// layout (8-row x 16-byte core matrices), so a pipeline stage is two bulk
// copies and every MMA is free of bank conflicts. B's nine planes follow each
// other in its rows: one MMA of A's plane i against B's planes 0 .. 8 - i
// (N = 32 (9 - i)) adds to the accumulators i .. 8, which are neighbouring
// TMEM columns, so a K step of 16 takes 10 MMAs.
#pragma once

#include <cuda.h>
#include <cstdint>
#include <vector>

#include "axi_common.cuh"
#include "tma.cuh"

namespace axi_sl {

constexpr int DIGITS = 9;
constexpr int BITS = 7;
constexpr int BM = 128;                              // rows of A per tile
constexpr int BN = 32;                               // rows of B per tile
constexpr int BK = 16;                               // K elements per stage
constexpr int A_STAGE = DIGITS * BM * BK * 2;        // 36864 bytes
constexpr int B_STAGE = DIGITS * BN * BK * 2;        // 9216 bytes
constexpr int STAGE_BYTES = A_STAGE + B_STAGE;
constexpr int NSTAGE = 5;
constexpr int CHUNK = 512 / BK;                      // K steps whose sums stay exact
constexpr int SMEM_BYTES = NSTAGE * STAGE_BYTES + 128 + 256;
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 32 * (2 + EPI_WARPS);

enum { ERR_PRODUCER = 7, ERR_MMA = 8, ERR_EPILOGUE = 9, ERR_DRAIN = 10 };
enum { KIND_A = 0, KIND_B = 1 };

// exponent of a row that holds a value which is not finite: its products are NaN
constexpr int EXP_NONFINITE = 1 << 20;

inline int pad_rows(int rows, int kind) {
  const int b = kind == KIND_A ? BM : BN;
  return (rows + b - 1) / b * b;
}
inline int k_steps(int K) { return (K + BK - 1) / BK; }

// Bytes of one sliced operand: the digit planes, then one exponent per row.
inline size_t plane_bytes(int rows, int K, int kind) {
  return (size_t)pad_rows(rows, kind) * k_steps(K) * BK * DIGITS * 2;
}
inline size_t slice_bytes(int rows, int K, int kind) {
  return plane_bytes(rows, K, kind) + (size_t)pad_rows(rows, kind) * sizeof(int);
}

// One operand to slice: src[row * rs + k * ks].
struct SliceJob {
  const double* src;
  long long rs, ks;
  int rows, K;
  int kind;
  int pad;
  uint8_t* planes;
  int* exps;
};

struct GemmJob {
  const uint8_t* a;
  const int* ea;
  const uint8_t* b;
  const int* eb;
  double* c;
  const double* scale;  // elementwise factor, row-major (M, N), or null
  int M, N, ldc;
  int nk;               // K steps
};

inline SliceJob slice_job(const double* src, long long rs, long long ks, int rows, int K, int kind,
                          void* dst) {
  SliceJob j;
  j.src = src; j.rs = rs; j.ks = ks; j.rows = rows; j.K = K; j.kind = kind; j.pad = 0;
  j.planes = static_cast<uint8_t*>(dst);
  j.exps = reinterpret_cast<int*>(j.planes + plane_bytes(rows, K, kind));
  return j;
}

// Items of the slicing kernel (8 rows each) and tiles of the product.
inline int slice_items(int rows, int kind) { return pad_rows(rows, kind) / 8; }
inline int gemm_tiles(int M, int N) { return ((M + BM - 1) / BM) * ((N + BN - 1) / BN); }
void append_slice_items(std::vector<int4>& items, int job, int rows, int kind);
void append_gemm_tiles(std::vector<int4>& tiles, int job, int M, int N, int K);
// longest main loop first, stable
void order_tiles(std::vector<int4>& tiles);

// The first operand's source / the output may be given per call (overrides,
// null: as in the job table; only for tables of one job).
int launch_slice(const SliceJob* jobs_dev, const int4* items_dev, int n_items, cudaStream_t s,
                 const double* src = nullptr, long long rs = 0);
int launch_gemm(const GemmJob* jobs_dev, const int4* tiles_dev, int n_tiles, int* err_dev,
                cudaStream_t s, double* c = nullptr, int ldc = 0);

// The four spectral products of one case on sliced operands (as C = A B^T):
//   0  X (nz, nr)   = Ezinv * in^T                 in   (nr, nz), row stride ld_in
//   1  Y (nr, nz)   = (Erinv_w * X^T) .* inv_eig
//   2  X (nz, nr)   = Ez * Y^T
//   3  out (nr, nz) = Er * X^T
// work: X then Y (2 nr nz doubles); slices: the B operand of the stage at
// hand (spectral_slice_bytes). basis: Ezinv, Erinv_w, Ez, Er as sliced A
// operands.
size_t spectral_slice_bytes(int nr, int nz);
void spectral_jobs(int nr, int nz, const double* in, long long ld_in, double* out, int ld_out,
                   double* work, void* slices, const void* const basis[4], const double* inv_eig,
                   SliceJob sl[4], GemmJob gm[4]);

}  // namespace axi_sl
