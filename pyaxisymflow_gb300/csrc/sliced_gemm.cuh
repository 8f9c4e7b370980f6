// FP64 matrix products on the tcgen05 tensor cores, by integer slicing.
//
//   C[M, N] = A[M, K] * B[N, K]^T   (FP64 in and out), optionally .* S[M, N]
//
// The method is the error-free slicing of Ozaki, Ogita, Oishi and Rump
// ("Error-free transformations of matrix multiplication by using fast
// routines of matrix multiplication", Numer. Algorithms 59, 2012): every row
// of an operand is scaled by a power of two to |x| < 1 and written as eight
// signed digits of radix 256,
//
//   x = sum_{i=0..7} d_i 2^(-6 - 8 i),  |d_i| <= 128     (62 bits below the row's
//                                                          power of two)
//
// each digit plane stored as 16-bit floats (small integers, exact). A product
// of two planes is a sum of integers of at most 2^14, so the FP32 accumulators
// of the tensor cores hold it exactly; the planes i, j with i + j = d <= 7
// share accumulator d. Over K = 128 the accumulators stay within
// 8 * 128 * 2^14 = 2^24, so all of them are exact; every 128 of K the epilogue
// adds them to integer sums (96 bits, exact for any K), which it rounds to
// FP64 once.
//
// A digit string that starts at the row's largest value keeps 53 bits of the
// elements within 2^9 of it and fewer of the smaller ones. Along z that is
// enough (every row of a z basis is flat), along r it is not: the columns of E_r
// grow with the mode where those of the field fall, so that the sums of the rows
// next to the axis hung on elements cut short (relative errors of psi 1e-13 in
// rows 1 to 3 and up to 1 in row 0). So a radial product is balanced: column m
// of its left operand is multiplied by 2^c(m) and row m of the field divided by
// it, 2^c(m) being the size of the field's largest value of index m in this
// call. Both are exact; the left operand's rows then rank the terms of the sums as
// they are. It costs the slicing of the radial bases in every call (a radial
// slicing launch of eight cases of 256 x 128 to 1024 x 512: 12.5 -> 22 us, their
// step 666 -> 714; the step of one 512 x 256 case 4.6 us, of a soft sphere on
// 1024 x 512 cells 12).
//
// Error against long double on the same bases, 64 to 1024 radial rows (and 300, 65),
// sources smooth at the axis, in a ring, white, within four cells of the axis,
// and one cosine mode (FP64 FMA products in brackets): psi 0.6-8e-16
// (1-51e-16), psi in rows 1 to 3 0.4-5e-16 (1-170e-16), in row 0, which the
// operator decouples, 0.5e-16 to 2e-14 (3e-16 to 1e-13), the largest u_z
// smaller or, where it is the rounding of psi at the outer wall, within 10 %.
//
// Why: GB300 executes FP64 at about 1.2 TFLOP/s and FP16 tensor work at about
// 2 PFLOP/s; 36 plane products cost 36 * 2 M N K FP16 operations. A solve (four
// products) takes, in us: 128 x 64 cells 41, 256 x 128 50, 512 x 256 68, 768 x 384
// 85, 1024 x 512 142, 2048 x 1024 724 (36 TFLOP/s of FP64 products, 1.28 PFLOP/s
// of FP16 ones). Steps with FP64 FMA products / with these: soft sphere on 1024 x
// 512 cells 4171 / 460, double engine at 512 x 256 with FP64 DCTs in z 300 / 133,
// with eigenvectors in z 553 / 134, at 2048 x 1024 (FP64 DCTs) 8062 / 1062.
//
// Operands are laid out by the slicing kernel exactly as shared memory wants
// them: per block of rows and per 16 K-elements one contiguous piece (A: 128
// rows, 32 KB; B: 32 or 16 rows) in the tensor core's unswizzled K-major
// layout (8-row x 16-byte core matrices), so a pipeline stage is two bulk
// copies and every MMA is free of bank conflicts. B's eight planes follow each
// other in its rows: one MMA of A's plane i against B's planes 0 .. 7 - i
// (N = 32 (8 - i)) adds to the accumulators i .. 7, which are neighbouring
// TMEM columns, so a K step of 16 takes 8 MMAs.
//
// Slicing and product kernels form a chain of programmatic dependent launches:
// a kernel sets up its barriers and TMEM or reads its item while its predecessor
// finishes.
#pragma once

#include <cuda.h>
#include <cstdint>
#include <vector>

#include "axi_common.cuh"
#include "tma.cuh"

namespace axi_sl {

constexpr int DIGITS = 8;
constexpr int BM = 128;                              // rows of A per tile
constexpr int BK = 16;                               // K elements per stage
constexpr int A_STAGE = DIGITS * BM * BK * 2;        // 32768 bytes
constexpr int NSTAGE = 5;
constexpr int CHUNK = 128 / BK;                      // K steps whose sums stay exact
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 32 * (2 + EPI_WARPS);

// Forms of a product launch: columns of C per tile (= rows of a block of B).
enum Form { FORM_WIDE = 0, FORM_NARROW = 1 };
constexpr int form_cols(int form) { return form == FORM_WIDE ? 32 : 16; }
constexpr int b_stage(int bn) { return DIGITS * bn * BK * 2; }

// exponent word of a row that holds a value which is not finite (larger than
// every biased exponent, shifted or not)
constexpr int NOT_FINITE = 1 << 20;
// balanced right operands carry their exponents this much higher
constexpr int BALANCE_BIAS = 2048;

enum { ERR_PRODUCER = 7, ERR_MMA = 8, ERR_EPILOGUE = 9, ERR_DRAIN = 10 };

// Sliced operands are laid out in blocks of `block` rows: BM for A, the tile
// width for B.
inline int pad_rows(int rows, int block) { return (rows + block - 1) / block * block; }
inline int k_steps(int K) { return (K + BK - 1) / BK; }

// Bytes of one sliced operand: the digit planes, then one word per row, the
// largest biased exponent of its values (NOT_FINITE: a value is not finite, and
// the row's products are NaN).
inline size_t plane_bytes(int rows, int K, int block) {
  return (size_t)pad_rows(rows, block) * k_steps(K) * BK * DIGITS * 2;
}
inline size_t slice_bytes(int rows, int K, int block) {
  return plane_bytes(rows, K, block) + (size_t)pad_rows(rows, block) * sizeof(int);
}

// One operand to slice: src[row * rs + k * ks].
struct SliceJob {
  const double* src;
  long long rs, ks;
  int rows, K;
  int block;     // rows per block of the layout
  int have_exps; // the product that wrote src also left its row exponents in exps
  uint8_t* planes;
  int* exps;
  int* clear;    // words that the next product's epilogue accumulates into
  int n_clear;
  int balance;   // 1 / -1: left / right operand of a balanced product, else 0
  const int* col_exps;  // balanced: largest biased exponent of the field per K index
};

struct GemmJob {
  const uint8_t* a;
  const int* ea;
  const uint8_t* b;
  const int* eb;
  double* c;
  const double* scale;  // elementwise factor, row-major (M, N), or null
  int* row_exps;        // largest exponent of each row of C, accumulated (or null)
  int* col_exps;        // the same of each column, of its finite values (or null)
  int M, N, ldc;
  int nk;               // K steps
  int exp_bias;         // of the operands' exponents together
};

inline SliceJob slice_job(const double* src, long long rs, long long ks, int rows, int K, int block,
                          void* planes, int* exps) {
  SliceJob j;
  j.src = src; j.rs = rs; j.ks = ks; j.rows = rows; j.K = K; j.block = block;
  j.have_exps = 0;
  j.planes = static_cast<uint8_t*>(planes);
  j.exps = exps;
  j.clear = nullptr;
  j.n_clear = 0;
  j.balance = 0;
  j.col_exps = nullptr;
  return j;
}
// The exponents behind the planes of an operand.
inline int* exps_of(void* planes, int rows, int K, int block) {
  return reinterpret_cast<int*>(static_cast<uint8_t*>(planes) + plane_bytes(rows, K, block));
}

// Items of the slicing kernel: 8 rows each, and a share of their K where the
// row groups of a launch alone would leave SMs idle (a row's largest exponent
// is then found by every share, unless the product before has left it).
inline int slice_groups(int rows, int block) { return pad_rows(rows, block) / 8; }
inline int slice_parts(int groups_of_launch, int K, int sms) {
  const int want = (2 * sms + groups_of_launch - 1) / groups_of_launch;
  const int most = (K + 255) / 256;
  return want < 1 ? 1 : want < most ? want : most;
}
// Tiles of the product.
inline int gemm_tiles(int M, int N, int form) {
  const int cols = form_cols(form);
  return ((M + BM - 1) / BM) * ((N + cols - 1) / cols);
}
// Form of a launch that has `narrow_tiles` tiles of 16 columns: narrow where they
// all run at once. Steps of the double engine (all four launches in one form), us,
// wide / narrow: 128 x 64 124 / 105, 256 x 128 133 / 111, eight of them 142 / 118,
// 512 x 256 (64 tiles a launch) 156 / 130, 768 x 384 (144) 190 / 154, three of 512
// x 256 (192) 201 / 203, 1024 x 512 (256) 251 / 271, 2048 x 1024 (1024) 1061 / 1174.
// A mix of uneven cases just above the line would gain 4 % by narrow tiles (176
// and 198 tiles: 202 / 194, 214 / 206).
inline int choose_form(int narrow_tiles, int sms) {
  return narrow_tiles <= sms ? FORM_NARROW : FORM_WIDE;
}
void append_slice_items(std::vector<int4>& items, int job, int rows, int block, int parts);
void append_gemm_tiles(std::vector<int4>& tiles, int job, int M, int N, int K, int form);
// longest main loop first, stable
void order_tiles(std::vector<int4>& tiles);

// The first operand's source / the output may be given per call (overrides,
// null: as in the job table; only for tables of one job). chained: as a
// programmatic dependent launch, which reads its tables ahead of its
// dependencies (not where the stream has only just copied them).
// A product whose bounded waits run out sets *err_dev and writes NaN; later waits
// on a set word give up early. err_begin: two words, of which the first slicing
// of a run clears [0] (the word of its products) after moving a code to [1].
int launch_slice(const SliceJob* jobs_dev, const int4* items_dev, int n_items, cudaStream_t s,
                 const double* src = nullptr, long long rs = 0, int* err_begin = nullptr,
                 bool chained = true);
int launch_gemm(const GemmJob* jobs_dev, const int4* tiles_dev, int n_tiles, int form,
                int* err_dev, cudaStream_t s, double* c = nullptr, int ldc = 0);

// The four spectral products of one case on sliced operands (as C = A B^T):
//   0  X (nz, nr)   = Ezinv * in^T                 in   (nr, nz), row stride ld_in
//   1  Y (nr, nz)   = (Erinv_w * X^T) .* inv_eig
//   2  X (nz, nr)   = Ez * Y^T
//   3  out (nr, nz) = Er * X^T
// work: X then Y (2 nr nz doubles); slices: the operands of the stage at hand
// (spectral_slice_bytes). basis: Ezinv and Ez as sliced A operands (0, 2);
// radial: Erinv_w and Er (nr, nr), row-major, which are balanced against the
// field and sliced on every call, in the launch that slices the field.
// sl: the field operands of the four stages, then the radial bases of stages 1
// and 3.
constexpr int SLICE_JOBS = 6;
size_t spectral_slice_bytes(int nr, int nz);
void spectral_jobs(int nr, int nz, const int form[4], const double* in, long long ld_in,
                   double* out, int ld_out, double* work, void* slices,
                   const void* const basis[4], const double* const radial[2],
                   const double* inv_eig, SliceJob sl[SLICE_JOBS], GemmJob gm[4]);
// Row groups of 8 that the slicing launch of a stage covers, and its items.
// `job0`: index of the case's first slicing job.
inline int stage_groups(int nr, int nz, int st, int form) {
  return st % 2 == 0 ? slice_groups(nr, form_cols(form))
                     : slice_groups(nz, form_cols(form)) + slice_groups(nr, BM);
}
inline void append_stage_items(std::vector<int4>& items, int job0, int nr, int nz, int st, int form,
                               int parts) {
  append_slice_items(items, job0 + st, st % 2 == 0 ? nr : nz, form_cols(form), parts);
  if (st % 2 == 1) append_slice_items(items, job0 + 4 + st / 2, nr, BM, parts);
}

}  // namespace axi_sl
