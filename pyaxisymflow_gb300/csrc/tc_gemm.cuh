// tcgen05 (5th-generation tensor core) GEMM with FP32-accurate 3xTF32 products.
//
//   C[M, N] = A[M, K] * B[N, K]^T        (both operands K-major, FP32 in HBM)
//
// Each operand is stored as a TF32 "hi" part (x rounded to TF32) and the
// TF32-rounded remainder "lo"; the tensor core accumulates
// hi*hi + hi*lo + lo*hi in FP32 in tensor memory, which restores close to
// FP32 accuracy (the dropped lo*lo term is near FP32 rounding).
//
// Persistent CTAs (one per SM) walk a list of 128 x BN output tiles (BN = 128
// or 64):
//   warp 0, one thread   TMA producer: cp.async.bulk.tensor tiles (128 or BN rows
//                        x 32 floats, 128-byte swizzle) of A_hi, A_lo, B_hi, B_lo
//                        into a 3- or 4-stage shared-memory ring (mbarrier
//                        complete_tx), continuous across tiles
//   warp 1, one thread   MMA issuer: 3 x 4 tcgen05.mma.kind::tf32 per stage into
//                        one of two 128-lane x BN-column FP32 accumulators in
//                        TMEM; tcgen05.commit releases stages and accumulators
//   warps 2-9            epilogue: tcgen05.ld (warp w reads TMEM lanes
//                        32 (w % 4) .., warps 2-5 the first half of the columns,
//                        warps 6-9 the second); plain outputs go out as one TMA store
//                        per 32 x 32 block (128-byte swizzled shared-memory
//                        box), the split and scaled forms through a per-warp
//                        shared-memory transpose and row-contiguous stores; it
//                        drains one accumulator while the MMAs fill the other
// Every mbarrier wait is bounded by a 1 s wall-clock limit; on expiry the
// kernel records an error code, drains its outstanding copies (bounded),
// frees its TMEM and returns.
#pragma once

#include <cuda.h>
#include <cstdint>

#include "axi_common.cuh"
#include "tma.cuh"


namespace axi_tc {

constexpr int BM = 128;
// Tiles of 128 x BN, 32 K floats (128-byte rows, 128-byte swizzle) per stage.
// BN is 128 where a launch has tiles for every SM and 64 where it has not
// (choose_cols): a narrow tile's stage takes less time, and its result,
// summed in the same order, is the same. Measured alternatives to the stage,
// both slower on the spectral products: 16-float stages with a 6-deep ring
// (64-byte swizzle; twice the barriers and copies per FLOP) and 128 x 256 tiles
// with two 96 KB stages (the ring too shallow to cover the operand loads).
// A stage takes 768 cycles at 128 columns (12 MMAs at the tensor rate) and 670
// at 64 (the issuing thread; 576 for the MMAs, bound by the reads of A), 1044
// for both before the issuer ran under elect.sync. Products of 512 x 256,
// 768 x 384 and 1024 x 512 cases together 12.1 / 14.6 -> 9.3 / 12.0 us.
constexpr int BKF = 32;                         // K floats per stage
constexpr int ROW_BYTES = BKF * 4;              // swizzle span of a tile row
constexpr int EPI_WARPS = 8;                    // two per TMEM lane quarter
constexpr int THREADS = 32 * (2 + EPI_WARPS);   // TMA warp, MMA warp, 8 epilogue warps
// epilogue staging: a 32 x 33-float transpose per warp, or (TMA stores) a
// 32 x 32-float 128-byte-swizzled box per warp at 4 KB strides
constexpr int EPI_STAGE_BYTES = EPI_WARPS * 32 * 33 * 4;
static_assert(EPI_WARPS * 4096 <= EPI_STAGE_BYTES, "TMA store boxes fit the staging region");
constexpr int A_BYTES = BM * ROW_BYTES;         // 16 KB per A operand tile
constexpr int b_bytes(int bn) { return bn * ROW_BYTES; }
constexpr int stage_bytes(int bn) { return 2 * (A_BYTES + b_bytes(bn)); }  // A_hi, A_lo, B_hi, B_lo
constexpr int stages(int bn) { return bn == 64 ? 4 : 3; }
constexpr int smem_bytes(int bn) {
  return stages(bn) * stage_bytes(bn) + 1024 + EPI_STAGE_BYTES + 256;
}
static_assert(smem_bytes(128) <= 227 * 1024 && smem_bytes(64) <= 227 * 1024,
              "shared memory of a block");

inline int tile_count(int M, int N, int bn) { return ((M + BM - 1) / BM) * ((N + bn - 1) / bn); }
// Tile columns of a launch, from its tile count at 64 columns: 64 where those
// tiles run at once, 128 otherwise (twice the operand loads per product: 64
// cases' radial products go from 77 / 119 to 125 / 148 us). 128 / 64 columns,
// us per launch: K = 500, 500 x 252, 8 / 16 tiles: 20.5 / 15.0; K = 128,
// 128 x 256 pair, 2 / 4 tiles: 11.7 / 8.4; five cases, 68 / 136 tiles: 18.0 /
// 14.8. 32 columns leave half of the epilogue idle and load A once more per
// tile: 18.5 and 11.0 us on the first two.
inline int choose_cols(int tiles64, int sms) { return tiles64 <= sms ? 64 : 128; }

// MODE_PAIR_ADD: the output is the float pair (c, c_lo) holding c + c_lo;
// the product is added to it and the pair renormalised (c the rounded sum,
// c_lo the exact remainder), so repeated additions keep about 48 bits.
enum { MODE_PLAIN = 0, MODE_SPLIT = 1, MODE_SCALE_SPLIT = 2, MODE_SCALE = 3, MODE_PAIR_ADD = 4 };
enum { ERR_PRODUCER = 1, ERR_MMA = 2, ERR_EPILOGUE = 3, ERR_DRAIN = 4 };

// One GEMM problem. Tensor maps are encoded on the host (cuTensorMapEncodeTiled)
// and live in global memory next to the job.
struct TcJob {
  CUtensorMap a_hi, a_lo, b_hi, b_lo;
  CUtensorMap c_map;   // MODE_PLAIN with c_tma: the output in 32 x 32 boxes for TMA stores
  float* c;            // output (MODE_PLAIN) or its hi part
  float* c_lo;         // lo part (split modes; MODE_PAIR_ADD: low part of the pair)
  const float* scale;  // elementwise factor, row-major (M, N) (MODE_SCALE*)
  int M, N, K, ldc;
  int mode;
  int c_tma;           // 1: the epilogue stores tiles through c_map. Every job of
                       // one launch must agree (the two store paths lay out the
                       // epilogue's shared memory differently).
};

// Nearest TF32 value of x (10 explicit mantissa bits, ties away from zero):
// the tensor core ignores the low 13 bits of an operand, so operands are
// rounded before they are stored.
__device__ __forceinline__ float tf32_round(float x) {
  return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xFFFFE000u);
}

// TF32 split: hi = nearest TF32 of x, lo = nearest TF32 of the exact
// remainder x - hi. hi + lo carries about 23 significant bits (truncating
// either part would lose two of them).
__device__ __forceinline__ void tf32_split(float x, float& hi, float& lo) {
  hi = tf32_round(x);
  lo = tf32_round(x - hi);
}

// Host: encode a 2-D K-major FP32 operand (rows x K, row stride ld floats)
// for box_rows x BKF-float boxes (BM for A, the tile columns for B) with the
// ROW_BYTES swizzle. Returns AXI status.
int encode_operand(CUtensorMap* map, const float* base, int rows, int K, int ld, int box_rows);

// Host: encode the output of a MODE_PLAIN job (rows x cols, row stride ld
// floats) for 32 x 32-float TMA stores with the 128-byte swizzle; sets
// job->c_tma. False (job untouched) when the output cannot be stored that way
// (base not 16-byte aligned or ld not a multiple of 4).
bool encode_output(TcJob* job);

// Host: complete a tile table (job, m0, n0, -) with each tile's k-block
// count (w = ceil(K / BKF), which the kernel reads instead of the job) and
// (with `sort`) order it longest main loop (largest K) first, stable within
// equal K. The persistent CTAs take tiles with a fixed stride, so the long
// tiles are spread over all SMs before the short ones.
void order_tiles_by_k(int4* tiles, int n, const TcJob* jobs, bool sort = true);

// Host: launch the grouped kernel over `n_tiles` (job, m0, n0, k-blocks) tiles
// of `cols` columns (those that the jobs' B operands are encoded for) with `ctas_percent` of the SMs as persistent CTAs (0: all of them).
// `pdl`: as a programmatic dependent launch.
int launch(const TcJob* jobs_dev, const int4* tiles_dev, int n_tiles, int cols, int* err_dev,
           cudaStream_t s, int ctas_percent = 0, bool pdl = false);

}  // namespace axi_tc
