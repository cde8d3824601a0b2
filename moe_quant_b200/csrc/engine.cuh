// Picks the arithmetic for a dense contraction: fp32 CUDA cores or tcgen05
// tensor cores on 16-bit planes.  One Engine lives for the duration of one
// C-ABI call and carves its scratch out of that call's workspace.
#pragma once

#include "gemm.cuh"

namespace mq {

// Scratch the tensor-core path needs for a GEMM whose operands are at most
// (M x K) and (K x N) fp32: the bf16 planes of both operands.
size_t engine_workspace_bytes(int64_t M, int64_t N, int64_t K, int math, int split);

// 16-bit planes of one GEMM operand, K-major: element (plane, row, k) at
// base[(plane * total_rows + row) * K_pad + k].  rows are padded to 128, k to 64, so that every
// TMA box is fully inside the buffer.  row0 / k0 shift the origin: the operand of a GEMM may be a
// window of a larger plane buffer (e.g. one 128-wide k range of the planes of the whole factor).
struct PlaneSet {
  uint16_t* base = nullptr;
  int planes = 0;
  int64_t total_rows = 0;  // batch * rows_pad
  int rows_pad = 0;        // rows one batch occupies
  int K_pad = 0;
  bool fp16 = false;
  int64_t row0 = 0;
  int k0 = 0;
};

inline int64_t pad_rows(int64_t rows) { return (rows + 127) / 128 * 128; }
inline int64_t pad_k(int64_t k) { return (k + 63) / 64 * 64; }
inline size_t plane_set_bytes(int64_t rows, int64_t K, int planes) {
  return align_up((size_t)planes * (size_t)pad_rows(rows) * (size_t)pad_k(K) * 2, 256);
}

// x -> hi + mid + lo with bf16 pieces; each residual is exact in fp32.
__device__ __forceinline__ void split_bf16x3(float x, uint16_t& hi, uint16_t& mid, uint16_t& lo) {
  const __nv_bfloat16 h = __float2bfloat16_rn(x);
  const float r1 = x - __bfloat162float(h);
  const __nv_bfloat16 m = __float2bfloat16_rn(r1);
  const float r2 = r1 - __bfloat162float(m);
  hi = __bfloat16_as_ushort(h);
  mid = __bfloat16_as_ushort(m);
  lo = __bfloat16_as_ushort(__float2bfloat16_rn(r2));
}

// x -> hi + lo with fp16 pieces: 22 significant bits while |x| lies in [2^-3, 2^15], an absolute error of
// 2^-25 below.  The callers scale by powers of two so that the largest values sit just under 2^14; what
// the pair drops is then at most 2^-39 of those.  The three products hi hi, hi lo, lo hi stand in for the
// six of three bf16 planes: half the tensor work and two thirds of the operand bytes.
__device__ __forceinline__ void split_half2(float x, uint16_t& hi, uint16_t& lo) {
  const __half h = __float2half_rn(x);
  hi = __half_as_ushort(h);
  lo = __half_as_ushort(__float2half_rn(x - __half2float(h)));
}

// 2^(14 - e) for |bound| in [2^(e-1), 2^e): scaled by it, values up to `bound` lie below 2^14 (2^126 at most, so that the inverse
// is a normal number too).  1 for zero, infinity and NaN.
__device__ __forceinline__ float scale_below_2_14(float bound) {
  const int b = (int)((__float_as_uint(bound) >> 23) & 0xFFu);
  if (b == 0 || b == 255) return 1.0f;
  int e = 14 - (b - 126);   // -114 ..
  e = e > 126 ? 126 : e;
  return __uint_as_float((uint32_t)(e + 127) << 23);
}

// Equilibration of a matrix to be factored: the power of two 2^(13 - n) with h / 4^n in [1, 4) for the diagonal
// entry h, so that the diagonal of  eq H eq  lies in [2^26, 2^28) and every entry of its triangular factor
// below 2^14, where a pair of fp16 planes holds 22 bits of all but the smallest.  Powers of two: the factorisation
// does the same fp32 operations, up to exponents, as on H itself.  1 where h is not a positive finite number.
__device__ __forceinline__ float equilibrating_power(float h) {
  if (!(h > 0.0f && h < INFINITY)) return 1.0f;
  const int e = ilogbf(h);   // floor(log2 h)
  int n = 13 - (e >= 0 ? e / 2 : -((1 - e) / 2));
  n = n < -60 ? -60 : (n > 60 ? 60 : n);
  return __uint_as_float((uint32_t)(n + 127) << 23);
}

// The `split` of a factorisation or a sweep: 1 and 2 keep that many bf16 planes; 3 and 4 are full precision, and work on pairs
// of fp16 planes (3 with three products, 4 with all four) or on three bf16 planes (six products).
// Pairs from 513 columns on: below there is no deep update, which is what pairs are for and
// where sums of 64 of k win back the bits that the operands lose: error of a layer's running values against fp64, pairs in units of
// three planes (mean of 12 seeds): 1.012 to 1.022 at 256 to 512 columns, 0.96 at 648, 0.90 from 2048 on.  Nor are they faster
// there: 2048 x 256 takes 135.5 us with pairs and 131.9 with three planes, 32768 x 512 551 and 531.
// The low pieces' product shows where the factorisation's sums cancel.  Tokens for 0.17 / 0.35 / 0.7 of the columns, the same error
// with three products: 1.07 / 1.00 / 0.93 at 4096 columns, 1.08 / 1.05 / 0.97 at 1024; with all four 0.99 / 0.95 / 0.90 and
// 1.01 / 0.99 / 0.95.  It costs 2048 x 7168 1.9 % (3889 -> 3962 us), 7168 x 16384 3.9 %.
constexpr int64_t PAIRS_FROM_COLUMNS = 512;
inline bool uses_pairs(int64_t C, int math, int split) {
  return (math & ~MQ_MATH_COMPACT) == MQ_MATH_TENSOR && (split == 3 || split == 4) && C > PAIRS_FROM_COLUMNS;
}
inline int plane_count(int split) { return split == 4 ? 3 : split; }

// Columns of a super-block of the sweep and of a super-panel of the factorisation.
constexpr int SUPER_COLUMNS = 512;
// Columns whose update of everything behind them (in front of them, in the factorisation) is applied together where operands are pairs.
constexpr int64_t PAIR_FAR_COLUMNS = 1024;
// ... provided that the first half's update by itself, `tiles` of 256 x 256, is more than one for each of the 74 CTA pairs.  Otherwise an update takes as long
// as one tile, and one tile of 1024 takes longer than one of 512 (1056 columns: 544 us instead of 535).
inline bool joint_update(long long tiles) { return tiles > 74; }

// Whether a sweep takes a super-block of SUPER_COLUMNS per launch (sweep_super.cu) instead of a 128-column tile and the update behind it.
// The factor's diagonal blocks of that size are then scaled as a whole.  Of one layer with 4096 columns (its quantization, us, tiles /
// super-blocks with one lane a row; four lanes take another 14 us off) 512 rows take 1574 / 1462, 1024 rows 1598 / 1485, 2048 rows 1670 / 1558; but with several layers in flight the super-blocks'
// SM time counts, and the two must agree to the last bit there: four experts of 512 x 4096 take 6.66 / 5.80 ms, 1024 x 4096 6.38 / 6.38,
// 1024 x 7168 11.53 / 11.57, 1536 x 7168 12.46 / 12.87, 2048 x 7168 13.9 / 15.3.
constexpr int64_t SUPER_BLOCK_ROWS = 1024;
inline bool sweep_by_super_blocks(int64_t R, int math) { return (math & ~MQ_MATH_COMPACT) == MQ_MATH_TENSOR && R <= SUPER_BLOCK_ROWS; }

// Tensor-core GEMM whose operands are already planes (d.A / d.B and their strides are ignored;
// d.K is the reduction length starting at k0 of each set).  Both sets must have the same
// number of planes.
int gemm_tensor_planes(const GemmDesc& d, const PlaneSet& A, const PlaneSet& B, cudaStream_t st);

// fp32 matrix (rows x K, element (r,k) at src[r*rs + k*cs]) -> planes, zero padded.
// only_k_blocks_before_rows: write only the part with k in a 128-block in front of the row's own
// 128-block (the strictly upper blocks of a triangular factor stored transposed); the rest of
// the buffer stays unwritten and must not be read.  row_div (optional, device): destination row r is
// divided by row_div[r] before the split.
int make_planes_f32(const float* src, int64_t rs, int64_t cs, int rows, int K, int planes, uint16_t* dst, PlaneSet* out,
                    cudaStream_t st, bool only_k_blocks_before_rows = false, const float* row_div = nullptr);

// The factor's blocks above the diagonal, transposed, as pairs of fp16 planes: destination row j, k = i holds
//   Utilde[i][j] * t_j,  Utilde[i][j] = U[i][j] / col_div[j] * eq[j] / eq[i]   (col_div, eq optional, else 1),
// t_j a power of two that brings the column's entries under 2^14: from the column's maximum (a pass of its own), or, where
// eq_bounds says that this is near enough, with the C factors eq of an equilibration followed by the smallest of them, from the
// bound 2^14 / eq[C] that every entry of U[i][j] / eq[i] keeps.  inv_t (2 C floats)
// receives 1 / t_j in its first half, the second is scratch.  Only k in the blocks of `own` columns (128 or SUPER_COLUMNS) in
// front of the row's own are written (and read), inv_t from the second such block on.
int make_factor_planes_half(const float* U, int64_t ldu, int C, uint16_t* dst, float* inv_t, const float* col_div, const float* eq,
                            bool eq_bounds, int own, PlaneSet* out, cudaStream_t st);

// Whether that bound is near enough, by the damping: diag(T) is at least sqrt(rel_damp mean(diag H)), so the bound exceeds Utilde's unit
// diagonal by at most 2 sqrt(C / rel_damp), 2^11.5 here, and what a pair of fp16 planes drops (2^-39 of it) stays below
// 2^-27 of the error it multiplies.  With less damping a column of small channels, in front of one that is 2^24 times as large,
// kept ten bits and less of its entries.
inline bool equilibration_bounds_factor(int64_t C, float rel_damp) { return (float)C <= 0x1p21f * rel_damp; }

// Tensor-core GEMM on fp32 operands that are split into `split` bf16 planes on the fly.
int gemm_tensor_f32(const GemmDesc& d, int split, Workspace ws, cudaStream_t st);

struct Engine {
  int math;
  int split;
  Workspace ws;  // private view of what is left of the call's workspace
  cudaStream_t st;
  Engine(int math_, int split_, const Workspace& remaining, cudaStream_t st_)
      : math(math_), split(split_), ws(remaining.base ? remaining.base + remaining.used : nullptr,
                                        remaining.base ? remaining.size - remaining.used : 0), st(st_) {}
  int gemm(const GemmDesc& d) {
    if (math == MQ_MATH_TENSOR) return gemm_tensor_f32(d, split, ws, st);
    return gemm_simt(d, MQ_F32, st);
  }
};

}  // namespace mq
