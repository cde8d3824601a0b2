// GPTQ column sweep.  Replaces the 2*C Triton launches and C/B cuBLAS calls of the
// reference's captured loop (src/gptq_loop.py:141-148) with, per 128-column tile,
// ONE sweep kernel plus ONE GEMM.
//
// (Up to 1024 rows a launch takes 512 columns instead: sweep_super.cu.)
//
// Sweep kernel: a CTA takes up to 64 weight rows through the tile in sub-blocks of sixteen columns.
// Column j is quantized as
//   q = clamp(floor(x/s + z + 0.5), 0, maxq)   y = round_to_dtype((q - z) s)   e = y - x
// (src/gptq_loop.py:28-40, src/quant_utils.py:30-49) and its error is applied to the columns
// behind it, w_k += Uhat[j,k] e (src/gptq_loop.py:83-88), with one fma per (j, k) in
// increasing j: the reference's order.  One thread per row runs the sixteen dependent steps of a
// sub-block; the other warps apply the errors to the rest of the tile.
//
// The errors of the tile (R x 128) go to a scratch matrix, on the tensor path as operand planes (pairs
// of fp16 planes in the inverse-free form of more than 512 columns, bf16 planes otherwise), and the lazy update
//   W[:, later] += E Uhat[tile, later]             (src/gptq_loop.py:148)
// is a GEMM: on the tensor path in two levels (the rest of the tile's 512-column super-block at
// once, everything behind the super-block once per super-block with all 512 errors of a row
// in the contraction), on the fp32 path one update of everything behind the tile.  Codes are
// written straight into the (R, C) uint8 result, so the transposes of src/gptq.py:191-199
// never happen.
#include "engine.cuh"
#include "mbarrier.cuh"
#include "profile.cuh"
#include "sweep.cuh"

namespace mq {

namespace {

constexpr int TILE = SWEEP_TILE;
constexpr int SUB = 16;                 // columns of a sub-block: one chain of quantisation steps per row
constexpr int N_SUB = TILE / SUB;
constexpr int SWEEP_THREADS = 256;
constexpr int MAX_ROWS = 64;            // rows of a CTA's group
constexpr int W_LD = TILE + 4;          // row stride of the running weights: a warp's 16-byte reads of 8 rows hit 32 banks
// Four tiles form a super-block of 512 columns.  Behind each tile only the rest of its own
// super-block takes the rank-128 update at once; the columns behind the super-block are updated
// once per super-block with all 512 errors of a row in one contraction, so a tile of W is read
// and written once per 512 instead of once per 128 swept columns.
constexpr int SUPER = SUPER_COLUMNS;

constexpr size_t sweep_smem_bytes(int rows, bool uniform, bool inverse_free) {
  return (size_t)(TILE * TILE + rows * W_LD * (inverse_free ? 2 : 1) + rows * (uniform ? N_SUB : 2 * SUB) * 4) * sizeof(float);
}

// One 128 x 128 tile of the factor (top-left element at `src`) -> shared memory, row-major, by
// asynchronous 16-byte copies, all in flight at once.  Quads that lie below the diagonal are not
// copied and not read; everything past nb becomes zero (a copy with source size 0).
__device__ __forceinline__ void stage_factor_tile(float* us, const float* __restrict__ src, int64_t ldu, int nb) {
  for (int idx = threadIdx.x; idx < TILE * TILE / 4; idx += blockDim.x) {
    const int j = idx >> 5, k4 = (idx & 31) * 4;
    if (k4 + 3 <= j) continue;
    const bool keep = j < nb && k4 < nb;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&us[j * TILE + k4]);
    const float* g = keep ? src + (int64_t)j * ldu + k4 : src;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(g), "r"(keep ? 16 : 0) : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// One 128-column tile of the sweep for up to MAX_ROWS rows per CTA, in eight sub-blocks of sixteen columns.
// Thread r < rows takes row r through sub-block c:
//   chain:  the sixteen columns in order, in registers: quantize column j, add e_j U[j, k] to the columns k behind
//           it inside the sub-block.  The only serial dependence is quantize(j) -> one FMA -> quantize(j + 1),
//           about fifteen operations;
//   next:   the sixteen errors go to the sixteen columns of sub-block c + 1, which it then holds.
// Meanwhile the other warps add the errors of sub-block c - 1 to the columns from sub-block c + 1 on: a lane
// keeps the 16 x 4 entries of the factor for its four columns in registers and walks the rows.  One barrier
// per sub-block hands the errors over and orders the two: before `next` touches sub-block c + 1 the other
// warps have added everything up to c - 1 there.  Every element so takes the errors in increasing column order
// with one FMA each, as a column-at-a-time recurrence does.
// What bounds a tile is the chain, 128 steps of 84 cycles whatever the number of rows (5.6 us), and handing the
// sub-blocks over, 700 to 1000 cycles each (3.4 us).  (Original weights that the chain loaded itself, a sub-block ahead, cost a sweep of
// 2048 x 7168 45 us of 1485, and staging them behind the wait for the update in front another 8; the scales are as well off behind it.  With
// sixteen or eight lanes per row and the row's tile in their registers, the owner of a chunk ran its chain while
// the others waited, and both the chain and the rest were one serial instruction stream: 19 us for 2048 rows,
// 36 us for 7168; one row per thread for everything, 30 us.  Now 15.7 and 19 us.)
// UNIFORM: the columns of a sub-block lie in one quantization group (group % 16 == 0).
// INVERSE_FREE (a.Worig given): U is the unit factor Utilde = Uhat^-1 and what is propagated is minus the
// total change of the column, -(y - w_original), instead of the error against the running value;
// x_j = w_j - sum_{i<j} (y_i - w_i) Utilde[i,j] is the same number as the reference's running weight
// (E Uhat = Y - W  <=>  E = (Y - W) Utilde).
template <int DT, bool UNIFORM, bool INVERSE_FREE>
__global__ void __launch_bounds__(SWEEP_THREADS, 1) sweep_tile_kernel(const SweepArgs a, const int group_rows) {
  using T = typename StorageOf<DT>::type;
  extern __shared__ __align__(16) float sweep_smem[];
  float* us = sweep_smem;                            // [TILE][TILE], strict upper triangle
  float* ws = sweep_smem + TILE * TILE;              // [group_rows][W_LD]: running weights, replaced by the errors as they become known
  float* wos = ws + group_rows * W_LD;               // INVERSE_FREE: [group_rows][W_LD], original weights
  // the grid of every row (scale, its reciprocal, zero point): UNIFORM [N_SUB][group_rows], one per sub-block;
  // otherwise [2][SUB][group_rows], the columns of two sub-blocks by turns
  float4* gs = reinterpret_cast<float4*>(ws + group_rows * W_LD * (INVERSE_FREE ? 2 : 1));
  const int nb = a.nb, i1 = a.i1, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float maxq = a.maxq;
  const bool wide_codes = (a.C & 15) == 0 && (reinterpret_cast<uintptr_t>(a.codes) & 15) == 0;
  const uint32_t group = (uint32_t)a.group;
  int row0 = blockIdx.x * group_rows, rows = a.R - row0 < group_rows ? a.R - row0 : group_rows;   // the grid has no CTA without rows
  auto grid_of = [&](int r, int j) {   // column j of the tile
    float s = 1.0f, z = a.zero_default;
    if (j < nb) {
      const int64_t off = (int64_t)(row0 + r) * a.s_rs + (int64_t)((uint32_t)(i1 + j) / group) * a.s_gs;
      s = __ldg(a.scale + off);
      if (a.zero) z = __ldg(a.zero + off);
    }
    return make_float4(s, 1.0f / s, z, 0.0f);
  };
  auto fill_columns = [&](int c, int from, int step) {   // !UNIFORM: the sixteen columns of sub-block c
    for (int idx = from; idx < rows * SUB; idx += step)
      gs[((c & 1) * SUB + (idx & (SUB - 1))) * group_rows + idx / SUB] = grid_of(idx / SUB, c * SUB + (idx & (SUB - 1)));
  };
  auto stage_rows = [&](float* dst, const float* __restrict__ src, int64_t ld) {   // this tile's columns of the group
    for (int idx = tid; idx < rows * (TILE / 4); idx += SWEEP_THREADS) {
      const int r = idx >> 5, k4 = (idx & 31) * 4;
      const bool keep = k4 < nb;
      const float* g = src + (int64_t)(row0 + r) * ld + i1 + (keep ? k4 : 0);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(&dst[r * W_LD + k4])), "l"(g), "r"(keep ? 16 : 0)
                   : "memory");
    }
  };
  auto fill_grid = [&] {
    if constexpr (UNIFORM) {
      for (int idx = tid; idx < rows * N_SUB; idx += SWEEP_THREADS) gs[(idx & 7) * group_rows + (idx >> 3)] = grid_of(idx >> 3, (idx & 7) * SUB);
    } else {
      fill_columns(0, tid, SWEEP_THREADS);
    }
  };
  // The factor and the original weights are constant during the sweep: they are staged before this grid waits for the
  // rank-128 update that precedes it in the stream (only W depends on that update).
  stage_factor_tile(us, a.U + (int64_t)i1 * a.ldu + i1, a.ldu, nb);
  if constexpr (INVERSE_FREE) stage_rows(wos, a.Worig, a.ldwo);
  chain_wait();
  chain_release();

  for (;;) {
    const int chain_warps = (rows + 31) >> 5;
    stage_rows(ws, a.W, a.ldw);
    asm volatile("cp.async.commit_group;" ::: "memory");
    fill_grid();
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    if (warp < chain_warps) {
      // ---- chains.  Lanes past the last row repeat it and store nothing.
      const bool valid = tid < rows;
      const int r = valid ? tid : rows - 1;
      const int64_t row = row0 + r;
      float* wrow = ws + r * W_LD;
      const float* worow = wos + r * W_LD;
      float w[SUB];
#pragma unroll
      for (int qd = 0; qd < SUB / 4; ++qd) {
        const float4 v = *reinterpret_cast<const float4*>(wrow + 4 * qd);
        w[4 * qd] = v.x; w[4 * qd + 1] = v.y; w[4 * qd + 2] = v.z; w[4 * qd + 3] = v.w;
      }
#pragma unroll 1
      for (int c = 0; c < N_SUB; ++c) {
        const int j0 = c * SUB;
        constexpr int NS = UNIFORM ? 1 : SUB;
        float sc[NS], zr[NS], rs[NS];
        if constexpr (UNIFORM) {
          const float4 g = gs[c * group_rows + r];
          sc[0] = g.x; rs[0] = g.y; zr[0] = g.z;
        } else {
#pragma unroll
          for (int t = 0; t < SUB; ++t) {
            const float4 g = gs[((c & 1) * SUB + t) * group_rows + r];
            sc[t] = g.x; rs[t] = g.y; zr[t] = g.z;
          }
        }
        float e[SUB];
        uint32_t cw[SUB / 4];
        float4 wo = make_float4(0.f, 0.f, 0.f, 0.f);
        const float* ud = us + j0 * TILE + j0;   // the sub-block's own 16 x 16 block of the factor
#pragma unroll
        for (int t = 0; t < SUB; ++t) {
          const float s_t = sc[UNIFORM ? 0 : t], z_t = zr[UNIFORM ? 0 : t], r_t = rs[UNIFORM ? 0 : t];
          float4 ur[SUB / 4];
#pragma unroll
          for (int qd = t >> 2; qd < SUB / 4; ++qd) {
            if (qd == (t >> 2) && (t & 3) == 3) continue;
            ur[qd] = *reinterpret_cast<const float4*>(ud + t * TILE + 4 * qd);
          }
          const float x = w[t];
          // x / s through the reciprocal and one residual correction (Markstein 1990): two FMAs on the chain
          float d = x * r_t;
          d = fmaf(fmaf(-s_t, d, x), r_t, d);
          // clamp first, then floor (the bounds are whole numbers, so the order does not matter): adding 2^23
          // with rounding towards minus infinity leaves the whole part, and the code in the low bits
          const float v = fminf(fmaxf((d + z_t) + 0.5f, 0.0f), maxq);
          const float big = __fadd_rd(v, 8388608.0f);
          const float q = big - 8388608.0f;
          const float y = round_through<DT>((q - z_t) * s_t);
          if (INVERSE_FREE && (t & 3) == 0) wo = *reinterpret_cast<const float4*>(worow + j0 + t);
          const float et = INVERSE_FREE ? ((t & 3) == 0 ? wo.x : (t & 3) == 1 ? wo.y : (t & 3) == 2 ? wo.z : wo.w) - y : y - x;
          e[t] = et;
          const uint32_t code = __float_as_uint(big) & 0xFFu;
          if ((t & 3) == 0) cw[t >> 2] = code;
          else cw[t >> 2] |= code << (8 * (t & 3));
          // the rest of t's own quad one by one, whole quads after it
          if ((t & 3) != 3) {
            const float4 u = ur[t >> 2];
            if ((t & 3) < 1) w[(t & ~3) + 1] = fmaf(u.y, et, w[(t & ~3) + 1]);
            if ((t & 3) < 2) w[(t & ~3) + 2] = fmaf(u.z, et, w[(t & ~3) + 2]);
            w[(t & ~3) + 3] = fmaf(u.w, et, w[(t & ~3) + 3]);
          }
          const float2 e2 = make_float2(et, et);
#pragma unroll
          for (int qd = (t >> 2) + 1; qd < SUB / 4; ++qd) {
            const float4 u = ur[qd];
            // packed fp32 FMA: two columns per instruction, each half an ordinary fma.rn
            const float2 p01 = __ffma2_rn(make_float2(u.x, u.y), e2, make_float2(w[4 * qd], w[4 * qd + 1]));
            const float2 p23 = __ffma2_rn(make_float2(u.z, u.w), e2, make_float2(w[4 * qd + 2], w[4 * qd + 3]));
            w[4 * qd] = p01.x; w[4 * qd + 1] = p01.y; w[4 * qd + 2] = p23.x; w[4 * qd + 3] = p23.y;
          }
        }
        if (valid) {
#pragma unroll
          for (int qd = 0; qd < SUB / 4; ++qd)
            *reinterpret_cast<float4*>(wrow + j0 + 4 * qd) = make_float4(e[4 * qd], e[4 * qd + 1], e[4 * qd + 2], e[4 * qd + 3]);
        }
        __syncthreads();
        if (c + 1 < N_SUB) {
          // ---- next: this row's errors on the columns of the following sub-block
#pragma unroll
          for (int qd = 0; qd < SUB / 4; ++qd) {
            const float4 v = *reinterpret_cast<const float4*>(wrow + j0 + SUB + 4 * qd);
            w[4 * qd] = v.x; w[4 * qd + 1] = v.y; w[4 * qd + 2] = v.z; w[4 * qd + 3] = v.w;
          }
#pragma unroll
          for (int t = 0; t < SUB; ++t) {
            const float2 e2 = make_float2(e[t], e[t]);
#pragma unroll
            for (int qd = 0; qd < SUB / 4; ++qd) {
              const float4 u = *reinterpret_cast<const float4*>(ud + t * TILE + SUB + 4 * qd);
              const float2 p01 = __ffma2_rn(make_float2(u.x, u.y), e2, make_float2(w[4 * qd], w[4 * qd + 1]));
              const float2 p23 = __ffma2_rn(make_float2(u.z, u.w), e2, make_float2(w[4 * qd + 2], w[4 * qd + 3]));
              w[4 * qd] = p01.x; w[4 * qd + 1] = p01.y; w[4 * qd + 2] = p23.x; w[4 * qd + 3] = p23.y;
            }
          }
        }
        // codes (and packed words) leave; a narrow last tile ends on a multiple of eight columns
        if (valid) {
          uint8_t* cdst = a.codes + row * a.C + i1 + j0;
          if (wide_codes && j0 + SUB <= nb) {
            *reinterpret_cast<uint4*>(cdst) = make_uint4(cw[0], cw[1], cw[2], cw[3]);
          } else {
#pragma unroll
            for (int qd = 0; qd < SUB / 4; ++qd)
              if (j0 + 4 * qd < nb) *reinterpret_cast<uint32_t*>(cdst + 4 * qd) = cw[qd];
          }
          if (a.packed) {
#pragma unroll
            for (int h = 0; h < SUB / 8; ++h)
              if (j0 + 8 * h < nb) a.packed[row * (a.C >> 3) + ((i1 + j0 + 8 * h) >> 3)] = (int32_t)pack_nibbles(cw[2 * h], cw[2 * h + 1]);
          }
          if (a.deq) {
            T* dq = static_cast<T*>(a.deq) + row * a.C + i1 + j0;
#pragma unroll
            for (int t = 0; t < SUB; ++t)
              if (j0 + t < nb)
                dq[t] = from_float<T>(((float)((cw[t >> 2] >> (8 * (t & 3))) & 0xFFu) - zr[UNIFORM ? 0 : t]) * sc[UNIFORM ? 0 : t]);
          }
        }
      }
    } else {
      // ---- the errors of sub-block c on the columns from sub-block c + 2 on.  `quads` column quads; the lanes of
      // a warp divide into rows of `span` lanes, so that few lanes idle as the region shrinks
      const int first = warp - chain_warps, helpers = SWEEP_THREADS / 32 - chain_warps;
#pragma unroll 1
      for (int c = 0; c < N_SUB; ++c) {
        const int j0 = c * SUB;
        const int quads = (TILE - 2 * SUB - j0) / 4;
        const int span = quads > 16 ? 32 : quads > 8 ? 16 : quads > 4 ? 8 : 4;
        const int quad = lane & (span - 1);
        const bool mine = quad < quads;
        const int k = j0 + 2 * SUB + 4 * quad;
        float4 u[SUB];
        if (mine) {
#pragma unroll
          for (int t = 0; t < SUB; ++t) u[t] = *reinterpret_cast<const float4*>(us + (j0 + t) * TILE + k);
        }
        if (!UNIFORM && c + 1 < N_SUB) fill_columns(c + 1, tid - 32 * chain_warps, SWEEP_THREADS - 32 * chain_warps);
        __syncthreads();
        if (mine) {
          const int per_warp = 32 / span;
          for (int r = first * per_warp + lane / span; r < rows; r += helpers * per_warp) {
            float* wr = ws + r * W_LD;
            float4 v = *reinterpret_cast<const float4*>(wr + k);
#pragma unroll
            for (int t4 = 0; t4 < SUB / 4; ++t4) {
              const float4 e4 = *reinterpret_cast<const float4*>(wr + j0 + 4 * t4);
              const float ev[4] = {e4.x, e4.y, e4.z, e4.w};
#pragma unroll
              for (int t = 0; t < 4; ++t) {
                const float4 uu = u[4 * t4 + t];
                const float2 e2 = make_float2(ev[t], ev[t]);
                const float2 p01 = __ffma2_rn(make_float2(uu.x, uu.y), e2, make_float2(v.x, v.y));
                const float2 p23 = __ffma2_rn(make_float2(uu.z, uu.w), e2, make_float2(v.z, v.w));
                v = make_float4(p01.x, p01.y, p23.x, p23.y);
              }
            }
            *reinterpret_cast<float4*>(wr + k) = v;
          }
        }
      }
    }
    __syncthreads();

    // ---- the errors of the tile (columns past nb are zero: the update may read all 128)
    for (int idx = tid; idx < rows * (TILE / 8); idx += SWEEP_THREADS) {
      const int r = idx >> 4, k = (idx & 15) * 8;
      const float4 lo4 = *reinterpret_cast<const float4*>(ws + r * W_LD + k), hi4 = *reinterpret_cast<const float4*>(ws + r * W_LD + k + 4);
      write_errors(a, row0 + r, k, lo4, hi4, lane);
    }
    row0 += gridDim.x * group_rows;
    if (row0 >= a.R) break;
    rows = a.R - row0 < group_rows ? a.R - row0 : group_rows;
    __syncthreads();   // the next group's weights replace the errors
    if constexpr (INVERSE_FREE) stage_rows(wos, a.Worig, a.ldwo);
  }
}

template <int DT>
int launch_sweep_tile(bool chained, bool uniform, int grid, int rows, cudaStream_t st, const SweepArgs& args) {
  const bool free = args.Worig != nullptr;
  auto* kernel = uniform ? (free ? sweep_tile_kernel<DT, true, true> : sweep_tile_kernel<DT, true, false>)
                         : (free ? sweep_tile_kernel<DT, false, true> : sweep_tile_kernel<DT, false, false>);
  MQ_CUDA(launch_chained(chained, kernel, dim3(grid), dim3(SWEEP_THREADS), sweep_smem_bytes(rows, uniform, free), st, args, rows));
  return MQ_OK;
}

template <int DT>
int configure_dtype() {
  constexpr int bytes = (int)sweep_smem_bytes(MAX_ROWS, false, true);
  MQ_CUDA(cudaFuncSetAttribute(sweep_tile_kernel<DT, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  MQ_CUDA(cudaFuncSetAttribute(sweep_tile_kernel<DT, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  MQ_CUDA(cudaFuncSetAttribute(sweep_tile_kernel<DT, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  MQ_CUDA(cudaFuncSetAttribute(sweep_tile_kernel<DT, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  return MQ_OK;
}

int configure_once() {
  static bool done[64] = {};
  int dev = 0;
  MQ_CUDA(cudaGetDevice(&dev));
  if (!done[dev & 63]) {
    MQ_TRY(configure_dtype<MQ_F32>());
    MQ_TRY(configure_dtype<MQ_BF16>());
    MQ_TRY(configure_dtype<MQ_F16>());
    done[dev & 63] = true;
  }
  return MQ_OK;
}

}  // namespace

// inverse_free: the sweep has the original weights and works on pairs of planes where uses_pairs says so.
size_t sweep_workspace_bytes(int64_t R, int64_t C, int math, int split, bool inverse_free) {
  if ((math & ~MQ_MATH_COMPACT) != MQ_MATH_TENSOR) return align_up((size_t)R * TILE * sizeof(float), 256);
  if (inverse_free && uses_pairs(C, math, split))
    return plane_set_bytes(R, PAIR_FAR_COLUMNS, 2) + plane_set_bytes(C, C, 2) + align_up((size_t)R * (PAIR_FAR_COLUMNS / TILE) * sizeof(float), 256) +
           align_up((size_t)C * 2 * sizeof(float), 256);
  return plane_set_bytes(R, SUPER, plane_count(split)) + plane_set_bytes(C, C, plane_count(split));
}

int gptq_sweep(float* W, int64_t R, int64_t C, int64_t ldw, const float* Uhat, int64_t ldu, const float* scale,
               const float* zero, int64_t group, int64_t s_rs, int64_t s_gs, int bits, int out_dtype, uint8_t* codes,
               void* deq, const float* Worig, int64_t ldwo, int math, int split, Workspace& ws, cudaStream_t st,
               const float* col_div, const float* eq, bool eq_bounds, int32_t* packed) {
  // col_div (tensor math only): above its diagonal 128-blocks Uhat holds the factor before its
  // columns were divided by col_div; the plane split divides where it reads it.  The diagonal
  // blocks, which the tiles read, are already scaled (blocks of SUPER columns where sweep_by_super_blocks says so).  eq (with col_div): what lies above is the factor
  // of the equilibrated matrix, entry (i, j) times eq[j] / eq[i] is the one of the matrix itself; eq_bounds: see
  // make_factor_planes_half.
  MQ_TRY(configure_once());
  const bool compact = (math & MQ_MATH_COMPACT) != 0;
  math &= ~MQ_MATH_COMPACT;
  const bool tensor = math == MQ_MATH_TENSOR;
  float* err = tensor ? nullptr : ws.take<float>((size_t)R * TILE);
  MQ_REQUIRE(tensor || err, MQ_ERR_WORKSPACE, "mq_gptq_sweep: workspace too small");
  MQ_REQUIRE(!tensor || (split >= 1 && split <= 4), MQ_ERR_ARGUMENT, "mq_gptq_sweep: split must be 1, 2, 3 or 4 (got %d)", split);
  const int all_products = split == 4 ? 1 : 0;   // of pairs
  split = plane_count(split);
  Engine eng(math, split, ws, st);
  // Tensor path: the factor is cut into transposed planes once (row n, k -> U[k][n]); the lazy
  // update of tile i1 then reads the window k in [i1, i1+128), rows n >= i2 of those planes,
  // and the sweep kernel writes its errors as planes itself.  No per-tile conversion passes.
  //
  // Inverse-free form at full precision (uses_pairs): the operands are pairs of fp16 planes, three
  // products instead of six (split_half2).  A power of two per row and tile brings the errors into fp16's
  // range, and one per column does so for the factor; the GEMM's epilogue takes both back exactly.  The
  // other form, which propagates y - x against the inverse, keeps three bf16 planes.
  const bool half = uses_pairs(C, math, split) && Worig != nullptr;
  MQ_REQUIRE(!eq || half || !tensor, MQ_ERR_ARGUMENT, "mq_gptq_sweep: an equilibrated factor needs the inverse-free form");
  const bool by_super = sweep_by_super_blocks(R, math);
  const int own = by_super ? SUPER : TILE;               // diagonal blocks of this size are already divided by col_div, and need no planes
  const int64_t far = half ? PAIR_FAR_COLUMNS : SUPER;   // columns whose update of everything behind them is applied together
  PlaneSet err_set, u_set;
  float *row_f = nullptr, *col_f = nullptr;
  if (half) {
    uint16_t* ep = ws.take<uint16_t>(plane_set_bytes(R, far, 2) / 2);
    uint16_t* up = ws.take<uint16_t>(plane_set_bytes(C, C, 2) / 2);
    row_f = ws.take<float>((size_t)R * (far / TILE));
    col_f = ws.take<float>((size_t)C * 2);
    MQ_REQUIRE(ep && up && row_f && col_f, MQ_ERR_WORKSPACE, "mq_gptq_sweep: workspace too small for the operand planes");
    err_set.base = ep; err_set.planes = 2; err_set.rows_pad = (int)pad_rows(R); err_set.total_rows = err_set.rows_pad;
    err_set.K_pad = (int)far; err_set.fp16 = true;
    MQ_TRY(make_factor_planes_half(Uhat, ldu, (int)C, up, col_f, col_div, eq, eq_bounds, own, &u_set, st));
  } else if (tensor && !(by_super && C <= SUPER)) {   // (a single super-block has no updates)
    uint16_t* ep = ws.take<uint16_t>(plane_set_bytes(R, SUPER, split) / 2);
    uint16_t* up = ws.take<uint16_t>(plane_set_bytes(C, C, split) / 2);
    MQ_REQUIRE(ep && up, MQ_ERR_WORKSPACE, "mq_gptq_sweep: workspace too small for the operand planes");
    err_set.base = ep; err_set.planes = split; err_set.rows_pad = (int)pad_rows(R); err_set.total_rows = err_set.rows_pad;
    err_set.K_pad = SUPER;
    // the lazy updates read Uhat[i1:i2, i2:]: only blocks strictly above the diagonal
    MQ_TRY(make_planes_f32(Uhat, 1, ldu, (int)C, (int)C, split, up, &u_set, st, true, col_div));
  }
  SweepArgs sa;
  sa.W = W; sa.ldw = ldw; sa.R = (int)R;
  sa.U = Uhat; sa.ldu = ldu;
  sa.scale = scale; sa.zero = zero; sa.group = group; sa.s_rs = s_rs; sa.s_gs = s_gs;
  sa.maxq = (float)((1 << bits) - 1);
  sa.zero_default = 0.5f * (float)(1 << bits);
  sa.codes = codes; sa.C = C;
  sa.packed = packed;
  sa.deq = deq; sa.err = err;
  MQ_TRY(engine_fault_word(&sa.fault));
  sa.Worig = Worig; sa.ldwo = ldwo;
  sa.err_planes = nullptr;
  sa.plane_stride = tensor ? err_set.total_rows * far : 0;
  sa.n_planes = half ? 2 : split;
  sa.err_ld = tensor ? (int)far : TILE;
  const bool uniform = group % SUB == 0;
  // Rows per CTA: the chain costs the same for 1 row and for 64, so a tile of 2048 rows takes 16.5 us on 148 SMs,
  // 17.4 on 74 and 19.0 on 48.  Alone, one CTA per SM; a caller with several layers in flight gives each
  // few SMs: eight streams, ms per layer with R / 148, R / 74, R / 44 and R / 22 rows per CTA (64 at most): 2048 x 7168 2.14, 1.79, 1.69
  // and 1.65, 7168 x 2048 0.528, 0.470, 0.470 and 0.474, 4096 x 4096 1.10, 0.94, 0.89 and 0.91.  Fewer than eight rows per CTA gain nothing.
  int rows = (int)ceil_div(R, compact ? 44 : 148);
  rows = rows < 8 ? 8 : (rows > MAX_ROWS ? MAX_ROWS : rows);
  const int64_t row_groups = ceil_div(R, rows);
  const int grid = (int)(row_groups < 148 ? row_groups : 148);

  const int64_t step = by_super ? SUPER : TILE;
  for (int64_t i1 = 0; i1 < C; i1 += step) {
    const int nb = (int)((C - i1) < step ? (C - i1) : step);
    {
      // The kernels stage their part of the factor before they wait for their predecessor: only a launch
      // that follows this loop's own update (which writes W, never the factor) may be chained.
      const bool chained = i1 > 0;
      // bytes the launch must move: W in, codes out, errors out, the triangle of Uhat once
      ProfScope prof(PROF_SWEEP_TILE, (double)R * nb * (4.0 + 1.0 + 4.0) + 2.0 * nb * nb, (double)R * nb * (nb - 1), st);
      sa.i1 = (int)i1; sa.nb = nb;
      if (tensor) sa.err_planes = err_set.base + (i1 % far);
      sa.row_f = half ? row_f + (i1 % far) / TILE * R : nullptr;
      if (by_super) {
        if (i1 + nb >= C) sa.err_planes = nullptr;   // nothing behind it
        MQ_TRY(sweep_super_block(chained, uniform, compact, out_dtype, sa, st));
      } else {
        switch (out_dtype) {
          case MQ_F32: MQ_TRY(launch_sweep_tile<MQ_F32>(chained, uniform, grid, rows, st, sa)); break;
          case MQ_BF16: MQ_TRY(launch_sweep_tile<MQ_BF16>(chained, uniform, grid, rows, st, sa)); break;
          default: MQ_TRY(launch_sweep_tile<MQ_F16>(chained, uniform, grid, rows, st, sa));
        }
      }
    }
    MQ_LAUNCH_CHECK();
    const int64_t i2 = i1 + nb;
    if (i2 >= C) break;
    if (!tensor) {
      GemmDesc g;
      g.A = err; g.a_rs = TILE; g.a_cs = 1;
      g.B = Uhat + i1 * ldu + i2; g.b_rs = ldu; g.b_cs = 1;
      g.C = W + i2; g.ldc = ldw;
      g.M = (int)R; g.N = (int)(C - i2); g.K = nb;
      g.alpha = 1.0f; g.beta = 1.0f;
      MQ_TRY(eng.gemm(g));
      continue;
    }
    const int64_t s0 = i1 / SUPER * SUPER;                        // first column of this super-block
    const int64_t s1 = (s0 + SUPER) < C ? (s0 + SUPER) : C;       // one past its last column
    if (i2 < s1) {
      // near: W[:, i2:s1] += E_tile Uhat[i1:i2, i2:s1]
      GemmDesc g;
      g.C = W + i2; g.ldc = ldw;
      g.M = (int)R; g.N = (int)(s1 - i2); g.K = nb;
      g.alpha = 1.0f; g.beta = 1.0f;
      g.compact = compact ? 1 : 0;
      g.all_products = all_products;
      g.row_f = sa.row_f; g.col_f = col_f ? col_f + i2 : nullptr;
      PlaneSet a = err_set, b = u_set;
      a.k0 = (int)(i1 % far);
      b.row0 = i2; b.k0 = (int)i1;
      MQ_TRY(gemm_tensor_planes(g, a, b, st));
    } else {
      // The super-block is done.  By itself: W[:, s1:] += E_super Uhat[s0:s1, s1:], all errors of the super-block in one contraction.
      // Where two go together, behind the first only the second takes its update, W[:, s1:f1] += E_super Uhat[s0:s1, s1:f1], and
      // everything behind both takes the errors of both: W[:, s1:] += E Uhat[f0:s1, s1:].
      const int64_t f0 = i1 / far * far, f1 = (f0 + far) < C ? (f0 + far) : C;
      const bool joint = far > SUPER && joint_update(ceil_div(R, 256) * ceil_div(C - f0 - SUPER, 256));
      const bool rest = joint && s1 < f1;
      const int64_t from = joint && !rest ? f0 : s0;
      GemmDesc g;
      g.C = W + s1; g.ldc = ldw;
      g.M = (int)R; g.N = (int)((rest ? f1 : C) - s1); g.K = (int)(s1 - from);
      g.alpha = 1.0f; g.beta = 1.0f;
      g.all_products = all_products;
      g.row_f = half ? row_f + (from - f0) / TILE * R : nullptr; g.row_f_step = R; g.col_f = col_f ? col_f + s1 : nullptr;
      PlaneSet a = err_set, b = u_set;
      a.k0 = (int)(from - f0);
      b.row0 = s1; b.k0 = (int)from;
      MQ_TRY(gemm_tensor_planes(g, a, b, st));
    }
  }
  return MQ_OK;
}

}  // namespace mq

extern "C" size_t mq_gptq_sweep_workspace_bytes(int64_t R, int64_t C, int math, int split) {
  if (R <= 0 || C <= 0) return 0;
  const size_t with_original = mq::sweep_workspace_bytes(R, C, math, split, true), without = mq::sweep_workspace_bytes(R, C, math, split, false);
  return with_original > without ? with_original : without;
}

extern "C" int mq_gptq_sweep(float* W, int64_t R, int64_t C, int64_t ldw, const float* Uhat, int64_t ldu,
                             const float* scale, const float* zero, int64_t group, int64_t row_stride,
                             int64_t group_stride, int bits, int out_dtype, uint8_t* codes, int32_t* packed, void* dequantized,
                             const float* W_original, int64_t ldwo, int math, int split, void* workspace,
                             size_t workspace_bytes, void* stream) {
  using namespace mq;
  MQ_REQUIRE(W && Uhat && scale && codes, MQ_ERR_ARGUMENT, "mq_gptq_sweep: null pointer");
  MQ_REQUIRE(R > 0 && C > 0 && ldw >= C && ldu >= C, MQ_ERR_ARGUMENT, "mq_gptq_sweep: bad shape R=%lld C=%lld ldw=%lld ldu=%lld",
             (long long)R, (long long)C, (long long)ldw, (long long)ldu);
  MQ_REQUIRE(group > 0 && C % group == 0, MQ_ERR_ARGUMENT, "mq_gptq_sweep: group %lld does not divide C=%lld", (long long)group,
             (long long)C);
  MQ_REQUIRE(bits >= 2 && bits <= 8, MQ_ERR_ARGUMENT, "mq_gptq_sweep: bits=%d", bits);
  MQ_REQUIRE(valid_dtype(out_dtype), MQ_ERR_ARGUMENT, "mq_gptq_sweep: bad dtype %d", out_dtype);
  MQ_REQUIRE(C % 8 == 0, MQ_ERR_UNSUPPORTED, "mq_gptq_sweep: C=%lld must be a multiple of 8", (long long)C);
  MQ_REQUIRE(ldw % 4 == 0 && ldu % 4 == 0 && aligned(W, 16) && aligned(Uhat, 16) && aligned(codes, 4), MQ_ERR_ALIGNMENT,
             "mq_gptq_sweep: W/Uhat need 16-byte alignment and leading dimensions that are multiples of 4");
  MQ_REQUIRE((math & ~MQ_MATH_COMPACT) == MQ_MATH_FP32 || (math & ~MQ_MATH_COMPACT) == MQ_MATH_TENSOR, MQ_ERR_ARGUMENT,
             "mq_gptq_sweep: bad math %d", math);
  Workspace ws(workspace, workspace_bytes);
  if (W_original) {
    MQ_REQUIRE(ldwo >= C && ldwo % 4 == 0 && aligned(W_original, 16) && W_original != W, MQ_ERR_ALIGNMENT,
               "mq_gptq_sweep: W_original must be a separate 16-byte aligned matrix with ldwo %% 4 == 0");
  }
  MQ_REQUIRE(!packed || (bits == 4 && !zero && aligned(packed, 4)), MQ_ERR_UNSUPPORTED,
             "mq_gptq_sweep: packed words need bits == 4, the symmetric zero point and a 4-byte aligned buffer");
  return gptq_sweep(W, R, C, ldw, Uhat, ldu, scale, zero, group, row_stride, group_stride, bits, out_dtype, codes,
                    dequantized, W_original, ldwo, math, split, ws, static_cast<cudaStream_t>(stream), nullptr, nullptr, false, packed);
}
