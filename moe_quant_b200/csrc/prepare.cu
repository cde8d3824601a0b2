// Hessian preparation (NaN guard, dead channels, zero-column masking, damping)
// and the symmetric absmax grid.  All of it is one or two passes over H / W, i.e.
// HBM-bound, and everything stays on the device: no host round trip for the
// `.any().item()` of the reference (src/gptq.py:141).
#include "engine.cuh"

namespace mq {

int launch_to_fp32(const void* src, int dtype, float* dst, int64_t n, cudaStream_t st);

// ---------------------------------------------------------------- NaN guard
__global__ void __launch_bounds__(256) nan_scan_kernel(const float* __restrict__ H, int64_t C, int64_t ldh,
                                                       mq_layer_flags* flags) {
  // C % 4 == 0 and ldh % 4 == 0 (checked on the host): rows are float4-addressable.  A thread
  // keeps its column and walks rows, four independent loads per step, no index division.
  const int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  bool bad = false;
  if (c < C) {
    const float* col = H + c;
    int64_t r = blockIdx.y;
    for (; r + 3 * (int64_t)gridDim.y < C; r += 4 * (int64_t)gridDim.y) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = __ldg(reinterpret_cast<const float4*>(col + (r + u * (int64_t)gridDim.y) * ldh));
#pragma unroll
      for (int u = 0; u < 4; ++u) bad |= (v[u].x != v[u].x) | (v[u].y != v[u].y) | (v[u].z != v[u].z) | (v[u].w != v[u].w);
    }
    for (; r < C; r += gridDim.y) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(col + r * ldh));
      bad |= (v.x != v.x) | (v.y != v.y) | (v.z != v.z) | (v.w != v.w);
    }
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0) atomicExch(&flags->nan_hessian, 1);
}

// Also clears the column flags (may be null) for the pass over the weights that follows.
__global__ void __launch_bounds__(256) identity_if_nan_kernel(float* __restrict__ H, int64_t C, int64_t ldh,
                                                              const mq_layer_flags* flags, int* __restrict__ nonzero) {
  int64_t n = C * C;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  if (nonzero)
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < C; i += stride) nonzero[i] = 0;
  if (flags->nan_hessian == 0) return;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    int64_t r = i / C, c = i - r * C;
    H[r * ldh + c] = (r == c) ? 1.0f : 0.0f;
  }
}

// ---------------------------------------------------------------- column masks
// nonzero[c] = 1 when any W[r, c] != 0.  Threads of a warp read consecutive columns.
__global__ void __launch_bounds__(256) column_nonzero_kernel(const float* __restrict__ W, int64_t R, int64_t C,
                                                             int64_t ldw, int rows_per_block,
                                                             int* __restrict__ nonzero) {
  int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  int64_t r0 = (int64_t)blockIdx.y * rows_per_block;
  int64_t r1 = r0 + rows_per_block < R ? r0 + rows_per_block : R;
  bool nz = false;
  for (int64_t r = r0; r < r1; ++r) nz |= (__ldg(W + r * ldw + c) != 0.0f);
  if (nz) nonzero[c] = 1;
}

// One block, everything that happens on the diagonal: lists the masked channels (diag(H)==0, or an all-zero weight
// column; list[0] = count, list[1..] = channel indices in any order), sets their diagonal to 1, adds
// rel_damp * mean(diag H) and, where eq is given, computes the equilibration of the damped diagonal
// (equilibrating_power); eq[C] is the smallest factor.
// The diagonal is read once, DIAG_KEEP values per thread in flight: with a pass per purpose (list, damping,
// equilibration) the three took 12 + 16 + 3 us at 7168 channels, all of it memory latency.
constexpr int DIAG_THREADS_PREP = 1024, DIAG_KEEP = 8;

__global__ void __launch_bounds__(DIAG_THREADS_PREP) diagonal_kernel(float* __restrict__ H, int64_t C, int64_t ldh,
                                                                     const int* __restrict__ nonzero, int* __restrict__ list,
                                                                     float rel_damp, float* __restrict__ eq, mq_layer_flags* flags) {
  __shared__ int n_masked, n_dead, n_zero, least;
  __shared__ float partial[32];
  __shared__ float damp_s;
  if (threadIdx.x == 0) { n_masked = n_dead = n_zero = 0; least = 0x7f7f7f7f; }
  __syncthreads();
  float acc = 0.0f, kept[DIAG_KEEP];
  for (int64_t c0 = threadIdx.x; c0 < C; c0 += (int64_t)DIAG_KEEP * DIAG_THREADS_PREP) {
    float h[DIAG_KEEP];
    int nz[DIAG_KEEP];
#pragma unroll
    for (int u = 0; u < DIAG_KEEP; ++u) {
      const int64_t c = c0 + (int64_t)u * DIAG_THREADS_PREP;
      h[u] = c < C ? H[c * ldh + c] : 0.0f;
      nz[u] = (c < C && nonzero != nullptr) ? nonzero[c] : 1;
    }
#pragma unroll
    for (int u = 0; u < DIAG_KEEP; ++u) {
      const int64_t c = c0 + (int64_t)u * DIAG_THREADS_PREP;
      if (c >= C) continue;
      // The reference zeroes W[:, dead] before looking for all-zero columns, so a dead
      // channel is always also a zero column (src/gptq.py:145-152, 224).
      const bool dead = h[u] == 0.0f;
      if (dead) atomicAdd(&n_dead, 1);
      if (dead || nz[u] == 0) {
        atomicAdd(&n_zero, 1);
        list[1 + atomicAdd(&n_masked, 1)] = (int)c;
        h[u] = 1.0f;
      }
      acc += h[u];
      if (c0 == threadIdx.x) kept[u] = h[u];
      else H[c * ldh + c] = h[u];                  // beyond the kept ones: written now, read again below
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) partial[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < (blockDim.x >> 5) ? partial[threadIdx.x] : 0.0f;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) {
      damp_s = rel_damp * (v / (float)C);
      list[0] = n_masked;
      flags->dead_channels = n_dead;
      flags->zero_columns = n_zero;
    }
  }
  __syncthreads();
  const float damp = damp_s;
  int mine = 0x7f7f7f7f;
  auto finish = [&](int64_t c, float h) {
    h += damp;
    H[c * ldh + c] = h;
    if (eq) {
      const float e = equilibrating_power(h);
      eq[c] = e;
      mine = min(mine, __float_as_int(e));         // positive floats order like their bits
    }
  };
#pragma unroll
  for (int u = 0; u < DIAG_KEEP; ++u) {
    const int64_t c = threadIdx.x + (int64_t)u * DIAG_THREADS_PREP;
    if (c < C) finish(c, kept[u]);
  }
  for (int64_t c = threadIdx.x + (int64_t)DIAG_KEEP * DIAG_THREADS_PREP; c < C; c += DIAG_THREADS_PREP) finish(c, H[c * ldh + c]);
  if (eq) {
    atomicMin(&least, mine);
    __syncthreads();
    if (threadIdx.x == 0) eq[C] = __int_as_float(least);
  }
}

// Rows and columns of the masked channels become those of the identity (the diagonal is
// diagonal_kernel's); their weight column becomes zero.
__global__ void __launch_bounds__(256) apply_mask_kernel(float* __restrict__ H, int64_t C, int64_t ldh,
                                                         float* __restrict__ W, int64_t R, int64_t ldw,
                                                         const int* __restrict__ list) {
  int n_masked = list[0];
  if (n_masked == 0) return;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int k = 0; k < n_masked; ++k) {
    int64_t c = list[1 + k];
    for (int64_t i = tid; i < C; i += stride) {
      if (i == c) continue;
      H[c * ldh + i] = 0.0f;
      H[i * ldh + c] = 0.0f;
    }
    if (W != nullptr) {
      for (int64_t r = tid; r < R; r += stride) W[r * ldw + c] = 0.0f;
    }
  }
}

// ---------------------------------------------------------------- absmax grid
// One warp walks one (row, group) segment at a time with float4 loads.
template <int DT>
__global__ void __launch_bounds__(256) absmax_scales_kernel(const float* __restrict__ W, int64_t R, int64_t C,
                                                            int64_t ldw, int64_t group, float two_over_maxq,
                                                            float* __restrict__ scale) {
  int64_t G = C / group;
  int64_t n_seg = R * G;
  int lane = threadIdx.x & 31;
  int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t seg = warp; seg < n_seg; seg += n_warps) {
    int64_t r = seg / G, gi = seg - r * G;
    const float* p = W + r * ldw + gi * group;
    float m = 0.0f;
    if ((group & 3) == 0) {
      for (int64_t k = lane * 4; k < group; k += 128) {
        float4 v = __ldg(reinterpret_cast<const float4*>(p + k));
        m = fmaxf(m, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
      }
    } else {
      for (int64_t k = lane; k < group; k += 32) m = fmaxf(m, fabsf(__ldg(p + k)));
    }
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) {
      // (2/maxq) * absmax, then + 1e-12, each rounded to fp32, then through the layer dtype:
      // the operation order of src/quant_utils.py:95-96.
      float s = __fadd_rn(__fmul_rn(two_over_maxq, m), 1e-12f);
      scale[seg] = round_through<DT>(s);
    }
  }
}

// ---------------------------------------------------------------- MSE scale search
// One warp per (row, group): the absmax scale s0 is shrunk by each candidate factor p_i,
//   s_i = round_to_dtype(s0 * p_i),  loss_i = sum_c |dequant(quant(x_c; s_i)) - x_c|^norm,
// and replaced by s0 * p_argmin rounded through the dtype (mse_scale_triton_kernel,
// src/quant_utils.py:104-139).  |d|^norm is exp(norm * log|d|) as in tl_pow (src/quant_utils.py:25-27),
// which is 0 for d == 0.  Of equal losses the first candidate wins; candidates with equal losses
// almost always have equal rounded scales, so the choice among them does not change the result.
//
// What bounds it is the number of (element, candidate) terms: two special-function operations and
// about fifteen fp32 operations each.  Three things keep that number and the cost of a term down,
// none of which changes a loss that decides anything:
//  * every term is non-negative and fp32 addition is monotone, so a candidate whose largest terms
//    alone reach the best loss so far cannot win.  The terms of the segment's largest and smallest
//    element, which the shrunk grids clip, are computed for 32 candidates at a time (one candidate
//    per lane); two thirds of the 100 candidates of a 128-wide group fall to them.  mse_scales_wide_kernel
//    compares the partial sum every eight elements per lane instead.
//  * the elements of a 32-, 64- or 128-wide group stay in registers over all candidates.
//  * x / s goes through the reciprocal of s, which the whole warp shares, and one residual correction
//    (Markstein 1990); scales so small or large that the residual could underflow keep the division.
// 7168 x 2048 bf16, groups of 128, 100 candidates: 2826 us before, about 715 us now (4394 -> 1951 us for the whole quantize call).
template <int DT>
__device__ __forceinline__ float mse_term(float x, float s, float rs, bool plain, float zero, float maxq, float norm) {
  float d;
  if (plain) {
    d = x * rs;
    d = fmaf(fmaf(-s, d, x), rs, d);
  } else {
    d = __fdiv_rn(x, s);
  }
  // clamp first, then floor (the bounds are whole numbers, so the order does not matter; NaN becomes 0
  // either way): adding 2^23 with rounding towards minus infinity leaves the whole part
  const float v = fminf(fmaxf(__fadd_rn(__fadd_rn(d, zero), 0.5f), 0.0f), maxq);
  const float q = __fadd_rd(v, 8388608.0f) - 8388608.0f;
  const float y = round_through<DT>(__fmul_rn(q - zero, s));
  return __expf(__logf(fabsf(y - x)) * norm);
}

// EPL: elements per lane of a group of 32 * EPL columns, held in registers; 0: any group.
template <int DT, int EPL>
__global__ void __launch_bounds__(256) mse_scales_kernel(const float* __restrict__ W, int64_t R, int64_t C, int64_t ldw,
                                                         int64_t group, float maxq, float zero,
                                                         const float* __restrict__ p, int p_size, float norm,
                                                         float* __restrict__ scale) {
  const int64_t G = C / group;
  const int64_t n_seg = R * G;
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t seg = warp; seg < n_seg; seg += n_warps) {
    const int64_t r = seg / G, gi = seg - r * G;
    const float* x = W + r * ldw + gi * group;
    const float s0 = scale[seg];
    float xr[EPL > 0 ? EPL : 1];
    float hi = -INFINITY, lo = INFINITY;
    if constexpr (EPL > 0) {
#pragma unroll
      for (int e = 0; e < EPL; ++e) {
        xr[e] = __ldg(x + lane + 32 * e);
        hi = fmaxf(hi, xr[e]);
        lo = fminf(lo, xr[e]);
      }
    } else {
      for (int64_t k = lane; k < group; k += 32) {
        const float xv = __ldg(x + k);
        hi = fmaxf(hi, xv);
        lo = fminf(lo, xv);
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    }
    float best = 0.0f;
    int best_i = -1;
    for (int i0 = 0; i0 < p_size; i0 += 32) {
      // A lower bound of candidate i0 + lane's loss.  The two terms may be summed in another order than in
      // the loss itself: the factor is far below the rounding of any sum over a row.  (A group of one
      // element has one term; an all-NaN segment leaves +-inf here, whose terms compare as NaN.)
      float bound = INFINITY, s_lane = 1.0f, rs_lane = 1.0f;
      if (i0 + lane < p_size) {
        s_lane = round_through<DT>(__fmul_rn(s0, __ldg(p + i0 + lane)));
        rs_lane = 1.0f / s_lane;
        const bool plain = s_lane > 1e-18f && s_lane < 1e18f;
        const float a = mse_term<DT>(hi, s_lane, rs_lane, plain, zero, maxq, norm);
        const float b = mse_term<DT>(lo, s_lane, rs_lane, plain, zero, maxq, norm);
        bound = hi != lo ? (a + b) * 0.9995f : a;
      }
      unsigned alive = __ballot_sync(0xffffffffu, bound < best);
      if (best_i < 0) alive = __ballot_sync(0xffffffffu, i0 + lane < p_size);
      while (alive) {
        const int j = __ffs(alive) - 1;
        alive &= alive - 1;
        const int i = i0 + j;
        const float s = __shfl_sync(0xffffffffu, s_lane, j), rs = __shfl_sync(0xffffffffu, rs_lane, j);
        const bool plain = s > 1e-18f && s < 1e18f;
        float loss = 0.0f;
        if constexpr (EPL > 0) {
#pragma unroll
          for (int e = 0; e < EPL; ++e) loss += mse_term<DT>(xr[e], s, rs, plain, zero, maxq, norm);
        } else {
          for (int64_t k = lane; k < group; k += 32) loss += mse_term<DT>(__ldg(x + k), s, rs, plain, zero, maxq, norm);
        }
        for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
        if (best_i < 0 || loss < best) {
          best = loss;
          best_i = i;
          alive &= __ballot_sync(0xffffffffu, bound < best);
        }
      }
    }
    if (lane == 0 && best_i >= 0) scale[seg] = round_through<DT>(__fmul_rn(s0, __ldg(p + best_i)));
  }
}

// A CTA per (row, group), its warps share out the candidates (mse_by_ctas: few or very wide groups).  Every warp takes candidate 0
// first, so that all start from the same best; a candidate's loss is summed by one warp in the order of the kernel above.  Of
// equal losses the first candidate wins.
template <int DT>
__global__ void __launch_bounds__(256) mse_scales_wide_kernel(const float* __restrict__ W, int64_t R, int64_t C, int64_t ldw, int64_t group,
                                                              float maxq, float zero, const float* __restrict__ p, int p_size, float norm,
                                                              float* __restrict__ scale) {
  __shared__ int shared_best;          // bits of the smallest loss so far: non-negative floats order like them
  __shared__ float w_best[8];
  __shared__ int w_index[8];
  const int64_t G = C / group, n_seg = R * G;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t seg = blockIdx.x; seg < n_seg; seg += gridDim.x) {
    const int64_t r = seg / G, gi = seg - r * G;
    const float* x = W + r * ldw + gi * group;
    const float s0 = scale[seg];
    if (threadIdx.x == 0) shared_best = 0x7f800000;
    __syncthreads();
    float best = 0.0f;
    int best_i = 0;
    // i = 0 for every warp, then warp + 1, warp + 9, ...
    for (int i = 0; i < p_size; i = i == 0 ? warp + 1 : i + 8) {
      const float s = round_through<DT>(__fmul_rn(s0, __ldg(p + i)));
      const float rs = 1.0f / s;
      const bool plain = s > 1e-18f && s < 1e18f;
      float loss = 0.0f;
      bool beaten = false;
      for (int64_t k0 = 0; k0 < group; k0 += 256) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int64_t k = k0 + u * 32 + lane;
          if (k < group) loss += mse_term<DT>(__ldg(x + k), s, rs, plain, zero, maxq, norm);
        }
        if (i > 0 && k0 + 256 < group) {
          float part = loss;
          for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
          // another warp's best may belong to a later candidate: only a larger loss is out for certain
          beaten = part >= best || part > __int_as_float(*reinterpret_cast<volatile int*>(&shared_best));
          beaten = __any_sync(0xffffffffu, beaten);
          if (beaten) break;
        }
      }
      if (beaten) continue;
      for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
      if (i == 0 || loss < best) {
        best = loss;
        best_i = i;
        if (lane == 0 && loss >= 0.0f) atomicMin(&shared_best, __float_as_int(loss));
      }
    }
    if (lane == 0) { w_best[warp] = best; w_index[warp] = best_i; }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 0; w < 8; ++w)
        if (w_best[w] < best || (w_best[w] == best && w_index[w] < best_i)) { best = w_best[w]; best_i = w_index[w]; }
      scale[seg] = round_through<DT>(__fmul_rn(s0, __ldg(p + best_i)));
    }
    __syncthreads();
  }
}

// A warp per segment needs about 0.28 us per column of the group however few there are, and its 64 warps per SM then finish
// together; the bound of the two extreme elements drops most candidates of a narrow group.  A CTA per segment shortens the
// serial stream, and its partial sums drop candidates of a wide group, where two elements say little.  The search alone, bf16, us by
// warps / by CTAs:
//   group  256:  1792 segments   86 / 109   4736  107 /  236    57344   900 / 2589
//   group  512:   896           141 /  99   2368  146 /  183    28672  1035 / 1891
//   group 1024:  1184           289 / 163   2960  357 /  356    14336  1214 / 1610
//   group 1536:  4096           755 / 685  16384 2192 / 2728
//   group 2048:  3072           852 / 655   7168 1710 / 1556    16384  3210 / 3604
//   group 4096:   500          1457 / 321   8192 5338 / 3689    16384 10328 / 7162
// The line lies at 1300 segments, and from 684 columns on at a number that grows with the square of the width.
inline bool mse_by_ctas(int64_t n_seg, int64_t group) { return group >= 256 && (n_seg < 1300 || n_seg < group * group / 360); }

template <int DT>
void launch_mse_scales(int grid, cudaStream_t st, const float* W, int64_t R, int64_t C, int64_t ldw, int64_t group, float maxq, float zero,
                       const float* p, int p_size, float norm, float* scale) {
  if (group == 128) mse_scales_kernel<DT, 4><<<grid, 256, 0, st>>>(W, R, C, ldw, group, maxq, zero, p, p_size, norm, scale);
  else if (group == 64) mse_scales_kernel<DT, 2><<<grid, 256, 0, st>>>(W, R, C, ldw, group, maxq, zero, p, p_size, norm, scale);
  else if (group == 32) mse_scales_kernel<DT, 1><<<grid, 256, 0, st>>>(W, R, C, ldw, group, maxq, zero, p, p_size, norm, scale);
  else if (const int64_t n_seg = R * (C / group); mse_by_ctas(n_seg, group)) {
    mse_scales_wide_kernel<DT><<<(unsigned)(n_seg < 148 * 8 ? n_seg : 148 * 8), 256, 0, st>>>(W, R, C, ldw, group, maxq, zero, p, p_size, norm, scale);
  } else mse_scales_kernel<DT, 0><<<grid, 256, 0, st>>>(W, R, C, ldw, group, maxq, zero, p, p_size, norm, scale);
}

// ---------------------------------------------------------------- the weights' way in
// One pass over the layer's weights: two fp32 copies (original and running), columns of dead channels (diag(H)==0,
// hdiag given) zeroed, flags of the columns that hold a non-zero, and the absmax scales of groups of 32,
// 64 or 128 columns (GROUP_LANES = lanes of 4 columns per group; 0: none).  A warp takes 128 columns of
// eight rows, four rows in flight.  As separate passes (conversion, column flags, absmax, copy) the same took
// 14 + 16 + 27 + 20 us for 2048 x 7168; the scales of 64-wide groups, half of whose warps' lanes idled, 49.
template <typename S, int GROUP_LANES>
__global__ void __launch_bounds__(256) weights_in_kernel(const S* __restrict__ src, int64_t R, int64_t C, float* __restrict__ run,
                                                         float* __restrict__ orig, const float* __restrict__ H, int64_t ldh,
                                                         int* __restrict__ nonzero, float two_over_maxq, int out_dtype,
                                                         float* __restrict__ scale) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t c = (int64_t)blockIdx.x * 128 + lane * 4;
  const bool in = c < C;   // C % 8 == 0: a lane is in or out as a whole; one that is out only takes part in the shuffles
  bool dead[4] = {false, false, false, false};
  if (H != nullptr && in) {
#pragma unroll
    for (int q = 0; q < 4; ++q) dead[q] = __ldg(H + (c + q) * (ldh + 1)) == 0.0f;
  }
  bool nz[4] = {false, false, false, false};
  const int64_t r_end = ((int64_t)blockIdx.y + 1) * 64 < R ? ((int64_t)blockIdx.y + 1) * 64 : R;
  for (int64_t r0 = (int64_t)blockIdx.y * 64 + warp * 8; r0 < r_end && r0 < (int64_t)blockIdx.y * 64 + warp * 8 + 8; r0 += 4) {
    float v[4][4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const S* p = src + (r0 + u) * C + c;
      const bool ok = in && r0 + u < r_end;
      if constexpr (sizeof(S) == 4) {
        const float4 x = ok ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[u][0] = x.x; v[u][1] = x.y; v[u][2] = x.z; v[u][3] = x.w;
      } else {
        union { uint2 w; S t[4]; } x;
        x.w = ok ? __ldg(reinterpret_cast<const uint2*>(p)) : make_uint2(0u, 0u);
#pragma unroll
        for (int q = 0; q < 4; ++q) v[u][q] = to_float(x.t[q]);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int64_t r = r0 + u;
      float m = 0.0f;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        nz[q] |= v[u][q] != 0.0f;
        if (dead[q]) v[u][q] = 0.0f;
        m = fmaxf(m, fabsf(v[u][q]));
      }
      if (r >= r_end) break;   // uniform in the warp
      if (in) {
        const float4 o = make_float4(v[u][0], v[u][1], v[u][2], v[u][3]);
        *reinterpret_cast<float4*>(run + r * C + c) = o;
        *reinterpret_cast<float4*>(orig + r * C + c) = o;
      }
      if constexpr (GROUP_LANES > 0) {
#pragma unroll
        for (int o = GROUP_LANES / 2; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (in && (lane & (GROUP_LANES - 1)) == 0) {
          const float s = __fadd_rn(__fmul_rn(two_over_maxq, m), 1e-12f);   // as in absmax_scales_kernel
          scale[r * (C / (4 * GROUP_LANES)) + c / (4 * GROUP_LANES)] =
              out_dtype == MQ_BF16 ? round_through<MQ_BF16>(s) : out_dtype == MQ_F16 ? round_through<MQ_F16>(s) : s;
        }
      }
    }
  }
  if (nonzero != nullptr && in) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (nz[q]) nonzero[c + q] = 1;
  }
}

template <typename S>
static int launch_weights_in(const void* src, int dtype, int64_t R, int64_t C, float* run, float* orig, const float* H, int64_t ldh,
                             int* nonzero, int64_t group, int bits, float* scale, cudaStream_t st) {
  const dim3 grid((unsigned)ceil_div(C, 128), (unsigned)ceil_div(R, 64));
  const float f = 2.0f / (float)((1 << bits) - 1);
  const S* p = static_cast<const S*>(src);
  switch (group) {
    case 32: weights_in_kernel<S, 8><<<grid, 256, 0, st>>>(p, R, C, run, orig, H, ldh, nonzero, f, dtype, scale); break;
    case 64: weights_in_kernel<S, 16><<<grid, 256, 0, st>>>(p, R, C, run, orig, H, ldh, nonzero, f, dtype, scale); break;
    case 128: weights_in_kernel<S, 32><<<grid, 256, 0, st>>>(p, R, C, run, orig, H, ldh, nonzero, f, dtype, scale); break;
    default: weights_in_kernel<S, 0><<<grid, 256, 0, st>>>(p, R, C, run, orig, H, ldh, nonzero, f, dtype, scale);
  }
  MQ_LAUNCH_CHECK();
  return MQ_OK;
}

// The layer's weights -> both fp32 copies and the scales.  H, nonzero: see weights_in_kernel (null for a tied layer).
int weights_in(const void* src, int dtype, int64_t R, int64_t C, float* run, float* orig, const float* H, int64_t ldh, int* nonzero,
               int64_t group, int bits, float* scale, cudaStream_t st) {
  // a weight view that starts off a 4-element boundary goes through an aligned copy of itself
  const bool vec = aligned(src, dtype == MQ_F32 ? 16 : 8);
  if (!vec) {
    MQ_TRY(launch_to_fp32(src, dtype, orig, R * C, st));
    MQ_TRY(launch_weights_in<float>(orig, dtype, R, C, run, orig, H, ldh, nonzero, group, bits, scale, st));
  } else {
    switch (dtype) {
      case MQ_F32: MQ_TRY(launch_weights_in<float>(src, dtype, R, C, run, orig, H, ldh, nonzero, group, bits, scale, st)); break;
      case MQ_BF16: MQ_TRY(launch_weights_in<__nv_bfloat16>(src, dtype, R, C, run, orig, H, ldh, nonzero, group, bits, scale, st)); break;
      default: MQ_TRY(launch_weights_in<__half>(src, dtype, R, C, run, orig, H, ldh, nonzero, group, bits, scale, st));
    }
  }
  if (group != 32 && group != 64 && group != 128) MQ_TRY(mq_absmax_scales(run, R, C, C, group, bits, dtype, scale, st));
  return MQ_OK;
}

// ---------------------------------------------------------------- fp32 working copy
template <typename T>
__global__ void __launch_bounds__(256) to_fp32_kernel(const T* __restrict__ src, float* __restrict__ dst, int64_t n) {
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) dst[i] = to_float(src[i]);
}

int launch_to_fp32(const void* src, int dtype, float* dst, int64_t n, cudaStream_t st) {
  if (n == 0) return MQ_OK;
  int grid = (int)(ceil_div(n, 256) < 148 * 8 ? ceil_div(n, 256) : 148 * 8);
  switch (dtype) {
    case MQ_F32:
      MQ_CUDA(cudaMemcpyAsync(dst, src, n * sizeof(float), cudaMemcpyDeviceToDevice, st));
      return MQ_OK;
    case MQ_BF16:
      to_fp32_kernel<<<grid, 256, 0, st>>>(static_cast<const __nv_bfloat16*>(src), dst, n);
      break;
    case MQ_F16:
      to_fp32_kernel<<<grid, 256, 0, st>>>(static_cast<const __half*>(src), dst, n);
      break;
    default:
      set_error("bad dtype %d", dtype);
      return MQ_ERR_ARGUMENT;
  }
  MQ_LAUNCH_CHECK();
  return MQ_OK;
}

}  // namespace mq

namespace mq {

// Flags cleared, NaN guard, column flags (may be null) cleared.
int scan_hessian(float* H, int64_t C, int64_t ldh, int* nonzero, mq_layer_flags* flags, cudaStream_t st) {
  MQ_CUDA(cudaMemsetAsync(flags, 0, sizeof(mq_layer_flags), st));
  const unsigned gx = (unsigned)ceil_div(C / 4, 256);
  unsigned gy = (unsigned)(148 * 8 / gx);
  if (gy < 1) gy = 1;
  if ((int64_t)gy > C) gy = (unsigned)C;
  nan_scan_kernel<<<dim3(gx, gy), 256, 0, st>>>(H, C, ldh, flags);
  MQ_LAUNCH_CHECK();
  identity_if_nan_kernel<<<148 * 4, 256, 0, st>>>(H, C, ldh, flags, nonzero);
  MQ_LAUNCH_CHECK();
  return MQ_OK;
}

int mask_and_damp(float* H, int64_t C, int64_t ldh, float* W, int64_t R, int64_t ldw, const int* nonzero, int* list, float rel_damp,
                  float* eq, mq_layer_flags* flags, cudaStream_t st) {
  diagonal_kernel<<<1, DIAG_THREADS_PREP, 0, st>>>(H, C, ldh, nonzero, list, rel_damp, eq, flags);
  MQ_LAUNCH_CHECK();
  apply_mask_kernel<<<148, 256, 0, st>>>(H, C, ldh, W, R, ldw, list);
  MQ_LAUNCH_CHECK();
  return MQ_OK;
}

// The whole preparation of a layer: H masked and damped, eq (may be null) its equilibration, the weights as two
// fp32 copies and the scales.
int prepare_layer(const void* Wsrc, int dtype, int64_t R, int64_t C, float* run, float* orig, float* H, int64_t ldh, int64_t group, int bits,
                  float rel_damp, float* scale, float* eq, mq_layer_flags* flags, void* prep, cudaStream_t st) {
  int* nonzero = static_cast<int*>(prep);
  int* list = nonzero + align_up((size_t)C * sizeof(int), 256) / sizeof(int);
  MQ_TRY(scan_hessian(H, C, ldh, nonzero, flags, st));
  MQ_TRY(weights_in(Wsrc, dtype, R, C, run, orig, H, ldh, nonzero, group, bits, scale, st));
  return mask_and_damp(H, C, ldh, nullptr, R, C, nonzero, list, rel_damp, eq, flags, st);
}

}  // namespace mq

extern "C" size_t mq_hessian_prepare_workspace_bytes(int64_t C) {
  if (C < 0) return 0;
  // nonzero[C] + list[1 + C], each rounded up to 256 bytes
  return mq::align_up((size_t)C * sizeof(int), 256) + mq::align_up((size_t)(C + 1) * sizeof(int), 256);
}

extern "C" int mq_hessian_prepare(float* H, int64_t C, int64_t ldh, float* W, int64_t R, int64_t ldw, float rel_damp,
                                  mq_layer_flags* flags, void* workspace, size_t workspace_bytes, void* stream) {
  using namespace mq;
  MQ_REQUIRE(H && flags, MQ_ERR_ARGUMENT, "mq_hessian_prepare: null H or flags");
  MQ_REQUIRE(C > 0 && ldh >= C, MQ_ERR_ARGUMENT, "mq_hessian_prepare: bad C=%lld ldh=%lld", (long long)C, (long long)ldh);
  MQ_REQUIRE(C % 4 == 0 && ldh % 4 == 0 && aligned(H, 16), MQ_ERR_ALIGNMENT,
             "mq_hessian_prepare: needs C %% 4 == 0, ldh %% 4 == 0 and a 16-byte aligned H");
  if (W) MQ_REQUIRE(R > 0 && ldw >= C, MQ_ERR_ARGUMENT, "mq_hessian_prepare: bad R=%lld ldw=%lld", (long long)R, (long long)ldw);
  Workspace ws(workspace, workspace_bytes);
  int* nonzero = ws.take<int>(C);
  int* list = ws.take<int>(C + 1);
  MQ_REQUIRE(nonzero && list, MQ_ERR_WORKSPACE, "mq_hessian_prepare: workspace of %zu bytes is too small", workspace_bytes);
  cudaStream_t st = static_cast<cudaStream_t>(stream);

  MQ_TRY(scan_hessian(H, C, ldh, W ? nonzero : nullptr, flags, st));
  if (W) {
    const int rows_per_block = 64;
    dim3 grid((unsigned)ceil_div(C, 256), (unsigned)ceil_div(R, rows_per_block));
    column_nonzero_kernel<<<grid, 256, 0, st>>>(W, R, C, ldw, rows_per_block, nonzero);
    MQ_LAUNCH_CHECK();
  }
  return mask_and_damp(H, C, ldh, W, R, ldw, W ? nonzero : nullptr, list, rel_damp, nullptr, flags, st);
}

extern "C" int mq_absmax_scales(const float* W, int64_t R, int64_t C, int64_t ldw, int64_t group, int bits,
                                int out_dtype, float* scale, void* stream) {
  using namespace mq;
  MQ_REQUIRE(W && scale, MQ_ERR_ARGUMENT, "mq_absmax_scales: null pointer");
  MQ_REQUIRE(R > 0 && C > 0 && ldw >= C, MQ_ERR_ARGUMENT, "mq_absmax_scales: bad shape R=%lld C=%lld ldw=%lld",
             (long long)R, (long long)C, (long long)ldw);
  MQ_REQUIRE(group > 0 && C % group == 0, MQ_ERR_ARGUMENT, "mq_absmax_scales: group %lld does not divide C=%lld",
             (long long)group, (long long)C);
  MQ_REQUIRE(bits >= 2 && bits <= 8, MQ_ERR_ARGUMENT, "mq_absmax_scales: bits=%d", bits);
  MQ_REQUIRE(valid_dtype(out_dtype), MQ_ERR_ARGUMENT, "mq_absmax_scales: bad dtype %d", out_dtype);
  if (group % 4 == 0) {
    MQ_REQUIRE(aligned(W, 16) && ldw % 4 == 0, MQ_ERR_ALIGNMENT, "mq_absmax_scales: W must be 16-byte aligned with ldw %% 4 == 0");
  }
  float two_over_maxq = 2.0f / (float)((1 << bits) - 1);
  int64_t n_seg = R * (C / group);
  int grid = (int)(ceil_div(n_seg, 8) < 148 * 8 ? ceil_div(n_seg, 8) : 148 * 8);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (out_dtype) {
    case MQ_F32:
      absmax_scales_kernel<MQ_F32><<<grid, 256, 0, st>>>(W, R, C, ldw, group, two_over_maxq, scale);
      break;
    case MQ_BF16:
      absmax_scales_kernel<MQ_BF16><<<grid, 256, 0, st>>>(W, R, C, ldw, group, two_over_maxq, scale);
      break;
    default:
      absmax_scales_kernel<MQ_F16><<<grid, 256, 0, st>>>(W, R, C, ldw, group, two_over_maxq, scale);
  }
  MQ_LAUNCH_CHECK();
  return MQ_OK;
}

extern "C" int mq_mse_scales(const float* W, int64_t R, int64_t C, int64_t ldw, int64_t group, int bits, int out_dtype,
                             const float* shrink, int n_shrink, float norm, float* scale, void* stream) {
  using namespace mq;
  MQ_REQUIRE(W && scale && shrink, MQ_ERR_ARGUMENT, "mq_mse_scales: null pointer");
  MQ_REQUIRE(R > 0 && C > 0 && ldw >= C && n_shrink > 0, MQ_ERR_ARGUMENT, "mq_mse_scales: bad shape R=%lld C=%lld ldw=%lld n=%d",
             (long long)R, (long long)C, (long long)ldw, n_shrink);
  MQ_REQUIRE(group > 0 && C % group == 0, MQ_ERR_ARGUMENT, "mq_mse_scales: group %lld does not divide C=%lld",
             (long long)group, (long long)C);
  MQ_REQUIRE(bits >= 2 && bits <= 8, MQ_ERR_ARGUMENT, "mq_mse_scales: bits=%d", bits);
  MQ_REQUIRE(valid_dtype(out_dtype), MQ_ERR_ARGUMENT, "mq_mse_scales: bad dtype %d", out_dtype);
  const float maxq = (float)((1 << bits) - 1), zero = 0.5f * (float)(1 << bits);
  const int64_t n_seg = R * (C / group);
  const int grid = (int)(ceil_div(n_seg, 8) < 148 * 8 ? ceil_div(n_seg, 8) : 148 * 8);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (out_dtype) {
    case MQ_F32:
      launch_mse_scales<MQ_F32>(grid, st, W, R, C, ldw, group, maxq, zero, shrink, n_shrink, norm, scale);
      break;
    case MQ_BF16:
      launch_mse_scales<MQ_BF16>(grid, st, W, R, C, ldw, group, maxq, zero, shrink, n_shrink, norm, scale);
      break;
    default:
      launch_mse_scales<MQ_F16>(grid, st, W, R, C, ldw, group, maxq, zero, shrink, n_shrink, norm, scale);
  }
  MQ_LAUNCH_CHECK();
  return MQ_OK;
}

// ---------------------------------------------------------------------------- no-allocation variant
// Some hosts of this library have no way to hand over scratch memory: a plain C program that
// was given nothing but the H and W pointers by another runtime, a plug-in running inside a
// process whose allocator it must not call (all device memory already belongs to a pool it
// does not control), or code on a path where cudaMalloc's implicit device synchronisation is
// not acceptable.  For them the channel lists of the preparation step live in this
// file-scope array instead of a caller workspace.  It is sized for kNoAllocMaxChannels
// input channels (about 256 KB) and every GPU that loads the library carries it until the
// process exits.
namespace mq {
constexpr int64_t kNoAllocMaxChannels = 32768;
constexpr size_t kNoAllocScratchBytes = ((kNoAllocMaxChannels * 4 + 255) / 256) * 256 + (((kNoAllocMaxChannels + 1) * 4 + 255) / 256) * 256;
static __device__ __align__(256) unsigned char g_prepare_scratch[kNoAllocScratchBytes];
}  // namespace mq

extern "C" int mq_hessian_prepare_noalloc(float* H, int64_t C, int64_t ldh, float* W, int64_t R, int64_t ldw,
                                          float rel_damp, mq_layer_flags* flags, void* stream) {
  using namespace mq;
  MQ_REQUIRE(C > 0, MQ_ERR_ARGUMENT, "mq_hessian_prepare_noalloc: bad C=%lld", (long long)C);
  MQ_REQUIRE(C <= kNoAllocMaxChannels, MQ_ERR_UNSUPPORTED,
             "mq_hessian_prepare_noalloc: C=%lld is beyond the built-in scratch (%lld channels); "
             "use mq_hessian_prepare with a caller-provided workspace",
             (long long)C, (long long)kNoAllocMaxChannels);
  MQ_REQUIRE(mq_hessian_prepare_workspace_bytes(C) <= kNoAllocScratchBytes, MQ_ERR_UNSUPPORTED,
             "mq_hessian_prepare_noalloc: built-in scratch too small for C=%lld", (long long)C);
  // In host code the array's name is only a handle; the kernels need its device address,
  // which differs per GPU.  Looked up once per device, with that device current.
  static void* device_address[64] = {};
  int dev = -1;
  MQ_CUDA(cudaGetDevice(&dev));
  MQ_REQUIRE(dev >= 0 && dev < 64, MQ_ERR_UNSUPPORTED, "mq_hessian_prepare_noalloc: device ordinal %d not supported", dev);
  if (device_address[dev] == nullptr) {
    void* p = nullptr;
    MQ_CUDA(cudaGetSymbolAddress(&p, g_prepare_scratch));
    MQ_REQUIRE(p != nullptr, MQ_ERR_CUDA, "mq_hessian_prepare_noalloc: no device address for the built-in scratch");
    device_address[dev] = p;
  }
  // Same kernels, same order as mq_hessian_prepare; the zero-initialised parts of the scratch
  // (column flags, list length) are cleared by that sequence on every call.
  return mq_hessian_prepare(H, C, ldh, W, R, ldw, rel_damp, flags, device_address[dev], kNoAllocScratchBytes, stream);
}
