// Shared by the sweep's kernels: the argument block of a launch, and how the errors leave.
#pragma once

#include <utility>

#include "engine.cuh"

namespace mq {

constexpr int SWEEP_TILE = 128;

// eight codes below 16, held as bytes in two words (lowest byte = first column) -> one word of nibbles
__device__ __forceinline__ uint32_t pack_nibbles(uint32_t lo4, uint32_t hi4) {
  const uint32_t w = (lo4 & 0xFu) | ((lo4 >> 4) & 0xF0u) | ((lo4 >> 8) & 0xF00u) | ((lo4 >> 12) & 0xF000u);
  const uint32_t v = (hi4 & 0xFu) | ((hi4 >> 4) & 0xF0u) | ((hi4 >> 8) & 0xF00u) | ((hi4 >> 12) & 0xF000u);
  return w | (v << 16);
}

struct SweepArgs {
  float* W; int64_t ldw; int R;
  const float* U; int64_t ldu;
  const float* scale; const float* zero; int64_t group, s_rs, s_gs;
  float maxq, zero_default;
  uint8_t* codes; int64_t C;
  int32_t* packed;   // optional (R, C/8) int32: the same codes, eight 4-bit nibbles per word
  void* deq; float* err;
  int i1, nb;
  const float* Worig; int64_t ldwo;
  uint16_t* err_planes; int64_t plane_stride; int n_planes;
  int err_ld;   // row stride of err / err_planes (both already point at this launch's k window)
  // not null: the errors are written as two fp16 planes, each row scaled by a power of two of its own for every tile,
  // whose inverse goes to row_f[tile * R + row]
  float* row_f;
  int* fault;   // the device's word for waits that were given up
};

// Eight errors of row `gr`, columns k .. k + 7 of the super-block; the sixteen lanes of a half warp hold the 128 of a tile.
__device__ __forceinline__ void write_errors(const SweepArgs& a, int64_t gr, int k, const float4 lo4, const float4 hi4, int lane) {
  const float e[8] = {lo4.x, lo4.y, lo4.z, lo4.w, hi4.x, hi4.y, hi4.z, hi4.w};
  if (!a.err_planes) {
    float4* dst = reinterpret_cast<float4*>(a.err + gr * a.err_ld + k);
    dst[0] = lo4;
    dst[1] = hi4;
    return;
  }
  uint32_t p0[4], p1[4], p2[4];
  if (a.row_f) {
    // The largest error of the row's 128 comes just under 2^14, so that a pair holds 22 bits of every error down to 2^-17 of
    // it; the sixteen lanes of a row agree on it.  (One power of two per row of the matrix cost a row whose groups differ
    // by 2^20 the last bits of its small groups: 13 to 16 times the error of three bf16 planes there.)
    float m = 0.0f;
#pragma unroll
    for (int t = 0; t < 8; ++t) m = fmaxf(m, fabsf(e[t]));
    const unsigned half_warp = 0xffffu << (lane & 16);
    for (int o = 8; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(half_warp, m, o));
    const float rho = scale_below_2_14(m);
    if ((lane & 15) == 0) a.row_f[(int64_t)(k / SWEEP_TILE) * a.R + gr] = 1.0f / rho;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      uint16_t h0, l0, h1, l1;
      split_half2(e[2 * t] * rho, h0, l0);
      split_half2(e[2 * t + 1] * rho, h1, l1);
      p0[t] = (uint32_t)h0 | ((uint32_t)h1 << 16);
      p1[t] = (uint32_t)l0 | ((uint32_t)l1 << 16);
    }
  } else {
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      uint16_t h0, m0, l0, h1, m1, l1;
      split_bf16x3(e[2 * t], h0, m0, l0);
      split_bf16x3(e[2 * t + 1], h1, m1, l1);
      p0[t] = (uint32_t)h0 | ((uint32_t)h1 << 16);
      p1[t] = (uint32_t)m0 | ((uint32_t)m1 << 16);
      p2[t] = (uint32_t)l0 | ((uint32_t)l1 << 16);
    }
  }
  uint16_t* dst = a.err_planes + gr * a.err_ld + k;
  *reinterpret_cast<uint4*>(dst) = make_uint4(p0[0], p0[1], p0[2], p0[3]);
  if (a.n_planes > 1) *reinterpret_cast<uint4*>(dst + a.plane_stride) = make_uint4(p1[0], p1[1], p1[2], p1[3]);
  if (a.n_planes > 2) *reinterpret_cast<uint4*>(dst + 2 * a.plane_stride) = make_uint4(p2[0], p2[1], p2[2], p2[3]);
}

// A launch over up to SUPER_COLUMNS columns and all rows (sweep_super.cu).
int sweep_super_block(bool chained, bool uniform, bool compact, int out_dtype, const SweepArgs& args, cudaStream_t st);

}  // namespace mq
