// int4 -> int32 packing in the compressed-tensors layout, and the matching
// dequantizer.  Both are pure bandwidth kernels: every byte of the code matrix is
// read once with 16-byte loads, every output byte written once.
//
// Replaces pack_weight -> compressed_tensors.pack_to_int32
// (pack_quantized_model.py:57-75) and dequantize_linear_weight
// (src/quant_utils.py:243-256).
#include "common.cuh"
#include "profile.cuh"

namespace mq {

constexpr int kPackThreads = 256;

__device__ __forceinline__ uint32_t pack8(uint32_t lo4, uint32_t hi4) {
  // lo4 holds codes c0..c3 as bytes (c0 lowest), hi4 holds c4..c7.  With every code
  // < 16 the sum of shifted codes equals the OR of the nibbles.
  uint32_t w = (lo4 & 0xFu) | ((lo4 >> 4) & 0xF0u) | ((lo4 >> 8) & 0xF00u) | ((lo4 >> 12) & 0xF000u);
  uint32_t v = (hi4 & 0xFu) | ((hi4 >> 4) & 0xF0u) | ((hi4 >> 8) & 0xF00u) | ((hi4 >> 12) & 0xF000u);
  return w | (v << 16);
}

// Fast path: symmetric (zero == 8, nibble == code), C % 16 == 0, 16-byte aligned base.
// One thread turns 16 codes into two words, four such vectors per trip with all four loads
// issued before the first is used: a 22 MB matrix is one short wave of CTAs, so what counts is
// how many bytes every thread has in flight, not how many trips it makes.
constexpr int kPackUnroll = 4;
__global__ void __launch_bounds__(kPackThreads) pack_int4_vec16(const uint4* __restrict__ codes,
                                                                uint2* __restrict__ packed, int64_t n_vec) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n_vec; i0 += stride * kPackUnroll) {
    uint4 c[kPackUnroll];
#pragma unroll
    for (int u = 0; u < kPackUnroll; ++u) {
      const int64_t i = i0 + u * stride;
      c[u] = i < n_vec ? __ldcs(codes + i) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int u = 0; u < kPackUnroll; ++u) {
      const int64_t i = i0 + u * stride;
      if (i < n_vec) __stcs(packed + i, make_uint2(pack8(c[u].x, c[u].y), pack8(c[u].z, c[u].w)));
    }
  }
}

// General path: any C, optional per-group int8 zero points.  One thread per word.
// Follows the library arithmetic literally: u = uint8(int8(code) - zero + 8), the
// word is the wrapping int32 sum of u << 4i, columns past C contribute 0.
__global__ void __launch_bounds__(kPackThreads) pack_int4_general(const uint8_t* __restrict__ codes, int64_t R,
                                                                  int64_t C, const int8_t* __restrict__ zero,
                                                                  int64_t group, int32_t* __restrict__ packed) {
  int64_t words_per_row = (C + 7) / 8;
  int64_t n = R * words_per_row;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t n_groups = zero ? C / group : 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    int64_t r = i / words_per_row;
    int64_t k = i - r * words_per_row;
    uint32_t w = 0;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      int64_t c = k * 8 + t;
      if (c < C) {
        int8_t v = (int8_t)codes[r * C + c];
        int8_t z = zero ? zero[r * n_groups + c / group] : (int8_t)8;
        uint8_t u = (uint8_t)(int8_t)(v - z + 8);
        w += (uint32_t)u << (4 * t);
      }
    }
    packed[i] = (int32_t)w;
  }
}

// Fast path: groups that are a multiple of 16 / sizeof(out) columns wide, 16-byte aligned output.  A thread
// turns VEC codes (8 for 16-bit outputs, 4 for fp32) into one 16-byte store, four such vectors per trip
// with all loads issued before the first is used; the lanes of a warp read and write consecutive
// bytes.  Scale and zero are read in the type the caller keeps them in (a conversion pass over each
// cost a launch of 6 us), and one 32-bit division finds the group of a whole vector.  The element
// loop below spends its time on a 64-bit division per element and on 2-byte stores.  7168 x 2048
// bf16, groups of 128 (44 MB): 37 us in the element loop; dequantize and pack together, as called
// from Python, 52 -> 33 us, which is then the host's time.
constexpr int kDeqUnroll = 4;
template <int DT, typename S>
__global__ void __launch_bounds__(256) dequantize_vec_kernel(const uint8_t* __restrict__ codes, uint32_t n_vec, uint32_t vec_per_group,
                                                             const S* __restrict__ scale, const S* __restrict__ zero_pts, float zero,
                                                             typename StorageOf<DT>::type* __restrict__ out) {
  using T = typename StorageOf<DT>::type;
  constexpr int VEC = 16 / sizeof(T);
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint64_t i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < n_vec; i0 += (uint64_t)stride * kDeqUnroll) {
    uint32_t c[kDeqUnroll][VEC / 4];
    float s[kDeqUnroll], z[kDeqUnroll];
#pragma unroll
    for (int u = 0; u < kDeqUnroll; ++u) {
      const uint64_t i = i0 + (uint64_t)u * stride;
      if (i < n_vec) {
        if constexpr (VEC == 8) {
          const uint2 v = __ldcs(reinterpret_cast<const uint2*>(codes) + i);
          c[u][0] = v.x; c[u][1] = v.y;
        } else {
          c[u][0] = __ldcs(reinterpret_cast<const uint32_t*>(codes) + i);
        }
        const uint32_t g = (uint32_t)i / vec_per_group;
        s[u] = to_float(scale[g]);
        z[u] = zero_pts ? to_float(zero_pts[g]) : zero;
      }
    }
#pragma unroll
    for (int u = 0; u < kDeqUnroll; ++u) {
      const uint64_t i = i0 + (uint64_t)u * stride;
      if (i >= n_vec) break;
      union { T t[VEC]; uint4 q; } o;
#pragma unroll
      for (int k = 0; k < VEC; ++k) o.t[k] = from_float<T>(((float)((c[u][k >> 2] >> (8 * (k & 3))) & 0xFFu) - z[u]) * s[u]);
      reinterpret_cast<uint4*>(out)[i] = o.q;
    }
  }
}

// General path: groups of any width.
template <int DT, typename S>
__global__ void __launch_bounds__(256) dequantize_kernel(const uint8_t* __restrict__ codes, int64_t R, int64_t C,
                                                         const S* __restrict__ scale,
                                                         const S* __restrict__ zero_pts, int64_t group, float zero,
                                                         typename StorageOf<DT>::type* __restrict__ out) {
  using T = typename StorageOf<DT>::type;
  int64_t n = R * C;
  int64_t G = C / group;
  int64_t stride = (int64_t)gridDim.x * blockDim.x * 4;
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4; i < n; i += stride) {
    // C % 4 == 0 is checked on the host, so four consecutive elements share a row.
    int64_t r = i / C;
    int64_t c = i - r * C;
    uint32_t q4 = *reinterpret_cast<const uint32_t*>(codes + i);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      int64_t gi = r * G + (c + t) / group;
      float s = to_float(scale[gi]);
      float z = zero_pts ? to_float(zero_pts[gi]) : zero;
      float q = (float)((q4 >> (8 * t)) & 0xFFu);
      out[i + t] = from_float<T>((q - z) * s);
    }
  }
}

static int grid_for(int64_t work_items, int threads) {
  int64_t blocks = ceil_div(work_items, threads);
  int64_t cap = 148 * 8;
  return (int)(blocks < 1 ? 1 : (blocks > cap ? cap : blocks));
}

}  // namespace mq

extern "C" int mq_pack_int4(const uint8_t* codes, int64_t R, int64_t C, const int8_t* zero_i8, int64_t group,
                            int32_t* packed, void* stream) {
  using namespace mq;
  MQ_REQUIRE(R >= 0 && C >= 0, MQ_ERR_ARGUMENT, "mq_pack_int4: negative shape R=%lld C=%lld", (long long)R, (long long)C);
  if (R == 0 || C == 0) return MQ_OK;
  MQ_REQUIRE(codes && packed, MQ_ERR_ARGUMENT, "mq_pack_int4: null pointer");
  MQ_REQUIRE(aligned(packed, 4), MQ_ERR_ALIGNMENT, "mq_pack_int4: packed must be 4-byte aligned");
  if (zero_i8) {
    MQ_REQUIRE(group > 0 && C % group == 0, MQ_ERR_ARGUMENT, "mq_pack_int4: group %lld does not divide C=%lld",
               (long long)group, (long long)C);
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  ProfScope prof(PROF_PACK, 1.5 * (double)R * (double)C, 0.0, st);
  if (!zero_i8 && C % 16 == 0 && aligned(codes, 16) && aligned(packed, 8)) {
    int64_t n_vec = R * C / 16;
    pack_int4_vec16<<<grid_for(ceil_div(n_vec, kPackUnroll), kPackThreads), kPackThreads, 0, st>>>(
        reinterpret_cast<const uint4*>(codes), reinterpret_cast<uint2*>(packed), n_vec);
  } else {
    int64_t n = R * ((C + 7) / 8);
    pack_int4_general<<<grid_for(n, kPackThreads), kPackThreads, 0, st>>>(codes, R, C, zero_i8, group, packed);
  }
  MQ_LAUNCH_CHECK();
  return MQ_OK;
}

namespace mq {

template <int DT, typename S>
static int launch_dequantize(const uint8_t* codes, int64_t R, int64_t C, const void* scale, const void* zero_pts, int64_t group,
                             float zero, void* out, cudaStream_t st) {
  using T = typename StorageOf<DT>::type;
  constexpr int VEC = 16 / sizeof(T);
  const int64_t n_vec = R * C / VEC;
  if (group % VEC == 0 && aligned(codes, VEC) && aligned(out, 16) && n_vec < ((int64_t)1 << 32)) {
    dequantize_vec_kernel<DT, S><<<grid_for(ceil_div(n_vec, kDeqUnroll), 256), 256, 0, st>>>(
        codes, (uint32_t)n_vec, (uint32_t)(group / VEC), static_cast<const S*>(scale), static_cast<const S*>(zero_pts), zero,
        static_cast<T*>(out));
  } else {
    dequantize_kernel<DT, S><<<grid_for(R * C / 4, 256), 256, 0, st>>>(codes, R, C, static_cast<const S*>(scale),
                                                                       static_cast<const S*>(zero_pts), group, zero, static_cast<T*>(out));
  }
  MQ_LAUNCH_CHECK();
  return MQ_OK;
}

template <typename S>
static int dispatch_dequantize(int out_dtype, const uint8_t* codes, int64_t R, int64_t C, const void* scale, const void* zero_pts,
                               int64_t group, float zero, void* out, cudaStream_t st) {
  switch (out_dtype) {
    case MQ_F32: return launch_dequantize<MQ_F32, S>(codes, R, C, scale, zero_pts, group, zero, out, st);
    case MQ_BF16: return launch_dequantize<MQ_BF16, S>(codes, R, C, scale, zero_pts, group, zero, out, st);
    default: return launch_dequantize<MQ_F16, S>(codes, R, C, scale, zero_pts, group, zero, out, st);
  }
}

}  // namespace mq

extern "C" int mq_dequantize_typed(const uint8_t* codes, int64_t R, int64_t C, const void* scale, const void* zero_pts, int scale_dtype,
                                   int64_t group, int bits, int out_dtype, void* out, void* stream) {
  using namespace mq;
  MQ_REQUIRE(R >= 0 && C >= 0, MQ_ERR_ARGUMENT, "mq_dequantize: negative shape");
  if (R == 0 || C == 0) return MQ_OK;
  MQ_REQUIRE(codes && scale && out, MQ_ERR_ARGUMENT, "mq_dequantize: null pointer");
  MQ_REQUIRE(bits >= 2 && bits <= 8, MQ_ERR_ARGUMENT, "mq_dequantize: bits=%d", bits);
  MQ_REQUIRE(valid_dtype(out_dtype) && valid_dtype(scale_dtype), MQ_ERR_ARGUMENT, "mq_dequantize: bad dtype %d", out_dtype);
  MQ_REQUIRE(group > 0 && C % group == 0, MQ_ERR_ARGUMENT, "mq_dequantize: group %lld does not divide C=%lld",
             (long long)group, (long long)C);
  MQ_REQUIRE(C % 4 == 0 && aligned(codes, 4), MQ_ERR_UNSUPPORTED, "mq_dequantize: needs C %% 4 == 0 and 4-byte aligned codes");
  const float zero = 0.5f * (float)(1 << bits);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (scale_dtype) {
    case MQ_F32: return dispatch_dequantize<float>(out_dtype, codes, R, C, scale, zero_pts, group, zero, out, st);
    case MQ_BF16: return dispatch_dequantize<__nv_bfloat16>(out_dtype, codes, R, C, scale, zero_pts, group, zero, out, st);
    default: return dispatch_dequantize<__half>(out_dtype, codes, R, C, scale, zero_pts, group, zero, out, st);
  }
}

extern "C" int mq_dequantize(const uint8_t* codes, int64_t R, int64_t C, const float* scale, const float* zero_pts,
                             int64_t group, int bits, int out_dtype, void* out, void* stream) {
  return mq_dequantize_typed(codes, R, C, scale, zero_pts, MQ_F32, group, bits, out_dtype, out, stream);
}

// ---------------------------------------------------------------------------- column permutation
// out[r, j] = src[rows[r], cols[j] / group]  (rows null: r).  The activation order reads the Hessian, the weights and the
// replicated scales through a permutation and brings the codes back through its inverse
// (src/gptq.py:180-187).  A CTA stages a source row in shared memory with whole loads and gathers from there, so that
// global memory only sees rows; an element-wise gather of a 7168 x 7168 matrix took 590 us (the whole activation-order call 5255 -> 4880 us).
namespace mq {

constexpr int64_t kPermuteStageBytes = 96 * 1024;

template <typename T, bool STAGED>
__global__ void __launch_bounds__(256) permute_columns_kernel(const T* __restrict__ src, int64_t ld, const int* __restrict__ rows,
                                                              const int* __restrict__ cols, uint32_t group, int64_t R, int C_in, int C_out,
                                                              T* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char permute_smem[];
  T* stage = reinterpret_cast<T*>(permute_smem);
  for (int64_t r = blockIdx.x; r < R; r += gridDim.x) {
    const T* row = src + (rows ? (int64_t)rows[r] : r) * ld;
    if constexpr (STAGED) {
      const bool vec = (reinterpret_cast<uintptr_t>(row) & 15) == 0;
      constexpr int V = 16 / sizeof(T);
      const int whole = vec ? C_in / V : 0;
      for (int i = threadIdx.x; i < whole; i += blockDim.x) reinterpret_cast<uint4*>(stage)[i] = __ldg(reinterpret_cast<const uint4*>(row) + i);
      for (int i = whole * V + threadIdx.x; i < C_in; i += blockDim.x) stage[i] = row[i];
      __syncthreads();
    }
    T* dst = out + r * C_out;
    for (int j = threadIdx.x * 4; j < C_out; j += blockDim.x * 4) {
      T v[4];
#pragma unroll
      for (int t = 0; t < 4; ++t)
        if (j + t < C_out) {
          const uint32_t c = (uint32_t)__ldg(cols + j + t);
          const uint32_t k = group == 1 ? c : c / group;
          v[t] = STAGED ? stage[k] : row[k];
        }
      if ((C_out & 3) == 0 && (reinterpret_cast<uintptr_t>(out) & (4 * sizeof(T) - 1)) == 0) {
        if constexpr (sizeof(T) == 4) *reinterpret_cast<uint4*>(dst + j) = make_uint4(v[0], v[1], v[2], v[3]);
        else *reinterpret_cast<uint32_t*>(dst + j) = (uint32_t)v[0] | ((uint32_t)v[1] << 8) | ((uint32_t)v[2] << 16) | ((uint32_t)v[3] << 24);
      } else {
#pragma unroll
        for (int t = 0; t < 4; ++t)
          if (j + t < C_out) dst[j + t] = v[t];
      }
    }
    if constexpr (STAGED) __syncthreads();
  }
}

template <typename T>
static int launch_permute(const void* src, int64_t ld, const int* rows, const int* cols, int64_t group, int64_t R, int64_t C_in, int64_t C_out,
                          void* out, cudaStream_t st) {
  const unsigned grid = (unsigned)(R < 148 * 8 ? R : 148 * 8);
  const int64_t bytes = C_in * (int64_t)sizeof(T);
  if (bytes <= kPermuteStageBytes) {
    static bool done[64] = {};
    int dev = 0;
    MQ_CUDA(cudaGetDevice(&dev));
    if (!done[dev & 63]) {
      MQ_CUDA(cudaFuncSetAttribute(permute_columns_kernel<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPermuteStageBytes));
      done[dev & 63] = true;
    }
    permute_columns_kernel<T, true><<<grid, 256, (size_t)align_up((size_t)bytes, 16), st>>>(static_cast<const T*>(src), ld, rows, cols, (uint32_t)group,
                                                                                            R, (int)C_in, (int)C_out, static_cast<T*>(out));
  } else {
    permute_columns_kernel<T, false><<<grid, 256, 0, st>>>(static_cast<const T*>(src), ld, rows, cols, (uint32_t)group, R, (int)C_in, (int)C_out,
                                                           static_cast<T*>(out));
  }
  MQ_LAUNCH_CHECK();
  return MQ_OK;
}

}  // namespace mq

extern "C" int mq_permute_columns(const void* src, int elem_bytes, int64_t ld, const int32_t* rows, const int32_t* cols, int64_t group, int64_t R,
                                  int64_t C_in, int64_t C_out, void* out, void* stream) {
  using namespace mq;
  MQ_REQUIRE(R >= 0 && C_in >= 0 && C_out >= 0 && ld >= C_in && group > 0, MQ_ERR_ARGUMENT, "mq_permute_columns: bad shape R=%lld C=%lld",
             (long long)R, (long long)C_in);
  if (R == 0 || C_out == 0) return MQ_OK;
  MQ_REQUIRE(src && cols && out && C_in < (1ll << 31) && C_out < (1ll << 31), MQ_ERR_ARGUMENT, "mq_permute_columns: null pointer or too wide");
  MQ_REQUIRE(elem_bytes == 1 || (elem_bytes == 4 && aligned(src, 4) && aligned(out, 4)), MQ_ERR_UNSUPPORTED,
             "mq_permute_columns: elements of 1 or 4 bytes, aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (elem_bytes == 4) return launch_permute<uint32_t>(src, ld, rows, cols, group, R, C_in, C_out, out, st);
  return launch_permute<uint8_t>(src, ld, rows, cols, group, R, C_in, C_out, out, st);
}
