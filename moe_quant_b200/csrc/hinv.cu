// Uhat = row-normalised upper Cholesky factor of H^-1, computed without ever
// forming H^-1:
//
//   H = T T^T with T upper triangular (a Cholesky factorisation that starts at the
//   bottom-right corner), so chol_upper(H^-1) = T^-1 and, after dividing each row
//   by its diagonal,  Uhat = diag(T) T^-1 = (T diag(T)^-1)^-1.
//
// One factorisation (C^3/3 flop) and one unit-triangular inverse (C^3/3) replace
// the reference's potrf + potri + potrf (src/linalg_utils.py:12,
// src/gptq.py:237-242; about 4C^3/3 flop).
//
// Blocked right-looking factorisation with 128-wide panels processed from the last
// panel to the first:
//   1. the 128x128 diagonal block, one CTA, and
//   2. the panel above it, substitution against that block: both in one launch (factor_panel_kernel) when the
//                              layer has the GPU to itself, else chol_diag_rev_kernel and trsm_rows_kernel;
//   3. GEMMs (GemmDesc)      : trailing update of the upper triangle; on the tensor path in
//                              levels (the rest of the panel's 512-column super-panel at once,
//                              what lies in front of it once per super-panel or two, with
//                              all of their columns in the contraction).
// The inverse is built by inverting the 128x128 diagonal blocks (same substitution
// kernel on identity rows) and then merging neighbouring blocks pairwise,
//   inv([A B; 0 D]) = [A^-1, -A^-1 B D^-1; 0, D^-1],
// log2(C/128) levels of two batched GEMMs each.
#include "gemm.cuh"
#include "engine.cuh"
#include "mbarrier.cuh"
#include "profile.cuh"

namespace mq {

namespace {

constexpr int NB = 128;  // panel width
constexpr int SUPER_PANELS = 4;               // panels whose update of what lies in front of them is applied together
constexpr int SUPER_NB = SUPER_PANELS * NB;
static_assert(SUPER_NB == SUPER_COLUMNS, "a super-panel");

// ------------------------------------------------------------------ diagonal block
// D (nb x nb, upper triangle valid) -> T_d upper with D = T_d T_d^T, by one CTA, eight pivots at a time (a "leaf", columns
// 8kt..8kt+7, the last one first).  What bounds it is the chain of 128 pivots, so everything else is kept out of its way:
//   chain (2 warps)   : thread t holds rows t and t + 64 of the leaf's column strip in registers.  It factors its own copy of the
//                       8x8 leaf (the same arithmetic in every thread, no communication inside the chain of 8 pivots) and
//                       solves its rows against it; their results are final.  Then it brings its rows of the NEXT leaf's
//                       strip up to date itself and goes on;
//   helpers (4 warps) : meanwhile take the rank-8 update of the columns in front of the next leaf.  A thread keeps one 8x8
//                       tile in registers from the load to the end and hands it over when its columns come next.  Tiles are
//                       dealt out by columns, so whole warps retire;
//   writer (1 warp)   : takes finished strips to global memory, 32 columns (128-byte rows) at a time.
// One barrier per leaf orders the first two: chain(kt) runs beside update(kt + 1).  Every element takes its updates in the
// order of the leaves with one FMA per column.
// What counts beside the chain is the 128 bytes a cycle at which shared memory answers, broadcasts included: two rows per chain thread and
// 8x8 tiles halve what is read (with one row and 4x4 tiles a leaf took 1780 cycles).  Now a leaf takes 1300: 460 to 540 for the
// pivots, 200 to put the strip down, 350 for the next strip, 100 to 240 to exchange the leaf; the block 15.0 us (21.4 with all threads
// updating the block in shared memory between two barriers per leaf, and no look-ahead).
constexpr int PAN_HALF = 80;                // rows of a strip column in shared memory: quads of rows 8i.. first, of rows 8i + 4.. from here on,
constexpr int PAN_LD = PAN_HALF + NB / 2;   // so that neither a row per lane nor eight rows per lane meet bank conflicts
constexpr int DIAG_LD = NB + 4;             // row stride of the finished block in shared memory
constexpr int CHAIN_THREADS = NB / 2;
constexpr int HELP_THREADS = 128;           // 14 * 15 / 2 = 105 tiles in front of the last two leaves
constexpr int DIAG_THREADS = CHAIN_THREADS + HELP_THREADS + 32;
constexpr int DIAG_SMEM_FLOATS = NB * DIAG_LD + 4 * 8 * PAN_LD + 64;
constexpr size_t kDiagSmem = (size_t)DIAG_SMEM_FLOATS * sizeof(float) + (NB / 8) * sizeof(uint64_t);

__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ int pan_pos(int row) { return ((row >> 2) & 1) * PAN_HALF + (row >> 3) * 4 + (row & 3); }

// The memory of a CTA that factors a block.  Finished leaves stay in T, and ready[leaf] tells whoever takes them on.
struct DiagShared {
  float* T;         // [NB][DIAG_LD]: the finished strips
  float* pan;       // [2][8][PAN_LD]: the strip just solved, by kt & 1
  float* next;      // [2][8][PAN_LD]: what the helpers hand over, by strip & 1
  float* leaf;      // [8][8]
  uint64_t* ready;  // [NB / 8] barriers
  __device__ __forceinline__ explicit DiagShared(float* smem)
      : T(smem), pan(T + NB * DIAG_LD), next(pan + 2 * 8 * PAN_LD), leaf(next + 2 * 8 * PAN_LD), ready(reinterpret_cast<uint64_t*>(leaf + 64)) {}
  __device__ __forceinline__ void init() const {   // one thread, before the CTA's first barrier
    for (int k = 0; k < NB / 8; ++k) mbar_init(smem_u32(ready + k), CHAIN_THREADS / 32);
  }
};

// Called by the first DIAG_THREADS threads of a CTA after DiagShared::init.  diag receives the block's diagonal.
__device__ __forceinline__ void factor_diag_block(const DiagShared sh, float* __restrict__ blk, int64_t ld, int nb, int k_global,
                                                  float* __restrict__ diag, mq_layer_flags* flags, int* fault) {
  const int t = threadIdx.x;
  const int kt0 = ((nb + 7) >> 3) - 1;                // the last leaf; rows and columns past nb read as the identity
  // A whole, 16-byte aligned block moves as float4.
  const bool vec = nb == NB && (ld & 3) == 0 && (reinterpret_cast<uintptr_t>(blk) & 15) == 0;
  auto load4 = [&](int r, int c) {
    if (vec) return *reinterpret_cast<const float4*>(blk + (int64_t)r * ld + c);
    float e[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) e[q] = (r < nb && c + q < nb) ? blk[(int64_t)r * ld + c + q] : (r == c + q ? 1.0f : 0.0f);
    return make_float4(e[0], e[1], e[2], e[3]);
  };
  if (t < CHAIN_THREADS) {
    float x[2][8], y[2][8];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int row = t + 64 * h;
        const float4 v = row < 8 * kt0 + 8 ? load4(row, 8 * kt0 + 4 * q) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 u = row < 8 * kt0 ? load4(row, 8 * kt0 - 8 + 4 * q) : make_float4(0.f, 0.f, 0.f, 0.f);
        x[h][4 * q] = v.x; x[h][4 * q + 1] = v.y; x[h][4 * q + 2] = v.z; x[h][4 * q + 3] = v.w;
        y[h][4 * q] = u.x; y[h][4 * q + 1] = u.y; y[h][4 * q + 2] = u.z; y[h][4 * q + 3] = u.w;
      }
    const int p0 = pan_pos(t), p1 = pan_pos(t + 64);
#pragma unroll 1
    for (int kt = kt0;; --kt) {
      const int li = ((t - 8 * kt) & 63) < 8 ? (t & 7) : -1;   // row of the leaf that this thread holds, as its row number lh
      const int lh = kt >> 3;
      if (li >= 0) {
#pragma unroll
        for (int q = 0; q < 2; ++q)
          *reinterpret_cast<float4*>(sh.leaf + li * 8 + 4 * q) =
              lh ? make_float4(x[1][4 * q], x[1][4 * q + 1], x[1][4 * q + 2], x[1][4 * q + 3])
                 : make_float4(x[0][4 * q], x[0][4 * q + 1], x[0][4 * q + 2], x[0][4 * q + 3]);
      }
      bar_sync(1, CHAIN_THREADS);
      float L[8][8];   // L[i][j] = leaf element (row 8kt+i, column 8kt+j), i <= j
#pragma unroll
      for (int i = 7; i >= 0; --i) {
        const float4 hi = *reinterpret_cast<const float4*>(sh.leaf + i * 8 + 4);
        L[i][4] = hi.x; L[i][5] = hi.y; L[i][6] = hi.z; L[i][7] = hi.w;
      }
#pragma unroll
      for (int i = 3; i >= 0; --i) {
        const float4 lo = *reinterpret_cast<const float4*>(sh.leaf + i * 8);
        L[i][0] = lo.x; L[i][1] = lo.y; L[i][2] = lo.z; L[i][3] = lo.w;
      }
      // The 8 pivots are one straight line of code (no branch), so that the scheduler can put
      // the row arithmetic of pivot kk into the latency of pivot kk-1's rsqrt chain.  The rows
      // of the leaf itself, and those below it, run the row arithmetic too.  A pivot that is not positive
      // turns what follows into NaN; it is reported, and the whole factor is replaced.
      int fail = 0;
      float* pb = sh.pan + (kt & 1) * 8 * PAN_LD;
      const bool in[2] = {t < 8 * kt + 8, t + 64 < 8 * kt + 8};
#pragma unroll
      for (int kk = 7; kk >= 0; --kk) {
        const float d = L[kk][kk];
        fail = (!(d > 0.0f) && fail == 0) ? kk + 1 : fail;   // also catches NaN
        float r;                       // d is a positive, normal pivot: the hardware approximation, refined below
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
        r = r * fmaf(-0.5f * d * r, r, 1.5f);  // one Newton step: r = 1/sqrt(d) to about 1 ulp
        L[kk][kk] = d * r;
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (i < kk) L[i][kk] *= r;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (i <= j && j < kk) L[i][j] = fmaf(-L[i][kk], L[j][kk], L[i][j]);
        // these rows above the leaf: p_kk = x_kk / T[kk][kk]; x_j -= p_kk T[j][kk]  (j < kk)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float pv = x[h][kk] * r;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (j < kk) x[h][j] = fmaf(-pv, L[j][kk], x[h][j]);
          // A row of the leaf goes through the same operations as its copy in L: it is the factor from its diagonal on.
          x[h][kk] = t + 64 * h > 8 * kt + kk ? 0.0f : pv;
          if (in[h]) pb[kk * PAN_LD + (h ? p1 : p0)] = x[h][kk];
        }
      }
      if (t == 0 && fail != 0 && kt * 8 + fail - 1 < nb) atomicCAS(&flags->not_positive, 0, k_global + kt * 8 + fail);
      if (kt > 0) bar_sync(2, CHAIN_THREADS + HELP_THREADS);
      // the strip is final
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (in[h]) {
          float* dst = sh.T + (t + 64 * h) * DIAG_LD + 8 * kt;
          *reinterpret_cast<float4*>(dst) = make_float4(x[h][0], x[h][1], x[h][2], x[h][3]);
          *reinterpret_cast<float4*>(dst + 4) = make_float4(x[h][4], x[h][5], x[h][6], x[h][7]);
        }
      __syncwarp();
      if ((t & 31) == 0) mbar_arrive(smem_u32(sh.ready + kt));
      if (kt == 0) break;
      // the next strip: what the helpers have done to it, then this leaf
      if (kt < kt0) {
        const float* nx = sh.next + ((kt - 1) & 1) * 8 * PAN_LD;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          y[0][j] = nx[j * PAN_LD + p0];
          y[1][j] = nx[j * PAN_LD + p1];
        }
      }
      const int pn = pan_pos(8 * kt - 8);   // rows 8kt-8.. of the strip: the next leaf's columns
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        const float4 lo = *reinterpret_cast<const float4*>(&pb[kk * PAN_LD + pn]);
        const float4 hi = *reinterpret_cast<const float4*>(&pb[kk * PAN_LD + pn + PAN_HALF]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float2 n = make_float2(-x[h][kk], -x[h][kk]);
          // two columns per instruction (packed fp32 FMA: each half is an ordinary fma.rn)
          const float2 q0 = __ffma2_rn(n, make_float2(lo.x, lo.y), make_float2(y[h][0], y[h][1]));
          const float2 q1 = __ffma2_rn(n, make_float2(lo.z, lo.w), make_float2(y[h][2], y[h][3]));
          const float2 q2 = __ffma2_rn(n, make_float2(hi.x, hi.y), make_float2(y[h][4], y[h][5]));
          const float2 q3 = __ffma2_rn(n, make_float2(hi.z, hi.w), make_float2(y[h][6], y[h][7]));
          y[h][0] = q0.x; y[h][1] = q0.y; y[h][2] = q1.x; y[h][3] = q1.y;
          y[h][4] = q2.x; y[h][5] = q2.y; y[h][6] = q3.x; y[h][7] = q3.y;
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) x[h][kk] = y[h][kk];
    }
    // the diagonal (T is complete; its rows are other threads')
    bar_sync(1, CHAIN_THREADS);
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (t + 64 * h < nb) diag[t + 64 * h] = sh.T[(t + 64 * h) * (DIAG_LD + 1)];
  } else if (t < CHAIN_THREADS + HELP_THREADS) {
    // tile (mi, mj), mi <= mj, in the order of the columns
    const int id = t - CHAIN_THREADS;
    int mj = (int)((sqrtf(8.0f * id + 1.0f) - 1.0f) * 0.5f);
    if ((mj + 1) * (mj + 2) / 2 <= id) ++mj;
    if (mj * (mj + 1) / 2 > id) --mj;
    const int mi = id - mj * (mj + 1) / 2;
    const bool mine = mj < kt0 - 1;     // the last two strips belong to the chain from the start
    float c[8][8];
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const float4 v = mine ? load4(8 * mi + a, 8 * mj + 4 * q) : make_float4(0.f, 0.f, 0.f, 0.f);
        c[a][4 * q] = v.x; c[a][4 * q + 1] = v.y; c[a][4 * q + 2] = v.z; c[a][4 * q + 3] = v.w;
      }
#pragma unroll 1
    for (int kt = kt0; kt > 0; --kt) {
      bar_sync(2, CHAIN_THREADS + HELP_THREADS);
      if (!mine || mj >= kt - 1) continue;          // columns in front of the next strip
      const float* pb = sh.pan + (kt & 1) * 8 * PAN_LD;
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        const float4 i0 = *reinterpret_cast<const float4*>(pb + kk * PAN_LD + 4 * mi);
        const float4 i1 = *reinterpret_cast<const float4*>(pb + kk * PAN_LD + PAN_HALF + 4 * mi);
        const float4 j0 = *reinterpret_cast<const float4*>(pb + kk * PAN_LD + 4 * mj);
        const float4 j1 = *reinterpret_cast<const float4*>(pb + kk * PAN_LD + PAN_HALF + 4 * mj);
        const float pi[8] = {i0.x, i0.y, i0.z, i0.w, i1.x, i1.y, i1.z, i1.w};
        const float2 pj[4] = {make_float2(j0.x, j0.y), make_float2(j0.z, j0.w), make_float2(j1.x, j1.y), make_float2(j1.z, j1.w)};
#pragma unroll
        for (int a = 0; a < 8; ++a) {
          const float2 n = make_float2(-pi[a], -pi[a]);
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const float2 q = __ffma2_rn(n, pj[b], make_float2(c[a][2 * b], c[a][2 * b + 1]));
            c[a][2 * b] = q.x; c[a][2 * b + 1] = q.y;
          }
        }
      }
      if (mj == kt - 2) {
        float* nx = sh.next + (mj & 1) * 8 * PAN_LD;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          *reinterpret_cast<float4*>(nx + j * PAN_LD + 4 * mi) = make_float4(c[0][j], c[1][j], c[2][j], c[3][j]);
          *reinterpret_cast<float4*>(nx + j * PAN_LD + PAN_HALF + 4 * mi) = make_float4(c[4][j], c[5][j], c[6][j], c[7][j]);
        }
      }
    }
  } else {
    // finished columns, 32 at a time: eight lanes a row
    const int lane = t & 31;
    for (int kt = kt0; kt >= 0; --kt) {
      if (!mbar_wait(smem_u32(sh.ready + kt), 0, fault, 63)) return;
      if (kt & 3) continue;
      const int c = 8 * kt + (lane & 7) * 4;
      if (c >= nb) continue;
      for (int r = lane >> 3; r < nb; r += 4) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);      // below the diagonal tiles
        if ((r >> 3) <= (c >> 3)) v = *reinterpret_cast<const float4*>(sh.T + r * DIAG_LD + c);
        if (vec) {
          *reinterpret_cast<float4*>(blk + (int64_t)r * ld + c) = v;
        } else {
          const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (c + q < nb) blk[(int64_t)r * ld + c + q] = e[q];
        }
      }
    }
  }
}

__global__ void __launch_bounds__(DIAG_THREADS, 1) chol_diag_rev_kernel(float* __restrict__ blk, int64_t ld, int nb, int k_global,
                                                                     float* __restrict__ diag, mq_layer_flags* flags, int* fault) {
  extern __shared__ __align__(16) float smem[];
  const DiagShared sh(smem);
  if (threadIdx.x == 0) {
    sh.init();
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  chain_wait();
  chain_release();
  factor_diag_block(sh, blk, ld, nb, k_global, diag, flags, fault);
}

// ------------------------------------------------------------------ substitution
// Solves P T^T = A row by row, T the (nb x nb) upper-triangular block at `tblk`:
//   for k = nb-1 .. 0:  p_k = a_k / T[k,k];  a_j -= p_k T[j,k]  (j < k).
// One warp per row; lane l holds columns 4l..4l+3.  T is staged transposed in shared
// memory so that a lane reads the four T[j,k] it needs as one float4.
// IDENTITY: the right-hand side is I and the result is stored transposed, which
// yields T^-1 (upper triangular) in `rows`.
constexpr int TT_LD = NB + 4;

// a / d through the reciprocal and one residual correction (Markstein 1990)
__device__ __forceinline__ float quotient(float a, float d, float rd) {
  const float q = a * rd;
  return fmaf(fmaf(-d, q, a), rd, q);
}

// Four neighbouring entries of a solved row as operand planes: a pair of fp16 planes (the equilibrated factor's entries lie
// below 2^14) or up to three bf16 planes.
__device__ __forceinline__ void store_planes(const float (&a)[4], uint16_t* dst, int64_t plane_stride, int n_planes, int half) {
  uint16_t p0[4], p1[4], p2[4];
  if (half) {
#pragma unroll
    for (int q = 0; q < 4; ++q) split_half2(a[q], p0[q], p1[q]);
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q) split_bf16x3(a[q], p0[q], p1[q], p2[q]);
  }
  auto put = [&](uint16_t* to, const uint16_t (&v)[4]) {
    *reinterpret_cast<uint2*>(to) = make_uint2((uint32_t)v[0] | ((uint32_t)v[1] << 16), (uint32_t)v[2] | ((uint32_t)v[3] << 16));
  };
  put(dst, p0);
  if (half || n_planes > 1) put(dst + plane_stride, p1);
  if (!half && n_planes > 2) put(dst + 2 * plane_stride, p2);
}

template <bool IDENTITY>
__global__ void __launch_bounds__(256) trsm_rows_kernel(const float* __restrict__ tblk, int64_t ldt, int64_t t_bs,
                                                        float* __restrict__ rows, int64_t ldr, int64_t r_bs,
                                                        int nrows, int nb_full, int n_total,
                                                        uint16_t* __restrict__ planes, int64_t plane_stride, int n_planes,
                                                        int plane_ld, int half) {
  extern __shared__ __align__(16) float smem[];
  float* TT = smem;                // [NB][TT_LD], TT[k][j] = T[j][k] for j < k, else 0
  float* dg = smem + NB * TT_LD;   // [NB] diagonal of T
  float* rdg = dg + NB;            // [NB] its reciprocal
  const int b = blockIdx.y;
  int nb = nb_full;
  if (n_total > 0) {  // batched over diagonal blocks: the last one may be narrower
    int left = n_total - b * nb_full;
    nb = left < nb_full ? left : nb_full;
    if (IDENTITY) nrows = nb;
  }
  tblk += (int64_t)b * t_bs;
  rows += (int64_t)b * r_bs;
  // Four rows per warp at a time share each shared-memory read of TT and give the scheduler four
  // independent shuffle/FMA chains.
  constexpr int ROWS = 4;
  const int lane = threadIdx.x & 31;
  const int warps_per_block = blockDim.x >> 5;
  const int r_first = ROWS * (blockIdx.x * warps_per_block + (threadIdx.x >> 5));
  float a[ROWS][4];
  // The rows of the panel were final before the diagonal block in front of this launch was
  // factored (that kernel writes only the block), so the first rows are fetched before this grid
  // waits for it; the block itself is staged after the wait.
  if (!IDENTITY) {
#pragma unroll
    for (int h = 0; h < ROWS; ++h) {
      const int r = r_first + h;
      if (r < nrows && lane * 4 < nb) {
        float4 v = *reinterpret_cast<const float4*>(rows + (int64_t)r * ldr + lane * 4);
        a[h][0] = v.x; a[h][1] = v.y; a[h][2] = v.z; a[h][3] = v.w;
      } else {
        a[h][0] = a[h][1] = a[h][2] = a[h][3] = 0.0f;
      }
    }
  }
  chain_wait();
  chain_release();
  {
    // Up to 16 independent float4 loads per thread plus the diagonal are issued before any is used
    // (one memory latency for the block); quads that lie below the diagonal are zeros in the
    // staged form and are not loaded.  float4 index: row j = idx % 128, columns
    // k4..k4+3; consecutive threads take consecutive rows so that the transposed shared-memory
    // stores hit 32 different banks.
    float4 v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int idx = threadIdx.x + i * 256;
      const int j = idx & 127, k4 = (idx >> 7) * 4;
      v[i] = (j < nb && k4 < nb && k4 + 3 > j) ? __ldg(reinterpret_cast<const float4*>(tblk + (int64_t)j * ldt + k4))
                                 : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (threadIdx.x < NB) {
      const int k = threadIdx.x;
      const float d = k < nb ? __ldg(tblk + (int64_t)k * ldt + k) : 1.0f;
      dg[k] = d;
      rdg[k] = 1.0f / d;
    }
    __syncthreads();
    // The block is staged with every column already divided by its diagonal entry
    // (TT[k][j] = T[j][k] / T[k][k], zero for j >= k), so a substitution step is
    // a_j -= a_k * TT[k][j]: no division and no write-back of a_k inside the chain; the quotients
    // p_k = a_k / T[k][k] are formed once at the end.
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const int idx = threadIdx.x + i * 256;
      const int j = idx & 127, k4 = (idx >> 7) * 4;
      const float4 r4 = *reinterpret_cast<const float4*>(&rdg[k4]);
      const float e[4] = {v[i].x * r4.x, v[i].y * r4.y, v[i].z * r4.z, v[i].w * r4.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) TT[(k4 + q) * TT_LD + j] = (j < k4 + q && k4 + q < nb) ? e[q] : 0.0f;
    }
  }
  __syncthreads();
  for (int r0 = r_first; r0 < nrows; r0 += ROWS * gridDim.x * warps_per_block) {
#pragma unroll
    for (int h = 0; h < ROWS; ++h) {
      const int r = r0 + h;
      if (IDENTITY) {
#pragma unroll
        for (int q = 0; q < 4; ++q) a[h][q] = (lane * 4 + q == r) ? 1.0f : 0.0f;
      } else if (r0 == r_first) {
        // fetched before the wait
      } else if (r < nrows && lane * 4 < nb) {
        float4 v = *reinterpret_cast<const float4*>(rows + (int64_t)r * ldr + lane * 4);
        a[h][0] = v.x; a[h][1] = v.y; a[h][2] = v.z; a[h][3] = v.w;
      } else {
        a[h][0] = a[h][1] = a[h][2] = a[h][3] = 0.0f;
      }
    }
    for (int kq = (nb >> 2) - 1; kq >= 0; --kq) {
#pragma unroll
      for (int kk = 3; kk >= 0; --kk) {
        const float4 tt = *reinterpret_cast<const float4*>(&TT[(kq * 4 + kk) * TT_LD + lane * 4]);
#pragma unroll
        for (int h = 0; h < ROWS; ++h) {
          const float ak = __shfl_sync(0xffffffffu, a[h][kk], kq);
          // packed fp32 FMA: two columns per instruction, each half an ordinary fma.rn
          const float2 nak = make_float2(-ak, -ak);
          const float2 lo = __ffma2_rn(nak, make_float2(tt.x, tt.y), make_float2(a[h][0], a[h][1]));
          const float2 hi = __ffma2_rn(nak, make_float2(tt.z, tt.w), make_float2(a[h][2], a[h][3]));
          a[h][0] = lo.x; a[h][1] = lo.y; a[h][2] = hi.x; a[h][3] = hi.y;
        }
      }
    }
    {
      const float4 d4 = *reinterpret_cast<const float4*>(&dg[lane * 4]);
      const float4 r4 = *reinterpret_cast<const float4*>(&rdg[lane * 4]);
      const float dd[4] = {d4.x, d4.y, d4.z, d4.w}, rr[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
      for (int h = 0; h < ROWS; ++h)
#pragma unroll
        for (int q = 0; q < 4; ++q) a[h][q] = quotient(a[h][q], dd[q], rr[q]);
    }
    if (lane * 4 < nb) {
#pragma unroll
      for (int h = 0; h < ROWS; ++h) {
        const int r = r0 + h;
        if (r >= nrows) continue;
        if (IDENTITY) {
          // result row r is column r of T^-1
#pragma unroll
          for (int q = 0; q < 4; ++q) rows[(int64_t)(lane * 4 + q) * ldr + r] = a[h][q];
        } else {
          *reinterpret_cast<float4*>(rows + (int64_t)r * ldr + lane * 4) = make_float4(a[h][0], a[h][1], a[h][2], a[h][3]);
        }
      }
    }
    if (!IDENTITY && planes) {
      // the updates read this panel as operand planes (row, k = column inside the panel)
#pragma unroll
      for (int h = 0; h < ROWS; ++h) {
        const int r = r0 + h;
        if (r >= nrows) continue;
        if (lane * 4 >= nb) a[h][0] = a[h][1] = a[h][2] = a[h][3] = 0.0f;
        store_planes(a[h], planes + (int64_t)r * plane_ld + lane * 4, plane_stride, n_planes, half);   // `planes` points at this panel's k window
      }
    }
  }
}

// ------------------------------------------------------------------ one panel in one launch
// The diagonal block and the solve of the rows above it, for a caller whose layer has the GPU to itself.  The block is a chain
// on one SM, and the solve takes its columns in the order in which the block produces them, the last ones first: so one CTA
// factors the block and passes every strip of eight columns on as it becomes final, and the others follow it strip by strip,
// each with its rows in registers (a warp has RPW rows, a lane four columns of them).  When the block is done the solve is one strip
// behind it.
// Which CTA factors is settled by a ticket, so that it is one that runs: the others wait for it, it waits for nobody.  Waits are bounded.
// The arithmetic is that of trsm_rows_kernel, column by column: a_j -= a_k (T[j,k] / T[k,k]), the quotients at the end.
// A panel takes 16.9 us with 32 rows per CTA, 19.0 with 64 (4705 rows and more), where the two launches took 21.4 + 12.9 (the block now takes 15.0)
// and the gap between them: 2048 x 7168 4242 -> 3498 us, 7168 x 2048 1154 -> 978.  One warp that fetches the strips is not enough (46 us a panel: a
// strip is under way for 2 to 3 us, poll and load, and a new one is there every 0.7).  With several layers in flight the solving CTAs hold
// their SMs while they wait, so compact launches keep the two kernels.  (Callers that run layers on streams of their own without saying so
// are still better off than with two kernels: 2048 x 7168 on two / eight streams 2358 / 2095 us a layer against 2810 / 2190, 1024 x 4096 964 / 771
// against 1221 / 816, the other steps since then included.)
constexpr int PANEL_WARPS = 8;                             // of a solving CTA
constexpr int FETCH_WARPS = 4;                             // the strips' way takes longer than the next strip: several fetch, by turns
constexpr int PANEL_THREADS = (PANEL_WARPS + FETCH_WARPS) * 32;
constexpr int STRIP_WORDS = (NB / 8) * NB * 8;             // one block on its way: [leaf][column pair][row][column]
constexpr size_t kPanelSmem = 120 * 1024;                  // more than half of an SM: the block's CTA shares its SM with none
static_assert(PANEL_THREADS >= DIAG_THREADS + 32, "the block's CTA has a warp to spare that passes the strips on");
static_assert(kPanelSmem >= kDiagSmem && kPanelSmem >= (size_t)(NB * (NB + 4) + 2 * NB) * sizeof(float), "either role fits");

struct PanelArgs {
  float* blk;          // the diagonal block
  float* rows;         // the rows above it (nrows x nb)
  int64_t ld;
  int nb, nrows, k_global;
  float* diag;         // of the block
  mq_layer_flags* flags;
  uint16_t* planes;    // the result as operand planes (this panel's k window)
  int64_t plane_stride;
  int n_planes, plane_ld, half;
  int* ticket;         // zero before the launch
  uint64_t* strips;    // STRIP_WORDS; no word carries `tag` before the launch
  uint32_t tag;
  int* fault;
};

// Strips of the block on their way to other CTAs: 64-bit words of value and tag, each written and read whole, so that a word whose
// tag is right carries its value with it and neither side needs a fence.
__device__ __forceinline__ void store_tagged(uint64_t* dst, float a, float b, uint32_t tag) {
  const uint64_t t = (uint64_t)tag << 32;
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(dst), "l"(t | __float_as_uint(a)), "l"(t | __float_as_uint(b)) : "memory");
}
__device__ __forceinline__ void load_tagged(const uint64_t* src, uint64_t& a, uint64_t& b) {
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(src) : "memory");
}
// columns 8 kt + 2 q and the next of a row
__device__ __forceinline__ uint64_t* strip_words(uint64_t* strips, int kt, int q, int row) { return strips + ((int64_t)(kt * 4 + q) * NB + row) * 2; }

// one warp of the block's CTA
__device__ __forceinline__ void publish_strips(const DiagShared sh, const PanelArgs& p, int lane) {
  for (int kt = ((p.nb + 7) >> 3) - 1; kt >= 0; --kt) {
    if (!mbar_wait(smem_u32(sh.ready + kt), 0, p.fault, 64)) return;
    // as the solve wants them: divided by the diagonal above it (times the reciprocal), the diagonal itself, zeros below
    const int k = 8 * kt + (lane & 7);
    const float mine = 1.0f / sh.T[k * (DIAG_LD + 1)];
    float rd[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) rd[q] = __shfl_sync(0xffffffffu, mine, q);
    for (int row = lane; row < 8 * kt + 8; row += 32) {
      const float4 lo = *reinterpret_cast<const float4*>(sh.T + row * DIAG_LD + 8 * kt), hi = *reinterpret_cast<const float4*>(sh.T + row * DIAG_LD + 8 * kt + 4);
      float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = row < 8 * kt + q ? v[q] * rd[q] : v[q];
#pragma unroll
      for (int q = 0; q < 4; ++q) store_tagged(strip_words(p.strips, kt, q, row), v[2 * q], v[2 * q + 1], p.tag);
    }
  }
}

// One of the warps of a solving CTA that bring strips from global memory to TT, dg and rdg; full[kt] says that strip kt is there.
__device__ __forceinline__ void fetch_strips(const PanelArgs& p, float* TT, float* dg, float* rdg, uint32_t full0, int which, int lane) {
#pragma unroll 1
  for (int kt = ((p.nb + 7) >> 3) - 1 - which; kt >= 0; kt -= FETCH_WARPS) {
    uint64_t v[4][8];
    WaitLimit limit;
    const uint64_t none = (uint64_t)p.tag << 32;
    for (uint32_t it = 0;; ++it) {
      // one word (of those passed on last) until it is there, then all of them
      uint64_t a = none, b = none;
      if (lane == 0) load_tagged(strip_words(p.strips, kt, 3, 8 * kt + 7), a, b);
      bool ok = __shfl_sync(0xffffffffu, (uint32_t)(a >> 32), 0) == p.tag;
      if (ok) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            v[i][2 * q] = v[i][2 * q + 1] = none;
            if (lane + 32 * i < 8 * kt + 8) load_tagged(strip_words(p.strips, kt, q, lane + 32 * i), v[i][2 * q], v[i][2 * q + 1]);
          }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int q = 0; q < 8; ++q) ok = ok && (uint32_t)(v[i][q] >> 32) == p.tag;
        if (__all_sync(0xffffffffu, ok)) break;
      }
      int gone = 0;
      if ((it & 255u) == 255u && lane == 0) gone = limit.expired(p.fault, 61);
      if (__shfl_sync(0xffffffffu, gone, 0)) return;   // the solving warps give up by themselves
    }
    float d = 1.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int row = lane + 32 * i;
      if (row >= 8 * kt + 8) continue;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        float x = __uint_as_float((uint32_t)v[i][q]);
        if (row == 8 * kt + q) {
          d = x;
          x = 0.0f;
        }
        TT[(8 * kt + q) * TT_LD + row] = x;
      }
    }
    if (((lane - 8 * kt) & 31) < 8) {   // the leaf's rows
      const int k = 8 * kt + ((lane - 8 * kt) & 31);
      dg[k] = d;
      rdg[k] = 1.0f / d;
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(full0 + 8 * kt);
  }
}

template <int RPW>
__global__ void __launch_bounds__(PANEL_THREADS, 1) factor_panel_kernel(const PanelArgs p) {
  extern __shared__ __align__(16) float smem[];
  __shared__ __align__(8) uint64_t full[NB / 8];
  __shared__ int role;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const DiagShared sh(smem);
  if (t == 0) {
    role = atomicAdd(p.ticket, 1);
    for (int k = 0; k < NB / 8; ++k) mbar_init(smem_u32(&full[k]), 1);
    sh.init();
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  chain_wait();
  chain_release();
  if (role == 0) {
    if (t < DIAG_THREADS) factor_diag_block(sh, p.blk, p.ld, p.nb, p.k_global, p.diag, p.flags, p.fault);
    else if (warp == DIAG_THREADS / 32) publish_strips(sh, p, lane);
    return;
  }
  float* TT = smem;                // [NB][TT_LD], TT[k][j] = T[j][k] / T[k][k] for j < k, else 0 (up to the end of k's leaf)
  float* dg = smem + NB * TT_LD;   // [NB] diagonal of T
  float* rdg = dg + NB;            // [NB] its reciprocal
  if (warp >= PANEL_WARPS) {
    fetch_strips(p, TT, dg, rdg, smem_u32(&full[0]), warp - PANEL_WARPS, lane);
    return;
  }
  const int kt0 = ((p.nb + 7) >> 3) - 1;
  // ---- the rows
  const int groups = (int)gridDim.x - 1;
  for (int r0 = ((role - 1) * PANEL_WARPS + warp) * RPW; r0 < p.nrows; r0 += groups * PANEL_WARPS * RPW) {
    float a[RPW][4];
#pragma unroll
    for (int h = 0; h < RPW; ++h) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r0 + h < p.nrows && lane * 4 < p.nb) v = *reinterpret_cast<const float4*>(p.rows + (int64_t)(r0 + h) * p.ld + lane * 4);
      a[h][0] = v.x; a[h][1] = v.y; a[h][2] = v.z; a[h][3] = v.w;
    }
#pragma unroll 1
    for (int kt = kt0; kt >= 0; --kt) {
      if (!mbar_wait(smem_u32(&full[kt]), 0, p.fault, 62)) return;
#pragma unroll
      for (int kk = 7; kk >= 0; --kk) {
        float4 tt = make_float4(0.f, 0.f, 0.f, 0.f);     // columns behind the leaf are done
        if (lane < 2 * kt + 2) tt = *reinterpret_cast<const float4*>(&TT[(8 * kt + kk) * TT_LD + lane * 4]);
#pragma unroll
        for (int h = 0; h < RPW; ++h) {
          const float ak = __shfl_sync(0xffffffffu, a[h][kk & 3], 2 * kt + (kk >> 2));
          // packed fp32 FMA: two columns per instruction, each half an ordinary fma.rn
          const float2 nak = make_float2(-ak, -ak);
          const float2 lo = __ffma2_rn(nak, make_float2(tt.x, tt.y), make_float2(a[h][0], a[h][1]));
          const float2 hi = __ffma2_rn(nak, make_float2(tt.z, tt.w), make_float2(a[h][2], a[h][3]));
          a[h][0] = lo.x; a[h][1] = lo.y; a[h][2] = hi.x; a[h][3] = hi.y;
        }
      }
    }
    const bool in = lane * 4 < p.nb;
    float4 d4 = make_float4(1.f, 1.f, 1.f, 1.f), r4 = d4;
    if (in) {
      d4 = *reinterpret_cast<const float4*>(&dg[lane * 4]);
      r4 = *reinterpret_cast<const float4*>(&rdg[lane * 4]);
    }
    const float dd[4] = {d4.x, d4.y, d4.z, d4.w}, rr[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
    for (int h = 0; h < RPW; ++h) {
#pragma unroll
      for (int q = 0; q < 4; ++q) a[h][q] = quotient(a[h][q], dd[q], rr[q]);
      if (r0 + h >= p.nrows) continue;
      if (in) *reinterpret_cast<float4*>(p.rows + (int64_t)(r0 + h) * p.ld + lane * 4) = make_float4(a[h][0], a[h][1], a[h][2], a[h][3]);
      store_planes(a[h], p.planes + (int64_t)(r0 + h) * p.plane_ld + lane * 4, p.plane_stride, p.n_planes, p.half);
    }
  }
}

// ------------------------------------------------------------------ small passes
// T -> T diag(T)^-1 on the upper triangle (unit diagonal), zeros below it.
// upper_only: what lies entirely below the diagonal is left as it is instead of being zeroed
// (the layer path never reads it).
__device__ __forceinline__ void scale_quad(float* __restrict__ H, int64_t ld, const float* __restrict__ diag,
                                           const float* __restrict__ eq, int64_t r, int64_t c) {
  // four columns c..c+3 of row r; what lies entirely below the diagonal is written without being read
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
  if (c + 3 >= r) {
    const float4 v = *reinterpret_cast<const float4*>(H + r * ld + c);
    const float4 d = *reinterpret_cast<const float4*>(diag + c);
    // equilibrated: entry (r, c) of the matrix's own factor is eq[c] / eq[r] times this one's (powers of two)
    float4 e = make_float4(1.f, 1.f, 1.f, 1.f);
    if (eq) {
      const float er = 1.0f / __ldg(eq + r);
      const float4 ec = __ldg(reinterpret_cast<const float4*>(eq + c));
      e = make_float4(ec.x * er, ec.y * er, ec.z * er, ec.w * er);
    }
    o.x = (c + 0 > r) ? v.x / d.x * e.x : (c + 0 == r ? 1.0f : 0.0f);
    o.y = (c + 1 > r) ? v.y / d.y * e.y : (c + 1 == r ? 1.0f : 0.0f);
    o.z = (c + 2 > r) ? v.z / d.z * e.z : (c + 2 == r ? 1.0f : 0.0f);
    o.w = (c + 3 > r) ? v.w / d.w * e.w : (c + 3 == r ? 1.0f : 0.0f);
  }
  *reinterpret_cast<float4*>(H + r * ld + c) = o;
}

// The end of an unscaled factorisation: the diagonal blocks of `own` columns divided by diag(T)
// (the sweep kernels read them; the blocks above are divided by whoever splits them into planes).  A warp takes a row.
__global__ void __launch_bounds__(256) finish_diag_blocks_kernel(float* __restrict__ H, int64_t C, int64_t ld, int own,
                                                                const float* __restrict__ diag, const float* __restrict__ eq) {
  const int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (r >= C) return;
  const int64_t end = (r / own + 1) * own < C ? (r / own + 1) * own : C;   // C % 8 == 0: quads are whole
  for (int64_t c = r / 4 * 4 + (threadIdx.x & 31) * 4; c < end; c += 128) scale_quad(H, ld, diag, eq, r, c);
}

__global__ void __launch_bounds__(256) scale_columns_kernel(float* __restrict__ H, int64_t C, int64_t ld,
                                                            const float* __restrict__ diag, const float* __restrict__ eq,
                                                            int upper_only) {
  const int64_t r = blockIdx.y;
  if ((C & 3) == 0 && (ld & 3) == 0 && (reinterpret_cast<uintptr_t>(H) & 15) == 0) {
    for (int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4; c < C; c += (int64_t)gridDim.x * blockDim.x * 4) {
      if (upper_only && c + 3 < r) continue;
      scale_quad(H, ld, diag, eq, r, c);
    }
    return;
  }
  for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < C; c += (int64_t)gridDim.x * blockDim.x) {
    float v = H[r * ld + c];
    H[r * ld + c] = (c > r) ? v / diag[c] * (eq ? eq[c] / eq[r] : 1.0f) : (c == r ? 1.0f : 0.0f);
  }
}

// The equilibration of H (equilibrating_power) for callers that hand over H alone; eq[C] receives the smallest
// factor (positive floats order like their bits; preset by the host).
__global__ void __launch_bounds__(256) equilibration_kernel(const float* __restrict__ H, int64_t C, int64_t ld, float* __restrict__ eq) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const float v = i < C ? equilibrating_power(H[i * ld + i]) : 1.0f;
  if (i < C) eq[i] = v;
  const int least = __reduce_min_sync(0xffffffffu, i < C ? __float_as_int(v) : 0x7f7f7f7f);
  if ((threadIdx.x & 31) == 0) atomicMin(reinterpret_cast<int*>(eq + C), least);
}

// dst[r][c] = src[r][c] * eq[r] * eq[c] from the start of row r's diagonal 128-block on (dst may be src; eq may
// be null: a copy).  ld % 4 == 0, 16-byte aligned.
__global__ void __launch_bounds__(256) scaled_upper_blocks_kernel(const float* __restrict__ src, int64_t lds, float* __restrict__ dst,
                                                                  int64_t ldd, int64_t C, const float* __restrict__ eq) {
  const int64_t r = blockIdx.y;
  const float er = eq ? __ldg(eq + r) : 1.0f;
  for (int64_t c = (r / NB) * NB + ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4; c < C; c += (int64_t)gridDim.x * blockDim.x * 4) {
    float4 v = *reinterpret_cast<const float4*>(src + r * lds + c);
    if (eq) {
      const float4 ec = __ldg(reinterpret_cast<const float4*>(eq + c));
      v = make_float4(v.x * er * ec.x, v.y * er * ec.y, v.z * er * ec.z, v.w * er * ec.w);
    }
    *reinterpret_cast<float4*>(dst + r * ldd + c) = v;
  }
}

// diag(T) of the matrix itself from that of the equilibrated one
__global__ void __launch_bounds__(256) unscale_diag_kernel(float* __restrict__ diag, const float* __restrict__ eq, int64_t C) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < C) diag[i] = diag[i] / eq[i];
}

__global__ void __launch_bounds__(256) identity_if_failed_kernel(float* __restrict__ U, int64_t C, int64_t ld,
                                                                 const mq_layer_flags* flags, float* __restrict__ diag) {
  if (flags->not_positive == 0) return;
  // with the identity as factor its column scaling is 1 as well (a caller that was handed the
  // unscaled factor divides by it)
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < C; i += (int64_t)gridDim.x * blockDim.x) diag[i] = 1.0f;
  int64_t n = C * C;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    int64_t r = i / C, c = i - r * C;
    U[r * ld + c] = (r == c) ? 1.0f : 0.0f;
  }
}

constexpr size_t kTrsmSmem = (size_t)(NB * TT_LD + 2 * NB) * sizeof(float);

int configure_once() {
  static bool done[64] = {};
  int dev = 0;
  MQ_CUDA(cudaGetDevice(&dev));
  if (!done[dev & 63]) {
    MQ_CUDA(cudaFuncSetAttribute(chol_diag_rev_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDiagSmem));
    MQ_CUDA(cudaFuncSetAttribute(factor_panel_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPanelSmem));
    MQ_CUDA(cudaFuncSetAttribute(factor_panel_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPanelSmem));
    MQ_CUDA(cudaFuncSetAttribute(factor_panel_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPanelSmem));
    MQ_CUDA(cudaFuncSetAttribute(trsm_rows_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrsmSmem));
    MQ_CUDA(cudaFuncSetAttribute(trsm_rows_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrsmSmem));
    done[dev & 63] = true;
  }
  return MQ_OK;
}

}  // namespace

static long long upper_pair_tiles(int64_t C) {
  const int64_t n = ceil_div(C, 256);
  return n * (n + 1) / 2;
}

// Columns whose update of everything in front of them is applied together.  1024 with pairs: what bounds those updates is the way of
// every tile out of its SM, whatever their depth (see umma_pair_kernel); with the sweep's, an attention block
// takes 28.5 instead of 30.0 ms, four experts 13.0 instead of 13.6.  The factor's error against fp64 (4104 to 9224 columns, means of five
// Hessians) is 0.985 to 0.998 of that with 512 where tokens are at least as many as columns, 0.988 to 1.009 with half to three quarters
// as many, up to 1.034 with a twelfth: the partial sums of sixteen slabs outgrow what they leave of the matrix.  So only callers that
// say so (many_tokens) go that deep.
static int far_columns(int64_t C, int math, int split, bool many_tokens) {
  return many_tokens && uses_pairs(C, math, split) && split == 3 ? (int)PAIR_FAR_COLUMNS : SUPER_NB;
}

// what the CTAs of factor_panel_kernel tell one another: the strips of the block in flight, a ticket per panel
static size_t panel_sync_bytes(int64_t C) {
  return align_up(STRIP_WORDS * sizeof(uint64_t) + (size_t)ceil_div(C, NB) * sizeof(int), 256);
}

// enough for either depth
size_t factor_workspace_bytes(int64_t C, int math, int split) {
  if (math != MQ_MATH_TENSOR) return 0;
  return plane_set_bytes(C, far_columns(C, math, split, true), uses_pairs(C, math, split) ? 2 : plane_count(split)) + align_up((size_t)(C + 1) * sizeof(float), 256) + panel_sync_bytes(C);
}

// One panel: the block and the rows above it (factor_panel_kernel).  Eight warps of RPW rows a CTA, one CTA per SM at most.
static int launch_panel(bool chained, const PanelArgs& a, cudaStream_t st) {
  auto launch = [&](auto* kernel, int rpw) {
    const int64_t groups = ceil_div(a.nrows, PANEL_WARPS * rpw);
    const unsigned grid = 1 + (unsigned)(groups < 147 ? groups : 147);
    return launch_chained(chained, kernel, dim3(grid), dim3(PANEL_THREADS), kPanelSmem, st, a);
  };
  if (a.nrows <= 147 * PANEL_WARPS * 4) MQ_CUDA(launch(factor_panel_kernel<4>, 4));
  else if (a.nrows <= 147 * PANEL_WARPS * 8) MQ_CUDA(launch(factor_panel_kernel<8>, 8));
  else MQ_CUDA(launch(factor_panel_kernel<16>, 16));
  return MQ_OK;
}

static int launch_solve(const float* dblk, int64_t ldh, float* rows, int nrows, int nb, uint16_t* planes, int64_t plane_stride, int split,
                        bool half, int plane_ld, bool compact, cudaStream_t st) {
  // 32 rows per CTA (one group of four rows per warp); compact launches: 64 rows, half the CTAs
  // and half the copies of the diagonal block (462 against 454-459 layers/s on eight streams)
  const int grid = compact ? (int)ceil_div(nrows, 64) : (int)(ceil_div(nrows, 32) < 148 * 2 ? ceil_div(nrows, 32) : 148 * 2);
  ProfScope prof(PROF_TRSM, (double)nrows * nb * nb, 0.0, st);
  MQ_CUDA(launch_chained(true, trsm_rows_kernel<false>, dim3(grid, 1), dim3(256), kTrsmSmem, st, dblk, ldh, (int64_t)0, rows, ldh, (int64_t)0,
                         nrows, nb, 0, planes, plane_stride, split, plane_ld, half ? 1 : 0));
  MQ_LAUNCH_CHECK();
  return MQ_OK;
}

static int equilibration(const float* H, int64_t C, int64_t ldh, float* eq, cudaStream_t st) {
  MQ_CUDA(cudaMemsetAsync(eq + C, 0x7f, sizeof(float), st));
  equilibration_kernel<<<(unsigned)ceil_div(C, 256), 256, 0, st>>>(H, C, ldh, eq);
  MQ_LAUNCH_CHECK();
  return MQ_OK;
}

int copy_upper_scaled(const float* src, int64_t lds, float* dst, int64_t ldd, int64_t C, const float* eq, cudaStream_t st) {
  scaled_upper_blocks_kernel<<<dim3(8, (unsigned)C), 256, 0, st>>>(src, lds, dst, ldd, C, eq);
  MQ_LAUNCH_CHECK();
  return MQ_OK;
}

size_t hinv_workspace_bytes(int64_t C, int math, int split) {
  size_t bytes = align_up((size_t)C * sizeof(float), 256);          // diag
  bytes += align_up((size_t)C * (size_t)C * sizeof(float), 256);    // merge scratch
  size_t a = engine_workspace_bytes(C, C, C, math, plane_count(split)), b = factor_workspace_bytes(C, math, split);
  bytes += a > b ? a : b;
  return bytes;
}

// H (damped, symmetric; upper triangle read) -> unit upper factor Utilde = T diag(T)^-1 in place,
// zeros below the diagonal (upper_only: the part below the diagonal blocks is neither read nor written;
// unscaled, if not 0: only the diagonal blocks of that many columns are scaled; above them T itself is left in place and the caller
// divides column c by diag[c] where it reads it).  diag (C floats, device) receives diag(T).  On a non-positive pivot
// flags->not_positive is set and the result is replaced by I.
// eq (uses_pairs only): H has been equilibrated by the caller (copy_upper_scaled) with these
// factors; unscaled then leaves the equilibrated factor above the diagonal blocks and its diagonal in diag.
// Null: where pairs are used the matrix is equilibrated here and everything is given back in H's own units.
int chol_unit_factor(float* H, int64_t C, int64_t ldh, float* diag, int math, int split, mq_layer_flags* flags,
                     Workspace& ws, cudaStream_t st, bool upper_only, int unscaled, const float* eq) {
  MQ_TRY(configure_once());
  const int compact = (math & MQ_MATH_COMPACT) ? 1 : 0;   // the panel solves and the rank-128 strips look at it
  const bool many_tokens = (math & MQ_MATH_MANY_TOKENS) != 0;
  math &= ~(MQ_MATH_COMPACT | MQ_MATH_MANY_TOKENS);
  MQ_REQUIRE(math != MQ_MATH_TENSOR || (split >= 1 && split <= 4), MQ_ERR_ARGUMENT, "factorisation: split must be 1, 2, 3 or 4 (got %d)", split);
  const bool half = uses_pairs(C, math, split);   // pairs of fp16 planes (split_half2)
  const int all_products = half && split == 4 ? 1 : 0;
  const int far_nb = far_columns(C, math, split, many_tokens), far_panels = far_nb / NB;
  split = plane_count(split);
  MQ_REQUIRE(!eq || half, MQ_ERR_ARGUMENT, "factorisation: an equilibrated matrix needs pairs of planes");
  Workspace local(ws.base ? ws.base + ws.used : nullptr, ws.base ? ws.size - ws.used : 0);
  const bool own_units = half && !eq;
  if (own_units) {
    MQ_REQUIRE(!unscaled, MQ_ERR_ARGUMENT, "factorisation: an unscaled factor needs the caller's equilibration");
    float* own = local.take<float>(C + 1);
    MQ_REQUIRE(own, MQ_ERR_WORKSPACE, "factorisation: workspace too small");
    MQ_TRY(equilibration(H, C, ldh, own, st));
    MQ_TRY(copy_upper_scaled(H, ldh, H, ldh, C, own, st));
    eq = own;
  }
  const int P = (int)ceil_div(C, NB);
  // Tensor path: the panel solve writes its result as planes too, and the rank-128 update
  // P P^T reads one plane set as both operands.
  const bool tensor = math == MQ_MATH_TENSOR;
  {
    // ---- right-looking in levels, last panel first.  Four panels form a super-panel of 512
    // columns.  Behind each panel only the columns of its own super-panel that are still to be
    // factored take their rank-128 update at once (a strip at most 384 wide); what lies in
    // front of the super-panel is updated with all 512 columns of it in one contraction.  Where far_columns says so
    // two super-panels go together: behind the first only the second takes its update (512 deep), and everything
    // in front of both takes one with all 1024 columns, so a tile of the trailing matrix moves once per 1024 columns.  Tensor path: the panel solve writes its result as operand
    // planes too (k window of its panel inside the plane buffer), and the updates read one
    // plane set as both operands.
    PlaneSet pset;
    if (tensor) {
      const int planes = half ? 2 : split;
      pset.base = local.take<uint16_t>(plane_set_bytes(C, far_nb, planes) / 2);
      MQ_REQUIRE(pset.base, MQ_ERR_WORKSPACE, "factorisation: workspace too small for the panel planes");
      pset.planes = planes; pset.rows_pad = (int)pad_rows(C); pset.total_rows = pset.rows_pad; pset.K_pad = far_nb;
      pset.fp16 = half;
    }
    // A caller with several layers in flight gives each few SMs, and the solving CTAs would hold theirs while they wait.
    const bool together = tensor && !compact && P > 1;
    uint64_t* strips = nullptr;
    int *tickets = nullptr, *fault = nullptr;
    MQ_TRY(engine_fault_word(&fault));
    if (together) {
      strips = local.take<uint64_t>(panel_sync_bytes(C) / sizeof(uint64_t));
      MQ_REQUIRE(strips, MQ_ERR_WORKSPACE, "factorisation: workspace too small for the panels' strips");
      tickets = reinterpret_cast<int*>(strips + STRIP_WORDS);
      MQ_CUDA(cudaMemsetAsync(strips, 0, panel_sync_bytes(C), st));
    }
    Engine eng(math, split, local, st);   // fp32 math
    for (int p = P - 1; p >= 0; --p) {
      const int p_lo = (p / SUPER_PANELS) * SUPER_PANELS;      // first (lowest) panel of this super-panel
      const int64_t k0 = (int64_t)p_lo * NB;                   // first column of the super-panel
      const int64_t k1 = (int64_t)p * NB;
      const int nb = (int)((C - k1) < NB ? (C - k1) : NB);
      const int f_lo = (p / far_panels) * far_panels;          // first panel of those whose far update is applied together
      const int kwin = (p - f_lo) * NB;                        // this panel's k window in the plane buffer
      float* dblk = H + k1 * ldh + k1;
      if (together && k1 > 0) {
        PanelArgs pa;
        pa.blk = dblk; pa.rows = H + k1; pa.ld = ldh;
        pa.nb = nb; pa.nrows = (int)k1; pa.k_global = (int)k1;
        pa.diag = diag + k1; pa.flags = flags;
        pa.planes = pset.base + kwin; pa.plane_stride = pset.total_rows * (int64_t)far_nb;
        pa.n_planes = split; pa.plane_ld = far_nb; pa.half = half ? 1 : 0;
        pa.ticket = tickets + p; pa.strips = strips; pa.tag = (uint32_t)(p + 1);
        pa.fault = fault;
        ProfScope prof(PROF_CHOL_DIAG, (double)nb * nb * nb / 3.0 + (double)k1 * nb * nb, 0.0, st);
        MQ_TRY(launch_panel(p < P - 1, pa, st));
      } else {
        ProfScope prof(PROF_CHOL_DIAG, (double)nb * nb * nb / 3.0, 0.0, st);
        MQ_CUDA(launch_chained(true, chol_diag_rev_kernel, dim3(1), dim3(DIAG_THREADS), kDiagSmem, st, dblk, ldh, nb, (int)k1, diag + k1, flags, fault));
      }
      MQ_LAUNCH_CHECK();
      if (k1 == 0) break;
      if (!together) {
        MQ_TRY(launch_solve(dblk, ldh, H + k1, (int)k1, nb, tensor ? pset.base + kwin : nullptr, tensor ? pset.total_rows * (int64_t)far_nb : 0,
                            split, half, far_nb, compact != 0, st));
      }
      if (!tensor) {
        GemmDesc g;
        g.A = H + k1; g.a_rs = ldh; g.a_cs = 1;
        g.B = H + k1; g.b_rs = 1; g.b_cs = ldh;
        g.C = H; g.ldc = ldh;
        g.M = (int)k1; g.N = (int)k1; g.K = nb;
        g.alpha = -1.0f; g.beta = 1.0f;
        g.upper_tiles_only = 1;
        MQ_TRY(eng.gemm(g));
        continue;
      }
      if (p > p_lo) {
        // near: H[0:k1, k0:k1] -= P P[k0:k1]^T, the rest of this super-panel
        GemmDesc g;
        g.C = H + k0; g.ldc = ldh;
        g.M = (int)k1; g.N = (int)(k1 - k0); g.K = nb;
        g.alpha = -1.0f; g.beta = 1.0f;
        g.compact = compact;
        g.all_products = all_products;
        PlaneSet a = pset, b = pset;
        a.k0 = kwin;
        b.k0 = kwin; b.row0 = k0;
        MQ_TRY(gemm_tensor_planes(g, a, b, st));
      } else if (k0 > 0) {
        const int64_t f0 = (int64_t)f_lo * NB;
        const int p_hi = (p_lo + SUPER_PANELS - 1) < (P - 1) ? (p_lo + SUPER_PANELS - 1) : (P - 1);
        const int f_hi = (f_lo + far_panels - 1) < (P - 1) ? (f_lo + far_panels - 1) : (P - 1);
        GemmDesc g;
        g.ldc = ldh;
        g.alpha = -1.0f; g.beta = 1.0f;
        g.all_products = all_products;
        g.k_round = NB;   // partial sums per panel meet in round-to-nearest adds, as in a one-level loop
        PlaneSet a = pset, b = pset;
        a.k0 = b.k0 = (p_lo - f_lo) * NB;
        const bool joint = far_nb > SUPER_NB && joint_update(upper_pair_tiles((int64_t)(f_lo + SUPER_PANELS) * NB));
        if (!joint) {
          // H[0:k0, 0:k0] -= P_S P_S^T over the columns of this super-panel, tiles on and above the diagonal
          g.C = H;
          g.M = (int)k0; g.N = (int)k0; g.K = (p_hi - p_lo + 1) * NB;
          g.upper_tiles_only = 1;
        } else if (p_lo > f_lo) {
          // H[0:k0, f0:k0] -= P_S P_S[f0:k0]^T over the columns of this super-panel: the rest of those that go together
          g.C = H + f0;
          g.M = (int)k0; g.N = (int)(k0 - f0); g.K = (p_hi - p_lo + 1) * NB;
          b.row0 = f0;
        } else {
          // H[0:k0, 0:k0] -= P P^T over all columns of those, tiles on and above the diagonal
          g.C = H;
          g.M = (int)k0; g.N = (int)k0; g.K = (f_hi - f_lo + 1) * NB;
          g.upper_tiles_only = 1;
        }
        MQ_TRY(gemm_tensor_planes(g, a, b, st));
      }
    }
  }
  // ---- T -> unit-diagonal factor
  if (unscaled) {
    finish_diag_blocks_kernel<<<(unsigned)ceil_div(C, 8), 256, 0, st>>>(H, C, ldh, unscaled, diag, eq);
    MQ_LAUNCH_CHECK();
  } else {
    const unsigned gx = (unsigned)(ceil_div(C, 256) < 8 ? ceil_div(C, 256) : 8);
    scale_columns_kernel<<<dim3(gx, (unsigned)C), 256, 0, st>>>(H, C, ldh, diag, eq, upper_only ? 1 : 0);
    MQ_LAUNCH_CHECK();
  }
  if (own_units) {
    unscale_diag_kernel<<<(unsigned)ceil_div(C, 256), 256, 0, st>>>(diag, eq, C);
    MQ_LAUNCH_CHECK();
  }
  identity_if_failed_kernel<<<148 * 4, 256, 0, st>>>(H, C, ldh, flags, diag);
  MQ_LAUNCH_CHECK();
  return MQ_OK;
}

int hinv_upper(float* H, int64_t C, int64_t ldh, float* Uhat, int64_t ldu, float* diag_out, int math, int split,
               mq_layer_flags* flags, Workspace& ws, cudaStream_t st) {
  float* diag = ws.take<float>(C);
  float* scratch = ws.take<float>((size_t)C * C);
  MQ_REQUIRE(diag && scratch, MQ_ERR_WORKSPACE, "mq_hinv_upper: workspace too small");
  // The factor is the result here and no sweep averages its error: with three products it is 1.00 to 1.02 of that of three planes
  // (648 to 4096 columns, as many tokens), with all four 0.98 to 1.00.
  MQ_TRY(chol_unit_factor(H, C, ldh, diag, math, split == 3 ? 4 : split, flags, ws, st, false, 0, nullptr));
  if (diag_out) MQ_CUDA(cudaMemcpyAsync(diag_out, diag, C * sizeof(float), cudaMemcpyDeviceToDevice, st));
  Engine eng(math, plane_count(split), ws, st);
  const int P = (int)ceil_div(C, NB);
  // ---- inverse of the unit factor: invert the diagonal blocks, then merge pairs of blocks
  MQ_CUDA(cudaMemsetAsync(Uhat, 0, (size_t)C * ldu * sizeof(float), st));
  trsm_rows_kernel<true><<<dim3(4, P), 256, kTrsmSmem, st>>>(H, ldh, (int64_t)NB * (ldh + 1), Uhat, ldu,
                                                             (int64_t)NB * (ldu + 1), NB, NB, (int)C, nullptr, 0, 0, NB, 0);
  MQ_LAUNCH_CHECK();
  for (int64_t s = NB; s < C; s *= 2) {
    const int batch = (int)ceil_div(C - s, 2 * s);
    GemmDesc g1;  // scratch block = B D^-1
    g1.A = H + s; g1.a_rs = ldh; g1.a_cs = 1; g1.a_bs = 2 * s * (ldh + 1);
    g1.B = Uhat + s * ldu + s; g1.b_rs = ldu; g1.b_cs = 1; g1.b_bs = 2 * s * (ldu + 1);
    g1.C = scratch + s; g1.ldc = C; g1.c_bs = 2 * s * (C + 1);
    g1.M = (int)s; g1.N = (int)s; g1.K = (int)s;
    g1.alpha = 1.0f; g1.beta = 0.0f;
    g1.b_upper = 1;
    g1.batch = batch; g1.n_total = (int)(C - s); g1.n_step = (int)(2 * s); g1.k_follows_n = 1;
    MQ_TRY(eng.gemm(g1));
    GemmDesc g2;  // off-diagonal block = -A^-1 (scratch block)
    g2.A = Uhat; g2.a_rs = ldu; g2.a_cs = 1; g2.a_bs = 2 * s * (ldu + 1);
    g2.B = scratch + s; g2.b_rs = C; g2.b_cs = 1; g2.b_bs = 2 * s * (C + 1);
    g2.C = Uhat + s; g2.ldc = ldu; g2.c_bs = 2 * s * (ldu + 1);
    g2.M = (int)s; g2.N = (int)s; g2.K = (int)s;
    g2.alpha = -1.0f; g2.beta = 0.0f;
    g2.a_upper = 1;
    g2.batch = batch; g2.n_total = (int)(C - s); g2.n_step = (int)(2 * s);
    MQ_TRY(eng.gemm(g2));
  }
  identity_if_failed_kernel<<<148 * 4, 256, 0, st>>>(Uhat, C, ldu, flags, diag);
  MQ_LAUNCH_CHECK();
  return MQ_OK;
}

}  // namespace mq

extern "C" size_t mq_hinv_upper_workspace_bytes(int64_t C, int math, int split) {
  if (C <= 0) return 0;
  return mq::hinv_workspace_bytes(C, math, split);
}

extern "C" int mq_hinv_upper(float* H, int64_t C, int64_t ldh, float* Uhat, int64_t ldu, float* diag_out, int math, int split,
                             mq_layer_flags* flags, void* workspace, size_t workspace_bytes, void* stream) {
  using namespace mq;
  MQ_REQUIRE(H && Uhat && flags, MQ_ERR_ARGUMENT, "mq_hinv_upper: null pointer");
  MQ_REQUIRE(C > 0 && ldh >= C && ldu >= C, MQ_ERR_ARGUMENT, "mq_hinv_upper: bad C=%lld ldh=%lld ldu=%lld", (long long)C,
             (long long)ldh, (long long)ldu);
  MQ_REQUIRE(C % 8 == 0, MQ_ERR_UNSUPPORTED, "mq_hinv_upper: C=%lld must be a multiple of 8", (long long)C);
  MQ_REQUIRE(ldh % 4 == 0 && ldu % 4 == 0 && aligned(H, 16) && aligned(Uhat, 16), MQ_ERR_ALIGNMENT,
             "mq_hinv_upper: H and Uhat must be 16-byte aligned with leading dimensions that are multiples of 4");
  MQ_REQUIRE(math == MQ_MATH_FP32 || math == MQ_MATH_TENSOR, MQ_ERR_ARGUMENT, "mq_hinv_upper: bad math %d", math);
  Workspace ws(workspace, workspace_bytes);
  return hinv_upper(H, C, ldh, Uhat, ldu, diag_out, math, split, flags, ws, static_cast<cudaStream_t>(stream));
}

extern "C" size_t mq_chol_unit_factor_workspace_bytes(int64_t C, int math, int split) {
  if (C <= 0) return 0;
  return mq::align_up((size_t)C * sizeof(float), 256) + mq::factor_workspace_bytes(C, math & ~MQ_MATH_MANY_TOKENS, split);
}

extern "C" int mq_chol_unit_factor(float* H, int64_t C, int64_t ldh, float* diag_out, int math, int split,
                                   mq_layer_flags* flags, void* workspace, size_t workspace_bytes, void* stream) {
  using namespace mq;
  MQ_REQUIRE(H && flags, MQ_ERR_ARGUMENT, "mq_chol_unit_factor: null pointer");
  MQ_REQUIRE(C > 0 && ldh >= C, MQ_ERR_ARGUMENT, "mq_chol_unit_factor: bad C=%lld ldh=%lld", (long long)C, (long long)ldh);
  MQ_REQUIRE(C % 8 == 0, MQ_ERR_UNSUPPORTED, "mq_chol_unit_factor: C=%lld must be a multiple of 8", (long long)C);
  MQ_REQUIRE(ldh % 4 == 0 && aligned(H, 16), MQ_ERR_ALIGNMENT, "mq_chol_unit_factor: H must be 16-byte aligned, ldh %% 4 == 0");
  const int base_math = math & ~MQ_MATH_MANY_TOKENS;
  MQ_REQUIRE(base_math == MQ_MATH_FP32 || base_math == MQ_MATH_TENSOR, MQ_ERR_ARGUMENT, "mq_chol_unit_factor: bad math %d", math);
  Workspace ws(workspace, workspace_bytes);
  float* diag = ws.take<float>(C);
  MQ_REQUIRE(diag, MQ_ERR_WORKSPACE, "mq_chol_unit_factor: workspace too small");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  MQ_TRY(chol_unit_factor(H, C, ldh, diag, math, split, flags, ws, st, false, 0, nullptr));
  if (diag_out) MQ_CUDA(cudaMemcpyAsync(diag_out, diag, C * sizeof(float), cudaMemcpyDeviceToDevice, st));
  return MQ_OK;
}
