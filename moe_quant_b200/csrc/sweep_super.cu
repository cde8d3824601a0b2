// The column sweep, a super-block of 512 columns per launch (see sweep.cu for the recurrence and for when).
#include "engine.cuh"
#include "mbarrier.cuh"
#include "sweep.cuh"

namespace mq {

namespace {

constexpr int TILE = SWEEP_TILE;
constexpr int SUB = 16;                 // columns of a sub-block: one chain of quantisation steps per row
constexpr int SUPER = SUPER_COLUMNS;
// Warp 0 runs the chains, warps 1 to 3 fetch what the next sub-blocks need, warps 4 to 11 apply the errors.
// A chain keeps the 136 entries of its 16 x 16 triangle in registers, so that they are there when a step needs them: with the
// 128 registers a thread that all could have alike, a sub-block took 5300 cycles instead of 2900.  (With eight warps of 255 registers,
// and twice as many columns per helper, 2048 x 7168 took 1500 us instead of 1260: too few warps in flight.)
constexpr int SUPER_THREADS = 384;
constexpr int FETCHERS = 3, HELPERS = 8;
constexpr int SUPER_REGS = 168, CHAIN_REGS = 248, HELPER_REGS = 128;   // a thread: at the launch, and how the warpgroups divide them
static_assert((1 + FETCHERS) * CHAIN_REGS + HELPERS * HELPER_REGS <= SUPER_THREADS / 32 * SUPER_REGS, "the registers of the launch are all there are");
// Rows of a CTA: eight; a caller with several layers in flight gives each half of the GPU (eight streams, four experts of
// 4096 x 1024 at 74 / 148 CTAs: 6.38 / 7.08 ms).
constexpr int ROWS = 8, COMPACT_CTAS = 74;
constexpr int MAX_ROWS = ((int)SUPER_BLOCK_ROWS + COMPACT_CTAS - 1) / COMPACT_CTAS;
static_assert(SUPER_BLOCK_ROWS <= 148 * ROWS && MAX_ROWS >= ROWS, "a CTA has one group of rows");
constexpr int W_LD = SUPER + 4;         // row stride of the running weights: a warp's 16-byte reads of 8 rows hit 32 banks
constexpr int SLOTS = 3;                // slabs (sixteen rows of the factor) in shared memory: one in use, one there, one on its way
constexpr int SLAB = SUB * SUPER;
constexpr int SLAB_FAULT = 65;          // code of a slab that did not arrive
constexpr int WO_LD = SUB + 4;          // row stride of the original weights of a sub-block

constexpr size_t super_smem_bytes(int rows, bool uniform) {
  return (size_t)(SLOTS * SLAB + rows * W_LD + rows * 2 * WO_LD + rows * 2 * ((uniform ? 1 : SUB) + 1) * 4) * sizeof(float);
}
static_assert(super_smem_bytes(MAX_ROWS, false) <= 227 * 1024 - 64, "shared memory of a CTA");

// Rows 16c .. 16c + 15 of the super-block's part of the factor (`src`: its top-left element), from their diagonal block on,
// -> shared memory [SUB][SUPER], a bulk copy per row, complete on `bar`.  Called by a whole warp.  What lies below the diagonal is
// copied but not used; rows and columns past nb (a multiple of eight) keep what was there and reach no column in front of nb.
__device__ __forceinline__ void fetch_slab(float* slab, uint32_t bar, const float* __restrict__ src, int64_t ldu, int nb, int c) {
  const int t = threadIdx.x & 31, j0 = c * SUB;
  const int rows = nb - j0 < SUB ? nb - j0 : SUB;
  const uint32_t bytes = (uint32_t)(nb - j0) * 4;
  if (t == 0) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes * rows) : "memory");
  __syncwarp();
  if (t < rows)
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(&slab[t * SUPER + j0])),
                 "l"(src + (int64_t)(j0 + t) * ldu + j0), "r"(bytes), "r"(bar)
                 : "memory");
}

// four columns take e times the factor's entries u: packed fp32 FMAs, each half an ordinary fma.rn
__device__ __forceinline__ void fma4(float4& v, const float4 u, const float e) {
  const float2 e2 = make_float2(e, e);
  const float2 p01 = __ffma2_rn(make_float2(u.x, u.y), e2, make_float2(v.x, v.y));
  const float2 p23 = __ffma2_rn(make_float2(u.z, u.w), e2, make_float2(v.z, v.w));
  v = make_float4(p01.x, p01.y, p23.x, p23.y);
}

// Up to 512 columns of the sweep for up to MAX_ROWS rows per CTA, in sub-blocks of sixteen columns.
// Thread r < rows takes row r through sub-block c:
//   chain:  the sixteen columns in order, in registers: quantize column j, add e_j U[j, k] to the columns k behind
//           it inside the sub-block.  The only serial dependence is quantize(j) -> one FMA -> quantize(j + 1),
//           about fifteen operations;
//   next:   the sixteen errors go to the sixteen columns of sub-block c + 1, which it then holds.
// Meanwhile the other warps add the errors of sub-block c - 1 to the columns from sub-block c + 1 on: a lane
// keeps the 16 x 4 entries of the factor for its four columns in registers and walks the rows.  One barrier
// per sub-block hands the errors over and orders the two: before `next` touches sub-block c + 1 the other
// warps have added everything up to c - 1 there.  The columns of the current 128-column tile so take the errors in increasing
// column order with one FMA each, as a column-at-a-time recurrence does.  Those behind it collect what
// they receive, sixteen products at a time, and get it added to their running value once, when their tile
// comes next: the value goes back to W (which so holds every tile as it was when its turn came).
// The factor passes through three slabs of sixteen rows, 32 KB down to 1 KB each, fetched two sub-blocks ahead.
//
// What bounds a super-block is the chain, 512 steps of 94 cycles, and handing the sub-blocks over (the next one's sixteen columns take a lane
// by itself 600 cycles, and 900 while the helpers read shared memory): 2800 cycles per sub-block, 47 us, whatever the number of rows;
// 45 us with up to eight rows per CTA.  As four tiles and three rank-128 updates the same columns take 4 x 16.5 + 3 x 8.5 us: 512 x 4096 is
// quantized in 1452 us instead of 1574, 500 x 1056 in 417 instead of 533.  With more rows per CTA than are taken now the helpers' FMAs take over (2048 rows on 74 SMs:
// 59 us), where the tensor cores' updates are the better way; far products on mma.sync, from planes in shared memory, took longer
// still (49 rows per CTA: 141 us against 121).
// UNIFORM: the columns of a sub-block lie in one quantization group (group % 16 == 0).
// QUARTERS: at most eight rows (`next` by four lanes a row: a sweep of 512 x 4096 takes 534 us instead of 551).
// INVERSE_FREE (a.Worig given): U is the unit factor Utilde = Uhat^-1 and what is propagated is minus the
// total change of the column, -(y - w_original), instead of the error against the running value;
// x_j = w_j - sum_{i<j} (y_i - w_i) Utilde[i,j] is the same number as the reference's running weight
// (E Uhat = Y - W  <=>  E = (Y - W) Utilde).
template <int DT, bool UNIFORM, bool INVERSE_FREE, bool QUARTERS>
__global__ void __launch_bounds__(SUPER_THREADS, 1) sweep_super_kernel(const SweepArgs a, const int group_rows) {
  using T = typename StorageOf<DT>::type;
  extern __shared__ __align__(16) float sweep_smem[];
  __shared__ __align__(8) uint64_t slab_bars[SLOTS];
  float* us = sweep_smem;                 // [SLOTS][SUB][SUPER]
  float* ws = us + SLOTS * SLAB;          // [group_rows][W_LD]: running weights (behind the current tile: what they have received), replaced by the errors
  float* wos = ws + group_rows * W_LD;    // [2][group_rows][WO_LD]: original weights of two sub-blocks by turns
  // the grid of every row (scale, its reciprocal, zero point) for two sub-blocks by turns: UNIFORM [2][group_rows], otherwise [2][SUB][group_rows]
  float4* gs = reinterpret_cast<float4*>(wos + 2 * group_rows * WO_LD);
  uint4* cs = reinterpret_cast<uint4*>(gs + 2 * group_rows * (UNIFORM ? 1 : SUB));   // [2][group_rows]: codes of two sub-blocks by turns
  const int nb = a.nb, i1 = a.i1, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n_sub = (nb + SUB - 1) / SUB;
  const float* factor = a.U + (int64_t)i1 * a.ldu + i1;
  // Slabs are warp 3's business alone: it starts the copies and waits for them, and the block's barriers tell the others.
  // The factor is constant during the sweep: its first slabs are fetched before this grid waits for the
  // update that precedes it in the stream (only W depends on that update).
  const uint32_t slab_full = smem_u32(slab_bars);   // [SLOTS]
  uint32_t slab_phases = 0;                         // of warp 3: the parity that the next wait for a slot waits for
  auto fetch_first_slabs = [&] {
    fetch_slab(us, slab_full, factor, a.ldu, nb, 0);
    if (n_sub > 1) fetch_slab(us + SLAB, slab_full + 8, factor, a.ldu, nb, 1);
  };
  auto wait_slab = [&](int slot) {
    if (!mbar_wait_lane(slab_full + 8 * slot, (slab_phases >> slot) & 1, a.fault, SLAB_FAULT)) {
      // given up: what has been started still ends before the block does
      for (const uint64_t t0 = global_ns(); !mbar_try(slab_full + 8 * slot, (slab_phases >> slot) & 1) && global_ns() - t0 < 100000000ull;) {}
    }
    slab_phases ^= 1u << slot;
  };
  if (warp == 3) {
    if (lane == 0)
      for (int i = 0; i < SLOTS; ++i) mbar_init(slab_full + 8 * i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    fetch_first_slabs();
  }
  chain_wait();
  chain_release();
  const float maxq = a.maxq;
  const bool wide_codes = (a.C & 15) == 0 && (reinterpret_cast<uintptr_t>(a.codes) & 15) == 0;
  const uint32_t group = (uint32_t)a.group;
  int row0 = blockIdx.x * group_rows, rows = 0;

  auto fill_grid = [&](int c, int from, int step) {   // of sub-block c
    constexpr int PER_ROW = UNIFORM ? 1 : SUB, AT_ONCE = UNIFORM ? 1 : 4;   // loads under way
    for (int first = from; first < rows * PER_ROW; first += AT_ONCE * step) {
      float s[AT_ONCE], z[AT_ONCE];
#pragma unroll
      for (int u = 0; u < AT_ONCE; ++u) {
        const int idx = first + u * step, r = idx / PER_ROW, j = c * SUB + (idx & (PER_ROW - 1));
        s[u] = 1.0f; z[u] = a.zero_default;
        if (r < rows && j < nb) {
          const int64_t off = (int64_t)(row0 + r) * a.s_rs + (int64_t)((uint32_t)(i1 + j) / group) * a.s_gs;
          s[u] = __ldg(a.scale + off);
          if (a.zero) z[u] = __ldg(a.zero + off);
        }
      }
#pragma unroll
      for (int u = 0; u < AT_ONCE; ++u) {
        const int idx = first + u * step, r = idx / PER_ROW;
        if (r < rows) gs[((c & 1) * PER_ROW + (idx & (PER_ROW - 1))) * group_rows + r] = make_float4(s[u], 1.0f / s[u], z[u], 0.0f);
      }
    }
  };
  auto stage_original = [&](int c, int from, int step) {   // sub-block c of every row
    if constexpr (INVERSE_FREE) {
      for (int idx = from; idx < rows * (SUB / 4); idx += step) {
        const int r = idx / (SUB / 4), k4 = (idx & (SUB / 4 - 1)) * 4;
        const bool keep = c * SUB + k4 < nb;
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&wos[((c & 1) * group_rows + r) * WO_LD + k4]);
        const float* g = a.Worig + (int64_t)(row0 + r) * a.ldwo + i1 + (keep ? c * SUB + k4 : 0);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(g), "r"(keep ? 16 : 0) : "memory");
      }
    }
  };
  // The launch has a CTA for every group of rows, so the loops over groups below end after the first.  They stay because
  // without them the compiler spills 17 registers of the helpers' (227 KB of shared memory leave no L1): a sweep of 1024 x 4096 takes 610 us instead
  // of 548, compact 699 instead of 598, 512 x 4096 568 instead of 536.
  auto begin_group = [&] {   // all warps: everything that the first two sub-blocks of rows row0 .. need
    rows = a.R - row0 < group_rows ? a.R - row0 : group_rows;
    if (warp == 3 && row0 != (int)blockIdx.x * group_rows) fetch_first_slabs();
    for (int idx = tid; idx < rows * (TILE / 4); idx += SUPER_THREADS) {
      const int r = idx >> 5, k4 = (idx & 31) * 4;
      const bool keep = k4 < nb;
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&ws[r * W_LD + k4]);
      const float* g = a.W + (int64_t)(row0 + r) * a.ldw + i1 + (keep ? k4 : 0);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(g), "r"(keep ? 16 : 0) : "memory");
    }
    stage_original(0, tid, SUPER_THREADS);
    stage_original(1, tid, SUPER_THREADS);
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (nb > TILE)
      for (int idx = tid; idx < rows * ((SUPER - TILE) / 4); idx += SUPER_THREADS) {
        const int r = idx / ((SUPER - TILE) / 4);
        *reinterpret_cast<float4*>(&ws[r * W_LD + TILE + (idx - r * ((SUPER - TILE) / 4)) * 4]) = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    fill_grid(0, tid, SUPER_THREADS);
    fill_grid(1, tid, SUPER_THREADS);
    if (warp == 3) {
      wait_slab(0);
      if (n_sub > 1) wait_slab(1);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
  };
  const bool errors_leave = a.err_planes || a.err;
  auto leave = [&](int k0, int r_begin, int r_end, int from, int step) {   // the errors of the tile at k0; sixteen lanes have a row
    for (int idx = r_begin * (TILE / 8) + from; idx < r_end * (TILE / 8); idx += step) {
      const int r = idx >> 4, k = k0 + (idx & 15) * 8;
      const float4 lo4 = *reinterpret_cast<const float4*>(ws + r * W_LD + k), hi4 = *reinterpret_cast<const float4*>(ws + r * W_LD + k + 4);
      write_errors(a, row0 + r, k, lo4, hi4, lane);
    }
  };
  auto end_group = [&] {   // all warps
    __syncthreads();
    if (errors_leave) leave(nb - TILE, 0, rows, tid, SUPER_THREADS);
    __syncthreads();   // the next group's weights replace the errors
  };

  if (warp < 4) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(CHAIN_REGS));
    for (; row0 < a.R; row0 += gridDim.x * group_rows) {
      begin_group();
      if (warp > 0) {
        // ---- what sub-block c + 2 needs, and the errors of the tiles that are done, a part of the rows at a time
        const int from = tid - 32, step = 32 * FETCHERS;
        int slot = 1;   // of slab c + 1
#pragma unroll 1
        for (int c = 0; c < n_sub; ++c) {
          if (warp == 3 && c > 0 && c + 1 < n_sub) wait_slab(slot);
          asm volatile("cp.async.wait_group 0;" ::: "memory");   // original weights of sub-block c + 1
          __syncthreads();
          // the chains have left slab c - 1, and hold the grid and the weights of sub-block c
          slot = slot == SLOTS - 1 ? 0 : slot + 1;
          if (c + 2 < n_sub) {
            if (warp == 3) fetch_slab(us + slot * SLAB, slab_full + 8 * slot, factor, a.ldu, nb, c + 2);
            stage_original(c + 2, from, step);
            asm volatile("cp.async.commit_group;" ::: "memory");
            fill_grid(c + 2, from, step);
          }
          // codes (and packed words) leave; a narrow last tile ends on a multiple of eight columns.  (From the chain: a sweep of 512 x 4096
          // took 562 us instead of 545.)
          if (from < rows) {
            const int j0 = c * SUB;
            const int64_t row = row0 + from;
            const uint4 code = cs[(c & 1) * group_rows + from];
            const uint32_t cw[SUB / 4] = {code.x, code.y, code.z, code.w};
            uint8_t* cdst = a.codes + row * a.C + i1 + j0;
            if (wide_codes && j0 + SUB <= nb) {
              *reinterpret_cast<uint4*>(cdst) = code;
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
          }
          constexpr int PER_TILE = TILE / SUB;
          if (errors_leave && c >= PER_TILE) {
            const int part = c % PER_TILE;
            leave((c / PER_TILE - 1) * TILE, rows * part / PER_TILE, rows * (part + 1) / PER_TILE, from, step);
          }
        }
      } else {
      // ---- chains.  Lanes past the last row repeat it and store nothing.  QUARTERS: four lanes have the same row; each runs
      // its chain, and brings a quad of the next columns up to date.
      const int own_row = QUARTERS ? lane & 7 : lane;
      const bool valid = lane < rows;
      const int r = own_row < rows ? own_row : rows - 1;
      const int64_t row = row0 + r;
      float* wrow = ws + r * W_LD;
      float* wglobal = a.W + row * a.ldw + i1;
      float w[SUB];
#pragma unroll
      for (int qd = 0; qd < SUB / 4; ++qd) {
        const float4 v = *reinterpret_cast<const float4*>(wrow + 4 * qd);
        w[4 * qd] = v.x; w[4 * qd + 1] = v.y; w[4 * qd + 2] = v.z; w[4 * qd + 3] = v.w;
      }
      int slot = 0;
#pragma unroll 1
      for (int c = 0; c < n_sub; ++c) {
        const int j0 = c * SUB;
        const bool enters = ((c + 1) * SUB) % TILE == 0;   // the following sub-block is the first of its tile
        float4 grid = gs[((c & 1) * (UNIFORM ? 1 : SUB)) * group_rows + r];
        float e[SUB];
        uint32_t cw[SUB / 4];
        const float* worow = wos + ((c & 1) * group_rows + r) * WO_LD;
        float4 wo = make_float4(0.f, 0.f, 0.f, 0.f);
        const float* ud = us + slot * SLAB + j0;   // the sub-block's own 16 x 16 block of the factor
        slot = slot == SLOTS - 1 ? 0 : slot + 1;
#pragma unroll
        for (int t = 0; t < SUB; ++t) {
          if (!UNIFORM && t > 0) grid = gs[((c & 1) * SUB + t) * group_rows + r];
          const float s_t = grid.x, r_t = grid.y, z_t = grid.z;
          float4 ur[SUB / 4];
#pragma unroll
          for (int qd = t >> 2; qd < SUB / 4; ++qd) {
            if (qd == (t >> 2) && (t & 3) == 3) continue;
            ur[qd] = *reinterpret_cast<const float4*>(ud + t * SUPER + 4 * qd);
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
          if (INVERSE_FREE && (t & 3) == 0) wo = *reinterpret_cast<const float4*>(worow + t);
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
#pragma unroll
          for (int qd = (t >> 2) + 1; qd < SUB / 4; ++qd) {
            float4 wq = make_float4(w[4 * qd], w[4 * qd + 1], w[4 * qd + 2], w[4 * qd + 3]);
            fma4(wq, ur[qd], et);
            w[4 * qd] = wq.x; w[4 * qd + 1] = wq.y; w[4 * qd + 2] = wq.z; w[4 * qd + 3] = wq.w;
          }
        }
        auto write_dequantized = [&] {
          if (!a.deq) return;
          T* dq = static_cast<T*>(a.deq) + row * a.C + i1 + j0;
#pragma unroll
          for (int t = 0; t < SUB; ++t) {
            if (!UNIFORM) grid = gs[((c & 1) * SUB + t) * group_rows + r];
            if (j0 + t < nb) dq[t] = from_float<T>(((float)((cw[t >> 2] >> (8 * (t & 3))) & 0xFFu) - grid.z) * grid.x);
          }
        };
        if (!UNIFORM && valid) write_dequantized();   // behind the barrier the table belongs to sub-block c + 2
        if (valid) {
          cs[(c & 1) * group_rows + r] = make_uint4(cw[0], cw[1], cw[2], cw[3]);
#pragma unroll
          for (int qd = 0; qd < SUB / 4; ++qd)
            *reinterpret_cast<float4*>(wrow + j0 + 4 * qd) = make_float4(e[4 * qd], e[4 * qd + 1], e[4 * qd + 2], e[4 * qd + 3]);
        }
        __syncthreads();
        if (c + 1 < n_sub) {
          // ---- next: this row's errors on the columns of the following sub-block
          if constexpr (QUARTERS) {
            const int at = j0 + SUB + 4 * (lane >> 3);
            float4 v = enters ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4*>(wrow + at);
#pragma unroll
            for (int t = 0; t < SUB; ++t) fma4(v, *reinterpret_cast<const float4*>(ud + t * SUPER + at - j0), e[t]);
            if (enters) {
              const float4 got = *reinterpret_cast<const float4*>(wrow + at);
              v = make_float4(got.x + v.x, got.y + v.y, got.z + v.z, got.w + v.w);
              if (own_row < rows && at < nb) *reinterpret_cast<float4*>(wglobal + at) = v;
            }
#pragma unroll
            for (int qd = 0; qd < SUB / 4; ++qd) {
              const int from = own_row + 8 * qd;
              w[4 * qd] = __shfl_sync(0xffffffffu, v.x, from); w[4 * qd + 1] = __shfl_sync(0xffffffffu, v.y, from);
              w[4 * qd + 2] = __shfl_sync(0xffffffffu, v.z, from); w[4 * qd + 3] = __shfl_sync(0xffffffffu, v.w, from);
            }
          } else {
            float4 v[SUB / 4];
#pragma unroll
            for (int qd = 0; qd < SUB / 4; ++qd)
              v[qd] = enters ? make_float4(0.f, 0.f, 0.f, 0.f) : *reinterpret_cast<const float4*>(wrow + j0 + SUB + 4 * qd);
#pragma unroll
            for (int t = 0; t < SUB; ++t)
#pragma unroll
              for (int qd = 0; qd < SUB / 4; ++qd) fma4(v[qd], *reinterpret_cast<const float4*>(ud + t * SUPER + SUB + 4 * qd), e[t]);
            if (enters) {
#pragma unroll
              for (int qd = 0; qd < SUB / 4; ++qd) {
                const float4 got = *reinterpret_cast<const float4*>(wrow + j0 + SUB + 4 * qd);
                v[qd] = make_float4(got.x + v[qd].x, got.y + v[qd].y, got.z + v[qd].z, got.w + v[qd].w);
                if (valid && j0 + SUB + 4 * qd < nb) *reinterpret_cast<float4*>(wglobal + j0 + SUB + 4 * qd) = v[qd];
              }
            }
#pragma unroll
            for (int qd = 0; qd < SUB / 4; ++qd) { w[4 * qd] = v[qd].x; w[4 * qd + 1] = v[qd].y; w[4 * qd + 2] = v[qd].z; w[4 * qd + 3] = v[qd].w; }
          }
        }
        if (UNIFORM && valid) write_dequantized();
      }
      }
      end_group();
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(HELPER_REGS));
    for (; row0 < a.R; row0 += gridDim.x * group_rows) {
      begin_group();
      // ---- the errors of sub-block c on the columns from sub-block c + 2 on.  More than 32 column quads: the warps divide into
      // the chunks of 32; fewer: the lanes of a warp divide into rows of `span` lanes, so that few lanes idle as the region shrinks
      const int hw = warp - 4;
      int slot = 0;
#pragma unroll 1
      for (int c = 0; c < n_sub; ++c) {
        const int j0 = c * SUB;
        const int quads = (n_sub * SUB - 2 * SUB - j0) / 4;
        const int chunks = quads > 96 ? 4 : quads > 64 ? 3 : quads > 32 ? 2 : 1;
        const int span = quads > 16 ? 32 : quads > 8 ? 16 : quads > 4 ? 8 : 4;
        const int quad = hw % chunks * 32 + (lane & (span - 1));
        const int per_warp = 32 / span, row_step = (HELPERS - hw % chunks + chunks - 1) / chunks * per_warp;
        const bool mine = quad < quads;
        const int k = j0 + 2 * SUB + 4 * quad;
        const bool near = k / TILE == j0 / TILE;
        // The tile of these columns is the next one: their own value joins what they have received.  Its first sub-block, which
        // the chains take after this one's errors, is ready one sub-block earlier.
        const bool first = (k & (TILE - 1)) < SUB;
        const bool enters = first ? (j0 + 2 * SUB) % TILE == 0 && k - j0 < 3 * SUB : (j0 + SUB) % TILE == 0 && k - j0 < SUB + TILE;
        float4 u[SUB];
        if (mine) {
#pragma unroll
          for (int t = 0; t < SUB; ++t) u[t] = *reinterpret_cast<const float4*>(us + slot * SLAB + t * SUPER + k);
        }
        slot = slot == SLOTS - 1 ? 0 : slot + 1;
        __syncthreads();
        // N rows at a time: a row by itself is a chain of sixteen FMAs
        auto update = [&](int r, auto n_rows) {
          constexpr int N = decltype(n_rows)::value;
          float* wr = ws + r * W_LD + k;
          const int ld = row_step * W_LD;
          float4 v[N];
#pragma unroll
          for (int i = 0; i < N; ++i) v[i] = near ? *reinterpret_cast<const float4*>(wr + i * ld) : make_float4(0.f, 0.f, 0.f, 0.f);
          const float* er = ws + r * W_LD + j0;
#pragma unroll
          for (int t4 = 0; t4 < SUB / 4; ++t4) {
            float4 e4[N];
#pragma unroll
            for (int i = 0; i < N; ++i) e4[i] = *reinterpret_cast<const float4*>(er + i * ld + 4 * t4);
#pragma unroll
            for (int i = 0; i < N; ++i) fma4(v[i], u[4 * t4], e4[i].x);
#pragma unroll
            for (int i = 0; i < N; ++i) fma4(v[i], u[4 * t4 + 1], e4[i].y);
#pragma unroll
            for (int i = 0; i < N; ++i) fma4(v[i], u[4 * t4 + 2], e4[i].z);
#pragma unroll
            for (int i = 0; i < N; ++i) fma4(v[i], u[4 * t4 + 3], e4[i].w);
          }
          if (!near) {
#pragma unroll
            for (int i = 0; i < N; ++i) {
              const float4 got = *reinterpret_cast<const float4*>(wr + i * ld);
              v[i] = make_float4(got.x + v[i].x, got.y + v[i].y, got.z + v[i].z, got.w + v[i].w);
            }
            if (enters && k < nb) {
              float* wg = a.W + (int64_t)(row0 + r) * a.ldw + i1 + k;
#pragma unroll
              for (int i = 0; i < N; ++i) {
                const float4 x = *reinterpret_cast<const float4*>(wg + (int64_t)i * row_step * a.ldw);
                v[i] = make_float4(x.x + v[i].x, x.y + v[i].y, x.z + v[i].z, x.w + v[i].w);
              }
              if (!first) {
#pragma unroll
                for (int i = 0; i < N; ++i) *reinterpret_cast<float4*>(wg + (int64_t)i * row_step * a.ldw) = v[i];
              }
            }
          }
#pragma unroll
          for (int i = 0; i < N; ++i) *reinterpret_cast<float4*>(wr + i * ld) = v[i];
        };
        int r = mine ? hw / chunks * per_warp + lane / span : rows;
        for (; r + 3 * row_step < rows; r += 4 * row_step) update(r, std::integral_constant<int, 4>{});
        for (; r + row_step < rows; r += 2 * row_step) update(r, std::integral_constant<int, 2>{});
        if (r < rows) update(r, std::integral_constant<int, 1>{});
      }
      end_group();
    }
  }
}

template <int DT>
int launch(bool chained, bool uniform, int grid, int rows, cudaStream_t st, const SweepArgs& args) {
  const bool free = args.Worig != nullptr;
  auto pick = [&](auto quarters) {
    constexpr bool Q = decltype(quarters)::value;
    return uniform ? (free ? sweep_super_kernel<DT, true, true, Q> : sweep_super_kernel<DT, true, false, Q>)
                   : (free ? sweep_super_kernel<DT, false, true, Q> : sweep_super_kernel<DT, false, false, Q>);
  };
  auto* kernel = rows <= ROWS ? pick(std::true_type{}) : pick(std::false_type{});
  MQ_CUDA(launch_chained(chained, kernel, dim3(grid), dim3(SUPER_THREADS), super_smem_bytes(rows, uniform), st, args, rows));
  return MQ_OK;
}

template <int DT, bool QUARTERS>
int configure_kernels() {
  constexpr int bytes = (int)super_smem_bytes(MAX_ROWS, true), by_column = (int)super_smem_bytes(MAX_ROWS, false);
  MQ_CUDA(cudaFuncSetAttribute(sweep_super_kernel<DT, true, true, QUARTERS>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  MQ_CUDA(cudaFuncSetAttribute(sweep_super_kernel<DT, true, false, QUARTERS>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  MQ_CUDA(cudaFuncSetAttribute(sweep_super_kernel<DT, false, true, QUARTERS>, cudaFuncAttributeMaxDynamicSharedMemorySize, by_column));
  MQ_CUDA(cudaFuncSetAttribute(sweep_super_kernel<DT, false, false, QUARTERS>, cudaFuncAttributeMaxDynamicSharedMemorySize, by_column));
  return MQ_OK;
}

template <int DT>
int configure_dtype() {
  MQ_TRY((configure_kernels<DT, true>()));
  return configure_kernels<DT, false>();
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

int sweep_super_block(bool chained, bool uniform, bool compact, int out_dtype, const SweepArgs& args, cudaStream_t st) {
  MQ_TRY(configure_once());
  const int spread = (int)ceil_div(args.R, COMPACT_CTAS), rows = compact && spread > ROWS ? spread : ROWS;
  const int grid = (int)ceil_div(args.R, rows);
  switch (out_dtype) {
    case MQ_F32: return launch<MQ_F32>(chained, uniform, grid, rows, st, args);
    case MQ_BF16: return launch<MQ_BF16>(chained, uniform, grid, rows, st, args);
    default: return launch<MQ_F16>(chained, uniform, grid, rows, st, args);
  }
}

}  // namespace mq
