// GPTQ row kernel: column-by-column quantisation with Hessian error feedback, several weight rows per CTA.
//
// Inputs are what the host prepared once per matrix: the column-permuted weights Wp [rows, cols] (activation order),
// the upper Cholesky factor U [cols, cols] of the inverse permuted Hessian, and one fixed scale per row and clip candidate (the
// caller keeps the best candidate per row).  A (row, candidate) pair is a row of its own here.  Rows are independent, so the only serial
// dimension is the column index, and what bounds the kernel is the chain of dependent operations along it.
//   * One warp per row walks a 128-column block (4 values per lane in registers, the current one broadcast with a shuffle,
//     the rank-1 feedback reads U from a shared 128x128 tile). The two divisions of a column sit on the chain: each is a
//     multiplication by a reciprocal and two fused corrections (`div_rn`) instead of the general routine.
//   * The block's 128 errors must reach every column right of it. The next block needs them at once (`near`: all warps of the CTA,
//     each thread a column of a row at a time); the columns beyond are updated by the 12 warps that own no row while the row warps
//     already walk the next block (`far`), off the chain. An element of U is loaded once per group of rows (four or eight).
// Small form: four rows and 16 warps per CTA, two diagonal tiles, of which the far warps fetch the next; 512 rows spread over 128 SMs.
// Large form: up to 20 rows, five per scheduler, and 32 warps; one diagonal tile, fetched during the near update. It is for more rows
// than four per SM, such as five clip candidates of one matrix, and is bound by issue slots as much as by the chain.
// 512 x 1536, 6-bit: one candidate 0.20 ms, five in one launch 0.85 ms. Before: eight rows per CTA, every warp doing the far updates of
// its row by itself, 2.42 ms for one; four rows with near and far update in one phase between two blocks 0.53 ms.
// The arithmetic inside a block is written with explicitly rounded operations (no fused multiply-add) so that the
// codes match the float32 reference except where the two summation orders of the trailing update differ.
//
// Reference behaviour: the full-Hessian GPTQ of records/track_10min_16mb/2026-03-25_ValCalib_GPTQ_XSA_BigramHash3072/
// train_gpt.py:1171-1224 (block size 128, act-order, per-row clip candidates).
#include <cuda_runtime.h>
#include <stdint.h>

#include "pgb.h"

namespace pgb {

namespace {
constexpr int GQ_ROWS = 4;                   // rows of the small form
constexpr int GQ_MAX_ROWS = 20;              // rows of the large one
constexpr int GQ_FAR_THREADS = 384;
constexpr int GQ_GROUP_SMALL = 4, GQ_GROUP_LARGE = 8;      // rows that share one pass over U in the far update
constexpr int GQ_BLOCK = 128;
constexpr int GQ_TILE = GQ_BLOCK * GQ_BLOCK;

// The code of x: sign(x) floor(|x| + 1/2) within [qmin, qmax]. The limits are whole numbers, so clamping may come first; below 2^23
// adding and subtracting 2^23 with the first addition rounded down is a floor (two additions where `floorf` is a slower
// conversion). NaN stays NaN: `walk_block` recognises by it what `div_rn` does not cover.
__device__ __forceinline__ float code_of(float x, float qmin, float qmax) {
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(x) : "f"(qmin));
  asm("min.NaN.f32 %0, %0, %1;" : "+f"(x) : "f"(qmax));
  return copysignf(__fsub_rn(__fadd_rd(__fadd_rn(fabsf(x), 0.5f), 8388608.f), 8388608.f), x);
}

// a / b rounded to nearest, given r = 1 / b rounded to nearest: a first quotient, its remainder, one correction (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", 1990). The theorem asks for a first quotient within
// one ulp, and a * r can be 1.5 ulp off; but only significand pairs whose quotient lies within 4.5 / 2^24 ulp of the middle between
// two floats could then round wrongly, and all 52,333,588 pairs within 9 / 2^24 were checked: none does. NaN where the first
// quotient is infinite or b outside [2^-60, 2^60] (`short_reciprocal`). A dividend below 2^-102, whose remainder is not exact,
// may give a quotient (below 2^-42) that is an ulp off.
__device__ __forceinline__ float div_rn(float a, float b, float r) {
  const float q = __fmul_rn(a, r);
  return __fmaf_rn(__fmaf_rn(-q, b, a), r, q);
}
__device__ __forceinline__ float short_reciprocal(float b) {
  const float m = fabsf(b);
  return m >= 0x1p-60f && m <= 0x1p60f ? __frcp_rn(b) : __int_as_float(0x7fffffff);
}

// One row's walk over a block with the general division: what `walk_block` falls back to. The row's values are updated in place.
__device__ __noinline__ void walk_general(const float* tile, float* w_row, int8_t* q_row, float* e_row, int lane, int nb, float s, float qmin, float qmax) {
  for (int j = 0; j < nb; ++j) {
    const float* u_row = tile + j * GQ_BLOCK;
    __syncwarp();
    const float w = w_row[j], x = __fdiv_rn(w, s);
    const float q = fminf(fmaxf(copysignf(floorf(fabsf(x) + 0.5f), x), qmin), qmax);      // NaN: qmin
    const float err = __fdiv_rn(__fsub_rn(w, __fmul_rn(q, s)), u_row[j]);
    if (lane == 0) {
      q_row[j] = (int8_t)q;
      e_row[j] = err;
    }
    for (int c = j + 1 + lane; c < nb; c += 32) w_row[c] = __fsub_rn(w_row[c], __fmul_rn(err, u_row[c]));
  }
}

// One row's walk over a block of 128 columns (`WHOLE`) or the last nb < 128 columns: without the end test of the ragged form
// the shared-memory reads of later columns move ahead of the dependency chain. A quotient that `div_rn` does not cover leaves NaN
// in its column's error and so in every later column's: the block is then walked again.
template <bool WHOLE>
__device__ __forceinline__ void walk_block(const float* __restrict__ tile, const float* __restrict__ sR, float* w_row, int8_t* q_row, float* e_row,
                                           int lane, int nb, float s, float rs, float qmin, float qmax) {
  float reg[4], err = 0.f;
#pragma unroll
  for (int ii = 0; ii < 4; ++ii) {
    const int c = ii * 32 + lane;
    reg[ii] = (WHOLE || c < nb) ? w_row[c] : 0.f;
  }
#pragma unroll
  for (int ii = 0; ii < 4; ++ii) {
    float my_q = 0.f, my_e = 0.f;
#pragma unroll 8
    for (int jj = 0; jj < 32; ++jj) {
      const int j = ii * 32 + jj;
      if (!WHOLE && j >= nb) break;                                        // uniform across the warp
      const float* u_row = tile + j * GQ_BLOCK;
      const float w = __shfl_sync(0xffffffffu, reg[ii], jj);
      const float q = code_of(div_rn(w, s, rs), qmin, qmax);
      err = div_rn(__fsub_rn(w, __fmul_rn(q, s)), u_row[j], sR[j]);
      if (lane == jj) {
        my_q = q;
        my_e = err;
      }
#pragma unroll
      for (int i2 = 0; i2 < 4; ++i2)
        if (i2 >= ii) {
          // columns left of j are finished: what the upper triangle's zeros would subtract from them is never read again
          const int c = i2 * 32 + lane;
          reg[i2] = __fsub_rn(reg[i2], __fmul_rn(err, u_row[c]));
        }
    }
    const int c = ii * 32 + lane;
    if (WHOLE || c < nb) {
      q_row[c] = (int8_t)my_q;
      e_row[c] = my_e;
    }
  }
  if (err != err) walk_general(tile, w_row, q_row, e_row, lane, nb, s, qmin, qmax);
}

template <int BYTES>
__device__ __forceinline__ void gq_copy(float* smem_dst, const float* gmem_src, bool valid) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(gmem_src), "n"(BYTES), "r"(valid ? BYTES : 0) : "memory");
}

// `rows` counts (candidate, row) pairs, candidate-major; R of them per CTA (one warp each), then 12 warps for the far updates.
// The small form's one CTA per SM may use 128 registers a thread; told only its threads, the compiler kept to 64 and spilled on the
// chain (512 x 1536: 0.26 ms instead of 0.19).
template <int GROUP, int MAX_THREADS, bool TWO_TILES>
__global__ void __launch_bounds__(MAX_THREADS, TWO_TILES ? 1 : 0)
gptq_rows_kernel(const float* __restrict__ Wp, const float* __restrict__ U, const float* __restrict__ scales, int8_t* __restrict__ Q, int rows,
                 int weight_rows, int cols, int R, float qmin, float qmax) {
  extern __shared__ __align__(16) float sm[];
  float* sU = sm;                                   // diagonal tiles of U, [128][128] each: this block's and, with two, the next one's
  float* sR = sU + (TWO_TILES ? 2 : 1) * GQ_TILE;   // [128] reciprocals of the current tile's diagonal
  float* sE = sR + GQ_BLOCK;                        // 2 x [R][128] scaled errors of a block
  float* sW = sE + 2 * R * GQ_BLOCK;                // [R][cols] working rows
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, threads = blockDim.x;
  const int row0 = blockIdx.x * R;
  const int live = min(R, rows - row0);
  for (int r = warp; r < R; r += threads / 32) {
    const float* src = Wp + (size_t)((row0 + min(r, live - 1)) % weight_rows) * cols;
    for (int c = lane; c < cols; c += 32) sW[r * cols + c] = r < live ? src[c] : 0.f;
  }
  for (int i = threadIdx.x; i < 2 * R * GQ_BLOCK; i += threads) sE[i] = 0.f;
  const bool wide = (cols & 3) == 0 && (reinterpret_cast<uintptr_t>(U) & 15) == 0;      // rows of U start on 16-byte boundaries
  auto load_tile = [&](int i1, int t, int nthreads) {    // elements outside the matrix read as zero
    const int nb = min(GQ_BLOCK, cols - i1);
    float* dst = sU + (TWO_TILES ? ((i1 / GQ_BLOCK) & 1) * GQ_TILE : 0);
    if (wide) {
      for (int idx = t * 4; idx < GQ_TILE; idx += nthreads * 4) {
        const int j = idx >> 7, c = idx & 127;
        const bool in = j < nb && c < nb;
        gq_copy<16>(dst + idx, in ? U + (size_t)(i1 + j) * cols + i1 + c : U, in);
      }
    } else {
      for (int idx = t; idx < GQ_TILE; idx += nthreads) {
        const int j = idx >> 7, c = idx & 127;
        const bool in = j < nb && c < nb;
        gq_copy<4>(dst + idx, in ? U + (size_t)(i1 + j) * cols + i1 + c : U, in);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto reciprocals = [&](int i1) {
    const float* tile = sU + (TWO_TILES ? ((i1 / GQ_BLOCK) & 1) * GQ_TILE : 0);
    if (threadIdx.x < min(GQ_BLOCK, cols - i1)) sR[threadIdx.x] = short_reciprocal(tile[threadIdx.x * (GQ_BLOCK + 1)]);
  };
  load_tile(0, threadIdx.x, threads);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  reciprocals(0);
  __syncthreads();
  const float s = warp < live ? scales[row0 + warp] : 1.f;
  const float rs = short_reciprocal(s);
  for (int i1 = 0; i1 < cols; i1 += GQ_BLOCK) {
    const int nb = min(GQ_BLOCK, cols - i1);
    const int buf = (i1 / GQ_BLOCK) & 1;
    if (warp < R) {
      if (warp < live) {
        const float* tile = sU + (TWO_TILES ? buf * GQ_TILE : 0);
        float* e_row = sE + (buf * R + warp) * GQ_BLOCK;
        float* w_row = sW + warp * cols + i1;
        int8_t* q_row = Q + (size_t)(row0 + warp) * cols + i1;
        if (nb == GQ_BLOCK) walk_block<true>(tile, sR, w_row, q_row, e_row, lane, nb, s, rs, qmin, qmax);
        else walk_block<false>(tile, sR, w_row, q_row, e_row, lane, nb, s, rs, qmin, qmax);
      }
    } else {
      const int t = threadIdx.x - 32 * R;
      if (TWO_TILES && i1 + GQ_BLOCK < cols) load_tile(i1 + GQ_BLOCK, t, GQ_FAR_THREADS);
      if (i1 > 0) {
        // far: the previous block's errors into the columns beyond this block, w[r][c] -= sum_j err[r][j] * U[j][c]
        for (int c = i1 + GQ_BLOCK + t; c < cols; c += GQ_FAR_THREADS) {
          const float* u = U + (size_t)(i1 - GQ_BLOCK) * cols + c;
          for (int r0 = 0; r0 < live; r0 += GROUP) {
            const float* e_prev = sE + ((buf ^ 1) * R + r0) * GQ_BLOCK;
            const int rn = min(GROUP, R - r0);              // R is a multiple of 4: a group may be half full
            float a[GROUP][4] = {};
#pragma unroll 4
            for (int j = 0; j < GQ_BLOCK; j += 4) {
              const float u0 = __ldg(u + (size_t)j * cols), u1 = __ldg(u + (size_t)(j + 1) * cols), u2 = __ldg(u + (size_t)(j + 2) * cols),
                          u3 = __ldg(u + (size_t)(j + 3) * cols);
#pragma unroll
              for (int r = 0; r < GROUP; ++r) {
                if (r >= 4 && r >= rn) break;
                const float4 e = *reinterpret_cast<const float4*>(e_prev + r * GQ_BLOCK + j);
                a[r][0] = fmaf(e.x, u0, a[r][0]);
                a[r][1] = fmaf(e.y, u1, a[r][1]);
                a[r][2] = fmaf(e.z, u2, a[r][2]);
                a[r][3] = fmaf(e.w, u3, a[r][3]);
              }
            }
#pragma unroll
            for (int r = 0; r < GROUP; ++r)
              if (r < 4 || r < rn) sW[(r0 + r) * cols + c] -= (a[r][0] + a[r][1]) + (a[r][2] + a[r][3]);
          }
        }
      }
      if (TWO_TILES) asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();                                // this block's errors and the far updates (and the next of two tiles) are visible
    if (i1 + GQ_BLOCK >= cols) break;
    if (!TWO_TILES) load_tile(i1 + GQ_BLOCK, threadIdx.x, threads);
    if (TWO_TILES) reciprocals(i1 + GQ_BLOCK);
    // near: this (whole) block's errors into the next block's columns
    for (int i = threadIdx.x; i < R * GQ_BLOCK; i += threads) {
      const int r = i >> 7, c = i1 + GQ_BLOCK + (i & 127);
      if (c < cols) {
        const float* e_row = sE + (buf * R + r) * GQ_BLOCK;
        const float* u = U + (size_t)i1 * cols + c;
        float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll 8
        for (int j = 0; j < GQ_BLOCK; j += 4) {
          const float4 e = *reinterpret_cast<const float4*>(e_row + j);
          a0 = fmaf(e.x, __ldg(u + (size_t)j * cols), a0);
          a1 = fmaf(e.y, __ldg(u + (size_t)(j + 1) * cols), a1);
          a2 = fmaf(e.z, __ldg(u + (size_t)(j + 2) * cols), a2);
          a3 = fmaf(e.w, __ldg(u + (size_t)(j + 3) * cols), a3);
        }
        sW[r * cols + c] -= (a0 + a1) + (a2 + a3);
      }
    }
    if (!TWO_TILES) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
      reciprocals(i1 + GQ_BLOCK);
    }
    __syncthreads();
  }
}

size_t gq_smem(int R, int cols, bool two_tiles) {
  return ((two_tiles ? 2 : 1) * (size_t)GQ_TILE + GQ_BLOCK + 2 * (size_t)R * GQ_BLOCK + (size_t)R * cols) * sizeof(float);
}

template <int GROUP, int MAX_THREADS, bool TWO_TILES>
void gq_launch(const float* Wp, const float* U, const float* scales, int8_t* Q, int rows, int weight_rows, int cols, int R, float qmin, float qmax,
               cudaStream_t st) {
  auto kern = gptq_rows_kernel<GROUP, MAX_THREADS, TWO_TILES>;
  const size_t smem = gq_smem(R, cols, TWO_TILES);
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  kern<<<(rows + R - 1) / R, 32 * R + GQ_FAR_THREADS, smem, st>>>(Wp, U, scales, Q, rows, weight_rows, cols, R, qmin, qmax);
}
}  // namespace

void gptq_rows(const float* Wp, const float* U, const float* scales, int8_t* Q, int candidates, int rows, int cols, int bits, cudaStream_t st) {
  if (rows <= 0 || cols <= 0 || candidates <= 0) return;
  if (bits < 2 || bits > 8) throw std::runtime_error("gptq_rows: bits must be in 2..8");
  if ((long long)rows * candidates > 0x7fffffffll) throw std::runtime_error("gptq_rows: too many rows");
  const size_t limit = 227 * 1024;
  if (gq_smem(GQ_ROWS, cols, true) > limit)
    throw std::runtime_error("gptq_rows: rows of more than " + std::to_string((limit - gq_smem(GQ_ROWS, 0, true)) / sizeof(float) / GQ_ROWS) +
                             " columns do not fit in shared memory");
  const float qmax = (float)((1 << (bits - 1)) - 1), qmin = -(float)(1 << (bits - 1));
  const int total = rows * candidates;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // A CTA's time grows more slowly than its rows (one round of 1,536 columns: 4 rows 0.20 ms, 8 0.34, 12 0.52, 16 0.63, 20 0.82), so
  // the fewest rounds win: four rows per CTA while those fit in one round, else as many as shared memory allows, evened out over the
  // rounds. ms this way / in rounds of the small form: 1,184 rows 0.34 / 0.38, 1,776 0.53 / 0.57, 2,368 0.64 / 0.75, 2,960 0.84 / 0.93,
  // 5,920 1.67 / 1.85. (Four rows in the large form, two CTAs per SM, measured 0.31, 0.53, 0.60, 0.80 and 1.47; not used.)
  int R = GQ_ROWS;
  if ((total + GQ_ROWS - 1) / GQ_ROWS > sms) {
    int most = GQ_MAX_ROWS;
    while (most > GQ_ROWS && gq_smem(most, cols, false) > limit) most -= 4;
    const int rounds = (total + sms * most - 1) / (sms * most);
    R = std::min(most, ((total + sms * rounds - 1) / (sms * rounds) + 3) / 4 * 4);
  }
  if (R == GQ_ROWS) gq_launch<GQ_GROUP_SMALL, 32 * GQ_ROWS + GQ_FAR_THREADS, true>(Wp, U, scales, Q, total, rows, cols, R, qmin, qmax, st);
  else gq_launch<GQ_GROUP_LARGE, 32 * GQ_MAX_ROWS + GQ_FAR_THREADS, false>(Wp, U, scales, Q, total, rows, cols, R, qmin, qmax, st);
}

}  // namespace pgb
