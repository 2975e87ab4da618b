// The factor that GPTQ's error feedback runs on: U with inv(H) = U^T U, U upper triangular, from the damped Hessian with its columns in
// activation order. With rows and columns in reverse order, H = L L^T and U is inv(L) reversed again. In fp64, like the library
// factorisation and triangular solve it replaces.
//
// One cooperative launch. The matrix is cut into 64 x 64 tiles; step k factorises tile (k, k) and inverts the factor (one CTA), then
// every CTA takes tiles: L_ik = A_ik inv(L_kk)^T and row k of the inverse, X_kj = inv(L_kk) Y_kj, then the updates A_ij -= L_ik L_jk^T and
// Y_ij -= L_ik X_kj. So the inverse grows with the factor and costs no steps of its own. What bounds it is the chain of columns
// inside the diagonal tiles (a reciprocal and a rank-1 update each) and two grid barriers a step; the update of
// the next diagonal tile and its factorisation run beside the other updates.
#include <cuda_runtime.h>
#include <stdint.h>

#include "pgb.h"

namespace pgb {

namespace {
constexpr int FB = 64;                        // tile
constexpr int FT = 256;                       // threads: 16 x 16, each 2 x 2 pairs of rows and columns of a tile
constexpr int FP = FB + 2;                    // pitch of a tile in shared memory (doubles)
constexpr size_t FSMEM = 2 * (size_t)FB * FP * sizeof(double);
constexpr unsigned long long F_WAIT_NS = 2000000000ull;

struct FactorParams {
  const float* H;                             // [c][c] damped
  const long long* order;                     // [c]: row i of the factorised matrix is row order[i] of H
  double* A;                                  // [n][n] work: becomes L (lower tiles)
  double* Y;                                  // [n][n] work: becomes inv(L)
  double* dinv;                               // [64][64] inverse of the current diagonal factor
  float* U;                                   // [c][c]
  int* info;                                  // {0: factorised, k > 0: the leading minor of order k is not positive, -1: a wait ran out; barrier counter}
  int c, nb;
};

// All CTAs; bounded: false once a CTA did not come within two seconds.
__device__ bool grid_barrier(const FactorParams& p, unsigned target) {
  __shared__ int good;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    unsigned* counter = reinterpret_cast<unsigned*>(p.info + 1);
    atomicAdd(counter, 1u);
    unsigned seen;
    unsigned long long t0 = 0, t = 0;
    int ok = 1;
    for (int spin = 0;; ++spin) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
      if (seen >= target) break;
      if ((spin & 255) == 255) {
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        if (t0 == 0) t0 = t;
        if (t - t0 > F_WAIT_NS) {
          atomicExch(p.info, -1);
          ok = 0;
          break;
        }
      }
    }
    __threadfence();
    good = ok;
  }
  __syncthreads();
  return good != 0;
}

struct Lane {
  int r, c;                                   // this thread's rows r, r + 1, r + 32, r + 33 and columns likewise
  __device__ Lane() {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    c = 2 * ((lane & 7) + 8 * (warp & 1));
    r = 2 * ((lane >> 3) + 4 * (warp >> 1));
  }
  __device__ int row(int i) const { return r + (i & 1) + 32 * (i >> 1); }
  __device__ int col(int i) const { return c + (i & 1) + 32 * (i >> 1); }
};

// s[k][r] = g[r][k], or s[k][c] = g[k][c]
template <bool TRANSPOSE>
__device__ void load_tile(double* s, const double* g, size_t ld) {
#pragma unroll
  for (int it = 0; it < FB * FB / 2 / FT; ++it) {
    const int idx = it * FT + threadIdx.x;
    if constexpr (TRANSPOSE) {
      const int k = 2 * ((idx & 3) + 4 * ((idx >> 5) & 7)), r = ((idx >> 2) & 7) + 8 * (idx >> 8);
      const double2 x = __ldcg(reinterpret_cast<const double2*>(g + r * ld + k));
      s[k * FP + r] = x.x;
      s[(k + 1) * FP + r] = x.y;
    } else {
      const int k = idx >> 5, c = 2 * (idx & 31);
      *reinterpret_cast<double2*>(s + k * FP + c) = __ldcg(reinterpret_cast<const double2*>(g + k * ld + c));
    }
  }
}

// acc[i][j] += sum_k sa[k][row i] sb[k][col j]
__device__ __forceinline__ void tile_mma(const double* sa, const double* sb, const Lane& t, double (&acc)[4][4]) {
#pragma unroll 8
  for (int k = 0; k < FB; ++k) {
    const double2 a0 = *reinterpret_cast<const double2*>(sa + k * FP + t.r), a1 = *reinterpret_cast<const double2*>(sa + k * FP + t.r + 32);
    const double2 b0 = *reinterpret_cast<const double2*>(sb + k * FP + t.c), b1 = *reinterpret_cast<const double2*>(sb + k * FP + t.c + 32);
    const double a[4] = {a0.x, a0.y, a1.x, a1.y}, b[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
  }
}

__device__ __forceinline__ void store_tile(double* g, size_t ld, const Lane& t, const double (&acc)[4][4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h)
      __stcg(reinterpret_cast<double2*>(g + t.row(i) * ld + t.c + 32 * h), make_double2(acc[i][2 * h], acc[i][2 * h + 1]));
}

// g -= sa^T sb
__device__ __forceinline__ void update_tile(double* g, size_t ld, const double* sa, const double* sb, const Lane& t) {
  double acc[4][4] = {};
  double2 old[4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) old[i][h] = __ldcg(reinterpret_cast<const double2*>(g + t.row(i) * ld + t.c + 32 * h));
  tile_mma(sa, sb, t, acc);
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      acc[i][2 * h] = old[i][h].x - acc[i][2 * h];
      acc[i][2 * h + 1] = old[i][h].y - acc[i][2 * h + 1];
    }
  store_tile(g, ld, t, acc);
}

// row tile `ti` and column tile `tj` of inv(L), reversed, into U
__device__ __forceinline__ void write_u(const FactorParams& p, int ti, int tj, const Lane& t, const double (&x)[4][4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = ti * FB + t.row(i), c = tj * FB + t.col(j);
      if (r < p.c && c < p.c) p.U[(size_t)(p.c - 1 - r) * p.c + (p.c - 1 - c)] = (float)x[i][j];
    }
}

// 1 / x to a few units in the last place: the single-precision reciprocal r, then r (1 + e + e^2) with e = 1 - x r, |e| < 2^-22. Three
// dependent fp64 operations (each ~40 clocks) where the rounded reciprocal has more than twice as many.
__device__ __forceinline__ double reciprocal(double x) {
  if (!(fabs(x) > 0x1p-100 && fabs(x) < 0x1p100)) return __drcp_rn(x);
  float r0;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"((float)x));
  const double r = (double)r0;
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

// inv of the diagonal blocks of 2 W from those of W in `sa` (zeros above the diagonal); `sb` holds M. Each thread has NC columns of a row, two
// sums for each.
template <int W>
__device__ __forceinline__ void double_inverse(double* sa, const double* sb) {
  constexpr int PER = FT / (FB / (2 * W)), NC = W * W / PER;
  const int o = (threadIdx.x / PER) * 2 * W, w = threadIdx.x % PER, r = w / (W / NC), c = (w % (W / NC)) * NC;
  double s[NC][2] = {};
#pragma unroll 8
  for (int q = 0; q < W; ++q) {
    const double m = sb[(o + W + r) * FP + o + q];
#pragma unroll
    for (int i = 0; i < NC; ++i) s[i][q & 1] = fma(m, sa[(o + q) * FP + o + c + i], s[i][q & 1]);
  }
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    sa[(o + r) * FP + o + W + c + i] = s[i][0] + s[i][1];
    s[i][0] = s[i][1] = 0.0;
  }
  __syncthreads();
#pragma unroll 8
  for (int q = 0; q < W; ++q) {
    const double m = sa[(o + W + r) * FP + o + W + q];
#pragma unroll
    for (int i = 0; i < NC; ++i) s[i][q & 1] = fma(m, sa[(o + q) * FP + o + W + c + i], s[i][q & 1]);
  }
#pragma unroll
  for (int i = 0; i < NC; ++i) sa[(o + W + r) * FP + o + c + i] = -(s[i][0] + s[i][1]);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < NC; ++i) sa[(o + r) * FP + o + W + c + i] = 0.0;      // the product in between stood right of the diagonal
  __syncthreads();
}

// Factor of the diagonal tile (this thread's 4 x 4 part in `a`) and its inverse. The columns stay unscaled while the tile is reduced, A = M D M^T
// with M unit lower triangular: a column then costs one reciprocal on the chain instead of a reciprocal root. Sixteen columns at a time are
// reduced by one warp in registers (two rows a lane; a column's values reach the others by shuffle), then all warps update the rest
// of the tile. inv(M) comes from its 16 x 16 diagonal blocks by doubling, inv([P 0; Q R]) = [inv(P) 0; -inv(R) Q inv(P) inv(R)], and the
// roots of D at the end. A tile takes 23 us, 12 of them the columns of its panels. (Column by column with the whole CTA, a barrier
// and a reciprocal in every thread each, a matrix of 1,536 took 1,103 us; so 895, the library's factorisation and solve 1,860.)
__device__ void factor_tile(const FactorParams& p, int k, double* sa, double* sb, const Lane& t, const double (&a)[4][4]) {
  __shared__ double d[FB], rs[FB];                     // D and its reciprocal roots
  constexpr int PW = 16;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) sa[t.row(i) * FP + t.col(j)] = a[i][j];
  __syncthreads();
#pragma unroll 1
  for (int c0 = 0; c0 < FB; c0 += PW) {
    if (warp == 0) {
      double x0[PW], x1[PW];                           // rows `lane` and `lane + 32`
#pragma unroll
      for (int j = 0; j < PW; ++j) {
        x0[j] = sa[lane * FP + c0 + j];
        x1[j] = sa[(lane + 32) * FP + c0 + j];
      }
      const bool hi = c0 >= 32;
#pragma unroll
      for (int j = 0; j < PW; ++j) {
        const double mine = hi ? x1[j] : x0[j];
        double v[PW];                                  // the column's values in the panel's own rows, its row by symmetry
#pragma unroll
        for (int q = j; q < PW; ++q) v[q] = __shfl_sync(0xffffffffu, mine, (c0 + q) & 31);
        const double rd = reciprocal(v[j]);
        const double m0 = lane > c0 + j ? x0[j] * rd : 0.0, m1 = lane + 32 > c0 + j ? x1[j] * rd : 0.0;
#pragma unroll
        for (int q = j + 1; q < PW; ++q) {
          x0[q] = fma(-m0, v[q], x0[q]);
          x1[q] = fma(-m1, v[q], x1[q]);
        }
        sb[lane * FP + c0 + j] = lane == c0 + j ? 1.0 : m0;
        sb[(lane + 32) * FP + c0 + j] = lane + 32 == c0 + j ? 1.0 : m1;
        sa[lane * FP + c0 + j] = x0[j];
        sa[(lane + 32) * FP + c0 + j] = x1[j];
        if (lane == 0) {
          d[c0 + j] = v[j];
          if (!(v[j] > 0.0)) atomicCAS(p.info, 0, k * FB + c0 + j + 1);
        }
      }
    }
    __syncthreads();
    const int r0 = c0 + PW + (threadIdx.x >> 4), q0 = c0 + PW + (threadIdx.x & 15);
    // all of this thread's sums at once, rows past the end clamped and not stored: a branch in here would put every step's latency in a row
    double u[3][3] = {};
#pragma unroll
    for (int q = 0; q < PW; ++q) {
      double mr[3], ac[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        mr[i] = sb[min(r0 + PW * i, FB - 1) * FP + c0 + q];
        ac[i] = sa[min(q0 + PW * i, FB - 1) * FP + c0 + q];
      }
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) u[i][j] = fma(mr[i], ac[j], u[i][j]);
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
      if (r0 + PW * i < FB)
#pragma unroll
        for (int j = 0; j <= i; ++j) sa[(r0 + PW * i) * FP + q0 + PW * j] -= u[i][j];
    __syncthreads();
  }
  // inverses of the 16 x 16 diagonal blocks: a warp each, a lane per column
  if (warp < FB / PW && lane < PW) {
    const int o = warp * PW;
    double x[PW];
#pragma unroll
    for (int i = 0; i < PW; ++i) x[i] = i == lane ? 1.0 : 0.0;
#pragma unroll
    for (int i = 0; i < PW; ++i)
#pragma unroll
      for (int r = i + 1; r < PW; ++r) x[r] = fma(-sb[(o + r) * FP + o + i], x[i], x[r]);
#pragma unroll
    for (int i = 0; i < PW; ++i) sa[(o + i) * FP + o + lane] = x[i];
  }
  if (threadIdx.x >= FT - FB) rs[threadIdx.x - (FT - FB)] = 1.0 / sqrt(d[threadIdx.x - (FT - FB)]);
  __syncthreads();
  // from blocks of W to blocks of 2 W; the product in between stands in the unused block right of the diagonal
  double_inverse<PW>(sa, sb);
  double_inverse<2 * PW>(sa, sb);
  // inv(L) = D^-1/2 inv(M)
  double x[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) x[i][j] = sa[t.row(i) * FP + t.col(j)] * rs[t.row(i)];
  store_tile(p.dinv, FB, t, x);
  write_u(p, k, k, t, x);
  store_tile(p.Y + ((size_t)k * FB) * (p.nb * FB) + (size_t)k * FB, (size_t)p.nb * FB, t, x);
}

__global__ void __launch_bounds__(FT, 1) gptq_factor_kernel(const FactorParams p) {
  extern __shared__ __align__(16) double fsm[];
  double* sa = fsm;
  double* sb = fsm + FB * FP;
  const int n = p.nb * FB, nb = p.nb;
  const size_t ld = n;
  const Lane t;
  unsigned phase = 0;
  auto tile = [&](double* m, int i, int j) { return m + (size_t)i * FB * ld + (size_t)j * FB; };
  auto load_update = [&](int i, int j, int k, bool inverse) {      // A_ij -= L_ik L_jk^T, or Y_ij -= L_ik X_kj
    __syncthreads();
    load_tile<true>(sa, tile(p.A, i, k), ld);
    if (inverse) load_tile<false>(sb, tile(p.Y, k, j), ld);
    else load_tile<true>(sb, tile(p.A, j, k), ld);
    __syncthreads();
  };
  // the permuted matrix in fp64, a unit diagonal behind its last column
  for (size_t i = (size_t)blockIdx.x * FT + threadIdx.x; i < (size_t)n * n; i += (size_t)gridDim.x * FT) {
    const int r = (int)(i / n), c = (int)(i - (size_t)r * n);
    if (r / FB >= c / FB) {
      double v = r == c ? 1.0 : 0.0;
      if (r < p.c && c < p.c) v = (double)p.H[(size_t)p.order[r] * p.c + p.order[c]];
      p.A[i] = v;
      p.Y[i] = 0.0;
    }
  }
  for (size_t i = (size_t)blockIdx.x * FT + threadIdx.x; i < (size_t)p.c * p.c; i += (size_t)gridDim.x * FT) p.U[i] = 0.f;
  if (!grid_barrier(p, ++phase * gridDim.x)) return;
  for (int k = -1; k < nb; ++k) {
    if (k >= 0) {
      // column k of L and row k of the inverse
      const int tasks = nb - 1;
      for (int w = (int)blockIdx.x; w < tasks; w += gridDim.x) {
        const bool inverse = w < k;
        const int i = inverse ? w : w + 1;
        __syncthreads();
        double acc[4][4] = {};
        if (inverse) {                        // X_ki = inv(L_kk) Y_ki
          load_tile<true>(sa, p.dinv, FB);
          load_tile<false>(sb, tile(p.Y, k, i), ld);
        } else {                              // L_ik = A_ik inv(L_kk)^T
          load_tile<true>(sa, tile(p.A, i, k), ld);
          load_tile<true>(sb, p.dinv, FB);
        }
        __syncthreads();
        tile_mma(sa, sb, t, acc);
        if (inverse) {
          store_tile(tile(p.Y, k, i), ld, t, acc);
          write_u(p, k, i, t, acc);
        } else {
          store_tile(tile(p.A, i, k), ld, t, acc);
        }
      }
      if (!grid_barrier(p, ++phase * gridDim.x)) return;
    }
    if (k + 1 == nb) break;
    // updates of the tiles below and right of k; the first CTA takes the next diagonal tile and factorises it
    if (blockIdx.x == 0) {
      double acc[4][4];
      double* g = tile(p.A, k + 1, k + 1);
      if (k >= 0) {
        load_update(k + 1, k + 1, k, false);
        update_tile(g, ld, sa, sb, t);
        __syncthreads();
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = __ldcg(g + t.row(i) * ld + t.col(j));
      factor_tile(p, k + 1, sa, sb, t, acc);
    } else if (k >= 0) {
      const int m = nb - 1 - k;               // tile rows left
      const int upd = m * (m + 1) / 2 - 1, inv = m * (k + 1);
      for (int w = (int)blockIdx.x - 1; w < upd + inv; w += gridDim.x - 1) {
        int i, j;
        if (w < upd) {
          i = (int)((sqrtf(8.f * (w + 1) + 1.f) - 1.f) * 0.5f);
          while ((i + 1) * (i + 2) / 2 <= w + 1) ++i;
          while (i * (i + 1) / 2 > w + 1) --i;
          j = w + 1 - i * (i + 1) / 2;
          load_update(k + 1 + i, k + 1 + j, k, false);
          update_tile(tile(p.A, k + 1 + i, k + 1 + j), ld, sa, sb, t);
        } else {
          i = (w - upd) / (k + 1);
          j = (w - upd) - i * (k + 1);
          load_update(k + 1 + i, j, k, true);
          update_tile(tile(p.Y, k + 1 + i, j), ld, sa, sb, t);
        }
      }
    }
    if (!grid_barrier(p, ++phase * gridDim.x)) return;
  }
}
}  // namespace

size_t gptq_factor_work_doubles(int c) {
  const size_t n = ((size_t)c + FB - 1) / FB * FB;
  return 2 * n * n + FB * FB;
}

void gptq_factor(const float* H, const long long* order, double* work, float* U, int* info, int c, cudaStream_t st) {
  if (c <= 0) throw std::runtime_error("gptq_factor: empty matrix");
  FactorParams p;
  p.H = H;
  p.order = order;
  p.U = U;
  p.info = info;
  p.c = c;
  p.nb = (c + FB - 1) / FB;
  const size_t n = (size_t)p.nb * FB;
  p.A = work;
  p.Y = work + n * n;
  p.dinv = work + 2 * n * n;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaFuncSetAttribute(gptq_factor_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FSMEM);
  const int tiles = p.nb * (p.nb + 1) / 2 + p.nb;
  const int grid = std::max(2, std::min(sms, tiles));
  void* args[] = {&p};
  if (cudaMemsetAsync(info, 0, 2 * sizeof(int), st) != cudaSuccess ||
      cudaLaunchCooperativeKernel((const void*)gptq_factor_kernel, dim3(grid), dim3(FT), args, FSMEM, st) != cudaSuccess)
    throw std::runtime_error("gptq_factor: the launch was refused");
}

}  // namespace pgb
