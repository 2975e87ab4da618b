// Persistent warp-specialised bf16 GEMM for sm_100a: TMA -> shared memory -> tcgen05.mma -> TMEM -> epilogue.
//
//   D[b][m][n] = epilogue( sum_k A[b][m][k] * B[b][n][k] )
//
// Both operands may be stored K-contiguous ("K-major", [rows][K]) or row-contiguous along M/N
// ("MN-major", [K][rows]); the tensor core reads either through the shared-memory descriptor, so the
// three GEMMs of a linear layer need no transposes:
//   forward  Y = X W^T         A = X  [T][K]  K-major     B = W  [N][K]  K-major
//   dX = dY W                  A = dY [T][N]  K-major     B = W  [N][K]  MN-major (reduction over N)
//   dW = dY^T X                A = dY [T][N]  MN-major    B = X  [T][K]  MN-major (reduction over T, split-K)
// It replaces the cuBLAS calls of the reference's GEMM engine
// (parameter-golf-rs/crates/pg-kernels/src/gemm.rs:158-179,501-698) and the elementwise kernels that
// follow them, which become epilogues here.
//
// CTA = 10 warps: warp 0 issues TMA loads, warp 1 owns TMEM and issues the MMAs (one elected lane),
// warps 2..9 read the accumulator back (tcgen05.ld, one row per thread) and run the epilogue. Two
// accumulators (2 x BN TMEM columns) let the epilogue of tile i overlap the main loop of tile i+1.
// Tile 128 x BN x 64, BN in {64, 128, 256} (`pick_tile`), 256 x 256 by a pair of CTAs in most of the 256-column forms (`tile_ctas`);
// grid = min(#tiles, #SMs); tile index = n fastest so CTAs working at the same time share the rows of the large operand in L2. The 64-column form has four epilogue warps (6 warps in all).
#include <cmath>

#include "common.cuh"
#include "launch.h"
#include "pgb.h"
#include "tma_host.h"

namespace pgb {

constexpr int BM = 128;
constexpr int BK = 64;
// TMA warp, MMA warp, epilogue warps: two per TMEM lane quarter (one for 64 columns, so that a warp still owns whole heads)
constexpr int epi_warps(int bn) { return bn == 64 ? 4 : 8; }
constexpr int gemm_threads(int bn) { return 64 + 32 * epi_warps(bn); }
// 256-column tiles are computed by two CTAs on neighbouring SMs: 256 rows, 128 in each one's tensor memory, each holding its own rows of A
// and half of B's columns in shared memory. A K step then pulls 32 KB through L2 per CTA instead of 48, which is what bounds the
// large products (98,304 x 1536 x 512: 1.8 GB of operands). us alone / in pairs, 98,304 rows: 512 columns from 1536 125 / 111, with
// the residual 139 / 127, 512 from 1024 94 / 82; weight gradients of 512 x 1536 119 / 109. Not where a short sum meets a second operand:
// the output stage is then the longer part, and a pair's two have to wait for each other (activation gradient from 512 195 / 217).
constexpr int tile_ctas(int bn, int epi) { return bn == 256 && epi != EPI_RESID_BF16 && epi != EPI_MUL_ACTGRAD && epi != EPI_MUL_ACTROOT ? 2 : 1; }

struct GemmKernelParams {
  int M, N, K, batch;
  int tiles_m, tiles_n, splits, kb_per_split, kb_total;
  long long ldd, stride_d;
  long long ld_aux, stride_aux;
  void* D;
  void* D2;
  const void* aux;
  const float* colscale;
  float alpha, beta, slope;
  int* status;
  const int* wait_flag;   // optional: B (the weights) is valid once *wait_flag >= wait_value (peer ranks push it)
  int wait_value;
  int seg_rows[2];        // fp32 epilogues: rows >= seg_rows[k] (> 0) are written to seg_D[k] as row m - seg_rows[k]
  float* seg_D[2];
  int aligned;             // rows of the bf16 outputs and of the second operand start on 16-byte boundaries
  int aux_l2_prefetch;     // the producer warp pulls the next tile's second operand into L2 through `map_x`
  const float* batch_sumsq;   // optional: alpha and beta of batch b are multiplied by 1 / (sqrt(batch_sumsq[b]) + 1e-7) ^ sumsq_pow
  int sumsq_pow;
  const float* rope_cos;      // EPI_QKV_NORM_ROPE
  const float* rope_sin;
  const float* head_gain;
  int q_heads, qk_heads, rope_half, seq_len, raw_qk;
  float norm_eps;
  uint32_t* signs;            // EPI_ACT_SQ_SIGN, EPI_MUL_ACTROOT
  float* row_part;            // EPI_AXPBY_BF16: sums of squares out; EPI_ACT_SQ_SIGN: in (norm_parts per row)
  float* row_factor;          // EPI_ACT_SQ_SIGN: out; EPI_MUL_ACTROOT: in
  int norm_parts;
  float norm_scale;
};

constexpr int STG_PITCH = 64;
constexpr int STG_WARP_BYTES = 32 * STG_PITCH;      // one 32-row x 32-column bf16 chunk

// Epilogue staging: two chunk-sized slots per epilogue warp, first behind the operand stages so that they start on the 512 bytes their
// swizzle repeats after. Without a second operand they hold outputs on their way out, in turn. With one, a slot first receives a
// chunk of it (cp.async, two chunks ahead of its use), is read, then stages the output chunk in place.
constexpr int SGN_BYTES = 32 * 4;                   // the sign words of one chunk
template <int BN, int EPI>
struct GemmSmem {
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int CTAS = tile_ctas(BN, EPI);
  static constexpr int B_ROWS = BN / CTAS;
  static constexpr int B_BYTES = B_ROWS * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = BN == 64 ? 8 : BN == 128 || CTAS == 2 ? 6 : 4;     // pairs with five and four slots: 512 columns from 1536 118 us, not 111
  static constexpr int TILE_BYTES = STAGES * STAGE_BYTES;
  static constexpr int STG_BYTES = epi_warps(BN) * 2 * STG_WARP_BYTES;
  static constexpr int SGN_TOTAL = EPI == EPI_MUL_ACTROOT ? epi_warps(BN) * 2 * SGN_BYTES : 0;
  static constexpr int BAR_BYTES = 256;             // 2 per stage, 4 for the accumulators, two words
  // the declaration aligns the memory to 1024 bytes; slack for it stays where there is room
  static constexpr int TOTAL = TILE_BYTES + STG_BYTES + BAR_BYTES + SGN_TOTAL + (SGN_TOTAL ? 0 : 1024);
  static_assert(8 * (2 * STAGES + 4) + 8 <= BAR_BYTES, "barriers");
  static_assert(TOTAL <= 227 * 1024, "shared memory of one CTA");
};

__device__ __forceinline__ float act_fn(float x, float slope) { return x >= 0.f ? x : slope * x; }

// epilogues that read a second [M][N] bf16 operand
constexpr bool epi_has_aux(int epi) { return epi == EPI_AXPBY_BF16 || epi == EPI_RESID_BF16 || epi == EPI_MUL_ACTGRAD || epi == EPI_MUL_ACTROOT; }

// Relative error below 2^-22; its results are rounded to bf16. Without the handling of denormal arguments (roots below 1e-19), which
// costs the activation gradient of 98,304 x 1536 20 us.
__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int EPI>
__device__ __forceinline__ void epilogue_chunk(const GemmKernelParams& p, float alpha, float beta, int b, int m, int n0, const uint32_t (&r)[32]) {
  // One thread: row m, columns n0 .. n0+31 of batch b. Caller guarantees m < M.
  const bool full = (n0 + 32 <= p.N);
  const long long off = (long long)b * p.stride_d + (long long)m * p.ldd + n0;
  float v[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);

  if constexpr (EPI == EPI_F32 || EPI == EPI_F32_ATOMIC) {
    float* d = reinterpret_cast<float*>(p.D) + off;
    // one product, several output matrices (e.g. the packed QKV weight gradient lands in three gradient banks)
    if (p.seg_rows[1] > 0 && m >= p.seg_rows[1]) d = p.seg_D[1] + (long long)b * p.stride_d + (long long)(m - p.seg_rows[1]) * p.ldd + n0;
    else if (p.seg_rows[0] > 0 && m >= p.seg_rows[0]) d = p.seg_D[0] + (long long)b * p.stride_d + (long long)(m - p.seg_rows[0]) * p.ldd + n0;
    if (full && ((reinterpret_cast<uintptr_t>(d) & 15) == 0)) {
#pragma unroll
      for (int i = 0; i < 32; i += 4) {
        float4 q = make_float4(v[i] * alpha, v[i + 1] * alpha, v[i + 2] * alpha, v[i + 3] * alpha);
        if constexpr (EPI == EPI_F32) *reinterpret_cast<float4*>(d + i) = q;
        else atomicAdd(reinterpret_cast<float4*>(d + i), q);
      }
    } else {
      for (int i = 0; i < 32; ++i)
        if (n0 + i < p.N) {
          if constexpr (EPI == EPI_F32) d[i] = v[i] * alpha;
          else atomicAdd(d + i, v[i] * alpha);
        }
    }
    return;
  } else {
    __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(p.D) + off;
    const long long aoff = (long long)b * p.stride_aux + (long long)m * p.ld_aux + n0;
    const bool vec = full && ((reinterpret_cast<uintptr_t>(d) & 15) == 0);
    float a[32];
    if constexpr (EPI == EPI_AXPBY_BF16 || EPI == EPI_RESID_BF16 || EPI == EPI_MUL_ACTGRAD) {
      const __nv_bfloat16* ap = reinterpret_cast<const __nv_bfloat16*>(p.aux) + aoff;
      if (vec && ((reinterpret_cast<uintptr_t>(ap) & 15) == 0)) {
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
          const uint4 q = *reinterpret_cast<const uint4*>(ap + i);
          float2 f0 = unpack_bf16x2(q.x), f1 = unpack_bf16x2(q.y), f2 = unpack_bf16x2(q.z), f3 = unpack_bf16x2(q.w);
          a[i] = f0.x; a[i + 1] = f0.y; a[i + 2] = f1.x; a[i + 3] = f1.y;
          a[i + 4] = f2.x; a[i + 5] = f2.y; a[i + 6] = f3.x; a[i + 7] = f3.y;
        }
      } else {
        for (int i = 0; i < 32; ++i) a[i] = (n0 + i < p.N) ? __bfloat162float(ap[i]) : 0.f;
      }
    }
    float o[32];
    float o2[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      if constexpr (EPI == EPI_BF16) o[i] = v[i] * alpha;
      if constexpr (EPI == EPI_AXPBY_BF16) o[i] = alpha * v[i] + beta * a[i];
      if constexpr (EPI == EPI_RESID_BF16) o[i] = a[i] + ((n0 + i < p.N) ? p.colscale[n0 + i] : 0.f) * v[i];
      if constexpr (EPI == EPI_ACT_SQ) {
        // the pre-activation is stored in bf16 and the activation is computed from that stored value,
        // so the backward pass (which reads it back) sees exactly the same argument
        float h = __bfloat162float(__float2bfloat16(v[i]));
        float t = act_fn(h, p.slope);
        o[i] = h;
        o2[i] = t * t;
      }
      if constexpr (EPI == EPI_MUL_ACTGRAD) {
        float h = a[i];
        o[i] = v[i] * 2.f * act_fn(h, p.slope) * (h >= 0.f ? 1.f : p.slope);
      }
    }
    if (vec) {
#pragma unroll
      for (int i = 0; i < 32; i += 8)
        *reinterpret_cast<uint4*>(d + i) = make_uint4(pack_bf16x2(o[i], o[i + 1]), pack_bf16x2(o[i + 2], o[i + 3]),
                                                      pack_bf16x2(o[i + 4], o[i + 5]), pack_bf16x2(o[i + 6], o[i + 7]));
      if constexpr (EPI == EPI_ACT_SQ) {
        __nv_bfloat16* d2 = reinterpret_cast<__nv_bfloat16*>(p.D2) + off;
#pragma unroll
        for (int i = 0; i < 32; i += 8)
          *reinterpret_cast<uint4*>(d2 + i) = make_uint4(pack_bf16x2(o2[i], o2[i + 1]), pack_bf16x2(o2[i + 2], o2[i + 3]),
                                                         pack_bf16x2(o2[i + 4], o2[i + 5]), pack_bf16x2(o2[i + 6], o2[i + 7]));
      }
    } else {
      for (int i = 0; i < 32; ++i)
        if (n0 + i < p.N) {
          d[i] = __float2bfloat16(o[i]);
          if constexpr (EPI == EPI_ACT_SQ) (reinterpret_cast<__nv_bfloat16*>(p.D2) + off)[i] = __float2bfloat16(o2[i]);
        }
    }
  }
}

// Aligned bf16 epilogue. A thread owns one accumulator row, but 16-byte accesses of 32 different rows per instruction touch half a
// sector each, so chunks of 32 rows x 64 bytes go through shared memory. An output without a second operand leaves by a TMA store:
// one thread asks, and the warp neither computes addresses nor waits (98,304 rows: QKV 138 us with loads and stores of its own, 125 so;
// 1,024 columns 98 and 92). With a second operand the warp copies by itself, 8 rows x 64 contiguous bytes per instruction: the
// operand's, the output's and the prefetch's boxes of 64-byte rows are more than the TMA has time for beside the main loop's (the
// activation gradient took 211 us that way, 195 so).
// The chunk is XOR-swizzled: the 16-byte piece p of row r sits at piece p ^ ((r >> 1) & 3), the 64-byte swizzle of the tensor maps,
// under which all these access patterns (8 consecutive rows x one piece, 2 rows x 4 pieces, the TMA's) are free of bank conflicts.
__device__ __forceinline__ int stg_off(int row, int piece) { return row * STG_PITCH + ((piece ^ ((row >> 1) & 3)) << 4); }

// Outputs of one chunk: this thread's row of 32 values, packed. `ax` is the row of the second operand, `sg` its sign word.
template <int EPI>
__device__ __forceinline__ void epilogue_math(const GemmKernelParams& p, float alpha, float beta, int m_base, int lane, int n0, const uint32_t (&r)[32],
                                              const uint32_t (&ax)[16], uint32_t sg, float rf, uint32_t (&pk)[16], uint32_t (&pk2)[16]) {
  float a[32];
  if constexpr (epi_has_aux(EPI)) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float2 f = unpack_bf16x2(ax[i]);
      a[2 * i] = f.x; a[2 * i + 1] = f.y;
    }
  }
  float o[32], o2[32];
  float cs[32];
  if constexpr (EPI == EPI_RESID_BF16) {
    if ((reinterpret_cast<uintptr_t>(p.colscale + n0) & 15) == 0) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 t = __ldcg(reinterpret_cast<const float4*>(p.colscale + n0) + i);
        cs[4 * i] = t.x; cs[4 * i + 1] = t.y; cs[4 * i + 2] = t.z; cs[4 * i + 3] = t.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < 32; ++i) cs[i] = p.colscale[n0 + i];
    }
  }
  if constexpr (EPI == EPI_MUL_ACTROOT) {
    // aux = bf16(t^2) with t = leaky_relu(h): the root, rounded to bf16, is |t| itself (t has 8 significant bits, and its square was
    // off by at most half a unit of 8 bits, which moves the root by less than half a unit; `test_activation_root` goes through all t).
    const float pos = 2.f, neg = -2.f * p.slope;
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      const float2 t = unpack_bf16x2(pack_bf16x2(sqrt_approx(a[i]), sqrt_approx(a[i + 1])));
      o[i] = __uint_as_float(r[i]) * rf * (t.x * ((sg >> i) & 1u ? neg : pos));
      o[i + 1] = __uint_as_float(r[i + 1]) * rf * (t.y * ((sg >> (i + 1)) & 1u ? neg : pos));
    }
  }
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const float v = __uint_as_float(r[i]);
    if constexpr (EPI == EPI_BF16) o[i] = v * alpha;
    if constexpr (EPI == EPI_AXPBY_BF16) o[i] = alpha * v + beta * a[i];
    if constexpr (EPI == EPI_RESID_BF16) o[i] = a[i] + cs[i] * v;
    if constexpr (EPI == EPI_MUL_ACTGRAD) {
      const float h = a[i];
      o[i] = v * 2.f * act_fn(h, p.slope) * (h >= 0.f ? 1.f : p.slope);
    }
  }
  bool packed = false;
  if constexpr (EPI == EPI_ACT_SQ_SIGN) {
    packed = true;
    const __nv_bfloat162 sl = __float2bfloat162_rn(p.slope);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const __nv_bfloat162 hb = __floats2bfloat162_rn(__uint_as_float(r[2 * i]) * rf, __uint_as_float(r[2 * i + 1]) * rf);
      const __nv_bfloat162 t = __hmax2(hb, __hmul2(hb, sl));
      const __nv_bfloat162 sq = __hmul2(t, t);
      pk[i] = *reinterpret_cast<const uint32_t*>(&sq);
    }
    if (p.signs != nullptr) {
      uint32_t w = 0;
#pragma unroll
      for (int i = 31; i >= 0; --i) w = __funnelshift_l(r[i], w, 1);       // the factor and rounding to bf16 keep the sign
      if (m_base + lane < p.M) p.signs[(size_t)(n0 >> 5) * p.M + m_base + lane] = w;
    }
  }
  if constexpr (EPI == EPI_ACT_SQ) {
    // With a slope that is zero or a power of two, slope*h is exact in bf16 and the square of a bf16 value rounds
    // once either way, so the whole activation can run on packed bf16 pairs with bit-identical results.
    if ((__float_as_uint(p.slope) & 0x007fffffu) == 0u && p.slope >= 0.f && p.slope < 1.f) {
      packed = true;
      const __nv_bfloat162 sl = __float2bfloat162_rn(p.slope);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const __nv_bfloat162 hb = __floats2bfloat162_rn(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
        const __nv_bfloat162 t = __hmax2(hb, __hmul2(hb, sl));
        const __nv_bfloat162 sq = __hmul2(t, t);
        pk[i] = *reinterpret_cast<const uint32_t*>(&hb);
        pk2[i] = *reinterpret_cast<const uint32_t*>(&sq);
      }
    }
  }
  if (!packed) {
    if constexpr (EPI == EPI_ACT_SQ) {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float h = __bfloat162float(__float2bfloat16(__uint_as_float(r[i])));
        const float t = act_fn(h, p.slope);
        o[i] = h;
        o2[i] = t * t;
      }
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      pk[i] = pack_bf16x2(o[2 * i], o[2 * i + 1]);
      if constexpr (EPI == EPI_ACT_SQ) pk2[i] = pack_bf16x2(o2[2 * i], o2[2 * i + 1]);
    }
  }
}

// Half-split rotary on the first 2*HALF of a head's 64 values, tables [seq_len][HALF] (the layout of `qk_norm_rope_fwd`).
template <int HALF>
__device__ __forceinline__ void rope_head(float (&x)[64], const float* __restrict__ cosT, const float* __restrict__ sinT, int pos) {
  if constexpr (HALF > 0) {
    const float4* c4 = reinterpret_cast<const float4*>(cosT + (size_t)pos * HALF);
    const float4* s4 = reinterpret_cast<const float4*>(sinT + (size_t)pos * HALF);
#pragma unroll
    for (int i = 0; i < HALF; i += 4) {
      const float4 c = __ldg(c4 + i / 4), sn = __ldg(s4 + i / 4);
      const float cc[4] = {c.x, c.y, c.z, c.w}, ss[4] = {sn.x, sn.y, sn.z, sn.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float x1 = x[i + e], x2 = x[i + e + HALF];
        x[i + e] = x1 * cc[e] + x2 * ss[e];
        x[i + e + HALF] = x2 * cc[e] - x1 * ss[e];
      }
    }
  }
}

// EPI_QKV_NORM_ROPE on one head (two 32-column chunks) of 32 rows: the raw projection goes to D; for query and key heads the
// RMS-normalised, rotated and (queries) gain-scaled head goes to D2. The norm is taken of the bf16-rounded projection, the
// values the backward recomputes it from. Replaces a pass over the projection (`qk_norm_rope_fwd`, kept for the LoRA path);
// same math as the reference's fused QK kernels (parameter-golf-rs/crates/pg-kernels/src/gpu_kernels.rs:2640-2822).
template <typename Put>
__device__ __forceinline__ void epilogue_qkv_head(const GemmKernelParams& p, int m_base, int lane, int n0, const uint32_t (&ra)[32],
                                                  const uint32_t (&rb)[32], Put put) {
  uint32_t pk[32];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    pk[i] = pack_bf16x2(__uint_as_float(ra[2 * i]) * p.alpha, __uint_as_float(ra[2 * i + 1]) * p.alpha);
    pk[16 + i] = pack_bf16x2(__uint_as_float(rb[2 * i]) * p.alpha, __uint_as_float(rb[2 * i + 1]) * p.alpha);
  }
  const int head = n0 >> 6;
  if (p.raw_qk || head >= p.qk_heads) {
    put(pk, 0, n0);
    put(pk + 16, 0, n0 + 32);
  }
  if (head >= p.qk_heads) return;                  // value heads: the projection as it is (warp-uniform)
  float x[64];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const float2 f = unpack_bf16x2(pk[i]);
    x[2 * i] = f.x;
    x[2 * i + 1] = f.y;
    ss += f.x * f.x + f.y * f.y;
  }
  const float inv = rsqrtf(ss * (1.f / 64.f) + p.norm_eps);
#pragma unroll
  for (int i = 0; i < 64; ++i) x[i] *= inv;
  const int row = min(m_base + lane, p.M - 1);
  const int pos = row % p.seq_len;
  switch (p.rope_half) {
    case 8: rope_head<8>(x, p.rope_cos, p.rope_sin, pos); break;
    case 16: rope_head<16>(x, p.rope_cos, p.rope_sin, pos); break;
    case 32: rope_head<32>(x, p.rope_cos, p.rope_sin, pos); break;
    default: break;
  }
  const float g = (head < p.q_heads && p.head_gain != nullptr) ? p.head_gain[head] : 1.f;
#pragma unroll
  for (int i = 0; i < 32; ++i) pk[i] = pack_bf16x2(x[2 * i] * g, x[2 * i + 1] * g);     // one rounding, at the store
  put(pk, 1, n0);
  put(pk + 16, 1, n0 + 32);
}

template <int BN, bool A_KMAJOR, bool B_KMAJOR, int EPI>
__global__ void __launch_bounds__(gemm_threads(BN), 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_d, const __grid_constant__ CUtensorMap map_d2,
                    const GemmKernelParams p) {
  using S = GemmSmem<BN, EPI>;
  constexpr int STAGES = S::STAGES;
  constexpr uint32_t TMEM_COLS = 2 * BN;            // 128, 256 or 512: two accumulators
  constexpr bool PAIR = S::CTAS == 2;
  constexpr int TILE_M = BM * S::CTAS;
  const int rank = PAIR ? (int)(blockIdx.x & 1) : 0;          // which CTA of the pair; the first one issues the MMAs of both
  const int first_tile = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, tile_step = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + S::TILE_BYTES + S::STG_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], S::CTAS * epi_warps(BN));       // one arrival per epilogue warp, of both CTAs
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc<PAIR>(tmem_slot, TMEM_COLS);
    tmem_relinquish<PAIR>();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_b);
  }
  tc_fence_before();
  if constexpr (PAIR) cluster_sync();               // the other CTA's barriers are set up before anything arrives on them
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  chain_next();
  chain_wait();

  const int tiles_per_batch = p.tiles_m * p.tiles_n * p.splits;
  const int total_tiles = tiles_per_batch * p.batch;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      if (p.wait_flag != nullptr) {
        // The weight operand is written by peer GPUs (parameter all-gather fused here): poll the per-layer
        // ready counter, bounded, then order the peer's generic-proxy stores before this CTA's TMA reads.
        int seen;
        asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(seen) : "l"(p.wait_flag) : "memory");
        if (seen < p.wait_value) {
          const uint64_t t0 = globaltimer_ns();
          while (true) {
            asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(seen) : "l"(p.wait_flag) : "memory");
            if (seen >= p.wait_value) break;
            if (globaltimer_ns() - t0 > PGB_WAIT_LIMIT_NS) {
              *abort_flag = 1;
              report(p.status, ST_WAIT_FLAG, p.wait_value);
              ok = false;
              break;
            }
            __nanosleep(128);
          }
        }
        asm volatile("fence.proxy.async.global;" ::: "memory");
      }
      for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
        const int b = tile / tiles_per_batch;
        int r = tile - b * tiles_per_batch;
        const int split = r / (p.tiles_m * p.tiles_n);
        r -= split * p.tiles_m * p.tiles_n;
        const int tm = r / p.tiles_n, tn = r - tm * p.tiles_n;
        const int m0 = tm * TILE_M + rank * BM, n0 = tn * BN + rank * S::B_ROWS;
        const int kb0 = split * p.kb_per_split;
        const int kb1 = min(kb0 + p.kb_per_split, p.kb_total);
        if (p.aux_l2_prefetch && tile + tile_step < total_tiles) {
          // The epilogue warps read the second operand of this CTA's NEXT tile while they finish this one; ask for it now
          // so that those reads find it in L2.
          const int nt = tile + tile_step;
          const int pb = nt / tiles_per_batch;
          int pr = nt - pb * tiles_per_batch;
          pr -= (pr / (p.tiles_m * p.tiles_n)) * p.tiles_m * p.tiles_n;
          const int ptm = pr / p.tiles_n, ptn = pr - ptm * p.tiles_n;
#pragma unroll
          for (int j = 0; j < BN / 64; ++j)
            if (ptn * BN + 64 * j < p.N) tma_prefetch_l2_3d(&map_x, ptn * BN + 64 * j, ptm * TILE_M + rank * BM, pb);
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.status, ST_WAIT_EMPTY, kb)) { ok = false; break; }
          uint8_t* sa = smem + stage * S::STAGE_BYTES;
          uint8_t* sb = sa + S::A_BYTES;
          if (rank == 0) mbar_expect_tx(&full_bar[stage], S::CTAS * S::STAGE_BYTES);      // the bytes of both CTAs' loads
          if constexpr (A_KMAJOR) {
            tma_load_3d<PAIR>(sa, &map_a, &full_bar[stage], kb * BK, m0, b);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_3d<PAIR>(sa + j * 8192, &map_a, &full_bar[stage], m0 + 64 * j, kb * BK, b);
          }
          if constexpr (B_KMAJOR) {
            tma_load_3d<PAIR>(sb, &map_b, &full_bar[stage], kb * BK, n0, b);
          } else {
#pragma unroll
            for (int j = 0; j < S::B_ROWS / 64; ++j) tma_load_3d<PAIR>(sb + j * 8192, &map_b, &full_bar[stage], n0 + 64 * j, kb * BK, b);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      if (!ok) {
        // drain: every stage whose load may still be in flight (a pair's loads all report to the first CTA, which the other outlives)
        if (rank == 0)
          for (int s = 0; s < STAGES; ++s) mbar_drain(&full_bar[s], (s < stage) ? phase : (phase ^ 1));
      } else if constexpr (PAIR) {
        // the last arrivals of the other CTA's MMA thread on this CTA's barriers are in before it leaves
        for (int i = 0; i < STAGES; ++i) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag, p.status, ST_WAIT_EMPTY, -1)) break;
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (rank == 0 && elect_one()) {
      constexpr uint32_t IDESC = make_idesc_bf16(TILE_M, BN, A_KMAJOR ? 0 : 1, B_KMAJOR ? 0 : 1);
      // operand descriptors of stage 0; a stage or K step only adds to their address field
      const uint64_t da0 = A_KMAJOR ? make_smem_desc(smem_u32(smem), 16, 1024) : make_smem_desc(smem_u32(smem), 8192, 1024);
      const uint64_t db0 = B_KMAJOR ? make_smem_desc(smem_u32(smem) + S::A_BYTES, 16, 1024) : make_smem_desc(smem_u32(smem) + S::A_BYTES, 8192, 1024);
      constexpr uint32_t A_STEP = (A_KMAJOR ? 32 : 2048) >> 4, B_STEP = (B_KMAJOR ? 32 : 2048) >> 4;
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
        int r = tile % tiles_per_batch;
        const int split = r / (p.tiles_m * p.tiles_n);
        const int kb0 = split * p.kb_per_split;
        const int kb1 = min(kb0 + p.kb_per_split, p.kb_total);
        if (!mbar_wait(&tempty_bar[acc], acc_phase ^ 1, abort_flag, p.status, ST_WAIT_TMEM_EMPTY, tile)) { ok = false; break; }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + acc * BN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&full_bar[stage], phase, abort_flag, p.status, ST_WAIT_FULL, kb)) { ok = false; break; }
          tc_fence_after();
          const uint32_t at = (uint32_t)stage * (S::STAGE_BYTES >> 4);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) umma_ss<PAIR>(tmem_d, da0 + at + k * A_STEP, db0 + at + k * B_STEP, IDESC, (kb > kb0 || k > 0) ? 1u : 0u);
          umma_commit<PAIR>(&empty_bar[stage]);
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma_commit<PAIR>(&tfull_bar[acc]);
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..9; 2..5 for 64 columns)
    const int quarter = warp & 3;                 // TMEM lane quarter this warp may access
    const int half = (warp - 2) >> 2;             // which half of the tile's columns
    uint8_t* slots = smem + S::TILE_BYTES + (warp - 2) * 2 * STG_WARP_BYTES;
    uint8_t* sgn = smem + S::TILE_BYTES + S::STG_BYTES + S::BAR_BYTES + (warp - 2) * 2 * SGN_BYTES;      // sign words beside each slot
    const bool leader = elect_one();              // issues this warp's stores and waits for them
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    constexpr bool HAS_AUX = epi_has_aux(EPI);
    constexpr int CH = BN / 8 / epi_warps(BN);    // 32-column chunks per epilogue warp (the warps of a quarter split the columns)
    constexpr bool BF16_OUT = !(EPI == EPI_F32 || EPI == EPI_F32_ATOMIC);
    const int c_begin = half * CH;
    auto tile_coords = [&](int tile, int& b, int& tm, int& tn) {
      b = tile / tiles_per_batch;
      int r = tile - b * tiles_per_batch;
      const int split = r / (p.tiles_m * p.tiles_n);
      r -= split * p.tiles_m * p.tiles_n;
      tm = r / p.tiles_n;
      tn = r - tm * p.tiles_n;
    };
    auto fill = [&](uint8_t* slot, const uint32_t* x) {
#pragma unroll
      for (int i = 0; i < 4; ++i) *reinterpret_cast<uint4*>(slot + stg_off(lane, i)) = make_uint4(x[4 * i], x[4 * i + 1], x[4 * i + 2], x[4 * i + 3]);
    };
    // A chunk of output by TMA: into a slot once the store that last left it has read it, then out.
    int out = 1;
    auto put = [&](const uint32_t* x, int second, int b, int m_base, int col) {
      out ^= 1;
      uint8_t* slot = slots + out * STG_WARP_BYTES;
      if (leader) bulk_wait_read<1>();                     // the latest store is the other slot's
      __syncwarp();
      fill(slot, x);
      fence_proxy_async();
      __syncwarp();
      if (leader) {
        if (m_base < p.M) tma_store_3d(second ? &map_d2 : &map_d, slot, col, m_base, b);
        bulk_commit();                                     // also of nothing: the wait above counts groups
      }
    };
    // Second operand: a 32-row x 32-column chunk goes into one of this warp's two staging slots with 16-byte asynchronous
    // copies (8 rows x 64 contiguous bytes per instruction), one commit group per chunk, two chunks ahead of its use
    // (across the tile boundary too), so its DRAM latency hides behind the chunks processed meanwhile. cp.async is used
    // rather than loads into registers because pending register loads share the warp's few scoreboard counters with the
    // shared-memory and tensor-memory traffic of those chunks, which then wait for DRAM as well. The slot is read by the
    // thread that owns the row, reused in place to stage the output chunk, and refilled once the stores have read it.
    const bool aux_async = HAS_AUX && p.aligned;
    auto whole = [&](int tn, int cc) { return tn * BN + (c_begin + cc) * 32 + 32 <= p.N; };
    auto issue_aux = [&](int b, int tm, int tn, int cc) {
      if constexpr (HAS_AUX) {
        if (whole(tn, cc)) {
          const int n0 = tn * BN + (c_begin + cc) * 32, m_base = tm * TILE_M + rank * BM + quarter * 32;
          uint8_t* slot = slots + (cc & 1) * STG_WARP_BYTES;
          const __nv_bfloat16* ap = reinterpret_cast<const __nv_bfloat16*>(p.aux) + (long long)b * p.stride_aux + n0 + (lane & 3) * 8;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int row = m_base + i * 8 + (lane >> 2);
            if (row < p.M) cp_async16(slot + stg_off(i * 8 + (lane >> 2), lane & 3), ap + (long long)row * p.ld_aux);
          }
          if constexpr (EPI == EPI_MUL_ACTROOT) {
            if (p.signs != nullptr && m_base + lane < p.M)
              cp_async4(sgn + (cc & 1) * SGN_BYTES + lane * 4, p.signs + (size_t)(n0 >> 5) * p.M + m_base + lane);
          }
        }
        cp_async_commit();          // one group per chunk, also when nothing was copied: the wait below counts groups
      }
    };
    static_assert(CH % 2 == 0, "slot parity and the halves of a 64-column sum of squares follow the chunk index within the tile");
    // The factor of this thread's row. For the next tile it is asked for before the last chunk of this one and used after it.
    constexpr bool ROW_FACTOR = EPI == EPI_ACT_SQ_SIGN || EPI == EPI_MUL_ACTROOT;
    constexpr int PARTS = EPI == EPI_ACT_SQ_SIGN ? 8 : 1;       // read in one go; wider rows are summed in further rounds
    auto ask_factor = [&](int m, float (&q)[PARTS]) {
      if constexpr (ROW_FACTOR) {
        const int mm = min(m, p.M - 1);
        if constexpr (EPI == EPI_MUL_ACTROOT) q[0] = p.row_factor ? __ldcg(p.row_factor + mm) : 1.f;
        else if (p.row_part) {
#pragma unroll
          for (int k = 0; k < PARTS; ++k) q[k] = k < p.norm_parts ? __ldcg(p.row_part + (size_t)k * p.M + mm) : 0.f;
        }
      }
    };
    auto take_factor = [&](int m, const float (&q)[PARTS]) {
      if constexpr (EPI == EPI_MUL_ACTROOT) return q[0];
      if (!ROW_FACTOR || !p.row_part) return 1.f;
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < PARTS; ++k) s += q[k];
      for (int k = PARTS; k < p.norm_parts; ++k) s += __ldcg(p.row_part + (size_t)k * p.M + min(m, p.M - 1));
      return p.norm_scale * rsqrtf(s / p.K + p.norm_eps);
    };
    float asked[PARTS] = {};
    if constexpr (ROW_FACTOR) {
      if (first_tile < total_tiles) {
        int b0, tm0, tn0;
        tile_coords(first_tile, b0, tm0, tn0);
        ask_factor(tm0 * TILE_M + rank * BM + quarter * 32 + lane, asked);
      }
    }
    float sumsq = 0.f;                            // of this thread's row in the 64 columns under way (AXPBY with `row_part`)
    if (aux_async && first_tile < total_tiles) {
      int b0, tm0, tn0;
      tile_coords(first_tile, b0, tm0, tn0);
      issue_aux(b0, tm0, tn0, 0);
      issue_aux(b0, tm0, tn0, 1);
    }
    for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
      int b, tm, tn;
      tile_coords(tile, b, tm, tn);
      const int next = tile + tile_step;
      int nb = 0, ntm = 0, ntn = 0;
      if (next < total_tiles) tile_coords(next, nb, ntm, ntn);
      const int m_base = tm * TILE_M + rank * BM + quarter * 32, m = m_base + lane;
      const uint32_t taddr = tmem_base + acc * BN + ((uint32_t)(quarter * 32) << 16);
      float alpha = p.alpha, beta = p.beta;
      if (p.batch_sumsq != nullptr) {
        // Newton-Schulz on an un-normalised input: the matrix norm enters as a per-matrix factor of the whole output
        const float inv = 1.f / (sqrtf(p.batch_sumsq[b]) + 1e-7f);
        const float f = p.sumsq_pow == 2 ? inv * inv : inv;
        alpha *= f;
        beta *= f;
      }
      const float rf = take_factor(m, asked);
      if constexpr (EPI == EPI_ACT_SQ_SIGN) {
        if (p.row_factor && tn == 0 && half == 0 && m < p.M) p.row_factor[m] = rf;
      }
      if (!mbar_wait(&tfull_bar[acc], acc_phase, abort_flag, p.status, ST_WAIT_TMEM_FULL, tile)) { ok = false; break; }
      tc_fence_after();
      if constexpr (EPI == EPI_QKV_NORM_ROPE) {
        // one head (two chunks) at a time: the norm needs all 64 values of the row before either chunk can be written
#pragma unroll
        for (int cc = 0; cc < CH; cc += 2) {
          const int c = c_begin + cc;
          const int n0 = tn * BN + c * 32;
          if (n0 < p.N) {                         // warp-uniform; N is a multiple of 64 (checked on the host)
            uint32_t ra[32], rb[32];
            PGB_TMEM_LD32(taddr + c * 32, ra);
            PGB_TMEM_LD32(taddr + c * 32 + 32, rb);
            PGB_TMEM_WAIT_LD32(ra);
            PGB_TMEM_WAIT_LD32(rb);
            epilogue_qkv_head(p, m_base, lane, n0, ra, rb, [&](const uint32_t* x, int second, int col) { put(x, second, b, m_base, col); });
          }
        }
      } else {
#pragma unroll
      for (int cc = 0; cc < CH; ++cc) {
        const int c = c_begin + cc;
        const int n0 = tn * BN + c * 32;
        if constexpr (ROW_FACTOR) {
          if (cc == CH - 1 && next < total_tiles) ask_factor(ntm * TILE_M + rank * BM + quarter * 32 + lane, asked);
        }
        if (n0 < p.N) {                           // warp-uniform
          uint32_t rr[32];
          PGB_TMEM_LD32(taddr + c * 32, rr);
          if constexpr (HAS_AUX) {
            if (aux_async) {                      // two groups are pending; this chunk's is the older one
              cp_async_wait<1>();
              __syncwarp();
            }
          }
          PGB_TMEM_WAIT_LD32(rr);
          bool done = false;
          if constexpr (BF16_OUT) {
            if (p.aligned && whole(tn, cc)) {
              uint32_t ax[16], pk[16], pk2[16];
              uint32_t sg = 0;
              if constexpr (HAS_AUX) {
                uint8_t* slot = slots + (cc & 1) * STG_WARP_BYTES;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  const uint4 q = *reinterpret_cast<const uint4*>(slot + stg_off(lane, i));
                  ax[4 * i] = q.x; ax[4 * i + 1] = q.y; ax[4 * i + 2] = q.z; ax[4 * i + 3] = q.w;
                }
                if constexpr (EPI == EPI_MUL_ACTROOT) {
                  if (p.signs != nullptr) sg = *reinterpret_cast<const uint32_t*>(sgn + (cc & 1) * SGN_BYTES + lane * 4);
                }
                epilogue_math<EPI>(p, alpha, beta, m_base, lane, n0, rr, ax, sg, rf, pk, pk2);
                if constexpr (EPI == EPI_AXPBY_BF16) {
                  if (p.row_part) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                      const float2 f = unpack_bf16x2(pk[i]);
                      sumsq = fmaf(f.x, f.x, fmaf(f.y, f.y, sumsq));
                    }
                    if (cc & 1) {
                      if (m < p.M) p.row_part[(size_t)(n0 >> 6) * p.M + m] = sumsq;
                      sumsq = 0.f;
                    }
                  }
                }
                fill(slot, pk);
                __syncwarp();
                __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(p.D) + (long long)b * p.stride_d + n0 + (lane & 3) * 8;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  const int lr = i * 8 + (lane >> 2);
                  if (m_base + lr < p.M) *reinterpret_cast<uint4*>(d + (long long)(m_base + lr) * p.ldd) = *reinterpret_cast<const uint4*>(slot + stg_off(lr, lane & 3));
                }
              } else {
                epilogue_math<EPI>(p, alpha, beta, m_base, lane, n0, rr, ax, sg, rf, pk, pk2);
                put(pk, 0, b, m_base, n0);
                if constexpr (EPI == EPI_ACT_SQ) put(pk2, 1, b, m_base, n0);
              }
              done = true;
            }
          }
          if constexpr (EPI != EPI_ACT_SQ_SIGN && EPI != EPI_MUL_ACTROOT) {      // the host refuses what is not aligned
            if (!done && m < p.M) epilogue_chunk<EPI>(p, alpha, beta, b, m, n0, rr);
          }
        }
        if constexpr (HAS_AUX) {
          if (aux_async) {
            __syncwarp();                         // every lane is done with this slot
            if (cc + 2 < CH) issue_aux(b, tm, tn, cc + 2);
            else if (next < total_tiles) issue_aux(nb, ntm, ntn, cc + 2 - CH);
            else cp_async_commit();
          }
        }
      }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_first<PAIR>(&tempty_bar[acc]);
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
    if (leader) bulk_wait_all();                  // the stores have read their slots, and their writes are complete
  }

  tc_fence_before();
  if constexpr (PAIR) cluster_sync();               // neither CTA's shared or tensor memory is used by the other any more
  else __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc<PAIR>(tmem_base, TMEM_COLS);
  }
}

// ---- host side --------------------------------------------------------------------------------------------------
static int g_num_sms = 0;

static int num_sms() {
  if (!g_num_sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_num_sms <= 0) g_num_sms = 148;
  }
  return g_num_sms;
}

static CUtensorMap operand_map(const void* ptr, bool kmajor, int rows, int K, long long ld, long long batch_stride, int batch,
                               int tile_rows) {
  uint64_t dims[3];
  uint64_t strides[2];
  uint32_t box[3];
  if (kmajor) {         // memory [batch][rows][K]
    dims[0] = (uint64_t)K; dims[1] = (uint64_t)rows; dims[2] = (uint64_t)batch;
    box[0] = BK; box[1] = (uint32_t)tile_rows; box[2] = 1;
  } else {              // memory [batch][K][rows]
    dims[0] = (uint64_t)rows; dims[1] = (uint64_t)K; dims[2] = (uint64_t)batch;
    box[0] = 64; box[1] = BK; box[2] = 1;
  }
  strides[0] = (uint64_t)ld * 2;
  strides[1] = (uint64_t)(batch > 1 ? batch_stride : (long long)dims[1] * ld) * 2;
  return make_tmap_bf16(ptr, 3, dims, strides, box);
}

struct GemmMaps {
  CUtensorMap a, b, x, d, d2;      // operands, second operand of the epilogue (prefetch only), outputs
};

// [batch][M][N] bf16 in chunks of 32 x 32, the unit in which an epilogue warp writes
static CUtensorMap chunk_map(const void* ptr, const GemmArgs& a, long long ld, long long batch_stride) {
  const uint64_t dims[3] = {(uint64_t)a.N, (uint64_t)a.M, (uint64_t)a.batch};
  const uint64_t strides[2] = {(uint64_t)ld * 2, (uint64_t)(a.batch > 1 ? batch_stride : (long long)a.M * ld) * 2};
  const uint32_t box[3] = {32, 32, 1};
  return make_tmap_bf16(ptr, 3, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B);
}

template <int BN, bool AK, bool BKM, int EPI>
static void launch_variant(const GemmMaps& m, const GemmKernelParams& p, int grid, long long chain_rows, cudaStream_t stream) {
  auto kern = gemm_tcgen05_kernel<BN, AK, BKM, EPI>;
  static bool configured[64] = {};          // the attribute is a per-device property of the kernel
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || !configured[dev]) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmSmem<BN, EPI>::TOTAL);
    if (dev >= 0 && dev < 64) configured[dev] = true;
  }
  launch_chained_clusters(chain_rows, tile_ctas(BN, EPI), kern, grid, gemm_threads(BN), GemmSmem<BN, EPI>::TOTAL, stream, m.a, m.b, m.x, m.d, m.d2, p);
}

template <int BN, int EPI>
static void launch_major(const GemmArgs& a, const GemmMaps& m, const GemmKernelParams& p, int grid,
                         cudaStream_t stream) {
  if (a.a_kmajor && a.b_kmajor) launch_variant<BN, true, true, EPI>(m, p, grid, a.chain_rows, stream);
  else if (a.a_kmajor && !a.b_kmajor) launch_variant<BN, true, false, EPI>(m, p, grid, a.chain_rows, stream);
  else if constexpr (BN == 64) throw std::runtime_error("gemm: 64-column tiles take row-major activations");
  else if (!a.a_kmajor && a.b_kmajor) launch_variant<BN, false, true, EPI>(m, p, grid, a.chain_rows, stream);
  else launch_variant<BN, false, false, EPI>(m, p, grid, a.chain_rows, stream);
}

template <int BN>
static void launch_epi(const GemmArgs& a, const GemmMaps& m, const GemmKernelParams& p, int grid,
                       cudaStream_t stream) {
  if constexpr (BN != 64) {
    switch (a.epi) {
      case EPI_F32: launch_major<BN, EPI_F32>(a, m, p, grid, stream); return;
      case EPI_F32_ATOMIC: launch_major<BN, EPI_F32_ATOMIC>(a, m, p, grid, stream); return;
      case EPI_RESID_BF16: launch_major<BN, EPI_RESID_BF16>(a, m, p, grid, stream); return;
      default: break;
    }
  }
  switch (a.epi) {
    case EPI_BF16: launch_major<BN, EPI_BF16>(a, m, p, grid, stream); break;
    case EPI_AXPBY_BF16: launch_major<BN, EPI_AXPBY_BF16>(a, m, p, grid, stream); break;
    case EPI_ACT_SQ: launch_major<BN, EPI_ACT_SQ>(a, m, p, grid, stream); break;
    case EPI_MUL_ACTGRAD: launch_major<BN, EPI_MUL_ACTGRAD>(a, m, p, grid, stream); break;
    case EPI_QKV_NORM_ROPE:
      if (!(a.a_kmajor && a.b_kmajor)) throw std::runtime_error("gemm: the QKV epilogue takes row-major activations and [N][K] weights");
      launch_variant<BN, true, true, EPI_QKV_NORM_ROPE>(m, p, grid, a.chain_rows, stream);
      break;
    case EPI_ACT_SQ_SIGN:
      if (!(a.a_kmajor && a.b_kmajor)) throw std::runtime_error("gemm: the activation with signs takes row-major activations and [N][K] weights");
      launch_variant<BN, true, true, EPI_ACT_SQ_SIGN>(m, p, grid, a.chain_rows, stream);
      break;
    case EPI_MUL_ACTROOT:
      if (!(a.a_kmajor && !a.b_kmajor)) throw std::runtime_error("gemm: the activation gradient from the root takes row-major gradients and [K][N] weights");
      launch_variant<BN, true, false, EPI_MUL_ACTROOT>(m, p, grid, a.chain_rows, stream);
      break;
    default: throw std::runtime_error("gemm: unknown epilogue");
  }
}

struct TilePlan {
  int bn, splits;
};

// Tile width and number of K splits by estimated time, in SM clocks. An item (one tile, one K split) costs 540 / 285 / 245 clocks
// per 64-deep K step of a 256 / 128 / 64 column tile (a 64-column MMA is bound by its operand reads) plus an epilogue; a round of
// items beyond the first costs 0.8 of that, since a main loop overlaps the epilogue before it. A pair's items are twice as tall and
// there are half as many places for them. The constants were fitted to products of 1024 to 98,304 rows on the model's sites and order the
// widths as measured there (us with launch, cold caches, 256 / 128 / 64 columns):
//   M = 2048,  N = 1536, K = 512   14 / 12 / 14          M = 4096, N = 512, K = 1536   20 / 16 / 18
//   M = 16384, N = 512,  K = 1536  35 / 37 / 41          M = 98304, N = 512, K = 1024  80 / 100
// The output stages of the activation and the QKV product are longer than the plain one: with the same figure for all, 2,048 rows of the up
// projection and 4,480 of the QKV product took pairs (one scored window 799 us, now 773; logits of 5 x 896 1,007 and 955).
// With a second operand (AXPBY) a pair's output stage is the longer part unless the sum is long: M = 98304, N = 512: K = 512 84 / 72,
// K = 1536 123 / 145; M = 16384, K = 512 24 / 23.
// A narrower tile has to win by 8 %: it reads the activations from L2 more often than the model counts.
// Weight gradients (fp32 adds): every split adds a whole tile to the output in L2 (~52 clocks per column), so one round with as many
// splits as fill the SMs beats two rounds (512x1536 from 4096 rows: 3 splits of 128-column tiles 10.4 us, 6 splits 12.3), and narrow tiles win while the sum is short.
static int tile_count(const GemmArgs& a, int bn) {
  const int rows = BM * tile_ctas(bn, a.epi);
  return ((a.M + rows - 1) / rows) * ((a.N + bn - 1) / bn) * a.batch;
}

static TilePlan pick_tile(const GemmArgs& a, int kb_total, int sms) {
  TilePlan best{0, 1};
  double best_cost = 0.0;
  const bool atomic = a.epi == EPI_F32_ATOMIC;
  for (int bn : {256, 128, 64}) {
    if (a.tile_n > 0 && bn != a.tile_n) continue;
    if (a.tile_n <= 0 && bn == 256 && a.N <= 128) continue;
    if (bn == 64 && (!a.a_kmajor || a.epi == EPI_F32 || a.epi == EPI_RESID_BF16 || atomic)) continue;
    const int base = tile_count(a, bn), units = sms / tile_ctas(bn, a.epi);
    const double step = bn == 256 ? 540.0 : bn == 128 ? 285.0 : 245.0;
    const bool busy = a.epi == EPI_ACT_SQ_SIGN || a.epi == EPI_QKV_NORM_ROPE;
    const double wide = a.epi == EPI_AXPBY_BF16 ? 7500.0 : busy ? 6000.0 : 4900.0;
    const double epi = atomic ? 52.0 * bn : bn == 256 ? wide : bn == 128 ? 2900.0 : 2000.0;
    int last = 0;
    for (int waves : {1, 2, 3}) {
      int splits = std::max(1, a.splits);
      if (atomic && a.splits <= 0) splits = std::min(std::max(1, kb_total / 4), std::max(1, waves * units / base));
      if (splits == last) continue;
      last = splits;
      const int rounds = (base * splits + units - 1) / units;
      const double cost = (step * ((kb_total + splits - 1) / splits) + epi) * (1.0 + 0.8 * (rounds - 1));
      if (best.bn == 0 || cost < 0.92 * best_cost) {
        best = {bn, splits};
        best_cost = cost;
      }
    }
  }
  if (best.bn == 0) throw std::runtime_error("gemm: no tile of this width for this product");
  return best;
}

void gemm_bf16(const GemmArgs& a, cudaStream_t stream) {
  if (a.M <= 0 || a.N <= 0 || a.K <= 0 || a.batch <= 0) throw std::runtime_error("gemm: empty problem");
  if ((a.lda % 8) || (a.ldb % 8)) throw std::runtime_error("gemm: leading dimensions must be multiples of 8 elements");
  GemmKernelParams p;
  p.M = a.M; p.N = a.N; p.K = a.K; p.batch = a.batch;
  p.kb_total = (a.K + BK - 1) / BK;
  const TilePlan plan = pick_tile(a, p.kb_total, num_sms());
  const int bn = plan.bn, splits = plan.splits;
  p.tiles_m = (a.M + BM * tile_ctas(bn, a.epi) - 1) / (BM * tile_ctas(bn, a.epi));
  p.tiles_n = (a.N + bn - 1) / bn;
  if (splits > 1 && a.epi != EPI_F32_ATOMIC) throw std::runtime_error("gemm: split-K needs the atomic fp32 epilogue");
  p.kb_per_split = (p.kb_total + splits - 1) / splits;
  p.splits = (p.kb_total + p.kb_per_split - 1) / p.kb_per_split;
  p.ldd = a.ldd; p.stride_d = a.stride_d;
  p.ld_aux = a.ld_aux; p.stride_aux = a.stride_aux;
  p.D = a.D; p.D2 = a.D2; p.aux = a.aux; p.colscale = a.colscale;
  p.alpha = a.alpha; p.beta = a.beta; p.slope = a.slope;
  p.status = a.status;
  p.wait_flag = a.wait_flag;
  p.wait_value = a.wait_value;
  p.batch_sumsq = a.batch_sumsq;
  p.sumsq_pow = a.sumsq_pow;
  for (int k = 0; k < 2; ++k) {
    p.seg_rows[k] = a.seg_rows[k];
    p.seg_D[k] = a.seg_D[k];
  }
  if ((a.seg_rows[0] > 0 || a.seg_rows[1] > 0) && !(a.epi == EPI_F32 || a.epi == EPI_F32_ATOMIC))
    throw std::runtime_error("gemm: row segments need an fp32 epilogue");
  p.rope_cos = a.rope_cos;
  p.rope_sin = a.rope_sin;
  p.head_gain = a.head_gain;
  p.q_heads = a.q_heads;
  p.qk_heads = a.q_heads + a.kv_heads;
  p.rope_half = a.rope_dims / 2;
  p.seq_len = a.seq_len;
  p.raw_qk = a.raw_qk;
  p.norm_eps = a.norm_eps;
  p.signs = a.signs;
  p.row_part = a.epi == EPI_ACT_SQ_SIGN ? const_cast<float*>(a.norm_part) : a.row_part;
  p.row_factor = a.row_factor;
  p.norm_parts = a.K / 64;
  p.norm_scale = a.norm_scale;
  if ((a.row_part && (a.epi != EPI_AXPBY_BF16 || a.N % 64 || a.batch != 1)) || (a.norm_part && (a.epi != EPI_ACT_SQ_SIGN || a.K % 64)) ||
      (a.row_factor && !(a.epi == EPI_MUL_ACTROOT || (a.epi == EPI_ACT_SQ_SIGN && a.norm_part))))
    throw std::runtime_error("gemm: row sums and factors go with un-batched products of a multiple of 64 columns and their own epilogues");
  if (a.epi == EPI_ACT_SQ_SIGN || a.epi == EPI_MUL_ACTROOT) {
    int e = 0;
    const bool slope_ok = a.slope == 0.f || (a.slope > 0.f && a.slope < 1.f && std::frexp(a.slope, &e) == 0.5f);
    if (a.batch != 1 || a.N % 32 || (a.ldd % 8) || (reinterpret_cast<uintptr_t>(a.D) & 15) || !slope_ok ||
        (a.epi == EPI_MUL_ACTROOT && (a.aux == nullptr || (a.ld_aux % 8) || (reinterpret_cast<uintptr_t>(a.aux) & 15) || (a.slope > 0.f && !a.signs))))
      throw std::runtime_error("gemm: the activation with signs needs 16-byte aligned rows, N a multiple of 32 and a slope of 0 or a power of two below 1");
  }
  if (a.epi == EPI_QKV_NORM_ROPE) {
    const bool rope_ok = a.rope_dims == 0 || ((a.rope_dims == 16 || a.rope_dims == 32 || a.rope_dims == 64) && a.rope_cos && a.rope_sin &&
                                              (reinterpret_cast<uintptr_t>(a.rope_cos) & 15) == 0 && (reinterpret_cast<uintptr_t>(a.rope_sin) & 15) == 0);
    if (a.batch != 1 || a.D2 == nullptr || a.N != (a.q_heads + 2 * a.kv_heads) * 64 || a.seq_len <= 0 || !rope_ok || (a.ldd % 8) ||
        (reinterpret_cast<uintptr_t>(a.D) & 15) || (reinterpret_cast<uintptr_t>(a.D2) & 15))
      throw std::runtime_error("gemm: the QKV epilogue needs heads of 64, rope_dims in {0,16,32,64}, 16-byte aligned outputs of one row pitch and a sequence length");
  }
  GemmMaps m;
  m.a = operand_map(a.A, a.a_kmajor, a.M, a.K, a.lda, a.stride_a, a.batch, BM);
  m.b = operand_map(a.B, a.b_kmajor, a.N, a.K, a.ldb, a.stride_b, a.batch, bn / tile_ctas(bn, a.epi));
  const int total = p.tiles_m * p.tiles_n * p.splits * a.batch;
  const int grid = std::min(total, num_sms() / tile_ctas(bn, a.epi)) * tile_ctas(bn, a.epi);
  auto rows_ok = [&](const void* ptr, long long ld, long long stride) {
    return (reinterpret_cast<uintptr_t>(ptr) & 15) == 0 && ld % 8 == 0 && (a.batch == 1 || stride % 8 == 0);
  };
  const bool aux = a.aux != nullptr && epi_has_aux(a.epi), two = a.D2 != nullptr && (a.epi == EPI_ACT_SQ || a.epi == EPI_QKV_NORM_ROPE);
  p.aligned = rows_ok(a.D, a.ldd, a.stride_d) && (!two || rows_ok(a.D2, a.ldd, a.stride_d)) && (!aux || rows_ok(a.aux, a.ld_aux, a.stride_aux));
  if (a.row_part && !p.aligned) throw std::runtime_error("gemm: row sums need 16-byte aligned rows");
  const bool stores = p.aligned && !aux && a.epi != EPI_F32 && a.epi != EPI_F32_ATOMIC;
  m.d = stores ? chunk_map(a.D, a, a.ldd, a.stride_d) : m.a;
  m.d2 = stores && two ? chunk_map(a.D2, a, a.ldd, a.stride_d) : m.a;
  // L2 prefetch of the epilogue's second operand ([batch][M][N] bf16, row pitch ld_aux) one tile ahead of its readers
  p.aux_l2_prefetch = p.aligned && aux && total > grid / tile_ctas(bn, a.epi) ? 1 : 0;
  m.x = p.aux_l2_prefetch ? operand_map(a.aux, true, a.M, a.N, a.ld_aux, a.stride_aux, a.batch, BM) : m.a;
  if (bn == 256) launch_epi<256>(a, m, p, grid, stream);
  else if (bn == 128) launch_epi<128>(a, m, p, grid, stream);
  else launch_epi<64>(a, m, p, grid, stream);
}

}  // namespace pgb
