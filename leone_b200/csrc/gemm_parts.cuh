// Shared by the tcgen05 products: tile geometry, the parameters of one product, the work units
// of a launch and the epilogues that finish sums into outputs (all device code is inline).
#pragma once
#include "tc_common.cuh"

namespace leone {
namespace tc {

constexpr int kTileW = 128;     // weight rows per tile = MMA M
constexpr int kTileK = 64;      // one 128-byte swizzle row of bf16
constexpr int kGemmThreads = 192;

// Up to 64 tokens per tile a block keeps about 100 KB of stages, so two blocks (of this kernel
// or of this one and the next) share an SM: while one drains its epilogue the other already
// streams weights.  Larger token tiles take the whole SM.
constexpr int pow2_at_least(int v) {
  int p = 32;
  while (p < v) p *= 2;
  return p;
}
template <int BN> struct GemmCfg {
  static constexpr int kStageBytes = kTileW * kTileK * 2 + BN * kTileK * 2;
  static constexpr int kStages = BN <= 16 ? 5 : BN <= 32 ? 5 : BN <= 64 ? 4 : BN <= 128 ? 6 : 4;
  static constexpr int kBlocksPerSm = BN <= 64 ? 2 : 1;
  static constexpr int kTmemCols = pow2_at_least(2 * BN);      // two accumulators, BN columns apart
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*alignment*/ + 256 /*barriers*/;
};

// Decode-sized token tiles in cluster mode push their partial sums into the shared memory of the
// block that finishes the rows (see the kernel): that block needs an inbox beside its stages, one
// slot of [BN columns][32 rows] floats per (chunk it owns, rank): at most 8 slots.
template <int BN, bool kSwap, bool kCluster> constexpr bool gemm_pushes() { return kCluster && kSwap && BN <= 16; }
template <int BN, bool kSwap, bool kCluster> constexpr int gemm_smem_bytes() {
  return GemmCfg<BN>::kSmemBytes + (gemm_pushes<BN, kSwap, kCluster>() ? 8 * BN * 32 * 4 : 0);
}

struct GemmParams {
  void* out;
  const float* residual;
  int M, N, K, ldc;
  int epilogue;
  int splits;        // K is split this many ways ...
  int full_tiles;    // ... for tiles at or past this index; earlier tiles are not split
  float* workspace;
  int* counters;
  int* status;
  long long* trace;  // optional: 8 nanosecond time stamps per block (see leone_gemm_tc_set_trace)
  // RMSNorm around the product (swapped orientation), so that a norm between two products
  // needs no kernel of its own.  The product before the norm (fp32 output, epilogue 1 or 2)
  // also writes norm_out_x[m][n] = bf16(out[m][n] * norm_out_w[n]) and, per 32 weight rows, the
  // sum of out[m][n]^2 into norm_out_ss[(n / 32)][m]; the product after the norm reads
  // norm_out_x as its token operand and scales every output of token m by
  // rsqrt(sum_p norm_in_ss[p][m] / K + norm_eps), which is W . rmsnorm(out).
  __nv_bfloat16* norm_out_x;
  const float* norm_out_w;
  float* norm_out_ss;
  int ld_norm_out;
  const float* norm_in_ss;
  int norm_in_parts;
  float norm_eps;
  int l2_ahead;      // k-blocks of weights past the early stages that the producer asks the L2 for
  // The gate's shape of epilogue 3: g' sigmoid(slope g' (1 + cubic g'^2)) (u' + shift) with g' = min(g, limit)
  // and u' = clamp(u, -limit, limit).  gate_plain: slope 1, no limit, shift and cubic 0 (SwiGLU).
  int gate_plain;
  float gate_slope, gate_limit, gate_shift, gate_cubic;
  // One fp32 number per weight row added to its sums (before a gate, a residual or a norm after the product), or
  // null.
  const float* bias;
};

// Host side: the gate fields from an optional {slope, limit, shift, cubic} (null: SwiGLU).
inline void set_gate_shape(GemmParams& p, const float* shape) {
  p.gate_plain = shape == nullptr ? 1 : 0;
  p.gate_slope = shape == nullptr ? 1.f : shape[0];
  p.gate_limit = shape == nullptr ? INFINITY : shape[1];
  p.gate_shift = shape == nullptr ? 0.f : shape[2];
  p.gate_cubic = shape == nullptr ? 0.f : shape[3];
}

__device__ __forceinline__ long long global_ns() {
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t)::"memory");
  return t;
}
__device__ __forceinline__ void stamp(const GemmParams& p, int slot) {
  if (p.trace != nullptr) p.trace[(size_t)blockIdx.x * 8 + slot] = global_ns();
}

// Work units in launch order: the unsplit tiles first, then `splits` units per remaining tile.
// Splitting only the tiles of the last, partly filled round keeps every SM busy without
// paying the partial-sum round trip on the others.
struct Unit {
  int tile, split, nsplit;
};
__device__ __forceinline__ Unit unit_of(int u, const GemmParams& p) {
  if (u < p.full_tiles) return Unit{u, 0, 1};
  const int r = u - p.full_tiles;
  return Unit{p.full_tiles + r / p.splits, r % p.splits, p.splits};
}

// SwiGLU of a gate and an up value for a bf16 result: g / (1 + e^-g) * u with the fast exponential
// and division (a few units in the last place of fp32, far below the rounding to bf16; e^-g = inf
// gives g * 0).
__device__ __forceinline__ float silu_mul(float g, float u) { return __fdividef(g, 1.f + __expf(-g)) * u; }
// The same with the gate's shape from the parameters (a block-uniform branch).
__device__ __forceinline__ float gate_mul(const GemmParams& p, float g, float u) {
  if (p.gate_plain) return silu_mul(g, u);
  g = fminf(g, p.gate_limit);
  u = fminf(fmaxf(u, -p.gate_limit), p.gate_limit);
  const float z = p.gate_slope * g * fmaf(p.gate_cubic * g, g, 1.f);
  return __fdividef(g, 1.f + __expf(-z)) * (u + p.gate_shift);
}

// v[j] += bias[n + j] for 16 weight rows from n on, a multiple of 16 (every thread of a warp reads the same addresses).
__device__ __forceinline__ void add_bias16(const GemmParams& p, float* v, int n) {
  if (n + 16 <= p.N) {
    const float4* b = reinterpret_cast<const float4*>(p.bias + n);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 q = __ldg(b + j);
      v[4 * j] += q.x; v[4 * j + 1] += q.y; v[4 * j + 2] += q.z; v[4 * j + 3] += q.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (n + j < p.N) v[j] += p.bias[n + j];
  }
}

// Swapped orientation: the thread that owns weight row n finishes NC token columns
// m0 + c .. m0 + c + NC - 1 whose sums are in v (r: the residual values, fetched by the caller
// before anything is stored, because the residual may be the output itself).
// gw_known: the following norm's weight of row n if the caller fetched it already (else null).
template <int NC>
__device__ __forceinline__ void finish_swapped(const GemmParams& p, float (&v)[NC], const float (&r)[NC],
                                               int n, int m0, int c, int lane, const float* rs_s,
                                               const float* gw_known = nullptr) {
  if (p.norm_in_ss != nullptr) {
#pragma unroll
    for (int j = 0; j < NC; ++j) v[j] *= rs_s[c + j];
  }
  if (p.bias != nullptr) {
    const float b = n < p.N ? p.bias[n] : 0.f;
#pragma unroll
    for (int j = 0; j < NC; ++j) v[j] += b;
  }
  if (p.epilogue == 3) {
    // rows come in groups of 32: 16 gate rows (lanes 0-15) then their 16 up rows (lanes 16-31).
    // The halves of the warp swap one value per pair of token columns, so that the lower half
    // finishes the even column and the upper half the odd one (half the arithmetic of letting
    // the lower half finish both, and every store is 32 lanes wide).
    const int col = (n >> 5) * 16 + (lane & 15);
    const bool low = lane < 16;
    static_assert(NC % 2 == 0, "token columns are finished in pairs");
#pragma unroll
    for (int j = 0; j < NC; j += 2) {
      const float x = __shfl_xor_sync(0xffffffffu, low ? v[j + 1] : v[j], 16);
      const float g = low ? v[j] : x, u = low ? x : v[j + 1];
      const int m = m0 + c + j + (low ? 0 : 1);
      if (n < p.N && m < p.M) ((__nv_bfloat16*)p.out)[(size_t)m * p.ldc + col] = __float2bfloat16_rn(gate_mul(p, g, u));
    }
    return;
  }
  if (n < p.N) {
    if (p.epilogue == 2) {
#pragma unroll
      for (int j = 0; j < NC; ++j) v[j] += r[j];
    }
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      const int m = m0 + c + j;
      if (m < p.M) {
        const size_t o = (size_t)m * p.ldc + n;
        if (p.epilogue == 0) ((__nv_bfloat16*)p.out)[o] = __float2bfloat16_rn(v[j]);
        else ((float*)p.out)[o] = v[j];
      }
    }
  }
  if (p.norm_out_x != nullptr) {
    // the operand of the product after the following norm, and this warp's 32 rows' share of
    // the sums of squares (the lanes of a warp are 32 consecutive weight rows)
    const float gw = gw_known != nullptr ? *gw_known : n < p.N ? p.norm_out_w[n] : 0.f;
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      const int m = m0 + c + j;
      const float val = n < p.N ? v[j] : 0.f;
      if (n < p.N && m < p.M) p.norm_out_x[(size_t)m * p.ld_norm_out + n] = __float2bfloat16_rn(val * gw);
      float sq = val * val;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
      if (lane == 0 && m < p.M && n < p.N) p.norm_out_ss[(size_t)(n >> 5) * p.M + m] = sq;
    }
  }
}
template <int NC>
__device__ __forceinline__ void fetch_residual(const GemmParams& p, float (&r)[NC], int n, int m0, int c) {
  if (p.epilogue == 2 && n < p.N) {
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      const int m = m0 + c + j;
      r[j] = m < p.M ? p.residual[(size_t)m * p.ldc + n] : 0.f;
    }
  }
}

// The residual values that finish_token_major32 would add to token row m, weight rows n .. n+31
// (zeros where there are none), so that the caller can have them in flight early.
__device__ __forceinline__ void fetch_residual32(const GemmParams& p, float (&r)[32], int m, int n) {
#pragma unroll
  for (int j = 0; j < 32; ++j) r[j] = 0.f;
  if (p.epilogue != 2 || m >= p.M || n >= p.N) return;
  const size_t o = (size_t)m * p.ldc + n;
  if (n + 32 <= p.N && (p.ldc & 3) == 0) {
    const float4* res = reinterpret_cast<const float4*>(p.residual + o);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float4 q = res[j];
      r[4 * j] = q.x; r[4 * j + 1] = q.y; r[4 * j + 2] = q.z; r[4 * j + 3] = q.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (n + j < p.N) r[j] = p.residual[o + j];
  }
}

// Token-major form, splits summed inside a cluster: 32 finished sums of token row m for the weight
// rows n .. n+31 (n a multiple of 32) go out through the product's epilogue.  No folded norm.
// residual_added: the caller has added the residual already (fetch_residual32).
__device__ __forceinline__ void finish_token_major32(const GemmParams& p, float (&v)[32], int m, int n,
                                                     bool residual_added = false) {
  if (m >= p.M || n >= p.N) return;
  const bool vec_ok = (p.ldc & 7) == 0;
  if (p.bias != nullptr) {
    add_bias16(p, v, n);
    add_bias16(p, v + 16, n + 16);
  }
  if (p.epilogue == 3) {                                 // 16 gate columns, then their 16 up columns
    __nv_bfloat16* orow = (__nv_bfloat16*)p.out + (size_t)m * p.ldc;
    const int col = n >> 1;
    uint32_t packed[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float a = gate_mul(p, v[2 * j], v[16 + 2 * j]);
      const float b = gate_mul(p, v[2 * j + 1], v[16 + 2 * j + 1]);
      __nv_bfloat162 v2 = __floats2bfloat162_rn(a, b);
      packed[j] = *reinterpret_cast<uint32_t*>(&v2);
    }
    if (vec_ok) {
      uint4* dst = reinterpret_cast<uint4*>(orow + col);
      dst[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
      dst[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) *reinterpret_cast<uint32_t*>(orow + col + 2 * j) = packed[j];
    }
    return;
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int nn = n + 16 * h;
    if (nn >= p.N) break;
    float* vv = v + 16 * h;
    const size_t o = (size_t)m * p.ldc + nn;
    const bool full = nn + 16 <= p.N && vec_ok;
    if (p.epilogue == 0) {
      __nv_bfloat16* dst = (__nv_bfloat16*)p.out + o;
      if (full) {
        uint32_t packed[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          __nv_bfloat162 v2 = __floats2bfloat162_rn(vv[2 * j], vv[2 * j + 1]);
          packed[j] = *reinterpret_cast<uint32_t*>(&v2);
        }
        reinterpret_cast<uint4*>(dst)[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        reinterpret_cast<uint4*>(dst)[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
      } else {
        for (int j = 0; j < 16 && nn + j < p.N; ++j) dst[j] = __float2bfloat16_rn(vv[j]);
      }
    } else {
      float* dst = (float*)p.out + o;
      if (full) {
        if (p.epilogue == 2 && !residual_added) {
          const float4* res = reinterpret_cast<const float4*>(p.residual + o);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float4 r = res[j];
            vv[4 * j] += r.x; vv[4 * j + 1] += r.y; vv[4 * j + 2] += r.z; vv[4 * j + 3] += r.w;
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
          reinterpret_cast<float4*>(dst)[j] = make_float4(vv[4 * j], vv[4 * j + 1], vv[4 * j + 2], vv[4 * j + 3]);
      } else {
        for (int j = 0; j < 16 && nn + j < p.N; ++j) {
          if (p.epilogue == 2 && !residual_added) vv[j] += p.residual[o + j];
          dst[j] = vv[j];
        }
      }
    }
  }
}


// Token-major form: the thread that owns token row m finishes the tile's bn weight rows from n0
// on (tile n_tile; bn a multiple of 16, of 32 with the SwiGLU epilogue), 16 at a time, from tensor
// memory at taddr: the norm's factor before, the product's epilogue, and the operand and sum of
// squares of a norm after it.  Warp-wide (the loads from tensor memory are), so every thread of
// the warp calls it, rows past M too.
__device__ __forceinline__ void finish_token_major_row(const GemmParams& p, uint32_t taddr, int m, int n0,
                                                       int n_tile, const int bn) {
  const bool vec_ok = (p.ldc & 7) == 0;
  // the norm before this product: this row's factor from the parts the product before left
  float rs = 1.f;
  if (p.norm_in_ss != nullptr) {
    float ss = 0.f;
    if (m < p.M)
      for (int q = 0; q < p.norm_in_parts; ++q) ss += p.norm_in_ss[(size_t)q * p.M + m];
    rs = rsqrtf(ss / (float)p.K + p.norm_eps);
  }
  // the norm after this product: this row's sum of squares over the tile's columns, and
  // bf16(out * weight) beside the output (token-major: one part per tile of BN columns)
  float ssq = 0.f;
  auto norm_out16 = [&](const float (&val)[16], int n) {      // 16 finished outputs from column n
    if (p.norm_out_x != nullptr && m < p.M && n < p.N) {
      uint32_t packed[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float a = n + 2 * j < p.N ? val[2 * j] : 0.f, b = n + 2 * j + 1 < p.N ? val[2 * j + 1] : 0.f;
        ssq = fmaf(a, a, fmaf(b, b, ssq));
        __nv_bfloat162 v2 = __floats2bfloat162_rn(a * (n + 2 * j < p.N ? p.norm_out_w[n + 2 * j] : 0.f),
                                                  b * (n + 2 * j + 1 < p.N ? p.norm_out_w[n + 2 * j + 1] : 0.f));
        packed[j] = *reinterpret_cast<uint32_t*>(&v2);
      }
      __nv_bfloat16* xrow = p.norm_out_x + (size_t)m * p.ld_norm_out + n;
      if (n + 16 <= p.N && (p.ld_norm_out & 7) == 0) {
        reinterpret_cast<uint4*>(xrow)[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        reinterpret_cast<uint4*>(xrow)[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
      } else {
        for (int j = 0; j < 16 && n + j < p.N; ++j)
          xrow[j] = __float2bfloat16_rn(val[j] * p.norm_out_w[n + j]);
      }
    }
  };
  if (p.epilogue == 3) {
    __nv_bfloat16* orow = (__nv_bfloat16*)p.out + (size_t)m * p.ldc;
    for (int c = 0; c < bn; c += 32) {             // 16 gate columns, then their 16 up columns
      float g[16], u[16];
      tmem_ld16(taddr + c, g);
      tmem_ld16(taddr + c + 16, u);
      if (p.norm_in_ss != nullptr) {
#pragma unroll
        for (int j = 0; j < 16; ++j) { g[j] *= rs; u[j] *= rs; }
      }
      if (p.bias != nullptr && n0 + c < p.N) {     // (rows come in whole groups of 32)
        add_bias16(p, g, n0 + c);
        add_bias16(p, u, n0 + c + 16);
      }
      const int col = (n0 + c) >> 1;
      if (m < p.M && n0 + c < p.N) {
        uint32_t packed[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float a = gate_mul(p, g[2 * j], u[2 * j]);
          const float b = gate_mul(p, g[2 * j + 1], u[2 * j + 1]);
          __nv_bfloat162 v2 = __floats2bfloat162_rn(a, b);
          packed[j] = *reinterpret_cast<uint32_t*>(&v2);
        }
        if (vec_ok) {
          uint4* dst = reinterpret_cast<uint4*>(orow + col);
          dst[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
          dst[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) *reinterpret_cast<uint32_t*>(orow + col + 2 * j) = packed[j];
        }
      }
    }
  } else if (p.epilogue == 2 && vec_ok && n0 + bn <= p.N) {
    // fp32 out = acc + residual for a whole row of the tile: the residual is fetched three
    // chunks ahead of its use, so its latency is paid once per row, not once per chunk
    // (the residual may be the output itself: a chunk is read before it is written, and
    // chunks do not overlap).  The branch is the same for every thread of the block, as
    // the warp-wide tensor-memory loads need; rows past M read row 0 and store nothing.
    constexpr int kAhead = 3;
    const bool row_ok = m < p.M;
    const size_t row_at = (size_t)(row_ok ? m : 0) * p.ldc + n0;
    const float4* res = reinterpret_cast<const float4*>(p.residual + row_at);
    float4* dst = reinterpret_cast<float4*>((float*)p.out + row_at);
    const int chunks = bn / 16;
    float4 rb[kAhead][4];
#pragma unroll
    for (int a = 0; a < kAhead; ++a) {
      if (a < chunks) {
#pragma unroll
        for (int j = 0; j < 4; ++j) rb[a][j] = res[a * 4 + j];
      }
    }
    for (int i0 = 0; i0 < chunks; i0 += kAhead) {
#pragma unroll
      for (int a = 0; a < kAhead; ++a) {        // chunk i0 + a uses and refills slot a
        const int i = i0 + a;
        if (i >= chunks) break;
        float v[16];
        tmem_ld16(taddr + i * 16, v);
        float4 r[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) r[j] = rb[a][j];
        if (i + kAhead < chunks) {
#pragma unroll
          for (int j = 0; j < 4; ++j) rb[a][j] = res[(i + kAhead) * 4 + j];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          v[4 * j] += r[j].x; v[4 * j + 1] += r[j].y; v[4 * j + 2] += r[j].z; v[4 * j + 3] += r[j].w;
        }
        if (p.bias != nullptr) add_bias16(p, v, n0 + i * 16);
        if (row_ok) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            dst[i * 4 + j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
        norm_out16(v, n0 + i * 16);
      }
    }
  } else {
    for (int c = 0; c < bn; c += 16) {
      float v[16];
      tmem_ld16(taddr + c, v);
      const int n = n0 + c;
      if (m >= p.M || n >= p.N) continue;
      if (p.norm_in_ss != nullptr) {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] *= rs;
      }
      if (p.bias != nullptr) add_bias16(p, v, n);
      const size_t o = (size_t)m * p.ldc + n;
      const bool full = n + 16 <= p.N && vec_ok;
      if (p.epilogue == 0) {
        __nv_bfloat16* dst = (__nv_bfloat16*)p.out + o;
        if (full) {
          uint32_t packed[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            __nv_bfloat162 v2 = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
            packed[j] = *reinterpret_cast<uint32_t*>(&v2);
          }
          reinterpret_cast<uint4*>(dst)[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
          reinterpret_cast<uint4*>(dst)[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
        } else {
          for (int j = 0; j < 16 && n + j < p.N; ++j) dst[j] = __float2bfloat16_rn(v[j]);
        }
      } else {
        float* dst = (float*)p.out + o;
        if (full) {
          if (p.epilogue == 2) {
            const float4* res = reinterpret_cast<const float4*>(p.residual + o);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float4 r = res[j];
              v[4 * j] += r.x; v[4 * j + 1] += r.y; v[4 * j + 2] += r.z; v[4 * j + 3] += r.w;
            }
          }
#pragma unroll
          for (int j = 0; j < 4; ++j)
            reinterpret_cast<float4*>(dst)[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        } else {
          for (int j = 0; j < 16 && n + j < p.N; ++j) {
            if (p.epilogue == 2) v[j] += p.residual[o + j];
            dst[j] = v[j];
          }
        }
        norm_out16(v, n);
      }
    }
  }
  if (p.norm_out_x != nullptr && m < p.M) p.norm_out_ss[(size_t)n_tile * p.M + m] = ssq;
}
template <int BN>
__device__ __forceinline__ void finish_token_major_row(const GemmParams& p, uint32_t taddr, int m, int n0,
                                                       int n_tile) {
  finish_token_major_row(p, taddr, m, n0, n_tile, BN);
}

// The row's factor of a norm before the product (1 without one).
__device__ __forceinline__ float norm_in_factor(const GemmParams& p, int m) {
  if (p.norm_in_ss == nullptr) return 1.f;
  float ss = 0.f;
  if (m < p.M) {
#pragma unroll 8
    for (int q = 0; q < p.norm_in_parts; ++q) ss += p.norm_in_ss[(size_t)q * p.M + m];
  }
  return rsqrtf(ss / (float)p.K + p.norm_eps);
}

constexpr int kBoxBytes = 32 * 128;                // a warp's shared memory for finish_rows
constexpr int kResidualAhead = 2;                  // chunks of residual values in flight ahead of their use

// The residual values of one chunk of 32 columns, as finish_rows' lanes own them: rows 4 i + lane / 8, columns 4 (lane % 8) ..
__device__ __forceinline__ void fetch_residual_chunk(const GemmParams& p, float4 (&r)[8], int m0, int n, int c, int c_hi, bool vec) {
  const int lane = threadIdx.x & 31, col = n + c + 4 * (lane & 7);
  const bool here = c + 4 * (lane & 7) < c_hi;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int m = m0 + 4 * i + (lane >> 3);
    r[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!here || m >= p.M) continue;
    const float* src = p.residual + (size_t)m * p.ldc + col;
    if (vec && col + 4 <= p.N) {
      r[i] = *reinterpret_cast<const float4*>(src);
    } else {
      if (col < p.N) r[i].x = src[0];
      if (col + 1 < p.N) r[i].y = src[1];
      if (col + 2 < p.N) r[i].z = src[2];
      if (col + 3 < p.N) r[i].w = src[3];
    }
  }
}

// Token-major form, the epilogue of pairs and of narrow tiles: a warp finishes its 32 token rows (m0 ..; tensor memory at `taddr`, lane = row) for
// the accumulator columns [c_lo, c_hi) of the tile whose first weight row is n0 (multiples of 16, of 32 with the gate).
// Sums go through 4 KB of the warp's own shared memory, 32 rows of 128 bytes with their 16-byte pieces swizzled by the row, so
// that every access to global memory is four rows of 128 bytes side by side.  (A thread per row, as above, touches 32 rows with
// 16 bytes each: half sectors, and 32 cache lines an instruction.)
//
// A product's kernel runs once in a layer, with the step's other kernels in between, so the code of its epilogue comes from memory
// again: what every tile of the gate executes is kept short (a loop over 16 outputs at a time, the edges of tiles and unaligned rows
// in paths of their own).  12288 x 2048 with the gate in a step of 1,027 tokens 54.7 us with the loop unrolled, 42.8 as it is (48.8
// with a thread a row); at 64 tokens 22.9 and 10.3.  (The unrolled one over and over, its code at hand: 44.9.)
//
// `ready`: waits until the accumulator is complete (false: gave up); the first residual values are requested before it.
// Called by whole warps.  `squares(s)`: s[i] is the sum of squares of output row m0 + 4 i + lane / 8 over these
// columns, for the norm after the product (the row's eight lanes have it).
template <class Ready, class Squares>
__device__ __forceinline__ bool finish_rows(const GemmParams& p, uint32_t taddr, int m0, int n0, int c_lo, int c_hi,
                                            uint32_t box, Ready ready, Squares squares) {
  const int lane = threadIdx.x & 31;
  const uint32_t mine = box + lane * 128;                             // this thread's row of the box
  const int sw = lane & 7;
  const int row_out = lane >> 3, unit = lane & 7;                     // on the way out: rows 4 i + row_out, 16-byte piece `unit`
  if (m0 >= p.M) return ready();                                      // no such tokens: nothing to store
  const float rs = norm_in_factor(p, m0 + lane);
  auto put = [&](int u, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(mine + ((u ^ sw) << 4)), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
  };
  auto get = [&](int i) {
    const int r = 4 * i + row_out;
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(box + r * 128 + ((unit ^ (r & 7)) << 4)) : "memory");
    return v;
  };
  auto pack = [](float a, float b) {
    __nv_bfloat162 v2 = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v2);
  };
  if (p.epilogue == 1 || p.epilogue == 2) {
    const bool vec = ((p.ldc & 3) | ((uintptr_t)p.out & 15) | ((uintptr_t)p.residual & 15)) == 0;
    const bool vec_x = ((p.ld_norm_out & 3) | ((uintptr_t)p.norm_out_x & 7)) == 0;
    float4 ahead[kResidualAhead][8];
    float ssq[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) ssq[i] = 0.f;
    if (p.epilogue == 2) {
#pragma unroll
      for (int a = 0; a < kResidualAhead; ++a)
        if (c_lo + 32 * a < c_hi) fetch_residual_chunk(p, ahead[a], m0, n0, c_lo + 32 * a, c_hi, vec);
    }
    if (!ready()) return false;
    for (int c0 = c_lo; c0 < c_hi; c0 += 32 * kResidualAhead) {
#pragma unroll
      for (int a = 0; a < kResidualAhead; ++a) {                      // chunk c uses and refills slot a
        const int c = c0 + 32 * a;
        if (c >= c_hi) break;
        uint32_t r[32];
        const bool whole = c + 32 <= c_hi;
        if (whole) tmem_ld32_issue(taddr + c, r);
        else tmem_ld16_issue(taddr + c, r);
        tmem_ld_wait();
        __syncwarp();                                                 // the chunk before has left the box
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          if (q == 1 && !whole) break;
          float v[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[16 * q + j]) * rs;
          if (p.bias != nullptr) add_bias16(p, v, n0 + c + 16 * q);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            put(4 * q + j, __float_as_uint(v[4 * j]), __float_as_uint(v[4 * j + 1]), __float_as_uint(v[4 * j + 2]),
                __float_as_uint(v[4 * j + 3]));
        }
        __syncwarp();
        const int n = n0 + c + 4 * unit;
        const bool here = c + 4 * unit < c_hi && n < p.N, full = vec && n + 4 <= p.N;
        float w[4] = {0.f, 0.f, 0.f, 0.f};
        if (p.norm_out_x != nullptr && here) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (n + j < p.N) w[j] = __ldg(p.norm_out_w + n + j);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int m = m0 + 4 * i + row_out;
          const uint4 raw = get(i);
          float4 v = make_float4(__uint_as_float(raw.x), __uint_as_float(raw.y), __uint_as_float(raw.z), __uint_as_float(raw.w));
          if (p.epilogue == 2) {
            v.x += ahead[a][i].x;
            v.y += ahead[a][i].y;
            v.z += ahead[a][i].z;
            v.w += ahead[a][i].w;
          }
          if (!here || m >= p.M) continue;
          float* dst = (float*)p.out + (size_t)m * p.ldc + n;
          if (full) {
            *reinterpret_cast<float4*>(dst) = v;
          } else {
            dst[0] = v.x;
            if (n + 1 < p.N) dst[1] = v.y; else v.y = 0.f;
            if (n + 2 < p.N) dst[2] = v.z; else v.z = 0.f;
            if (n + 3 < p.N) dst[3] = v.w; else v.w = 0.f;
          }
          if (p.norm_out_x != nullptr) {
            ssq[i] = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, ssq[i]))));
            __nv_bfloat16* x = p.norm_out_x + (size_t)m * p.ld_norm_out + n;
            if (full && vec_x) {
              *reinterpret_cast<uint2*>(x) = make_uint2(pack(v.x * w[0], v.y * w[1]), pack(v.z * w[2], v.w * w[3]));
            } else {
              x[0] = __float2bfloat16_rn(v.x * w[0]);
              if (n + 1 < p.N) x[1] = __float2bfloat16_rn(v.y * w[1]);
              if (n + 2 < p.N) x[2] = __float2bfloat16_rn(v.z * w[2]);
              if (n + 3 < p.N) x[3] = __float2bfloat16_rn(v.w * w[3]);
            }
          }
        }
        if (p.epilogue == 2 && c + 32 * kResidualAhead < c_hi)
          fetch_residual_chunk(p, ahead[a], m0, n0, c + 32 * kResidualAhead, c_hi, vec);
      }
    }
    if (p.norm_out_x != nullptr) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        float s = ssq[i];
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        ssq[i] = s;
      }
      squares(ssq);
    }
    return true;
  }
  // bfloat16 outputs: 64 of them a chunk, from 64 accumulator columns or, with the gate, from 128
  if (!ready()) return false;
  const bool gated = p.epilogue == 3;
  const bool vec = ((p.ldc & 7) | ((uintptr_t)p.out & 15)) == 0;
  const int step = gated ? 128 : 64;
  const int n_out = gated ? p.N >> 1 : p.N;
#pragma unroll 1
  for (int c = c_lo; c < c_hi; c += step) {
    __syncwarp();                                                     // the chunk before has left the box
    const int parts = min(step, c_hi - c) / (gated ? 32 : 16);        // 16 outputs each
#pragma unroll 1
    for (int h = 0; h < parts; ++h) {
      uint32_t r[32];
      float v[16];
      if (gated) {
        const int at = c + 32 * h;
        tmem_ld32_issue(taddr + at, r);
        tmem_ld_wait();
        float u[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          v[j] = __uint_as_float(r[j]) * rs;
          u[j] = __uint_as_float(r[16 + j]) * rs;
        }
        if (__builtin_expect(p.bias != nullptr, 0) && n0 + at < p.N) {
          add_bias16(p, v, n0 + at);
          add_bias16(p, u, n0 + at + 16);
        }
        if (__builtin_expect(p.gate_plain, 1)) {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = silu_mul(v[j], u[j]);
        } else {
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = gate_mul(p, v[j], u[j]);
        }
      } else {
        const int at = c + 16 * h;
        tmem_ld16_issue(taddr + at, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]) * rs;
        if (__builtin_expect(p.bias != nullptr, 0)) add_bias16(p, v, n0 + at);
      }
      put(2 * h, pack(v[0], v[1]), pack(v[2], v[3]), pack(v[4], v[5]), pack(v[6], v[7]));
      put(2 * h + 1, pack(v[8], v[9]), pack(v[10], v[11]), pack(v[12], v[13]), pack(v[14], v[15]));
    }
    __syncwarp();
    const int first = gated ? (n0 + c) >> 1 : n0 + c, n = first + 8 * unit, m1 = m0 + row_out;
    const bool here = n < n_out && unit < 2 * parts;
    __nv_bfloat16* dst = (__nv_bfloat16*)p.out + (size_t)m1 * p.ldc + n;
    if (__all_sync(0xffffffffu, !here || (vec && n + 8 <= n_out))) {
#pragma unroll
      for (int i = 0; i < 8; ++i, dst += 4 * (size_t)p.ldc) {
        const uint4 v = get(i);
        if (here && m1 + 4 * i < p.M) *reinterpret_cast<uint4*>(dst) = v;
      }
    } else {
#pragma unroll 1
      for (int i = 0; i < 8; ++i, dst += 4 * (size_t)p.ldc) {
        const uint4 v = get(i);
        if (!here || m1 + 4 * i >= p.M) continue;
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (n + j < n_out) dst[j] = __ushort_as_bfloat16((unsigned short)(w[j >> 1] >> (16 * (j & 1))));
      }
    }
  }
  return true;
}

}  // namespace tc
}  // namespace leone
