// C[M,N] = A[M,K] * W[N,K]^T in 32 bits on tensor cores: the 32-bit product of prompt steps (gemm_simt.cu has the others).
//
// Every operand is the sum of two numbers of 11 significant bits, x = hi + lo + r with |lo| <= 2^-11 |x| and |r| <= 2^-23 |x| (both
// rounded to nearest), and a product of two is hi hi + hi lo + lo hi; the dropped lo lo is at most 2^-22 of it, of either
// sign, so that a product is within about 2^-21 (of sums of normal inputs the drops are 8e-8 in the 2-norm).  The three run as
// tcgen05.mma kind::tf32, whose operands these numbers are exactly.  What tensor cores lose is in their sums, not in
// the products, so sums stay short there: hi hi of 64 k is summed in tensor memory (8 additions) and then added to fp32
// registers, which hold the running sum over K; the small products (2^-12 of the result) are summed in tensor memory to the
// end.  Measured against 64 bits (K 2,048 to 6,144, normal inputs): 2.1e-7 to 2.7e-7,
// of which 1.5e-7 is a bias towards zero (the sums in tensor memory are cut off, not rounded); a chain of fp32 FMA over 32-k tiles
// with two sums an output 5.7e-7 to 9.9e-7.
//
// A word that is not finite has no such terms, a word near the least normal number loses its second one, and products beyond
// the range of fp32 cancel as inf - inf; outputs whose rows hold such words (terms_suffice) are formed from the operands in
// global memory instead, with fp32 FMA in the order of k.
//
// A block owns 128 tokens x 128 weight rows.  Warp 0 brings 32 k of both operands at a time by TMA (128-byte swizzle, four stages).
// Warps 2..5 split the tokens' words and leave both terms in tensor memory, from where the MMAs read their A operand; warps
// 6..9 replace the weights' words by their hi terms and leave the lo terms beside them (the same place in a second tile, so
// nothing depends on the swizzle); warp 1 issues the MMAs, warps 10..17 add up.  Bound by shared memory: 32 KB in, 32 KB read and
// 32 KB written by the split, 48 KB read by the MMAs, 144 KB at 128 bytes a cycle for 768 cycles of MMAs.  (With the tokens' terms
// in shared memory too it was 224 KB, and 70 us where this takes 57.)
// Where tiles are fewer than SMs a cluster of `splits` blocks shares a tile's K: every block leaves its sums in its own shared
// memory, and each adds a share of the rows over the ranks, in rank order.  Every wait is bounded.
// Measured (509 tokens): 12,288 x 2,048 170 us (150 TFLOP/s), 4,096 x 2,048 56 us, 2,048 x 6,144 88 us (two splits); tiles of packed
// FMA (fma.rn.f32x2, 8 x 8 sums a thread) 617, 206 and 320 us.
#include "gemm_f32.h"
#include "tc_common.cuh"

namespace leone {
namespace tc {

constexpr int kFtM = 128, kFtN = 128, kFtK = 32, kFtStages = 4;
constexpr int kFtSplitWarps = 8, kFtSumWarps = 8, kFtThreads = 32 * (2 + kFtSplitWarps + kFtSumWarps);
constexpr int kFtTile = kFtM * kFtK * 4;                  // the tokens' words, the weights' hi terms, their lo terms
constexpr int kFtStage = 3 * kFtTile;
// tensor memory: two sums of hi hi, the sum of the small products, two sets of the tokens' hi and lo terms
constexpr int kFtSmall = 2 * kFtN, kFtTerms = 3 * kFtN, kFtTermCols = 2 * kFtK;
constexpr int kFtPitch = kFtN + 4;                        // floats of a row of the tile's sums
constexpr int kFtSmem = kFtStages * kFtStage + 1024 + 256;
static_assert(kFtM * kFtPitch * 4 <= kFtStages * kFtStage, "the sums fit where the stages were");

// The nearest number of 11 significant bits (of two as near the larger), in integer steps: the conversion instruction runs at a
// fraction of their rate.  For finite words; the caller looks for the others in the words' magnitudes.
__device__ __forceinline__ uint32_t to_tf32(float x) { return (__float_as_uint(x) + 0x1000u) & 0xffffe000u; }

// The two terms hold a word to 2^-23 of it while the second stays above the least normal number, and products and sums must stay
// below the largest: what an output can meet is told by the largest magnitudes of its token's and its weight row's words
// (over the block's K).  lo, hi: the least but zero, and the largest, of several weight rows.  False too for an infinity or a NaN.
constexpr float kFtLeast = 0x1p-100f, kFtMostProduct = 0x1p110f, kFtMostWord = 0x1p126f;
__device__ __forceinline__ bool terms_suffice(float x, float lo, float hi) {
  if (x == 0.f || hi == 0.f) return x < kFtMostWord && hi < kFtMostWord;
  return x >= kFtLeast && x < kFtMostWord && lo >= kFtLeast && hi < kFtMostWord && x * hi < kFtMostProduct && x * lo >= kFtLeast;
}
__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
  hi = to_tf32(x);
  lo = to_tf32(x - __uint_as_float(hi));
}
// The largest magnitude of words in two running maxima of three operands an instruction: as signed integers the largest
// positive word wins, as unsigned ones the largest negative, if there is one.
struct Largest {
  int s = 0;
  uint32_t u = 0;
  __device__ __forceinline__ void add(const float4& x) {
    s = __vimax3_s32(__vimax3_s32(s, __float_as_int(x.x), __float_as_int(x.y)), __float_as_int(x.z), __float_as_int(x.w));
    u = __vimax3_u32(__vimax3_u32(u, __float_as_uint(x.x), __float_as_uint(x.y)), __float_as_uint(x.z), __float_as_uint(x.w));
  }
  __device__ __forceinline__ uint32_t magnitude() const { return max((uint32_t)s, u & 0x7fffffffu); }
};
// D[tmem] (+)= A[tmem] * B[smem]^T: row m of A in lane m, an element a column.
__device__ __forceinline__ void umma_tf32(uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// 16 consecutive 32-bit columns of this thread's lane.
__device__ __forceinline__ void tmem_store16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// tf32 x tf32 -> fp32, both operands K-major.
__host__ __device__ constexpr uint32_t instr_desc_tf32(int m, int n) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__global__ void __launch_bounds__(kFtThreads, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const float* A,
                   const float* W, float* C, const float* residual, const float* bias, int M, int N, int K, int lda,
                   int ldw, int ldc, int splits, int* status) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t tiles_base = (raw + 1023u) & ~1023u;
  uint8_t* tiles = smem_raw + (tiles_base - raw);
  uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + kFtStages * kFtStage);
  const uint32_t raw_full0 = smem_u32(bars), split_full0 = raw_full0 + 8 * kFtStages, empty0 = split_full0 + 8 * kFtStages;
  const uint32_t sum_full0 = empty0 + 8 * kFtStages, sum_empty0 = sum_full0 + 16, terms_empty0 = sum_empty0 + 16;
  __shared__ uint32_t tmem_holder;
  __shared__ int gave_up;
  __shared__ uint32_t x_most[kFtM], w_most[kFtN], w_low, w_high;      // magnitudes: of every row, and over the weight rows
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = splits > 1 ? (int)cluster_ctarank() : 0;
  const int m0 = blockIdx.y * kFtM, n0 = (blockIdx.x / splits) * kFtN;
  const int steps = (K + kFtK - 1) / kFtK;
  const int first = (int)((long long)steps * rank / splits), last = (int)((long long)steps * (rank + 1) / splits);
  if (threadIdx.x == 0) {
    gave_up = 0;
    w_low = 0x7f7fffffu;
    w_high = 0;
    for (int s = 0; s < kFtStages; ++s) {
      mbar_init(raw_full0 + 8 * s, 1);
      mbar_init(split_full0 + 8 * s, kFtSplitWarps);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(sum_full0 + 8 * b, 1);
      mbar_init(sum_empty0 + 8 * b, kFtSumWarps);
      mbar_init(terms_empty0 + 8 * b, 1);
    }
    mbar_fence_init();
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_w);
  }
  __syncthreads();
  if (warp == 1) tmem_alloc(smem_u32(&tmem_holder), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_holder;
  volatile int* giveup = &gave_up;
  pdl_trigger();

  if (warp == 0) {
    // ---------------- copies: the first stages' weights before the wait for the kernel before this one ----------------
    if (elect_one()) {
      const int early = min(kFtStages, last - first);
      for (int i = 0; i < early; ++i) {
        mbar_expect_tx(raw_full0 + 8 * i, 2 * kFtTile);
        tma_load_2d(tiles_base + i * kFtStage + kFtTile, &map_w, raw_full0 + 8 * i, (first + i) * kFtK, n0);
      }
      pdl_wait();
      int stage = 0;
      uint32_t phase = 0;
      for (int step = first; step < last; ++step) {
        const uint32_t bar = raw_full0 + 8 * stage, dst = tiles_base + stage * kFtStage;
        if (step - first >= early) {
          if (!mbar_wait(empty0 + 8 * stage, phase ^ 1, giveup)) break;
          mbar_expect_tx(bar, 2 * kFtTile);
          tma_load_2d(dst + kFtTile, &map_w, bar, step * kFtK, n0);
        }
        tma_load_2d(dst, &map_a, bar, step * kFtK, m0);
        if (++stage == kFtStages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMAs ----------------
    if (elect_one()) {
      const uint32_t idesc = instr_desc_tf32(kFtM, kFtN);
      const uint32_t small = tmem_base + kFtSmall;
      int stage = 0;
      uint32_t phase = 0;
      for (int step = first; step < last; ++step) {
        const int i = step - first, pair = i >> 1, buf = pair & 1;
        if ((i & 1) == 0 && !mbar_wait(sum_empty0 + 8 * buf, ((pair >> 1) & 1) ^ 1, giveup)) break;
        if (!mbar_wait(split_full0 + 8 * stage, phase, giveup)) break;
        tc_fence_after();
        const uint32_t at = tiles_base + stage * kFtStage, big = tmem_base + buf * kFtN;
        const uint32_t a_hi = tmem_base + kFtTerms + (i & 1) * kFtTermCols, a_lo = a_hi + kFtK;
        const uint64_t w_hi = smem_desc_sw128(at + kFtTile), w_lo = smem_desc_sw128(at + 2 * kFtTile);
#pragma unroll
        for (int k = 0; k < kFtK / 8; ++k) {
          umma_tf32(big, a_hi + 8 * k, w_hi + 2 * k, idesc, (i & 1) || k > 0 ? 1u : 0u);
          umma_tf32(small, a_hi + 8 * k, w_lo + 2 * k, idesc, i > 0 || k > 0 ? 1u : 0u);
          umma_tf32(small, a_lo + 8 * k, w_hi + 2 * k, idesc, 1u);
        }
        umma_commit(terms_empty0 + 8 * (i & 1));
        umma_commit(empty0 + 8 * stage);
        if ((i & 1) || step + 1 == last) umma_commit(sum_full0 + 8 * buf);
        if (++stage == kFtStages) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp < 6) {
    // ---------------- split of the tokens: a thread's row of 32 words, both terms to its lane of tensor memory ----------------
    const int quarter = warp & 3, row = quarter * 32 + lane;
    int stage = 0;
    uint32_t phase = 0;
    Largest most;
    for (int step = first; step < last; ++step) {
      const int i = step - first;
      bool ok = mbar_wait(terms_empty0 + 8 * (i & 1), ((i >> 1) & 1) ^ 1, giveup) && mbar_wait(raw_full0 + 8 * stage, phase, giveup);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      const float4* words = reinterpret_cast<const float4*>(tiles + stage * kFtStage + row * 128);
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + kFtTerms + (i & 1) * kFtTermCols;
#pragma unroll
      for (int c0 = 0; c0 < 8; c0 += 4) {
        uint32_t h[16], l[16];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float4 x = words[(c0 + c) ^ (row & 7)];            // the 128-byte swizzle: 16-byte pieces by row
          most.add(x);
          split_tf32(x.x, h[4 * c], l[4 * c]);
          split_tf32(x.y, h[4 * c + 1], l[4 * c + 1]);
          split_tf32(x.z, h[4 * c + 2], l[4 * c + 2]);
          split_tf32(x.w, h[4 * c + 3], l[4 * c + 3]);
        }
        tmem_store16(taddr + 4 * c0, h);
        tmem_store16(taddr + kFtK + 4 * c0, l);
      }
      if (step + 1 == last) x_most[row] = most.magnitude();
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(split_full0 + 8 * stage);
      if (++stage == kFtStages) { stage = 0; phase ^= 1; }
    }
  } else if (warp < 2 + kFtSplitWarps) {
    // ---------------- split of the weights: words to hi terms in place, lo terms in the next tile ----------------
    const int at = (warp - 6) * 32 + lane;
    constexpr int kPieces = kFtTile / 16 / 128;            // a thread's, each of another row
    int stage = 0;
    uint32_t phase = 0;
    Largest most[kPieces];
    for (int step = first; step < last; ++step) {
      bool ok = mbar_wait(raw_full0 + 8 * stage, phase, giveup);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      float4* words = reinterpret_cast<float4*>(tiles + stage * kFtStage + kFtTile);
      uint4* hi = reinterpret_cast<uint4*>(words);
      uint4* lo = hi + kFtTile / 16;
#pragma unroll
      for (int j = 0; j < kPieces; ++j) {
        const int i = at + j * 128;
        const float4 x = words[i];
        uint4 h, l;
        most[j].add(x);
        split_tf32(x.x, h.x, l.x);
        split_tf32(x.y, h.y, l.y);
        split_tf32(x.z, h.z, l.z);
        split_tf32(x.w, h.w, l.w);
        hi[i] = h;
        lo[i] = l;
      }
      if (step + 1 == last) {
#pragma unroll
    for (int j = 0; j < kPieces; ++j) {                    // a row's eight pieces are neighbouring lanes'
      uint32_t m = most[j].magnitude();
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
      if ((lane & 7) == 0) {
        w_most[(at + j * 128) / 8] = m;
        atomicMax(&w_high, m);
        if (m != 0) atomicMin(&w_low, m);
      }
    }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(split_full0 + 8 * stage);
      if (++stage == kFtStages) { stage = 0; phase ^= 1; }
    }
  } else {
    // ---------------- sums: a thread holds half of a token's row of the tile ----------------
    const int quarter = warp & 3, half = (warp - 2 - kFtSplitWarps) >> 2;        // (a warp reads the 32 lanes of tensor memory of its number mod 4)
    const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + half * (kFtN / 2);
    float acc[kFtN / 2];
#pragma unroll
    for (int j = 0; j < kFtN / 2; ++j) acc[j] = 0.f;
    auto add = [&](uint32_t at) {
#pragma unroll
      for (int c = 0; c < kFtN / 2; c += 16) {
        float v[16];
        tmem_ld16(at + c, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) acc[c + j] += v[j];
      }
    };
    const int pairs = (last - first + 1) / 2;
    bool ok = true;
    for (int pair = 0; pair < pairs; ++pair) {
      const int buf = pair & 1;
      ok = mbar_wait(sum_full0 + 8 * buf, (pair >> 1) & 1, giveup);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      add(taddr + buf * kFtN);
      if (pair + 1 == pairs) add(taddr + kFtSmall);      // the last commit covers the small products too
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(sum_empty0 + 8 * buf);
    }
    pdl_wait();
    // (every MMA is done, so the stages are free)
    const int row = quarter * 32 + lane;
    float* dst = reinterpret_cast<float*>(tiles) + row * kFtPitch + half * (kFtN / 2);
#pragma unroll
    for (int c = 0; c < kFtN / 2; c += 4) *reinterpret_cast<float4*>(dst + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
    const float x = __uint_as_float(x_most[row]);
    if (!terms_suffice(x, __uint_as_float(w_low), __uint_as_float(w_high))) {
      const float* a = A + (size_t)min(m0 + row, M - 1) * lda;
      for (int c = 0; c < kFtN / 2; ++c) {
        const float most = __uint_as_float(w_most[half * (kFtN / 2) + c]);
        if (terms_suffice(x, most, most)) continue;
        const float* w = W + (size_t)min(n0 + half * (kFtN / 2) + c, N - 1) * ldw;
        float sum = 0.f;
        for (int k = first * kFtK; k < min(last * kFtK, K); ++k) sum = fmaf(a[k], w[k], sum);
        dst[c] = sum;
      }
    }
  }
  __syncwarp();
  if (splits > 1) cluster_sync_all();
  else __syncthreads();
  if (warp < 2 + kFtSplitWarps) pdl_wait();              // (they write too)
  const bool wide = ldc % 4 == 0 && (((uintptr_t)C | (uintptr_t)residual) & 15) == 0;
  for (int i = rank * kFtThreads + threadIdx.x; i < kFtM * kFtN / 4; i += splits * kFtThreads) {
    const int r = i / (kFtN / 4), c = (i % (kFtN / 4)) * 4;
    float v[4] = {0.f, 0.f, 0.f, 0.f};
    if (splits == 1) {
      const float4 x = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(tiles) + r * kFtPitch + c);
      v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    } else {
      for (int u = 0; u < splits; ++u) {
        const uint32_t at = cluster_map(tiles_base + (r * kFtPitch + c) * 4, u);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] += cluster_ld_f32(at + 4 * j);
      }
    }
    const int m = m0 + r, n = n0 + c;
    if (m >= M) continue;
    float* out = C + (size_t)m * ldc + n;
    if (wide && n + 3 < N) {
      if (bias != nullptr)
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] += bias[n + j];
      if (residual != nullptr) {
        const float4 x = *reinterpret_cast<const float4*>(residual + (size_t)m * ldc + n);
        v[0] += x.x; v[1] += x.y; v[2] += x.z; v[3] += x.w;
      }
      *reinterpret_cast<float4*>(out) = make_float4(v[0], v[1], v[2], v[3]);
      continue;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (n + j >= N) break;
      if (bias != nullptr) v[j] += bias[n + j];
      if (residual != nullptr) v[j] += residual[(size_t)m * ldc + n + j];
      out[j] = v[j];
    }
  }
  tc_fence_before();
  if (splits > 1) cluster_sync_all();                    // a block's sums stay until everyone has read them
  else __syncthreads();
  if (threadIdx.x == 0 && gave_up) set_status(status, kWaitTimeout, blockIdx.x, 50);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// Row-major fp32 matrix, tiles of [128, 32] with 128-byte swizzle.
inline int make_map_f32(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (fn == nullptr) return kRefusedSize;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * 4};
  cuuint32_t box[2] = {kFtK, 128};
  cuuint32_t elem[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, elem,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : kRefusedAlignment;
}

}  // namespace tc

int gemm_f32_tc(const float* a, const float* w, float* c, const float* residual, const float* bias, int m, int n, int k,
                int lda, int ldw, int ldc, int* status, cudaStream_t stream) {
  using namespace tc;
  CUtensorMap map_a, map_w;
  int e = make_map_f32(&map_a, a, m, k, lda);
  if (e == 0) e = make_map_f32(&map_w, w, n, k, ldw);
  if (e != 0) return e;
  static const cudaError_t ready = cudaFuncSetAttribute(gemm_f32_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFtSmem);
  if (ready != cudaSuccess) return (int)ready;
  const int tiles_n = (n + kFtN - 1) / kFtN, tiles_m = (m + kFtM - 1) / kFtM;
  if (tiles_m > 65535) return kRefusedSize;
  // As many splits as run at once (74 clusters of two, 33 of four, 15 of eight with a block an SM), while a block keeps at
  // least eight steps.
  const long long tiles = (long long)tiles_n * tiles_m;
  int splits = 1;
  while (splits < 8 && tiles <= (splits == 1 ? 74 : splits == 2 ? 33 : 15) && (k + kFtK - 1) / kFtK >= splits * 2 * 8) splits *= 2;
  const dim3 grid(tiles_n * splits, tiles_m);
  if (splits == 1)
    return launch_kernel(gemm_f32_tc_kernel, grid, dim3(kFtThreads), kFtSmem, stream, map_a, map_w, a, w, c, residual, bias, m, n, k,
                         lda, ldw, ldc, 1, status);
  return launch_kernel_cluster(gemm_f32_tc_kernel, grid, dim3(kFtThreads), kFtSmem, stream, dim3(splits, 1, 1), map_a, map_w, a, w, c,
                               residual, bias, m, n, k, lda, ldw, ldc, splits, status);
}

}  // namespace leone
