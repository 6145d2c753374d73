// Attention through a cached latent for prompt portions on the 5th-generation tensor cores: rows of 576 elements, of which the first
// 512 are the value (a rank of 512 and a rotated part of 64).
//
// The formulas of attention_latent_mma.cu: all heads share the cache rows as keys and their first elements as values; fp32 online
// softmax with the per-head sink as one more score; an output gate.  That kernel's mma.sync tiles hold the heads of one token (16 rows)
// and read every key row once for each product from shared memory: bound by that traffic at a tenth of the tensor cores' rate.  Here
// a tile of queries is eight tokens of a sequence by 16 heads, 128 rows.
//
// A block owns one tile of queries and half of the value columns: 128 x 512 sums would be all of tensor memory, so two blocks share a
// tile, each with the scores for itself (1.5 times the operations of one block, none of the traffic between two).  Tensor memory: the sums
// O (256 columns), two tiles of scores S of 64 keys (64 each; the probabilities P as bfloat16 pairs over their first half), and the
// first 256 elements of the queries (128), which makes room in shared memory for two tiles of keys:
//   S(t) = Q K(t)^T      keys K-major as they lie in the pages; the queries' first four pieces of 64 elements from tensor memory, the
//                        other five from shared memory
//   O += P(t) V(t)       V is the same tile read MN-major (a key a row), P from tensor memory
// issued as S(t + 1), PV(t), so that the tensor cores have the next scores to make while the softmax of a tile runs.
//
// Warps: 0-3 softmax, a thread a row; 4 issues the MMAs; 5-8 gather tiles of keys from the pages with 16-byte asynchronous copies
// that write the 128-byte-swizzled layout (TMA copies of a page's 16 rows by 64 elements, 36 of them a tile, took 216 us in place of 196).  Every wait
// is bounded.
//
// A tile's chain bounds it (the gather of 73 KB, scores, softmax), not the tensor cores.  One sequence of 2,048 tokens, 16 heads, a
// window of 1,024: 415 us in the mma.sync form, 197 in this (0.17 of the bf16 rate, from 0.08); a prompt of the eight-layer decoder
// with two such layers 4.51 to 4.08 ms.  Its error against 64 bits is no larger than that form's.
// A tile walks its keys alone, so few tokens behind many keys take the other form, which splits them over blocks (8 tokens behind 16,384:
// 824 us here, 150 there); the rule and its measurements are latent_times in ops/cuda.py.
#include "tc_common.cuh"

namespace leone {
namespace latent_tc {

using namespace leone::tc;

constexpr int kRows = 128, kKeys = 64, kHeads = 16, kTokens = kRows / kHeads;
constexpr int kDk = 576, kDv = 512, kPieces = kDk / 64, kTmemPieces = 4, kSmemPieces = kPieces - kTmemPieces;
constexpr int kHalf = kDv / 2;
constexpr int kPieceQ = kRows * 128, kPieceK = kKeys * 128;      // bytes of 64 elements of a tile
constexpr int kTileK = kPieces * kPieceK;
constexpr int kColS = kHalf, kColQ = kHalf + 2 * kKeys;          // tensor memory columns
constexpr int kLoadWarp0 = 5, kLoadThreads = 128;
constexpr int kThreads = kLoadWarp0 * 32 + kLoadThreads;
constexpr int kSmem = kSmemPieces * kPieceQ + 2 * kTileK + 1024 /*alignment*/ + 128 /*barriers*/;
constexpr float kLog2e = 1.4426950408889634f;

struct Params {
  const __nv_bfloat16* q;          // [n_tokens, heads, 576]
  const __nv_bfloat16* pool;       // [num_pages, page_tokens, 576]
  __nv_bfloat16* out;              // [n_tokens, heads, 512]
  const int* block_table;
  int table_width;
  const int* q_start;
  const int* ctx_len;
  int heads;
  float scale;
  int window;
  const void* sink;                // [heads] or null
  int sink_bf16;
  const __nv_bfloat16* gate;       // [n_tokens, >= heads] or null
  int ldg;
  int page_tokens, num_pages;
  int* status;
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// MN-major operand: a row of 128 bytes per K index, the next 64 MN elements `stride` bytes further (128-byte swizzle).
__device__ __forceinline__ uint64_t smem_desc_mn_sw128(uint32_t addr, uint32_t stride) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((stride >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)(1024u >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
__device__ __forceinline__ void umma_a_tmem(uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__global__ void __launch_bounds__(kThreads, 1)
attention_latent_tc_kernel(const Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  const uint32_t q_s = base, k_s = q_s + kSmemPieces * kPieceQ, bars = k_s + 2 * kTileK;
  const uint32_t bar_q = bars, bar_k = bars + 8, bar_free = bars + 24, bar_s = bars + 40, bar_p = bars + 56, bar_o = bars + 72;
  __shared__ uint32_t tmem_holder;
  __shared__ int gave_up, bad;
  __shared__ int row_s[2 * kKeys];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    gave_up = 0;
    bad = 0;
    mbar_init(bar_q, 4);
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_k + 8 * b, kLoadThreads / 32);
      mbar_init(bar_free + 8 * b, 1);
      mbar_init(bar_s + 8 * b, 1);
      mbar_init(bar_p + 8 * b, 4);
    }
    mbar_init(bar_o, 1);
    mbar_fence_init();
  }
  if (warp == 4) tmem_alloc(smem_u32(&tmem_holder), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_holder;
  volatile int* giveup = &gave_up;
  pdl_trigger();
  pdl_wait();

  // the tiles with the most keys first; neighbouring blocks are the two halves of one tile
  const int seq = blockIdx.z, h0 = blockIdx.y * kHeads;
  const int half = blockIdx.x & 1, tile = (int)(gridDim.x >> 1) - 1 - (int)(blockIdx.x >> 1);
  const int q0 = p.q_start[seq], q_len = p.q_start[seq + 1] - q0;
  const int tok0 = tile * kTokens;
  if (tok0 < q_len) {                                            // block-uniform
    const int start = p.ctx_len[seq] - q_len;
    const int first_pos = start + tok0, last_pos = start + min(q_len, tok0 + kTokens) - 1;
    const int lo = p.window > 0 ? max(0, first_pos - p.window + 1) : 0;
    const int tile0 = lo / kKeys * kKeys, n = (last_pos - tile0) / kKeys + 1;

    if (warp == 4) {
      // ---------------- MMA issuer ----------------
      if (elect_one()) {
        constexpr uint32_t idesc_s = instr_desc_bf16(kRows, kKeys), idesc_o = instr_desc_bf16(kRows, kHalf) | (1u << 16);
        auto issue_s = [&](int t) {
          const uint32_t k_t = k_s + (t & 1) * kTileK, d = tmem + kColS + (t & 1) * kKeys;
#pragma unroll
          for (int c = 0; c < kPieces; ++c) {
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
              const uint64_t b = smem_desc_sw128(k_t + c * kPieceK + ks * 32);
              if (c < kTmemPieces) umma_a_tmem(d, tmem + kColQ + c * 32 + ks * 8, b, idesc_s, c + ks > 0 ? 1u : 0u);
              else umma_bf16(d, smem_desc_sw128(q_s + (c - kTmemPieces) * kPieceQ + ks * 32), b, idesc_s, 1u);
            }
          }
          umma_commit(bar_s + 8 * (t & 1));
        };
        auto issue_pv = [&](int t) {
          const uint32_t v_t = k_s + (t & 1) * kTileK + half * (kHalf / 64) * kPieceK;
#pragma unroll
          for (int ks = 0; ks < kKeys / 16; ++ks)                // 16 keys: 8 columns of P, 16 rows of V
            umma_a_tmem(tmem, tmem + kColS + (t & 1) * kKeys + ks * 8, smem_desc_mn_sw128(v_t + ks * 2048, kPieceK), idesc_o,
                        t + ks > 0 ? 1u : 0u);
        };
        auto keys_there = [&](int t) { return mbar_wait(bar_k + 8 * (t & 1), (t >> 1) & 1, giveup); };
        bool ok = mbar_wait(bar_q, 0, giveup) && keys_there(0);
        if (ok) {
          tc_fence_after();
          issue_s(0);
        }
        for (int t = 0; t < n && ok; ++t) {
          if (t + 1 < n) {
            ok = keys_there(t + 1);
            if (!ok) break;
            tc_fence_after();
            issue_s(t + 1);
          }
          ok = mbar_wait(bar_p + 8 * (t & 1), (t >> 1) & 1, giveup);
          if (!ok) break;
          tc_fence_after();
          issue_pv(t);
          umma_commit(bar_free + 8 * (t & 1));
          if (t == n - 1) umma_commit(bar_o);
        }
      }
    } else if (warp >= kLoadWarp0) {
      // ---------------- the warps that gather tiles of keys ----------------
      const int lt = tid - kLoadWarp0 * 32;
      const int* table = p.block_table + (size_t)seq * p.table_width;
      // The row of key j in the pool, or -1 where no query reads it: such rows are zeros in the tile (what a page holds there
      // may be anything, and zero times it is not zero then).
      auto row_of = [&](int j) {
        if (j < lo || j > last_pos) return -1;
        const int blk = j / p.page_tokens, page = blk < p.table_width ? table[blk] : -1;
        if (page < 0 || page >= p.num_pages) {
          set_status(p.status, kBadPage, q0 + tok0, page, j);
          bad = 1;
          __threadfence_block();
          return -1;
        }
        return page * p.page_tokens + j % p.page_tokens;
      };
      int next_row = lt < kKeys ? row_of(tile0 + lt) : -1;       // looked up a tile ahead
      bool ok = true;
      for (int t = 0; t < n; ++t) {
        int* rows = row_s + (t & 1) * kKeys;
        if (lt < kKeys) {
          rows[lt] = next_row;
          if (t + 1 < n) next_row = row_of(tile0 + (t + 1) * kKeys + lt);
        }
        if (t >= 2 && ok && !mbar_wait(bar_free + 8 * (t & 1), ((t >> 1) - 1) & 1, giveup)) ok = false;
        named_barrier_sync(1, kLoadThreads);                     // the tile's rows are known
        const uint32_t dst = k_s + (t & 1) * kTileK;
#pragma unroll 4
        for (int i = lt; i < kKeys * (kDk / 8); i += kLoadThreads) {
          const int r = i / (kDk / 8), u = i - r * (kDk / 8);    // 16-byte piece u of row r
          const int row = rows[r];
          const __nv_bfloat16* src = p.pool + (size_t)(row < 0 ? 0 : row) * kDk + u * 8;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + (u >> 3) * kPieceK + r * 128 + (((u & 7) ^ (r & 7)) << 4)),
                       "l"(src), "r"(row < 0 ? 0 : 16) : "memory");
        }
        asm volatile("cp.async.commit_group;\n cp.async.wait_group 0;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_k + 8 * (t & 1));
      }
    } else {
      // ---------------- softmax: a thread per query row ----------------
      const int row = warp * 32 + lane, tok = tok0 + row / kHeads, head = h0 + row % kHeads;
      const bool here = tok < q_len && head < p.heads;
      const int pos = here ? start + tok : -1;
      const uint32_t t_lane = tmem + ((uint32_t)(warp * 32) << 16);
      {
        const uint4* src = reinterpret_cast<const uint4*>(p.q + ((size_t)(q0 + (here ? tok : tok0)) * p.heads + (here ? head : h0)) * kDk);
#pragma unroll
        for (int c = 0; c < kTmemPieces * 2; ++c) {              // 32 elements: 16 columns
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint4 v = here ? src[c * 4 + i] : make_uint4(0, 0, 0, 0);
            w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
          }
          tmem_st16(t_lane + kColQ + c * 16, w);
        }
#pragma unroll
        for (int i = 0; i < kSmemPieces * 8; ++i) {
          const uint4 v = here ? src[kTmemPieces * 8 + i] : make_uint4(0, 0, 0, 0);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(q_s + (i >> 3) * kPieceQ + row * 128 + (((i & 7) ^ (row & 7)) << 4)),
                       "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
        }
        tmem_st_wait();
        fence_proxy_async();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_q);
      }
      const float sl2 = p.scale * kLog2e;
      float m_run = -INFINITY, l_run = 0.f;
      if (p.sink != nullptr && here) {                           // the sink is the first score
        m_run = (p.sink_bf16 ? __bfloat162float(((const __nv_bfloat16*)p.sink)[head]) : ((const float*)p.sink)[head]) * kLog2e;
        l_run = m_run == -INFINITY ? 0.f : 1.f;                  // (a sink of -inf, or one that is after the factor, has no weight)
      }
      const int first_seen = p.window > 0 ? max(0, pos - p.window + 1) : 0;
      bool ok = true;
      for (int t = 0; t < n; ++t) {
        const uint32_t t_s = t_lane + kColS + (t & 1) * kKeys;
        const int j0 = tile0 + t * kKeys;
        if (ok && !mbar_wait(bar_s + 8 * (t & 1), (t >> 1) & 1, giveup)) ok = false;
        tc_fence_after();
        const bool whole = j0 + kKeys - 1 <= first_pos && (p.window <= 0 || j0 > last_pos - p.window);   // seen whole by every row
        uint32_t sc[64];
        tmem_ld32_issue(t_s, sc);
        tmem_ld32_issue(t_s + 32, sc + 32);
        tmem_ld_wait();
        if (!whole) {
#pragma unroll
          for (int i = 0; i < 64; ++i)
            if (j0 + i > pos || j0 + i < first_seen) sc[i] = __float_as_uint(-INFINITY);
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 64; ++i) mx[i & 3] = fmaxf(mx[i & 3], __uint_as_float(sc[i]));
        const float tile_max = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sl2;      // the scale is positive
        float alpha = 1.f;
        if (m_run == -INFINITY) {
          m_run = tile_max;
        } else if (tile_max > m_run) {                           // (exactly: the largest weight so far is then 1 and not rounded)
          alpha = ex2(m_run - tile_max);
          m_run = tile_max;
          l_run *= alpha;
        }
        if (t > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {    // warp-uniform: the loads and stores are collective
          // O is at rest once the product of the tile before is done
          bool rest = ok && mbar_wait(bar_free + 8 * ((t - 1) & 1), ((t - 1) >> 1) & 1, giveup);
          rest = __all_sync(0xffffffffu, rest);
          tc_fence_after();
          if (rest) {
#pragma unroll 1
            for (int c = 0; c < kHalf; c += 32) {
              uint32_t r[32];
              tmem_ld32_issue(t_lane + c, r);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) * alpha);
              tmem_st16(t_lane + c, r);
              tmem_st16(t_lane + c + 16, r + 16);
            }
          } else {
            ok = false;
          }
        }
        const float shift = m_run == -INFINITY ? 0.f : -m_run;
        float l[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 2; ++c) {                            // 32 keys: 16 columns of P
          uint32_t w[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const float a = ex2(fmaf(__uint_as_float(sc[32 * c + 2 * i]), sl2, shift)),
                        b = ex2(fmaf(__uint_as_float(sc[32 * c + 2 * i + 1]), sl2, shift));
            __nv_bfloat162 v2 = __floats2bfloat162_rn(a, b);
            w[i] = *reinterpret_cast<uint32_t*>(&v2);
            // the sum is of the rounded weights, those that the values are multiplied with
            l[i & 3] += __uint_as_float(w[i] << 16) + __uint_as_float(w[i] & 0xffff0000u);
          }
          tmem_st16(t_s + c * 16, w);
        }
        l_run += (l[0] + l[1]) + (l[2] + l[3]);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_p + 8 * (t & 1));
      }
      if (ok && !mbar_wait(bar_o, 0, giveup)) ok = false;
      ok = __all_sync(0xffffffffu, ok);
      tc_fence_after();
      if (ok) {
        const bool zeros = *(volatile int*)&bad != 0;            // (a sum that is NaN stays one: its outputs are too)
        float f = l_run > 0.f ? 1.f / l_run : 0.f;
        if (p.gate != nullptr && here) f *= 1.f / (1.f + expf(-__bfloat162float(p.gate[(size_t)(q0 + tok) * p.ldg + head])));
        uint4* dst = reinterpret_cast<uint4*>(p.out + ((size_t)(q0 + (here ? tok : tok0)) * p.heads + (here ? head : h0)) * kDv + half * kHalf);
        for (int c = 0; c < kHalf; c += 32) {
          uint32_t r[32];
          tmem_ld32_issue(t_lane + c, r);
          tmem_ld_wait();
          if (here) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              uint32_t w[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                __nv_bfloat162 v2 = __floats2bfloat162_rn(__uint_as_float(r[8 * q + 2 * i]) * f, __uint_as_float(r[8 * q + 2 * i + 1]) * f);
                w[i] = zeros ? 0u : *reinterpret_cast<uint32_t*>(&v2);
              }
              dst[c / 8 + q] = make_uint4(w[0], w[1], w[2], w[3]);
            }
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (gave_up) {
    if (tid == 0) set_status(p.status, kWaitTimeout, blockIdx.x, 7);
    // let tile copies that are still in flight land before the block's memory goes away
    const long long began = clock64();
    while (clock64() - began < 200000) {}
    __syncthreads();
  }
  if (warp == 4) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace latent_tc
}  // namespace leone

using namespace leone;

// Rows of 576 elements with values of 512.
extern "C" int leone_attention_latent_tc_supported(int dk, int dv) { return dk == latent_tc::kDk && dv == latent_tc::kDv; }

// q, out, gate: the rows that q_start counts; sequences of any number of tokens.
extern "C" int leone_attention_latent_tc(const void* q, void* out, const void* pool, const int* block_table, int table_width,
                                         const int* q_start, const int* ctx_len, int n_seqs, int max_q_len, int heads, int dk, int dv,
                                         float scale, int window, const void* sink, int sink_dtype, const void* gate, int ldg,
                                         int page_tokens, int num_pages, int* status, cudaStream_t stream) {
  using namespace latent_tc;
  if (n_seqs <= 0 || max_q_len <= 0) return 0;
  if (!leone_attention_latent_tc_supported(dk, dv) || heads <= 0 || table_width <= 0 || page_tokens <= 0 || num_pages <= 0 || (long long)num_pages * page_tokens > 0x7fffffff || n_seqs > 65535 ||
      (heads + kHeads - 1) / kHeads > 65535 || !(scale > 0.f))
    return kRefusedSize;
  if (sink_dtype != 0 && sink_dtype != 1) return kRefusedDtype;
  if (((uintptr_t)q | (uintptr_t)out | (uintptr_t)pool) & 15) return kRefusedAlignment;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(attention_latent_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const Params p{(const __nv_bfloat16*)q, (const __nv_bfloat16*)pool, (__nv_bfloat16*)out, block_table, table_width, q_start, ctx_len, heads, scale, window, sink,
                 sink_dtype, (const __nv_bfloat16*)gate, ldg, page_tokens, num_pages, status};
  const dim3 grid(2 * ((max_q_len + kTokens - 1) / kTokens), (heads + kHeads - 1) / kHeads, n_seqs);
  return launch_kernel(attention_latent_tc_kernel, grid, dim3(kThreads), (size_t)kSmem, stream, p);
}
