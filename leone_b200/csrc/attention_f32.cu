// Causal grouped-query attention over a paged cache in 32 bits, head sizes 64 and 128: the fp32 path's attention where
// the sizes allow it (attention_generic.cu takes every size).
//
// The query at absolute position p reads keys lo..p of its own sequence (lo = 0, or p - window + 1), found through the
// block table; kv_head = q_head / (n_q / n_kv); score = (q.k) * scale; softmax and sums in fp32, running over key tiles in
// ascending order (crates/leone/src/cpu.rs:2299-2421; the mask is the loop bound, :2372).  A row's arithmetic depends on
// its own sequence only; splits of a sequence's keys in decode steps change the grouping of the sums, so rounding only.
#include "common.cuh"

namespace leone {
namespace attn32 {

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  const int bytes = valid ? 16 : 0;        // 0: zeros, the source is not read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void fma2(float2& acc, float2 a, float2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(reinterpret_cast<unsigned long long&>(acc))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
}

struct Params {
  const float* qkv;
  int row_stride;
  float* out;
  int out_stride;
  const float* k_pool;
  const float* v_pool;
  const int* block_table;
  int table_width;
  const int* q_start;
  const int* ctx_len;
  int n_q, n_kv;
  float scale;
  int window, page_tokens, num_pages;
  int* status;
};

// Row of the pools that holds position j of sequence s for kv head `kvh`, or -1 (reported) if its page is not valid.
__device__ __forceinline__ long long key_row(const Params& p, int s, int kvh, int j, int row) {
  const int blk = j / p.page_tokens;
  const int page = blk < p.table_width ? p.block_table[(size_t)s * p.table_width + blk] : -1;
  if (page < 0 || page >= p.num_pages) {
    set_status(p.status, kBadPage, row, page, j);
    return -1;
  }
  return ((long long)page * p.n_kv + kvh) * p.page_tokens + (j - blk * p.page_tokens);
}

// ---- prompt portions -----------------------------------------------------------------------------------------
// Bound by the FMA pipes: 4 * D operations per (row, key) pair.  A block owns 64 rows (tokens x heads of one kv head's
// group, so a key tile serves the whole group) and walks tiles of 64 keys; 256 threads own 4 x 4 scores and 4 rows x D / 16
// output columns each.  Rows lie in shared memory as in global memory, padded by 4 floats (8 neighbouring rows' 16-byte
// pieces cover all banks); products run on fma.rn.f32x2, over pairs of k for the scores and pairs of columns for the
// outputs.  Keys of the next tile are copied while the outputs of this one are summed, values while the scores are.
// Measured: 509 tokens, 16 heads on 8 of 128: 70 us; the any-size kernel (a block per token and head, which reads every key for
// itself) 1,155 us.
constexpr int kRowsQ = 64, kKeys = 64;

template <bool B> struct Masked { static constexpr bool value = B; };
template <int D>
struct PromptShape {
  static constexpr int kPitch = D + 4, kPitchP = kKeys + 4;
  static constexpr size_t kSmem = (size_t)((kRowsQ + kKeys) * kPitch + kKeys * D + kRowsQ * kPitchP) * sizeof(float);
};

template <int D>
__global__ void __launch_bounds__(256, 1)
attention_f32_prompt_kernel(const Params p) {
  using S = PromptShape<D>;
  constexpr int kCols = D / 16;                 // output columns a thread owns, in runs of 4 at 4 tx, 64 + 4 tx
  constexpr int kPieces = D / 4;                // 16-byte pieces of a row
  extern __shared__ __align__(16) float smem[];
  __shared__ long long key_rows[2][kKeys];
  float* q_s = smem;
  float* k_s = q_s + kRowsQ * S::kPitch;
  float* v_s = k_s + kKeys * S::kPitch;
  float* p_s = v_s + kKeys * D;
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = lane & 15, ty = warp * 2 + (lane >> 4);
  const int s = blockIdx.z, kvh = blockIdx.y, g = p.n_q / p.n_kv;
  const int q0 = p.q_start[s], q_len = p.q_start[s + 1] - q0, start = p.ctx_len[s] - q_len;
  // the longest rows (the last tile) first: the blocks of a grid start in order
  const int tile = gridDim.x - 1 - blockIdx.x;
  const int row0 = tile * kRowsQ, rows = q_len * g;
  if (row0 >= rows) return;
  if (start < 0) {
    if (tid == 0) set_status(p.status, kBadPosition, q0, start);
    return;
  }
  const int last_row = min(row0 + kRowsQ, rows) - 1;
  const int hi = start + last_row / g;                                     // the last position any row sees
  const int lo = p.window > 0 ? max(0, start + row0 / g - p.window + 1) : 0;   // the first

  const uint32_t q_at = (uint32_t)__cvta_generic_to_shared(q_s), k_at = (uint32_t)__cvta_generic_to_shared(k_s),
                 v_at = (uint32_t)__cvta_generic_to_shared(v_s);
  for (int i = tid; i < kRowsQ * kPieces; i += 256) {
    const int r = i / kPieces, c = (i % kPieces) * 4, row = row0 + r;
    const bool ok = row < rows;
    const float* src = p.qkv;
    if (ok) src += (size_t)(q0 + row / g) * p.row_stride + (size_t)(kvh * g + row % g) * D + c;
    cp_async16(q_at + (uint32_t)(r * S::kPitch + c) * 4, src, ok);
  }
  auto look_up = [&](int j0, int buf) {
    if (tid < kKeys) key_rows[buf][tid] = j0 + tid <= hi ? key_row(p, s, kvh, j0 + tid, q0) : -1;
  };
  auto load = [&](const float* pool, uint32_t dst, int pitch, int buf) {
    for (int i = tid; i < kKeys * kPieces; i += 256) {
      const int r = i / kPieces, c = (i % kPieces) * 4;
      const long long row = key_rows[buf][r];
      cp_async16(dst + (uint32_t)(r * pitch + c) * 4, row >= 0 ? pool + row * D + c : pool, row >= 0);
    }
  };
  const int tiles = (hi - lo) / kKeys + 1;
  look_up(lo, 0);
  __syncthreads();
  load(p.k_pool, k_at, S::kPitch, 0);
  cp_commit();

  float m_run[4], l_run[4];
  float2 acc[4][kCols / 2];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m_run[i] = -INFINITY;
    l_run[i] = 0.f;
#pragma unroll
    for (int c = 0; c < kCols / 2; ++c) acc[i][c] = make_float2(0.f, 0.f);
  }
  int pos[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) pos[i] = start + min(row0 + ty + 16 * i, rows - 1) / g;

  for (int t = 0; t < tiles; ++t) {
    const int j0 = lo + t * kKeys, buf = t & 1;
    cp_wait<0>();
    __syncthreads();                       // keys have landed; the values' and the weights' readers are done
    load(p.v_pool, v_at, D, buf);
    cp_commit();
    if (t + 1 < tiles) look_up(j0 + kKeys, buf ^ 1);
    float2 sc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) sc[i][j] = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int d = 0; d < D; d += 4) {
      float4 b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = *(const float4*)(k_s + (tx + 16 * j) * S::kPitch + d);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 a = *(const float4*)(q_s + (ty + 16 * i) * S::kPitch + d);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          fma2(sc[i][j], make_float2(a.x, a.y), make_float2(b[j].x, b[j].y));
          fma2(sc[i][j], make_float2(a.z, a.w), make_float2(b[j].z, b[j].w));
        }
      }
    }
    bool there[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) there[j] = key_rows[buf][tx + 16 * j] >= 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int first = p.window > 0 ? pos[i] - p.window + 1 : 0;
      float v[4], top = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = j0 + tx + 16 * j;
        v[j] = there[j] && key <= pos[i] && key >= first ? (sc[i][j].x + sc[i][j].y) * p.scale : -INFINITY;
        top = fmaxf(top, v[j]);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
      const float m_new = fmaxf(m_run[i], top);
      const float base = m_new == -INFINITY ? 0.f : m_new;       // a row that has seen no key yet: all weights 0
      const float alpha = expf(m_run[i] - base);
      m_run[i] = m_new;
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float w = expf(v[j] - base);
        sum += w;
        p_s[(ty + 16 * i) * S::kPitchP + tx + 16 * j] = w;
      }
      l_run[i] = l_run[i] * alpha + sum;
#pragma unroll
      for (int c = 0; c < kCols / 2; ++c) {
        acc[i][c].x *= alpha;
        acc[i][c].y *= alpha;
      }
    }
    cp_wait<0>();
    __syncthreads();                       // values have landed, weights are written, the keys' readers are done
    if (t + 1 < tiles) load(p.k_pool, k_at, S::kPitch, buf ^ 1);
    cp_commit();
    // Of a tile on the diagonal or at the window's edge a row takes its own keys only: a masked key's weight is 0, but its value
    // may be infinite.  (A missing page's values are zeros.)
    auto add = [&](auto some_masked) {
#pragma unroll 2
      for (int j = 0; j < kKeys; j += 4) {
        float w[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) *(float4*)w[i] = *(const float4*)(p_s + (ty + 16 * i) * S::kPitchP + j);
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          float4 v[kCols / 4];
#pragma unroll
          for (int c = 0; c < kCols / 4; ++c) v[c] = *(const float4*)(v_s + (j + jj) * D + 64 * c + 4 * tx);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 ww = make_float2(w[i][jj], w[i][jj]);
            const int key = j0 + j + jj;
            if (decltype(some_masked)::value && (key > pos[i] || (p.window > 0 && key <= pos[i] - p.window))) continue;
#pragma unroll
            for (int c = 0; c < kCols / 4; ++c) {
              fma2(acc[i][2 * c], ww, make_float2(v[c].x, v[c].y));
              fma2(acc[i][2 * c + 1], ww, make_float2(v[c].z, v[c].w));
            }
          }
        }
      }
    };
    if (j0 + kKeys - 1 > start + row0 / g || (p.window > 0 && j0 <= hi - p.window)) add(Masked<true>());
    else add(Masked<false>());
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float l = l_run[i];
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    const int row = row0 + ty + 16 * i;
    if (row >= rows) continue;
    const float inv = l > 0.f ? 1.f / l : 0.f;
    float* dst = p.out + (size_t)(q0 + row / g) * p.out_stride + (size_t)(kvh * g + row % g) * D;
#pragma unroll
    for (int c = 0; c < kCols / 4; ++c)
      *(float4*)(dst + 64 * c + 4 * tx) =
          make_float4(acc[i][2 * c].x * inv, acc[i][2 * c].y * inv, acc[i][2 * c + 1].x * inv, acc[i][2 * c + 1].y * inv);
  }
}

// ---- one token a sequence --------------------------------------------------------------------------------------
// Bound by the keys' and values' bytes.  A cluster of `splits` blocks owns a (sequence, kv head, up to GT heads of its
// group); the warps of all its blocks take runs of eight keys in turn (four with eight heads).  A lane holds D / 32 elements of every
// query and reads its piece of a run's keys and values, each a whole row per warp, all at once; the rows of the next run are
// looked up meanwhile.  With few short sequences the time is a chain of such reads, one after another, so runs are short and
// many warps are at work: runs of 32 keys in steps of four took a sequence of 300 through eight reads in a row, these
// through three.  Every warp keeps its own running maximum, sum and outputs; a block's meet in shared memory, then the blocks' across
// the cluster, in rank order.  Measured in the step of 4
// sequences of 300, 16 heads on 8 of 128: 17 us before the next kernel can start with runs of 32, 8 with runs of 8 (the
// any-size kernel 74).
constexpr int kWarps = 4, kMostSplits = 8;

template <int D, int GT>
__global__ void __launch_bounds__(kWarps * 32)
attention_f32_decode_kernel(const Params p, int head_groups, int splits) {
  constexpr int E = D / 32;                     // elements of a row a lane holds
  __shared__ float m_s[kWarps][GT], l_s[kWarps][GT];
  __shared__ __align__(16) float o_s[kWarps][GT][D];
  __shared__ float m_b[GT], l_b[GT];            // of the whole block
  constexpr int kRun = GT <= 4 ? 8 : 4;         // keys a warp reads at a time
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = splits > 1 ? (int)cluster_ctarank() : 0;
  const int s = blockIdx.z, kvh = blockIdx.y / head_groups, g = p.n_q / p.n_kv;
  const int h0 = (blockIdx.y % head_groups) * GT, heads = min(GT, g - h0);
  const int row = p.q_start[s], pos = p.ctx_len[s] - 1;
  const int lo = p.window > 0 ? max(0, pos - p.window + 1) : 0;
  if (pos < 0 && tid == 0) set_status(p.status, kBadPosition, row, pos);
  float q[GT][E], acc[GT][E], m_run[GT], l_run[GT];
#pragma unroll
  for (int h = 0; h < GT; ++h) {
    m_run[h] = -INFINITY;
    l_run[h] = 0.f;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      acc[h][e] = 0.f;
      q[h][e] = h < heads ? p.qkv[(size_t)row * p.row_stride + (size_t)(kvh * g + h0 + h) * D + lane * E + e] : 0.f;
    }
  }
  auto piece = [&](const float* src, float* dst) {
    if constexpr (E == 4) {
      const float4 v = *(const float4*)src;
      dst[0] = v.x; dst[1] = v.y; dst[2] = v.z; dst[3] = v.w;
    } else {
      const float2 v = *(const float2*)src;
      dst[0] = v.x; dst[1] = v.y;
    }
  };
  const int step = splits * kWarps * kRun;
  auto lookup = [&](int j0) { return lane < kRun && j0 + lane <= pos ? key_row(p, s, kvh, j0 + lane, row) : -1ll; };
  int j0 = lo + (rank * kWarps + warp) * kRun;
  long long mine = lookup(j0);
  for (; j0 <= pos; j0 += step) {
    long long at[kRun];
    float k[kRun][E], v[kRun][E];
#pragma unroll
    for (int i = 0; i < kRun; ++i) {
      at[i] = __shfl_sync(0xffffffffu, mine, i);
      piece(p.k_pool + (at[i] < 0 ? 0 : at[i]) * D + lane * E, k[i]);
    }
#pragma unroll
    for (int i = 0; i < kRun; ++i) piece(p.v_pool + (at[i] < 0 ? 0 : at[i]) * D + lane * E, v[i]);
    mine = lookup(j0 + step);
#pragma unroll
    for (int i = 0; i < kRun; ++i)
      if (at[i] < 0)
#pragma unroll
        for (int e = 0; e < E; ++e) v[i][e] = 0.f;         // another row's value may be infinite
    float sc[kRun * GT];
#pragma unroll
    for (int h = 0; h < GT; ++h)
#pragma unroll
      for (int i = 0; i < kRun; ++i) {
        float a = 0.f;
#pragma unroll
        for (int e = 0; e < E; ++e) a = fmaf(q[h][e], k[i][e], a);
        sc[h * kRun + i] = a;
      }
    warp_sum_scatter<kRun * GT, 16>(sc, lane);
#pragma unroll
    for (int h = 0; h < GT; ++h) {
      float w[kRun], top = -INFINITY;
#pragma unroll
      for (int i = 0; i < kRun; ++i) {
        w[i] = __shfl_sync(0xffffffffu, sc[0], (h * kRun + i) * (32 / (kRun * GT))) * p.scale;
        if (at[i] < 0) w[i] = -INFINITY;
        top = fmaxf(top, w[i]);
      }
      const float m_new = fmaxf(m_run[h], top);
      const float base = m_new == -INFINITY ? 0.f : m_new;
      const float alpha = expf(m_run[h] - base);
      m_run[h] = m_new;
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < kRun; ++i) {
        w[i] = expf(w[i] - base);
        sum += w[i];
      }
      l_run[h] = l_run[h] * alpha + sum;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        float a = acc[h][e] * alpha;
#pragma unroll
        for (int i = 0; i < kRun; ++i) a = fmaf(w[i], v[i][e], a);
        acc[h][e] = a;
      }
    }
  }
#pragma unroll
  for (int h = 0; h < GT; ++h) {
    if (lane == 0) {
      m_s[warp][h] = m_run[h];
      l_s[warp][h] = l_run[h];
    }
#pragma unroll
    for (int e = 0; e < E; ++e) o_s[warp][h][lane * E + e] = acc[h][e];
  }
  __syncthreads();
  // The block's warps become one: thread tid owns elements tid, tid + 128, .. of the heads' outputs and leaves them in warp 0's place
  // (nobody else reads those elements; the maxima and sums go to a place of their own).
  for (int i = tid; i < GT * D; i += kWarps * 32) {
    const int h = i / D, c = i % D;
    float top = -INFINITY, l = 0.f, o = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) top = fmaxf(top, m_s[w][h]);
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      if (m_s[w][h] == -INFINITY) continue;
      const float f = expf(m_s[w][h] - top);
      l += f * l_s[w][h];
      o += f * o_s[w][h][c];
    }
    o_s[0][h][c] = o;
    if (c == 0) {
      m_b[h] = top;
      l_b[h] = l;
    }
    if (splits == 1 && h < heads)
      p.out[(size_t)row * p.out_stride + (size_t)(kvh * g + h0 + h) * D + c] = l > 0.f ? o / l : 0.f;
  }
  if (splits == 1) return;
  cluster_sync_all();
  const uint32_t m_at = (uint32_t)__cvta_generic_to_shared(m_b), l_at = (uint32_t)__cvta_generic_to_shared(l_b),
                 o_at = (uint32_t)__cvta_generic_to_shared(&o_s[0][0][0]);
  // The cluster's threads share out the heads' elements; a thread's loads from the other blocks are in flight together.
  for (int i = rank * kWarps * 32 + tid; i < heads * D; i += splits * kWarps * 32) {
    const int h = i / D, c = i % D;
    float m[kMostSplits], l[kMostSplits], o[kMostSplits], top = -INFINITY, sum = 0.f, out = 0.f;
#pragma unroll
    for (int r = 0; r < kMostSplits; ++r) {
      if (r < splits) {
        m[r] = cluster_ld_f32(cluster_map(m_at + h * 4, r));
        l[r] = cluster_ld_f32(cluster_map(l_at + h * 4, r));
        o[r] = cluster_ld_f32(cluster_map(o_at + (h * D + c) * 4, r));
      }
    }
#pragma unroll
    for (int r = 0; r < kMostSplits; ++r)
      if (r < splits) top = fmaxf(top, m[r]);
#pragma unroll
    for (int r = 0; r < kMostSplits; ++r) {
      if (r >= splits || m[r] == -INFINITY) continue;
      const float f = expf(m[r] - top);
      sum += f * l[r];
      out += f * o[r];
    }
    p.out[(size_t)row * p.out_stride + (size_t)(kvh * g + h0 + h) * D + c] = sum > 0.f ? out / sum : 0.f;
  }
  cluster_sync_all();                      // a block's sums stay until everyone has read them
}

template <int D>
int launch_prompt(const Params& p, int n_seqs, int max_q_len, cudaStream_t stream) {
  static const cudaError_t ready = cudaFuncSetAttribute(attention_f32_prompt_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                        (int)PromptShape<D>::kSmem);
  if (ready != cudaSuccess) return (int)ready;
  const long long tiles = ((long long)max_q_len * (p.n_q / p.n_kv) + kRowsQ - 1) / kRowsQ;
  if (tiles > 0x7fffffff) return kRefusedSize;
  return launch_kernel(attention_f32_prompt_kernel<D>, dim3((unsigned)tiles, p.n_kv, n_seqs), dim3(256), PromptShape<D>::kSmem,
                       stream, p);
}

template <int D, int GT>
int launch_decode(const Params& p, int n_seqs, int max_ctx, cudaStream_t stream) {
  const int groups = (p.n_q / p.n_kv + GT - 1) / GT;
  if ((long long)p.n_kv * groups > 65535) return kRefusedSize;
  // Splits until two blocks an SM are there, while every warp of a split has two runs of its own.
  int splits = 1;
  const long long blocks = (long long)n_seqs * p.n_kv * groups;
  while (splits < kMostSplits && blocks * splits < 2 * 148 && max_ctx > splits * kWarps * 16) splits *= 2;
  const dim3 grid(splits, p.n_kv * groups, n_seqs);
  if (splits == 1)
    return launch_kernel(attention_f32_decode_kernel<D, GT>, grid, dim3(kWarps * 32), 0, stream, p, groups, 1);
  return launch_kernel_cluster(attention_f32_decode_kernel<D, GT>, grid, dim3(kWarps * 32), 0, stream, dim3(splits, 1, 1), p,
                               groups, splits);
}

}  // namespace attn32
}  // namespace leone

using namespace leone;

// Rows of q_start[s] .. q_start[s + 1] are sequence s's tokens, the last of them at position ctx_len[s] - 1.  `max_q_len` 1:
// the decode form.  q rows and `out` start on 16 bytes, strides are multiples of 4 floats.
extern "C" int leone_attention_f32(const float* qkv, int row_stride, float* out, int out_stride, const float* k_pool,
                                   const float* v_pool, const int* block_table, int table_width, const int* q_start,
                                   const int* ctx_len, int n_seqs, int max_q_len, int max_ctx, int n_q, int n_kv, int d,
                                   float scale, int window, int page_tokens, int num_pages, int* status,
                                   cudaStream_t stream) {
  if (n_seqs <= 0) return 0;
  if (n_q <= 0 || n_kv <= 0 || n_q % n_kv != 0 || n_kv > 65535 || n_seqs > 65535 || page_tokens <= 0 || table_width <= 0 ||
      max_q_len <= 0 || (d != 64 && d != 128))
    return kRefusedSize;
  if (row_stride % 4 != 0 || out_stride % 4 != 0 || (uintptr_t)qkv % 16 != 0 || (uintptr_t)out % 16 != 0 ||
      (uintptr_t)k_pool % 16 != 0 || (uintptr_t)v_pool % 16 != 0)
    return kRefusedAlignment;
  const attn32::Params p = {qkv, row_stride, out, out_stride, k_pool, v_pool, block_table, table_width, q_start, ctx_len,
                            n_q, n_kv, scale, window, page_tokens, num_pages, status};
  if (max_q_len > 1)
    return d == 64 ? attn32::launch_prompt<64>(p, n_seqs, max_q_len, stream) : attn32::launch_prompt<128>(p, n_seqs, max_q_len, stream);
  const int g = n_q / n_kv;
#define DECODE(GT) \
  (d == 64 ? attn32::launch_decode<64, GT>(p, n_seqs, max_ctx, stream) : attn32::launch_decode<128, GT>(p, n_seqs, max_ctx, stream))
  if (g == 1) return DECODE(1);
  if (g == 2) return DECODE(2);
  if (g <= 4) return DECODE(4);
  return DECODE(8);
#undef DECODE
}
