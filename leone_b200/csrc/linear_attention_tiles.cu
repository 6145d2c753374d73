// Linear attention with a decaying state (linear_attention.cu) for prompt portions in bfloat16 runs: 64 tokens at a
// time as matrix products, every operand and sum in fp32 (packed FMA).
//
// With d the head's decay, S the state before a chunk of n <= 64 tokens and q, k, v the silu of their projections:
//
//   o_t = d^(t+1) S^T q_t + sum_{s <= t} d^(t-s) (q_t . k_s) v_s        S' = d^n S + sum_s k_s (d^(n-1-s) v_s)^T
//
// Four passes: (1) every chunk that another follows sums its own k v^T; (2) a pass over a sequence's chunks turns
// these into the states that chunks start from; (3) outputs per chunk; (4) the state after the last chunk, to the slot.
// A step of portions of one chunk is (3) and (4).  A chunk's products are in no other sequence's, sums run in the order of the
// tokens or channels, and products of a token with later ones are left out, not multiplied by zero: an infinite value
// of a later token does not reach an earlier one.  The powers of d are products in fp64, rounded once.
//
// Why fp32: tensor cores take q, k, v and the state as sums of short terms.  Two bfloat16 terms (2^-17 of an operand) were further
// from 64 bits than the walk (outputs 1.5e-6 to 5e-6 in the 2-norm; the walk 0.8e-7 at 60 tokens to 4.9e-7 at 2,048, this 0.8e-7
// to 1.9e-7; states 1.5e-6 to 5e-6, 1.3e-7 to 5.0e-7, 0.8e-7 to 1.6e-7), and an infinity has no such terms.
// Bound by the FMA pipes and by latency: (3) is 1.6 M multiply-adds a chunk and head of 128 x 128 where the walk takes 2.1 M, one
// after another; (1) 1.0 M.  A block is 256 threads with 8 x 8 outputs each, in (3) of half of the sums, two blocks an SM; the
// state comes through shared memory in slabs of 8 channels, two slabs ahead.
// Measured (16 heads of 128 x 128): 2,048 tokens 131 us ((1) 39, (2) 11, (3) 72, (4) 15; the walk, in chunks of 64, 349), 500 tokens 53
// (140), 77 tokens 47 (89), 16 sequences of 200 tokens 215 (545).
#include "common.cuh"

namespace leone {

constexpr int kLtTokens = 64, kLtThreads = 256, kLtMostDim = 128;
constexpr int kLtPitch = kLtMostDim + 4;           // floats of a row of q and k: 8 neighbouring rows' 16-byte pieces cover all banks
constexpr int kLtPitchA = kLtTokens + 4;           // of a row of the weighted scores
constexpr int kLtSlab = 8, kLtSlabs = 3;           // channels of the state in a slab, slabs in shared memory

struct LinTileParams {
  const __nv_bfloat16* proj;   // [n_tokens, ld]: projections of q, k (heads x dim each) and v (heads x vdim)
  int ld, q_off, k_off, v_off;
  float* out;                  // fp32 [n_tokens, ldo], head h at columns h * vdim
  int ldo;
  float* state;                // [n_slots, heads, dim, vdim]
  const int* q_start;
  const int* slot_ids;
  const float* decay;          // [heads]
  int n_seqs, heads, dim, vdim, n_slots;
  float* chunk_state;          // [entries, heads, dim, vdim]: one for every chunk but a sequence's first
  int* status;
};

// The sequence and chunk of number z: its tokens, and its place among the chunks that have an entry of chunk_state.
struct LinChunk { int seq, t0, n, first, last, entry; };

// Called by whole warps: 32 sequences at a time.
__device__ __forceinline__ bool find_chunk(const LinTileParams& p, int z, LinChunk& c) {
  const int lane = threadIdx.x & 31;
  int chunks_before = 0, entries_before = 0;
  for (int b0 = 0; b0 < p.n_seqs; b0 += 32) {
    const int b = b0 + lane;
    const int from = b < p.n_seqs ? p.q_start[b] : 0, to = b < p.n_seqs ? p.q_start[b + 1] : 0;
    const int mine = (to - from + kLtTokens - 1) / kLtTokens, entries = max(mine - 1, 0);
    int upto = mine, entries_upto = entries;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, upto, o), y = __shfl_up_sync(0xffffffffu, entries_upto, o);
      if (lane >= o) {
        upto += x;
        entries_upto += y;
      }
    }
    const unsigned there = __ballot_sync(0xffffffffu, z < chunks_before + upto);
    if (there != 0) {
      const int at = __ffs(there) - 1;
      const int chunk = z - (chunks_before + __shfl_sync(0xffffffffu, upto - mine, at));
      const int end = __shfl_sync(0xffffffffu, to, at);
      c.seq = b0 + at;
      c.t0 = __shfl_sync(0xffffffffu, from, at) + chunk * kLtTokens;
      c.n = min(kLtTokens, end - c.t0);
      c.first = chunk == 0;
      c.last = c.t0 + c.n == end;
      c.entry = entries_before + __shfl_sync(0xffffffffu, entries_upto - entries, at) + chunk - 1;    // (the first chunk has none)
      return true;
    }
    chunks_before += __shfl_sync(0xffffffffu, upto, 31);
    entries_before += __shfl_sync(0xffffffffu, entries_upto, 31);
  }
  return false;
}

__device__ __forceinline__ void fma2(float2& acc, float2 a, float2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(reinterpret_cast<unsigned long long&>(acc))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
}
// d^n, rounded once; a decay above one may overflow: 0 times it must stay 0.
__device__ __forceinline__ float power(float d, int n) {
  double f = 1.0, b = (double)d;
  for (; n > 0; n >>= 1, b *= b)
    if (n & 1) f *= b;
  return (float)fmin(f, 3.0e38);
}
// The silu of 8 projections, times w.
__device__ __forceinline__ void silu8(uint4 raw, float* dst, float w = 1.f) {
  const uint32_t in[4] = {raw.x, raw.y, raw.z, raw.w};
  float v[8];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    v[2 * e] = silu_branchless(__uint_as_float(in[e] << 16)) * w;
    v[2 * e + 1] = silu_branchless(__uint_as_float(in[e] & 0xffff0000u)) * w;
  }
  *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
  *reinterpret_cast<float4*>(dst + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
__device__ __forceinline__ float2 twice(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 lower(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 upper(const float4& v) { return make_float2(v.z, v.w); }

// (1) and (4): k v^T of a chunk's tokens.  FINAL: of every sequence's last chunk, on top of the state that it starts from.  A thread
// owns 4 * DH channels (4 ty .. and 64 + 4 ty ..) times 4 * VH columns; blockIdx.z counts (slice of columns, slice of channels).
template <int DH, int VH, bool FINAL>
__global__ void __launch_bounds__(kLtThreads, 2)
linear_attention_update_kernel(const LinTileParams p) {
  pdl_trigger();
  pdl_wait();
  constexpr int D = 64 * DH, V = 64 * VH;
  extern __shared__ __align__(16) float smem[];
  float* k_s = smem;                               // [kLtTokens][D]
  float* v_s = k_s + kLtTokens * D;                // [kLtTokens][V], weighted
  float* pow_s = v_s + kLtTokens * V;              // d^0 .. d^64
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int dim = p.dim, vdim = p.vdim, d_slices = (dim + D - 1) / D;
  const int h = blockIdx.y, v0 = (blockIdx.z / d_slices) * V, d0 = (blockIdx.z % d_slices) * D;
  LinChunk c;
  if (!find_chunk(p, blockIdx.x, c) || c.last != (FINAL ? 1 : 0)) return;
  const int slot = p.slot_ids[c.seq];
  if (slot < 0 || slot >= p.n_slots) return;       // (reported with the outputs)
  if (tid <= kLtTokens) pow_s[tid] = power(p.decay[h], tid);
  __syncthreads();
  const __nv_bfloat16* k_src = p.proj + (size_t)c.t0 * p.ld + p.k_off + (size_t)h * dim + d0;
  const __nv_bfloat16* v_src = p.proj + (size_t)c.t0 * p.ld + p.v_off + (size_t)h * vdim + v0;
  const int cols = min(V, vdim - v0);
  const uint4 zero = make_uint4(0, 0, 0, 0);       // silu(0) = 0
#pragma unroll 4
  for (int i = tid; i < c.n * (D / 8); i += kLtThreads) {
    const int t = i / (D / 8), d = (i % (D / 8)) * 8;
    silu8(d0 + d < dim ? *reinterpret_cast<const uint4*>(k_src + (size_t)t * p.ld + d) : zero, k_s + t * D + d);
  }
#pragma unroll 4
  for (int i = tid; i < c.n * (V / 8); i += kLtThreads) {
    const int t = i / (V / 8), v = (i % (V / 8)) * 8;
    silu8(v < cols ? *reinterpret_cast<const uint4*>(v_src + (size_t)t * p.ld + v) : zero, v_s + t * V + v, pow_s[c.n - 1 - t]);
  }
  __syncthreads();
  float2 acc[4 * DH][2 * VH];
#pragma unroll
  for (int i = 0; i < 4 * DH; ++i)
#pragma unroll
    for (int j = 0; j < 2 * VH; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll 4
  for (int t = 0; t < c.n; ++t) {
    float4 k[DH], v[VH];
#pragma unroll
    for (int a = 0; a < DH; ++a) k[a] = *reinterpret_cast<const float4*>(k_s + t * D + 64 * a + 4 * ty);
#pragma unroll
    for (int a = 0; a < VH; ++a) v[a] = *reinterpret_cast<const float4*>(v_s + t * V + 64 * a + 4 * tx);
#pragma unroll
    for (int a = 0; a < DH; ++a) {
      const float kk[4] = {k[a].x, k[a].y, k[a].z, k[a].w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int b = 0; b < VH; ++b) {
          fma2(acc[4 * a + i][2 * b], twice(kk[i]), lower(v[b]));
          fma2(acc[4 * a + i][2 * b + 1], twice(kk[i]), upper(v[b]));
        }
    }
  }
  const size_t per_head = (size_t)dim * vdim;
  float* slot_state = p.state + ((size_t)slot * p.heads + h) * per_head;
  // a chunk's own sum stands where the state that it leads to will
  float* to = FINAL ? slot_state : p.chunk_state + ((size_t)(c.entry + 1) * p.heads + h) * per_head;
  const float* from = !FINAL ? nullptr : c.first ? slot_state : p.chunk_state + ((size_t)c.entry * p.heads + h) * per_head;
  const float keep = pow_s[c.n];
#pragma unroll
  for (int i = 0; i < 4 * DH; ++i) {
    const int d = d0 + 64 * (i / 4) + 4 * ty + i % 4;
    if (d >= dim) continue;
#pragma unroll
    for (int b = 0; b < VH; ++b) {
      const int v = 64 * b + 4 * tx;
      if (v >= cols) continue;
      const size_t at = (size_t)d * vdim + v0 + v;
      float4 s = make_float4(acc[i][2 * b].x, acc[i][2 * b].y, acc[i][2 * b + 1].x, acc[i][2 * b + 1].y);
      if (FINAL) {
        const float4 old = *reinterpret_cast<const float4*>(from + at);
        s = make_float4(fmaf(keep, old.x, s.x), fmaf(keep, old.y, s.y), fmaf(keep, old.z, s.z), fmaf(keep, old.w, s.w));
      }
      *reinterpret_cast<float4*>(to + at) = s;
    }
  }
}

// (2): a thread per 4 elements of a sequence's state walks the entries of its chunks.
__global__ void __launch_bounds__(256)
linear_attention_states_kernel(const LinTileParams p) {
  pdl_trigger();
  pdl_wait();
  constexpr int kAhead = 8;
  __shared__ int first_s;
  const int s = blockIdx.y, lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    int before = 0;
    for (int b = lane; b < s; b += 32) before += max((p.q_start[b + 1] - p.q_start[b] + kLtTokens - 1) / kLtTokens - 1, 0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if (lane == 0) first_s = before;
  }
  __syncthreads();
  const int entries = (p.q_start[s + 1] - p.q_start[s] + kLtTokens - 1) / kLtTokens - 1;
  const int slot = p.slot_ids[s];
  const size_t per_seq = (size_t)p.heads * p.dim * p.vdim;
  const size_t e = ((size_t)blockIdx.x * 256 + threadIdx.x) * 4;
  if (entries <= 0 || slot < 0 || slot >= p.n_slots || e >= per_seq) return;
  const float f = power(p.decay[e / ((size_t)p.dim * p.vdim)], kLtTokens);
  float4 run = *reinterpret_cast<const float4*>(p.state + (size_t)slot * per_seq + e);
  float* at = p.chunk_state + (size_t)first_s * per_seq + e;
  for (int c0 = 0; c0 < entries; c0 += kAhead) {
    float4 own[kAhead];
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
      if (c0 + i < entries) own[i] = *reinterpret_cast<const float4*>(at + (size_t)(c0 + i) * per_seq);
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
      if (c0 + i < entries) {
        run = make_float4(fmaf(f, run.x, own[i].x), fmaf(f, run.y, own[i].y), fmaf(f, run.z, own[i].z), fmaf(f, run.w, own[i].w));
        *reinterpret_cast<float4*>(at + (size_t)(c0 + i) * per_seq) = run;
      }
  }
}

// (3): two groups of 128 threads; a thread owns tokens ty, 8 + ty, .. 56 + ty times 4 * VH columns, of every other four channels and
// tokens that are summed, so every warp has the same share of the tokens' triangle and no sum is a chain of more than
// 96 (the walk's are of 16 channels); the groups' halves meet in shared memory.  (Chains of 192 were 1.2e-7 to 2.5e-7 from 64 bits,
// in the same time.)
template <int VH> struct LinOutLayout {
  static constexpr int V = 64 * VH;
  static constexpr int kFloats = 2 * kLtTokens * kLtPitch + kLtTokens * V + kLtSlabs * kLtSlab * V + kLtTokens + 4;
};
static_assert(kLtTokens * kLtPitchA <= kLtTokens * kLtPitch, "the scores fit where the keys were");

template <int VH>
__global__ void __launch_bounds__(kLtThreads, 2)
linear_attention_outputs_kernel(const LinTileParams p) {
  pdl_trigger();
  pdl_wait();
  constexpr int V = 64 * VH;
  extern __shared__ __align__(16) float smem[];
  float* q_s = smem;                               // [kLtTokens][kLtPitch]
  float* k_s = q_s + kLtTokens * kLtPitch;         // the same; later the weighted scores, [kLtTokens][kLtPitchA]
  float* v_s = k_s + kLtTokens * kLtPitch;         // [kLtTokens][V]
  float* s_s = v_s + kLtTokens * V;                // [kLtSlabs][kLtSlab][V]
  float* pow_s = s_s + kLtSlabs * kLtSlab * V;     // d^0 .. d^64
  const int tid = threadIdx.x, tx = tid & 15, group = tid >> 7, ty = tid >> 4 & 7;
  const int h = blockIdx.y, v0 = blockIdx.z * V, dim = p.dim, vdim = p.vdim;
  LinChunk c;
  if (!find_chunk(p, blockIdx.x, c)) return;
  const int slot = p.slot_ids[c.seq];
  if (slot < 0 || slot >= p.n_slots) {
    if (tid == 0) set_status(p.status, kBadSequence, c.seq, slot);
    return;
  }
  const int cols = min(V, vdim - v0), nt = c.n;
  const size_t per_head = (size_t)dim * vdim;
  const float* s_src = (c.first ? p.state + ((size_t)slot * p.heads + h) * per_head
                                : p.chunk_state + ((size_t)c.entry * p.heads + h) * per_head) + v0;
  const uint32_t s_at = (uint32_t)__cvta_generic_to_shared(s_s);
  auto request = [&](int slab) {
    if (slab * kLtSlab < dim)
      for (int i = tid; i < kLtSlab * V / 4; i += kLtThreads) {
        const int d = i / (V / 4), v = (i % (V / 4)) * 4;
        const int bytes = v < cols ? 16 : 0;       // 0: zeros, the source is not read
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s_at + (uint32_t)(((slab % kLtSlabs) * kLtSlab + d) * V + v) * 4),
                     "l"(bytes ? s_src + (size_t)(slab * kLtSlab + d) * vdim + v : s_src), "r"(bytes) : "memory");
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int s = 0; s < kLtSlabs - 1; ++s) request(s);
  if (tid <= kLtTokens) pow_s[tid] = power(p.decay[h], tid);
  const __nv_bfloat16* q_src = p.proj + (size_t)c.t0 * p.ld + p.q_off + (size_t)h * dim;
  const __nv_bfloat16* k_src = p.proj + (size_t)c.t0 * p.ld + p.k_off + (size_t)h * dim;
  const __nv_bfloat16* v_src = p.proj + (size_t)c.t0 * p.ld + p.v_off + (size_t)h * vdim + v0;
  const uint4 zero = make_uint4(0, 0, 0, 0);       // silu(0) = 0: rows past the chunk's tokens are not stored
  const int pieces = dim / 8;
#pragma unroll 4
  for (int i = tid; i < kLtTokens * pieces; i += kLtThreads) {
    const int t = i / pieces, d = (i - t * pieces) * 8;
    const uint4 rq = t < nt ? *reinterpret_cast<const uint4*>(q_src + (size_t)t * p.ld + d) : zero;
    const uint4 rk = t < nt ? *reinterpret_cast<const uint4*>(k_src + (size_t)t * p.ld + d) : zero;
    silu8(rq, q_s + t * kLtPitch + d);
    silu8(rk, k_s + t * kLtPitch + d);
  }
#pragma unroll 4
  for (int i = tid; i < kLtTokens * (V / 8); i += kLtThreads) {
    const int t = i / (V / 8), v = (i % (V / 8)) * 8;
    silu8(t < nt && v < cols ? *reinterpret_cast<const uint4*>(v_src + (size_t)t * p.ld + v) : zero, v_s + t * V + v);
  }
  __syncthreads();
  {
    // scores of tokens row + 16 i with tokens tx + 16 j, j <= i, each in eight sums
    const int row = tid >> 4;
    float2 sc[4][4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) sc[i][j][e] = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int d = 0; d < dim; d += 8) {
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        float4 a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          a[i] = *reinterpret_cast<const float4*>(q_s + (row + 16 * i) * kLtPitch + d + 2 * e);
          b[i] = *reinterpret_cast<const float4*>(k_s + (tx + 16 * i) * kLtPitch + d + 2 * e);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j <= i; ++j) {
            fma2(sc[i][j][e], lower(a[i]), lower(b[j]));
            fma2(sc[i][j][e + 1], upper(a[i]), upper(b[j]));
          }
      }
    }
    __syncthreads();                               // the keys are read
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j) {
        const int t = row + 16 * i, s = tx + 16 * j;
        float sum[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[e] = sc[i][j][e].x + sc[i][j][e].y;
        k_s[t * kLtPitchA + s] = ((sum[0] + sum[1]) + (sum[2] + sum[3])) * pow_s[max(t - s, 0)];
      }
  }
  // the read-out of the state before these tokens: four channels of a slab a group
  float2 acc[8][2 * VH];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 2 * VH; ++j) acc[i][j] = make_float2(0.f, 0.f);
  const int slabs = dim / kLtSlab;
  for (int slab = 0; slab < slabs; ++slab) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kLtSlabs - 2) : "memory");
    __syncthreads();                               // this slab has landed, the last one's readers are done (and the scores are there)
    request(slab + kLtSlabs - 1);
    const float* rows = s_s + ((slab % kLtSlabs) * kLtSlab + 4 * group) * V;
#pragma unroll
    for (int d = 0; d < 4; d += 2) {
      float2 q[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) q[i] = *reinterpret_cast<const float2*>(q_s + (ty + 8 * i) * kLtPitch + slab * kLtSlab + 4 * group + d);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float4 s[VH];
#pragma unroll
        for (int b = 0; b < VH; ++b) s[b] = *reinterpret_cast<const float4*>(rows + (d + e) * V + 64 * b + 4 * tx);
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int b = 0; b < VH; ++b) {
            fma2(acc[i][2 * b], twice(e ? q[i].y : q[i].x), lower(s[b]));
            fma2(acc[i][2 * b + 1], twice(e ? q[i].y : q[i].x), upper(s[b]));
          }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float f = pow_s[ty + 8 * i + 1];
#pragma unroll
    for (int j = 0; j < 2 * VH; ++j) {
      acc[i][j].x *= f;
      acc[i][j].y *= f;
    }
  }
  // the chunk's own tokens up to each one: four of eight a group
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (8 * j >= nt) break;
#pragma unroll
    for (int e2 = 0; e2 < 4; e2 += 2) {
      const int s0 = 4 * group + e2;
      float2 a[8];
#pragma unroll
      for (int i = j; i < 8; ++i) a[i] = *reinterpret_cast<const float2*>(k_s + (ty + 8 * i) * kLtPitchA + 8 * j + s0);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float4 v[VH];
#pragma unroll
        for (int b = 0; b < VH; ++b) v[b] = *reinterpret_cast<const float4*>(v_s + (8 * j + s0 + e) * V + 64 * b + 4 * tx);
#pragma unroll
        for (int i = j; i < 8; ++i) {
          if (i > j || s0 + e <= ty) {
#pragma unroll
            for (int b = 0; b < VH; ++b) {
              fma2(acc[i][2 * b], twice(e ? a[i].y : a[i].x), lower(v[b]));
              fma2(acc[i][2 * b + 1], twice(e ? a[i].y : a[i].x), upper(v[b]));
            }
          }
        }
      }
    }
  }
  // each group finishes four of a thread's tokens: the other group's part of them comes through where the queries were
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if ((i < 4) == (group == 1)) {
#pragma unroll
      for (int b = 0; b < VH; ++b)
        *reinterpret_cast<float4*>(q_s + (ty + 8 * i) * kLtPitch + 64 * b + 4 * tx) =
            make_float4(acc[i][2 * b].x, acc[i][2 * b].y, acc[i][2 * b + 1].x, acc[i][2 * b + 1].y);
    }
  __syncthreads();
  float* dst = p.out + (size_t)c.t0 * p.ldo + (size_t)h * vdim + v0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int t = ty + 8 * i;
    if ((i < 4) != (group == 0) || t >= nt) continue;
#pragma unroll
    for (int b = 0; b < VH; ++b)
      if (64 * b + 4 * tx < cols) {
        const float4 o = *reinterpret_cast<const float4*>(q_s + t * kLtPitch + 64 * b + 4 * tx);
        *reinterpret_cast<float4*>(dst + (size_t)t * p.ldo + 64 * b + 4 * tx) =
            make_float4(acc[i][2 * b].x + o.x, acc[i][2 * b].y + o.y, acc[i][2 * b + 1].x + o.z, acc[i][2 * b + 1].y + o.w);
      }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

}  // namespace leone

using namespace leone;

// 1 if these kernels take the sizes (rows of 16-byte loads).
extern "C" int leone_linear_attention_tiles_supported(int dim, int vdim) {
  return dim > 0 && dim <= kLtMostDim && dim % 8 == 0 && vdim > 0 && vdim % 8 == 0 && vdim <= 16384 * 64;
}

// The arguments of leone_linear_attention with bfloat16 proj.  n_chunks: the sum over sequences of ceil(tokens / 64); entries: the
// same with one less for every sequence that has tokens; chunk_state: fp32 [entries, heads, dim, vdim].  ld and the offsets
// are multiples of 8, ldo of 4.
extern "C" int leone_linear_attention_tiles(const void* proj, int ld, int q_off, int k_off, int v_off, float* out, int ldo,
                                            float* state, const int* q_start, const int* slot_ids, const float* decay,
                                            int n_seqs, int heads, int dim, int vdim, int n_slots, int n_chunks, int entries,
                                            float* chunk_state, int* status, cudaStream_t stream) {
  if (n_seqs <= 0 || n_chunks <= 0) return 0;
  if (!leone_linear_attention_tiles_supported(dim, vdim) || heads <= 0 || heads > 65535 || n_seqs > 65535 || entries < 0 ||
      (entries > 0 && chunk_state == nullptr))
    return kRefusedSize;
  if (ld % 8 || q_off % 8 || k_off % 8 || v_off % 8 || ldo % 4 ||
      (((uintptr_t)proj | (uintptr_t)out | (uintptr_t)state | (uintptr_t)chunk_state) & 15))
    return kRefusedAlignment;
  const LinTileParams p = {(const __nv_bfloat16*)proj, ld, q_off, k_off, v_off, out, ldo, state, q_start, slot_ids, decay,
                           n_seqs, heads, dim, vdim, n_slots, chunk_state, status};
  int code = 0;
#define RUN(KERNEL, FLOATS, SLICES)                                                                                         \
  do {                                                                                                                      \
    constexpr int smem = (int)sizeof(float) * (FLOATS);                                                                     \
    static const cudaError_t ready = cudaFuncSetAttribute(KERNEL, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);       \
    if (ready != cudaSuccess) return (int)ready;                                                                            \
    code = launch_kernel(KERNEL, dim3(n_chunks, heads, SLICES), dim3(kLtThreads), smem, stream, p);                         \
    if (code != 0) return code;                                                                                             \
  } while (0)
#define UPDATE(DH, VH, FINAL)                                                                                               \
  do {                                                                                                                      \
    constexpr auto kernel = linear_attention_update_kernel<DH, VH, FINAL>;                                                  \
    RUN(kernel, kLtTokens * 64 * (DH + VH) + kLtTokens + 4,                                                                 \
        ((vdim + 64 * VH - 1) / (64 * VH)) * ((dim + 64 * DH - 1) / (64 * DH)));                                            \
  } while (0)
  if (entries > 0) {
    // many chunks: a block takes a whole head of 128 x 128
    if (dim <= 64 && vdim <= 64) UPDATE(1, 1, false);
    else if (dim <= 64) UPDATE(1, 2, false);
    else if (vdim <= 64) UPDATE(2, 1, false);
    else UPDATE(2, 2, false);
    const size_t per_seq = (size_t)heads * dim * vdim;
    code = launch_kernel(linear_attention_states_kernel, dim3((unsigned)((per_seq / 4 + 255) / 256), n_seqs), dim3(256), 0, stream, p);
    if (code != 0) return code;
  }
  if (vdim <= 64) {
    constexpr auto kernel = linear_attention_outputs_kernel<1>;
    RUN(kernel, LinOutLayout<1>::kFloats, 1);
  } else {
    constexpr auto kernel = linear_attention_outputs_kernel<2>;
    RUN(kernel, LinOutLayout<2>::kFloats, (vdim + 127) / 128);
  }
  // A chunk a sequence: tiles of 64 x 64 while that makes more blocks at once, a head a block beyond (16 sequences of 64 tokens,
  // 16 heads of 128: the call 61 us against 69; one sequence of 60 tokens 48 against 32).
  if (dim > 64 && vdim > 64 && (long long)n_seqs * heads > 148) UPDATE(2, 2, true);
  else UPDATE(1, 1, true);
#undef UPDATE
#undef RUN
  return code;
}
