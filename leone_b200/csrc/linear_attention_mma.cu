// Linear attention with a decaying state (linear_attention.cu) for prompt portions in bfloat16 runs: 64 tokens at a
// time as matrix products on tensor cores (mma.sync m16n8k16).
//
// With d the head's decay, S the state before 64 tokens and q, k, v the silu of their projections (fp32):
//
//   o_t = d^(t+1) S^T q_t + sum_{s <= t} d^(t-s) (q_t . k_s) v_s        S' = d^64 S + sum_s k_s (d^(63-s) v_s)^T
//
// Every fp32 operand (q, k, v, the state, the weighted scores and values) enters as two bfloat16 terms, hi + lo (2^-17 of it,
// where the projections in front of it are rounded to 2^-9), and a product of two is three MMAs: hi hi, hi lo, lo hi.  Sums
// and the state stay fp32; the powers of d are products of fp32 factors, as in the walk, so nothing is a quotient of decays.
//
// Why: the walk is bound by instructions of the CUDA cores (two multiply-adds per state element and token, once more for
// the chunks' contributions); as products the same work is 20 times fewer instructions, and loading, silu and splitting a
// tile's operands (shared by its 64 tokens) is about half of what is left.  A block owns (64 value columns, head, chunk of
// tokens); two blocks an SM hide each other's loads, since 106 KB of operands leave no room for a second tile.  Warp w keeps
// rows 16 w .. 16 w + 15 of S^T as accumulator fragments, which are at the same time the A operand of the read-out; of the
// scores it forms tokens 16 w .. 16 w + 15.  Long portions run chunk-parallel: contributions per chunk (the same kernel
// without outputs, from a zero state), the pass over the chunks that gated linear attention has, outputs per chunk.
// Measured (2,048 tokens, 16 heads of 128 x 128, chunks of 128): contributions 25 us, pass 7, outputs 66, together 98 us; the walk, in
// chunks of 64, 344 us.
#include "gla_parts.cuh"
#include "mma_tile.cuh"

namespace leone {

constexpr int kLmTokens = 64, kLmThreads = 128, kLmCols = 64;
constexpr int kLmPV = kLmCols + 8, kLmPA = kLmTokens + 8;              // bfloat16 per row of v and of the scores

struct LinAttnParams {
  const __nv_bfloat16* proj;   // [n_tokens, ld]: projections of q, k (heads x dim each) and v (heads x vdim)
  int ld, q_off, k_off, v_off;
  float* out;                  // fp32 [n_tokens, ldo], head h at columns h * vdim
  int ldo;
  float* state;                // [n_slots, heads, dim, vdim]
  const int* q_start;
  const int* slot_ids;
  const float* decay;          // [heads]
  int n_seqs, heads, dim, vdim, n_slots, chunk;
  float* chunk_state;          // [chunks, heads, dim, vdim]
  float* chunk_decay;          // [chunks, heads, dim], equal along dim
  int* status;
};

template <int KD, bool OUT> struct LmLayout {
  static constexpr int PD = KD * 16 + 8;                               // bfloat16 per row of q and k
  static constexpr int kK = kLmTokens * PD, kV = kLmTokens * kLmPV, kA = kLmTokens * kLmPA;   // elements of one term
  static constexpr size_t bytes = 2 * (size_t)(2 * ((OUT ? 2 : 1) * kK + kV + (OUT ? kA : 0))) + sizeof(float) * (kLmTokens + 4);
};

__device__ __forceinline__ float silu_split(float z) { return __fdividef(z, 1.f + __expf(-z)); }

// 8 projections to the silu's two terms.
__device__ __forceinline__ void silu_terms(uint4 raw, __nv_bfloat16* hi, __nv_bfloat16* lo) {
  const uint32_t in[4] = {raw.x, raw.y, raw.z, raw.w};
  uint32_t h[4], l[4];
#pragma unroll
  for (int e = 0; e < 4; ++e)
    split_pair(silu_split(__uint_as_float(in[e] << 16)), silu_split(__uint_as_float(in[e] & 0xffff0000u)), h[e], l[e]);
  *reinterpret_cast<uint4*>(hi) = make_uint4(h[0], h[1], h[2], h[3]);
  *reinterpret_cast<uint4*>(lo) = make_uint4(l[0], l[1], l[2], l[3]);
}

template <int KD, bool OUT>
__global__ void __launch_bounds__(kLmThreads, 2)
linear_attention_mma_kernel(const LinAttnParams p) {
  pdl_trigger();
  pdl_wait();
  using L = LmLayout<KD, OUT>;
  constexpr int PD = L::PD, NT = 2 * KD;
  constexpr uint32_t kLoK = L::kK * 2, kLoV = L::kV * 2, kLoA = L::kA * 2;   // bytes from a hi term to its lo term
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __nv_bfloat16* k_s = reinterpret_cast<__nv_bfloat16*>(smem_raw);
  __nv_bfloat16* v_s = k_s + 2 * L::kK;
  __nv_bfloat16* q_s = v_s + 2 * L::kV;
  __nv_bfloat16* a_s = q_s + (OUT ? 2 * L::kK : 0);
  float* pow_s = reinterpret_cast<float*>(a_s + (OUT ? 2 * L::kA : 0));      // d^0 .. d^64
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, tq = lane & 3, mi = lane >> 3;
  const int dim = p.dim, vdim = p.vdim, h = blockIdx.y, v0 = blockIdx.x * kLmCols;
  GlaSpan sp;
  if (!gla_span(p, blockIdx.z, sp)) return;
  if (!OUT && sp.last) return;                     // the last chunk's contribution is never needed
  const int slot = p.slot_ids[sp.seq];
  if (slot < 0 || slot >= p.n_slots) {
    if (tid == 0) set_status(p.status, kBadSequence, sp.seq, slot);
    return;
  }
  const size_t per_head = (size_t)dim * vdim;
  float* slot_state = p.state + ((size_t)slot * p.heads + h) * per_head;
  float* mine = p.chunk > 0 ? p.chunk_state + ((size_t)blockIdx.z * p.heads + h) * per_head : slot_state;
  float* s_out = !OUT ? mine : (sp.last ? slot_state : nullptr);
  const int cols = min(kLmCols, vdim - v0);
  const bool owner = warp * 16 < cols;             // (warp-uniform) this warp holds rows of the state
  const float dec = p.decay[h];
  if (tid <= kLmTokens) {
    float f = 1.f;
    for (int i = 0; i < tid; ++i) f *= dec;
    pow_s[tid] = fminf(f, 3.0e38f);                // (a decay above one may overflow: 0 times it must stay 0)
  }
  float S[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int v = warp * 16 + g + (i >> 1) * 8, d = n * 8 + 2 * tq + (i & 1);
      S[n][i] = OUT && v < cols && d < dim ? mine[(size_t)d * vdim + v0 + v] : 0.f;
    }
  const __nv_bfloat16* k_src = p.proj + p.k_off + (size_t)h * dim;
  const __nv_bfloat16* q_src = p.proj + p.q_off + (size_t)h * dim;
  const __nv_bfloat16* v_src = p.proj + p.v_off + (size_t)h * vdim + v0;
  const uint32_t k_at = (uint32_t)__cvta_generic_to_shared(k_s), v_at = (uint32_t)__cvta_generic_to_shared(v_s),
                 q_at = (uint32_t)__cvta_generic_to_shared(q_s), a_at = (uint32_t)__cvta_generic_to_shared(a_s);
  const uint4 zero = make_uint4(0, 0, 0, 0);       // silu(0) = 0: rows and columns past the end carry nothing
  float kept = 1.f;

  for (int tb = sp.t0; tb < sp.t1; tb += kLmTokens) {
    const int nt = min(kLmTokens, sp.t1 - tb);
    __syncthreads();                               // the last tile's operands are read
#pragma unroll 4
    for (int i = tid; i < kLmTokens * 2 * KD; i += kLmThreads) {
      const int tt = i / (2 * KD), d = (i - tt * 2 * KD) * 8;
      const bool ok = tt < nt && d < dim;
      const size_t at = (size_t)(tb + (ok ? tt : 0)) * p.ld + (ok ? d : 0);
      const uint4 rk = ok ? *reinterpret_cast<const uint4*>(k_src + at) : zero;
      const uint4 rq = OUT && ok ? *reinterpret_cast<const uint4*>(q_src + at) : zero;
      silu_terms(rk, k_s + tt * PD + d, k_s + L::kK + tt * PD + d);
      if (OUT) silu_terms(rq, q_s + tt * PD + d, q_s + L::kK + tt * PD + d);
    }
#pragma unroll
    for (int i = tid; i < kLmTokens * (kLmCols / 8); i += kLmThreads) {
      const int tt = i >> 3, c = (i & 7) * 8;
      const bool ok = tt < nt && c < cols;
      silu_terms(ok ? *reinterpret_cast<const uint4*>(v_src + (size_t)(tb + tt) * p.ld + c) : zero, v_s + tt * kLmPV + c,
                 v_s + L::kV + tt * kLmPV + c);
    }
    __syncthreads();
    float Y[8][4];
    if (OUT) {
      // the scores of this warp's 16 tokens and the tokens up to them
      float G[8][4];
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) G[n][i] = 0.f;
#pragma unroll
      for (int k = 0; k < KD; ++k) {
        uint32_t qh[4], ql[4];
        const uint32_t at = q_at + ((warp * 16 + (lane & 15)) * PD + (lane >> 4) * 8 + k * 16) * 2;
        ldsm4(at, qh[0], qh[1], qh[2], qh[3]);
        ldsm4(at + kLoK, ql[0], ql[1], ql[2], ql[3]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (j <= warp) {
            uint32_t bh[4], bl[4];
            const uint32_t kt = k_at + ((j * 16 + (lane & 7) + (mi >> 1) * 8) * PD + (mi & 1) * 8 + k * 16) * 2;
            ldsm4(kt, bh[0], bh[1], bh[2], bh[3]);
            ldsm4(kt + kLoK, bl[0], bl[1], bl[2], bl[3]);
#pragma unroll
            for (int nn = 0; nn < 2; ++nn) {
              mma16816(G[2 * j + nn], ql[0], ql[1], ql[2], ql[3], bh[2 * nn], bh[2 * nn + 1]);
              mma16816(G[2 * j + nn], qh[0], qh[1], qh[2], qh[3], bl[2 * nn], bl[2 * nn + 1]);
              mma16816(G[2 * j + nn], qh[0], qh[1], qh[2], qh[3], bh[2 * nn], bh[2 * nn + 1]);
            }
          }
        }
      }
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        if ((n >> 1) <= warp) {
          const int s = n * 8 + 2 * tq;
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int t = warp * 16 + g + r * 8;
            const float u0 = s <= t ? G[n][2 * r] * pow_s[t - s] : 0.f;
            const float u1 = s + 1 <= t ? G[n][2 * r + 1] * pow_s[t - s - 1] : 0.f;
            uint32_t hi, lo;
            split_pair(u0, u1, hi, lo);
            *reinterpret_cast<uint32_t*>(a_s + t * kLmPA + s) = hi;
            *reinterpret_cast<uint32_t*>(a_s + L::kA + t * kLmPA + s) = lo;
          }
        }
      }
      // the read-out of the state before these tokens
#pragma unroll
      for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) Y[n][i] = 0.f;
      if (owner) {
#pragma unroll
        for (int k = 0; k < KD; ++k) {
          uint32_t sh[4], sl[4];
          split_pair(S[2 * k][0], S[2 * k][1], sh[0], sl[0]);
          split_pair(S[2 * k][2], S[2 * k][3], sh[1], sl[1]);
          split_pair(S[2 * k + 1][0], S[2 * k + 1][1], sh[2], sl[2]);
          split_pair(S[2 * k + 1][2], S[2 * k + 1][3], sh[3], sl[3]);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint32_t ch[4], cl[4];
            const uint32_t at = q_at + ((j * 16 + (lane & 7) + (mi >> 1) * 8) * PD + (mi & 1) * 8 + k * 16) * 2;
            ldsm4(at, ch[0], ch[1], ch[2], ch[3]);
            ldsm4(at + kLoK, cl[0], cl[1], cl[2], cl[3]);
#pragma unroll
            for (int nn = 0; nn < 2; ++nn) {
              mma16816(Y[2 * j + nn], sl[0], sl[1], sl[2], sl[3], ch[2 * nn], ch[2 * nn + 1]);
              mma16816(Y[2 * j + nn], sh[0], sh[1], sh[2], sh[3], cl[2 * nn], cl[2 * nn + 1]);
              mma16816(Y[2 * j + nn], sh[0], sh[1], sh[2], sh[3], ch[2 * nn], ch[2 * nn + 1]);
            }
          }
        }
#pragma unroll
        for (int n = 0; n < 8; ++n) {
          const float e0 = pow_s[n * 8 + 2 * tq + 1], e1 = pow_s[n * 8 + 2 * tq + 2];
          Y[n][0] *= e0;
          Y[n][1] *= e1;
          Y[n][2] *= e0;
          Y[n][3] *= e1;
        }
      }
      __syncthreads();                             // the scores are there
    }
    const float keep = pow_s[nt];
    kept *= keep;
    if (owner) {
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) S[n][i] *= keep;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t vh[4], vl[4];
        const uint32_t vt = v_at + ((k * 16 + (lane & 7) + (mi >> 1) * 8) * kLmPV + (mi & 1) * 8 + warp * 16) * 2;
        ldsm4_trans(vt, vh[0], vh[1], vh[2], vh[3]);
        ldsm4_trans(vt + kLoV, vl[0], vl[1], vl[2], vl[3]);
        if (OUT) {
#pragma unroll
          for (int j = k; j < 4; ++j) {
            uint32_t bh[4], bl[4];
            const uint32_t at = a_at + ((j * 16 + (lane & 7) + (mi >> 1) * 8) * kLmPA + (mi & 1) * 8 + k * 16) * 2;
            ldsm4(at, bh[0], bh[1], bh[2], bh[3]);
            ldsm4(at + kLoA, bl[0], bl[1], bl[2], bl[3]);
#pragma unroll
            for (int nn = 0; nn < 2; ++nn) {
              mma16816(Y[2 * j + nn], vl[0], vl[1], vl[2], vl[3], bh[2 * nn], bh[2 * nn + 1]);
              mma16816(Y[2 * j + nn], vh[0], vh[1], vh[2], vh[3], bl[2 * nn], bl[2 * nn + 1]);
              mma16816(Y[2 * j + nn], vh[0], vh[1], vh[2], vh[3], bh[2 * nn], bh[2 * nn + 1]);
            }
          }
        }
        // S^T += (w v)^T k, a token's value weighed by what is left of it after the tile's last token
        uint32_t wh[4], wl[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int s = k * 16 + (i >> 1) * 8 + 2 * tq;
          const float w0 = pow_s[max(nt - 1 - s, 0)], w1 = pow_s[max(nt - 2 - s, 0)];
          split_pair((__uint_as_float(vh[i] << 16) + __uint_as_float(vl[i] << 16)) * w0,
                     (__uint_as_float(vh[i] & 0xffff0000u) + __uint_as_float(vl[i] & 0xffff0000u)) * w1, wh[i], wl[i]);
        }
#pragma unroll
        for (int j = 0; j < KD; ++j) {
          uint32_t bh[4], bl[4];
          const uint32_t kt = k_at + ((k * 16 + (lane & 7) + (mi & 1) * 8) * PD + j * 16 + (mi >> 1) * 8) * 2;
          ldsm4_trans(kt, bh[0], bh[1], bh[2], bh[3]);
          ldsm4_trans(kt + kLoK, bl[0], bl[1], bl[2], bl[3]);
#pragma unroll
          for (int nn = 0; nn < 2; ++nn) {
            mma16816(S[2 * j + nn], wl[0], wl[1], wl[2], wl[3], bh[2 * nn], bh[2 * nn + 1]);
            mma16816(S[2 * j + nn], wh[0], wh[1], wh[2], wh[3], bl[2 * nn], bl[2 * nn + 1]);
            mma16816(S[2 * j + nn], wh[0], wh[1], wh[2], wh[3], bh[2 * nn], bh[2 * nn + 1]);
          }
        }
      }
      if (OUT) {
        float* dst = p.out + (size_t)h * vdim + v0 + warp * 16 + g;
        const bool in0 = warp * 16 + g < cols, in1 = warp * 16 + g + 8 < cols;
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int t = n * 8 + 2 * tq + i;
            if (t < nt) {
              if (in0) dst[(size_t)(tb + t) * p.ldo] = Y[n][i];
              if (in1) dst[(size_t)(tb + t) * p.ldo + 8] = Y[n][2 + i];
            }
          }
      }
    }
  }
  if (s_out != nullptr && owner) {
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int v = warp * 16 + g + (i >> 1) * 8, d = n * 8 + 2 * tq + (i & 1);
        if (v < cols && d < dim) s_out[(size_t)d * vdim + v0 + v] = S[n][i];
      }
  }
  if (!OUT && blockIdx.x == 0) {
    float* dst = p.chunk_decay + ((size_t)blockIdx.z * p.heads + h) * dim;
    for (int d = tid; d < dim; d += kLmThreads) dst[d] = fminf(kept, 3.0e38f);
  }
}

}  // namespace leone

using namespace leone;

// 1 if the tensor-core form takes these sizes (rows of 16-byte loads).
extern "C" int leone_linear_attention_mma_supported(int dim, int vdim) {
  return dim > 0 && dim <= 128 && dim % 8 == 0 && vdim > 0 && vdim % 8 == 0;
}

// The arguments of leone_linear_attention with bfloat16 proj.  chunk: a multiple of 64 with scratch chunk_state fp32 [n_chunks,
// heads, dim, vdim] and chunk_decay fp32 [n_chunks, heads, dim], or 0.  ld and the offsets must be multiples of 8.
extern "C" int leone_linear_attention_mma(const void* proj, int ld, int q_off, int k_off, int v_off, float* out, int ldo,
                                          float* state, const int* q_start, const int* slot_ids, const float* decay,
                                          int n_seqs, int heads, int dim, int vdim, int n_slots, int chunk, int n_chunks,
                                          float* chunk_state, float* chunk_decay, int* status, cudaStream_t stream) {
  if (n_seqs <= 0) return 0;
  if (!leone_linear_attention_mma_supported(dim, vdim) || heads <= 0 || heads > 65535 || n_seqs > 65535) return kRefusedSize;
  if (chunk < 0 || (chunk > 0 && (chunk % kLmTokens != 0 || n_chunks <= 0 || n_chunks > 65535 || chunk_state == nullptr ||
                                  chunk_decay == nullptr)))
    return kRefusedSize;
  if (ld % 8 || q_off % 8 || k_off % 8 || v_off % 8 || ((uintptr_t)proj & 15) ||
      (((uintptr_t)state | (uintptr_t)chunk_state) & 15))
    return kRefusedAlignment;
  LinAttnParams p = {(const __nv_bfloat16*)proj, ld, q_off, k_off, v_off, out, ldo, state, q_start, slot_ids, decay, n_seqs,
                     heads, dim, vdim, n_slots, chunk, chunk_state, chunk_decay, status};
  const int slices = (vdim + kLmCols - 1) / kLmCols, grid_z = chunk > 0 ? n_chunks : n_seqs;
  int code = 0;
#define RUN(KD, OUT)                                                                                                       \
  do {                                                                                                                     \
    constexpr size_t smem = LmLayout<KD, OUT>::bytes;                                                                      \
    static const cudaError_t ready = cudaFuncSetAttribute(linear_attention_mma_kernel<KD, OUT>,                            \
                                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);         \
    if (ready != cudaSuccess) return (int)ready;                                                                           \
    code = launch_kernel(linear_attention_mma_kernel<KD, OUT>, dim3(slices, heads, grid_z), dim3(kLmThreads), smem, stream, p); \
  } while (0)
#define RUN_D(OUT)                     \
  do {                                 \
    if (dim <= 32) RUN(2, OUT);        \
    else if (dim <= 64) RUN(4, OUT);   \
    else if (dim <= 96) RUN(6, OUT);   \
    else RUN(8, OUT);                  \
  } while (0)
  if (chunk > 0) {
    RUN_D(false);
    if (code != 0) return code;
    GlaParams pass = {};
    pass.state = state;
    pass.q_start = q_start;
    pass.slot_ids = slot_ids;
    pass.heads = heads;
    pass.dim = dim;
    pass.vdim = vdim;
    pass.chunk = chunk;
    pass.n_seqs = n_seqs;
    pass.n_slots = n_slots;
    pass.chunk_state = chunk_state;
    pass.chunk_decay = chunk_decay;
    code = launch_gla_prefix(pass, stream);
    if (code != 0) return code;
  }
  RUN_D(true);
#undef RUN_D
#undef RUN
  return code;
}
