// C[M,N] = A[M,K] * W[N,K]^T on CUDA cores with fp32 FMA accumulation.
//
// This is the matrix product of the true 32-bit path (no tensor cores, no
// reduced-precision mode) and the any-size product of the bfloat16 path for
// shapes the tensor-core kernel refuses.  y[r] = sum_c W[r,c] x[c], weights
// row-major [out][in] (crates/leone/src/cpu.rs:1622-1640).
//
// Three forms, chosen by leone_gemm_simt from dtype, sizes and alignment:
//  * gemm_rows: 32 bits, up to 8 tokens.  A stream over the weights;
//  * gemm_tile: 32 bits, more tokens.  Tiles of 16 to 128 tokens x 128 weight rows, split along K over a
//    thread-block cluster where the tiles alone would leave SMs idle;
//  * gemm_simt_kernel: bfloat16, and any size or alignment (4-byte loads).
// In every form a row of C is computed from its own row of A only.  How its sum over k is grouped depends on the
// form and the split, so a token's result in another batch differs by fp32 rounding at most.
//
// Epilogues: 0 store in the input type; 1 store fp32; 2 store fp32 = acc + residual
// (residual may alias the output: each element is read then written by one thread).  bias: fp32 [N] added to
// the sums before them, or null.
#include "common.cuh"

namespace leone {

constexpr int BM = 64, BN = 64, BK = 16;

template <typename T, int EPI>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const T* __restrict__ A, const T* __restrict__ W, void* Cv,
                 const float* residual, const float* __restrict__ bias, int M, int N, int K, int lda, int ldw, int ldc) {
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int ty = tid >> 4, tx = tid & 15;
  const int lr = tid >> 2, lk = (tid & 3) * 4;   // loader: row within tile, first k
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  const T* a_row = A + (size_t)(m0 + lr) * lda;
  const T* w_row = W + (size_t)(n0 + lr) * ldw;
  const bool a_ok = m0 + lr < M, w_ok = n0 + lr < N;
  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = k0 + lk + i;
      As[lk + i][lr] = (a_ok && k < K) ? to_float<T>(a_row[k]) : 0.f;
      Ws[lk + i][lr] = (w_ok && k < K) ? to_float<T>(w_row[k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Ws[k][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= N) continue;
      const size_t o = (size_t)m * ldc + n;
      if (bias != nullptr) acc[i][j] += bias[n];
      if (EPI == 0) ((T*)Cv)[o] = from_float<T>(acc[i][j]);
      else if (EPI == 1) ((float*)Cv)[o] = acc[i][j];
      else ((float*)Cv)[o] = acc[i][j] + residual[o];
    }
  }
}

// ---- 32 bits, few tokens: a stream over the weights ---------------------------------------------------------
// Bound by the weights' bytes up to 4 tokens, by the loads of the tokens' rows (which come from the L1) at 8.  A block owns
// R weight rows and up to MT tokens; its 256 threads take every 256th 16-byte piece of a row, so 8 warps share a row's
// K and a row of 2,048 is two loads a thread and row, the second requested before the first is used.  The weights are not
// kept in the L1.  The sums of the 256 threads meet by halving exchanges and in shared memory, in a fixed order.  Weights of the first round are
// requested before the kernel waits for its predecessor.
// Measured (K 2,048, weights from memory): 12,288 rows at 1 / 4 / 8 tokens 16.6 / 18.7 / 27.7 us (6.1 / 5.4 / 3.6 TB/s), 2,048 rows
// of K 6,144 at 4 tokens 12 us; the any-size kernel, whose 64 x 64 tiles walk K one after another, took 204 us for the first kind
// and 308 us for the second (a decode step of 4 tokens of the 1.7B shape 31.5 ms, now 2.4).
__device__ __forceinline__ float4 ld_stream(const float* p) {
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

template <int MT, int R>
__global__ void __launch_bounds__(256, MT == 8 ? 3 : 4)
gemm_rows_kernel(const float* A, const float* __restrict__ W, float* C, const float* residual,
                 const float* __restrict__ bias, int M, int N, int K, int lda, int ldw, int ldc) {
  constexpr int V = R * MT;
  static_assert((V & (V - 1)) == 0 && V <= 64, "the exchanges halve the values");
  __shared__ float part[8][V];
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // token chunks are the fast index: the blocks that share weight rows run beside one another
  const int m0 = blockIdx.x * MT, n0 = blockIdx.y * R;
  const int pieces = K >> 2;
  const float* w_row[R];
#pragma unroll
  for (int r = 0; r < R; ++r) w_row[r] = W + (size_t)min(n0 + r, N - 1) * ldw;
  float4 w[R];
  if (tid < pieces) {
#pragma unroll
    for (int r = 0; r < R; ++r) w[r] = ld_stream(w_row[r] + 4 * tid);
  }
  float acc[V];
#pragma unroll
  for (int i = 0; i < V; ++i) acc[i] = 0.f;
  pdl_wait();
  for (int c = tid; c < pieces; c += 256) {
    float4 next[R];
    if (c + 256 < pieces) {
#pragma unroll
      for (int r = 0; r < R; ++r) next[r] = ld_stream(w_row[r] + 4 * (c + 256));
    }
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const float4 x = *(const float4*)(A + (size_t)min(m0 + m, M - 1) * lda + 4 * c);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float a = acc[r * MT + m];
        a = fmaf(w[r].x, x.x, a);
        a = fmaf(w[r].y, x.y, a);
        a = fmaf(w[r].z, x.z, a);
        acc[r * MT + m] = fmaf(w[r].w, x.w, a);
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) w[r] = next[r];
  }
  warp_sum_scatter<V, 16>(acc, lane);
  if constexpr (V > 32) {
    part[warp][lane * 2] = acc[0];
    part[warp][lane * 2 + 1] = acc[1];
  } else {
    if (lane % (32 / V) == 0) part[warp][lane / (32 / V)] = acc[0];
  }
  __syncthreads();
  if (tid < V) {
    float sum = part[0][tid];
#pragma unroll
    for (int i = 1; i < 8; ++i) sum += part[i][tid];
    const int n = n0 + tid / MT, m = m0 + tid % MT;
    if (n < N && m < M) {
      if (bias != nullptr) sum += bias[n];
      const size_t o = (size_t)m * ldc + n;
      if (residual != nullptr) sum += residual[o];
      C[o] = sum;
    }
  }
}

// ---- 32 bits, tiles ------------------------------------------------------------------------------------------
// Bound by what shared memory delivers to registers (a register of a warp a cycle and SM) and by the FMA pipes, which
// reach their rate with fma.rn.f32x2 only: scalar FMA stopped at half of it.  A thread owns 8 tokens x 8 weight rows;
// both operands lie in shared memory as they do in global memory (k contiguous, rows padded to 36 floats, so that 8
// neighbouring rows' 16-byte pieces cover all banks), brought by 16-byte cp.async.  A thread reads 4 k of a row at once and
// keeps two sums per output, over even and over odd k, which are the two halves of the packed FMA: no operand has to be
// duplicated.  (With k as the slow index and sums paired over weight rows, 8 x 16 a thread, duplicating the tokens' values
// cost more than the fewer loads saved: 36 TFLOP/s at 1,024 tokens against 42.)
// Where the tiles are fewer than the SMs, a cluster of `splits` blocks shares a tile's K: every block leaves its sums in
// its own shared memory, and each adds a share of the tile's rows over the ranks, in rank order.
// Measured (K 2,048, 509 tokens): 12,288 rows 617 us (41 TFLOP/s of about 74), 4,096 rows 207 us, 2,048 rows 115 us (two
// splits); the any-size kernel 22 TFLOP/s.
constexpr int kTileN = 128, kTileK = 32, kPitch = kTileK + 4;

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  const int bytes = valid ? 16 : 0;        // 0: the 16 bytes are filled with zeros, the source is not read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void fma2(float2& acc, float2 a, float2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(reinterpret_cast<unsigned long long&>(acc))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
}

template <int BM>
struct TileShape {
  static constexpr int kThreads = 2 * BM;                       // 16 along the weight rows, BM / 8 along the tokens
  static constexpr int kThreadsM = BM / 8;
  static constexpr int kStages = BM >= 128 ? 4 : 3;
  static constexpr int kStageFloats = (BM + kTileN) * kPitch;
  static constexpr size_t kSmem = (size_t)kStages * kStageFloats * sizeof(float);
  static_assert(kStages * kStageFloats >= BM * kTileN, "the tile's sums fit where the stages were");
};

template <int BM>
__global__ void __launch_bounds__(2 * BM, BM >= 128 ? 1 : 2)
gemm_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, float* C, const float* residual,
                 const float* __restrict__ bias, int M, int N, int K, int lda, int ldw, int ldc, int splits) {
  using S = TileShape<BM>;
  extern __shared__ __align__(16) float tile_smem[];
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = splits > 1 ? (int)cluster_ctarank() : 0;
  const int m0 = blockIdx.y * BM, n0 = (blockIdx.x / splits) * kTileN;
  const int tx = (warp & 1) * 8 + (lane & 7), ty = (warp >> 1) * 4 + (lane >> 3);   // a warp: 8 along n, 4 along m
  const int steps = (K + kTileK - 1) / kTileK;
  const int first = (int)((long long)steps * rank / splits), last = (int)((long long)steps * (rank + 1) / splits);

  const uint32_t base = (uint32_t)__cvta_generic_to_shared(tile_smem);
  // a stage: BM rows of A, then 128 rows of W, 8 pieces of 16 bytes a row
  constexpr int kRowsAtOnce = S::kThreads / 8;
  const int lr = tid >> 3, lk = (tid & 7) * 4;
  auto load_w = [&](int step, int stage) {
    const int k = step * kTileK + lk;
#pragma unroll
    for (int i = 0; i < kTileN / kRowsAtOnce; ++i) {
      const int row = lr + i * kRowsAtOnce;
      const bool ok = n0 + row < N && k < K;
      cp_async16(base + (uint32_t)(stage * S::kStageFloats + (BM + row) * kPitch + lk) * 4,
                 ok ? W + (size_t)(n0 + row) * ldw + k : W, ok);
    }
  };
  auto load_a = [&](int step, int stage) {
    const int k = step * kTileK + lk;
#pragma unroll
    for (int i = 0; i < BM / kRowsAtOnce; ++i) {
      const int row = lr + i * kRowsAtOnce;
      const bool ok = m0 + row < M && k < K;
      cp_async16(base + (uint32_t)(stage * S::kStageFloats + row * kPitch + lk) * 4,
                 ok ? A + (size_t)(m0 + row) * lda + k : A, ok);
    }
  };
  // the weights of the first stages do not depend on the kernel before this one
#pragma unroll
  for (int s = 0; s < S::kStages - 1; ++s)
    if (first + s < last) load_w(first + s, s);
  pdl_wait();
#pragma unroll
  for (int s = 0; s < S::kStages - 1; ++s) {
    if (first + s < last) load_a(first + s, s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  float2 acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = make_float2(0.f, 0.f);

  int stage = 0;
  for (int step = first; step < last; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(S::kStages - 2) : "memory");
    __syncthreads();                       // this stage has landed for everyone, and the one before it has been read
    const int ahead = step + S::kStages - 1, free_stage = stage == 0 ? S::kStages - 1 : stage - 1;
    if (ahead < last) {
      load_w(ahead, free_stage);
      load_a(ahead, free_stage);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* As = tile_smem + stage * S::kStageFloats;
    const float* Ws = As + BM * kPitch;
#pragma unroll
    for (int k = 0; k < kTileK; k += 4) {
      float4 b[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) b[j] = *(const float4*)(Ws + (tx + j * 16) * kPitch + k);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 a = *(const float4*)(As + (ty + i * S::kThreadsM) * kPitch + k);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          fma2(acc[i][j], make_float2(a.x, a.y), make_float2(b[j].x, b[j].y));
          fma2(acc[i][j], make_float2(a.z, a.w), make_float2(b[j].z, b[j].w));
        }
      }
    }
    stage = stage == S::kStages - 1 ? 0 : stage + 1;
  }

  auto finish = [&](int m, int n, float sum) {
    if (m >= M || n >= N) return;
    if (bias != nullptr) sum += bias[n];
    const size_t o = (size_t)m * ldc + n;
    if (residual != nullptr) sum += residual[o];
    C[o] = sum;
  };
  if (splits == 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) finish(m0 + ty + i * S::kThreadsM, n0 + tx + j * 16, acc[i][j].x + acc[i][j].y);
    return;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();                         // no copy and no reader is left in the stages
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) tile_smem[(ty + i * S::kThreadsM) * kTileN + tx + j * 16] = acc[i][j].x + acc[i][j].y;
  cluster_sync_all();
  for (int at = rank * S::kThreads + tid; at < BM * kTileN; at += splits * S::kThreads) {
    float sum = 0.f;
    for (int r = 0; r < splits; ++r) sum += cluster_ld_f32(cluster_map(base + at * 4, r));
    finish(m0 + at / kTileN, n0 + at % kTileN, sum);
  }
  cluster_sync_all();                      // a block's sums stay until everyone has read them
}

// How many ways a tile's K is split: until the blocks fill the places the SMs have, while a block keeps at least eight
// steps of 32 (a split costs a pass of the tile's sums through shared memory and two cluster barriers).
inline int tile_splits(long long tiles, int k, int places) {
  int splits = 1;
  while (splits < 8 && tiles * splits * 2 <= places && (k + kTileK - 1) / kTileK >= splits * 2 * 8) splits *= 2;
  return splits;
}

template <int BM>
int launch_tile(const float* a, const float* w, float* c, const float* residual, const float* bias, int m, int n, int k,
                int lda, int ldw, int ldc, cudaStream_t stream) {
  using S = TileShape<BM>;
  static const cudaError_t ready =
      cudaFuncSetAttribute(gemm_tile_kernel<BM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::kSmem);
  if (ready != cudaSuccess) return (int)ready;
  const int tiles_n = (n + kTileN - 1) / kTileN, tiles_m = (m + BM - 1) / BM;
  if (tiles_m > 65535) return kRefusedSize;
  const int splits = tile_splits((long long)tiles_n * tiles_m, k, BM >= 128 ? 148 : 2 * 148);
  const dim3 grid(tiles_n * splits, tiles_m);
  if (splits == 1)
    return launch_kernel(gemm_tile_kernel<BM>, grid, dim3(S::kThreads), S::kSmem, stream, a, w, c, residual, bias, m, n, k,
                         lda, ldw, ldc, 1);
  return launch_kernel_cluster(gemm_tile_kernel<BM>, grid, dim3(S::kThreads), S::kSmem, stream, dim3(splits, 1, 1), a, w,
                               c, residual, bias, m, n, k, lda, ldw, ldc, splits);
}

// The 32-bit product with 16-byte loads.  Up to 24 tokens the stream is faster, read again for every 8 tokens (its blocks share
// the weights through the L2): 12,288 x 2,048 at 24 tokens 73 us, the tile 118 us at 32 and still 120 us at 64; one tile of 64
// tokens up to 64, above it 128 (65 tokens 207 us against 240 in two tiles of 64).
inline int launch_f32(const float* a, const float* w, float* c, const float* residual, const float* bias, int m, int n,
                      int k, int lda, int ldw, int ldc, cudaStream_t stream) {
#define ROWS(MT, R)                                                                                                    \
  launch_kernel(gemm_rows_kernel<MT, R>, dim3((m + MT - 1) / MT, (n + R - 1) / R), dim3(256), 0, stream, a, w, c,      \
                residual, bias, m, n, k, lda, ldw, ldc)
  if (m <= 24 && n <= 65535 * 4) {
    if (m == 1) return ROWS(1, 4);
    if (m == 2) return ROWS(2, 4);
    if (m <= 4) return ROWS(4, 4);
    return ROWS(8, 4);
  }
#undef ROWS
  return m <= 64 ? launch_tile<64>(a, w, c, residual, bias, m, n, k, lda, ldw, ldc, stream)
                 : launch_tile<128>(a, w, c, residual, bias, m, n, k, lda, ldw, ldc, stream);
}

}  // namespace leone

using namespace leone;

extern "C" int leone_gemm_simt(int dtype, int epilogue, const void* a, const void* w, void* c,
                               const float* residual, const float* bias, int m, int n, int k, int lda,
                               int ldw, int ldc, cudaStream_t stream) {
  if (m <= 0 || n <= 0) return 0;
  if (k <= 0 || lda < k || ldw < k || ldc < n) return kRefusedSize;
  if (epilogue == 2 && residual == nullptr) return kRefusedSize;
  if (dtype == 0 && (epilogue < 0 || epilogue > 2)) return kRefusedSize;
  // 16-byte loads of both operands; anything else runs on the any-size kernel
  if (dtype == 0 && k % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (uintptr_t)a % 16 == 0 && (uintptr_t)w % 16 == 0)
    return launch_f32((const float*)a, (const float*)w, (float*)c, epilogue == 2 ? residual : nullptr, bias, m, n, k, lda,
                      ldw, ldc, stream);
  dim3 grid((n + BN - 1) / BN, (m + BM - 1) / BM);
  if (grid.y > 65535) return kRefusedSize;
#define LAUNCH(T, E)                                                                       \
  gemm_simt_kernel<T, E><<<grid, 256, 0, stream>>>((const T*)a, (const T*)w, c, residual, bias, m, \
                                                   n, k, lda, ldw, ldc)
  if (dtype == 0) {
    if (epilogue == 0) LAUNCH(float, 0);
    else if (epilogue == 1) LAUNCH(float, 1);
    else if (epilogue == 2) LAUNCH(float, 2);
    else return kRefusedSize;
  } else if (dtype == 1) {
    if (epilogue == 0) LAUNCH(__nv_bfloat16, 0);
    else if (epilogue == 1) LAUNCH(__nv_bfloat16, 1);
    else if (epilogue == 2) LAUNCH(__nv_bfloat16, 2);
    else return kRefusedSize;
  } else {
    return kRefusedDtype;
  }
#undef LAUNCH
  return launch_result();
}
