// C[M,N] = A[M,K] * W[N,K]^T on CUDA cores with fp32 FMA accumulation, and the choice of the 32-bit product's form.
//
// This is the matrix product of the 32-bit path for few tokens and for any size or alignment, and the any-size product
// of the bfloat16 path for shapes the tensor-core kernel refuses.  y[r] = sum_c W[r,c] x[c], weights
// row-major [out][in] (crates/leone/src/cpu.rs:1622-1640).
//
// Three forms, chosen by leone_gemm_simt from dtype, sizes and alignment:
//  * gemm_rows: 32 bits, up to 24 tokens.  A stream over the weights;
//  * gemm_f32_tc.cu: 32 bits, more tokens, K of 256 and more.  Tiles on tensor cores, operands split into two terms;
//  * gemm_simt_kernel: bfloat16, and any size or alignment (4-byte loads).
// In every form a row of C is computed from its own row of A only.  How its sum over k is grouped depends on the
// form and the split, so a token's result in another batch differs by fp32 rounding at most.
//
// Epilogues: 0 store in the input type; 1 store fp32; 2 store fp32 = acc + residual
// (residual may alias the output: each element is read then written by one thread).  bias: fp32 [N] added to
// the sums before them, or null.
#include "common.cuh"
#include "gemm_f32.h"

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

// The 32-bit product with 16-byte loads of up to 24 tokens: the stream is read again for every 8 tokens (its blocks share the
// weights through the L2), tensor cores take the same time for any part of a tile of 128.  One line for all shapes, where a layer's four
// products break even: at 24 tokens 27 / 15 / 73 / 37 us here (152) and 29 / 26 / 58 / 51 there (164; at 25) for 4,096, 2,048 and
// 12,288 rows of 2,048 and 2,048 of 6,144; the next 8 tokens cost the stream a third more.
constexpr int kStreamTokens = 24;
// From here on the tensor cores' sums are nearer to 64 bits than a chain of FMA is (2.1e-7 at any K against 2.8e-7 at 256, growing
// with its root; below, a chain is as near, and the product is small).
constexpr int kTensorCoresFrom = 256;

inline int launch_rows(const float* a, const float* w, float* c, const float* residual, const float* bias, int m, int n,
                       int k, int lda, int ldw, int ldc, cudaStream_t stream) {
#define ROWS(MT, R)                                                                                                    \
  launch_kernel(gemm_rows_kernel<MT, R>, dim3((m + MT - 1) / MT, (n + R - 1) / R), dim3(256), 0, stream, a, w, c,      \
                residual, bias, m, n, k, lda, ldw, ldc)
  if (m == 1) return ROWS(1, 4);
  if (m == 2) return ROWS(2, 4);
  if (m <= 4) return ROWS(4, 4);
  return ROWS(8, 4);
#undef ROWS
}

}  // namespace leone

using namespace leone;

extern "C" int leone_gemm_simt(int dtype, int epilogue, const void* a, const void* w, void* c,
                               const float* residual, const float* bias, int m, int n, int k, int lda,
                               int ldw, int ldc, int* status, cudaStream_t stream) {
  if (m <= 0 || n <= 0) return 0;
  if (k <= 0 || lda < k || ldw < k || ldc < n) return kRefusedSize;
  if (epilogue == 2 && residual == nullptr) return kRefusedSize;
  if (dtype == 0 && (epilogue < 0 || epilogue > 2)) return kRefusedSize;
  // 16-byte loads of both operands; anything else runs on the any-size kernel
  if (dtype == 0 && k % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (uintptr_t)a % 16 == 0 && (uintptr_t)w % 16 == 0) {
    const float *x = (const float*)a, *y = (const float*)w, *r = epilogue == 2 ? residual : nullptr;
    if (m <= kStreamTokens && n <= 65535 * 4)
      return launch_rows(x, y, (float*)c, r, bias, m, n, k, lda, ldw, ldc, stream);
    if (k >= kTensorCoresFrom) {
      const int code = gemm_f32_tc(x, y, (float*)c, r, bias, m, n, k, lda, ldw, ldc, status, stream);
      if (code >= 0) return code;          // (refused: nothing was launched)
    }
  }
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
