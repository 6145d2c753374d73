// The grouped products of the routed experts (experts.cu) on tcgen05 for steps of many pairs in bfloat16.
//
// The pairs (token, choice) are sorted by expert; a tile is 128 pairs of one expert (MMA M) times 256 weight rows (MMA N):
//   mode 0  128 rows of the gate matrix and the same 128 of the up matrix: act = silu(g) u in the epilogue
//   mode 1  256 rows of the up matrix of an ungated expert: act = max(u, 0)^2
//   mode 2  256 rows of the down matrix: the pair's row of fp32 sums, times its weight
// The tokens' rows are copied into sorted order first (12 us at 8,192 pairs of 2,048; gathering them as they are loaded, with
// cp.async.bulk.tensor tile::gather4, cost 70 us more: its 32 instructions a k-block take longer than the k-block's MMAs).
// Persistent, one block an SM, which walks tiles with the row tiles of an expert side by side, so that its weights are read
// from memory once: warp 0 loads (three stages of 16 + 32 KB), warp 1 issues tcgen05.mma, warps 2..9 finish a tile out of one
// of the two accumulators in tensor memory while the other is filled.  Every wait is bounded and reports into the
// status word.
//
// Why this split: the mma.sync form computes 64 x 64 tiles and is bound by ldmatrix and the copies from the L2 (32 KB of operands
// per 1 M multiply-adds, here 48 KB per 8 M), and the legacy tensor path has a quarter of the rate.  128 rows of pairs on
// the M side waste the rest of an expert's last tile, a quarter of the work at 256 pairs an expert.
// Measured (all launches of a layer's experts, 2,048 tokens; before: the mma.sync form): 32 experts of 512, 4 chosen, width 2,048
// 131 us (265); ungated 32 of 768 126 us (284); 64 experts of 1,024, 6 chosen, width 4,096 507 us (1,345).
#include "experts_tc.h"
#include "tc_common.cuh"

namespace leone {
namespace tc {

constexpr int kExRows = 128, kExCols = 256, kExK = 64, kExStages = 3, kExThreads = 320;
constexpr int kExRowBytes = 256, kExRowPitch = kExRowBytes + 16;       // what a thread of the epilogue stages of its row at a time
constexpr int kExStageA = kExRows * kExK * 2, kExStageB = kExCols * kExK * 2, kExStage = kExStageA + kExStageB;
constexpr int kExSmem = kExStages * kExStage + 1024 + 256 + 2 * kExRows * kExRowPitch;

struct ExpertParams {
  const int* offsets;          // [experts + 1]: sorted rows of every expert
  const int* order;            // [pairs]: sorted row -> pair
  const float* weight;         // [pairs]
  void* out;                   // modes 0, 1: bf16 [pairs, cols] by sorted row; mode 2: fp32 [pairs, cols] by pair
  int experts, top;
  int cols, K;                 // output columns (weight rows of one expert), inner size
  int scale_input, mode;
  int* status;
};

// sorted[row] = x[token of the row's pair].  (What the kernels before this one write is not declared read-only: such a load
// may be moved ahead of the wait for them.  The count of rows is the first thing read, so it would be.)
__global__ void __launch_bounds__(256)
experts_sort_rows_kernel(const __nv_bfloat16* x, int ldx, int width, int top, const int* order, const int* total,
                         __nv_bfloat16* sorted) {
  pdl_trigger();
  pdl_wait();
  const int pieces = width / 8, rows = *static_cast<const volatile int*>(total);
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)(order[r] / top) * ldx);
    uint4* dst = reinterpret_cast<uint4*>(sorted + (size_t)r * width);
    for (int i = threadIdx.x; i < pieces; i += 256) dst[i] = src[i];
  }
}

__global__ void __launch_bounds__(kExThreads, 1)
experts_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                  const __grid_constant__ CUtensorMap map_w2, const ExpertParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t tiles_base = (raw + 1023u) & ~1023u;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + (tiles_base - raw) + kExStages * kExStage);
  const uint32_t full0 = smem_u32(bars), empty0 = full0 + 8 * kExStages;
  const uint32_t acc_full0 = empty0 + 8 * kExStages, acc_empty0 = acc_full0 + 16;
  __shared__ uint32_t tmem_holder;
  __shared__ int gave_up;
  __shared__ int first_tile[kExpertsTcMost + 1];        // row tiles before every expert
  __shared__ int first_row[kExpertsTcMost + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    gave_up = 0;
    for (int s = 0; s < kExStages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full0 + 8 * b, 1);
      mbar_init(acc_empty0 + 8 * b, 8);
    }
    mbar_fence_init();
    tma_prefetch_desc(&map_x);
    tma_prefetch_desc(&map_w);
  }
  pdl_trigger();
  pdl_wait();                                          // the pairs' grouping is the kernel before this one
  for (int e = threadIdx.x; e <= p.experts; e += kExThreads) first_row[e] = p.offsets[e];
  __syncthreads();
  if (warp == 1) tmem_alloc(smem_u32(&tmem_holder), 512);
  if (warp == 0) {
    int run = 0;
    for (int e0 = 0; e0 < p.experts; e0 += 32) {
      const int e = e0 + lane;
      const int n = e < p.experts ? (first_row[e + 1] - first_row[e] + kExRows - 1) / kExRows : 0;
      int upto = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int before = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += before;
      }
      if (e < p.experts) first_tile[e] = run + upto - n;
      run += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (lane == 0) first_tile[p.experts] = run;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_holder;
  volatile int* giveup = &gave_up;
  const int cols_per_tile = p.mode == 0 ? kExCols / 2 : kExCols;
  const int n_tiles = (p.cols + cols_per_tile - 1) / cols_per_tile;
  const int total = first_tile[p.experts] * n_tiles;
  const int k_blocks = (p.K + kExK - 1) / kExK;
  // Tile t: row tiles are the fast index within an expert's columns (the same weights, back to back).
  auto locate = [&](int t, int& expert, int& row0, int& n0) {
    int lo = 0, hi = p.experts - 1;                    // the last expert whose first tile is at or before t's
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (first_tile[mid] * n_tiles <= t) lo = mid;
      else hi = mid - 1;
    }
    expert = lo;
    const int rows = first_tile[lo + 1] - first_tile[lo], in = t - first_tile[lo] * n_tiles;
    row0 = first_row[lo] + (in % rows) * kExRows;
    n0 = (in / rows) * cols_per_tile;
  };

  if (warp == 0) {
    // ---------------- producer ----------------
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
        int expert, row0, n0;
        locate(t, expert, row0, n0);
        const int w_row = expert * p.cols + n0;
        for (int kb = 0; kb < k_blocks; ++kb) {
          ok = mbar_wait(empty0 + 8 * stage, phase ^ 1, giveup);
          if (!ok) break;
          const uint32_t dst = tiles_base + stage * kExStage, bar = full0 + 8 * stage;
          mbar_expect_tx(bar, kExStage);
          tma_load_2d(dst, &map_x, bar, kb * kExK, row0);            // (rows of the next experts come along; nobody stores them)
          tma_load_2d(dst + kExStageA, &map_w, bar, kb * kExK, w_row);
          if (p.mode == 0) tma_load_2d(dst + kExStageA + kExStageB / 2, &map_w2, bar, kb * kExK, w_row);
          if (++stage == kExStages) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (elect_one()) {
      const uint32_t idesc = instr_desc_bf16(kExRows, kExCols);
      int stage = 0, it = 0;
      uint32_t phase = 0;
      for (int t = blockIdx.x; t < total && !*giveup; t += gridDim.x, ++it) {
        const int buf = it & 1;
        if (!mbar_wait(acc_empty0 + 8 * buf, (((it >> 1) & 1) ^ 1), giveup)) break;
        tc_fence_after();
        bool ok = true;
        for (int kb = 0; kb < k_blocks; ++kb) {
          if (!mbar_wait(full0 + 8 * stage, phase, giveup)) { ok = false; break; }
          const uint32_t a_addr = tiles_base + stage * kExStage;
          umma_k64(tmem_base + buf * kExCols, desc_low(a_addr), desc_low(a_addr + kExStageA), idesc, kb > 0 ? 1u : 0u);
          umma_commit(empty0 + 8 * stage);
          if (++stage == kExStages) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        umma_commit(acc_full0 + 8 * buf);
      }
    }
  } else {
    // ---------------- epilogue: two threads finish a pair's row of the tile, half of the columns each ----------------
    // A thread leaves up to 256 bytes of its row in shared memory, and the warp writes the 32 rows one after another: whole
    // lines, where stores from the registers would touch 32 rows, 16 bytes of each, an instruction.  (A bulk copy a row
    // took about 60 cycles each, 8 us a tile of the down product.)
    const int quarter = warp & 3;                      // lanes 32 * quarter .. of tensor memory
    const int half = (warp - 2) >> 2;
    const uint32_t staged = full0 + 256 + (uint32_t)(half * kExRows + quarter * 32) * kExRowPitch, staged_row = staged + lane * kExRowPitch;
    const int elem = p.mode == 2 ? 4 : 2, chunk = min(cols_per_tile / 2, kExRowBytes / elem);
    int it = 0;
    for (int t = blockIdx.x; t < total && !*giveup; t += gridDim.x, ++it) {
      int expert, row0, n0;
      locate(t, expert, row0, n0);
      const int row = row0 + quarter * 32 + lane, end = first_row[expert + 1];
      const int pair = row < end ? p.order[row] : 0;
      const float w = p.mode == 1 || (p.mode == 0) != (p.scale_input != 0) ? 1.f : p.weight[pair];
      uint8_t* dst = static_cast<uint8_t*>(p.out) + ((size_t)(p.mode == 2 ? pair : row) * p.cols + n0) * elem;
      const int buf = it & 1;
      bool ok = mbar_wait(acc_full0 + 8 * buf, (it >> 1) & 1, giveup);
      ok = __all_sync(0xffffffffu, ok);                // the loads from tensor memory are warp-wide
      if (!ok) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * kExCols;
      for (int c0 = half * (cols_per_tile / 2); c0 < (half + 1) * (cols_per_tile / 2); c0 += chunk) {
        __syncwarp();                                  // the last rows have been read
        for (int c = c0; c < c0 + chunk; c += 16) {
          uint32_t a[16], b[16];
          tmem_ld16_issue(taddr + c, a);
          if (p.mode == 0) tmem_ld16_issue(taddr + kExCols / 2 + c, b);
          tmem_ld_wait();
          uint32_t v[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float s = __uint_as_float(a[j]);
            float f;
            if (p.mode == 0) {
              f = silu_branchless(round_to<__nv_bfloat16>(s * w)) * round_to<__nv_bfloat16>(__uint_as_float(b[j]) * w);
            } else if (p.mode == 1) {
              const float u = fmaxf(round_to<__nv_bfloat16>(s), 0.f);
              f = u * u;
            } else {
              f = s * w;
            }
            v[j] = __float_as_uint(f);
          }
          const uint32_t at = staged_row + (uint32_t)(c - c0) * elem;
          if (p.mode == 2) {
#pragma unroll
            for (int j = 0; j < 16; j += 4)
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + 4 * j), "r"(v[j]), "r"(v[j + 1]), "r"(v[j + 2]),
                           "r"(v[j + 3]) : "memory");
          } else {
#pragma unroll
            for (int j = 0; j < 16; j += 8) {
              uint32_t q[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const __nv_bfloat162 two = __floats2bfloat162_rn(__uint_as_float(v[j + 2 * i]), __uint_as_float(v[j + 2 * i + 1]));
                q[i] = *reinterpret_cast<const uint32_t*>(&two);
              }
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + 2 * j), "r"(q[0]), "r"(q[1]), "r"(q[2]), "r"(q[3])
                           : "memory");
            }
          }
        }
        __syncwarp();
        const int bytes = min(chunk, p.cols - n0 - c0) * elem;               // (columns come in eights: whole pieces of 16)
        const int lanes = chunk * elem / 16, sub = lane / lanes, at = (lane % lanes) * 16;      // 8 or 16 lanes a row
        const unsigned long long mine = reinterpret_cast<unsigned long long>(dst);
        for (int r = 0; r < 32; r += 32 / lanes) {
          const unsigned long long to = __shfl_sync(0xffffffffu, mine, r + sub);
          if (row0 + quarter * 32 + r + sub < end && at < bytes) {
            uint4 v;
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                         : "r"(staged + (uint32_t)(r + sub) * kExRowPitch + at));
            *reinterpret_cast<uint4*>(to + (size_t)c0 * elem + at) = v;
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty0 + 8 * buf);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && gave_up) set_status(p.status, kWaitTimeout, blockIdx.x, 40 + p.mode);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace tc
}  // namespace leone

using namespace leone;

// One grouped product.  mode 0: x [n_tokens, ldx], w = gate, w2 = up, out bf16 [pairs, cols]; mode 1: w = up; mode 2: x = act
// bf16 [pairs, K], w = down, out fp32 [pairs, cols].  w: [experts, cols, K].  sorted: room for bf16 [pairs, K] (modes 0 and 1).
// All rows start on 16 bytes.
int leone::experts_tc_product(int mode, const void* x, int ldx, const void* w, const void* w2, const int* offsets, const int* order,
                              const float* weight, int n_tokens, int experts, int top, int cols, int K, int scale_input, void* out,
                              void* sorted, int* status, cudaStream_t stream) {
  using namespace leone::tc;
  const long long pairs = (long long)n_tokens * top;
  CUtensorMap mx, mw, mw2;
  int e = make_tensor_map_2d(&mx, mode == 2 ? x : sorted, pairs, K, K, kExRows);
  if (e == 0) e = make_tensor_map_2d(&mw, w, (uint64_t)experts * cols, K, K, mode == 0 ? kExCols / 2 : kExCols);
  if (e == 0 && mode == 0) e = make_tensor_map_2d(&mw2, w2, (uint64_t)experts * cols, K, K, kExCols / 2);
  if (e != 0) return e;
  if (mode != 0) mw2 = mw;
  static const cudaError_t ready = cudaFuncSetAttribute(experts_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kExSmem);
  if (ready != cudaSuccess) return (int)ready;
  if (mode != 2) {
    e = launch_kernel(experts_sort_rows_kernel, dim3((unsigned)(pairs < 148 * 8 ? pairs : 148 * 8)), dim3(256), 0, stream,
                      (const __nv_bfloat16*)x, ldx, K, top, order, offsets + experts, (__nv_bfloat16*)sorted);
    if (e != 0) return e;
  }
  const ExpertParams p = {offsets, order, weight, out, experts, top, cols, K, scale_input, mode, status};
  const int per = mode == 0 ? kExCols / 2 : kExCols;
  const long long most = (pairs / kExRows + (experts < pairs ? experts : pairs)) * ((cols + per - 1) / per);
  return launch_kernel(experts_tc_kernel, dim3((unsigned)(most < 148 ? most : 148)), dim3(kExThreads), kExSmem, stream, mx, mw, mw2,
                       p);
}
