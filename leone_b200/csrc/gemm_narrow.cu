// out[M,N] = x[M,K] * w[N,K]^T in bfloat16 where the product has too few tiles of the other kernels to fill the chip.
//
// The token-major form on single SMs with tiles as narrow as it takes: up to 128 tokens ride the MMA's M side, and a tile has
// just so many weight rows (a multiple of 16 from 16 to 256) that the tiles fill the SMs once, unsplit.  The other way to fill them,
// a split of K, pays an exchange of fp32 partial tiles after the last MMA (4 to 8 us: a cluster barrier, then loads through
// distributed shared memory or the L2), which is more than these products' weights take to arrive.  A narrow tile reads the tokens'
// operand more often, but that comes out of the L2 while the weights come from memory.
//
// Warp 0 loads (TMA, 128-byte swizzle; the token tile only as many rows as there are tokens, in whole groups of eight: the MMA reads
// 128 rows whatever they hold, and a row reaches nothing but its own sums, which are not stored), warp 1 issues tcgen05.mma, the
// others finish rows (finish_rows).  Two accumulators where a block has several tiles.  Every wait is bounded.
//
// All of K is added in one accumulator, as in every unsplit product: a relative error against 64 bits of 2.1e-6 at K 2048 and 4.4e-6
// at 4096, where a split, whose shorter sums meet in fp32, has 0.2 to 2.1e-6.  The operands' rounding to bfloat16 is 2e-3, and
// the logits of whole steps are as far from 64 bits in either form.
#include "gemm_parts.cuh"

namespace leone {
namespace tc {

constexpr int kNarrowEpilogueWarps = 4;
constexpr int kNarrowThreads = 64 + 32 * kNarrowEpilogueWarps;
constexpr int kNarrowMaxStages = 12;
constexpr int kNarrowOther = 1024 /*alignment*/ + 256 /*barriers*/ + kNarrowEpilogueWarps * kBoxBytes;

struct NarrowShape {
  int token_rows, blocks, a_bytes, b_bytes, stages, smem_bytes, columns;      // blocks: k-blocks of a stage, a_bytes and b_bytes of one
};
// `most`: tiles of the block with the most of them
__host__ __device__ inline NarrowShape narrow_shape(int m, int bn, int k_blocks, int most) {
  NarrowShape c;
  c.token_rows = m >= kTileW ? kTileW : (m + 7) / 8 * 8;
  c.a_bytes = c.token_rows * kTileK * 2;
  c.b_bytes = bn * kTileK * 2;
  const int room = 227 * 1024 - 64 - kNarrowOther;
  // Two k-blocks a stage where that leaves four stages: what a stage costs the thread that issues its MMAs (the wait for its data,
  // the commit) is then paid once for eight MMAs.
  c.blocks = k_blocks > 1 && room / (2 * (c.a_bytes + c.b_bytes)) >= 4 ? 2 : 1;
  c.stages = room / (c.blocks * (c.a_bytes + c.b_bytes));
  const int all = (k_blocks + c.blocks - 1) / c.blocks * most;
  if (c.stages > kNarrowMaxStages) c.stages = kNarrowMaxStages;
  if (c.stages > all) c.stages = all;
  c.smem_bytes = c.stages * c.blocks * (c.a_bytes + c.b_bytes) + kNarrowOther;
  c.columns = pow2_at_least(most > 1 ? 2 * bn : bn);
  return c;
}

__global__ void __launch_bounds__(kNarrowThreads, 1)
gemm_narrow_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const GemmParams p,
                   const int BN, const NarrowShape cfg) {
  const int kStages = cfg.stages, blocks = cfg.blocks, stage_bytes = blocks * (cfg.a_bytes + cfg.b_bytes);
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t tiles_base = (raw + 1023u) & ~1023u;
  const uint32_t bars = tiles_base + kStages * stage_bytes;
  // barriers: full[kStages], empty[kStages], acc_full[2], acc_empty[2]
  const uint32_t full0 = bars, empty0 = full0 + 8 * kStages, acc_full0 = empty0 + 8 * kStages, acc_empty0 = acc_full0 + 16;
  __shared__ uint32_t tmem_holder;
  __shared__ int gave_up;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m_tiles = (p.M + kTileW - 1) / kTileW, n_tiles = (p.N + BN - 1) / BN;
  const int total = m_tiles * n_tiles, k_blocks = (p.K + kTileK - 1) / kTileK;
  if (threadIdx.x == 0) {
    gave_up = 0;
    for (int s = 0; s < kStages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full0 + 8 * b, 1);
      mbar_init(acc_empty0 + 8 * b, kNarrowEpilogueWarps);
    }
    mbar_fence_init();
    tma_prefetch_desc(&map_w);
    tma_prefetch_desc(&map_x);
  }
  if (warp == 1) tmem_alloc(smem_u32(&tmem_holder), cfg.columns);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_holder;
  volatile int* giveup = &gave_up;
  pdl_trigger();

  if (warp == 0) {
    // The weights are older than the kernels before this one: those of the first stages are requested at once, the L2 is asked for
    // the next ones, and only then does the producer wait for the predecessor, whose output is the token operand.
    if (elect_one()) {
      // where the next stage's data comes from: tile t, k-block kb
      struct Cursor { int t, kb, m, n; };
      auto start = [&](Cursor& c) {
        c.kb = 0;
        c.m = c.t % m_tiles * kTileW;
        c.n = c.t / m_tiles * BN;
      };
      auto advance = [&](Cursor& c) {
        if ((c.kb += blocks) >= k_blocks) {
          c.t += gridDim.x;
          start(c);
        }
      };
      auto load_w = [&](const Cursor& c, uint32_t dst, uint32_t bar) {
        const int here = min(blocks, k_blocks - c.kb);
        mbar_expect_tx(bar, (uint32_t)(here * (cfg.a_bytes + cfg.b_bytes)));
        for (int i = 0; i < here; ++i)
          tma_load_2d(dst + blocks * cfg.a_bytes + i * cfg.b_bytes, &map_w, bar, (c.kb + i) * kTileK, c.n);
      };
      auto load_x = [&](const Cursor& c, uint32_t dst, uint32_t bar) {
        for (int i = 0; i < min(blocks, k_blocks - c.kb); ++i) tma_load_2d(dst + i * cfg.a_bytes, &map_x, bar, (c.kb + i) * kTileK, c.m);
      };
      Cursor c{(int)blockIdx.x, 0, 0, 0};
      start(c);
      const Cursor first = c;
      int early = 0;
      for (; early < kStages && c.t < total; ++early, advance(c)) load_w(c, tiles_base + early * stage_bytes, full0 + 8 * early);
      for (int ahead = p.l2_ahead; ahead > 0 && c.t < total; ahead -= blocks, advance(c))
        for (int i = 0; i < min(blocks, k_blocks - c.kb); ++i) tma_prefetch_2d(&map_w, (c.kb + i) * kTileK, c.n);
      pdl_wait();
      c = first;
      for (int i = 0; i < early; ++i, advance(c)) load_x(c, tiles_base + i * stage_bytes, full0 + 8 * i);
      uint32_t dst = tiles_base, bar = full0, phase = 0;         // (the ring was filled once where anything is left)
      for (; c.t < total; advance(c)) {
        if (!mbar_wait(bar + 8 * kStages, phase, giveup)) break;
        load_w(c, dst, bar);
        load_x(c, dst, bar);
        dst += stage_bytes;
        bar += 8;
        if (bar == empty0) {
          dst = tiles_base;
          bar = full0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = instr_desc_bf16(kTileW, BN);
      const uint32_t first = desc_low(tiles_base), step = stage_bytes >> 4;
      const uint32_t a_step = cfg.a_bytes >> 4, b_step = cfg.b_bytes >> 4, b_at = blocks * a_step;
      uint32_t a = first, bar = full0, phase = 0;
      int it = 0;
      for (int t = blockIdx.x; t < total && !*giveup; t += gridDim.x, ++it) {
        const int buf = it & 1;
        if (!mbar_wait(acc_empty0 + 8 * buf, ((it >> 1) & 1) ^ 1, giveup)) break;
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + buf * BN;
        uint32_t sum = 0;                              // the first MMA of a tile sets the accumulator
        int left = k_blocks;
        for (; left > 0; left -= blocks) {
          if (!mbar_wait(bar, phase, giveup)) break;
          umma_k64(tmem_d, a, a + b_at, idesc, sum);
          sum = 1;
          if (blocks == 2 && left > 1) umma_k64(tmem_d, a + a_step, a + b_at + b_step, idesc, 1);
          umma_commit(bar + 8 * kStages);
          bar += 8;
          a += step;
          if (bar == empty0) {
            bar = full0;
            a = first;
            phase ^= 1;
          }
        }
        if (left > 0) break;                           // a wait ran out
        umma_commit(acc_full0 + 8 * buf);
      }
    }
  } else {
    const int quarter = warp & 3;                     // tensor memory lanes 32 * quarter .. +31
    const uint32_t box = bars + 256 + (warp - 2) * kBoxBytes;
    int it = 0;
    pdl_wait();                                       // outputs and residual may be in use until here
    for (int t = blockIdx.x; t < total && !*giveup; t += gridDim.x, ++it) {
      const int m_tile = t % m_tiles, n_tile = t / m_tiles, buf = it & 1;
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * BN;
      auto complete = [&]() {
        bool ok = mbar_wait(acc_full0 + 8 * buf, (it >> 1) & 1, giveup);
        ok = __all_sync(0xffffffffu, ok);             // the loads from tensor memory are warp-wide
        if (ok) tc_fence_after();
        return ok;
      };
      if (!finish_rows(p, taddr, m_tile * kTileW + quarter * 32, n_tile * BN, 0, BN, box, complete, [](const float (&)[8]) {})) break;
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty0 + 8 * buf);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (gave_up) {
    if (threadIdx.x == 0) set_status(p.status, kWaitTimeout, blockIdx.x, 6);
    // let tile copies that are still in flight land before the block's memory goes away
    const long long start = clock64();
    while (clock64() - start < 200000) {}
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, cfg.columns);
  }
}

}  // namespace tc
}  // namespace leone

using namespace leone;
using namespace leone::tc;

// The arguments and epilogues of leone_gemm_pair (0 bf16, 1 fp32, 2 fp32 += residual, 3 gate) with tiles of 128 tokens x `width` weight
// rows (a multiple of 16 from 16 to 256, of 32 with the gate); a norm before the product, none after it.  (The callers' rules
// take it for products without a norm on either side.)
extern "C" int leone_gemm_narrow(const void* x, const void* w, void* out, const float* residual, int m, int n, int k, int ldx,
                                 int ldw, int ldc, int epilogue, int width, int* status, int sm_count,
                                 const float* norm_in_ss, int norm_in_parts, float norm_eps, const float* gate_shape,
                                 const float* bias, cudaStream_t stream) {
  if (m <= 0 || n <= 0) return 0;
  if (k <= 0 || (k % 8) != 0 || (ldx % 8) != 0 || (ldw % 8) != 0) return kRefusedAlignment;
  if (epilogue < 0 || epilogue > 3 || sm_count < 1 || width < 16 || width > 256 || (width % 16) != 0) return kRefusedSize;
  if (epilogue == 2 && residual == nullptr) return kRefusedSize;
  if (epilogue == 3 && ((n % 32) != 0 || (width % 32) != 0)) return kRefusedSize;
  if (norm_in_ss != nullptr && norm_in_parts < 1) return kRefusedSize;
  if ((uintptr_t)bias & 15) return kRefusedAlignment;
  const int k_blocks = (k + kTileK - 1) / kTileK;
  const long long total = (long long)((n + width - 1) / width) * ((m + kTileW - 1) / kTileW);
  if (total > 0x7fffffff) return kRefusedSize;
  const int grid = (int)(total < sm_count ? total : sm_count), most = (int)((total + grid - 1) / grid);
  const NarrowShape cfg = narrow_shape(m, width, k_blocks, most > 64 ? 64 : most);
  if (cfg.stages < 2 && (k_blocks + cfg.blocks - 1) / cfg.blocks * (long long)most >= 2) return kRefusedSize;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_narrow_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 64);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  CUtensorMap mw, mx;
  int r = make_tensor_map_2d(&mw, w, (uint64_t)n, (uint64_t)k, (uint64_t)ldw, (uint32_t)width);
  if (r != 0) return r;
  r = make_tensor_map_2d(&mx, x, (uint64_t)m, (uint64_t)k, (uint64_t)ldx, (uint32_t)cfg.token_rows);
  if (r != 0) return r;
  GemmParams p{out, residual, m, n, k, ldc, epilogue, 1, 0, nullptr, nullptr, status, nullptr,
               nullptr, nullptr, nullptr, 0, norm_in_ss, norm_in_parts, norm_eps, 8};
  set_gate_shape(p, gate_shape);
  p.bias = bias;
  return launch_kernel(gemm_narrow_kernel, dim3((unsigned)grid), dim3(kNarrowThreads), (size_t)cfg.smem_bytes, stream, mw, mx, p,
                       width, cfg);
}
