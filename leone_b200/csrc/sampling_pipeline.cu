// The sampler's truncation stages on the device, in fp64.
//
// The reference builds a sampling distribution on the host in f64 (crates/leone/src/sampler.rs:
// 451-469): finite logits sorted descending (ties: lower id first), weights exp(l/T - l_max/T)
// normalised (:501-530); the stages that read raw logits (top-n-sigma, min-k) first (:532-553),
// then every other stage in the order given, each seeing the renormalised survivors of the one
// before and never emptying the set (:555-612); the token is then drawn by scanning the whole
// row in id order with u = uniform(seed, position, Select) (:803-857).  The same here:
//
//   sort      one row = P (a power of two >= vocab) pairs (fp64 key, id): a stable radix sort of the
//             fp32 logits, or, where the keys are fp64 or a row is short, a bitonic network (tiles of 2,048
//             pairs in shared memory, larger strides in global memory); a list that starts with a top-k
//             of up to 1,024 finds and sorts those k alone
//   stages    one block per row walks the stage list over the sorted row with block-wide
//             fp64 sums and scans; "typical" needs a second sort (by |surprise - entropy|),
//             so the stage list is cut there and the host entry launches the pieces in order
//   select    probabilities scattered back to id order, id-order scan against u
//
// Stage types: 0 top-k, 1 top-p, 2 min-p, 3 top-a, 4 tail-free, 5 typical, 6 epsilon, 7 eta,
// 8 min-k, 9 top-n-sigma.
#include <cmath>
#include <climits>
#include "common.cuh"

namespace leone {
namespace samp {

constexpr int kTile = 2048;          // pairs a block sorts in shared memory
constexpr int kThreads = 1024;
constexpr int kMaxStages = 16;

enum Stage { kTopK = 0, kTopP, kMinP, kTopA, kTailFree, kTypical, kEpsilon, kEta, kMinK, kTopNSigma };

struct Stages {
  int n;
  int type[kMaxStages];
  double value[kMaxStages];
};

// Per-row views into the scratch area.
struct Row {
  double* keys;     // [P] sorted raw logits (descending); -inf past the finite ones
  int* order;       // [P] their ids
  double* kept;     // [P] probabilities of the survivors, in the same order
  double* skeys;    // [P] second sort: -score
  int* sidx;        // [P] second sort: slot
  double* aux_f;    // [P]
  int* aux_i;       // [P]
  double* dense;    // [vocab] probabilities in id order
  int* n;           // survivors
};

__host__ __device__ inline size_t row_bytes(int P, int vocab) {
  return (size_t)P * (8 + 4 + 8 + 8 + 4 + 8 + 4) + (size_t)((vocab + 1) / 2 * 2) * 8 + 16;
}
__host__ __device__ inline Row row_of(uint8_t* scratch, int row, int P, int vocab) {
  uint8_t* b = scratch + (size_t)row * row_bytes(P, vocab);
  Row r;
  r.keys = (double*)b; b += (size_t)P * 8;
  r.kept = (double*)b; b += (size_t)P * 8;
  r.skeys = (double*)b; b += (size_t)P * 8;
  r.aux_f = (double*)b; b += (size_t)P * 8;
  r.dense = (double*)b; b += (size_t)((vocab + 1) / 2 * 2) * 8;
  r.order = (int*)b; b += (size_t)P * 4;
  r.sidx = (int*)b; b += (size_t)P * 4;
  r.aux_i = (int*)b; b += (size_t)P * 4;
  r.n = (int*)b;
  return r;
}

// The order of a sorted row: larger key first, equal keys by smaller id.
__device__ __forceinline__ bool precedes(double ka, int ia, double kb, int ib) {
  return ka > kb || (ka == kb && ia < ib);
}

// ---- sort ----------------------------------------------------------------------------------
// row_map (or null): row r of this call works on row row_map[r] of `logits`.
__global__ void sort_init_logits_kernel(const float* __restrict__ logits, const int* __restrict__ row_map,
                                        int vocab, int P, uint8_t* scratch) {
  const int row = blockIdx.y;
  const Row r = row_of(scratch, row, P, vocab);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *r.n = 0;
  if (i >= P) return;
  const int src = row_map != nullptr ? row_map[row] : row;
  const float v = i < vocab ? logits[(size_t)src * vocab + i] : NAN;
  const bool ok = i < vocab && isfinite(v);
  r.keys[i] = ok ? (double)v : -INFINITY;
  r.order[i] = ok ? i : vocab + i;            // the excluded ones sort last, in a fixed order
}

__global__ void count_finite_kernel(int vocab, int P, uint8_t* scratch) {
  // after the sort: the finite keys are a prefix
  const int row = blockIdx.y;
  const Row r = row_of(scratch, row, P, vocab);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P) return;
  const bool here = r.order[i] < vocab;
  const bool next = i + 1 < P && r.order[i + 1] < vocab;
  if (here && !next) *r.n = i + 1;
}

// All passes with stride below the tile for the levels k_first..k_last, in shared memory.
__global__ void __launch_bounds__(kThreads)
bitonic_tile_kernel(int which, int vocab, int P, int n_sort, uint8_t* scratch, int k_first, int k_last) {
  __shared__ double sk[kTile];
  __shared__ int si[kTile];
  const Row r = row_of(scratch, blockIdx.y, P, vocab);
  double* keys = which ? r.skeys : r.keys;
  int* idx = which ? r.sidx : r.order;
  const int tile = n_sort < kTile ? n_sort : kTile;
  const int base = blockIdx.x * tile;
  for (int t = threadIdx.x; t < tile; t += blockDim.x) {
    sk[t] = keys[base + t];
    si[t] = idx[base + t];
  }
  __syncthreads();
  for (int k = k_first; k <= k_last; k <<= 1) {
    int j = k >> 1;
    if (j > (tile >> 1)) j = tile >> 1;
    for (; j >= 1; j >>= 1) {
      for (int t = threadIdx.x; t < (tile >> 1); t += blockDim.x) {
        const int i = 2 * j * (t / j) + (t % j), l = i + j;
        const bool up = ((base + i) & k) == 0;
        const double ka = sk[i], kb = sk[l];
        const int ia = si[i], ib = si[l];
        const bool swap = up ? precedes(kb, ib, ka, ia) : precedes(ka, ia, kb, ib);
        if (swap) {
          sk[i] = kb; si[i] = ib;
          sk[l] = ka; si[l] = ia;
        }
      }
      __syncthreads();
    }
  }
  for (int t = threadIdx.x; t < tile; t += blockDim.x) {
    keys[base + t] = sk[t];
    idx[base + t] = si[t];
  }
}

// One pass with a stride of at least a tile.
__global__ void bitonic_global_kernel(int which, int vocab, int P, int n_sort, uint8_t* scratch, int k, int j) {
  const Row r = row_of(scratch, blockIdx.y, P, vocab);
  double* keys = which ? r.skeys : r.keys;
  int* idx = which ? r.sidx : r.order;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (n_sort >> 1)) return;
  const int i = 2 * j * (t / j) + (t % j), l = i + j;
  const bool up = (i & k) == 0;
  const double ka = keys[i], kb = keys[l];
  const int ia = idx[i], ib = idx[l];
  const bool swap = up ? precedes(kb, ib, ka, ia) : precedes(ka, ia, kb, ib);
  if (swap) {
    keys[i] = kb; idx[i] = ib;
    keys[l] = ka; idx[l] = ia;
  }
}

// Sorts the first n_sort (a power of two) pairs of every row's first or second pair of arrays.
static int sort_rows(int which, int vocab, int P, int n_sort, int rows, uint8_t* scratch, cudaStream_t stream) {
  const int tile = n_sort < kTile ? n_sort : kTile;
  bitonic_tile_kernel<<<dim3(n_sort / tile, rows), kThreads, 0, stream>>>(which, vocab, P, n_sort, scratch, 2, tile);
  for (int k = 2 * tile; k <= n_sort; k <<= 1) {
    for (int j = k >> 1; j >= tile; j >>= 1)
      bitonic_global_kernel<<<dim3((n_sort / 2 + 255) / 256, rows), 256, 0, stream>>>(which, vocab, P, n_sort,
                                                                                       scratch, k, j);
    bitonic_tile_kernel<<<dim3(n_sort / tile, rows), kThreads, 0, stream>>>(which, vocab, P, n_sort, scratch, k, k);
  }
  return (int)cudaGetLastError();
}

// ---- block-wide fp64 helpers (one block of kThreads per row) ----------------------------------
struct Shared {
  double f[32];
  int i[32];
  double total;
  int result;
};

__device__ __forceinline__ double block_sum(double v, Shared& sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) sh.f[warp] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) t += sh.f[w];
    sh.total = t;
  }
  __syncthreads();
  return sh.total;
}

// Exclusive prefix of v over the threads, in thread order; *total gets the sum.
__device__ __forceinline__ double block_scan(double v, Shared& sh, double* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const double up = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += up;
  }
  __syncthreads();
  if (lane == 31) sh.f[warp] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    double run = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) {
      const double s = sh.f[w];
      sh.f[w] = run;
      run += s;
    }
    sh.total = run;
  }
  __syncthreads();
  *total = sh.total;
  return sh.f[warp] + incl - v;
}

__device__ __forceinline__ int block_min(int v, Shared& sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if (lane == 0) sh.i[warp] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    int m = INT_MAX;
    for (int w = 0; w < kThreads / 32; ++w) m = min(m, sh.i[w]);
    sh.result = m;
  }
  __syncthreads();
  return sh.result;
}

__device__ __forceinline__ int block_sum_int(int v, Shared& sh) {
  return (int)(block_sum((double)v, sh) + 0.5);
}

// This thread's contiguous share of [0, n).
__device__ __forceinline__ void chunk_of(int n, int* lo, int* hi) {
  const int c = (n + kThreads - 1) / kThreads;
  *lo = min(n, (int)threadIdx.x * c);
  *hi = min(n, *lo + c);
}

__device__ double sum_of(const double* a, int n, Shared& sh) {
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += kThreads) s += a[i];
  return block_sum(s, sh);
}

__device__ double entropy_of(const double* kept, int n, Shared& sh) {
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += kThreads) {
    const double p = kept[i];
    if (p > 0.0) s += -p * log(p);
  }
  return block_sum(s, sh);
}

// How many leading entries are at least `floor` (kept is non-increasing, so they are a prefix).
__device__ int threshold_keep(const double* kept, int n, double floor, Shared& sh) {
  int first_below = n;
  for (int i = threadIdx.x; i < n; i += kThreads)
    if (!(kept[i] >= floor)) { first_below = i; break; }
  return block_min(first_below, sh);
}

// First index whose running sum of f(i) satisfies `reached`, scanning [0, count) in order.
template <typename F, typename R>
__device__ int first_where(int count, F f, R reached, Shared& sh) {
  int lo, hi;
  chunk_of(count, &lo, &hi);
  double local = 0.0;
  for (int i = lo; i < hi; ++i) local += f(i);
  double total;
  double run = block_scan(local, sh, &total);
  int found = INT_MAX;
  for (int i = lo; i < hi; ++i) {
    run += f(i);
    if (reached(run)) { found = i; break; }
  }
  return block_min(found, sh);
}

__device__ void renormalize(double* kept, int n, Shared& sh) {
  const double total = sum_of(kept, n, sh);
  for (int i = threadIdx.x; i < n; i += kThreads) kept[i] /= total;
  __syncthreads();
}

// ---- the k best of a row ------------------------------------------------------------------------
// A block per row, in place of ordering the whole row.  Bound by two readings of the row through one SM (about 5 us each at
// 151,936 logits); a full sort moves the row 36 times.  Every thread keeps the largest of its share of the row; the k-th
// largest of the 1,024 such maxima is a lower bound of the row's k-th largest value, so few values reach it; those
// are collected and sorted as 64-bit words (value as an ordered integer, then the smaller id first).  Where more
// reach it than fit (a few threads hold most of the best values, or thousands of ties), the k-th value and the
// last id among its ties are found bit by bit with counts over the row.
// Measured with all that follows (64 rows of 151,936 logits, top-k 40 and top-p): 2.29 ms with tiles of 2,048 sorted and their
// heads gathered, now 0.24 ms of which the host's share is most.
constexpr int kMaxTopK = 1024, kCandidates = 4096;

// Finite values in order; 0 for the others.  (-0 and 0 are equal keys.)
__device__ __forceinline__ unsigned ordered(float v) {
  if (!isfinite(v)) return 0u;
  const unsigned u = __float_as_uint(v + 0.f);
  return u & 0x80000000u ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float from_ordered(unsigned o) {
  return __uint_as_float(o & 0x80000000u ? o & 0x7fffffffu : ~o);
}

__global__ void __launch_bounds__(kThreads)
top_k_kernel(const float* __restrict__ logits, const int* __restrict__ row_map, int vocab, int P, uint8_t* scratch, int k) {
  __shared__ unsigned long long cand[kCandidates];
  __shared__ Shared sh;
  __shared__ int count_s;
  const int row = blockIdx.x, tid = threadIdx.x;
  const Row r = row_of(scratch, row, P, vocab);
  const float* l = logits + (size_t)(row_map != nullptr ? row_map[row] : row) * vocab;
  unsigned top = 0;
  int finite = 0;
#pragma unroll 8
  for (int i = tid; i < vocab; i += kThreads) {
    const unsigned o = ordered(l[i]);
    finite += o != 0;
    top = max(top, o);
  }
  finite = block_sum_int(finite, sh);
  const int want = min(k, finite);
  if (tid == 0) {
    *r.n = want;
    count_s = 0;
  }
  if (want == 0) return;
  // the largest bound that at least `want` threads reach (1, the least finite value's lower neighbour, if too few do)
  unsigned bound = 0;
  for (int b = 31; b >= 0; --b) {
    const unsigned t = bound | 1u << b;
    if (__syncthreads_count(top >= t) >= want) bound = t;
  }
  bound = max(bound, 1u);
#pragma unroll 8
  for (int i = tid; i < vocab; i += kThreads) {
    const unsigned o = ordered(l[i]);
    if (o >= bound) {
      const int at = atomicAdd(&count_s, 1);
      if (at < kCandidates) cand[at] = (unsigned long long)o << 32 | (0xffffffffu - (unsigned)i);
    }
  }
  __syncthreads();
  int count = count_s;
  if (count > kCandidates) {
    auto reach = [&](unsigned t) {
      int c = 0;
      for (int i = tid; i < vocab; i += kThreads) c += ordered(l[i]) >= t;
      return block_sum_int(c, sh);
    };
    unsigned kth = 0;
    for (int b = 31; b >= 0; --b)
      if (reach(kth | 1u << b) >= want) kth |= 1u << b;
    const int ties = want - (kth == 0xffffffffu ? 0 : reach(kth + 1));       // at least one
    // the id of the last tie that belongs: the largest t with fewer than `ties` ties below it
    unsigned last = 0;
    for (int b = 30; b >= 0; --b) {
      const unsigned t = last | 1u << b;
      int c = 0;
      for (int i = tid; i < vocab; i += kThreads) c += ordered(l[i]) == kth && (unsigned)i < t;
      if (block_sum_int(c, sh) < ties) last = t;
    }
    if (tid == 0) count_s = 0;
    __syncthreads();
    for (int i = tid; i < vocab; i += kThreads) {
      const unsigned o = ordered(l[i]);
      if (o > kth || (o == kth && (unsigned)i <= last))
        cand[atomicAdd(&count_s, 1)] = (unsigned long long)o << 32 | (0xffffffffu - (unsigned)i);
    }
    __syncthreads();
    count = count_s;                       // = want
  }
  int n_sort = 2;
  while (n_sort < count) n_sort <<= 1;
  for (int i = count + tid; i < n_sort; i += kThreads) cand[i] = 0;
  __syncthreads();
  for (int size = 2; size <= n_sort; size <<= 1)
    for (int j = size >> 1; j >= 1; j >>= 1) {
      for (int t = tid; t < (n_sort >> 1); t += kThreads) {
        const int i = 2 * j * (t / j) + (t % j);
        const unsigned long long a = cand[i], b = cand[i + j];
        if ((i & size) == 0 ? a < b : a > b) {
          cand[i] = b;
          cand[i + j] = a;
        }
      }
      __syncthreads();
    }
  for (int i = tid; i < want; i += kThreads) {
    r.keys[i] = (double)from_ordered((unsigned)(cand[i] >> 32));
    r.order[i] = (int)(0xffffffffu - (unsigned)cand[i]);
  }
}

// ---- radix sort of the logits ---------------------------------------------------------------------
// Four passes over 8 bits of the ordered logit, each a count per tile of 4,096 entries, a scan of the counts in (digit, tile)
// order, and a stable scatter; ids start in order, so equal logits stay in id order.  Bound by the row's bytes, moved 5
// times (the bitonic network moves them 36 times).  The entries that are not finite come last; the others are counted in *r.n.
// Measured, 50 rows of 151,936 logits: 0.73 ms (scatters 0.49, counts 0.20); the network 4.2 ms.  A row of one tile of the network
// (2,048) or less stays with it: one launch.
constexpr int kRadixTile = 4096, kRadixThreads = 256, kRadixItems = kRadixTile / kRadixThreads;

struct RadixRow {
  const unsigned* key_in;      // null: the first pass reads the logits
  const int* id_in;
  unsigned* key_out;           // null: the last pass writes r.keys and r.order
  int* id_out;
  int* counts;                 // [256][tiles]
};
__device__ __forceinline__ RadixRow radix_row(const Row& r, int P, int pass) {
  unsigned* keys = reinterpret_cast<unsigned*>(r.skeys);              // two of P
  RadixRow x;
  x.key_in = pass == 0 ? nullptr : keys + (pass & 1 ? 0 : P);
  x.id_in = pass & 1 ? r.sidx : r.aux_i;
  x.key_out = pass == 3 ? nullptr : keys + (pass & 1 ? P : 0);
  x.id_out = pass & 1 ? r.aux_i : r.sidx;
  x.counts = reinterpret_cast<int*>(r.aux_f);
  return x;
}
// Larger logits first: the digit counted from the top.
__device__ __forceinline__ int radix_digit(unsigned key, int pass) { return 255 - (int)(key >> (8 * pass) & 255u); }

__global__ void __launch_bounds__(kRadixThreads)
radix_count_kernel(const float* __restrict__ logits, const int* __restrict__ row_map, int vocab, int P, uint8_t* scratch, int pass) {
  __shared__ int hist[256];
  __shared__ int finite_s;
  const int row = blockIdx.y, tid = threadIdx.x, tiles = gridDim.x;
  const Row r = row_of(scratch, row, P, vocab);
  const RadixRow x = radix_row(r, P, pass);
  const float* l = logits + (size_t)(row_map != nullptr ? row_map[row] : row) * vocab;
  hist[tid] = 0;
  if (tid == 0) finite_s = 0;
  __syncthreads();
  int finite = 0;
#pragma unroll
  for (int j = 0; j < kRadixItems; ++j) {
    const int i = blockIdx.x * kRadixTile + j * kRadixThreads + tid;
    if (i >= vocab) continue;
    const unsigned key = pass == 0 ? ordered(l[i]) : x.key_in[i];
    finite += key != 0;
    // lanes with the same digit add once: most logits share their upper digits
    const int digit = radix_digit(key, pass);
    const unsigned peers = __match_any_sync(__activemask(), digit);
    if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&hist[digit], __popc(peers));
  }
  if (pass == 0 && finite > 0) atomicAdd(&finite_s, finite);
  __syncthreads();
  x.counts[tid * tiles + blockIdx.x] = hist[tid];
  if (pass == 0 && tid == 0) atomicAdd(r.n, finite_s);
}

__global__ void __launch_bounds__(kThreads)
radix_scan_kernel(int vocab, int P, uint8_t* scratch, int tiles) {
  __shared__ int warp_sum[kThreads / 32];
  const Row r = row_of(scratch, blockIdx.x, P, vocab);
  int* counts = reinterpret_cast<int*>(r.aux_f);
  const int n = 256 * tiles, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int lo, hi;
  chunk_of(n, &lo, &hi);
  int local = 0;
  for (int i = lo; i < hi; ++i) local += counts[i];
  int upto = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int before = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += before;
  }
  if (lane == 31) warp_sum[warp] = upto;
  __syncthreads();
  int run = upto - local;
  for (int w = 0; w < warp; ++w) run += warp_sum[w];
  for (int i = lo; i < hi; ++i) {
    const int c = counts[i];
    counts[i] = run;
    run += c;
  }
}

__global__ void __launch_bounds__(kRadixThreads)
radix_scatter_kernel(const float* __restrict__ logits, const int* __restrict__ row_map, int vocab, int P, uint8_t* scratch, int pass) {
  constexpr int kWarps = kRadixThreads / 32;
  __shared__ int where[kWarps][256];               // per warp: how many of a digit so far, then where its first one goes
  const int row = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tiles = gridDim.x;
  const Row r = row_of(scratch, row, P, vocab);
  const RadixRow x = radix_row(r, P, pass);
  const float* l = logits + (size_t)(row_map != nullptr ? row_map[row] : row) * vocab;
  for (int i = tid; i < kWarps * 256; i += kRadixThreads) (&where[0][0])[i] = 0;
  __syncthreads();
  // a warp's entries are neighbours, 32 at a time, so ranks within the warp follow the row's order
  unsigned key[kRadixItems];
  int id[kRadixItems], rank[kRadixItems];
  const int first = blockIdx.x * kRadixTile + warp * 32 * kRadixItems + lane;
#pragma unroll
  for (int j = 0; j < kRadixItems; ++j) {
    const int i = first + 32 * j;
    const bool in = i < vocab;
    key[j] = !in ? 0u : pass == 0 ? ordered(l[i]) : x.key_in[i];
    id[j] = !in ? -1 : pass == 0 ? i : x.id_in[i];
  }
#pragma unroll
  for (int j = 0; j < kRadixItems; ++j) {
    const bool in = id[j] >= 0;
    const int digit = radix_digit(key[j], pass);
    const unsigned peers = __match_any_sync(0xffffffffu, in ? digit : 256 + lane);
    int before = 0;
    if (in) before = where[warp][digit];
    __syncwarp();
    rank[j] = before + __popc(peers & ((1u << lane) - 1u));
    if (in && lane == __ffs(peers) - 1) where[warp][digit] = before + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  {
    int run = x.counts[tid * tiles + blockIdx.x];  // one digit a thread
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const int c = where[w][tid];
      where[w][tid] = run;
      run += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kRadixItems; ++j) {
    if (id[j] < 0) continue;
    const int to = where[warp][radix_digit(key[j], pass)] + rank[j];
    if (pass == 3) {
      r.keys[to] = key[j] == 0 ? -INFINITY : (double)from_ordered(key[j]);
      r.order[to] = key[j] == 0 ? vocab + id[j] : id[j];
    } else {
      x.key_out[to] = key[j];
      x.id_out[to] = id[j];
    }
  }
}

__global__ void zero_counts_kernel(int rows, int vocab, int P, uint8_t* scratch) {
  const int row = blockIdx.x * blockDim.x + threadIdx.x;
  if (row < rows) *row_of(scratch, row, P, vocab).n = 0;
}

static int radix_sort_rows(const float* logits, const int* row_map, int vocab, int P, int rows, uint8_t* scratch,
                           cudaStream_t stream) {
  const int tiles = (vocab + kRadixTile - 1) / kRadixTile;
  zero_counts_kernel<<<(rows + 255) / 256, 256, 0, stream>>>(rows, vocab, P, scratch);
  for (int pass = 0; pass < 4; ++pass) {
    radix_count_kernel<<<dim3(tiles, rows), kRadixThreads, 0, stream>>>(logits, row_map, vocab, P, scratch, pass);
    radix_scan_kernel<<<rows, kThreads, 0, stream>>>(vocab, P, scratch, tiles);
    radix_scatter_kernel<<<dim3(tiles, rows), kRadixThreads, 0, stream>>>(logits, row_map, vocab, P, scratch, pass);
  }
  return (int)cudaGetLastError();
}

// ---- the stages -------------------------------------------------------------------------------
// begin != 0: raw-logit stages, weights, normalisation; then stages [s0, s1) (raw ones skipped).
__global__ void __launch_bounds__(kThreads)
stages_kernel(int vocab, int P, uint8_t* scratch, const double* __restrict__ temperature, Stages st,
              int begin, int s0, int s1) {
  __shared__ Shared sh;
  const Row r = row_of(scratch, blockIdx.x, P, vocab);
  int n = *r.n;
  __syncthreads();
  if (n <= 0) return;
  const double* keys = r.keys;
  double* kept = r.kept;
  if (begin) {
    for (int s = 0; s < st.n; ++s) {
      if (st.type[s] == kTopNSigma && n >= 2) {
        const double mean = sum_of(keys, n, sh) / (double)n;
        double v = 0.0;
        for (int i = threadIdx.x; i < n; i += kThreads) {
          const double d = keys[i] - mean;
          v += d * d;
        }
        const double dev = sqrt(block_sum(v, sh) / (double)n);
        if (isfinite(dev)) {
          const double cut = keys[0] - st.value[s] * dev;
          n = max(1, threshold_keep(keys, n, cut, sh));
        }
      } else if (st.type[s] == kMinK && n >= 2) {
        const double range = keys[0] - keys[n - 1] + 1e-8;
        if (isfinite(range) && range > 0.0) {
          // the rank with the largest (gap / range) / rank; of equal ones the lowest
          double best = -INFINITY;
          int cliff = INT_MAX;
          for (int rank = 1 + threadIdx.x; rank < n; rank += kThreads) {
            const double w = ((keys[rank - 1] - keys[rank]) / range) / (double)rank;
            if (w > best) { best = w; cliff = rank; }
          }
          // block-wide: largest value, then the lowest rank that has it
          double m = best;
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
          __syncthreads();
          if ((threadIdx.x & 31) == 0) sh.f[threadIdx.x >> 5] = m;
          __syncthreads();
          m = sh.f[0];
          for (int w = 1; w < kThreads / 32; ++w) m = fmax(m, sh.f[w]);
          __syncthreads();
          cliff = block_min(best == m ? cliff : INT_MAX, sh);
          const double fb = floor(st.value[s] / range);
          const int fallback = (isfinite(fb) && fb >= 0.0) ? (int)fmin(fb, (double)n) : n;
          n = min(n, max(1, max(cliff, fallback)));
        }
      }
    }
    const double t = temperature[blockIdx.x];
    const double top = keys[0] / t;
    for (int i = threadIdx.x; i < n; i += kThreads) kept[i] = exp(keys[i] / t - top);
    __syncthreads();
    renormalize(kept, n, sh);
  }
  for (int s = s0; s < s1; ++s) {
    const int type = st.type[s];
    const double value = st.value[s];
    int keep = n;
    if (type == kTopK) {
      keep = (int)fmin(value, (double)n);
    } else if (type == kTopP) {
      const int at = first_where(n, [&](int i) { return kept[i]; }, [&](double c) { return c >= value; }, sh);
      keep = at == INT_MAX ? n : at + 1;
    } else if (type == kMinP) {
      keep = threshold_keep(kept, n, value * kept[0], sh);
    } else if (type == kTopA) {
      keep = threshold_keep(kept, n, value * kept[0] * kept[0], sh);
    } else if (type == kEpsilon) {
      keep = threshold_keep(kept, n, value, sh);
    } else if (type == kEta) {
      const double h = entropy_of(kept, n, sh);
      keep = threshold_keep(kept, n, fmin(value, sqrt(value) * exp(-h)), sh);
    } else if (type == kTailFree) {
      if (n >= 3) {
        auto second = [&](int i) { return fabs(kept[i] - 2.0 * kept[i + 1] + kept[i + 2]); };
        double local = 0.0;
        for (int i = threadIdx.x; i < n - 2; i += kThreads) local += second(i);
        const double total = block_sum(local, sh);
        if (total > 0.0 && isfinite(total)) {
          const int at = first_where(n - 2, [&](int i) { return second(i) / total; },
                                     [&](double c) { return !(c <= value); }, sh);
          keep = 1 + (at == INT_MAX ? n - 2 : at);
        }
      }
    } else {
      continue;                       // raw stages ran at the beginning; typical is the host's cut
    }
    n = max(1, min(n, keep));
    __syncthreads();
    renormalize(kept, n, sh);
  }
  if (threadIdx.x == 0) *r.n = n;
}

// Typical, first half: the keys of the second sort (ascending |surprise - entropy|, then slot).
__global__ void __launch_bounds__(kThreads)
typical_scores_kernel(int vocab, int P, uint8_t* scratch) {
  __shared__ Shared sh;
  const Row r = row_of(scratch, blockIdx.x, P, vocab);
  const int n = *r.n;
  const double h = entropy_of(r.kept, n, sh);
  for (int i = threadIdx.x; i < P; i += kThreads) {
    if (i < n) {
      const double score = fabs(-log(r.kept[i]) - h);
      r.skeys[i] = score == score ? -score : -INFINITY;
      r.sidx[i] = i;
    } else {
      r.skeys[i] = -INFINITY;
      r.sidx[i] = P + i;
    }
  }
}

// Typical, second half: slots in score order until their mass reaches `mass`; the survivors
// keep their descending order.
__global__ void __launch_bounds__(kThreads)
typical_select_kernel(int vocab, int P, uint8_t* scratch, double mass) {
  __shared__ Shared sh;
  const Row r = row_of(scratch, blockIdx.x, P, vocab);
  const int n = *r.n;
  __syncthreads();
  if (n <= 0) return;
  const int at = first_where(n, [&](int i) { return r.kept[r.sidx[i]]; }, [&](double c) { return c >= mass; }, sh);
  const int m = at == INT_MAX ? n : at + 1;
  for (int i = threadIdx.x; i < n; i += kThreads) r.aux_i[i] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < m; i += kThreads) r.aux_i[r.sidx[i]] = 1;
  __syncthreads();
  // compaction in slot order; the second sort's keys are no longer needed: their place holds
  // the survivors' ids meanwhile
  int* ids = reinterpret_cast<int*>(r.skeys);
  int lo, hi;
  chunk_of(n, &lo, &hi);
  int local = 0;
  for (int i = lo; i < hi; ++i) local += r.aux_i[i];
  double total;
  int pos = (int)(block_scan((double)local, sh, &total) + 0.5);
  for (int i = lo; i < hi; ++i)
    if (r.aux_i[i]) {
      r.aux_f[pos] = r.kept[i];
      ids[pos] = r.order[i];
      ++pos;
    }
  __syncthreads();
  for (int i = threadIdx.x; i < m; i += kThreads) {
    r.kept[i] = r.aux_f[i];
    r.order[i] = ids[i];
  }
  __syncthreads();
  renormalize(r.kept, m, sh);
  if (threadIdx.x == 0) *r.n = m;
}

// Mirostat v2's filter (crates/leone/src/sampler.rs:383-420): of the distribution the stages
// left (the target), the tokens whose surprise -ln p is at most the row's current maximum are
// kept and renormalised (the most probable one if none is); the target's probabilities stay in
// aux_f so that the draw can report the chosen token's.
__global__ void __launch_bounds__(kThreads)
surprise_filter_kernel(int vocab, int P, uint8_t* scratch, const double* __restrict__ maximum_surprise) {
  __shared__ Shared sh;
  const Row r = row_of(scratch, blockIdx.x, P, vocab);
  const int n = *r.n;
  __syncthreads();
  if (n <= 0) return;
  const double mu = maximum_surprise[blockIdx.x];
  int first_out = n;
  for (int i = threadIdx.x; i < n; i += kThreads) r.aux_f[i] = r.kept[i];
  for (int i = threadIdx.x; i < n; i += kThreads)
    if (!(-log(r.kept[i]) <= mu)) { first_out = i; break; }
  const int keep = max(1, block_min(first_out, sh));
  renormalize(r.kept, keep, sh);
  if (threadIdx.x == 0) *r.n = keep;
}

__device__ __forceinline__ unsigned long long splitmix64(unsigned long long v) {
  unsigned long long z = v + 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

constexpr int kFewSurvivors = 1024;

// Probabilities back in id order, and the draw: the first id whose running sum exceeds u, else
// the last id with any probability.
__global__ void __launch_bounds__(kThreads)
select_kernel(int vocab, int P, uint8_t* scratch, const long long* __restrict__ seeds,
              const long long* __restrict__ positions, int* __restrict__ out, const int* __restrict__ row_map,
              double* __restrict__ probs, double* __restrict__ chosen_prob) {
  __shared__ Shared sh;
  const int row = blockIdx.x;
  const int dst = row_map != nullptr ? row_map[row] : row;      // where the row's id goes
  const Row r = row_of(scratch, row, P, vocab);
  const int n = *r.n;
  const unsigned long long purpose = 0xbf58476d1ce4e5b9ull;
  const unsigned long long mixed =
      splitmix64((unsigned long long)seeds[row] ^ splitmix64((unsigned long long)positions[row] ^ purpose));
  const double u = (double)(mixed >> 11) * (1.0 / 9007199254740992.0);
  int token;
  if (n > 0 && n <= kFewSurvivors && probs == nullptr) {
    // few survivors: sorted by id here instead of scattered over the vocabulary.  The sums are the other branch's,
    // whose zeros change none of them: a thread's share of the ids in order, from the prefix of the shares before it.
    __shared__ int ids[kFewSurvivors];
    __shared__ double p[kFewSurvivors];
    int n_sort = 2;
    while (n_sort < n) n_sort <<= 1;
    for (int i = threadIdx.x; i < n_sort; i += kThreads) {
      ids[i] = i < n ? r.order[i] : INT_MAX;
      p[i] = i < n ? r.kept[i] : 0.0;
    }
    __syncthreads();
    for (int size = 2; size <= n_sort; size <<= 1)
      for (int j = size >> 1; j >= 1; j >>= 1) {
        for (int t = threadIdx.x; t < (n_sort >> 1); t += kThreads) {
          const int i = 2 * j * (t / j) + (t % j);
          const int a = ids[i], b = ids[i + j];
          if ((i & size) == 0 ? a > b : a < b) {
            ids[i] = b;
            ids[i + j] = a;
            const double pa = p[i];
            p[i] = p[i + j];
            p[i + j] = pa;
          }
        }
        __syncthreads();
      }
    auto first_at_least = [&](int id) {
      int lo = 0, hi = n;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (ids[mid] < id) lo = mid + 1;
        else hi = mid;
      }
      return lo;
    };
    int lo, hi;
    chunk_of(vocab, &lo, &hi);
    const int from = first_at_least(lo), to = first_at_least(hi);
    double local = 0.0, total;
    int last = -1;
    for (int i = from; i < to; ++i) {
      local += p[i];
      if (p[i] > 0.0) last = ids[i];
    }
    double run = block_scan(local, sh, &total);
    int found = INT_MAX;
    if (lo < hi && (from == to || ids[from] != lo) && u < run) found = lo;
    for (int i = from; i < to && found == INT_MAX; ++i) {
      run += p[i];
      if (u < run) found = ids[i];
    }
    const int at = block_min(found, sh);
    last = -block_min(-last, sh);
    token = at == INT_MAX ? last : at;
  } else {
    for (int i = threadIdx.x; i < vocab; i += kThreads) r.dense[i] = 0.0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += kThreads) r.dense[r.order[i]] = r.kept[i];
    __syncthreads();
    if (probs != nullptr)
      for (int i = threadIdx.x; i < vocab; i += kThreads) probs[(size_t)row * vocab + i] = r.dense[i];
    if (n <= 0) {
      if (threadIdx.x == 0) out[dst] = -1;
      return;
    }
    const double* dense = r.dense;
    const int at = first_where(vocab, [&](int i) { return dense[i]; }, [&](double c) { return u < c; }, sh);
    int last = -1;
    for (int i = threadIdx.x; i < vocab; i += kThreads)
      if (dense[i] > 0.0) last = i;
    last = -block_min(-last, sh);
    token = at == INT_MAX ? last : at;             // a zero entry cannot make the sum pass u
  }
  if (threadIdx.x == 0) out[dst] = token;
  if (chosen_prob != nullptr)                      // the token's probability before the surprise filter
    for (int i = threadIdx.x; i < n; i += kThreads)
      if (r.order[i] == token) chosen_prob[row] = r.aux_f[i];
}

// Penalties from the decode history, before the sampler (crates/leone/src/penalty.rs:163-206).
// The host has walked the history (it owns it) and lists, per (row, token), how often the token
// occurs in the row's window and the largest repeated-suffix (DRY) penalty that reaches it; the
// arithmetic on the logits is done here, in fp64 as there: a seen token's logit is divided by
// the repetition factor if positive, multiplied if not, then loses the presence penalty once
// and the frequency penalty per occurrence, and is rounded to fp32; the DRY penalty is then
// subtracted from that.
__global__ void penalize_kernel(float* __restrict__ logits, int vocab, int n, const int* __restrict__ rows,
                                const int* __restrict__ tokens, const int* __restrict__ counts,
                                const double* __restrict__ dry, const double* __restrict__ repetition,
                                const double* __restrict__ presence, const double* __restrict__ frequency) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  const int row = rows[e], token = tokens[e];
  if (token < 0 || token >= vocab) return;
  float* at = logits + (size_t)row * vocab + token;
  float logit = *at;
  const double rep = repetition[row], pres = presence[row], freq = frequency[row];
  if (counts[e] > 0 && (rep != 1.0 || pres != 0.0 || freq != 0.0)) {
    double value = (double)logit;
    value = value > 0.0 ? value / rep : value * rep;
    value -= pres;
    value -= freq * (double)counts[e];
    logit = (float)value;
  }
  if (dry[e] > 0.0) logit = (float)((double)logit - dry[e]);
  *at = logit;
}

}  // namespace samp
}  // namespace leone

using namespace leone;
using namespace leone::samp;

static int pow2_at_least(int v) {
  int p = 2;
  while (p < v) p <<= 1;
  return p;
}

// Bytes of scratch for `rows` rows of `vocab` logits.
extern "C" long long leone_sample_truncated_scratch(int rows, int vocab) {
  return (long long)rows * (long long)row_bytes(pow2_at_least(vocab), vocab);
}

// logits: fp32 [rows, vocab]; temperature: fp64 [rows] (> 0); seeds, positions: int64 [rows];
// the stage list (types and values, in the order they apply) is the same for all rows; out: int32
// sampled ids; probs: fp64 [rows, vocab] or null, the distribution the draw was made from.
// row_map: int32 [rows] or null: row r of the call reads logits row row_map[r] and writes
// out[row_map[r]] (a subset of a step's rows is sampled in place, without gathering it first).
// maximum_surprise: fp64 [rows] or null: Mirostat v2's filter after the stages; chosen_prob (fp64
// [rows], with it) gets the drawn token's probability before that filter.
extern "C" int leone_sample_truncated(const float* logits, int rows, int vocab, const double* temperature,
                                      const long long* seeds, const long long* positions, int n_stages,
                                      const int* types, const double* values, void* scratch, int* out,
                                      double* probs, const double* maximum_surprise, double* chosen_prob,
                                      const int* row_map, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (vocab <= 0 || n_stages < 0 || n_stages > kMaxStages) return kRefusedSize;
  Stages st;
  st.n = n_stages;
  for (int s = 0; s < n_stages; ++s) {
    if (types[s] < 0 || types[s] > kTopNSigma) return kRefusedSize;
    st.type[s] = types[s];
    st.value[s] = values[s];
  }
  const int P = pow2_at_least(vocab);
  uint8_t* sc = static_cast<uint8_t*>(scratch);
  // A list that starts with a top-k and has no raw-logit stage needs only the row's k best pairs.  (A larger k than a block
  // collects orders the whole row.)
  bool raw = false;
  for (int s = 0; s < n_stages; ++s) raw = raw || st.type[s] == kMinK || st.type[s] == kTopNSigma;
  int e;
  if (!raw && n_stages > 0 && st.type[0] == kTopK && st.value[0] <= kMaxTopK) {
    top_k_kernel<<<rows, kThreads, 0, stream>>>(logits, row_map, vocab, P, sc, (int)st.value[0]);
  } else if (P > kTile) {
    e = radix_sort_rows(logits, row_map, vocab, P, rows, sc, stream);
    if (e != 0) return e;
  } else {
    sort_init_logits_kernel<<<dim3((P + 255) / 256, rows), 256, 0, stream>>>(logits, row_map, vocab, P, sc);
    e = sort_rows(0, vocab, P, P, rows, sc, stream);
    if (e != 0) return e;
    count_finite_kernel<<<dim3((P + 255) / 256, rows), 256, 0, stream>>>(vocab, P, sc);
  }
  int done = 0;
  bool begun = false;
  while (true) {
    int cut = done;
    while (cut < n_stages && st.type[cut] != kTypical) ++cut;
    stages_kernel<<<rows, kThreads, 0, stream>>>(vocab, P, sc, temperature, st, begun ? 0 : 1, done, cut);
    begun = true;
    if (cut >= n_stages) break;
    typical_scores_kernel<<<rows, kThreads, 0, stream>>>(vocab, P, sc);
    e = sort_rows(1, vocab, P, P, rows, sc, stream);
    if (e != 0) return e;
    typical_select_kernel<<<rows, kThreads, 0, stream>>>(vocab, P, sc, st.value[cut]);
    done = cut + 1;
  }
  if (maximum_surprise != nullptr) {
    if (chosen_prob == nullptr) return kRefusedSize;
    surprise_filter_kernel<<<rows, kThreads, 0, stream>>>(vocab, P, sc, maximum_surprise);
  }
  select_kernel<<<rows, kThreads, 0, stream>>>(vocab, P, sc, seeds, positions, out, row_map, probs,
                                               maximum_surprise != nullptr ? chosen_prob : nullptr);
  return (int)cudaGetLastError();
}

// logits: fp32 [.., vocab], changed in place at the n listed (row, token) entries (each at most
// once); counts: occurrences in the row's window (0: only the DRY penalty applies); dry: the DRY
// penalty (0: none); repetition, presence, frequency: fp64 per row.
extern "C" int leone_penalize(float* logits, int vocab, int n, const int* rows, const int* tokens,
                              const int* counts, const double* dry, const double* repetition,
                              const double* presence, const double* frequency, cudaStream_t stream) {
  if (n <= 0) return 0;
  if (vocab <= 0) return kRefusedSize;
  penalize_kernel<<<(n + 255) / 256, 256, 0, stream>>>(logits, vocab, n, rows, tokens, counts, dry, repetition,
                                                      presence, frequency);
  return (int)cudaGetLastError();
}
