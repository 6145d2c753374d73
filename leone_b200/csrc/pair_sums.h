// The order in which the two epilogue warps of a quarter (32 token rows) of a pair's tile pass a tile's sums of squares: the second
// warp writes its half's sums and arrives on a barrier, the first waits for it and adds its own.  Plain C++, host and device
// (the hand-over can be walked through without a GPU).
//
// One barrier and one place in shared memory for each accumulator buffer and quarter.  A warp counts the hand-overs in which it took
// part, per buffer, and not the block's tiles: where the 32 rows lie past the last token there is none.  (Both warps of a quarter
// skip the same tiles.)  The barrier cannot complete twice before it is waited for: the second warp comes to a buffer
// again only after the first has released it, which it does behind its wait.
#pragma once

#ifdef __CUDACC__
#define LEONE_HD __host__ __device__ __forceinline__
#else
#define LEONE_HD inline
#endif

namespace leone {

constexpr int kSumsBarriers = 8;      // two buffers by four quarters

struct SumsHandover {
  unsigned phases = 0;                // bit b: parity of the next hand-over in buffer b

  LEONE_HD static int place(int buf, int quarter) { return buf * 4 + quarter; }
  // This warp's next hand-over in the buffer: the parity to wait for.
  LEONE_HD unsigned next(int buf) {
    const unsigned parity = (phases >> buf) & 1u;
    phases ^= 1u << buf;
    return parity;
  }
};

}  // namespace leone
