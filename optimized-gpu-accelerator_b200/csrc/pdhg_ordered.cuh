// Sums in a fixed serial order: one block per sum.
//
// A sum whose every partial result is defined (left to right from zero, each
// step rounded) is a chain of dependent additions, so one thread adds.  What
// a lone thread reading global memory pays beside that chain is one load
// latency per few terms (34 ns a term measured for the power iteration's
// norms: 1,076 us for 24 LPs of up to 31,250 columns).  Here the block's
// other warps fetch the next kOrderedChunk terms, coalesced, into shared
// memory while thread 0 folds the current ones from there: the chain alone is
// left (the same norms: 159 us, 10 cycles a term; the certified bound of 61
// cases over 5,220 terms, with directed rounding: 1,002 -> 78 us).
#pragma once

#include <cstdint>

namespace b2p {

constexpr int kOrderedThreads = 128;
constexpr int kOrderedChunk = 1024;

// load(i): term i (any thread but those of warp 0); fold(s, terms, count):
// the sum s after `count` more terms (thread 0).  The result is valid on
// thread 0.  Every thread of the block (kOrderedThreads) must call.
template <class Load, class Fold>
__device__ __forceinline__ double ordered_sum(int64_t len, Load&& load, Fold&& fold) {
  __shared__ __align__(16) double buf[2][kOrderedChunk];
  double s = 0.0;
  const int64_t chunks = (len + kOrderedChunk - 1) / kOrderedChunk;
  // step c fetches chunk c and folds chunk c - 1
  for (int64_t c = 0; c <= chunks; ++c) {
    if (threadIdx.x >= 32) {
      const int64_t beg = c * kOrderedChunk;
      const int64_t end = beg + kOrderedChunk < len ? beg + kOrderedChunk : len;
      for (int64_t i = beg + threadIdx.x - 32; i < end; i += kOrderedThreads - 32) buf[c & 1][i - beg] = load(i);
    } else if (threadIdx.x == 0 && c > 0) {
      const int64_t left = len - (c - 1) * kOrderedChunk;
      s = fold(s, buf[(c - 1) & 1], static_cast<int>(left < kOrderedChunk ? left : kOrderedChunk));
    }
    __syncthreads();
  }
  return s;
}

}  // namespace b2p
