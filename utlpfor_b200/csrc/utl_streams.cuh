// utl_streams.cuh -- the stream of a block in a batch's table.
#pragma once
#include "utl_device.cuh"

namespace utl {

// Stream of block b (largest s with block_start[s] <= b).
__device__ __forceinline__ int stream_of(const uint64_t* bstart, int n_streams, int64_t b) {
  int lo = 0, hi = n_streams;
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if ((int64_t)bstart[mid] <= b) lo = mid;
    else hi = mid;
  }
  return lo;
}
// The same by the whole warp, each round probing 32 evenly spaced streams at
// once: two dependent loads for 1000 streams where the bisection takes ten.
__device__ __forceinline__ int warp_stream_of(const uint64_t* bstart, int n_streams, int64_t b, int lane) {
  int lo = 0, hi = n_streams;
  while (hi - lo > 1) {
    const int step = (hi - lo + 31) >> 5;
    const int64_t p = (int64_t)lo + (int64_t)lane * step;
    const unsigned m = __ballot_sync(kFull, p < hi && (lane == 0 || (int64_t)bstart[p] <= b));
    lo += (31 - __clz(m)) * step;
    hi = min(hi, lo + step);
  }
  return lo;
}
// The same, knowing the stream s0 of an earlier block: galloping from s0
// (consecutive blocks are nearly always in the same or the next stream).
__device__ __forceinline__ int stream_from(const uint64_t* bstart, int n_streams, int s0, int64_t b) {
  int lo = s0, step = 1;
  while (lo + step < n_streams && (int64_t)bstart[lo + step] <= b) {
    lo += step;
    step <<= 1;
  }
  int hi = min(n_streams, lo + step);
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if ((int64_t)bstart[mid] <= b) lo = mid;
    else hi = mid;
  }
  return lo;
}
}  // namespace utl
