// Groups in the order of their first rows, without a sort: when every group's
// first row is a different row of one stream, a bitmap over the stream's rows
// with one bit per group, and the number of bits before a group's own, give
// the group's place.
#pragma once

#include <cstdint>

namespace kdb {

// One word of the bitmap: the bits of 32 rows, and the groups whose first
// row lies before them.
struct FirstWord {
  uint32_t bits;
  uint32_t before;
};
static_assert(sizeof(FirstWord) == 8, "FirstWord layout");

constexpr int kOrderThreads = 256;
constexpr int kOrderWords = 4 * kOrderThreads;  // bitmap words per CTA (one chunk)
constexpr int64_t kOrderRows = 32LL * kOrderWords;  // rows of one chunk

// One CTA of kOrderThreads threads fills `before` in the words of chunk
// `chunk` (counted from `first_chunk`, whose words start at `w`); the
// counts of bits of the chunks before it are groups[first_chunk ... chunk).
// Every thread returns the number of bits up to and including its own words
// (the last thread's of the last chunk is the total).
__device__ __forceinline__ uint32_t OrderChunk(FirstWord* __restrict__ w, const uint32_t* __restrict__ groups,
                                               int first_chunk, int chunk) {
  __shared__ uint32_t earlier[kOrderThreads / 32], wsum[kOrderThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t e = 0;
  for (int c = first_chunk + threadIdx.x; c < chunk; c += kOrderThreads) e += groups[c];
  uint4* v = reinterpret_cast<uint4*>(w + static_cast<int64_t>(chunk - first_chunk) * kOrderWords + 4 * threadIdx.x);
  uint4 a = v[0], b = v[1];  // two words each
  const uint32_t c0 = __popc(a.x), c1 = __popc(a.z), c2 = __popc(b.x), c3 = __popc(b.z);
  const uint32_t mine = c0 + c1 + c2 + c3;
  uint32_t incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
    e += __shfl_xor_sync(0xffffffffu, e, o);
  }
  if (lane == 31) wsum[warp] = incl;
  if (lane == 0) earlier[warp] = e;
  __syncthreads();
  uint32_t run = incl - mine;
  for (int k = 0; k < kOrderThreads / 32; k++) run += earlier[k] + (k < warp ? wsum[k] : 0u);
  a.y = run;
  a.w = run + c0;
  b.y = run + c0 + c1;
  b.w = run + c0 + c1 + c2;
  v[0] = a;
  v[1] = b;
  return run + mine;
}

}  // namespace kdb
