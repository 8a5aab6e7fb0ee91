// Byte volumes at any address, read as aligned words.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace bm {

// A byte volume at any address, read as aligned words.
struct ByteVolume {
  const uint32_t* words;  // the word that holds the first byte
  int lead;               // bytes of it before the first
  long long end;          // one past the last byte, from words
  __device__ ByteVolume(const uint8_t* p, long long n)
      : words(reinterpret_cast<const uint32_t*>(p - (reinterpret_cast<uintptr_t>(p) & 3u))),
        lead((int)(reinterpret_cast<uintptr_t>(p) & 3u)),
        end(n + lead) {}
};

// A word that the volume does not fill, from the bytes it has (0 for the others).
static __device__ __noinline__ uint32_t edge_word(const uint32_t* words, int lead, long long end, long long k) {
  uint32_t w = 0u;
  for (int j = 0; j < 4; ++j) {
    const long long i = 4 * k + j;
    if (i >= lead && i < end) w |= (uint32_t) reinterpret_cast<const uint8_t*>(words)[i] << (8 * j);
  }
  return w;
}

// Bytes at .. at + 15 of the volume (0 past its end).  Five word loads a lane
// measured faster than one 16-byte load and the next lane's words by shuffles (x
// pass of 417 x 333 x 379 79 against 91 us).
__device__ __forceinline__ uint4 load16(const ByteVolume& v, long long at) {
  const long long k = (at + v.lead) >> 2;
  const uint32_t by = (uint32_t)(at + v.lead) % 4u * 8u;
  uint32_t w[5];
  if (4 * k >= v.lead && 4 * k + 20 <= v.end) {
#pragma unroll
    for (int j = 0; j < 5; ++j) w[j] = __ldg(v.words + k + j);
  } else {
#pragma unroll 1
    for (int j = 0; j < 5; ++j) {
      const uint32_t e = edge_word(v.words, v.lead, v.end, k + j);
#pragma unroll
      for (int i = 0; i < 5; ++i) w[i] = i == j ? e : w[i];
    }
  }
  return make_uint4(__funnelshift_r(w[0], w[1], by), __funnelshift_r(w[1], w[2], by), __funnelshift_r(w[2], w[3], by),
                    __funnelshift_r(w[3], w[4], by));
}

}  // namespace bm
