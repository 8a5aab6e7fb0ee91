// Where an overflowing disc list lies: its first entry's index in the pool, kept
// in the first slot of the patch's own list.
#pragma once

#include <cuda_runtime.h>

namespace bm {

// 64 bits: the pool of a volume of 2^32 voxels may hold more than 2^32 entries.
__host__ __device__ inline uint2 disc_place(unsigned long long first) {
  uint2 slot;
  slot.x = (unsigned)first;
  slot.y = (unsigned)(first >> 32);
  return slot;
}

__host__ __device__ inline unsigned long long disc_first(uint2 slot) {
  return ((unsigned long long)slot.y << 32) | slot.x;
}

}  // namespace bm
