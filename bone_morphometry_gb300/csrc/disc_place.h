// Where an overflowing disc list lies: its first entry's index in the pool, kept
// in the first word of the patch's own list.
#pragma once

#include <cuda_runtime.h>

namespace bm {

// The pool of a volume of 2^32 voxels may hold more than 2^32 entries, so its
// segments start at multiples of 4 and a place counts in fours: 2^34 entries.
// (A 64-bit place in both words of the slot cost the painting 0.5 %: 3.89 against
// 3.87 ms for both phases of 512^3.)
constexpr unsigned kPoolAlign = 4;

// Entries of the pool that a list of n takes.
__host__ __device__ inline unsigned disc_segment(unsigned n) { return (n + kPoolAlign - 1) / kPoolAlign * kPoolAlign; }

__host__ __device__ inline unsigned disc_place(unsigned long long first) { return (unsigned)(first / kPoolAlign); }

__host__ __device__ inline unsigned long long disc_first(unsigned place) {
  return (unsigned long long)place * kPoolAlign;
}

}  // namespace bm
