// How far a disc's planes and a chord's rows reach before a neighbour's cover them.
#pragma once

#include <cuda_runtime.h>

namespace bm {

// The last t with a disc (or chord) of squared radius rho - t^2 not covered by
// that of the neighbour one step up, rho' - (t - 1)^2, gain = rho' - rho: covered
// where gain >= 1 - 2 t, or (not strict: an equal value) where gain > 1 - 2 t.
__host__ __device__ inline int cut_above(int gain, bool larger) {
  return larger ? -((gain - 1) >> 1) - 1 : (1 - gain) >> 1;
}
// The first t not covered by the neighbour one step down: covered where gain >= 1 + 2 t.
__host__ __device__ inline int cut_below(int gain) { return (gain + 1) >> 1; }

}  // namespace bm
