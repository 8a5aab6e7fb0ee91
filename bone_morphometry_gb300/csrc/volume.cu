// Voxel counts of volume_metrics (metrics.rs:123-132, 166-202).
//
// The first kernel packs the ROI and the ROI-clipped bone into bitmasks, 16
// voxels per lane and rows of a warp (or less), at any address, and counts both; the
// second finds the boundary voxels 32 at a time from seven words.  The inputs
// are read once (2 bytes a voxel); the masks, an eighth of that, stay in L2.
// 430 x 389 x 401: 611 us a voxel per thread with byte loads, 92 four voxels per
// thread with the neighbours from L1 and L2, 70 here.
#include "bytes.h"
#include "kernels.h"

namespace bm {

namespace {

constexpr int kPackWarps = 8;
constexpr int kEdgeZ = 8;  // planes a thread counts

// Bit i: byte i is not 0.
__device__ __forceinline__ uint32_t nonzero4(uint32_t v) {
  return ((__vcmpne4(v, 0u) & 0x01010101u) * 0x01020408u) >> 24 & 0xfu;
}
__device__ __forceinline__ uint32_t nonzero16(const uint4& v) {
  return nonzero4(v.x) | (nonzero4(v.y) << 4) | (nonzero4(v.z) << 8) | (nonzero4(v.w) << 12);
}

// Adds the block's sum of v to *out.
__device__ __forceinline__ void add_block(uint32_t v, unsigned long long* out) {
  __shared__ unsigned long long part[kPackWarps];
  unsigned long long t = v;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kPackWarps; ++w) t += part[w];
    if (t) atomicAdd(out, t);
  }
}

// 2^LG lanes take a row (an even number, of which pairs make a word), so that a
// warp takes several rows of a narrow volume: 512 x 512 x 2 73 us with a warp per
// row, 20 here, 512 x 512 x 128 74 and 32.
template <int LG>
__global__ void __launch_bounds__(kPackWarps * 32)
pack_rows_kernel(const uint8_t* __restrict__ bone, const uint8_t* __restrict__ roi, Dims dm,
                 uint32_t* __restrict__ rbits, uint32_t* __restrict__ bbits, unsigned long long* __restrict__ out) {
  const ByteVolume vr(roi, dm.n()), vb(bone, dm.n());
  const int lane = threadIdx.x & 31, nw = dm.nw(), nvec = (dm.w + 15) >> 4;
  constexpr int kSeg = 1 << LG;
  const long long rows = (long long)dm.h * dm.d;
  uint32_t n_roi = 0, n_bone = 0;  // 2^32 voxels over many threads: 32 bits hold a thread's
  for (long long row0 = (long long)blockIdx.x * kPackWarps + (threadIdx.x >> 5); (row0 << (5 - LG)) < rows;
       row0 += (long long)gridDim.x * kPackWarps) {
    const long long row = (row0 << (5 - LG)) + (lane >> LG);
    for (int v0 = 0; v0 < nvec; v0 += kSeg) {
      const int v = LG == 5 || row < rows ? v0 + (lane & (kSeg - 1)) : nvec;
      uint32_t r = 0, b = 0;
      if (v < nvec) {
        const long long at = row * dm.w + 16 * v;
        const uint4 R = load16(vr, at), B = load16(vb, at);
        r = nonzero16(R) & (dm.w - 16 * v >= 16 ? 0xffffu : (1u << (dm.w - 16 * v)) - 1u);  // voxels of this row
        b = nonzero16(B) & r;
      }
      const uint32_t both = r | (b << 16), next = __shfl_down_sync(0xffffffffu, both, 1);
      n_roi += __popc(r);
      n_bone += __popc(b);
      if (!(lane & 1) && v < nvec) {  // an odd number of 16-voxel groups ends on a half word: its upper half is empty
        const uint32_t up = v + 1 < nvec ? next : 0u;
        rbits[row * nw + (v >> 1)] = __byte_perm(both, up, 0x5410);
        bbits[row * nw + (v >> 1)] = __byte_perm(both, up, 0x7632);
      }
    }
  }
  add_block(n_roi, out);
  add_block(n_bone, out + 1);
}

__global__ void __launch_bounds__(kPackWarps * 32)
boundary_kernel(const uint32_t* __restrict__ rbits, const uint32_t* __restrict__ bbits, Dims dm,
                unsigned long long* __restrict__ out) {
  const int nw = dm.nw(), plane = nw * dm.h;  // < 2^26
  const int p = blockIdx.x * (kPackWarps * 32) + threadIdx.x;
  const int z1 = min(((int)blockIdx.y + 1) * kEdgeZ, dm.d);
  uint32_t n = 0;
  if (p < plane) {
    const int c = p % nw;
    for (int z = blockIdx.y * kEdgeZ; z < z1; ++z) {
      const long long i = (long long)z * plane + p;
      const uint32_t b = bbits[i];
      if (!b) continue;
      const uint32_t r = rbits[i];
      // what lies outside the volume is outside the ROI
      uint32_t inner = (r << 1 | (c > 0 ? rbits[i - 1] >> 31 : 0u)) & (r >> 1 | (c + 1 < nw ? rbits[i + 1] << 31 : 0u));
      inner &= (p >= nw ? rbits[i - nw] : 0u) & (p + nw < plane ? rbits[i + nw] : 0u);
      inner &= (z > 0 ? rbits[i - plane] : 0u) & (z + 1 < dm.d ? rbits[i + plane] : 0u);
      n += __popc(b & ~inner);
    }
  }
  add_block(n, out + 2);
}

}  // namespace

namespace {
// The fewest lanes that hold a row.
template <int LG>
void pack_rows(const uint8_t* bone, const uint8_t* roi, Dims dm, uint32_t* rbits, uint32_t* bbits,
               unsigned long long* out, cudaStream_t s) {
  if constexpr (LG < 5) {
    if (dm.w > 16 << LG) return pack_rows<LG + 1>(bone, roi, dm, rbits, bbits, out, s);
  }
  constexpr long long kRows = kPackWarps << (5 - LG);  // of a block
  long long blocks = ((long long)dm.h * dm.d + kRows - 1) / kRows;
  if (blocks > 152 * 12) blocks = 152 * 12;
  pack_rows_kernel<LG><<<(unsigned)blocks, kPackWarps * 32, 0, s>>>(bone, roi, dm, rbits, bbits, out);
}
}  // namespace

cudaError_t launch_volume_counts(const uint8_t* bone, const uint8_t* roi, Dims dm, uint32_t* rbits, uint32_t* bbits,
                                 unsigned long long* out, cudaStream_t s, unsigned long long* launches) {
  pack_rows<1>(bone, roi, dm, rbits, bbits, out, s);
  const int plane = dm.nw() * dm.h;
  boundary_kernel<<<dim3((unsigned)((plane + kPackWarps * 32 - 1) / (kPackWarps * 32)),
                         (unsigned)((dm.d + kEdgeZ - 1) / kEdgeZ)),
                    kPackWarps * 32, 0, s>>>(rbits, bbits, dm, out);
  *launches += 2;
  return cudaGetLastError();
}

}  // namespace bm
