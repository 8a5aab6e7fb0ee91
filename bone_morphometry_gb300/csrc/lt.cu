// Local thickness on sm_103a (local_thickness.rs:16-358): search templates,
// distance ridge, sphere fill, surface cleanup, phase mask and the exact
// statistics of the scaled map (metrics.rs:204-241).
#include "kernels.h"

namespace bm {

namespace {

// floor(sqrt(v)) exactly: float estimate, then integer fix-up (same contract
// as integer_sqrt, local_thickness.rs:339-348).
__device__ __forceinline__ uint32_t isqrt_u32(uint32_t v) {
  uint32_t r = (uint32_t)sqrtf((float)v);
  while ((unsigned long long)(r + 1) * (r + 1) <= v) ++r;
  while ((unsigned long long)r * r > v) --r;
  return r;
}

__device__ __forceinline__ uint32_t csqrt_u32(uint32_t v) {  // ceiling_sqrt, :351-358
  const uint32_t f = isqrt_u32(v);
  return f * f == v ? f : f + 1;
}

// One warp per r^2: lanes split k, loop j; the three offsets of
// create_templates (local_thickness.rs:67-73) share one integer sqrt.
__global__ void __launch_bounds__(256) lut_kernel(uint4* __restrict__ lut, uint32_t lo, uint32_t hi) {
  const int lane = threadIdx.x & 31;
  const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long rr = (long long)lo + wid; rr <= (long long)hi; rr += nwarps) {
    const uint32_t R = (uint32_t)rr;
    const uint32_t rad = isqrt_u32(R) + 1;
    uint32_t m0 = 0, m1 = 0, m2 = 0;
    for (uint32_t k = lane; k <= rad; k += 32) {
      const uint32_t kk = k * k;
      if (kk > R) break;
      const uint32_t k1 = (k + 1) * (k + 1);
      for (uint32_t j = 0; j <= rad; ++j) {
        const uint32_t kj = kk + j * j;
        if (kj > R) break;
        const uint32_t i1 = isqrt_u32(R - kj) + 1;
        const uint32_t ii = i1 * i1;
        const uint32_t j1 = (j + 1) * (j + 1);
        m0 = max(m0, kk + j * j + ii);
        m1 = max(m1, kk + j1 + ii);
        m2 = max(m2, k1 + j1 + ii);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      m0 = max(m0, __shfl_xor_sync(0xffffffffu, m0, o));
      m1 = max(m1, __shfl_xor_sync(0xffffffffu, m1, o));
      m2 = max(m2, __shfl_xor_sync(0xffffffffu, m2, o));
    }
    if (lane == 0) {
      // (2.0_f64 * sqrt(r2 as f64)) as f32, local_thickness.rs:206
      const float dia = __double2float_rn(2.0 * sqrt((double)R));
      lut[R] = make_uint4(m0, m1, m2, __float_as_uint(dia));
    }
  }
}

// One warp per ridge ball; lanes take the (z, y) rows of the clipped box and
// walk their chord |dx| <= isqrt(r2 - dy^2 - dz^2) (local_thickness.rs:172-202).
__global__ void __launch_bounds__(256)
fill_kernel(const uint2* __restrict__ ridges, const Counters* __restrict__ ctr, Dims dm,
            uint32_t* __restrict__ fillmap) {
  const unsigned long long nr = ctr->ridges;
  const int lane = threadIdx.x & 31;
  const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  const long long sl = (long long)dm.w * dm.h;
  for (long long i = wid; i < (long long)nr; i += nwarps) {
    const uint2 rec = ridges[i];
    const long long idx = rec.x;
    const uint32_t R = rec.y;
    const int z = (int)(idx / sl);
    const long long rem = idx - (long long)z * sl;
    const int y = (int)(rem / dm.w);
    const int x = (int)(rem - (long long)y * dm.w);
    const int rad = (int)csqrt_u32(R);
    const int zs = max(z - rad, 0), ze = min(z + rad, dm.d - 1);
    const int ys = max(y - rad, 0), ye = min(y + rad, dm.h - 1);
    const int ny = ye - ys + 1;
    const int rows = (ze - zs + 1) * ny;
    for (int r = lane; r < rows; r += 32) {
      const int zz = zs + r / ny;
      const int yy = ys + r % ny;
      const uint32_t dz = (uint32_t)abs(zz - z), dy = (uint32_t)abs(yy - y);
      const uint32_t dyz = dz * dz + dy * dy;
      if (dyz > R) continue;
      const int half = (int)isqrt_u32(R - dyz);
      const int x0 = max(x - half, 0), x1 = min(x + half, dm.w - 1);
      uint32_t* rowp = fillmap + ((long long)zz * dm.h + yy) * dm.w;
      for (int xx = x0; xx <= x1; ++xx) atomicMax(rowp + xx, R);
    }
  }
}



// NEIGHBORS_26 of local_thickness.rs:285-312 (Fiji's visitation order), which
// fixes the order of the f32 sum in cleanup pass 2; constant so that the
// unrolled loop addresses shared memory with immediate offsets.
__device__ constexpr signed char kN26c[26][3] = {
    {0, 0, -1}, {0, 0, 1},  {0, -1, 0}, {0, 1, 0},   {-1, 0, 0},  {1, 0, 0},  {0, 1, -1},
    {0, 1, 1},  {1, -1, 0}, {1, 1, 0},  {-1, 0, 1},  {1, 0, 1},   {0, -1, -1}, {0, -1, 1},
    {-1, -1, 0}, {-1, 1, 0}, {-1, 0, -1}, {1, 0, -1}, {1, 1, 1},   {1, -1, 1}, {-1, 1, 1},
    {-1, -1, 1}, {1, 1, -1}, {1, -1, -1}, {-1, 1, -1}, {-1, -1, -1}};

// Surface cleanup (local_thickness.rs:210-281), phase mask (:31-43), f32
// calibration and exact moment sums (metrics.rs:215-226).
//
// Pass 1 keeps a nonzero value without a zero 26-neighbour ("interior"); pass 2
// gives every other nonzero voxel the mean diameter of its interior neighbours,
// summed in NEIGHBORS_26 order with IEEE f32 adds and one IEEE division.  Both
// work on row-padded bitmasks (layout of the selection bits): the fill writes
// the diameters 2 sqrt(r^2) and their nonzero mask, interior_kernel erodes the
// mask, and cleanup_kernel reads one diameter per voxel.  Only the selected voxels that are not interior (the phase's skin)
// look at their neighbours; they are collected per warp and handled 32 at a
// time, so that the 26 gathers run on full warps.
//
// Bound by instruction issue (64% active, 47% of the warps).  Per phase, with
// the erosion: 0.44 ms on 512^3 and 3.9 ms on 1024^3, where a fused kernel that
// staged a halo of 2 around 32 x 16 x 8 tiles took 1.35 and 8.6 ms.

// Diameters and nonzero bits of an r^2 map whose fill does not write them (one
// warp per word; dmap may be fm's own memory).
__global__ void __launch_bounds__(256)
diameter_kernel(const uint32_t* fm, Dims dm, long long words, const float* __restrict__ dia, float* dmap,
                uint32_t* __restrict__ nzbits) {
  const int lane = threadIdx.x & 31, nw = dm.nw();
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < words; i += nwarps) {
    const long long row = i / nw;
    const int x = (int)(i - row * nw) * 32 + lane;
    const uint32_t v = x < dm.w ? fm[row * dm.w + x] : 0u;
    if (x < dm.w) dmap[row * dm.w + x] = __ldg(dia + v);
    const unsigned m = __ballot_sync(0xffffffffu, v != 0u);
    if (lane == 0) nzbits[i] = m;
  }
}

// interior = nonzero and no zero 26-neighbour (neighbours outside the volume do
// not count): the nonzero mask eroded by 3 x 3 x 3.  A thread takes one word
// through kErodeZ planes, with each plane's word eroded along x and y once.
constexpr int kErodeZ = 4;

__global__ void __launch_bounds__(256)
interior_kernel(const uint32_t* __restrict__ nzbits, Dims dm, uint32_t* __restrict__ inbits) {
  const int nw = dm.nw();
  const long long cols = (long long)nw * dm.h;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cols) return;
  const int y = (int)(i / nw), c = (int)(i - (long long)y * nw);
  const int z0 = blockIdx.y * kErodeZ, z1 = min(z0 + kErodeZ, dm.d);
  const int tail = dm.w - (nw - 1) * 32;
  const uint32_t beyond = tail < 32 ? ~0u << tail : 0u;  // bits past the row's end, in its last word
  // the word eroded along x and y; own: the word itself
  auto plane = [&](int z, uint32_t& own) -> uint32_t {
    own = 0u;
    if (z < 0 || z >= dm.d) return ~0u;
    uint32_t m = ~0u;
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy) {
      if (y + dy < 0 || y + dy >= dm.h) continue;
      const uint32_t* row = nzbits + ((long long)z * dm.h + y + dy) * nw + c;
      const uint32_t l = c > 0 ? row[-1] : ~0u, r = c + 1 < nw ? row[1] : ~0u;
      uint32_t q = row[0];
      if (dy == 0) own = q;
      if (c + 1 == nw) q |= beyond;
      m &= q & __funnelshift_l(l, q, 1) & __funnelshift_r(q, r, 1);
    }
    return m;
  };
  uint32_t own, next, unused;
  uint32_t lo = plane(z0 - 1, unused), mid = plane(z0, own);
  for (int z = z0; z < z1; ++z) {
    const uint32_t hi = plane(z + 1, next);
    inbits[((long long)z * dm.h + y) * nw + c] = lo & mid & hi & own;
    lo = mid;
    mid = hi;
    own = next;
  }
}

constexpr int kCleanThreads = 256;
constexpr int kCleanWarps = kCleanThreads / 32;
constexpr int kCleanRows = 8;  // rows of 32 voxels a warp takes at a time (their loads are in flight together)

// Exact moment sums of one thread: the values with one f32 exponent are added
// up as mantissas and squared mantissas (a run), and a run joins the fixed-point
// sums, or the block's per-exponent sums outside their span, when it ends.
struct Moments {
  unsigned long long fx1 = 0;
  unsigned __int128 fx2 = 0;
  unsigned long long s1 = 0, s2 = 0;
  uint32_t base = 0, hidden = 0;  // the run's exponent field in place, and its values' hidden bit
  uint32_t mx = 0;

  __device__ __forceinline__ void flush(StatsAccum& sacc, int e_lo) {
    const uint32_t e = max(base >> 23, 1u), sh = e - (uint32_t)e_lo;
    if (sh <= (uint32_t)kFixedSpan) {
      fx1 += s1 << sh;
      fx2 += (unsigned __int128)s2 << (2 * sh);
    } else if (s1) {
      atomicAdd(&sacc.sum_m[e], s1);
      atomicAdd(&sacc.sq_hi[e], s2 >> 24);
      atomicAdd(&sacc.sq_lo[e], s2 & 0xffffffull);
    }
    s1 = s2 = 0;
  }

  // v > 0.  A run must end (flush) within 2^16 values: their squares fill s2.
  __device__ __forceinline__ void add(float v, StatsAccum& sacc, int e_lo) {
    const uint32_t bits = __float_as_uint(v);
    mx = max(mx, bits);
    if (bits - base > 0x7fffffu) {  // another exponent
      flush(sacc, e_lo);
      base = bits & 0xff800000u;
      hidden = base ? 0x800000u : 0u;
    }
    const uint32_t m = (bits - base) + hidden;
    s1 += m;
    s2 += (unsigned long long)m * m;
  }
};

// limb[at ..] += v with carries, by atomics (the total is the same in any order).
__device__ __forceinline__ void add_limbs(unsigned long long* limb, int limbs, int at, unsigned long long v) {
  for (; v && at < limbs; ++at) {
    const unsigned long long old = atomicAdd(&limb[at], v);
    v = old + v < old ? 1ull : 0ull;
  }
}

__global__ void __launch_bounds__(kCleanThreads, 4)
cleanup_kernel(const float* __restrict__ dmap, const uint32_t* __restrict__ selbits,
               const uint32_t* __restrict__ inbits, Dims dm, VoxelDecoder vd, float scale,
               float* __restrict__ outmap, StatsAccum* __restrict__ acc, int e_lo,
               int nyt, long long units) {
  __shared__ StatsAccum sacc;
  __shared__ uint32_t queue[kCleanWarps][32 + 32 * kCleanRows];  // skin voxels a warp holds back until 32 are ready
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned below = (1u << lane) - 1u;
  for (int i = tid; i < 256; i += kCleanThreads) {
    sacc.sum_m[i] = 0;
    sacc.sq_hi[i] = 0;
    sacc.sq_lo[i] = 0;
  }
  if (tid == 0) {
    sacc.count = 0;
    sacc.max_bits = 0;
  }
  __syncthreads();
  const int nw = dm.nw();
  const int slice = dm.w * dm.h;  // < 2^30 (dimensions are at most 32768)
  Moments mom;
  uint32_t count = 0, since = 0;  // this lane's selected voxels; values added since a run was ended for its length
  uint32_t* q = queue[warp];
  int nq = 0;
  const long long nwarps = (long long)gridDim.x * kCleanWarps;
  // a unit: 32 x, kCleanRows rows of one plane
  for (long long u = (long long)blockIdx.x * kCleanWarps + warp;; u += nwarps) {
    const bool done = u >= units;
    if (!done) {
      const int c = (int)(u % nw);
      const long long yz = u / nw;
      const int y0 = (int)(yz % nyt) * kCleanRows, z = (int)(yz / nyt);
      const int rows = min(kCleanRows, dm.h - y0);
      const long long row0 = (long long)z * dm.h + y0;
      const int x = c * 32 + lane;
      uint32_t sel = 0u, keep = 0u, skin = 0u;  // lane r: the words of row r
      if (lane < rows) {
        sel = selbits[(row0 + lane) * nw + c];
        const uint32_t in = inbits[(row0 + lane) * nw + c];
        keep = sel & in;
        skin = sel & ~in;
        count += __popc(sel);  // every selected voxel has a value: its own ball covers it
      }
      const uint32_t first = (uint32_t)(row0 * dm.w) + (uint32_t)x;
      if (!__any_sync(0xffffffffu, sel != 0u)) {  // nothing selected: the masked map is 0
        if (outmap)
          for (int r = 0; r < rows; ++r)
            if (x < dm.w) outmap[first + (uint32_t)(r * dm.w)] = 0.0f;
      } else {
        float d[kCleanRows];
#pragma unroll
        for (int r = 0; r < kCleanRows; ++r)
          d[r] = (__shfl_sync(0xffffffffu, keep, r) >> lane) & 1u ? __ldg(dmap + (first + (uint32_t)(r * dm.w))) : 0.0f;
#pragma unroll
        for (int r = 0; r < kCleanRows; ++r) {
          const uint32_t skins = __shfl_sync(0xffffffffu, skin, r);
          const bool is_skin = (skins >> lane) & 1u;
          const uint32_t at = first + (uint32_t)(r * dm.w);
          if (outmap && r < rows && x < dm.w && !is_skin) outmap[at] = d[r];
          if (d[r] > 0.0f) mom.add(__fmul_rn(d[r], scale), sacc, e_lo);
          if (skins) {
            if (is_skin) q[nq + __popc(skins & below)] = at;
            nq += __popc(skins);
          }
        }
        if ((since += kCleanRows) > 60000u) {
          mom.flush(sacc, e_lo);
          since = 0;
        }
        __syncwarp();
      }
    }
    while (nq >= 32 || (done && nq > 0)) {
      const int take = min(nq, 32);
      nq -= take;
      const uint32_t at = q[nq + min(lane, take - 1)];
      int x, y, z;
      vd(at, x, y, z);
      // interior flags of the 3 x 3 x 3 neighbourhood, bit (dz + 1) * 9 + (dy + 1) * 3 + (dx + 1)
      uint32_t cube = 0;
      const int c0 = (x - 1) >> 5, c1 = (x + 1) >> 5;
#pragma unroll
      for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy) {
          const bool rin = (unsigned)(z + dz) < (unsigned)dm.d && (unsigned)(y + dy) < (unsigned)dm.h;
          const uint32_t* row = inbits + ((long long)(z + dz) * dm.h + (y + dy)) * nw;
          const uint32_t w0 = rin && c0 >= 0 ? row[c0] : 0u, w1 = rin && c1 < nw ? row[c1] : 0u;
          cube |= (__funnelshift_r(w0, w1, (x - 1) & 31) & 7u) << ((dz + 1) * 9 + (dy + 1) * 3);
        }
      // an absent neighbour adds 0, which changes no bit of the sum
      float sum = 0.0f;
      constexpr int kHalf = 13;
#pragma unroll
      for (int h = 0; h < 26; h += kHalf) {
        float g[kHalf];
#pragma unroll
        for (int k = 0; k < kHalf; ++k) {  // NEIGHBORS_26 order (compile-time offsets)
          const int dx = kN26c[h + k][0], dy = kN26c[h + k][1], dz = kN26c[h + k][2];
          const int ci = (dz + 1) * 9 + (dy + 1) * 3 + (dx + 1);
          g[k] = (cube >> ci) & 1u ? __ldg(dmap + (at + (uint32_t)(dz * slice + dy * dm.w + dx))) : 0.0f;
        }
#pragma unroll
        for (int k = 0; k < kHalf; ++k) sum = __fadd_rn(sum, g[k]);
      }
      const float val = cube ? __fdiv_rn(sum, (float)__popc(cube)) : __ldg(dmap + at);
      if (lane < take) {
        if (outmap) outmap[at] = val;
        if (val > 0.0f) mom.add(__fmul_rn(val, scale), sacc, e_lo);
      }
      ++since;
      __syncwarp();
    }
    if (done) break;
  }
  mom.flush(sacc, e_lo);
  if (count) atomicAdd(&sacc.count, (unsigned long long)count);
  if (mom.mx) atomicMax(&sacc.max_bits, mom.mx);
  // this CTA's fixed-point sums
  unsigned long long fx1 = mom.fx1, f2lo = (unsigned long long)mom.fx2, f2hi = (unsigned long long)(mom.fx2 >> 64);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    fx1 += __shfl_xor_sync(0xffffffffu, fx1, o);
    const unsigned long long olo = __shfl_xor_sync(0xffffffffu, f2lo, o);
    const unsigned long long ohi = __shfl_xor_sync(0xffffffffu, f2hi, o);
    const unsigned long long lo = f2lo + olo;
    f2hi += ohi + (lo < f2lo ? 1u : 0u);
    f2lo = lo;
  }
  __shared__ unsigned long long s_fx[kCleanWarps][3];
  if (lane == 0) {
    s_fx[warp][0] = fx1;
    s_fx[warp][1] = f2lo;
    s_fx[warp][2] = f2hi;
  }
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < kCleanWarps; ++w) {
      s_fx[0][0] += s_fx[w][0];
      const unsigned long long lo = s_fx[0][1] + s_fx[w][1];
      s_fx[0][2] += s_fx[w][2] + (lo < s_fx[0][1] ? 1u : 0u);
      s_fx[0][1] = lo;
    }
    add_limbs(acc->fx_s1, 2, 0, s_fx[0][0]);
    add_limbs(acc->fx_s2, 3, 0, s_fx[0][1]);
    add_limbs(acc->fx_s2, 3, 1, s_fx[0][2]);
  }
  for (int i = tid; i < 256; i += kCleanThreads) {
    if (sacc.sum_m[i]) atomicAdd(&acc->sum_m[i], sacc.sum_m[i]);
    if (sacc.sq_hi[i]) atomicAdd(&acc->sq_hi[i], sacc.sq_hi[i]);
    if (sacc.sq_lo[i]) atomicAdd(&acc->sq_lo[i], sacc.sq_lo[i]);
  }
  if (tid == 0) {
    if (sacc.count) atomicAdd(&acc->count, sacc.count);
    if (sacc.max_bits) atomicMax(&acc->max_bits, sacc.max_bits);
  }
}

// Distance ridge (local_thickness.rs:104-167) on 32 x 8 x 8 tiles with the
// distance map staged with a halo of 1 (out-of-volume neighbours are skipped,
// as in the reference's bounds checks).  A selected voxel (d > 0) is a ridge
// unless some 26-neighbour's d reaches the search template of its own r^2
// (offset class = number of nonzero components).
constexpr int kRTX = 32, kRTY = 8, kRTZ = 8;
constexpr int kRSX = kRTX + 2, kRSY = kRTY + 2, kRSZ = kRTZ + 2;

__global__ void __launch_bounds__(256)
ridge_tile_kernel(const uint32_t* __restrict__ dist, const uint32_t* __restrict__ selbits, Dims dm,
                  const uint4* __restrict__ lut, uint2* __restrict__ ridges, Counters* __restrict__ ctr,
                  uint32_t* __restrict__ occ, uint32_t* __restrict__ ridgebits, int ntx, int nty, int ntz) {
  __shared__ uint32_t D[kRSZ * kRSY * kRSX];
  __shared__ uint32_t s_wcnt[8];
  __shared__ unsigned long long s_base;
  __shared__ uint32_t s_tile;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long ntiles = (long long)ntx * nty * ntz;
  const int nw = dm.nw();
  // tiles are taken from a counter as CTAs free up (their costs vary widely)
  for (;;) {
    __syncthreads();  // every thread has read s_tile
    if (tid == 0) s_tile = atomicAdd(&ctr->tile_next, 1u);
    __syncthreads();
    const long long tile = s_tile;
    if (tile >= ntiles) break;
    const int tx = (int)(tile % ntx), ty = (int)((tile / ntx) % nty), tz = (int)(tile / ((long long)ntx * nty));
    const int x0 = tx * kRTX, y0 = ty * kRTY, z0 = tz * kRTZ;
    // ridges are selected voxels: a tile without any has none
    bool any_sel = false;
    if (tid < kRTZ * kRTY) {
      const int z = z0 + tid / kRTY, y = y0 + tid % kRTY;
      if (z < dm.d && y < dm.h) any_sel = selbits[((long long)z * dm.h + y) * nw + tx] != 0u;
    }
    if (!__syncthreads_or(any_sel)) continue;
    // stage the distance map with halo 1: one row of 34 per warp step, loads
    // of all the warp's rows issued before the stores
    constexpr int kRidgeRows = (kRSZ * kRSY + 7) / 8;  // 13 (the last step covers 4 rows)
    constexpr int kRBatch = 5;
#pragma unroll
    for (int b = 0; b < kRidgeRows; b += kRBatch) {
      uint32_t v[kRBatch], v2[kRBatch];
#pragma unroll
      for (int j = 0; j < kRBatch; ++j) {
        const int r = warp + 8 * (b + j);
        const int z = z0 - 1 + r / kRSY, y = y0 - 1 + r % kRSY;
        const bool rin = b + j < kRidgeRows && r < kRSZ * kRSY && z >= 0 && z < dm.d && y >= 0 && y < dm.h;
        const uint32_t* row = dist + ((long long)z * dm.h + y) * dm.w;
        const int x = x0 - 1 + lane, xb = x0 + 31 + lane;
        v[j] = (rin && x >= 0 && x < dm.w) ? row[x] : 0u;
        v2[j] = (lane < 2 && rin && xb < dm.w) ? row[xb] : 0u;
      }
#pragma unroll
      for (int j = 0; j < kRBatch; ++j) {
        const int r = warp + 8 * (b + j);
        if (b + j < kRidgeRows && r < kRSZ * kRSY) {
          uint32_t* srow = D + r * kRSX;
          srow[lane] = v[j];
          if (lane < 2) srow[32 + lane] = v2[j];
        }
      }
    }
    __syncthreads();
    // ridge masks of this warp's 8 rows, then one global slot reservation per tile
    unsigned mk[kRTZ * kRTY / 8];
    int wcount = 0;
#pragma unroll
    for (int k = 0; k < kRTZ * kRTY / 8; ++k) {
      const int r = warp + 8 * k;
      const int oz = r / kRTY, oy = r % kRTY;
      const int z = z0 + oz, y = y0 + oy, x = x0 + lane;
      bool ridge = false;
      if (z < dm.d && y < dm.h && x < dm.w) {
        const int sx = lane + 1, sy = oy + 1, sz = oz + 1;
        const uint32_t R = D[(sz * kRSY + sy) * kRSX + sx];
        if (R > 0u) {
          const uint4 t = lut[R];
          ridge = true;
          // neighbours outside the volume hold 0 and never reach a template (>= 4)
#pragma unroll
          for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
            for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
              for (int dx = -1; dx <= 1; ++dx) {
                if (dx == 0 && dy == 0 && dz == 0) continue;
                const int c = (dx != 0) + (dy != 0) + (dz != 0);
                const uint32_t thr = c == 1 ? t.x : (c == 2 ? t.y : t.z);
                if (D[((sz + dz) * kRSY + sy + dy) * kRSX + sx + dx] >= thr) ridge = false;
              }
        }
      }
      mk[k] = __ballot_sync(0xffffffffu, ridge);
      wcount += __popc(mk[k]);
      if (ridgebits && lane == 0 && z < dm.d && y < dm.h) ridgebits[((long long)z * dm.h + y) * nw + tx] = mk[k];
    }
    if (lane == 0) s_wcnt[warp] = (uint32_t)wcount;
    __syncthreads();
    if (tid == 0) {
      uint32_t tot = 0;
      for (int w = 0; w < 8; ++w) {
        const uint32_t c = s_wcnt[w];
        s_wcnt[w] = tot;
        tot += c;
      }
      s_base = tot ? atomicAdd(&ctr->ridges, (unsigned long long)tot) : 0ull;
    }
    __syncthreads();
    unsigned long long slot = s_base + s_wcnt[warp];
#pragma unroll
    for (int k = 0; k < kRTZ * kRTY / 8; ++k) {
      const unsigned m = mk[k];
      if ((m >> lane) & 1u) {
        const int r = warp + 8 * k;
        const int oz = r / kRTY, oy = r % kRTY;
        const int z = z0 + oz, y = y0 + oy, x = x0 + lane;
        const uint32_t R = D[((oz + 1) * kRSY + oy + 1) * kRSX + lane + 1];
        ridges[slot + __popc(m & ((1u << lane) - 1u))] =
            make_uint2((uint32_t)(((long long)z * dm.h + y) * dm.w + x), R);
        if (occ && occ[R] == 0u) occ[R] = 1u;
      }
      slot += __popc(m);
    }
  }
}

__global__ void dia_extract_kernel(const uint4* __restrict__ lut, uint32_t n, float* __restrict__ dia) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    dia[i] = __uint_as_float(lut[i].w);
}

inline unsigned grid_for(long long work, int per_block, int cap) {
  long long b = (work + per_block - 1) / per_block;
  if (b < 1) b = 1;
  if (b > cap) b = cap;
  return (unsigned)b;
}

}  // namespace

cudaError_t launch_lut(uint4* lut, uint32_t lo, uint32_t hi, cudaStream_t s, unsigned long long* launches) {
  if (hi < lo) return cudaSuccess;
  const long long count = (long long)hi - lo + 1;
  lut_kernel<<<grid_for(count, 8, 152 * 16), 256, 0, s>>>(lut, lo, hi);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launch_dia_table(const uint4* lut, uint32_t n, float* dia, cudaStream_t s, unsigned long long* launches) {
  dia_extract_kernel<<<grid_for(n, 256, 1024), 256, 0, s>>>(lut, n, dia);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launch_ridges(const uint32_t* dist, const uint32_t* selbits, Dims dm, const uint4* lut, uint2* ridges,
                          Counters* ctr, uint32_t* occ, uint32_t* ridgebits, cudaStream_t s,
                          unsigned long long* launches) {
  const int ntx = (dm.w + kRTX - 1) / kRTX, nty = (dm.h + kRTY - 1) / kRTY, ntz = (dm.d + kRTZ - 1) / kRTZ;
  const long long tiles = (long long)ntx * nty * ntz;
  ridge_tile_kernel<<<resident_grid<ridge_tile_kernel>(256, tiles), 256, 0, s>>>(dist, selbits, dm, lut, ridges, ctr,
                                                                                 occ, ridgebits, ntx, nty, ntz);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launch_fill(const uint2* ridges, const Counters* ctr, unsigned long long max_ridges, Dims dm,
                        uint32_t* fillmap, cudaStream_t s, unsigned long long* launches) {
  fill_kernel<<<grid_for((long long)max_ridges, 8, 152 * 32), 256, 0, s>>>(ridges, ctr, dm, fillmap);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launch_diameters(const uint32_t* fillmap, Dims dm, const float* dia, float* dmap, uint32_t* nzbits,
                             cudaStream_t s, unsigned long long* launches) {
  const long long words = (long long)dm.nw() * dm.h * dm.d;
  diameter_kernel<<<grid_for(words, 8, 152 * 16), 256, 0, s>>>(fillmap, dm, words, dia, dmap, nzbits);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launch_cleanup(const float* dmap, const uint32_t* selbits, const uint32_t* nzbits, uint32_t* inbits, Dims dm,
                           float scale, float* outmap, StatsAccum* acc, int e_lo, cudaStream_t s,
                           unsigned long long* launches) {
  const long long cols = (long long)dm.nw() * dm.h;
  interior_kernel<<<dim3((unsigned)((cols + 255) / 256), (unsigned)((dm.d + kErodeZ - 1) / kErodeZ)), 256, 0, s>>>(
      nzbits, dm, inbits);
  const int nyt = (dm.h + kCleanRows - 1) / kCleanRows;
  const long long units = (long long)dm.nw() * nyt * dm.d;
  const unsigned g = resident_grid<cleanup_kernel>(kCleanThreads, (units + kCleanWarps - 1) / kCleanWarps);
  cleanup_kernel<<<g, kCleanThreads, 0, s>>>(dmap, selbits, inbits, dm, VoxelDecoder::of(dm), scale, outmap, acc, e_lo,
                                             nyt, units);
  *launches += 2;
  return cudaGetLastError();
}

}  // namespace bm
