// Exact squared Euclidean distance transform on sm_103a (edt.rs:57-156).
//
// The reference computes the Felzenszwalb-Huttenlocher lower envelope in f64
// with INF = 1e30 and rounds; on integer inputs every comparison it makes is
// exact and INF parabolas never reach the envelope inside a line that has a
// finite one, so its output is the mathematically exact squared EDT.  The GPU
// computes the same values with integers only:
//   pass x : distance to the nearest non-selected voxel of the row, from a
//            bitmask of the row (ballot + clz/ffs), squared;
//   pass y, z : lower envelope of the parabolas (q - p)^2 + f(p) with the
//            intersection test done by int64 cross-multiplication; lines
//            whose every entry is "no site" (kInfSq) stay kInfSq.
#include <cuda.h>  // CUtensorMap and its enums (types only; the encoder comes from the runtime)
#include <cudaTypedefs.h>

#include <climits>
#include <cstdint>

#include "bytes.h"
#include "kernels.h"

namespace bm {

namespace {

template <int MODE>
__device__ __forceinline__ bool selected_at(const uint8_t* __restrict__ a, const uint8_t* __restrict__ b,
                                            long long i) {
  if (MODE == SEL_FOREGROUND) return a[i] != 0;
  if (MODE == SEL_BACKGROUND) return a[i] == 0;
  if (MODE == SEL_BONE_IN_ROI) return b[i] != 0 && a[i] != 0;
  return b[i] != 0 && a[i] == 0;
}

constexpr int kXWarps = 8;
constexpr int kXMaxSmem = kXWarps * 3 * 1024 * 4;  // rows of 32768 voxels
constexpr int kNoLeft = -(1 << 20);  // sentinels: no site on that side (w <= 32768)
constexpr int kNoRight = 1 << 21;

// Second half of the x pass for one row whose site bitmask (1 = non-selected
// voxel) is in mask[0 .. nw): two warp scans give lastpos[c], the highest
// site position in words <= c, and firstpos[c], the lowest in words >= c, so
// that every voxel finds its nearest site on each side without branching:
// inside its own word from the bits below / above it, else from the neighbour
// word's entry.
__device__ __forceinline__ void x_row_scans(const uint32_t* mask, int* lastpos, int* firstpos, int nw, int lane) {
  int carry = kNoLeft;
  for (int c0 = 0; c0 < nw; c0 += 32) {
    const int c = c0 + lane;
    const uint32_t m = c < nw ? mask[c] : 0u;
    int v = m ? c * 32 + 31 - __clz(m) : kNoLeft;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v = max(v, t);
    }
    v = max(v, carry);
    if (c < nw) lastpos[c] = v;
    carry = __shfl_sync(0xffffffffu, v, 31);
  }
  carry = kNoRight;
  for (int c0 = ((nw - 1) >> 5) << 5; c0 >= 0; c0 -= 32) {
    const int c = c0 + lane;
    const uint32_t m = c < nw ? mask[c] : 0u;
    int v = m ? c * 32 + __ffs(m) - 1 : kNoRight;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_down_sync(0xffffffffu, v, o);
      if (lane + o < 32) v = min(v, t);
    }
    v = min(v, carry);
    if (c < nw) firstpos[c] = v;
    carry = __shfl_sync(0xffffffffu, v, 0);
  }
  __syncwarp();
}

// Squared distance of voxel x to the nearer of its sites left / right
// (kInfSq when neither exists; 0 when x is a site).
__device__ __forceinline__ uint32_t x_dist(bool site, int x, int left, int right) {
  const int g = min(x - left, right - x);
  return site ? 0u : (g >= (1 << 20) ? kInfSq : (uint32_t)g * (uint32_t)g);
}

// One voxel per lane per word: one coalesced 128-byte store per word.
__device__ __forceinline__ void x_row_distances(const uint32_t* mask, int* lastpos, int* firstpos, int nw, int w,
                                                int lane, uint32_t* __restrict__ orow) {
  x_row_scans(mask, lastpos, firstpos, nw, lane);
  const uint32_t below = (1u << lane) - 1u, above = ~((2u << lane) - 1u);  // lane 31: above = 0
#pragma unroll 1
  for (int c = 0; c < nw; ++c) {
    const int x = c * 32 + lane;
    const uint32_t m = mask[c];
    const int lprev = c > 0 ? lastpos[c - 1] : kNoLeft;
    const int rnext = c + 1 < nw ? firstpos[c + 1] : kNoRight;
    const uint32_t lo = m & below, hi = m & above;
    const int left = lo ? c * 32 + 31 - __clz(lo) : lprev;
    const int right = hi ? c * 32 + __ffs(hi) - 1 : rnext;
    if (x < w) orow[x] = x_dist((m >> lane) & 1u, x, left, right);
  }
  __syncwarp();
}

// Four adjacent voxels per lane (rows whose length is a multiple of 16 and
// whose start is 16-byte aligned): the nearest site left of the first voxel
// and right of the last come from the word and scan entries as above, the
// others follow from the three bits between them; one 16-byte store per lane,
// 512 bytes per warp.
__device__ __forceinline__ void x_row_distances4(const uint32_t* mask, int* lastpos, int* firstpos, int nw, int w,
                                                 int lane, uint32_t* __restrict__ orow) {
  x_row_scans(mask, lastpos, firstpos, nw, lane);
  const int b = (lane & 7) * 4;  // first bit of this lane's voxels in their word
  const uint32_t below = (1u << b) - 1u, above = ~((2u << (b + 3)) - 1u);  // b + 3 = 31: above = 0
#pragma unroll 1
  for (int x0 = 0; x0 < w; x0 += 128) {
    const int x = x0 + 4 * lane;
    if (x < w) {
      const int c = x >> 5;
      const uint32_t m = mask[c];
      const int cb = c * 32 + b;
      const uint32_t lo = m & below, hi = m & above;
      const int l0 = lo ? c * 32 + 31 - __clz(lo) : (c > 0 ? lastpos[c - 1] : kNoLeft);
      const int r3 = hi ? c * 32 + __ffs(hi) - 1 : (c + 1 < nw ? firstpos[c + 1] : kNoRight);
      const uint32_t bits = m >> b;  // this lane's 4 voxels in bits 0..3
      const int l1 = (bits & 1u) ? cb : l0;
      const int l2 = (bits & 2u) ? cb + 1 : l1;
      const int l3 = (bits & 4u) ? cb + 2 : l2;
      const int r2 = (bits & 8u) ? cb + 3 : r3;
      const int r1 = (bits & 4u) ? cb + 2 : r2;
      const int r0 = (bits & 2u) ? cb + 1 : r1;
      uint4 v;
      v.x = x_dist(bits & 1u, x, l0, r0);
      v.y = x_dist(bits & 2u, x + 1, l1, r1);
      v.z = x_dist(bits & 4u, x + 2, l2, r2);
      v.w = x_dist(bits & 8u, x + 3, l3, r3);
      *reinterpret_cast<uint4*>(orow + x) = v;
    }
  }
  __syncwarp();
}

// One warp per x row.  Shared memory per warp: site bitmask of the row and, per
// word, the nearest site position at-or-before / at-or-after it.
template <int MODE>
__global__ void __launch_bounds__(kXWarps * 32)
edt_x_kernel(const uint8_t* __restrict__ a, const uint8_t* __restrict__ b, Dims dm, uint32_t* __restrict__ out,
             uint32_t* __restrict__ selbits, Counters* __restrict__ ctr) {
  extern __shared__ uint32_t smem[];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nw = dm.nw();
  uint32_t* mask = smem + (size_t)warp * 3 * nw;
  int* lastpos = reinterpret_cast<int*>(mask + nw);
  int* firstpos = lastpos + nw;
  const long long rows = (long long)dm.h * dm.d;
  unsigned long long sites = 0;

  for (long long row = (long long)blockIdx.x * kXWarps + warp; row < rows;
       row += (long long)gridDim.x * kXWarps) {
    const long long base = row * dm.w;
    for (int c = 0; c < nw; ++c) {
      const int x = c * 32 + lane;
      const bool in = x < dm.w;
      const bool s = in && selected_at<MODE>(a, b, base + x);
      const unsigned site = __ballot_sync(0xffffffffu, in && !s);
      const unsigned selw = __ballot_sync(0xffffffffu, s);
      if (lane == 0) {
        mask[c] = site;
        selbits[row * nw + c] = selw;
        sites += __popc(site);
      }
    }
    __syncwarp();
    x_row_distances(mask, lastpos, firstpos, nw, dm.w, lane, out + base);
  }
  if (lane == 0 && sites) atomicAdd(&ctr->sites, sites);
}

// 4-bit selection mask of the 4 voxels in a (bone) and b (roi) words:
// per byte, the MODE predicate, packed to bits 0..3.
template <int MODE>
__device__ __forceinline__ uint32_t sel4(uint32_t a, uint32_t b) {
  const uint32_t nza = __vcmpne4(a, 0u), nzb = __vcmpne4(b, 0u);  // 0xff per nonzero byte
  uint32_t m;
  if (MODE == SEL_FOREGROUND) m = nza;
  else if (MODE == SEL_BACKGROUND) m = ~nza;
  else if (MODE == SEL_BONE_IN_ROI) m = nzb & nza;
  else m = nzb & ~nza;
  m &= 0x01010101u;
  return (m * 0x01020408u) >> 24 & 0xfu;  // bytes 0..3 -> bits 0..3
}

// The x pass for rows whose bytes are 16-byte aligned (w a multiple of 16 and
// aligned inputs): each lane loads 16 voxels of bone and roi at once and the
// lanes' 16-bit masks pair up into the row's 32-bit words; the distances are
// then computed four adjacent voxels per lane (16-byte stores).
template <int MODE>
__global__ void __launch_bounds__(kXWarps * 32, 5)
edt_x_vec_kernel(const uint8_t* __restrict__ a, const uint8_t* __restrict__ b, Dims dm, uint32_t* __restrict__ out,
                 uint32_t* __restrict__ selbits, Counters* __restrict__ ctr) {
  extern __shared__ uint32_t smem[];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nw = dm.nw();
  uint32_t* mask = smem + (size_t)warp * 3 * nw;
  int* lastpos = reinterpret_cast<int*>(mask + nw);
  int* firstpos = lastpos + nw;
  const long long rows = (long long)dm.h * dm.d;
  const bool two = MODE == SEL_BONE_IN_ROI || MODE == SEL_MARROW_IN_ROI;
  unsigned long long sites = 0;

  for (long long row = (long long)blockIdx.x * kXWarps + warp; row < rows;
       row += (long long)gridDim.x * kXWarps) {
    const long long base = row * dm.w;
    const uint4* av = reinterpret_cast<const uint4*>(a + base);
    const uint4* bv = two ? reinterpret_cast<const uint4*>(b + base) : nullptr;
    const int nvec = dm.w >> 4;  // 16 voxels per uint4
    for (int v0 = 0; v0 < nvec; v0 += 32) {
      const int v = v0 + lane;
      uint32_t s16 = 0, t16 = 0;
      if (v < nvec) {
        const uint4 A = av[v];
        const uint4 B = two ? bv[v] : make_uint4(0u, 0u, 0u, 0u);
        s16 = sel4<MODE>(A.x, B.x) | (sel4<MODE>(A.y, B.y) << 4) | (sel4<MODE>(A.z, B.z) << 8) |
              (sel4<MODE>(A.w, B.w) << 12);
        t16 = ~s16 & 0xffffu;  // all 16 voxels lie inside the row
      }
      const uint32_t s_hi = __shfl_down_sync(0xffffffffu, s16, 1);
      const uint32_t t_hi = __shfl_down_sync(0xffffffffu, t16, 1);
      if (!(lane & 1) && v < nvec) {
        const int c = v >> 1;  // word index: voxels 32c .. 32c + 31
        // a row of 16k voxels with k odd ends on a half word: its upper half is empty
        const bool full = v + 1 < nvec;
        const uint32_t sw = s16 | (full ? s_hi << 16 : 0u);
        const uint32_t tw = t16 | (full ? t_hi << 16 : 0u);
        mask[c] = tw;
        selbits[row * nw + c] = sw;
        sites += __popc(tw);
      }
    }
    __syncwarp();
    x_row_distances4(mask, lastpos, firstpos, nw, dm.w, lane, out + base);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sites += __shfl_xor_sync(0xffffffffu, sites, o);
  if (lane == 0 && sites) atomicAdd(&ctr->sites, sites);
}

// One thread per line; consecutive threads take consecutive x so that every
// load and store of the line data is a coalesced row.  The envelope stack
// (position, f) lives in global scratch, k-major, and is cached by L1/L2.
// Out uint16_t: a map with strides of its own, values beyond 16 bits cut to
// 0xffff, beside the whole values in wide (at in's strides).
template <class Out>
__global__ void __launch_bounds__(256)
edt_line_kernel(const uint32_t* __restrict__ in, Out* __restrict__ out, uint32_t* __restrict__ wide, int n,
                long long stride, int w, long long outer, long long out_stride, long long out_outer, long long nlines,
                uint32_t* __restrict__ spos, uint32_t* __restrict__ sf, Counters* __restrict__ ctr, int track_max,
                const uint8_t* __restrict__ only) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t localmax = 0;
  if (t < nlines && (only == nullptr || only[t])) {
    const long long base = (t / w) * outer + (t % w);
    Out* to = out + (t / w) * out_outer + (t % w);
    auto put = [&](int q, uint32_t v) {
      to[(long long)q * out_stride] = (Out)(sizeof(Out) == 2 ? min(v, 0xffffu) : v);
      if (sizeof(Out) == 2) wide[base + (long long)q * stride] = v;
    };
    int k = -1;
    long long p1 = 0, F1 = 0;  // stack top
    long long p0 = 0, F0 = 0;  // entry below the top (valid when k >= 1)
    constexpr int kAhead = 4;  // inputs in flight
    uint32_t next[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) next[u] = u < n ? in[base + (long long)u * stride] : kInfSq;
    for (int q = 0; q < n; ++q) {
      const uint32_t fq = next[0];
#pragma unroll
      for (int u = 0; u + 1 < kAhead; ++u) next[u] = next[u + 1];
      next[kAhead - 1] = q + kAhead < n ? in[base + (long long)(q + kAhead) * stride] : kInfSq;
      if (fq == kInfSq) continue;
      const long long Fq = (long long)fq + (long long)q * q;
      while (k >= 1 && (Fq - F1) * (p1 - p0) <= (F1 - F0) * ((long long)q - p1)) {
        --k;
        p1 = p0;
        F1 = F0;
        if (k >= 1) {
          p0 = spos[(long long)(k - 1) * nlines + t];
          F0 = (long long)sf[(long long)(k - 1) * nlines + t] + p0 * p0;
        }
      }
      ++k;
      spos[(long long)k * nlines + t] = (uint32_t)q;
      sf[(long long)k * nlines + t] = fq;
      p0 = p1;
      F0 = F1;
      p1 = q;
      F1 = Fq;
    }
    if (k < 0) {
      for (int q = 0; q < n; ++q) put(q, kInfSq);
    } else {
      int j = 0;
      long long pj = spos[t];
      uint32_t fj = sf[t];
      long long Fj = (long long)fj + pj * pj;
      long long pn = 0, Fn = 0;
      uint32_t fn = 0;
      if (k >= 1) {
        pn = spos[nlines + t];
        fn = sf[nlines + t];
        Fn = (long long)fn + pn * pn;
      }
      for (int q = 0; q < n; ++q) {
        while (j < k && (Fn - Fj) < 2LL * q * (pn - pj)) {
          ++j;
          pj = pn;
          fj = fn;
          Fj = Fn;
          if (j < k) {
            pn = spos[(long long)(j + 1) * nlines + t];
            fn = sf[(long long)(j + 1) * nlines + t];
            Fn = (long long)fn + pn * pn;
          }
        }
        const long long dq = q - pj;
        const uint32_t v = (uint32_t)(dq * dq) + fj;
        put(q, v);
        localmax = max(localmax, v);
      }
    }
  }
  if (track_max) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) localmax = max(localmax, __shfl_xor_sync(0xffffffffu, localmax, o));
    if ((threadIdx.x & 31) == 0 && localmax) atomicMax(&ctr->rmax, localmax);
  }
}

// Windowed y / z pass.  d(q) = min_p (q - p)^2 + f(p), and p = q already gives
// f(q), so only |q - p| <= isqrt(f(q) - 1) can improve it: every output is an
// exact minimum over a window whose width is bounded by its own input value.
// A CTA owns 32 consecutive x of one line-row and kWinTL consecutive outputs
// along the axis; it stages those inputs in shared memory as 128-byte rows,
// then a halo on each side as wide as the largest window it needs (at most
// kWinHalo).  Each lane computes four adjacent outputs q .. q+3 of its column
// at once: the loads at q - e and q + 3 + e serve all four (at distances
// k + e and 3 - k + e for output q + k), so a scan step costs two shared loads
// for four outputs.  The scan runs outwards until e^2 reaches the largest of
// the four minima.  Lines with an output whose window exceeds the halo (or
// that have no site at all, f = kInfSq) are marked in `redo`; the
// lower-envelope kernel recomputes exactly those lines afterwards.
constexpr int kWinTL = 128;
constexpr int kWinHalo = 64;
constexpr int kWinThreads = 256;
constexpr int kWinWarps = kWinThreads / 32;
constexpr int kWinGroup = 4;  // adjacent outputs per lane
static_assert(kWinTL == kWinWarps * kWinGroup * 4, "four groups of four outputs per warp");
static_assert(kInfSq + (kWinHalo + 6u) * (kWinHalo + 6u) > kInfSq, "the window scan adds distance^2 to kInfSq");

// floor(sqrt(f)) + 2 >= isqrt(f - 1) + 1 for f >= 1: the halo that f needs,
// from the hardware reciprocal square root (error far below one).
__device__ __forceinline__ uint32_t halo_need(uint32_t f) {
  const float ff = (float)f;
  return (uint32_t)(ff * rsqrtf(ff)) + 2u;
}

// One scan step at offset e: left candidate L = f(q - e), right R = f(q + 3 + e).
__device__ __forceinline__ void win_step(uint32_t L, uint32_t R, uint32_t e, uint32_t& b0, uint32_t& b1,
                                         uint32_t& b2, uint32_t& b3) {
  const uint32_t s0 = e * e, s1 = s0 + 2u * e + 1u, s2 = s1 + 2u * e + 3u, s3 = s2 + 2u * e + 5u;
  b0 = __viaddmin_u32(L, s0, __viaddmin_u32(R, s3, b0));
  b1 = __viaddmin_u32(L, s1, __viaddmin_u32(R, s2, b1));
  b2 = __viaddmin_u32(L, s2, __viaddmin_u32(R, s1, b2));
  b3 = __viaddmin_u32(L, s3, __viaddmin_u32(R, s0, b3));
}

// Whether a flag of rows q0 .. q0 + kWinTL - 1 (of n, w flags each) is set in
// the block's 32 columns, x being the thread's own (block-wide vote).
__device__ __forceinline__ bool any_flag(const uint8_t* __restrict__ only, int q0, int n, int x, int w) {
  bool any = false;
  for (int q = q0 + (int)(threadIdx.x >> 5); q < min(q0 + kWinTL, n); q += kWinWarps)
    any = any || (x < w && only[(long long)q * w + x]);
  return __syncthreads_or(any);
}

__global__ void __launch_bounds__(kWinThreads)
edt_window_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, int n, long long stride, int w,
                  long long outer_stride, int nxt, int nchunk, uint8_t* __restrict__ redo, Counters* __restrict__ ctr,
                  int track_max, const uint8_t* __restrict__ only) {
  __shared__ uint32_t buf[(kWinTL + 2 * kWinHalo) * 32];
  __shared__ uint32_t s_need;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long bid = blockIdx.x;
  const int xt = (int)(bid % nxt);
  const int chunk = (int)((bid / nxt) % nchunk);
  const long long orow = bid / ((long long)nxt * nchunk);
  const int x = xt * 32 + lane;
  const bool xin = x < w;
  const long long base = orow * outer_stride + x;
  const int q0 = chunk * kWinTL;
  if (only && !any_flag(only, q0, n, x, w)) return;
  if (threadIdx.x == 0) s_need = 0u;
  __syncthreads();
  // centre rows (loads of the warp's 16 rows issued before their use)
  uint32_t need = 0;  // halo rows this block needs: from its largest finite value
  constexpr int kPer = kWinTL / kWinWarps;  // 16
  uint32_t f[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int q = q0 + warp + kWinWarps * j;
    f[j] = (xin && q < n) ? in[base + (long long)q * stride] : kInfSq;
  }
  uint32_t fmax = 0;  // largest finite value (the halo bound grows with it)
  bool inf = false;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const uint32_t v = f[j];
    inf = inf || v == kInfSq;
    fmax = max(fmax, v == kInfSq ? 0u : v);
    buf[(kWinHalo + warp + kWinWarps * j) * 32 + lane] = v;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) fmax = max(fmax, __shfl_xor_sync(0xffffffffu, fmax, o));
  inf = __any_sync(0xffffffffu, inf);
  if (lane == 0) {
    need = inf ? 0xffffu : (fmax ? halo_need(fmax) : 0u);
    atomicMax(&s_need, need);
  }
  __syncthreads();
  const int halo = (int)min(s_need, (uint32_t)kWinHalo);
  for (int i = warp; i < halo; i += kWinWarps) {
    const int ql = q0 - 1 - i, qr = q0 + kWinTL + i;
    const uint32_t l = (xin && ql >= 0) ? in[base + (long long)ql * stride] : kInfSq;
    const uint32_t r = (xin && qr < n) ? in[base + (long long)qr * stride] : kInfSq;
    buf[(kWinHalo - 1 - i) * 32 + lane] = l;
    buf[(kWinHalo + kWinTL + i) * 32 + lane] = r;
  }
  __syncthreads();
  uint32_t localmax = 0;
  bool bad = false;
#pragma unroll 1
  for (int j = 0; j < kPer / kWinGroup; ++j) {
    const int i = kWinGroup * (warp + kWinWarps * j);  // first of the group's rows (warp-uniform)
    const int q = q0 + i;
    if (!xin || q >= n) continue;
    const int m = min(kWinGroup, n - q);  // outputs inside the line
    const uint32_t* col = buf + (kWinHalo + i) * 32 + lane;
    const uint32_t c0 = col[0], c1 = col[32], c2 = col[64], c3 = col[96];
    // the group's own values (rows past the line end hold kInfSq)
    uint32_t b0 = __viaddmin_u32(c1, 1u, __viaddmin_u32(c2, 4u, __viaddmin_u32(c3, 9u, c0)));
    uint32_t b1 = __viaddmin_u32(c0, 1u, __viaddmin_u32(c2, 1u, __viaddmin_u32(c3, 4u, c1)));
    uint32_t b2 = __viaddmin_u32(c0, 4u, __viaddmin_u32(c1, 1u, __viaddmin_u32(c3, 1u, c2)));
    uint32_t b3 = __viaddmin_u32(c0, 9u, __viaddmin_u32(c1, 4u, __viaddmin_u32(c2, 1u, c3)));
    if (m < 4) {  // outputs past the line end take no part in the stopping test
      b3 = 0u;
      if (m < 3) b2 = 0u;
      if (m < 2) b1 = 0u;
    }
    // after offsets 1 .. e-1 every candidate within distance e of every output
    // has been tried, so the scan stops once e^2 reaches the largest minimum
    bool done = true;
    int e = 1;
    uint32_t mx = max(max(b0, b1), max(b2, b3));
    while ((uint32_t)(e * e) < mx) {
      if (e + 3 <= halo) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          win_step(col[-(e + u) * 32], col[(3 + e + u) * 32], (uint32_t)(e + u), b0, b1, b2, b3);
        e += 4;
      } else {
        if (e > halo) {
          done = false;
          break;
        }
        win_step(col[-e * 32], col[(3 + e) * 32], (uint32_t)e, b0, b1, b2, b3);
        ++e;
      }
      mx = max(max(b0, b1), max(b2, b3));
    }
    if (!done) {
      bad = true;
      continue;
    }
    uint32_t* op = out + base + (long long)q * stride;
    op[0] = b0;
    if (m > 1) op[stride] = b1;
    if (m > 2) op[2 * stride] = b2;
    if (m > 3) op[3 * stride] = b3;
    localmax = max(localmax, mx);
  }
  if (bad) {
    redo[orow * (long long)w + x] = 1u;
    if (track_max) ctr->z_redo = 1u;
  }
  if (track_max) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) localmax = max(localmax, __shfl_xor_sync(0xffffffffu, localmax, o));
    if (lane == 0 && localmax) atomicMax(&ctr->rmax, localmax);
  }
}


// ---- TMA-staged window pass -------------------------------------------------
// Same computation as edt_window_kernel, with the staging done by the tensor
// memory accelerator: one thread issues a single 3-D tiled copy of the block's
// 128 output rows plus a full 64-row halo on each side (256 rows of 32 x,
// 32 KB) into shared memory and every thread waits on the copy's mbarrier.
// Rows outside the line arrive zero-filled and are set to kInfSq ("no site")
// by the blocks at the line ends.  The per-thread load, staging and halo
// sizing work of the plain kernel disappears; the scan may always run to the
// full halo.  Needs w a multiple of 4 (16-byte row pitch) and 16-byte aligned
// buffers; other volumes, and the z pass, take edt_window_kernel.
constexpr int kTmaRows = kWinTL + 2 * kWinHalo;
static_assert(kTmaRows <= 256, "a TMA box dimension is at most 256");
constexpr long long kWaitCycles = 4000000000ll;  // ~2 s at 2 GHz: a copy that has not landed by then never will

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Bounded wait for phase `parity` of the mbarrier at `bar`: false once `limit`
// cycles have passed (limit 0: gives up before the first try).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, long long limit) {
  const long long t0 = clock64();
  for (;;) {
    if (clock64() - t0 >= limit) return false;
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
}

__global__ void __launch_bounds__(kWinThreads)
edt_window_tma_kernel(const __grid_constant__ CUtensorMap tin, uint32_t* __restrict__ out, int axis, int n,
                      long long stride, int w, long long outer_stride, int nxt, int nchunk,
                      uint8_t* __restrict__ redo, Counters* __restrict__ ctr, int track_max, long long wait_limit,
                      const uint8_t* __restrict__ only) {
  __shared__ alignas(128) uint32_t buf[kTmaRows * 32];
  __shared__ alignas(8) unsigned long long bar;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long bid = blockIdx.x;
  const int xt = (int)(bid % nxt);
  const int chunk = (int)((bid / nxt) % nchunk);
  const int orow = (int)(bid / ((long long)nxt * nchunk));
  const int x = xt * 32 + lane;
  const bool xin = x < w;
  const int q0 = chunk * kWinTL;
  if (only && !any_flag(only, q0, n, x, w)) return;
  const uint32_t b = smem_u32(&bar);
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int c0 = xt * 32, ql = q0 - kWinHalo;  // x start: 128-byte multiple; rows may start below 0
    const int c1 = axis == 1 ? ql : orow, c2 = axis == 1 ? orow : ql;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(kTmaRows * 32 * 4)
                 : "memory");
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_u32(buf)), "l"(reinterpret_cast<unsigned long long>(&tin)), "r"(c0), "r"(c1), "r"(c2), "r"(b)
        : "memory");
  }
  const bool landed = mbar_wait(b, 0u, wait_limit);
  if (!__syncthreads_and(landed)) {
    // the copy did not complete in time: report it, give the copy in flight a
    // second wait with the full bound (it writes into this block's shared
    // memory) and leave
    if (threadIdx.x == 0) atomicOr(&ctr->status, 1u);
    mbar_wait(b, 0u, kWaitCycles);
    return;
  }
  if (q0 < kWinHalo || q0 + kWinTL + kWinHalo > n) {
    for (int k = threadIdx.x; k < kTmaRows * 32; k += kWinThreads) {
      const int q = q0 - kWinHalo + (k >> 5);
      if (q < 0 || q >= n) buf[k] = kInfSq;
    }
    __syncthreads();
  }
  const long long base = (long long)orow * outer_stride + x;
  uint32_t localmax = 0;
  bool bad = false;
#pragma unroll 1
  for (int j = 0; j < kWinTL / (kWinGroup * kWinWarps); ++j) {
    const int i = kWinGroup * (warp + kWinWarps * j);
    const int q = q0 + i;
    if (!xin || q >= n) continue;
    const int m = min(kWinGroup, n - q);
    const uint32_t* col = buf + (kWinHalo + i) * 32 + lane;
    const uint32_t c0 = col[0], c1 = col[32], c2 = col[64], c3 = col[96];
    uint32_t b0 = __viaddmin_u32(c1, 1u, __viaddmin_u32(c2, 4u, __viaddmin_u32(c3, 9u, c0)));
    uint32_t b1 = __viaddmin_u32(c0, 1u, __viaddmin_u32(c2, 1u, __viaddmin_u32(c3, 4u, c1)));
    uint32_t b2 = __viaddmin_u32(c0, 4u, __viaddmin_u32(c1, 1u, __viaddmin_u32(c3, 1u, c2)));
    uint32_t b3 = __viaddmin_u32(c0, 9u, __viaddmin_u32(c1, 4u, __viaddmin_u32(c2, 1u, c3)));
    if (m < 4) {
      b3 = 0u;
      if (m < 3) b2 = 0u;
      if (m < 2) b1 = 0u;
    }
    bool done = true;
    int e = 1;
    uint32_t mx = max(max(b0, b1), max(b2, b3));
    while ((uint32_t)(e * e) < mx) {
      if (e + 3 <= kWinHalo) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          win_step(col[-(e + u) * 32], col[(3 + e + u) * 32], (uint32_t)(e + u), b0, b1, b2, b3);
        e += 4;
      } else {
        if (e > kWinHalo) {
          done = false;
          break;
        }
        win_step(col[-e * 32], col[(3 + e) * 32], (uint32_t)e, b0, b1, b2, b3);
        ++e;
      }
      mx = max(max(b0, b1), max(b2, b3));
    }
    if (!done) {
      bad = true;
      continue;
    }
    uint32_t* op = out + base + (long long)q * stride;
    op[0] = b0;
    if (m > 1) op[stride] = b1;
    if (m > 2) op[2 * stride] = b2;
    if (m > 3) op[3 * stride] = b3;
    localmax = max(localmax, mx);
  }
  if (bad) {
    redo[(long long)orow * w + x] = 1u;
    if (track_max) ctr->z_redo = 1u;
  }
  if (track_max) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) localmax = max(localmax, __shfl_xor_sync(0xffffffffu, localmax, o));
    if (lane == 0 && localmax) atomicMax(&ctr->rmax, localmax);
  }
}

// ---- 16-bit passes ----------------------------------------------------------
// The transform while every squared distance is at most kNearMax = 65^2: the
// x and y results in 16 bits at a padded row pitch, two adjacent voxels of x
// per register, so that the maps between the passes are half as large and a
// scan step serves eight outputs instead of four.  A value up to kNearMax is
// exact in every pass, and a larger one only says that the true value is at
// least kNearMax: the row distance is cut at kReach, rows outside the volume
// read kFar16, and the y pass stores what it has once it has tried its 64 rows
// on either side (a candidate beyond them adds at least 65^2).  A minimum of at
// most kNearMax can only have come from exact candidates, so the z pass' outputs
// up to kNearMax are exact too; it flags the lines that hold others, and the
// 32-bit passes compute those (launch_edt_x, launch_edt_window, then
// launch_edt_redo or launch_edt_near_redo).
//
// 512^3, 15 % foreground: 754 us with 32-bit passes, 445 here (x 106, y 129,
// z 172; the maps' bytes alone take 260 at the copy rate, the rest is issue).
// 417 x 333 x 379 (rows at any address): 673 us, 333 here (79, 102, 115; the x
// pass 125 from single bytes, a ballot per 32).  Where 36 to 94 % of the volume
// lies beyond 65 voxels of a site, so that the 32-bit passes run as well, 1.23-2.70
// ms before and 1.18-2.68 here; small volumes all of which lie beyond lose 20 us.
constexpr uint32_t kNearMax = (kWinHalo + 1) * (kWinHalo + 1);
constexpr uint32_t kFar16 = 40000;
constexpr int kReach = 190, kReachWords = 6;
constexpr uint32_t kPair = 0x10001u;
static_assert(32 * kReachWords >= kReach, "a site beyond the words looked at is at least kReach away");
static_assert((kReach + 7) * (kReach + 7) <= (int)kFar16 && kReach * kReach > (int)kNearMax, "far rows stay far");
static_assert(kFar16 + (kWinHalo + 6) * (kWinHalo + 6) < 65536, "the window scan adds distance^2 to kFar16");

// The x pass: a warp per row, eight voxels per lane.  A voxel's distance is the
// least of three: to a site among its lane's eight voxels (a table by their
// bits), to the nearest site left of them and right of them.
template <int MODE, bool VEC>
__global__ void __launch_bounds__(kXWarps * 32, VEC ? 6 : 5)
edt_x_near_kernel(const uint8_t* __restrict__ a, const uint8_t* __restrict__ b, Dims dm, int pitch,
                  uint16_t* __restrict__ out, uint32_t* __restrict__ selbits, Counters* __restrict__ ctr) {
  extern __shared__ uint32_t smem[];
  __shared__ uint4 s_inside[256];
  static_assert(kXWarps * 32 == 256, "a table entry per thread");
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nw = dm.nw();
  uint32_t* mask = smem + (size_t)warp * nw;  // the row's sites
  const long long rows = (long long)dm.h * dm.d;
  const bool two = MODE == SEL_BONE_IN_ROI || MODE == SEL_MARROW_IN_ROI;
  const ByteVolume ba(a, dm.n()), bb(two ? b : a, dm.n());
  unsigned long long sites = 0;
  {
    const uint32_t t = threadIdx.x;
    uint32_t v[4];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t lo = t & ((2u << i) - 1u), hi = t >> i;  // bits at or below, at or above
      const int l = lo ? i - (31 - __clz(lo)) : 255, r = hi ? __ffs(hi) - 1 : 255;
      const uint32_t g = (uint32_t)min(l, r);
      if (i & 1) v[i >> 1] |= g << 16;
      else v[i >> 1] = g;
    }
    s_inside[t] = make_uint4(v[0], v[1], v[2], v[3]);
  }
  __syncthreads();

  for (long long row = (long long)blockIdx.x * kXWarps + warp; row < rows;
       row += (long long)gridDim.x * kXWarps) {
    const long long base = row * dm.w;
    const int nvec = (dm.w + 15) >> 4;  // 16 voxels per lane
    for (int v0 = 0; v0 < nvec; v0 += 32) {
      const int v = v0 + lane;
      uint32_t s16 = 0, t16 = 0;
      if (v < nvec) {
        const long long at = base + 16 * v;
        const uint4 A = VEC ? __ldg(reinterpret_cast<const uint4*>(a + at)) : load16(ba, at);
        const uint4 B = !two  ? make_uint4(0u, 0u, 0u, 0u)
                        : VEC ? __ldg(reinterpret_cast<const uint4*>(b + at))
                              : load16(bb, at);
        const uint32_t inside = dm.w - 16 * v >= 16 ? 0xffffu : (1u << (dm.w - 16 * v)) - 1u;  // voxels of this row
        s16 = (sel4<MODE>(A.x, B.x) | (sel4<MODE>(A.y, B.y) << 4) | (sel4<MODE>(A.z, B.z) << 8) |
               (sel4<MODE>(A.w, B.w) << 12)) & inside;
        t16 = ~s16 & inside;
      }
      const uint32_t s_hi = __shfl_down_sync(0xffffffffu, s16, 1);
      const uint32_t t_hi = __shfl_down_sync(0xffffffffu, t16, 1);
      if (!(lane & 1) && v < nvec) {
        const int c = v >> 1;  // word index: voxels 32c .. 32c + 31
        // an odd number of 16-voxel groups ends on a half word: its upper half is empty
        const bool full = v + 1 < nvec;
        const uint32_t tw = t16 | (full ? t_hi << 16 : 0u);
        mask[c] = tw;
        selbits[row * nw + c] = s16 | (full ? s_hi << 16 : 0u);
        sites += __popc(tw);
      }
    }
    __syncwarp();
    const int bit = (lane & 3) * 8;  // first bit of this lane's voxels in their word
    const uint32_t below = (1u << bit) - 1u, above = ~((2u << (bit + 7)) - 1u);  // bit + 7 = 31: above = 0
    uint4* orow = reinterpret_cast<uint4*>(out + row * pitch);
#pragma unroll 1
    for (int x0 = 0; x0 < dm.w; x0 += 256) {
      const int x = x0 + 8 * lane;
      if (x < dm.w) {
        const int c = x >> 5;
        const uint32_t m = mask[c];
        // the nearest site on either side, no further than kReachWords words away
        uint32_t lo = m & below, hi = m & above;
        int cl = c, cr = c;
#pragma unroll 1
        while (lo == 0u && cl > max(c - kReachWords, 0)) lo = mask[--cl];
#pragma unroll 1
        while (hi == 0u && cr < min(c + kReachWords, nw - 1)) hi = mask[++cr];
        const int left = lo ? cl * 32 + 31 - __clz(lo) : kNoLeft, right = hi ? cr * 32 + __ffs(hi) - 1 : kNoRight;
        const uint32_t dl = (uint32_t)min(x - left, kReach) * kPair, dr = (uint32_t)min(right - x - 7, kReach) * kPair;
        const uint4 in8 = s_inside[(m >> bit) & 0xffu];
        auto square = [&](uint32_t inside, uint32_t i) {  // of voxels i and i + 1 of the eight
          const uint32_t g = __viaddmin_u16x2(dl, i * kPair + 0x10000u,
                                              __viaddmin_u16x2(dr, (7u - i) * kPair - 0x10000u, inside));
          const uint32_t g0 = g & 0xffffu, g1 = g >> 16;
          return g1 * (g & 0xffff0000u) + g0 * g0;
        };
        uint4 v = make_uint4(square(in8.x, 0), square(in8.y, 2), square(in8.z, 4), square(in8.w, 6));
        if (x + 8 > dm.w) {  // the padding holds zeros
          const int k = dm.w - x;
          auto cut = [&](uint32_t p, int i) { return k >= i + 2 ? p : k == i + 1 ? p & 0xffffu : 0u; };
          v = make_uint4(cut(v.x, 0), cut(v.y, 2), cut(v.z, 4), cut(v.w, 6));
        }
        orow[x >> 3] = v;
        if (x + 8 < pitch && x + 8 >= dm.w) orow[(x >> 3) + 1] = make_uint4(0u, 0u, 0u, 0u);
      }
    }
    __syncwarp();
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sites += __shfl_xor_sync(0xffffffffu, sites, o);
  if (lane == 0 && sites) atomicAdd(&ctr->sites, sites);
}

// Four adjacent outputs of a lane's two columns (col: the group's first row in
// shared memory, 32 pairs per row); m: how many lie inside the line; halo: rows
// staged on either side, a multiple of 4.  Returns the largest of the outputs.
__device__ __forceinline__ uint32_t near_group(const uint32_t* col, int m, int halo, uint32_t (&b)[4]) {
  const uint32_t c0 = col[0], c1 = col[32], c2 = col[64], c3 = col[96];
  b[0] = __viaddmin_u16x2(c1, kPair, __viaddmin_u16x2(c2, 4 * kPair, __viaddmin_u16x2(c3, 9 * kPair, c0)));
  b[1] = __viaddmin_u16x2(c0, kPair, __viaddmin_u16x2(c2, kPair, __viaddmin_u16x2(c3, 4 * kPair, c1)));
  b[2] = __viaddmin_u16x2(c0, 4 * kPair, __viaddmin_u16x2(c1, kPair, __viaddmin_u16x2(c3, kPair, c2)));
  b[3] = __viaddmin_u16x2(c0, 9 * kPair, __viaddmin_u16x2(c1, 4 * kPair, __viaddmin_u16x2(c2, kPair, c3)));
  if (m < 4) {  // outputs past the line end take no part in the stopping test
    b[3] = 0u;
    if (m < 3) b[2] = 0u;
    if (m < 2) b[1] = 0u;
  }
  // after offsets 1 .. e-1 every candidate within distance e of every output
  // has been tried, so the scan stops once e^2 reaches the largest minimum
  uint32_t mx = __vmaxu2(__vimax3_u16x2(b[0], b[1], b[2]), b[3]);
  const uint32_t *lp = col - 32, *rp = col + 4 * 32;
#pragma unroll 1
  for (uint32_t e = 1, t = kPair; e <= (uint32_t)halo && __vmaxu2(mx, t) != t; e += 4, lp -= 4 * 32, rp += 4 * 32) {
    uint32_t sq[8];  // (e + k)^2
    sq[0] = t;
#pragma unroll
    for (uint32_t k = 0; k < 7; ++k) sq[k + 1] = sq[k] + 2u * e * kPair + (2u * k + 1u) * kPair;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint32_t L = lp[-u * 32], R = rp[u * 32];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        b[k] = __viaddmin_u16x2(L, sq[u + k], __viaddmin_u16x2(R, sq[u + 3 - k], b[k]));
    }
    t = sq[4];
    mx = __vmaxu2(__vimax3_u16x2(b[0], b[1], b[2]), b[3]);
  }
  return mx;
}

// The y or z pass over 64 columns and kWinTL outputs per block, the input
// staged by every thread, with a halo as wide as the largest value needs.
// in: pairs; strides in pairs.  WIDE: the 32-bit result at the volume's own
// pitch, else pairs again.
template <bool Z, bool WIDE>
__global__ void __launch_bounds__(kWinThreads, 6)
edt_near_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, int n, long long stride, int pairs,
                long long outer, int nxt, int nchunk, int w, long long out_stride, uint8_t* __restrict__ redo,
                Counters* __restrict__ ctr) {
  __shared__ uint32_t buf[(kWinTL + 2 * kWinHalo) * 32];
  __shared__ uint32_t s_max[kWinWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long bid = blockIdx.x;
  const int xt = (int)(bid % nxt);
  const int chunk = (int)((bid / nxt) % nchunk);
  const long long orow = bid / ((long long)nxt * nchunk);
  const int px = xt * 32 + lane;
  const bool pin = px < pairs;
  const long long base = orow * outer + px;
  const int q0 = chunk * kWinTL;
  constexpr int kPer = kWinTL / kWinWarps;  // 16
  uint32_t f[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int q = q0 + warp + kWinWarps * j;
    f[j] = q < n ? (pin ? in[base + (long long)q * stride] : 0u) : kFar16 * kPair;
  }
  uint32_t top = 0;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    if (q0 + warp + kWinWarps * j < n) top = __vmaxu2(top, f[j]);
    buf[(kWinHalo + warp + kWinWarps * j) * 32 + lane] = f[j];
  }
  top = __reduce_max_sync(0xffffffffu, max(top & 0xffffu, top >> 16));
  if (lane == 0) s_max[warp] = top;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kWinWarps; ++k) top = max(top, s_max[k]);
  const int halo = top ? (int)min((halo_need(top) + 3u) & ~3u, (uint32_t)kWinHalo) : 0;
  uint32_t least = kFar16 * kPair;
  if (Z && top > kNearMax)
#pragma unroll
    for (int j = 0; j < kPer; ++j) least = __vminu2(least, f[j]);
  for (int i = warp; i < halo; i += kWinWarps) {
    const int ql = q0 - 1 - i, qr = q0 + kWinTL + i;
    const uint32_t l = ql >= 0 ? (pin ? in[base + (long long)ql * stride] : 0u) : kFar16 * kPair;
    const uint32_t r = qr < n ? (pin ? in[base + (long long)qr * stride] : 0u) : kFar16 * kPair;
    buf[(kWinHalo - 1 - i) * 32 + lane] = l;
    buf[(kWinHalo + kWinTL + i) * 32 + lane] = r;
    least = __vminu2(least, __vminu2(l, r));
  }
  const int x = 2 * px;
  uint32_t localmax = 0;
  uint32_t far = 0;  // the lane's columns with an output beyond kNearMax
  // a block that stages nothing up to kNearMax holds no output up to it either
  // (columns of the padding stage zeros)
  const bool some = !Z || top <= kNearMax || (pin && min(least & 0xffffu, least >> 16) <= kNearMax);
  if (!__syncthreads_or(some)) {
    if (x < w) redo[orow * w + x] = 1u;
    if (x + 1 < w) redo[orow * w + x + 1] = 1u;
    if (threadIdx.x == 0) ctr->z_redo = 1u;
    return;
  }
#pragma unroll 1
  for (int j = 0; j < kPer / kWinGroup; ++j) {
    const int i = kWinGroup * (warp + kWinWarps * j);
    const int q = q0 + i;
    if (!pin || q >= n) continue;
    const int m = min(kWinGroup, n - q);
    uint32_t b[4];
    const uint32_t mx = near_group(buf + (kWinHalo + i) * 32 + lane, m, halo, b);
    if (Z) {
      const uint32_t m0 = mx & 0xffffu, m1 = mx >> 16;
      if (m0 > kNearMax) far |= 1u;
      else localmax = max(localmax, m0);
      if (m1 > kNearMax) far |= 2u;
      else localmax = max(localmax, m1);
    }
    if (WIDE) {
      uint32_t* op = out + orow * w + x + (long long)q * out_stride;
#pragma unroll
      for (int k = 0; k < kWinGroup; ++k, op += out_stride) {
        if (k >= m) break;
        if (x < w) op[0] = b[k] & 0xffffu;
        if (x + 1 < w) op[1] = b[k] >> 16;
      }
    } else {
      uint32_t* op = out + base + (long long)q * stride;
#pragma unroll
      for (int k = 0; k < kWinGroup; ++k)
        if (k < m) op[k * stride] = b[k];
    }
  }
  if (Z) {
    if (far) {
      if (far & 1u) redo[orow * w + x] = 1u;
      if (far & 2u) redo[orow * w + x + 1] = 1u;
      ctr->z_redo = 1u;
    }
    localmax = __reduce_max_sync(0xffffffffu, localmax);
    if (lane == 0 && localmax) atomicMax(&ctr->rmax, localmax);
  }
}

// The y pass staged by one TMA copy per block, as edt_window_tma_kernel.
__global__ void __launch_bounds__(kWinThreads)
edt_near_tma_kernel(const __grid_constant__ CUtensorMap tin, uint32_t* __restrict__ out, int n, int pairs, int nxt,
                    int nchunk, Counters* __restrict__ ctr, long long wait_limit) {
  __shared__ alignas(128) uint32_t buf[kTmaRows * 32];
  __shared__ alignas(8) unsigned long long bar;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long bid = blockIdx.x;
  const int xt = (int)(bid % nxt);
  const int chunk = (int)((bid / nxt) % nchunk);
  const int plane = (int)(bid / ((long long)nxt * nchunk));
  const int px = xt * 32 + lane;
  const int q0 = chunk * kWinTL;
  const uint32_t b = smem_u32(&bar);
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(kTmaRows * 32 * 4)
                 : "memory");
    // x start: 64 16-bit values, a multiple of 128 bytes; rows may start below 0
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_u32(buf)), "l"(reinterpret_cast<unsigned long long>(&tin)), "r"(xt * 64), "r"(q0 - kWinHalo),
        "r"(plane), "r"(b)
        : "memory");
  }
  const bool landed = mbar_wait(b, 0u, wait_limit);
  if (!__syncthreads_and(landed)) {  // as in edt_window_tma_kernel
    if (threadIdx.x == 0) atomicOr(&ctr->status, 1u);
    mbar_wait(b, 0u, kWaitCycles);
    return;
  }
  const int before = kWinHalo - q0, inside = n - q0 + kWinHalo;  // the box's rows before the line; up to its end
  if (before > 0 || inside < kTmaRows) {
    for (int k = threadIdx.x; k < before * 32; k += kWinThreads) buf[k] = kFar16 * kPair;
    for (int k = inside * 32 + threadIdx.x; k < kTmaRows * 32; k += kWinThreads) buf[k] = kFar16 * kPair;
    __syncthreads();
  }
  if (px >= pairs) return;
#pragma unroll 1
  for (int j = 0; j < kWinTL / (kWinGroup * kWinWarps); ++j) {
    const int i = kWinGroup * (warp + kWinWarps * j);
    const int q = q0 + i;
    if (q >= n) continue;
    const int m = min(kWinGroup, n - q);
    uint32_t v[4];
    near_group(buf + (kWinHalo + i) * 32 + lane, m, kWinHalo, v);
    uint32_t* op = out + ((long long)plane * n + q) * pairs + px;
#pragma unroll
    for (int k = 0; k < kWinGroup; ++k)
      if (k < m) op[(long long)k * pairs] = v[k];
  }
}

// The lines along z that redo does not flag, from 16 to 32 bits (a thread per
// line and kWidenZ planes; bytes alone bound it).
constexpr int kWidenZ = 64;
__global__ void __launch_bounds__(256)
edt_widen_kernel(const uint16_t* __restrict__ narrow, uint32_t* __restrict__ wide, Dims dm, int pitch,
                 const uint8_t* __restrict__ redo) {
  const int x = blockIdx.x * 256 + threadIdx.x, y = blockIdx.y, z0 = blockIdx.z * kWidenZ;
  if (x >= dm.w || redo[(long long)y * dm.w + x]) return;
  const uint16_t* from = narrow + ((long long)z0 * dm.h + y) * pitch + x;
  uint32_t* to = wide + ((long long)z0 * dm.h + y) * dm.w + x;
  const int planes = min(kWidenZ, dm.d - z0);
#pragma unroll 8
  for (int z = 0; z < planes; ++z)
    to[(long long)z * dm.w * dm.h] = from[(long long)z * pitch * dm.h];
}

}  // namespace

size_t edt_scratch_bytes(Dims dm) {
  // two u32 arrays (position, f) of line-length x line-count for the larger pass
  const long long y_pass = (long long)dm.h * dm.w * dm.d;
  return (size_t)y_pass * 2 * sizeof(uint32_t);
}

template <int MODE>
cudaError_t launch_edt_x_mode(const uint8_t* a, const uint8_t* b, Dims dm, uint32_t* out, uint32_t* selbits,
                              Counters* ctr, unsigned blocks, size_t smem, cudaStream_t s) {
  const bool two = MODE == SEL_BONE_IN_ROI || MODE == SEL_MARROW_IN_ROI;
  const bool vec = dm.w % 16 == 0 && (reinterpret_cast<uintptr_t>(a) & 15u) == 0 &&
                   (!two || (reinterpret_cast<uintptr_t>(b) & 15u) == 0) &&
                   (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
  if (vec) {
    if (smem > 48 * 1024) {
      cudaError_t e =
          cudaFuncSetAttribute(edt_x_vec_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kXMaxSmem);
      if (e != cudaSuccess) return e;
    }
    edt_x_vec_kernel<MODE><<<blocks, kXWarps * 32, smem, s>>>(a, b, dm, out, selbits, ctr);
  } else {
    if (smem > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(edt_x_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kXMaxSmem);
      if (e != cudaSuccess) return e;
    }
    edt_x_kernel<MODE><<<blocks, kXWarps * 32, smem, s>>>(a, b, dm, out, selbits, ctr);
  }
  return cudaGetLastError();
}

cudaError_t launch_edt_x(const uint8_t* a, const uint8_t* b, int mode, Dims dm, uint32_t* out,
                         uint32_t* selbits, Counters* ctr, cudaStream_t s, unsigned long long* launches) {
  const long long rows = (long long)dm.h * dm.d;
  long long blocks = (rows + kXWarps - 1) / kXWarps;
  if (blocks > 152 * 64) blocks = 152 * 64;
  const size_t smem = (size_t)kXWarps * 3 * dm.nw() * sizeof(uint32_t);
  cudaError_t e;
  switch (mode) {
    case SEL_FOREGROUND:
      e = launch_edt_x_mode<SEL_FOREGROUND>(a, b, dm, out, selbits, ctr, (unsigned)blocks, smem, s);
      break;
    case SEL_BACKGROUND:
      e = launch_edt_x_mode<SEL_BACKGROUND>(a, b, dm, out, selbits, ctr, (unsigned)blocks, smem, s);
      break;
    case SEL_BONE_IN_ROI:
      e = launch_edt_x_mode<SEL_BONE_IN_ROI>(a, b, dm, out, selbits, ctr, (unsigned)blocks, smem, s);
      break;
    default:
      e = launch_edt_x_mode<SEL_MARROW_IN_ROI>(a, b, dm, out, selbits, ctr, (unsigned)blocks, smem, s);
      break;
  }
  ++*launches;
  return e;
}

cudaError_t launch_edt_line(int axis, const uint32_t* in, uint32_t* out, Dims dm, void* scratch, Counters* ctr,
                            cudaStream_t s, unsigned long long* launches) {
  int n;
  long long stride, outer, nlines;
  if (axis == 1) {
    n = dm.h;
    stride = dm.w;
    outer = (long long)dm.w * dm.h;
    nlines = (long long)dm.w * dm.d;
  } else {
    n = dm.d;
    stride = (long long)dm.w * dm.h;
    outer = dm.w;
    nlines = (long long)dm.w * dm.h;
  }
  uint32_t* spos = static_cast<uint32_t*>(scratch);
  uint32_t* sf = spos + (size_t)nlines * n;
  const long long blocks = (nlines + 255) / 256;
  edt_line_kernel<<<(unsigned)blocks, 256, 0, s>>>(in, out, nullptr, n, stride, dm.w, outer, stride, outer, nlines, spos, sf,
                                                   ctr, axis == 2 ? 1 : 0, nullptr);
  ++*launches;
  return cudaGetLastError();
}

namespace {

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }();
  return fn;
}

// Tensor map of a u32 volume (x fastest) whose box is 32 x by `rows` along the
// pass axis; false when the volume or buffer does not meet TMA's rules.
bool window_map(CUtensorMap* map, const uint32_t* vol, Dims dm, int axis, unsigned rows) {
  if (dm.w % 4 != 0 || (reinterpret_cast<uintptr_t>(vol) & 15u) != 0) return false;
  const PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)dm.w, (cuuint64_t)dm.h, (cuuint64_t)dm.d};
  const cuuint64_t pitch[2] = {(cuuint64_t)dm.w * 4, (cuuint64_t)dm.w * dm.h * 4};
  const cuuint32_t box[3] = {32u, axis == 1 ? rows : 1u, axis == 1 ? 1u : rows};
  const cuuint32_t unit[3] = {1u, 1u, 1u};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, const_cast<uint32_t*>(vol), dims, pitch, box, unit,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tensor map of a 16-bit map of pitch edt_near_pitch(w): boxes of 64 x by kTmaRows y.
bool near_map(CUtensorMap* map, const uint16_t* vol, Dims dm) {
  const PFN_cuTensorMapEncodeTiled_v12000 enc = tensor_map_encoder();
  if (!enc || (reinterpret_cast<uintptr_t>(vol) & 15u) != 0) return false;
  const cuuint64_t pitch = (cuuint64_t)edt_near_pitch(dm.w);
  const cuuint64_t dims[3] = {pitch, (cuuint64_t)dm.h, (cuuint64_t)dm.d};
  const cuuint64_t strides[2] = {pitch * 2, pitch * dm.h * 2};
  const cuuint32_t box[3] = {64u, (cuuint32_t)kTmaRows, 1u};
  const cuuint32_t unit[3] = {1u, 1u, 1u};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, const_cast<uint16_t*>(vol), dims, strides, box, unit,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

namespace {

struct Lines {  // the lines along an axis
  int n;                          // length
  long long stride, outer, rows;  // step along a line, step between rows of lines, rows
  long long count;                // lines
};

Lines lines_of(int axis, Dims dm) {
  const long long w = dm.w, wh = w * dm.h;
  return axis == 1 ? Lines{dm.h, w, wh, dm.d, w * dm.d} : Lines{dm.d, wh, w, dm.h, wh};
}

}  // namespace

cudaError_t launch_edt_window(int axis, const uint32_t* in, uint32_t* out, Dims dm, uint8_t* redo, Counters* ctr,
                              long long wait_cycles, const uint8_t* only, cudaStream_t s,
                              unsigned long long* launches) {
  const Lines l = lines_of(axis, dm);
  const int nxt = (dm.w + 31) / 32;
  const int nchunk = (l.n + kWinTL - 1) / kWinTL;
  const long long blocks = (long long)nxt * nchunk * l.rows;
  // TMA staging for the y pass only: a z-pass box spans 256 rows a whole
  // slice apart (a different page each), which the copy engine translates one
  // by one; there the per-thread loads measured faster (2.2 against 3.0 ms on
  // 1024^3 bone).
  CUtensorMap map;
  if (axis == 1 && window_map(&map, in, dm, axis, kTmaRows)) {
    edt_window_tma_kernel<<<(unsigned)blocks, kWinThreads, 0, s>>>(map, out, axis, l.n, l.stride, dm.w, l.outer, nxt,
                                                                   nchunk, redo, ctr, axis == 2 ? 1 : 0,
                                                                   wait_cycles < 0 ? kWaitCycles : wait_cycles, only);
  } else {
    edt_window_kernel<<<(unsigned)blocks, kWinThreads, 0, s>>>(in, out, l.n, l.stride, dm.w, l.outer, nxt, nchunk, redo,
                                                               ctr, axis == 2 ? 1 : 0, only);
  }
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launch_edt_redo(int axis, const uint32_t* in, uint32_t* out, Dims dm, void* scratch, const uint8_t* redo,
                            Counters* ctr, cudaStream_t s, unsigned long long* launches) {
  const Lines l = lines_of(axis, dm);
  uint32_t* spos = static_cast<uint32_t*>(scratch);
  uint32_t* sf = spos + (size_t)l.count * l.n;
  edt_line_kernel<<<(unsigned)((l.count + 255) / 256), 256, 0, s>>>(in, out, nullptr, l.n, l.stride, dm.w, l.outer,
                                                                   l.stride, l.outer, l.count, spos, sf, ctr,
                                                                   axis == 2 ? 1 : 0, redo);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launch_edt_near_redo(const uint32_t* in, uint16_t* out, uint32_t* wide, Dims dm, void* scratch, const uint8_t* redo,
                                 Counters* ctr, cudaStream_t s, unsigned long long* launches) {
  const Lines l = lines_of(2, dm);
  const long long pitch = edt_near_pitch(dm.w);
  uint32_t* spos = static_cast<uint32_t*>(scratch);
  uint32_t* sf = spos + (size_t)l.count * l.n;
  edt_line_kernel<<<(unsigned)((l.count + 255) / 256), 256, 0, s>>>(in, out, wide, l.n, l.stride, dm.w, l.outer,
                                                                   pitch * dm.h, pitch, l.count, spos, sf, ctr, 1, redo);
  ++*launches;
  return cudaGetLastError();
}

cudaError_t launch_edt_widen(const uint16_t* narrow, uint32_t* wide, Dims dm, const uint8_t* redo, cudaStream_t s,
                             unsigned long long* launches) {
  const dim3 grid((unsigned)((dm.w + 255) / 256), (unsigned)dm.h, (unsigned)((dm.d + kWidenZ - 1) / kWidenZ));
  edt_widen_kernel<<<grid, 256, 0, s>>>(narrow, wide, dm, edt_near_pitch(dm.w), redo);
  ++*launches;
  return cudaGetLastError();
}

int edt_near_pitch(int w) { return (w + 15) & ~15; }

template <int MODE>
cudaError_t launch_edt_x_near_mode(const uint8_t* a, const uint8_t* b, Dims dm, uint16_t* out, uint32_t* selbits,
                                   Counters* ctr, unsigned blocks, cudaStream_t s) {
  const bool two = MODE == SEL_BONE_IN_ROI || MODE == SEL_MARROW_IN_ROI;
  const size_t smem = (size_t)kXWarps * dm.nw() * sizeof(uint32_t);  // at most 32 KB, beside the table's 4
  const bool vec = dm.w % 16 == 0 && (reinterpret_cast<uintptr_t>(a) & 15u) == 0 &&
                   (!two || (reinterpret_cast<uintptr_t>(b) & 15u) == 0);
  auto kernel = vec ? edt_x_near_kernel<MODE, true> : edt_x_near_kernel<MODE, false>;
  kernel<<<blocks, kXWarps * 32, smem, s>>>(a, b, dm, edt_near_pitch(dm.w), out, selbits, ctr);
  return cudaGetLastError();
}

cudaError_t launch_edt_near_xy(const uint8_t* a, const uint8_t* b, int mode, Dims dm, uint16_t* xmap, uint16_t* ymap,
                               uint32_t* selbits, Counters* ctr, long long wait_cycles, bool x_pass, cudaStream_t s,
                               unsigned long long* launches) {
  ++*launches;
  if (x_pass) {
    // enough rows per warp that the table is not what a block spends its time on
    long long blocks = ((long long)dm.h * dm.d + kXWarps - 1) / kXWarps;
    if (blocks > 152 * 12) blocks = 152 * 12;
    switch (mode) {
      case SEL_FOREGROUND:
        return launch_edt_x_near_mode<SEL_FOREGROUND>(a, b, dm, xmap, selbits, ctr, (unsigned)blocks, s);
      case SEL_BACKGROUND:
        return launch_edt_x_near_mode<SEL_BACKGROUND>(a, b, dm, xmap, selbits, ctr, (unsigned)blocks, s);
      case SEL_BONE_IN_ROI:
        return launch_edt_x_near_mode<SEL_BONE_IN_ROI>(a, b, dm, xmap, selbits, ctr, (unsigned)blocks, s);
      default:
        return launch_edt_x_near_mode<SEL_MARROW_IN_ROI>(a, b, dm, xmap, selbits, ctr, (unsigned)blocks, s);
    }
  }
  const int pairs = edt_near_pitch(dm.w) / 2;
  const int nxt = (pairs + 31) / 32, nchunk = (dm.h + kWinTL - 1) / kWinTL;
  const unsigned blocks = (unsigned)((long long)nxt * nchunk * dm.d);
  const uint32_t* in = reinterpret_cast<const uint32_t*>(xmap);
  uint32_t* out = reinterpret_cast<uint32_t*>(ymap);
  CUtensorMap map;
  if (near_map(&map, xmap, dm)) {
    edt_near_tma_kernel<<<blocks, kWinThreads, 0, s>>>(map, out, dm.h, pairs, nxt, nchunk, ctr,
                                                       wait_cycles < 0 ? kWaitCycles : wait_cycles);
  } else {
    edt_near_kernel<false, false><<<blocks, kWinThreads, 0, s>>>(in, out, dm.h, pairs, pairs, (long long)pairs * dm.h, nxt,
                                                          nchunk, dm.w, 0, nullptr, ctr);
  }
  return cudaGetLastError();
}

cudaError_t launch_edt_near_z(const uint16_t* ymap, uint32_t* wide, uint16_t* narrow, Dims dm, uint8_t* redo,
                              Counters* ctr, cudaStream_t s, unsigned long long* launches) {
  const int pairs = edt_near_pitch(dm.w) / 2;
  const int nxt = (pairs + 31) / 32, nchunk = (dm.d + kWinTL - 1) / kWinTL;
  auto kernel = wide ? edt_near_kernel<true, true> : edt_near_kernel<true, false>;
  kernel<<<(unsigned)((long long)nxt * nchunk * dm.h), kWinThreads, 0, s>>>(
      reinterpret_cast<const uint32_t*>(ymap), wide ? wide : reinterpret_cast<uint32_t*>(narrow), dm.d,
      (long long)pairs * dm.h, pairs, pairs, nxt, nchunk, dm.w, (long long)dm.w * dm.h, redo, ctr);
  ++*launches;
  return cudaGetLastError();
}

}  // namespace bm
