// Exact order statistics and moment sums of a thickness map (metrics.rs:204-298).
//
// The reference keeps the finite positive f32 values and selects the k-th
// smallest with select_nth_unstable (total order on floats).  Positive finite
// floats order like their bit patterns, so the k-th value is found by a
// two-level radix select on the 32-bit pattern: a histogram of the high 16
// bits over the whole map, then, for the bins that hold the wanted ranks, a
// histogram of the low 16 bits.  The ranks are followed through both on the
// device, so that a call reads back ten values; they are exact, and the
// interpolation that follows on the host (in f64, then f32 calibration) is the
// reference's arithmetic on the reference's operands.
#include "kernels.h"

namespace bm {

namespace {

__device__ __forceinline__ bool positive_finite(uint32_t b) { return b != 0u && b < 0x7f800000u; }

constexpr int kHiBins = 0x7f80;  // high halves of the positive finite values
static_assert(kHiBins % 4 == 0 && kHiBins <= 32 * 1024, "read 16 bytes at a time, 32 bins per thread");
constexpr int kLoBins = 65536;

// Calls f(b0, b1, b2, b3) on the map's words four at a time (16-byte loads when
// the map allows them; the words past its end are 0).
template <class F>
__device__ __forceinline__ void each_four(const uint32_t* __restrict__ map, long long n, F&& f) {
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x, nth = (long long)gridDim.x * blockDim.x;
  const bool vec = (reinterpret_cast<uintptr_t>(map) & 15u) == 0;
  const long long quads = (n + 3) / 4;
  const int lane = threadIdx.x & 31;
  auto load = [&](long long q0) {
    const long long i = 4 * (q0 + lane);
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (vec && i + 4 <= n) {
      v = __ldg(reinterpret_cast<const uint4*>(map + i));
    } else {
      if (i < n) v.x = map[i];
      if (i + 1 < n) v.y = map[i + 1];
      if (i + 2 < n) v.z = map[i + 2];
      if (i + 3 < n) v.w = map[i + 3];
    }
    return v;
  };
  // whole warps stay together: f may use warp-wide operations.  Two steps' words
  // are in flight beside the one in hand.
  const long long first = tid - lane;
  uint4 v = load(first), next = load(first + nth);
  for (long long q0 = first; q0 < quads; q0 += nth) {
    const uint4 after = load(q0 + 2 * nth);
    f(v.x, v.y, v.z, v.w);
    v = next;
    next = after;
  }
}

// Adds runs of equal keys among four neighbours at once: neighbouring voxels of
// a thickness map often share a value, and equal addresses in a warp serialise.
template <class Add>
__device__ __forceinline__ void add_runs(const uint32_t (&key)[4], const bool (&ok)[4], Add&& add) {
  uint32_t cur = key[0], c = ok[0] ? 1u : 0u;
#pragma unroll
  for (int j = 1; j < 4; ++j) {
    if (ok[j] && (c == 0u || key[j] == cur)) {
      cur = key[j];
      ++c;
    } else if (ok[j]) {
      add(cur, c);
      cur = key[j];
      c = 1u;
    }
  }
  if (c) add(cur, c);
}

// hist[hi16] += 1 for every positive finite value: counted in shared memory (one
// CTA of 1024 threads per SM holds all 32640 bins), then added to the global
// histogram.  Counting straight into global memory, one atomic per distinct key
// and warp, took 2.03 ms on 33.5 M values of which 35% count (0.036 ms here).
__global__ void __launch_bounds__(1024)
hist_hi_kernel(const uint32_t* __restrict__ map, long long n, uint32_t* __restrict__ hist) {
  extern __shared__ uint32_t h[];
  for (int i = threadIdx.x; i < kHiBins; i += blockDim.x) h[i] = 0u;
  __syncthreads();
  each_four(map, n, [&](uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    const uint32_t key[4] = {a >> 16, b >> 16, c >> 16, d >> 16};
    const bool ok[4] = {positive_finite(a), positive_finite(b), positive_finite(c), positive_finite(d)};
    add_runs(key, ok, [&](uint32_t k, uint32_t m) { atomicAdd(&h[k], m); });
  });
  __syncthreads();
  for (int i = threadIdx.x; i < kHiBins; i += blockDim.x)
    if (h[i]) atomicAdd(&hist[i], h[i]);
}

// The bins among bins[0 .. nbins) that hold the ranks (0-based), one CTA of 1024
// threads: every thread sums PER consecutive bins (16-byte loads, all in
// flight), a scan finds the thread of each rank, and a warp per rank scans that
// thread's bins.  found(r, bin, rank inside the bin) is called by one thread
// per rank (by none for a rank past the total).
template <int PER, class F>
__device__ __forceinline__ void find_ranks(const uint32_t* __restrict__ bins, int nbins, const unsigned long long* ranks,
                                           int nranks, F&& found) {
  static_assert(PER % 32 == 0, "whole warps scan a thread's bins");
  __shared__ unsigned long long warps[32], start[kQuantileRanks];
  __shared__ int owner[kQuantileRanks];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid < nranks) owner[tid] = -1;
  unsigned long long sum = 0;
#pragma unroll
  for (int j = 0; j < PER; j += 4) {
    const int b = tid * PER + j;
    const uint4 v = b < nbins ? __ldg(reinterpret_cast<const uint4*>(bins + b)) : make_uint4(0u, 0u, 0u, 0u);
    sum += (unsigned long long)v.x + v.y + v.z + v.w;
  }
  unsigned long long incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) warps[warp] = incl;
  __syncthreads();
  unsigned long long before = incl - sum;
  for (int w = 0; w < warp; ++w) before += warps[w];
  for (int r = 0; r < nranks; ++r)
    if (ranks[r] >= before && ranks[r] < before + sum) {
      owner[r] = tid;
      start[r] = before;
    }
  __syncthreads();
  if (warp >= nranks || owner[warp] < 0) return;
  const unsigned long long want = ranks[warp] - start[warp];
  unsigned long long base = 0;
#pragma unroll
  for (int j = 0; j < PER; j += 32) {
    const int b = owner[warp] * PER + j + lane;
    const uint32_t c = b < nbins ? bins[b] : 0u;
    unsigned long long in = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long u = __shfl_up_sync(0xffffffffu, in, o);
      if (lane >= o) in += u;
    }
    if (want >= base + in - c && want < base + in) found(warp, b, want - (base + in - c));
    base += __shfl_sync(0xffffffffu, in, 31);
  }
}

// High bins of the ranks: q->target = the distinct ones, q->slot / q->resid =
// each rank's index into them and its rank inside the bin.
__global__ void __launch_bounds__(1024) select_hi_kernel(const uint32_t* __restrict__ hist,
                                                         const unsigned long long* __restrict__ count,
                                                         QuantileState* q) {
  __shared__ uint32_t bin[kQuantileRanks];
  __shared__ unsigned long long rank[kQuantileRanks];
  if (threadIdx.x < kQuantileRanks) {
    bin[threadIdx.x] = 0xffffffffu;
    const unsigned long long n = *count;
    unsigned long long r[2] = {~0ull, ~0ull};  // no such rank
    if (n) quantile_ranks((int)threadIdx.x / 2, n, &r[0], &r[1]);
    rank[threadIdx.x] = threadIdx.x & 1 ? r[1] : r[0];
  }
  __syncthreads();
  find_ranks<32>(hist, kHiBins, rank, kQuantileRanks, [&](int r, int b, unsigned long long resid) {
    bin[r] = (uint32_t)b;
    q->resid[r] = resid;
  });
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t n = 0;
    for (int r = 0; r < kQuantileRanks; ++r) {
      uint32_t j = 0;
      while (j < n && q->target[j] != bin[r]) ++j;
      if (j == n) q->target[n++] = bin[r];
      q->slot[r] = j;
    }
    q->targets = n;
  }
}

// For target j (hi16 value), hist[j * 65536 + lo16] += 1.  A thickness map has
// few different values, each of them many times: a CTA counts the first key that
// falls on each of kHotKeys places in shared memory, the others in the global
// histogram.  Marrow map of 251 x 187 x 203: 40 us with every run of equal keys
// counted there, 15 here.
constexpr int kHotKeys = 1024;
__global__ void __launch_bounds__(512)
hist_lo_kernel(const uint32_t* __restrict__ map, long long n, const QuantileState* __restrict__ q,
               uint32_t* __restrict__ hist) {
  __shared__ uint32_t slots[kHiBins / 4];  // a byte per high bin: its target, or 0xff
  __shared__ uint32_t hot[kHotKeys], times[kHotKeys];
  uint8_t* slot = reinterpret_cast<uint8_t*>(slots);
  for (int i = threadIdx.x; i < kHiBins / 4; i += blockDim.x) slots[i] = 0xffffffffu;
  for (int i = threadIdx.x; i < kHotKeys; i += blockDim.x) {
    hot[i] = 0xffffffffu;
    times[i] = 0u;
  }
  __syncthreads();
  if (threadIdx.x < q->targets && q->target[threadIdx.x] < (uint32_t)kHiBins)
    slot[q->target[threadIdx.x]] = (uint8_t)threadIdx.x;
  __syncthreads();
  each_four(map, n, [&](uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    const uint32_t v[4] = {a, b, c, d};
    uint32_t key[4];
    bool ok[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t s = positive_finite(v[j]) ? slot[v[j] >> 16] : 0xffu;
      ok[j] = s != 0xffu;
      key[j] = s * (uint32_t)kLoBins + (v[j] & 0xffffu);
    }
    add_runs(key, ok, [&](uint32_t k, uint32_t m) {
      const uint32_t at = k * 2654435769u >> 22;  // 10 bits of a multiplicative hash
      uint32_t owner = *static_cast<volatile uint32_t*>(&hot[at]);
      if (owner == 0xffffffffu) {
        owner = atomicCAS(&hot[at], 0xffffffffu, k);
        if (owner == 0xffffffffu) owner = k;
      }
      if (owner == k) atomicAdd(&times[at], m);
      else atomicAdd(&hist[k], m);
    });
  });
  __syncthreads();
  for (int i = threadIdx.x; i < kHotKeys; i += blockDim.x)
    if (times[i]) atomicAdd(&hist[hot[i]], times[i]);
}

// q->bits[r] = the value of rank r (one CTA per rank); 0xffffffff: no such rank.
__global__ void __launch_bounds__(1024) select_lo_kernel(const uint32_t* __restrict__ hist, QuantileState* q) {
  const int r = blockIdx.x;
  const uint32_t slot = q->slot[r], hi = q->target[slot];
  if (threadIdx.x == 0) q->bits[r] = 0xffffffffu;
  __syncthreads();
  if (hi >= (uint32_t)kHiBins) return;
  find_ranks<kLoBins / 1024>(hist + (size_t)slot * kLoBins, kLoBins, &q->resid[r], 1,
                             [&](int, int b, unsigned long long) { q->bits[r] = (hi << 16) | (uint32_t)b; });
}

// Exact moment sums of f32(raw * scale) over the finite positive raw values
// (metrics.rs:215-226), same accumulator as the cleanup kernel.  A warp adds
// its values in fixed point relative to the largest exponent it meets first
// (span of 16 exponents: squares shifted by at most 30 bits, 78 bits each and 96
// a thread, no atomics); values outside go to the block's
// per-exponent sums one by one.  At the end the fixed-point totals are split
// into the per-exponent sums too: 2^15 units of exponent e are one of e + 15.
constexpr int kMomentSpan = 15;

__global__ void __launch_bounds__(256)
moments_kernel(const uint32_t* __restrict__ map, long long n, float scale, StatsAccum* __restrict__ acc) {
  __shared__ unsigned long long s1[256], sh[256], sl[256];
  __shared__ unsigned long long scount;
  __shared__ uint32_t smax;
  for (int i = threadIdx.x; i < 256; i += blockDim.x) s1[i] = sh[i] = sl[i] = 0;
  if (threadIdx.x == 0) {
    scount = 0;
    smax = 0;
  }
  __syncthreads();
  uint32_t thread_cnt = 0;
  unsigned long long fx1 = 0;
  uint32_t f0 = 0, f1 = 0, f2 = 0;  // the fixed-point sum of squares
  uint32_t mx = 0, base = 0;  // base: the exponent of the fixed-point unit (0: not chosen yet; the same in all lanes)
  each_four(map, n, [&](uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    const uint32_t raw[4] = {a, b, c, d};
    uint32_t v[4];
    uint32_t top;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool ok = positive_finite(raw[j]);
      v[j] = ok ? __float_as_uint(__fmul_rn(__uint_as_float(raw[j]), scale)) : 0u;
      thread_cnt += ok;
    }
    top = __vimax3_u32(v[0], v[1], max(v[2], v[3]));
    mx = max(mx, top);
    if (base == 0u) {
      const uint32_t e = __reduce_max_sync(0xffffffffu, top) >> 23;
      if (e) base = min(e > 12u ? e - 12u : 1u, 255u - kMomentSpan);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t e = max(v[j] >> 23, 1u), m = (v[j] & 0x7fffffu) | (v[j] >> 23 ? 0x800000u : 0u);
      const uint32_t s = e - base;
      const unsigned long long m2 = (unsigned long long)m * m;
      if (base && s <= (uint32_t)kMomentSpan) {
        const uint32_t w0 = (uint32_t)m2, w1 = (uint32_t)(m2 >> 32), by = 2u * s;
        fx1 += (unsigned long long)m << s;
        asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, %5;"
            : "+r"(f0), "+r"(f1), "+r"(f2)
            : "r"(w0 << by), "r"(__funnelshift_l(w0, w1, by)), "r"(__funnelshift_l(w1, 0u, by)));
      } else if (m) {
        atomicAdd(&s1[e], (unsigned long long)m);
        atomicAdd(&sh[e], m2 >> 24);
        atomicAdd(&sl[e], m2 & 0xffffffull);
      }
    }
  });
  unsigned long long cnt = thread_cnt, lo = (unsigned long long)f1 << 32 | f0, hi = f2;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    fx1 += __shfl_xor_sync(0xffffffffu, fx1, o);
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    const unsigned long long ol = __shfl_xor_sync(0xffffffffu, lo, o), oh = __shfl_xor_sync(0xffffffffu, hi, o);
    const unsigned long long t = lo + ol;
    hi += oh + (t < lo ? 1u : 0u);
    lo = t;
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((threadIdx.x & 31) == 0 && cnt) {
    atomicAdd(&scount, cnt);
    atomicMax(&smax, mx);
    if (base) {
      const unsigned __int128 rest = (((unsigned __int128)hi << 64) | lo) >> (2 * kMomentSpan);
      atomicAdd(&s1[base], fx1 & ((1ull << kMomentSpan) - 1ull));
      atomicAdd(&s1[base + kMomentSpan], fx1 >> kMomentSpan);
      atomicAdd(&sl[base], lo & 0xffffffull);
      atomicAdd(&sh[base], (lo >> 24) & ((1ull << (2 * kMomentSpan - 24)) - 1ull));
      atomicAdd(&sl[base + kMomentSpan], (unsigned long long)rest & 0xffffffull);
      atomicAdd(&sh[base + kMomentSpan], (unsigned long long)(rest >> 24));
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 256; i += blockDim.x) {
    if (s1[i]) atomicAdd(&acc->sum_m[i], s1[i]);
    if (sh[i]) atomicAdd(&acc->sq_hi[i], sh[i]);
    if (sl[i]) atomicAdd(&acc->sq_lo[i], sl[i]);
  }
  if (threadIdx.x == 0) {
    if (scount) atomicAdd(&acc->count, scount);
    if (smax) atomicMax(&acc->max_bits, smax);
  }
}

// CTAs for n words at per_cta words each, at most cap.
inline unsigned ctas_for(long long n, long long per_cta, long long cap) {
  long long b = (n + per_cta - 1) / per_cta;
  if (b > cap) b = cap;
  return (unsigned)(b < 1 ? 1 : b);
}

}  // namespace

cudaError_t launch_moments(const float* map, long long n, float scale, StatsAccum* acc, cudaStream_t s,
                           unsigned long long* launches) {
  moments_kernel<<<ctas_for(n, 4096, 152 * 6), 256, 0, s>>>(reinterpret_cast<const uint32_t*>(map), n, scale, acc);
  ++*launches;
  return cudaGetLastError();
}

size_t quantile_scratch_words() { return (size_t)kHiBins + (size_t)kQuantileRanks * kLoBins; }

cudaError_t launch_quantiles(const float* map, long long n, const unsigned long long* count, uint32_t* scratch,
                             QuantileState* q, cudaStream_t s, unsigned long long* launches) {
  const uint32_t* words = reinterpret_cast<const uint32_t*>(map);
  uint32_t* lo = scratch + kHiBins;
  const size_t hi_bytes = (size_t)kHiBins * sizeof(uint32_t);
  cudaError_t e = cudaMemsetAsync(scratch, 0, quantile_scratch_words() * sizeof(uint32_t), s);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(hist_hi_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hi_bytes);
  if (e != cudaSuccess) return e;
  hist_hi_kernel<<<ctas_for(n, 16384, 152), 1024, hi_bytes, s>>>(words, n, scratch);
  select_hi_kernel<<<1, 1024, 0, s>>>(scratch, count, q);
  hist_lo_kernel<<<ctas_for(n, 8192, 152 * 4), 512, 0, s>>>(words, n, q, lo);
  select_lo_kernel<<<kQuantileRanks, 1024, 0, s>>>(lo, q);
  *launches += 4;
  return cudaGetLastError();
}

}  // namespace bm
