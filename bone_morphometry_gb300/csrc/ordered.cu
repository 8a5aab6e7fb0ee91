// The statistics' f64 sums in the reference's own order (metrics.rs:215-226).
//
// nonzero_stats adds v = (raw * scale_f32) as f64 and v * v, one value after
// the other in index order, into two f64 accumulators.  Its mean and SD are
// functions of those two rounded sums, so reproducing them bit for bit means
// reproducing every rounding of that sequence.  This file does it in parallel.
//
// The idea.  Let s be the running sum.  While s stays inside one binade
// [2^E, 2^(E+1)), every representable value there is a multiple of
// U = 2^(E-52), so s + v rounds to s + (v rounded to a multiple of U) -- an
// integer increment of s/U that depends on v and E only, except when v's
// remainder is exactly U/2: then round-to-nearest-even picks the increment
// that makes s/U even, which depends on the parity of s/U.  So within one
// binade an element is a function of the parity P of s/U:
//     P -> (increment(P), new parity(P)),
// and a run of elements composes into a function of the same shape (two
// 64-bit increments and two parity bits).  Composition is associative, so
// runs reduce in parallel, in order.  A run's function is valid if s/U after
// it is at most 2^53 (every intermediate state then stayed in the binade, or
// reached 2^(E+1) exactly, which both roundings agree on); otherwise the run
// crossed into the next binade and its elements are replayed.
//
// The pipeline.  The map is cut into chunks of kChunk voxels in index order,
// 32 chunks make a block.
//   1. approximate sums of v and v*v per chunk (f32, on values scaled by a
//      power of two), per block and per 32, 1024 and 32768 blocks (fixed point);
//   2. per chunk, the binade the running sum is predicted to stay in (from the
//      approximate prefix, with a relative margin) and the chunk's function for
//      that binade.  Without a tie a value's increment does not depend on the
//      parity, and increments add up in any order: the lanes sum them.  A chunk
//      with a tie (or +inf) is folded in order.  Per block of 32 chunks, and on
//      further levels of 32, the composition when all share one binade;
//   3. a walker per sum.  The blocks whose composition is invalid -- the ~30
//      binade crossings -- are listed by step 2; the walker's warps compose the
//      runs of blocks between them, and inside each of them the chunks before
//      the first and after the last unpredicted chunk.  Then they follow the
//      sequence from s = 0 together: a composed run is one integer addition, an
//      unpredicted chunk is replayed, a value per thread: a scan of the
//      increments finds the value that leaves the binade, and that one is added
//      with an f64 addition, the reference's own operation.
// Every step the walker takes is checked against the exact state, and where a
// prediction does not hold it goes through the levels and, at worst, replays
// every chunk: a wrong prediction costs time, never exactness.  No per-value
// f64 arithmetic outside the crossings: the GB300's f64 rate is a small
// fraction of its f32 and integer rates.  Not a reference function: the
// reference's loop is serial (metrics.rs:215-226).
//
// Per map, against an earlier form (a serial fold per chunk, a one-CTA scan, a
// one-warp walker that went through the levels): 0.07 against 0.22 ms on
// 64 x 56 x 72, 0.26 against 0.50 ms on 33.5 M values, 0.51 against 0.90 ms on
// 512^3.  The second step is bound by the integer ALU pipe, the walker by the
// latency of its replays, some thousand cycles a round of which the 64-bit
// shifts that make the increments are the largest part.  128^3, bone and marrow
// phase: 84 and 97 thousand cycles for the sum, 104 and 127 for the squares; 110
// and 125, 118 and 146 with a round of four barriers per binade of a chunk and a
// reduction per run of predicted chunks.  The chunks' values in shared memory
// beforehand gave nothing.
#include <climits>
#include <cstdint>

#include "kernels.h"

namespace bm {

namespace {

constexpr int kChunk = 256;                      // voxels per chunk
constexpr unsigned long long kTwo53 = 1ull << 53;
constexpr unsigned long long kSat = 1ull << 54;  // saturated increment: never valid
// Relative margin of the binade prediction.  The approximate prefix sums come
// from f32 chunk sums in fixed point (errors of ~2^-21 of a chunk each,
// shrinking relative to the prefix as it grows); the sequential sum differs
// from the exact prefix by ~sqrt(k) 2^-53.  A miss only sends a chunk to the
// replay.
constexpr int kMarginBits = 24;
// Fixed-point scale of the approximate sums (values scaled into [1, 2)):
// 2^24 units per unit, so a 2^32-voxel map's sums of squares fit 64 bits.
constexpr int kFixBits = 24;
constexpr float kFix = 16777216.0f;

// meta word of a function: 0 = invalid (no prediction); bit 2 = identity valid
// in every binade; else bits 3.. hold E + 2048; bits 0, 1 = out parity for
// input parity 0, 1.
struct Fn {
  unsigned long long i0, i1;
  uint32_t meta;
};

__device__ __forceinline__ unsigned long long sat_add(unsigned long long a, unsigned long long b) {
  const unsigned long long c = a + b;
  return (c >= kSat || c < a) ? kSat : c;
}

__device__ __forceinline__ Fn fn_identity() { return Fn{0ull, 0ull, 4u | 2u}; }

__device__ __forceinline__ uint32_t meta_of(int E, uint32_t o0, uint32_t o1) {
  return ((uint32_t)(E + 2048) << 3) | o0 | (o1 << 1);
}

// F then G.  Binades: an identity-everywhere side takes the other's; two
// different binades, or an invalid side, give invalid.
__device__ __forceinline__ Fn compose(const Fn& F, const Fn& G) {
  if (F.meta == 0u || G.meta == 0u) return Fn{0ull, 0ull, 0u};
  const uint32_t f0 = F.meta & 1u, f1 = (F.meta >> 1) & 1u;
  Fn H;
  H.i0 = sat_add(F.i0, f0 ? G.i1 : G.i0);
  H.i1 = sat_add(F.i1, f1 ? G.i1 : G.i0);
  const uint32_t h0 = (G.meta >> f0) & 1u, h1 = (G.meta >> f1) & 1u;
  const bool fw = (F.meta & 4u) != 0u, gw = (G.meta & 4u) != 0u;
  uint32_t ebits;
  if (fw && gw) {
    ebits = 4u;
  } else if (fw) {
    ebits = G.meta & ~7u;
  } else if (gw) {
    ebits = F.meta & ~7u;
  } else {
    if ((F.meta >> 3) != (G.meta >> 3)) return Fn{0ull, 0ull, 0u};
    ebits = F.meta & ~7u;
  }
  H.meta = ebits | h0 | (h1 << 1);
  return H;
}

__device__ __forceinline__ Fn shfl_fn(const Fn& f, int src) {
  Fn r;
  r.i0 = __shfl_sync(0xffffffffu, f.i0, src);
  r.i1 = __shfl_sync(0xffffffffu, f.i1, src);
  r.meta = __shfl_sync(0xffffffffu, f.meta, src);
  return r;
}

__device__ __forceinline__ Fn shfl_down_fn(const Fn& f, int o) {
  Fn r;
  r.i0 = __shfl_down_sync(0xffffffffu, f.i0, o);
  r.i1 = __shfl_down_sync(0xffffffffu, f.i1, o);
  r.meta = __shfl_down_sync(0xffffffffu, f.meta, o);
  return r;
}

// In-order reduction of the warp's 32 functions (lane 0 first); result in lane 0.
__device__ __forceinline__ Fn warp_reduce_fn(Fn f, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const Fn g = shfl_down_fn(f, o);
    if ((lane & (2 * o - 1)) == 0 && lane + o < 32) f = compose(f, g);
  }
  return f;
}

// The value nonzero_stats adds for a map entry (metrics.rs:216-224): v =
// raw * scale_f32 in f32, then x = v as f64 (or x * x for the sum of squares,
// exact in f64), as an integer mantissa and a power of two, x = M * 2^k (M = 0
// when the entry is skipped or v is 0; k = INT_MAX marks +inf).
struct Term {
  unsigned long long M;
  int k;
};

__device__ __forceinline__ Term term(float raw, float scale, bool sq) {
  Term t{0ull, 0};
  if (!(raw > 0.0f) || !isfinite(raw)) return t;
  const uint32_t b = __float_as_uint(__fmul_rn(raw, scale));
  const uint32_t ef = (b >> 23) & 0xffu;
  unsigned long long m = b & 0x7fffffu;
  if (ef == 0xffu) {  // the f32 product overflowed: +inf
    t.M = ~0ull;
    t.k = INT_MAX;
    return t;
  }
  if (ef) m |= 1ull << 23;
  if (m == 0) return t;
  const int e = (ef ? (int)ef : 1) - 150;
  t.M = sq ? m * m : m;
  t.k = sq ? 2 * e : e;
  return t;
}

// x itself, for the additions made in f64 (a binade crossing, the first value).
__device__ __forceinline__ double term_value(float raw, float scale, bool sq) {
  const double v = (double)__fmul_rn(raw, scale);
  return sq ? __dmul_rn(v, v) : v;
}

__device__ __forceinline__ int binade_of(double s) {
  return (int)((__double_as_longlong(s) >> 52) & 0x7ff) - 1023;
}

__device__ __forceinline__ unsigned long long units_of(double s) {  // s / 2^(E-52), in [2^52, 2^53)
  return ((unsigned long long)__double_as_longlong(s) & ((1ull << 52) - 1ull)) | (1ull << 52);
}

__device__ __forceinline__ double from_units(unsigned long long u, int E) {  // u in [2^52, 2^53]
  if (u == kTwo53) return __longlong_as_double((long long)(E + 1 + 1023) << 52);
  return __longlong_as_double(((long long)(E + 1023) << 52) | (long long)(u & ((1ull << 52) - 1ull)));
}

// Apply f to s (s > 0, finite); false (s unchanged) when f does not hold there.
__device__ __forceinline__ bool apply_fn(const Fn& f, double& s) {
  if (f.meta == 0u) return false;
  if (f.meta & 4u) return true;  // identity
  const int E = binade_of(s);
  if ((int)(f.meta >> 3) - 2048 != E) return false;
  const unsigned long long u = units_of(s);
  const unsigned long long nu = sat_add(u, (u & 1ull) ? f.i1 : f.i0);
  if (nu > kTwo53) return false;
  s = from_units(nu, E);
  return true;
}

__device__ __forceinline__ void load8(const float* __restrict__ map, long long n, long long base, float (&v)[8]) {
  if (base + 8 <= n && (reinterpret_cast<uintptr_t>(map + base) & 15u) == 0) {
    const float4 a = *reinterpret_cast<const float4*>(map + base);
    const float4 b = *reinterpret_cast<const float4*>(map + base + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = base + j < n ? map[base + j] : 0.0f;
  }
}

// Clamped f32 exponent field of the map's largest value v = raw * scale_f32.
__device__ __forceinline__ int max_exponent_field(uint32_t maxbits) {
  const int ef = (int)((maxbits >> 23) & 0xffu);
  return ef < 1 ? 1 : ef > 253 ? 253 : ef;
}

// Power of two that brings the largest value of the map into [1, 2): the
// approximate sums run in f32 on values scaled by it (no overflow, even for
// their squares).
__device__ __forceinline__ float norm_factor(uint32_t maxbits) {
  return __uint_as_float((uint32_t)(254 - max_exponent_field(maxbits)) << 23);  // 2^(127 - ef)
}

__device__ __forceinline__ unsigned long long to_fixed(float x) {
  return (unsigned long long)__fmul_rn(x, kFix);
}

constexpr int kSumLevels = 4;      // approximate sums: blocks, and groups of 32, 1024 and 32768 blocks
// Chunks per warp (32 / CPW warps take the 32 chunks of a block): 4 in the first
// step and 8 in the second (4: 1.07 instead of 1.03 ms for the sums of both
// phases of 512^3), or 1 for maps of fewer than kSmallMap values, which are bound
// by a warp's latency.
constexpr long long kSmallMap = 1ll << 22;
constexpr float kEmptyChunk = -0.0f;  // approximate sum of a chunk without values (others have no sign)

struct Sums {
  unsigned long long* s[kSumLevels];
  unsigned long long* q[kSumLevels];
};

// 1. Approximate sums per chunk of v and v^2 (scaled by norm_factor, in f32),
// and per block and group of blocks (fixed point; the groups' sums start at 0).
// One CTA per block; all loads of a warp's chunks are in flight together.
template <int CPW>
__global__ void __launch_bounds__(1024 / CPW)
osum_chunk_kernel(const float* __restrict__ map, long long n, float scale, long long nchunks,
                  const uint32_t* __restrict__ maxbits, float* __restrict__ cs, float* __restrict__ cq, Sums sums) {
  __shared__ unsigned long long sh_s, sh_q;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long blk = blockIdx.x, c0 = blk * 32 + warp * CPW;
  if (threadIdx.x == 0) sh_s = sh_q = 0ull;
  __syncthreads();
  const float nf = norm_factor(*maxbits);
  float v[CPW][8];
#pragma unroll
  for (int j = 0; j < CPW; ++j) load8(map, n, (c0 + j) * kChunk + lane * 8, v[j]);
  unsigned long long ts = 0, tq = 0;
#pragma unroll
  for (int j = 0; j < CPW; ++j) {
    float s = 0.0f, q = 0.0f;
    bool any = false;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const float raw = v[j][t];
      const bool ok = raw > 0.0f && isfinite(raw);
      const float x = ok ? __fmul_rn(__fmul_rn(raw, scale), nf) : 0.0f;
      any = any || ok;
      s += x;
      q += x * x;
    }
    const bool some = __any_sync(0xffffffffu, any);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, o);
      q += __shfl_xor_sync(0xffffffffu, q, o);
    }
    if (lane == 0 && c0 + j < nchunks) {
      cs[c0 + j] = some ? s : kEmptyChunk;
      cq[c0 + j] = q;
    }
    ts += to_fixed(s);
    tq += to_fixed(q);
  }
  if (lane == 0) {
    if (ts) atomicAdd(&sh_s, ts);
    if (tq) atomicAdd(&sh_q, tq);
  }
  __syncthreads();
#pragma unroll
  for (int L = 0; L < kSumLevels; ++L) {
    if (threadIdx.x != L) continue;
    if (L == 0) {
      sums.s[0][blk] = sh_s;
      sums.q[0][blk] = sh_q;
    } else {
      if (sh_s) atomicAdd(sums.s[L] + (blk >> (5 * L)), sh_s);
      if (sh_q) atomicAdd(sums.q[L] + (blk >> (5 * L)), sh_q);
    }
  }
}

// Sum of everything before block blk (whole warp; the same in all lanes).
__device__ __forceinline__ unsigned long long prefix_of(unsigned long long* const (&lv)[kSumLevels], long long blk,
                                                        int lane) {
  unsigned long long t = 0;
#pragma unroll
  for (int L = 0; L < kSumLevels; ++L) {
    const long long at = blk >> (5 * L), first = L + 1 < kSumLevels ? at & ~31ll : 0ll;
    for (long long i = first + lane; i < at; i += 32) t += lv[L][i];  // at most once below the top level
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

// Binade the running sum is predicted to stay in from P to S, both approximate
// (f32 chunk sums in fixed point, hence the margin); 2^(eshift - kFixBits) is
// their unit.  INT_MIN: none.  Integers only: GB300 retires two f64 operations
// per SM and clock.
__device__ __forceinline__ int predict(unsigned long long P, unsigned long long S, int eshift) {
  if (P == 0ull) return INT_MIN;
  const unsigned long long lo = P - (P >> kMarginBits) - 1ull, hi = S + (S >> kMarginBits) + 1ull;
  if (lo == 0ull) return INT_MIN;
  const int e0 = 63 - __clzll((long long)lo), e1 = 63 - __clzll((long long)hi);
  return e0 == e1 ? e0 - kFixBits + eshift : INT_MIN;
}

struct Level {
  unsigned long long* i0;
  unsigned long long* i1;
  uint32_t* meta;
};

__device__ __forceinline__ void store_fn(const Level& L, long long i, const Fn& f) {
  L.i0[i] = f.i0;
  L.i1[i] = f.i1;
  L.meta[i] = f.meta;
}

__device__ __forceinline__ Fn load_fn(const Level& L, long long i) { return Fn{L.i0[i], L.i1[i], L.meta[i]}; }

// A chunk's function accumulated element by element by one thread: the
// increments and output parities for input parity 0 and 1 (no saturation
// needed inside a chunk: kChunk increments of at most 2^54 fit 64 bits).
struct Acc {
  unsigned long long i0, i1;
  uint32_t o0, o1;
};

// Adds the element M * 2^k to acc for the binade whose ulp is 2^em52; mbits
// bounds M (M < 2^mbits).
__device__ __forceinline__ void acc_elem(Acc& A, unsigned long long M, int k, int em52, int mbits) {
  if (k == INT_MAX) {  // +inf: never within a binade
    A.i0 = A.i1 = kSat;
    return;
  }
  const int sh = em52 - k;
  unsigned long long c;
  if (sh <= 0) {
    c = (sh <= -54 || (M >> (54 + sh)) != 0) ? kSat : (M << -sh);  // M * 2^-sh >= 2^54: saturated
  } else if (sh > mbits) {
    return;  // below half an ulp: lost
  } else {
    const unsigned long long a = M >> sh, rem = M & ((1ull << sh) - 1ull), half = 1ull << (sh - 1);
    if (rem == half) {  // a tie: the increment that leaves s/U even, for each input parity
      A.i0 += a + ((A.o0 + a) & 1ull);
      A.i1 += a + ((A.o1 + a) & 1ull);
      A.o0 = 0u;
      A.o1 = 0u;
      return;
    }
    c = a + (rem > half ? 1ull : 0ull);
  }
  A.i0 += c;
  A.i1 += c;
  A.o0 ^= (uint32_t)(c & 1ull);
  A.o1 ^= (uint32_t)(c & 1ull);
}

// A run whose total increment does not depend on the parity.
__device__ __forceinline__ Fn plain_fn(unsigned long long inc, int E) {
  if (E == INT_MIN) return Fn{0ull, 0ull, 0u};
  const uint32_t p = (uint32_t)(inc & 1ull);
  if (inc > kSat) inc = kSat;
  return Fn{inc, inc, meta_of(E, p, p ^ 1u)};
}

__device__ __forceinline__ Fn acc_fn(const Acc& A, bool any, int E) {
  if (!any) return fn_identity();
  if (E == INT_MIN) return Fn{0ull, 0ull, 0u};
  return Fn{A.i0 >= kSat ? kSat : A.i0, A.i1 >= kSat ? kSat : A.i1, meta_of(E, A.o0, A.o1)};
}

constexpr int kMaxLevels = 8;
constexpr int kMaxMixed = 256;  // blocks with a crossing the walker prepares (more: it goes through all levels)

struct Walk {
  Level lv[kMaxLevels];  // lv[0]: chunks; lv[L]: blocks of 32^L chunks
  long long cnt[kMaxLevels];
  int nlev;
  uint32_t* mixed;  // [0]: number of blocks without a valid composition, then their indexes (any order)
};

// The functions of chunk c folded in order (whole warp; the same in all lanes):
// lane l folds values 8 l .. 8 l + 7, then the lanes' functions are composed.
struct FnPair {
  Fn s, q;
};
__device__ __noinline__ FnPair ordered_fold(const float* __restrict__ map, long long n, float scale, long long c, int es,
                                            int eq, int lane) {
  float w[8];
  load8(map, n, c * kChunk + lane * 8, w);
  Acc a{0ull, 0ull, 0u, 1u}, q{0ull, 0ull, 0u, 1u};
  bool has = false;
#pragma unroll 1
  for (int t = 0; t < 8; ++t) {
    float v = w[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) v = t == j ? w[j] : v;
    const Term x = term(v, scale, false);
    if (!x.M) continue;
    has = true;
    const bool inf = x.k == INT_MAX;
    if (es != INT_MIN) acc_elem(a, x.M, x.k, es - 52, 24);
    if (eq != INT_MIN) acc_elem(q, inf ? x.M : x.M * x.M, inf ? INT_MAX : 2 * x.k, eq - 52, 48);
  }
  return FnPair{shfl_fn(warp_reduce_fn(acc_fn(a, has, es), lane), 0),
                shfl_fn(warp_reduce_fn(acc_fn(q, has, eq), lane), 0)};
}

// v << n, 0 for n >= 32.
__device__ __forceinline__ uint32_t shifted_left(uint32_t v, uint32_t n) {
  uint32_t r;
  asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(v), "r"(n));
  return r;
}

// Sum over the warp (modulo 2^64), in parts whose sums fit 32 bits.
__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
  const uint32_t lo = (uint32_t)v, hi = (uint32_t)(v >> 32);
  const uint32_t a = __reduce_add_sync(0xffffffffu, lo & 0xffffu), b = __reduce_add_sync(0xffffffffu, lo >> 16);
  const uint32_t h = __reduce_add_sync(0xffffffffu, hi);
  return a + ((unsigned long long)b << 16) + ((unsigned long long)h << 32);
}

// 2. Functions of every chunk, for both sums, and of every block.  One CTA per
// block; a chunk without values is not read again.
template <int CPW>
__global__ void __launch_bounds__(1024 / CPW)
osum_fn_kernel(const float* __restrict__ map, long long n, float scale, long long nchunks,
               const uint32_t* __restrict__ maxbits, const float* __restrict__ cs, const float* __restrict__ cq,
               Sums sums, Walk ws, Walk wq) {
  __shared__ Fn sh[2][32];
  __shared__ int binade[2][32];
  static_assert(CPW <= 16, "two warps predict");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long blk = blockIdx.x, b0 = blk * 32;
  const float my_s = b0 + lane < nchunks ? cs[b0 + lane] : kEmptyChunk;
  const unsigned filled = __ballot_sync(0xffffffffu, __float_as_uint(my_s) != __float_as_uint(kEmptyChunk));
  const bool vec = (reinterpret_cast<uintptr_t>(map) & 15u) == 0;
  auto load = [&](int j, float (&x)[8]) {  // any order within the chunk: coalesced
    const int c = warp * CPW + j;
    const long long at = (b0 + c) * kChunk + lane * 4;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long long i = at + h * 128;
      if (!((filled >> c) & 1u)) {
        x[4 * h] = x[4 * h + 1] = x[4 * h + 2] = x[4 * h + 3] = 0.0f;
      } else if (vec && i + 4 <= n) {
        const float4 y = *reinterpret_cast<const float4*>(map + i);
        x[4 * h] = y.x; x[4 * h + 1] = y.y; x[4 * h + 2] = y.z; x[4 * h + 3] = y.w;
      } else {
#pragma unroll
        for (int t = 0; t < 4; ++t) x[4 * h + t] = i + t < n ? map[i + t] : 0.0f;
      }
    }
  };
  float next[8];
  load(0, next);
  // the chunks' predicted binades: those of the sum by warp 0, of the squares by warp 1
  if (warp < 2) {
    int e = INT_MIN;
    if (filled) {
      const float* approx = warp ? cq : cs;
      const unsigned long long mine = b0 + lane < nchunks ? to_fixed(approx[b0 + lane]) : 0ull;
      unsigned long long p = mine;  // inclusive scan within the block
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long u = __shfl_up_sync(0xffffffffu, p, o);
        if (lane >= o) p += u;
      }
      p += prefix_of(warp ? sums.q : sums.s, blk, lane);
      // the approximate sums are of values scaled by 2^(127 - ef): undo it in the binade
      const int shift = max_exponent_field(*maxbits) - 127;
      e = predict(p - mine, p, warp ? 2 * shift : shift);
    }
    binade[warp][lane] = e;
  }
  __syncthreads();
#pragma unroll 1
  for (int j = 0; j < CPW; ++j) {
    float v[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) v[t] = next[t];
    if (j + 1 < CPW) load(j + 1, next);
    const int c = warp * CPW + j;
    if (!((filled >> c) & 1u)) {
      if (lane == 0) {
        sh[0][c] = sh[1][c] = fn_identity();
        if (b0 + c < nchunks) {
          store_fn(ws.lv[0], b0 + c, fn_identity());
          store_fn(wq.lv[0], b0 + c, fn_identity());
        }
      }
      continue;
    }
    const int es = binade[0][c], eq = binade[1][c];
    // M = 0 (an increment of 0) for the entries that are skipped
    uint32_t bits[8], top = 0u, low = ~0u;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const bool ok = __float_as_uint(v[t]) - 1u < 0x7f7fffffu;  // positive and finite
      bits[t] = ok ? __float_as_uint(__fmul_rn(v[t], scale)) : 0u;
    }
#pragma unroll
    for (int t = 0; t < 8; t += 2) {
      top = __vimax3_u32(top, bits[t], bits[t + 1]);
      low = __vimin3_u32(low, bits[t] - 1u, bits[t + 1] - 1u);  // (the skipped ones go to the top)
    }
    top = __reduce_max_sync(0xffffffffu, top) >> 23;
    low = (__reduce_min_sync(0xffffffffu, low) + 1u) >> 23;
    // The usual chunk: normal values over at most 8 binades.  In units of the
    // lowest one's ulp 2^k a value is a 31-bit integer m, and all are rounded
    // at the same bit: m at bit sha, m^2 (one multiplication that adds half an
    // ulp too) at bit shq.
    const int k = (int)low - 150;
    const int sha = es == INT_MIN ? 0 : es - 52 - k, shq = eq == INT_MIN ? 40 : eq - 52 - 2 * k;
    Fn fs, fq;
    bool odd = true;
    unsigned long long A = 0, Q = 0;
    if (low > 0u && top < 255u && top - low <= 7u && sha >= -23 && sha <= 31 && shq >= 1 && shq <= 62) {
      const unsigned ra = (unsigned)max(sha, 0);
      const uint32_t half_a = (1u << ra) >> 1, mask_a = (1u << ra) - 1u, tie_a = ra ? 0u : 1u;
      const unsigned long long half_q = 1ull << (shq - 1);
      const uint32_t base = low << 23;
      odd = false;
      auto sum = [&](auto&& shift_q) {
        uint32_t pair = 0;
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          // (a skipped entry's 0 - base is shifted by 258 or more: 0)
          const uint32_t m = shifted_left((bits[t] & 0x7fffffu) | 0x800000u, (bits[t] - base) >> 23);
          const uint32_t ta = m + half_a;
          odd = odd || (ta & mask_a) == tie_a;
          if (t & 1) A += pair + (ta >> ra);  // each below 2^31
          else pair = ta >> ra;
          shift_q((unsigned long long)m * m + half_q);
        }
      };
      if (shq >= 32) {
        const unsigned rq = (unsigned)shq - 32u;
        const uint32_t mask = (1u << rq) - 1u;
        sum([&](unsigned long long tq) {
          const uint32_t hi = (uint32_t)(tq >> 32);
          odd = odd || ((hi & mask) | (uint32_t)tq) == 0u;
          Q += hi >> rq;
        });
      } else {
        const unsigned rq = (unsigned)shq;
        const uint32_t mask = (1u << rq) - 1u;
        sum([&](unsigned long long tq) {
          odd = odd || ((uint32_t)tq & mask) == 0u;
          Q += tq >> rq;
        });
      }
      if (sha < 0) A <<= -sha;
    }
    if (!__any_sync(0xffffffffu, odd)) {
      A = warp_sum(A);
      Q = warp_sum(Q);
      fs = plain_fn(A, es);
      fq = plain_fn(Q, eq);
    } else {
      const FnPair f = ordered_fold(map, n, scale, b0 + c, es, eq, lane);
      fs = f.s;
      fq = f.q;
    }
    if (lane == 0) {
      sh[0][c] = b0 + c < nchunks ? fs : fn_identity();
      sh[1][c] = b0 + c < nchunks ? fq : fn_identity();
      if (b0 + c < nchunks) {
        store_fn(ws.lv[0], b0 + c, fs);
        store_fn(wq.lv[0], b0 + c, fq);
      }
    }
  }
  __syncthreads();
  if (warp > 1) return;
  // warp 0 composes the sum's block function, warp 1 that of the squares
  const Walk& W = warp ? wq : ws;
  const Fn f = warp_reduce_fn(sh[warp][lane], lane);
  if (lane > 0) return;
  store_fn(W.lv[1], blk, f);
  if (f.meta == 0u) {
    const uint32_t p = atomicAdd(&W.mixed[0], 1u);
    if (p < kMaxMixed) W.mixed[1 + p] = (uint32_t)blk;
  }
}

// Next aggregate level: compositions of 32 consecutive entries.
__global__ void __launch_bounds__(256) osum_level_kernel(Level s_in, Level q_in, long long n_in, Level s_out,
                                                         Level q_out) {
  const int lane = threadIdx.x & 31;
  const long long blk = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long i = blk * 32 + lane;
  if (blk * 32 >= n_in) return;
  const Fn fs = warp_reduce_fn(i < n_in ? load_fn(s_in, i) : fn_identity(), lane);
  const Fn fq = warp_reduce_fn(i < n_in ? load_fn(q_in, i) : fn_identity(), lane);
  if (lane == 0) {
    store_fn(s_out, blk, fs);
    store_fn(q_out, blk, fq);
  }
}

// What a run of values adds to a state in units of its binade's ulp, when the
// state is even (inc) and when it is odd (inc + d, d = (int)w >> 2); bits 0 and
// 1 of w: the parity after it.
struct Step {
  unsigned long long inc;
  uint32_t w;
};

constexpr uint32_t kStay = 2u;  // w of a run that adds nothing

__device__ __forceinline__ unsigned long long after_step(unsigned long long u, const Step& f) {
  return u + f.inc + (unsigned long long)((u & 1ull) ? (long long)((int)f.w >> 2) : 0ll);
}

__device__ __forceinline__ Step then(const Step& f, const Step& g) {
  const int d = (int)g.w >> 2, d0 = f.w & 1u ? d : 0, d1 = f.w & 2u ? d : 0;
  const uint32_t o0 = (g.w >> (f.w & 1u)) & 1u, o1 = (g.w >> ((f.w >> 1) & 1u)) & 1u;
  return Step{f.inc + g.inc + (unsigned long long)(long long)d0,
              ((uint32_t)(((int)f.w >> 2) + d1 - d0) << 2) | (o1 << 1) | o0};
}

// Inclusive scan over the warp.
__device__ __forceinline__ void scan_steps(Step& f, int lane) {
#pragma unroll 1
  for (int o = 1; o < 32; o <<= 1) {
    const Step g{__shfl_up_sync(0xffffffffu, f.inc, o), __shfl_up_sync(0xffffffffu, f.w, o)};
    if (lane >= o) f = then(g, f);
  }
}

// Shared memory of a replay; the halves are used in turn.
struct Replay {
  unsigned long long total[2][2][kChunk / 32];  // of the warps' values, in the state's binade and in the next
  uint32_t ties[2][kChunk / 32];                // bit 0: a tie in the state's binade, bit 1: in the next
  Step step[kChunk / 32];                       // the warps' values with their ties
  unsigned long long rest[2];
  double s[2];
  int next[2];
  uint32_t has[kChunk / 32];
  double first;
};

// Replays chunk c from state s exactly as the reference adds, by a CTA of kChunk
// threads that all hold s, a value per thread.  In s's binade every value is an
// increment; a scan of them gives the state after each value, and the first
// value that leaves the binade (or the first value at all, s = 0) is added with
// an f64 addition, the reference's own operation (metrics.rs:223-224).  The
// values after it go on in the next binade, whose increments are scanned beside
// the first ones: a chunk with one crossing and no tie takes one round of two
// barriers.  An increment that is a tie depends on the parity before it: where
// there are any, the warps scan their values as functions of the parity.
__device__ __noinline__ double replay_chunk(const float* __restrict__ map, long long n, float scale, bool sq,
                                            long long c, double s, Replay& sh) {
  constexpr int kWarps = kChunk / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long at = c * kChunk + tid;
  const float raw = at < n ? map[at] : 0.0f;
  const Term t = term(raw, scale, sq);
  const bool inf = t.k == INT_MAX;
  int start = 0;     // the first value not yet added
  __syncthreads();   // the last replay's results have been read
  if (s == 0.0) {
    const unsigned has = __ballot_sync(0xffffffffu, t.M != 0ull);
    if (lane == 0) sh.has[warp] = has;
    __syncthreads();
    int b = kChunk;
#pragma unroll
    for (int w = kWarps - 1; w >= 0; --w)
      if (sh.has[w]) b = w * 32 + __ffs(sh.has[w]) - 1;
    if (b == kChunk) return s;
    if (tid == b) sh.first = term_value(raw, scale, sq);
    __syncthreads();
    s = sh.first;
    start = b + 1;
  }
#pragma unroll 1
  for (int turn = 0; start < kChunk; turn ^= 1) {
    if (!isfinite(s)) return s;  // +inf stays +inf
    const int E = binade_of(s), sft = E - 52 - (inf ? 0 : t.k);
    // a, and what is left below it: nothing, less than, exactly or more than half an ulp
    unsigned long long a = 0;
    bool left = false, tie = false;
    uint32_t up = 0;
    if (t.M != 0ull && tid >= start) {
      if (inf || sft <= -54 || (sft < 0 && (t.M >> (54 + sft)) != 0ull)) {
        a = kSat;  // leaves the binade
      } else if (sft <= 0) {
        a = t.M << -sft;
      } else if (sft <= 48) {
        a = t.M >> sft;
        const unsigned long long rem = t.M << (64 - sft);  // M < 2^48: at the top of 64 bits
        left = rem != 0ull;
        tie = rem == 1ull << 63;
        up = rem > 1ull << 63 ? 1u : 0u;
      } else {
        left = true;
      }
    }
    const uint32_t odd = (uint32_t)a & 1u;
    unsigned long long f = a + up, g = (a >> 1) + (odd && left ? 1u : 0u);
    const uint32_t ties =
        (__any_sync(0xffffffffu, tie) ? 1u : 0u) | (__any_sync(0xffffffffu, odd && !left) ? 2u : 0u);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long f2 = __shfl_up_sync(0xffffffffu, f, o), g2 = __shfl_up_sync(0xffffffffu, g, o);
      if (lane >= o) {
        f += f2;
        g += g2;
      }
    }
    if (lane == 31) {
      sh.total[turn][0][warp] = f;
      sh.total[turn][1][warp] = g;
      sh.ties[turn][warp] = ties;
    }
    __syncthreads();
    uint32_t all = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) all |= sh.ties[turn][w];
    Step own{f, kStay};
    if (all & 1u) {
      const unsigned long long inc = a + up;
      const uint32_t p = (uint32_t)(inc & 1ull);
      own = tie ? (p ? Step{inc + 1ull, (uint32_t)-4} : Step{inc, 4u}) : Step{inc, p | ((p ^ 1u) << 1)};
      scan_steps(own, lane);
      if (lane == 31) sh.step[warp] = own;
      __syncthreads();
    }
    unsigned long long u = units_of(s), before = 0;
    int wb = -1;  // the warp whose values leave the binade: the states only grow
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const unsigned long long v = all & 1u ? after_step(u, sh.step[w]) : u + sh.total[turn][0][w];
      if (wb < 0 && v > kTwo53) {
        wb = w;
        before = u;
      }
      u = v;
    }
    if (wb < 0) return from_units(u, E);
    if (warp == wb) {
      const unsigned long long after = all & 1u ? after_step(before, own) : before + f;
      const int b = __popc(__ballot_sync(0xffffffffu, after <= kTwo53));
      const unsigned long long prev = __shfl_up_sync(0xffffffffu, after, 1);
      if (lane == b) {
        sh.s[turn] = __dadd_rn(from_units(lane ? prev : before, E), term_value(raw, scale, sq));
        sh.next[turn] = wb * 32 + b + 1;
        sh.rest[turn] = sh.total[turn][1][wb] - g;
      }
    }
    __syncthreads();
    s = sh.s[turn];
    start = sh.next[turn];
    if (!(all & 2u) && isfinite(s) && binade_of(s) == E + 1) {
      u = units_of(s) + sh.rest[turn];
#pragma unroll
      for (int w = 0; w < kWarps; ++w)
        if (w > wb) u += sh.total[turn][1][w];
      if (u <= kTwo53) return from_units(u, E + 1);
    }
  }
  return s;
}

// The walker's state is the same in all its threads: every warp makes the same
// steps, and the replays are theirs together.
//
// Follows the sequence through one block whose chunk functions the lanes hold
// (lane j: chunk c0 + j; identity past the map's end), from lane p to lane e.
__device__ __noinline__ double walk_block(const float* __restrict__ map, long long n, float scale, bool sq,
                                          long long c0, const Fn& f, int p, int e, double s, int lane, Replay& sh) {
  // the runs between unpredicted chunks, composed at once: run's lane t holds
  // the chunks from the one after the last unpredicted before t (or p) up to t
  const unsigned bad = __ballot_sync(0xffffffffu, f.meta == 0u);
  const unsigned upto = bad & ((2u << lane) - 1u);
  const int first = max(p, upto ? 32 - __clz(upto) : 0);
  Fn run = first <= lane ? f : fn_identity();
#pragma unroll 1
  for (int o = 1; o < 32; o <<= 1) {
    const Fn g = shfl_fn(run, lane - o);
    if (lane - o >= first) run = compose(g, run);
  }
  while (p <= e) {
    if (!isfinite(s)) break;
    const unsigned next = bad >> p;  // p <= 31
    const int q = min(next ? p + __ffs(next) - 1 : 32, e + 1);  // chunks p .. q - 1 are predicted
    if (q > p) {
      if (!apply_fn(shfl_fn(run, q - 1), s)) break;
      p = q;
      continue;
    }
    s = replay_chunk(map, n, scale, sq, c0 + p, s, sh);
    ++p;
  }
  // where a prediction does not hold
  while (p <= e) {
    if (!isfinite(s)) break;
    const int E = s == 0.0 ? INT_MIN : binade_of(s);
    const bool ok = (f.meta & 4u) || (E != INT_MIN && f.meta != 0u && (int)(f.meta >> 3) - 2048 == E);
    const unsigned stop = __ballot_sync(0xffffffffu, lane >= p && (!ok || lane > e));
    const int t = stop ? __ffs(stop) - 1 : 32;  // chunks p .. t - 1 qualify
    if (t > p) {
      const bool run = lane >= p && lane < t;
      double s2 = s;
      bool moved = E == INT_MIN;  // empty chunks before the first value
      if (!moved) {
        const Fn r = shfl_fn(warp_reduce_fn(run ? f : fn_identity(), lane), 0);
        moved = apply_fn(r, s2);
      }
      if (moved) {
        s = s2;
        p = t;
        continue;
      }
      const Fn f0 = shfl_fn(f, p);  // the run left the binade somewhere: its first chunk alone
      if (t > p + 1 && apply_fn(f0, s)) {
        ++p;
        continue;
      }
    }
    s = replay_chunk(map, n, scale, sq, c0 + p, s, sh);
    ++p;
  }
  return s;
}

// Follows the sequence over chunks c .. end - 1 from state s: the highest level
// whose entry starts at c, does not pass `end` and applies, up to 32 entries of
// it at a time, or a replay of one chunk.
__device__ __noinline__ double walk_range(const float* __restrict__ map, long long n, float scale, bool sq,
                                          const Walk& W, long long c, long long end, double s, int lane, Replay& sh) {
  while (c < end) {
    if (!isfinite(s)) break;  // a value overflowed to +inf: the sum stays +inf
    bool moved = false;
    for (int L = W.nlev - 1; L >= 0 && !moved; --L) {
      const int lg = 5 * L;
      const long long span = 1ll << lg;
      if (c & (span - 1)) continue;
      const long long q = c >> lg;
      // up to 32 entries of this level, but not past the next block of level
      // L + 1, and only whole ones before `end` (the map's last entry may be short)
      long long qe = min((q / 32 + 1) * 32, end >= W.cnt[0] ? W.cnt[L] : end >> lg);
      if (L + 1 == W.nlev) qe = min(q + 32, end >= W.cnt[0] ? W.cnt[L] : end >> lg);
      if (q >= qe) continue;
      const long long i = q + lane;
      const Fn f = i < qe ? load_fn(W.lv[L], i) : Fn{0ull, 0ull, 0u};
      const int E = s == 0.0 ? INT_MIN : binade_of(s);
      const bool ok = (f.meta & 4u) || (E != INT_MIN && f.meta != 0u && (int)(f.meta >> 3) - 2048 == E);
      const unsigned okm = __ballot_sync(0xffffffffu, ok);
      const int t = (~okm) ? __ffs(~okm) - 1 : 32;  // entries 0 .. t-1 qualify
      if (t == 0) continue;
      if (E == INT_MIN) {  // empty chunks before the first value
        c = min((q + t) * span, end);
        moved = true;
        break;
      }
      Fn r = warp_reduce_fn(lane < t ? f : fn_identity(), lane);
      r = shfl_fn(r, 0);
      double s2 = s;
      if (apply_fn(r, s2)) {
        s = s2;
        c = min((q + t) * span, end);
        moved = true;
      } else if (t > 1) {
        // the run left the binade somewhere: take its first entry alone
        const Fn f0 = shfl_fn(f, 0);
        s2 = s;
        if (apply_fn(f0, s2)) {
          s = s2;
          c = min((q + 1) * span, end);
          moved = true;
        }
      }
    }
    if (!moved) {
      s = replay_chunk(map, n, scale, sq, c, s, sh);
      ++c;
    }
  }
  return s;
}

// Composition of level-1 entries a .. b - 1 (whole warp), through the levels.
__device__ Fn compose_blocks(const Walk& W, long long a, long long b, int lane) {
  Fn front = fn_identity(), back = fn_identity();
  for (int L = 1; a < b; ++L) {
    const bool top = L + 1 >= W.nlev;
    const long long head = top ? b : min((a + 31) & ~31ll, b);  // entries up to the next whole group
    for (; a < head; a += 32) {
      const Fn f = a + lane < head ? load_fn(W.lv[L], a + lane) : fn_identity();
      front = compose(front, shfl_fn(warp_reduce_fn(f, lane), 0));
      if (head - a < 32) {
        a = head;
        break;
      }
    }
    if (a >= b) break;
    const long long tail = b & ~31ll;  // a is a multiple of 32 and below b
    if (tail < b) {
      const Fn f = tail + lane < b ? load_fn(W.lv[L], tail + lane) : fn_identity();
      back = compose(shfl_fn(warp_reduce_fn(f, lane), 0), back);
      b = tail;
    }
    a >>= 5;
    b >>= 5;
  }
  return compose(front, back);
}

constexpr int kWalkWarps = kChunk / 32;

// 3. The walker: block 0 follows the sum of values, block 1 the sum of squares.
__global__ void __launch_bounds__(kWalkWarps * 32)
osum_walk_kernel(const float* __restrict__ map, long long n, float scale, Walk ws, Walk wq, double* __restrict__ out) {
  __shared__ uint32_t at[kMaxMixed];                  // the mixed blocks in order
  __shared__ Fn gap[kMaxMixed + 1];                   // the blocks before each of them (and after the last)
  __shared__ Fn pre[kMaxMixed], suf[kMaxMixed];       // their chunks before the first / after the last unpredicted one
  __shared__ uint8_t first[kMaxMixed], last[kMaxMixed];
  __shared__ Replay replay;
  const bool sq = blockIdx.x == 1;
  const Walk& W = sq ? wq : ws;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long nchunks = W.cnt[0], nblocks = W.cnt[1];
  const int nm = (int)W.mixed[0];
  if (nm > kMaxMixed) {  // many wrong predictions: through all levels
    const double s = walk_range(map, n, scale, sq, W, 0, nchunks, 0.0, lane, replay);
    if (tid == 0) out[sq ? 1 : 0] = s;
    return;
  }
  for (int i = tid; i < nm; i += kWalkWarps * 32) {
    const uint32_t me = W.mixed[1 + i];
    int r = 0;
    for (int j = 0; j < nm; ++j) r += W.mixed[1 + j] < me ? 1 : 0;
    at[r] = me;
  }
  __syncthreads();
  for (int t = warp; t < 2 * nm + 1; t += kWalkWarps) {
    const int i = t >> 1;
    if (t & 1) {  // inside mixed block i
      const long long c = (long long)at[i] * 32 + lane;
      const Fn f = c < nchunks ? load_fn(W.lv[0], c) : fn_identity();
      const unsigned bad = __ballot_sync(0xffffffffu, f.meta == 0u);
      const int a = bad ? __ffs(bad) - 1 : 32, b = bad ? 31 - __clz(bad) : 31;
      const Fn p = warp_reduce_fn(lane < a ? f : fn_identity(), lane);
      const Fn q = warp_reduce_fn(lane > b ? f : fn_identity(), lane);
      if (lane == 0) {
        pre[i] = p;
        suf[i] = q;
        first[i] = (uint8_t)a;
        last[i] = (uint8_t)b;
      }
      for (unsigned left = bad; left; left &= left - 1u) {  // the values about to be replayed
        const long long v = ((long long)at[i] * 32 + __ffs(left) - 1) * kChunk + lane * 8;
        if (v < n) asm volatile("prefetch.global.L1 [%0];" ::"l"(map + v));
      }
    } else {  // between mixed blocks i - 1 and i
      const long long a = i ? (long long)at[i - 1] + 1 : 0, b = i < nm ? (long long)at[i] : nblocks;
      const Fn f = compose_blocks(W, a, b, lane);
      if (lane == 0) gap[i] = f;
    }
  }
  __syncthreads();
  double s = 0.0;
  long long block = 0;
  for (int i = 0; i <= nm; ++i) {
    const long long m = i < nm ? (long long)at[i] : nblocks;
    if (m > block && !apply_fn(gap[i], s))
      s = walk_range(map, n, scale, sq, W, block * 32, min(m * 32, nchunks), s, lane, replay);
    if (i == nm) break;
    const long long c0 = m * 32;
    const int a = first[i], b = last[i];
    if (a == b && apply_fn(pre[i], s)) {  // the usual case: one unpredicted chunk
      s = replay_chunk(map, n, scale, sq, c0 + a, s, replay);
      if (apply_fn(suf[i], s)) {
        block = m + 1;
        continue;
      }
      const Fn f = c0 + lane < nchunks ? load_fn(W.lv[0], c0 + lane) : fn_identity();
      s = walk_block(map, n, scale, sq, c0, f, b + 1, 31, s, lane, replay);
    } else {
      const Fn f = c0 + lane < nchunks ? load_fn(W.lv[0], c0 + lane) : fn_identity();
      s = walk_block(map, n, scale, sq, c0, f, 0, 31, s, lane, replay);
    }
    block = m + 1;
  }
  if (tid == 0) out[sq ? 1 : 0] = s;
}

// Entry counts of the levels: chunks, then blocks of 32 per level up to a
// single entry; at least two levels.
int level_counts(long long nchunks, long long* cnt) {
  int nlev = 0;
  long long c = nchunks;
  for (;;) {
    cnt[nlev++] = c;
    if ((nlev >= 2 && c == 1) || nlev == kMaxLevels) break;
    c = (c + 31) / 32;
  }
  return nlev;
}

}  // namespace

namespace {

// The scratch memory's parts, in order; base null: sizes only.
struct Parts {
  char* base;
  size_t used = 0;
  template <class T>
  T* take(long long count) {
    char* r = base ? base + used : nullptr;
    used += ((size_t)count * sizeof(T) + 255) & ~(size_t)255;
    return reinterpret_cast<T*>(r);
  }
};

struct Plan {
  float *cs, *cq;
  Sums sums;
  Walk ws, wq;
  size_t zero_at, zero_bytes;  // the part that starts at 0: group sums, mixed lists
  size_t bytes;
};

Plan plan_of(long long n, void* scratch) {
  const long long nchunks = n > 0 ? (n + kChunk - 1) / kChunk : 1, nblocks = (nchunks + 31) / 32;
  Parts p{static_cast<char*>(scratch)};
  Plan r{};
  r.cs = p.take<float>(nchunks);
  r.cq = p.take<float>(nchunks);
  r.sums.s[0] = p.take<unsigned long long>(nblocks);
  r.sums.q[0] = p.take<unsigned long long>(nblocks);
  long long cnt[kMaxLevels];
  const int nlev = level_counts(nchunks, cnt);
  r.ws.nlev = r.wq.nlev = nlev;
  for (int L = 0; L < nlev; ++L)
    for (Walk* w : {&r.ws, &r.wq}) {
      w->lv[L].i0 = p.take<unsigned long long>(cnt[L]);
      w->lv[L].i1 = p.take<unsigned long long>(cnt[L]);
      w->lv[L].meta = p.take<uint32_t>(cnt[L]);
      w->cnt[L] = cnt[L];
    }
  r.zero_at = p.used;
  for (int L = 1; L < kSumLevels; ++L) {
    const long long groups = ((nblocks - 1) >> (5 * L)) + 1;
    r.sums.s[L] = p.take<unsigned long long>(groups);
    r.sums.q[L] = p.take<unsigned long long>(groups);
  }
  r.ws.mixed = p.take<uint32_t>(1 + kMaxMixed);
  r.wq.mixed = p.take<uint32_t>(1 + kMaxMixed);
  r.zero_bytes = p.used - r.zero_at;
  r.bytes = p.used;
  return r;
}

}  // namespace

size_t ordered_sum_scratch_bytes(long long n) { return plan_of(n, nullptr).bytes; }

cudaError_t launch_ordered_sums(const float* map, long long n, float scale, const uint32_t* maxbits, void* scratch,
                                double* out, cudaStream_t s, unsigned long long* launches) {
  if (n <= 0) return cudaMemsetAsync(out, 0, 2 * sizeof(double), s);
  const Plan p = plan_of(n, scratch);
  const long long nchunks = p.ws.cnt[0];
  const unsigned blocks = (unsigned)p.ws.cnt[1];
  cudaError_t e = cudaMemsetAsync(static_cast<char*>(scratch) + p.zero_at, 0, p.zero_bytes, s);
  if (e != cudaSuccess) return e;
  if (n < kSmallMap) {
    osum_chunk_kernel<1><<<blocks, 1024, 0, s>>>(map, n, scale, nchunks, maxbits, p.cs, p.cq, p.sums);
    osum_fn_kernel<1><<<blocks, 1024, 0, s>>>(map, n, scale, nchunks, maxbits, p.cs, p.cq, p.sums, p.ws, p.wq);
  } else {
    osum_chunk_kernel<4><<<blocks, 256, 0, s>>>(map, n, scale, nchunks, maxbits, p.cs, p.cq, p.sums);
    osum_fn_kernel<8><<<blocks, 128, 0, s>>>(map, n, scale, nchunks, maxbits, p.cs, p.cq, p.sums, p.ws, p.wq);
  }
  *launches += 3;
  for (int L = 2; L < p.ws.nlev; ++L) {
    osum_level_kernel<<<(unsigned)((p.ws.cnt[L] + 7) / 8), 256, 0, s>>>(p.ws.lv[L - 1], p.wq.lv[L - 1], p.ws.cnt[L - 1],
                                                                       p.ws.lv[L], p.wq.lv[L]);
    ++*launches;
  }
  osum_walk_kernel<<<2, kWalkWarps * 32, 0, s>>>(map, n, scale, p.ws, p.wq, out);
  return cudaGetLastError();
}

}  // namespace bm
