// Separable sphere fill (local_thickness.rs:104-202) for sm_103a.
//
// The map to compute is F(v) = max { R : a ridge ball (centre c, squared
// radius R) with |v - c|^2 <= R }, on selected and non-selected voxels alike.
// The test splits by axis: with rho = R - (z - c_z)^2 the ball meets plane z in
// the disc of squared radius rho around (c_x, c_y), and with R - ... - (y -
// c_y)^2 the disc meets row y in a chord.  So the fill runs in two passes, the
// idea of the separable local thickness algorithm of Lovric and others, with
// the lists cut down at each pass by tests that never change the maximum:
//
//   disc_list_kernel   per column (x, y), the discs of its ridge balls at every
//     plane z.  Of the discs (R, rho) of one column and plane, one whose R and
//     rho are both no larger than another's paints nothing of its own; and one
//     whose rho is covered by a disc of the next column over (rho' >= the
//     largest |u + o|^2 over the lattice points |u|^2 <= rho, o the offset)
//     with R' >= R neither.  What is left is a list per 32 x 8 patch and plane.
//   disc_paint_kernel  per 64 x TY tile of a plane, the chords of its discs
//     into a reversed sparse table: a chord of length L writes max R into two
//     cells of level floor(log2 L); the levels are pushed down at the end.
//
// On a 192^3 crop of the 512^3 workload's generator (marrow phase) a ball
// centre meets 5.6 planes per selected voxel and 58.7 rows; the lists hold
// 0.85 discs with 7.4 rows per selected voxel.  Nothing depends
// on the order of the balls, so there is no sort by radius, no list of balls
// per tile and no barrier between radii, and the non-selected voxels on a
// ball's sphere (rho = 0 at the end) come out of the same passes.
#include "disc_cuts.h"
#include "disc_place.h"
#include "kernels.h"

namespace bm {

namespace {

__device__ __forceinline__ uint32_t floor_sqrt(uint32_t t) {
  // t <= kDiscMaxR2 = 127^2.  sqrt(t + 1/2) is at least 1/(4 * 127) = 2e-3 away
  // from every whole number, far more than the error of the hardware reciprocal
  // root (2^-22 relative: 3e-5), so its floor is floor(sqrt(t)).  The conversions
  // go through the f32 mantissa (2^23 + t), which leaves one special-function
  // operation.
  const float f = __uint_as_float(0x4b000000u | t) - 8388607.5f;
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
  return __float_as_uint(__fadd_rz(f * r, 8388608.0f)) & 0x7fffffu;
}

// ---- ridge map --------------------------------------------------------------
// Distance ridge (local_thickness.rs:104-167) as a u16 map: twice the squared
// distance (0 for a non-selected voxel), plus 1 for a ridge voxel.  Two
// adjacent voxels of x per register.  A warp owns 60 x (its outer lanes hold the
// x neighbours) and ROWS rows and walks NZ planes upwards; each plane's rows are
// loaded once and reduced to the maxima that the face, edge and corner tests of
// three planes share, in registers.
//
// Bound by issue and by the gather of the bounds (two per register of selected
// voxels): both phases of 512^3 595 us with a voxel per lane from a 32-bit map,
// 412 here (bytes alone: 160).
constexpr int kMapPairs = 30;
constexpr int kMapWarps = 4;

template <int ROWS, int NZ>
__global__ void __launch_bounds__(kMapWarps * 32)
ridge_map_kernel(const uint32_t* __restrict__ dist, int pairs, int h, int d, const uint2* __restrict__ thr,
                 uint32_t* __restrict__ out, int nxt, int nyt, int nzt) {
  const int lane = threadIdx.x & 31;
  const long long wid = (long long)blockIdx.x * kMapWarps + (threadIdx.x >> 5);
  if (wid >= (long long)nxt * nyt * nzt) return;
  const int xt = (int)(wid % nxt), yt = (int)((wid / nxt) % nyt), zt = (int)(wid / ((long long)nxt * nyt));
  const int x = xt * kMapPairs - 1 + lane, y0 = yt * ROWS, z0 = zt * NZ;
  const int z1 = min(z0 + NZ, d);
  const bool xin = x >= 0 && x < pairs, xout = lane >= 1 && lane <= kMapPairs && x < pairs;
  const long long slice = (long long)pairs * h;
  const uint32_t* src = dist + (long long)(y0 - 1) * pairs + x;
  uint32_t* dst = out + (long long)y0 * pairs + x;
  auto load = [&](int z, uint32_t (&c)[ROWS + 2]) {
    const bool zin = xin && z >= 0 && z < d;
    const uint32_t* p = src + (long long)z * slice;
#pragma unroll
    for (int r = 0; r < ROWS + 2; ++r) c[r] = zin && y0 - 1 + r >= 0 && y0 - 1 + r < h ? p[r * pairs] : 0u;
  };
  // of two voxels and their plane: themselves, their in-plane face neighbours, their in-plane corner neighbours
  struct PlaneMax {
    uint32_t c, m, s;
  };
  auto reduce = [&](const uint32_t (&c)[ROWS + 2], PlaneMax (&p)[ROWS]) {
    uint32_t a[ROWS + 2];  // max of the two x neighbours
#pragma unroll
    for (int r = 0; r < ROWS + 2; ++r) {
      const uint32_t before = __shfl_up_sync(0xffffffffu, c[r], 1), after = __shfl_down_sync(0xffffffffu, c[r], 1);
      a[r] = __vmaxu2(__byte_perm(before, c[r], 0x5432), __byte_perm(c[r], after, 0x5432));
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
      p[r] = PlaneMax{c[r + 1], __vimax3_u16x2(a[r + 1], c[r], c[r + 2]), __vmaxu2(a[r], a[r + 2])};
  };
  uint32_t c[ROWS + 2];
  PlaneMax mid[ROWS], hi[ROWS];
  uint32_t face[ROWS], edge[ROWS], corner[ROWS];  // of plane z, without plane z + 1
  load(z0 - 1, c);
  reduce(c, hi);
  load(z0, c);
  reduce(c, mid);
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
    face[r] = __vmaxu2(mid[r].m, hi[r].c);
    edge[r] = __vmaxu2(mid[r].s, hi[r].m);
    corner[r] = hi[r].s;
  }
  load(z0 + 1, c);
  for (int z = z0; z < z1; ++z) {
    reduce(c, hi);
    if (z + 1 < z1) load(z + 2, c);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const uint32_t R = mid[r].c;
      uint32_t v = 0u;
      if (R) {
        const uint2 t0 = __ldg(thr + (R & 0xffffu)), t1 = __ldg(thr + (R >> 16));  // {face | edge << 16, corner}
        const uint32_t tf = __byte_perm(t0.x, t1.x, 0x5410), te = __byte_perm(t0.x, t1.x, 0x7632),
                       tc = __byte_perm(t0.y, t1.y, 0x5410);
        // a half is 0 where all three maxima are at most their bounds
        const uint32_t over = (__vimax3_u16x2(face[r], hi[r].c, tf) ^ tf) | (__vimax3_u16x2(edge[r], hi[r].m, te) ^ te) |
                              (__vimax3_u16x2(corner[r], hi[r].s, tc) ^ tc);
        v = 2u * R;
        if (!(over & 0xffffu) && (R & 0xffffu)) v |= 1u;
        if (!(over >> 16) && (R >> 16)) v |= 0x10000u;
      }
      if (xout && y0 + r < h) dst[(long long)z * slice + r * pairs] = v;
      face[r] = __vmaxu2(hi[r].m, mid[r].c);
      edge[r] = __vmaxu2(hi[r].s, mid[r].m);
      corner[r] = mid[r].s;
      mid[r] = hi[r];
    }
  }
}

// thr[R] = the largest values that pass the ridge map's three tests of R: its
// search templates (lut, at least 1) less 1;
// tmpl[rho] = the largest |u + o|^2 over the 2-D lattice points |u|^2 <= rho for
// o = (1, 0) in the low and o = (1, 1) in the high half.
__global__ void disc_tables_kernel(const uint4* __restrict__ lut, uint32_t n, uint2* __restrict__ thr,
                                   uint32_t* __restrict__ tmpl) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint4 t = lut[i];
    thr[i] = make_uint2((min(t.x, 0x10000u) - 1u) | ((min(t.y, 0x10000u) - 1u) << 16), min(t.z, 0x10000u) - 1u);
    uint32_t face = 0, corner = 0;
    for (uint32_t a = 0; a * a <= i; ++a) {
      const uint32_t b = floor_sqrt(i - a * a);
      face = max(face, (a + 1) * (a + 1) + b * b);
      corner = max(corner, (a + 1) * (a + 1) + (b + 1) * (b + 1));
    }
    tmpl[i] = min(face, 0xffffu) | (min(corner, 0xffffu) << 16);
  }
}

// ---- disc lists -------------------------------------------------------------
constexpr int kListThreads = 512;
constexpr int kListWarps = kListThreads / 32;
constexpr int kCols = kDiscPX * kDiscPY;   // columns of the patch
constexpr int kRowPad = kDiscPX + 2;       // per-plane table with an empty border of one cell
constexpr int kPlaneCells = (kDiscPY + 2) * kRowPad;
constexpr int kRunLen = 3;                 // planes per run
constexpr int kWalk = 6;                   // planes a thread walks per step
constexpr int kCentres = 4096;             // ball centres a CTA keeps from its first walk
// centres and runs a warp holds back until 32 are ready
constexpr int kCentreQueue = 32 + 32 * kWalk, kRunQueue = 64;

// Cell of patch column c in a plane of the padded table.
__device__ __forceinline__ int cell_of(uint32_t c) { return (int)(c >> 5) * kRowPad + kRowPad + (int)(c & 31u) + 1; }

// One CTA per patch of 32 x 8 columns and NZ planes.  Its threads walk the
// ridge map's columns through the planes and a halo of the largest radius; the
// ball centres they meet are collected per warp, handled 32 at a time, and kept
// for the second step (up to kCentres; beyond, the columns are walked again).
//
// Cut along z: the planes of a centre's discs end where the ball of one of its
// two neighbours in the column covers them, ridge voxel or not (a ball that is
// not on the ridge lies in a larger one that is).  For the neighbour above, with
// R' >= R, rho' - rho grows along z, so it covers this centre's discs from some
// plane on, and the one below up to some plane (of two equal discs the lower
// one stays).  First step: every disc left enters a table of the largest rho of its
// column and plane.  Second step, a thread per run of up to kRunLen discs:
//   - a disc that its own column's largest disc covers (R' >= R, rho' >= rho)
//     or that of one of the six neighbouring columns at x -+ 1 is left out;
//   - the rows of the others are cut at the largest discs of the columns at
//     y -+ 1, as the planes were along z.
// At any row, each of these tests leaves a chord out only for one with R' > R, or
// with R' = R and a larger squared half-length (or an equal one and a lower
// centre).  So of the chords of the largest R that contain a voxel one is left:
// no chain of tests among them closes.
//
// Per selected voxel of the 192^3 marrow phase: 1.55 discs enter the table, 0.85
// discs with 7.4 rows are listed.  Cutting at ridge voxels alone enters 2.0,
// at every centre of the column 1.5, and lists as many; testing the six columns
// at x -+ 2 too lists 0.79 with 6.7 rows, for as much time as it saves.
//
// A plane with more than kDiscSlots discs gets a segment of the overflow pool
// and a third step.
template <int NZ>
__global__ void __launch_bounds__(kListThreads, 2)
disc_list_kernel(const uint16_t* __restrict__ rmap, int pitch, Dims dm, int H, const uint32_t* __restrict__ tmpl, int npx, int npy,
                 uint32_t* __restrict__ hdr, uint2* __restrict__ ent, uint2* __restrict__ pool,
                 unsigned long long pool_cap, Counters* __restrict__ ctr) {
  extern __shared__ uint32_t smem[];
  uint32_t* largest = smem;  // NZ x kPlaneCells: rho << 16 | R
  uint2* centres = reinterpret_cast<uint2*>(largest + NZ * kPlaneCells);  // kCentres
  uint2* queues = centres + kCentres;
  static_assert(NZ <= 32, "a bit per plane");
  __shared__ uint32_t s_count[NZ], s_full, s_centres;  // s_full: planes whose list goes to the pool
  __shared__ uint2* s_dst[NZ];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned below = (1u << lane) - 1u;
  const long long bid = blockIdx.x;
  const int px = (int)(bid % npx), py = (int)((bid / npx) % npy), pz = (int)(bid / ((long long)npx * npy));
  const int z0 = pz * NZ, nz = min(NZ, dm.d - z0);
  const long long slice = (long long)pitch * dm.h;
  const long long plane_hdrs = (long long)npx * npy;
  const long long first_hdr = (long long)z0 * plane_hdrs + (long long)py * npx + px;
  constexpr int kParts = kListThreads / kCols;  // threads per column, each on a part of the planes
  const int cell = tid & (kCols - 1), part = tid / kCols;
  const int x = px * kDiscPX + lane, y = py * kDiscPY + (cell >> 5);
  const bool in = x < dm.w && y < dm.h;
  const uint16_t* src = rmap + (long long)y * pitch + x;
  const int za = max(z0 - H, 0), zb = min(z0 + nz + H, dm.d);
  const int per = (zb - za + kParts - 1) / kParts;
  const int w0 = za + part * per, w1 = min(w0 + per, zb);  // planes this thread walks
  uint2* cq = queues + warp * (kCentreQueue + kRunQueue);
  uint2* rq = cq + kCentreQueue;
  for (int i = tid; i < NZ * kPlaneCells; i += kListThreads) largest[i] = 0u;
  if (tid < NZ) {
    s_count[tid] = 0u;
    s_dst[tid] = ent + (first_hdr + (long long)tid * plane_hdrs) * kDiscSlots;
  }
  if (tid == 0) s_full = s_centres = 0u;
  __syncthreads();
  for (int pass = 0; pass < 3; ++pass) {
    const int kept = pass ? (int)s_centres : 0;
    const bool cached = pass && kept <= kCentres;  // else the columns are walked again
    const uint32_t planes = pass == 2 ? s_full : ~0u;
    int n = 0, nr = 0, z = w0, ci = warp * 32;
    uint32_t v[kWalk + 2];  // planes z - 1 .. z + kWalk
    auto at = [&](int z) -> uint32_t { return in && z >= 0 && z < dm.d ? src[(long long)z * slice] : 0u; };
    uint32_t ahead[kWalk];  // the next step's planes, in flight during this one
    if (!cached) {
      v[0] = at(w0 - 1);
      v[1] = at(w0);
#pragma unroll
      for (int j = 0; j < kWalk; ++j) ahead[j] = at(w0 + 1 + j);
    }
    for (bool final = false; !final;) {
      if (cached) {
        n = max(min(kept - ci, 32), 0);
        final = ci + kListThreads >= kept;
      } else {
#pragma unroll
        for (int j = 0; j < kWalk; ++j) v[2 + j] = ahead[j];
        if (z + kWalk < w1) {
#pragma unroll
          for (int j = 0; j < kWalk; ++j) ahead[j] = at(z + kWalk + 1 + j);
        }
#pragma unroll
        for (int j = 0; j < kWalk; ++j) {
          const int k = z + j - z0;
          const uint32_t R = v[1 + j] & 1u ? v[1 + j] >> 1 : 0u;
          const int far = k < 0 ? -k : max(k - (nz - 1), 0);
          const bool have = z + j < w1 && R != 0u && (int)R >= far * far;  // a centre whose ball meets the planes
          const unsigned m = __ballot_sync(0xffffffffu, have);
          if (have)  // {R | R above << 16, R below | (k + 128) << 15 | column << 24}
            cq[n + __popc(m & below)] = make_uint2(
                R | ((v[2 + j] >> 1) << 16), (v[j] >> 1) | ((uint32_t)(k + 128) << 15) | ((uint32_t)cell << 24));
          n += __popc(m);
        }
        v[0] = v[kWalk];
        v[1] = v[kWalk + 1];
        z += kWalk;
        final = z >= w1;
        __syncwarp();
      }
      while (n >= (final ? 1 : cached ? 1 : 32) || (final && nr > 0)) {
        const int take = min(n, 32);
        n -= take;
        const uint2* from = cached ? centres + ci : cq + n;
        const uint2 c = from[max(min(lane, take - 1), 0)];
        ci += kListThreads;
        const int R = (int)(c.x & 0x7fffu), k = (int)((c.y >> 15) & 511u) - 128;
        const uint32_t cc = c.y >> 24;
        // the planes lo .. hi of its discs
        const int rad = (int)floor_sqrt((uint32_t)R);
        const int up = (int)(c.x >> 16) - R, dn = (int)(c.y & 0x7fffu) - R;
        int hi = min(rad, cut_above(up, up > 0)), lo = max(-rad, cut_below(dn));
        if (up < 0) hi = rad;
        if (dn < 0) lo = -rad;
        lo = max(lo + k, 0);
        hi = lane < take ? min(hi + k, nz - 1) : -1;
        if (pass == 0) {
          const unsigned m = __ballot_sync(0xffffffffu, lo <= hi);
          uint32_t base = 0;
          if (lane == 0 && m) base = atomicAdd(&s_centres, (uint32_t)__popc(m));
          base = __shfl_sync(0xffffffffu, base, 0) + __popc(m & below);
          if (lo <= hi && base < kCentres) centres[base] = c;
          uint32_t* P = largest + lo * kPlaneCells + cell_of(cc);
          for (int i = lo; i <= hi; ++i, P += kPlaneCells)
            atomicMax(P, ((uint32_t)(R - (i - k) * (i - k)) << 16) | (uint32_t)R);
          __syncwarp();
          continue;
        }
        // runs {R | column << 16 | length << 24, first plane | (first plane - centre's + 128) << 8}
        for (bool last = false; !last;) {
          const int run = min(kRunLen, hi - lo + 1);
          const unsigned m = __ballot_sync(0xffffffffu, run > 0 && (planes >> lo & ((1u << run) - 1u)) != 0u);
          if (m >> lane & 1u)
            rq[nr + __popc(m & below)] = make_uint2(
                (uint32_t)R | (cc << 16) | ((uint32_t)run << 24),
                (uint32_t)lo | ((uint32_t)(lo - k + 128) << 8));
          nr += __popc(m);
          lo += kRunLen;
          __syncwarp();
          // a full warp of runs, or what is left at the very end
          last = !__any_sync(0xffffffffu, lo <= hi);
          const bool flush = last && n == 0 && final;
          if (nr < 32 && !(flush && nr > 0)) continue;
          const int rtake = min(nr, 32);
          nr -= rtake;
          const uint2 r = rq[nr + min(lane, rtake - 1)];
          const int Rr = (int)(r.x & 0x7fffu), len = lane < rtake ? (int)(r.x >> 24) : 0;
          const uint32_t rc = (r.x >> 16) & 255u;
          const int k0 = (int)(r.y & 63u), t0 = (int)(r.y >> 8) - 128;
          const uint32_t* P = largest + k0 * kPlaneCells + cell_of(rc);
#pragma unroll 1
          for (int j = 0; j < kRunLen; ++j, P += kPlaneCells) {
            const int t = t0 + j, kk = k0 + j;
            const int rho = Rr - t * t;
            bool keep = j < len;
            int ylo = 0, yhi = 0;
            if (keep) {
              const uint32_t own = ((uint32_t)rho << 16) | (uint32_t)Rr, p = P[0];
              const uint32_t T = __ldg(tmpl + rho);
              const uint32_t nf = (T << 16) | (uint32_t)Rr, nc = (T & 0xffff0000u) | (uint32_t)Rr;
              bool covered = p != own && __vminu2(p, own) == own;
              covered |= __vminu2(P[-1], nf) == nf;
              covered |= __vminu2(P[1], nf) == nf;
              covered |= __vminu2(P[-kRowPad - 1], nc) == nc;
              covered |= __vminu2(P[-kRowPad + 1], nc) == nc;
              covered |= __vminu2(P[kRowPad - 1], nc) == nc;
              covered |= __vminu2(P[kRowPad + 1], nc) == nc;
              const uint32_t a = P[kRowPad], b = P[-kRowPad];
              const int h = (int)floor_sqrt((uint32_t)rho), ra = (int)(a & 0xffffu), rb = (int)(b & 0xffffu);
              yhi = ra >= Rr ? min(h, cut_above((int)(a >> 16) - rho, ra > Rr)) : h;
              ylo = rb >= Rr ? max(-h, cut_below((int)(b >> 16) - rho)) : -h;
              keep = !covered && ylo <= yhi && (planes >> kk & 1u);
            }
            // one counter update per plane and warp
            const unsigned grp = __match_any_sync(0xffffffffu, keep ? kk : -1);
            const int leader = __ffs(grp) - 1;
            uint32_t slot = 0;
            if (keep && lane == leader) slot = atomicAdd(&s_count[kk], (uint32_t)__popc(grp));
            slot = __shfl_sync(0xffffffffu, slot, leader) + __popc(grp & below);
            if (keep && (pass == 2 || slot < kDiscSlots))
              s_dst[kk][slot] = make_uint2(((uint32_t)Rr << 16) | (uint32_t)rho,
                                           rc | ((uint32_t)(ylo + 128) << 8) | ((uint32_t)(yhi + 128) << 16));
          }
          __syncwarp();
          last = last && !(flush && nr > 0);
        }
      }
    }
    __syncthreads();
    if (pass == 0) continue;
    if (pass == 2) break;
    // headers: a warp per plane finds the plane's reach
    for (int k = warp; k < nz; k += kListWarps) {
      uint32_t r = 0;
      for (int i = lane; i < kPlaneCells; i += 32) r = max(r, largest[k * kPlaneCells + i]);
      r = __reduce_max_sync(0xffffffffu, r >> 16);
      if (lane == 0) {
        const uint32_t cnt = s_count[k];
        uint2* list = s_dst[k];
        uint32_t h = cnt | (cnt ? floor_sqrt(r) << 16 : 0u);
        s_dst[k] = nullptr;
        if (cnt > kDiscSlots) {
          const unsigned long long first = atomicAdd(&ctr->disc_pool, (unsigned long long)disc_segment(cnt));
          if (first + cnt <= pool_cap) {
            list[0].x = disc_place(first);
            s_dst[k] = pool + first;
            s_count[k] = 0u;
            atomicOr(&s_full, 1u << k);
          } else {
            ctr->disc_overflow = 1u;
            h = 0u;
          }
        }
        hdr[first_hdr + (long long)k * plane_hdrs] = h;
      }
    }
    __syncthreads();
    if (!s_full) break;
  }
}

// ---- disc painting ----------------------------------------------------------
constexpr int kPaintX = 64;
constexpr int kPaintStride = kPaintX + 1;  // words per row: consecutive rows fall into different banks
constexpr int kPaintPatches = (kPaintX / kDiscPX + 2 * (kDiscMaxHalo / kDiscPX + 1)) *
                              (64 / kDiscPY + 2 * (kDiscMaxHalo / kDiscPY + 1));  // in reach of a tile of up to 64 rows
constexpr int kPaintUnits = 1024;          // units of work the tile's disc lists are split into (at most)
constexpr int kPaintAhead = 2;             // entries a lane loads at a time
static_assert(kPaintAhead == 2, "the loop below picks one of two");
constexpr int kQueue = 64;                 // discs a warp holds back until 32 are ready

// Bound by issue (66 to 76 % of the cycles at two CTAs an SM).  Of a 64-row tile's
// warp instructions about half are chords in the marrow phase of the 512^3
// generator, an eighth in the bone phase; the rest is per tile and list, so
// lists are taken without divisions or empty halves and the levels pushed down
// two voxels at a time: both phases of 512^3 4.04 -> 3.88 ms.  Cutting the discs'
// rows at the columns to the sides too leaves 17 % fewer of them, which saved
// the painting 0.24 ms and cost the lists 0.28.
template <int TY>
__global__ void __launch_bounds__(8 * TY, 64 / TY * 2)
disc_paint_kernel(const uint32_t* __restrict__ hdr, const uint2* __restrict__ ent, const uint2* __restrict__ pool,
                  Dims dm, int H, int kmax, int npx, int npy, int ntx, int nty, const float* __restrict__ dia,
                  float* __restrict__ dmap, uint32_t* __restrict__ nzbits, uint32_t* __restrict__ fillmap) {
  extern __shared__ __align__(16) uint32_t lev[];  // (kmax + 1) levels of TY rows
  constexpr int kPlane = TY * kPaintStride;
  constexpr int kPaintThreads = 8 * TY, kPaintWarps = kPaintThreads / 32;
  __shared__ uint2 chord[kPaintX + 1];  // by length: word offsets of its level and of its second cell
  __shared__ uint2 queue[kPaintWarps][kQueue];
  __shared__ uint32_t s_list[kPaintPatches], s_unit[kPaintUnits], s_patches, s_discs, s_units, s_next;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long bid = blockIdx.x;
  const int tx = (int)(bid % ntx), ty = (int)((bid / ntx) % nty), z = (int)(bid / ((long long)ntx * nty));
  const int x0 = tx * kPaintX, y0 = ty * TY;
  const long long first = ((long long)z * dm.h + y0) * dm.w + x0;
  float* out = dmap + first;
  const int nw = dm.nw();
  uint32_t* outbits = nzbits + ((long long)z * dm.h + y0) * nw + (x0 >> 5);
  const int px0 = max(x0 - H, 0) / kDiscPX, px1 = min(x0 + kPaintX - 1 + H, dm.w - 1) / kDiscPX;
  const int py0 = max(y0 - H, 0) / kDiscPY, py1 = min(y0 + TY - 1 + H, dm.h - 1) / kDiscPY;
  const int nhx = px1 - px0 + 1, nh = nhx * (py1 - py0 + 1);
  const long long zh = (long long)z * npx * npy;
  if (tid == 0) s_patches = s_discs = s_units = s_next = 0u;
  __syncthreads();
  // the patches whose discs reach the tile: place << 16 | count
  for (int i = tid; i < nh; i += kPaintThreads) {
    const int ry = i / nhx, rx = i - ry * nhx, px = px0 + rx, py = py0 + ry;
    const uint32_t h = __ldg(hdr + zh + (long long)py * npx + px);
    const int reach = (int)(h >> 16), bx = px * kDiscPX, by = py * kDiscPY;
    if (h != 0u && bx - reach <= x0 + kPaintX - 1 && bx + kDiscPX - 1 + reach >= x0 && by - reach <= y0 + TY - 1 &&
        by + kDiscPY - 1 + reach >= y0) {
      s_list[atomicAdd(&s_patches, 1u)] = ((uint32_t)(ry << 8 | rx) << 16) | (h & 0xffffu);
      atomicAdd(&s_discs, h & 0xffffu);
    }
  }
  __syncthreads();
  const int patches = (int)s_patches;
  const int vx = min(kPaintX, dm.w - x0), vy = min(TY, dm.h - y0);
  if (patches == 0) {  // no disc in reach: all zero
    for (int y = warp; y < vy; y += kPaintWarps)
      for (int x = lane; x < vx; x += 32) {
        out[(long long)y * dm.w + x] = 0.0f;
        if (fillmap) fillmap[first + (long long)y * dm.w + x] = 0u;
        if (lane == 0) outbits[(long long)y * nw + (x >> 5)] = 0u;
      }
    return;
  }
  static_assert(kPlane % 4 == 0, "cleared 16 bytes at a time");
  for (int i = tid; i < (kmax + 1) * kPlane / 4; i += kPaintThreads)
    reinterpret_cast<uint4*>(lev)[i] = make_uint4(0u, 0u, 0u, 0u);
  // units of `unit` discs, taken by the warps as they finish one: short enough
  // that no warp is left alone with a long list, and at most kPaintUnits
  uint32_t unit = 32 * kPaintAhead;
  while (s_discs / unit + patches > kPaintUnits) unit *= 2;
  for (int i = tid; i < patches; i += kPaintThreads) {
    const uint32_t parts = ((s_list[i] & 0xffffu) + unit - 1) / unit, base = atomicAdd(&s_units, parts);
    for (uint32_t j = 0; j < parts; ++j) s_unit[base + j] = ((uint32_t)i << 16) | j;
  }
  if (tid <= kPaintX) {
    const int k = min(31 - __clz(max(tid, 1)), kmax);
    chord[tid] = make_uint2((uint32_t)(k * kPlane), (uint32_t)(tid - (1 << k)));
  }
  __syncthreads();
  const unsigned below = (1u << lane) - 1u;
  uint2* q = queue[warp];
  const uint2* list = nullptr;
  uint32_t count = 0, e0 = 0;
  int bx = 0, by = 0, nq = 0;
  for (bool done = false; !done;) {
    if (e0 >= count) {
      uint32_t next = 0;
      if (lane == 0) next = atomicAdd(&s_next, 1u);
      next = __shfl_sync(0xffffffffu, next, 0);
      done = next >= s_units;
      count = e0 = 0;
      if (!done) {
        const uint32_t u = s_unit[next], item = s_list[u >> 16];
        e0 = (u & 0xffffu) * unit;
        count = min(e0 + unit, item & 0xffffu);
        const int px = px0 + (int)((item >> 16) & 255u), py = py0 + (int)(item >> 24);
        list = ent + (zh + (long long)py * npx + px) * kDiscSlots;
        if ((item & 0xffffu) > kDiscSlots) list = pool + disc_first(__ldg(&list->x));
        bx = px * kDiscPX - x0;
        by = py * kDiscPY - y0;
      }
    }
    // discs that meet the tile: {R << 16 | rho, centre, rows}
    uint2 e[kPaintAhead];
#pragma unroll
    for (int j = 0; j < kPaintAhead; ++j) {
      const uint32_t i = e0 + 32 * j + lane;
      e[j] = i < count ? __ldg(list + i) : make_uint2(0u, 0u);
    }
    e0 += 32 * kPaintAhead;
    // (one round more than the unit has, with nothing in it, where the queue is to be emptied)
    const int rounds = done ? 1 : count + 32 * kPaintAhead - e0 > 32 ? 2 : 1;
#pragma unroll 1
    for (int j = 0; j < rounds; ++j) {
      const uint2 d = j ? e[1] : e[0];
      const int cx = bx + (int)(d.y & 31u), cy = by + (int)((d.y >> 5) & 7u);
      const int r = (int)floor_sqrt(d.x & 0xffffu);
      const int ya = max(cy + (int)((d.y >> 8) & 255u) - 128, 0);
      const int yb = min(cy + (int)(d.y >> 16) - 128, TY - 1);
      const bool hit = d.x != 0u && cx + r >= 0 && cx - r < kPaintX && ya <= yb;
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (hit)
        q[nq + __popc(m & below)] =
            make_uint2(d.x, (uint32_t)(cx + 256) | ((uint32_t)(cy + 256) << 10) | ((uint32_t)ya << 20) |
                                   ((uint32_t)yb << 26));
      nq += __popc(m);
      __syncwarp();
      while (nq >= 32 || (done && nq > 0)) {
        const int take = min(nq, 32);
        nq -= take;
        // the rows of the discs one after the other, two to a lane: a lane's disc
        // is the last one that starts at or before its rows
        const uint2 it = q[nq + min(lane, take - 1)];
        const int ya = (int)((it.y >> 20) & 63u);
        const int pairs = lane < take ? ((int)(it.y >> 26) - ya + 2) >> 1 : 0;
        int end = pairs;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int u = __shfl_up_sync(0xffffffffu, end, o);
          if (lane >= o) end += u;
        }
        const int start = end - pairs, total = __shfl_sync(0xffffffffu, end, 31);
        const int first = ya - 2 * start;  // row = first + 2 * position
        int before = 0;                    // discs that start before s
        for (int s = 0; s < total; s += 32) {
          const unsigned at = (unsigned)(start - s);
          const unsigned starts = __reduce_or_sync(0xffffffffu, pairs > 0 && at < 32u ? 1u << at : 0u);
          const int owner = before + __popc(starts & (2u * below + 1u)) - 1;
          before += __popc(starts);
          const uint32_t ox = __shfl_sync(0xffffffffu, it.x, owner), oy = __shfl_sync(0xffffffffu, it.y, owner);
          const int y = __shfl_sync(0xffffffffu, first, owner) + 2 * (s + lane);
          if (s + lane < total) {
            const uint32_t R = ox >> 16;
            const int cx = (int)(oy & 1023u) - 256, dy = y - (int)((oy >> 10) & 1023u) + 256;
            const int t0 = (int)(ox & 0xffffu) - dy * dy, t1 = t0 - 2 * dy - 1;
            const bool two = y < (int)(oy >> 26);
            const int h0 = (int)floor_sqrt((uint32_t)t0), h1 = (int)floor_sqrt((uint32_t)max(t1, 0));
            const int xa0 = max(cx - h0, 0), len0 = min(cx + h0, kPaintX - 1) - xa0 + 1;
            const int xa1 = max(cx - h1, 0), len1 = two ? min(cx + h1, kPaintX - 1) - xa1 + 1 : 0;
            uint32_t* row = lev + y * kPaintStride;
            if (len0 > 0) {
              const uint2 off = chord[len0];
              uint32_t* p = row + off.x + xa0;
              uint32_t* p2 = p + off.y;
              atomicMax(p, R);
              atomicMax(p2, R);
            }
            if (len1 > 0) {
              const uint2 off = chord[len1];
              uint32_t* p = row + kPaintStride + off.x + xa1;
              uint32_t* p2 = p + off.y;
              atomicMax(p, R);
              atomicMax(p2, R);
            }
          }
        }
        __syncwarp();
      }
    }
  }
  __syncthreads();
  // push the levels down: a cell of level k covers 2^k voxels, so it passes to
  // the two cells of level k - 1 at its own place and 2^(k-1) further
  for (int y = warp; y < vy; y += kPaintWarps) {
    const uint32_t* row = lev + y * kPaintStride;
    uint32_t v = 0u;  // voxels lane (low half) and lane + 32: squared radii fit 16 bits
    for (int k = kmax; k >= 0; --k) {
      const uint32_t* lk = row + k * kPlane;
      const uint32_t own = lk[lane] | (lk[lane + 32] << 16);
      uint32_t moved = 0u;
      if (k < kmax) {
        const int s = 1 << k;  // the shift of level k + 1's second cell
        moved = __shfl_sync(0xffffffffu, v, (lane - s) & 31);
        if (lane < s) moved <<= 16;  // voxel lane + 32 - s
      }
      v = __vimax3_u16x2(v, moved, own);
    }
    const uint32_t a = v & 0xffffu, b = v >> 16;
    const long long at = (long long)y * dm.w + lane;
    if (lane < vx) {
      out[at] = __ldg(dia + a);
      if (fillmap) fillmap[first + at] = a;
    }
    if (lane + 32 < vx) {
      out[at + 32] = __ldg(dia + b);
      if (fillmap) fillmap[first + at + 32] = b;
    }
    const unsigned ma = __ballot_sync(0xffffffffu, lane < vx && a != 0u);
    const unsigned mb = __ballot_sync(0xffffffffu, lane + 32 < vx && b != 0u);
    if (lane == 0) outbits[(long long)y * nw] = ma;
    if (lane == 0 && vx > 32) outbits[(long long)y * nw + 1] = mb;
  }
}

}  // namespace

size_t disc_header_count(Dims dm) {
  const size_t npx = (dm.w + kDiscPX - 1) / kDiscPX, npy = (dm.h + kDiscPY - 1) / kDiscPY;
  return npx * npy * (size_t)dm.d;
}

// Entries per voxel that the pool took for the marrow phase of 300 x 256 x 288
// (BV/TV 0.15, sigma 4 to 20), by the largest squared radius: 350 0.011, 603 0.095,
// 1334 0.31, 2153 0.65, 4237 1.25; a third to half of that at BV/TV 0.4.
size_t disc_pool_entries(Dims dm, uint32_t rmax) {
  const unsigned long long n = (unsigned long long)dm.n(), want = n * rmax / 2800;
  return (size_t)((want < 2 * n ? want : 2 * n) + 4096);
}

cudaError_t launch_disc_tables(const uint4* lut, uint32_t n, uint2* thr, uint32_t* tmpl, cudaStream_t s,
                               unsigned long long* launches) {
  unsigned blocks = (n + 127) / 128;
  disc_tables_kernel<<<blocks ? blocks : 1, 128, 0, s>>>(lut, n, thr, tmpl);
  ++*launches;
  return cudaGetLastError();
}

namespace {
template <int ROWS, int NZ>
cudaError_t ridge_map_rows(const uint16_t* dist, Dims dm, const uint2* thr, uint16_t* rmap, cudaStream_t s) {
  const int pairs = edt_near_pitch(dm.w) / 2;
  const int nxt = (pairs + kMapPairs - 1) / kMapPairs, nyt = (dm.h + ROWS - 1) / ROWS, nzt = (dm.d + NZ - 1) / NZ;
  const long long warps = (long long)nxt * nyt * nzt;
  ridge_map_kernel<ROWS, NZ><<<(unsigned)((warps + kMapWarps - 1) / kMapWarps), kMapWarps * 32, 0, s>>>(
      reinterpret_cast<const uint32_t*>(dist), pairs, dm.h, dm.d, thr, reinterpret_cast<uint32_t*>(rmap), nxt, nyt,
      nzt);
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_ridge_map(const uint16_t* dist, Dims dm, const uint2* thr, uint16_t* rmap, cudaStream_t s,
                             unsigned long long* launches) {
  ++*launches;
  // 4 rows and 32 planes a warp load fewer halos, 2 and 4 give more warps; both
  // phases: 128^3 59 and 27 us, 187 x 203 x 251 67 and 59, 301 x 190 x 253 80 and 83,
  // 320^3 142 and 162, 512^3 411 and 574.  The line lies below where the two meet
  // for a call alone: fewer halos are less work, which counts where specimens
  // overlap (16 of 96 to 384 voxels an edge 9.11 ms, 9.17 with the line at 3 * 2^22).
  return dm.n() >= (1ll << 23) ? ridge_map_rows<4, 32>(dist, dm, thr, rmap, s)
                               : ridge_map_rows<2, 4>(dist, dm, thr, rmap, s);
}

namespace {
int halo_of(uint32_t rmax) {
  int h = 0;
  while ((h + 1) * (h + 1) <= (int)rmax) ++h;
  return h;
}

template <int NZ>
cudaError_t list_planes(const uint16_t* rmap, Dims dm, int H, const uint32_t* tmpl, int npx, int npy, uint32_t* hdr,
                        uint2* ent, uint2* pool, size_t pool_cap, Counters* ctr, cudaStream_t s) {
  constexpr size_t smem = (size_t)NZ * kPlaneCells * sizeof(uint32_t) +
                          ((size_t)kCentres + kListWarps * (kCentreQueue + kRunQueue)) * sizeof(uint2);
  const long long blocks = (long long)npx * npy * ((dm.d + NZ - 1) / NZ);
  cudaError_t e = cudaFuncSetAttribute(disc_list_kernel<NZ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  disc_list_kernel<NZ><<<(unsigned)blocks, kListThreads, smem, s>>>(rmap, edt_near_pitch(dm.w), dm, H, tmpl, npx, npy, hdr, ent, pool,
                                                                    pool_cap, ctr);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_disc_lists(const uint16_t* rmap, Dims dm, uint32_t rmax, const uint32_t* tmpl, uint32_t* hdr,
                              uint2* ent, uint2* pool, size_t pool_cap, Counters* ctr, cudaStream_t s,
                              unsigned long long* launches) {
  const int H = halo_of(rmax);
  const int npx = (dm.w + kDiscPX - 1) / kDiscPX, npy = (dm.h + kDiscPY - 1) / kDiscPY;
  ++*launches;
  // 32 planes per CTA share the walk through the halo.  Where such CTAs would
  // leave half of the SMs idle, 8: lists of both phases of 56 x 64 x 72 (42
  // CTAs) 47 us with 32 planes, 36 with 16, 28 with 8; 72 x 81 x 97 (132 CTAs) 23 with any of
  // them; 128^3 (256 CTAs) 78, 73, 82; 200 x 180 x 251 191, 225, 311.
  if ((long long)npx * npy * ((dm.d + 31) / 32) <= 76)
    return list_planes<8>(rmap, dm, H, tmpl, npx, npy, hdr, ent, pool, pool_cap, ctr, s);
  return list_planes<32>(rmap, dm, H, tmpl, npx, npy, hdr, ent, pool, pool_cap, ctr, s);
}

namespace {
template <int TY>
cudaError_t paint_rows(const uint32_t* hdr, const uint2* ent, const uint2* pool, Dims dm, int H, const float* dia,
                       float* dmap, uint32_t* nzbits, uint32_t* fillmap, cudaStream_t s) {
  int kmax = 0;  // largest level a chord of at most min(2 H + 1, 64) voxels writes (two cells of 32 cover 64)
  while (kmax < 5 && (2 << kmax) <= 2 * H + 1) ++kmax;
  const int npx = (dm.w + kDiscPX - 1) / kDiscPX, npy = (dm.h + kDiscPY - 1) / kDiscPY;
  const int ntx = (dm.w + kPaintX - 1) / kPaintX, nty = (dm.h + TY - 1) / TY;
  const size_t level = (size_t)TY * kPaintStride * sizeof(uint32_t);
  // the attribute is the kernel's, not the launch's: always its largest value,
  // so that calls on other threads with other radii cannot lower it in between
  cudaError_t e = cudaFuncSetAttribute(disc_paint_kernel<TY>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(6 * level));
  if (e != cudaSuccess) return e;
  disc_paint_kernel<TY><<<(unsigned)((long long)ntx * nty * dm.d), 8 * TY, (kmax + 1) * level, s>>>(
      hdr, ent, pool, dm, H, kmax, npx, npy, ntx, nty, dia, dmap, nzbits, fillmap);
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_disc_paint(const uint32_t* hdr, const uint2* ent, const uint2* pool, Dims dm, uint32_t rmax,
                              const float* dia, float* dmap, uint32_t* nzbits, uint32_t* fillmap, cudaStream_t s,
                              unsigned long long* launches) {
  ++*launches;
  const int H = halo_of(rmax);
  // Tiles of 64 rows take a list that reaches two of 32 once, those of 32 are twice
  // as many.  Both phases: 64^3 28.0 and 26.7 us, 90 x 97 x 95 45.3 and 41.0, 128^3
  // 61.4 and 63.2; 320^3 (smoothing of 4 voxels) 0.80 and 0.88 ms, 512^3 (5) 3.44 and
  // 3.81.  With smaller balls 32 rows stay ahead a little longer (smoothing of 3.5:
  // 160^3 122 and 115 us, 256^3 380 and 376, 320^3 728 and 718).
  return dm.n() >= (1ll << 22) ? paint_rows<64>(hdr, ent, pool, dm, H, dia, dmap, nzbits, fillmap, s)
                               : paint_rows<32>(hdr, ent, pool, dm, H, dia, dmap, nzbits, fillmap, s);
}

}  // namespace bm
