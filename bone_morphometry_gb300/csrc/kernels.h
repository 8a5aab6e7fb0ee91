// Host-side launchers of the device kernels (one declaration per kernel family).
#pragma once

#include <atomic>
#include <cmath>

#include "bm_internal.h"

namespace bm {

// Grid of a persistent (tile-looping) kernel: as many CTAs as the current
// device keeps resident at once, at most one per tile.  A kernel is always
// launched with the same block size and no dynamic shared memory, so the number
// is looked up once per device (its constant, kept for the process).
template <auto kKernel>
inline unsigned resident_grid(int threads, long long tiles) {
  constexpr int kDevices = 64;
  static std::atomic<long long> known[kDevices];
  int dev = 0;
  cudaGetDevice(&dev);
  long long g = dev < kDevices ? known[dev].load(std::memory_order_relaxed) : 0;
  if (g == 0) {
    int sms = 0, per = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kKernel, threads, 0);
    g = (long long)(per > 0 ? per : 1) * (sms > 0 ? sms : 1);
    if (dev < kDevices) known[dev].store(g, std::memory_order_relaxed);
  }
  if (g > tiles) g = tiles;
  if (g < 1) g = 1;
  return (unsigned)g;
}

// Bytes of device scratch the EDT line passes need for a volume.
size_t edt_scratch_bytes(Dims dm);

// First EDT pass (x rows): phase selection from the inputs (mode), the 1-D
// distance to the nearest non-selected voxel of the row, squared (kInfSq when
// the row has none), the row-padded selection bitmask, and the site count.
cudaError_t launch_edt_x(const uint8_t* a, const uint8_t* b, int mode, Dims dm, uint32_t* out,
                         uint32_t* selbits, Counters* ctr, cudaStream_t s, unsigned long long* launches);

// Lower-envelope pass along y (axis 1) or z (axis 2).  The z pass also
// records the maximum squared distance in ctr->rmax.
cudaError_t launch_edt_line(int axis, const uint32_t* in, uint32_t* out, Dims dm, void* scratch,
                            Counters* ctr, cudaStream_t s, unsigned long long* launches);

// Windowed y (axis 1) / z (axis 2) pass.  Lines it cannot bound are flagged in
// redo (one byte per line, zeroed by the caller; the z pass also sets
// ctr->z_redo) and left to launch_edt_redo.  wait_cycles: limit of the TMA
// copy's first bounded wait (< 0: the default, about 2 s); a block that gives up
// sets ctr->status.  only (the y pass; may be null): the flags of the z pass; the
// blocks whose columns have none are left out.
cudaError_t launch_edt_window(int axis, const uint32_t* in, uint32_t* out, Dims dm, uint8_t* redo, Counters* ctr,
                              long long wait_cycles, const uint8_t* only, cudaStream_t s,
                              unsigned long long* launches);
// The exact lower envelope of the flagged lines (scratch: edt_scratch_bytes).
cudaError_t launch_edt_redo(int axis, const uint32_t* in, uint32_t* out, Dims dm, void* scratch, const uint8_t* redo,
                            Counters* ctr, cudaStream_t s, unsigned long long* launches);

// The 16-bit passes (squared distances up to 65^2): x (x_pass) or y of a volume
// or slab of planes, and z.  Maps of edt_near_pitch(w) * h * d values, 16-byte
// aligned.  The z pass flags the lines that hold larger distances in redo and
// ctr->z_redo; the 32-bit passes compute those.
int edt_near_pitch(int w);
cudaError_t launch_edt_near_xy(const uint8_t* a, const uint8_t* b, int mode, Dims dm, uint16_t* xmap, uint16_t* ymap,
                               uint32_t* selbits, Counters* ctr, long long wait_cycles, bool x_pass, cudaStream_t s,
                               unsigned long long* launches);
// wide (32 bits at the volume's pitch) or narrow (16 bits at edt_near_pitch): the one not null.
cudaError_t launch_edt_near_z(const uint16_t* ymap, uint32_t* wide, uint16_t* narrow, Dims dm, uint8_t* redo,
                              Counters* ctr, cudaStream_t s, unsigned long long* launches);
// The flagged lines of a narrow result, from the 32-bit y pass' output; in 32
// bits in wide too.
cudaError_t launch_edt_near_redo(const uint32_t* in, uint16_t* out, uint32_t* wide, Dims dm, void* scratch,
                                 const uint8_t* redo, Counters* ctr, cudaStream_t s, unsigned long long* launches);
// The other lines of a narrow result into wide.
cudaError_t launch_edt_widen(const uint16_t* narrow, uint32_t* wide, Dims dm, const uint8_t* redo, cudaStream_t s,
                             unsigned long long* launches);

// out (zeroed): ROI voxels, ROI-clipped bone voxels, and those of them with a
// 6-neighbour outside the volume or the ROI (metrics.rs:166-202).  rbits, bbits:
// a row-padded bitmask each (nw * h * d words).
cudaError_t launch_volume_counts(const uint8_t* bone, const uint8_t* roi, Dims dm, uint32_t* rbits, uint32_t* bbits,
                                 unsigned long long* out, cudaStream_t s, unsigned long long* launches);

// Search-template table entries lut[r2] for r2 in [lo, hi]:
// {scan_cube(1,0,0), scan_cube(1,1,0), scan_cube(1,1,1), f32 bits of 2*sqrt(r2)}.
cudaError_t launch_lut(uint4* lut, uint32_t lo, uint32_t hi, cudaStream_t s, unsigned long long* launches);

// Distance-ridge extraction: appends {linear index, r2} records and, when occ
// is not null, sets occ[r2] = 1 for every ridge r2.  When ridgebits is not null, writes the ridge bitmask
// rows (layout of selbits) of every tile with a selected voxel (the caller
// zeroes it first).
cudaError_t launch_ridges(const uint32_t* dist, const uint32_t* selbits, Dims dm, const uint4* lut, uint2* ridges,
                          Counters* ctr, uint32_t* occ, uint32_t* ridgebits, cudaStream_t s,
                          unsigned long long* launches);

// Site values by reverse chain passes: the non-selected voxels a ridge sphere
// reaches are exactly the nearest sites of the ridge voxel, reached through
// the argmins of the z, y and x passes.  launch_chain_z: for every ridge
// voxel c (ridgebits) and every z' with g(x, y, z') + (z - z')^2 = m(c),
// chain(x, y, z') = max(., m(c)) (chain zeroed by the caller).
// launch_chain_y: for every (x, y, z') with chain > 0 and every y' with
// f(x, y', z') + (y - y')^2 = g(x, y, z'), the x pass's nearest sites x' of
// (x, y', z') get sites(x', y', z') = max(., chain): run on the tile fill's
// map, whose non-selected voxels are 0, it adds what launch_sites would.
// f, g, m: the x, y and z pass outputs.  halo: rows staged on each side, at
// least isqrt(largest ridge r2) + 1; the largest ridge r2 must be below
// kChainMaxR2.
constexpr int kChainMaxR2 = 2048;
constexpr int kChainMaxHalo = 46;  // isqrt(kChainMaxR2 - 1) + 1
cudaError_t launch_chain_z(const uint32_t* g, const uint32_t* m, const uint32_t* ridgebits, uint32_t* chain, Dims dm,
                           int halo, cudaStream_t s, unsigned long long* launches);
cudaError_t launch_chain_y(const uint32_t* f, const uint32_t* g, const uint32_t* chain, const uint32_t* selbits,
                           uint32_t* sites, Dims dm, int halo, cudaStream_t s, unsigned long long* launches);

// Sphere fill: atomic max of r2 over every voxel of each ridge ball (any phase).
cudaError_t launch_fill(const uint2* ridges, const Counters* ctr, unsigned long long max_ridges, Dims dm,
                        uint32_t* fillmap, cudaStream_t s, unsigned long long* launches);

// Cleanup passes 1 and 2, phase mask, optional f32 map, exact statistics.
// dmap: the fill's diameters 2*sqrt(r2) (0 where no ball reaches); nzbits: its
// nonzero voxels as a row-padded bitmask; inbits: scratch of its size.  The
// separable fill writes both; launch_diameters makes them of an r2 map (dmap
// may be the map's memory).  dia: f32 diameters by r2 (launch_dia_table).
// Values whose f32 exponent lies in [e_lo, e_lo + kFixedSpan] are summed in
// fixed point (acc->fx_s1, fx_s2); the others go to acc's per-exponent sums.
cudaError_t launch_diameters(const uint32_t* fillmap, Dims dm, const float* dia, float* dmap, uint32_t* nzbits,
                             cudaStream_t s, unsigned long long* launches);
cudaError_t launch_cleanup(const float* dmap, const uint32_t* selbits, const uint32_t* nzbits, uint32_t* inbits, Dims dm,
                           float scale, float* outmap, StatsAccum* acc, int e_lo, cudaStream_t s,
                           unsigned long long* launches);
cudaError_t launch_dia_table(const uint4* lut, uint32_t n, float* dia, cudaStream_t s, unsigned long long* launches);

// Separable fill (discs.cu), for squared radii up to kDiscMaxR2: offsets from a
// ball's centre are kept in 8 bits.
constexpr int kDiscMaxHalo = 127;
constexpr uint32_t kDiscMaxR2 = kDiscMaxHalo * kDiscMaxHalo;
constexpr int kDiscPX = 32, kDiscPY = 8;   // columns per list patch
constexpr uint32_t kDiscSlots = 384;       // discs per patch and plane (1.5 per column)
size_t disc_header_count(Dims dm);
// thr / tmpl: n entries by squared radius, from the search templates.
cudaError_t launch_disc_tables(const uint4* lut, uint32_t n, uint2* thr, uint32_t* tmpl, cudaStream_t s,
                               unsigned long long* launches);
// The distance ridge of a 16-bit distance map as one: twice the squared
// distance, plus 1 for ridge voxels.  Both at edt_near_pitch, the padding 0.
cudaError_t launch_ridge_map(const uint16_t* dist, Dims dm, const uint2* thr, uint16_t* rmap, cudaStream_t s,
                             unsigned long long* launches);
// Disc lists: hdr[patch] = count | reach << 16 for every 32 x 8 patch of every
// plane (disc_header_count), its discs {R << 16 | rho, column | (first row +
// 128) << 8 | (last row + 128) << 16} (rows from the centre's) at
// ent[patch * kDiscSlots].  A patch with more than kDiscSlots discs has them at
// pool[disc_first(ent[patch * kDiscSlots].x)]; a pool that is too small (disc_pool_entries:
// a first estimate) sets ctr->disc_overflow and leaves lists out; ctr->disc_pool,
// 0 beforehand, has the entries wanted in either case.
size_t disc_pool_entries(Dims dm, uint32_t rmax);
cudaError_t launch_disc_lists(const uint16_t* rmap, Dims dm, uint32_t rmax, const uint32_t* tmpl, uint32_t* hdr,
                              uint2* ent, uint2* pool, size_t pool_cap, Counters* ctr, cudaStream_t s,
                              unsigned long long* launches);
// The fill's diameters (selected voxels and the sites that spheres reach, 0
// elsewhere; dia: diameters by r^2), their nonzero voxels as a row-padded
// bitmask and, when fillmap is not null, the r^2 map.
cudaError_t launch_disc_paint(const uint32_t* hdr, const uint2* ent, const uint2* pool, Dims dm, uint32_t rmax,
                              const float* dia, float* dmap, uint32_t* nzbits, uint32_t* fillmap, cudaStream_t s,
                              unsigned long long* launches);

// Tile-owned fill (fill.cu).
// Rows of y per fill tile: 64 for volumes of at least kFillTallMinVoxels (fewer
// ball entries per voxel), 32 from kFillMidMinVoxels, else 16 (more tiles: a
// small volume's fill is bound by its tiles' serial chains); requested = 16,
// 32 or 64 forces it.
int fill_tile_rows(Dims dm, int requested);
long long fill_tile_count(Dims dm, int ty);
size_t scan_scratch_words(long long n);
// Exclusive scan of n u32 values (out may alias in); scratch of scan_scratch_words(n).
cudaError_t launch_scan(const uint32_t* in, uint32_t* out, long long n, uint32_t* scratch, cudaStream_t s,
                        unsigned long long* launches);
// occ[0..rmax+1] (occ[rmax+1] == 0) -> rank_desc / rvals / info->nR.
// rgeo[rank] = {r2, ceil sqrt, floor sqrt, 0} for every rank.
cudaError_t launch_rank(const uint32_t* occ, uint32_t* rank_desc, uint32_t rmax, uint32_t* rvals, uint4* rgeo,
                        FillInfo* info, uint32_t* scan_scratch, cudaStream_t s, unsigned long long* launches);
// ty: the fill tile's rows of y (fill_tile_rows).
cudaError_t launch_bin(bool count, const uint2* ridges, const Counters* ctr, unsigned long long max_ridges,
                       const uint32_t* rank_desc, FillInfo* info, Dims dm, int ty, uint32_t* counts,
                       const uint32_t* offsets, uint32_t* entries, cudaStream_t s, unsigned long long* launches);
// Sphere lattice-point table: count (surf_cnt[r2]) or fill (surf_pts from surf_off[r2]) for r2 in [lo, hi].
cudaError_t launch_surf(bool count, uint32_t lo, uint32_t hi, uint32_t* surf_cnt, const uint32_t* surf_off,
                        uint32_t* surf_pts, cudaStream_t s, unsigned long long* launches);
// Selected voxels of every tile from the binned balls; non-selected voxels get 0.
// selbits: the phase's row-padded selection bitmask (edt_x output).
// order_scratch: tile_order_words(dm, ty) words (the tiles' processing order).
size_t tile_order_words(Dims dm, int ty);
cudaError_t launch_tile_fill(const uint32_t* entries, const uint32_t* offsets, const uint32_t* rvals,
                             const uint4* rgeo, const FillInfo* info, const uint32_t* selbits, Dims dm, int ty,
                             uint32_t* order_scratch, uint32_t* fillmap, cudaStream_t s, unsigned long long* launches);
// Non-selected voxels on each ridge's sphere: atomic max of r2 (after the tile
// fill).  surf_off / surf_pts: the lattice-point table covering every ridge r2;
// small: 8 lanes per ridge instead of 16 (spheres of about 40 points or fewer).
cudaError_t launch_sites(const uint2* ridges, const Counters* ctr, unsigned long long max_ridges,
                         const uint32_t* selbits, const uint32_t* surf_off, const uint32_t* surf_pts, bool small,
                         Dims dm, uint32_t* fillmap, cudaStream_t s, unsigned long long* launches);

// The sum and the sum of squares of x = f32(raw * scale) as f64 over the finite
// positive raw values of map[0 .. n), each accumulated in index order with one
// f64 rounding per value -- the reference's own sequence (metrics.rs:215-224),
// reproduced exactly (ordered.cu).  out[0] = sum, out[1] = sum of squares.
// maxbits: device pointer to the f32 bits of the largest such value (the
// statistics accumulator's max_bits), which scales the approximate sums.
size_t ordered_sum_scratch_bytes(long long n);
cudaError_t launch_ordered_sums(const float* map, long long n, float scale, const uint32_t* maxbits, void* scratch,
                                double* out, cudaStream_t s, unsigned long long* launches);

// Exact moment sums of f32(raw * scale) over the finite positive raw values.
cudaError_t launch_moments(const float* map, long long n, float scale, StatsAccum* acc, cudaStream_t s,
                           unsigned long long* launches);
// Exact order statistics (quantile.cu): q->bits[r] = the f32 bits of the value
// of rank q->rank[r] (0-based) among the finite positive values of map[0 .. n);
// 0xffffffff when there is none.  scratch: quantile_scratch_words() words.
constexpr int kQuantileRanks = 10;
struct QuantileState {
  unsigned long long resid[kQuantileRanks];  // rank inside its high bin
  uint32_t target[kQuantileRanks];           // the distinct high bins
  uint32_t slot[kQuantileRanks];             // each rank's index into target
  uint32_t targets;
  uint32_t bits[kQuantileRanks];             // out
};
size_t quantile_scratch_words();
// count: the number of positive finite values, known when the launch runs.
cudaError_t launch_quantiles(const float* map, long long n, const unsigned long long* count, uint32_t* scratch,
                             QuantileState* q, cudaStream_t s, unsigned long long* launches);
// The two 0-based ranks that quantile i (median, P10, P25, P75, P90) of `count`
// values lies between, and its place between them (metrics.rs:247-251, 278-288).
__host__ __device__ inline double quantile_ranks(int i, unsigned long long count, unsigned long long* lo,
                                                 unsigned long long* hi) {
  const double p = i == 0 ? 0.5 : i == 1 ? 0.1 : i == 2 ? 0.25 : i == 3 ? 0.75 : 0.9;
  const double position = p * (double)(count - 1), f = floor(position);
  *lo = (unsigned long long)f;
  *hi = (unsigned long long)ceil(position);
  return position - f;
}

}  // namespace bm
