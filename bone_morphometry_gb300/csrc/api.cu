// C ABI of libbm_gb300 (include/bm.h): context, buffer cache, the per-phase
// pipeline and the drop-in entry points for edt.rs / local_thickness.rs /
// metrics.rs.
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <new>
#include <thread>
#include <vector>

#include "exact_sum.h"
#include "kernels.h"

using namespace bm;

namespace {

thread_local std::string g_create_error;

struct CallError {
  int status;
};

void set_err(bm_ctx* ctx, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  if (ctx) ctx->last_error = buf;
  else g_create_error = buf;
}

[[noreturn]] void fail(bm_ctx* ctx, int status, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  ctx->last_error = buf;
  throw CallError{status};
}

void check(bm_ctx* ctx, cudaError_t e, const char* what) {
  if (e == cudaSuccess) return;
  const int st = (e == cudaErrorMemoryAllocation) ? BM_ERR_OOM : BM_ERR_CUDA;
  cudaGetLastError();  // clear a sticky-free error so the context stays usable
  fail(ctx, st, "%s: %s", what, cudaGetErrorString(e));
}

// Whether this allocation is the one that bm_ctx_fail_allocation asked to fail.
bool refused(bm_ctx* ctx, const char* what) {
  if (ctx->fail_what.empty() || ctx->fail_what != what || ctx->fail_skip-- > 0) return false;
  ctx->fail_what.clear();
  return true;
}

void* ensure(bm_ctx* ctx, Buffer& b, size_t bytes, const char* what) {
  if (bytes == 0) bytes = 16;
  if (b.bytes >= bytes) return b.ptr;
  if (b.ptr) {
    cudaFree(b.ptr);
    b.ptr = nullptr;
    b.bytes = 0;
  }
  void* p = nullptr;
  cudaError_t e = refused(ctx, what) ? cudaErrorMemoryAllocation : cudaMalloc(&p, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    fail(ctx, BM_ERR_OOM, "device allocation of %zu bytes for %s failed: %s", bytes, what, cudaGetErrorString(e));
  }
  b.ptr = p;
  b.bytes = bytes;
  return p;
}

void release(Buffer& b) {
  if (b.ptr) cudaFree(b.ptr);
  b.ptr = nullptr;
  b.bytes = 0;
}

const char* const kFamilyName[KF_COUNT] = {"count_roi", "edt_x",     "edt_y",           "edt_z",
                                            "templates", "ridge",     "fill",            "fill_rank",
                                            "fill_bin",  "fill_sites",      "cleanup_final",
                                            "quantile",  "stats_order"};

cudaEvent_t pooled_event(bm_ctx* ctx) {
  if (!ctx->event_pool.empty()) {
    cudaEvent_t e = ctx->event_pool.back();
    ctx->event_pool.pop_back();
    return e;
  }
  cudaEvent_t e = nullptr;
  check(ctx, cudaEventCreate(&e), "event create");
  return e;
}

// Launch through `launch` (a callable returning cudaError_t); while profiling,
// bracket it with events on the launching stream.
template <class L>
void timed(bm_ctx* ctx, int family, cudaStream_t s, const char* what, L&& launch) {
  if (!ctx->profiling) {
    check(ctx, launch(), what);
    return;
  }
  cudaEvent_t a = pooled_event(ctx), b = pooled_event(ctx);
  check(ctx, cudaEventRecord(a, s), "event record");
  check(ctx, launch(), what);
  check(ctx, cudaEventRecord(b, s), "event record");
  ctx->prof.push_back(ProfRec{family, a, b});
}

void fold_profile(bm_ctx* ctx) {
  for (const ProfRec& r : ctx->prof) {
    float ms = 0.f;
    if (cudaEventSynchronize(r.stop) == cudaSuccess && cudaEventElapsedTime(&ms, r.start, r.stop) == cudaSuccess) {
      ctx->prof_ms[r.family] += ms;
      ctx->prof_n[r.family] += 1;
    }
    cudaGetLastError();
    ctx->event_pool.push_back(r.start);
    ctx->event_pool.push_back(r.stop);
  }
  ctx->prof.clear();
}

// volume.rs:12-34 plus the library's own limits (u32 linear ridge index, u32
// squared distances whose search templates cannot overflow u32).
Dims check_dims(bm_ctx* ctx, size_t w, size_t h, size_t d) {
  if (w < 2 || h < 2 || d < 2)
    fail(ctx, BM_ERR_DIMS, "all dimensions must be at least 2 for 3-D morphometry; got %zux%zux%zu", w, h, d);
  if (w > 32768 || h > 32768 || d > 32768)
    fail(ctx, BM_ERR_DIMS, "dimension above 32768 is not supported; got %zux%zux%zu", w, h, d);
  const unsigned long long n = (unsigned long long)w * h * d;
  if (n >= 0xFFFFFFFFull)
    fail(ctx, BM_ERR_DIMS, "volume of %llu voxels exceeds the 2^32-1 voxel limit", n);
  const unsigned long long r2 =
      (unsigned long long)(w - 1) * (w - 1) + (unsigned long long)(h - 1) * (h - 1) +
      (unsigned long long)(d - 1) * (d - 1);
  if (r2 >= (1ull << 30)) fail(ctx, BM_ERR_DIMS, "largest squared distance %llu exceeds 2^30", r2);
  return Dims{(int)w, (int)h, (int)d};
}

const char* phase_name(int phase) { return phase == BM_PHASE_BACKGROUND ? "background" : "foreground"; }

// The tables by squared radius: search templates, diameters, and those of the
// separable fill.  All are made before any takes its place in the context, so
// that a failure on the way leaves the context with the tables that it had.
void ensure_lut(bm_ctx* ctx, uint32_t rmax) {
  if (ctx->lut_max >= rmax && ctx->lut.ptr) return;
  // grow to at least twice the current size so repeated growth stays amortised
  uint32_t target = rmax;
  if (ctx->lut.ptr && target < ctx->lut_max * 2u) target = ctx->lut_max * 2u;
  if (target < 1024) target = 1024;
  const size_t n = (size_t)target + 1, nd = std::min<size_t>(target, kDiscMaxR2) + 1;
  struct Tables {
    Buffer lut, dia, thr, tmpl;
    ~Tables() {
      for (Buffer* b : {&lut, &dia, &thr, &tmpl}) release(*b);
    }
  } t;
  uint4* lut = static_cast<uint4*>(ensure(ctx, t.lut, n * sizeof(uint4), "template table"));
  float* dia = static_cast<float*>(ensure(ctx, t.dia, n * sizeof(float), "diameter table"));
  uint2* thr = static_cast<uint2*>(ensure(ctx, t.thr, nd * sizeof(uint2), "disc tables"));
  uint32_t* tmpl = static_cast<uint32_t*>(ensure(ctx, t.tmpl, nd * sizeof(uint32_t), "disc tables"));
  uint32_t lo = 0;
  if (ctx->lut.ptr) {
    check(ctx, cudaMemcpyAsync(lut, ctx->lut.ptr, ((size_t)ctx->lut_max + 1) * sizeof(uint4), cudaMemcpyDeviceToDevice,
                               ctx->stream),
          "template table copy");
    lo = ctx->lut_max + 1;
  }
  timed(ctx, KF_TEMPLATES, ctx->stream, "template kernel",
        [&] { return launch_lut(lut, lo, target, ctx->stream, &ctx->launches); });
  check(ctx, launch_dia_table(lut, (uint32_t)n, dia, ctx->stream, &ctx->launches), "diameter table");
  timed(ctx, KF_TEMPLATES, ctx->stream, "disc tables",
        [&] { return launch_disc_tables(lut, (uint32_t)nd, thr, tmpl, ctx->stream, &ctx->launches); });
  // the phase that reads the tables may run on another stream
  check(ctx, cudaStreamSynchronize(ctx->stream), "template tables");
  std::swap(ctx->lut, t.lut);
  std::swap(ctx->lutf, t.dia);
  std::swap(ctx->discthr, t.thr);
  std::swap(ctx->disctmpl, t.tmpl);
  ctx->lut_max = target;
}

void ensure_surf(bm_ctx* ctx, uint32_t rmax);

// Sphere fill of one phase into F (u32 r^2 map): tile-owned fill, or the
// per-ball atomic scatter when the (ball, tile) entry count would not fit u32.
// f, g, m: the x, y and z pass outputs (kept for the chain passes); ridgebits:
// the ridge bitmask; m is free for reuse once the chain_z pass has read it.
// Returns the map the fill wrote: F, or m's buffer when F is g's (g is still
// needed by the chain_y pass that follows the fill).
uint32_t* fill_phase(bm_ctx* ctx, Dims dm, const uint2* ridges, Counters* ctr, unsigned long long max_ridges,
                     uint32_t rmax, const uint32_t* occ, const uint32_t* selbits, const uint32_t* f,
                     const uint32_t* g, uint32_t* m, const uint32_t* ridgebits, uint32_t* F, cudaStream_t s) {
  const size_t rwords = (size_t)rmax + 2;
  uint32_t* rank = static_cast<uint32_t*>(ensure(ctx, ctx->rank, rwords * 4, "r2 ranks"));
  uint32_t* rvals = static_cast<uint32_t*>(ensure(ctx, ctx->rvals, rwords * 4, "r2 values"));
  uint4* rgeo = static_cast<uint4*>(ensure(ctx, ctx->rgeo, rwords * sizeof(uint4), "r2 geometry"));
  FillInfo* info = static_cast<FillInfo*>(ensure(ctx, ctx->fillinfo, sizeof(FillInfo), "fill info"));
  uint32_t* scratch = static_cast<uint32_t*>(ensure(ctx, ctx->scanscratch, scan_scratch_words((long long)rwords) * 4,
                                                    "scan scratch"));
  check(ctx, cudaMemsetAsync(info, 0, sizeof(FillInfo), s), "memset");
  timed(ctx, KF_FILL_RANK, s, "rank kernel",
        [&] { return launch_rank(occ, rank, rmax, rvals, rgeo, info, scratch, s, &ctx->launches); });
  FillInfo hi;
  check(ctx, cudaMemcpyAsync(&hi, info, sizeof hi, cudaMemcpyDeviceToHost, s), "fill info readback");
  check(ctx, cudaStreamSynchronize(s), "rank kernel");
  const int ty = fill_tile_rows(dm, ctx->fill_rows);
  const long long tiles = fill_tile_count(dm, ty);
  const long long nbins = tiles * (long long)hi.nR;
  uint32_t* counts = static_cast<uint32_t*>(ensure(ctx, ctx->bincounts, ((size_t)nbins + 1) * 4, "bin counts"));
  uint32_t* offsets = static_cast<uint32_t*>(ensure(ctx, ctx->binoffsets, ((size_t)nbins + 1) * 4, "bin offsets"));
  scratch = static_cast<uint32_t*>(ensure(ctx, ctx->scanscratch, scan_scratch_words(nbins + 1) * 4, "scan scratch"));
  check(ctx, cudaMemsetAsync(counts, 0, ((size_t)nbins + 1) * 4, s), "memset");
  if (hi.nR > 0) {
    timed(ctx, KF_FILL_BIN, s, "bin count kernel", [&] {
      return launch_bin(true, ridges, ctr, max_ridges, rank, info, dm, ty, counts, nullptr, nullptr, s,
                        &ctx->launches);
    });
  }
  timed(ctx, KF_FILL_BIN, s, "bin scan",
        [&] { return launch_scan(counts, offsets, nbins + 1, scratch, s, &ctx->launches); });
  check(ctx, cudaMemcpyAsync(&hi, info, sizeof hi, cudaMemcpyDeviceToHost, s), "fill info readback");
  check(ctx, cudaStreamSynchronize(s), "bin kernels");
  if (hi.total_entries >= 0xFFFFFFFFull || rmax > kSurfMaxR2 || hi.nR >= 0xFFFFu) {
    check(ctx, cudaMemsetAsync(F, 0, (size_t)dm.n() * 4, s), "memset");
    timed(ctx, KF_FILL, s, "fill kernel",
          [&] { return launch_fill(ridges, ctr, max_ridges, dm, F, s, &ctx->launches); });
    return F;
  }
  uint32_t* entries = static_cast<uint32_t*>(
      ensure(ctx, ctx->binentries, ((size_t)hi.total_entries + 1) * 4, "bin entries"));
  if (hi.nR > 0) {
    timed(ctx, KF_FILL_BIN, s, "bin scatter kernel", [&] {
      return launch_bin(false, ridges, ctr, max_ridges, rank, info, dm, ty, counts, offsets, entries, s,
                        &ctx->launches);
    });
  }
  // Sites: the site kernel's half-warp steps over the ridge spheres' lattice
  // points (35-55 ps each, measured), or the two chain passes (9-17 ps a
  // voxel, bounded halo): chains above 0.2 steps per voxel.  The 512^3
  // workload's phases sit at 0.07 (bone) and 0.62 (marrow), the 1024^3
  // plate generator's at 0.10 and 0.28.
  const int halo = (int)std::sqrt((double)rmax) + 1;
  const bool chains_fit = f && g && m && ridgebits && rmax < (uint32_t)kChainMaxR2;
  const bool auto_chains = (double)hi.site_steps > 0.2 * (double)dm.n();
  const bool chains = chains_fit && (ctx->site_method == BM_SITES_CHAINS ||
                                     (ctx->site_method == BM_SITES_AUTO && auto_chains));
  uint32_t* chain = nullptr;
  if (chains) {
    const size_t nbytes = (size_t)dm.n() * 4;
    chain = static_cast<uint32_t*>(ensure(ctx, ctx->chainmap, nbytes, "chain map"));
    check(ctx, cudaMemsetAsync(chain, 0, nbytes, s), "memset");
    timed(ctx, KF_FILL_SITES, s, "chain z pass",
          [&] { return launch_chain_z(g, m, ridgebits, chain, dm, halo, s, &ctx->launches); });
    if (F == g) F = m;  // the z pass output has been read; g must outlive the fill
  } else {
    ensure_surf(ctx, rmax);
  }
  uint32_t* order = static_cast<uint32_t*>(ensure(ctx, ctx->tileorder, tile_order_words(dm, ty) * 4, "tile order"));
  timed(ctx, KF_FILL, s, "tile fill kernel", [&] {
    return launch_tile_fill(entries, offsets, rvals, rgeo, info, selbits, dm, ty, order, F, s, &ctx->launches);
  });
  if (chains) {
    timed(ctx, KF_FILL_SITES, s, "chain y pass",
          [&] { return launch_chain_y(f, g, chain, selbits, F, dm, halo, s, &ctx->launches); });
  } else {
    // 8 lanes per ridge when the spheres average at most 2.5 half-warp steps
    // (about 40 lattice points): half-warps would idle on their last step
    const bool small_spheres = 2 * hi.site_steps <= 5 * hi.ridges;
    timed(ctx, KF_FILL_SITES, s, "site kernel", [&] {
      return launch_sites(ridges, ctr, max_ridges, selbits, static_cast<const uint32_t*>(ctx->surf_off.ptr),
                          static_cast<const uint32_t*>(ctx->surf_pts.ptr), small_spheres, dm, F, s,
                          &ctx->launches);
    });
  }
  return F;
}

// Lattice points of every sphere |d|^2 = r2 for r2 <= rmax, cached per context.
void ensure_surf(bm_ctx* ctx, uint32_t rmax) {
  if (ctx->surf_off.ptr && ctx->surf_max >= rmax) return;
  uint32_t target = rmax < 1024 ? 1024 : rmax;
  if (target > kSurfMaxR2) target = kSurfMaxR2 > rmax ? kSurfMaxR2 : rmax;
  cudaStream_t s = ctx->stream;
  const long long n = (long long)target + 2;
  Buffer cnt;
  uint32_t* c = static_cast<uint32_t*>(ensure(ctx, cnt, (size_t)n * 4, "sphere table"));
  try {
    release(ctx->surf_off);
    release(ctx->surf_pts);
    ctx->surf_max = 0;
    uint32_t* off = static_cast<uint32_t*>(ensure(ctx, ctx->surf_off, (size_t)n * 4, "sphere table"));
    uint32_t* scratch = static_cast<uint32_t*>(ensure(ctx, ctx->scanscratch, scan_scratch_words(n) * 4, "scan"));
    check(ctx, cudaMemsetAsync(c, 0, (size_t)n * 4, s), "memset");
    check(ctx, launch_surf(true, 0, target, c, nullptr, nullptr, s, &ctx->launches), "sphere table");
    check(ctx, launch_scan(c, off, n, scratch, s, &ctx->launches), "sphere table");
    uint32_t total = 0;
    check(ctx, cudaMemcpyAsync(&total, off + target + 1, 4, cudaMemcpyDeviceToHost, s), "sphere table");
    check(ctx, cudaStreamSynchronize(s), "sphere table");
    uint32_t* pts = static_cast<uint32_t*>(ensure(ctx, ctx->surf_pts, ((size_t)total + 1) * 4, "sphere table"));
    check(ctx, launch_surf(false, 0, target, nullptr, off, pts, s, &ctx->launches), "sphere table");
    check(ctx, cudaStreamSynchronize(s), "sphere table");
  } catch (...) {
    release(cnt);
    release(ctx->surf_off);
    release(ctx->surf_pts);
    throw;
  }
  release(cnt);
  ctx->surf_max = target;
}

// Page-locked readback area of a context: copies into it return at once, so a
// phase's work is queued to its end without a wait.
struct Readback {
  Counters ctr;                   // after the distance transform
  PhaseOut out;                   // at the end of the phase
  unsigned long long counts[3];   // ROI counts; volume counts
  QuantileState quantile;
};

Readback& readback(bm_ctx* ctx) { return *static_cast<Readback*>(ctx->pinned); }

PhaseOut* phase_out(bm_ctx* ctx, size_t flags = 0) {
  return static_cast<PhaseOut*>(ensure(ctx, ctx->phaseout, sizeof(PhaseOut) + flags, "phase results"));
}

// The reference's sequential f64 sums of the calibrated map values
// (metrics.rs:215-224) into out->osum, on stream s, after out->acc has its
// maximum.
void ordered_sums(bm_ctx* ctx, const float* d_map, long long n, float scale, PhaseOut* out, cudaStream_t s) {
  void* scratch = ensure(ctx, ctx->ordscratch, ordered_sum_scratch_bytes(n), "ordered-sum scratch");
  timed(ctx, KF_STATS_ORDER, s, "ordered sums", [&] {
    return launch_ordered_sums(d_map, n, scale, &out->acc.max_bits, scratch, out->osum, s, &ctx->launches);
  });
}

// The order statistics of the quantiles of d_map's finite positive values
// (metrics.rs:242-288), whose number out->acc holds by then, and their readback.
void queue_quantiles(bm_ctx* ctx, const float* d_map, long long n, const PhaseOut* out, cudaStream_t s) {
  uint32_t* hist = static_cast<uint32_t*>(ensure(ctx, ctx->qhist, quantile_scratch_words() * 4, "quantile histograms"));
  QuantileState* dq = static_cast<QuantileState*>(ensure(ctx, ctx->qtargets, sizeof(QuantileState), "quantile ranks"));
  timed(ctx, KF_QUANTILE, s, "quantiles",
        [&] { return launch_quantiles(d_map, n, &out->acc.count, hist, dq, s, &ctx->launches); });
  check(ctx, cudaMemcpyAsync(&readback(ctx).quantile, dq, sizeof(QuantileState), cudaMemcpyDeviceToHost, s),
        "quantile readback");
}

// One phase: EDT (+ local thickness unless edt_only, + the reference-order
// statistics sums when stats).  d_a / d_b are the device inputs for `mode`;
// results optionally go to d_edt (u32 EDT), d_map (f32 masked diameters) and
// d_sq (u32 propagated r^2).
//
// The steps only queue work, but for the two waits: prepare, xy (slab by slab
// where the inputs arrive so), z; wait_edt, whose largest radius sizes and
// chooses what follows; fill; finish, which waits for the results.  The two
// phases of a call are stepped in turn by one host thread, each on its own
// context.  A thread started per call, pageable readbacks and a wait for the ROI
// counts before either phase took 111 us more of a 64 x 56 x 72 call (235 us now)
// and 141 more of a 128^3 one from host inputs with quantiles (450).
struct Phase {
  // set by the caller
  bm_ctx* ctx;
  Dims dm;
  const uint8_t* d_a;
  const uint8_t* d_b;
  int mode;
  cudaStream_t s;
  bool edt_only = false, stats = false;
  bool quantiles = false;  // with stats
  uint32_t* d_edt = nullptr;
  float* d_map = nullptr;
  uint32_t* d_sq = nullptr;
  float scale = 1.0f;

  // results
  Counters hc{};
  StatsAccum acc;
  double osum[2] = {0.0, 0.0};

  // x pass output (kept for the chain passes), y pass input; then the ridge map,
  // or the flagged lines in 32 bits; then the f32 map, where the caller wants none
  uint32_t* A = nullptr;
  uint32_t* B = nullptr;        // y pass output; then the fill's diameters
  uint32_t* E = nullptr;        // z pass output
  uint32_t* selbits = nullptr;  // selection bits
  PhaseOut* out = nullptr;
  uint8_t* yflags = nullptr;    // per-line flags of the windowed passes
  uint8_t* zflags = nullptr;
  bool near = false;            // the 16-bit passes first
  bool separable = false;
  bool left_separable = false;  // there was no memory for the lists
  uint32_t* hdr = nullptr;      // disc lists
  uint2* ent = nullptr;
  uint2* pool = nullptr;
  int e_lo = 0;

  size_t voxels() const { return (size_t)dm.n(); }
  size_t bits_bytes() const { return (size_t)dm.nw() * dm.h * dm.d * sizeof(uint32_t); }

  size_t narrow_bytes() const { return (size_t)edt_near_pitch(dm.w) * dm.h * dm.d * 2; }
  size_t map_bytes() const { return std::max(voxels() * 4, near ? narrow_bytes() : 0); }
  size_t lists_bytes() const { return disc_header_count(dm) * kDiscSlots * sizeof(uint2); }
  size_t flag_bytes() const { return (size_t)dm.w * (dm.h + dm.d); }  // lines along y and z

  // A forced site method or tile height asks for the tile fill.
  bool tiles_asked() const { return ctx->site_method != BM_SITES_AUTO || ctx->fill_rows != 0; }

  // What the separable fill leaves of a budgeted phase's bytes for its pool.
  size_t pool_room() const {
    if (!ctx->budgeted) return SIZE_MAX;
    const size_t limit = phase_limit_bytes(voxels());
    const size_t held = 2 * std::max(voxels() * 4, narrow_bytes()) + narrow_bytes() + lists_bytes() +
                        disc_header_count(dm) * 4 + 3 * bits_bytes() + ordered_sum_scratch_bytes(dm.n()) +
                        quantile_scratch_words() * 4 + sizeof(PhaseOut) + flag_bytes();
    return held < limit ? limit - held : 0;
  }

  // The 16-bit rows are padded to 16 voxels and the lists to 32 x 8 columns: of
  // a volume a few voxels wide they would take many times its size (two voxels
  // wide 48 and 200 bytes a voxel).  Such a volume keeps them while they are
  // small: 512 x 512 x 2 local thickness 442 us, 770 with the tile fill.
  bool narrow_fits() const {
    constexpr size_t kSmall = 1ull << 30;
    if (edt_only) return narrow_bytes() <= std::max(voxels() * 4, kSmall);
    return lists_bytes() <= std::max(voxels() * 24, kSmall) && pool_room() > 0;
  }

  // Buffers, and everything the phase accumulates into zeroed.
  void prepare() {
    // the 16-bit passes, but where the caller has asked for the tile fill (its
    // chain passes read the 32-bit maps)
    near = (edt_only || !tiles_asked()) && narrow_fits();
    A = static_cast<uint32_t*>(ensure(ctx, ctx->dist, edt_only && near ? narrow_bytes() : map_bytes(), "distance map"));
    B = static_cast<uint32_t*>(ensure(ctx, ctx->dist2, map_bytes(), "distance map"));
    selbits = static_cast<uint32_t*>(ensure(ctx, ctx->selbits, bits_bytes(), "selection bits"));
    out = phase_out(ctx, flag_bytes());
    yflags = reinterpret_cast<uint8_t*>(out + 1);
    zflags = yflags + (size_t)dm.w * dm.d;
    // local thickness keeps the x pass output (the chain passes read it): the z
    // pass then writes its own map, in 16 bits for the separable fill
    E = d_edt ? d_edt
              : static_cast<uint32_t*>(ensure(ctx, ctx->edtmap, near ? narrow_bytes() : voxels() * 4, "distance map"));
    check(ctx, cudaMemsetAsync(out, 0, sizeof(PhaseOut) + flag_bytes(), s), "memset");
  }

  // Envelope scratch of the flagged lines, in the memory that the disc lists take
  // after them (allocated at their size where they may follow).
  void* line_scratch() {
    const size_t lists_follow = near && !edt_only && !left_separable ? lists_bytes() : 0;
    return ensure(ctx, ctx->discent, std::max(edt_scratch_bytes(dm), lists_follow), "envelope scratch");
  }

  // The x and y passes of planes z0 .. z1-1: both work within a plane, so a slab
  // of planes is a volume of its own (every offset is a whole number of planes,
  // which keeps the 16-byte alignment of rows whose width is a multiple of 4).
  // The counters accumulate over slabs.
  void xy(int z0, int z1) {
    const Dims sd{dm.w, dm.h, z1 - z0};
    const long long off = (long long)z0 * dm.w * dm.h;
    const uint8_t* a = d_a + off;
    const uint8_t* b = d_b ? d_b + off : nullptr;
    uint32_t* sel = selbits + (long long)z0 * dm.h * dm.nw();
    if (near) {
      const long long off16 = (long long)z0 * edt_near_pitch(dm.w) * dm.h;
      uint16_t* xmap = reinterpret_cast<uint16_t*>(A) + off16;
      uint16_t* ymap = reinterpret_cast<uint16_t*>(B) + off16;
      for (const bool x_pass : {true, false})
        timed(ctx, x_pass ? KF_EDT_X : KF_EDT_Y, s, x_pass ? "edt x pass" : "edt y pass", [&] {
          return launch_edt_near_xy(a, b, mode, sd, xmap, ymap, sel, &out->ctr, ctx->wait_cycles, x_pass, s,
                                    &ctx->launches);
        });
      return;
    }
    wide_xy(sd, a, b, sel, off, yflags + (long long)z0 * dm.w, nullptr);
  }

  // The 32-bit x and y passes; only: the z lines whose tiles the y pass is for (null: all).
  void wide_xy(Dims sd, const uint8_t* a, const uint8_t* b, uint32_t* sel, long long off, uint8_t* flags,
               const uint8_t* only) {
    A = static_cast<uint32_t*>(ensure(ctx, ctx->dist, voxels() * 4, "distance map"));
    timed(ctx, KF_EDT_X, s, "edt x pass",
          [&] { return launch_edt_x(a, b, mode, sd, A + off, sel, &out->ctr, s, &ctx->launches); });
    void* lines = line_scratch();
    timed(ctx, KF_EDT_Y, s, "edt y pass", [&] {
      const cudaError_t e =
          launch_edt_window(1, A + off, B + off, sd, flags, &out->ctr, ctx->wait_cycles, only, s, &ctx->launches);
      if (e != cudaSuccess) return e;
      return launch_edt_redo(1, A + off, B + off, sd, lines, flags, &out->ctr, s, &ctx->launches);
    });
  }

  void z() {
    timed(ctx, KF_EDT_Z, s, "edt z pass", [&] {
      if (near)
        return launch_edt_near_z(reinterpret_cast<const uint16_t*>(B), d_edt, reinterpret_cast<uint16_t*>(E), dm,
                                 zflags, &out->ctr, s, &ctx->launches);
      return launch_edt_window(2, B, E, dm, zflags, &out->ctr, ctx->wait_cycles, nullptr, s, &ctx->launches);
    });
    read_counters();
  }

  void read_counters() {
    check(ctx, cudaMemcpyAsync(&readback(ctx).ctr, &out->ctr, sizeof(Counters), cudaMemcpyDeviceToHost, s),
          "counter readback");
  }

  void wait_edt() {
    check(ctx, cudaStreamSynchronize(s), "edt");
    hc = readback(ctx).ctr;
    if (hc.z_redo && !hc.status && hc.sites) {  // (without a site every line is flagged: refused below)
      // the flagged lines, from 32-bit x and y passes
      const unsigned long long sites = hc.sites;
      if (near) wide_xy(dm, d_a, d_b, selbits, 0, yflags, zflags);
      void* lines = line_scratch();
      timed(ctx, KF_EDT_Z, s, "edt z lines", [&] {
        if (near && !d_edt)
          return launch_edt_near_redo(B, reinterpret_cast<uint16_t*>(E), A, dm, lines, zflags, &out->ctr, s,
                                      &ctx->launches);
        return launch_edt_redo(2, B, E, dm, lines, zflags, &out->ctr, s, &ctx->launches);
      });
      read_counters();
      check(ctx, cudaStreamSynchronize(s), "edt");
      hc = readback(ctx).ctr;
      hc.sites = sites;  // counted twice by two x passes
    }
    if (hc.status) fail(ctx, BM_ERR_TIMEOUT, "a bounded device-side wait of the distance transform ran out");
    if (hc.sites == 0) {
      const int phase = (mode == SEL_BACKGROUND) ? BM_PHASE_BACKGROUND : BM_PHASE_FOREGROUND;
      fail(ctx, BM_ERR_ALL_SELECTED,
           "distance transform is undefined for an all-%s volume unless an exterior convention is specified",
           phase_name(phase));
    }
    // The separable fill (discs.cu) up to radius 127, where its packed discs end.
    separable = near && !edt_only && hc.rmax <= kDiscMaxR2;
  }

  // No memory for the lists: the tile fill in the memory that they hold.  None of
  // their kernels may be in flight.
  void leave_separable() {
    ctx->last_error.clear();
    separable = false;
    left_separable = true;
    for (Buffer* b : {&ctx->dischdr, &ctx->discent, &ctx->discpool}) release(*b);
  }

  // Local thickness, after wait_edt: lists, then paint, queued to their end (but
  // for the tile fill's own waits).
  void lists() {
    ensure_lut(ctx, hc.rmax);
    if (!separable) return;
    // a budgeted context's phase holds either fill's buffers
    if (ctx->budgeted)
      for (Buffer* b : {&ctx->chainmap, &ctx->ridges, &ctx->ridgebits, &ctx->bincounts, &ctx->binoffsets, &ctx->binentries})
        release(*b);
    uint16_t* rmap = reinterpret_cast<uint16_t*>(A);  // the y pass has read it
    try {
      const size_t count = disc_header_count(dm);
      hdr = static_cast<uint32_t*>(ensure(ctx, ctx->dischdr, count * 4, "disc headers"));
      ent = static_cast<uint2*>(ensure(ctx, ctx->discent, lists_bytes(), "disc lists"));
      const size_t first = disc_pool_entries(dm, hc.rmax) * sizeof(uint2);
      pool = static_cast<uint2*>(ensure(ctx, ctx->discpool, std::min(first, pool_room()), "disc pool"));
    } catch (const CallError& e) {
      if (e.status != BM_ERR_OOM) throw;
      leave_separable();
      return;
    }
    const size_t pool_cap = ctx->discpool.bytes / sizeof(uint2);
    const uint2* thr = static_cast<const uint2*>(ctx->discthr.ptr);
    const uint32_t* tmpl = static_cast<const uint32_t*>(ctx->disctmpl.ptr);
    timed(ctx, KF_RIDGE, s, "ridge map", [&] {
      return launch_ridge_map(reinterpret_cast<const uint16_t*>(E), dm, thr, rmap, s, &ctx->launches);
    });
    timed(ctx, KF_FILL_BIN, s, "disc lists", [&] {
      return launch_disc_lists(rmap, dm, hc.rmax, tmpl, hdr, ent, pool, pool_cap, &out->ctr, s, &ctx->launches);
    });
  }

  void paint() {
    if (!separable) {
      tile_fill();
      return;
    }
    uint32_t* nzbits = static_cast<uint32_t*>(ensure(ctx, ctx->nzbits, bits_bytes(), "nonzero bits"));
    const float* dia = static_cast<const float*>(ctx->lutf.ptr);
    float* dmap = reinterpret_cast<float*>(B);  // the y pass output has been read
    timed(ctx, KF_FILL, s, "disc painting", [&] {
      return launch_disc_paint(hdr, ent, pool, dm, hc.rmax, dia, dmap, nzbits, d_sq, s, &ctx->launches);
    });
    cleanup(dmap, nzbits);
  }

  // The whole transform in 32 bits, for the tile fill after the 16-bit passes.
  // Beyond the separable fill's radius the flagged lines are in A already, and the
  // chain passes, which read the x and y passes' maps, do not run.
  void widen() {
    if (hc.rmax > kDiscMaxR2) {
      timed(ctx, KF_EDT_Z, s, "edt z lines", [&] {
        return launch_edt_widen(reinterpret_cast<const uint16_t*>(E), A, dm, zflags, s, &ctx->launches);
      });
      E = A;
      return;
    }
    E = static_cast<uint32_t*>(ensure(ctx, ctx->edtmap, voxels() * 4, "distance map"));
    check(ctx, cudaMemsetAsync(yflags, 0, flag_bytes(), s), "memset");
    wide_xy(dm, d_a, d_b, selbits, 0, yflags, nullptr);
    void* lines = line_scratch();
    timed(ctx, KF_EDT_Z, s, "edt z pass", [&] {
      const cudaError_t e =
          launch_edt_window(2, B, E, dm, zflags, &out->ctr, ctx->wait_cycles, nullptr, s, &ctx->launches);
      if (e != cudaSuccess) return e;
      return launch_edt_redo(2, B, E, dm, lines, zflags, &out->ctr, s, &ctx->launches);
    });
    read_counters();
    check(ctx, cudaStreamSynchronize(s), "edt");
    if (readback(ctx).ctr.status)
      fail(ctx, BM_ERR_TIMEOUT, "a bounded device-side wait of the distance transform ran out");
  }

  void tile_fill() {
    if (ctx->budgeted)
      for (Buffer* b : {&ctx->dischdr, &ctx->discpool}) release(*b);
    if (near) widen();
    const uint4* lut = static_cast<const uint4*>(ctx->lut.ptr);
    const float* dia = static_cast<const float*>(ctx->lutf.ptr);
    const unsigned long long selected = voxels() - hc.sites;
    uint32_t* nzbits = static_cast<uint32_t*>(ensure(ctx, ctx->nzbits, bits_bytes(), "nonzero bits"));
    uint2* ridges = static_cast<uint2*>(ensure(ctx, ctx->ridges, (selected + 1) * sizeof(uint2), "ridge list"));
    const size_t rwords = (size_t)hc.rmax + 2;
    uint32_t* occ = static_cast<uint32_t*>(ensure(ctx, ctx->occ, rwords * 4, "r2 flags"));
    check(ctx, cudaMemsetAsync(occ, 0, rwords * 4, s), "memset");
    uint32_t* rbits = static_cast<uint32_t*>(ensure(ctx, ctx->ridgebits, bits_bytes(), "ridge bits"));
    check(ctx, cudaMemsetAsync(rbits, 0, bits_bytes(), s), "memset");
    timed(ctx, KF_RIDGE, s, "ridge kernel",
          [&] { return launch_ridges(E, selbits, dm, lut, ridges, &out->ctr, occ, rbits, s, &ctx->launches); });
    // E is the context's map: the chain passes may reuse it
    static_assert(kChainMaxR2 <= kDiscMaxR2, "no chain passes after a widened transform");
    uint32_t* F = fill_phase(ctx, dm, ridges, &out->ctr, selected, hc.rmax, occ, selbits, E == A ? nullptr : A, B, E,
                             rbits, d_sq ? d_sq : B, s);
    float* dmap = reinterpret_cast<float*>(F == d_sq ? B : F);
    timed(ctx, KF_CLEAN_FINAL, s, "diameters",
          [&] { return launch_diameters(F, dm, dia, dmap, nzbits, s, &ctx->launches); });
    cleanup(dmap, nzbits);
  }

  // Cleanup, statistics and the readback that ends the phase, from the fill's
  // diameters and nonzero bits.
  void cleanup(const float* dmap, const uint32_t* nzbits) {
    uint32_t* inbits = static_cast<uint32_t*>(ensure(ctx, ctx->inbits, bits_bytes(), "interior bits"));
    // every value of the map is at least 2 * scale (diameters are >= 2), so its
    // f32 exponent is at least that of 2 * scale: the fixed-point base
    const float two_s = 2.0f * scale;
    uint32_t tb;
    std::memcpy(&tb, &two_s, 4);
    const int e2s = (int)(tb >> 23);
    e_lo = (e2s >= 1 && e2s + kFixedSpan <= 254) ? e2s : 4096;  // 4096: no fixed-point path
    // the statistics' sums and quantiles read the f32 map: kept in A when the caller wants none
    float* cmap = stats && !d_map ? reinterpret_cast<float*>(A) : d_map;
    timed(ctx, KF_CLEAN_FINAL, s, "cleanup", [&] {
      return launch_cleanup(dmap, selbits, nzbits, inbits, dm, scale, cmap, &out->acc, e_lo, s, &ctx->launches);
    });
    if (stats) ordered_sums(ctx, cmap, dm.n(), scale, out, s);
    if (quantiles) queue_quantiles(ctx, cmap, dm.n(), out, s);
    check(ctx, cudaMemcpyAsync(&readback(ctx).out, out, sizeof(PhaseOut), cudaMemcpyDeviceToHost, s), "stats readback");
  }

  void finish() {
    check(ctx, cudaStreamSynchronize(s), "local thickness");
    if (separable && readback(ctx).out.ctr.disc_overflow) {
      // the lists' pool ran out: again with one of the size that they wanted, or,
      // where there is no memory (or no room in the budget) for it, with the tile
      // fill in the lists' memory
      const unsigned long long wanted = readback(ctx).out.ctr.disc_pool;
      check(ctx, cudaMemsetAsync(&out->acc, 0, sizeof(StatsAccum), s), "memset");
      check(ctx, cudaMemsetAsync(&out->ctr.disc_pool, 0, sizeof(out->ctr.disc_pool), s), "memset");
      check(ctx, cudaMemsetAsync(&out->ctr.disc_overflow, 0, sizeof(out->ctr.disc_overflow), s), "memset");
      try {
        const size_t room = pool_room();
        if (wanted * sizeof(uint2) > room) throw CallError{BM_ERR_OOM};
        ensure(ctx, ctx->discpool, std::min<size_t>((wanted + wanted / 8) * sizeof(uint2), room), "disc pool");
        lists();
      } catch (const CallError& e) {
        if (e.status != BM_ERR_OOM) throw;
        leave_separable();
      }
      paint();
      check(ctx, cudaStreamSynchronize(s), "local thickness");
    }
    const PhaseOut& r = readback(ctx).out;
    acc = r.acc;
    if (e_lo != 4096) acc.fx_elo = e_lo;
    osum[0] = r.osum[0];
    osum[1] = r.osum[1];
  }
};

// A whole phase, one step after the other.
void run_phase(Phase& p) {
  p.prepare();
  p.xy(0, p.dm.d);
  p.z();
  p.wait_edt();
  if (p.edt_only) return;
  p.lists();
  p.paint();
  p.finish();
}

// nonzero_stats (metrics.rs:228-241; quantile fields NaN) from the reference's
// own sequential sums osum = {sum, sum of squares}; the exact sums are
// reported beside them.
int finish_stats(bm_ctx* ctx, const StatsAccum& a, const double* osum, bm_stats* out) {
  if (a.count == 0) {
    set_err(ctx, "cannot compute statistics because the selected phase is empty");
    return BM_ERR_EMPTY;
  }
  double xsum, xss;
  exact_sums_to_double(a, &xsum, &xss);
  const double sum = osum[0], ss = osum[1];
  const double c = (double)a.count;
  const double mean = sum / c;
  const double centered = (c * ss - sum * sum) / c;
  const double sd = (a.count > 1 && centered > 0.0) ? std::sqrt(centered / (c - 1.0)) : 0.0;
  float mxf;
  std::memcpy(&mxf, &a.max_bits, 4);
  if (out) {
    out->count = a.count;
    out->mean = mean;
    out->standard_deviation = sd;
    out->maximum = (double)mxf;
    out->median = out->percentile_10 = out->percentile_25 = out->percentile_75 = out->percentile_90 = NAN;
    out->interquartile_range = NAN;
    out->coefficient_of_variation = sd / mean;
    out->sum = sum;
    out->sum_of_squares = ss;
    out->exact_sum = xsum;
    out->exact_sum_of_squares = xss;
  }
  return BM_OK;
}

// Quantiles (metrics.rs:242-298) from the order statistics that queue_quantiles
// left: median, P10, P25, P75, P90 by numpy-linear interpolation, then
// (q as f32 * scale_f32) as f64; IQR = P75 - P25.
void finish_quantiles(bm_ctx* ctx, const QuantileState& qs, unsigned long long count, double scale, bm_stats* out) {
  const float sf = (float)scale;
  double q[5];
  for (int i = 0; i < 5; ++i) {
    unsigned long long rank[2];
    const double frac = quantile_ranks(i, count, &rank[0], &rank[1]);
    double v[2];
    for (int j = 0; j < 2; ++j) {
      const uint32_t bits = qs.bits[2 * i + j];
      if (bits == 0xffffffffu) fail(ctx, BM_ERR_CUDA, "quantile rank %llu beyond the %llu values", rank[j], count);
      float f;
      std::memcpy(&f, &bits, 4);
      v[j] = (double)f;
    }
    const double qv = v[0] + frac * (v[1] - v[0]);  // metrics.rs:289
    q[i] = (double)((float)qv * sf);                // metrics.rs:290
  }
  out->median = q[0];
  out->percentile_10 = q[1];
  out->percentile_25 = q[2];
  out->percentile_75 = q[3];
  out->percentile_90 = q[4];
  out->interquartile_range = q[3] - q[2];
}

int nonzero_stats_impl(bm_ctx* ctx, const float* d_values, size_t n, double scale, unsigned flags, bm_stats* out,
                       cudaStream_t s) {
  PhaseOut* po = phase_out(ctx);
  check(ctx, cudaMemsetAsync(po, 0, sizeof(PhaseOut), s), "memset");
  timed(ctx, KF_QUANTILE, s, "moments kernel",
        [&] { return launch_moments(d_values, (long long)n, (float)scale, &po->acc, s, &ctx->launches); });
  ordered_sums(ctx, d_values, (long long)n, (float)scale, po, s);
  if (flags & BM_FLAG_QUANTILES) queue_quantiles(ctx, d_values, (long long)n, po, s);
  PhaseOut& r = readback(ctx).out;
  check(ctx, cudaMemcpyAsync(&r, po, sizeof(PhaseOut), cudaMemcpyDeviceToHost, s), "stats readback");
  check(ctx, cudaStreamSynchronize(s), "moments kernel");
  const int st = finish_stats(ctx, r.acc, r.osum, out);
  if (st) return st;
  if (flags & BM_FLAG_QUANTILES) finish_quantiles(ctx, readback(ctx).quantile, r.acc.count, scale, out);
  return BM_OK;
}

template <class F>
int guarded(bm_ctx* ctx, F&& f) {
  if (!ctx) return BM_ERR_INVALID;
  std::lock_guard<std::mutex> lock(ctx->mu);
  ctx->last_error.clear();
  try {
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e != cudaSuccess) {
      cudaGetLastError();
      fail(ctx, BM_ERR_CUDA, "cudaSetDevice: %s", cudaGetErrorString(e));
    }
    return f();
  } catch (const CallError& ce) {
    return ce.status;
  } catch (const std::bad_alloc&) {
    ctx->last_error = "host allocation failed";
    return BM_ERR_OOM;
  }
}

cudaStream_t pick_stream(bm_ctx* ctx, void* stream) {
  return stream ? static_cast<cudaStream_t>(stream) : ctx->stream;
}

int edt_device_impl(bm_ctx* ctx, const uint8_t* d_vol, Dims dm, int phase, uint32_t* d_out, cudaStream_t s) {
  Phase p{ctx, dm, d_vol, nullptr, phase == BM_PHASE_BACKGROUND ? SEL_BACKGROUND : SEL_FOREGROUND, s};
  p.edt_only = true;
  p.d_edt = d_out;
  run_phase(p);
  return BM_OK;
}

int lt_device_impl(bm_ctx* ctx, const uint8_t* d_vol, Dims dm, int phase, float* d_out, uint32_t* d_sq,
                   cudaStream_t s) {
  Phase p{ctx, dm, d_vol, nullptr, phase == BM_PHASE_BACKGROUND ? SEL_BACKGROUND : SEL_FOREGROUND, s};
  p.d_map = d_out;
  p.d_sq = d_sq;
  run_phase(p);
  return BM_OK;
}

void check_phase(bm_ctx* ctx, int phase) {
  if (phase != BM_PHASE_FOREGROUND && phase != BM_PHASE_BACKGROUND)
    fail(ctx, BM_ERR_INVALID, "phase must be 0 (foreground) or 1 (background); got %d", phase);
}

// Nonzero bytes of a word, as a multiple of 8 (0xff per nonzero byte, then
// one population count).
__device__ __forceinline__ unsigned nz8(uint32_t v) { return (unsigned)__popc(__vcmpne4(v, 0u)); }
__device__ __forceinline__ unsigned both8(uint32_t r, uint32_t b) {
  return (unsigned)__popc(__vcmpne4(r, 0u) & __vcmpne4(b, 0u));
}

// ROI voxels and ROI-clipped bone voxels (the bails of metrics.rs:70-99).
// With both volumes 16-byte aligned, every thread reads two 16-byte words of
// each per step (bytes in flight for the HBM rate); the last n % 32 bytes and
// unaligned inputs take the byte loop.
__global__ void count_roi_kernel(const uint8_t* __restrict__ bone, const uint8_t* __restrict__ roi, long long n,
                                 unsigned long long* __restrict__ out) {
  unsigned long long in_roi = 0, bone_in = 0;
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nth = (long long)gridDim.x * blockDim.x;
  long long head = 0;
  if (((reinterpret_cast<uintptr_t>(bone) | reinterpret_cast<uintptr_t>(roi)) & 15u) == 0) {
    const uint4* R = reinterpret_cast<const uint4*>(roi);
    const uint4* B = reinterpret_cast<const uint4*>(bone);
    const long long pairs = n / 32;
    unsigned long long r8 = 0, b8 = 0;
    for (long long i = tid; i < pairs; i += nth) {
      const uint4 r0 = __ldcs(R + 2 * i), r1 = __ldcs(R + 2 * i + 1);
      const uint4 b0 = __ldcs(B + 2 * i), b1 = __ldcs(B + 2 * i + 1);
      r8 += nz8(r0.x) + nz8(r0.y) + nz8(r0.z) + nz8(r0.w) + nz8(r1.x) + nz8(r1.y) + nz8(r1.z) + nz8(r1.w);
      b8 += both8(r0.x, b0.x) + both8(r0.y, b0.y) + both8(r0.z, b0.z) + both8(r0.w, b0.w) + both8(r1.x, b1.x) +
            both8(r1.y, b1.y) + both8(r1.z, b1.z) + both8(r1.w, b1.w);
    }
    in_roi = r8 >> 3;
    bone_in = b8 >> 3;
    head = pairs * 32;
  }
  for (long long i = head + tid; i < n; i += nth) {
    const bool r = roi[i] != 0;
    in_roi += r;
    bone_in += (r && bone[i] != 0);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    in_roi += __shfl_xor_sync(0xffffffffu, in_roi, o);
    bone_in += __shfl_xor_sync(0xffffffffu, bone_in, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (in_roi) atomicAdd(&out[0], in_roi);
    if (bone_in) atomicAdd(&out[1], bone_in);
  }
}

int volume_metrics_impl(bm_ctx* ctx, const uint8_t* d_bone, const uint8_t* d_roi, Dims dm, const double* sp,
                        bm_volume_metrics* out, cudaStream_t s) {
  for (int i = 0; i < 3; ++i)
    if (!std::isfinite(sp[i]) || sp[i] <= 0.0)
      fail(ctx, BM_ERR_SPACING, "voxel spacings must be finite and positive; got [%g, %g, %g]", sp[0], sp[1], sp[2]);
  unsigned long long* dc = reinterpret_cast<unsigned long long*>(phase_out(ctx));
  const size_t bits = (size_t)dm.nw() * dm.h * dm.d * sizeof(uint32_t);
  uint32_t* rbits = static_cast<uint32_t*>(ensure(ctx, ctx->selbits, bits, "ROI bits"));
  uint32_t* bbits = static_cast<uint32_t*>(ensure(ctx, ctx->nzbits, bits, "bone bits"));
  check(ctx, cudaMemsetAsync(dc, 0, 24, s), "memset");
  timed(ctx, KF_COUNT_ROI, s, "volume counts",
        [&] { return launch_volume_counts(d_bone, d_roi, dm, rbits, bbits, dc, s, &ctx->launches); });
  unsigned long long* hc = readback(ctx).counts;
  check(ctx, cudaMemcpyAsync(hc, dc, 24, cudaMemcpyDeviceToHost, s), "count readback");
  check(ctx, cudaStreamSynchronize(s), "volume counts");
  const double voxel_volume = ((1.0 * sp[0]) * sp[1]) * sp[2];  // metrics.rs:123 (product)
  out->roi_voxels = hc[0];
  out->bone_voxels = hc[1];
  out->boundary_bone_voxels = hc[2];
  out->bone_volume = (double)hc[1] * voxel_volume;
  out->total_volume = (double)hc[0] * voxel_volume;
  out->bone_volume_fraction = out->bone_volume / out->total_volume;
  out->roi_boundary_bone_fraction = (double)hc[2] / (double)hc[1];
  return BM_OK;
}

// The context's twin (created on first use, with the parent's profiling state).
bm_ctx* twin_of(bm_ctx* ctx) {
  if (!ctx->inputs_ready) check(ctx, cudaEventCreateWithFlags(&ctx->inputs_ready, cudaEventDisableTiming), "event");
  if (ctx->twin) return ctx->twin;
  bm_ctx* t = nullptr;
  const int st = bm_ctx_create(ctx->device, &t);
  if (st != BM_OK) fail(ctx, st, "second stream context creation failed");
  t->profiling = ctx->profiling;
  t->site_method = ctx->site_method;
  t->fill_rows = ctx->fill_rows;
  t->wait_cycles = ctx->wait_cycles;
  t->budgeted = ctx->budgeted;
  ctx->twin = t;
  return t;
}

// metrics.rs:70-78, and the library's flags
void check_call(bm_ctx* ctx, double spacing, unsigned flags) {
  if (!std::isfinite(spacing) || spacing <= 0.0)
    fail(ctx, BM_ERR_SPACING, "voxel spacings must be finite and positive; got [%g, %g, %g]", spacing, spacing,
         spacing);
  if (flags & ~(unsigned)(BM_FLAG_QUANTILES | BM_FLAG_BONEJ_ROI))
    fail(ctx, BM_ERR_INVALID, "unknown flags 0x%x", flags);
}

bool phases_side_by_side(const bm_ctx* ctx, Dims dm) { return ctx->split_phases && dm.n() <= kSplitMaxVoxels; }

void count_roi(bm_ctx* ctx, const uint8_t* d_bone, const uint8_t* d_roi, long long n, PhaseOut* out, cudaStream_t s) {
  timed(ctx, KF_COUNT_ROI, s, "count kernel", [&] {
    count_roi_kernel<<<152 * 8, 256, 0, s>>>(d_bone, d_roi, n, out->roi);
    ++ctx->launches;
    return cudaGetLastError();
  });
}

void read_roi_counts(bm_ctx* ctx, const PhaseOut* out, cudaStream_t s) {
  check(ctx, cudaMemcpyAsync(readback(ctx).counts, out->roi, sizeof out->roi, cudaMemcpyDeviceToHost, s),
        "count readback");
  check(ctx, cudaEventRecord(ctx->counted, s), "event record");
}

// Waits for the ROI counts; the bails of metrics.rs:79-99.
void check_roi_counts(bm_ctx* ctx, long long n, unsigned flags) {
  check(ctx, cudaEventSynchronize(ctx->counted), "count kernel");
  const unsigned long long roi = readback(ctx).counts[0], bone = readback(ctx).counts[1];
  if (roi == 0) fail(ctx, BM_ERR_ROI_EMPTY, "ROI mask contains no included voxels");
  if ((flags & BM_FLAG_BONEJ_ROI) && roi == (unsigned long long)n)
    fail(ctx, BM_ERR_ROI_FULL, "BoneJ compatibility mode requires an ROI mask with both inside and outside voxels");
  if (bone == 0) fail(ctx, BM_ERR_NO_BONE, "ROI contains no bone voxels");
  if (bone == roi) fail(ctx, BM_ERR_NO_MARROW, "ROI contains no marrow voxels");
}

// Runs steps of the twin's phase; its error is reported on this context.
template <class F>
void on_twin(bm_ctx* ctx, bm_ctx* tw, F&& f) {
  try {
    f();
  } catch (const CallError&) {
    ctx->last_error = tw->last_error;
    throw;
  }
}

// On every exit from bm_tbth_tbsp: nothing of the call is left in flight (no
// copy from the caller's buffers, no pass reading the inputs), and the twin's
// launches count as this context's.
struct CallFence {
  bm_ctx* ctx;
  bm_ctx* twin;
  cudaStream_t s;
  bool done = false;  // everything has been waited for
  ~CallFence() {
    if (!done) {
      if (ctx->upload_stream) cudaStreamSynchronize(ctx->upload_stream);
      cudaStreamSynchronize(s);
      if (twin) cudaStreamSynchronize(twin->stream);
    }
    if (twin) {
      ctx->launches += twin->launches;
      twin->launches = 0;
    }
  }
};

int report_phase(const Phase& p, bm_ctx* ctx, double spacing, bm_stats* out) {
  const int st = finish_stats(ctx, p.acc, p.osum, out);
  if (st == BM_OK && p.quantiles) finish_quantiles(ctx, readback(p.ctx).quantile, p.acc.count, spacing, out);
  return st;
}

// bm_tbth_tbsp on device inputs.  feed: queues the ROI counts (into the bone
// phase's out) and the x and y passes of the bone phase and, side by side, of
// the marrow phase; the bails are checked once the z passes are queued behind
// them (the passes only write the phases' own buffers).
template <class Feed>
int tbth_phases(bm_ctx* ctx, const uint8_t* d_bone, const uint8_t* d_roi, Dims dm, double spacing, unsigned flags,
                bm_stats* th, bm_stats* sp, float* d_thmap, float* d_spmap, cudaStream_t s, Feed&& feed) {
  const long long N = dm.n();
  const bool want_q = (flags & BM_FLAG_QUANTILES) != 0;
  // The two phases are independent: the marrow phase runs on the twin context
  // (its own stream and buffers), so that their kernels overlap on the GPU.
  // Results and errors are reported in the reference's order (bone first).
  // Side by side only while one phase cannot fill the GPU: on 1024^3 the two
  // phases' kernels compete (59.9 ms against 55.9 ms one after the other), on
  // 512^3 and below they fill each other's gaps.
  bm_ctx* tw = phases_side_by_side(ctx, dm) ? twin_of(ctx) : nullptr;
  bm_ctx* mctx = tw ? tw : ctx;
  CallFence fence{ctx, tw, s};
  Phase bone{ctx, dm, d_bone, d_roi, SEL_BONE_IN_ROI, s};
  Phase marrow{mctx, dm, d_bone, d_roi, SEL_MARROW_IN_ROI, tw ? tw->stream : s};
  bone.stats = marrow.stats = true;
  bone.quantiles = want_q && th;
  marrow.quantiles = want_q && sp;
  bone.scale = marrow.scale = (float)spacing;  // metrics.rs:213
  bone.d_map = d_thmap;
  marrow.d_map = d_spmap;
  if (tw) {
    check(ctx, cudaEventRecord(ctx->inputs_ready, s), "event record");
    check(ctx, cudaStreamWaitEvent(tw->stream, ctx->inputs_ready, 0), "stream wait");
  }
  bone.prepare();
  if (tw) on_twin(ctx, tw, [&] { marrow.prepare(); });
  feed(bone, tw ? &marrow : nullptr);
  bone.z();
  if (tw) on_twin(ctx, tw, [&] { marrow.z(); });
  check_roi_counts(ctx, N, flags);

  bone.wait_edt();
  if (!tw) {
    bone.lists();
    bone.paint();
    bone.finish();
    int st = report_phase(bone, ctx, spacing, th);
    if (st) return st;
    run_phase(marrow);
    fence.done = true;
    return report_phase(marrow, ctx, spacing, sp);
  }
  int twin_status = BM_OK;
  auto try_twin = [&](auto&& f) {
    if (twin_status != BM_OK) return;
    try {
      f();
    } catch (const CallError& e) {
      twin_status = e.status;
    } catch (const std::bad_alloc&) {
      tw->last_error = "host allocation failed";
      twin_status = BM_ERR_OOM;
    }
  };
  try_twin([&] {
    marrow.wait_edt();
  });
  // Decided here, once: a phase may turn to the tile fill later, in finish, when
  // its lists' pool cannot grow.
  const bool queued = bone.separable && marrow.separable;
  if (twin_status == BM_OK && !queued) {
    // the tile fill waits for its own counts: a host thread for each phase
    std::thread thread([&] {
      try_twin([&] {
        const cudaError_t e = cudaSetDevice(tw->device);
        check(tw, e, "cudaSetDevice");
        marrow.lists();
        marrow.paint();
        marrow.finish();
      });
    });
    struct Join {
      std::thread& t;
      ~Join() { t.join(); }
    } join{thread};
    bone.lists();
    bone.paint();
    bone.finish();
  } else {
    // In turns and the marrow phase, whose balls are larger as a rule, first:
    // neither phase's kernels wait for all the other's launches (64^3 242 us, 255
    // with the bone phase queued whole and first; 128^3 364 and 375; 256^3 1306 and
    // 1332; 300 x 310 x 290 2.01 and 2.03 ms).  Where kernels outlast launches the
    // bone phase first, so that the phases are at different kernels (400 x 410 x 390
    // 4.41 ms, 4.49 in turns; 512^3 9.17 and 9.33).
    const bool turns = N < (1ll << 25);
    if (turns) try_twin([&] { marrow.lists(); });
    bone.lists();
    if (turns) try_twin([&] { marrow.paint(); });
    bone.paint();
    if (!turns) try_twin([&] { marrow.lists(), marrow.paint(); });
    bone.finish();
  }
  int st = report_phase(bone, ctx, spacing, th);
  if (st) return st;
  if (queued) try_twin([&] { marrow.finish(); });
  if (twin_status != BM_OK) {
    ctx->last_error = tw->last_error;
    throw CallError{twin_status};
  }
  fence.done = true;
  return report_phase(marrow, ctx, spacing, sp);
}

int tbth_device_impl(bm_ctx* ctx, const uint8_t* d_bone, const uint8_t* d_roi, Dims dm, double spacing,
                     unsigned flags, bm_stats* th, bm_stats* sp, float* d_thmap, float* d_spmap, cudaStream_t s) {
  check_call(ctx, spacing, flags);
  auto feed = [&](Phase& bone, Phase* marrow) {
    count_roi(ctx, d_bone, d_roi, dm.n(), bone.out, s);
    read_roi_counts(ctx, bone.out, s);
    bone.xy(0, dm.d);
    if (marrow) on_twin(ctx, marrow->ctx, [&] { marrow->xy(0, dm.d); });
  };
  try {
    return tbth_phases(ctx, d_bone, d_roi, dm, spacing, flags, th, sp, d_thmap, d_spmap, s, feed);
  } catch (const CallError& e) {
    if (e.status != BM_ERR_OOM) throw;
    // a bail comes before a failed allocation of the phases' buffers
    const std::string message = ctx->last_error;
    PhaseOut* out = phase_out(ctx);
    check(ctx, cudaMemsetAsync(out, 0, sizeof(PhaseOut), s), "memset");
    count_roi(ctx, d_bone, d_roi, dm.n(), out, s);
    read_roi_counts(ctx, out, s);
    check_roi_counts(ctx, dm.n(), flags);
    ctx->last_error = message;
    throw;
  }
}

uint8_t* stage_input(bm_ctx* ctx, Buffer& b, const uint8_t* host, size_t n, cudaStream_t s) {
  uint8_t* d = static_cast<uint8_t*>(ensure(ctx, b, n, "input volume"));
  check(ctx, cudaMemcpyAsync(d, host, n, cudaMemcpyHostToDevice, s), "input upload");
  return d;
}

// bm_tbth_tbsp from host inputs of at least kPipeMinVoxels: bone and ROI go up
// on a copy stream in kPipeSlabs slabs of planes, and each slab's ROI counts
// and x and y passes (of both phases when they run side by side, else of the
// bone phase) start as soon as the slab has landed, so that the transfer hides
// most of those passes.  The bails are checked once every slab is counted; the
// passes that ran before them only wrote the phases' own buffers.
constexpr long long kPipeMinVoxels = 1ll << 22;
constexpr int kPipeSlabs = 8;

int tbth_host_pipelined(bm_ctx* ctx, const uint8_t* bone, const uint8_t* roi, Dims dm, double spacing, unsigned flags,
                        bm_stats* th, bm_stats* sp, float* d_th, float* d_sp, cudaStream_t s) {
  check_call(ctx, spacing, flags);
  const size_t N = (size_t)dm.n();
  uint8_t* d_bone = static_cast<uint8_t*>(ensure(ctx, ctx->in_a, N, "input volume"));
  uint8_t* d_roi = static_cast<uint8_t*>(ensure(ctx, ctx->in_b, N, "input volume"));
  if (!ctx->upload_stream)
    check(ctx, cudaStreamCreateWithFlags(&ctx->upload_stream, cudaStreamNonBlocking), "stream create");
  while ((int)ctx->slab_ready.size() < kPipeSlabs) {
    cudaEvent_t e = nullptr;
    check(ctx, cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "event create");
    ctx->slab_ready.push_back(e);
  }
  return tbth_phases(ctx, d_bone, d_roi, dm, spacing, flags, th, sp, d_th, d_sp, s, [&](Phase& bp, Phase* mp) {
    const int K = dm.d < kPipeSlabs ? dm.d : kPipeSlabs;
    const size_t plane = (size_t)dm.w * dm.h;
    for (int k = 0; k < K; ++k) {
      const int z0 = (int)((long long)dm.d * k / K), z1 = (int)((long long)dm.d * (k + 1) / K);
      const size_t off = (size_t)z0 * plane, len = (size_t)(z1 - z0) * plane;
      check(ctx, cudaMemcpyAsync(d_bone + off, bone + off, len, cudaMemcpyHostToDevice, ctx->upload_stream),
            "input upload");
      check(ctx, cudaMemcpyAsync(d_roi + off, roi + off, len, cudaMemcpyHostToDevice, ctx->upload_stream),
            "input upload");
      check(ctx, cudaEventRecord(ctx->slab_ready[k], ctx->upload_stream), "event record");
      check(ctx, cudaStreamWaitEvent(s, ctx->slab_ready[k], 0), "stream wait");
      count_roi(ctx, d_bone + off, d_roi + off, (long long)len, bp.out, s);
      bp.xy(z0, z1);
      if (mp) on_twin(ctx, mp->ctx, [&] {
        check(mp->ctx, cudaStreamWaitEvent(mp->s, ctx->slab_ready[k], 0), "stream wait");
        mp->xy(z0, z1);
      });
    }
    read_roi_counts(ctx, bp.out, s);
  });
}

}  // namespace

namespace bm {
// Message returned by bm_last_error(NULL, ...) on this thread (used by the
// entry points that take no context).
void set_thread_error(const char* msg) { g_create_error = msg; }

// The per-call working buffers of a context (released by bm_ctx_trim; the
// cached tables stay).
std::vector<Buffer*> work_buffers(bm_ctx* ctx) {
  return {&ctx->in_a,      &ctx->in_b,       &ctx->dist,        &ctx->dist2,   &ctx->edtmap,
          &ctx->chainmap,  &ctx->fillmap,    &ctx->selbits,     &ctx->ridgebits, &ctx->ridges, &ctx->phaseout,
          &ctx->outmap,    &ctx->outmap2,     &ctx->occ,     &ctx->rank,   &ctx->rvals,
          &ctx->bincounts, &ctx->binoffsets, &ctx->binentries,  &ctx->scanscratch, &ctx->qhist,
          &ctx->qtargets,  &ctx->qmap,       &ctx->rgeo,        &ctx->ordscratch,
          &ctx->tileorder, &ctx->dischdr,     &ctx->discent, &ctx->discpool,
          &ctx->nzbits,    &ctx->inbits};
}

size_t cached_bytes(const bm_ctx* ctx) {
  size_t t = 0;
  for (const Buffer* b : work_buffers(const_cast<bm_ctx*>(ctx))) t += b->bytes;
  if (ctx->twin) t += cached_bytes(ctx->twin);
  return t;
}
}  // namespace bm

extern "C" {

int bm_ctx_create(int device, bm_ctx** out) {
  if (!out) return BM_ERR_INVALID;
  *out = nullptr;
  int ndev = 0;
  cudaError_t e = cudaGetDeviceCount(&ndev);
  if (e != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    set_err(nullptr, "no CUDA device available: %s", e == cudaSuccess ? "device count is 0" : cudaGetErrorString(e));
    return BM_ERR_NO_DEVICE;
  }
  if (device < 0 || device >= ndev) {
    set_err(nullptr, "device %d out of range (0..%d)", device, ndev - 1);
    return BM_ERR_INVALID;
  }
  bm_ctx* ctx = new (std::nothrow) bm_ctx();
  if (!ctx) return BM_ERR_OOM;
  ctx->device = device;
  e = cudaSetDevice(device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&ctx->num_sms, cudaDevAttrMultiProcessorCount, device);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ctx->counted, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaMallocHost(&ctx->pinned, sizeof(Readback));
  if (e != cudaSuccess) {
    cudaGetLastError();
    if (ctx->counted) cudaEventDestroy(ctx->counted);
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
    set_err(nullptr, "context creation failed: %s", cudaGetErrorString(e));
    delete ctx;
    return BM_ERR_CUDA;
  }
  *out = ctx;
  return BM_OK;
}

int bm_ctx_trim(bm_ctx* ctx) {
  return guarded(ctx, [&]() -> int {
    cudaStreamSynchronize(ctx->stream);
    if (ctx->twin) bm_ctx_trim(ctx->twin);
    for (Buffer* b : work_buffers(ctx)) release(*b);
    return BM_OK;
  });
}

void bm_ctx_destroy(bm_ctx* ctx) {
  if (!ctx) return;
  {
    std::lock_guard<std::mutex> plock(ctx->pool_mu);
    if (ctx->pool) pool_destroy(ctx->pool);
    ctx->pool = nullptr;
  }
  {
    std::lock_guard<std::mutex> lock(ctx->mu);
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    if (ctx->twin) bm_ctx_destroy(ctx->twin);
    ctx->twin = nullptr;
    if (ctx->inputs_ready) cudaEventDestroy(ctx->inputs_ready);
    if (ctx->counted) cudaEventDestroy(ctx->counted);
    if (ctx->pinned) cudaFreeHost(ctx->pinned);
    if (ctx->upload_stream) {
      cudaStreamSynchronize(ctx->upload_stream);
      cudaStreamDestroy(ctx->upload_stream);
    }
    for (cudaEvent_t e : ctx->slab_ready) cudaEventDestroy(e);
    for (Buffer* b : work_buffers(ctx)) release(*b);
    for (Buffer* b : {&ctx->lut, &ctx->fillinfo}) release(*b);
    for (const ProfRec& r : ctx->prof) {
      cudaEventDestroy(r.start);
      cudaEventDestroy(r.stop);
    }
    for (cudaEvent_t e : ctx->event_pool) cudaEventDestroy(e);
    release(ctx->surf_off);
    release(ctx->surf_pts);
    release(ctx->lutf);
    release(ctx->discthr);
    release(ctx->disctmpl);
    if (ctx->stream) cudaStreamDestroy(ctx->stream);
  }
  delete ctx;
}

const char* bm_status_string(int status) {
  switch (status) {
    case BM_OK: return "ok";
    case BM_ERR_ALL_SELECTED: return "all voxels selected";
    case BM_ERR_DIMS: return "invalid dimensions";
    case BM_ERR_OOM: return "out of device memory";
    case BM_ERR_CUDA: return "CUDA error";
    case BM_ERR_TIMEOUT: return "device wait timed out";
    case BM_ERR_INVALID: return "invalid argument";
    case BM_ERR_EMPTY: return "empty phase";
    case BM_ERR_ROI_EMPTY: return "empty ROI";
    case BM_ERR_NO_BONE: return "no bone in ROI";
    case BM_ERR_NO_MARROW: return "no marrow in ROI";
    case BM_ERR_NO_DEVICE: return "no CUDA device";
    case BM_ERR_SPACING: return "invalid spacing";
    case BM_ERR_ROI_FULL: return "ROI has no outside voxels";
    case BM_ERR_BUSY: return "busy";
    default: return "unknown status";
  }
}

size_t bm_last_error(const bm_ctx* ctx, char* buf, size_t len) {
  const std::string& s = ctx ? ctx->last_error : g_create_error;
  if (buf && len) {
    const size_t n = s.size() < len - 1 ? s.size() : len - 1;
    std::memcpy(buf, s.data(), n);
    buf[n] = 0;
  }
  return s.size();
}

uint64_t bm_ctx_launch_count(const bm_ctx* ctx) { return ctx ? ctx->launches : 0; }

int bm_ctx_set_concurrent_phases(bm_ctx* ctx, int on) {
  return guarded(ctx, [&]() -> int {
    ctx->split_phases = on != 0;
    return BM_OK;
  });
}

int bm_ctx_set_site_method(bm_ctx* ctx, int method) {
  return guarded(ctx, [&]() -> int {
    if (method != BM_SITES_AUTO && method != BM_SITES_SPHERES && method != BM_SITES_CHAINS)
      fail(ctx, BM_ERR_INVALID, "site method must be 0 (auto), 1 (spheres) or 2 (chains); got %d", method);
    ctx->site_method = method;
    if (ctx->twin) ctx->twin->site_method = method;
    return BM_OK;
  });
}

int bm_ctx_set_fill_tile_rows(bm_ctx* ctx, int rows) {
  return guarded(ctx, [&]() -> int {
    if (rows != 0 && rows != 16 && rows != 32 && rows != 64)
      fail(ctx, BM_ERR_INVALID, "fill tile rows must be 0 (by volume size), 16, 32 or 64; got %d", rows);
    ctx->fill_rows = rows;
    if (ctx->twin) ctx->twin->fill_rows = rows;
    return BM_OK;
  });
}

int bm_ctx_set_wait_cycles(bm_ctx* ctx, long long cycles) {
  return guarded(ctx, [&]() -> int {
    ctx->wait_cycles = cycles < 0 ? -1 : cycles;
    if (ctx->twin) ctx->twin->wait_cycles = ctx->wait_cycles;
    return BM_OK;
  });
}

int bm_ctx_fail_allocation(bm_ctx* ctx, const char* what, int skip) {
  return guarded(ctx, [&]() -> int {
    if (skip < 0) fail(ctx, BM_ERR_INVALID, "skip must not be negative; got %d", skip);
    ctx->fail_what = what ? what : "";
    ctx->fail_skip = skip;
    return BM_OK;
  });
}

int bm_profile_enable(bm_ctx* ctx, int on) {
  return guarded(ctx, [&]() -> int {
    fold_profile(ctx);
    if (on) {
      for (int i = 0; i < KF_COUNT; ++i) {
        ctx->prof_ms[i] = 0.0;
        ctx->prof_n[i] = 0;
      }
    }
    ctx->profiling = on != 0;
    if (ctx->twin) bm_profile_enable(ctx->twin, on);
    return BM_OK;
  });
}

int bm_profile_read(bm_ctx* ctx, bm_kernel_time* out, size_t cap, size_t* count) {
  return guarded(ctx, [&]() -> int {
    fold_profile(ctx);
    if (ctx->twin) {  // the twin's kernels count as this context's
      bm_ctx* t = ctx->twin;
      std::lock_guard<std::mutex> tl(t->mu);
      fold_profile(t);
      for (int i = 0; i < KF_COUNT; ++i) {
        ctx->prof_ms[i] += t->prof_ms[i];
        ctx->prof_n[i] += t->prof_n[i];
        t->prof_ms[i] = 0.0;
        t->prof_n[i] = 0;
      }
    }
    size_t n = 0;
    for (int i = 0; i < KF_COUNT; ++i) {
      if (out && n < cap) {
        std::memset(out[n].name, 0, sizeof out[n].name);
        std::strncpy(out[n].name, kFamilyName[i], sizeof out[n].name - 1);
        out[n].launches = ctx->prof_n[i];
        out[n].total_ms = ctx->prof_ms[i];
      }
      ++n;
    }
    if (count) *count = n;
    return BM_OK;
  });
}

int bm_edt_sq_device(bm_ctx* ctx, const uint8_t* d_volume, size_t width, size_t height, size_t depth, int phase,
                     uint32_t* d_out, void* stream) {
  return guarded(ctx, [&]() -> int {
    if (!d_volume || !d_out) fail(ctx, BM_ERR_INVALID, "null pointer");
    check_phase(ctx, phase);
    const Dims dm = check_dims(ctx, width, height, depth);
    return edt_device_impl(ctx, d_volume, dm, phase, d_out, pick_stream(ctx, stream));
  });
}

int bm_edt_sq(bm_ctx* ctx, const uint8_t* volume, size_t width, size_t height, size_t depth, int phase,
              uint32_t* out) {
  return guarded(ctx, [&]() -> int {
    if (!volume || !out) fail(ctx, BM_ERR_INVALID, "null pointer");
    check_phase(ctx, phase);
    const Dims dm = check_dims(ctx, width, height, depth);
    const size_t N = (size_t)dm.n();
    cudaStream_t s = ctx->stream;
    uint8_t* d_in = stage_input(ctx, ctx->in_a, volume, N, s);
    uint32_t* d_out = static_cast<uint32_t*>(ensure(ctx, ctx->fillmap, N * 4, "output"));
    edt_device_impl(ctx, d_in, dm, phase, d_out, s);
    check(ctx, cudaMemcpyAsync(out, d_out, N * 4, cudaMemcpyDeviceToHost, s), "result download");
    check(ctx, cudaStreamSynchronize(s), "result download");
    return BM_OK;
  });
}

int bm_local_thickness_device(bm_ctx* ctx, const uint8_t* d_volume, size_t width, size_t height, size_t depth,
                              int phase, float* d_out, uint32_t* d_squared_thickness, void* stream) {
  return guarded(ctx, [&]() -> int {
    if (!d_volume || !d_out) fail(ctx, BM_ERR_INVALID, "null pointer");
    check_phase(ctx, phase);
    const Dims dm = check_dims(ctx, width, height, depth);
    return lt_device_impl(ctx, d_volume, dm, phase, d_out, d_squared_thickness, pick_stream(ctx, stream));
  });
}

int bm_local_thickness(bm_ctx* ctx, const uint8_t* volume, size_t width, size_t height, size_t depth, int phase,
                       float* out, uint32_t* squared_thickness) {
  return guarded(ctx, [&]() -> int {
    if (!volume || !out) fail(ctx, BM_ERR_INVALID, "null pointer");
    check_phase(ctx, phase);
    const Dims dm = check_dims(ctx, width, height, depth);
    const size_t N = (size_t)dm.n();
    cudaStream_t s = ctx->stream;
    uint8_t* d_in = stage_input(ctx, ctx->in_a, volume, N, s);
    float* d_out = static_cast<float*>(ensure(ctx, ctx->outmap, N * 4, "output"));
    uint32_t* d_sq = squared_thickness ? static_cast<uint32_t*>(ensure(ctx, ctx->fillmap, N * 4, "output")) : nullptr;
    lt_device_impl(ctx, d_in, dm, phase, d_out, d_sq, s);
    check(ctx, cudaMemcpyAsync(out, d_out, N * 4, cudaMemcpyDeviceToHost, s), "result download");
    if (squared_thickness)
      check(ctx, cudaMemcpyAsync(squared_thickness, d_sq, N * 4, cudaMemcpyDeviceToHost, s), "result download");
    check(ctx, cudaStreamSynchronize(s), "result download");
    return BM_OK;
  });
}

int bm_nonzero_stats_device(bm_ctx* ctx, const float* d_values, size_t n, double scale, unsigned flags,
                            bm_stats* out, void* stream) {
  return guarded(ctx, [&]() -> int {
    if (!d_values || !out) fail(ctx, BM_ERR_INVALID, "null pointer");
    if (flags & ~(unsigned)BM_FLAG_QUANTILES) fail(ctx, BM_ERR_INVALID, "unknown flags 0x%x", flags);
    cudaStream_t s = pick_stream(ctx, stream);
    return nonzero_stats_impl(ctx, d_values, n, scale, flags, out, s);
  });
}

int bm_nonzero_stats(bm_ctx* ctx, const float* values, size_t n, double scale, unsigned flags, bm_stats* out) {
  return guarded(ctx, [&]() -> int {
    if (!values || !out) fail(ctx, BM_ERR_INVALID, "null pointer");
    if (flags & ~(unsigned)BM_FLAG_QUANTILES) fail(ctx, BM_ERR_INVALID, "unknown flags 0x%x", flags);
    cudaStream_t s = ctx->stream;
    float* d = static_cast<float*>(ensure(ctx, ctx->qmap, (n ? n : 1) * 4, "values"));
    if (n) check(ctx, cudaMemcpyAsync(d, values, n * 4, cudaMemcpyHostToDevice, s), "values upload");
    return nonzero_stats_impl(ctx, d, n, scale, flags, out, s);
  });
}

int bm_volume_metrics_device(bm_ctx* ctx, const uint8_t* d_bone, const uint8_t* d_roi, size_t width, size_t height,
                             size_t depth, const double spacing_um[3], bm_volume_metrics* out, void* stream) {
  return guarded(ctx, [&]() -> int {
    if (!d_bone || !d_roi || !spacing_um || !out) fail(ctx, BM_ERR_INVALID, "null pointer");
    const Dims dm = check_dims(ctx, width, height, depth);
    return volume_metrics_impl(ctx, d_bone, d_roi, dm, spacing_um, out, pick_stream(ctx, stream));
  });
}

int bm_volume_metrics_compute(bm_ctx* ctx, const uint8_t* bone, const uint8_t* roi, size_t width, size_t height,
                              size_t depth, const double spacing_um[3], bm_volume_metrics* out) {
  return guarded(ctx, [&]() -> int {
    if (!bone || !roi || !spacing_um || !out) fail(ctx, BM_ERR_INVALID, "null pointer");
    const Dims dm = check_dims(ctx, width, height, depth);
    const size_t N = (size_t)dm.n();
    cudaStream_t s = ctx->stream;
    const uint8_t* d_bone = stage_input(ctx, ctx->in_a, bone, N, s);
    const uint8_t* d_roi = stage_input(ctx, ctx->in_b, roi, N, s);
    return volume_metrics_impl(ctx, d_bone, d_roi, dm, spacing_um, out, s);
  });
}

int bm_tbth_tbsp_device(bm_ctx* ctx, const uint8_t* d_bone, const uint8_t* d_roi, size_t width, size_t height,
                        size_t depth, double spacing_um, unsigned flags, bm_stats* thickness, bm_stats* spacing,
                        float* d_thickness_map, float* d_spacing_map, void* stream) {
  return guarded(ctx, [&]() -> int {
    if (!d_bone || !d_roi) fail(ctx, BM_ERR_INVALID, "null pointer");
    const Dims dm = check_dims(ctx, width, height, depth);
    return tbth_device_impl(ctx, d_bone, d_roi, dm, spacing_um, flags, thickness, spacing, d_thickness_map,
                            d_spacing_map, pick_stream(ctx, stream));
  });
}

int bm_tbth_tbsp(bm_ctx* ctx, const uint8_t* bone, const uint8_t* roi, size_t width, size_t height, size_t depth,
                 double spacing_um, unsigned flags, bm_stats* thickness, bm_stats* spacing, float* thickness_map,
                 float* spacing_map) {
  return guarded(ctx, [&]() -> int {
    if (!bone || !roi) fail(ctx, BM_ERR_INVALID, "null pointer");
    const Dims dm = check_dims(ctx, width, height, depth);
    const size_t N = (size_t)dm.n();
    cudaStream_t s = ctx->stream;
    float* d_th = thickness_map ? static_cast<float*>(ensure(ctx, ctx->outmap, N * 4, "output")) : nullptr;
    float* d_sp = spacing_map ? static_cast<float*>(ensure(ctx, ctx->outmap2, N * 4, "output")) : nullptr;
    int st;
    if ((long long)N >= kPipeMinVoxels) {
      st = tbth_host_pipelined(ctx, bone, roi, dm, spacing_um, flags, thickness, spacing, d_th, d_sp, s);
    } else {
      const uint8_t* d_bone = stage_input(ctx, ctx->in_a, bone, N, s);
      const uint8_t* d_roi = stage_input(ctx, ctx->in_b, roi, N, s);
      st = tbth_device_impl(ctx, d_bone, d_roi, dm, spacing_um, flags, thickness, spacing, d_th, d_sp, s);
    }
    if (st) return st;
    if (thickness_map)
      check(ctx, cudaMemcpyAsync(thickness_map, d_th, N * 4, cudaMemcpyDeviceToHost, s), "result download");
    if (spacing_map)
      check(ctx, cudaMemcpyAsync(spacing_map, d_sp, N * 4, cudaMemcpyDeviceToHost, s), "result download");
    check(ctx, cudaStreamSynchronize(s), "result download");
    return BM_OK;
  });
}

}  // extern "C"
