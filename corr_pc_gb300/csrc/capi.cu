// capi.cu -- the C ABI (include/corrpc.h): contexts, catalogue upload with the
// on-device cell list, per-job set-up (the reference's corels2 rules, exact
// thresholds and FP32 guard bands), work-unit construction and launches.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <cstdlib>
#include <exception>
#include <map>
#include <memory>
#include <stdexcept>
#include <string>
#include <system_error>
#include <thread>
#include <tuple>
#include <vector>

#include "../../include/corrpc.h"
#include "cpc_device.cuh"
#include "host_helpers.h"
#include "param_check.h"
#include "kernels.h"

using namespace cpc;

// initial capacity of the FP64 edge queue (entries); it grows when a count
// needs more
#ifndef CPC_EDGE_QUEUE_INIT
#define CPC_EDGE_QUEUE_INIT (1ull << 24)
#endif

namespace {

// message of the calling thread's last failing call (entry points without a context)
thread_local std::string g_err;

template <class T>
struct DevBuf {
  T *p = nullptr;
  size_t n = 0;
  DevBuf() = default;
  DevBuf(const DevBuf &) = delete;
  DevBuf &operator=(const DevBuf &) = delete;
  ~DevBuf() { reset(); }
  void reset() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
  cudaError_t alloc(size_t count) {
    if (count <= n && p) return cudaSuccess;
    reset();
    if (count == 0) count = 1;
    cudaError_t e = cudaMalloc(&p, sizeof(T) * count);
    if (e != cudaSuccess) {
      p = nullptr;
      return e;
    }
    n = count;
    return cudaSuccess;
  }
};

struct Slot {
  bool valid = false;
  int64_t n = 0;
  bool has_e = false, exact_f32 = true;
  double wmax = 1.0, wmin = 1.0, emax = 0.0, cmax = 0.0, phimax = 0.0;
  uint64_t version = 0;
  // grid this cell list was built with
  int ncx = 0, ncy = 0, n_reg = 1, kcells = 0;
  bool auto_k = true;  // kcells is automatic, not a width that the caller set
  double cw_x = 0, cw_y = 0, row_density = 0;
  // device, cell order
  DevBuf<float4> pos, shp, ewt, aux;
  DevBuf<float> zlo, zf;
  DevBuf<double> x, y, z, w, e1, e2, phi, e3;
  DevBuf<int32_t> jk;
  DevBuf<uint8_t> keep;
  DevBuf<int64_t> orig;
  DevBuf<uint8_t> aflag;  // corels1 scan-start flags of each row (cell order)
  DevBuf<int> bk_start, bk_end, bk_region, col_begin, col_end;
  DevBuf<float> bk_zmin, bk_zmax;
  // host copies used to build work units
  std::vector<float4> h_pos;
  std::vector<int> h_bk_start, h_bk_end, h_bk_region;
  // z-ordered FP64 copy for the plain kernel (built on first use)
  bool zbuilt = false;
  DevBuf<double> zx, zy, zz, zw, ze1, ze2, zphi, ze3;
  DevBuf<int32_t> zjk;
  DevBuf<uint8_t> zkeep, zaflag;
  DevBuf<int64_t> zorig;
  // sky (coordinates 0): x, y, z, w, e1, e2, phi, jk, keep, orig above hold the
  // redshift-ordered catalogue; these the sky-only per-galaxy quantities
  bool sky = false;
  DevBuf<double> dc, da, sd, cd, rar, decr, win;
  // cell order (SkyFast): sorted by (region, keep flag, sky cell, redshift)
  DevBuf<unsigned char> sky_pack;  // every array of sky_f, one allocation and one copy
  SkyFast sky_f{};
  bool sky_mono = false;      // the rows' redshift window bounds rise with the redshift
  double dcmax = 0;           // largest |D_C| (error bound of the float Pi)
  double damin = 0, damax = 0;  // range of D_A
  double sky_mag = 0;         // largest window bound or coordinate of the float tests
  double sky_zw = 0;          // mean width of the rows' windows in scaled redshift
  double sky_fz = 0;          // mean share of the catalogue inside a row's redshift window
  double sky_hw = 0, sky_area = 0;  // mean half width of the rows' Dec windows; area (degrees)
  int sky_nkey = 0;           // (region, keep flag) keys with galaxies
  std::vector<int> hc_zidx;   // redshift-ordered position of each cell-ordered row
  std::vector<float> hc_z;    // scaled redshift, cell order
  std::vector<int4> hc_bk;    // buckets
  std::vector<SkyTileRows> hc_tiles;  // tiles over every row (built by the first count)
  std::vector<int> hc_tile_key;       // their bucket keys
  std::vector<float4> hc_bwin, hc_box;  // per bucket: union of its rows' RA/Dec windows; its box
  // host copies in the same order for the host edge tier
  std::vector<double> hs_ra, hs_dec, hs_dc, hs_da, hs_w, hs_e1, hs_e2, hs_phi;
  std::vector<int32_t> hs_jk;
  std::vector<uint8_t> hs_keep;
  std::vector<int64_t> hs_orig;  // input row of each redshift-ordered row (row samples)
};

// device buffers of one job of a sky launch: its histogram block, fixed-point
// sums, counters, host-tier queue and row sample
struct SkyJobBufs {
  DevBuf<unsigned long long> num, fix, counters, hq_n, xq_n;
  DevBuf<double> sums;
  DevBuf<int2> hq, xq;
  DevBuf<int> rows;
  DevBuf<SkyTileRows> tiles;
};

// a box job's histogram block and counters
struct AccumBufs {
  DevBuf<unsigned long long> num, counters;
  DevBuf<double> sums;
};

struct UnitCache {
  uint64_t v1 = 0, v2 = 0;
  int s1 = -1, s2 = -1, wpi = 0, tile = 0, twin = 0, variant = 0;
  uint64_t id = 0;  // of this list's contents: never given twice in the process
  std::vector<UnitDesc> units;  // job field filled at launch
};

}  // namespace

namespace {
struct JobPlan;  // one planned count (below)
}  // namespace

struct cpc_ctx {
  int64_t pref_n = -1;  // preferred_cells for a largest catalogue of pref_n rows
  int pref_k = 2;
  cpc_params p{};
  std::vector<double> H, dA;
  std::string err;
  Slot slots[kMaxSlots];
  uint64_t version_ctr = 0;
  double ps = 0, rsize = 0;
  double thr_rp[kMaxRp + 1];
  double thr_pi[kMaxPi + 1];
  int tune_k = 0, tune_wpi = 0, tune_tile = 0;
  int device = 0, sm_count = 152;
  cudaStream_t st = nullptr;
  cudaStream_t st2 = nullptr;  // beside st, for launches that may overlap (sky_run)
  cudaEvent_t e0 = nullptr, e1 = nullptr, e2 = nullptr;
  cudaEvent_t e_in = nullptr, e_done = nullptr;  // cpc_count_async ordering
  // scratch
  DevBuf<JobDev> d_jobs;
  DevBuf<UnitDesc> d_units;
  std::vector<uint64_t> units_key;  // what d_units holds (enqueue_fast)
  DevBuf<unsigned int> d_unit_ctr;
  DevBuf<QEntry> d_queue;
  DevBuf<unsigned long long> d_qcount;
  unsigned long long qcap = 0;
  double q_per_unit = 0;  // most pairs any count queued per work unit (queue sizing)
  size_t last_units = 0;  // work units of the last fast launch
  std::vector<std::unique_ptr<AccumBufs>> accum;  // one per job of this context in a launch
  // sky launches: one buffer set per job of the launch, the unit queue
  std::vector<std::unique_ptr<SkyJobBufs>> sky_bufs;
  DevBuf<SkyUnit> d_sky_units;
  DevBuf<unsigned long long> d_sky_ctr;
  // sort scratch
  DevBuf<uint64_t> d_keys, d_ktmp;
  DevBuf<uint32_t> d_vals, d_vtmp, d_hist, d_bucket;
  DevBuf<unsigned long long> d_census;
  // upload scratch: a catalogue in input order, its checks and statistics
  DevBuf<double> u_x, u_y, u_z, u_w, u_e1, u_e2, u_phi, u_prob, u_e3;
  DevBuf<int32_t> u_jk;
  DevBuf<uint8_t> u_keep, u_flag;
  DevBuf<int64_t> u_orig;
  DevBuf<UploadStats> d_ustats;
  UploadStats h_ustats{};
  std::vector<UnitCache> unit_cache;
  // a count enqueued by cpc_count_async, collected by cpc_count_finish
  int pending = 0;  // 0 none, 1 fast engine, 2 FP64 engine
  std::vector<JobPlan> pending_jobs;
  int64_t launches = 0;  // kernels launched by this context (all entry points)
  // work-unit shard of the fast box engine (cpc_set_shard)
  int shard = 0, n_shards = 1;
  // whether two box slots hold the same galaxies in the same order (twin jobs),
  // for the slot pair and versions last compared; CPC_TWIN=0 turns twin jobs off
  int twin_s1 = -1, twin_s2 = -1;
  uint64_t twin_v1 = 0, twin_v2 = 0;
  bool twin_same = false;
  int twin_on = 1;
  int last_twin = 0;  // the last fast count ran a twin job
  DevBuf<unsigned> d_differ;
  // CUDA graph of the fast engine's device work (zeroing, pair kernels,
  // recheck), replayed while every value baked into it stays the same
  int graph_on = 1;
  cudaGraphExec_t gexec = nullptr;
  std::vector<uint64_t> gkey;
  int64_t graph_captures = 0, graph_replays = 0;
};

namespace {

// Record msg as the context's (and the library's) last error and return s.  A
// message that cannot be stored (out of host memory) leaves the old one.
cpc_status fail(cpc_ctx *c, cpc_status s, const std::string &msg) noexcept {
  try {
    if (c) c->err = msg;
    g_err = msg;
  } catch (...) {
  }
  return s;
}

// The status of a C++ exception that reached an entry point (called from its
// catch block): no exception crosses the C ABI.  A stream capture left open
// by the interrupted call is closed so that the context stays usable.
cpc_status host_exception(cpc_ctx *c) noexcept {
  if (c && c->st) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(c->st, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone) {
      cudaGraph_t g = nullptr;
      cudaStreamEndCapture(c->st, &g);
      if (g) cudaGraphDestroy(g);
      cudaGetLastError();
    }
  }
  try {
    throw;
  } catch (const std::bad_alloc &) {
    return fail(c, CPC_ERR_NOMEM, "host allocation failed");
  } catch (const std::length_error &) {
    return fail(c, CPC_ERR_NOMEM, "host allocation too large");
  } catch (const std::exception &e) {
    return fail(c, CPC_ERR_HOST, std::string("host error: ") + e.what());
  } catch (...) {
    return fail(c, CPC_ERR_HOST, "host error");
  }
}

cpc_status cuda_fail(cpc_ctx *c, cudaError_t e, const char *where) {
  std::string m = std::string(where) + ": " + cudaGetErrorString(e);
  if (e == cudaErrorMemoryAllocation) return fail(c, CPC_ERR_NOMEM, m);
  if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) return fail(c, CPC_ERR_NODEVICE, m);
  return fail(c, CPC_ERR_CUDA, m);
}

#define CK(expr, where)                              \
  do {                                               \
    cudaError_t _e = (expr);                         \
    if (_e != cudaSuccess) return cuda_fail(c, _e, where); \
  } while (0)

// Run f(begin, end, part) over [0, n) in contiguous chunks on the host's cores
// (one chunk per thread, part < 64, at least min_chunk items each; in the
// calling thread when n is small).  Parts whose thread cannot be started run in
// the calling thread; the first exception thrown by a part is rethrown here
// after every part has finished.
template <class F>
void host_parallel(int64_t n, F &&f, int64_t min_chunk = 16384) {
  const int64_t hw = std::max(1u, std::thread::hardware_concurrency());
  const int T = (int)std::max<int64_t>(1, std::min<int64_t>({hw, 64, n / min_chunk}));
  if (T <= 1) {
    f((int64_t)0, n, 0);
    return;
  }
  std::exception_ptr errs[64];
  auto part = [&f, &errs, n, T](int t) {
    try {
      f(n * t / T, n * (t + 1) / T, t);
    } catch (...) {
      errs[t] = std::current_exception();
    }
  };
  std::vector<std::thread> th;
  th.reserve(T);
  int t = 0;
  for (; t < T; t++) {
    try {
      th.emplace_back(part, t);
    } catch (const std::system_error &) {
      break;
    }
  }
  for (; t < T; t++) part(t);
  for (auto &x : th) x.join();
  for (int k = 0; k < T; k++)
    if (errs[k]) std::rethrow_exception(errs[k]);
}

// float ULP at magnitude v (v > 0)
double ulpf(double v) {
  if (!(v > 0)) return std::ldexp(1.0, -149);
  int ex;
  std::frexp(v, &ex);  // v = m * 2^ex, m in [0.5, 1)
  return std::ldexp(1.0, ex - 1 - 23);
}
float f_up(double v) {
  float f = (float)v;
  if ((double)f < v) f = std::nextafter(f, INFINITY);
  return f;
}
float f_down(double v) {
  float f = (float)v;
  if ((double)f > v) f = std::nextafter(f, -INFINITY);
  return f;
}

cpc_status validate_params(cpc_ctx *c, const cpc_params &p) {
  if (const char *m = param_error(p)) return fail(c, CPC_ERR_INVALID, m);
  return CPC_OK;
}

// corels2's pair-type rules (corr.cpp:226-296) and corel choice
// (initialization.cpp:699-752).
struct JobRule {
  int corel, gws, swapped;
};
int job_rule(const cpc_params &p, cpc_pair_kind kind, int64_t n1, int64_t n2, JobRule &r) {
  int gws = 0;
  switch (kind) {
    case CPC_PAIR_DRS: case CPC_PAIR_RSRD: case CPC_PAIR_RSRS: gws = 0; break;
    case CPC_PAIR_SRD: case CPC_PAIR_SD: case CPC_PAIR_SRS: gws = 2; break;
    default: return -1;
  }
  int corel;
  if (kind == CPC_PAIR_RSRS || kind == CPC_PAIR_RSRD || p.which_corr == 0) corel = COREL_DD;
  else if (p.which_corr == 1) corel = COREL_SD;
  else if (p.which_corr == 2) corel = (kind == CPC_PAIR_SD) ? COREL_SS : COREL_SD;
  else corel = COREL_DK + (p.which_corr - 3);  // 3 DK, 4 SK, 5 ED
  if (corel == COREL_SS && p.estimator != 0) corel = COREL_SSA;
  r.swapped = 0;
  if (n2 > n1) {
    r.swapped = 1;
    if (gws == 2) gws = 1; else if (gws == 1) gws = 2;
  }
  r.corel = corel;
  r.gws = gws;
  return 0;
}

// corels1's rules (corr.cpp:103-216): g_with_shape = 1, no swap; corel by
// choose_corel_func (initialization.cpp:490-520) with do_RsRs or do_SS set.
int job_rule_auto(const cpc_params &p, cpc_pair_kind kind, JobRule &r) {
  int corel;
  if (kind == CPC_PAIR_RSRS) corel = COREL_DD;
  else if (kind == CPC_PAIR_SS)
    corel = p.which_corr == 0 ? COREL_DD : p.which_corr <= 2 ? COREL_SS : COREL_DK + (p.which_corr - 3);
  else return -1;
  if (corel == COREL_SS && p.estimator != 0) corel = COREL_SSA;
  r.swapped = 0;
  r.corel = corel;
  r.gws = 1;
  return 0;
}

void fill_views(Slot &s, FCat &f, DCat &d) {
  f.n = s.n;
  f.pos = s.pos.p;
  f.shp = s.shp.p;
  f.ewt = s.ewt.p;
  f.aux = s.aux.p;
  f.zlo = s.zlo.p;
  f.zf = s.zf.p;
  f.keep = s.keep.p;
  f.aflag = s.aflag.p;
  f.bk_start = s.bk_start.p;
  f.bk_end = s.bk_end.p;
  f.bk_region = s.bk_region.p;
  f.bk_zmin = s.bk_zmin.p;
  f.bk_zmax = s.bk_zmax.p;
  f.col_begin = s.col_begin.p;
  f.col_end = s.col_end.p;
  d.n = s.n;
  d.x = s.x.p; d.y = s.y.p; d.z = s.z.p; d.w = s.w.p;
  d.e1 = s.e1.p; d.e2 = s.e2.p; d.phi = s.phi.p; d.e3 = s.e3.p;
  d.jk = s.jk.p; d.keep = s.keep.p; d.orig = s.orig.p; d.aflag = s.aflag.p;
}

// z window offsets of lim_calc_xyz (PB_calcs.cpp:12-28): [p_min, p_max], or
// [-r_max, r_max] for coordinates 7 (p_min, p_max then bound mu)
double wz_lo(const cpc_params &p) { return p.coordinates == 7 ? -p.bin_r_max : p.p_min; }
double wz_hi(const cpc_params &p) { return p.coordinates == 7 ? p.bin_r_max : p.p_max; }

// error bound (absolute, per coordinate difference) of the FP32 separations
double eps_abs(const cpc_ctx *c, const Slot &a, const Slot &b) {
  const cpc_params &p = c->p;
  const double L = p.periodic_box_size;
  const double cmax = std::max({a.cmax, b.cmax, L});
  double e = 0;
  if (!(a.exact_f32 && b.exact_f32)) e += ulpf(cmax);
  const double wmax = std::max({p.bin_r_max, wz_hi(p), -wz_lo(p)});
  if (p.periodic_box && !(wmax <= 0.45 * L)) e += ulpf(2 * cmax);
  return e;
}

struct JobPlan {
  cpc_ctx *c;
  cpc_pair_kind kind;
  int s1, s2;  // after the swap
  JobRule rule;
  int wpi, tile;
  int variant;  // of the fast kernel (kernels.h)
  int64_t row_stride, row_offset;
  cpc_accum *out;
  JobDev jd;
  bool empty;
};

// every weight of both catalogues is 1: the weight sum is the count (the fast
// kernel keeps no words for it)
int unit_weights(const Slot &a, const Slot &b) {
  return (a.wmax == 1.0 && a.wmin == 1.0 && b.wmax == 1.0 && b.wmin == 1.0) ? 1 : 0;
}

// A context's unit shard replaced for the autotuner's trials, restored when the
// trials end (or on any early return).
struct ShardOverride {
  cpc_ctx *c;
  int shard, n_shards;
  bool active = true;
  ShardOverride(cpc_ctx *ctx, int sh, int nsh) : c(ctx), shard(ctx->shard), n_shards(ctx->n_shards) {
    c->shard = sh;
    c->n_shards = nsh;
  }
  void restore() {
    if (!active) return;
    c->shard = shard;
    c->n_shards = n_shards;
    active = false;
  }
  ~ShardOverride() { restore(); }
};

// Whether box slots sa and sb hold the same galaxies in the same (cell) order:
// positions, weights, shapes, orientations, regions and input rows identical
// (the keep flags, drawn from rand() per read, may differ).  A cross term of a
// catalogue with itself, uploaded as two samples, is such a pair.  Compared on
// the device, cached per slot versions.
bool slots_twin(cpc_ctx *c, int sa, int sb) {
  if (sa == sb) return true;
  Slot &A = c->slots[sa], &B = c->slots[sb];
  if (!A.valid || !B.valid || A.sky || B.sky || A.n != B.n || A.has_e != B.has_e ||
      A.kcells != B.kcells || A.ncx != B.ncx || A.ncy != B.ncy || A.n_reg != B.n_reg)
    return false;
  if (c->twin_s1 == sa && c->twin_s2 == sb && c->twin_v1 == A.version && c->twin_v2 == B.version)
    return c->twin_same;
  const int64_t n = A.n;
  bool same = false;
  if (c->d_differ.alloc(1) == cudaSuccess &&
      cudaMemsetAsync(c->d_differ.p, 0, sizeof(unsigned), c->st) == cudaSuccess) {
    const std::pair<const void *, const void *> arr8[] = {
        {A.x.p, B.x.p}, {A.y.p, B.y.p}, {A.z.p, B.z.p}, {A.w.p, B.w.p}, {A.e1.p, B.e1.p},
        {A.e2.p, B.e2.p}, {A.phi.p, B.phi.p}, {A.e3.p, B.e3.p}, {A.orig.p, B.orig.p}};
    bool ok = true;
    for (const auto &ab : arr8)
      ok = ok && launch_bytes_differ(ab.first, ab.second, 8 * n, c->d_differ.p, c->st) ==
                     cudaSuccess;
    ok = ok && launch_bytes_differ(A.jk.p, B.jk.p, 4 * n, c->d_differ.p, c->st) == cudaSuccess;
    unsigned d = 1;
    if (ok && cudaMemcpyAsync(&d, c->d_differ.p, sizeof d, cudaMemcpyDeviceToHost, c->st) ==
                  cudaSuccess &&
        cudaStreamSynchronize(c->st) == cudaSuccess)
      same = d == 0;
    c->launches += ok ? 10 : 0;
  }
  c->twin_s1 = sa;
  c->twin_s2 = sb;
  c->twin_v1 = A.version;
  c->twin_v2 = B.version;
  c->twin_same = same;
  return same;
}

// Whether a box cross term counts as a twin job: the fast engine on every
// outer row (no row sample), coordinates 6, a corel whose other order differs
// only in the fields FieldMap::a lists (density_density, shape_shape), a Pi
// binning symmetric about 0 and twin slots.  Symmetric: the exact thresholds
// satisfy |thr[k] + thr[npi - k]| <= 2^-24 |thr| + 1e-13 L (the reference's
// floor((Pi - p_min) / p_size) leaves them a few ulps from exact symmetry),
// a quarter of the guard of the fast path's Pi bands at most, so the other
// order of every pair the fast path bins has Pi bin npi - 1 - bin.
bool twin_job(cpc_ctx *c, const JobRule &rule, int s1, int s2, int64_t rs, int64_t ro,
              int auto_mode) {
  const cpc_params &p = c->p;
  if (!c->twin_on || auto_mode || rs > 1 || ro != 0 || p.coordinates != 6) return false;
  if (rule.corel != COREL_DD && rule.corel != COREL_SS && rule.corel != COREL_SSA) return false;
  const int npi = p.n_p_bin;
  if (npi < 1 || npi > kMaxPi) return false;
  const double tol_abs = 1e-13 * p.periodic_box_size;
  for (int k = 0; k <= npi; k++) {
    const double a = c->thr_pi[k], b = c->thr_pi[npi - k];
    if (!(std::fabs(a + b) <= std::ldexp(1.0, -24) * std::max(std::fabs(a), std::fabs(b)) + tol_abs))
      return false;
  }
  return slots_twin(c, s1, s2);
}

// Constants of the mixed-precision path of a box job (BoxConst): error bounds of
// the float separations (ea: the absolute error of a coordinate difference, from
// positions that are not float32 values or image shifts that round) against the
// reference's double values.
void box_consts(const cpc_ctx *c, const Slot &g1, const Slot &g2, JobDev &J) {
  const cpc_params &p = c->p;
  const int nrp = p.n_bins, npi = p.n_p_bin;
  const bool rmu = p.coordinates == 7;
  const double L = p.periodic_box_size, eps = std::ldexp(1.0, -24);
  const double ea = eps_abs(c, g1, g2);
  const double z0 = J.wz_lo, z1 = J.wz_hi, zm = std::max(std::fabs(z0), std::fabs(z1));
  const double dtiny = 1e-12 * (L + std::max({p.bin_r_max, z1, -z0}));
  BoxConst &K = J.bc;
  // window: one rounding per difference, one of xyc - m or zh - |dz|, those of
  // the bounds, and of z1 + zc where the z window is not symmetric; doubled
  const double z_mid = 0.5 * (z0 + z1), cmax = std::max({g1.cmax, g2.cmax, L});
  // (a window symmetric but for rounding is taken as symmetric)
  const double zc = std::fabs(z_mid) <= std::ldexp(zm, -20) ? 0.0 : z_mid;
  K.xyc = (float)p.bin_r_max;
  K.zc = (float)zc;
  K.zh = (float)(0.5 * (z1 - z0));
  K.guard = f_up(2 * (ea + 4 * eps * std::max(p.bin_r_max, zm) +
                      (zc != 0 ? ulpf(cmax + std::fabs(zc)) : std::fabs(z_mid)) + dtiny));
  // r^2: each squared difference within (2 eps + 2 ea / r) of its share, two more
  // roundings; relative 2^-21 and twice the absolute part
  const double nterm = rmu ? 3.0 : 2.0;
  auto gr = [&](double T) {
    return 8 * eps * T * T + 2.0 * std::sqrt(nterm) * T * ea + nterm * ea * ea + 1e-12 * T * T;
  };
  const double lo = c->thr_rp[0], hi = c->thr_rp[nrp];
  K.rej_lo = f_down(lo * lo - gr(lo));
  K.rej_hi = f_up(hi * hi + gr(hi));
  auto certain = [](double E) { return E < 0.5 ? f_down(0.5 - E) : -1.0f; };
  {
    const double s = 1.0 / c->ps, o = -p.p_min * s - 0.5;
    const double map = 3 * eps * (npi + std::fabs(o) + 1) + 1e-9;  // roundings of the map
    K.pi_s = (float)s;
    K.pi_o = (float)o;
    K.pi_abs = 0.0f;
    if (!rmu) {
      K.pi_in = certain((2 * eps * zm + 2 * ea + dtiny) * s + map);
    } else {  // mu = dz / r, |mu| <= 1: relative 2^-21 (rsqrtf 2 ulp) and 3 ea / r
      const double tmax = std::max({1.0, std::fabs(p.p_min), std::fabs(p.p_max)});
      K.pi_in = certain(8 * eps * tmax * s + map);
      K.pi_abs = f_up((4 * ea * tmax + dtiny + 1e-30) * s);
    }
  }
  {
    double E, o;
    K.rp_abs = 0.0f;
    if (p.lin_bin) {
      const double s = 1.0 / c->rsize;
      o = -p.bin_r_min * s - 0.5;
      K.rp_s = (float)s;
      E = (6 * eps * p.bin_r_max + std::sqrt(nterm) * 2 * ea + dtiny) * s +
          4 * eps * (nrp + std::fabs(o) + p.bin_r_max * s + 1) + 1e-7;
    } else {
      const double s = nrp / (2.0 * std::log2(p.bin_r_max / p.bin_r_min));
      const double l0 = 2.0 * std::log2(p.bin_r_min);
      const double lm = std::max(std::fabs(l0), std::fabs(2.0 * std::log2(p.bin_r_max)));
      o = -l0 * s - 0.5;
      K.rp_s = (float)s;
      // log2 r^2: relative 8 eps of r^2; __log2f within 2 ulp (2^-21.4 near 1)
      E = s * (8 * eps / M_LN2 + std::max(4 * eps * lm, 8e-7) + 2 * eps * lm) +
          3 * eps * (nrp + std::fabs(o) + 1) + 1e-7;
      K.rp_abs = f_up(s * 1.01 * (2 * std::sqrt(nterm) * ea + 1e-30) / M_LN2 * 1.05);
      if (!(ea > 0)) K.rp_abs = 0.0f;
      // the exact thresholds must be the edges of this map
      for (int k = 0; k <= nrp; k++)
        if (!(std::fabs((2.0 * std::log2(c->thr_rp[k]) - l0) * s - k) < 1e-7)) E = 1.0;
    }
    K.rp_o = (float)o;
    K.rp_in = certain(E);
  }
}

// Model of the kernel's time, by which a job's cell width, kernel variant and the
// z extent of its chunks of rows are chosen.  Per row of a chunk of r rows (of
// lam rows per unit of z): r / 32 + 1/4 rounds of lanes over r on each candidate of the
// chunk's z range, kap of them per unit of z (the quarter is the staging and the
// lanes left idle); four rounds of 32 lanes per 32 pairs that bin; and each unit's set-up
// and flush, about 500 such rounds of a 256-thread block.  With fewer units than
// the GPU holds blocks, blocks wait.
// Measured against fixed rules (the smallest blocks of at least 11 bins, chunks of
// half the window or a quarter of the z range, k = 2 but for sparse tiles) over
// drawn boxes: the kernel with fixed rules 1.38 times as fast as before it was
// rewritten, with the model 1.7 to 1.9; kappa of 20,000 rows in 288 buckets 0.86 ->
// 0.17 ms, a batch of w++ boxes of up to 9,000 rows 4.0 -> 1.3; the 200k wg+ box,
// whose tiles are full either way, 13.8 -> 13.5.
// The model sees the catalogues, the binning and a fixed number of SMs (a GB300's),
// never the device: contexts that count shards of the same pairs (cpc_set_shard)
// must cut them into the same units.
constexpr int kModelSMs = 152;
struct ChunkModel {
  double kap, heavy, zw, ps, n, slots, unit, scale;
  int npi, wpi;
  bool rmu, narrow;
  ChunkModel(const cpc_ctx *c, double n1, double n2, double cell, int twin, int variant, int w) {
    const cpc_params &p = c->p;
    const double L = p.periodic_box_size, r = p.bin_r_max, d = n2 / (L * L * L);
    const double side = std::min(L, 2 * r + 2 * cell);
    zw = wz_hi(p) - (twin ? 0.0 : wz_lo(p));
    kap = d * side * side;
    heavy = 4.0 / 32 * d * M_PI * r * r * zw;
    ps = c->ps;
    n = n1;
    npi = p.n_p_bin;
    wpi = w;
    rmu = p.coordinates == 7;
    narrow = !rmu && wpi < npi;
    slots = (double)kModelSMs * fast_variant_blocks(variant);
    unit = 500.0 * 4 / fast_variant_blocks(variant);
    scale = variant == 1 ? 1.0 : variant == 2 ? 1.05 : 1.1;  // wider blocks wait for one another
  }
  // Pi range that the pairs of a narrow unit may cover: it starts anywhere in the
  // window's first bin and ends anywhere in its last.
  double window() const { return (wpi - 2) * ps; }
  double cost(double lam, double *extent = nullptr) const {
    double best = INFINITY;
    for (const double f : {0.125, 0.1875, 0.25, 0.375, 0.5, 0.625, 0.75}) {
      const double E = narrow ? std::min({f * window(), window() - ps, zw}) : f * zw;
      const double r0 = std::max(1.0, lam * E), r = r0 / std::ceil(r0 / kTileThreads);
      const double units =
          narrow ? std::max(1.0, (zw + E) / std::max(ps, window() - E)) : 1.0;
      const double t = kap * (zw + E) * (1.0 / 32 + 0.25 / r) + heavy + unit * units / r;
      const double slices = rmu ? std::ceil((double)npi / wpi) : 1.0;  // all of it, per mu slice
      const double idle = slots / std::max(1.0, n / r * units * slices);
      const double total = scale * t * slices * std::max(1 + 0.2 * idle, idle);
      if (total < best) {
        best = total;
        if (extent) *extent = E;
      }
    }
    return best;
  }
};

// Smallest window (coordinates 7: any mu slice): what always fits a block.
int min_window(const cpc_params &p, int twin) { return p.coordinates == 7 ? 1 : twin ? 5 : 8; }

struct Variant {
  int variant = 0, wpi = 0;  // 0: the smallest window fits no variant's share of an SM
  double cost = 0;
};
// The variant for a job of n1 x n2 rows: of the widest window that each holds,
// the one the model finds fastest.
Variant choose_variant(const cpc_ctx *c, int corel, int auto_mode, int unit_w, int twin, double n1,
                       double n2, double cell, double lam) {
  const cpc_params &p = c->p;
  const int jk = p.do_jk ? 1 : 0, wmin = min_window(p, twin);
  Variant best;
  for (int v = 1; v <= 3; v++) {
    const size_t budget = fast_block_smem(v) - fast_static_smem_bytes(corel, jk, v, twin) - 1024;
    auto bytes = [&](int w) {
      return fast_smem_bytes(corel, jk, p.n_bins, w, auto_mode, unit_w, twin, v);
    };
    // (the bytes are linear in the window)
    const size_t b0 = bytes(0), bin = bytes(1) - b0;
    const int w = std::min(p.n_p_bin, std::max(wmin, budget > b0 ? (int)((budget - b0) / bin) : 0));
    if (bytes(w) > budget || (best.variant && w <= best.wpi)) continue;
    const double t = ChunkModel(c, n1, n2, cell, twin, v, w).cost(lam);
    if (!best.variant || t < best.cost) best = Variant{v, w, t};
  }
  return best;
}

// Cell width (r_max / k) when none is set, from the largest catalogue of the
// context (or the n rows of an upload), so that every count of the context uses
// one width and a catalogue is rebuilt at most when a larger one comes: 2, or 1
// where the model finds it as fast within a tenth, with the rows spread evenly
// over the columns and jackknife cubes (k = 1 quadruples a bucket's rows, for
// 16 / 9 of the candidates).  Measured, k = 1 over 2: wgg of 20,000 points 0.71, 12
// boxes of L = 3.3 r_max 1.0, w++ boxes of 9,000 rows 0.5; 200k wg+ box 1.07, ED 1.14.
int preferred_cells(cpc_ctx *c, int64_t n = 0) {
  const cpc_params &p = c->p;
  for (const Slot &s : c->slots)
    if (s.valid && !s.sky) n = std::max(n, s.n);
  if (c->pref_n == n) return c->pref_k;
  const double L = p.periodic_box_size;
  const int corel = p.which_corr < 3 ? COREL_DD + p.which_corr : COREL_DK + (p.which_corr - 3);
  auto cost = [&](int k) {
    const double cols = std::max(1.0, std::floor(L / (p.bin_r_max / k)));
    const double cuts = cols + (p.do_jk ? std::cbrt((double)p.n_jk) - 1 : 0);
    return choose_variant(c, corel, 0, 0, 0, (double)n, (double)n, L / cols, n / (cuts * cuts * L)).cost;
  };
  c->pref_n = n;
  c->pref_k = cost(1) < 1.1 * cost(2) ? 1 : 2;
  return c->pref_k;
}

// The automatic cell width.  Of a context that counts shards it is r_max / 2,
// whatever the context holds: the units that the shards share out are those of the
// cell lists, and each shard's context may hold other catalogues beside the counted
// ones.  (Shards pay for large catalogues, which take r_max / 2 anyway.)
int automatic_cells(cpc_ctx *c, int64_t n = 0) {
  return c->n_shards > 1 ? 2 : preferred_cells(c, n);
}

cpc_status rebuild_cells(cpc_ctx *c, Slot &s, int k);

// The box catalogues in these slots on one grid: where their widths differ, that of
// the context's present setting, which they then keep, so that no two counts rebuild
// a slot in turn (results do not depend on it).
cpc_status same_grid(cpc_ctx *c, const std::vector<int> &slots) {
  bool same = true;
  for (int q : slots) same = same && c->slots[q].kcells == c->slots[slots[0]].kcells;
  if (same) return CPC_OK;
  const int k = c->tune_k > 0 ? c->tune_k : automatic_cells(c);
  for (int q : slots) {
    Slot &s = c->slots[q];
    if (!s.valid || s.sky) continue;
    const cpc_status st = s.kcells == k ? CPC_OK : rebuild_cells(c, s, k);
    if (st != CPC_OK) return st;
    s.auto_k = c->tune_k == 0;
  }
  return CPC_OK;
}

// Every catalogue of automatic width on the width that the context's state asks for
// now: after an upload or a shard, so that no count has to rebuild a list.
cpc_status settle_cells(cpc_ctx *c) {
  for (Slot &s : c->slots) {
    if (!s.valid || s.sky || !s.auto_k || s.kcells == automatic_cells(c)) continue;
    const cpc_status st = rebuild_cells(c, s, automatic_cells(c));
    if (st != CPC_OK) return st;
  }
  return CPC_OK;
}

// allow_twin: false for the cell-list FP64 comparison engine, which counts every
// order and keeps the plain job's window.  one_grid: same_grid was called for every
// job of the context (a batch plans them all before it counts: none may rebuild a
// slot that another one was planned on).
cpc_status plan_job(cpc_ctx *c, cpc_pair_kind kind, int slot_g1, int slot_g2, int64_t rs,
                    int64_t ro, cpc_accum *out, JobPlan &jp, int auto_mode = 0,
                    bool allow_twin = true, bool one_grid = false) {
  if (slot_g1 < 0 || slot_g1 >= kMaxSlots || slot_g2 < 0 || slot_g2 >= kMaxSlots)
    return fail(c, CPC_ERR_INVALID, "slot out of range");
  Slot &A = c->slots[slot_g1], &B = c->slots[slot_g2];
  if (!A.valid || !B.valid) return fail(c, CPC_ERR_STATE, "count before upload");
  if (!out || !out->num || !out->sums) return fail(c, CPC_ERR_INVALID, "null output arrays");
  const cpc_params &p = c->p;
  jp.c = c;
  jp.kind = kind;
  jp.out = out;
  jp.row_stride = rs > 1 ? rs : 1;
  jp.row_offset = ro;
  if ((auto_mode ? job_rule_auto(p, kind, jp.rule) : job_rule(p, kind, A.n, B.n, jp.rule)) != 0)
    return fail(c, CPC_ERR_INVALID, "bad pair kind");
  jp.s1 = jp.rule.swapped ? slot_g2 : slot_g1;
  jp.s2 = jp.rule.swapped ? slot_g1 : slot_g2;
  Slot &g1 = c->slots[jp.s1], &g2 = c->slots[jp.s2];
  if (!one_grid) {
    const cpc_status st = same_grid(c, {jp.s1, jp.s2});
    if (st != CPC_OK) return st;
  }
  if (g1.ncx != g2.ncx || g1.ncy != g2.ncy || g1.n_reg != g2.n_reg)
    return fail(c, CPC_ERR_STATE, "catalogues were uploaded with different cell grids");
  jp.empty = (A.n == 0 || B.n == 0);
  const int nrp = p.n_bins, npi = p.n_p_bin;
  const int jk = p.do_jk ? 1 : 0;
  // block-local Pi window: as many Pi bins as fit a block's shared memory.  With
  // coordinates 7 the mu bins have no locality in z: a block holds every mu bin
  // when they fit (else the units are repeated over slices of wpi mu bins)
  const bool rmu = p.coordinates == 7;
  // twin job: each unordered pair once, both orders added (its block holds the
  // other order's histograms too, so the window is narrower; it covers only
  // the pair order with g2 ahead, whose units span half the Pi range)
  const int twin =
      (allow_twin && !jp.empty && twin_job(c, jp.rule, jp.s1, jp.s2, rs, ro, auto_mode)) ? 1 : 0;
  const int wmin = min_window(p, twin);
  // The kernel variant (block size) and its window.  A window set by
  // cpc_set_tuning takes the smallest blocks whose share of an SM it fits.
  const int uw = unit_weights(g1, g2);
  int wpi = 0, variant = 0;
  if (c->tune_wpi > 0 && !rmu) {
    wpi = std::min(npi, c->tune_wpi);
    auto bytes = [&](int v, int w) {
      return fast_smem_bytes(jp.rule.corel, jk, nrp, w, auto_mode, uw, twin, v);
    };
    auto fixed = [&](int v) { return fast_static_smem_bytes(jp.rule.corel, jk, v, twin); };
    for (variant = 1; variant <= 3; variant++)
      if (bytes(variant, wpi) <= fast_block_smem(variant) - fixed(variant) - 1024) break;
    if (variant > 3) {  // fewer blocks per SM, of the variant with the least staging
      variant = 1;
      // histograms of up to 200 KB are accepted, and narrowed beside the staging
      const size_t room = 227 * 1024 - fixed(1);
      if (fast_window_bytes(jp.rule.corel, jk, nrp, wpi, uw, twin) <= 200 * 1024)
        while (wpi > 1 && bytes(1, wpi) > room) wpi--;
    }
  } else {
    const Variant b = choose_variant(c, jp.rule.corel, auto_mode, uw, twin, (double)g1.n,
                                     (double)g2.n, g1.cw_x, g1.row_density);
    variant = b.variant ? b.variant : 3;  // (else the smallest window in the largest blocks)
    wpi = b.variant ? b.wpi : wmin;
  }
  if (!rmu && wpi < npi && wpi < wmin) wpi = std::min(npi, wmin);
  jp.wpi = wpi;
  jp.variant = variant;
  jp.tile = kTileThreads;

  JobDev &J = jp.jd;
  std::memset(&J, 0, sizeof J);
  fill_views(g1, J.f1, J.d1);
  fill_views(g2, J.f2, J.d2);
  J.corel = jp.rule.corel;
  J.gws = jp.rule.gws;
  J.twin = twin;
  J.which_corr = p.which_corr;
  J.estimator = p.estimator;
  J.do_jk = jk;
  J.n_jk = p.n_jk;
  J.periodic = p.periodic_box ? 1 : 0;
  J.coordinates = p.coordinates;
  J.nrp = nrp;
  J.npi = npi;
  J.wpi = wpi;
  J.lin_bin = p.lin_bin ? 1 : 0;
  J.box_same_keep = 1;  // jk_check_PB (jk.cpp:64-71) for coordinates 6
  J.auto_mode = auto_mode;
  J.has_lo = (g1.exact_f32 && g2.exact_f32) ? 0 : 1;
  J.rmu = rmu ? 1 : 0;
  J.ncx = g1.ncx;
  J.ncy = g1.ncy;
  J.row_stride = jp.row_stride;
  J.row_offset = jp.row_offset;
  const double L = p.periodic_box_size;
  J.L = L;
  J.Lf = (float)L;
  J.rmin = p.bin_r_min;
  J.rmax = p.bin_r_max;
  J.pmin = p.p_min;
  J.pmax = p.p_max;
  J.wz_lo = wz_lo(p);
  J.wz_hi = wz_hi(p);
  J.ps = c->ps;
  J.rsize = c->rsize;
  for (int k = 0; k <= nrp; k++) J.thr[k] = c->thr_rp[k];
  box_consts(c, g1, g2, J);
  // fixed-point scales: field f's terms are rint(v 2^S_f) with
  // |v_f| 2^S_f <= 2^29 / (1 + 2^-12) < 2^29 - 2^17 (see pair_fast.cu); S_f
  // from a bound on |v_f| (emax bounds |e|, so every rotated ellipticity)
  {
    const double wm = std::max(g1.wmax, 1e-30) * std::max(g2.wmax, 1e-30);
    const double em = std::max({g1.emax, g2.emax, 1e-30});
    // |phi - theta| folded (calcs.cpp:97-105): phi = -10 for galaxies read
    // without shapes gives values outside [0, pi/2]
    const double tm = std::max(M_PI / 2, std::max(g1.phimax, g2.phimax) + M_PI);
    const double tm2 = (jp.rule.corel == COREL_SSA) ? 2 * tm : tm;
    double vb[kNF];
    vb[0] = wm;
    vb[1] = vb[3] = wm * em;
    vb[2] = vb[4] = wm * wm * em * em;
    vb[5] = vb[7] = vb[9] = wm * em * em;
    vb[6] = vb[8] = vb[10] = wm * wm * em * em * em * em;
    vb[11] = tm2;
    vb[12] = 2 * tm * tm;
    if (jp.rule.corel == COREL_ED) {  // cos^2 <= |e|^2 <= 3 max|e_k|^2
      vb[11] = std::max(1.0, 3 * em * em);
      vb[12] = vb[11] * vb[11];
    }
    for (int f = 0; f < kNF; f++) {
      const double v = std::max(vb[f] * (1.0 + 1.0 / 4096.0), 1e-30);
      int S = 29 - (int)std::ceil(std::log2(v));
      S = std::min(60, std::max(-60, S));
      J.qscale[f] = (float)std::ldexp(1.0, S);
      J.inv_qscale[f] = std::ldexp(1.0, -S);
    }
  }
  J.unit_w = unit_weights(g1, g2);
  return CPC_OK;
}

// tiles of g1 rows and their units (cached per slot versions and window).  The
// context keeps the lists last used, 8 or those of the `jobs` jobs that the present
// launch has of it: a list goes only when newer ones fill the cache.
const UnitCache &build_units(JobPlan &jp, size_t jobs) {
  cpc_ctx *c = jp.c;
  for (auto it = c->unit_cache.begin(); it != c->unit_cache.end(); ++it) {
    const UnitCache &uc = *it;
    if (uc.s1 == jp.s1 && uc.s2 == jp.s2 && uc.v1 == c->slots[jp.s1].version &&
        uc.v2 == c->slots[jp.s2].version && uc.wpi == jp.wpi && uc.tile == jp.tile &&
        uc.twin == jp.jd.twin && uc.variant == jp.variant) {
      std::rotate(it, it + 1, c->unit_cache.end());
      return c->unit_cache.back();
    }
  }
  while (c->unit_cache.size() >= std::max<size_t>(8, jobs))
    c->unit_cache.erase(c->unit_cache.begin());
  c->unit_cache.emplace_back();
  UnitCache &uc = c->unit_cache.back();
  uc.s1 = jp.s1;
  uc.s2 = jp.s2;
  uc.v1 = c->slots[jp.s1].version;
  uc.v2 = c->slots[jp.s2].version;
  uc.wpi = jp.wpi;
  uc.tile = jp.tile;
  uc.twin = jp.jd.twin;
  uc.variant = jp.variant;
  static std::atomic<uint64_t> next_id{1};
  uc.id = next_id++;
  const cpc_params &p = c->p;
  const Slot &g1 = c->slots[jp.s1];
  const double L = p.periodic_box_size;
  const double ps = c->ps;
  const int npi = p.n_p_bin, wpi = jp.wpi;
  const double cmax = std::max(g1.cmax, L);
  const double ea = eps_abs(c, g1, c->slots[jp.s2]);
  const bool rmu = p.coordinates == 7;
  const double zw0 = wz_lo(p), zw1 = wz_hi(p);
  const double guard = 4 * ulpf(2 * cmax) + 2 * ea + std::ldexp(1.0, -20) * (std::fabs(zw0) + std::fabs(zw1) + p.bin_r_max);
  // chunk extents by the bucket's rows per unit of z, in steps of a quarter octave
  const Slot &g2 = c->slots[jp.s2];
  const ChunkModel model(c, (double)g1.n, (double)g2.n, g1.cw_x, jp.jd.twin, jp.variant, wpi);
  constexpr int kOne = 64;  // entry of one row per z range
  double extents[2 * kOne + 1];
  for (int q = 0; q <= 2 * kOne; q++)
    model.cost(std::exp2(0.25 * (q - kOne)) / model.zw, &extents[q]);
  const int ncx = g1.ncx, ncy = g1.ncy;
  const double inv_cwx = 1.0 / g1.cw_x, inv_cwy = 1.0 / g1.cw_y;
  std::vector<UnitDesc> &units = uc.units;
  units.clear();
  const int nb = (int)g1.h_bk_start.size();
  // buckets are independent: contiguous bucket ranges on the host's cores, each
  // into its own list, concatenated in bucket order (the serial order)
  std::vector<std::vector<UnitDesc>> part_units(64);
  host_parallel(nb, [&](int64_t b_lo, int64_t b_hi, int part) {
    std::vector<UnitDesc> &units = part_units[part];
    for (int b = (int)b_lo; b < (int)b_hi; b++) {
      const int s = g1.h_bk_start[b], e = g1.h_bk_end[b];
      int i = s;
      const double ext = std::max<double>((double)g1.h_pos[e - 1].z - g1.h_pos[s].z, ps);
      const double lq = 4 * std::log2((e - s) / ext * model.zw) + kOne;
      const double extent = extents[(int)std::lrint(std::min(std::max(lq, 0.0), 2.0 * kOne))];
      while (i < e) {
        // z-chunk, dealt round-robin into tiles of <= tile rows
        const float z0 = g1.h_pos[i].z;
        int j = i + 1;
        while (j < e && (double)g1.h_pos[j].z - z0 <= extent) j++;
        float bx0 = INFINITY, bx1 = -INFINITY, by0 = INFINITY, by1 = -INFINITY;
        for (int k = i; k < j; k++) {
          bx0 = std::min(bx0, g1.h_pos[k].x);
          bx1 = std::max(bx1, g1.h_pos[k].x);
          by0 = std::min(by0, g1.h_pos[k].y);
          by1 = std::max(by1, g1.h_pos[k].y);
        }
        const int m = j - i;
        const int nt = (m + jp.tile - 1) / jp.tile;
        const double zt0 = g1.h_pos[i].z, zt1 = g1.h_pos[j - 1].z;
        const double rg = p.bin_r_max + guard;
        int cx0 = (int)std::floor((bx0 - rg) * inv_cwx), cx1 = (int)std::floor((bx1 + rg) * inv_cwx);
        int cy0 = (int)std::floor((by0 - rg) * inv_cwy), cy1 = (int)std::floor((by1 + rg) * inv_cwy);
        if (p.periodic_box) {
          cx0 = std::max(cx0, -ncx); cx1 = std::min(cx1, 2 * ncx - 1);
          cy0 = std::max(cy0, -ncy); cy1 = std::min(cy1, 2 * ncy - 1);
        } else {
          cx0 = std::max(cx0, 0); cx1 = std::min(cx1, ncx - 1);
          cy0 = std::max(cy0, 0); cy1 = std::min(cy1, ncy - 1);
        }
        // twin jobs: only candidates ahead of the rows (Pi >= 0; the other order
        // is added with each pair)
        const double Zlo = zt0 + (jp.jd.twin ? 0.0 : zw0) - guard, Zhi = zt1 + zw1 + guard;
        for (int k = 0; k < nt; k++) {
          UnitDesc u;
          std::memset(&u, 0, sizeof u);
          u.g1_start = i + k;
          u.g1_stride = nt;
          u.g1_count = (m - k + nt - 1) / nt;
          u.region = g1.h_bk_region[b];
          u.cx_lo = cx0; u.cx_hi = cx1; u.cy_lo = cy0; u.cy_hi = cy1;
          int U = 1;
          if (model.narrow)
            U = std::max(1, (int)std::ceil((Zhi - Zlo) /
                                           std::max(ps, model.window() - (zt1 - zt0))));
          // coordinates 7: one unit per slice of wpi mu bins; each pair is taken by
          // the slice holding its bin (pair_fast.cu)
          for (int base = 0; base < (rmu ? npi : 1); base += wpi)
            for (int q = 0; q < U; q++) {
              u.zlo = (q == 0) ? Zlo : Zlo + (Zhi - Zlo) * q / U;
              u.zhi = (q == U - 1) ? Zhi : Zlo + (Zhi - Zlo) * (q + 1) / U;
              u.n2_base = base;
              if (model.narrow)
                u.n2_base = std::max(
                    0, std::min((int)std::floor((u.zlo - zt1 - guard - p.p_min) / ps), npi - wpi));
              units.push_back(u);
            }
        }
        i = j;
      }
    }
  }, 512);  // a bucket's units take microseconds: threads pay for large catalogues
  size_t total = 0;
  for (const auto &v : part_units) total += v.size();
  units.reserve(total);
  for (const auto &v : part_units) units.insert(units.end(), v.begin(), v.end());
  return uc;
}

cpc_status ensure_scratch(cpc_ctx *c, size_t n_units, size_t n_jobs) {
  if (n_units > c->d_units.n) c->units_key.clear();  // the list held goes, even if this fails
  CK(c->d_units.alloc(n_units), "alloc units");
  CK(c->d_jobs.alloc(n_jobs), "alloc jobs");
  CK(c->d_unit_ctr.alloc(1), "alloc counter");
  CK(c->d_qcount.alloc(1), "alloc queue counter");
  if (!c->d_queue.p) {
    c->qcap = CPC_EDGE_QUEUE_INIT;
    // CPC_EDGE_QUEUE_INIT in the environment (a positive entry count) starts the
    // context with another capacity: tests use a small one to drive the overflow
    // path (grow, count again)
    if (const char *ev = std::getenv("CPC_EDGE_QUEUE_INIT")) {
      const long long v = std::atoll(ev);
      if (v > 0) c->qcap = (unsigned long long)v;
    }
    cudaError_t e = c->d_queue.alloc(c->qcap);
    if (e != cudaSuccess) {
      cudaGetLastError();
      c->qcap = 1ull << 20;
      CK(c->d_queue.alloc(c->qcap), "alloc edge queue");
    }
  }
  return CPC_OK;
}

size_t accum_cells(const cpc_ctx *c) {
  const cpc_params &p = c->p;
  return (size_t)(1 + (p.do_jk ? p.n_jk : 0)) * p.n_bins * p.n_p_bin;
}

// The histogram block and counters of a box job: the context's q-th (the jobs of one
// context in a batch have one each)
cpc_status alloc_accum(JobPlan &jp, size_t q) {
  cpc_ctx *c = jp.c;
  const size_t cells = accum_cells(c);
  while (c->accum.size() <= q) c->accum.emplace_back(new AccumBufs());
  AccumBufs &a = *c->accum[q];
  CK(a.num.alloc(cells), "alloc accum");
  CK(a.sums.alloc(cells * kNF), "alloc accum");
  CK(a.counters.alloc(4), "alloc counters");
  jp.jd.acc_num = a.num.p;
  jp.jd.acc_sums = a.sums.p;
  jp.jd.counters = a.counters.p;
  return CPC_OK;
}

cpc_status zero_accum(const JobPlan &jp, cudaStream_t st) {
  cpc_ctx *c = jp.c;
  const size_t cells = accum_cells(c);
  CK(cudaMemsetAsync(jp.jd.acc_num, 0, sizeof(unsigned long long) * cells, st), "memset");
  CK(cudaMemsetAsync(jp.jd.acc_sums, 0, sizeof(double) * cells * kNF, st), "memset");
  CK(cudaMemsetAsync(jp.jd.counters, 0, sizeof(unsigned long long) * 4, st), "memset");
  return CPC_OK;
}

// the histogram block and counters in device buffers num / sums / counters
cpc_status fetch_accum_from(cpc_ctx *c, const unsigned long long *num, const double *sums,
                            const unsigned long long *counters, cpc_accum *out, cudaStream_t st,
                            int unit_w) {
  const cpc_params &p = c->p;
  const size_t n_hist = 1 + (p.do_jk ? p.n_jk : 0);
  const size_t cells = n_hist * p.n_bins * p.n_p_bin;
  unsigned long long cnt[4];
  CK(cudaMemcpyAsync(out->num, num, sizeof(int64_t) * cells, cudaMemcpyDeviceToHost, st), "D2H");
  CK(cudaMemcpyAsync(out->sums, sums, sizeof(double) * cells * kNF, cudaMemcpyDeviceToHost, st), "D2H");
  CK(cudaMemcpyAsync(cnt, counters, sizeof cnt, cudaMemcpyDeviceToHost, st), "D2H");
  CK(cudaStreamSynchronize(st), "sync");
  if (unit_w)
    for (size_t k = 0; k < cells; k++) out->sums[k * kNF] = (double)out->num[k];
  out->n_window = (int64_t)(cnt[0] + cnt[1]);
  out->n_rechecked = (int64_t)cnt[2];
  int64_t nb = 0;
  const size_t c0 = (size_t)p.n_bins * p.n_p_bin;
  for (size_t k = 0; k < c0; k++) nb += out->num[k];
  out->n_binned = nb;
  return CPC_OK;
}

cpc_status fetch_accum(const JobPlan &jp, cudaStream_t st, int unit_w) {
  return fetch_accum_from(jp.c, jp.jd.acc_num, jp.jd.acc_sums, jp.jd.counters, jp.out, st, unit_w);
}

cpc_status build_zorder(cpc_ctx *c, Slot &s) {
  if (s.zbuilt) return CPC_OK;
  const int64_t n = s.n;
  cudaStream_t st = c->st;
  CK(c->d_keys.alloc(n), "alloc");
  CK(c->d_ktmp.alloc(n), "alloc");
  CK(c->d_vals.alloc(n), "alloc");
  CK(c->d_vtmp.alloc(n), "alloc");
  CK(c->d_hist.alloc(radix_hist_words(n)), "alloc");
  CK(c->d_census.alloc(8 * 256), "alloc");
  CK(launch_z_keys(n, s.z.p, c->d_keys.p, c->d_vals.p, st), "z keys");
  CK(radix_sort_pairs(n, c->d_keys.p, c->d_vals.p, c->d_ktmp.p, c->d_vtmp.p, c->d_hist.p,
                      c->d_census.p, st, &c->launches), "z sort");
  c->launches += 2;  // z keys + gather
  CK(s.zx.alloc(n), "alloc"); CK(s.zy.alloc(n), "alloc"); CK(s.zz.alloc(n), "alloc");
  CK(s.zw.alloc(n), "alloc"); CK(s.ze1.alloc(n), "alloc"); CK(s.ze2.alloc(n), "alloc");
  CK(s.zphi.alloc(n), "alloc"); CK(s.zjk.alloc(n), "alloc"); CK(s.zkeep.alloc(n), "alloc");
  CK(s.zorig.alloc(n), "alloc"); CK(s.ze3.alloc(n), "alloc");
  GatherIn in{s.x.p, s.y.p, s.z.p, s.w.p, s.e1.p, s.e2.p, s.phi.p, s.jk.p, s.keep.p, s.e3.p};
  GatherOut out{};
  out.x = s.zx.p; out.y = s.zy.p; out.z = s.zz.p; out.w = s.zw.p;
  out.e1 = s.ze1.p; out.e2 = s.ze2.p; out.phi = s.zphi.p; out.e3 = s.ze3.p; out.jk = s.zjk.p;
  out.keep = s.zkeep.p; out.orig = s.zorig.p; out.orig_in = s.orig.p;
  CK(launch_gather(n, c->d_keys.p, c->d_vals.p, in, out, st), "z gather");
  CK(s.zaflag.alloc(n), "alloc");
  CK(launch_gather_u8(n, c->d_vals.p, s.aflag.p, s.zaflag.p, st), "z gather");
  c->launches += 1;
  CK(cudaStreamSynchronize(st), "sync");
  s.zbuilt = true;
  return CPC_OK;
}

DCat zview(Slot &s) {
  DCat d;
  d.n = s.n;
  d.x = s.zx.p; d.y = s.zy.p; d.z = s.zz.p; d.w = s.zw.p;
  d.e1 = s.ze1.p; d.e2 = s.ze2.p; d.phi = s.zphi.p; d.e3 = s.ze3.p;
  d.jk = s.zjk.p; d.keep = s.zkeep.p; d.orig = s.zorig.p; d.aflag = s.zaflag.p;
  return d;
}

// the plain FP64 kernel: enqueue on the context's stream, then fetch
cpc_status enqueue_plain(JobPlan &jp) {
  cpc_ctx *c = jp.c;
  cpc_status s;
  if ((s = alloc_accum(jp, 0)) != CPC_OK) return s;
  if ((s = zero_accum(jp, c->st)) != CPC_OK) return s;
  CK(cudaEventRecord(c->e0, c->st), "event");
  if (jp.empty) {
    CK(cudaEventRecord(c->e1, c->st), "event");
    return CPC_OK;
  }
  Slot &g1 = c->slots[jp.s1], &g2 = c->slots[jp.s2];
  if ((s = build_zorder(c, g1)) != CPC_OK) return s;
  if ((s = build_zorder(c, g2)) != CPC_OK) return s;
  if ((s = ensure_scratch(c, 1, 1)) != CPC_OK) return s;
  DCat a = zview(g1), b = zview(g2);
  jp.jd.d1 = a;
  jp.jd.d2 = b;
  CK(cudaMemcpyAsync(c->d_jobs.p, &jp.jd, sizeof(JobDev), cudaMemcpyHostToDevice, c->st), "H2D job");
  CK(launch_plain_fp64(c->d_jobs.p, a, b, c->st), "plain fp64 kernel");
  c->launches += 1;
  CK(cudaEventRecord(c->e1, c->st), "event");
  return CPC_OK;
}

cpc_status finish_plain(JobPlan &jp) {
  cpc_ctx *c = jp.c;
  cpc_status s;
  if ((s = fetch_accum(jp, c->st, 0)) != CPC_OK) return s;
  float ms = 0;
  CK(cudaEventElapsedTime(&ms, c->e0, c->e1), "event time");
  jp.out->kernel_ms = ms;
  jp.out->pair_kernel_ms = ms;
  return CPC_OK;
}

cpc_status run_plain(JobPlan &jp) {
  const cpc_status s = enqueue_plain(jp);
  return s != CPC_OK ? s : finish_plain(jp);
}

// fast engine over one or more jobs (one persistent launch per corel group):
// enqueue on the first context's stream, then wait, check the edge queue and
// fetch
cpc_status run_fast(std::vector<JobPlan> &jobs, int grow_attempt = 0);

// one persistent launch of the fast kernel over a range of the unit list
struct FastGroup {
  int corel, jk, variant, grid;
  size_t first, n_units, smem;
  FastScales sc;
  int auto_pairs;  // the group holds corels1 jobs (their rules in shared memory)
  int twin;        // the group's jobs are twin jobs (their own kernel)
};

// The device work of one fast count, in stream order on st: zero every job's
// histogram block and counters, the edge-queue counter, then per group the
// unit counter and the persistent kernel, then the FP64 recheck.  rec_flags
// records the timing events (cudaEventRecordExternal inside a capture, so
// that they become event nodes of the graph).
cpc_status fast_body(cpc_ctx *c0, std::vector<JobPlan> &jobs, const std::vector<FastGroup> &gs,
                     cudaStream_t st, unsigned rec_flags) {
  cpc_ctx *c = c0;
  for (size_t k = 0; k < jobs.size(); k++) {
    const cpc_status s = zero_accum(jobs[k], st);
    if (s != CPC_OK) return s;
  }
  CK(cudaMemsetAsync(c0->d_qcount.p, 0, sizeof(unsigned long long), st), "memset");
  CK(cudaEventRecordWithFlags(c0->e0, st, rec_flags), "event");
  for (const FastGroup &g : gs) {
    CK(cudaMemsetAsync(c0->d_unit_ctr.p, 0, sizeof(unsigned int), st), "memset");
    CK(launch_fast(g.corel, g.jk, g.variant, g.twin, c0->d_jobs.p, c0->d_units.p + g.first,
                   (int)g.n_units,
                   c0->d_unit_ctr.p, c0->d_queue.p, c0->d_qcount.p, c0->qcap, g.sc, g.smem,
                   g.grid, g.auto_pairs, st),
       "fast kernel");
  }
  CK(cudaEventRecordWithFlags(c0->e2, st, rec_flags), "event");
  CK(launch_recheck(c0->d_jobs.p, c0->d_queue.p, c0->d_qcount.p, c0->qcap, c0->sm_count * 8, st),
     "recheck kernel");
  CK(cudaEventRecordWithFlags(c0->e1, st, rec_flags), "event");
  return CPC_OK;
}

// Everything fast_body bakes into its launches: buffer addresses and sizes,
// queue capacity, and each group's kernel, unit range, grid and shared memory.
std::vector<uint64_t> fast_graph_key(cpc_ctx *c0, const std::vector<JobPlan> &jobs,
                                     const std::vector<FastGroup> &gs) {
  std::vector<uint64_t> k;
  auto put = [&](uint64_t v) { k.push_back(v); };
  put((uint64_t)(uintptr_t)c0->st);
  put((uint64_t)(uintptr_t)c0->d_jobs.p);
  put((uint64_t)(uintptr_t)c0->d_units.p);
  put((uint64_t)(uintptr_t)c0->d_unit_ctr.p);
  put((uint64_t)(uintptr_t)c0->d_queue.p);
  put((uint64_t)(uintptr_t)c0->d_qcount.p);
  put(c0->qcap);
  put((uint64_t)c0->sm_count);
  put(jobs.size());
  for (const JobPlan &jp : jobs) {
    put((uint64_t)(uintptr_t)jp.jd.acc_num);
    put((uint64_t)(uintptr_t)jp.jd.acc_sums);
    put((uint64_t)(uintptr_t)jp.jd.counters);
    put(accum_cells(jp.c));
  }
  put(gs.size());
  for (const FastGroup &g : gs) {
    put((uint64_t)g.corel);
    put((uint64_t)g.jk);
    put((uint64_t)g.variant);
    put((uint64_t)g.grid);
    put(g.first);
    put(g.n_units);
    put(g.smem);
    put((uint64_t)g.auto_pairs);
    put((uint64_t)g.twin);
    for (int f = 0; f < kNF; f++) {  // the scales are kernel parameters too
      uint32_t b;
      std::memcpy(&b, &g.sc.qs[f], sizeof b);
      put(b);
    }
  }
  return k;
}

void drop_graph(cpc_ctx *c) {
  if (c->gexec) cudaGraphExecDestroy(c->gexec);
  c->gexec = nullptr;
  c->gkey.clear();
}

// Launch the fast count's device work: replay the context's graph when it was
// captured for the same key, else capture it anew (or launch directly when
// graphs are off or the capture fails, which turns graphs off for the context).
cpc_status launch_fast_body(cpc_ctx *c0, std::vector<JobPlan> &jobs,
                            const std::vector<FastGroup> &gs) {
  cpc_ctx *c = c0;
  cudaStream_t st = c0->st;
  const int64_t n_launch = (int64_t)gs.size() + 1;
  if (!c0->graph_on) {
    const cpc_status s = fast_body(c0, jobs, gs, st, cudaEventRecordDefault);
    if (s == CPC_OK) c0->launches += n_launch;
    return s;
  }
  std::vector<uint64_t> key = fast_graph_key(c0, jobs, gs);
  if (!c0->gexec || key != c0->gkey) {
    drop_graph(c0);
    cudaGraph_t g = nullptr;
    CK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal), "begin capture");
    const cpc_status s = fast_body(c0, jobs, gs, st, cudaEventRecordExternal);
    const cudaError_t e_end = cudaStreamEndCapture(st, &g);
    cudaGraphExec_t ex = nullptr;
    cudaError_t e_inst = cudaErrorUnknown;
    if (s == CPC_OK && e_end == cudaSuccess && g) e_inst = cudaGraphInstantiate(&ex, g, 0);
    if (g) cudaGraphDestroy(g);
    if (s != CPC_OK || e_end != cudaSuccess || e_inst != cudaSuccess) {
      // capture unavailable here: direct launches from now on
      cudaGetLastError();
      if (ex) cudaGraphExecDestroy(ex);
      c0->graph_on = 0;
      const cpc_status s2 = fast_body(c0, jobs, gs, st, cudaEventRecordDefault);
      if (s2 == CPC_OK) c0->launches += n_launch;
      return s2;
    }
    c0->gexec = ex;
    c0->gkey = std::move(key);
    c0->graph_captures++;
  }
  CK(cudaGraphLaunch(c0->gexec, st), "graph launch");
  c0->graph_replays++;
  c0->launches += n_launch;
  return CPC_OK;
}

cpc_status enqueue_fast(std::vector<JobPlan> &jobs) {
  cpc_ctx *c0 = jobs[0].c;
  cpc_ctx *c = c0;
  cudaStream_t st = c0->st;
  std::map<cpc_ctx *, size_t> n_of;  // jobs of each context so far
  for (JobPlan &jp : jobs) {
    const cpc_status s = alloc_accum(jp, n_of[jp.c]++);
    if (s != CPC_OK) return s;
  }
  // group by kernel instantiation: corel, jackknife, twin, variant
  using Inst = std::tuple<int, int, int, int>;
  std::map<Inst, std::vector<int>> groups;
  for (size_t k = 0; k < jobs.size(); k++)
    if (!jobs[k].empty)
      groups[Inst(jobs[k].jd.corel, jobs[k].jd.do_jk, jobs[k].jd.twin,
                  jobs[k].jd.all_exact ? 0 : jobs[k].variant)].push_back((int)k);
  // the launches' unit ranges, and what identifies the list that they make up: a
  // context that counts the same pairs again finds it on the device (copying the
  // units of the 2M w++ box took 6 ms a call, of the 200k wg+ box 0.5 of 14.3)
  size_t total_units = 0;
  std::vector<std::pair<size_t, size_t>> ranges;
  std::vector<Inst> gkeys;
  std::vector<std::vector<int>> members;
  std::vector<uint64_t> key;
  for (auto &g : groups) {
    const size_t b = total_units;
    for (int k : g.second) {
      const UnitCache &uc = build_units(jobs[k], n_of[jobs[k].c]);
      // this context's shard of the units (cpc_set_shard): every n_shards-th
      // unit from `shard`; the units partition the pairs, so the shards' blocks
      // sum to the whole count
      const size_t nsh = (size_t)jobs[k].c->n_shards, sh = (size_t)jobs[k].c->shard;
      key.insert(key.end(), {uc.id, (uint64_t)k, nsh, sh});
      total_units += uc.units.size() > sh ? (uc.units.size() - sh + nsh - 1) / nsh : 0;
    }
    ranges.push_back({b, total_units});
    gkeys.push_back(g.first);
    members.push_back(g.second);
  }
  cpc_status s;
  if ((s = ensure_scratch(c0, std::max<size_t>(1, total_units), jobs.size())) != CPC_OK) return s;
  if (key != c0->units_key) {
    c0->units_key.clear();
    std::vector<UnitDesc> all;
    all.reserve(total_units);
    for (const auto &m : members)
      for (int k : m) {
        const std::vector<UnitDesc> &u = build_units(jobs[k], n_of[jobs[k].c]).units;
        const size_t nsh = (size_t)jobs[k].c->n_shards;
        for (size_t ui = (size_t)jobs[k].c->shard; ui < u.size(); ui += nsh) {
          UnitDesc d = u[ui];
          d.job = k;
          const int64_t ncol = (int64_t)(d.cx_hi - d.cx_lo + 1) * (d.cy_hi - d.cy_lo + 1);
          if (ncol < 1 || ncol > kFastMaxCols || d.g1_count < 1 || d.g1_count > kTileThreads)
            return fail(c, CPC_ERR_INVALID, "work unit outside kernel limits (too many neighbour columns)");
          all.push_back(d);
        }
      }
    if (total_units)
      CK(cudaMemcpyAsync(c0->d_units.p, all.data(), sizeof(UnitDesc) * total_units,
                         cudaMemcpyHostToDevice, st), "H2D units");
    c0->units_key = std::move(key);
  }
  // size the edge queue from the rate earlier counts of this context queued
  // (per unit): a count whose queue overflows is run again, which a full count
  // after sharded or sampled ones would otherwise pay
  {
    const double need = c0->q_per_unit * (double)total_units * 1.25;
    if (need > (double)c0->qcap && need < 4e9) {
      unsigned long long cap = c0->qcap;
      while ((double)cap < need) cap *= 2;
      c0->d_queue.reset();
      CK(c0->d_queue.alloc(cap), "alloc edge queue");
      c0->qcap = cap;
    }
  }
  c0->last_units = total_units;
  c0->last_twin = 0;
  for (const JobPlan &jp : jobs) c0->last_twin |= jp.jd.twin;
  std::vector<JobDev> jds(jobs.size());
  for (size_t k = 0; k < jobs.size(); k++) jds[k] = jobs[k].jd;
  CK(cudaMemcpyAsync(c0->d_jobs.p, jds.data(), sizeof(JobDev) * jds.size(), cudaMemcpyHostToDevice, st), "H2D jobs");
  std::vector<FastGroup> gs;
  for (size_t g = 0; g < ranges.size(); g++) {
    const int corel = std::get<0>(gkeys[g]), jk = std::get<1>(gkeys[g]), twin = std::get<2>(gkeys[g]),
              variant = std::get<3>(gkeys[g]);
    size_t smem = 0;  // the largest any job of the group needs
    FastScales sc;    // per field the smallest scale of the group's jobs
    int auto_pairs = 0;
    for (int f = 0; f < kNF; f++) {
      sc.qs[f] = INFINITY;
      sc.iqs[f] = 0.0;
    }
    for (int k : members[g]) auto_pairs |= jobs[k].jd.auto_mode ? 1 : 0;
    for (int k : members[g]) {
      const JobPlan &jp = jobs[k];
      smem = std::max(smem, fast_smem_bytes(corel, jk, jp.jd.nrp, jp.wpi, auto_pairs,
                                            jp.jd.unit_w, jp.jd.twin, variant));
      for (int f = 0; f < kNF; f++)
        if (jp.jd.qscale[f] < sc.qs[f]) {
          sc.qs[f] = jp.jd.qscale[f];
          sc.iqs[f] = jp.jd.inv_qscale[f];
        }
    }
    const size_t n_units = ranges[g].second - ranges[g].first;
    if (n_units == 0) continue;
    const int bps = fast_blocks(corel, jk, variant, smem, twin);
    if (bps <= 0) return fail(c, CPC_ERR_INVALID, "fast kernel does not fit on an SM with these bins");
    const int grid = (int)std::min<int64_t>((int64_t)c0->sm_count * bps, (int64_t)n_units);
    gs.push_back(
        FastGroup{corel, jk, variant, grid, ranges[g].first, n_units, smem, sc, auto_pairs, twin});
  }
  return launch_fast_body(c0, jobs, gs);
}

cpc_status finish_fast(std::vector<JobPlan> &jobs, int grow_attempt) {
  cpc_ctx *c0 = jobs[0].c;
  cpc_ctx *c = c0;
  cudaStream_t st = c0->st;
  cpc_status s;
  CK(cudaStreamSynchronize(st), "fast kernels");
  float ms = 0, pms = 0;
  CK(cudaEventElapsedTime(&ms, c0->e0, c0->e1), "event time");
  CK(cudaEventElapsedTime(&pms, c0->e0, c0->e2), "event time");
  unsigned long long qn = 0;
  CK(cudaMemcpy(&qn, c0->d_qcount.p, sizeof qn, cudaMemcpyDeviceToHost), "D2H");
  if (c0->last_units > 0 && !jobs[0].jd.all_exact)  // (the FP64 comparison queues every pair)
    c0->q_per_unit = std::max(c0->q_per_unit, (double)qn / (double)c0->last_units);
  if (qn > c0->qcap) {
    // the edge queue overflowed: grow it to hold every queued pair and count
    // again (the queued set does not depend on the order of execution)
    if (grow_attempt) return fail(c, CPC_ERR_NOMEM, "edge queue overflow after growing it");
    unsigned long long cap = c0->qcap;
    while (cap < qn) cap *= 2;
    c0->d_queue.reset();
    CK(c0->d_queue.alloc(cap), "alloc edge queue");
    c0->qcap = cap;
    return run_fast(jobs, 1);
  }
  for (size_t k = 0; k < jobs.size(); k++) {
    if ((s = fetch_accum(jobs[k], st, jobs[k].jd.unit_w)) != CPC_OK) return s;
    jobs[k].out->kernel_ms = ms;
    jobs[k].out->pair_kernel_ms = pms;
  }
  return CPC_OK;
}

cpc_status run_fast(std::vector<JobPlan> &jobs, int grow_attempt) {
  const cpc_status s = enqueue_fast(jobs);
  return s != CPC_OK ? s : finish_fast(jobs, grow_attempt);
}

// Cell list of slot s from a catalogue held in the context's upload buffers
// (u_x .. u_flag; orig_in maps their rows to input rows, null = identity):
// grid of columns r_max / k wide, keys, radix sort, gather into the slot, the
// bucket and column tables.  check_stats: the upload's device checks must pass.
cpc_status build_cells(cpc_ctx *c, Slot &s, int64_t n, int k, const int64_t *orig_in,
                       bool check_stats) {
  const cpc_params &p = c->p;
  const double L = p.periodic_box_size;
  const size_t nn = std::max<int64_t>(n, 1);
  cudaStream_t st = c->st;
  DevBuf<double> &ox = c->u_x, &oy = c->u_y, &oz = c->u_z, &ow = c->u_w, &oe1 = c->u_e1,
                 &oe2 = c->u_e2, &ophi = c->u_phi, &oe3 = c->u_e3;
  DevBuf<int32_t> &ojk = c->u_jk;
  DevBuf<uint8_t> &okeep = c->u_keep, &oflag = c->u_flag;
  // grid: columns of width >= r_max / k over [0, box)
  int nc = (int)std::floor(L / (p.bin_r_max / k));
  nc = std::max(1, std::min(nc, 2048));
  s.ncx = s.ncy = nc;
  s.cw_x = s.cw_y = L / nc;
  s.kcells = k;
  s.n_reg = p.do_jk ? p.n_jk : 1;
  if ((double)nc * nc * s.n_reg >= 4294967295.0) return fail(c, CPC_ERR_INVALID, "too many cell buckets");
  CK(c->d_keys.alloc(nn), "alloc"); CK(c->d_ktmp.alloc(nn), "alloc");
  CK(c->d_vals.alloc(nn), "alloc"); CK(c->d_vtmp.alloc(nn), "alloc");
  CK(c->d_hist.alloc(radix_hist_words(nn)), "alloc");
  CK(c->d_census.alloc(8 * 256), "alloc");
  CK(c->d_bucket.alloc(nn), "alloc");
  CK(s.pos.alloc(nn), "alloc"); CK(s.shp.alloc(nn), "alloc"); CK(s.zf.alloc(nn), "alloc");
  CK(s.ewt.alloc(nn), "alloc"); CK(s.aux.alloc(nn), "alloc"); CK(s.zlo.alloc(nn), "alloc"); CK(s.e3.alloc(nn), "alloc");
  CK(s.x.alloc(nn), "alloc"); CK(s.y.alloc(nn), "alloc"); CK(s.z.alloc(nn), "alloc");
  CK(s.w.alloc(nn), "alloc"); CK(s.e1.alloc(nn), "alloc"); CK(s.e2.alloc(nn), "alloc");
  CK(s.phi.alloc(nn), "alloc"); CK(s.jk.alloc(nn), "alloc"); CK(s.keep.alloc(nn), "alloc");
  CK(s.orig.alloc(nn), "alloc");
  CK(launch_cell_keys(n, ox.p, oy.p, oz.p, ojk.p, 1.0 / s.cw_x, 1.0 / s.cw_y, s.ncx, s.ncy, s.n_reg,
                      c->d_keys.p, c->d_vals.p, st), "cell keys");
  CK(radix_sort_pairs(n, c->d_keys.p, c->d_vals.p, c->d_ktmp.p, c->d_vtmp.p, c->d_hist.p,
                      c->d_census.p, st, &c->launches), "radix sort");
  if (n > 0) c->launches += 2;  // cell keys + gather
  GatherIn in{ox.p, oy.p, oz.p, ow.p, oe1.p, oe2.p, ophi.p, ojk.p, okeep.p, oe3.p};
  GatherOut go{};
  go.pos = s.pos.p; go.shp = s.shp.p; go.ewt = s.ewt.p; go.aux = s.aux.p; go.zlo = s.zlo.p; go.zf = s.zf.p;
  go.bucket = c->d_bucket.p;
  go.x = s.x.p; go.y = s.y.p; go.z = s.z.p; go.w = s.w.p; go.e1 = s.e1.p; go.e2 = s.e2.p;
  go.e3 = s.e3.p;
  go.phi = s.phi.p; go.jk = s.jk.p; go.keep = s.keep.p; go.orig = s.orig.p; go.orig_in = orig_in;
  CK(launch_gather(n, c->d_keys.p, c->d_vals.p, in, go, st), "gather");
  CK(s.aflag.alloc(nn), "alloc");
  if (n > 0) {
    CK(launch_gather_u8(n, c->d_vals.p, oflag.p, s.aflag.p, st), "gather");
    c->launches += 1;
  }
  // buckets on the host
  std::vector<uint32_t> hb(n);
  s.h_pos.resize(n);
  if (n > 0) {
    CK(cudaMemcpyAsync(hb.data(), c->d_bucket.p, 4 * n, cudaMemcpyDeviceToHost, st), "D2H");
    CK(cudaMemcpyAsync(s.h_pos.data(), s.pos.p, sizeof(float4) * n, cudaMemcpyDeviceToHost, st), "D2H");
  }
  CK(cudaStreamSynchronize(st), "upload");
  if (check_stats) {  // the device checks (first failing row of each kind) and statistics
    const UploadStats &u = c->h_ustats;
    static const char *what[4] = {"non-finite position", "position outside [0, box_size]",
                                  "non-finite weight, ellipticity or phi",
                                  "jackknife label out of range"};
    int kind = -1;
    for (int q = 0; q < 4; q++)
      if (u.bad_row[q] != ~0ull && (kind < 0 || u.bad_row[q] < u.bad_row[kind])) kind = q;
    if (kind >= 0)
      return fail(c, CPC_ERR_RANGE,
                  std::string(what[kind]) + " at row " + std::to_string(u.bad_row[kind]));
    double v;
    std::memcpy(&v, &u.cmax_bits, 8); s.cmax = v;
    std::memcpy(&v, &u.wmax_bits, 8); s.wmax = v;
    std::memcpy(&v, &u.emax_bits, 8); s.emax = v;
    std::memcpy(&v, &u.phimax_bits, 8); s.phimax = v;
    s.wmin = n > 0 ? from_orderable_key(u.wmin_key) : 1.0;
    s.exact_f32 = u.not_f32 == 0;
  }
  s.h_bk_start.clear(); s.h_bk_end.clear(); s.h_bk_region.clear();
  std::vector<float> bz0, bz1;
  const int ncol = s.ncx * s.ncy;
  std::vector<int> cb(ncol, 0), ce(ncol, 0);
  // bucket starts (rows whose key differs from the previous row's), found in
  // chunks on the host's cores and concatenated in row order
  std::vector<std::vector<int64_t>> part_starts(64);
  host_parallel(n, [&](int64_t b0, int64_t b1, int part) {
    for (int64_t i = b0; i < b1; i++)
      if (i == 0 || hb[i] != hb[i - 1]) part_starts[part].push_back(i);
  }, 1 << 20);  // a cheap pass: threads only pay for millions of rows
  std::vector<int64_t> starts;
  for (const auto &v : part_starts) starts.insert(starts.end(), v.begin(), v.end());
  for (size_t q = 0; q < starts.size(); q++) {
    const int64_t i = starts[q], j = q + 1 < starts.size() ? starts[q + 1] : n;
    const int b = (int)s.h_bk_start.size();
    const int col = (int)(hb[i] / s.n_reg), reg = (int)(hb[i] % s.n_reg);
    if (ce[col] == 0 && cb[col] == 0) cb[col] = b;
    ce[col] = b + 1;
    s.h_bk_start.push_back((int)i);
    s.h_bk_end.push_back((int)j);
    s.h_bk_region.push_back(reg);
    bz0.push_back(s.h_pos[i].z);
    bz1.push_back(s.h_pos[j - 1].z);
  }
  // columns with no bucket: empty range
  for (int q = 0; q < ncol; q++)
    if (ce[q] == 0) cb[q] = 0;
  const size_t nbk = std::max<size_t>(1, s.h_bk_start.size());
  CK(s.bk_start.alloc(nbk), "alloc"); CK(s.bk_end.alloc(nbk), "alloc");
  CK(s.bk_region.alloc(nbk), "alloc"); CK(s.bk_zmin.alloc(nbk), "alloc");
  CK(s.bk_zmax.alloc(nbk), "alloc"); CK(s.col_begin.alloc(ncol), "alloc");
  CK(s.col_end.alloc(ncol), "alloc");
  const size_t nb = s.h_bk_start.size();
  if (nb) {
    CK(cudaMemcpyAsync(s.bk_start.p, s.h_bk_start.data(), 4 * nb, cudaMemcpyHostToDevice, st), "H2D");
    CK(cudaMemcpyAsync(s.bk_end.p, s.h_bk_end.data(), 4 * nb, cudaMemcpyHostToDevice, st), "H2D");
    CK(cudaMemcpyAsync(s.bk_region.p, s.h_bk_region.data(), 4 * nb, cudaMemcpyHostToDevice, st), "H2D");
    CK(cudaMemcpyAsync(s.bk_zmin.p, bz0.data(), 4 * nb, cudaMemcpyHostToDevice, st), "H2D");
    CK(cudaMemcpyAsync(s.bk_zmax.p, bz1.data(), 4 * nb, cudaMemcpyHostToDevice, st), "H2D");
  }
  CK(cudaMemcpyAsync(s.col_begin.p, cb.data(), 4 * ncol, cudaMemcpyHostToDevice, st), "H2D");
  CK(cudaMemcpyAsync(s.col_end.p, ce.data(), 4 * ncol, cudaMemcpyHostToDevice, st), "H2D");
  CK(cudaStreamSynchronize(st), "upload");
  // rows per unit of z that the buckets' rows see, on average
  double dens = 0;
  for (size_t b = 0; b < nb; b++) {
    const double m = s.h_bk_end[b] - s.h_bk_start[b];
    dens += m * m / std::max<double>((double)bz1[b] - bz0[b], c->ps);
  }
  s.row_density = dens / (double)nn;
  s.valid = true;
  return CPC_OK;
}

// Rebuild a box slot's cell list with columns r_max / k wide from its own
// device arrays (the autotuner's cell-size candidates).
cpc_status rebuild_cells(cpc_ctx *c, Slot &s, int k) {
  const int64_t n = s.n;
  const size_t nn = std::max<int64_t>(n, 1);
  cudaStream_t st = c->st;
  CK(c->u_x.alloc(nn), "alloc"); CK(c->u_y.alloc(nn), "alloc"); CK(c->u_z.alloc(nn), "alloc");
  CK(c->u_w.alloc(nn), "alloc"); CK(c->u_e1.alloc(nn), "alloc"); CK(c->u_e2.alloc(nn), "alloc");
  CK(c->u_phi.alloc(nn), "alloc"); CK(c->u_jk.alloc(nn), "alloc"); CK(c->u_keep.alloc(nn), "alloc");
  CK(c->u_flag.alloc(nn), "alloc"); CK(c->u_orig.alloc(nn), "alloc"); CK(c->u_e3.alloc(nn), "alloc");
  if (n > 0) {
    auto d2d = [&](void *d, const void *h, size_t bytes) {
      return cudaMemcpyAsync(d, h, bytes, cudaMemcpyDeviceToDevice, st);
    };
    CK(d2d(c->u_x.p, s.x.p, 8 * n), "D2D"); CK(d2d(c->u_y.p, s.y.p, 8 * n), "D2D");
    CK(d2d(c->u_z.p, s.z.p, 8 * n), "D2D"); CK(d2d(c->u_w.p, s.w.p, 8 * n), "D2D");
    CK(d2d(c->u_e1.p, s.e1.p, 8 * n), "D2D"); CK(d2d(c->u_e2.p, s.e2.p, 8 * n), "D2D");
    CK(d2d(c->u_phi.p, s.phi.p, 8 * n), "D2D"); CK(d2d(c->u_jk.p, s.jk.p, 4 * n), "D2D");
    CK(d2d(c->u_keep.p, s.keep.p, n), "D2D"); CK(d2d(c->u_flag.p, s.aflag.p, n), "D2D");
    CK(d2d(c->u_orig.p, s.orig.p, 8 * n), "D2D");
    CK(d2d(c->u_e3.p, s.e3.p, 8 * n), "D2D");
  }
  s.valid = false;
  s.zbuilt = false;
  s.version = ++c->version_ctr;
  return build_cells(c, s, n, k, c->u_orig.p, false);
}

// A context's tuning and cell widths during the autotuners' trials: put back when the
// trials end without a choice (an error return).  A slot whose rebuild fails stays
// invalid, as after a failed upload.
struct TuneTrials {
  cpc_ctx *c;
  int k, wpi;
  bool active = true;
  struct Cells {
    int k;
    bool automatic;
  } cells[kMaxSlots];
  explicit TuneTrials(cpc_ctx *ctx) : c(ctx), k(ctx->tune_k), wpi(ctx->tune_wpi) {
    for (int q = 0; q < kMaxSlots; q++) cells[q] = {c->slots[q].kcells, c->slots[q].auto_k};
  }
  ~TuneTrials() {
    if (!active) return;
    c->tune_k = k;
    c->tune_wpi = wpi;
    for (int q = 0; q < kMaxSlots; q++) {
      Slot &s = c->slots[q];
      s.auto_k = cells[q].automatic;
      try {
        if (s.valid && !s.sky && s.kcells != cells[q].k) rebuild_cells(c, s, cells[q].k);
      } catch (...) {
        s.valid = false;
      }
    }
  }
};

// A box slot on cells r_max / k wide that no later upload changes (the autotuners).
cpc_status set_cells(cpc_ctx *c, Slot &s, int k) {
  const cpc_status st = s.kcells == k ? CPC_OK : rebuild_cells(c, s, k);
  if (st == CPC_OK) s.auto_k = false;
  return st;
}

// ---------------------------------------------------------------------------
// sky path (coordinates 0)
// ---------------------------------------------------------------------------

SkyParams sky_params(const cpc_ctx *c) {
  const cpc_params &p = c->p;
  SkyParams sp;
  sp.H = c->H.data();
  sp.dA = c->dA.data();
  sp.n_table = (int64_t)std::min(c->H.size(), c->dA.size());
  sp.dz = p.dz;
  sp.z_max = p.z_max;
  sp.z_sep_max = p.z_sep_max;
  sp.p_min = p.p_min;
  sp.p_max = p.p_max;
  sp.p_size = c->ps;
  sp.r_min = p.bin_r_min;
  sp.r_max = p.bin_r_max;
  sp.r_size = c->rsize;
  sp.lin_bin = p.lin_bin ? 1 : 0;
  sp.n_bins = p.n_bins;
  sp.n_p_bin = p.n_p_bin;
  return sp;
}

// Scaled redshift of the fast kernel's window tests: a power of two that puts
// [0, z_max] on the scale of the angles in degrees, so that one float guard
// serves the three window tests.
double sky_z_scale(const cpc_params &p) {
  return std::ldexp(1.0, (int)std::floor(std::log2(256.0 / std::max(p.z_max, 1e-6))));
}

// Cell order of a redshift-ordered sky catalogue (s.hs_*; zs its redshifts, wins
// its row windows): rows sorted by (jackknife region, keep flag, sky cell of the
// region, redshift), and the buckets (non-empty cells).  A region's cells divide
// its RA x Dec box evenly, sized so that a cell holds about 96 rows (three row
// passes of a warp) in a quarter of the redshift window, between an eighth
// and three quarters of the mean angular window: smaller cells would only
// shorten the candidate runs, larger ones test candidates far outside.
void sky_cell_order(cpc_ctx *c, Slot &s, const std::vector<double> &zs,
                    const std::vector<double> &wins) {
  const cpc_params &p = c->p;
  const int64_t n = s.n;
  const int nreg = p.do_jk ? p.n_jk : 1;
  const double zk = sky_z_scale(p);
  struct Reg {
    double a0 = 1e300, a1 = -1e300, d0 = 1e300, d1 = -1e300, ix = 0, iy = 0;
    int64_t n = 0, base = 0;
    int nx = 1, ny = 1;
  };
  std::vector<Reg> reg(nreg);
  for (int64_t k = 0; k < n; k++) {
    Reg &r = reg[p.do_jk ? s.hs_jk[k] : 0];
    r.a0 = std::min(r.a0, s.hs_ra[k]);
    r.a1 = std::max(r.a1, s.hs_ra[k]);
    r.d0 = std::min(r.d0, s.hs_dec[k]);
    r.d1 = std::max(r.d1, s.hs_dec[k]);
    r.n++;
  }
  // mean window of a sample of rows: half width in Dec, width in redshift, and
  // the share of the catalogue inside it
  double hw = 0, zw = 0, fz = 0;
  int64_t m = 0;
  for (int64_t k = 0; k < n; k += std::max<int64_t>(1, n / 512), m++) {
    const double z0 = wins[k], z1 = wins[n + k];
    hw += 0.5 * (wins[5 * n + k] - wins[4 * n + k]);
    zw += z1 - z0;
    fz += (double)(std::upper_bound(zs.begin(), zs.end(), z1) -
                   std::lower_bound(zs.begin(), zs.end(), z0)) / (double)n;
  }
  if (m) {
    hw /= m;
    zw /= m;
    fz /= m;
  }
  s.sky_zw = zw * zk;
  s.sky_fz = fz;
  s.sky_hw = hw;
  s.sky_area = 0;
  int64_t cells = 0;
  for (Reg &r : reg) {
    r.base = cells;
    if (r.n > 0) {
      const double cosd = std::cos(0.5 * (r.d0 + r.d1) * M_PI / 180.0);
      const double ex = std::max((r.a1 - r.a0) * std::max(cosd, 1e-3), 1e-9);
      const double ey = std::max(r.d1 - r.d0, 1e-9);
      s.sky_area += ex * ey;
      double sz = std::sqrt(96.0 * ex * ey / (std::max(1e-9, 0.25 * fz) * (double)r.n));
      sz = std::min(std::max(sz, hw / 8), 0.75 * hw);
      if (sz > 0) {
        const double lim = std::max(1.0, std::sqrt((double)r.n / 8.0));
        r.nx = (int)std::min(lim, std::max(1.0, std::round(ex / sz)));
        r.ny = (int)std::min(lim, std::max(1.0, std::round(ey / sz)));
      }
      r.ix = r.nx / std::max(r.a1 - r.a0, 1e-30);
      r.iy = r.ny / std::max(r.d1 - r.d0, 1e-30);
    }
    cells += 2ll * r.nx * r.ny;
  }
  std::vector<int64_t> start((size_t)cells + 1, 0);
  std::vector<int64_t> id(n);
  host_parallel(n, [&](int64_t b0, int64_t b1, int) {
    for (int64_t k = b0; k < b1; k++) {
      const Reg &r = reg[p.do_jk ? s.hs_jk[k] : 0];
      const int cx = std::min(r.nx - 1, (int)((s.hs_ra[k] - r.a0) * r.ix));
      const int cy = std::min(r.ny - 1, (int)((s.hs_dec[k] - r.d0) * r.iy));
      id[k] = r.base + (s.hs_keep[k] ? (int64_t)r.nx * r.ny : 0) + (int64_t)cy * r.nx + cx;
    }
  });
  for (int64_t k = 0; k < n; k++) start[id[k] + 1]++;
  for (int64_t q = 0; q < cells; q++) start[q + 1] += start[q];
  s.hc_bk.clear();
  for (int g = 0; g < nreg; g++) {
    const int64_t nc = (int64_t)reg[g].nx * reg[g].ny;
    for (int64_t q = 0; q < 2 * nc; q++) {
      const int64_t b = reg[g].base + q;
      if (start[b + 1] > start[b])
        s.hc_bk.push_back(make_int4((int)start[b], (int)start[b + 1], 2 * g + (q >= nc ? 1 : 0), 0));
    }
  }
  s.sky_nkey = 0;
  for (size_t b = 0; b < s.hc_bk.size(); b++)
    s.sky_nkey += b == 0 || s.hc_bk[b].z != s.hc_bk[b - 1].z;
  s.hc_zidx.resize(n);
  s.hc_z.resize(n);
  for (int64_t k = 0; k < n; k++) s.hc_zidx[start[id[k]]++] = (int)k;
  host_parallel(n, [&](int64_t b0, int64_t b1, int) {
    for (int64_t q = b0; q < b1; q++) s.hc_z[q] = (float)(zs[s.hc_zidx[q]] * zk);
  });
}

// Upload a sky catalogue: per-galaxy windows and angles on the host (C
// library, exactly the reference's values), redshift order from the device
// radix sort, then every array in that order on the device and on the host.
cpc_status sky_upload(cpc_ctx *c, int slot, const cpc_catalog *cat) {
  const cpc_params &p = c->p;
  const int64_t n = cat->n;
  if (n > 0 && (!cat->dc || !cat->da))
    return fail(c, CPC_ERR_INVALID, "sky catalogues need dc and da (distance-table lookups)");
  Slot &s = c->slots[slot];
  s.valid = false;
  s.zbuilt = false;
  s.sky = true;
  s.n = n;
  s.version = ++c->version_ctr;
  const SkyParams sp = sky_params(c);
  std::vector<double> w(n, 1.0), e1(n, 0.0), e2(n, 0.0), phi(n, -10.0);
  std::vector<double> rar(n), decr(n), sd(n), cd(n), win(6 * (size_t)n);
  std::vector<int32_t> jk(n, 0);
  std::vector<uint8_t> keep(n, 0);
  s.has_e = cat->e1 && cat->e2;
  // per row, on the host's cores: the read-path checks (the first failing row
  // in input order is reported), the statistics that size the fixed-point
  // scales, the angles and the lim_calc_sky window with the C library
  struct Part {
    int64_t bad = -1;
    std::string msg;
    double wmax = 0, wmin = 1e300, emax = 0, phimax = 0;
  };
  const int kMaxParts = 64;
  // rows worth a thread: about 0.1 us each of trigonometry and window tables
  const int64_t kSkyRows = 1024;
  std::vector<Part> parts(kMaxParts);
  host_parallel(n, [&](int64_t b0, int64_t b1, int part) {
    Part &P = parts[part];
    for (int64_t i = b0; i < b1; i++) {
      auto bad = [&](const std::string &m) {
        P.bad = i;
        P.msg = m;
      };
      const double ra = cat->x[i], dec = cat->y[i], z = cat->z[i];
      if (!std::isfinite(ra) || !std::isfinite(dec) || !std::isfinite(z) ||
          !std::isfinite(cat->dc[i]) || !std::isfinite(cat->da[i])) {
        bad("non-finite position or distance at row " + std::to_string(i));
        return;
      }
      if (z < 0 || z > p.z_max) {  // read_dat.cpp:228-234
        bad("redshift outside [0, z_max] at row " + std::to_string(i));
        return;
      }
      if (cat->w) {
        if (!std::isfinite(cat->w[i])) { bad("non-finite weight"); return; }
        w[i] = cat->w[i];
      }
      if (s.has_e) {
        if (!std::isfinite(cat->e1[i]) || !std::isfinite(cat->e2[i])) {
          bad("non-finite ellipticity");
          return;
        }
        e1[i] = cat->e1[i];
        e2[i] = cat->e2[i];
      }
      if (cat->phi) {
        if (!std::isfinite(cat->phi[i])) { bad("non-finite phi"); return; }
        phi[i] = cat->phi[i];
      }
      if (p.do_jk) {
        const int r = cat->jk[i];
        if (r < 0 || r >= p.n_jk) {
          bad("jackknife label out of range at row " + std::to_string(i));
          return;
        }
        jk[i] = r;
      }
      if (cat->jk_prob) keep[i] = cat->jk_prob[i] >= 0.5 ? 1 : 0;
      P.wmax = std::max(P.wmax, std::fabs(w[i]));
      P.wmin = std::min(P.wmin, w[i]);
      P.emax = std::max(P.emax, std::sqrt(e1[i] * e1[i] + e2[i] * e2[i]) * (1.0 + 1e-15));
      P.phimax = std::max(P.phimax, std::fabs(phi[i]));
      sky_angles(ra, dec, &rar[i], &decr[i], &sd[i], &cd[i]);
      double wv[6];
      const int rc = sky_window(sp, ra, dec, z, wv);
      if (rc == 1) {  // lim_calc_ra_dec exits the program here (sky_calcs.cpp:109-113)
        bad("window z_min above z_max at row " + std::to_string(i));
        return;
      }
      if (rc == 2) {
        bad("distance table too short for the window of row " + std::to_string(i));
        return;
      }
      for (int q = 0; q < 6; q++) win[(size_t)q * n + i] = wv[q];
    }
  }, kSkyRows);
  s.wmax = 0;
  s.wmin = n > 0 ? 1e300 : 1.0;
  s.emax = 0;
  s.phimax = 0;
  for (const Part &P : parts) {  // chunks are in input order: the first bad row
    if (P.bad >= 0) return fail(c, CPC_ERR_RANGE, P.msg);
    s.wmax = std::max(s.wmax, P.wmax);
    s.wmin = std::min(s.wmin, P.wmin);
    s.emax = std::max(s.emax, P.emax);
    s.phimax = std::max(s.phimax, P.phimax);
  }
  // redshift order (stable: ties keep the input order)
  cudaStream_t st = c->st;
  const size_t nn = std::max<int64_t>(n, 1);
  std::vector<uint32_t> perm(n);
  {
    DevBuf<double> oz;
    CK(oz.alloc(nn), "alloc");
    CK(c->d_keys.alloc(nn), "alloc"); CK(c->d_ktmp.alloc(nn), "alloc");
    CK(c->d_vals.alloc(nn), "alloc"); CK(c->d_vtmp.alloc(nn), "alloc");
    CK(c->d_hist.alloc(radix_hist_words(nn)), "alloc");
    CK(c->d_census.alloc(8 * 256), "alloc");
    if (n > 0) {
      CK(cudaMemcpyAsync(oz.p, cat->z, 8 * n, cudaMemcpyHostToDevice, st), "H2D");
      CK(launch_z_keys(n, oz.p, c->d_keys.p, c->d_vals.p, st), "z keys");
      c->launches += 1;
      CK(radix_sort_pairs(n, c->d_keys.p, c->d_vals.p, c->d_ktmp.p, c->d_vtmp.p, c->d_hist.p,
                          c->d_census.p, st, &c->launches), "z sort");
      CK(cudaMemcpyAsync(perm.data(), c->d_vals.p, 4 * n, cudaMemcpyDeviceToHost, st), "D2H");
    }
    CK(cudaStreamSynchronize(st), "sort");
  }
  std::vector<double> zs(n), sds(n), cds(n), rars(n), decrs(n);
  for (std::vector<double> *v : {&s.hs_ra, &s.hs_dec, &s.hs_dc, &s.hs_da, &s.hs_w, &s.hs_e1,
                                 &s.hs_e2, &s.hs_phi})
    v->resize(n);
  s.hs_jk.resize(n);
  s.hs_keep.resize(n);
  std::vector<int64_t> &orig = s.hs_orig;
  orig.resize(n);
  std::vector<double> wins(6 * (size_t)n);
  std::vector<uint8_t> aflag(n);
  host_parallel(n, [&](int64_t b0, int64_t b1, int) {
    for (int64_t k = b0; k < b1; k++) {
      const uint32_t o = perm[k];
      s.hs_ra[k] = cat->x[o];
      s.hs_dec[k] = cat->y[o];
      zs[k] = cat->z[o];
      s.hs_dc[k] = cat->dc[o];
      s.hs_da[k] = cat->da[o];
      s.hs_w[k] = w[o];
      s.hs_e1[k] = e1[o];
      s.hs_e2[k] = e2[o];
      s.hs_phi[k] = phi[o];
      sds[k] = sd[o];
      cds[k] = cd[o];
      rars[k] = rar[o];
      decrs[k] = decr[o];
      s.hs_jk[k] = jk[o];
      s.hs_keep[k] = keep[o];
      orig[k] = o;
      for (int q = 0; q < 6; q++) wins[(size_t)q * n + k] = win[(size_t)q * n + o];
      // corels1 scan start: row o + 1 (input order) against z_min of row o
      aflag[k] = (o + 1 < (uint32_t)n && !(cat->z[o + 1] < win[o])) ? kAutoStart0 : 0;
    }
  }, 4 * kSkyRows);
  s.hc_tiles.clear();
  s.hc_tile_key.clear();
  sky_cell_order(c, s, zs, wins);
  auto put = [&](DevBuf<double> &d, const std::vector<double> &h, size_t cnt) -> cudaError_t {
    cudaError_t e = d.alloc(std::max<size_t>(cnt, 1));
    if (e != cudaSuccess || cnt == 0) return e;
    return cudaMemcpyAsync(d.p, h.data(), 8 * cnt, cudaMemcpyHostToDevice, st);
  };
  CK(put(s.x, s.hs_ra, n), "sky upload"); CK(put(s.y, s.hs_dec, n), "sky upload");
  CK(put(s.z, zs, n), "sky upload"); CK(put(s.w, s.hs_w, n), "sky upload");
  CK(put(s.e1, s.hs_e1, n), "sky upload"); CK(put(s.e2, s.hs_e2, n), "sky upload");
  CK(put(s.phi, s.hs_phi, n), "sky upload"); CK(put(s.dc, s.hs_dc, n), "sky upload");
  CK(put(s.da, s.hs_da, n), "sky upload"); CK(put(s.sd, sds, n), "sky upload");
  CK(put(s.cd, cds, n), "sky upload"); CK(put(s.rar, rars, n), "sky upload");
  CK(put(s.decr, decrs, n), "sky upload"); CK(put(s.win, wins, 6 * (size_t)n), "sky upload");
  // float views for the fast kernel, in cell order: hi parts and the remainders
  const double zk = sky_z_scale(p);
  const size_t nbk = s.hc_bk.size();
  size_t pack_bytes = 0;
  auto room = [&](size_t bytes) {  // offset of an array in the packed views
    const size_t o = pack_bytes;
    pack_bytes += (bytes + 255) / 256 * 256;
    return o;
  };
  size_t off4[9], off2[2], off1[3];
  for (int q = 0; q < 7; q++) off4[q] = room(sizeof(float4) * n);
  for (int q = 7; q < 9; q++) off4[q] = room(sizeof(float4) * nbk);
  for (size_t &o : off2) o = room(sizeof(float2) * n);
  for (size_t &o : off1) o = room(sizeof(float) * n);
  const size_t off_bk = room(sizeof(int4) * nbk);
  std::unique_ptr<unsigned char[]> pack(new unsigned char[std::max<size_t>(pack_bytes, 1)]);
  auto at4 = [&](int q) { return reinterpret_cast<float4 *>(pack.get() + off4[q]); };
  auto at2 = [&](int q) { return reinterpret_cast<float2 *>(pack.get() + off2[q]); };
  float4 *su = at4(0), *sl = at4(1), *sw = at4(2), *sx = at4(3), *ss = at4(4), *sh = at4(5),
         *wb = at4(6), *box = at4(7), *bwin = at4(8);
  float2 *sph = at2(0), *wz = at2(1);
  float *zf = reinterpret_cast<float *>(pack.get() + off1[0]);
  float *dl = reinterpret_cast<float *>(pack.get() + off1[1]);
  int *zidx = reinterpret_cast<int *>(pack.get() + off1[2]);
  auto hi = [](double v) { return (float)v; };
  auto lo = [](double v) { return (float)(v - (double)(float)v); };
  struct Range {
    double dc = 0, da0 = 1e300, da1 = 0, mag = 0;
  };
  std::vector<Range> ranges(kMaxParts);
  host_parallel(n, [&](int64_t b0, int64_t b1, int part) {
    Range &R = ranges[part];
    for (int64_t q = b0; q < b1; q++) {
      const int64_t k = s.hc_zidx[q];
      const double ux = cds[k] * std::cos(rars[k]), uy = cds[k] * std::sin(rars[k]), uz = sds[k];
      const double dcv = s.hs_dc[k];
      R.dc = std::max(R.dc, std::fabs(dcv));
      R.da0 = std::min(R.da0, s.hs_da[k]);
      R.da1 = std::max(R.da1, std::fabs(s.hs_da[k]));
      su[q] = make_float4(hi(ux), hi(uy), hi(uz), (float)s.hs_da[k]);
      sl[q] = make_float4(lo(ux), lo(uy), lo(uz), lo(dcv));
      dl[q] = (float)(dcv - (double)hi(dcv) - (double)lo(dcv));  // exact: at most 6 bits
      sw[q] = make_float4(hi(s.hs_ra[k]), hi(s.hs_dec[k]), s.hc_z[q], hi(dcv));
      sx[q] = make_float4(lo(s.hs_ra[k]), lo(s.hs_dec[k]), (float)decrs[k], (float)s.hs_w[k]);
      zf[q] = s.hc_z[q];
      zidx[q] = s.hc_zidx[q];
      // weighted ellipticity and the half Dec angle's cosine and sine as hi +
      // lo parts (the compensated shape terms: cos of the pair's mean Dec is
      // cos(d1/2) cos(d2/2) - sin(d1/2) sin(d2/2))
      const double we1 = s.hs_w[k] * s.hs_e1[k], we2 = s.hs_w[k] * s.hs_e2[k];
      ss[q] = make_float4(hi(we1), hi(we2), lo(we1), lo(we2));
      const double ch = std::cos(decrs[k] / 2.0), sh2 = std::sin(decrs[k] / 2.0);
      sh[q] = make_float4(hi(ch), lo(ch), hi(sh2), lo(sh2));
      sph[q] = make_float2((float)s.hs_phi[k], lo(s.hs_w[k]));
      // windows as centre and half width; NaN bounds (lim_calc_ra_dec's acos out
      // of range gives two) pass every candidate, as in the reference
      float c2[3], h2[3];
      for (int m = 0; m < 3; m++) {
        const double f = m == 0 ? zk : 1.0;
        const double v0 = wins[(size_t)(2 * m) * n + k] * f, v1 = wins[(size_t)(2 * m + 1) * n + k] * f;
        if (std::isnan(v0) || std::isnan(v1)) {
          c2[m] = 0.0f;
          h2[m] = INFINITY;
          continue;
        }
        c2[m] = (float)(0.5 * (v0 + v1));
        h2[m] = (float)(0.5 * (v1 - v0));
        R.mag = std::max({R.mag, std::fabs(v0), std::fabs(v1)});
      }
      R.mag = std::max({R.mag, std::fabs(s.hs_ra[k]), std::fabs(s.hs_dec[k]),
                        std::fabs((double)s.hc_z[q])});
      wz[q] = make_float2(c2[0], h2[0]);
      wb[q] = make_float4(c2[1], h2[1], c2[2], h2[2]);
    }
  }, kSkyRows);
  s.dcmax = s.damax = s.sky_mag = 0;
  s.damin = 1e300;
  for (const Range &R : ranges) {
    s.dcmax = std::max(s.dcmax, R.dc);
    s.damin = std::min(s.damin, R.da0);
    s.damax = std::max(s.damax, R.da1);
    s.sky_mag = std::max(s.sky_mag, R.mag);
  }
  // the buckets' RA and Dec ranges, and those of their rows' windows
  s.hc_box.resize(nbk);
  s.hc_bwin.resize(nbk);
  host_parallel((int64_t)nbk, [&](int64_t b0, int64_t b1, int) {
    for (int64_t b = b0; b < b1; b++) {
      float4 r = make_float4(INFINITY, -INFINITY, INFINITY, -INFINITY), v = r;
      for (int q = s.hc_bk[b].x; q < s.hc_bk[b].y; q++) {
        r.x = std::min(r.x, sw[q].x);
        r.y = std::max(r.y, sw[q].x);
        r.z = std::min(r.z, sw[q].y);
        r.w = std::max(r.w, sw[q].y);
        v.x = std::min(v.x, wb[q].x - wb[q].y);
        v.y = std::max(v.y, wb[q].x + wb[q].y);
        v.z = std::min(v.z, wb[q].z - wb[q].w);
        v.w = std::max(v.w, wb[q].z + wb[q].w);
      }
      box[b] = s.hc_box[b] = r;
      bwin[b] = s.hc_bwin[b] = v;
    }
  }, 16);
  if (nbk) std::memcpy(pack.get() + off_bk, s.hc_bk.data(), sizeof(int4) * nbk);
  CK(s.sky_pack.alloc(std::max<size_t>(pack_bytes, 1)), "alloc");
  if (pack_bytes)
    CK(cudaMemcpyAsync(s.sky_pack.p, pack.get(), pack_bytes, cudaMemcpyHostToDevice, st), "H2D");
  {
    auto d4 = [&](int q) { return reinterpret_cast<const float4 *>(s.sky_pack.p + off4[q]); };
    auto d2 = [&](int q) { return reinterpret_cast<const float2 *>(s.sky_pack.p + off2[q]); };
    SkyFast &f = s.sky_f;
    f.su = d4(0); f.sl = d4(1); f.sw = d4(2); f.sx = d4(3); f.ss = d4(4); f.sh = d4(5);
    f.wb = d4(6); f.bk_box = d4(7); f.bk_win = d4(8);
    f.sp = d2(0); f.wz = d2(1);
    f.zf = reinterpret_cast<const float *>(s.sky_pack.p + off1[0]);
    f.dl = reinterpret_cast<const float *>(s.sky_pack.p + off1[1]);
    f.zidx = reinterpret_cast<const int *>(s.sky_pack.p + off1[2]);
    f.bk = reinterpret_cast<const int4 *>(s.sky_pack.p + off_bk);
    f.n_bk = (int)nbk;
  }
  // redshift window bounds that rise with the redshift (but for float rounding,
  // which the kernel's guard covers) can be searched
  s.sky_mono = true;
  const float tol = (float)(2.0 * ulpf(std::max(s.sky_mag, 1e-30)));
  for (const int4 &b : s.hc_bk) {
    float top = -INFINITY, bot = -INFINITY;  // largest bounds so far
    for (int q = b.x; q < b.y && s.sky_mono; q++) {
      const float u = wz[q].x + wz[q].y, l = wz[q].x - wz[q].y;
      s.sky_mono = u >= top - tol && l >= bot - tol;
      top = std::max(top, u);
      bot = std::max(bot, l);
    }
  }
  CK(s.jk.alloc(nn), "alloc"); CK(s.keep.alloc(nn), "alloc"); CK(s.orig.alloc(nn), "alloc");
  CK(s.aflag.alloc(nn), "alloc");
  if (n > 0) {
    CK(cudaMemcpyAsync(s.aflag.p, aflag.data(), n, cudaMemcpyHostToDevice, st), "H2D");
    CK(cudaMemcpyAsync(s.jk.p, s.hs_jk.data(), 4 * n, cudaMemcpyHostToDevice, st), "H2D");
    CK(cudaMemcpyAsync(s.keep.p, s.hs_keep.data(), n, cudaMemcpyHostToDevice, st), "H2D");
    CK(cudaMemcpyAsync(s.orig.p, orig.data(), 8 * n, cudaMemcpyHostToDevice, st), "H2D");
  }
  CK(cudaStreamSynchronize(st), "sky upload");
  s.valid = true;
  return CPC_OK;
}

// One sky corels2 call of a launch (several pair types may share one launch of
// the fast kernel): its job descriptor, device buffers and output.
struct SkyPlan {
  cpc_pair_kind kind;
  int s1, s2;  // slots after the swap rule
  JobRule rule;
  cpc_accum *out;
  JobDev J;
  bool empty;
  size_t cells, n_fix;
  // the outer rows' tiles (fast engine) and their keys; own_*: of a row sample or shard
  const std::vector<SkyTileRows> *tiles = nullptr;
  const std::vector<int> *keys = nullptr;
  bool all = false;  // tiles against every bucket, not region pair by region pair
  std::vector<SkyTileRows> own_tiles;
  std::vector<int> own_keys;
};

SkyView sky_view(Slot &s) {
  SkyView v;
  v.d.n = s.n;
  v.d.x = s.x.p; v.d.y = s.y.p; v.d.z = s.z.p; v.d.w = s.w.p;
  v.d.e1 = s.e1.p; v.d.e2 = s.e2.p; v.d.phi = s.phi.p;
  v.d.jk = s.jk.p; v.d.keep = s.keep.p; v.d.orig = s.orig.p; v.d.aflag = s.aflag.p;
  v.dc = s.dc.p; v.da = s.da.p; v.sd = s.sd.p; v.cd = s.cd.p;
  v.rar = s.rar.p; v.decr = s.decr.p; v.win = s.win.p;
  return v;
}

// Tiles of the fast sky kernel over the rows list[0 .. n_list) (cell positions
// in cell order; null: every row) of slot s.  A tile holds up to kSkyTile rows
// of one bucket within half the mean redshift window, or up to two of them until it
// has 64 rows: a tile's bucket searches and staging cost more than the tests of a
// wide redshift range (data x randoms of 20k x 200k, up to one window until 32 rows
// 7.08 ms, two and 64 6.42, three and 96 6.65; half a window and 32 rows 8.3).  Inside
// a bucket its size is a multiple of 32, so that no row pass has idle lanes.
void sky_tiles(const Slot &s, const int *list, int64_t n_list, std::vector<SkyTileRows> &tiles,
               std::vector<int> &keys) {
  tiles.clear();
  keys.clear();
  const float E = (float)(0.5 * s.sky_zw), Ehi = (float)(2 * s.sky_zw);
  auto z = [&](int64_t k) { return s.hc_z[list ? list[k] : k]; };
  int64_t i = 0;
  for (const int4 &b : s.hc_bk) {
    int64_t e = list ? i : b.y;
    while (list && e < n_list && list[e] < b.y) e++;
    while (i < e) {
      const float z0 = z(i);
      int64_t j = i + 1;
      while (j < e && j - i < kSkyTile && (z(j) - z0 <= E || (j - i < 64 && z(j) - z0 <= Ehi))) j++;
      if (j < e && j - i > 32) j -= (j - i) & 31;
      tiles.push_back(SkyTileRows{(int)i, (int)(j - i)});
      keys.push_back(b.z);
      i = j;
    }
  }
}

// Work units of job m of a sky launch from its tiles (bucket keys `keys`): every
// pair of a row key and a candidate key whose boxes meet, its tiles in `parts`
// runs; or (all) every tile against all candidate buckets.  Returns the number
// of (row key, candidate key) pairs.
size_t sky_units(const Slot &g1, const Slot &g2, const std::vector<int> &keys, int m, int parts,
                 int slices, double guard, bool flip, bool all, std::vector<SkyUnit> &units) {
  auto runs = [](size_t n, auto key, auto &&f) {  // runs of equal keys
    for (size_t a = 0; a < n;) {
      size_t e = a + 1;
      while (e < n && key(e) == key(a)) e++;
      f(a, e);
      a = e;
    }
  };
  struct Key {
    int key, bk0, bk1;
    float4 box;
  };
  auto key_boxes = [&](const Slot &s, const std::vector<float4> &boxes) {
    std::vector<Key> v;
    runs(s.hc_bk.size(), [&](size_t b) { return s.hc_bk[b].z; }, [&](size_t a, size_t e) {
      Key k{s.hc_bk[a].z, (int)a, (int)e, boxes[a]};
      for (size_t b = a + 1; b < e; b++) {
        k.box.x = std::min(k.box.x, boxes[b].x);
        k.box.y = std::max(k.box.y, boxes[b].y);
        k.box.z = std::min(k.box.z, boxes[b].z);
        k.box.w = std::max(k.box.w, boxes[b].w);
      }
      v.push_back(k);
    });
    return v;
  };
  // k1: the tiles' keys, k2: the candidates'; the windows are g1's
  const std::vector<Key> k1 = flip ? key_boxes(g2, g2.hc_box) : key_boxes(g1, g1.hc_bwin);
  const std::vector<Key> k2 = flip ? key_boxes(g1, g1.hc_bwin) : key_boxes(g2, g2.hc_box);
  const int nbk = (int)(flip ? g1 : g2).hc_bk.size();
  if (flip) slices = 1;
  size_t pairs = 0;
  auto emit = [&](int t0, int t1, int key, int b0, int b1) {
    for (int q = 0; q < parts; q++) {
      const int a = t0 + (int)((int64_t)(t1 - t0) * q / parts);
      const int e = t0 + (int)((int64_t)(t1 - t0) * (q + 1) / parts);
      if (a < e)
        for (int sl = 0; sl < slices; sl++)
          units.push_back(SkyUnit{m, a, e, key, b0, b1, all ? 1 : 0, sl, slices});
    }
    pairs++;
  };
  size_t q1 = 0;
  const float g = (float)(4 * guard);
  runs(keys.size(), [&](size_t t) { return keys[t]; }, [&](size_t t0, size_t t1) {
    const int key = keys[t0];
    if (all) {
      for (size_t t = t0; t < t1; t++) emit((int)t, (int)t + 1, key, 0, nbk);
      return;
    }
    while (k1[q1].key != key) q1++;  // both in bucket order
    const float4 w = k1[q1].box;
    for (const Key &y : k2)
      if (y.box.x <= w.y + g && y.box.y >= w.x - g && y.box.z <= w.w + g && y.box.w >= w.z - g)
        emit((int)t0, (int)t1, key, y.bk0, y.bk1);
  });
  return pairs;
}

// Constants of the mixed-precision path of a sky job (SkyConst).  A bin index is
// rint(s x + o) of a float x; it is certain when s x + o is farther from the next
// half-integer (a bin edge) than the error bound E of the whole evaluation
// against the reference's double value.
void sky_consts(const cpc_ctx *c, const Slot &g1, const Slot &g2, JobDev &J) {
  const cpc_params &p = c->p;
  const int nrp = p.n_bins, npi = p.n_p_bin;
  SkyConst &K = J.sk;
  const double eps = std::ldexp(1.0, -24);
  // window tests h - |x - c|: the coordinate, the centre and the half width are
  // within half an ulp of their double values, x - c within another half (|x - c|
  // is h there) and the last difference is exact near zero; doubled
  K.guard = f_up(4.0 * ulpf(std::max({g1.sky_mag, g2.sky_mag, 1e-30})));
  const double dcm = std::max(g1.dcmax, g2.dcmax);
  const double damin = std::min(g1.damin, g2.damin), damax = std::max(g1.damax, g2.damax);
  const double pe = 12 * eps * dcm + 1e-30;
  K.pi_c = (float)(0.5 * (p.p_min + p.p_max));
  K.pi_h = f_up(0.5 * (p.p_max - p.p_min) + pe + 2 * ulpf(std::fabs(p.p_min) + std::fabs(p.p_max)));
  // Pi from hi + lo distances is within 2^-23 |Pi| + 2^-46 max D_C (doubled here)
  {
    const double Pm = std::max(std::fabs(p.p_min), std::fabs(p.p_max));
    const double o = -p.p_min / c->ps - 0.5;
    K.pi_s = (float)(1.0 / c->ps);
    K.pi_o = (float)o;
    const double E = (4 * eps * Pm + 4e-14 * dcm + 1e-30) / c->ps +
                     4 * eps * (npi + std::fabs(o) + 1) + 1e-9;
    K.pi_in = E < 0.5 ? f_down(0.5 - E) : -1.0f;
    const double v0 = std::floor((0.0 - p.p_min) / c->ps);  // corel_bin (corels.cpp:26)
    K.pi_zero = v0 >= 0 && v0 < npi ? (int)v0 : -1;
  }
  // r_p certainly outside, from t = chord^2 (D_A1 + D_A2)^2 of float unit vectors
  // (chord within 4e-7): r_p < r_hi implies t < t_hi, r_p >= r_lo implies t >= t_lo
  const double r_lo = c->thr_rp[0], r_hi = c->thr_rp[nrp];
  {
    const double h = 2 * r_hi + 8e-7 * damax;
    K.t_hi = f_up(h * h * (1 + 1e-5));
    // a clamped pair (theta < 1.42e-5) has r_p = 0, which bins when thr_0 <= 0
    if (r_lo <= 0 && r_hi < 1e-4 * damax) K.t_hi = INFINITY;
    K.t_lo = -1.0f;
    if (r_lo > 0 && damin > 0 && r_lo < 0.5 * damin) {
      const double th = r_lo / damin, l = 2 * r_lo * (1 - th * th / 24) - 8e-7 * damax;
      if (l > 0) K.t_lo = f_down(l * l * (1 - 1e-5));
    }
  }
  // r_p from the hi + lo chord: its series or asinf, the D_A sum (< 1.5e-6), and
  // the reference's own sum = cos(theta) rounding through acos, at most 4e-7 for
  // chords above 1e-4 (smaller ones take the FP64 path): 2.1e-6 relative
  {
    const double rel = 2.1e-6;
    double E, o;
    if (p.lin_bin) {
      const double s = 1.0 / c->rsize;
      o = -p.bin_r_min * s - 0.5;
      K.rp_s = (float)(0.5 * s);
      E = rel * p.bin_r_max * s + 6 * eps * (nrp + std::fabs(o) + p.bin_r_max * s + 1) + 1e-7;
    } else {
      // log2 of (2 r_p)^2: __log2f is within 2 ulp (4e-6 for |log2| < 32)
      const double s = nrp / (2.0 * std::log2(p.bin_r_max / p.bin_r_min));
      const double l0 = 2.0 + 2.0 * std::log2(p.bin_r_min);
      o = -l0 * s - 0.5;
      K.rp_s = (float)s;
      E = s * (2 * rel / M_LN2 + 4e-6 + 4 * eps * (std::fabs(l0) + 32)) +
          4 * eps * (nrp + std::fabs(o) + 1) + 1e-7;
      // the exact thresholds must be the edges of this map
      for (int k = 0; k <= nrp; k++)
        if (!(std::fabs((2.0 + 2.0 * std::log2(c->thr_rp[k]) - l0) * s - k) < 1e-7)) E = 1.0;
    }
    K.rp_o = (float)o;
    K.rp_in = E < 0.5 ? f_down(0.5 - E) : -1.0f;
  }
}

// Entries for the undecided pairs of `rows` rows of g1 against g2: their window pairs,
// by the share of g2 in a mean window, times twice the rates met (pair_sky.cu).  Too
// few cost time, not pairs: randoms x randoms of 1M rows leave 5e6, all but a fixed
// 2^20 of which went to single lanes (304 ms, 292 with room for them).
size_t sky_queue(const Slot &g1, const Slot &g2, double rows, bool counts) {
  const double sky = std::min(1.0, 4 * g1.sky_hw * g1.sky_hw / std::max(g2.sky_area, 1e-30));
  const double want = rows * (double)g2.n * g1.sky_fz * sky * (counts ? 1.0 / 4096 : 1.0 / 200);
  if (!(want > (double)kSkyExactQueue)) return kSkyExactQueue;
  return (size_t)std::min(want, (double)kSkyExactQueueMax);
}

// Plan job k of a sky launch: the corels2 rules, the bands and fixed-point
// scales of the mixed-precision path, zeroed device buffers (set k), the row
// sample as a list of g1 rows.
cpc_status sky_plan(cpc_ctx *c, cpc_pair_kind kind, int slot_g1, int slot_g2, int64_t rs,
                    int64_t ro, cpc_engine engine, cpc_accum *out, int auto_mode, size_t k,
                    SkyPlan &P) {
  if (slot_g1 < 0 || slot_g1 >= kMaxSlots || slot_g2 < 0 || slot_g2 >= kMaxSlots)
    return fail(c, CPC_ERR_INVALID, "slot out of range");
  Slot &A = c->slots[slot_g1], &B = c->slots[slot_g2];
  if (!A.valid || !B.valid || !A.sky || !B.sky) return fail(c, CPC_ERR_STATE, "count before upload");
  if (!out || !out->num || !out->sums) return fail(c, CPC_ERR_INVALID, "null output arrays");
  const cpc_params &p = c->p;
  JobRule rule;
  if ((auto_mode ? job_rule_auto(p, kind, rule) : job_rule(p, kind, A.n, B.n, rule)) != 0)
    return fail(c, CPC_ERR_INVALID, "bad pair kind");
  const int s1 = rule.swapped ? slot_g2 : slot_g1, s2 = rule.swapped ? slot_g1 : slot_g2;
  Slot &g1 = c->slots[s1], &g2 = c->slots[s2];
  P.kind = kind;
  P.s1 = s1;
  P.s2 = s2;
  P.rule = rule;
  P.out = out;
  P.empty = A.n == 0 || B.n == 0;  // corr.cpp:273-277
  P.cells = (size_t)(1 + (p.do_jk ? p.n_jk : 0)) * p.n_bins * p.n_p_bin;
  P.n_fix = P.cells * kNF;
  out->kernel_ms = out->pair_kernel_ms = 0;
  while (c->sky_bufs.size() <= k) c->sky_bufs.emplace_back(new SkyJobBufs());
  SkyJobBufs &Bf = *c->sky_bufs[k];
  cudaStream_t st = c->st;
  CK(Bf.num.alloc(P.cells), "alloc histograms");
  CK(Bf.sums.alloc(P.cells * kNF), "alloc histograms");
  CK(Bf.counters.alloc(4), "alloc counters");
  CK(cudaMemsetAsync(Bf.num.p, 0, sizeof(unsigned long long) * P.cells, st), "memset");
  CK(cudaMemsetAsync(Bf.sums.p, 0, sizeof(double) * P.cells * kNF, st), "memset");
  CK(cudaMemsetAsync(Bf.counters.p, 0, sizeof(unsigned long long) * 4, st), "memset");
  JobDev &J = P.J;
  std::memset(&J, 0, sizeof J);
  J.acc_num = Bf.num.p;
  J.acc_sums = Bf.sums.p;
  J.counters = Bf.counters.p;
  if (P.empty) return CPC_OK;
  J.corel = rule.corel;
  J.gws = rule.gws;
  J.which_corr = p.which_corr;
  J.estimator = p.estimator;
  J.do_jk = p.do_jk ? 1 : 0;
  J.n_jk = p.n_jk;
  J.coordinates = 0;
  J.nrp = p.n_bins;
  J.npi = p.n_p_bin;
  J.lin_bin = p.lin_bin ? 1 : 0;
  J.box_same_keep = 0;  // jk_check_sky (jk.cpp:53-57)
  J.auto_mode = auto_mode;
  J.row_stride = rs > 1 ? rs : 1;
  J.row_offset = ro;
  J.rmin = p.bin_r_min;
  J.rmax = p.bin_r_max;
  J.pmin = p.p_min;
  J.pmax = p.p_max;
  J.ps = c->ps;
  J.rsize = c->rsize;
  for (int q = 0; q <= p.n_bins; q++) J.thr[q] = c->thr_rp[q];
  sky_consts(c, g1, g2, J);
  // fixed-point scales of the fast kernel: terms rint(v 2^S_f),
  // |v| 2^S_f <= 2^30 / (1 + 2^-12); the global sums keep a low and a high
  // 64-bit word per bin and field (2^48 terms per bin, checked after the count)
  {
    const double wm = std::max(g1.wmax, 1e-30) * std::max(g2.wmax, 1e-30);
    const double em = std::max({g1.emax, g2.emax, 1e-30});
    const double tm = std::max(M_PI / 2, std::max(g1.phimax, g2.phimax) + M_PI);
    const double tm2 = (rule.corel == COREL_SSA) ? 2 * tm : tm;
    double vb[kNF];
    vb[0] = wm;
    vb[1] = vb[3] = wm * em;
    vb[2] = vb[4] = wm * wm * em * em;
    vb[5] = vb[7] = vb[9] = wm * em * em;
    vb[6] = vb[8] = vb[10] = wm * wm * em * em * em * em;
    vb[11] = tm2;
    vb[12] = 2 * tm * tm;
    for (int f = 0; f < kNF; f++) {
      const double v = std::max(vb[f] * (1.0 + 1.0 / 4096.0), 1e-30);
      int S = 30 - (int)std::ceil(std::log2(v));
      S = std::min(60, std::max(-60, S));
      J.qscale[f] = (float)std::ldexp(1.0, S);
      J.inv_qscale[f] = std::ldexp(1.0, -S);
    }
    J.unit_w = (engine == CPC_ENGINE_FAST && g1.wmax == 1.0 && g1.wmin == 1.0 &&
                g2.wmax == 1.0 && g2.wmin == 1.0) ? 1 : 0;
  }
  CK(Bf.fix.alloc(2 * P.n_fix), "alloc fixed-point sums");  // low words, then high words
  CK(cudaMemsetAsync(Bf.fix.p, 0, sizeof(unsigned long long) * 2 * P.n_fix, st), "memset");
  J.acc_fix = Bf.fix.p;
  J.acc_fixh = Bf.fix.p + P.n_fix;
  J.sky1 = sky_view(g1);
  J.sky2 = sky_view(g2);
  J.sf1 = g1.sky_f;
  J.sf2 = g2.sky_f;
  CK(Bf.hq.alloc(kSkyHostQueue), "alloc host queue");
  CK(Bf.hq_n.alloc(1), "alloc");
  CK(cudaMemsetAsync(Bf.hq_n.p, 0, sizeof(unsigned long long), st), "memset");
  J.sk.hist_smem = sky_hist_fits(J.corel, J.unit_w, p.n_bins * p.n_p_bin) ? 1 : 0;
  J.hq = Bf.hq.p;
  J.hq_n = Bf.hq_n.p;
  // the outer rows as tiles.  A row sample (input index i with i % rs == ro) or a
  // work shard of the fast engine (cpc_set_shard: redshift-ordered positions k
  // with k % n_shards == shard) lists its rows first.
  // Against a g2 of at most half as many galaxies (data against randoms) the
  // tiles hold g2's and the candidates are g1's, whose runs then fill the warps.
  J.row_list = nullptr;
  const int W = c->n_shards;
  if (engine == CPC_ENGINE_FAST) {
    // A region pair's unit pays for itself from about 40 pairs per bin on (counts
    // alone, whose pairs cost one global add: 300); below, and with too many keys
    // to pair up on the host, the units are tiles against every bucket.  RsRd of
    // 15k randoms in 100 regions (8 per bin): 0.95 ms by pairs, 0.30 by tiles; of
    // 200k (1,400): 14.8 and 21.0.  SRd of 8k x 40k (11): 2.08 and 1.43; of 20k x
    // 200k (140): 7.1 and 15.2.
    {
      const double k1 = std::max(1, g1.sky_nkey), k2 = std::max(1, g2.sky_nkey);
      const double rows = (double)g1.n / (double)std::max<int64_t>(1, rs) / W;
      P.all = rows / k1 * ((double)g2.n / k2) * g2.sky_fz <
                  (J.corel == COREL_DD ? 300.0 : 40.0) * p.n_bins * p.n_p_bin ||
              k1 * k2 > 4e6;
    }
    if (W <= 1 && rs <= 1) {
      J.sk.flip = !P.all && !auto_mode && g1.sky_mono && g2.n * 2 <= g1.n ? 1 : 0;
      Slot &gt = J.sk.flip ? g2 : g1;
      if (gt.hc_tiles.empty()) sky_tiles(gt, nullptr, gt.n, gt.hc_tiles, gt.hc_tile_key);
      P.tiles = &gt.hc_tiles;
      P.keys = &gt.hc_tile_key;
    } else {
      std::vector<int> rows;
      rows.reserve((size_t)(g1.n / std::max<int64_t>(1, rs) / W + 1));
      for (int64_t q = 0; q < g1.n; q++) {
        const int i = g1.hc_zidx[q];
        if ((W <= 1 || i % W == c->shard) && (rs <= 1 || ((g1.hs_orig[i] - ro) % rs) == 0))
          rows.push_back((int)q);
      }
      sky_tiles(g1, rows.data(), (int64_t)rows.size(), P.own_tiles, P.own_keys);
      P.tiles = &P.own_tiles;
      P.keys = &P.own_keys;
      CK(Bf.rows.alloc(std::max<size_t>(rows.size(), 1)), "alloc row sample");
      if (!rows.empty())
        CK(cudaMemcpyAsync(Bf.rows.p, rows.data(), sizeof(int) * rows.size(),
                           cudaMemcpyHostToDevice, st), "H2D");
      CK(cudaStreamSynchronize(st), "sync");  // rows is a host temporary
      J.row_list = Bf.rows.p;
    }
    CK(Bf.tiles.alloc(std::max<size_t>(P.tiles->size(), 1)), "alloc tiles");
    if (!P.tiles->empty())
      CK(cudaMemcpyAsync(Bf.tiles.p, P.tiles->data(), sizeof(SkyTileRows) * P.tiles->size(),
                         cudaMemcpyHostToDevice, st), "H2D");
    J.tiles = Bf.tiles.p;
    {
      const double rows = (double)g1.n / (double)std::max<int64_t>(1, rs) / W;
      const size_t want = sky_queue(g1, g2, rows, J.corel == COREL_DD && J.unit_w);
      if (want > kSkyExactQueue && Bf.xq.alloc(want) != cudaSuccess) cudaGetLastError();
      CK(Bf.xq.alloc(kSkyExactQueue), "alloc undecided pairs");
      J.xq_cap = Bf.xq.n;
    }
    CK(Bf.xq_n.alloc(1), "alloc");
    CK(cudaMemsetAsync(Bf.xq_n.p, 0, sizeof(unsigned long long), st), "memset");
    J.xq = Bf.xq.p;
    J.xq_n = Bf.xq_n.p;
  }
  return CPC_OK;
}

// The host edge tier of a finished job: the pairs the GPU queued are binned with
// the C library in the reference's operation order and added to the output.
cpc_status sky_finish(cpc_ctx *c, SkyPlan &P, size_t k, cpc_engine engine, float ms) {
  const cpc_params &p = c->p;
  cpc_accum *out = P.out;
  SkyJobBufs &Bf = *c->sky_bufs[k];
  cpc_status st_;
  if ((st_ = fetch_accum_from(c, Bf.num.p, Bf.sums.p, Bf.counters.p, out, c->st,
                              P.empty ? 0 : P.J.unit_w)) != CPC_OK)
    return st_;
  out->kernel_ms = out->pair_kernel_ms = ms;
  if (P.empty) return CPC_OK;
  if (engine != CPC_ENGINE_FP64) {
    // the low and high fixed-point words hold 2^48 terms of |u| < 2^30 per bin
    for (size_t q = 0; q < P.cells; q++)
      if ((unsigned long long)out->num[q] >= (1ull << 48))
        return fail(c, CPC_ERR_RANGE,
                    "a sky bin holds 2^48 pairs or more: its fixed-point sums may overflow; "
                    "count the term in row samples (row_stride)");
  }
  unsigned long long nq = 0;
  CK(cudaMemcpy(&nq, Bf.hq_n.p, sizeof nq, cudaMemcpyDeviceToHost), "D2H");
  if (nq > kSkyHostQueue)
    return fail(c, CPC_ERR_RANGE, "too many pairs within the trigonometry error bound of a bin edge");
  std::vector<int2> q(nq);
  if (nq) CK(cudaMemcpy(q.data(), Bf.hq.p, sizeof(int2) * nq, cudaMemcpyDeviceToHost), "D2H");
  const JobRule &rule = P.rule;
  Slot &g1 = c->slots[P.s1], &g2 = c->slots[P.s2];
  // host edge tier: the reference's own arithmetic with the C library
  const SkyParams sp = sky_params(c);
  const int nb = p.n_bins, npb = p.n_p_bin;
  const size_t hstride = (size_t)nb * npb;
  for (const int2 &e : q) {
    const int i = e.x, j = e.y;
    int n1, n2;
    if (sky_bin(sp, g1.hs_ra[i], g1.hs_dec[i], g1.hs_dc[i], g1.hs_da[i], g2.hs_ra[j],
                g2.hs_dec[j], g2.hs_dc[j], g2.hs_da[j], &n1, &n2) != 2)
      continue;
    const double wt = g1.hs_w[i] * g2.hs_w[j];
    const double theta = rule.corel == COREL_DD
                             ? 0.0 : sky_orient(g1.hs_ra[i], g1.hs_dec[i], g2.hs_ra[j], g2.hs_dec[j]);
    double f[kNF];
    pair_values(rule.corel, rule.gws, wt, theta, PairGal{g1.hs_e1[i], g1.hs_e2[i], g1.hs_phi[i]},
                PairGal{g2.hs_e1[j], g2.hs_e2[j], g2.hs_phi[j]}, f);
    const size_t cell = (size_t)n1 * npb + n2;
    out->num[cell] += 1;
    for (int k = 0; k < kNF; k++) out->sums[cell * kNF + k] += f[k];
    if (!p.do_jk) continue;
    const int r1 = g1.hs_jk[i], r2 = g2.hs_jk[j];
    int k1 = g1.hs_keep[i], k2 = g2.hs_keep[j];
    if (r1 == r2) k2 = 0;
    const int rr[2] = {r1, r2}, kk[2] = {k1, k2};
    for (int t = 0; t < 2; t++) {
      if (!kk[t]) continue;
      const size_t hc = (size_t)(1 + rr[t]) * hstride + cell;
      out->num[hc] += 1;
      out->sums[hc * kNF] += f[0];
      if (p.which_corr == 0) continue;
      for (int k = 1; k < kNF; k += 2) out->sums[hc * kNF + k] += f[k];
    }
  }
  int64_t nbin = 0;
  for (size_t q2 = 0; q2 < hstride; q2++) nbin += out->num[q2];
  out->n_binned = nbin;
  out->n_rechecked = (int64_t)nq;
  return CPC_OK;
}

// Sky counts (coordinates 0) of one context: the fast engine runs the units of
// every job (sky_tile_kernel), then the fixed-point blocks are converted and each
// job's host edge tier runs; the FP64 engine runs the plain kernel per job.
cpc_status sky_run(cpc_ctx *c, std::vector<SkyPlan> &plans, cpc_engine engine) {
  const cpc_params &p = c->p;
  cudaStream_t st = c->st;
  cpc_status st_;
  if ((st_ = ensure_scratch(c, 1, plans.size())) != CPC_OK) return st_;
  std::vector<JobDev> jd;
  std::vector<size_t> idx;  // plan of each launched job
  for (size_t k = 0; k < plans.size(); k++) {
    if (plans[k].empty) continue;
    jd.push_back(plans[k].J);
    idx.push_back(k);
  }
  // bound on |sum_gpu - sum_libm|: cos differs by <= 3 ulp (CUDA 2 + C library
  // 1), one more ulp from each of the product and the sum, doubled
  const double esum = 8.0 * std::ldexp(1.0, -52);
  CK(cudaEventRecord(c->e0, st), "event");
  if (!jd.empty()) {
    CK(cudaMemcpyAsync(c->d_jobs.p, jd.data(), sizeof(JobDev) * jd.size(), cudaMemcpyHostToDevice,
                       st), "H2D jobs");
    if (engine == CPC_ENGINE_FP64) {
      for (size_t m = 0; m < jd.size(); m++) {
        Slot &g1 = c->slots[plans[idx[m]].s1], &g2 = c->slots[plans[idx[m]].s2];
        CK(launch_sky_fp64(c->d_jobs.p + m, sky_view(g1), sky_view(g2), jd[m].hq, jd[m].hq_n,
                           kSkyHostQueue, esum, st), "sky kernel");
        c->launches += 1;
      }
    } else {
      // the units of every job, split until each block finds about six of them:
      // first a key pair's tiles, then the redshift range of its candidates.  Each
      // instantiation (0 counts, 1 shape x density, 2 shape x shape) has its range of
      // the list, counts first: their units (randoms against randoms) are the longest,
      // and last they cost 5% in few regions.
      std::vector<SkyUnit> units;
      size_t end[3] = {0, 0, 0};  // of the units of each
      auto set_of = [&](const JobDev &J) {
        return J.corel == COREL_DD ? 0 : J.corel == COREL_SD ? 1 : 2;
      };
      auto build = [&](int parts, int slices) {
        size_t pairs = 0;
        units.clear();
        for (int q = 0; q < 3; q++) {
          for (size_t m = 0; m < jd.size(); m++) {
            const SkyPlan &P = plans[idx[m]];
            if (set_of(jd[m]) == q)
              pairs += sky_units(c->slots[P.s1], c->slots[P.s2], *P.keys, (int)m, parts, slices,
                                 jd[m].sk.guard, jd[m].sk.flip != 0, P.all, units);
          }
          end[q] = units.size();
        }
        return pairs;
      };
      const size_t want = (size_t)c->sm_count * 24;
      const size_t pairs = build(1, 1);
      if (pairs && units.size() < want) {
        const int parts = (int)((want + pairs - 1) / pairs);
        build(parts, 1);
        if (units.size() < want / 2)
          build(parts, (int)std::min<size_t>(4, want / std::max<size_t>(1, units.size())));
      }
      // A launch per instantiation: counts keep four blocks per SM of 64 registers,
      // shape terms three of 80 (20k x 200k: 30.6 ms in one launch, 28.6 in two).  The
      // second goes on a stream of its own, so that its blocks follow the first's as
      // they end.  Ranges of fewer than about eight units a block share a launch: a
      // coarse list leaves blocks idle at the end of each (8k x 53k in 25 regions,
      // 1,300 units of counts: 2.45 ms in one, 2.73 in two).
      const size_t kRange = (size_t)c->sm_count * 32;
      struct Range {
        size_t first, n;
        int set;
      };
      std::vector<Range> ranges;
      for (int q = 0; q < 3; q++) {
        const size_t first = q ? end[q - 1] : 0, n = end[q] - first;
        if (n == 0) continue;
        if (!ranges.empty() && (ranges.back().n < kRange || n < kRange)) {
          ranges.back().n += n;
          ranges.back().set = q;
        } else {
          ranges.push_back(Range{first, n, q});
        }
      }
      CK(c->d_sky_units.alloc(units.size()), "alloc units");
      CK(c->d_sky_ctr.alloc(3), "alloc");
      if (!units.empty())
        CK(cudaMemcpyAsync(c->d_sky_units.p, units.data(), sizeof(SkyUnit) * units.size(),
                           cudaMemcpyHostToDevice, st), "H2D");
      CK(cudaMemsetAsync(c->d_sky_ctr.p, 0, 3 * sizeof(unsigned long long), st), "memset");
      if (ranges.size() > 1) {
        if (!c->st2) CK(cudaStreamCreateWithFlags(&c->st2, cudaStreamNonBlocking), "stream");
        CK(cudaEventRecord(c->e_in, st), "event");
        CK(cudaStreamWaitEvent(c->st2, c->e_in, 0), "stream wait");
      }
      std::reverse(ranges.begin(), ranges.end());  // (counts, of the small blocks, fill in)
      cudaError_t launched = cudaSuccess;
      for (size_t q = 0; q < ranges.size() && launched == cudaSuccess; q++) {
        size_t hist_words = 1;
        for (const JobDev &J : jd)
          if (J.sk.hist_smem && set_of(J) <= ranges[q].set)
            hist_words = std::max(hist_words,
                                  sky_hist_words(J.corel, J.unit_w, p.n_bins * p.n_p_bin));
        launched = launch_sky_tile(c->d_jobs.p, c->d_sky_units.p + ranges[q].first,
                                   (int)ranges[q].n, ranges[q].set, hist_words,
                                   c->d_sky_ctr.p + q, kSkyHostQueue, esum, c->sm_count,
                                   q & 1 ? c->st2 : st);
        if (launched == cudaSuccess) c->launches += 1;
      }
      // st goes on after st2, also where a launch failed: a later count reuses the buffers
      if (ranges.size() > 1) {
        CK(cudaEventRecord(c->e_done, c->st2), "event");
        CK(cudaStreamWaitEvent(st, c->e_done, 0), "stream wait");
      }
      CK(launched, "sky kernel");
      for (size_t m = 0; m < jd.size(); m++) {
        const SkyPlan &P = plans[idx[m]];
        CK(launch_sky_finish((int64_t)P.n_fix, jd[m].acc_fix, jd[m].acc_fixh, jd[m].acc_sums,
                             c->d_jobs.p + m, kSkyHostQueue, esum, st), "fixed-point sums");
        c->launches += 1;
      }
    }
  }
  CK(cudaEventRecord(c->e1, st), "event");
  CK(cudaEventSynchronize(c->e1), "sync");
  float ms = 0;
  CK(cudaEventElapsedTime(&ms, c->e0, c->e1), "event time");
  for (size_t k = 0; k < plans.size(); k++)
    if ((st_ = sky_finish(c, plans[k], k, engine, ms)) != CPC_OK) return st_;
  return CPC_OK;
}

// one sky corels2 call
cpc_status sky_count(cpc_ctx *c, cpc_pair_kind kind, int slot_g1, int slot_g2, int64_t rs,
                     int64_t ro, cpc_engine engine, cpc_accum *out, int auto_mode = 0) {
  std::vector<SkyPlan> plans(1);
  cpc_status s = sky_plan(c, kind, slot_g1, slot_g2, rs, ro, engine, out, auto_mode, 0, plans[0]);
  if (s != CPC_OK) return s;
  return sky_run(c, plans, engine);
}

}  // namespace

extern "C" {

const char *cpc_version(void) { return "corr_pc_gb300 0.1 (sm_103a)"; }

const char *cpc_last_error(const cpc_ctx *ctx) {
  if (ctx) return ctx->err.c_str();
  return g_err.c_str();
}

cpc_status cpc_create(cpc_ctx **out, const cpc_params *params) try {
  if (!out || !params) return fail(nullptr, CPC_ERR_INVALID, "null argument");
  *out = nullptr;
  cpc_status s = validate_params(nullptr, *params);
  if (s != CPC_OK) return s;
  std::unique_ptr<cpc_ctx> c(new (std::nothrow) cpc_ctx());
  if (!c) return fail(nullptr, CPC_ERR_NOMEM, "host allocation failed");
  c->p = *params;
  if (params->H_z && params->n_table > 0) {
    c->H.assign(params->H_z, params->H_z + params->n_table);
    c->p.H_z = c->H.data();
  }
  if (params->dA_z && params->n_table > 0) {
    c->dA.assign(params->dA_z, params->dA_z + params->n_table);
    c->p.dA_z = c->dA.data();
  }
  const cpc_params &p = c->p;
  c->ps = (p.p_max - p.p_min) / (p.n_p_bin);
  if (p.lin_bin) c->rsize = (p.bin_r_max - p.bin_r_min) / p.n_bins;
  else c->rsize = (std::log10(p.bin_r_max) - std::log10(p.bin_r_min)) / p.n_bins;
  int rc = rp_thresholds(p.lin_bin, p.n_bins, p.bin_r_min, p.bin_r_max, c->thr_rp);
  if (rc != 0) return fail(nullptr, CPC_ERR_INVALID, "r_p bin thresholds could not be derived (non-monotone bin function)");
  rc = pi_thresholds(p.n_p_bin, p.p_min, p.p_max, c->thr_pi);
  if (rc != 0) return fail(nullptr, CPC_ERR_INVALID, "Pi bin thresholds could not be derived");
  cudaError_t e = cudaGetDevice(&c->device);
  if (e != cudaSuccess) return cuda_fail(nullptr, e, "cudaGetDevice");
  e = cudaDeviceGetAttribute(&c->sm_count, cudaDevAttrMultiProcessorCount, c->device);
  if (e != cudaSuccess) return cuda_fail(nullptr, e, "device attribute");
  if (const char *ev = std::getenv("CPC_TWIN")) c->twin_on = std::atoi(ev) != 0 ? 1 : 0;
  e = cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking);
  if (e != cudaSuccess) return cuda_fail(nullptr, e, "stream");
  e = cudaEventCreate(&c->e0);
  if (e == cudaSuccess) e = cudaEventCreate(&c->e1);
  if (e == cudaSuccess) e = cudaEventCreate(&c->e2);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&c->e_in, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&c->e_done, cudaEventDisableTiming);
  if (e != cudaSuccess) return cuda_fail(nullptr, e, "event");
  *out = c.release();
  return CPC_OK;
} catch (...) {
  return host_exception(nullptr);
}

cpc_status cpc_destroy(cpc_ctx *c) try {
  if (!c) return CPC_OK;
  cudaStreamSynchronize(c->st);
  if (c->st2) cudaStreamSynchronize(c->st2);
  drop_graph(c);
  if (c->e0) cudaEventDestroy(c->e0);
  if (c->e1) cudaEventDestroy(c->e1);
  if (c->e2) cudaEventDestroy(c->e2);
  if (c->e_in) cudaEventDestroy(c->e_in);
  if (c->e_done) cudaEventDestroy(c->e_done);
  if (c->st) cudaStreamDestroy(c->st);
  if (c->st2) cudaStreamDestroy(c->st2);
  delete c;
  return CPC_OK;
} catch (...) {
  return host_exception(c);
}

cpc_status cpc_accum_shape(const cpc_ctx *c, int *n_hist, int *n_bins, int *n_p_bin) {
  if (!c) return fail(nullptr, CPC_ERR_INVALID, "null context");
  if (n_hist) *n_hist = 1 + (c->p.do_jk ? c->p.n_jk : 0);
  if (n_bins) *n_bins = c->p.n_bins;
  if (n_p_bin) *n_p_bin = c->p.n_p_bin;
  return CPC_OK;
}

// a count enqueued by cpc_count_async must be collected first
static bool busy(cpc_ctx *c) {
  if (!c || !c->pending) return false;
  fail(c, CPC_ERR_STATE, "a count is pending: call cpc_count_finish first");
  return true;
}

cpc_status cpc_set_tuning(cpc_ctx *c, int cells_per_rmax, int pi_window, int tile) {
  if (!c) return fail(nullptr, CPC_ERR_INVALID, "null context");
  if (busy(c)) return CPC_ERR_STATE;
  if (cells_per_rmax < 0 || cells_per_rmax > kMaxCellsPerRmax || pi_window < 0 ||
      (tile != 0 && tile != kTileThreads))
    return fail(c, CPC_ERR_INVALID, "tuning values out of range");
  c->tune_k = cells_per_rmax;
  c->tune_wpi = pi_window;
  c->tune_tile = tile;
  return CPC_OK;
}

cpc_status cpc_upload(cpc_ctx *c, int slot, const cpc_catalog *cat) try {
  if (!c || !cat) return fail(c, CPC_ERR_INVALID, "null argument");
  if (busy(c)) return CPC_ERR_STATE;
  if (slot < 0 || slot >= kMaxSlots) return fail(c, CPC_ERR_INVALID, "slot out of range");
  const cpc_params &p = c->p;
  const int64_t n = cat->n;
  if (n < 0 || n >= 2147483647LL) return fail(c, CPC_ERR_INVALID, "catalogue size out of range");
  if (n > 0 && (!cat->x || !cat->y || !cat->z)) return fail(c, CPC_ERR_INVALID, "null positions");
  if (p.do_jk && n > 0 && !cat->jk) return fail(c, CPC_ERR_INVALID, "jackknife labels required (do_jk=1)");
  if (p.coordinates == 0) return sky_upload(c, slot, cat);
  Slot &s = c->slots[slot];
  s.sky = false;
  s.valid = false;
  s.zbuilt = false;
  s.n = n;
  s.version = ++c->version_ctr;
  const double L = p.periodic_box_size;
  s.has_e = cat->e1 || cat->e2 || cat->e3;
  cudaStream_t st = c->st;
  // the caller's arrays, in input order, in context buffers reused by every
  // upload; absent optional arrays get the reference's defaults on the device
  // (w 1, e 0, phi -10, region 0)
  const size_t nn = std::max<int64_t>(n, 1);
  DevBuf<double> &ox = c->u_x, &oy = c->u_y, &oz = c->u_z, &ow = c->u_w, &oe1 = c->u_e1,
                 &oe2 = c->u_e2, &ophi = c->u_phi, &oprob = c->u_prob, &oe3 = c->u_e3;
  DevBuf<int32_t> &ojk = c->u_jk;
  DevBuf<uint8_t> &okeep = c->u_keep, &oflag = c->u_flag;
  CK(oe3.alloc(nn), "alloc");
  CK(ox.alloc(nn), "alloc"); CK(oy.alloc(nn), "alloc"); CK(oz.alloc(nn), "alloc");
  CK(ow.alloc(nn), "alloc"); CK(oe1.alloc(nn), "alloc"); CK(oe2.alloc(nn), "alloc");
  CK(ophi.alloc(nn), "alloc"); CK(oprob.alloc(nn), "alloc"); CK(ojk.alloc(nn), "alloc");
  CK(okeep.alloc(nn), "alloc"); CK(oflag.alloc(nn), "alloc");
  CK(c->d_ustats.alloc(1), "alloc");
  UploadStats init;
  for (int q = 0; q < 4; q++) init.bad_row[q] = ~0ull;
  init.cmax_bits = init.wmax_bits = init.emax_bits = init.phimax_bits = 0;
  init.wmin_key = ~0ull;
  init.not_f32 = 0;
  c->h_ustats = init;
  if (n > 0) {
    auto h2d = [&](void *d, const void *h, size_t bytes) {
      return cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, st);
    };
    CK(h2d(ox.p, cat->x, 8 * n), "H2D");
    CK(h2d(oy.p, cat->y, 8 * n), "H2D");
    CK(h2d(oz.p, cat->z, 8 * n), "H2D");
    CK(cat->w ? h2d(ow.p, cat->w, 8 * n) : launch_fill_f64(n, 1.0, ow.p, st), "weights");
    // e1 alone carries kappa (which_corr 3, 4)
    CK(cat->e1 ? h2d(oe1.p, cat->e1, 8 * n) : cudaMemsetAsync(oe1.p, 0, 8 * n, st), "e1");
    CK(cat->e2 ? h2d(oe2.p, cat->e2, 8 * n) : cudaMemsetAsync(oe2.p, 0, 8 * n, st), "e2");
    CK(cat->phi ? h2d(ophi.p, cat->phi, 8 * n) : launch_fill_f64(n, -10.0, ophi.p, st), "phi");
    CK(cat->e3 ? h2d(oe3.p, cat->e3, 8 * n) : cudaMemsetAsync(oe3.p, 0, 8 * n, st), "e3");
    CK(p.do_jk ? h2d(ojk.p, cat->jk, 4 * n) : cudaMemsetAsync(ojk.p, 0, 4 * n, st), "labels");
    if (cat->jk_prob) CK(h2d(oprob.p, cat->jk_prob, 8 * n), "H2D");
    CK(h2d(c->d_ustats.p, &c->h_ustats, sizeof(UploadStats)), "H2D");
    PrepIn pin;
    pin.n = n;
    pin.x = ox.p; pin.y = oy.p; pin.z = oz.p; pin.w = cat->w ? ow.p : nullptr;
    pin.e1 = s.has_e ? oe1.p : nullptr; pin.e2 = s.has_e ? oe2.p : nullptr;
    pin.phi = cat->phi ? ophi.p : nullptr; pin.jk_prob = cat->jk_prob ? oprob.p : nullptr;
    pin.jk = p.do_jk ? ojk.p : nullptr;
    pin.e3 = cat->e3 ? oe3.p : nullptr;
    pin.L = L;
    pin.wz_lo = wz_lo(p);
    pin.n_jk = p.n_jk;
    CK(launch_prep_catalog(pin, okeep.p, oflag.p, c->d_ustats.p, st), "catalogue checks");
    c->launches += 1;
    CK(cudaMemcpyAsync(&c->h_ustats, c->d_ustats.p, sizeof(UploadStats), cudaMemcpyDeviceToHost,
                       st), "D2H");
  }
  s.auto_k = c->tune_k == 0;
  const cpc_status built =
      build_cells(c, s, n, s.auto_k ? automatic_cells(c, n) : c->tune_k, nullptr, true);
  return built == CPC_OK ? settle_cells(c) : built;
} catch (...) {
  return host_exception(c);
}

cpc_status cpc_count(cpc_ctx *c, cpc_pair_kind kind, int slot_g1, int slot_g2, cpc_engine engine,
                     int64_t row_stride, int64_t row_offset, cpc_accum *out) try {
  if (!c) return fail(nullptr, CPC_ERR_INVALID, "null context");
  if (busy(c)) return CPC_ERR_STATE;
  if (engine != CPC_ENGINE_FAST && engine != CPC_ENGINE_FP64 && engine != CPC_ENGINE_CELL_FP64)
    return fail(c, CPC_ERR_INVALID, "unknown engine");
  if (kind == CPC_PAIR_SS)
    return fail(c, CPC_ERR_INVALID, "CPC_PAIR_SS pairs one catalogue: use cpc_count_auto");
  // sky: mixed-precision tile kernel (fast) or plain FP64 kernel, both with
  // the FP64 path and the host edge tier for the pairs that can bin
  if (c->p.coordinates == 0) {
    if (engine == CPC_ENGINE_CELL_FP64)
      return fail(c, CPC_ERR_INVALID, "the cell-list FP64 engine counts box pairs only");
    return sky_count(c, kind, slot_g1, slot_g2, row_stride, row_offset, engine, out);
  }
  std::vector<JobPlan> jobs(1);
  cpc_status s = plan_job(c, kind, slot_g1, slot_g2, row_stride, row_offset, out, jobs[0], 0,
                          engine == CPC_ENGINE_FAST);
  if (s != CPC_OK) return s;
  if (engine == CPC_ENGINE_FP64) return run_plain(jobs[0]);
  jobs[0].jd.all_exact = engine == CPC_ENGINE_CELL_FP64 ? 1 : 0;
  return run_fast(jobs);
} catch (...) {
  return host_exception(c);
}

cpc_status cpc_count_async(cpc_ctx *c, cpc_pair_kind kind, int slot_g1, int slot_g2,
                           cpc_engine engine, int64_t row_stride, int64_t row_offset,
                           void *stream) try {
  if (!c) return fail(nullptr, CPC_ERR_INVALID, "null context");
  if (busy(c)) return CPC_ERR_STATE;
  if (engine != CPC_ENGINE_FAST && engine != CPC_ENGINE_FP64)
    return fail(c, CPC_ERR_INVALID, "unknown engine");
  if (kind == CPC_PAIR_SS)
    return fail(c, CPC_ERR_INVALID, "CPC_PAIR_SS pairs one catalogue: use cpc_count_auto");
  if (c->p.coordinates == 0)
    return fail(c, CPC_ERR_INVALID,
                "sky counts finish on the host (edge tier): use cpc_count for coordinates 0");
  cudaStream_t user = reinterpret_cast<cudaStream_t>(stream);
  std::vector<JobPlan> jobs(1);
  cpc_accum placeholder{};  // plan_job checks the output arrays; the real ones come at finish
  int64_t dummy_num = 0;
  double dummy_sums = 0;
  placeholder.num = &dummy_num;
  placeholder.sums = &dummy_sums;
  cpc_status s = plan_job(c, kind, slot_g1, slot_g2, row_stride, row_offset, &placeholder, jobs[0]);
  if (s != CPC_OK) return s;
  jobs[0].out = nullptr;
  // the count follows the caller's earlier work on `stream`
  CK(cudaEventRecord(c->e_in, user), "event");
  CK(cudaStreamWaitEvent(c->st, c->e_in, 0), "stream wait");
  s = engine == CPC_ENGINE_FP64 ? enqueue_plain(jobs[0]) : enqueue_fast(jobs);
  if (s != CPC_OK) return s;
  // and the caller's later work on `stream` follows the count
  CK(cudaEventRecord(c->e_done, c->st), "event");
  CK(cudaStreamWaitEvent(user, c->e_done, 0), "stream wait");
  c->pending = engine == CPC_ENGINE_FP64 ? 2 : 1;
  c->pending_jobs = std::move(jobs);
  return CPC_OK;
} catch (...) {
  return host_exception(c);
}

cpc_status cpc_count_finish(cpc_ctx *c, cpc_accum *out) try {
  if (!c) return fail(nullptr, CPC_ERR_INVALID, "null context");
  if (!c->pending) return fail(c, CPC_ERR_STATE, "no count is pending");
  if (!out || !out->num || !out->sums) return fail(c, CPC_ERR_INVALID, "null output arrays");
  std::vector<JobPlan> jobs = std::move(c->pending_jobs);
  const int mode = c->pending;
  c->pending = 0;
  c->pending_jobs.clear();
  jobs[0].out = out;
  return mode == 2 ? finish_plain(jobs[0]) : finish_fast(jobs, 0);
} catch (...) {
  return host_exception(c);
}

cpc_status cpc_count_auto(cpc_ctx *c, cpc_pair_kind kind, int slot, cpc_engine engine,
                          int64_t row_stride, int64_t row_offset, cpc_accum *out) try {
  if (!c) return fail(nullptr, CPC_ERR_INVALID, "null context");
  if (busy(c)) return CPC_ERR_STATE;
  if (engine != CPC_ENGINE_FAST && engine != CPC_ENGINE_FP64)
    return fail(c, CPC_ERR_INVALID, "unknown engine");
  if (kind != CPC_PAIR_SS && kind != CPC_PAIR_RSRS)
    return fail(c, CPC_ERR_INVALID, "auto pairs: kind must be CPC_PAIR_SS or CPC_PAIR_RSRS");
  if (c->p.data_sorted != 0 && c->p.data_sorted != 1)
    return fail(c, CPC_ERR_INVALID, "auto pairs: data_sorted must be 0 or 1");
  const int mode = c->p.data_sorted == 1 ? 2 : 1;
  if (c->p.coordinates == 0)
    return sky_count(c, kind, slot, slot, row_stride, row_offset, engine, out, mode);
  std::vector<JobPlan> jobs(1);
  cpc_status s = plan_job(c, kind, slot, slot, row_stride, row_offset, out, jobs[0], mode);
  if (s != CPC_OK) return s;
  if (engine == CPC_ENGINE_FP64) return run_plain(jobs[0]);
  return run_fast(jobs);
} catch (...) {
  return host_exception(c);
}

// Pi windows the autotuner tries: for 256, 512 and 1024 threads per block the largest
// window whose histograms fit, and three quarters of it (more, narrower units).
// With coordinates 7 the mu window is automatic (every mu bin when they fit):
// only the cell width is tuned.
std::vector<int> tune_windows(const cpc_params &p, int corel, int unit_w, int twin) {
  std::vector<int> ws;
  if (p.coordinates == 7) return {0};
  const int wmin = twin ? 5 : 8;
  const int jk = p.do_jk ? 1 : 0, nrp = p.n_bins, npi = p.n_p_bin;
  for (int v = 1; v <= 3; v++) {
    const size_t budget =
        fast_block_smem(v) - fast_static_smem_bytes(corel, jk, v, twin) - 1024;
    int w = npi;
    while (w > 1 && fast_smem_bytes(corel, jk, nrp, w, 0, unit_w, twin, v) > budget) w--;
    if (fast_smem_bytes(corel, jk, nrp, w, 0, unit_w, twin, v) > budget) continue;
    for (int cand : {w, (3 * w + 3) / 4}) {
      if (cand < std::min(npi, wmin)) continue;
      if (std::find(ws.begin(), ws.end(), cand) == ws.end()) ws.push_back(cand);
    }
    if (w == npi) break;  // every Pi bin fits: larger blocks gain nothing
  }
  if (ws.empty()) ws.push_back(0);
  return ws;
}

cpc_status cpc_autotune(cpc_ctx *c, cpc_pair_kind kind, int slot_g1, int slot_g2,
                        int64_t sample_stride, int *cells_per_rmax, int *pi_window) try {
  if (!c) return fail(nullptr, CPC_ERR_INVALID, "null context");
  if (busy(c)) return CPC_ERR_STATE;
  const cpc_params &p = c->p;
  if (slot_g1 < 0 || slot_g1 >= kMaxSlots || slot_g2 < 0 || slot_g2 >= kMaxSlots)
    return fail(c, CPC_ERR_INVALID, "slot out of range");
  if (!c->slots[slot_g1].valid || !c->slots[slot_g2].valid)
    return fail(c, CPC_ERR_STATE, "autotune before upload");
  if (c->slots[slot_g1].sky) {  // the sky kernel has no cell or window knobs
    if (cells_per_rmax) *cells_per_rmax = 0;
    if (pi_window) *pi_window = 0;
    return CPC_OK;
  }
  int nh, nb, npb;
  cpc_accum_shape(c, &nh, &nb, &npb);
  std::vector<int64_t> num((size_t)nh * nb * npb);
  std::vector<double> sums(num.size() * kNF);
  cpc_accum acc{};
  acc.num = num.data();
  acc.sums = sums.data();
  const int ks[5] = {2, 3, 4, 5, 6};
  std::vector<int> ws;
  {
    JobRule rule;
    if (job_rule(p, kind, c->slots[slot_g1].n, c->slots[slot_g2].n, rule) != 0)
      return fail(c, CPC_ERR_INVALID, "bad pair kind");
    const int s1 = rule.swapped ? slot_g2 : slot_g1, s2 = rule.swapped ? slot_g1 : slot_g2;
    ws = tune_windows(p, rule.corel, unit_weights(c->slots[slot_g1], c->slots[slot_g2]),
                      twin_job(c, rule, s1, s2, 1, 0, 0) ? 1 : 0);
  }
  // the trials count every sample_stride-th work unit (a unit shard: whole
  // tiles, so each trial's per-unit costs are those of the full count)
  const int64_t stride = std::max<int64_t>(1, sample_stride);
  const int automatic = automatic_cells(c);
  ShardOverride so(c, 0, (int)std::min<int64_t>(stride, 1 << 30));
  TuneTrials trials(c);
  // time of a pair on cells r_max / k (w 0: the automatic window and variant); the
  // first run builds the work units, the next two are timed (the faster counts)
  auto trial = [&](int k, int w, double &t) -> cpc_status {
    cpc_status s;
    t = INFINITY;
    c->tune_k = k;
    c->tune_wpi = w;
    if ((s = set_cells(c, c->slots[slot_g1], k)) != CPC_OK) return s;
    if ((s = set_cells(c, c->slots[slot_g2], k)) != CPC_OK) return s;
    for (int rep = 0; rep < 3; rep++) {
      if (cpc_count(c, kind, slot_g1, slot_g2, CPC_ENGINE_FAST, 1, 0, &acc) != CPC_OK) break;
      if (rep) t = std::min(t, (double)acc.pair_kernel_ms);
    }
    return CPC_OK;
  };
  cpc_status s;
  double untuned, best = INFINITY;
  if ((s = trial(automatic, 0, untuned)) != CPC_OK) return s;
  int bk = automatic, bw = 0;
  for (int k : ks)
    for (int w : ws) {
      double t;
      if ((s = trial(k, w, t)) != CPC_OK) return s;
      if (t < best) {
        best = t;
        bk = k;
        bw = w;
      }
    }
  so.restore();
  if (cells_per_rmax) *cells_per_rmax = bk;
  if (pi_window) *pi_window = bw;
  if (std::min(untuned, best) == INFINITY) return CPC_OK;  // no trial ran: as before
  trials.active = false;
  if (untuned <= best) {  // no pair is faster
    c->tune_k = c->tune_wpi = 0;
    for (Slot &sl : c->slots) sl.auto_k = true;
    return settle_cells(c);
  }
  // keep the best: every box slot on the chosen grid (counts pair slots of one grid)
  c->tune_k = bk;
  c->tune_wpi = bw;
  for (int q = 0; q < kMaxSlots; q++) {
    Slot &sl = c->slots[q];
    if (sl.valid && !sl.sky) {
      const cpc_status s = set_cells(c, sl, bk);
      if (s != CPC_OK) return s;
    }
  }
  return CPC_OK;
} catch (...) {
  return host_exception(c);
}

// The batch of cpc_count_batch on every row_stride-th outer row of each job.
cpc_status count_batch_rows(int n_jobs, cpc_ctx *const *ctxs, const cpc_pair_kind *kinds,
                            const int *slots_g1, const int *slots_g2, cpc_accum *outs,
                            int64_t row_stride) {
  std::map<cpc_ctx *, std::vector<int>> used;  // the slots that each context's jobs read
  for (int k = 0; k < n_jobs; k++) {
    if (ctxs[k]->device != ctxs[0]->device) return fail(ctxs[k], CPC_ERR_INVALID, "batch spans devices");
    for (const int q : {slots_g1[k], slots_g2[k]})
      if (q >= 0 && q < kMaxSlots) used[ctxs[k]].push_back(q);
  }
  for (const auto &u : used) {
    const cpc_status s = same_grid(u.first, u.second);
    if (s != CPC_OK) return s;
  }
  std::vector<JobPlan> jobs(n_jobs);
  for (int k = 0; k < n_jobs; k++) {
    const cpc_status s = plan_job(ctxs[k], kinds[k], slots_g1[k], slots_g2[k], row_stride, 0,
                                  &outs[k], jobs[k], 0, true, true);
    if (s != CPC_OK) return s;
  }
  return run_fast(jobs);
}

cpc_status cpc_autotune_batch(int n_jobs, cpc_ctx *const *ctxs, const cpc_pair_kind *kinds,
                              const int *slots_g1, const int *slots_g2, int64_t sample_stride,
                              int *cells_per_rmax, int *pi_window) try {
  if (n_jobs <= 0 || !ctxs || !kinds || !slots_g1 || !slots_g2)
    return fail(nullptr, CPC_ERR_INVALID, "bad batch arguments");
  for (int k = 0; k < n_jobs; k++) {
    if (!ctxs[k]) return fail(nullptr, CPC_ERR_INVALID, "null context in batch");
    if (busy(ctxs[k])) return CPC_ERR_STATE;
    const cpc_ctx *c = ctxs[k];
    if (slots_g1[k] < 0 || slots_g1[k] >= kMaxSlots || slots_g2[k] < 0 || slots_g2[k] >= kMaxSlots)
      return fail(ctxs[k], CPC_ERR_INVALID, "slot out of range");
    if (!c->slots[slots_g1[k]].valid || !c->slots[slots_g2[k]].valid)
      return fail(ctxs[k], CPC_ERR_STATE, "autotune before upload");
    if (c->slots[slots_g1[k]].sky || c->p.coordinates != ctxs[0]->p.coordinates ||
        c->p.n_bins != ctxs[0]->p.n_bins || c->p.n_p_bin != ctxs[0]->p.n_p_bin ||
        c->p.which_corr != ctxs[0]->p.which_corr)
      return fail(ctxs[k], CPC_ERR_INVALID,
                  "batch autotuning needs box jobs with one binning and which_corr");
  }
  JobRule rule;
  {
    const cpc_ctx *c0 = ctxs[0];
    if (job_rule(c0->p, kinds[0], c0->slots[slots_g1[0]].n, c0->slots[slots_g2[0]].n, rule) != 0)
      return fail(ctxs[0], CPC_ERR_INVALID, "bad pair kind");
  }
  int unit_w = 1, twin = 1;
  for (int k = 0; k < n_jobs; k++) {
    cpc_ctx *c = ctxs[k];
    unit_w &= unit_weights(c->slots[slots_g1[k]], c->slots[slots_g2[k]]);
    JobRule rk;
    if (job_rule(c->p, kinds[k], c->slots[slots_g1[k]].n, c->slots[slots_g2[k]].n, rk) != 0)
      return fail(c, CPC_ERR_INVALID, "bad pair kind");
    const int s1 = rk.swapped ? slots_g2[k] : slots_g1[k], s2 = rk.swapped ? slots_g1[k] : slots_g2[k];
    twin &= twin_job(c, rk, s1, s2, 1, 0, 0) ? 1 : 0;
  }
  const std::vector<int> ws = tune_windows(ctxs[0]->p, rule.corel, unit_w, twin);
  std::vector<std::vector<int64_t>> nums(n_jobs);
  std::vector<std::vector<double>> sums(n_jobs);
  std::vector<cpc_accum> accs(n_jobs);
  for (int k = 0; k < n_jobs; k++) {
    int nh, nb, npb;
    cpc_accum_shape(ctxs[k], &nh, &nb, &npb);
    nums[k].resize((size_t)nh * nb * npb);
    sums[k].resize(nums[k].size() * kNF);
    accs[k] = cpc_accum{};
    accs[k].num = nums[k].data();
    accs[k].sums = sums[k].data();
  }
  // the trials count every sample_stride-th work unit of each context (unit
  // shards: whole tiles, so each trial's per-unit costs are those of the full
  // count)
  const int64_t stride = std::max<int64_t>(1, sample_stride);
  std::vector<int> automatic;  // cell width of each job's context
  for (int k = 0; k < n_jobs; k++) automatic.push_back(automatic_cells(ctxs[k]));
  std::vector<std::unique_ptr<ShardOverride>> sos;
  std::vector<std::unique_ptr<TuneTrials>> trials;
  for (int k = 0; k < n_jobs; k++) {
    bool seen = false;
    for (const auto &so : sos) seen = seen || so->c == ctxs[k];
    if (seen) continue;
    sos.emplace_back(new ShardOverride(ctxs[k], 0, (int)std::min<int64_t>(stride, 1 << 30)));
    trials.emplace_back(new TuneTrials(ctxs[k]));
  }
  // every slot a job reads, on cells r_max / kc (0: each context's automatic width)
  auto regrid = [&](int kc, int w) -> cpc_status {
    for (int k = 0; k < n_jobs; k++) {
      ctxs[k]->tune_k = kc ? kc : automatic[k];
      ctxs[k]->tune_wpi = w;
      for (int sl : {slots_g1[k], slots_g2[k]}) {
        const cpc_status st = set_cells(ctxs[k], ctxs[k]->slots[sl], ctxs[k]->tune_k);
        if (st != CPC_OK) return st;
      }
    }
    return CPC_OK;
  };
  // time of the batch so; the first run builds the work units, the next two are timed
  // (the faster counts)
  auto trial = [&](int kc, int w, double &t) -> cpc_status {
    t = INFINITY;
    const cpc_status s = regrid(kc, w);
    for (int rep = 0; rep < 3 && s == CPC_OK; rep++) {
      if (count_batch_rows(n_jobs, ctxs, kinds, slots_g1, slots_g2, accs.data(), 1) != CPC_OK)
        break;
      if (rep) t = std::min(t, (double)accs[0].pair_kernel_ms);
    }
    return s;
  };
  cpc_status s;
  double untuned, best = INFINITY;
  if ((s = trial(0, 0, untuned)) != CPC_OK) return s;
  int bk = automatic[0], bw = 0;
  for (int kc : {2, 3, 4, 5, 6})
    for (int w : ws) {
      double t;
      if ((s = trial(kc, w, t)) != CPC_OK) return s;
      if (t < best) {
        best = t;
        bk = kc;
        bw = w;
      }
    }
  sos.clear();  // the contexts' own shards again
  if (cells_per_rmax) *cells_per_rmax = bk;
  if (pi_window) *pi_window = bw;
  if (std::min(untuned, best) == INFINITY) return CPC_OK;  // no trial ran: as before
  for (const auto &t : trials) t->active = false;
  if (!(untuned <= best)) return regrid(bk, bw);
  for (int k = 0; k < n_jobs; k++) {  // no pair is faster
    ctxs[k]->tune_k = ctxs[k]->tune_wpi = 0;
    for (Slot &sl : ctxs[k]->slots) sl.auto_k = true;
    if ((s = settle_cells(ctxs[k])) != CPC_OK) return s;
  }
  return CPC_OK;
} catch (...) {
  return host_exception(n_jobs > 0 && ctxs ? ctxs[0] : nullptr);
}

cpc_status cpc_count_batch(int n_jobs, cpc_ctx *const *ctxs, const cpc_pair_kind *kinds,
                           const int *slots_g1, const int *slots_g2, cpc_accum *outs) try {
  if (n_jobs <= 0 || !ctxs || !kinds || !slots_g1 || !slots_g2 || !outs)
    return fail(nullptr, CPC_ERR_INVALID, "bad batch arguments");
  for (int k = 0; k < n_jobs; k++)
    if (busy(ctxs[k])) return CPC_ERR_STATE;
  for (int k = 0; k < n_jobs; k++)
    if (!ctxs[k]) return fail(nullptr, CPC_ERR_INVALID, "null context in batch");
  for (int k = 0; k < n_jobs; k++)
    if (ctxs[k]->p.coordinates == 0) {
      bool one_ctx = true;
      for (int m = 0; m < n_jobs; m++) one_ctx = one_ctx && ctxs[m] == ctxs[0];
      if (one_ctx) {  // the pair types of one sky run: one launch of the fast kernel
        cpc_ctx *c = ctxs[0];
        std::vector<SkyPlan> plans(n_jobs);
        for (int m = 0; m < n_jobs; m++) {
          const cpc_status s = sky_plan(c, kinds[m], slots_g1[m], slots_g2[m], 1, 0,
                                        CPC_ENGINE_FAST, &outs[m], 0, (size_t)m, plans[m]);
          if (s != CPC_OK) return s;
        }
        return sky_run(c, plans, CPC_ENGINE_FAST);
      }
      for (int m = 0; m < n_jobs; m++) {  // sky jobs of several contexts: one launch each
        const cpc_status s = cpc_count(ctxs[m], kinds[m], slots_g1[m], slots_g2[m],
                                       CPC_ENGINE_FAST, 1, 0, &outs[m]);
        if (s != CPC_OK) return s;
      }
      return CPC_OK;
    }
  return count_batch_rows(n_jobs, ctxs, kinds, slots_g1, slots_g2, outs, 1);
} catch (...) {
  return host_exception(n_jobs > 0 && ctxs ? ctxs[0] : nullptr);
}

cpc_status cpc_host_rand_uniform(uint32_t seed, int64_t skip, int64_t n, double *out) try {
  if (n < 0 || skip < 0 || (n > 0 && !out)) return fail(nullptr, CPC_ERR_INVALID, "bad arguments");
  std::vector<int32_t> r(n);
  glibc_rand_stream(seed, skip, n, r.data());
  for (int64_t i = 0; i < n; i++) out[i] = r[i] / (2147483647 + 1.);
  return CPC_OK;
} catch (...) {
  return host_exception(nullptr);
}

cpc_status cpc_host_elip_angle(int64_t n, const double *e1, const double *e2, double *phi) try {
  if (n < 0 || (n > 0 && (!e1 || !e2 || !phi))) return fail(nullptr, CPC_ERR_INVALID, "bad arguments");
  for (int64_t i = 0; i < n; i++) phi[i] = elip_angle(e1[i], e2[i]);
  return CPC_OK;
} catch (...) {
  return host_exception(nullptr);
}

cpc_status cpc_host_rp_thresholds(const cpc_params *p, double *thr) try {
  if (!p || !thr) return fail(nullptr, CPC_ERR_INVALID, "null argument");
  if (p->n_bins <= 0 || p->n_bins > kMaxRp) return fail(nullptr, CPC_ERR_INVALID, "n_bins out of range");
  const int rc = rp_thresholds(p->lin_bin, p->n_bins, p->bin_r_min, p->bin_r_max, thr);
  return rc == 0 ? CPC_OK : fail(nullptr, CPC_ERR_INVALID, "threshold derivation failed");
} catch (...) {
  return host_exception(nullptr);
}

cpc_status cpc_set_shard(cpc_ctx *c, int shard, int n_shards) try {
  if (!c) return fail(nullptr, CPC_ERR_INVALID, "null context");
  if (busy(c)) return CPC_ERR_STATE;
  if (n_shards < 1 || shard < 0 || shard >= n_shards)
    return fail(c, CPC_ERR_INVALID, "shard must satisfy 0 <= shard < n_shards");
  c->shard = shard;
  c->n_shards = n_shards;
  return settle_cells(c);
} catch (...) {
  return host_exception(c);
}

cpc_status cpc_set_graph_replay(cpc_ctx *c, int enable) try {
  if (!c) return fail(nullptr, CPC_ERR_INVALID, "null context");
  if (busy(c)) return CPC_ERR_STATE;
  cudaStreamSynchronize(c->st);
  drop_graph(c);
  c->graph_on = enable ? 1 : 0;
  return CPC_OK;
} catch (...) {
  return host_exception(c);
}

cpc_status cpc_graph_stats(const cpc_ctx *c, int64_t *captures, int64_t *replays) {
  if (!c) return fail(nullptr, CPC_ERR_INVALID, "null context");
  if (captures) *captures = c->graph_captures;
  if (replays) *replays = c->graph_replays;
  return CPC_OK;
}

cpc_status cpc_set_twin(cpc_ctx *c, int enable) try {
  if (!c) return fail(nullptr, CPC_ERR_INVALID, "null context");
  if (busy(c)) return CPC_ERR_STATE;
  c->twin_on = enable ? 1 : 0;
  return CPC_OK;
} catch (...) {
  return host_exception(c);
}

cpc_status cpc_last_twin(const cpc_ctx *c, int *twin) {
  if (!c || !twin) return fail(nullptr, CPC_ERR_INVALID, "null argument");
  *twin = c->last_twin;
  return CPC_OK;
}

cpc_status cpc_launch_count(const cpc_ctx *c, int64_t *launches) {
  if (!c || !launches) return fail(nullptr, CPC_ERR_INVALID, "null argument");
  *launches = c->launches;
  return CPC_OK;
}

cpc_status cpc_host_pi_thresholds(const cpc_params *p, double *thr) try {
  if (!p || !thr) return fail(nullptr, CPC_ERR_INVALID, "null argument");
  if (p->n_p_bin <= 0 || p->n_p_bin > kMaxPi) return fail(nullptr, CPC_ERR_INVALID, "n_p_bin out of range");
  const int rc = pi_thresholds(p->n_p_bin, p->p_min, p->p_max, thr);
  return rc == 0 ? CPC_OK : fail(nullptr, CPC_ERR_INVALID, "threshold derivation failed");
} catch (...) {
  return host_exception(nullptr);
}

}  // extern "C"
