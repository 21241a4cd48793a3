// pair_sky.cu -- sky pair loop (coordinates 0) on the GPU in double precision.
//
// The reference's sky path (corr.cpp:350-423 with lim_calc_sky and
// do_pair_sorted): for each g1 row a window in redshift, Dec and RA computed
// from the distance table (sky_calcs.cpp:105-196); g2 scanned in redshift
// order from the window's lower edge to its upper edge; Dec then RA tests;
// then corel_bin with Pi = DC2 - DC1 (calcs.cpp:126-132) and
// r_p = acos(sin d1 sin d2 + cos d1 cos d2 cos(a1 - a2)) (DA1 + DA2) / 2
// (sky_calcs.cpp:24-31, 91-96), and the jackknife rule jk_check_sky.
//
// Exactness.  The windows, sin/cos of Dec and the angles in radians are
// computed once per galaxy on the host with the C library (exactly the
// reference's values), so every window test and the Pi bin are exact here.
// Only cos(a1 - a2) and acos come from CUDA's math library, whose results can
// differ from the C library's by a few ulps; near sum = 1 acos amplifies that
// by 1/sin(theta).  Each pair gets a rigorous bound on the r_p difference
// (esum on the cosine sum, propagated through acos and the product) and every
// pair whose r_p lies within that bound of a bin threshold, or whose sum lies
// within esum of the reference's clamp at 0.9999999999, is appended to a host
// queue and binned there with the C library.  All other pairs are binned here
// against the exact host-derived thresholds, so the integer counts equal the
// reference's.  D_C is a row of the distance table, so 0.2% of the pairs have
// Pi = 0 exactly, often a bin edge: counts of unit weights recognise them by equal
// D_C (three float parts) and take their bin from the host, else they take the FP64
// path.  Shape sums use CUDA's atan/cos/sin (within 1e-6).
//
// Two kernels:
//  * sky_fp64_kernel -- the plain FP64 kernel: one thread per g1 row, every
//    window pair through the FP64 path, global atomics (CPC_ENGINE_FP64).
//  * sky_tile_kernel -- the fast kernel (CPC_ENGINE_FAST).  Catalogues are held
//    in cell order (jackknife region, keep flag, sky cell of the region,
//    redshift).  A unit is a run of row tiles of one region against the buckets
//    of one partner region: whole buckets outside the tile's windows are
//    skipped, a run of the others is cut to the tile's redshift range, and the
//    block histogram holds one region pair, so the jackknife attribution costs
//    a flush and nothing per pair.  Each warp stages its own candidates,
//    broadcasts them to 32 rows at a time (one per lane) and keeps a bit per
//    test; the surviving pairs are queued by a prefix sum of the bit counts and
//    evaluated 32 at a time with every lane busy: Pi and r_p in FP32 from hi+lo
//    floats, their bins from the linear maps of Pi and log2 r_p with one error
//    bound each (no table lookups), compensated shape terms (pair_df.cuh).
//    Undecided windows and bins go to a queue that sky_finish_kernel evaluates
//    in FP64 (behind it the host tier).
//
//    Counts (RsRd) are bound by instruction issue (81% of issue slots: 34
//    instructions per 32 window tests, 120 per 32 binned pairs), data against
//    randoms by the latency of bucket searches and staging (61%).  Four terms of
//    20k data and 200k randoms, 100 regions, 1.44e9 binned pairs: 113.8 ms before (a
//    warp per row scanning its whole redshift range, every corel in one
//    128-register kernel, the partner's region by global atomics per pair), 29.1 ms
//    now; counts alone 8.4e10 pairs/s.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <climits>

#include "cpc_device.cuh"
#include "field_map.cuh"
#include "kernels.h"
#include "pair_df.cuh"

namespace cpc {

// number of thresholds thr[0..nrp] that are <= v
__device__ inline int thr_count(const JobDev &J, double v) {
  if (!(v >= J.thr[0])) return 0;
  int lo = 0, hi = J.nrp + 1;  // thr[lo] <= v, thr[hi] > v (hi = nrp+1: none)
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (v >= J.thr[mid]) lo = mid; else hi = mid;
  }
  return lo + 1;
}

__global__ void __launch_bounds__(128)
sky_fp64_kernel(const JobDev *__restrict__ jobp, SkyView a, SkyView b, int2 *hq,
                unsigned long long *hq_n, unsigned long long hq_cap, double esum) {
  const JobDev &J = *jobp;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t n1 = a.d.n, n2 = b.d.n;
  if (i >= n1) return;
  if (J.row_stride > 1 && ((a.d.orig[i] - J.row_offset) % J.row_stride) != 0) return;
  // corels1: the scan from row i + 1 must pass the lower redshift bound (sorted)
  if (J.auto_mode == 2 && !(a.d.aflag[i] & kAutoStart0)) return;
  const int64_t oi = a.d.orig[i];
  const double z_min = a.win[i], z_max = a.win[n1 + i];
  const double ra_min = a.win[2 * n1 + i], ra_max = a.win[3 * n1 + i];
  const double dec_min = a.win[4 * n1 + i], dec_max = a.win[5 * n1 + i];
  const double ra1 = a.d.x[i], dec1 = a.d.y[i];
  const double dc1 = a.dc[i], da1 = a.da[i], sd1 = a.sd[i], cd1 = a.cd[i];
  const double rar1 = a.rar[i], decr1 = a.decr[i];
  // first g2 row with redshift >= z_min
  int64_t lo = 0, hi = n2;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (b.d.z[mid] < z_min) lo = mid + 1; else hi = mid;
  }
  const double kClamp = 0.9999999999;        // dA_calc (sky_calcs.cpp:28)
  const double kEps = 2.220446049250313e-16;  // 2^-52
  unsigned long long nwin = 0;
  for (int64_t j = lo; j < n2; j++) {
    const double z2 = b.d.z[j];
    if (z2 > z_max) break;
    if (J.auto_mode && !(b.d.orig[j] > oi)) continue;  // corels1: partners after row i
    const double dec2 = b.d.y[j];
    if (dec2 > dec_max || dec2 < dec_min) continue;
    const double ra2 = b.d.x[j];
    if (ra2 < ra_min || ra2 > ra_max) continue;  // NaN bounds pass, as in the reference
    nwin++;
    // Pi bin (exact)
    const double dP = __dsub_rn(b.dc[j], dc1);
    const double v2 = floor(__ddiv_rn(__dsub_rn(dP, J.pmin), J.ps));
    if (!(v2 >= 0.0) || v2 >= (double)J.npi) continue;
    // great-circle separation
    const double cdel = cos(__dsub_rn(rar1, b.rar[j]));
    const double sum = __dadd_rn(__dmul_rn(sd1, b.sd[j]), __dmul_rn(__dmul_rn(cd1, b.cd[j]), cdel));
    bool amb = fabs(sum - kClamp) <= esum;
    double daR = 0.0, tol = 0.0;
    if (!(sum > kClamp)) {
      const double th = acos(sum);
      daR = __ddiv_rn(__dmul_rn(th, __dadd_rn(da1, b.da[j])), 2.0);
      const double st = sin(th);
      // |d theta| <= esum / sin(theta) + a few ulps of theta (both acos)
      const double rel = esum / fmax(st * th, 1e-300) + 8.0 * kEps;
      tol = 2.0 * daR * rel;
    }
    const int k = thr_count(J, daR);
    if (!amb && tol > 0.0) amb = thr_count(J, daR - tol) != k || thr_count(J, daR + tol) != k;
    if (amb) {
      const unsigned long long q = atomicAdd(hq_n, 1ull);
      if (q < hq_cap) hq[q] = make_int2((int)i, (int)j);
      continue;
    }
    if (k < 1 || k > J.nrp) continue;
    // values (angle_orient_axis_sky, sky_calcs.cpp:13-22) and accumulation
    const double wt = __dmul_rn(a.d.w[i], b.d.w[j]);
    double theta = 0.0;
    if (J.corel != COREL_DD)
      theta = atan((dec2 - dec1) / ((ra2 - ra1) * cos((decr1 + b.decr[j]) / 2.0)));
    double f[kNF];
    pair_values(J.corel, J.gws, wt, theta, PairGal{a.d.e1[i], a.d.e2[i], a.d.phi[i]},
                PairGal{b.d.e1[j], b.d.e2[j], b.d.phi[j]}, f);
    exact_accumulate(J, a.d, i, b.d, j, k - 1, (int)v2, f);
  }
  if (nwin) atomicAdd(&J.counters[1], nwin);
}

// ---------------------------------------------------------------------------
// fast kernel
// ---------------------------------------------------------------------------

constexpr int kSkyThreads = 256;
constexpr int kSkyWarps = kSkyThreads / 32;
// candidate slots per warp: 32 for launches of counts alone; with shapes 16, and
// 24 for the counts beside them, so that three blocks fit an SM
__host__ __device__ constexpr int sky_cand(int set, bool shapes) {
  return set == 0 ? 32 : shapes ? 16 : 24;
}
constexpr int kSkySeg = 256;            // candidate buckets taken at a time
// per-warp ring of pairs awaiting the heavy step: a pass over cand - 1 candidates
// adds at most 32 of them each to fewer than 32 left over
__host__ __device__ constexpr int sky_ring(int cand) { return 32 * cand; }
// pairs a block may add to a bin between flushes: |u| < 2^30 splits into words
// below 2^15 - 7 and low ones within 2^14 + 2^12 (df32.cuh), so 2^16 of them stay
// within a signed 32-bit word
constexpr int kSkyFlushPairs = 1 << 16;
static_assert((long long)kSkyFlushPairs * ((1 << 15) - 7) < 1ll << 31,
              "high words stay within 31 bits");
static_assert((long long)kSkyFlushPairs * ((1 << 14) + (1 << 12)) < 1ll << 31,
              "low words stay within 31 bits");
// The same for counts of unit weights, which have no such words: what is pending and
// the next candidates' pairs, each at most this many, stay within an int.
constexpr int kSkyFlushCounts = 1 << 29;
static_assert(2ll * kSkyFlushCounts <= INT_MAX, "pairs pending in a histogram fit an int");
constexpr unsigned kSkyEdge = 0x8000u;  // queue entry: the window test is undecided

// Jackknife attribution of a sky pair: jk_check_sky (jk.cpp:53-57), each
// region whose galaxy has jk_prob >= 0.5 (same region: g1's only).
__device__ __forceinline__ int sky_regions(int r1, int keep1, int r2, int keep2, int rs[2]) {
  int n = 0;
  if (keep1) rs[n++] = r1;
  if (r2 != r1 && keep2) rs[n++] = r2;
  return n;
}

// n pairs of one bin whose FP64 values sum to f, into the full sample: global FP64
// atomics (rare pairs)
__device__ __forceinline__ void sky_add_full(const JobDev &J, int64_t cell, unsigned n,
                                             const double f[kNF]) {
  const int nf = J.corel == COREL_DD ? 1 : kNF;
  atomicAdd(&J.acc_num[cell], (unsigned long long)n);
  for (int q = 0; q < nf; q++)
    if (f[q] != 0) atomicAdd(&J.acc_sums[cell * kNF + q], f[q]);
}
// A pair's FP64 values into its jackknife regions (corel_jk1, jk.cpp:138-171); i, j:
// redshift-ordered positions.
__device__ __forceinline__ void sky_add_regions(const JobDev &J, int64_t i, int64_t j,
                                                int64_t cell, const double f[kNF]) {
  if (!J.do_jk) return;
  const DCat &a = J.sky1.d, &b = J.sky2.d;
  const int64_t hstride = (int64_t)J.nrp * J.npi;
  int rs[2];
  const int nr = sky_regions(a.jk[i], a.keep[i], b.jk[j], b.keep[j], rs);
  for (int t = 0; t < nr; t++) {
    const int64_t hc = (int64_t)(1 + rs[t]) * hstride + cell;
    atomicAdd(&J.acc_num[hc], 1ull);
    double *sj = J.acc_sums + hc * kNF;
    if (f[0] != 0) atomicAdd(&sj[0], f[0]);
    if (J.which_corr == 0 || J.corel == COREL_DD) continue;
    for (int q = 1; q < kNF; q += 2)
      if (f[q] != 0) atomicAdd(&sj[q], f[q]);
  }
}

// Add x (a term rint(v 2^S_f), |v| 2^S_f < 2^30, or a block's partial sum of
// terms) to the global fixed-point sum of one bin and field: its low 15 bits
// (0 .. 2^15 - 1) into word lo, its arithmetic shift x >> 15 into word hi.
// Terms have |x| < 2^30 and a block's partial sum holds fewer than 2^33 of them,
// so a bin takes 2^48 terms before either word can overflow; the value is
// hi 2^15 + lo (sky_finish_kernel).
__device__ __forceinline__ void fix_add(unsigned long long *lo, unsigned long long *hi,
                                        long long x) {
  const unsigned long long l = (unsigned long long)x & 0x7FFFull;
  const long long h = x >> 15;
  if (l) atomicAdd(lo, l);
  if (h) atomicAdd(hi, (unsigned long long)h);
}

// FP64 path of one window pair whose Pi and r_p may fall in the bins: exact Pi bin,
// great-circle r_p, ambiguity test.  The pair's bin, or -1: none, or left to the host
// tier.  i, j: redshift-ordered positions.
__device__ __forceinline__ int sky_bin_fp64(const JobDev &J, int64_t i, int64_t j,
                                            unsigned long long hq_cap, double esum) {
  const SkyView &a = J.sky1, &b = J.sky2;
  const double dP = __dsub_rn(b.dc[j], a.dc[i]);
  const double v2 = floor(__ddiv_rn(__dsub_rn(dP, J.pmin), J.ps));
  if (!(v2 >= 0.0) || v2 >= (double)J.npi) return -1;
  const double cdel = cos(__dsub_rn(a.rar[i], b.rar[j]));
  const double sum =
      __dadd_rn(__dmul_rn(a.sd[i], b.sd[j]), __dmul_rn(__dmul_rn(a.cd[i], b.cd[j]), cdel));
  const double kClamp = 0.9999999999;
  const double kEps = 2.220446049250313e-16;
  bool amb = fabs(sum - kClamp) <= esum;
  double daR = 0.0, tol = 0.0;
  if (!(sum > kClamp)) {
    const double th = acos(sum);
    daR = __ddiv_rn(__dmul_rn(th, __dadd_rn(a.da[i], b.da[j])), 2.0);
    const double rel = esum / fmax(sin(th) * th, 1e-300) + 8.0 * kEps;
    tol = 2.0 * daR * rel;
  }
  const int k = thr_count(J, daR);
  if (!amb && tol > 0.0) amb = thr_count(J, daR - tol) != k || thr_count(J, daR + tol) != k;
  if (amb) {
    const unsigned long long q = atomicAdd(J.hq_n, 1ull);
    if (q < hq_cap) J.hq[q] = make_int2((int)i, (int)j);
    return -1;
  }
  return k < 1 || k > J.nrp ? -1 : (k - 1) * J.npi + (int)v2;
}
__device__ __forceinline__ void sky_values_fp64(const JobDev &J, int64_t i, int64_t j,
                                                double f[kNF]) {
  const SkyView &a = J.sky1, &b = J.sky2;
  const double wt = __dmul_rn(a.d.w[i], b.d.w[j]);
  double theta = 0.0;
  if (J.corel != COREL_DD)
    theta = atan((b.d.y[j] - a.d.y[i]) /
                 ((b.d.x[j] - a.d.x[i]) * cos((a.decr[i] + b.decr[j]) / 2.0)));
  pair_values(J.corel, J.gws, wt, theta, PairGal{a.d.e1[i], a.d.e2[i], a.d.phi[i]},
              PairGal{b.d.e1[j], b.d.e2[j], b.d.phi[j]}, f);
}

// A pair the mixed-precision path leaves undecided (positions i, j): the exact double
// window first when that test is the undecided one (edge), then the FP64 path.
__device__ __forceinline__ int sky_exact_bin(const JobDev &J, int64_t i, int64_t j, bool edge,
                                             unsigned long long hq_cap, double esum) {
  if (edge) {
    const double *win = J.sky1.win;
    const int64_t n1 = J.sky1.d.n;
    const double z2 = J.sky2.d.z[j], dec2 = J.sky2.d.y[j], ra2 = J.sky2.d.x[j];
    if (z2 < win[i] || z2 > win[n1 + i]) return -1;
    if (dec2 > win[5 * n1 + i] || dec2 < win[4 * n1 + i]) return -1;
    if (ra2 < win[2 * n1 + i] || ra2 > win[3 * n1 + i]) return -1;  // NaN bounds pass
    atomicAdd(&J.counters[1], 1ull);
  }
  return sky_bin_fp64(J, i, j, hq_cap, esum);
}
// The same pair (cell positions i1, j2) binned and added.
__device__ __noinline__ void sky_pair_exact(const JobDev &J, int i1, int j2, bool edge,
                                            unsigned long long hq_cap, double esum) {
  const int64_t i = J.sf1.zidx[i1], j = J.sf2.zidx[j2];
  const int cell = sky_exact_bin(J, i, j, edge, hq_cap, esum);
  if (cell < 0) return;
  double f[kNF];
  sky_values_fp64(J, i, j, f);
  sky_add_full(J, cell, 1, f);
  sky_add_regions(J, i, j, cell, f);
}

// Undecided pairs (about 1 in 10^4, and with weights or shapes those of equal D_C, 1
// in 400) are queued and evaluated by sky_finish_kernel with every lane busy:
// evaluated here, one lane of a warp at a time, they kept the FP64 pipe 62% busy and
// took half of the kernel's time.  Past the queue's end (sized by sky_queue) they
// are evaluated here all the same.
__device__ __forceinline__ void sky_undecided(const JobDev &J, int i1, int j2, bool edge,
                                              unsigned long long hq_cap, double esum) {
  const unsigned long long pos = atomicAdd(J.xq_n, 1ull);
  if (pos < J.xq_cap) J.xq[pos] = make_int2(edge ? ~i1 : i1, j2);
  else sky_pair_exact(J, i1, j2, edge, hq_cap, esum);
}

// first index in [lo, hi) that is not below (below(i): true, then false)
template <class P>
__device__ __forceinline__ int sky_lower_bound(const P &below, int lo, int hi) {
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (below(mid)) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Static shared memory of a block.
struct SkyShared {
  int unit;
  int wcnt[kSkyWarps];
  float red[kSkyTile / 32][6];
  int seg_a[kSkySeg], seg_key[kSkySeg], seg_pre[kSkySeg + 1];
  int key[kSkyThreads];     // bucket key of each staged candidate
  // tile rows, then candidate slots: cell position, third part of D_C (SkyFast::dl)
  int pos[kSkyTile + kSkyThreads];
  float d3[kSkyTile + kSkyThreads];
  int rorig[kSkyTile];      // corels1: input row of each tile row
  float qs[kNF];            // fixed-point scales of the unit's job
  SkyConst k;               // and its constants
};

// Dynamic shared memory before the histogram: the views of the tile rows and of
// the candidate slots (16-byte views su, sw, sl, sx; the windows; with shapes ss,
// sh, sp) and the pair queues
__host__ __device__ constexpr size_t sky_stage_bytes(int set, bool shapes) {
  return (size_t)(kSkyTile + kSkyWarps * sky_cand(set, shapes)) *
             (5 * 16 + 8 + (shapes ? 2 * 16 + 8 : 0)) +
         (size_t)kSkyWarps * sky_ring(sky_cand(set, shapes)) * 2;
}
// Offset of the block histogram: behind the staging of every corel of the launch,
// so that a block that goes from one job's unit to another's finds it zero.
__host__ __device__ constexpr size_t sky_hist_off(int set) {
  return set > 0 && sky_stage_bytes(set, true) > sky_stage_bytes(set, false)
             ? sky_stage_bytes(set, true) : sky_stage_bytes(set, false);
}
// 32-bit words of a bin of the block histogram: the count, then a high and a
// low word per field
__host__ __device__ constexpr int sky_bin_words(int fm, int f0) { return 1 + 2 * (fm - f0); }

// Add the block histogram to the job's global fixed-point block -- the full
// sample, region xreg (the tile's, when its rows are kept) and the partner
// region yreg (each -1: none) -- and zero it.
template <int C>
__device__ __noinline__ void sky_flush(const JobDev &J, unsigned *H, int xreg, int yreg) {
  using F = FieldMap<C>;
  const int ncell = J.nrp * J.npi, f0 = J.unit_w ? 1 : 0;
  const int SW = sky_bin_words(F::FM, f0);
  const bool regf = J.which_corr != 0 && C != COREL_DD;
  const int64_t hx = xreg >= 0 ? (int64_t)(1 + xreg) * ncell : -1;
  const int64_t hy = yreg >= 0 ? (int64_t)(1 + yreg) * ncell : -1;
  for (int c = threadIdx.x; c < ncell; c += kSkyThreads) {
    unsigned *h = H + c * SW;
    const unsigned n = h[0];
    if (!n) continue;
    h[0] = 0u;
    atomicAdd(&J.acc_num[c], (unsigned long long)n);
    if (hx >= 0) atomicAdd(&J.acc_num[hx + c], (unsigned long long)n);
    if (hy >= 0) atomicAdd(&J.acc_num[hy + c], (unsigned long long)n);
    const unsigned bias = n * kMagicBits;
    for (int f = f0; f < F::FM; f++) {
      const int o = 1 + 2 * (f - f0), fld = F::m(f);
      const long long x = fixed_sum(h + o, bias);
      h[o] = 0u;
      h[o + 1] = 0u;
      if (x == 0) continue;
      const bool rf = fld == 0 || ((fld & 1) && regf);
      const int64_t m = (int64_t)c * kNF + fld;
      fix_add(&J.acc_fix[m], &J.acc_fixh[m], x);
      if (rf && hx >= 0) fix_add(&J.acc_fix[hx * kNF + m], &J.acc_fixh[hx * kNF + m], x);
      if (rf && hy >= 0) fix_add(&J.acc_fix[hy * kNF + m], &J.acc_fixh[hy * kNF + m], x);
    }
  }
}

// One unit: a run of row tiles of one (jackknife region, keep flag), up to
// kSkyTile g1 rows each, against the candidate buckets [bk0, bk1) that a tile's
// windows reach, or one of n_slices redshift slices of them.  The buckets are
// those of one partner region where the host can pair the regions up: the
// block histogram then holds one (region, partner region) pair, whose
// attribution is done once per flush instead of per pair.
template <int C, int SET>
__device__ __forceinline__ void sky_unit(const SkyUnit &U, const JobDev &J, unsigned char *smem,
                                         unsigned *H, SkyShared &S, unsigned long long hq_cap,
                                         double esum) {
  using F = FieldMap<C>;
  constexpr bool kShapes = C != COREL_DD;
  constexpr int kCand = sky_cand(SET, kShapes);
  const unsigned FULL = 0xffffffffu;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const unsigned lt_mask = (1u << lane) - 1u;
  // views, the tile rows' at [0, kSkyTile), the candidate slots' behind them
  constexpr int kRec = kSkyTile + kSkyWarps * kCand;
  float4 *v_u = reinterpret_cast<float4 *>(smem);
  float4 *v_w = v_u + kRec, *v_l = v_w + kRec, *v_x = v_l + kRec, *v_b = v_x + kRec;
  float4 *v_s = v_b + kRec, *v_h = v_s + (kShapes ? kRec : 0);
  float2 *v_z = reinterpret_cast<float2 *>(v_h + (kShapes ? kRec : 0));
  float2 *v_p = v_z + kRec;
  constexpr int kRing = sky_ring(kCand);
  unsigned short *wq =
      reinterpret_cast<unsigned short *>(v_p + (kShapes ? kRec : 0)) + wid * kRing;

  // the tile rows' catalogue and the candidates' (flip: g2 and g1)
  const bool flip = J.sk.flip != 0;
  const SkyFast &fa = flip ? J.sf2 : J.sf1, &fb = flip ? J.sf1 : J.sf2;
  const float guard = J.sk.guard, pi_c = J.sk.pi_c, pi_h = J.sk.pi_h, t_hi = J.sk.t_hi;
  if (t < kNF) S.qs[t] = J.qscale[t];
  if (t == 0) S.k = J.sk;
  const int nrp = J.nrp, npi = J.npi, ncell = nrp * npi;
  const int f0 = J.unit_w ? 1 : 0;
  const int SW = sky_bin_words(F::FM, f0);
  const bool jk = J.do_jk != 0, regf = J.which_corr != 0 && kShapes;
  const bool hsm = J.sk.hist_smem != 0;
  const int auto_mode = J.auto_mode;
  const int gws = J.gws;
  const bool uw = J.unit_w != 0, lin = J.lin_bin != 0;
  const int xreg = U.key >> 1;
  const bool xkeep = (U.key & 1) != 0;
  unsigned nwin = 0;
  // an upper bound of the pairs in the histogram, and the regions that take
  // them at the flush (the tile's, the candidates'; -1: none)
  int pending = 0, cur_x = -1, cur_y = -1;
  const int flush_pairs = (F::FM > f0) ? kSkyFlushPairs : kSkyFlushCounts;
  for (int ti = U.tile0; ti < U.tile1; ti++) {
  const SkyTileRows T = J.tiles[ti];
  const int W = (T.count + 31) >> 5;
  // tiles of at most 16 (8) rows: 2 (4) candidate streams per warp
  const int rlanes = T.count <= 8 ? 8 : T.count <= 16 ? 16 : 32;
  const int nsub = 32 / rlanes, sub = lane / rlanes, rl = lane & (rlanes - 1);
  // ---- the tile's rows; slot tr = s * 32 + l holds tile row l * W + s, so the
  // lanes of a pass are spread over the tile ----
  float un[6] = {INFINITY, INFINITY, INFINITY, INFINITY, INFINITY, INFINITY};
  if (t < kSkyTile) {
    const int q = (t & 31) * W + (t >> 5);
    // no row: every window test fails
    float4 b = make_float4(0.f, 0.f, 0.f, 0.f), w = make_float4(0.f, 0.f, INFINITY, 0.f);
    float2 z = make_float2(0.f, -INFINITY);
    if ((t >> 5) < W && q < T.count) {
      int i1 = T.start + q;
      if (J.row_list) i1 = J.row_list[i1];
      v_u[t] = fa.su[i1];
      w = fa.sw[i1];
      v_l[t] = fa.sl[i1];
      v_x[t] = fa.sx[i1];
      S.pos[t] = i1;
      if (!kShapes && uw) S.d3[t] = fa.dl[i1];
      if (kShapes) {
        v_s[t] = fa.ss[i1];
        v_h[t] = fa.sh[i1];
        v_p[t] = fa.sp[i1];
      }
      bool ok = true;
      if (auto_mode) {
        const int zi = fa.zidx[i1];
        S.rorig[t] = (int)J.sky1.d.orig[zi];
        // corels1, sorted: the scan from row i + 1 must pass the lower bound
        if (auto_mode == 2) ok = (J.sky1.d.aflag[zi] & kAutoStart0) != 0;
      }
      if (flip) {
        un[0] = w.x; un[1] = -w.x; un[2] = w.y; un[3] = -w.y; un[4] = w.z; un[5] = -w.z;
      } else if (ok) {
        b = fa.wb[i1];
        z = fa.wz[i1];
        un[0] = b.x - b.y; un[1] = -(b.x + b.y);
        un[2] = b.z - b.w; un[3] = -(b.z + b.w);
        un[4] = z.x - z.y; un[5] = -(z.x + z.y);
      }
    } else {
      v_u[t] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    v_w[t] = w;
    v_b[t] = b;
    v_z[t] = z;
#pragma unroll
    for (int q6 = 0; q6 < 6; q6++) {
      for (int o = 16; o > 0; o >>= 1) un[q6] = fminf(un[q6], __shfl_xor_sync(FULL, un[q6], o));
      if (lane == 0) S.red[wid][q6] = un[q6];
    }
  }
  __syncthreads();
  // the union of the rows' windows (flip: the range of the rows), widened by the
  // guard
  auto uni = [&](int q6) {
    float v = S.red[0][q6];
    for (int w = 1; w < kSkyTile / 32; w++) v = fminf(v, S.red[w][q6]);
    return v;
  };
  const float g2 = 4.0f * guard;
  const float ra_lo = uni(0) - g2, ra_hi = g2 - uni(1), de_lo = uni(2) - g2, de_hi = g2 - uni(3);
  float z_lo = uni(4) - g2, z_hi = g2 - uni(5);
  {  // this unit's redshift slice, half-open (the last one closed by the guard)
    const float d = (z_hi - z_lo) / (float)U.n_slices, z0 = z_lo;
    if (U.slice > 0) z_lo = z0 + d * (float)U.slice;
    if (U.slice + 1 < U.n_slices) z_hi = z0 + d * (float)(U.slice + 1);
  }

  int b0 = U.bk0;
  while (b0 < U.bk1) {
    // ---- the next candidate buckets (in region order) and their runs inside
    // the redshift range ----
    int ns = 0;
    while (b0 < U.bk1 && ns + kSkyThreads <= kSkySeg) {
      const int b = b0 + t;
      int a = 0, e = 0, key = 0;
      if (b < U.bk1) {
        // the bucket's box (flip: the union of its rows' windows)
        const float4 bx = flip ? fb.bk_win[b] : fb.bk_box[b];
        const int4 bk = fb.bk[b];
        key = bk.z;
        if (bx.x <= ra_hi && bx.y >= ra_lo && bx.z <= de_hi && bx.w >= de_lo) {
          if (!flip) {
            a = sky_lower_bound([&](int i) { return fb.zf[i] < z_lo; }, bk.x, bk.y);
            e = sky_lower_bound([&](int i) { return fb.zf[i] < z_hi; }, a, bk.y);
          } else {  // rows whose redshift window reaches the tile (monotone bounds)
            a = sky_lower_bound([&](int i) { return fb.wz[i].x + fb.wz[i].y < z_lo; }, bk.x, bk.y);
            e = sky_lower_bound([&](int i) { return fb.wz[i].x - fb.wz[i].y <= z_hi; }, a, bk.y);
          }
        }
      }
      const unsigned m = __ballot_sync(FULL, e > a);
      if (lane == 0) S.wcnt[wid] = __popc(m);
      __syncthreads();
      int pos = ns + __popc(m & lt_mask), tot = 0;
      for (int w = 0; w < kSkyWarps; w++) {
        const int v = S.wcnt[w];
        if (w < wid) pos += v;
        tot += v;
      }
      if (e > a) {
        S.seg_a[pos] = a;
        S.seg_pre[pos] = e - a;
        S.seg_key[pos] = key;
      }
      ns += tot;
      b0 += kSkyThreads;
      __syncthreads();
    }
    if (wid == 0) {  // exclusive prefix of the run lengths
      int run = 0;
      for (int k0 = 0; k0 < ns; k0 += 32) {
        const int v = k0 + lane < ns ? S.seg_pre[k0 + lane] : 0;
        int s = v;
        for (int o = 1; o < 32; o <<= 1) {
          const int u = __shfl_up_sync(FULL, s, o);
          if (lane >= o) s += u;
        }
        if (k0 + lane < ns) S.seg_pre[k0 + lane] = run + s - v;
        run += __shfl_sync(FULL, s, 31);
      }
      if (lane == 0) S.seg_pre[ns] = run;
    }
    __syncthreads();

    int k = 0;
    while (k < ns) {  // groups of one (region, keep flag); U.all: one of every bucket
      const int key = S.seg_key[k];
      int g = k + 1;
      while (g < ns && (U.all || S.seg_key[g] == key)) g++;
      const int yreg = key >> 1;
      const int gN = S.seg_pre[g] - S.seg_pre[k];
      // jk_check_sky (jk.cpp:53-57): g1's region takes the pair when g1 is kept,
      // g2's when g2 is kept and in another region
      const bool other = yreg != xreg;
      const bool xj = jk && xkeep && (other || !flip);  // (U.all is never flipped)
      const bool yj = jk && (key & 1) != 0 && (other || flip);
      // Where the candidates' region gets its pairs: from the histogram at its
      // flush; or (U.all: few pairs per region pair) each pair adds its own terms
      // to the global block, the candidates of every region in one group.  A
      // flush touches up to ncell bins and a pair's own update a third of one, but
      // a region pair's unit has its fixed cost too (sky_run's choice).
      const bool ydir = !hsm || U.all != 0;
      const int want_x = xj ? xreg : -1, want_y = yj && !ydir ? yreg : -1;
      const int cap = max(kSkyThreads, flush_pairs / T.count);
      for (int base = 0; base < gN; base += cap) {
        const int nc = min(cap, gN - base);
        if (pending &&
            (want_x != cur_x || want_y != cur_y || pending + T.count * nc > flush_pairs)) {
          __syncthreads();
          sky_flush<C>(J, H, cur_x, cur_y);
          pending = 0;
          __syncthreads();
        }
        cur_x = want_x;
        cur_y = want_y;
        if (hsm) pending += T.count * nc;
        // this warp's candidates: positions p = wid (mod nw) of the chunk, in
        // nbw batches of at most kCand - 1 strided over its share (columns and
        // redshifts mixed, so that a warp's pairs fall in different bins)
        const int nw = min(kSkyWarps, max(1, nc >> 3));
        const int share = wid < nw ? (nc - wid + nw - 1) / nw : 0;
        const int nbw = (share + kCand - 2) / (kCand - 1);
        const int c0 = kSkyTile + wid * kCand;
        for (int bw = 0; bw < nbw; bw++) {
          const int nk = (share - bw + nbw - 1) / nbw;
          const int slot = c0 + lane;
          if (lane < nk) {
            const int p = S.seg_pre[k] + base + (lane * nbw + bw) * nw + wid;
            int lo = k, hi = g;  // run lo with pre[lo] <= p < pre[lo + 1]
            while (hi - lo > 1) {
              const int mid = (lo + hi) >> 1;
              if (S.seg_pre[mid] <= p) lo = mid; else hi = mid;
            }
            const int j2 = S.seg_a[lo] + (p - S.seg_pre[lo]);
            S.key[slot - kSkyTile] = S.seg_key[lo];
            S.pos[slot] = j2;
            if (!kShapes && uw) S.d3[slot] = fb.dl[j2];
            v_u[slot] = fb.su[j2];
            v_w[slot] = fb.sw[j2];
            v_l[slot] = fb.sl[j2];
            if (kShapes || !uw) v_x[slot] = fb.sx[j2];
            if (kShapes) {
              v_s[slot] = fb.ss[j2];
              v_h[slot] = fb.sh[j2];
              v_p[slot] = fb.sp[j2];
            }
            if (flip) {
              v_b[slot] = fb.wb[j2];
              v_z[slot] = fb.wz[j2];
            }
            if (auto_mode)  // corels1 (never flipped): the candidate's input row
              v_z[slot].x = __int_as_float((int)J.sky2.d.orig[fb.zidx[j2]]);
          } else if (lane < kCand) {  // no candidate: outside every redshift window
            v_u[slot] = make_float4(0.f, 0.f, 0.f, 0.f);
            v_w[slot] = make_float4(0.f, 0.f, INFINITY, 0.f);
            v_b[slot] = make_float4(0.f, 0.f, 0.f, 0.f);
            v_z[slot] = make_float2(0.f, -INFINITY);  // (as an input row: 0)
          }
          __syncwarp();
          // ---- window tests of every (row, candidate), 32 rows at a time: a
          // candidate is broadcast to the rows of the lanes, a bit per step marks
          // the pairs that may bin.  After a pass each lane queues its pairs
          // (a prefix sum of the bit counts gives its place): one row against
          // candidates spread over the group, which fall in different bins ----
          const int nks = (nk + nsub - 1) / nsub;
          int pass = 0, qhead = 0, qtail = 0;
          for (;;) {
            if (qtail - qhead < 32 && pass < W) {
              const int tr = pass * 32 + rl;
              unsigned mask = 0u, emask = 0u;
              const float4 u1 = v_u[tr], w1 = v_w[tr];
              unsigned bit = 1u;
              if (!flip) {
                const float4 wb = v_b[tr];
                const float2 wz = v_z[tr];
                const float dc1 = w1.w + pi_c;
                const int ro = auto_mode ? S.rorig[tr] : 0;
                const float4 *cp = v_w + c0 + sub;
#pragma unroll 4
                for (int s = 0; s < nks; s++) {
                  const float4 a = cp[0], v = cp[-kRec];  // v_w, v_u
                  // distance inside the window, the smallest of the three
                  const float da = wb.y - fabsf(a.x - wb.x), dd = wb.w - fabsf(a.y - wb.z);
                  const float dr = wz.y - fabsf(a.z - wz.x);
                  const float d = fminf(fminf(da, dd), dr);
                  const float dx = u1.x - v.x, dy = u1.y - v.y, dz = u1.z - v.z;
                  const float c2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                  const float ds = u1.w + v.w;
                  const float tt = c2 * (ds * ds);
                  const float pf = a.w - dc1;
                  bool in = d > guard, edge = fabsf(d) <= guard;
                  if (auto_mode) {  // corels1: partners after the row
                    const bool ord = __float_as_int(v_z[c0 + sub + s * nsub].x) > ro;
                    in = in && ord;
                    edge = edge && ord;
                  }
                  if (in) nwin++;
                  if (in && fabsf(pf) <= pi_h && tt < t_hi) mask |= bit;
                  if (edge) emask |= bit;
                  bit += bit;
                  cp += nsub;
                }
              } else {  // the candidates' windows against the row
                const float dc2 = w1.w - pi_c;
                const float4 *cp = v_u + c0 + sub;
                const float2 *zp = v_z + c0 + sub;
#pragma unroll 4
                for (int s = 0; s < nks; s++) {
                  const float4 v = cp[0], wb = cp[4 * kRec];  // v_u, v_b
                  const float2 wz = zp[0];
                  const float dc1 = cp[kRec].w;               // v_w
                  const float da = wb.y - fabsf(w1.x - wb.x), dd = wb.w - fabsf(w1.y - wb.z);
                  const float dr = wz.y - fabsf(w1.z - wz.x);
                  const float d = fminf(fminf(da, dd), dr);
                  const float dx = u1.x - v.x, dy = u1.y - v.y, dz = u1.z - v.z;
                  const float c2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                  const float ds = u1.w + v.w;
                  const float tt = c2 * (ds * ds);
                  const float pf = dc2 - dc1;
                  const bool in = d > guard;
                  if (in) nwin++;
                  if (in && fabsf(pf) <= pi_h && tt < t_hi) mask |= bit;
                  if (fabsf(d) <= guard) emask |= bit;
                  bit += bit;
                  cp += nsub;
                  zp += nsub;
                }
              }
              const int cnt = __popc(mask) + __popc(emask);
              int sum = cnt;
              for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(FULL, sum, o);
                if (lane >= o) sum += u;
              }
              unsigned pos = (unsigned)(qtail + sum - cnt);  // qtail < 2 kRing
              if (pos >= kRing) pos -= kRing;
              const unsigned en = (unsigned)tr | (unsigned)(sub << 7);
              while (mask) {
                const int s = 31 - __clz(mask);
                mask ^= 1u << s;
                wq[pos] = (unsigned short)(en + ((unsigned)(s * nsub) << 7));
                if (++pos == kRing) pos = 0;
              }
              while (emask) {
                const int s = 31 - __clz(emask);
                emask ^= 1u << s;
                wq[pos] = (unsigned short)((en + ((unsigned)(s * nsub) << 7)) | kSkyEdge);
                if (++pos == kRing) pos = 0;
              }
              qtail += __shfl_sync(FULL, sum, 31);
              pass++;
              __syncwarp();
              continue;
            }
            const int take = min(32, qtail - qhead);
            if (take == 0) break;
            if (lane < take) {
              // ---- heavy step for one queued pair ----
              const int qp = qhead + lane;
              const unsigned en = wq[qp >= kRing ? qp - kRing : qp];
              const int er = en & 127, ec = c0 + ((en >> 7) & 31);
              const int a1 = flip ? ec : er, a2 = flip ? er : ec;  // g1, g2
              const float4 u1 = v_u[a1], l1 = v_l[a1], u2 = v_u[a2], l2 = v_l[a2];
              const float4 w1 = v_w[a1], w2 = v_w[a2];
              // Pi from hi + lo comoving distances, its bin from the linear map
              const float pf = (w2.w - w1.w) + (l2.w - l1.w);
              const float v2 = fmaf(pf, S.k.pi_s, S.k.pi_o);
              const float m2 = v2 + kMagic;
              int n2 = __float_as_int(m2) - (int)kMagicBits;
              bool pi_ok = fabsf(v2 - (m2 - kMagic)) <= S.k.pi_in;
              // equal D_C (all three parts: common, as D_C is a distance-table row): Pi is
              // exactly 0, here a bin edge.  Where the pair adds a count and nothing else,
              // its bin is all there is to know; other pairs' values stay FP64
              if (!kShapes && uw && !pi_ok && pf == 0.0f && w1.w == w2.w && l1.w == l2.w &&
                  S.d3[a1] == S.d3[a2]) {
                n2 = S.k.pi_zero;
                pi_ok = true;
              }
              // chord of the hi + lo unit vectors; (2 asin(c / 2))^2 as its series
              // (c^2 <= 1/16: the first omitted term is 5e-9 of the sum)
              const float dx = (u1.x - u2.x) + (l1.x - l2.x);
              const float dy = (u1.y - u2.y) + (l1.y - l2.y);
              const float dz = (u1.z - u2.z) + (l1.z - l2.z);
              const float c2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
              float th2 = fmaf(c2, fmaf(c2, fmaf(c2, 1.0f / 560.0f, 1.0f / 90.0f), 1.0f / 12.0f),
                               1.0f) * c2;
              if (c2 > 0.0625f) {
                // (within 0.32 rad of the antipode the chord's rounding is too much of
                // theta: undecided)
                const float th = 2.0f * asinf(0.5f * sqrtf(c2));
                th2 = c2 < 3.9f ? th * th : __int_as_float(0x7fc00000);
              }
              const float ds = u1.w + u2.w;
              const float r4 = th2 * (ds * ds);  // (2 r_p)^2
              const float v1 = lin ? fmaf(sqrtf(r4), S.k.rp_s, S.k.rp_o)
                                   : fmaf(__log2f(r4), S.k.rp_s, S.k.rp_o);
              const float m1 = v1 + kMagic;
              const int n1 = __float_as_int(m1) - (int)kMagicBits;
              // undecided: near a Pi or r_p edge, or a separation so small that
              // the reference's own rounding of cos theta matters
              const float tt = c2 * (ds * ds);
              const bool amb =
                  !(pi_ok && fabsf(v1 - (m1 - kMagic)) <= S.k.rp_in && c2 >= 1e-8f) &&
                  tt >= S.k.t_lo;
              bool bin = tt >= S.k.t_lo && (unsigned)n1 < (unsigned)nrp && (unsigned)n2 < (unsigned)npi;
              bool exact = amb || (en & kSkyEdge);
              df32 X{0.f, 0.f}, ddec{0.f, 0.f};
              float4 x1, x2;
              if (kShapes || !uw) {
                x1 = v_x[a1];
                x2 = v_x[a2];
              }
              float4 h1, h2;
              if (kShapes && bin && !exact) {
                // tangent-plane separation: X = dRA cos(mean Dec), Y = dDec (hi + lo
                // degrees; the cosine from the half angles), as double-floats
                h1 = v_h[a1];
                h2 = v_h[a2];
                const df32 dra = df_diff_hl(w2.x, x2.x, w1.x, x1.x);
                ddec = df_diff_hl(w2.y, x2.y, w1.y, x1.y);
                const df32 cm = df_sub(df_mul(df32{h1.x, h1.y}, df32{h2.x, h2.y}),
                                       df_mul(df32{h1.z, h1.w}, df32{h2.z, h2.w}));
                X = df_mul(dra, cm);
                // coincident on the sky: atan(0/0), the FP64 path
                exact = X.h == 0.0f && ddec.h == 0.0f;
              }
              if (exact) {
                sky_undecided(J, S.pos[a1], S.pos[a2], (en & kSkyEdge) != 0, hq_cap, esum);
              } else if (bin) {
                const int cell = n1 * npi + n2;
                float v[kNF];
                df32 vd[kNF];
                if (!uw) v[0] = x1.w * x2.w;
                if (kShapes) {
                  // theta = atan(dDec / (dRA cos(mean Dec))) (sky_calcs.cpp:13-22)
                  df32 c, sn;
                  df_cos_sin_2theta(X, ddec, c, sn);
                  const float theta = atanf(__fdividef(ddec.h, X.h));
                  const float4 e1 = v_s[a1], e2 = v_s[a2];
                  const float2 p1 = v_p[a1], p2 = v_p[a2];
                  const DfGal g1{{e1.x, e1.z}, {e1.y, e1.w}, {x1.w, p1.y}, p1.x};
                  const DfGal g2{{e2.x, e2.z}, {e2.y, e2.w}, {x2.w, p2.y}, p2.x};
                  df_pair_terms<C>(c, sn, theta, g1, g2, gws, uw, vd, v);
                }
                unsigned wh[F::FM], wl[F::FM];
#pragma unroll
                for (int f = 0; f < F::FM; f++) {
                  if (f < f0) continue;
                  const int q = F::m(f);
                  if (df_field(C, q)) df_to_words(vd[q], S.qs[q], wh[f], wl[f]);
                  else f_to_words(v[q], S.qs[q], wh[f], wl[f]);
                }
                auto term = [&](int f) {  // the integer rint(v 2^S)
                  return (long long)((int)(wh[f] - kMagicBits) * 32768 + (int)(wl[f] - kMagicBits));
                };
                if (hsm) {
                  unsigned *h = H + cell * SW;
                  atomicAdd(h, 1u);
                  // even lanes add the high word first, odd lanes the low word, so
                  // lanes that hit one bin split over two banks
                  const bool odd = (lane & 1) != 0;
                  unsigned *ha = h + 1 - 2 * f0 + (odd ? 1 : 0), *hb = h + 2 - 2 * f0 - (odd ? 1 : 0);
#pragma unroll
                  for (int f = 0; f < F::FM; f++) {
                    if (f < f0) continue;
                    atomicAdd(ha + 2 * f, odd ? wl[f] : wh[f]);
                    atomicAdd(hb + 2 * f, odd ? wh[f] : wl[f]);
                  }
                }
                // straight to the global block: the partner's region of a sparse
                // group; with no room for a block histogram, everything
                auto direct = [&](int64_t h0, bool all) {
                  atomicAdd(&J.acc_num[h0 + cell], 1ull);
#pragma unroll
                  for (int f = 0; f < F::FM; f++) {
                    const int q = F::m(f);
                    if (f < f0 || !(all || q == 0 || ((q & 1) && regf))) continue;
                    const int64_t o = (h0 + cell) * kNF + q;
                    fix_add(&J.acc_fix[o], &J.acc_fixh[o], term(f));
                  }
                };
                if (!hsm) {
                  direct(0, true);
                  if (xj) direct((int64_t)(1 + xreg) * ncell, false);
                }
                if (ydir && jk) {
                  const int ky = S.key[ec - kSkyTile], yr = ky >> 1;
                  if ((ky & 1) && (yr != xreg || flip)) direct((int64_t)(1 + yr) * ncell, false);
                }
              }
            }
            qhead += take;
            if (qhead >= kRing) {
              qhead -= kRing;
              qtail -= kRing;
            }
            __syncwarp();
          }
          __syncwarp();  // every lane is done with the slots before restaging
        }
      }
      k = g;
    }
    __syncthreads();  // the run tables are free
  }
  __syncthreads();  // the row slots are free
  }
  if (pending) sky_flush<C>(J, H, cur_x, cur_y);
  {
    unsigned v = nwin;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(FULL, v, o);
    if (lane == 0 && v) atomicAdd(&J.counters[1], (unsigned long long)v);
  }
}

// Every job of a launch: the units of all jobs in one queue.  SET: the corels
// the instantiation holds (0 density_density; 1 also shape_density; 2 also
// shape_shape), so that a run of counts alone keeps few registers.
template <int SET, int MINB>
__global__ void __launch_bounds__(kSkyThreads, MINB)
sky_tile_kernel(const JobDev *__restrict__ jobs, const SkyUnit *__restrict__ units, int n_units,
                unsigned long long *ctr, unsigned long long hq_cap, double esum, int hist_off,
                int hist_words) {
  extern __shared__ __align__(16) unsigned char sky_smem[];
  __shared__ SkyShared S;
  unsigned *H = reinterpret_cast<unsigned *>(sky_smem + hist_off);
  for (int k = threadIdx.x; k < hist_words; k += kSkyThreads) H[k] = 0u;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) S.unit = (int)atomicAdd(ctr, 1ull);
    __syncthreads();
    const int u = S.unit;
    if (u >= n_units) break;
    const SkyUnit U = units[u];
    const JobDev &J = jobs[U.job];
    const int C = J.corel;
    if (SET == 0 || C == COREL_DD) {
      sky_unit<COREL_DD, SET>(U, J, sky_smem, H, S, hq_cap, esum);
    } else if (SET >= 1 && C == COREL_SD) {
      sky_unit<COREL_SD, SET>(U, J, sky_smem, H, S, hq_cap, esum);
    } else if (SET >= 2) {
      if (C == COREL_SS) sky_unit<COREL_SS, SET>(U, J, sky_smem, H, S, hq_cap, esum);
      else sky_unit<COREL_SSA, SET>(U, J, sky_smem, H, S, hq_cap, esum);
    }
  }
}

// Per job, after the pair kernel: the undecided pairs on the FP64 path, and
// the fixed-point block added to the FP64 sums, sums[i] += (hi[i] 2^15 + lo[i])
// 2^-S_f, f = i mod kNF (fix_add).
__global__ void sky_finish_kernel(int64_t n, const unsigned long long *__restrict__ lo,
                                  const unsigned long long *__restrict__ hi,
                                  double *__restrict__ sums, const JobDev *__restrict__ jobp,
                                  unsigned long long hq_cap, double esum) {
  const JobDev &J = *jobp;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  // The pairs of equal D_C fall in one Pi bin: a warp adds its pairs of one bin
  // together, else the few addresses of that bin's full sample take turns, 2.5 ns
  // a pair (100k x 1M shape x density, 6.6e6 such pairs: 114 ms in all, added so 102).
  // A few thousand pairs do not wait longer than the adding takes (8 us a job).
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const bool shapes = J.corel != COREL_DD;
  const int64_t nx = (int64_t)min(*J.xq_n, J.xq_cap);
  const bool together = nx >= 8192;
  for (int64_t base = i0 - lane; base < nx; base += step) {
    int cell = -1;
    double f[kNF];
    for (int q = 0; q < kNF; q++) f[q] = 0.0;
    if (base + lane < nx) {
      const int2 e = J.xq[base + lane];
      const bool edge = e.x < 0;
      const int64_t i = J.sf1.zidx[edge ? ~e.x : e.x], j = J.sf2.zidx[e.y];
      cell = sky_exact_bin(J, i, j, edge, hq_cap, esum);
      if (cell >= 0) {
        sky_values_fp64(J, i, j, f);
        sky_add_regions(J, i, j, cell, f);
      }
    }
    unsigned same = together ? __match_any_sync(FULL, cell) : 1u << lane;
    if (cell < 0) same = 0u;
    const bool first = same && lane == __ffs(same) - 1;
    // the first lane of a bin adds the others' values, one of them a turn
    unsigned rest = first ? same & (same - 1) : 0u;
    while (__any_sync(FULL, rest != 0u)) {
      const int l = rest ? __ffs(rest) - 1 : lane;
      const bool add = rest != 0u;
#pragma unroll
      for (int q = 0; q < kNF; q++) {
        if (q > 0 && !shapes) break;
        const double v = __shfl_sync(FULL, f[q], l);
        if (add) f[q] += v;
      }
      rest &= rest - 1;
    }
    if (first) sky_add_full(J, cell, __popc(same), f);
  }
  for (int64_t i = i0; i < n; i += step) {
    const unsigned long long l = lo[i];
    const long long h = (long long)hi[i];
    if (l != 0 || h != 0)
      atomicAdd(&sums[i], fma((double)h, 32768.0, (double)l) * J.inv_qscale[i % kNF]);
  }
}

cudaError_t launch_sky_finish(int64_t n, const unsigned long long *lo,
                              const unsigned long long *hi, double *sums, const JobDev *job,
                              unsigned long long hq_cap, double esum, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const int64_t blocks = std::min<int64_t>((n + 255) / 256, 4096);
  sky_finish_kernel<<<(unsigned)blocks, 256, 0, st>>>(n, lo, hi, sums, job, hq_cap, esum);
  return cudaGetLastError();
}

// Words of the block histogram a job of this corel needs, and whether the
// histogram (behind the staging buffers) fits a block at two blocks per SM.
size_t sky_hist_words(int corel, int unit_w, int ncell) {
  const int fm = corel == COREL_DD ? FieldMap<COREL_DD>::FM
                 : corel == COREL_SD ? FieldMap<COREL_SD>::FM
                 : corel == COREL_SS ? FieldMap<COREL_SS>::FM : FieldMap<COREL_SSA>::FM;
  return (size_t)sky_bin_words(fm, unit_w ? 1 : 0) * ncell;
}
bool sky_hist_fits(int corel, int unit_w, int ncell) {
  return sky_hist_off(corel == COREL_DD ? 0 : 1) + 4 * sky_hist_words(corel, unit_w, ncell) +
             sizeof(SkyShared) + 1024 <= (size_t)(228 * 1024) / 2;
}

template <int SET, int MINB>
static cudaError_t launch_sky_t(const JobDev *jobs, const SkyUnit *units, int n_units,
                                size_t hist_words, unsigned long long *ctr,
                                unsigned long long hq_cap, double esum, int sm_count,
                                cudaStream_t st) {
  auto kern = sky_tile_kernel<SET, MINB>;
  const size_t off = sky_hist_off(SET), smem = off + 4 * hist_words;
  cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int bps = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kern, kSkyThreads, smem);
  if (e != cudaSuccess) return e;
  if (bps < 1) return cudaErrorInvalidConfiguration;
  const int grid = (int)std::min<long long>((long long)sm_count * bps, n_units);
  kern<<<grid, kSkyThreads, smem, st>>>(jobs, units, n_units, ctr, hq_cap, esum, (int)off,
                                        (int)hist_words);
  return cudaGetLastError();
}

cudaError_t launch_sky_tile(const JobDev *jobs, const SkyUnit *units, int n_units, int set,
                            size_t hist_words, unsigned long long *ctr,
                            unsigned long long hq_cap, double esum, int sm_count,
                            cudaStream_t st) {
  if (n_units <= 0) return cudaSuccess;
  if (set == 0)
    return launch_sky_t<0, 4>(jobs, units, n_units, hist_words, ctr, hq_cap, esum, sm_count, st);
  if (set == 1)
    return launch_sky_t<1, 3>(jobs, units, n_units, hist_words, ctr, hq_cap, esum, sm_count, st);
  return launch_sky_t<2, 2>(jobs, units, n_units, hist_words, ctr, hq_cap, esum, sm_count, st);
}

cudaError_t launch_sky_fp64(const JobDev *job, const SkyView &a, const SkyView &b, int2 *hq,
                            unsigned long long *hq_n, unsigned long long hq_cap, double esum,
                            cudaStream_t st) {
  const int64_t blocks = (a.d.n + 127) / 128;
  if (blocks == 0) return cudaSuccess;
  sky_fp64_kernel<<<(unsigned)blocks, 128, 0, st>>>(job, a, b, hq, hq_n, hq_cap, esum);
  return cudaGetLastError();
}

}  // namespace cpc
