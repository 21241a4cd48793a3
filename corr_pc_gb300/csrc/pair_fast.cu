// pair_fast.cu -- the mixed-precision pair-counting kernel (sm_103a).
//
// One persistent launch drains a device work queue of "units".  A unit is a
// tile of up to kTile g1 rows from one (column, jackknife region) bucket and
// z-chunk, paired with every g2 candidate of the neighbouring columns inside
// the unit's shifted-z range.  A block keeps the tile's rows in shared memory;
// each warp stages its own batches of candidates and tests them against every
// row, in W passes of 32 rows (one row per lane; the lanes of a warp are spread
// over the tile).  Candidates are strided over their (partner region, image
// shift) group, so that a batch mixes columns and redshifts.
//
// Light pass (every candidate, broadcast to 32 rows): FP32 separations with the
// image shift applied exactly; the distance inside the reference's window is
// one number, compared with a guard both ways, and a bit per step keeps the
// pairs that may bin.  After a pass each lane queues its pairs (a prefix sum of
// the bit counts).  Heavy step (32 queued pairs, all lanes busy): r_p and Pi bins
// from linear maps of Pi and log2 r^2 with an error bound each, shape values,
// histogram updates.
//
// Measured (GB300, before -> now): kernel of the 200k wg+ box 17.9 -> 13.5 ms,
// kappa 11.6 -> 7.3, ED 7.0 -> 4.1; w++ twin of 2M points 567 -> 420, weighted w++
// (60k x 151k) 6.9 -> 5.2, 12 uneven w++ boxes 58 -> 25; wgg of 20,000 points
// 0.36 -> 0.12.  What gave it: one bit per test instead of a queue push per step
// (67 -> 24 instructions a step), maps instead of band tables, records of words
// at constant offsets added with their bias (no split of the fixed-point term),
// four-way order of the reductions, unit set-up by scans instead of serial
// loops, no barrier per thousand candidates, blocks of 512 and 1024 threads
// that share a wider histogram, and units cut by a model of their cost (capi.cu).  Bound now by the shared-memory reductions for
// the shape corels (74-78% of the pipe: a bin's pairs are serialised, see
// order4) and by instruction issue (87%) for kappa, ED and counts.
//
// Precision: a pair is resolved on this path only when it is farther than a
// rigorous error bound from every decision boundary (the r_p / Pi window,
// every r_p and Pi bin edge); otherwise it is appended to an edge queue and
// re-evaluated with the reference's exact double-precision arithmetic
// (recheck_kernel), so integer counts are bit-identical with the reference.
//
// Accumulation: block-private histograms over (r_p bin, block-local Pi window)
// in shared memory -- the full sample ("main"), the cross-region pairs that the
// tile's own jackknife region does NOT take ("NX": that region's sums are main
// minus NX, so the pairs it takes, most of them, cost no update of their own) and
// one other region ("Y", the partner's region for cross-region pairs); the corels
// of few fields keep a main histogram per attribution instead (by_class) -- with
// 32-bit counts and fixed-point sums split over two 32-bit words per field
// (exact integer addition, order independent), flushed to the FP64 global
// histogram block when the pairs added since the last flush could overflow a
// word (below) and at the end of the unit.  The terms of the fields whose sums
// cancel (rotated ellipticities and their products, kappa) are computed in
// compensated single precision (pair_df.cuh) and quantised at 2^-29 of their
// bound, so every bin sum matches the reference's double-precision sum to
// about 1e-9 of the field's bound.
#include <cuda_runtime.h>
#include <stdint.h>
#include <atomic>
#include <climits>

#include "cpc_device.cuh"
#include "field_map.cuh"
#include "kernels.h"
#include "pair_df.cuh"

namespace cpc {

constexpr int kTile = kTileThreads;          // g1 rows per tile
// Kernel variants: block size and blocks per SM (32 warps per SM at 64 registers;
// the FP64 comparison engine 16 at 128).  Wider blocks share a histogram among
// more warps, which widens its Pi window (choose_variant chooses).
__host__ __device__ constexpr int variant_threads(int v) { return v == 3 ? 1024 : v == 2 ? 512 : 256; }
__host__ __device__ constexpr int variant_blocks(int v) { return v == 3 ? 1 : v == 1 ? 4 : 2; }
constexpr int kMaxSeg = kFastMaxSeg;
constexpr int kMaxCols = kFastMaxCols;
static_assert(kMaxSeg == 256, "one candidate slot per thread");
// Candidate slots per warp: 32; 16 for the corels with many fields, whose
// staging and queue come out of the Pi window's shared memory (kappa with 32
// instead of 16: 8.6 -> 7.6 ms on the 200k box; weighted w++: 5.4 -> 6.0).  A
// warp's queue takes a pass over cand - 1 candidates, at most 32 pairs each, and
// fewer than 32 left over.
__host__ __device__ constexpr int cand_slots(int corel) {
  return corel == COREL_SD || corel == COREL_SS || corel == COREL_SSA ? 16 : 32;
}
__host__ __device__ constexpr int ring_size(int corel) { return 32 * cand_slots(corel); }

// Dynamic shared memory of the candidate staging: positions, then (for the
// corels with values) the weighted ellipticities or orientation and the aux
// view (x lo, y lo, phi, w lo) of each staged candidate, and the pair queues.
__host__ __device__ constexpr size_t stage_bytes(int corel, int warps) {
  return sizeof(float4) * (corel == COREL_DD ? 1 : 3) * warps * cand_slots(corel) +
         (corel == COREL_ED ? sizeof(float) * (warps * cand_slots(corel) + kTile) : 0) +  // z lo
         sizeof(unsigned short) * warps * ring_size(corel);
}
// Dynamic shared memory of the corels1 (auto pair) rules, after the staging:
// each staged candidate's input index and each row's thresholds per z image.
__host__ __device__ constexpr size_t auto_bytes(int corel, int warps) {
  return sizeof(int) * (warps * cand_slots(corel) + 3 * kTile);
}

// Block histograms: one record of 32-bit words per (r_p bin, window Pi bin) --
// the pair count, then per field a high and a low word (df_to_words) -- so that a
// pair's words are at compile-time offsets from one address.  Records have an
// odd number of words: the records' banks spread like their indices.  Twin jobs
// append the other order's order-dependent fields to the main record.  Unit
// weights (f0 = 1): field 0, equal to the count, has no words.
__host__ __device__ constexpr int rec_words(int fields, int f0, int fa) {
  return 1 + 2 * (fields - f0 + fa);
}

// With jackknife, the corels of few fields keep four main histograms a block, by
// which of its two regions take the pair (the tile's 1, the partner's 2): a pair adds one
// record instead of up to three, and pairs of one bin fall on four.  200k box:
// kappa 7.6 -> 7.3 ms, ED 4.27 -> 4.14.  Where the records are long the window
// pays: with the four, auto pairs of shapes 6.3 -> 6.9, weighted w++ 5.15 -> 5.07, wg+
// 13.5 -> 13.3; twin jobs would need sixteen.
__host__ __device__ constexpr bool by_class(int corel, int jk, int twin) {
  return jk && !twin && corel != COREL_SD && corel != COREL_SS && corel != COREL_SSA;
}
// Words from one class's record of a bin to the next class's: 8 banks on.
__host__ __device__ constexpr int class_stride(int words) { return words + ((8 - words) & 31); }

// Fields of a corel's main and region records.
static void record_fields(int corel, int *FM, int *FJ) {
  *FM = 1, *FJ = 1;
  if (corel == COREL_SD) { *FM = 7; *FJ = 4; }
  if (corel == COREL_SS) { *FM = 11; *FJ = 6; }
  if (corel == COREL_SSA) { *FM = 13; *FJ = 7; }
  if (corel == COREL_DK) { *FM = 2; *FJ = 2; }
  if (corel == COREL_SK) { *FM = 4; *FJ = 4; }
  if (corel == COREL_ED) { *FM = 3; *FJ = 2; }
}
// Bytes of a wpi-bin window of nrp r_p bins as one main record and two (twin: four)
// region records a bin: the measure by which a set window is too wide.
size_t fast_window_bytes(int corel, int do_jk, int nrp, int wpi, int unit_w, int twin) {
  int FM, FJ;
  record_fields(corel, &FM, &FJ);
  const int f0 = unit_w ? 1 : 0, FA = twin && corel == COREL_SS ? FieldMap<COREL_SS>::FA : 0;
  return 4ull * nrp * wpi *
         (rec_words(FM, f0, FA) + (do_jk ? rec_words(FJ, f0, 0) * (twin ? 4 : 2) : 0));
}
// Shared-memory bytes a block needs for a job: the staging, then the histograms
// (linear in wpi).
size_t fast_smem_bytes(int corel, int do_jk, int nrp, int wpi, int auto_pairs, int unit_w,
                       int twin, int variant) {
  const int warps = variant_threads(variant) / 32;
  const size_t b = stage_bytes(corel, warps) + (auto_pairs ? auto_bytes(corel, warps) : 0);
  if (!by_class(corel, do_jk, twin))
    return b + fast_window_bytes(corel, do_jk, nrp, wpi, unit_w, twin);
  int FM, FJ;
  record_fields(corel, &FM, &FJ);
  return b + 16ull * (nrp * wpi * rec_words(FM, unit_w ? 1 : 0, 0) + 31);
}

// Fixed-point sums in 32-bit shared words.  A term v of field f becomes the
// integer u = rint(v * 2^S_f), |u| < 2^29 (S_f from a bound on |v|), split into
// a high part of at most 2^14 and a signed low part of at most kLowTerm, each
// added with its bias (df_to_words) to its own 32-bit word with a plain
// reduction (no return value: no scoreboard wait).  A bin takes at most kBinTerms
// pairs between flushes, so that a word, read as a signed integer after its
// bin's count of biases is taken off, stays within 2^31 (df32.cuh): a block keeps a bound
// on the fullest bin (its last known maximum plus every pair tested since),
// finds the maximum when the bound could pass kBinTerms and flushes when the
// maximum itself could.  (Bounding the block's pair total instead flushed
// almost every thousand candidates.)
// Candidates a bin bound takes at a time: half of kBinTerms for a full tile
constexpr int kChunkTests = 1 << 16;
static_assert(kChunkTests <= kBinTerms, "a chunk fits a bin's words after a flush");
// Order of a lane's reductions.  Lanes of one instruction that hit the same bin
// are serialised (a cycle each), and the pairs of a tile concentrate on a few
// r_p bins: 32 pairs drawn from a (tile, group) of the 200k wg+ box put 6.2 on
// the fullest bank when every lane adds the same word, 4.7 when odd lanes take
// the two words of a field in the other order, 3.9 when the four words of two
// fields go in the order k ^ (lane & 3).  (Eight words: 3.5, for a third select
// per word.)
// The four words h0 l0 h1 l1 of two fields as this lane's 1st .. 4th.
__device__ __forceinline__ void order4(unsigned h0, unsigned l0, unsigned h1, unsigned l1, int lane,
                                       unsigned o[4]) {
  const bool a = lane & 1, b = lane & 2;
  const unsigned x0 = a ? l0 : h0, x1 = a ? h0 : l0, x2 = a ? l1 : h1, x3 = a ? h1 : l1;
  o[0] = b ? x2 : x0;
  o[1] = b ? x3 : x1;
  o[2] = b ? x0 : x2;
  o[3] = b ? x1 : x3;
}

__device__ __forceinline__ int floordiv(int a, int b) {
  int q = a / b;
  if ((a % b != 0) && ((a < 0) != (b < 0))) --q;
  return q;
}

// first index in [lo, hi) with zf[idx] >= v
__device__ __forceinline__ int lower_bound_f(const float *zf, int lo, int hi, float v) {
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(zf + mid) < v) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Append a pair to the FP64 edge queue.  Entries past the capacity are only
// counted: the host then grows the queue and runs the job again (the set of
// queued pairs is deterministic), so the kernel never needs an inline FP64
// path of its own.
__device__ __forceinline__ void enqueue(int job, int64_t i1, int64_t j2, int code, QEntry *q,
                                        unsigned long long *qcount, unsigned long long qcap) {
  const unsigned long long pos = atomicAdd(qcount, 1ull);
  if (pos < qcap) {
    QEntry e;
    e.job = job;
    e.i1 = (int)i1;
    e.j2 = (int)j2;
    e.shift = code;
    q[pos] = e;
  }
}

// Flush a region histogram (jackknife fields) into the global FP64 block at
// histogram index h, and zero it.  mirror: the histogram holds the other order
// of twin pairs, whose Pi bin is npi - 1 - (the window's bin).
template <class FMAP>
__device__ __noinline__ void flush_region(unsigned *H, int NB, int wpi, int npi, int nrp,
                                          int n2_base, int h, int f0, const double *s_iqs,
                                          const JobDev &J, bool mirror) {
  const int64_t hb = (int64_t)h * nrp * npi;
  const int S = rec_words(FMAP::FJ, f0, 0);
  for (int lb = threadIdx.x; lb < NB; lb += blockDim.x) {
    unsigned *r = H + lb * S;
    const unsigned n = r[0];
    if (!n) continue;
    const int n2 = n2_base + lb % wpi;
    const int64_t cell = hb + (int64_t)(lb / wpi) * npi + (mirror ? npi - 1 - n2 : n2);
    atomicAdd(&J.acc_num[cell], (unsigned long long)n);
    r[0] = 0u;
    const unsigned bias = n * kMagicBits;
#pragma unroll
    for (int g = 0; g < FMAP::FJ; g++) {
      if (g < f0) continue;  // field 0 of unit weights: no words
      unsigned *w = r + 1 + 2 * (g - f0);
      const int fld = FMAP::j(g);
      const long long v = fixed_sum(w, bias);
      if (v != 0) atomicAdd(&J.acc_sums[cell * kNF + fld], (double)v * s_iqs[fld]);
      w[0] = 0u;
      w[1] = 0u;
    }
  }
}

// A block's histograms: main; with jackknife the pairs the tile's own region
// does not take (nx) and the partner's region (y); in a twin job the same two of
// the other order, indexed by the window bin of the pair's own order.
struct BlockHist {
  unsigned *main, *nx, *y, *tnx, *ty;
};

// Flush the main histogram (into h = 0) and the tile's region (into hx): the
// region takes main minus NX, in exact integer arithmetic; zero both.  Twin
// blocks also add the other order of each bin's pairs to the mirrored Pi bin
// npi - 1 - n2: the same count and order-independent sums, its own
// order-dependent sums, and its own tile-region exclusions.
template <class FMAP, bool TW>
__device__ __noinline__ void flush_main_x(const BlockHist &B, int NB, int wpi, int npi, int nrp,
                                          int n2_base, int hx, bool jk, int f0,
                                          const double *s_iqs, const JobDev &J) {
  constexpr int FM = FMAP::FM, FJ = FMAP::FJ, FA = TW ? FMAP::FA : 0;
  const int64_t hsz = (int64_t)nrp * npi;
  const int S = rec_words(FM, f0, FA), SJ = rec_words(FJ, f0, 0);
  for (int lb = threadIdx.x; lb < NB; lb += blockDim.x) {
    unsigned *r = B.main + lb * S;
    const unsigned n = r[0];
    if (!n) continue;  // no pair in this bin since the last flush: every word is 0
    const int n1 = lb / wpi, elk = lb - n1 * wpi;
    const int64_t cell = (int64_t)n1 * npi + n2_base + elk;
    atomicAdd(&J.acc_num[cell], (unsigned long long)n);
    r[0] = 0u;
    const unsigned bias = n * kMagicBits;
    long long tm[FM];
#pragma unroll
    for (int f = 0; f < FM; f++) {
      tm[f] = 0;
      if (f < f0) continue;  // field 0 of unit weights: no words
      unsigned *w = r + 1 + 2 * (f - f0);
      tm[f] = fixed_sum(w, bias);
      w[0] = 0u;
      w[1] = 0u;
      const int fld = FMAP::m(f);
      if (tm[f] != 0) atomicAdd(&J.acc_sums[cell * kNF + fld], (double)tm[f] * s_iqs[fld]);
    }
    long long ta[FA > 0 ? FA : 1];
    const int64_t cm = (int64_t)n1 * npi + (npi - 1 - (n2_base + elk));
    if (TW) {
      atomicAdd(&J.acc_num[cm], (unsigned long long)n);
#pragma unroll
      for (int i = 0; i < FA; i++) {
        unsigned *w = r + 1 + 2 * (FM - f0 + i);
        ta[i] = fixed_sum(w, bias);
        w[0] = 0u;
        w[1] = 0u;
      }
#pragma unroll
      for (int f = 0; f < FM; f++) {
        if (f < f0) continue;
        const int ap = FA > 0 ? asym_pos<FMAP>(f) : -1;
        const long long v = ap >= 0 ? ta[ap] : tm[f];
        const int fld = FMAP::m(f);
        if (v != 0) atomicAdd(&J.acc_sums[cm * kNF + fld], (double)v * s_iqs[fld]);
      }
    }
    if (!jk) continue;
#pragma unroll
    for (int o = 0; o < (TW ? 2 : 1); o++) {  // the pair's own order, then the other
      unsigned *x = (o == 0 ? B.nx : B.tnx) + lb * SJ;
      const int64_t xc = (int64_t)hx * hsz + (o == 0 ? cell : cm);
      const unsigned nx = x[0], xb = nx * kMagicBits;
      x[0] = 0u;
      if (n - nx) atomicAdd(&J.acc_num[xc], (unsigned long long)(n - nx));
#pragma unroll
      for (int g = 0; g < FJ; g++) {
        if (g < f0) continue;
        unsigned *w = x + 1 + 2 * (g - f0);
        const long long tn = fixed_sum(w, xb);
        w[0] = 0u;
        w[1] = 0u;
        const int ap = (FA > 0 && o == 1) ? asym_pos<FMAP>(FMAP::jm(g)) : -1;
        const long long tx = (ap >= 0 ? ta[ap] : tm[FMAP::jm(g)]) - tn;
        const int fld = FMAP::j(g);
        if (tx != 0) atomicAdd(&J.acc_sums[xc * kNF + fld], (double)tx * s_iqs[fld]);
      }
    }
  }
}

// Flush of a block with class histograms (by_class; CS: class_stride): the pairs
// that the partner's region hy takes, whose classes are then folded into those that
// it does not take, and when `all` is set the full sample and the tile's region hx.
// Integer sums throughout; zeroes what it flushes.
template <class FMAP>
__device__ __noinline__ void flush_classes(unsigned *H, int CS, int NB, int wpi, int npi, int nrp,
                                           int n2_base, int hx, int hy, bool all, int f0,
                                           const double *s_iqs, const JobDev &J) {
  constexpr int FM = FMAP::FM, FJ = FMAP::FJ;
  const int64_t hsz = (int64_t)nrp * npi;
  const int S = rec_words(FM, f0, 0);
  for (int lb = threadIdx.x; lb < NB; lb += blockDim.x) {
    unsigned *r0 = H + lb * S, *r1 = r0 + CS, *r2 = r1 + CS, *r3 = r2 + CS;
    const int64_t cell = (int64_t)(lb / wpi) * npi + n2_base + lb % wpi;
    const unsigned n2 = r2[0], n3 = r3[0];
    if (n2 | n3) {
      const int64_t yc = (int64_t)hy * hsz + cell;
      atomicAdd(&J.acc_num[yc], (unsigned long long)(n2 + n3));
#pragma unroll
      for (int g = 0; g < FJ; g++) {
        if (g < f0) continue;
        const int o = 1 + 2 * (FMAP::jm(g) - f0), fld = FMAP::j(g);
        const long long v = fixed_sum(r2 + o, n2 * kMagicBits) + fixed_sum(r3 + o, n3 * kMagicBits);
        if (v != 0) atomicAdd(&J.acc_sums[yc * kNF + fld], (double)v * s_iqs[fld]);
      }
      for (int w = 0; w < S; w++) {
        r0[w] += r2[w];
        r1[w] += r3[w];
        r2[w] = 0u;
        r3[w] = 0u;
      }
    }
    if (!all) continue;
    const unsigned n0 = r0[0], n1 = r1[0];
    if (!(n0 | n1)) continue;
    const int64_t xc = (int64_t)hx * hsz + cell;
    atomicAdd(&J.acc_num[cell], (unsigned long long)(n0 + n1));
    if (n1) atomicAdd(&J.acc_num[xc], (unsigned long long)n1);
    r0[0] = 0u;
    r1[0] = 0u;
    long long tx[FM];
#pragma unroll
    for (int f = 0; f < FM; f++) {
      tx[f] = 0;
      if (f < f0) continue;  // field 0 of unit weights: no words
      const int o = 1 + 2 * (f - f0), fld = FMAP::m(f);
      tx[f] = fixed_sum(r1 + o, n1 * kMagicBits);
      const long long v = fixed_sum(r0 + o, n0 * kMagicBits) + tx[f];
      if (v != 0) atomicAdd(&J.acc_sums[cell * kNF + fld], (double)v * s_iqs[fld]);
      r0[o] = r0[o + 1] = r1[o] = r1[o + 1] = 0u;
    }
#pragma unroll
    for (int g = 0; g < FJ; g++) {
      if (g < f0) continue;
      const long long v = tx[FMAP::jm(g)];
      const int fld = FMAP::j(g);
      if (v != 0) atomicAdd(&J.acc_sums[xc * kNF + fld], (double)v * s_iqs[fld]);
    }
  }
}

constexpr unsigned kEdgeFlag = 0x8000u;  // queue entry: near the window edge

// VAR: the variant (variant_threads; 0: the FP64 comparison engine).  TW: twin jobs (every job
// of the launch), compiled apart so that the other jobs' kernel carries none of
// the twin code.
template <int C, bool JK, int VAR, bool TW>
__global__ void __launch_bounds__(variant_threads(VAR), variant_blocks(VAR))
fast_pairs_kernel(const JobDev *__restrict__ jobs, const UnitDesc *__restrict__ units,
                  int n_units, unsigned int *__restrict__ unit_ctr, QEntry *__restrict__ queue,
                  unsigned long long *__restrict__ qcount, unsigned long long qcap,
                  const __grid_constant__ FastScales sc, int zero_words, int auto_smem) {
  using F = FieldMap<C>;
  constexpr int kThreads = variant_threads(VAR), kWarps = kThreads / 32;
  constexpr int kCand = cand_slots(C), kSlots = kWarps * kCand, kRing = ring_size(C);
  constexpr int FA = TW ? F::FA : 0;
  const unsigned FULL = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem[];
  float4 *s_pos = reinterpret_cast<float4 *>(smem);
  // s_rshp / s_shp hold the weighted ellipticities (ewt) for the corels with
  // shape terms and the orientation (shp) for ED; s_aux: x lo, y lo, phi, w lo
  float4 *s_shp = s_pos + kSlots, *s_aux = s_shp + kSlots;
  // ED: z lo parts of the staged candidates and of the tile's rows
  float *s_zlo = reinterpret_cast<float *>(s_pos + (C == COREL_DD ? 1 : 3) * kSlots);
  float *s_rzlo = s_zlo + kSlots;
  unsigned short *wq =
      reinterpret_cast<unsigned short *>(C == COREL_ED ? s_rzlo + kTile : s_zlo) +
      (threadIdx.x >> 5) * kRing;
  // corels1 rules (launches with auto-pair jobs only): the input index of each
  // staged candidate; per row and z image (index sz + 1) a threshold on the
  // partner's input index: -1 every partner (and every pair outside corels1),
  // the row's own index: partners after it, INT_MAX: none
  int *s_orig = auto_smem ? reinterpret_cast<int *>(smem + stage_bytes(C, kWarps)) : nullptr;
  int *s_rothr = auto_smem ? s_orig + kSlots : nullptr;
  unsigned *hist = reinterpret_cast<unsigned *>(smem + stage_bytes(C, kWarps) +
                                                (auto_smem ? auto_bytes(C, kWarps) : 0));
  // the candidate slots of a unit, used only while the staging buffer is idle
  // (between the unit's slot set-up barriers, before any candidate is staged)
  int *s_slot_b = reinterpret_cast<int *>(s_pos);
  int *s_slot_info = s_slot_b + kMaxSeg;
  static_assert(2 * kMaxSeg * sizeof(int) <= kSlots * sizeof(float4), "slot tables fit the staging");

  __shared__ int s_unit, s_nseg, s_ngrp;
  __shared__ float s_zr[2][3];  // the unit's candidate z range per z image
  __shared__ int s_cnt[kMaxCols + 1];
  // candidate runs sorted by (partner region, image): start, prefix of the
  // lengths, key; s_grp: first run of each group of one key
  __shared__ int s_run_a[kMaxSeg], s_pre[kMaxSeg + 1], s_key[kMaxSeg], s_grp[kMaxSeg + 1];
  __shared__ __align__(16) int s_comp[kMaxSeg];
  __shared__ int s_jidx[kSlots];
  __shared__ unsigned char s_keep[kSlots];
  // twin jobs: the other role's keep flag of each staged candidate (g1's) and of
  // each tile row (g2's)
  __shared__ unsigned char s_keep2[TW ? kSlots : 1];
  __shared__ unsigned long long s_red[kWarps];
  __shared__ int s_max[2];  // pairs in the fullest bin, by turns
  // the tile's g1 rows, for the heavy step (any lane may process any row)
  __shared__ float4 s_rpos[kTile], s_rshp[C == COREL_DD ? 1 : kTile], s_raux[C == COREL_DD ? 1 : kTile];
  __shared__ unsigned char s_rkeep[kTile], s_rkeep2[TW ? kTile : 1];

  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  for (int k = t; k < zero_words; k += kThreads) hist[k] = 0u;
  if (t < 2) s_max[t] = 0;
  int bound = 0, turn = 0;  // bound of the pairs in any bin; the s_max in use
  __syncthreads();

  for (;;) {
    if (t == 0) s_unit = (int)atomicAdd(unit_ctr, 1u);
    __syncthreads();
    const int u = s_unit;
    if (u >= n_units) break;
    const UnitDesc U = units[u];
    const JobDev &J = jobs[U.job];
    const int nrp = J.nrp, wpi = J.wpi, npi = J.npi, NB = nrp * wpi;
    const int f0 = J.unit_w ? 1 : 0;
    const int S = rec_words(F::FM, f0, FA), SJ = rec_words(F::FJ, f0, 0);
    constexpr bool kClasses = by_class(C, JK, TW);
    const int CS = class_stride(NB * S);
    BlockHist B;
    B.main = hist;
    B.nx = B.main + NB * S;
    B.y = B.nx + NB * SJ;
    B.tnx = B.y + NB * SJ;
    B.ty = B.tnx + NB * SJ;

    // ---- the tile's g1 rows, in shared memory.  Row slot tr = s * 32 + l holds
    // tile row q = l * W + s (s < W): a warp holds slots s * 32 .. s * 32 + 31 in
    // its pass s, so its lanes are spread over the whole tile and simultaneous
    // pairs of a warp fall in different Pi bins.  Every warp tests its own
    // candidates against every row, one pass of 32 rows at a time; tiles of at
    // most 16 (8) rows take 2 (4) candidates per step. ----
    const int W = (U.g1_count + 31) >> 5;
    const int rlanes = U.g1_count <= 8 ? 8 : U.g1_count <= 16 ? 16 : 32;
    const int nsub = 32 / rlanes, sub = lane / rlanes, rl = lane & (rlanes - 1);
    // hi + lo positions for the orientation angle (raw separations) and the ED
    // separation
    constexpr bool kTheta = C == COREL_SD || C == COREL_SS || C == COREL_SSA || C == COREL_SK;
    const bool has_lo = (kTheta || C == COREL_ED) && J.has_lo;
    const bool rmu = J.rmu != 0, lin = J.lin_bin != 0;
    // VAR == 0: the cell-list FP64 comparison engine (CPC_ENGINE_CELL_FP64): every
    // candidate inside the outer window bounds is evaluated by the FP64 path,
    // inline, with global atomics (no FP32 value, no shared histogram)
    constexpr bool all_exact = VAR == 0;
    // jackknife attribution: jk_check_PB (the box's rule; this kernel runs box
    // jobs only)
    const int gws = J.gws;
    if (t < kTile && (t >> 5) < W) {
      const int q = (t & 31) * W + (t >> 5);
      // a row that is not counted is infinitely far: every window test fails
      float4 p = make_float4(0.f, 0.f, INFINITY, 0.f);
      unsigned char af = 0;
      int oi = 0;
      if (q < U.g1_count) {
        const int64_t i1 = (int64_t)U.g1_start + (int64_t)q * U.g1_stride;
        p = J.f1.pos[i1];
        if (J.auto_mode) {
          oi = (int)J.d1.orig[i1];  // input index (corels1)
          af = J.f1.aflag[i1];      // corels1 scan-start flags
        }
        if (J.row_stride > 1 && (J.d1.orig[i1] - J.row_offset) % J.row_stride != 0) p.z = INFINITY;
        if (C != COREL_DD) {
          s_rshp[t] = C == COREL_ED ? J.f1.shp[i1] : J.f1.ewt[i1];
          s_raux[t] = J.f1.aux[i1];
        }
        if (C == COREL_ED && has_lo) s_rzlo[t] = J.f1.zlo[i1];
        if (JK) s_rkeep[t] = J.f1.keep[i1];
        if (JK && TW) s_rkeep2[t] = J.f2.keep[i1];
      }
      s_rpos[t] = p;
      if (auto_smem)
        for (int z = -1; z <= 1; z++)
          s_rothr[(z + 1) * kTile + t] = auto_image_all(J.auto_mode, z, af) ? -1
                                         : auto_image_gt(J.auto_mode, z, af) ? oi : INT_MAX;
    }
    if (t < 6) s_zr[t / 3][t % 3] = (float)((t < 3 ? U.zlo : U.zhi) - J.L * (t % 3 - 1));
    const float Lf = J.Lf;
    const float xyc = J.bc.xyc, zc = J.bc.zc, zh = J.bc.zh, gd = J.bc.guard;
    const float rej_hi = J.bc.rej_hi;
    const int n2_base = U.n2_base;
    unsigned nwin = 0, nself = 0;  // window pairs of this thread's rows; pairs of a row with itself
    __syncthreads();

    // ---- enumerate candidate slots: (column, bucket, sz) overlapping the unit's z range ----
    const int ncxu = U.cx_hi - U.cx_lo + 1;
    const int ncol = ncxu * (U.cy_hi - U.cy_lo + 1);
    const int nsz_lo = J.periodic ? -1 : 0, nsz_hi = J.periodic ? 1 : 0;
    // f(bucket, sz, code) for every slot of column c, in order
    auto slots = [&](int c, auto &&f) {
      const int cx = U.cx_lo + c % ncxu, cy = U.cy_lo + c / ncxu;
      const int sx = J.periodic ? floordiv(cx, J.ncx) : 0, sy = J.periodic ? floordiv(cy, J.ncy) : 0;
      if (sx < -1 || sx > 1 || sy < -1 || sy > 1) return;
      const int col = (cy - sy * J.ncy) * J.ncx + (cx - sx * J.ncx);
      const int b1 = J.f2.col_end[col];
      for (int b = J.f2.col_begin[col]; b < b1; b++) {
        const float bz0 = J.f2.bk_zmin[b], bz1 = J.f2.bk_zmax[b];
        for (int sz = nsz_lo; sz <= nsz_hi; sz++)
          if (bz1 >= s_zr[0][sz + 1] && bz0 < s_zr[1][sz + 1]) f(b, shift_code(sx, sy, sz));
      }
    };
    for (int c = t; c < ncol; c += kThreads) {
      int cnt = 0;
      slots(c, [&](int, int) { cnt++; });
      s_cnt[c] = cnt;
    }
    __syncthreads();
    if (wid == 0) {  // exclusive prefix over the columns
      int run = 0;
      for (int c0 = 0; c0 < ncol; c0 += 32) {
        const int v = c0 + lane < ncol ? s_cnt[c0 + lane] : 0;
        int p = v;
        for (int o = 1; o < 32; o <<= 1) {
          const int w = __shfl_up_sync(FULL, p, o);
          if (lane >= o) p += w;
        }
        if (c0 + lane < ncol) s_cnt[c0 + lane] = run + p - v;
        run += __shfl_sync(FULL, p, 31);
      }
      if (lane == 0) s_cnt[ncol] = run;
    }
    __syncthreads();
    const int total_slots = s_cnt[ncol];
    int cur_y = -1;        // region held in the Y histogram
    // y: what the region in Y took; all: the rest too
    auto flush = [&](bool y, bool all) {
      if constexpr (kClasses) {
        flush_classes<F>(hist, CS, NB, wpi, npi, nrp, n2_base, 1 + U.region, 1 + cur_y, all, f0,
                         sc.iqs, J);
      } else {
        if (all)
          flush_main_x<F, TW>(B, NB, wpi, npi, nrp, n2_base, 1 + U.region, JK, f0, sc.iqs, J);
        if (JK && y) {
          flush_region<F>(B.y, NB, wpi, npi, nrp, n2_base, 1 + cur_y, f0, sc.iqs, J, false);
          if (TW)
            flush_region<F>(B.ty, NB, wpi, npi, nrp, n2_base, 1 + cur_y, f0, sc.iqs, J, true);
        }
      }
    };

    for (int chunk0 = 0; chunk0 < total_slots; chunk0 += kMaxSeg) {
      const int nslot = min(kMaxSeg, total_slots - chunk0);
      for (int c = t; c < ncol; c += kThreads) {
        int pos = s_cnt[c] - chunk0;
        if (pos >= kMaxSeg || s_cnt[c + 1] <= chunk0) continue;
        slots(c, [&](int b, int code) {
          if (pos >= 0 && pos < kMaxSeg) {
            s_slot_b[pos] = b;
            s_slot_info[pos] = code;
          }
          pos++;
        });
      }
      __syncthreads();
      {  // a run per thread of the first kMaxSeg, ranked by (partner region, image)
        int a = 0, len = 0, comp = INT_MAX;
        if (t < nslot) {
          const int b = s_slot_b[t], code = s_slot_info[t];
          const int sz = code / 9 - 1;
          // twin jobs test each unordered pair once, in the order whose g2 is
          // ahead of g1: image -1 candidates are the other order of image +1
          // pairs of their own tiles
          if (!(TW && sz < 0)) {
            const int bs = J.f2.bk_start[b], be = J.f2.bk_end[b];
            a = lower_bound_f(J.f2.zf, bs, be, s_zr[0][sz + 1]);
            len = lower_bound_f(J.f2.zf, a, be, s_zr[1][sz + 1]) - a;
            if (len > 0) comp = (J.f2.bk_region[b] * 27 + code) * kMaxSeg + t;
          }
        }
        if (t < kMaxSeg) s_comp[t] = comp;
        const unsigned any = __ballot_sync(FULL, comp != INT_MAX);
        __syncthreads();
        int r = 0;
        if (any) {
          const int n4 = (nslot + 3) >> 2;
          for (int m = 0; m < n4; m++) {
            const int4 v = reinterpret_cast<const int4 *>(s_comp)[m];
            r += (v.x < comp) + (v.y < comp) + (v.z < comp) + (v.w < comp);
          }
        }
        if (comp != INT_MAX) {
          s_run_a[r] = a;
          s_pre[r] = len;
          s_key[r] = comp / kMaxSeg;
        }
        if (t == 0) s_nseg = 0;
        __syncthreads();
        if (lane == 0 && any) atomicAdd(&s_nseg, __popc(any));
      }
      __syncthreads();
      if (wid == 0) {  // prefix of the run lengths, first run of each group
        const int n = s_nseg;
        int run = 0, ng = 0;
        for (int k0 = 0; k0 < n; k0 += 32) {
          const int k = k0 + lane;
          const int v = k < n ? s_pre[k] : 0;
          int p = v;
          for (int o = 1; o < 32; o <<= 1) {
            const int w = __shfl_up_sync(FULL, p, o);
            if (lane >= o) p += w;
          }
          const bool first = k < n && (k == 0 || s_key[k] != s_key[k - 1]);
          const unsigned m = __ballot_sync(FULL, first);
          if (k < n) s_pre[k] = run + p - v;
          if (first) s_grp[ng + __popc(m & ((1u << lane) - 1u))] = k;
          ng += __popc(m);
          run += __shfl_sync(FULL, p, 31);
        }
        if (lane == 0) {
          s_pre[n] = run;
          s_grp[ng] = n;
          s_ngrp = ng;
        }
      }
      __syncthreads();

      for (int gi = 0; gi < s_ngrp; gi++) {
        const int k = s_grp[gi], g = s_grp[gi + 1];
        const int key = s_key[k];
        const int region2 = key / 27, code = key % 27;
        int sx, sy, sz;
        shift_decode(code, sx, sy, sz);
        const bool same_region = region2 == U.region;
        const int gN = s_pre[g] - s_pre[k];
        if (JK && !same_region && cur_y != region2) {
          if (cur_y >= 0) {
            __syncthreads();
            flush(true, false);
            __syncthreads();
          }
          cur_y = region2;
        }
        // g2-side shift for -1 images (x2 - L exact for the candidates that can
        // reach the window), g1-side shift for +1 images (x1 - L exact for
        // x1 >= L/2)
        const float g2sx = sx == -1 ? Lf : 0.f, g2sy = sy == -1 ? Lf : 0.f, g2sz = sz == -1 ? Lf : 0.f;
        const float g1sx = sx == 1 ? Lf : 0.f, g1sy = sy == 1 ? Lf : 0.f, g1sz = sz == 1 ? Lf : 0.f;
        // twin jobs, image 0: the order with the larger z of g2 (the sign of a
        // float difference is exact; ties by the image shift in y, then x, then
        // the index)
        const int tie_dir = sy != 0 ? sy : sx;
        const float zmin = !TW || sz != 0 ? -INFINITY : tie_dir > 0 ? -1e-45f : 0.0f;
        const bool tie0 = TW && sz == 0 && tie_dir == 0;

        const int chunk = kChunkTests / 32 / W;
        for (int base = 0; base < gN; base += chunk) {
          const int nc = min(chunk, gN - base);
          if (!all_exact && bound + 32 * W * nc > kBinTerms) {  // (block-uniform)
            int m = 0;
            __syncthreads();
            for (int lb = t; lb < NB; lb += kThreads) {
              const unsigned *r = hist + lb * S;
              m = max(m, (int)(kClasses ? r[0] + r[CS] + r[2 * CS] + r[3 * CS] : r[0]));
            }
            m = __reduce_max_sync(FULL, m);
            if (lane == 0 && m > 0) atomicMax(&s_max[turn], m);
            if (t == 0) s_max[turn ^ 1] = 0;
            __syncthreads();
            bound = s_max[turn];
            turn ^= 1;
            if (bound + 32 * W * nc > kBinTerms) {
              flush(cur_y >= 0, true);
              bound = 0;
              __syncthreads();
            }
          }
          bound += 32 * W * nc;
          // this warp's share of the chunk, positions p = wid (mod nw), in nbw
          // batches of at most kCand - 1 candidates strided over it (columns and
          // redshifts mixed, so that a warp's pairs fall in different bins),
          // staged in the warp's own slots c0 .. (read by this warp only: no block
          // barrier)
          const int c0 = wid * kCand;
          const int nw = min(kWarps, max(1, nc >> 3));
          const int share = wid < nw ? (nc - wid + nw - 1) / nw : 0;
          const int nbw = (share + kCand - 2) / (kCand - 1);
          for (int bw = 0; bw < nbw; bw++) {
            const int nk = (share - bw + nbw - 1) / nbw;  // 1 .. kCand - 1
            if (lane < kCand) {
              const int slot = c0 + lane;
              // no candidate: infinitely far from every row (absent rows too)
              float4 q2 = make_float4(0.f, 0.f, -INFINITY, 0.f);
              if (lane < nk) {
                const int p = s_pre[k] + base + (lane * nbw + bw) * nw + wid;
                int lo = k, hi = g;  // run lo with s_pre[lo] <= p < s_pre[lo + 1]
                while (hi - lo > 1) {
                  const int mid = (lo + hi) >> 1;
                  if (s_pre[mid] <= p) lo = mid; else hi = mid;
                }
                const int j2 = s_run_a[lo] + (p - s_pre[lo]);
                q2 = J.f2.pos[j2];
                q2.x -= g2sx;
                q2.y -= g2sy;
                q2.z -= g2sz;
                if (C != COREL_DD) {
                  s_shp[slot] = C == COREL_ED ? J.f2.shp[j2] : J.f2.ewt[j2];
                  s_aux[slot] = J.f2.aux[j2];
                }
                if (C == COREL_ED && has_lo) s_zlo[slot] = J.f2.zlo[j2];
                s_jidx[slot] = j2;
                if (auto_smem && J.auto_mode) s_orig[slot] = (int)J.d2.orig[j2];
                if (JK) s_keep[slot] = J.f2.keep[j2];
                if (JK && TW) s_keep2[slot] = J.f1.keep[j2];
              }
              s_pos[slot] = q2;
            }
            __syncwarp();

            // ---- window tests: a candidate at a time against the lanes' rows, a
            // bit per step for the pairs that may bin and one for those near the
            // window's edge; after a pass each lane queues its pairs (a prefix
            // sum of the bit counts gives its place) and the heavy step runs
            // while 32 are queued (all lanes busy) ----
            const int nks = (nk + nsub - 1) / nsub;
            int pass = 0, qhead = 0, qtail = 0;
            for (;;) {
              if (qtail - qhead < 32 && pass < W) {
                const int tr = pass * 32 + rl;
                unsigned mask = 0u, emask = 0u;
                {
                  const float4 p1 = s_rpos[tr];
                  const float x1 = p1.x - g1sx, y1 = p1.y - g1sy, z1 = (p1.z - g1sz) + zc;
                  const int othr = auto_smem ? s_rothr[(sz + 1) * kTile + tr] : -1;
                  const float4 *cp = s_pos + c0 + sub;
                  unsigned bit = 1u;
#pragma unroll 4
                  for (int st = 0; st < nks; st++) {
                    const float4 p2 = cp[0];
                    const float dz = p2.z - z1, dx = x1 - p2.x, dy = y1 - p2.y;
                    // distance inside the window, the smaller of the two
                    const float d =
                        fminf(zh - fabsf(dz), xyc - fmaxf(fabsf(dx), fabsf(dy)));
                    float r2 = fmaf(dx, dx, dy * dy);
                    if (rmu) r2 = fmaf(dz, dz, r2);
                    bool in = d > gd, edge = fabsf(d) <= gd;
                    if (TW) {
                      bool ahead = dz > zmin;
                      if (tie0 && dz == 0.0f) {
                        const int j2 = s_jidx[c0 + sub + st * nsub];
                        const int i1 = U.g1_start + (rl * W + pass) * U.g1_stride;
                        ahead = j2 >= i1;
                        if (j2 == i1 && d > gd) nself++;
                      }
                      in = in && ahead;
                      edge = edge && ahead;
                    }
                    if (auto_smem && othr >= 0) {
                      const bool ord = s_orig[c0 + sub + st * nsub] > othr;
                      in = in && ord;
                      edge = edge && ord;
                    }
                    if (all_exact) {
                      edge = edge || in;
                    } else {
                      if (in) nwin++;
                      // r_p^2 (or r^2 of coordinates 7) certainly above the bins?
                      if (in && r2 < rej_hi) mask |= bit;
                    }
                    if (edge) emask |= bit;
                    bit += bit;
                    cp += nsub;
                  }
                }
                const int cnt = __popc(mask) + __popc(emask);
                int sum = cnt;
                for (int o = 1; o < 32; o <<= 1) {
                  const int v = __shfl_up_sync(FULL, sum, o);
                  if (lane >= o) sum += v;
                }
                unsigned pos = (unsigned)(qtail + sum - cnt);  // qtail < 2 kRing
                if (pos >= kRing) pos -= kRing;
                const unsigned en = (unsigned)tr | (unsigned)(sub << 7);
                while (mask) {
                  const int st = 31 - __clz(mask);
                  mask ^= 1u << st;
                  wq[pos] = (unsigned short)(en + ((unsigned)(st * nsub) << 7));
                  if (++pos == kRing) pos = 0;
                }
                while (emask) {
                  const int st = 31 - __clz(emask);
                  emask ^= 1u << st;
                  wq[pos] = (unsigned short)((en + ((unsigned)(st * nsub) << 7)) | kEdgeFlag);
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
                const bool edge = (en & kEdgeFlag) != 0;
                const float4 r1 = s_rpos[er];
                const float4 p2 = s_pos[ec];
                const float hdz = p2.z - (r1.z - g1sz);
                const float hdx = (r1.x - g1sx) - p2.x;
                const float hdy = (r1.y - g1sy) - p2.y;
                float r2 = fmaf(hdx, hdx, hdy * hdy);
                // the bins from the linear maps of Pi (or mu) and log2 r^2 (or r):
                // the nearest integer, certain when farther from the next
                // half-integer than the error bound (BoxConst)
                float lim2 = J.bc.pi_in, lim1 = J.bc.rp_in, v2;
                if (rmu) {
                  // coordinates 7: r = |(dx, dy, dz)|, mu = dz / r (r_mu_calc)
                  r2 = fmaf(hdz, hdz, r2);
                  const float ri = rsqrtf(r2);
                  v2 = fmaf(hdz * ri, J.bc.pi_s, J.bc.pi_o);
                  lim2 -= J.bc.pi_abs * ri;
                  lim1 -= J.bc.rp_abs * ri;
                } else {
                  v2 = fmaf(hdz, J.bc.pi_s, J.bc.pi_o);
                  if (J.bc.rp_abs > 0.0f) lim1 -= J.bc.rp_abs * rsqrtf(r2);
                }
                const float m2 = v2 + kMagic;
                const int n2 = __float_as_int(m2) - (int)kMagicBits;
                const float v1 = lin ? fmaf(sqrtf(r2), J.bc.rp_s, J.bc.rp_o)
                                     : fmaf(__log2f(r2), J.bc.rp_s, J.bc.rp_o);
                const float m1 = v1 + kMagic;
                const int n1 = __float_as_int(m1) - (int)kMagicBits;
                bool amb = !(fabsf(v2 - (m2 - kMagic)) <= lim2 && fabsf(v1 - (m1 - kMagic)) <= lim1);
                // a block holds the bins [n2_base, n2_base + wpi) of Pi; of mu, each
                // pair belongs to the unit whose slice holds its estimated bin
                // (clamped), the others skip it
                const int elk = n2 - n2_base;
                const int n2c = min(max(n2, 0), npi - 1) - n2_base;
                const bool own = !rmu || (unsigned)n2c < (unsigned)wpi;
                bool bin = r2 >= J.bc.rej_lo;  // else certainly below the bins
                if (!amb) {
                  bin = bin && (unsigned)n1 < (unsigned)nrp && (unsigned)n2 < (unsigned)npi;
                  amb = (unsigned)elk >= (unsigned)wpi;
                }
                // raw (un-shifted) separation for the orientation angle
                // (angle_orient_axis_PB); coincident positions give atan(0/0) in
                // the reference: those pairs take the exact path
                // The separation is a double-float: the exact difference of the
                // float hi parts, plus the lo parts for inputs that are not
                // float32 values (renormalised); it is zero only when the
                // positions coincide.
                df32 dxr{0.f, 0.f}, dyr{0.f, 0.f};
                if (kTheta) {
                  const float x2r = p2.x + g2sx, y2r = p2.y + g2sy;  // x2, y2 restored exactly
                  if (has_lo) {
                    const float4 a1 = s_raux[er], a2 = s_aux[ec];
                    dxr = df_diff_hl(x2r, a2.x, r1.x, a1.x);
                    dyr = df_diff_hl(y2r, a2.y, r1.y, a1.y);
                  } else {
                    dxr = two_diff(x2r, r1.x);
                    dyr = two_diff(y2r, r1.y);
                  }
                  if (dxr.h == 0.0f && dyr.h == 0.0f) amb = true;
                }
                // ED: the shifted separation g1 - (g2 + L*PB) (ED_calc_PB) from
                // hi + lo positions; a zero separation gives 0/0 in the reference
                float sxe = 0.f, sye = 0.f, sze = 0.f, see = 1.f;
                if (C == COREL_ED) {
                  sxe = hdx;
                  sye = hdy;
                  sze = -hdz;
                  if (has_lo) {
                    const float4 a1 = s_raux[er], a2 = s_aux[ec];
                    sxe += a1.x - a2.x;
                    sye += a1.y - a2.y;
                    sze += s_rzlo[er] - s_zlo[ec];
                  }
                  see = fmaf(sxe, sxe, fmaf(sye, sye, sze * sze));
                  if (!(see > 0.0f)) amb = true;
                }
                // twin jobs: a row paired with itself has no other order; it takes
                // the exact path (its count is not mirrored)
                bool tself = false;
                if (TW && tie0 && hdz == 0.0f) {
                  const int i1 = U.g1_start + (((er & 31) * W) + (er >> 5)) * U.g1_stride;
                  tself = s_jidx[ec] == i1;
                  if (tself) amb = true;
                }
                if (all_exact) {
                  // the comparison engine: the reference's double arithmetic for
                  // every candidate (window, bins, values), global FP64 atomics.
                  // With coordinates 7 every mu slice visits the pair: the window
                  // count is kept from slice 0 only, the pair's values go in by the
                  // slice that holds its exact mu bin
                  const int64_t gi1 = (int64_t)U.g1_start +
                                      (int64_t)(((er & 31) * W) + (er >> 5)) * U.g1_stride;
                  const int64_t gj2 = s_jidx[ec];
                  int xn1, xn2;
                  const int r = exact_classify(J, J.d1, gi1, J.d2, gj2, sx, sy, sz, xn1, xn2);
                  if (r >= 1) nwin++;
                  if (r == 2 && (!rmu || (xn2 >= n2_base && xn2 < n2_base + wpi))) {
                    double f[kNF];
                    exact_values(J, J.d1, gi1, J.d2, gj2, sx, sy, sz, f);
                    exact_accumulate(J, J.d1, gi1, J.d2, gj2, xn1, xn2, f);
                  }
                } else if (own && (edge || (bin && amb))) {
                  // near the window edge (not yet counted) or a bin edge (window
                  // counted): exact FP64 evaluation
                  const int64_t gi1 = (int64_t)U.g1_start +
                                      (int64_t)(((er & 31) * W) + (er >> 5)) * U.g1_stride;
                  enqueue(U.job, gi1, s_jidx[ec], edge ? code : (code | kWindowCounted), queue,
                          qcount, qcap);
                  // twin jobs: the other order, (g1 = the candidate, g2 = the row)
                  // at the opposite image
                  if (TW && !tself) {
                    const int mcode = shift_code(-sx, -sy, -sz);
                    enqueue(U.job, s_jidx[ec], gi1, edge ? mcode : (mcode | kWindowCounted), queue,
                            qcount, qcap);
                  }
                } else if (own && bin) {
                  const int lb = n1 * wpi + elk;
                  // per-field terms: v (float) for every field, vd (double-float)
                  // for the fields whose sums cancel (df_field)
                  float v[kNF];
                  df32 vd[kNF];
                  // twin jobs: the other order's order-dependent terms (shape_shape)
                  float vm[FA > 0 ? kNF : 1];
                  df32 vdm[FA > 0 ? kNF : 1];
                  v[0] = r1.w * p2.w;
                  if (C == COREL_ED) {
                    const float4 es = gws == 2 ? s_shp[ec] : s_rshp[er];
                    const float dot = fmaf(es.x, sxe, fmaf(es.y, sye, es.w * sze));
                    v[11] = __fdividef(dot * dot, see);
                    v[12] = v[11] * v[11];
                  } else if (C != COREL_DD) {
                    // (w e1, w e2) hi and lo parts, the weight's lo part and phi
                    const float4 ea = s_rshp[er], eb = s_shp[ec];
                    const float4 xa = s_raux[er], xb = s_aux[ec];
                    const DfGal g1{{ea.x, ea.z}, {ea.y, ea.w}, {r1.w, xa.w}, xa.z};
                    const DfGal g2{{eb.x, eb.z}, {eb.y, eb.w}, {p2.w, xb.w}, xb.z};
                    df32 c2{0.f, 0.f}, s2v{0.f, 0.f};
                    float theta = 0.f;
                    if (kTheta) {
                      df_cos_sin_2theta(dxr, dyr, c2, s2v);
                      if (C != COREL_SK) theta = atanf(__fdividef(dyr.h, dxr.h));
                    }
                    if constexpr (FA > 0)
                      df_pair_terms<C>(c2, s2v, theta, g1, g2, gws, J.unit_w != 0, vd, v, vdm, vm);
                    else
                      df_pair_terms<C>(c2, s2v, theta, g1, g2, gws, J.unit_w != 0, vd, v);
                  }
                  // the words of the main fields; those of two fields at a time go in
                  // this lane's order (order4), a single field's by lane parity
                  unsigned wh[F::FM], wl[F::FM];
#pragma unroll
                  for (int f = 0; f < F::FM; f++) {
                    const int q = F::m(f);
                    if (df_field(C, q)) df_to_words(vd[q], sc.qs[q], wh[f], wl[f]);
                    else f_to_words(v[q], sc.qs[q], wh[f], wl[f]);
                  }
                  const int odd = lane & 1, r4 = lane & 3;
                  auto add1 = [&](unsigned *w, unsigned h, unsigned l) {
                    atomicAdd(w + odd, odd ? l : h);
                    atomicAdd(w + 1 - odd, odd ? h : l);
                  };
                  auto add2 = [&](unsigned *w, unsigned h0, unsigned l0, unsigned h1, unsigned l1) {
                    unsigned o[4];
                    order4(h0, l0, h1, l1, lane, o);
                    atomicAdd(w + r4, o[0]);
                    atomicAdd(w + (1 ^ r4), o[1]);
                    atomicAdd(w + (2 ^ r4), o[2]);
                    atomicAdd(w + (3 ^ r4), o[3]);
                  };
                  // field f's words are at r0 + 2 f
                  unsigned *rec = hist + lb * S;
                  // jk_check_PB (jk.cpp:64-71): the tile's region takes a same-region
                  // pair and a cross-region pair whose row is kept; the partner's
                  // region takes a cross-region pair whose partner is kept
                  if (kClasses)
                    rec += (same_region ? 1 : (s_rkeep[er] ? 1 : 0) + (s_keep[ec] ? 2 : 0)) * CS;
                  unsigned *r0 = rec + 1 - 2 * f0;
                  atomicAdd(rec, 1u);
                  if (f0 == 0) add1(r0, wh[0], wl[0]);
#pragma unroll
                  for (int f = 1; f + 1 < F::FM; f += 2)
                    add2(r0 + 2 * f, wh[f], wl[f], wh[f + 1], wl[f + 1]);
                  if constexpr (F::FM > 1 && F::FM % 2 == 0)
                    add1(r0 + 2 * (F::FM - 1), wh[F::FM - 1], wl[F::FM - 1]);
                  unsigned xh[FA > 0 ? FA : 1], xl[FA > 0 ? FA : 1];
                  if constexpr (FA > 0) {
                    // the other order's order-dependent terms
                    static_assert(FA % 2 == 0, "order-dependent fields in pairs");
#pragma unroll
                    for (int i = 0; i < FA; i++) {
                      const int q = F::m(F::a(i));
                      if (df_field(C, q)) df_to_words(vdm[q], sc.qs[q], xh[i], xl[i]);
                      else f_to_words(vm[q], sc.qs[q], xh[i], xl[i]);
                    }
#pragma unroll
                    for (int i = 0; i < FA; i += 2)
                      add2(r0 + 2 * (F::FM + i), xh[i], xl[i], xh[i + 1], xl[i + 1]);
                  }
                  if (JK && !kClasses && !same_region) {
                    // (the tile's region: main - NX)
                    auto region = [&](unsigned *h, bool other) {
                      unsigned *q = h + lb * SJ, *q0 = q + 1 - 2 * f0;
                      atomicAdd(q, 1u);
#pragma unroll
                      for (int j = 0; j < F::FJ; j++) {
                        if (j < f0) continue;
                        const int ap = (FA > 0 && other) ? asym_pos<F>(F::jm(j)) : -1;
                        if (ap >= 0) add1(q0 + 2 * j, xh[ap < 0 ? 0 : ap], xl[ap < 0 ? 0 : ap]);
                        else add1(q0 + 2 * j, wh[F::jm(j)], wl[F::jm(j)]);
                      }
                    };
                    if (!s_rkeep[er]) region(B.nx, false);
                    if (s_keep[ec]) region(B.y, false);
                    if (TW) {
                      // the other order (g1 = the candidate, g2 = the row): the tile's
                      // region takes it when the row is kept in the g2 role, the
                      // partner's region when the candidate is kept in the g1 role
                      if (!s_rkeep2[er]) region(B.tnx, true);
                      if (s_keep2[ec]) region(B.ty, true);
                    }
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
            __syncwarp();  // every lane is done with the staged slots before restaging
          }
        }
      }
      __syncthreads();  // the run tables and staging are free
    }

    // ---- flush main, X and the last Y ----
    flush(cur_y >= 0, true);
    bound = 0;
    // window-pair counter (once per pair: mu slices other than the first skip it)
    {
      unsigned long long v =
          (rmu && n2_base != 0) ? 0ull : (TW ? 2ull * nwin - nself : (unsigned long long)nwin);
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(FULL, v, o);
      if (lane == 0) s_red[wid] = v;
      __syncthreads();
      if (t == 0) {
        unsigned long long sm = 0;
        for (int w = 0; w < kWarps; w++) sm += s_red[w];
        if (sm) atomicAdd(&J.counters[0], sm);
      }
    }
    __syncthreads();
  }
}

// Exact FP64 re-evaluation of the edge queue.
__global__ void recheck_kernel(const JobDev *__restrict__ jobs, const QEntry *__restrict__ queue,
                               const unsigned long long *__restrict__ qcount,
                               unsigned long long qcap) {
  const unsigned long long n = min(*qcount, qcap);
  for (unsigned long long idx = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n;
       idx += (unsigned long long)gridDim.x * blockDim.x) {
    const QEntry e = queue[idx];
    const JobDev &J = jobs[e.job];
    int sx, sy, sz, n1, n2;
    shift_decode(e.shift & kShiftMask, sx, sy, sz);
    const int r = exact_classify(J, J.d1, e.i1, J.d2, e.j2, sx, sy, sz, n1, n2);
    atomicAdd(&J.counters[2], 1ull);
    if (r == 0) continue;
    if (!(e.shift & kWindowCounted)) atomicAdd(&J.counters[1], 1ull);
    if (r == 2) {
      double f[kNF];
      exact_values(J, J.d1, e.i1, J.d2, e.j2, sx, sy, sz, f);
      exact_accumulate(J, J.d1, e.i1, J.d2, e.j2, n1, n2, f);
    }
  }
}

// ---- host-side launchers (called from capi.cu) ----
// Calls fn.run<C, JK, VAR, TW>() for the runtime corel, jackknife flag and variant.
template <int C, bool TW, class Fn>
static auto dispatch_var(int jk, int var, const Fn &fn) -> decltype(fn.template run<C, true, 1, TW>()) {
  if (var == 3) return jk ? fn.template run<C, true, 3, TW>() : fn.template run<C, false, 3, TW>();
  if (var == 2) return jk ? fn.template run<C, true, 2, TW>() : fn.template run<C, false, 2, TW>();
  if constexpr (!TW)
    if (var == 0) return jk ? fn.template run<C, true, 0, TW>() : fn.template run<C, false, 0, TW>();
  return jk ? fn.template run<C, true, 1, TW>() : fn.template run<C, false, 1, TW>();
}
template <class Fn>
static auto dispatch(int corel, int jk, int var, int twin, const Fn &fn)
    -> decltype(fn.template run<0, false, 1, false>()) {
  // twin jobs: density_density and shape_shape
  if (twin && var != 0) {
    if (corel == COREL_SS) return dispatch_var<COREL_SS, true>(jk, var, fn);
    if (corel == COREL_SSA) return dispatch_var<COREL_SSA, true>(jk, var, fn);
    return dispatch_var<COREL_DD, true>(jk, var, fn);
  }
  switch (corel) {
    case COREL_SD: return dispatch_var<COREL_SD, false>(jk, var, fn);
    case COREL_SS: return dispatch_var<COREL_SS, false>(jk, var, fn);
    case COREL_SSA: return dispatch_var<COREL_SSA, false>(jk, var, fn);
    case COREL_DK: return dispatch_var<COREL_DK, false>(jk, var, fn);
    case COREL_SK: return dispatch_var<COREL_SK, false>(jk, var, fn);
    case COREL_ED: return dispatch_var<COREL_ED, false>(jk, var, fn);
    default: return dispatch_var<COREL_DD, false>(jk, var, fn);
  }
}

struct LaunchFast {
  const JobDev *jobs;
  const UnitDesc *units;
  int n_units;
  unsigned int *unit_ctr;
  QEntry *q;
  unsigned long long *qcount, qcap;
  const FastScales *sc;
  size_t smem;
  int grid;
  int auto_pairs;
  cudaStream_t st;
  template <int C, bool JK, int VAR, bool TW>
  cudaError_t run() const {
    auto kern = fast_pairs_kernel<C, JK, VAR, TW>;
    cudaError_t err =
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    constexpr int kThr = variant_threads(VAR);
    const int zero_words = (int)((smem - stage_bytes(C, kThr / 32) -
                                  (auto_pairs ? auto_bytes(C, kThr / 32) : 0)) / 4);
    kern<<<grid, kThr, smem, st>>>(jobs, units, n_units, unit_ctr, q, qcount, qcap, *sc,
                                   zero_words, auto_pairs);
    return cudaGetLastError();
  }
};

struct Occupancy {
  size_t smem;
  template <int C, bool JK, int VAR, bool TW>
  int run() const {
    auto kern = fast_pairs_kernel<C, JK, VAR, TW>;
    int nb = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, variant_threads(VAR), smem) !=
            cudaSuccess)
      return 0;
    return nb;
  }
};

cudaError_t launch_fast(int corel, int jk, int variant, int twin, const JobDev *jobs,
                        const UnitDesc *units, int n_units, unsigned int *unit_ctr, QEntry *q,
                        unsigned long long *qcount, unsigned long long qcap,
                        const FastScales &sc, size_t smem, int grid, int auto_pairs,
                        cudaStream_t st) {
  if (corel < COREL_DD || corel > COREL_ED) return cudaErrorInvalidValue;
  return dispatch(corel, jk, variant, twin,
                  LaunchFast{jobs, units, n_units, unit_ctr, q, qcount, qcap, &sc, smem, grid,
                             auto_pairs, st});
}

struct StaticSmem {
  template <int C, bool JK, int VAR, bool TW>
  size_t run() const {
    cudaFuncAttributes a;
    const cudaError_t e = cudaFuncGetAttributes(&a, fast_pairs_kernel<C, JK, VAR, TW>);
    return e == cudaSuccess ? a.sharedSizeBytes : 24 * 1024;
  }
};
// Static shared memory of a block, asked of the runtime once per kernel.
size_t fast_static_smem_bytes(int corel, int jk, int variant, int twin) {
  static std::atomic<size_t> known[COREL_ED + 1][2][4][2];
  std::atomic<size_t> &k = known[corel][jk ? 1 : 0][variant][twin ? 1 : 0];
  size_t b = k.load(std::memory_order_relaxed);
  if (!b) k.store(b = dispatch(corel, jk, variant, twin, StaticSmem{}), std::memory_order_relaxed);
  return b;
}

// Blocks per SM of a variant with this much dynamic shared memory (0: none fit).
int fast_blocks(int corel, int jk, int variant, size_t smem, int twin) {
  if (corel < COREL_DD || corel > COREL_ED) return 0;
  return dispatch(corel, jk, variant, twin, Occupancy{smem});
}

cudaError_t launch_recheck(const JobDev *jobs, const QEntry *q, const unsigned long long *qcount,
                           unsigned long long qcap, int grid, cudaStream_t st) {
  recheck_kernel<<<grid, 256, 0, st>>>(jobs, q, qcount, qcap);
  return cudaGetLastError();
}

int fast_variant_blocks(int variant) { return variant_blocks(variant); }
size_t fast_block_smem(int variant) { return (size_t)(228 * 1024) / variant_blocks(variant); }
}  // namespace cpc
