// Host check of the fixed-point words of the pair kernels (df_to_words, f_to_words
// and fixed_sum of corr_pc_gb300/csrc/df32.cuh), built by tests/test_fixed_words.py
// with g++ -ffp-contract=off.  Prints what it found; exits 1 on a failure.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <random>

#include "df32.cuh"
#include "pair_df.cuh"

using namespace cpc;

static int bad = 0;
static void expect(bool ok, const char *what, double v) {
  std::printf("%s %s (%g)\n", ok ? "ok" : "BAD", what, v);
  if (!ok) bad = 1;
}
static int word(unsigned w) { return (int)(w - kMagicBits); }

// n times the words of one term, as reductions of 32 bits add them
static long long repeated(unsigned hi, unsigned lo, unsigned n) {
  const unsigned w[2] = {hi * n, lo * n};
  return fixed_sum(w, n * kMagicBits);
}

int main() {
  std::mt19937_64 g(11);
  std::uniform_real_distribution<double> U(-1.0, 1.0);
  for (const int S : {29, 30}) {  // box and sky: terms up to 2^S / (1 + 2^-12)
    const double top = std::ldexp(1.0, S) / (1.0 + 1.0 / 4096.0);
    const int high = S == 29 ? 1 << 14 : (1 << 15) - 8;
    double worst = 0, worst_f = 0;
    int hi_max = 0, lo_max = 0;
    for (int it = 0; it < 400000; it++) {
      const double v = it < 4 ? (it & 1 ? -1.0 : 1.0) : U(g) * std::exp2(-20.0 * std::fabs(U(g)) * (it & 1));
      const float h = (float)(v * top * std::ldexp(1.0, -S));
      const float l = (float)(U(g) * std::ldexp(std::fabs((double)h), -21));  // 8 ulps of h
      const float qs = std::ldexp(1.0f, S);
      unsigned a, b;
      df_to_words(df32{h, l}, qs, a, b);
      worst = std::max(worst, std::fabs((double)word(a) * 32768.0 + word(b) -
                                        ((double)h + l) * std::ldexp(1.0, S)));
      hi_max = std::max(hi_max, std::abs(word(a)));
      unsigned c, d;
      f_to_words(h, qs, c, d);
      worst_f = std::max(worst_f, std::fabs((double)word(c) * 32768.0 + word(d) -
                                            (double)h * std::ldexp(1.0, S)));
      lo_max = std::max(lo_max, std::abs(word(d)));
    }
    // one rounding to a quantum, one of r + l 2^S (a float below 2^15: 2^-9)
    expect(worst <= 0.5 + 1.0 / 512, "df_to_words: quanta off", worst);
    expect(worst_f <= 0.5, "f_to_words: quanta off", worst_f);
    expect(hi_max <= high, "high word", hi_max);
    expect(lo_max <= 1 << 14, "low word of a float term", lo_max);
  }
  // the low parts of rotated, weighted terms and their products at the bound
  {
    double worst = 0;
    for (int it = 0; it < 400000; it++) {
      const double a = M_PI * U(g), p = M_PI * U(g), q = M_PI * U(g), r = std::exp2(4 * U(g));
      auto split = [](double v) { return df32{(float)v, (float)(v - (float)v)}; };
      df32 c, s, ep, ex, fp, fx;
      df_cos_sin_2theta(split(r * std::cos(a)), split(r * std::sin(a)), c, s);
      df_rotate(c, s, split(std::cos(p)), split(std::sin(p)), ep, ex);
      df_rotate(c, s, split(std::cos(q)), split(std::sin(q)), fp, fx);
      for (const df32 v : {ep, ex, df_mul(ep, fp), df_mul(ex, fx), df_mul(ep, fx)})
        worst = std::max(worst, std::fabs((double)v.l));
    }
    worst *= std::ldexp(1.0, 29);
    expect(worst <= kLowTerm - (1 << 14), "low part of a term in quanta", worst);
  }
  // a bin's words filled with the extreme terms: the largest high and low words, and
  // the term whose low part alone passes 2^14 + 1
  for (const int sh : {-1, 1})
    for (const int sl : {-1, 1})
      for (const int hi : {0, 8193, 1 << 14})
        for (const int lo : {1 << 14, (1 << 14) + 16, kLowTerm}) {
          const unsigned a = (unsigned)(sh * hi) + kMagicBits, b = (unsigned)(sl * lo) + kMagicBits;
          const long long want = (long long)kBinTerms * (sh * hi * 32768ll + sl * lo);
          const long long got = repeated(a, b, (unsigned)kBinTerms);
          if (got != want) expect(false, "a full bin's sum is off by", (double)(got - want));
        }
  {
    unsigned a, b;
    df_to_words(df32{268451840.0f, 16.0f}, 1.0f, a, b);  // 2^28 + 2^14 and its l
    expect(word(b) == 16400, "a low word above 2^14 + 1", word(b));
    const long long want = (long long)kBinTerms * 268451856ll;
    expect(repeated(a, b, (unsigned)kBinTerms) == want, "a full bin of it", (double)want);
  }
  return bad;
}
