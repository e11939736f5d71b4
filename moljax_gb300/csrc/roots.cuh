// Host tables of roots of unity and of Bluestein's chirp and filter, in double-double arithmetic
// (a value is the unevaluated sum h + l; error-free sums and products of Knuth and Dekker).
//
// A table is the same for every row and step, so the errors of its entries do not average out, and
// an angle rounded to FP64 is off by up to 7e-16 at 2 pi: a chirp exp(-i pi j^2 / n) formed from it,
// and a filter transformed in FP64, gave the FP64 Bluestein transforms twice the error of their own
// arithmetic (a pair of 1999 x 6 points 7.9e-16, 4.8e-16 with these tables).  The long double
// functions, which the Arm host runs in software, take ten to thirty times as long (4096^2
// FP64 plan: 5.8 ms, 0.4 ms here).
#pragma once

#include <math.h>

#include <utility>
#include <vector>

namespace mjx {

struct DD { double h, l; };

inline DD dd_fast(double a, double b) {  // |a| >= |b|
  const double s = a + b;
  return {s, b - (s - a)};
}
inline DD dd_add(DD a, DD b) {
  const double s = a.h + b.h, t = s - a.h;
  return dd_fast(s, ((a.h - (s - t)) + (b.h - t)) + (a.l + b.l));
}
inline DD dd_neg(DD a) { return {-a.h, -a.l}; }
inline DD dd_mul(DD a, DD b) {
  const double p = fma(a.h, b.h, 0.0);  // rounded here: a host compiler may fuse a plain product into a sum
  return dd_fast(p, fma(a.h, b.h, -p) + (a.h * b.l + a.l * b.h));
}
inline DD dd_div(DD a, double d) {
  const double q = a.h / d;
  return dd_fast(q, (fma(-q, d, a.h) + a.l) / d);
}

// cos and sin of x, 0 <= x <= pi, by their power series
inline void dd_cis(DD x, DD* c, DD* s) {
  const DD x2 = dd_neg(dd_mul(x, x));
  DD tc = {1.0, 0.0}, ts = x;
  *c = tc;
  *s = ts;
  for (int k = 1; k < 30 && (fabs(tc.h) > 1e-33 || fabs(ts.h) > 1e-33); ++k) {
    tc = dd_div(dd_mul(tc, x2), (2.0 * k - 1.0) * (2.0 * k));
    ts = dd_div(dd_mul(ts, x2), (2.0 * k) * (2.0 * k + 1.0));
    *c = dd_add(*c, tc);
    *s = dd_add(*s, ts);
  }
}

// cos and sin of 2 pi j / m for j = 0 .. m - 1: up to pi / 2 (pi for an odd m) each the product of
// two entries of short tables, the rest by symmetry.
struct Roots {
  std::vector<DD> c, s;
  explicit Roots(int m) : c(m), s(m) {
    const DD pi2 = {6.283185307179586, 2.4492935982947064e-16};
    const int half = m / 2, top = m % 2 ? half : m / 4;
    int B = 1;
    while (B * B < top + 1) B <<= 1;
    std::vector<DD> hc(top / B + 1), hs(top / B + 1);
    for (int b = 0; b < B && b <= top; ++b) dd_cis(dd_div(dd_mul(pi2, {(double)b, 0.0}), m), &c[b], &s[b]);
    for (int a = 1; a <= top / B; ++a) dd_cis(dd_div(dd_mul(pi2, {(double)a * B, 0.0}), m), &hc[a], &hs[a]);
    for (int j = B; j <= top; ++j) {
      const int a = j / B, b = j - a * B;
      c[j] = dd_add(dd_mul(hc[a], c[b]), dd_neg(dd_mul(hs[a], s[b])));
      s[j] = dd_add(dd_mul(hs[a], c[b]), dd_mul(hc[a], s[b]));
    }
    if (m % 4 == 0) { c[top] = {0.0, 0.0}; s[top] = {1.0, 0.0}; }
    for (int j = top + 1; j <= half && j < m; ++j) { c[j] = dd_neg(c[half - j]); s[j] = s[half - j]; }
    for (int j = half + 1; j < m; ++j) { c[j] = c[m - j]; s[j] = dd_neg(s[m - j]); }
  }
};

// radix-2 FFT in place, F = DD or double
template <typename F>
struct HostFft {
  static void run(std::vector<F>& re, std::vector<F>& im, const Roots& r) {
    const int L = (int)re.size();
    for (int i = 1, j = 0; i < L; ++i) {
      int bit = L >> 1;
      for (; j & bit; bit >>= 1) j ^= bit;
      j ^= bit;
      if (i < j) { std::swap(re[i], re[j]); std::swap(im[i], im[j]); }
    }
    for (int len = 2; len <= L; len <<= 1)
      for (int k = 0; k < len / 2; ++k) {
        const F wr = pick(r.c[k * (L / len)]), wi = pick(r.s[k * (L / len)]);  // w = wr - i wi
        for (int u = k; u < L; u += len) {
          const int v = u + len / 2;
          const F xr = k ? add(mul(re[v], wr), mul(im[v], wi)) : re[v], xi = k ? sub(mul(im[v], wr), mul(re[v], wi)) : im[v];
          re[v] = sub(re[u], xr); im[v] = sub(im[u], xi);
          re[u] = add(re[u], xr); im[u] = add(im[u], xi);
        }
      }
  }
  static F pick(DD a) { F f; set(f, a); return f; }
  static void set(double& f, DD a) { f = a.h; }
  static void set(DD& f, DD a) { f = a; }
  static double add(double a, double b) { return a + b; }
  static double sub(double a, double b) { return a - b; }
  static double mul(double a, double b) { return a * b; }
  static DD add(DD a, DD b) { return dd_add(a, b); }
  static DD sub(DD a, DD b) { return dd_add(a, dd_neg(b)); }
  static DD mul(DD a, DD b) { return dd_mul(a, b); }
  static double value(double a) { return a; }
  static double value(DD a) { return a.h; }
};

// Bluestein's filter FFT_L(b) / L, b[j] = exp(i pi j^2 / n) for |j| < n, from the roots q of 2 n and r of L
template <typename F>
inline void bluestein_filter(int n, const Roots& q, const Roots& r, std::vector<double>* bhat) {
  const int L = (int)r.c.size();
  std::vector<F> re(L), im(L);
  for (int j = 0; j < n; ++j) {
    const int k = (int)(((long long)j * j) % (2LL * n));  // exp(i pi j^2 / n), conj of the chirp
    const F c = HostFft<F>::pick(q.c[k]), s = HostFft<F>::pick(q.s[k]);
    re[j] = c; im[j] = s;
    if (j > 0) { re[L - j] = c; im[L - j] = s; }
  }
  HostFft<F>::run(re, im, r);
  bhat->resize(2 * (size_t)L);
  for (int j = 0; j < L; ++j) {  // L is a power of two: exact
    (*bhat)[2 * j] = HostFft<F>::value(re[j]) / L;
    (*bhat)[2 * j + 1] = HostFft<F>::value(im[j]) / L;
  }
}

// The tables of a DFT of length n by transforms of length L (a power of two, roots r), re and im
// interleaved: chirp[j] = exp(-i pi j^2 / n) and the filter; `wide`: the filter's transform in
// double-double, for FP64 plans.
inline void bluestein_tables(int n, const Roots& r, bool wide, std::vector<double>* chirp, std::vector<double>* bhat) {
  const Roots q(2 * n);
  chirp->resize(2 * (size_t)n);
  for (int j = 0; j < n; ++j) {
    const int k = (int)(((long long)j * j) % (2LL * n));
    (*chirp)[2 * j] = q.c[k].h;
    (*chirp)[2 * j + 1] = -q.s[k].h;
  }
  if (wide) bluestein_filter<DD>(n, q, r, bhat);
  else bluestein_filter<double>(n, q, r, bhat);
}

}  // namespace mjx
