// dst_tables.h -- host construction of the DST-I tables of dst_core.h, in
// FP64 with exactly reduced angles (one libm rounding per entry).
#pragma once

#include <cmath>
#include <utility>
#include <vector>

#include "dst_core.h"
#include "dst_fx.h"

namespace qgw {

// sin(pi * m / N) for integer m, reduced exactly to [0, pi/2]
inline double sinpi_frac(long m, long N) {
  long r = m % (2 * N);
  if (r < 0) r += 2 * N;
  double sg = 1.0;
  if (r >= N) { r -= N; sg = -1.0; }
  if (2 * r > N) r = N - r;
  return sg * std::sin(M_PI * (double)r / (double)N);
}
// cos(pi m / N) = sin(pi (2m + N) / (2N))
inline double cospi_frac(long m, long N) { return sinpi_frac(2 * m + N, 2 * N); }

struct DstTablesHost {
  std::vector<double> tw, pre, spl, twp;  // interleaved (x, y) pairs
  std::vector<double> sj;                 // sin(pi j / M), j = 0..H
  // the warp transform's tables (H = 256, 512; one dummy pair otherwise):
  std::vector<double> twd;  // DIF twiddles: w_H^(n1 k2) at (k2-1) S0 + n1, then w_H^(8 n1 k2) at 7 S0 + (k2-1) S1 + n1
  std::vector<double> sjp;  // (s_{2m}, s_{2m+1}), m < H
};

// tw: H entries, twp: H - R0 entries, pre: H+1 entries, spl: H/2+1 entries
inline DstTablesHost build_dst_tables(int M) {
  const int H = M / 2;
  DstTablesHost t;
  t.tw.resize(2 * (size_t)H);
  for (int m = 0; m < H; ++m) {
    // 2 pi m / H = pi (2m) / H
    t.tw[2 * m] = cospi_frac(2L * m, H);
    t.tw[2 * m + 1] = -sinpi_frac(2L * m, H);
  }
  const DstGeom g = make_geom(M);
  t.twp.assign(2 * (size_t)(g.npass ? H - g.radix[0] : 0) + 2, 0.0);
  fill_pass_twiddles(g, t.tw.data(), t.twp.data());
  t.pre.resize(2 * (size_t)(H + 1));
  t.sj.resize((size_t)H + 1);
  for (int j = 0; j <= H; ++j) {
    const double s = sinpi_frac(j, M);
    t.pre[2 * j] = s + 0.5;
    t.pre[2 * j + 1] = s - 0.5;
    t.sj[j] = s;
  }
  t.spl.resize(2 * (size_t)(H / 2 + 1));
  for (int k = 0; k <= H / 2; ++k) {
    t.spl[2 * k] = cospi_frac(2L * k, M);
    t.spl[2 * k + 1] = sinpi_frac(2L * k, M);
  }
  t.twd.assign(2, 0.0);
  t.sjp.assign(2, 0.0);
  if (H == 256 || H == 512) {
    const int S0 = H / 8, S1 = H / 64;
    t.twd.assign(2 * (size_t)7 * (S0 + S1), 0.0);
    for (int k2 = 1; k2 < 8; ++k2) {
      for (int n1 = 0; n1 < S0; ++n1) {
        const int e = (k2 - 1) * S0 + n1, m = (n1 * k2) % H;
        t.twd[2 * e] = t.tw[2 * m];
        t.twd[2 * e + 1] = t.tw[2 * m + 1];
      }
      for (int n1 = 0; n1 < S1; ++n1) {
        const int e = 7 * S0 + (k2 - 1) * S1 + n1, m = (8 * n1 * k2) % H;
        t.twd[2 * e] = t.tw[2 * m];
        t.twd[2 * e + 1] = t.tw[2 * m + 1];
      }
    }
    t.sjp.resize(2 * (size_t)H);
    for (int m = 0; m < H; ++m) {
      const int j0 = 2 * m, j1 = 2 * m + 1;
      t.sjp[2 * m] = t.sj[j0 <= H ? j0 : M - j0];
      t.sjp[2 * m + 1] = t.sj[j1 <= H ? j1 : M - j1];
    }
  }
  return t;
}

// cos and -sin of pi m / N scaled by 2^b, b <= 63, N up to 2^14, by
// their Taylor series in 64-bit fixed point to 2^-61: the fixed-point
// transform (dst_fx.h) rounds at 2^-57, so it would feel the rounding of a
// double.  At b = 63 a value of +1 does not fit (no table holds one).
inline Q4 sincospi_fixed(long m, long N, int b) {
  typedef unsigned long long u64;
  auto hi = [](u64 a, u64 c) { return (u64)(((unsigned __int128)a * c) >> 64); };
  long r = m % (2 * N);
  if (r < 0) r += 2 * N;
  const bool half = r >= N;  // both signs change
  if (half) r -= N;
  const bool refl = 2 * r > N;  // the cosine's changes
  if (refl) r = N - r;
  const bool swap = 4 * r > N;
  const long a = swap ? N - 2 * r : 2 * r;  // the angle is pi a / (2 N), at most pi / 4
  // pi / 4 in units of 2^-64, times 2 a / N <= 1
  const u64 pi4 = 0xC90FDAA22168C235ull;
  const u64 t = (u64)(((unsigned __int128)pi4 * (u64)(2 * a)) / (u64)N);
  const u64 t2 = hi(t, t);
  u64 s = ~0ull, c = ~0ull;  // 1 - 2^-64
  for (int k = 11; k >= 1; --k) {
    s = ~0ull - hi(t2 / (u64)((2 * k) * (2 * k + 1)), s);
    c = ~0ull - hi(t2 / (u64)((2 * k - 1) * (2 * k)), c);
  }
  s = hi(t, s);
  // round from 2^-64 to 2^-b
  const int n = 64 - b;
  u64 S = a == 0 ? 0 : (s >> n) + ((s >> (n - 1)) & 1), C = a == 0 ? 1ull << b : (c >> n) + ((c >> (n - 1)) & 1);
  if (swap) std::swap(S, C);
  // two's complement negation carries 2^63 to the value -1 has
  Q4 w;
  w.x = q2_const((fx_t)(half != refl ? 0 - C : C));
  w.y = q2_const((fx_t)(half ? S : 0 - S));
  return w;
}

// The tables of the fixed-point transform (dst_fx.h) of geometry g, into
// arrays of fx_twq_len, H/2 + 1 and H + 1 entries.
inline size_t fx_twq_len(const DstGeom& g) { return (size_t)(g.npass ? g.H - g.radix[0] : 0) + 1; }
inline void fill_fx_twiddles(const DstGeom& g, Q4* twq) {
  int Ns = g.radix[0];
  for (int p = 1; p < g.npass; ++p) {
    const int R = g.radix[p];
    for (int q = 1; q < R; ++q)
      for (int k = 0; k < Ns; ++k) twq[(Ns - g.radix[0]) + (q - 1) * Ns + k] = sincospi_fixed(2L * q * k, (long)Ns * R, 62);
    Ns *= R;
  }
}
inline void fill_fx_tables(const DstGeom& g, Q4* twq, Q4* spq, Q2* nsj) {
  const int H = g.H, M = g.M;
  fill_fx_twiddles(g, twq);
  spq[0] = Q4{};
  for (int k = 1; k <= H / 2; ++k) spq[k] = sincospi_fixed(2L * k, M, 63);
  for (int j = 0; j <= H; ++j) nsj[j] = sincospi_fixed(j, M, 63).y;
}
// The chirp-z tables of g (g.blue): bc (M entries), bz (L = g.H entries) and
// bz's exponent.  bz is the transform's own FFT of the conjugate chirp, run
// with the device's work items; twq: g's pass twiddles.
inline int fill_fx_blue(const DstGeom& g, const Q4* twq, Q4* bc, Q4* bz) {
  const int M = g.M, L = g.H;
  std::vector<C2<fx_t>> a((size_t)pc<double>(L) + 1, C2<fx_t>{0, 0}), b(a.size());
  auto join = [](Q2 q) { return ((fx_t)q.h << 32) + q.l; };
  for (int m = 0; m < M; ++m) {
    const long e = ((long)m * m) % (4L * M);  // exp(i pi e / 2M)
    bc[m] = sincospi_fixed(-e, 2L * M, 62);
    // b at d mod L, d in (-M, M): conj(c_|d|)
    const Q4 w = sincospi_fixed(e, 2L * M, 58);
    a[pc<double>(m)].x = a[pc<double>((L - m) % L)].x = join(w.x);
    a[pc<double>(m)].y = a[pc<double>((L - m) % L)].y = join(w.y);
  }
  C2<fx_t>*src = a.data(), *dst = b.data();
  int Ns = 1, drop = 0;
  unsigned int mag = 0;
  for (int p = 0; p < g.npass; ++p) {
    const int R = g.radix[p], s = p ? fx_pass_shift(mag) : 0;
    if (p) drop += 2 - s;
    mag = 0;
    for (int i = 0; i < L / R; ++i)
      mag |= fx_stockham_dispatch(R, src, dst, i, i % Ns, Ns, L, s, twq + (p ? Ns - g.radix[0] : 0));
    Ns *= R;
    std::swap(src, dst);
  }
  double mx = 0;
  for (int k = 0; k < L; ++k) mx = std::fmax(mx, std::hypot((double)src[pc<double>(k)].x, (double)src[pc<double>(k)].y));
  int e;
  std::frexp(mx, &e);  // modulus < 2^e: up to 2^62
  const int up = 62 - e;
  for (int k = 0; k < L; ++k) {
    const C2<fx_t> v = fx_shift2(src[pc<double>(k)], up);
    bz[k] = Q4{q2_const(v.x), q2_const(v.y)};
  }
  return 62 - 58 + drop - up;  // value = bz 2^(drop - 58 - up)
}
struct FxTablesHost {
  std::vector<Q4> twq, spq, bc, bz;
  std::vector<Q2> nsj;
  int be = 0;
};
inline FxTablesHost build_fx_tables(const DstGeom& g) {
  FxTablesHost t;
  t.twq.resize(fx_twq_len(g));
  t.spq.resize((size_t)g.H / 2 + 1);
  t.nsj.resize((size_t)g.H + 1);
  if (g.blue) {
    fill_fx_twiddles(g, t.twq.data());
    t.bc.resize(g.M);
    t.bz.resize(g.H);
    t.be = fill_fx_blue(g, t.twq.data(), t.bc.data(), t.bz.data());
  } else {
    fill_fx_tables(g, t.twq.data(), t.spq.data(), t.nsj.data());
  }
  return t;
}

// Whether a projection runs in fixed point (modes_core.h): at most 20 terms,
// and the largest entries of the matrix's columns within a factor of 20.
// Per layer, what the projections give psi is then no larger than with FP64
// sums: 20 layers of ratio 1.3 (factor 17) 1.3 against 2.0 units of 2^-53 at
// the worst field; 16 of ratio 1.5 (factor 23) 8 against 3, 32 of ratio 1.3
// 20 against 5.
inline bool modes_fixed_ok(int nl, const double* mat) {
  if (nl > 20) return false;
  double lo = 0, hi = 0;
  for (int l = 0; l < nl; ++l) {
    double mx = 0;
    for (int m = 0; m < nl; ++m) mx = std::fmax(mx, std::fabs(mat[(size_t)m * nl + l]));
    lo = l ? std::fmin(lo, mx) : mx;
    hi = std::fmax(hi, mx);
  }
  return lo > 0 && hi <= 20 * lo && hi < 1e150 && lo > 1e-150;
}
// A projection matrix (nl x nl, row m: output m) in fixed point: every column
// by the power of two k of its largest entry (the largest column's 0), then
// every row by its largest entry.  e: 2 nl, as ModeTable's.
inline void fill_mode_table(int nl, const double* mat, Q2* c, int* e) {
  int* k = e + nl;
  int top = -10000;
  for (int l = 0; l < nl; ++l) {
    double mx = 0;
    for (int m = 0; m < nl; ++m) mx = std::fmax(mx, std::fabs(mat[(size_t)m * nl + l]));
    std::frexp(mx, &k[l]);
    top = k[l] > top ? k[l] : top;
  }
  for (int l = 0; l < nl; ++l) k[l] -= top;
  for (int m = 0; m < nl; ++m) {
    double mx = 0;
    for (int l = 0; l < nl; ++l) mx = std::fmax(mx, std::ldexp(std::fabs(mat[(size_t)m * nl + l]), -k[l]));
    std::frexp(mx, &e[m]);
    for (int l = 0; l < nl; ++l)
      c[m * nl + l] = q2_const((fx_t)std::nearbyint(std::ldexp(mat[(size_t)m * nl + l], 60 - e[m] - k[l])));
  }
}

}  // namespace qgw
