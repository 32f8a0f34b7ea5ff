// dst_fx.h -- the FP64 path's DST-I in 64-bit block fixed point: the same
// half-length transform as dst_core.h, with every value of a row an integer
// times one power of two that the row's own data set.
//
// Why: this chip issues two FP64 operations per clock and SM, but 64-128
// integer ones.  A 1024-point DST is 18 FP64 operations per point; in
// integers its additions cost two instructions each on the wide pipes and
// its products six (fx_mul), and none runs on the FP64 pipe.
//
// Accuracy: a row enters at 59 bits below its largest value, additions are
// exact, and before each pass's twiddle products the row is shifted to 2^61
// by its measured magnitude (the bitwise OR of |v| over the row), so each
// pass's products round at about 2^-57 of the row's rms, and the tables hold
// 62 bits.  The prefix sum of the odd outputs, which multiplies the
// roundings before it by about sqrt(M) and in floating point adds one per
// term, adds none.  The error against exact arithmetic is below the FP64
// transform's (tests/test_fixed_point.py).
//
// A value v of a row stands for v 2^e, e the row's exponent.  A row whose
// largest magnitude is infinite or NaN has every output NaN, a row of zeros
// every output zero; magnitudes below 2^-957 round to multiples of 2^-1015.
//
// Work items as in dst_core.h: one item of one phase, any order within a
// phase.  Buffers hold 8-byte values in the padded layout of doubles.
#pragma once

#include "dst_core.h"

namespace qgw {

typedef long long fx_t;
template <> struct QGW_ALIGN(16) C2<fx_t> { fx_t x, y; };

// A fixed-point constant h 2^32 + l, both halves signed, so that a product
// takes signed 32-bit multiplies only.
struct QGW_ALIGN(8) Q2 { int h, l; };
struct QGW_ALIGN(16) Q4 { Q2 x, y; };

QGW_HD Q2 q2_split(fx_t w) {
  Q2 q;
  q.l = (int)w;
  q.h = (int)(w >> 32) - (q.l >> 31);
  return q;
}
QGW_HD fx_t q2_join(Q2 q) { return (fx_t)((unsigned long long)(unsigned int)q.h << 32) + q.l; }
// of a constant: l is never -2^31 (fx_mul negates it)
QGW_HD Q2 q2_const(fx_t w) { return q2_split((int)w == (int)0x80000000 ? w + 1 : w); }

// Tables: twq the pass twiddles (cos, -sin) scaled by 2^62, in the order of
// fill_pass_twiddles; nsj -s_j scaled by 2^63, j <= H (s_H = 1 has no
// positive 2^63); spq (cos, -sin)(2 pi k / M) scaled by 2^63, 1 <= k <= H/2.
// A projection's constants (modes_core.h): c 2^-k = (h 2^32 + l) 2^(e - 60) <
// 2^e, e per row of the matrix, k <= 0 per column.
struct ModeTable {
  const Q2* c;   // nl x nl, row m: output m
  const int* e;  // e (nl), k (nl)
};
// Chirp-z lengths (dst_blue.h): twq of the L-point FFT, bc the chirp c_m
// scaled by 2^62, m < M, bz the transform of its conjugate scaled by 2^(62 - be).
struct FxTables {
  const Q4* twq;
  const Q2* nsj;
  const Q4* spq;
  const Q4 *bc, *bz;
  int be;
};

QGW_HD int fx_mh(int a, int b) {
#ifdef __CUDA_ARCH__
  return __mulhi(a, b);
#else
  return (int)(((long long)a * b) >> 32);
#endif
}
QGW_HD int fx_clz(unsigned int v) {
#ifdef __CUDA_ARCH__
  return __clz((int)v);
#else
  return v ? __builtin_clz(v) : 32;
#endif
}

// v w / 2^64 to within one unit: one 32 x 32 -> 64 product and the high
// words of the two cross products, one truncated down and the other, of the
// negated constant, up: the errors cancel on average and a zero gives zero
// (a constant added against two truncations down would be an error of one
// sign wherever a product is exact -- zeros, or a factor of one -- and a
// transform adds those up in one bin).  |v| < 2^61.5; no constant has l =
// -2^31.
QGW_HD fx_t fx_mul(fx_t v, Q2 w) {
  const Q2 a = q2_split(v);
  return (fx_t)a.h * w.h + (fx_t)(fx_mh(a.l, w.h) - fx_mh(a.h, -w.l));
}
// (x + iy) w / 2^64, |w| components at most 2^62.  UP: the truncations the
// other way round, which matters for a factor of one (l = 0), whose remaining
// one is then up instead of down: the members of a butterfly alternate.
template <bool UP = false> QGW_HD void fx_cmul(fx_t& x, fx_t& y, const Q4& w) {
  const Q2 a = q2_split(x), b = q2_split(y);
  int t1, t2;
  if (UP) {
    const int nx = -w.x.h, ny = -w.y.h;
    t1 = fx_mh(a.h, w.x.l) + fx_mh(b.l, ny) - fx_mh(a.l, nx) - fx_mh(b.h, w.y.l);
    t2 = fx_mh(a.h, w.y.l) + fx_mh(b.h, w.x.l) - fx_mh(a.l, ny) - fx_mh(b.l, nx);
  } else {
    const int nx = -w.x.l, ny = -w.y.l;
    t1 = fx_mh(a.l, w.x.h) + fx_mh(b.h, ny) - fx_mh(a.h, nx) - fx_mh(b.l, w.y.h);
    t2 = fx_mh(a.l, w.y.h) + fx_mh(b.l, w.x.h) - fx_mh(a.h, ny) - fx_mh(b.h, nx);
  }
  x = ((fx_t)a.h * w.x.h + (fx_t)t1) - (fx_t)b.h * w.y.h;
  y = (fx_t)b.h * w.x.h + ((fx_t)a.h * w.y.h + (fx_t)t2);
}
// v c for a constant c = B + f, |f| < 1/2, f scaled by 2^64
template <int B> QGW_HD fx_t fx_mulc(fx_t v, int h, int l) {
  Q2 f;
  f.h = h;
  f.l = l;
  const fx_t p = fx_mul(v, f);
  return B == 1 ? v + p : B == -1 ? p - v : p;
}

QGW_HD fx_t fx_shl(fx_t v, int s) { return (fx_t)((unsigned long long)v << s); }
// v / 2^n rounded, ties to even: the roundings of a row must not share a
// sign, or the prefix sum would add M of them up
QGW_HD fx_t fx_shr(fx_t v, int n) { return (v + ((((fx_t)1 << n) >> 1) - 1 + ((v >> n) & 1))) >> n; }
QGW_HD fx_t fx_shift(fx_t v, int s) { return s >= 0 ? fx_shl(v, s > 63 ? 63 : s) : s < -62 ? 0 : fx_shr(v, -s); }
QGW_HD fx_t fx_shr0(fx_t v, int n) { return n > 0 ? fx_shr(v, n) : v; }
QGW_HD unsigned int fx_mag(fx_t v) {  // OR of these over values: their magnitude's bits above 2^32
  const int h = (int)(v >> 32);
  return (unsigned int)(h ^ (h >> 31));
}

// ---- doubles in and out
constexpr int FX_EMIN = 66;    // smallest biased exponent a row is scaled to
constexpr int FX_EOFF = 1081;  // X = x 2^(FX_EOFF - E) < 2^59, E the row's largest biased exponent
constexpr int FX_NAN = 1 << 20;  // row exponent of a non-finite row
constexpr int FX_ZERO = -FX_NAN;  // and of a row of zeros (v 2^e is 0)
// the scale's biased exponent of a row from its largest high word
QGW_HD int fx_scale(unsigned int mx) { return (int)(mx >> 20) < FX_EMIN ? FX_EMIN : (int)(mx >> 20); }

// x 2^(1075 + UP - E) of a double's bits, truncated; E at least its biased
// exponent
template <int UP = 6> QGW_HD fx_t fx_from_bits(unsigned long long b, int E) {
  const unsigned int hi = (unsigned int)(b >> 32);
  int sh = E - (int)((hi >> 20) & 0x7ffu);
  sh = sh > 63 ? 63 : sh;
  const unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32 | (b & 0xffffffffull)) << UP;
  const fx_t v = (fx_t)(m >> sh);
  return (int)hi < 0 ? -v : v;
}
// v 2^e rounded to a double; e from fx_exp_ok's range (fx_to_bits) or any
QGW_HD bool fx_exp_ok(int e) { return e >= -1020 && e <= 900; }
QGW_HD unsigned long long fx_to_bits(fx_t v, int e) {
  const unsigned long long sg = (unsigned long long)v & 0x8000000000000000ull;
  unsigned long long m = (unsigned long long)(v < 0 ? -v : v);
  unsigned int hi = (unsigned int)(m >> 32);
  int n = fx_clz(hi);
  if (hi == 0) {
    hi = (unsigned int)m;
    n = 32 + fx_clz(hi);
  }
  m <<= (n & 63);
  m = (m >> 11) + ((m >> 10) & 1);  // 53 bits, rounded; a carry moves into the exponent
  return (hi == 0 ? 0 : ((unsigned long long)(1085 + e - n) << 52) + m) | sg;
}

// ---- phase 1: pre-processing of raw doubles, items j = 1..H.  y_j / 2 =
// (x_j - x_{M-j}) / 4 + s_j (x_j + x_{M-j}) / 2; returns the item's part of
// sum |X| in units of 2^41, rounded up.
QGW_HD unsigned int fx_pre_item(const unsigned long long* x, fx_t* y, int j, int M, int E, const Q2* nsj) {
  const fx_t a = fx_from_bits(x[pr<double>(j)], E), b = fx_from_bits(x[pr<double>(M - j)], E);
  const fx_t p = fx_mul(a + b, nsj[j]);
  const fx_t d = fx_shr(a - b, 2);
  y[pr<double>(j)] = d - p;
  if (2 * j != M) y[pr<double>(M - j)] = -d - p;
  if (j == 1) y[0] = 0;
  const unsigned int la = (fx_mag(a) >> 9) + 1, lb = (fx_mag(b) >> 9) + 1;
  return 2 * j != M ? la + lb : la;
}

// ---- phase 2: forward DFTs (exact but for the products)
QGW_HD fx_t fx_hs(fx_t v) { return fx_mulc<1>(v, -1257966796, -102865788); }  // v sqrt(1/2)
QGW_HD void fx_dft8(C2<fx_t>* v) {
  C2<fx_t> a[4], b[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) { a[r] = cadd(v[r], v[r + 4]); b[r] = csub(v[r], v[r + 4]); }
  dft4<fx_t>(a);
  v[0] = a[0]; v[2] = a[1]; v[4] = a[2]; v[6] = a[3];
  // odd outputs: DFT4(b0, W b1, W^2 b2, W^3 b3), W = (1 - i)/sqrt 2
  const fx_t p1x = fx_hs(b[1].x + b[1].y), p1y = fx_hs(b[1].y - b[1].x);
  const fx_t p3x = fx_hs(b[3].y - b[3].x), p3y = -fx_hs(b[3].x + b[3].y);
  b[1].x = p1x; b[1].y = p1y;
  b[2] = cmi(b[2]);
  b[3].x = p3x; b[3].y = p3y;
  dft4<fx_t>(b);
  v[1] = b[0]; v[3] = b[1]; v[5] = b[2]; v[7] = b[3];
}
QGW_HD void fx_dft3(C2<fx_t>* v) {
  const C2<fx_t> t = cadd(v[1], v[2]), d = csub(v[1], v[2]);
  C2<fx_t> m, p;
  m.x = v[0].x - ((t.x + 1) >> 1); m.y = v[0].y - ((t.y + 1) >> 1);
  p.x = fx_mulc<1>(d.x, -575416509, -1033546850); p.y = fx_mulc<1>(d.y, -575416509, -1033546850);  // sin(2 pi/3)
  v[0] = cadd(v[0], t);
  v[1].x = m.x + p.y; v[1].y = m.y - p.x;
  v[2].x = m.x - p.y; v[2].y = m.y + p.x;
}
QGW_HD fx_t fx_c51(fx_t v) { return fx_mulc<0>(v, 1327217885, -1079689717); }   // cos(2 pi/5)
QGW_HD fx_t fx_c52(fx_t v) { return fx_mulc<-1>(v, 820265763, 1079689717); }    // cos(4 pi/5)
QGW_HD fx_t fx_s51(fx_t v) { return fx_mulc<1>(v, -210210662, 581434099); }     // sin(2 pi/5)
QGW_HD fx_t fx_s52(fx_t v) { return fx_mulc<1>(v, -1770448860, -1429016722); }  // sin(4 pi/5)
QGW_HD void fx_dft5(C2<fx_t>* v) {
  const C2<fx_t> t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]);
  const C2<fx_t> d1 = csub(v[1], v[4]), d2 = csub(v[2], v[3]);
  C2<fx_t> a, b, p, q;
  a.x = v[0].x + fx_c51(t1.x) + fx_c52(t2.x); a.y = v[0].y + fx_c51(t1.y) + fx_c52(t2.y);
  b.x = v[0].x + fx_c52(t1.x) + fx_c51(t2.x); b.y = v[0].y + fx_c52(t1.y) + fx_c51(t2.y);
  p.x = fx_s51(d1.x) + fx_s52(d2.x); p.y = fx_s51(d1.y) + fx_s52(d2.y);
  q.x = fx_s52(d1.x) - fx_s51(d2.x); q.y = fx_s52(d1.y) - fx_s51(d2.y);
  v[0] = cadd(v[0], cadd(t1, t2));
  v[1].x = a.x + p.y; v[1].y = a.y - p.x;
  v[4].x = a.x - p.y; v[4].y = a.y + p.x;
  v[2].x = b.x + q.y; v[2].y = b.y - q.x;
  v[3].x = b.x - q.y; v[3].y = b.y + q.x;
}
// cos, sin of 2 pi e / 7, e = 1, 2, 3
QGW_HD fx_t fx_c7(fx_t v, int e) {
  return e == 1 ? fx_mulc<1>(v, -1617098988, 1601080166)
       : e == 2 ? fx_mulc<0>(v, -955720134, -76219603)
                : fx_mulc<-1>(v, 425335474, -1524860563);
}
QGW_HD fx_t fx_s7(fx_t v, int e) {
  return e == 1 ? fx_mulc<1>(v, -937026648, 787634270)
       : e == 2 ? fx_mulc<1>(v, -107683797, -951367907)
                : fx_mulc<0>(v, 1863516470, -961608703);
}
QGW_HD void fx_dft7(C2<fx_t>* v) {
  C2<fx_t> t[3], d[3], y[7];
  for (int n = 0; n < 3; ++n) { t[n] = cadd(v[n + 1], v[6 - n]); d[n] = csub(v[n + 1], v[6 - n]); }
  y[0] = cadd(v[0], cadd(t[0], cadd(t[1], t[2])));
  for (int k = 1; k <= 3; ++k) {
    C2<fx_t> a = v[0], p;
    p.x = 0; p.y = 0;
    for (int n = 1; n <= 3; ++n) {
      const int e = (n * k) % 7, f = e <= 3 ? e : 7 - e;
      a.x += fx_c7(t[n - 1].x, f); a.y += fx_c7(t[n - 1].y, f);
      const fx_t sx = fx_s7(d[n - 1].x, f), sy = fx_s7(d[n - 1].y, f);
      p.x += e <= 3 ? sx : -sx; p.y += e <= 3 ? sy : -sy;
    }
    y[k].x = a.x + p.y; y[k].y = a.y - p.x;
    y[7 - k].x = a.x - p.y; y[7 - k].y = a.y + p.x;
  }
  for (int k = 0; k < 7; ++k) v[k] = y[k];
}
template <int R> QGW_HD void fx_dft(C2<fx_t>* v) {
  if (R == 8) fx_dft8(v);
  else if (R == 4) dft4<fx_t>(v);
  else if (R == 2) dft2<fx_t>(v);
  else if (R == 3) fx_dft3(v);
  else if (R == 5) fx_dft5(v);
  else fx_dft7(v);
}

// The shift before a pass's twiddles, from the OR of fx_mag over the row:
// |v| 2^s < 2^61.  The components of a product (/ 4) are below 2^59.5 and a
// radix-8 butterfly's outputs below 2^62.5; so are the first pass's
// (|y / 2| < 2^59).
QGW_HD int fx_pass_shift(unsigned int mag) { return 29 - (32 - fx_clz(mag)); }

// the members' twiddles w^(q k) (tw: the pass's table, entry (q-1) Ns + k)
// on the row shifted by s; every member is divided by 4
template <int R> QGW_HD void fx_twiddle(C2<fx_t>* v, int k, int Ns, int s, const Q4* tw) {
  if (s >= 0) {
#pragma unroll
    for (int q = 0; q < R; ++q) {
      v[q].x = fx_shl(v[q].x, s);
      v[q].y = fx_shl(v[q].y, s);
    }
  } else {
#pragma unroll
    for (int q = 0; q < R; ++q) {
      v[q].x = fx_shr(v[q].x, -s);
      v[q].y = fx_shr(v[q].y, -s);
    }
  }
  v[0].x = fx_shr(v[0].x, 2);
  v[0].y = fx_shr(v[0].y, 2);
#pragma unroll
  for (int q = 1; q < R; ++q) {
    if (q & 1) fx_cmul<true>(v[q].x, v[q].y, tw[(q - 1) * Ns + k]);
    else fx_cmul<false>(v[q].x, v[q].y, tw[(q - 1) * Ns + k]);
  }
}
template <int R> QGW_HD unsigned int fx_mag_all(const C2<fx_t>* v) {
  unsigned int m = 0;
#pragma unroll
  for (int q = 0; q < R; ++q) m |= fx_mag(v[q].x) | fx_mag(v[q].y);
  return m;
}
// Stockham pass, item b (stockham_item_k's indices); returns the OR of its
// outputs' magnitudes
template <int R>
QGW_HD unsigned int fx_stockham_item(const C2<fx_t>* src, C2<fx_t>* dst, int b, int k, int Ns, int H, int s,
                                     const Q4* tw) {
  const int stride = H / R;
  C2<fx_t> v[R];
#pragma unroll
  for (int q = 0; q < R; ++q) v[q] = src[pc<double>(b + q * stride)];
  if (Ns > 1) fx_twiddle<R>(v, k, Ns, s, tw);
  fx_dft<R>(v);
  const int base = (b - k) * R + k;
#pragma unroll
  for (int q = 0; q < R; ++q) dst[pc<double>(base + q * Ns)] = v[q];
  return fx_mag_all<R>(v);
}
template <int R>
QGW_HD_NOINLINE unsigned int fx_stockham_item_far(const C2<fx_t>* src, C2<fx_t>* dst, int b, int k, int Ns, int H,
                                                  int s, const Q4* tw) {
#ifdef __CUDA_ARCH__
  // a function of its own does not see that its rows lie in shared memory
  __builtin_assume(__isShared(src));
  __builtin_assume(__isShared(dst));
#endif
  return fx_stockham_item<R>(src, dst, b, k, Ns, H, s, tw);
}
// tw: the table of the pass (twq + Ns - R0)
QGW_HD unsigned int fx_stockham_dispatch(int R, const C2<fx_t>* src, C2<fx_t>* dst, int b, int k, int Ns, int H, int s,
                                         const Q4* tw) {
  switch (R) {
    case 8: return fx_stockham_item_far<8>(src, dst, b, k, Ns, H, s, tw);
    case 4: return fx_stockham_item_far<4>(src, dst, b, k, Ns, H, s, tw);
    case 2: return fx_stockham_item_far<2>(src, dst, b, k, Ns, H, s, tw);
    case 3: return fx_stockham_item_far<3>(src, dst, b, k, Ns, H, s, tw);
    case 5: return fx_stockham_item_far<5>(src, dst, b, k, Ns, H, s, tw);
    default: return fx_stockham_item_far<7>(src, dst, b, k, Ns, H, s, tw);
  }
}

// ---- phase 3: split.  Shift s of Z: below 2^59 (a doubled difference
// enters a product), and so that |Y| <= 2 sum |X| stays below 2^62 (the
// prefix sums of the odd outputs are outputs, and wrapped intermediate sums
// of integers do no harm).  l1: sum of fx_pre_item's values; drop: the
// passes' sum of 2 - shift.
QGW_HD int fx_split_shift(unsigned int mag, unsigned int l1, int drop) {
  const int a = 27 - (32 - fx_clz(mag)), b = 21 - (32 - fx_clz(l1)) + drop;
  return a < b ? a : b;
}
// exponent of the row's outputs (mx: its largest high word)
QGW_HD int fx_row_exp(unsigned int mx, int drop, int s) {
  return mx == 0 ? FX_ZERO : mx >= 0x7ff00000u ? FX_NAN : fx_scale(mx) - FX_EOFF + 1 + drop - s;
}

QGW_HD int fx_exp_add(int ex, int d) { return ex == FX_NAN || ex == FX_ZERO ? ex : ex + d; }

QGW_HD void fx_split_pair(C2<fx_t> A, C2<fx_t> B, const Q4& cs, C2<fx_t>& lo, C2<fx_t>& hi) {
  const fx_t sr = A.x + B.x, si = A.y - B.y, dr = 2 * (A.x - B.x), di = 2 * (A.y + B.y);
  const fx_t P = fx_mul(di, cs.x) + fx_mul(dr, cs.y);  // c di - s dr
  const fx_t Q = fx_mul(dr, cs.x) - fx_mul(di, cs.y);  // c dr + s di
  lo.x = Q - si;  // Y_{2k}
  lo.y = sr + P;  // 2 R_k
  hi.x = Q + si;  // Y_{2(H-k)}
  hi.y = sr - P;  // 2 R_{H-k}
}
QGW_HD C2<fx_t> fx_shift2(C2<fx_t> v, int s) {
  v.x = fx_shift(v.x, s);
  v.y = fx_shift(v.y, s);
  return v;
}
QGW_HD void fx_split_item(const C2<fx_t>* Z, C2<fx_t>* o, int k, int H, int s, const Q4* spq) {
  if (k == 0) {
    const C2<fx_t> a = fx_shift2(Z[0], s);
    C2<fx_t> z0;
    z0.x = 0;
    z0.y = a.x + a.y;  // R_0
    o[0] = z0;
    return;
  }
  C2<fx_t> lo, hi;
  fx_split_pair(fx_shift2(Z[pc<double>(k)], s), fx_shift2(Z[pc<double>(H - k)], s), spq[k], lo, hi);
  o[pc<double>(k)] = lo;
  if (2 * k != H) o[pc<double>(H - k)] = hi;
}

// ---- real FFT of N = 2H reals (periodic.cuh's forms), scaled by 2: the split
// of Z (below 2^59) into 2 X_k, 2 X_{H-k}, 1 <= k <= H/2, cs = spq[k]
QGW_HD int fx_rsplit_shift(unsigned int mag) { return 27 - (32 - fx_clz(mag)); }
QGW_HD void fx_rsplit_pair(C2<fx_t> A, C2<fx_t> B, const Q4& cs, C2<fx_t>& xk, C2<fx_t>& xh) {
  const fx_t Pr = A.x + B.x, Pi = A.y - B.y, Qr = 2 * (A.x - B.x), Qi = 2 * (A.y + B.y);
  const fx_t Vr = fx_mul(Qi, cs.x) + fx_mul(Qr, cs.y);  // c Qi - s Qr
  const fx_t Vi = fx_mul(Qi, cs.y) - fx_mul(Qr, cs.x);  // -(c Qr + s Qi)
  xk.x = Pr + Vr; xk.y = Pi + Vi;
  xh.x = Pr - Vr; xh.y = Vi - Pi;
}
// and its inverse: conj Z'_k, conj Z'_{H-k} of X_k, X_{H-k} (below 2^59),
// divided by 8 (below 2^59 again)
QGW_HD void fx_rjoin_pair(C2<fx_t> a, C2<fx_t> b, const Q4& cs, C2<fx_t>& zk, C2<fx_t>& zh) {
  const fx_t Pr = a.x + b.x, Pi = a.y - b.y, Qr = 2 * (a.x - b.x), Qi = 2 * (a.y + b.y);
  const fx_t Ui = fx_mul(Qr, cs.x) + fx_mul(Qi, cs.y);  // c Qr - s Qi
  const fx_t Ur = fx_mul(Qr, cs.y) - fx_mul(Qi, cs.x);  // -(c Qi + s Qr)
  zk.x = fx_shr(Pr + Ur, 3); zk.y = -fx_shr(Pi + Ui, 3);
  zh.x = fx_shr(Pr - Ur, 3); zh.y = fx_shr(Pi - Ui, 3);
}
// item k = 0..H/2 of the join from raw doubles X (k complex values) to Z
QGW_HD C2<fx_t> fx_raw2(const C2<double>* x, int k, int E) {
  const unsigned long long* p = (const unsigned long long*)(x + pc<double>(k));
  C2<fx_t> v;
  v.x = fx_from_bits(p[0], E);
  v.y = fx_from_bits(p[1], E);
  return v;
}
QGW_HD void fx_rjoin_item(const C2<double>* X, C2<fx_t>* Z, int k, int H, int E, const Q4* spq) {
  C2<fx_t> a = fx_raw2(X, k, E), b = fx_raw2(X, H - k, E), zk, zh;
  if (k == 0) {
    // X_0 and X_H are real: Z'_0 = (X_0 + X_H) + i (X_0 - X_H)
    zk.x = fx_shr(a.x + b.x, 3);
    zk.y = -fx_shr(a.x - b.x, 3);
    Z[0] = zk;
    return;
  }
  fx_rjoin_pair(a, b, spq[k], zk, zh);
  Z[pc<double>(k)] = zk;
  if (2 * k != H) Z[pc<double>(H - k)] = zh;
}
QGW_HD void fx_rsplit_item(const C2<fx_t>* Z, C2<fx_t>* X, int k, int H, int s, const Q4* spq) {
  if (k == 0) {
    const C2<fx_t> a = fx_shift2(Z[0], s);
    C2<fx_t> x0, xH;
    x0.x = 2 * (a.x + a.y); x0.y = 0;
    xH.x = 2 * (a.x - a.y); xH.y = 0;
    X[0] = x0;
    X[pc<double>(H)] = xH;
    return;
  }
  C2<fx_t> xk, xh;
  fx_rsplit_pair(fx_shift2(Z[pc<double>(k)], s), fx_shift2(Z[pc<double>(H - k)], s), spq[k], xk, xh);
  X[pc<double>(k)] = xk;
  if (2 * k != H) X[pc<double>(H - k)] = xh;
}

// ---- chirp-z DST-I (dst_blue.h)
// z_m = x_m c_m (the value below 2^61, its product / 4), zero outside 1 <= m <
// M, of a raw row
QGW_HD void fx_chirp_item(const unsigned long long* x, C2<fx_t>* z, int m, int M, int E, const Q4* bc) {
  C2<fx_t> v;
  v.x = v.y = 0;
  if (m >= 1 && m < M) {
    const fx_t X = fx_from_bits<8>(x[pr<double>(m)], E);
    v.x = fx_mul(X, bc[m].x);
    v.y = fx_mul(X, bc[m].y);
  }
  z[pc<double>(m)] = v;
}
// conj(z_k bz_k) / 4 of the row shifted by s to below 2^61, in place
QGW_HD void fx_chirp_mul_item(C2<fx_t>* z, int k, int s, const Q4* bz) {
  C2<fx_t> v = fx_shift2(z[pc<double>(k)], s);
  fx_cmul(v.x, v.y, bz[k]);
  v.y = -v.y;
  z[pc<double>(k)] = v;
}
// Im(c_k conj d_k) / 4 of the row shifted by s, into y (index k); Y_k is 2 / L
// times it
QGW_HD void fx_chirp_out_item(const C2<fx_t>* d, fx_t* y, int k, int s, const Q4* bc) {
  if (k == 0) {
    y[0] = 0;
    return;
  }
  const C2<fx_t> v = fx_shift2(d[pc<double>(k)], s);
  y[pr<double>(k)] = fx_mul(v.x, bc[k].y) - fx_mul(v.y, bc[k].x);
}

}  // namespace qgw
