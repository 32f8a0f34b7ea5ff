// CPU check of the device DST-I building blocks (qgw_gb300/csrc/dst_core.h):
// runs every phase's work items in a plain loop, exactly as the kernels
// spread them over threads, and exposes the result through a C function.
#include <algorithm>
#include <cmath>
#include <vector>
#include <cstring>
#include "../../qgw_gb300/csrc/dst_tables.h"
#include "../../qgw_gb300/csrc/dst_warp.h"
#include "../../qgw_gb300/csrc/dst_blue.h"
#include "../../qgw_gb300/csrc/modes_core.h"
#include "../../qgw_gb300/csrc/rhs_core.h"

using namespace qgw;

template <typename T>
static void run(int M, int howmany, T* data) {
  DstGeom g = make_geom(M);
  DstTablesHost th = build_dst_tables(M);
  std::vector<T> tw(th.tw.begin(), th.tw.end()), pre(th.pre.begin(), th.pre.end()),
      spl(th.spl.begin(), th.spl.end());
  const C2<T>* TW = (const C2<T>*)tw.data();
  const C2<T>* PRE = (const C2<T>*)pre.data();
  const C2<T>* SPL = (const C2<T>*)spl.data();
  std::vector<T> A(padded_len<T>(M)), B(padded_len<T>(M));
  for (int r = 0; r < howmany; ++r) {
    T* x = data + (size_t)r * (M - 1);
    for (size_t j = 0; j < A.size(); ++j) A[j] = B[j] = T(777);  // pad slots must never be read
    for (int j = 0; j < M - 1; ++j) A[pr<T>(j + 1)] = x[j];      // x_j at index j
    A[pr<T>(0)] = T(12345);  // index 0 must never be read
    for (int j = 1; j <= g.H; ++j) dst_pre_item<T>(A.data(), B.data(), j, g, PRE);
    T* src = B.data();
    T* dst = A.data();
    int Ns = 1;
    for (int p = 0; p < g.npass; ++p) {
      const int R = g.radix[p];
      for (int b = 0; b < g.H / R; ++b)
        stockham_dispatch<T>(R, (const C2<T>*)src, (C2<T>*)dst, b, Ns, g.H, TW);
      Ns *= R;
      T* t = src; src = dst; dst = t;
    }
    // result in src; split into dst
    for (int k = 0; k <= g.H / 2; ++k) dst_split_item<T>((const C2<T>*)src, dst, k, g, SPL);
    std::vector<T> tot(g.nchunk);
    for (int c = 0; c < g.nchunk; ++c) tot[c] = dst_scan_chunk<T>(dst, c, g);
    T pref = T(0);
    for (int c = 0; c < g.nchunk; ++c) {
      if (c > 0) dst_scan_fix<T>(dst, c, pref, g);
      pref += tot[c];
    }
    for (int j = 0; j < M - 1; ++j) x[j] = dst[pr<T>(j + 1)];  // Y_k at index k
  }
}

// The one-warp transform (dst_warp.h) with its 32 lanes run one after the
// other inside each phase, every phase's reads done before its writes where
// the device code synchronises the warp in between; the lane-to-lane value
// of pass 1 (x_{M-2m}) taken as the device's shuffle delivers it.  The
// split's inputs are read through WarpDst::split_read (the digit-reversed
// positions) into a natural-order row, which the split and scan items of
// dst_core.h finish.
template <int LGH>
static void run_warp(int howmany, float* data) {
  using W = WarpDst<LGH>;
  constexpr int H = W::H, M = W::M, IPL = W::IPL, KPL = W::KPL;
  DstGeom g = make_geom(M);
  DstTablesHost th = build_dst_tables(M);
  std::vector<float> twd(th.twd.begin(), th.twd.end()), sjp(th.sjp.begin(), th.sjp.end()),
      spl(th.spl.begin(), th.spl.end());
  const C2<float>* TWD = (const C2<float>*)twd.data();
  const C2<float>* SJP = (const C2<float>*)sjp.data();
  const C2<float>* SPL = (const C2<float>*)spl.data();
  const int L = padded_len<float>(M);
  std::vector<F4> Abuf((L + 3) / 4), Bbuf((L + 3) / 4), Cbuf((L + 3) / 4);
  float* A = (float*)Abuf.data();
  float* B = (float*)Bbuf.data();
  float* Cr = (float*)Cbuf.data();
  static C2<float> own[32][IPL][8], mir[32][IPL][8], v[32][IPL][8];
  for (int r = 0; r < howmany; ++r) {
    float* x = data + (size_t)r * (M - 1);
    for (int j = 0; j < L; ++j) A[j] = B[j] = Cr[j] = 777.f;  // pad slots must never be read
    for (int j = 0; j < M - 1; ++j) A[pr<float>(j + 1)] = x[j];
    A[pr<float>(0)] = 12345.f;  // index 0 must never be read
    C2<float>* Z = (C2<float>*)A;
    for (int lane = 0; lane < 32; ++lane)
      for (int n2 = 0; n2 < 8; ++n2)
        for (int u = 0; u < IPL; ++u) W::p1_read(lane + 32 * u + W::S0 * n2, Z, own[lane][u][n2], mir[lane][u][n2]);
    for (int lane = 0; lane < 32; ++lane) {
      float prev = 0.f;
      for (int n2 = 0; n2 < 8; ++n2)
        for (int u = 0; u < IPL; ++u) {
          const int m = lane + 32 * u + W::S0 * n2;
          const float got = mir[(lane + 31) & 31][u][n2].x;  // __shfl_sync(.., (lane + 31) & 31)
          const float xm = lane > 0 ? got : prev;
          prev = got;
          v[lane][u][n2] = W::p1_pre(m, own[lane][u][n2], xm, mir[lane][u][n2].y, SJP[m]);
        }
    }
    for (int lane = 0; lane < 32; ++lane)
      for (int u = 0; u < IPL; ++u) W::p1_fft(lane + 32 * u, v[lane][u], TWD, Z);
    for (int lane = 0; lane < 32; ++lane) {
      C2<float> w2[8];
      W::p2_twiddles(lane % W::S1, TWD, w2);
      for (int u = 0; u < IPL; ++u) W::p2(lane + 32 * u, w2, Z);
    }
    for (int lane = 0; lane < 32; ++lane)
      for (int u = 0; u < 2; ++u) W::p3(lane + 32 * u, Z);
    C2<float>* N = (C2<float>*)B;
    for (int lane = 0; lane < 32; ++lane) {
      C2<float> Zl[KPL], Zh[KPL];
      W::split_read(lane, Z, Zl, Zh);
      for (int t = 0; t < KPL; ++t) {
        N[pc<float>(KPL * lane + t)] = Zl[t];
        N[pc<float>((lane == 0 && t == 0) ? H / 2 : H - KPL * lane - t)] = Zh[t];
      }
    }
    for (int k = 0; k <= H / 2; ++k) dst_split_item<float>((const C2<float>*)B, Cr, k, g, SPL);
    std::vector<float> tot(g.nchunk);
    for (int c = 0; c < g.nchunk; ++c) tot[c] = dst_scan_chunk<float>(Cr, c, g);
    float pref = 0.f;
    for (int c = 0; c < g.nchunk; ++c) {
      if (c > 0) dst_scan_fix<float>(Cr, c, pref, g);
      pref += tot[c];
    }
    for (int j = 0; j < M - 1; ++j) x[j] = Cr[pr<float>(j + 1)];
  }
}

// the one-warp transform for M = 512 and 1024; returns 0 for other lengths
// The fixed-point transform (dst_fx.h): raw doubles in, doubles out.
static void run_fx(int M, int howmany, double* data) {
  DstGeom g = make_geom(M);
  FxTablesHost fx = build_fx_tables(g);
  const int L = padded_len<double>(M), H = g.H;
  std::vector<fx_t> A(L), B(L);
  for (int r = 0; r < howmany; ++r) {
    double* x = data + (size_t)r * (M - 1);
    for (int j = 0; j < L; ++j) A[j] = B[j] = 777;  // pad slots must never be read
    unsigned int mx = 0;
    for (int j = 1; j < M; ++j) {
      std::memcpy(&A[pr<double>(j)], &x[j - 1], 8);
      const unsigned int h = (unsigned int)((unsigned long long)A[pr<double>(j)] >> 32) & 0x7fffffffu;
      mx = h > mx ? h : mx;
    }
    const int E = fx_scale(mx);
    unsigned int l1 = 0;
    for (int j = 1; j <= H; ++j)
      l1 += fx_pre_item((const unsigned long long*)A.data(), B.data(), j, M, E, fx.nsj.data());
    C2<fx_t>* src = (C2<fx_t>*)B.data();
    C2<fx_t>* dst = (C2<fx_t>*)A.data();
    int Ns = 1, drop = 0;
    unsigned int mag = 0;
    for (int p = 0; p < g.npass; ++p) {
      const int R = g.radix[p], s = p ? fx_pass_shift(mag) : 0;
      if (p) drop += 2 - s;
      mag = 0;
      for (int b = 0; b < H / R; ++b)
        mag |= fx_stockham_dispatch(R, src, dst, b, b % Ns, Ns, H, s, fx.twq.data() + (p ? Ns - g.radix[0] : 0));
      Ns *= R;
      C2<fx_t>* t = src; src = dst; dst = t;
    }
    const int s = fx_split_shift(mag, l1, drop), e = fx_row_exp(mx, drop, s);
    for (int k = 0; k <= H / 2; ++k) fx_split_item(src, dst, k, H, s, fx.spq.data());
    fx_t* o = (fx_t*)dst;
    for (int k = 1; k < H; ++k) o[pr<double>(2 * k + 1)] += o[pr<double>(2 * k - 1)];
    for (int j = 1; j < M; ++j) {
      const fx_t v = o[pr<double>(j)];
      if (e == FX_NAN) x[j - 1] = std::nan("");
      else if (fx_exp_ok(e)) { const unsigned long long b = fx_to_bits(v, e); std::memcpy(&x[j - 1], &b, 8); }
      else x[j - 1] = std::ldexp((double)v, e);
    }
  }
}
// The fixed-point chirp-z form.
static void run_fx_blue(int M, int howmany, double* data) {
  DstGeom g = make_geom_blue(M);
  FxTablesHost fx = build_fx_tables(g);
  const int Lc = g.H, ld = padded_len<double>(2 * Lc);
  std::vector<fx_t> A(ld), B(ld);
  auto passes = [&](C2<fx_t>*& src, C2<fx_t>*& dst, int& drop, unsigned int& mag) {
    int Ns = 1;
    for (int p = 0; p < g.npass; ++p) {
      const int R = g.radix[p], s = p ? fx_pass_shift(mag) : 0;
      if (p) drop += 2 - s;
      mag = 0;
      for (int b = 0; b < Lc / R; ++b)
        mag |= fx_stockham_dispatch(R, src, dst, b, b % Ns, Ns, Lc, s, fx.twq.data() + (p ? Ns - g.radix[0] : 0));
      Ns *= R;
      C2<fx_t>* t = src; src = dst; dst = t;
    }
  };
  for (int r = 0; r < howmany; ++r) {
    double* x = data + (size_t)r * (M - 1);
    for (int j = 0; j < ld; ++j) A[j] = B[j] = 777;
    unsigned int mx = 0;
    for (int j = 1; j < M; ++j) {
      std::memcpy(&A[pr<double>(j)], &x[j - 1], 8);
      const unsigned int h = (unsigned int)((unsigned long long)A[pr<double>(j)] >> 32) & 0x7fffffffu;
      mx = h > mx ? h : mx;
    }
    C2<fx_t>* src = (C2<fx_t>*)B.data();
    C2<fx_t>* dst = (C2<fx_t>*)A.data();
    for (int m = 0; m < Lc; ++m)
      fx_chirp_item((const unsigned long long*)A.data(), src, m, M, fx_scale(mx), fx.bc.data());
    int drop = 0;
    unsigned int mag = 0;
    passes(src, dst, drop, mag);
    int s = fx_pass_shift(mag);
    drop += 2 - s + fx.be;
    for (int k = 0; k < Lc; ++k) fx_chirp_mul_item(src, k, s, fx.bz.data());
    passes(src, dst, drop, mag);
    s = fx_pass_shift(mag);
    for (int k = 0; k < M; ++k) fx_chirp_out_item(src, (fx_t*)dst, k, s, fx.bc.data());
    int lg = 0;
    while ((1 << lg) < Lc) ++lg;
    const int e = fx_exp_add(fx_row_exp(mx, drop + 2 + 1 - lg, s), -1);
    for (int j = 1; j < M; ++j)
      x[j - 1] = e == FX_NAN ? std::nan("") : std::ldexp((double)((const fx_t*)dst)[pr<double>(j)], e);
  }
}
// DST-I by its definition in long double (at least 64 bits), one row
static void run_exact(int M, const double* x, long double* y) {
  std::vector<long double> s(2 * (size_t)M);
  const long double pi = 3.14159265358979323846264338327950288L;
  for (int m = 0; m < 2 * M; ++m) {
    int r = m % M;
    if (2 * r > M) r = M - r;
    s[m] = (m < M ? 1 : -1) * sinl(pi * r / M);
  }
  for (int k = 1; k < M; ++k) {
    long double t = 0;
    for (int j = 1; j < M; ++j) t += x[j - 1] * s[(long)j * k % (2 * M)];
    y[k - 1] = 2 * t;
  }
}

extern "C" int dst_warp_run_f32(int M, int howmany, float* data) {
  if (M == 512) run_warp<8>(howmany, data);
  else if (M == 1024) run_warp<9>(howmany, data);
  else return 0;
  return 1;
}

// The chirp-z form (dst_blue.h) of any length M >= 4, its phases as loops:
// chirp, L-point FFT (the Stockham items), multiply, FFT, output.
template <typename T>
static void run_blue(int M, int howmany, T* data) {
  const DstGeom g = make_geom_blue(M);
  const int L = g.H;
  DstTablesHost th = build_dst_tables(2 * L);  // twiddles of the L-point FFT
  std::vector<double> bcd, bzd;
  build_blue_tables(g, bcd, bzd);
  std::vector<T> tw(th.tw.begin(), th.tw.end()), bc(bcd.begin(), bcd.end()), bz(bzd.begin(), bzd.end());
  const C2<T>* TW = (const C2<T>*)tw.data();
  const C2<T>* BC = (const C2<T>*)bc.data();
  const C2<T>* BZ = (const C2<T>*)bz.data();
  const int ld = padded_len<T>(2 * L);
  std::vector<T> A(ld), B(ld);
  auto fft = [&](T* src, T* dst) -> T* {
    int Ns = 1;
    for (int p = 0; p < g.npass; ++p) {
      const int R = g.radix[p];
      for (int b = 0; b < L / R; ++b) stockham_dispatch<T>(R, (const C2<T>*)src, (C2<T>*)dst, b, Ns, L, TW);
      Ns *= R;
      T* t = src; src = dst; dst = t;
    }
    return src;
  };
  for (int r = 0; r < howmany; ++r) {
    T* x = data + (size_t)r * (M - 1);
    for (int j = 0; j < ld; ++j) A[j] = B[j] = T(777);
    for (int j = 0; j < M - 1; ++j) A[pr<T>(j + 1)] = x[j];
    A[pr<T>(0)] = T(12345);  // index 0 must never be read
    for (int m = 0; m < L; ++m) blue_chirp_item<T>(A.data(), (C2<T>*)B.data(), m, M, BC);
    T* O = fft(B.data(), A.data());
    for (int k = 0; k < L; ++k) blue_mul_item<T>((C2<T>*)O, k, BZ);
    T* D = fft(O, O == A.data() ? B.data() : A.data());
    T* out = D == A.data() ? B.data() : A.data();
    for (int k = 0; k < M; ++k) blue_out_item<T>((const C2<T>*)D, out, k, T(1) / T(L), BC);
    for (int j = 0; j < M - 1; ++j) x[j] = out[pr<T>(j + 1)];
  }
}
extern "C" void dst_blue_run_f64(int M, int howmany, double* data) { run_blue<double>(M, howmany, data); }
extern "C" void dst_blue_run_f32(int M, int howmany, float* data) { run_blue<float>(M, howmany, data); }

extern "C" void dst_core_run_f64(int M, int howmany, double* data) { run<double>(M, howmany, data); }
extern "C" void dst_core_run_f32(int M, int howmany, float* data) { run<float>(M, howmany, data); }

// pass-ordered twiddles (fill_pass_twiddles) against their definition:
// returns the number of mismatching entries, or -1 if the count is wrong
extern "C" int dst_core_check_twp(int M) {
  DstGeom g = make_geom(M);
  DstTablesHost th = build_dst_tables(M);
  const int H = g.H;
  int bad = 0, count = 0, Ns = g.radix[0];
  for (int p = 1; p < g.npass; ++p) {
    const int R = g.radix[p];
    for (int q = 1; q < R; ++q)
      for (int k = 0; k < Ns; ++k) {
        const int e = (Ns - g.radix[0]) + (q - 1) * Ns + k;
        const double ang = 2.0 * M_PI * ((double)q * k * (H / (Ns * R))) / H;
        if (std::fabs(th.twp[2 * e] - std::cos(ang)) > 1e-15 || std::fabs(th.twp[2 * e + 1] + std::sin(ang)) > 1e-15)
          ++bad;
        ++count;
      }
    Ns *= R;
  }
  if (count != (g.npass > 1 ? H - g.radix[0] : 0)) return -1;
  return bad;
}

// the transform lengths the library accepts (M even, M/2 a product of 2, 3, 5, 7)
extern "C" int dst_core_length_ok(int M) { return transform_length_ok(M) ? 1 : 0; }

// relative errors (2-norm, in units of 2^-53) of the FP64 and the fixed-point
// transform of one row
extern "C" void dst_fx_errors(int M, const double* x, double* err) {
  std::vector<long double> e(M - 1);
  run_exact(M, x, e.data());
  const bool blue = !transform_length_ok(M);
  for (int f = 0; f < 2; ++f) {
    std::vector<double> y(x, x + M - 1);
    if (f) blue ? run_fx_blue(M, 1, y.data()) : run_fx(M, 1, y.data());
    else blue ? run_blue<double>(M, 1, y.data()) : run<double>(M, 1, y.data());
    long double d = 0, n = 0;
    for (int k = 0; k < M - 1; ++k) {
      d += (y[k] - e[k]) * (y[k] - e[k]);
      n += e[k] * e[k];
    }
    err[f] = (double)(sqrtl(d / n) * 9007199254740992.0L);
  }
}
extern "C" void dst_fx_run(int M, int howmany, double* data) {
  transform_length_ok(M) ? run_fx(M, howmany, data) : run_fx_blue(M, howmany, data);
}

static unsigned long long bits_of(double v) {
  unsigned long long b;
  std::memcpy(&b, &v, 8);
  return b;
}
static double double_of(unsigned long long b) {
  double v;
  std::memcpy(&v, &b, 8);
  return v;
}
static double fx_double(fx_t v, int e) {
  return e == FX_NAN ? std::nan("") : fx_exp_ok(e) ? double_of(fx_to_bits(v, e)) : std::ldexp((double)v, e);
}
extern "C" int modes_fixed(int nl, const double* mat) { return modes_fixed_ok(nl, mat) ? 1 : 0; }
// The projection of a field x (nl layers of ny x nx) by mat: the errors of the
// FP64 sums and of the fixed-point ones (modes_core.h) against sums in long
// double, and those sums.
extern "C" void modes_errors(int nl, int ny, int nx, const double* mat, const double* x, double* err64, double* errfx,
                             double* exact) {
  std::vector<Q2> c((size_t)nl * nl);
  std::vector<int> e(2 * (size_t)nl);
  const int* k = e.data() + nl;
  fill_mode_table(nl, mat, c.data(), e.data());
  const size_t n = (size_t)ny * nx;
  std::vector<fx_t> v(nl);
  for (size_t p = 0; p < n; ++p) {
    const unsigned int turn = modes_turn((int)(p % nx), (int)(p / nx));
    ModeMax h = {};
    for (int l = 0; l < nl; ++l) modes_max(h, (unsigned int)(bits_of(x[l * n + p]) >> 32) & 0x7fffffffu, k[l]);
    for (int l = 0; l < nl; ++l) v[l] = modes_in(bits_of(x[l * n + p]), h, k[l], turn);
    for (int m = 0; m < nl; ++m) {
      long double t = 0;
      double f = 0;
      ModeAcc s = {};
      for (int l = 0; l < nl; ++l) {
        t += (long double)mat[m * nl + l] * x[l * n + p];
        f = std::fma(mat[m * nl + l], x[l * n + p], f);
        if (l & 1) modes_term<true>(s, modes_value<true>(v[l]), c[m * nl + l]);
        else modes_term<false>(s, modes_value<false>(v[l]), c[m * nl + l]);
        if ((l & 3) == 3 || l == nl - 1) modes_carry(s);
      }
      const double r = double_of(modes_turned(bits_of(fx_double(s.acc, modes_exp(h, e[m]))), turn));
      err64[m * n + p] = (double)(f - t);
      errfx[m * n + p] = (double)(r - t);
      exact[m * n + p] = (double)t;
    }
  }
}

// The Arakawa Jacobian (times 12 Delta^2) of a field of ny x nx points with a
// ring around it, in tiles of 32 x 16: the errors of the floating-point form
// and of the fixed-point one (rhs_core.h) against long double, and the latter.
extern "C" void jacobian_errors(int ny, int nx, const double* psi, const double* q, double* err64, double* errfx,
                                double* exact) {
  const int W = nx + 2;
  std::vector<fx_t> P((size_t)W * (ny + 2));
  std::vector<Q2> Q(P.size());
  auto hi = [](double v) { return (unsigned int)(bits_of(v) >> 32) & 0x7fffffffu; };
  for (int j0 = 0; j0 < ny; j0 += 16)
    for (int i0 = 0; i0 < nx; i0 += 32) {
      const int jn = std::min(ny, j0 + 16), in = std::min(nx, i0 + 32);
      unsigned int hp = 0, hq = 0;
      for (int y = j0; y < jn + 2; ++y)
        for (int x = i0; x < in + 2; ++x) {
          hp = std::max(hp, hi(psi[y * W + x]));
          hq = std::max(hq, hi(q[y * W + x]));
        }
      const int Ep = fx_scale(hp) + 2, Eq = fx_scale(hq);
      for (int y = j0; y < jn + 2; ++y)
        for (int x = i0; x < in + 2; ++x) {
          P[y * W + x] = fx_from_bits(bits_of(psi[y * W + x]), Ep);
          Q[y * W + x] = q2_split(fx_from_bits(bits_of(q[y * W + x]), Eq));
        }
      for (int j = j0; j < jn; ++j)
        for (int i = i0; i < in; ++i) {
          const int o = (j + 1) * W + i + 1;
          const double *p = psi + o, *z = q + o;
          int n;
          const fx_t v = fx_sum_value(fx_jacobian(fx_nine(P.data() + o, W), Q.data() + o, W), n);
          const double r = fx_double(v, Ep + Eq - 2 * FX_EOFF + 64 - n);
          double J = (p[1] - p[-1]) * (z[W] - z[-W]);
          J = std::fma(-(p[W] - p[-W]), z[1] - z[-1], J);
          J = std::fma(p[1], z[W + 1] - z[-W + 1], J);
          J = std::fma(-p[-1], z[W - 1] - z[-W - 1], J);
          J = std::fma(-p[W], z[W + 1] - z[W - 1], J);
          J = std::fma(p[-W], z[-W + 1] - z[-W - 1], J);
          J = std::fma(z[W], p[W + 1] - p[W - 1], J);
          J = std::fma(-z[-W], p[-W + 1] - p[-W - 1], J);
          J = std::fma(-z[1], p[W + 1] - p[-W + 1], J);
          J = std::fma(z[-1], p[W - 1] - p[-W - 1], J);
          auto d = [](const double* f, int a, int b) { return (long double)f[a] - f[b]; };
          // the coefficients of q sum to zero: of its differences
          const long double t = d(z, W, 0) * (d(p, 1, -1) + d(p, W + 1, W - 1)) - d(z, -W, 0) * (d(p, 1, -1) + d(p, -W + 1, -W - 1)) -
                                d(z, 1, 0) * (d(p, W, -W) + d(p, W + 1, -W + 1)) + d(z, -1, 0) * (d(p, W, -W) + d(p, W - 1, -W - 1)) +
                                d(z, W + 1, 0) * d(p, 1, W) + d(z, -W + 1, 0) * d(p, -W, 1) + d(z, W - 1, 0) * d(p, W, -1) +
                                d(z, -W - 1, 0) * d(p, -1, -W);
          err64[j * nx + i] = (double)(J - t);
          errfx[j * nx + i] = (double)(r - t);
          exact[j * nx + i] = (double)t;
        }
    }
}
