// rhs_core.h -- the arithmetic of the FP64 path's Arakawa Jacobian in fixed
// point (rhs_fx.cuh), for the kernel and for checks on the host.
//
// The Jacobian (src/domain.h:17-27) as a sum over the eight neighbours of q,
//   sum_n q_n C_n,  C_N = (psi_E - psi_W) + (psi_NE - psi_NW),
//   C_NE = psi_E - psi_N, ...
// whose C_n, differences of psi, sum to zero, so that of a smooth q most
// cancels.  The products are therefore kept whole (the four 32 x 32 -> 64
// products of their halves, of the lowest one its upper bits) and the sum
// rounds once, as it becomes a double; it is zero where every product is.
// Products cut to their high words, however the C_n are scaled, left 2^-54 of
// the largest |q C| a piece: of a smooth flow four to six times the FP64
// form's error, and the constant that stood for their truncation wherever q
// was zero.
#pragma once

#include "dst_fx.h"

namespace qgw {

// 2^32 hi + mid + 2^FX_SUM_LO lo, in units of 2^32
constexpr int FX_SUM_LO = 5;
struct FxSum {
  fx_t hi, mid;
  int lo;
};
// |a| <= 2^60, |b| < 2^59, eight terms: |mid| < 8 (2^59 + 2^58), |lo| <= 8 2^25
QGW_HD void fx_sum_add(FxSum& s, fx_t a, Q2 v) {
  const Q2 u = q2_split(a);
  s.hi += (fx_t)u.h * v.h;
  s.mid += (fx_t)u.h * v.l;
  s.mid += (fx_t)u.l * v.h;
  s.lo += fx_mh(u.l, v.l >> FX_SUM_LO);
}
// The sum as v 2^(64 - n): its leading bits, the rest jammed into the last
// one (neither up nor down).
QGW_HD fx_t fx_sum_value(const FxSum& s, int& n) {
  const fx_t mid = s.mid + (fx_t)s.lo * (1 << FX_SUM_LO), v = s.hi + (mid >> 32);
  const unsigned int f = (unsigned int)mid;
  n = fx_clz(fx_mag(v)) - 1;
  return fx_shl(v, n) | (fx_t)((unsigned long long)f >> (32 - n)) | (fx_t)((f << n) != 0);
}

// psi around a point
struct FxNine {
  fx_t c, e, w, n, s, ne, nw, se, sw;
};
QGW_HD FxNine fx_nine(const fx_t* p, int W) {
  return FxNine{p[0], p[1], p[-1], p[W], p[-W], p[W + 1], p[W - 1], p[-W + 1], p[-W - 1]};
}
// sum_n q_n C_n; q: the point in rows of W.  |psi| < 2^57, |q| < 2^59.
QGW_HD FxSum fx_jacobian(const FxNine& p, const Q2* q, int W) {
  FxSum J = {};
  const fx_t dx = p.e - p.w, dy = p.n - p.s;
  fx_sum_add(J, dx + (p.ne - p.nw), q[W]);
  fx_sum_add(J, (p.sw - p.se) - dx, q[-W]);
  fx_sum_add(J, (p.se - p.ne) - dy, q[1]);
  fx_sum_add(J, dy + (p.nw - p.sw), q[-1]);
  fx_sum_add(J, p.e - p.n, q[W + 1]);
  fx_sum_add(J, p.s - p.e, q[-W + 1]);
  fx_sum_add(J, p.n - p.w, q[W - 1]);
  fx_sum_add(J, p.w - p.s, q[-W - 1]);
  return J;
}

}  // namespace qgw
