// modes_core.h -- the arithmetic of the FP64 path's vertical projections
// (modes_fx.cuh), for the kernels and for checks on the host.
//
// The columns of the matrix are brought to like size by powers of two, which
// go to the values (thin layers' coefficients are small and their vorticity
// large).  A point's values then become integers below 2^61 by the largest of
// them, the coefficients integers below 2^60 by the largest of their row;
// products keep their high words and sums are exact, so the result does not
// depend on how outputs are grouped.  The error is about 2^-56 of the largest
// coefficient of the row times the largest value of the point, both as scaled.
// No term of an output need reach that: what columns of too unlike size lose
// by it is the reason for modes_fixed_ok's limits (dst_tables.h).
//
// Of a product's two cross terms one is truncated down and the other, of the
// negated value, up, the two taking turns from layer to layer.  Where one of
// them is exact -- a value of zero, or one of single precision, whose low word
// is zero -- the other's truncation is left, and at every point alike: its
// mean, which the inversion amplifies, would reach 1e-11 of psi with q in one
// of twenty layers.  So neighbouring points compute with opposite signs, and
// what is left alternates from point to point, at the wave number that the
// inversion damps most.
#pragma once

#include "dst_fx.h"

namespace qgw {

// the sign bit that point (i, j)'s values and results are turned by
QGW_HD unsigned int modes_turn(int i, int j) { return (unsigned int)(i + j) << 31; }
QGW_HD unsigned long long modes_turned(unsigned long long b, unsigned int turn) { return b ^ ((unsigned long long)turn << 32); }

// A point's largest high words, of the values as they are (which shows a
// non-finite one) and as scaled by 2^k (below zero: as good as none).
struct ModeMax {
  unsigned int raw;
  int hi;
};
QGW_HD void modes_max(ModeMax& h, unsigned int hi, int k) {
  const int s = (int)hi + k * (1 << 20);
  h.raw = hi > h.raw ? hi : h.raw;
  h.hi = s > h.hi ? s : h.hi;
}
// the value of bits b of a column scaled by 2^k
QGW_HD fx_t modes_in(unsigned long long b, const ModeMax& h, int k, unsigned int turn) {
  return fx_from_bits<8>(modes_turned(b, turn), fx_scale((unsigned int)h.hi) - k);
}
// exponent of the point's results
QGW_HD int modes_exp(const ModeMax& h, int ce) {
  return h.raw >= 0x7ff00000u ? FX_NAN : h.hi == 0 ? FX_ZERO : fx_scale((unsigned int)h.hi) - 1083 + ce + 4;
}
// A value as its halves and the negated one of the half whose cross term is
// truncated up: the low one (never -2^31) in even layers, the high one in odd
// ones.
struct ModeValue {
  Q2 v;
  int n;
};
template <bool ODD> QGW_HD ModeValue modes_value(fx_t x) {
  ModeValue m;
  m.v = q2_const(x);
  m.n = ODD ? -m.v.h : -m.v.l;
  return m;
}
// the terms of one output: acc (64 bits) and the cross terms' down and up
// truncated parts in units of 2^32, which hold four layers' (modes_carry)
struct ModeAcc {
  fx_t acc;
  int down, up;
};
template <bool ODD> QGW_HD void modes_term(ModeAcc& s, const ModeValue& x, Q2 c) {
  s.acc += (fx_t)x.v.h * c.h;
  s.down += ODD ? fx_mh(x.v.l, c.h) : fx_mh(x.v.h, c.l);
  s.up += ODD ? fx_mh(x.n, c.l) : fx_mh(x.n, c.h);
}
QGW_HD void modes_carry(ModeAcc& s) {
  s.acc += s.down - s.up;
  s.down = s.up = 0;
}

}  // namespace qgw
