// rhs_fx.cuh -- the RHS tile of the FP64 path in 64-bit fixed point (included
// by step_device.cuh; dst_fx.h holds the arithmetic).
//
// The tile's psi and q become integers of one power of two each, taken from
// the tile's own largest magnitudes.  The hyperviscosity sweeps, Laplacians
// and differences are then exact integer additions, and the Arakawa Jacobian
// a sum of whole products (rhs_core.h).  A point's few results become doubles
// at the end, for the coefficients (3-4 FP64 operations a point instead of
// 34).  1024^2 x 10 with three sweeps: 0.767 -> 0.312 ms (FP64 pipe 86% busy
// before; now integer instructions; with products cut to their high words
// 0.303).
//
// What stays in FP64 (rhs_tile_compute): edge tiles at walls with bc_fac !=
// 0, whose ghost values (2 bc_fac / Delta^2 psi at every sweep) exceed the
// interior ones by orders of magnitude, and the bottom layer over topography.
//
// Every tile is TX x 16 points here; a taller tile runs as bands of 16 rows,
// so that the scale of a point's tile does not depend on the tile shape.
#pragma once

#include "rhs_core.h"

namespace qgw {

constexpr int TYF = 16;

template <typename T> __device__ __forceinline__ bool rhs_fx_ok(const StepArgs<T>& a, bool edge, int k) {
  return sizeof(T) == 8 && !(edge && a.cbc > 0) && !(a.has_topo && k == a.nl - 1);
}

// in: the raw tile (zero or wrapped outside the domain), the block
// synchronised since it arrived; wk: the work buffers.  Returns the thread's
// CFL maximum |dpsi| as bits.
template <int R, bool EDGE>
__device__ __forceinline__ unsigned long long rhs_tile_fx(const StepArgs<double>& a, int i0, int j0, int k,
                                                          int step_index, const RhsIn<double>& in, double* wk) {
  using S = RhsShape<double, R, TYF>;
  constexpr int W = TW, HH = TYF + 2 * R, PW = TX + 2 * R, QW = TX + 2, QH = TYF + 2, XO = TOX, TS = S::TS;
  static_assert(S::TS + S::QS <= S::DIFFS, "the integer tiles lie where the FP64 form keeps its differences");
  fx_t* L0 = (fx_t*)wk;
  fx_t* L1 = L0 + TS;
  fx_t* P = L1 + TS;  // HH x W, psi with halo R
  Q2* Q = (Q2*)(P + TS);  // QH x W, q with halo 1
  __shared__ unsigned int rmax[2][NT / 32], rmag[NT / 32];
  const int tx = threadIdx.x, ty = threadIdx.y, tid = tx + ty * 32;
  const int nx = a.nx, ny = a.ny, pitch = a.pitch;
  const bool walls = EDGE && !a.periodic;

  // largest magnitudes, then integers: |P| < 2^57, |Q| < 2^59
  constexpr int NP = (PW * HH + NT - 1) / NT, NQ = (QW * QH + NT - 1) / NT;
  unsigned int hp = 0, hq = 0;
#pragma unroll
  for (int u = 0; u < NP; ++u) {
    const int w = tid + u * NT, y = w / PW, o = y * W + w - y * PW - R + XO;
    if (w < PW * HH) hp = max(hp, fx_hi(in.ps[o]));
  }
#pragma unroll
  for (int u = 0; u < NQ; ++u) {
    const int w = tid + u * NT, y = w / QW, o = y * W + w - y * QW - 1 + XO;
    if (w < QW * QH) hq = max(hq, fx_hi(in.qs[o]));
  }
  hp = __reduce_max_sync(0xffffffffu, hp);
  hq = __reduce_max_sync(0xffffffffu, hq);
  if (tx == 0) {
    rmax[0][ty] = hp;
    rmax[1][ty] = hq;
  }
  __syncthreads();
#pragma unroll
  for (int w = 0; w < NT / 32; ++w) {
    hp = max(hp, rmax[0][w]);
    hq = max(hq, rmax[1][w]);
  }
  const int Ep = fx_scale(hp) + 2, Eq = fx_scale(hq);
#pragma unroll
  for (int u = 0; u < NP; ++u) {
    const int w = tid + u * NT, y = w / PW, o = y * W + w - y * PW - R + XO;
    if (w < PW * HH) P[o] = fx_from_bits(__double_as_longlong(in.ps[o]), Ep);
  }
#pragma unroll
  for (int u = 0; u < NQ; ++u) {
    const int w = tid + u * NT, y = w / QW, o = y * W + w - y * QW - 1 + XO;
    if (w < QW * QH) Q[o] = q2_split(fx_from_bits(__double_as_longlong(in.qs[o]), Eq));
  }
  const int ep = Ep - FX_EOFF, eq = Eq - FX_EOFF;  // exponents of P and Q
  __syncthreads();

  // the Laplacian sweeps (calc_diff, src/dynamics.h:13-44) with a shrinking
  // halo, unscaled; at walls (bc_fac = 0 here) values outside the domain are
  // zero
  unsigned int lmag = 0;
  const int ksweep = a.nsweep;  // 0 or R
  const fx_t* Lp = P;
  fx_t* Lc = L0;
  int lsh = 0;  // the sweeps' right shift
#pragma unroll
  for (int s = 1; s <= R; ++s) {
    if (s > ksweep) break;
    const int Ws = TX + 2 * R - 2 * s, Hs = HH - 2 * s;
    const int cx = s - R + XO;
    auto lap = [&](int o, const fx_t c) {
      return ((Lp[o + 1] + Lp[o - 1]) + (Lp[o + W] + Lp[o - W])) - 4 * c;
    };
    auto point = [&](int yr, int xr) {
      const int o = (yr + s) * W + xr + cx;
      const fx_t c = Lp[o];
      fx_t v = lap(o, c);
      if (walls) {
        const int gi = i0 + xr + s - R, gj = j0 + yr + s - R;
        if (gi < 0 || gi >= nx || gj < 0 || gj >= ny) v = 0;
      }
      if (s == 1 && R > 1) lmag |= fx_mag(v);
      Lc[o] = v;
    };
    // the region's first 32 columns one row per warp, the rest after them
    for (int yr = ty; yr < Hs; yr += NT / 32) point(yr, tx);
    if (Ws > 32) {
      for (int w = tid; w < (Ws - 32) * Hs; w += NT) {
        const int yr = w / (Ws - 32);
        point(yr, 32 + w - yr * (Ws - 32));
      }
    }
    if (s < R) {
      if (s == 1) {
        lmag = __reduce_or_sync(0xffffffffu, lmag);
        if (tx == 0) rmag[ty] = lmag;
      }
      __syncthreads();
      if (s == 1) {
#pragma unroll
        for (int w = 0; w < NT / 32; ++w) lmag |= rmag[w];
        // each further sweep grows a value at most eightfold: room for them
        // (a rough psi only; a smooth one's Laplacian is far below it)
        lsh = 32 - fx_clz(lmag) + 32 + 3 * (R - 1) - 62;
        if (lsh > 0) {
          for (int w = tid; w < Ws * Hs; w += NT) {
            const int yr = w / Ws, o = (yr + s) * W + w - yr * Ws + cx;
            Lc[o] = fx_shr(Lc[o], lsh);
          }
          __syncthreads();
        } else {
          lsh = 0;
        }
      }
    }
    Lp = Lc;
    Lc = Lc == L0 ? L1 : L0;
  }
  // (a thread reads back the last sweep's values it wrote: that region is one
  // row of 32 points per warp, as below)
  // non-finite tiles and tiles of zeros, as the transforms mark them
  const bool bad = max(hp, hq) >= 0x7ff00000u;
  const int ed = bad ? FX_NAN : ep, el = bad ? FX_NAN : ep + lsh;
  const int ej = bad ? FX_NAN : (hp == 0 || hq == 0) ? FX_ZERO : ep + eq + 64;

  const size_t fs = (size_t)a.nl * a.lstride;
  int s0, s1, s2;
  slabs(step_index + 1, s0, s1, s2);
  double* fout = a.fab + s0 * fs + (size_t)k * a.lstride;
  const bool bottom = k == a.nl - 1;
  fx_t cfl = 0;
#pragma unroll
  for (int y = ty; y < TYF; y += NT / 32) {
    const int gi = i0 + tx, gj = j0 + y;
    if (EDGE && (gi >= nx || gj >= ny)) continue;
    const fx_t* p = P + (y + R) * W + tx + XO;
    const Q2* q = Q + (y + 1) * W + tx + XO;
    const FxNine ps = fx_nine(p, W);
    int jn;
    const fx_t J = fx_sum_value(fx_jacobian(ps, q, W), jn);
    const fx_t dx = ps.e - ps.w;
    // rhs, src/dynamics.h:55-58
    double f = fmaT(-a.inv12d2, fx_out(J, fx_exp_add(ej, -jn)), -(a.b2d * fx_out(dx, ed)));
    if (a.has_nu) {
      const fx_t lq = ((q2_join(q[1]) + q2_join(q[-1])) + (q2_join(q[W]) + q2_join(q[-W]))) - 4 * q2_join(q[0]);
      f = fmaT(a.nu_d2, fx_out(lq, bad ? FX_NAN : eq), f);
    }
    if (ksweep > 0) f = fmaT(a.nuh_scaled, fx_out(Lp[(y + R) * W + tx + XO], el), f);
    // surface wind (src/dynamics.h:66) and bottom drag (:67-69)
    if (k == 0 && a.has_wind) f += a.wind[gj];
    if (bottom && a.has_drag) f = fmaT(a.drag_d2, fx_out(((ps.e + ps.w) + (ps.n + ps.s)) - 4 * ps.c, ed), f);
    fout[(size_t)gj * pitch + gi] = f;
    // CFL (src/timestep.h:74-87): one-sided differences
    const fx_t du = ps.e - ps.c, dv = ps.n - ps.c;
    cfl = max(cfl, max(du < 0 ? -du : du, dv < 0 ? -dv : dv));
  }
  return absbits(fx_out(cfl, ed));
}

}  // namespace qgw
