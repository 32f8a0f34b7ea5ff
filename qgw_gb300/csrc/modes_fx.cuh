// modes_fx.cuh -- the FP64 path's vertical projections and row transforms
// (included by step_device.cuh).
//
// layers -> modes (src/elliptic.h:88-98) and modes -> layers (:140-147) act
// point by point and are linear, so each runs as a kernel of its own beside
// the row transforms: a thread holds one point's nl values, so every value is
// loaded and turned into fixed point once for all nl outputs, and the row
// kernel takes rows of any layer, several at a time.  (Inside the row kernels
// the projection cost nl FP64 multiply-adds a point, two thirds of their
// FP64-pipe-bound time, and shared memory held the rows of two modes only, so
// each pair of modes read the row's layers again.)  The extra pass over the
// spectral field mostly stays in L2.
//
// The arithmetic is modes_core.h's.  Runs of strongly graded profiles, whose
// matrix columns differ by more than it takes, or of more than 20 layers
// (modes_fixed_ok, dst_tables.h) keep FP64 sums (a.modes_fx = 0).
#pragma once

#include <type_traits>

#include "modes_core.h"

namespace qgw {

constexpr int MODES_NL = 16;  // layers a thread holds in registers, at most (more: read again per 8 outputs)

// what the forward projection does to q on the way
struct QUpdate {
  bool upd;                      // apply the pending AB3 update
  double c0, c1, c2;
  const double *f0, *f1, *f2;
  const double* field;           // stochastic forcing of layer 0 (null: none), * sqdt
  double sqdt;
  const double *r1, *r2;         // 4-D forcing records (null: none)
  double w1, w2, dt;
};
// (by one thread of a block: the square root and the record weights are a few
// dozen FP64 operations)
__device__ __forceinline__ QUpdate q_update(const StepArgs<double>& a, int step_mode) {
  const DevState* st = a.state;
  QUpdate u;
  u.upd = step_mode && st->pending;
  int s0, s1, s2;
  slabs(st->step_index, s0, s1, s2);
  u.c0 = st->c0;
  u.c1 = st->c1;
  u.c2 = st->c2;
  const size_t fs = (size_t)a.nl * a.lstride;
  u.f0 = a.fab + s0 * fs;
  u.f1 = a.fab + s1 * fs;
  u.f2 = a.fab + s2 * fs;
  u.field = u.upd && a.fr.on ? a.fr.field : nullptr;
  u.sqdt = u.field ? sqrt(st->dt) : 0.0;
  u.r1 = u.r2 = nullptr;
  u.w1 = u.w2 = u.dt = 0.0;
  if (u.upd && a.nrec > 0) {
    const Forc4D fw = forc4d_at(st->t_prev, a.dt_forc, a.nrec);
    u.r1 = a.frec + fw.i1 * fs;
    u.r2 = a.frec + fw.i2 * fs;
    u.w1 = fw.w1;
    u.w2 = fw.w2;
    u.dt = st->dt;
  }
  return u;
}
// q of layer l at point (i, j), o its offset in the run's layer: the run's
// field as it is (FK 0), with the pending update applied (1; 2: and forcing,
// src/timestep.h:138-163), or the caller's array (3); stored back in the last
// three cases.  FK is a compile-time choice outside the loop over layers:
// inside it the forcing's arithmetic ran predicated off in every iteration,
// five FP64 operations of eight.
template <int FK>
__device__ __forceinline__ double q_value(const StepArgs<double>& a, const QUpdate& u, int l, int j, int i, size_t o) {
  if constexpr (FK == 3) {
    const double v = a.qin[((size_t)l * (a.ny + 2) + j + 1) * (a.nx + 2) + i + 1];
    a.q[o] = v;
    return v;
  }
  double v = a.q[o];
  if constexpr (FK > 0) {
    v = ab3_plain<double>(v, u.c0, u.c1, u.c2, u.f0[o], u.f1[o], u.f2[o]);
    if constexpr (FK == 2) {
      if (u.field && l == 0) v = v + u.field[o] * u.sqdt;
      if (u.r1) v = v + forc4d_term<double>(u.r1, u.r2, o, u.w1, u.w2, u.dt);
    }
    a.q[o] = v;
  }
  return v;
}
// f(FK) of the case at hand
template <typename F> __device__ __forceinline__ void q_case(const StepArgs<double>& a, const QUpdate& u, F f) {
  if (a.qin) f(std::integral_constant<int, 3>{});
  else if (!u.upd) f(std::integral_constant<int, 0>{});
  else if (!u.field && !u.r1) f(std::integral_constant<int, 1>{});
  else f(std::integral_constant<int, 2>{});
}

// the terms of GO outputs for one value
template <int GO, bool ODD> __device__ __forceinline__ void modes_add(ModeAcc* s, fx_t x, const Q2* c) {
  const ModeValue v = modes_value<ODD>(x);
#pragma unroll
  for (int g = 0; g < GO; g += 2) {
    const Q4 cc = *reinterpret_cast<const Q4*>(c + g);
    modes_term<ODD>(s[g], v, cc.x);
    if (g + 1 < GO) modes_term<ODD>(s[g + 1 < GO ? g + 1 : g], v, cc.y);
  }
}
__device__ __forceinline__ double modes_out(const ModeAcc& s, int ex, unsigned int turn) {
  const double v = fx_out(s.acc, ex);
  return __longlong_as_double((long long)modes_turned((unsigned long long)__double_as_longlong(v), turn));
}

// One point of a run of NL layers; cs: the constants as [group][l][GE], GE =
// GO rounded up to even.
template <int NL> struct ModeShape {
  static constexpr int NG = NL > 8 ? 2 : 1, GO = (NL + NG - 1) / NG, GE = (GO + 1) & ~1;
  static constexpr int len = NG * NL * GE;
  static constexpr size_t bytes = len * sizeof(Q2) + NL * sizeof(int);  // and the columns' k
};
template <int NL> __device__ __forceinline__ void modes_stage(const ModeTable& tb, Q2* cs) {
  using S = ModeShape<NL>;
  for (int w = threadIdx.x; w < S::len; w += NT) {
    const int g = w % S::GE, l = w / S::GE % NL, n = w / (S::GE * NL), m = n * S::GO + g;
    cs[w] = g < S::GO && m < NL ? tb.c[m * NL + l] : Q2{0, 0};
  }
  if (threadIdx.x < NL) ((int*)(cs + S::len))[threadIdx.x] = tb.e[NL + threadIdx.x];
}
template <int NL, bool FWD>
__device__ __forceinline__ void modes_point(const StepArgs<double>& a, const ModeTable& tb, const QUpdate& u, int j,
                                            int i, const Q2* cs) {
  using S = ModeShape<NL>;
  const size_t o = (size_t)j * a.pitch + i;
  const double* src = FWD ? a.q : a.spec;
  double* dst = FWD ? a.spec : a.psi;
  const int* k = (const int*)(cs + S::len);
  double v[NL];
  ModeMax h = {};
  auto load = [&](auto value) {
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      v[l] = value(l, o + (size_t)l * a.lstride);
      modes_max(h, fx_hi(v[l]), k[l]);
    }
  };
  if constexpr (FWD)
    q_case(a, u, [&](auto fk) { load([&](int l, size_t ol) { return q_value<decltype(fk)::value>(a, u, l, j, i, ol); }); });
  else
    load([&](int, size_t ol) { return src[ol]; });
  grid_next();
  const unsigned int turn = modes_turn(i, j);
  fx_t x[NL];
#pragma unroll
  for (int l = 0; l < NL; ++l) x[l] = modes_in((unsigned long long)__double_as_longlong(v[l]), h, k[l], turn);
#pragma unroll
  for (int n = 0; n < S::NG; ++n) {
    ModeAcc s[S::GO] = {};
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      if (l & 1) modes_add<S::GO, true>(s, x[l], cs + (n * NL + l) * S::GE);
      else modes_add<S::GO, false>(s, x[l], cs + (n * NL + l) * S::GE);
      if ((l & 3) == 3 || l == NL - 1) {
#pragma unroll
        for (int g = 0; g < S::GO; ++g) modes_carry(s[g]);
      }
    }
#pragma unroll
    for (int g = 0; g < S::GO; ++g) {
      const int m = n * S::GO + g;
      if (m < NL) dst[o + (size_t)m * a.lstride] = modes_out(s[g], modes_exp(h, tb.e[m]), turn);
    }
  }
}
// The same for any nl, by the whole block (on: the thread has a point), in
// fixed point or, where a.modes_fx is 0, in FP64.  A block of GY = blockDim.y
// > 1 gives each of its points to GY threads, which take the layers in turns
// as q is brought up to date and then every GY-th group of outputs.  cs:
// shared memory, modes_any_bytes(nl, GY).
constexpr int MODES_GO = 8;  // outputs a thread forms at a time
constexpr size_t modes_any_bytes(int nl, int GY) {
  return sizeof(Q2) * MODES_GO * (size_t)nl * GY + (GY > 1 ? NT * sizeof(ModeMax) : 0);
}
template <bool FWD>
__device__ __forceinline__ void modes_point_any(const StepArgs<double>& a, const ModeTable& tb, const QUpdate& u,
                                                int j, int i, bool on, Q2* cs) {
  constexpr int GO = MODES_GO;
  const int nl = a.nl, y = threadIdx.y, GY = blockDim.y, tid = threadIdx.x + y * blockDim.x;
  const size_t o = (size_t)j * a.pitch + i;
  const double* src = FWD ? a.q : a.spec;
  double* dst = FWD ? a.spec : a.psi;
  const int* k = tb.e + nl;
  ModeMax h = {};
  auto load = [&](auto value) {
    for (int l = y; l < nl; l += GY) modes_max(h, fx_hi(value(l, o + (size_t)l * a.lstride)), k[l]);
  };
  if (on) {
    if constexpr (FWD)
      q_case(a, u, [&](auto fk) { load([&](int l, size_t ol) { return q_value<decltype(fk)::value>(a, u, l, j, i, ol); }); });
    else
      load([&](int, size_t ol) { return src[ol]; });
  }
  if (GY > 1) {
    ModeMax* hs = (ModeMax*)(cs + (size_t)nl * GO * GY);
    hs[tid] = h;
    __syncthreads();
    for (int g = 0; g < GY; ++g) {
      const ModeMax v = hs[g * blockDim.x + threadIdx.x];
      h.raw = max(h.raw, v.raw);
      h.hi = max(h.hi, v.hi);
    }
  }
  const unsigned int turn = modes_turn(i, j);
  const double* mat = FWD ? a.cl2m : a.cm2l;
  double* cd = (double*)cs;
  for (int b0 = 0; b0 < nl; b0 += GO * GY) {
    __syncthreads();
    for (int w = tid; w < nl * GO * GY; w += NT) {
      const int g = w % GO, l = w / GO % nl, m = b0 + w / (GO * nl) * GO + g, e = m * nl + l;
      if (a.modes_fx) cs[w] = m < nl ? tb.c[e] : Q2{0, 0};
      else cd[w] = m < nl ? mat[e] : 0.0;
    }
    __syncthreads();
    const int m0 = b0 + y * GO, c0 = y * nl;
    if (!on || m0 >= nl) continue;
    if (a.modes_fx) {
      ModeAcc s[GO] = {};
      for (int l = 0; l < nl; ++l) {
        const fx_t x = modes_in((unsigned long long)__double_as_longlong(src[o + (size_t)l * a.lstride]), h, k[l], turn);
        if (l & 1) modes_add<GO, true>(s, x, cs + (c0 + l) * GO);
        else modes_add<GO, false>(s, x, cs + (c0 + l) * GO);
        if ((l & 3) == 3 || l == nl - 1) {
#pragma unroll
          for (int g = 0; g < GO; ++g) modes_carry(s[g]);
        }
      }
#pragma unroll
      for (int g = 0; g < GO; ++g)
        if (m0 + g < nl) dst[o + (size_t)(m0 + g) * a.lstride] = modes_out(s[g], modes_exp(h, tb.e[m0 + g]), turn);
    } else {
      double acc[GO] = {};
      for (int l = 0; l < nl; ++l) {
        const double v = src[o + (size_t)l * a.lstride];
        double c[GO];
        ld_coefs<GO, double>(cd + (c0 + l) * GO, c);
#pragma unroll
        for (int g = 0; g < GO; ++g) acc[g] = fmaT(c[g], v, acc[g]);
      }
#pragma unroll
      for (int g = 0; g < GO; ++g)
        if (m0 + g < nl) dst[o + (size_t)(m0 + g) * a.lstride] = acc[g];
    }
  }
}

// The x-transform of nr rows of F, in place, forward or (INV) back: the
// fixed-point DST, the chirp-z DST (HL = -1), or (PER) the real FFT, whose
// spectral rows hold X_0..X_H as (re, im) pairs.  Row r is row j of layer l,
// l ny + j = r0 + r, or (row_j >= 0) row row_j of layer r0 + r.  A, B: nr row
// buffers each.  Starts and ends with the block synchronised.
template <bool PER, int HL, bool INV>
__device__ __forceinline__ void rows_f64(const StepArgs<double>& a, double* F, int r0, int nr, int row_j, double* A,
                                         double* B, double* tot) {
  FxScratch* sc = (FxScratch*)tot;
  const int ld = row_len<double>(a.gx), xo = PER ? 0 : 1;
  const int nin = PER && INV ? a.nx + 2 : a.nx, nout = PER && !INV ? a.nx + 2 : a.nx;
  auto row = [&](int r) {
    const int l = row_j >= 0 ? r0 + r : (r0 + r) / a.ny, j = row_j >= 0 ? row_j : r0 + r - l * a.ny;
    return F + (size_t)l * a.lstride + (size_t)j * a.pitch;
  };
  for (int n = 0; n < (HL == -1 ? 2 : 1); ++n) fx_clear(&sc[n]);
  __syncthreads();
  for (int r = 0; r < nr; ++r) {
    const double* src = row(r);
    unsigned int h = 0;
    for (int i = threadIdx.x; i < nin; i += NT) {
      const double v = src[i];
      A[r * ld + pr<double>(i + xo)] = v;
      h = max(h, fx_hi(v));
    }
    fx_note_max(sc, r, h);
  }
  __syncthreads();
  const fx_t* O;
  if constexpr (!PER) O = dst_fx<HL>(A, B, nr, ld, a.gx, a.fx, sc);
  else if constexpr (INV) O = fx_irfft(A, B, nr, ld, a.gx, a.fx, sc);
  else O = fx_rfft(A, B, nr, ld, a.gx, a.fx, sc);
  grid_next();
  for (int r = 0; r < nr; ++r) {
    double* dst = row(r);
    const int ex = sc->ex[r];
    for (int i = threadIdx.x; i < nout; i += NT) {
      const double v = fx_out(O[r * ld + pr<double>(i + xo)], ex);
      // the backward FFT's x_{2m+1} is minus its imaginary part
      dst[i] = PER && INV && (i & 1) ? -v : v;
    }
  }
  __syncthreads();
}

// Row j of an ensemble member: the projection of its points and the
// transforms of its layers' rows, G at a time, by one block.
template <bool PER, bool INV>
__device__ __forceinline__ void body_rows_f64(const StepArgs<double>& a, int step_mode, int j, unsigned char* smem_raw,
                                              double* tot) {
  if (step_mode && !a.state->active) return;
  const int G = INV ? a.G3 : a.G1, np = PER && INV ? a.nx + 2 : a.nx;
  double* A = (double*)(smem_raw + cst_bytes<double>(a.nl));
  double* B = A + (size_t)G * row_len<double>(a.gx);
  __shared__ QUpdate u;
  if (!INV && threadIdx.x == 0) u = q_update(a, step_mode);
  __syncthreads();
  for (int i0 = 0; i0 < np; i0 += NT)
    modes_point_any<!INV>(a, INV ? a.m2l : a.l2m, u, j, i0 + threadIdx.x, i0 + (int)threadIdx.x < np, (Q2*)smem_raw);
  __syncthreads();
  for (int l = 0; l < a.nl; l += G) rows_f64<PER, -2, INV>(a, INV ? a.psi : a.spec, l, min(G, a.nl - l), j, A, B, tot);
}

}  // namespace qgw
