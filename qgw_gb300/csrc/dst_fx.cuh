// dst_fx.cuh -- the block-wide fixed-point DST-I (dst_fx.h) of the FP64 row
// and column kernels: raw doubles of nrows rows in, integers and one exponent
// per row out.
//
// Per row the block keeps, in shared memory: the largest high word of the
// raw doubles (the caller notes it while it writes the rows), sum |X|, the OR
// of the magnitudes after each pass, and the output exponent.  Every thread
// derives a phase's shift from these after the block barrier that ends the
// phase before, so the shifts cost no barrier of their own.
//
// Measured at 1024^2 x 10 against the floating-point transforms (FP64 pipe
// 83-88% busy): columns 0.784 -> 0.227 ms; forward rows 0.640 -> 0.34 and
// inverse rows 0.551 -> 0.28, and with the projections in kernels of their own
// (modes_fx.cuh) 0.249 and 0.195 for both kernels; rel-L2 error of q after 10
// steps 2.3e-13 -> 3.3e-14.  Bound by integer instructions: a product is six
// (three multiplies, of which the wide one issues at 16 a clock and SM), a
// double to fixed point and back a dozen each.
#pragma once

#include "dst_fx.h"

namespace qgw {

constexpr int FX_NT = 256;    // threads per block
constexpr int FX_ROWS = 16;   // rows of one batched transform, at most
constexpr int FX_PASSES = 8;  // Stockham passes, at most (H <= 4096: 2 3^6)

struct FxScratch {
  unsigned int mx[FX_ROWS];               // largest |x|'s high word
  unsigned int l1[FX_ROWS];               // sum |X| (fx_pre_item)
  unsigned int mag[FX_PASSES][FX_ROWS];   // OR of fx_mag after pass p
  int ex[FX_ROWS];                        // output exponent
};

// clear what the next transform accumulates (before the barrier that precedes
// the first fx_note_max); the exponents stay
__device__ __forceinline__ void fx_clear(FxScratch* sc) {
  for (int w = threadIdx.x; w < (2 + FX_PASSES) * FX_ROWS; w += FX_NT) (&sc->mx[0])[w] = 0u;
}
__device__ __forceinline__ unsigned int fx_hi(double v) { return (unsigned int)__double2hiint(v) & 0x7fffffffu; }
// the warp's largest high word of a row joins the row's (whole warps)
__device__ __forceinline__ void fx_note_max(FxScratch* sc, int row, unsigned int hi) {
  const unsigned int m = __reduce_max_sync(0xffffffffu, hi);
  if ((threadIdx.x & 31) == 0) atomicMax(&sc->mx[row], m);
}
// an output as a double; ex the row's exponent.  (The hardware's 64-bit
// conversion runs at the FP64 rate of two a clock and SM: no faster in the
// transforms, and the RHS kernel went from 0.30 to 0.36 ms with it.)
static __device__ __noinline__ double fx_out_far(fx_t v, int ex) {
  return ex == FX_NAN ? __longlong_as_double(0x7ff8000000000000ll) : ldexp((double)v, ex);
}
__device__ __forceinline__ double fx_out(fx_t v, int ex) {
  return fx_exp_ok(ex) ? __longlong_as_double((long long)fx_to_bits(v, ex)) : fx_out_far(v, ex);
}

// OR (add) over the lanes of a warp that hold one row's items, once into the
// row's word.  NB: items per row, a power of two -- or 0: rows may change
// anywhere in the warp (lanes without an item bring 0).
template <int NB> __device__ __forceinline__ void fx_row_or(unsigned int* slot, int r, unsigned int m) {
  const int lane = threadIdx.x & 31;
  if constexpr (NB >= 32) {
    m = __reduce_or_sync(0xffffffffu, m);
    if (lane == 0) atomicOr(&slot[r], m);
  } else if constexpr (NB > 0) {
    const unsigned int group = ((1u << NB) - 1u) << (lane & ~(NB - 1));
    m = __reduce_or_sync(group, m);
    if ((lane & (NB - 1)) == 0) atomicOr(&slot[r], m);
  } else {
    if (__all_sync(0xffffffffu, r == __shfl_sync(0xffffffffu, r, 0))) {
      m = __reduce_or_sync(0xffffffffu, m);
      if (lane == 0) atomicOr(&slot[r], m);
    } else if (m) {
      atomicOr(&slot[r], m);
    }
  }
}
__device__ __forceinline__ void fx_row_add(unsigned int* slot, int r, unsigned int v) {
  if (__all_sync(0xffffffffu, r == __shfl_sync(0xffffffffu, r, 0))) {
    v = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0) atomicAdd(&slot[r], v);
  } else if (v) {
    atomicAdd(&slot[r], v);
  }
}

// The row's sum of 2 - shift over the passes
__device__ __forceinline__ int fx_drop(const FxScratch* sc, int r, int npass) {
  int d = 0;
  for (int p = 1; p < npass; ++p) d += 2 - fx_pass_shift(sc->mag[p - 1][r]);
  return d;
}

// ---- compile-time lengths H = 2^LGH >= 64
// One Stockham pass (StockhamItem's indices, dst_fixed.cuh) over all rows;
// RAW (the first pass): of raw doubles, whose largest high words mag_in holds.
// ONE: in place -- the block's threads take items of whole rows, one each or U
// of one row, and read all of them before any is written.
template <int R, int NS, int H, bool RAW = false, bool ONE = false>
__device__ __forceinline__ void fx_pass_fixed(const fx_t* src, fx_t* dst, int nrows, int ld, const Q4* tw,
                                              const unsigned int* mag_in, unsigned int* mag_out) {
  constexpr int NB = H / R, S = H / R;
  constexpr int LG = Pad<double>::LG, W = Pad<double>::W;
  auto pco = [](int e) { return e + W * (e >> LG); };
  static_assert(!ONE || ((FX_NT % NB == 0 || NB % FX_NT == 0) && NB >= 32), "a round is whole rows, and whole warps");
  if constexpr (ONE && NB > FX_NT) {  // a row a round, U items a thread
    constexpr int U = NB / FX_NT;
    for (int r = 0; r < nrows; ++r) {
      C2<fx_t>* row = (C2<fx_t>*)(src + r * ld);
      C2<fx_t> v[U][R];
      unsigned int m = 0;
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int q = 0; q < R; ++q) v[u][q] = row[pc<double>((int)threadIdx.x + u * FX_NT) + pco(q * S)];
      __syncthreads();
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int b = threadIdx.x + u * FX_NT, k = b & (NS - 1);
        fx_twiddle<R>(v[u], k, NS, fx_pass_shift(mag_in[r]), tw);
        fx_dft<R>(v[u]);
#pragma unroll
        for (int q = 0; q < R; ++q) row[pc<double>((b - k) * R + k) + pco(q * NS)] = v[u][q];
        m |= fx_mag_all<R>(v[u]);
      }
      fx_row_or<NB>(mag_out, r, m);
    }
    return;
  }
  const int n = nrows * NB;
  for (int w = threadIdx.x; ONE ? w - (int)threadIdx.x < n : w < n; w += FX_NT) {
    const int r = w / NB, b = w & (NB - 1), k = b & (NS - 1);
    const C2<fx_t>* in = (const C2<fx_t>*)(src + r * ld) + pc<double>(b);
    C2<fx_t>* out = (C2<fx_t>*)(dst + r * ld) + pc<double>((b - k) * R + k);
    C2<fx_t> v[R];
    if (!ONE || w < n) {
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = in[pco(q * S)];
    }
    if constexpr (ONE) {
      __syncthreads();
      if (w >= n) continue;
    }
    if constexpr (RAW) {
      const int E = fx_scale(mag_in[r]);
#pragma unroll
      for (int q = 0; q < R; ++q) {
        v[q].x = fx_from_bits((unsigned long long)v[q].x, E);
        v[q].y = fx_from_bits((unsigned long long)v[q].y, E);
      }
    }
    if constexpr (NS > 1) fx_twiddle<R>(v, k, NS, fx_pass_shift(mag_in[r]), tw);
    fx_dft<R>(v);
#pragma unroll
    for (int q = 0; q < R; ++q) out[pco(q * NS)] = v[q];
    fx_row_or<NB>(mag_out, r, fx_mag_all<R>(v));
  }
}

// The passes of the complex FFT of 2^LGH points from src, dst the second
// buffer; returns the buffer of the result, whose magnitudes are in
// sc->mag[passes - 1].  Ends with the block synchronised.
template <int LGH, bool RAW, bool ONE = false>
__device__ __forceinline__ fx_t* fx_passes_fixed(fx_t* src, fx_t* dst, int nrows, int ld, const Q4* tw, FxScratch* sc) {
  constexpr int H = 1 << LGH, NP8 = LGH / 3, RL = 1 << (LGH % 3);
  static_assert(LGH >= 6 && NP8 <= 4, "two to four radix-8 passes");
  auto turn = [&] {
    __syncthreads();
    fx_t* t = src;
    src = dst;
    dst = t;
  };
  fx_pass_fixed<8, 1, H, RAW, ONE>(src, dst, nrows, ld, nullptr, sc->mx, sc->mag[0]);
  turn();
  fx_pass_fixed<8, 8, H, false, ONE>(src, dst, nrows, ld, tw, sc->mag[0], sc->mag[1]);
  turn();
  if constexpr (NP8 >= 3) {
    fx_pass_fixed<8, 64, H, false, ONE>(src, dst, nrows, ld, tw + 56, sc->mag[1], sc->mag[2]);
    turn();
  }
  if constexpr (NP8 >= 4) {
    fx_pass_fixed<8, 512, H>(src, dst, nrows, ld, tw + 504, sc->mag[2], sc->mag[3]);
    turn();
  }
  if constexpr (RL > 1) {
    constexpr int NS = 1 << (3 * NP8);
    fx_pass_fixed<RL, NS, H, false, ONE>(src, dst, nrows, ld, tw + NS - 8, sc->mag[NP8 - 1], sc->mag[NP8]);
    turn();
  }
  return src;
}

// ONE (LGH = 9, 10): all in A, B unused.  Apart from the passes every item writes
// what it alone reads.  Half the shared memory, so a fourth block per SM at 64
// registers, for one more barrier a pass: 1024^2 x 10 columns 0.257 -> 0.227
// ms, rows 0.258 -> 0.254 and 0.197 -> 0.193; 2048^2 x 6 columns 0.782 ->
// 0.619, rows 0.571 -> 0.557 and 0.443 -> 0.430.
template <int LGH, bool ONE = false>
__device__ fx_t* dst_fx_fixed(double* A, double* B, int nrows, int ld, const FxTables& tb, FxScratch* sc) {
  constexpr int H = 1 << LGH, M = 2 * H, NP = LGH / 3 + (LGH % 3 ? 1 : 0);
  const int tid = threadIdx.x, lane = tid & 31;
  if (ONE) B = A;
  // pre-processing, A -> B
  for (int w = tid; w < nrows * H; w += FX_NT) {
    const int r = w >> LGH, j = (w & (H - 1)) + 1;
    const unsigned int l = fx_pre_item((const unsigned long long*)A + r * ld, (fx_t*)B + r * ld, j, M,
                                       fx_scale(sc->mx[r]), tb.nsj);
    const unsigned int t = __reduce_add_sync(0xffffffffu, l);
    if (lane == 0) atomicAdd(&sc->l1[r], t);
  }
  __syncthreads();
  fx_t* src = fx_passes_fixed<LGH, false, ONE>((fx_t*)B, (fx_t*)A, nrows, ld, tb.twq, sc);
  fx_t* dst = ONE ? src : src == (fx_t*)A ? (fx_t*)B : (fx_t*)A;
  // split: items k = 0..H/2-1, item 0 also k = H/2 (and R_0)
  {
    constexpr int KI = H / 2;
    for (int w = tid; w < nrows * KI; w += FX_NT) {
      const int r = w / KI, k = w & (KI - 1);
      const int drop = fx_drop(sc, r, NP), s = fx_split_shift(sc->mag[NP - 1][r], sc->l1[r], drop);
      const C2<fx_t>* Z = (const C2<fx_t>*)(src + r * ld);
      C2<fx_t>* o = (C2<fx_t>*)(dst + r * ld);
      const int kk = k == 0 ? KI : k, ia = pc<double>(kk), ib = pc<double>(H - kk);
      C2<fx_t> lo, hi;
      fx_split_pair(fx_shift2(Z[ia], s), fx_shift2(Z[ib], s), tb.spq[kk], lo, hi);
      o[ia] = lo;
      if (k == 0) {
        const C2<fx_t> a = fx_shift2(Z[0], s);
        hi.x = 0;
        hi.y = a.x + a.y;  // R_0
        o[0] = hi;
        sc->ex[r] = fx_row_exp(sc->mx[r], drop, s);
      } else {
        o[ib] = hi;
      }
    }
  }
  __syncthreads();
  // prefix sum of the odd outputs, one warp per row: lane c holds the chunk
  // of CH values from k = c CH in registers
  {
    constexpr int CH = H >= 256 ? H / 32 : 8, NC = H / CH;
    static_assert((2 * CH) % (2 * Pad<double>::P) == 0, "chunks of whole pad periods");
    for (int r = tid >> 5; r < nrows; r += FX_NT / 32) {
      fx_t* o = dst + r * ld + pr<double>(2 * CH * lane) + 1;
      fx_t v[CH], run = 0;
      if (lane < NC) {
#pragma unroll
        for (int t = 0; t < CH; ++t) v[t] = run = run + o[pr<double>(2 * t)];
      }
      fx_t incl = run;
#pragma unroll
      for (int of = 1; of < 32; of <<= 1) {
        const fx_t u = __shfl_up_sync(0xffffffffu, incl, of);
        if (lane >= of) incl += u;
      }
      const fx_t base = incl - run;
      if (lane < NC) {
#pragma unroll
        for (int t = 0; t < CH; ++t) o[pr<double>(2 * t)] = base + v[t];
      }
    }
  }
  __syncthreads();
  return dst;
}

// ---- any half-length that is a product of 2, 3, 5 and 7
// items w of a phase with n items a row, whole warps at a time: f(row, item,
// whether the lane has one)
template <typename F> __device__ __forceinline__ void fx_items(int nrows, int n, F f) {
  const int lane = threadIdx.x & 31;
  const unsigned int inv = 0xffffffffu / (unsigned int)n + 1;  // w / n exactly, w n < 2^32
  for (int w0 = threadIdx.x - lane; w0 < nrows * n; w0 += FX_NT) {
    const int w = min(w0 + lane, nrows * n - 1), r = n == 1 ? w : (int)__umulhi((unsigned int)w, inv);
    f(r, w - r * n, w0 + lane < nrows * n);
  }
}
template <bool RAW>
__device__ __forceinline__ fx_t* fx_passes_any(fx_t* src, fx_t* dst, int nrows, int ld, const DstGeom& g, const Q4* twq,
                                               FxScratch* sc) {
  const int H = g.H;
  if constexpr (RAW) {
    fx_items(nrows, H, [&](int r, int e, bool on) {
      if (!on) return;
      fx_t* p = src + r * ld + 2 * pc<double>(e);
      const int E = fx_scale(sc->mx[r]);
      p[0] = fx_from_bits((unsigned long long)p[0], E);
      p[1] = fx_from_bits((unsigned long long)p[1], E);
    });
    __syncthreads();
  }
  int Ns = 1;
  for (int p = 0; p < g.npass; ++p) {
    const int R = g.radix[p];
    const Q4* tw = twq + (p ? Ns - g.radix[0] : 0);
    const unsigned int inv = 0xffffffffu / (unsigned int)Ns + 1;
    fx_items(nrows, H / R, [&](int r, int b, bool on) {
      unsigned int m = 0;
      if (on)
        m = fx_stockham_dispatch(R, (const C2<fx_t>*)(src + r * ld), (C2<fx_t>*)(dst + r * ld), b,
                                 Ns == 1 ? 0 : b - Ns * (int)__umulhi((unsigned int)b, inv), Ns, H,
                                 p ? fx_pass_shift(sc->mag[p - 1][r]) : 0, tw);
      fx_row_or<0>(sc->mag[p], r, m);
    });
    __syncthreads();
    Ns *= R;
    fx_t* t = src;
    src = dst;
    dst = t;
  }
  return src;
}
static __device__ __noinline__ fx_t* dst_fx_any(double* A, double* B, int nrows, int ld, const DstGeom& g, const FxTables& tb,
                                                FxScratch* sc) {
  __builtin_assume(__isShared(A));
  __builtin_assume(__isShared(B));
  __builtin_assume(__isShared(sc));
  const int H = g.H, M = g.M, tid = threadIdx.x, lane = tid & 31;
  fx_items(nrows, H, [&](int r, int i, bool on) {
    unsigned int l = 0;
    if (on)
      l = fx_pre_item((const unsigned long long*)A + r * ld, (fx_t*)B + r * ld, i + 1, M, fx_scale(sc->mx[r]), tb.nsj);
    fx_row_add(sc->l1, r, l);
  });
  __syncthreads();
  fx_t* src = fx_passes_any<false>((fx_t*)B, (fx_t*)A, nrows, ld, g, tb.twq, sc);
  fx_t* dst = src == (fx_t*)A ? (fx_t*)B : (fx_t*)A;
  fx_items(nrows, H / 2 + 1, [&](int r, int k, bool on) {
    if (!on) return;
    const int drop = fx_drop(sc, r, g.npass), s = fx_split_shift(sc->mag[g.npass - 1][r], sc->l1[r], drop);
    fx_split_item((const C2<fx_t>*)(src + r * ld), (C2<fx_t>*)(dst + r * ld), k, H, s, tb.spq);
    if (k == 0) sc->ex[r] = fx_row_exp(sc->mx[r], drop, s);
  });
  __syncthreads();
  // prefix sum: one warp per row; a lane adds up its ceil(H / 32) odd outputs,
  // then writes their running sums on top of the lanes' before it
  const int ch = (H + 31) / 32, k0 = min(lane * ch, H), k1 = min(k0 + ch, H);
  for (int r = tid >> 5; r < nrows; r += FX_NT / 32) {
    fx_t* o = dst + r * ld;
    fx_t sum = 0;
    for (int k = k0; k < k1; ++k) sum += o[pr<double>(2 * k + 1)];
    fx_t incl = sum;
#pragma unroll
    for (int of = 1; of < 32; of <<= 1) {
      const fx_t u = __shfl_up_sync(0xffffffffu, incl, of);
      if (lane >= of) incl += u;
    }
    fx_t run = incl - sum;
    for (int k = k0; k < k1; ++k) {
      run += o[pr<double>(2 * k + 1)];
      o[pr<double>(2 * k + 1)] = run;
    }
  }
  __syncthreads();
  return dst;
}

// The complex FFT of g.H points (a power of two from 64 to 1024, or any
// supported length) of nrows rows: src raw doubles (RAW) or integers.
template <bool RAW>
__device__ __forceinline__ fx_t* fx_cfft(fx_t* src, fx_t* dst, int nrows, int ld, const DstGeom& g, const Q4* twq,
                                         FxScratch* sc) {
  switch (g.H) {
    case 64: return fx_passes_fixed<6, RAW>(src, dst, nrows, ld, twq, sc);
    case 128: return fx_passes_fixed<7, RAW>(src, dst, nrows, ld, twq, sc);
    case 256: return fx_passes_fixed<8, RAW>(src, dst, nrows, ld, twq, sc);
    case 512: return fx_passes_fixed<9, RAW>(src, dst, nrows, ld, twq, sc);
    case 1024: return fx_passes_fixed<10, RAW>(src, dst, nrows, ld, twq, sc);
    default: return fx_passes_any<RAW>(src, dst, nrows, ld, g, twq, sc);
  }
}
// Real FFT of raw rows (x_i at index i): 2 X_k, k = 0..H, as complex values at
// index k, with the rows' exponents (of X_k) in sc->ex; and the inverse, c2r,
// of raw spectral rows: x_{2m} = Re, x_{2m+1} = -Im of the value at index m.
__device__ __forceinline__ fx_t* fx_rfft(double* A, double* B, int nrows, int ld, const DstGeom& g, const FxTables& tb,
                                         FxScratch* sc) {
  const int H = g.H;
  fx_t* src = fx_cfft<true>((fx_t*)A, (fx_t*)B, nrows, ld, g, tb.twq, sc);
  fx_t* dst = src == (fx_t*)A ? (fx_t*)B : (fx_t*)A;
  fx_items(nrows, H / 2 + 1, [&](int r, int k, bool on) {
    if (!on) return;
    const int s = fx_rsplit_shift(sc->mag[g.npass - 1][r]);
    fx_rsplit_item((const C2<fx_t>*)(src + r * ld), (C2<fx_t>*)(dst + r * ld), k, H, s, tb.spq);
    // (fx_row_exp's exponent is one more than X's, and 2 X two: 2 X lies at
    // fx_row_exp - 1, X one below)
    if (k == 0) sc->ex[r] = fx_exp_add(fx_row_exp(sc->mx[r], fx_drop(sc, r, g.npass), s), -2);
  });
  __syncthreads();
  return dst;
}
__device__ __forceinline__ fx_t* fx_irfft(double* A, double* B, int nrows, int ld, const DstGeom& g, const FxTables& tb,
                                          FxScratch* sc) {
  const int H = g.H;
  fx_items(nrows, H / 2 + 1, [&](int r, int k, bool on) {
    if (on) fx_rjoin_item((const C2<double>*)(A + r * ld), (C2<fx_t>*)(B + r * ld), k, H, fx_scale(sc->mx[r]), tb.spq);
  });
  __syncthreads();
  fx_t* src = fx_cfft<false>((fx_t*)B, (fx_t*)A, nrows, ld, g, tb.twq, sc);
  if (threadIdx.x < nrows) {
    const int r = threadIdx.x;
    sc->ex[r] = fx_exp_add(fx_row_exp(sc->mx[r], fx_drop(sc, r, g.npass), 0), 2);
  }
  __syncthreads();
  return src;
}
// Chirp-z DST-I of raw rows (dst_blue.h), rows of L complex values, g.H = L;
// sc: two scratches.  The result Y_k at index k.
__device__ __forceinline__ fx_t* dst_fx_blue(double* A, double* B, int nrows, int ld, const DstGeom& g, const FxTables& tb,
                                             FxScratch* sc) {
  const int M = g.M, L = g.H;
  auto passes = [&](fx_t* src, fx_t* dst, FxScratch* s) {
    switch (L) {
      case 64: return fx_passes_fixed<6, false>(src, dst, nrows, ld, tb.twq, s);
      case 128: return fx_passes_fixed<7, false>(src, dst, nrows, ld, tb.twq, s);
      case 256: return fx_passes_fixed<8, false>(src, dst, nrows, ld, tb.twq, s);
      case 512: return fx_passes_fixed<9, false>(src, dst, nrows, ld, tb.twq, s);
      case 1024: return fx_passes_fixed<10, false>(src, dst, nrows, ld, tb.twq, s);
      case 2048: return fx_passes_fixed<11, false>(src, dst, nrows, ld, tb.twq, s);
      case 4096: return fx_passes_fixed<12, false>(src, dst, nrows, ld, tb.twq, s);
      default: return fx_passes_any<false>(src, dst, nrows, ld, g, tb.twq, s);
    }
  };
  fx_items(nrows, L, [&](int r, int m, bool on) {
    if (on)
      fx_chirp_item((const unsigned long long*)A + r * ld, (C2<fx_t>*)((fx_t*)B + r * ld), m, M, fx_scale(sc->mx[r]), tb.bc);
  });
  __syncthreads();
  fx_t* O = passes((fx_t*)B, (fx_t*)A, &sc[0]);
  fx_items(nrows, L, [&](int r, int k, bool on) {
    if (on) fx_chirp_mul_item((C2<fx_t>*)(O + r * ld), k, fx_pass_shift(sc[0].mag[g.npass - 1][r]), tb.bz);
  });
  __syncthreads();
  fx_t* D = passes(O, O == (fx_t*)A ? (fx_t*)B : (fx_t*)A, &sc[1]);
  fx_t* out = D == (fx_t*)A ? (fx_t*)B : (fx_t*)A;
  fx_items(nrows, M, [&](int r, int k, bool on) {
    if (!on) return;
    const int s = fx_pass_shift(sc[1].mag[g.npass - 1][r]);
    fx_chirp_out_item((const C2<fx_t>*)(D + r * ld), out + r * ld, k, s, tb.bc);
    if (k == 0) {
      // passes, product, passes, output (each product by a table / 4), 2 / L
      const int drop = fx_drop(&sc[0], r, g.npass) + (2 - fx_pass_shift(sc[0].mag[g.npass - 1][r])) + tb.be +
                       fx_drop(&sc[1], r, g.npass) + 2 + 1 - (31 - __clz(L));
      sc->ex[r] = fx_exp_add(fx_row_exp(sc->mx[r], drop, s), -1);
    }
  });
  __syncthreads();
  return out;
}

// DST-I of nrows raw rows in A (x_j at index j; the block synchronised since
// they were written, their largest high words noted), B the second buffer:
// returns the buffer that holds Y_k at index k as integers of the rows'
// exponents sc->ex.  HL: the half-length whose transform alone the kernel
// holds, 0 for those without a kernel of their own, -1 for the chirp-z lengths,
// -2 for all but these (the batched kernels, two buffers).
template <int HL>
__device__ __forceinline__ fx_t* dst_fx(double* A, double* B, int nrows, int ld, const DstGeom& g, const FxTables& tb,
                                        FxScratch* sc) {
  if constexpr (HL == 512) return dst_fx_fixed<9, true>(A, B, nrows, ld, tb, sc);
  if constexpr (HL == 1024) return dst_fx_fixed<10, true>(A, B, nrows, ld, tb, sc);
  if constexpr (HL == -1) return dst_fx_blue(A, B, nrows, ld, g, tb, sc);
  if constexpr (HL == -2) {
    if (g.H == 512) return dst_fx_fixed<9>(A, B, nrows, ld, tb, sc);
    if (g.H == 1024) return dst_fx_fixed<10>(A, B, nrows, ld, tb, sc);
  }
  switch (g.H) {
    case 64: return dst_fx_fixed<6>(A, B, nrows, ld, tb, sc);
    case 128: return dst_fx_fixed<7>(A, B, nrows, ld, tb, sc);
    case 256: return dst_fx_fixed<8>(A, B, nrows, ld, tb, sc);
    default: return dst_fx_any(A, B, nrows, ld, g, tb, sc);
  }
}

}  // namespace qgw
