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
// 83-88% busy): forward rows 0.64 -> 0.34 ms, columns 0.78 -> 0.28, inverse
// rows 0.55 -> 0.28; rel-L2 error of q after 10 steps 1.7e-13 -> 2.3e-14.
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

// The row's sum of 2 - shift over the passes, and the split's shift
__device__ __forceinline__ int fx_drop(const FxScratch* sc, int r, int npass) {
  int d = 0;
  for (int p = 1; p < npass; ++p) d += 2 - fx_pass_shift(sc->mag[p - 1][r]);
  return d;
}

// ---- compile-time lengths H = 2^LGH >= 64
// One Stockham pass (StockhamItem's indices, dst_fixed.cuh) over all rows.
template <int R, int NS, int H>
__device__ __forceinline__ void fx_pass_fixed(const fx_t* src, fx_t* dst, int nrows, int ld, const Q4* tw,
                                              const unsigned int* mag_in, unsigned int* mag_out) {
  constexpr int NB = H / R, S = H / R;
  constexpr int LG = Pad<double>::LG, W = Pad<double>::W;
  auto pco = [](int e) { return e + W * (e >> LG); };
  const int n = nrows * NB;
  for (int w = threadIdx.x; w < n; w += FX_NT) {
    const int r = w / NB, b = w & (NB - 1), k = b & (NS - 1);
    const C2<fx_t>* in = (const C2<fx_t>*)(src + r * ld) + pc<double>(b);
    C2<fx_t>* out = (C2<fx_t>*)(dst + r * ld) + pc<double>((b - k) * R + k);
    C2<fx_t> v[R];
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = in[pco(q * S)];
    if constexpr (NS > 1) fx_twiddle<R>(v, k, NS, fx_pass_shift(mag_in[r]), tw);
    fx_dft<R>(v);
#pragma unroll
    for (int q = 0; q < R; ++q) out[pco(q * NS)] = v[q];
    fx_row_or<NB>(mag_out, r, fx_mag_all<R>(v));
  }
}

template <int LGH>
__device__ fx_t* dst_fx_fixed(double* A, double* B, int nrows, int ld, const FxTables& tb, FxScratch* sc) {
  constexpr int H = 1 << LGH, M = 2 * H, NP8 = LGH / 3, RL = 1 << (LGH % 3), NP = NP8 + (RL > 1 ? 1 : 0);
  static_assert(LGH >= 6 && NP8 <= 3, "two or three radix-8 passes");
  const int tid = threadIdx.x, lane = tid & 31;
  // pre-processing, A -> B
  for (int w = tid; w < nrows * H; w += FX_NT) {
    const int r = w >> LGH, j = (w & (H - 1)) + 1;
    const unsigned int l = fx_pre_item((const unsigned long long*)A + r * ld, (fx_t*)B + r * ld, j, M,
                                       fx_scale(sc->mx[r]), tb.nsj);
    const unsigned int t = __reduce_add_sync(0xffffffffu, l);
    if (lane == 0) atomicAdd(&sc->l1[r], t);
  }
  __syncthreads();
  fx_t* src = (fx_t*)B;
  fx_t* dst = (fx_t*)A;
  auto turn = [&] {
    __syncthreads();
    fx_t* t = src;
    src = dst;
    dst = t;
  };
  fx_pass_fixed<8, 1, H>(src, dst, nrows, ld, nullptr, nullptr, sc->mag[0]);
  turn();
  fx_pass_fixed<8, 8, H>(src, dst, nrows, ld, tb.twq, sc->mag[0], sc->mag[1]);
  turn();
  if constexpr (NP8 == 3) {
    fx_pass_fixed<8, 64, H>(src, dst, nrows, ld, tb.twq + 56, sc->mag[1], sc->mag[2]);
    turn();
  }
  if constexpr (RL > 1) {
    constexpr int NS = 1 << (3 * NP8);
    fx_pass_fixed<RL, NS, H>(src, dst, nrows, ld, tb.twq + NS - 8, sc->mag[NP8 - 1], sc->mag[NP8]);
    turn();
  }
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
static __device__ __noinline__ fx_t* dst_fx_any(double* A, double* B, int nrows, int ld, const DstGeom& g, const FxTables& tb,
                                                FxScratch* sc) {
  const int H = g.H, M = g.M, tid = threadIdx.x, lane = tid & 31;
  // items w of a phase with n items a row, whole warps at a time: f(row,
  // item, whether the lane has one)
  auto items = [&](int n, auto f) {
    for (int w0 = tid - lane; w0 < nrows * n; w0 += FX_NT) {
      const int w = min(w0 + lane, nrows * n - 1), r = w / n;
      f(r, w - r * n, w0 + lane < nrows * n);
    }
  };
  items(H, [&](int r, int i, bool on) {
    unsigned int l = 0;
    if (on)
      l = fx_pre_item((const unsigned long long*)A + r * ld, (fx_t*)B + r * ld, i + 1, M, fx_scale(sc->mx[r]), tb.nsj);
    fx_row_add(sc->l1, r, l);
  });
  __syncthreads();
  fx_t* src = (fx_t*)B;
  fx_t* dst = (fx_t*)A;
  int Ns = 1;
  for (int p = 0; p < g.npass; ++p) {
    const int R = g.radix[p];
    const Q4* tw = tb.twq + (p ? Ns - g.radix[0] : 0);
    items(H / R, [&](int r, int b, bool on) {
      unsigned int m = 0;
      if (on)
        m = fx_stockham_dispatch(R, (const C2<fx_t>*)(src + r * ld), (C2<fx_t>*)(dst + r * ld), b, b % Ns, Ns, H,
                                 p ? fx_pass_shift(sc->mag[p - 1][r]) : 0, tw);
      fx_row_or<0>(sc->mag[p], r, m);
    });
    __syncthreads();
    Ns *= R;
    fx_t* t = src;
    src = dst;
    dst = t;
  }
  items(H / 2 + 1, [&](int r, int k, bool on) {
    if (!on) return;
    const int drop = fx_drop(sc, r, g.npass), s = fx_split_shift(sc->mag[g.npass - 1][r], sc->l1[r], drop);
    fx_split_item((const C2<fx_t>*)(src + r * ld), (C2<fx_t>*)(dst + r * ld), k, H, s, tb.spq);
    if (k == 0) sc->ex[r] = fx_row_exp(sc->mx[r], drop, s);
  });
  __syncthreads();
  // prefix sum: one warp per row, chunk by chunk of 32 odd outputs
  for (int r = tid >> 5; r < nrows; r += FX_NT / 32) {
    fx_t* o = dst + r * ld;
    fx_t carry = 0;
    for (int k0 = 0; k0 < H; k0 += 32) {
      const int k = k0 + lane;
      fx_t v = k < H ? o[pr<double>(2 * k + 1)] : 0;
#pragma unroll
      for (int of = 1; of < 32; of <<= 1) {
        const fx_t u = __shfl_up_sync(0xffffffffu, v, of);
        if (lane >= of) v += u;
      }
      v += carry;
      if (k < H) o[pr<double>(2 * k + 1)] = v;
      carry = __shfl_sync(0xffffffffu, v, 31);
    }
  }
  __syncthreads();
  return dst;
}

// DST-I of nrows raw rows in A (x_j at index j; the block synchronised since
// they were written, their largest high words noted), B the second buffer:
// returns the buffer that holds Y_k at index k as integers of the rows'
// exponents sc->ex.  HL: the half-length whose transform alone the kernel
// holds, or 0.
template <int HL>
__device__ __forceinline__ fx_t* dst_fx(double* A, double* B, int nrows, int ld, const DstGeom& g, const FxTables& tb,
                                        FxScratch* sc) {
  if constexpr (HL == 512) return dst_fx_fixed<9>(A, B, nrows, ld, tb, sc);
  switch (g.H) {
    case 64: return dst_fx_fixed<6>(A, B, nrows, ld, tb, sc);
    case 128: return dst_fx_fixed<7>(A, B, nrows, ld, tb, sc);
    case 256: return dst_fx_fixed<8>(A, B, nrows, ld, tb, sc);
    case 512: return dst_fx_fixed<9>(A, B, nrows, ld, tb, sc);
    case 1024: return dst_fx_fixed<10>(A, B, nrows, ld, tb, sc);
    default: return dst_fx_any(A, B, nrows, ld, g, tb, sc);
  }
}

}  // namespace qgw
