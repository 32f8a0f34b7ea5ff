// kernels.cu -- the single-run step kernels, the small kernels (begin,
// flush, forcing, boundary copies, budget) and their launchers; the device
// side they share with the ensemble kernels is step_device.cuh.
#include "step_device.cuh"

// The FP64 and the FP32c instantiations compile as two translation units
// (in parallel): this file compiled directly is part 1 (the FP64 kernels and
// the precision-free helpers), kernels_f32c.cu includes it as part 2 (the
// FP32c kernels).  The few non-template kernels are static to each unit.
#ifndef QGW_KERNELS_PART
#define QGW_KERNELS_PART 1
#endif

namespace qgw {

// ------------------------------------------------- single-run wrappers
// The row kernels of the FP32c path (FP64: k_modes and k_rows_f64 below).
// HL: 0, or the half-length whose transform alone the kernel holds (512:
// the 1024-point rows and columns of the common grid)
template <typename T, bool COMP, bool PER, int HL>
__global__ void __launch_bounds__(NT, 4) k_rows_fwd(StepArgs<T> a, int step_mode) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(16) T tot[tot_len<T>];
  grid_wait();
  body_rows_fwd<T, COMP, PER, HL>(a, step_mode, blockIdx.x, smem_raw + cst_bytes<T>(a.nl), tot, (T*)smem_raw);
}
// FP64, HL = 512, 1024: in place, four blocks per SM at 64 registers (dst_fx_fixed).
// CT: columns per tile (closed basin, and complex columns in FP64; the FP32
// periodic kernel takes two complex columns whatever CT)
template <typename T, bool COMP, bool PER, int CT, int HL>
__global__ void __launch_bounds__(NT, sizeof(T) == 8 && HL >= 512 ? 4 : 3) k_cols(const __grid_constant__ StepArgs<T> a, int step_mode) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(16) T tot[tot_len<T, HL>];
  grid_wait();
  if constexpr (PER && sizeof(T) == 8) body_cols_per_fx<CT>(a, step_mode, blockIdx.x, blockIdx.y, smem_raw, tot);
  else if constexpr (PER) body_cols_per<T, COMP>(a, step_mode, blockIdx.x, blockIdx.y, smem_raw);
  else body_cols<T, COMP, CT, HL>(a, step_mode, blockIdx.x, blockIdx.y, smem_raw, tot);
}
template <typename T> constexpr int CTD = ColsPer<T>::value;
// four blocks per SM (64 registers; at 1024^2 x 10 the kernel drops from
// 0.109 to 0.101 ms)
template <typename T, bool COMP, bool PER, int HL>
__global__ void __launch_bounds__(NT, 4) k_rows_inv(StepArgs<T> a, int step_mode) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(16) T tot[tot_len<T>];
  grid_wait();
  body_rows_inv<T, COMP, PER, HL>(a, step_mode, blockIdx.x, smem_raw + cst_bytes<T>(a.nl), tot, (T*)smem_raw,
                                  gridDim.y > 1 ? (int)blockIdx.y : -1);
}
// The RHS of a step: a persistent grid (a.rhs_grid blocks) over the
// ntx x nty x nl tiles (body_rhs_tiles); the FP64 path launches one block
// per tile (bound by its integer instructions; blocks that each load one
// tile overlap one another's loads without a second buffer).
template <typename T, bool COMP, int R, int TY>
__global__ void __launch_bounds__(NT, sizeof(T) == 4 ? 5 : 4) k_rhs(const __grid_constant__ StepArgs<T> a, int ntx,
                                                                    int nty) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ unsigned long long bar[4];
  // TMA destinations are 128-byte aligned (the launch adds 128 bytes)
  unsigned char* base = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  if (threadIdx.x == 0 && threadIdx.y == 0)
    for (int b = 0; b < 4; ++b) mbar_init(&bar[b]);
  grid_wait();
  __syncthreads();
  body_rhs_tiles<T, COMP, R, TY, rhs_nbuf<T>()>(a, ntx, nty, base, a.use_tma ? &a.tm[0] : nullptr, bar);
}

// FP64: the projections, one thread per point (NL: layers in registers; 0:
// any number, blockDim.y threads per point), and the row transforms (modes_fx.cuh).  The projections wait
// on their loads: five blocks per SM below eight layers (48 registers, few
// spills), four from there on.  Both forward kernels at three, four and five
// blocks: 1024^2 x 10 0.265, 0.256 and 0.258 ms, 768^2 x 8 0.182, 0.173 and
// 0.181, 1024^2 x 6 0.163, 0.157 and 0.155; at two to five, 512^2 x 12 0.124,
// 0.113, 0.107 and 0.115, 512^2 x 16 0.162, 0.150, 0.147 and 0.181.  Any number
// needs the registers (two and five: 256^2 x 20 0.081 and 0.141).
template <int NL, bool FWD>
__global__ void __launch_bounds__(NT, NL == 0 ? 2 : NL >= 8 ? 4 : 5) k_modes(const __grid_constant__ StepArgs<double> a, int step_mode) {
  grid_wait();
  if (step_mode && !a.state->active) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Q2* cs = (Q2*)smem_raw;
  const ModeTable& tb = FWD ? a.l2m : a.m2l;
  __shared__ QUpdate u;
  if (FWD && threadIdx.x == 0 && (NL > 0 || threadIdx.y == 0)) u = q_update(a, step_mode);
  if constexpr (NL > 0) modes_stage<NL>(tb, cs);
  __syncthreads();
  const int np = !FWD && a.periodic ? a.nx + 2 : a.nx;
  const int w = blockIdx.x * (NL > 0 ? NT : blockDim.x) + threadIdx.x, j = w / np, i = w - j * np;
  if constexpr (NL == 0) modes_point_any<FWD>(a, tb, u, j, i, j < a.ny, cs);
  else if (j < a.ny) modes_point<NL, FWD>(a, tb, u, j, i, cs);
}
template <bool PER, int HL, bool INV>
__global__ void __launch_bounds__(NT, HL >= 512 ? 4 : 3) k_rows_f64(const __grid_constant__ StepArgs<double> a, int step_mode) {
  grid_wait();
  if (step_mode && !a.state->active) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(16) double tot[tot_len<double, HL>];
  const int rows = INV ? a.RB3 : a.RB1, r0 = blockIdx.x * rows;
  double* A = (double*)smem_raw;
  rows_f64<PER, HL, INV>(a, INV ? a.psi : a.spec, r0, min(rows, a.nl * a.ny - r0), -1, A,
                         A + (size_t)rows * row_len<double>(a.gx), tot);
}

// ------------------------------------------------------- small kernels
static __global__ void k_begin(DevState* st, double t_out, double tend) {
  grid_wait();
  begin_state(st, t_out, tend, 0);
}

template <typename T, bool COMP>
// (a.qout: also writes the final q, joined to FP64, into the caller's array
// in the reference layout, its ring included)
__global__ void __launch_bounds__(NT) k_flush(StepArgs<T> a) {
  grid_wait();
  DevState* st = a.state;
  const bool pend = st->pending != 0;
  if (!pend && !a.qout) return;
  int s0, s1, s2;
  slabs(st->step_index, s0, s1, s2);
  const double c0 = st->c0, c1 = st->c1, c2 = st->c2;
  const double sqdt = sqrt(st->dt);
  const size_t fs = (size_t)a.nl * a.lstride;
  const T* f0 = a.fab + s0 * fs;
  const T* f1 = a.fab + s1 * fs;
  const T* f2 = a.fab + s2 * fs;
  const T* r1 = nullptr;
  const T* r2 = nullptr;
  T w1 = T(0), w2 = T(0);
  if (a.nrec > 0) {
    const Forc4D fw = forc4d_at(st->t_prev, a.dt_forc, a.nrec);
    r1 = a.frec + fw.i1 * fs;
    r2 = a.frec + fw.i2 * fs;
    w1 = (T)fw.w1;
    w2 = (T)fw.w2;
  }
  const int nxp2 = a.nx + 2;
  for (int row = blockIdx.x; row < a.nl * a.ny; row += gridDim.x) {
    const int l = row / a.ny, j = row - l * a.ny;
    const size_t o0 = (size_t)l * a.lstride + (size_t)j * a.pitch;
    // the caller's row, and the ring row that goes with the first and last:
    // zero at walls (no-slip rings do not come this way), wrapped if periodic
    double* out = a.qout ? a.qout + ((size_t)l * (a.ny + 2) + j + 1) * nxp2 : nullptr;
    for (int i = threadIdx.x; i < a.nx; i += NT) {
      const size_t o = o0 + i;
      // layer 0 also takes the stochastic forcing (src/timestep.h:143-150)
      const T* fo = (a.fr.on && l == 0) ? a.fr.field + o : nullptr;
      double v;
      if (COMP) {
        float hi = (float)a.q[o], lo = (float)a.qlo[o];
        if (pend) {
          const float d = ab3_increment((float)c0, (float)c1, (float)c2, (float)f0[o], (float)f1[o], (float)f2[o]);
          comp_add(hi, lo, d);
          if (fo) comp_add(hi, lo, (float)*fo * (float)sqdt);
          if (r1) comp_add(hi, lo, (float)forc4d_term<T>(r1, r2, o, w1, w2, (T)st->dt));
          a.q[o] = (T)hi;
          a.qlo[o] = (T)lo;
        }
        v = (double)hi + (double)lo;
      } else {
        T q = a.q[o];
        if (pend) {
          q = ab3_plain<T>(q, (T)c0, (T)c1, (T)c2, f0[o], f1[o], f2[o]);
          if (fo) q = q + *fo * (T)sqdt;
          if (r1) q = q + forc4d_term<T>(r1, r2, o, w1, w2, (T)st->dt);
          a.q[o] = q;
        }
        v = (double)q;
      }
      if (out) {
        auto put = [&](double* at, double x) {
          at[i + 1] = x;
          if (i == (a.periodic ? a.nx - 1 : 0)) at[0] = a.periodic ? x : 0.0;
          if (i == (a.periodic ? 0 : a.nx - 1)) at[nxp2 - 1] = a.periodic ? x : 0.0;
        };
        put(out, v);
        if (j == 0) put(out + (a.periodic ? a.ny : -1) * nxp2, a.periodic ? v : 0.0);
        if (j == a.ny - 1) put(out + (a.periodic ? -a.ny : 1) * nxp2, a.periodic ? v : 0.0);
      }
    }
  }
}

// the end of a call: nothing pending, and the scalars into the host's pinned
// copy (a copy of their own behind the kernels cost 5 us a call)
static __global__ void k_end(DevState* st, DevState* host) {
  grid_wait();
  if (threadIdx.x == 0) st->pending = 0;
  __syncthreads();
  static_assert(sizeof(DevState) % 4 == 0 && sizeof(DevState) <= 4 * 64, "one word per thread");
  if (threadIdx.x < sizeof(DevState) / 4) ((int*)host)[threadIdx.x] = ((const int*)st)[threadIdx.x];
}

// --------------------------------------------------- stochastic forcing
// F1: new ring amplitudes after each completed step (calc_forc,
// src/forcing.h:170-190): three draws per ring point from the C-library
// sequence in the order the reference consumes them (the logarithm's,
// the cosine's, the phase's), made by one thread chunk by chunk; the
// transcendental functions run on all threads.
constexpr double QGW_PI = 3.14159265358979323846;
constexpr int FORC_CHUNK = 1024;

template <typename T>
__global__ void __launch_bounds__(NT) k_forc_modes(StepArgs<T> a) {
  DevState* st = a.state;
  const ForcArgs<T>& f = a.fr;
  __shared__ uint32_t rv[3 * FORC_CHUNK];
  __shared__ GlibcRand g;
  __shared__ int go;
  const int tid = threadIdx.x;
  if (tid == 0) {
    go = st->forc_step != st->step_index;  // one field per completed step
    if (go) g = *f.rng;
  }
  __syncthreads();
  if (!go) return;
  for (int c0 = 0; c0 < f.nring; c0 += FORC_CHUNK) {
    const int nc = min(FORC_CHUNK, f.nring - c0);
    if (tid == 0)
      for (int k = 0; k < 3 * nc; ++k) rv[k] = glibc_rand_next(&g);
    __syncthreads();
    for (int k = tid; k < nc; k += NT) {
      const int ii = c0 + k;
      const int i = f.ring[2 * ii], j = f.ring[2 * ii + 1];
      const double rl = (double)rv[3 * k], rc = (double)rv[3 * k + 1], rp = (double)rv[3 * k + 2];
      const double nn = sqrt(-2. * log((rl + 1.) / (GLIBC_RAND_MAX + 2.))) * cos(2 * QGW_PI * rc / GLIBC_RAND_MAX);
      const double em = f.env * (f.sigma * nn);
      const double ph = rp / GLIBC_RAND_MAX * 2 * QGW_PI;
      T* d = f.spec + (size_t)j * f.fpitch + 2 * i;
      d[0] = (T)(em * cos(ph));
      d[1] = (T)(em * sin(ph));
    }
    __syncthreads();
  }
  if (tid == 0) {
    *f.rng = g;
    st->forc_step = st->step_index;
  }
}

// F2: backward complex FFT along j of two complex columns i per block
// (the first dimension of the NF x NF c2r, unnormalised); only the columns
// up to the ring's largest i: the others stay zero in both buffers.
template <typename T>
__global__ void __launch_bounds__(NT) k_forc_cols(StepArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const ForcArgs<T>& f = a.fr;
  const int ld = padded_len<T>(f.gy.M);
  T* A = (T*)smem_raw;
  T* B = A + 2 * ld;
  const int c4 = 4 * blockIdx.x;
  for (int j = threadIdx.x; j < f.NF; j += NT) {
    T v[4];
    load_cols<T, 4>(f.spec + (size_t)j * f.fpitch + c4, v);
    C2<T> z0, z1;
    z0.x = v[0]; z0.y = -v[1]; z1.x = v[2]; z1.y = -v[3];
    ((C2<T>*)A)[pc<T>(j)] = z0;
    ((C2<T>*)(A + ld))[pc<T>(j)] = z1;
  }
  __syncthreads();
  T* O = cfft_block<T>(A, B, 2, ld, f.gy, f.ty.tw);
  for (int j = threadIdx.x; j < f.NF; j += NT) {
    const C2<T> z0 = ((const C2<T>*)O)[pc<T>(j)];
    const C2<T> z1 = ((const C2<T>*)(O + ld))[pc<T>(j)];
    T v[4] = {z0.x, -z0.y, z1.x, -z1.y};
    store_cols<T, 4>(f.spec2 + (size_t)j * f.fpitch + c4, v);
  }
}

// F3: c2r along i of row j, written as the forcing of the run's interior
// row j (forc[i+1][j+1] = forc_p[j][i], src/forcing.h:196-200).
template <typename T>
__global__ void __launch_bounds__(NT) k_forc_rows(StepArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const ForcArgs<T>& f = a.fr;
  const int j = blockIdx.x;
  const int ld = padded_len<T>(f.gx.M);
  T* A = (T*)smem_raw;
  T* B = A + ld;
  const T* src = f.spec2 + (size_t)j * f.fpitch;
  for (int i = threadIdx.x; i < f.NF + 2; i += NT) A[pr<T>(i)] = src[i];
  __syncthreads();
  T* O = irfft_block<T>(A, B, 1, ld, f.gx, f.tx);
  T* dst = f.field + (size_t)j * a.pitch;
  for (int i = threadIdx.x; i < a.nx; i += NT) dst[i] = (i & 1) ? -O[pr<T>(i)] : O[pr<T>(i)];
}

template <typename T>
static void launch_forcing(const StepArgs<T>& a, cudaStream_t s) {
  const ForcArgs<T>& f = a.fr;
  if (!f.on) return;
  k_forc_modes<T><<<1, NT, 0, s>>>(a);
  k_forc_cols<T><<<f.col_blocks, NT, (size_t)4 * padded_len<T>(f.gy.M) * sizeof(T), s>>>(a);
  k_forc_rows<T><<<a.ny, NT, (size_t)2 * padded_len<T>(f.gx.M) * sizeof(T), s>>>(a);
}

#if QGW_KERNELS_PART == 1
// A new state's history: the three slabs of f (words: their 4-byte words) and
// the counters of the step.
static __global__ void __launch_bounds__(256) k_reset(DevState* st, unsigned int* fab, size_t words) {
  uint4* f4 = reinterpret_cast<uint4*>(fab);
  const size_t n4 = words / 4, t = (size_t)blockIdx.x * 256 + threadIdx.x;
  for (size_t i = t; i < n4; i += (size_t)gridDim.x * 256) f4[i] = make_uint4(0, 0, 0, 0);
  if (t < words - 4 * n4) fab[4 * n4 + t] = 0;
  if (t == 0) {
    st->maxbits = 0;
    st->done_blocks = 0;
    st->pending = 0;
    st->step_index = 0;
    st->forc_step = 0;
    st->nonfinite = 0;
    st->dev_error = 0;
  }
}
#endif
// Boundary copies: the reference layout (nl, ny+2, nx+2) in one contiguous
// device buffer (or the caller's host array) <-> the interior-only run
// layout, a row at a time.
// Four waves of blocks, so that the last one's rows even out: a stored q of
// 2048^2 x 6 from host memory 1.078 -> 1.055 ms, from the device 0.185 -> 0.168;
// q of 1024^2 x 10 into host memory 0.606 -> 0.597.
static inline int pack_blocks(int rows) { return std::min(rows, 152 * 32); }
template <typename T, bool SPLIT>
__global__ void __launch_bounds__(256) k_unpack(const double* __restrict__ full, T* __restrict__ dst,
                                                T* __restrict__ lo, int nx, int ny, int nl, int pitch) {
  for (int row = blockIdx.x; row < nl * ny; row += gridDim.x) {
    const int l = row / ny, j = row - l * ny;
    const double* src = full + ((size_t)l * (ny + 2) + (j + 1)) * (nx + 2) + 1;
    const size_t o0 = (size_t)row * pitch;
    for (int i = threadIdx.x; i < nx; i += 256) {
      const double v = src[i];
      if (SPLIT) {
        const float h = (float)v;
        dst[o0 + i] = (T)h;
        lo[o0 + i] = (T)(float)(v - (double)h);
      } else {
        dst[o0 + i] = (T)v;
      }
    }
  }
}
// The ring is what adjust_bc leaves after invert_pv (src/elliptic.h:152-153,
// src/domain.h:225-256,308-348): wrapped values in a periodic basin; at walls
// 0 (psi null) or c psi at the adjacent interior point, corners 0.  (On the
// host, its columns were one cache miss a point on memory the GPU had just
// written: 2 of 5 ms for the fields of 16 small runs.)
template <typename T>
__global__ void __launch_bounds__(256) k_pack(const T* __restrict__ src, const T* __restrict__ lo,
                                              const T* __restrict__ psi, double c, int periodic,
                                              double* __restrict__ full, int nx, int ny, int nl, int pitch) {
  for (int row = blockIdx.x; row < nl * (ny + 2); row += gridDim.x) {
    const int l = row / (ny + 2), jj = row - l * (ny + 2) - 1;
    // the interior row of the values (the adjacent one at walls)
    const bool iny = jj >= 0 && jj < ny;
    const int j = iny ? jj : periodic ? (jj < 0 ? ny - 1 : 0) : (jj < 0 ? 0 : ny - 1);
    const size_t o0 = ((size_t)l * ny + j) * pitch;
    double* dst = full + (size_t)row * (nx + 2);
    for (int i = threadIdx.x; i < nx + 2; i += 256) {
      const bool inx = i > 0 && i <= nx;
      const int g = inx ? i - 1 : periodic ? (i ? 0 : nx - 1) : (i ? nx - 1 : 0);
      const size_t o = o0 + g;
      double v = 0.0;
      if ((inx && iny) || periodic) v = (double)src[o] + (lo ? (double)lo[o] : 0.0);
      else if (psi && (inx || iny)) v = c * (double)psi[o];
      dst[i] = v;
    }
  }
}

// FP32c <-> FP64 conversions for the boundary copies
static __global__ void k_split_f64(const double* src, float* hi, float* lo, size_t n) {
  for (size_t w = blockIdx.x * (size_t)blockDim.x + threadIdx.x; w < n; w += (size_t)gridDim.x * blockDim.x) {
    const double x = src[w];
    const float h = (float)x;
    hi[w] = h;
    lo[w] = (float)(x - (double)h);
  }
}
static __global__ void k_join_f64(const float* hi, const float* lo, double* dst, size_t n) {
  for (size_t w = blockIdx.x * (size_t)blockDim.x + threadIdx.x; w < n; w += (size_t)gridDim.x * blockDim.x)
    dst[w] = (double)hi[w] + (lo ? (double)lo[w] : 0.0);
}

// FP64 diagnostics: per-block partial sums, then one block adds them up in a
// fixed order (bit-reproducible).
template <typename T>
__global__ void __launch_bounds__(NT) k_budget_partial(StepArgs<T> a, const double* wts, double* part) {
  __shared__ double red[4][NT];
  double ke = 0, en = 0, ens = 0, ww = 0;
  const size_t n = (size_t)a.nl * a.ny * a.nx;
  for (size_t w = blockIdx.x * (size_t)NT + threadIdx.x; w < n; w += (size_t)gridDim.x * NT) {
    const size_t row = w / a.nx;
    const int i = (int)(w - row * a.nx);
    const int l = (int)(row / a.ny);
    const int j = (int)(row - (size_t)l * a.ny);
    const size_t o = row * a.pitch + i;
    const double p = (double)a.psi[o];
    const double qv = (double)a.q[o] + (a.qlo ? (double)a.qlo[o] : 0.0);
    // closed basin: psi = 0 on the walls; periodic: the opposite side
    const double pe = (i + 1 < a.nx) ? (double)a.psi[o + 1] : (a.periodic ? (double)a.psi[o + 1 - a.nx] : 0.0);
    const double pn = (j + 1 < a.ny) ? (double)a.psi[o + a.pitch]
                                     : (a.periodic ? (double)a.psi[o - (size_t)(a.ny - 1) * a.pitch] : 0.0);
    const double u = (pe - p) / a.Delta, v = (pn - p) / a.Delta;
    const double wl = wts[l];
    ke += wl * 0.5 * (u * u + v * v);
    en -= wl * p * qv;
    ens += wl * qv * qv;
    if (l == 0 && a.wind) ww -= wl * p * (double)a.wind[j];
  }
  red[0][threadIdx.x] = ke; red[1][threadIdx.x] = en; red[2][threadIdx.x] = ens; red[3][threadIdx.x] = ww;
  __syncthreads();
  for (int s = NT / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s)
      for (int c = 0; c < 4; ++c) red[c][threadIdx.x] += red[c][threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x < 4) part[blockIdx.x * 4 + threadIdx.x] = red[threadIdx.x][0];
}

static __global__ void k_budget_final(const double* part, int nblk, double scale, double* out) {
  if (threadIdx.x < 4) {
    double s = 0;
    for (int b = 0; b < nblk; ++b) s += part[b * 4 + threadIdx.x];
    out[threadIdx.x] = s * scale;
  }
}

// ------------------------------------------------------------- launchers
// The dynamic shared-memory limit is a process-wide attribute of each kernel,
// shared by every run in the process; it is set to the device's opt-in
// maximum (never lowered) so that runs of different sizes can coexist.
[[maybe_unused]] static size_t rows_bytes(const StepArgs<double>& a) { return smem_rows_f64(a, std::max(a.RB1, a.RB3)); }
[[maybe_unused]] static size_t rows_bytes(const StepArgs<float>&) { return 0; }
// static shared memory of the row and column kernels, at most (with a margin
// in FP64: the sizes a run takes or refuses go by this)
template <typename T> constexpr size_t static_tot = sizeof(T) * GMAX * 32 + 64;
static_assert(sizeof(double) * tot_len<double, -1> <= static_tot<double>, "the chirp-z kernels' scratch");
template <typename T, bool COMP>
static cudaError_t set_attrs(const StepArgs<T>& a) {
  int dev = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return e;
  if (smem_rows<T, COMP>(a) + static_tot<T> > (size_t)optin || smem_cols<T, COMP>(a) + static_tot<T> > (size_t)optin ||
      smem_rows_inv<T, COMP>(a) + static_tot<T> > (size_t)optin || rhs_halo(a) > RHS_RMAX ||
      (sizeof(T) == 8 && rows_bytes(a) + static_tot<T> > (size_t)optin) ||
      smem_rhs<T>(a) + 1024 > (size_t)optin || smem_rhs_tiles<T>(a) + 1024 > (size_t)optin)
    return cudaErrorInvalidValue;
  const int lim = optin - (int)static_tot<T>;
  const void* columns[] = {
      (const void*)k_cols<T, COMP, false, CTD<T>, 0>,     (const void*)k_cols<T, COMP, false, CTD<T>, 512>,
      (const void*)k_cols<T, COMP, false, CTD<T> / 2, 0>, (const void*)k_cols<T, COMP, false, CTD<T> / 2, 512>,
      (const void*)k_cols<T, COMP, false, CTD<T> / 2, -1>, (const void*)k_cols<T, COMP, false, 1, -1>,
      (const void*)k_cols<T, COMP, true, CTD<T>, 0>,
      (const void*)k_cols<T, COMP, true, sizeof(T) == 8 ? 2 : CTD<T>, 0>};
  for (const void* f : columns)
    if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, lim))) return e;
  if constexpr (sizeof(T) == 8) {
    const void* rows[] = {(const void*)k_cols<T, COMP, false, CTD<T>, 1024>,
                          (const void*)k_cols<T, COMP, false, CTD<T> / 2, 1024>,
                          (const void*)k_rows_f64<false, 1024, false>, (const void*)k_rows_f64<false, 1024, true>,
                          (const void*)k_rows_f64<false, 0, false>,   (const void*)k_rows_f64<false, 0, true>,
                          (const void*)k_rows_f64<false, 512, false>, (const void*)k_rows_f64<false, 512, true>,
                          (const void*)k_rows_f64<false, -1, false>,  (const void*)k_rows_f64<false, -1, true>,
                          (const void*)k_rows_f64<true, 0, false>,    (const void*)k_rows_f64<true, 0, true>,
                          (const void*)k_modes<0, true>,              (const void*)k_modes<0, false>};
    for (const void* f : rows)
      if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, lim))) return e;
  } else {
    const void* rows[] = {(const void*)k_rows_fwd<T, COMP, false, 0>,   (const void*)k_rows_inv<T, COMP, false, 0>,
                          (const void*)k_rows_fwd<T, COMP, false, 512>, (const void*)k_rows_inv<T, COMP, false, 512>,
                          (const void*)k_rows_fwd<T, COMP, false, -1>,  (const void*)k_rows_inv<T, COMP, false, -1>,
                          (const void*)k_rows_fwd<T, COMP, true, 0>,    (const void*)k_rows_inv<T, COMP, true, 0>};
    for (const void* f : rows)
      if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, lim))) return e;
  }
  if ((e = cudaFuncSetAttribute(k_forc_cols<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim))) return e;
  if ((e = cudaFuncSetAttribute(k_forc_rows<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim))) return e;
  const int rl = optin - 1024;
  const void* rhs_kernels[] = {(const void*)k_rhs<T, COMP, 1, 16>, (const void*)k_rhs<T, COMP, 2, 16>,
                               (const void*)k_rhs<T, COMP, 3, 16>, (const void*)k_rhs<T, COMP, 4, 16>,
                               (const void*)k_rhs<T, COMP, 1, 32>, (const void*)k_rhs<T, COMP, 2, 32>,
                               (const void*)k_rhs<T, COMP, 3, 32>, (const void*)k_rhs<T, COMP, 4, 32>};
  for (const void* f : rhs_kernels)
    if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, rl)) != cudaSuccess) return e;
  return cudaSuccess;
}

// A step kernel's launch.  pdl: the kernel before it in the stream is one of
// a step too (or anything else: it then just completes first), and this one
// may be placed on the SMs before that has drained (grid_wait).  Kernels of
// small grids run 5-20 us, of which the launch gap was 2-3.
template <typename... P, typename... A>
static void launch(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, bool pdl, const A&... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = pdl ? 1 : 0;
  cudaLaunchKernelEx(&c, k, static_cast<P>(args)...);
}

// Threads that share a point in the projections of any number of layers, which
// read the layers again for every MODES_GO outputs: more of them where the
// points alone fill few blocks, as long as each has outputs and two blocks'
// constants fit an SM (or the blocks are fewer than the SMs).  Doubled up to 512
// blocks in FP64, up to one and a half per SM in fixed point, whose values each
// thread converts again.  Forward and inverse stage in ms, with one thread a
// point and as chosen: 64^2 x 128 2.24 and 0.40, 128^2 x 128 2.31 and
// 1.21, 256^2 x 64 1.26 and 1.11, 128^2 x 24 0.129 and 0.088, 64^2 x 17 0.093
// and 0.065; beyond the lines 384^2 x 24 0.517 with one and 0.523 with two,
// 256^2 x 17 0.136 and 0.141.
static inline int modes_any_split(const StepArgs<double>& a, size_t n) {
  const size_t few = (size_t)(a.modes_fx ? 228 : 512) * NT;
  int GY = 1;
  while (GY < 8 && GY * MODES_GO < a.nl && n * GY < few &&
         (modes_any_bytes(a.nl, 2 * GY) <= (size_t)110 * 1024 || 2 * GY * n <= (size_t)152 * NT))
    GY *= 2;
  return GY;
}

// FP64: a projection and the row transforms after it
template <bool FWD> static void launch_modes(const StepArgs<double>& a, int step_mode, bool pdl, cudaStream_t s) {
  const size_t n = (size_t)a.ny * (!FWD && a.periodic ? a.nx + 2 : a.nx);
  const dim3 grid((unsigned int)((n + NT - 1) / NT));
  switch (a.modes_fx ? a.nl : 0) {
#define QGW_MODES(N) \
  case N: launch(k_modes<N, FWD>, grid, dim3(NT), ModeShape<N>::bytes, s, pdl, a, step_mode); break;
    QGW_MODES(1) QGW_MODES(2) QGW_MODES(3) QGW_MODES(4) QGW_MODES(5) QGW_MODES(6) QGW_MODES(7) QGW_MODES(8)
    QGW_MODES(9) QGW_MODES(10) QGW_MODES(11) QGW_MODES(12) QGW_MODES(13) QGW_MODES(14) QGW_MODES(15) QGW_MODES(16)
#undef QGW_MODES
    default: {
      const int GY = modes_any_split(a, n), pts = NT / GY;
      launch(k_modes<0, FWD>, dim3((unsigned int)((n + pts - 1) / pts)), dim3(pts, GY), modes_any_bytes(a.nl, GY), s,
             pdl, a, step_mode);
      break;
    }
  }
}
template <bool INV> static void launch_rows(const StepArgs<double>& a, int step_mode, bool pdl, cudaStream_t s) {
  const int rows = INV ? a.RB3 : a.RB1;
  const size_t sm = smem_rows_f64(a, rows);
  const dim3 grid((a.nl * a.ny + rows - 1) / rows);
  if (a.periodic) launch(k_rows_f64<true, 0, INV>, grid, dim3(NT), sm, s, pdl, a, step_mode);
  else if (a.gx.blue) launch(k_rows_f64<false, -1, INV>, grid, dim3(NT), sm, s, pdl, a, step_mode);
  else if (a.gx.H == 512) launch(k_rows_f64<false, 512, INV>, grid, dim3(NT), sm, s, pdl, a, step_mode);
  else if (a.gx.H == 1024) launch(k_rows_f64<false, 1024, INV>, grid, dim3(NT), sm, s, pdl, a, step_mode);
  else launch(k_rows_f64<false, 0, INV>, grid, dim3(NT), sm, s, pdl, a, step_mode);
}

template <typename T, bool COMP>
static void launch_k1(const StepArgs<T>& a, int step_mode, bool pdl, cudaStream_t s) {
  if constexpr (sizeof(T) == 8) {
    launch_modes<true>(a, step_mode, pdl, s);
    launch_rows<false>(a, step_mode, pdl, s);
  } else {
    const size_t sm = smem_rows<T, COMP>(a);
    if (a.periodic) launch(k_rows_fwd<T, COMP, true, 0>, dim3(a.ny), dim3(NT), sm, s, pdl, a, step_mode);
    else if (a.gx.blue) launch(k_rows_fwd<T, COMP, false, -1>, dim3(a.ny), dim3(NT), sm, s, pdl, a, step_mode);
    else if (a.gx.H == 512) launch(k_rows_fwd<T, COMP, false, 512>, dim3(a.ny), dim3(NT), sm, s, pdl, a, step_mode);
    else launch(k_rows_fwd<T, COMP, false, 0>, dim3(a.ny), dim3(NT), sm, s, pdl, a, step_mode);
  }
}
template <typename T, bool COMP>
static void launch_k2(const StepArgs<T>& a, int step_mode, bool pdl, cudaStream_t s) {
  const int width = a.CT1 ? a.CT1 : col_width(a);
  const dim3 grid(a.periodic ? col_tiles(a) : (a.nx + width - 1) / width, a.nl);
  size_t sm = smem_cols<T, COMP>(a, width);
  if constexpr (sizeof(T) == 8) sm = sm / 2 * fx_bufs(a, a.gy);
  const bool wide = width == CTD<T>, h512 = a.gy.H == 512 && !a.gy.blue;
  if constexpr (sizeof(T) == 8) {
    if (a.periodic) {
      const int cc = per_cols(a);
      const dim3 tiles((a.gx.H + cc) / cc, a.nl);
      const size_t bytes = (size_t)2 * cc * row_len<T>(a.gy) * sizeof(T);
      if (cc == 4) launch(k_cols<T, COMP, true, 4, 0>, tiles, dim3(NT), bytes, s, pdl, a, step_mode);
      else launch(k_cols<T, COMP, true, 2, 0>, tiles, dim3(NT), bytes, s, pdl, a, step_mode);
      return;
    }
    if (a.gy.H == 1024 && !a.gy.blue) {
      if (wide) launch(k_cols<T, COMP, false, CTD<T>, 1024>, grid, dim3(NT), sm, s, pdl, a, step_mode);
      else launch(k_cols<T, COMP, false, CTD<T> / 2, 1024>, grid, dim3(NT), sm, s, pdl, a, step_mode);
      return;
    }
  }
  if (a.periodic) launch(k_cols<T, COMP, true, CTD<T>, 0>, grid, dim3(NT), sm, s, pdl, a, step_mode);
  else if (a.gy.blue && width == 1) launch(k_cols<T, COMP, false, 1, -1>, grid, dim3(NT), sm, s, pdl, a, step_mode);
  else if (a.gy.blue) launch(k_cols<T, COMP, false, CTD<T> / 2, -1>, grid, dim3(NT), sm, s, pdl, a, step_mode);
  else if (wide && h512) launch(k_cols<T, COMP, false, CTD<T>, 512>, grid, dim3(NT), sm, s, pdl, a, step_mode);
  else if (wide) launch(k_cols<T, COMP, false, CTD<T>, 0>, grid, dim3(NT), sm, s, pdl, a, step_mode);
  else if (h512) launch(k_cols<T, COMP, false, CTD<T> / 2, 512>, grid, dim3(NT), sm, s, pdl, a, step_mode);
  else launch(k_cols<T, COMP, false, CTD<T> / 2, 0>, grid, dim3(NT), sm, s, pdl, a, step_mode);
}
template <typename T, bool COMP>
static void launch_k3(const StepArgs<T>& a, int step_mode, bool pdl, cudaStream_t s) {
  if constexpr (sizeof(T) == 8) {
    launch_modes<false>(a, step_mode, pdl, s);
    launch_rows<true>(a, step_mode, pdl, s);
  } else {
    const size_t sm = smem_rows_inv<T, COMP>(a);
    // rows x layer groups: a row's groups read the same spectral rows, so
    // splitting them over blocks adds no traffic and evens out the SMs' loads
    const dim3 grid(a.ny, a.inv_split ? (a.nl + a.G3 - 1) / a.G3 : 1);
    if (a.periodic) launch(k_rows_inv<T, COMP, true, 0>, grid, dim3(NT), sm, s, pdl, a, step_mode);
    else if (a.gx.blue) launch(k_rows_inv<T, COMP, false, -1>, grid, dim3(NT), sm, s, pdl, a, step_mode);
    else if (a.gx.H == 512) launch(k_rows_inv<T, COMP, false, 512>, grid, dim3(NT), sm, s, pdl, a, step_mode);
    else launch(k_rows_inv<T, COMP, false, 0>, grid, dim3(NT), sm, s, pdl, a, step_mode);
  }
}
// tiles of the RHS kernel along x and y
template <typename T> static int rhs_ntx(const StepArgs<T>& a) { return (a.nx + TX - 1) / TX; }
template <typename T> static int rhs_nty(const StepArgs<T>& a) { return (a.ny + rhs_ty(a) - 1) / rhs_ty(a); }

template <typename T, bool COMP>
static void launch_rhs(const StepArgs<T>& a, bool pdl, cudaStream_t s) {
  const int ntx = rhs_ntx(a), nty = rhs_nty(a), ntiles = ntx * nty * a.nl;
  const int grid = (a.rhs_grid > 0 && a.rhs_grid < ntiles) ? a.rhs_grid : ntiles;
  // Tiles that stay in FP64 take several times as long as the others.  Placed
  // while the kernel before drains, all of a small grid's blocks crowd the SMs
  // that come free first and wait on their FP64 pipes: such a grid launches
  // plainly.  72^2 x 13 no-slip (195 tiles) a step of 99 -> 90 us, 192^2 x 3
  // with topography 95 -> 76, 384x240x3 120 -> 101; below 100 tiles (64^2 x 3:
  // 58 against 61) and above four blocks per SM (256^2 x 6: 89 against 92) the
  // overlap is worth more.
  if constexpr (sizeof(T) == 8)
    if ((a.cbc > 0 || a.has_topo) && ntiles >= 100 && ntiles < 608) pdl = false;
  const dim3 blk(32, 8);
  const size_t sm = smem_rhs_tiles(a);
  const bool t32 = rhs_ty(a) == 32;
  switch (rhs_halo(a)) {
    case 1:
      if (t32) launch(k_rhs<T, COMP, 1, 32>, grid, blk, sm, s, pdl, a, ntx, nty);
      else launch(k_rhs<T, COMP, 1, 16>, grid, blk, sm, s, pdl, a, ntx, nty);
      break;
    case 2:
      if (t32) launch(k_rhs<T, COMP, 2, 32>, grid, blk, sm, s, pdl, a, ntx, nty);
      else launch(k_rhs<T, COMP, 2, 16>, grid, blk, sm, s, pdl, a, ntx, nty);
      break;
    case 3:
      if (t32) launch(k_rhs<T, COMP, 3, 32>, grid, blk, sm, s, pdl, a, ntx, nty);
      else launch(k_rhs<T, COMP, 3, 16>, grid, blk, sm, s, pdl, a, ntx, nty);
      break;
    default:
      if (t32) launch(k_rhs<T, COMP, 4, 32>, grid, blk, sm, s, pdl, a, ntx, nty);
      else launch(k_rhs<T, COMP, 4, 16>, grid, blk, sm, s, pdl, a, ntx, nty);
      break;
  }
}

// Persistent grid of the RHS kernel: as many blocks as stay resident on the
// device at once (the occupancy of the run's halo and shared memory).
template <typename T, bool COMP>
static int rhs_grid(const StepArgs<T>& a) {
  int dev = 0, sms = 0, per = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 0;
  const size_t sm = smem_rhs_tiles(a);
  const int h = rhs_halo(a);
  const void* f = rhs_ty(a) == 32 ? (h == 1 ? (const void*)k_rhs<T, COMP, 1, 32> : h == 2 ? (const void*)k_rhs<T, COMP, 2, 32>
                                     : h == 3 ? (const void*)k_rhs<T, COMP, 3, 32> : (const void*)k_rhs<T, COMP, 4, 32>)
                                  : (h == 1 ? (const void*)k_rhs<T, COMP, 1, 16> : h == 2 ? (const void*)k_rhs<T, COMP, 2, 16>
                                     : h == 3 ? (const void*)k_rhs<T, COMP, 3, 16> : (const void*)k_rhs<T, COMP, 4, 16>);
  const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f, NT, sm);
  return (e == cudaSuccess && per > 0) ? per * sms : 0;
}

template <typename T, bool COMP>
static void launch_invert(const StepArgs<T>& a, int step_mode, bool pdl, cudaStream_t s) {
  launch_k1<T, COMP>(a, step_mode, pdl, s);
  launch_k2<T, COMP>(a, step_mode, pdl, s);
  launch_k3<T, COMP>(a, step_mode, pdl, s);
}

template <typename T, bool COMP>
static void launch_flush(const StepArgs<T>& a, DevState* host, cudaStream_t s) {
  const int blocks = std::min(a.nl * a.ny, 152 * 8);
  launch(k_flush<T, COMP>, dim3(blocks), dim3(NT), 0, s, true, a);
  launch(k_end, dim3(1), dim3(64), 0, s, true, a.state, host);
}

template <typename T, bool COMP>
static void launch_one(const StepArgs<T>& a, int which, cudaStream_t s) {
  if (which == 0) launch_k1<T, COMP>(a, 1, false, s);
  if (which == 1) launch_k2<T, COMP>(a, 1, false, s);
  if (which == 2) launch_k3<T, COMP>(a, 1, false, s);
  if (which == 3) launch_rhs<T, COMP>(a, false, s);
}

// ---- entry points used by api.cu (see kernels.h)
template <typename T>
static void budget_impl(const StepArgs<T>& a, const double* wts, double* part, int nblk, double scale, double* out,
                        cudaStream_t s) {
  k_budget_partial<T><<<nblk, NT, 0, s>>>(a, wts, part);
  k_budget_final<<<1, 32, 0, s>>>(part, nblk, scale, out);
}

#if QGW_KERNELS_PART == 1
void enqueue_begin(DevState* st, double t_out, double tend, cudaStream_t s) {
  launch(k_begin, dim3(1), dim3(1), 0, s, true, st, t_out, tend);
}

void enqueue_unpack_split(const double* full, float* hi, float* lo, int nx, int ny, int nl, int pitch,
                          cudaStream_t s) {
  k_unpack<float, true><<<pack_blocks(nl * ny), 256, 0, s>>>(full, hi, lo, nx, ny, nl, pitch);
}

void enqueue_pack_join(const float* hi, const float* lo, const float* psi, double c, int periodic, double* full, int nx,
                       int ny, int nl, int pitch, cudaStream_t s) {
  k_pack<float><<<pack_blocks(nl * (ny + 2)), 256, 0, s>>>(hi, lo, psi, c, periodic, full, nx, ny, nl, pitch);
}

int rhs_tile_x() { return TX; }

int rhs_box_width() { return TW; }

cudaError_t prepare_f64(const StepArgs<double>& a) { return set_attrs<double, false>(a); }

int rows_fit_f64(const StepArgs<double>& a, int want) {
  int dev = 0, optin = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
    return 1;
  while (want > 1 && smem_rows_f64(a, want) + static_tot<double> > (size_t)optin) --want;
  return want;
}

int rhs_grid_f64(const StepArgs<double>&) { return 0; }  // one block per tile

void enqueue_step_f64(const StepArgs<double>& a, cudaStream_t s) {
  launch_invert<double, false>(a, 1, true, s);
  launch_rhs<double, false>(a, true, s);
  launch_forcing<double>(a, s);
}

void enqueue_forcing_f64(const StepArgs<double>& a, cudaStream_t s) { launch_forcing<double>(a, s); }

void enqueue_invert_f64(const StepArgs<double>& a, bool pdl, cudaStream_t s) { launch_invert<double, false>(a, 0, pdl, s); }

void enqueue_flush_f64(const StepArgs<double>& a, DevState* host, cudaStream_t s) { launch_flush<double, false>(a, host, s); }

void enqueue_step_kernel_f64(const StepArgs<double>& a, int which, cudaStream_t s) { launch_one<double, false>(a, which, s); }

void enqueue_reset(DevState* st, void* fab, size_t bytes, cudaStream_t s) {
  const size_t blocks = (bytes / 16 + 255) / 256 + 1;
  k_reset<<<(int)std::min(blocks, (size_t)152 * 8), 256, 0, s>>>(st, (unsigned int*)fab, bytes / 4);
}
void enqueue_unpack_f64(const double* full, double* q, int nx, int ny, int nl, int pitch, cudaStream_t s) {
  k_unpack<double, false><<<pack_blocks(nl * ny), 256, 0, s>>>(full, q, nullptr, nx, ny, nl, pitch);
}

void enqueue_pack_f64(const double* src, const double* psi, double c, int periodic, double* full, int nx, int ny, int nl,
                      int pitch, cudaStream_t s) {
  k_pack<double><<<pack_blocks(nl * (ny + 2)), 256, 0, s>>>(src, nullptr, psi, c, periodic, full, nx, ny, nl, pitch);
}

void enqueue_split_f64(const double* src, float* hi, float* lo, size_t n, cudaStream_t s) {
  k_split_f64<<<1024, 256, 0, s>>>(src, hi, lo, n);
}

void enqueue_join_f64(const float* hi, const float* lo, double* dst, size_t n, cudaStream_t s) {
  k_join_f64<<<1024, 256, 0, s>>>(hi, lo, dst, n);
}

void enqueue_budget_f64(const StepArgs<double>& a, const double* w, double* part, int nblk, double scale, double* out,
                        cudaStream_t s) { budget_impl<double>(a, w, part, nblk, scale, out, s); }

int cols_per_tile_f64() { return ColsPer<double>::value; }

int rhs_tile_y_f64(const StepArgs<double>& a) { return rhs_ty(a); }

size_t smem_bytes_rows_f64(const StepArgs<double>& a) { return smem_rows<double, false>(a); }

size_t smem_bytes_cols_f64(const StepArgs<double>& a) { return smem_cols<double, false>(a); }

size_t smem_bytes_rhs_f64(const StepArgs<double>& a) { return smem_rhs_tiles<double>(a); }
#else
cudaError_t prepare_f32c(const StepArgs<float>& a) { return set_attrs<float, true>(a); }

int rhs_grid_f32c(const StepArgs<float>& a) { return rhs_grid<float, true>(a); }

void enqueue_step_f32c(const StepArgs<float>& a, cudaStream_t s) {
  launch_invert<float, true>(a, 1, true, s);
  launch_rhs<float, true>(a, true, s);
  launch_forcing<float>(a, s);
}

void enqueue_forcing_f32c(const StepArgs<float>& a, cudaStream_t s) { launch_forcing<float>(a, s); }

void enqueue_invert_f32c(const StepArgs<float>& a, bool pdl, cudaStream_t s) { launch_invert<float, true>(a, 0, pdl, s); }

void enqueue_flush_f32c(const StepArgs<float>& a, DevState* host, cudaStream_t s) { launch_flush<float, true>(a, host, s); }

void enqueue_step_kernel_f32c(const StepArgs<float>& a, int which, cudaStream_t s) { launch_one<float, true>(a, which, s); }

void enqueue_budget_f32c(const StepArgs<float>& a, const double* w, double* part, int nblk, double scale, double* out,
                         cudaStream_t s) { budget_impl<float>(a, w, part, nblk, scale, out, s); }

int cols_per_tile_f32c() { return ColsPer<float>::value; }

int rhs_tile_y_f32c(const StepArgs<float>& a) { return rhs_ty(a); }

size_t smem_bytes_rows_f32c(const StepArgs<float>& a) { return smem_rows<float, true>(a); }

size_t smem_bytes_cols_f32c(const StepArgs<float>& a) { return smem_cols<float, true>(a); }

size_t smem_bytes_rhs_f32c(const StepArgs<float>& a) { return smem_rhs_tiles<float>(a); }
#endif  // QGW_KERNELS_PART

}  // namespace qgw
