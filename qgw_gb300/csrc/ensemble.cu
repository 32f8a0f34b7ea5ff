// ensemble.cu -- batches of independent runs (uneven grids and layer
// counts) advanced together: one launch per step stage over all
// members, the four launches of a step captured once as a CUDA graph and
// replayed, and a project autotuner for the grid of each stage.
//
// Each member is a full qgw_run (own fields, own device scalars, own CFL
// counter); the batched kernels only change which block computes which
// member's work item, never the arithmetic, so a member's result is bitwise
// the same alone and in any batch.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <cstdlib>
#include <vector>

#include "../../include/qgw_gpu.h"
#include "kernels.h"
#include "qgw_device.cuh"
#include "run.h"
#include "ensemble_core.h"

struct qgw_ensemble {
  qgw::EnsembleCore core;  // owns its members
};

namespace {

int cuda_fail(cudaError_t e) {
  if (e == cudaSuccess) return QGW_OK;
  if (e == cudaErrorMemoryAllocation) return QGW_ERR_NOMEM;
  return QGW_ERR_CUDA;
}
#define CK(x)                                    \
  do {                                           \
    cudaError_t e_ = (x);                        \
    if (e_ != cudaSuccess) return cuda_fail(e_); \
  } while (0)

void drop_graph(qgw::EnsembleCore* e) {
  if (e->exec) cudaGraphExecDestroy(e->exec);
  if (e->graph) cudaGraphDestroy(e->graph);
  e->exec = nullptr;
  e->graph = nullptr;
}

int stage_occupancy(const qgw::EnsembleCore* e, int stage, size_t smem) {
  return e->precision == QGW_FP64 ? qgw::ens_blocks_per_sm_f64(stage, smem) : qgw::ens_blocks_per_sm_f32c(stage, smem);
}

// occupancy stage of the RHS kernel of halo radius r at the ensemble's tile
// height (3 + r for 16 rows, 7 + r for 32)
int rhs_stage(const qgw::EnsembleCore* e, int r) { return (e->sm.rhs_ty == 32 ? 7 : 3) + r; }

// persistent grid of each stage: bps blocks per SM, never more than can be
// resident at once (blocks beyond that would wait for a second wave); bps 0
// gives one block per work item
int stage_grid(const qgw::EnsembleCore* e, int total, int bps, int occ) {
  if (total <= 0) return 0;
  if (bps <= 0) return total;
  return std::max(1, std::min(total, e->nsm * std::min(bps, occ)));
}

void set_grids(qgw::EnsembleCore* e) {
  for (int s = 0; s < 3; ++s)
    e->grid[s] = std::max(1, stage_grid(e, e->total[s], e->bps[s], stage_occupancy(e, s, e->sm.bytes[s])));
  e->grid[3] = 0;
  for (int r = 1; r <= 4; ++r) {
    e->rhs_grid[r] = stage_grid(e, e->rhs_total[r], e->bps[3], stage_occupancy(e, rhs_stage(e, r), e->sm.rhs_bytes[r]));
    e->grid[3] += e->rhs_grid[r];
  }
}

// member table, per-stage work lists and shared-memory sizes
int build_tables(qgw::EnsembleCore* e) {
  const int n = (int)e->members.size();
  const int tx = qgw::rhs_tile_x();
  const size_t L = (size_t)n + 1;
  std::vector<int> lists(3 * L + 4 + 4 * (L + 4), 0);
  int* rows = lists.data();
  int* cols = rows + L;
  int* rhs = cols + L;
  int* tot = rhs + L;
  int* rr[5] = {nullptr, tot + 4, tot + 4 + (L + 4), tot + 4 + 2 * (L + 4), tot + 4 + 3 * (L + 4)};
  for (int i = 0; i < n; ++i) {
    const qgw_run* r = e->members[i];
    const int R = e->precision == QGW_FP64 ? qgw::rhs_halo_of_f64(r->a64) : qgw::rhs_halo_of_f32c(r->a32);
    const int ty = e->precision == QGW_FP64 ? qgw::rhs_tile_y_f64(r->a64) : qgw::rhs_tile_y_f32c(r->a32);
    const int tiles = ((r->nx + tx - 1) / tx) * ((r->ny + ty - 1) / ty) * r->nl;
    rows[i + 1] = rows[i] + r->ny;
    const int ctiles = e->precision == QGW_FP64 ? qgw::col_tiles_f64(r->a64) : qgw::col_tiles_f32c(r->a32);
    cols[i + 1] = cols[i] + ctiles * r->nl;
    rhs[i + 1] = rhs[i] + tiles;
    for (int h = 1; h <= 4; ++h) rr[h][i + 1] = rr[h][i] + (h == R ? tiles : 0);
  }
  tot[0] = rows[n];
  tot[1] = cols[n];
  tot[2] = rows[n];
  tot[3] = rhs[n];
  for (int s = 0; s < 4; ++s) e->total[s] = tot[s];
  for (int h = 1; h <= 4; ++h) {
    rr[h][L + 3] = rr[h][n];  // total[3] of the radius-h list
    e->rhs_total[h] = rr[h][n];
  }
  qgw::ens_core_free_tables(e);
  if (n == 0) return QGW_OK;
  CK(cudaMalloc(&e->d_lists, sizeof(int) * lists.size()));
  CK(cudaMemcpyAsync(e->d_lists, lists.data(), sizeof(int) * lists.size(), cudaMemcpyHostToDevice, e->stream));
  CK(cudaMalloc(&e->d_maxsteps, sizeof(int) * n));
  const int* d = e->d_lists;
  const int* drr[5] = {nullptr, d + (rr[1] - rows), d + (rr[2] - rows), d + (rr[3] - rows), d + (rr[4] - rows)};
  if (e->precision == QGW_FP64) {
    std::vector<qgw::StepArgs<double>> h(n);
    for (int i = 0; i < n; ++i) h[i] = e->members[i]->a64;
    CK(cudaMalloc(&e->d_members, sizeof(h[0]) * n));
    CK(cudaMemcpyAsync(e->d_members, h.data(), sizeof(h[0]) * n, cudaMemcpyHostToDevice, e->stream));
    e->sm = qgw::ens_smem_f64(h.data(), n);
    e->e64 = {(const qgw::StepArgs<double>*)e->d_members, d, d + L, d + 2 * L, d + 3 * L, n};
    for (int r = 1; r <= 4; ++r) e->r64[r] = {e->e64.members, d, d + L, drr[r], drr[r] + L, n};
  } else {
    std::vector<qgw::StepArgs<float>> h(n);
    for (int i = 0; i < n; ++i) h[i] = e->members[i]->a32;
    CK(cudaMalloc(&e->d_members, sizeof(h[0]) * n));
    CK(cudaMemcpyAsync(e->d_members, h.data(), sizeof(h[0]) * n, cudaMemcpyHostToDevice, e->stream));
    e->sm = qgw::ens_smem_f32c(h.data(), n);
    e->e32 = {(const qgw::StepArgs<float>*)e->d_members, d, d + L, d + 2 * L, d + 3 * L, n};
    for (int r = 1; r <= 4; ++r) e->r32[r] = {e->e32.members, d, d + L, drr[r], drr[r] + L, n};
  }
  set_grids(e);
  CK(cudaStreamSynchronize(e->stream));
  return QGW_OK;
}

void launch_step(qgw::EnsembleCore* e, int mask) {
  if (e->precision == QGW_FP64)
    qgw::ens_step_f64(e->e64, e->r64, e->sm, e->grid, e->rhs_grid, mask, e->periodic, e->stream);
  else qgw::ens_step_f32c(e->e32, e->r32, e->sm, e->grid, e->rhs_grid, mask, e->periodic, e->stream);
  // stochastic forcing: its own small launches per forced member, after the RHS
  if (mask & 8)
    for (qgw_run* r : e->members) {
      if (e->precision == QGW_FP64) {
        if (r->a64.fr.on) qgw::enqueue_forcing_f64(r->a64, e->stream);
      } else if (r->a32.fr.on) {
        qgw::enqueue_forcing_f32c(r->a32, e->stream);
      }
    }
}

int ensure_graph(qgw::EnsembleCore* e) {
  if (e->exec) return QGW_OK;
  CK(cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeThreadLocal));
  launch_step(e, 15);
  cudaGraph_t g = nullptr;
  CK(cudaStreamEndCapture(e->stream, &g));
  e->graph = g;
  CK(cudaGraphInstantiate(&e->exec, g, 0));
  return QGW_OK;
}

int read_states(qgw::EnsembleCore* e) {
  const int n = (int)e->members.size();
  e->h_states.resize(n);
  for (int i = 0; i < n; ++i)
    CK(cudaMemcpyAsync(&e->h_states[i], e->members[i]->d_state, sizeof(qgw::DevState), cudaMemcpyDeviceToHost,
                       e->stream));
  CK(cudaStreamSynchronize(e->stream));
  return QGW_OK;
}

}  // namespace

extern "C" {

int qgw_ensemble_create(int n, const qgw_params* params, int precision, qgw_ensemble** out) {
  if (!params || !out || n < 1) return QGW_ERR_PARAM;
  *out = nullptr;
  qgw_ensemble* ens = new qgw_ensemble();
  qgw::EnsembleCore* e = &ens->core;
  e->precision = precision;
  int dev = 0, rc = QGW_OK;
  auto fail = [&](int code) {
    qgw_ensemble_destroy(ens);
    return code;
  };
  if (cudaGetDevice(&dev) != cudaSuccess) return fail(QGW_ERR_CUDA);
  if (cudaDeviceGetAttribute(&e->nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return fail(QGW_ERR_CUDA);
  if (cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking) != cudaSuccess) return fail(QGW_ERR_CUDA);
  // one boundary kind per ensemble: the row and column kernels of a launch
  // use either the DST-I (closed basin) or the FFT (periodic)
  e->periodic = params[0].bc_fac == -1;
  for (int i = 0; i < n; ++i)
    if ((params[i].bc_fac == -1) != (e->periodic != 0)) return fail(QGW_ERR_UNSUPPORTED);
  for (int i = 0; i < n; ++i) {
    qgw_run* r = nullptr;
    if ((rc = qgw_create(&params[i], nullptr, nullptr, nullptr, nullptr, precision, &r))) return fail(rc);
    e->members.push_back(r);
  }
  if ((rc = qgw::ens_core_build(e))) return fail(rc);
  *out = ens;
  return QGW_OK;
}

void qgw_ensemble_destroy(qgw_ensemble* ens) {
  if (!ens) return;
  qgw::EnsembleCore* e = &ens->core;
  if (e->stream) cudaStreamSynchronize(e->stream);
  qgw::ens_core_free_tables(e);
  for (qgw_run* r : e->members) qgw_destroy(r);
  if (e->stream) cudaStreamDestroy(e->stream);
  delete ens;
}

int qgw_ensemble_size(qgw_ensemble* ens) { return ens ? (int)ens->core.members.size() : 0; }

qgw_run* qgw_ensemble_member(qgw_ensemble* ens, int i) {
  if (!ens || i < 0 || i >= (int)ens->core.members.size()) return nullptr;
  cudaStreamSynchronize(ens->core.stream);
  return ens->core.members[i];
}

}  // extern "C"

namespace qgw {

void ens_core_free_tables(EnsembleCore* e) {
  drop_graph(e);
  if (e->d_members) cudaFree(e->d_members);
  if (e->d_lists) cudaFree(e->d_lists);
  if (e->d_maxsteps) cudaFree(e->d_maxsteps);
  e->d_members = nullptr;
  e->d_lists = nullptr;
  e->d_maxsteps = nullptr;
}

// The members' RHS tile height in FP32c, unless a call chose one
// (rhs_rows_set): 32 rows where there are 16-row tiles for more than one wave
// of five blocks per SM.  The batched kernel holds one tile a block, so the
// taller tile's smaller halo costs no residency (the single run's ring of two
// tiles does lose blocks at radius 3): 16 members of 64^2 to 512^2, three
// draws, 480, 452 and 583 -> 444, 418 and 542 us a step (runs of one side
// within 0.3).  A single wave waits for its longest block: 8 members of 64^2 x
// 5 (320 tiles) 83.3 us in 32 rows, 81.4 in 16, one of 256^2 x 5 (640) 55.1
// and 53.0; 16 of 128^2 x 2 (1024) 108 and 111.  QGW_RHS_TILE_ROWS overrides.
static int default_rhs_rows(EnsembleCore* e) {
  if (e->precision == QGW_FP64 || e->rhs_rows_set || std::getenv("QGW_RHS_TILE_ROWS")) return QGW_OK;
  long long tiles = 0;
  for (const qgw_run* r : e->members)
    tiles += (long long)((r->nx + rhs_tile_x() - 1) / rhs_tile_x()) * ((r->ny + 15) / 16) * r->nl;
  qgw_shape want{};
  want.rhs_tile_rows = tiles > 5 * e->nsm ? 32 : 16;
  for (qgw_run* r : e->members) {
    qgw_shape sh{};
    qgw_get_shape(r, &sh);
    if (sh.rhs_tile_rows == want.rhs_tile_rows) continue;
    const int rc = qgw_set_shape(r, &want);
    if (rc && rc != QGW_ERR_PARAM) return rc;  // refused: it keeps 16
  }
  return QGW_OK;
}

// The batched kernels take the column-tile width and the RHS tile height
// as template arguments, one for all members: where members differ (a run
// whose long columns forced the narrower tile, a member set alone), every
// member takes the narrower width and, if their heights differ, 16 rows.
// No shape changes a result.
static int uniform_shape(EnsembleCore* e) {
  if (e->members.empty()) return QGW_OK;
  qgw_shape first{};
  for (qgw_run* r : e->members) r->a64.CT1 = r->a32.CT1 = 0;  // (a single run's choice)
  qgw_get_shape(e->members[0], &first);
  int ct = first.col_tile, ty = first.rhs_tile_rows;
  bool mixed = false;
  for (qgw_run* r : e->members) {
    qgw_shape sh{};
    qgw_get_shape(r, &sh);
    if (sh.col_tile != ct || sh.rhs_tile_rows != ty) mixed = true;
    ct = std::min(ct, sh.col_tile);
    if (sh.rhs_tile_rows != ty) ty = 16;
  }
  if (!mixed) return QGW_OK;
  qgw_shape want{};
  want.col_tile = ct;
  want.rhs_tile_rows = ty;
  for (qgw_run* r : e->members) {
    const int rc = qgw_set_shape(r, &want);
    if (rc) return rc;
  }
  return QGW_OK;
}

int ens_core_build(EnsembleCore* e) {
  const cudaError_t pe = e->precision == QGW_FP64 ? ens_prepare_f64() : ens_prepare_f32c();
  if (pe != cudaSuccess) return cuda_fail(pe);
  // the batched kernels hold the half-length transforms only: a member whose
  // grid needs the chirp-z form runs alone
  for (qgw_run* r : e->members) {
    const bool blue = e->precision == QGW_FP64 ? (r->a64.gx.blue || r->a64.gy.blue) : (r->a32.gx.blue || r->a32.gy.blue);
    if (blue) return QGW_ERR_UNSUPPORTED;
  }
  int rc = default_rhs_rows(e);
  if (rc || (rc = uniform_shape(e))) return rc;
  return build_tables(e);
}

int ens_core_step(EnsembleCore* e, int nsteps, const int* max_steps, bool use_graph) {
  const int n = (int)e->members.size();
  if (n == 0) return QGW_OK;
  for (qgw_run* r : e->members) {
    if (!r->has_q) return QGW_ERR_STATE;
    if (r->p.dt_forc_period != 0 && (r->precision == QGW_FP64 ? r->a64.nrec : r->a32.nrec) == 0)
      return QGW_ERR_STATE;  // 4-D forcing records not set
  }
  for (qgw_run* r : e->members) CK(cudaStreamSynchronize(r->stream));
  std::vector<int> ms(n, 0);
  if (max_steps) std::memcpy(ms.data(), max_steps, sizeof(int) * n);
  CK(cudaMemcpyAsync(e->d_maxsteps, ms.data(), sizeof(int) * n, cudaMemcpyHostToDevice, e->stream));
  if (e->precision == QGW_FP64) ens_begin_f64(e->e64, e->d_maxsteps, e->stream);
  else ens_begin_f32c(e->e32, e->d_maxsteps, e->stream);
  int rc;
  if (use_graph && (rc = ensure_graph(e))) return rc;
  const int chunk = 256;
  for (int done = 0; done < nsteps;) {
    const int k = std::min(chunk, nsteps - done);
    for (int s = 0; s < k; ++s) {
      if (use_graph) CK(cudaGraphLaunch(e->exec, e->stream));
      else launch_step(e, 15);
    }
    done += k;
    if (done < nsteps) {
      if ((rc = read_states(e))) return rc;
      bool any = false;
      for (const auto& st : e->h_states) any = any || st.active;
      if (!any) break;
    }
  }
  const int fgrid = std::max(1, std::min(e->total[0], e->nsm * 4));
  if (e->precision == QGW_FP64) ens_flush_f64(e->e64, fgrid, e->stream);
  else ens_flush_f32c(e->e32, fgrid, e->stream);
  CK(cudaGetLastError());
  return QGW_OK;
}

int ens_core_finish(EnsembleCore* e) { return read_states(e); }

}  // namespace qgw

extern "C" {

int qgw_ensemble_step(qgw_ensemble* ens, int nsteps, const int* max_steps, int use_graph, qgw_step_info* infos) {
  if (!ens || nsteps < 0) return QGW_ERR_PARAM;
  qgw::EnsembleCore* e = &ens->core;
  const int n = (int)e->members.size();
  int rc = qgw::ens_core_step(e, nsteps, max_steps, use_graph != 0);
  if (rc) return rc;
  if ((rc = qgw::ens_core_finish(e))) return rc;
  bool bad = false, timeout = false;
  for (int i = 0; i < n; ++i) {
    const qgw::DevState& s = e->h_states[i];
    bad = bad || s.nonfinite;
    timeout = timeout || s.dev_error;
    if (infos) {
      infos[i].time.t = s.t;
      infos[i].time.dt = s.dt;
      infos[i].time.dt0 = s.dt0;
      infos[i].time.dt1 = s.dt1;
      infos[i].time.DT_max = s.DT_max;
      infos[i].steps_taken = s.steps_taken;
      infos[i].stop_reason = s.stop_reason;
      infos[i].nonfinite = s.nonfinite;
    }
  }
  if (timeout) return QGW_ERR_TIMEOUT;  // a bounded device wait ran out
  return bad ? QGW_ERR_NAN : QGW_OK;
}

// A member's shape in the batched kernels, whose FP64 row kernels take rows of
// one grid row (G1, G3) where a single run's take rows of any layer.
static void member_shape(qgw_run* r, qgw_shape* sh) {
  qgw_get_shape(r, sh);
  if (r->precision != QGW_FP64) return;
  sh->row_group_fwd = r->a64.G1;
  sh->row_group_inv = r->a64.G3;
}

// The same work-tile shape for every member (qgw_set_shape), then the
// member table rebuilt; a member that refuses the shape leaves every member
// at its previous one.
static int ensemble_set_shape(qgw::EnsembleCore* e, const qgw_shape& sh) {
  const int n = (int)e->members.size();
  std::vector<qgw::StepArgs<double>> a64(n);
  std::vector<qgw::StepArgs<float>> a32(n);
  for (int i = 0; i < n; ++i) {
    a64[i] = e->members[i]->a64;
    a32[i] = e->members[i]->a32;
  }
  for (int i = 0; i < n; ++i) {
    const int rc = qgw_set_shape(e->members[i], &sh);
    if (rc) {
      for (int j = 0; j < i; ++j) {
        e->members[j]->a64 = a64[j];
        e->members[j]->a32 = a32[j];
      }
      return rc;
    }
  }
  if (sh.rhs_tile_rows) e->rhs_rows_set = true;
  return qgw::ens_core_build(e);
}

// Autotuner, coordinate descent timed over `trial_steps` whole steps per
// candidate (each choice measured in the context of the others: caches,
// the member states the step leaves behind): first the work-tile shape of
// every member -- RHS tile height, column-tile width, layers per block of the
// forward and of the inverse row kernels -- then the grid of
// each stage (blocks per SM).  Runs on the current state and then restores
// the members' time scalars; the trial steps advance q, so callers re-set
// q before the time loop.  best_ms[4] (optional) receives the step time
// after each stage's grid choice.
int qgw_ensemble_tune(qgw_ensemble* ens, int trial_steps, float* best_ms) {
  if (!ens || trial_steps < 1) return QGW_ERR_PARAM;
  qgw::EnsembleCore* e = &ens->core;
  for (qgw_run* r : e->members)
    if (!r->has_q) return QGW_ERR_STATE;
  const int n = (int)e->members.size();
  std::vector<qgw_time> saved(n);
  for (int i = 0; i < n; ++i) qgw_get_time(e->members[i], &saved[i]);
  std::vector<int> ms(n, 0);
  CK(cudaMemcpyAsync(e->d_maxsteps, ms.data(), sizeof(int) * n, cudaMemcpyHostToDevice, e->stream));
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  drop_graph(e);
  // mean step time of the current configuration
  auto trial = [&](float* out) -> int {
    if (e->precision == QGW_FP64) qgw::ens_begin_f64(e->e64, e->d_maxsteps, e->stream);
    else qgw::ens_begin_f32c(e->e32, e->d_maxsteps, e->stream);
    launch_step(e, 15);  // warm-up
    CK(cudaEventRecord(e0, e->stream));
    for (int t = 0; t < trial_steps; ++t) launch_step(e, 15);
    CK(cudaEventRecord(e1, e->stream));
    CK(cudaEventSynchronize(e1));
    float msr = 0;
    CK(cudaEventElapsedTime(&msr, e0, e1));
    *out = msr / trial_steps;
    return QGW_OK;
  };
  int rc;
  {
    const int ctd = e->precision == QGW_FP64 ? 4 : 8;
    const std::vector<int> cand[4] = {{16, 32}, {ctd, ctd / 2}, {2, 4, 8, 16}, {2, 3, 4, 5}};
    qgw_shape cur{};
    member_shape(e->members[0], &cur);
    int* field[4] = {&cur.rhs_tile_rows, &cur.col_tile, &cur.row_group_fwd, &cur.row_group_inv};
    for (int f = 0; f < 4; ++f) {
      float best = 1e30f;
      int best_v = *field[f];
      for (int v : cand[f]) {
        qgw_shape sh{};
        int* sf[4] = {&sh.rhs_tile_rows, &sh.col_tile, &sh.row_group_fwd, &sh.row_group_inv};
        *sf[f] = v;
        if (ensemble_set_shape(e, sh) != QGW_OK) continue;  // e.g. beyond the shared memory
        float msr;
        if ((rc = trial(&msr))) return rc;
        if (msr < best) { best = msr; best_v = v; }
      }
      qgw_shape sh{};
      int* sf[4] = {&sh.rhs_tile_rows, &sh.col_tile, &sh.row_group_fwd, &sh.row_group_inv};
      *sf[f] = best_v;
      if ((rc = ensemble_set_shape(e, sh))) return rc;
      *field[f] = best_v;
    }
    drop_graph(e);
  }
  const int cands[] = {0, 1, 2, 3, 4, 5, 6, 8};  // 0: one block per work item
  for (int s = 0; s < 4; ++s) {
    float best = 1e30f;
    int best_b = e->bps[s];
    int occ = 1;
    if (s < 3) occ = stage_occupancy(e, s, e->sm.bytes[s]);
    else
      for (int r = 1; r <= 4; ++r)
        if (e->rhs_total[r] > 0) occ = std::max(occ, stage_occupancy(e, rhs_stage(e, r), e->sm.rhs_bytes[r]));
    for (int b : cands) {
      if (b > occ) break;  // same grid as the resident maximum
      e->bps[s] = b;
      set_grids(e);
      float msr;
      if ((rc = trial(&msr))) return rc;
      if (msr < best) { best = msr; best_b = b; }
    }
    e->bps[s] = best_b;
    if (best_ms) best_ms[s] = best;
  }
  set_grids(e);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  // apply the last pending AB3 update of the trial steps
  const int fgrid = std::max(1, std::min(e->total[0], e->nsm * 4));
  if (e->precision == QGW_FP64) qgw::ens_flush_f64(e->e64, fgrid, e->stream);
  else qgw::ens_flush_f32c(e->e32, fgrid, e->stream);
  CK(cudaGetLastError());
  for (int i = 0; i < n; ++i) {
    qgw_run* r = e->members[i];
    qgw_set_time(r, &saved[i]);
  }
  return QGW_OK;
}

int qgw_ensemble_set_q(qgw_ensemble* ens, int i, const double* q) {
  qgw::EnsembleCore* e = ens ? &ens->core : nullptr;
  if (!e || i < 0 || i >= (int)e->members.size()) return QGW_ERR_PARAM;
  CK(cudaStreamSynchronize(e->stream));
  return qgw_set_q(e->members[i], q);
}

int qgw_ensemble_set_time(qgw_ensemble* ens, int i, const qgw_time* tm) {
  qgw::EnsembleCore* e = ens ? &ens->core : nullptr;
  if (!e || i < 0 || i >= (int)e->members.size()) return QGW_ERR_PARAM;
  CK(cudaStreamSynchronize(e->stream));
  return qgw_set_time(e->members[i], tm);
}

int qgw_ensemble_get(qgw_ensemble* ens, int i, double* psi, double* q) {
  qgw::EnsembleCore* e = ens ? &ens->core : nullptr;
  if (!e || i < 0 || i >= (int)e->members.size()) return QGW_ERR_PARAM;
  CK(cudaStreamSynchronize(e->stream));
  return qgw_get(e->members[i], psi, q);
}

int qgw_ensemble_set_forcing_records(qgw_ensemble* ens, int i, const double* rec, int nrec) {
  qgw::EnsembleCore* e = ens ? &ens->core : nullptr;
  if (!e || i < 0 || i >= (int)e->members.size()) return QGW_ERR_PARAM;
  CK(cudaStreamSynchronize(e->stream));
  const int rc = qgw_set_forcing_records(e->members[i], rec, nrec);
  return rc ? rc : qgw::ens_core_build(e);  // the member table holds the record pointers
}

int qgw_ensemble_set_shape(qgw_ensemble* ens, const qgw_shape* sh) {
  qgw::EnsembleCore* e = ens ? &ens->core : nullptr;
  if (!e || !sh) return QGW_ERR_PARAM;
  CK(cudaStreamSynchronize(e->stream));
  return ensemble_set_shape(e, *sh);
}

int qgw_ensemble_shape(qgw_ensemble* ens, int i, qgw_shape* sh) {
  qgw::EnsembleCore* e = ens ? &ens->core : nullptr;
  if (!e || !sh || i < 0 || i >= (int)e->members.size()) return QGW_ERR_PARAM;
  member_shape(e->members[i], sh);
  return QGW_OK;
}

int qgw_ensemble_grids(qgw_ensemble* ens, int* bps4) {
  qgw::EnsembleCore* e = ens ? &ens->core : nullptr;
  if (!e || !bps4) return QGW_ERR_PARAM;
  for (int s = 0; s < 4; ++s) bps4[s] = e->bps[s];
  return QGW_OK;
}

}  // extern "C"
