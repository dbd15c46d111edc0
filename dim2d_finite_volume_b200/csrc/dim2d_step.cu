// dim2d_step.cu -- one RK3-TVD time step on the device
// (td_integrator_class.f:103-161 with rk3tvd_steps_module.f:52-490).
//
// Buffers: A holds u^n.  Stage 1 writes B = A + dt L(A); stage 2 writes
// C = 3/4 A + 1/4 (B + dt L(B)); stage 3 writes B = 1/3 A + 2/3 (C + dt L(C));
// then A and B swap.  u^n stays intact in A until the last boundary pass,
// which the wall operator reads as nodes_tmp (bc_operators_wall_xy_class.f).
// A stage launch sets the ghost cells of its output itself (stage()).
#include <utility>

#include "dim2d_internal.h"

using namespace dim2d;

StageArgs make_stage_args(const dim2d_handle* h, const double* uin, double* uout, double dt,
                          int st) {
  StageArgs a{};
  a.uin = uin;
  a.u0 = h->A;
  a.uout = uout;
  a.f = h->f;
  a.dx = h->dx;
  a.dy = h->dy;
  a.rdx = h->rdx;
  a.rdy = h->rdy;
  a.dt = dt;
  a.stage = st;
  a.b = st == 2 ? 0.75 : (st == 3 ? 1.0 / 3.0 : 0.0);  // rk3tvd_steps_module.f:225,444
  a.periodic = h->periodic;
  a.wall_s = h->south_wall;
  a.variant = h->variant;
  a.open = h->open_mask;
  a.mixed = h->precision == DIM2D_MIXED;
  a.xmap0 = h->xmap0;
  // every other launch of a run of steps (A and B change places each step)
  a.reverse = (st & 1) ^ (h->A < h->B);
  a.mirror = h->mirror_sides;
  a.wall_runs = h->south_wall ? wall_run_count(h->f, h->open_mask) : 0;
  a.status = h->status;
  if (h->south_wall) a.wc = wall_coef(h->wall, h->k, h->dx, h->dy);
  a.wall = h->wall;
  a.k = h->k;
  a.c = strip_coef_of(h->k, h->rdx, h->rdy);
  a.cf = strip_coef_f32(a.c);
  return a;
}

static NodeBcArgs make_node_args(const dim2d_handle* h, const double* utmp, double* u) {
  NodeBcArgs a{};
  a.utmp = utmp;
  a.u = u;
  a.f = h->f;
  a.dx = h->dx;
  a.dy = h->dy;
  a.rdx = h->rdx;
  a.rdy = h->rdy;
  a.xmap0 = h->xmap0;
  a.south_wall = h->south_wall;
  a.corners_y = h->corners_y;
  a.open_w = h->open_w;
  a.open_e = h->open_e;
  a.open_n = h->open_n;
  a.status = h->status;
  a.wall = h->wall;
  a.k = h->k;
  return a;
}

int apply_bc_on_nodes(dim2d_handle* h, const double* nodes_tmp, double* nodes) {
  cudaError_t e = cudaSuccess;
  if (h->periodic) {
    e = launch_periodic_ghosts(nodes, h->f, h->stream);
    h->launches++;
  } else if (h->open_all) {
    return DIM2D_OK;  // no section of node type
  } else {
    e = launch_node_bc(make_node_args(h, nodes_tmp, nodes), h->stream);
    h->launches++;
  }
  if (e != cudaSuccess) return cuda_error(e, "apply_bc_on_nodes");
  return DIM2D_OK;
}

void prof_begin(dim2d_handle* h) {
  if (!h->prof) return;
  if (h->prof_used + 2 > h->prof_ev.size()) {
    for (int i = 0; i < 64; i++) {
      cudaEvent_t ev;
      if (cudaEventCreate(&ev) != cudaSuccess) {
        h->prof = false;
        return;
      }
      h->prof_ev.push_back(ev);
    }
  }
  cudaEventRecord(h->prof_ev[h->prof_used], h->stream);
}

void prof_end(dim2d_handle* h) {
  if (!h->prof) return;
  cudaEventRecord(h->prof_ev[h->prof_used + 1], h->stream);
  h->prof_used += 2;
}

// Read the wall status word (synchronising).  Non-zero = a wall ghost cell
// had no bracketed / converged root, where the reference stops.
int check_status(dim2d_handle* h) {
  if (h->pplan) {  // a persistent launch that stopped at a wait that ran out
    int rc = persist_error(*h->pplan);
    if (rc) return rc;
  }
  if (!h->south_wall || !h->status) return DIM2D_OK;
  unsigned int st = 0;
  cudaError_t e = cudaMemcpyAsync(&st, h->status, sizeof st, cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->stream);
  if (e != cudaSuccess) return cuda_error(e, "status");
  if (st)
    return set_error(DIM2D_ERR_WALL_ROOT,
                     "wall ghost cell: %s (status 0x%x)",
                     (st & 1u) ? "root not bracketed" : "Ridders' method did not converge", st);
  return DIM2D_OK;
}

cudaError_t launch_stage_work(dim2d_handle* h, const StageArgs& a, int mode) {
  // Callers count two kernels per stage in short runs of an untuned hedstrom_xy
  // field (dim2d_launch_count): there the corner cells follow in a launch of their
  // own.  Runs of eight steps, which are for speed, take one (rk3_steps).
  const bool corners_apart = a.open == OPEN_ALL && a.variant == 0 && h->corners_apart;
  StageArgs first = a;
  if (corners_apart) first.open &= ~OPEN_CORNERS;
  prof_begin(h);
  cudaError_t e =
      mode == 0 ? launch_time_dev(first, h->stream) : launch_interior_stage(first, h->stream);
  prof_end(h);
  h->launches++;
  if (e != cudaSuccess || !a.open) return e;
  if (corners_apart) {
    StageArgs corners = a;
    corners.open = OPEN_CORNERS;
    e = launch_open_runs(corners, mode, h->stream);
    h->launches++;
  } else if (!stage_fuses_open(a)) {
    e = launch_open_ghosts(a, h->stream);
    h->launches++;
  }
  return e;
}

static int stage(dim2d_handle* h, int st, const double* uin, double* uout, double dt) {
  // The stage launch leaves the ghost cells of its output set: periodic and
  // mirror images by the strips, open sections integrated like the interior
  // (x/y_borders widened, field_abstract_class.f:244-270), wall columns by
  // their runs.
  cudaError_t e = launch_stage_work(h, make_stage_args(h, uin, uout, dt, st), 1);
  return e == cudaSuccess ? DIM2D_OK : cuda_error(e, "rk3 stage");
}

int rk3_step(dim2d_handle* h, double dt) {
  int rc = stage(h, 1, h->A, h->B, dt);
  if (!rc) rc = stage(h, 2, h->B, h->C, dt);
  if (!rc) rc = stage(h, 3, h->C, h->B, dt);
  if (rc) return rc;
  std::swap(h->A, h->B);
  h->t += dt;  // field_class.f:70
  return DIM2D_OK;
}

cudaError_t wait_copy_if(dim2d_handle* h, const double* target) {
  if (!h->copy_pending || target != h->copy_src) return cudaSuccess;
  h->copy_pending = false;
  return cudaStreamWaitEvent(h->stream, h->copy_done, 0);
}

void drop_graphs(dim2d_handle* h) {
  for (auto& size : h->graph)
    for (StepGraph& g : size) {
      if (g.exec) cudaGraphExecDestroy(g.exec);
      g = StepGraph();
    }
}

// Capture `steps` RK3 steps into sg.  The capture runs
// rk3_step's host side (A/B swap, time += dt) without executing anything; it
// is rolled back, and the caller applies it per launch (replayed).  No
// kernel reads the field time, so one graph serves every time level.
static int capture_steps(dim2d_handle* h, double dt, StepGraph& sg, int steps) {
  if (sg.exec) cudaGraphExecDestroy(sg.exec);
  sg = StepGraph();
  double* const A0 = h->A;
  double* const B0 = h->B;
  const double t0 = h->t;
  const long long n0 = h->launches;
  cudaError_t e = cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeRelaxed);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return DIM2D_ERR_UNSUPPORTED;  // e.g. the legacy default stream
  }
  int rc = DIM2D_OK;
  for (int s = 0; s < steps && !rc; s++) rc = rk3_step(h, dt);
  cudaGraph_t g = nullptr;
  e = cudaStreamEndCapture(h->stream, &g);
  sg.launches = h->launches - n0;
  h->launches = n0;
  h->A = A0;
  h->B = B0;
  h->t = t0;
  cudaGraphExec_t x = nullptr;
  if (!rc && e == cudaSuccess && g) e = cudaGraphInstantiate(&x, g, 0);
  if (g) cudaGraphDestroy(g);
  if (rc || e != cudaSuccess || !x) {
    cudaGetLastError();
    return rc ? rc : DIM2D_ERR_UNSUPPORTED;
  }
  sg.exec = x;
  sg.A = A0;
  return DIM2D_OK;
}

// Stage-kernel variant 6: nsteps steps as one launch of the persistent
// kernel (dim2d_persist.cu) over this field alone -- stages pipelined band
// by band, no stage boundary across the field.  The tables are built on
// first use for this dt and the field's buffers, and rebuilt when either
// changes; dt_scale 0 makes the autotuner's dry step (stage buffers only,
// no swap, no time advance).
int persist_steps(dim2d_handle* h, double dt, int nsteps, double dt_scale) {
  if (nsteps <= 0) return DIM2D_OK;
  // the launch writes both buffers of the pair: pending copies land first
  if (h->copy_pending) {
    cudaError_t ew = cudaStreamWaitEvent(h->stream, h->copy_done, 0);
    if (ew != cudaSuccess) return cuda_error(ew, "step");
    h->copy_pending = false;
  }
  // a dry step keeps whatever dt the tables hold (its stages use dt * 0)
  const double pdt = dt_scale == 0.0 ? (h->pplan && h->pdt >= 0.0 ? h->pdt : 0.0) : dt;
  bool rebuild = !h->pplan || !h->pplan->valid || h->pdt != pdt;
  int step0 = 0;
  if (!rebuild) {
    // the tables hold the buffers as built; A/B swap with every step
    const PDomain& d0 = h->pdom0;
    if (h->A == d0.buf[0] && h->B == d0.buf[1] && h->C == d0.buf[2]) step0 = 0;
    else if (h->A == d0.buf[1] && h->B == d0.buf[0] && h->C == d0.buf[2]) step0 = 1;
    else rebuild = true;
  }
  if (rebuild) {
    if (!h->pplan) h->pplan = new PersistPlan();
    std::vector<dim2d_handle*> hs{h};
    std::vector<double> dts{pdt};
    int rc = persist_build(*h->pplan, hs, dts, 16, h->stream);
    if (rc) return rc;
    h->pdt = pdt;
    h->pdom0.buf[0] = h->A;
    h->pdom0.buf[1] = h->B;
    h->pdom0.buf[2] = h->C;
    step0 = 0;
  }
  prof_begin(h);
  cudaError_t e = persist_launch(*h->pplan, nsteps, step0, dt_scale, 2000000000ull, -1, h->stream);
  prof_end(h);
  if (e != cudaSuccess) return cuda_error(e, "persistent step");
  h->launches++;
  if (dt_scale != 0.0) {
    if (nsteps & 1) std::swap(h->A, h->B);
    for (int s = 0; s < nsteps; s++) h->t += dt;  // field_class.f:70, step by step
  }
  return DIM2D_OK;
}

static int run_steps(dim2d_handle* h, double dt, int nsteps) {
  const bool graphs = h->use_graphs && !h->prof;
  if (graphs && h->graph_dt != dt) {
    drop_graphs(h);
    h->graph_dt = dt;
  }
  for (int s = 0; s < nsteps;) {
    // stage 1 writes B: a pending asynchronous copy of B must land first.  One
    // of A overlaps the first step; the second writes A.
    const bool copying = h->copy_pending && h->copy_src == h->A;
    const int size = graph_size_for(copying ? 1 : nsteps - s);
    const int n = GRAPH_STEPS[size];
    // (200 steps of a 64^2 open field: 2532 us with the corner cells apart, 1849)
    h->corners_apart = size != 0;
    cudaError_t ew = wait_copy_if(h, h->B);
    if (ew != cudaSuccess) return cuda_error(ew, "step");
    if (graphs) {
      StepGraph* const slots = h->graph[size];
      StepGraph* g = nullptr;
      for (int i = 0; i < 2; i++)
        if (slots[i].exec && slots[i].A == h->A) g = &slots[i];
      if (!g) {
        StepGraph& free = slots[slots[0].exec && slots[0].A != h->A ? 1 : 0];
        if (capture_steps(h, dt, free, n) == DIM2D_OK) g = &free;
      }
      if (g) {
        cudaError_t e = cudaGraphLaunch(g->exec, h->stream);
        if (e != cudaSuccess) return cuda_error(e, "step graph");
        h->launches += g->launches;
        for (int i = 0; i < n; i++) {  // the host side of rk3_step
          std::swap(h->A, h->B);
          h->t += dt;  // field_class.f:70
        }
        s += n;
        continue;
      }
    }
    for (int i = 0; i < n; i++, s++) {
      int rc = rk3_step(h, dt);
      if (rc) return rc;
    }
  }
  return DIM2D_OK;
}

int rk3_steps(dim2d_handle* h, double dt, int nsteps) {
  if (h->variant == PERSIST_VARIANT) return persist_steps(h, dt, nsteps, 1.0);
  const int rc = run_steps(h, dt, nsteps);
  h->corners_apart = true;
  return rc;
}
