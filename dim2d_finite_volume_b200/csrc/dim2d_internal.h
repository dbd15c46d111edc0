// dim2d_internal.h -- host-side handle and helpers behind include/dim2d.h.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstdarg>
#include <vector>

#include "../../include/dim2d.h"
#include "dim2d_kernels.cuh"

// Work tables of the persistent kernel for a set of fields of one precision
// (dim2d_persist.cu): per-field descriptors, the per-step item list and the
// per-band strip+ghost item counts in device memory, and the launch
// counters.  The tables hold the fields' buffers as they were when built;
// launches pass the step parity since then.
struct PersistPlan {
  dim2d::PDomain* dom = nullptr;
  dim2d::PItem* items = nullptr;
  int* sg = nullptr;
  unsigned long long* ctr = nullptr;  // [0] next item, band counters, node counters
  unsigned int* ctl = nullptr;        // [0] abort flag, [1] error word
  long long items_per_step = 0;
  int nfields = 0;
  int nbands = 0;
  int rows = 0;   // rows per band / strip item
  int ctas = 0;   // CTAs of the last launch
  bool mixed = false;
  bool valid = false;
  dim2d::DimConst k{};
  dim2d::WallConst wall{};
};

// A captured graph of whole RK3 steps.
struct StepGraph {
  cudaGraphExec_t exec = nullptr;
  const double* A = nullptr;  // buffer that held u^n
  long long launches = 0;     // kernel launches in one replay
  int asked = 0;              // runs that could have replayed it (batches)
};
// Steps per graph: a run of n steps replays as many graphs of 8 as fit, then
// of 2 (both leave the buffer parity as it was), then of 1.  Between the
// kernels of one graph a launch costs less than between graphs: 512^2
// periodic 27.0 -> 24.7 us per step, 1024^2 72.5 -> 70.8.
constexpr int GRAPH_SIZES = 3;
constexpr int GRAPH_STEPS[GRAPH_SIZES] = {8, 2, 1};
inline int graph_size_for(int steps) { return steps >= 8 ? 0 : steps >= 2 ? 1 : 2; }

// Device time (ms) of one dry step of an autotuner, whose launches dry()
// issues on s and counts in *launches.  Where issuing a step takes the host more
// than half of the step's time, steps are replayed with `graphs`, as they will be
// in earnest: launched one by one they follow at the rate of the host, 15 us per
// step of a field, 60 us of a batch, and every shape takes as long (three periodic
// fields of 64^2 to 150^2 ended on a shape of 22 us per step, 13 on the best; one
// of 128^2 even on 65, 9).
template <typename Dry>
cudaError_t time_dry_step(cudaStream_t s, bool graphs, Dry dry, long long* launches, float* ms) {
  constexpr int STEPS = 2;
  auto steps = [&]() {
    cudaError_t r = cudaSuccess;
    for (int i = 0; i < STEPS && r == cudaSuccess; i++) r = dry();
    return r;
  };
  cudaGraphExec_t x = nullptr;
  long long per_replay = 0;
  auto run = [&]() {
    if (!x) return steps();
    *launches += per_replay;
    return cudaGraphLaunch(x, s);
  };
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  cudaError_t e = cudaEventCreate(&e0);
  if (e == cudaSuccess) e = cudaEventCreate(&e1);
  float issue = 0.f;
  auto measure = [&](int reps) {
    cudaError_t r = cudaEventRecord(e0, s);
    const auto t0 = std::chrono::steady_clock::now();
    for (int i = 0; i < reps && r == cudaSuccess; i++) r = run();
    const std::chrono::duration<float, std::milli> t = std::chrono::steady_clock::now() - t0;
    issue = t.count() / (float)(reps * STEPS);
    if (r == cudaSuccess) r = cudaEventRecord(e1, s);
    if (r == cudaSuccess) r = cudaEventSynchronize(e1);
    if (r == cudaSuccess) r = cudaEventElapsedTime(ms, e0, e1);
    *ms /= (float)(reps * STEPS);
    return r;
  };
  if (e == cudaSuccess) e = measure(1);  // warm-up
  if (e == cudaSuccess) e = measure(1);
  if (e == cudaSuccess && graphs && issue > 0.5f * *ms) {
    const long long n0 = *launches;
    if (cudaStreamBeginCapture(s, cudaStreamCaptureModeRelaxed) == cudaSuccess) {
      e = steps();
      cudaGraph_t g = nullptr;
      const cudaError_t ec = cudaStreamEndCapture(s, &g);
      if (e == cudaSuccess && ec == cudaSuccess && g) cudaGraphInstantiate(&x, g, 0);
      if (g) cudaGraphDestroy(g);
    }
    cudaGetLastError();  // a stream that cannot be captured: launched
    per_replay = *launches - n0;
    *launches = n0;
    // the least of four, some 0.15 ms each after the first
    if (x && e == cudaSuccess) e = run();
    float least = *ms;
    int reps = 1;
    for (int r = 0; r < 4 && x && e == cudaSuccess; r++) {
      e = measure(reps);
      least = std::min(least, *ms);
      reps = std::max(1, std::min(6, (int)(0.15f / (least * STEPS))));
    }
    *ms = least;
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  if (x) cudaGraphExecDestroy(x);
  return e;
}

struct dim2d_handle {
  int device = 0;
  dim2d_params p{};
  dim2d::DimConst k{};
  int precision = 0;
  int periodic = 0;
  int open_all = 0;  // hedstrom_xy: every section open, type bc_timedev
  int south_wall = 0;  // wall on S: wall_S_reflection, wall_S_open, half_wall_S_open
  int corners_y = 0;   // corner sections are reflection_y
  // open (Hedstrom) sections: dim2d::OPEN_* mask of the time-integrated ghost
  // sections (all of them for hedstrom_xy) and the open sides of the mixed
  // presets wall_S_open / half_wall_S_open
  int open_mask = 0;
  int open_w = 0, open_e = 0, open_n = 0;
  // dim2d::NODE_* sides whose ghost cells a node pass writes (mirrors, wall):
  // the persistent kernel's
  int node_sides = 0;
  // ... that are mirrors, whose images a stage launch writes itself
  int mirror_sides = 0;
  dim2d::WallConst wall{};
  unsigned int* status = nullptr;  // wall root status word (device)
  double xmap0 = 0, ymap0 = 0;     // x_map(1), y_map(1)
  int variant = 0;                 // stage-kernel variant (dim2d_set_variant)
  bool corners_apart = true;       // variant 0, hedstrom_xy: see launch_stage_work
  struct dim2d_batch* batch = nullptr;  // batch this field belongs to, if any
  // dim2d_download_async: side stream, its events, and the buffer being copied
  cudaStream_t copy_stream = nullptr;
  cudaEvent_t copy_ready = nullptr, copy_done = nullptr;
  const double* copy_src = nullptr;
  bool copy_pending = false;
  int bc_choice[8]{}, bc_type[8]{}, bc_order[8]{};
  int side_kind[8]{};
  dim2d::Field f{};
  // A = u^n (the field), B and C = stage buffers
  double* A = nullptr;
  double* B = nullptr;
  double* C = nullptr;
  double* td = nullptr;  // time_dev buffer, allocated on first use
  double* x_map = nullptr;
  double* y_map = nullptr;
  double* scalar = nullptr;  // [0] CFL reduction, [2] wall status word (status),
                             // [3] health word of a served request (health_word)
  double dx = 0, dy = 0, rdx = 0, rdy = 0;
  double x_min = 0, x_max = 0, y_min = 0, y_max = 0;
  double t = 0;
  bool uploaded = false;
  cudaStream_t stream = nullptr;
  cudaStream_t own_stream = nullptr;
  cudaStream_t pool = nullptr;  // buffers from the stream-ordered pool on this stream
  long long launches = 0;
  // captured step graphs by size and buffer parity (which buffer holds u^n);
  // valid for graph_dt, -1 invalidates them (set by anything that changes
  // kernel parameters)
  bool use_graphs = true;
  StepGraph graph[GRAPH_SIZES][2];
  double graph_dt = -1.0;
  // stage-kernel variant 6: the persistent kernel, tables built on first
  // use (pplan), steps since then (pparity)
  PersistPlan* pplan = nullptr;
  dim2d::PDomain pdom0{};  // buffers the tables were built with
  double pdt = -1.0;       // dt the tables hold (-1: rebuild)
  // live timing of the interior stage kernel (dim2d_profile)
  bool prof = false;
  std::vector<cudaEvent_t> prof_ev;  // start/stop pairs
  size_t prof_used = 0;
};

namespace dim2d {
int set_error(int code, const char* fmt, ...);
int cuda_error(cudaError_t e, const char* where);
DimConst make_const(const dim2d_params& p);
int pitch_for(int nx);
int resolve_sides(const int bc_choice[8], const int bc_type[8], int side_kind[8], int* periodic);
// 1 if all eight sections are hedstrom_choice with type bc_timedev
int all_open(const int bc_choice[8], const int bc_type[8]);
}  // namespace dim2d

// Mirror / south-wall configurations (library_config.py:58-115): returns 1
// and sets the flags when bc_choice/bc_type are reflection_xy or
// wall_S_reflection.
namespace dim2d {
int classify_mirrors(const int bc_choice[8], const int bc_type[8], int* south_wall,
                     int* corners_y);
// wall_S_open or half_wall_S_open (library_config.py:118-150): returns 1
// and sets *open_w (1 for wall_S_open, 0 for half_wall_S_open's mirror W);
// returns minus an error code (set_error) for a section order the kernels
// do not reproduce, 0 for any other configuration
int classify_open_wall(const int bc_choice[8], const int bc_type[8], const int bc_order[8],
                       int* open_w);
WallConst make_wall(const dim2d_params& p);
// dim2d_create; pool != nullptr: stream-ordered allocations on `pool`,
// which also becomes the field's stream
int create_field(const dim2d_params* p, int nx, int ny, const int bc_choice[8],
                 const int bc_type[8], const int bc_order[8], int precision, cudaStream_t pool,
                 dim2d_handle** out);
}  // namespace dim2d

// dim2d_step.cu
dim2d::StageArgs make_stage_args(const dim2d_handle* h, const double* uin, double* uout,
                                 double dt, int st);
int rk3_step(dim2d_handle* h, double dt);
// nsteps RK3 steps; each step replays a captured CUDA graph when graphs are
// enabled and the handle is not profiling
int rk3_steps(dim2d_handle* h, double dt, int nsteps);
// variant 6 (the persistent kernel): nsteps steps as one launch;
// dt_scale 0 = dry step of the autotuner
constexpr int PERSIST_VARIANT = 6;
int persist_steps(dim2d_handle* h, double dt, int nsteps, double dt_scale);
// the complete work of one stage (mode 1) or time derivative (mode 0): the
// stage kernel and, on open fields where the stage kernel does not cover
// them, the ghost-cell kernel; counts launches, profiles the stage kernel
cudaError_t launch_stage_work(dim2d_handle* h, const dim2d::StageArgs& a, int mode);
int apply_bc_on_nodes(dim2d_handle* h, const double* nodes_tmp, double* nodes);
int check_status(dim2d_handle* h);
// device word the serving loop's check sets: bit 0 a non-finite value in the
// field, bit 1 the wall status word set (zero at creation)
inline unsigned int* health_word(dim2d_handle* h) {
  return reinterpret_cast<unsigned int*>(h->scalar + 3);
}
// bracket one launch with profiling events (no-op unless h->prof)
void prof_begin(dim2d_handle* h);
void prof_end(dim2d_handle* h);
void drop_graphs(dim2d_handle* h);
// before work on h->stream writes `target`: wait for a pending
// dim2d_download_async copy whose source it is
cudaError_t wait_copy_if(dim2d_handle* h, const double* target);

// dim2d_persist.cu
void persist_free(PersistPlan& pl);
int persist_build(PersistPlan& pl, const std::vector<dim2d_handle*>& hs,
                  const std::vector<double>& dts, int rows, cudaStream_t s);
// nsteps steps of every field of the plan (dt_scale 0: dry steps that
// write only the stage buffers); step0 = steps taken since the build
cudaError_t persist_launch(PersistPlan& pl, int nsteps, int step0, double dt_scale,
                           unsigned long long wait_ns, long long withhold, cudaStream_t s);
// reads and clears the plan's error word (synchronous): DIM2D_ERR_TIMEOUT
// if a launch stopped at a wait that ran out
int persist_error(PersistPlan& pl);
