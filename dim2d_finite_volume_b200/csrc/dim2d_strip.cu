// dim2d_strip.cu -- fused RK3 stage, warp-streaming variant for sm_100a.
//
// Node quantities, face fluxes, divergence, body force and stage update of
// one RK stage (or the time derivative) in one pass over the state:
//   * a warp owns a strip of 30 interior columns and H rows and marches up
//     the strip one row per iteration; lane l holds column c0-1+l, so lanes
//     1..30 own the cells and lanes 0 and 31 their neighbours;
//   * what a cell needs of its own column stays in the lane's registers:
//     the state of row y, the node quantities of rows y and y+1, the bottom
//     face's flux.  What it needs of the columns beside it comes by warp
//     shuffle; state rows and u^n rows travel ahead of the warp into a
//     shared-memory ring (cp.async);
//   * node quantities (NodeQ) are chosen so that a face flux is made of their
//     sums and differences: products such as my v + P, rho u v and
//     (E + P) v are taken once per node instead of twice per face, and
//     Tcl - Tcap/We is one quantity, since both enter the energy flux by
//     their normal derivative with the factor 1/(Re Pr).  sqrt(1/We) is
//     folded into the density gradients, 1/We into the Laplacian.  Face
//     Laplacian and tangential derivatives are the sums of the two nodes'
//     halves (the reference's Mattsson stencils, regrouped);
//   * iteration y: copies of rows y+4 (state) and y+2 (u^n) are issued;
//     velocities of row y+1; x-face between columns x-1 and x of row y; the
//     other node quantities of row y+1; y-face between rows y and y+1; the
//     right x-face comes from lane+1, the bottom y-face is the top one of the
//     iteration before; update of cell (x, y).  Two rows per pass of the
//     loop, so that the values handed from row to row need no moves.
//
// Bound: instruction issue and FP64 latency at 4 warps per scheduler.  The
// form before this one kept node quantities in shared memory too and moved
// 165 128-byte wavefronts per warp and row through that pipe, against 121
// cycles of FP64 work; now a row costs 34 shuffles, 36 wavefronts of row data
// and 165 FP64 instructions instead of 242.  Measured per RK3 step (best
// shape): 1024^2 periodic 99.7 -> 70.1 us, 2048^2 open 321.7 -> 230, 2048^2 wall
// in mixed precision 324.8 -> 223 in runs of some 10 ms; longer ones at 2048^2
// reach the board's power limit (open 257 to 270).  Tried beside it: all
// rows prefetched into registers instead of the ring (periodic 85.7, more
// registers and 420 instead of 400 instructions per row), 20 warps per SM at
// 96 registers (92; spills), three or four rows per pass (as fast, larger).
//
// On a field with open sections the launch also integrates their ghost
// cells (open_run, one warp per run): they take the first CTAs of the grid, so
// that they overlap the strips.  Ghost and interior cells read the same input
// and write disjoint cells.
#include "dim2d_nodebc.cuh"

namespace dim2d {

namespace {

constexpr int SW = STRIP_COLS;  // cells per strip
constexpr int WARPS = 16;       // resident warps per SM (one warp per CTA, <= 128 registers)

// Every launch of a step is a programmatic dependent of the one before it on
// its stream: it lets its own dependent start before it ends and waits for the
// launch before it, complete and visible, before its first read
// (griddepcontrol.wait), so that launch latency and block scheduling overlap
// that launch's end.  The wait is what makes that launch's output visible: no
// kernel reads or writes a state before it, whatever ran in between (a launch
// that let its dependents start gives them no ordering by that alone).

template <typename T>
__device__ __forceinline__ T from_left(T v) {
  return __shfl_up_sync(0xffffffffu, v, 1);
}
template <typename T>
__device__ __forceinline__ T from_right(T v) {
  return __shfl_down_sync(0xffffffffu, v, 1);
}

// Asynchronous global -> shared copies (cp.async) through L2: the state rows
// and u^n rows ahead of the warp land in its shared-memory ring while it
// computes, without passing through registers.  (The L2 path is coherent:
// the persistent kernel rereads buffers that other SMs rewrite within its
// launch.)  Completion is per thread (commit / wait groups); a __syncwarp
// after the wait makes the whole row visible.
__device__ __forceinline__ void cp_async16(double* smem, const double* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(double* smem, const double* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
// wait until at most N of this thread's most recent groups are pending
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// The warp's ring: NS state rows (columns c0-2 .. c0+31 of 4 planes) and NU
// rows of u^n (columns c0-2 .. c0+29, same row length).
constexpr int RC = 34, NS = 5, NU = 3;
constexpr int ST_ROW = 4 * RC, UN_ROW = ST_ROW;
constexpr int WARP_DOUBLES = NS * ST_ROW + NU * UN_ROW;
constexpr int KEEP_AT = ST_ROW;  // what a wall run keeps (strip_warp)
extern __shared__ __align__(16) double g_ring[];

// The lane's part in copying a row: 16-byte pairs of columns c0-2 .. c0+29
// of two planes at once (lanes 0-15 one plane, 16-31 the next) and, by lanes
// 0..3, the pair of columns c0+30, c0+31 of one plane each.  Columns are
// clamped to the pitch, so no copy leaves the allocation; clamped values land
// in columns that only unused lanes read.  Needs an even pitch and 16-byte
// aligned planes (strip_layout_ok).
struct RowCopy {
  const double* src;  // the lane's first pair in the next row to copy
  size_t edge;        // from there to its pair of columns c0+30, c0+31
  int dst, edge_dst;  // their places in a ring row
  __device__ __forceinline__ RowCopy(const double* u, const Field& f, int c0, int row, int lane) {
    const int half = lane >> 4, pair = 2 * (lane & 15);
    const int col = min(c0 - 2 + pair, f.pitch - 2);
    src = u + (size_t)row * f.pitch + half * f.plane + col;
    edge = (size_t)lane * f.plane + (min(c0 + 30, f.pitch - 2) - col);
    dst = half * RC + pair;
    edge_dst = lane * RC + 32;
  }
  // the next state row into the ring row at `to`
  __device__ __forceinline__ void state(const Field& f, double* to, int lane) const {
    cp_async16(to + dst, src);
    cp_async16(to + dst + 2 * RC, src + 2 * f.plane);
    if (lane < 4) cp_async16(to + edge_dst, src + edge);
  }
  // the same for MODE 3: any pitch and alignment, 8 bytes a copy.  The 8-byte
  // form goes through L1, so its launches are plain ones: L1 is clean at their
  // start, and nothing rewrites their input while they run.
  __device__ __forceinline__ void narrow_state(const Field& f, const double* u, int c0, int row,
                                               double* to, int lane) const {
    const double* p = u + (size_t)row * f.pitch;
    const int col = min(c0 - 2 + lane, f.nx - 1), edge_col = min(c0 + 30 + (lane & 1), f.nx - 1);
#pragma unroll
    for (int v = 0; v < 4; v++) cp_async8(to + v * RC + lane, p + v * f.plane + col);
    if (lane < 8)
      cp_async8(to + (lane >> 1) * RC + 32 + (lane & 1), p + (lane >> 1) * f.plane + edge_col);
  }
  // the row at distance d (in u^n) into the ring row at `to`
  __device__ __forceinline__ void un(const Field& f, ptrdiff_t d, double* to) const {
    cp_async16(to + dst, src + d);
    cp_async16(to + dst + 2 * RC, src + d + 2 * f.plane);
  }
};

// Products that are added to something are written as fma, and products that
// must not be contracted as mul(), so that every instantiation of this code
// (one field, batch, persistent kernel) rounds alike.
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }

// Node quantities of one row in the lane's column.  T = double, or float for
// the face pass of the mixed-precision path; u, v, P, Tcl, 1/(3-rho) and
// Tcap are always evaluated in FP64.
template <typename T>
struct NodeQ {
  T r, mx, my, e;  // conservative values
  T u, v, p;       // velocity, pressure
  T qyy, qxy, hv;  // my v + P, mx v (= my u), (E + P) v
  T cp;            // 1.5/cv_r / (3 - rho)
  T lap;           // 1/We times half the density Laplacian
  T gx, gy;        // sqrt(1/We) times half the centred density gradient
  T dw;            // rho(x) - rho(x-1)
  double th;       // Tcl - Tcap/We, FP64 also in mixed precision
};

// Primitives as node_prim() (dim2d_prim_module.f:242-289, 425-453, 515-544,
// 1056-1071) with 1/rho and 1/(3-rho) from one reciprocal; Tcap = 0.5/rho
// |grad rho|^2 with centred gradients (:582-613).  First part: what the
// x-face of the row below takes from this row.
struct NodeUV {
  double inv, ir, u, v;
};
__device__ __forceinline__ NodeUV node_uv(double r, double mx, double my) {
  NodeUV n;
  const double tm = 3.0 - r;
  n.inv = reciprocal(r * tm);
  n.ir = tm * n.inv;
  n.u = mul(mx, n.ir);
  n.v = mul(my, n.ir);
  return n;
}
// the rest; dw = density difference to the west node, d1x, d1y = sums and
// d2x, d2y = differences of the density differences to both sides (the
// undivided centred first and second differences)
template <typename T>
__device__ __forceinline__ NodeQ<T> node(const NodeUV& n, double r, double mx, double my,
                                         double e, double dw, double d1x, double d2x, double d1y,
                                         double d2y, const StripCoef<double>& c) {
  const double cp = mul(c.c15cv * r, n.inv);
  const double m3r2 = mul(-3.0 * r, r);
  // W = E - rho|u|^2/2 + 3 rho^2
  const double w = fma(-0.5, fma(mx, n.u, my * n.v), e) - m3r2;
  const double p = fma(cp, w + w, m3r2);
  const double gx = mul(c.gx, d1x), gy = mul(c.gy, d1y);
  NodeQ<T> q;
  q.th = mul(n.ir, fma(-2.0, fma(gx, gx, gy * gy), w));
  q.lap = (T)fma(c.lx, d2x, c.ly * d2y);
  q.r = (T)r;
  q.mx = (T)mx;
  q.my = (T)my;
  q.e = (T)e;
  q.u = (T)n.u;
  q.v = (T)n.v;
  q.p = (T)p;
  q.qyy = fma(q.my, q.v, q.p);
  q.qxy = mul(q.mx, q.v);
  q.hv = mul(q.e + q.p, q.v);
  q.cp = (T)cp;
  q.gx = (T)gx;
  q.gy = (T)gy;
  q.dw = (T)dw;
  return q;
}

template <typename T>  // dw, de, ds, dn = density differences to the four nodes around
__device__ __forceinline__ NodeQ<T> node(const NodeUV& n, double r, double mx, double my,
                                         double e, double dw, double de, double ds, double dn,
                                         const StripCoef<double>& c) {
  return node<T>(n, r, mx, my, e, dw, de + dw, de - dw, dn + ds, dn - ds, c);
}

// the face pass's type and coefficients
template <bool MIX>
struct FaceType {
  using type = double;
};
template <>
struct FaceType<true> {
  using type = float;
};
__device__ __forceinline__ const StripCoef<double>& coef_of(const StageArgs& a, double) { return a.c; }
__device__ __forceinline__ const StripCoef<float>& coef_of(const StageArgs& a, float) { return a.cf; }

// Sums (s..) and differences (d..) of the two nodes' quantities at a face,
// in the face frame (n = normal, t = tangential).
template <typename T>
struct FaceSums {
  T smn, sqn, sqt;       // m_n, m_n u_n + P, m_t u_n
  double sh;             // (E + P) u_n - 2/(Re Pr) d/dn (Tcl - Tcap/We)
  T scp, scu;            // cp, cp u_n
  T sr, sun, sut;        // rho, u_n, u_t
  T dr, dun, dut;        // normal differences
  T gt;                  // scaled tangential density gradient
  T dunt, dutt;          // undivided tangential differences of u_n, u_t
  T lap;                 // Laplacian / We
};

// Twice the face flux of (mass, normal momentum, tangential momentum,
// energy); formulas of face_flux (dim2d_fluxes_module.f:103-541) on sums
// instead of averages.  tnn, tnt: viscous stress plus the capillary terms
// that enter the energy flux with the same velocity.
// The temperature term of the energy flux, which holds the third
// derivatives of the capillary part, is FP64 in mixed precision too (cth).
template <typename T>
__device__ __forceinline__ void face2(const FaceSums<T>& f, const FaceCoef<T>& c, T s, T F[3],
                                      double* F3) {
  const T drn = c.s * f.dr;
  const T drn2 = mul(drn, drn);
  const T t = fma(f.gt, f.gt, -drn2);
  const T g2 = fma(f.gt, f.gt, drn2);
  const T div = fma(c.dn, f.dun, c.dt * f.dutt);
  const T tnn = fma(T(0.5), t, fma(c.a1, f.dun, c.a2 * f.dutt));
  const T tnt = fma(-drn, f.gt, fma(c.b1, f.dunt, c.b2 * f.dut));
  F[0] = f.smn;
  F[1] = fma(T(-2), tnn, f.sqn) - fma(f.scp, g2, f.sr * f.lap);
  F[2] = fma(T(-2), tnt, f.sqt);
  const T cap = fma(-(f.sr * (s * drn)), div, fma(f.scu, g2, f.smn * f.lap));
  *F3 = f.sh - (double)fma(f.sun, tnn, fma(f.sut, tnt, cap));
}

// Twice the flux of the south wall's face (wall_face_flux,
// wall_xy_equilibrium_module.f:445-908): th = Tcl - Tcap/We of the first
// interior node, q = wall heat flux.  In FP64 from the sums on, also in mixed
// precision (the flux of the wall is not part of its FP32 face pass).
template <typename T>
__device__ __forceinline__ void wall_face2(const FaceSums<T>& f, const FaceCoef<double>& c,
                                           double th, double dy, double q, const DimConst& k,
                                           double F[3], double* F3) {
  const double tl = k.c38cv * th;
  const double t_half = 0.5 * (tl + (tl + dy * k.c38cv * k.re * k.pr * q));
  const double md = 0.5 * (double)f.sr, drn = c.s * (double)f.dr, gt = (double)f.gt;
  const double p = 8.0 * md * t_half / (3.0 - md) - 3.0 * (md * md);
  F[0] = 0.0;
  F[1] = 2.0 * p - ((double)f.sr * (double)f.lap + (gt * gt - drn * drn));
  F[2] = -2.0 * (c.b2 * (double)f.dut - drn * gt);
  *F3 = 2.0 * q;
}

// x-face between the lane's column and the one to the left, row y: n = node
// quantities of row y, ul, vl = the left column's velocity, gyu, gyv =
// undivided velocity differences across row y
template <typename T>
__device__ __forceinline__ FaceSums<T> x_sums(const NodeQ<T>& n, T ul, T vl, T gyu, T gyv,
                                              double cth) {
  FaceSums<T> f;
  const T cl = from_left(n.cp);
  f.smn = from_left(n.mx) + n.mx;
  const T qxx = fma(n.mx, n.u, n.p), hu = mul(n.e + n.p, n.u);
  f.sqn = from_left(qxx) + qxx;
  f.sqt = from_left(n.qxy) + n.qxy;
  if (sizeof(T) == sizeof(double))  // the low side's term travels whole: one exchange
    f.sh = from_left(fma(cth, n.th, (double)hu)) + fma(-cth, n.th, (double)hu);
  else
    f.sh = fma(-cth, n.th - from_left(n.th), (double)(from_left(hu) + hu));
  f.scp = cl + n.cp;
  f.scu = fma(cl, ul, n.cp * n.u);
  f.sr = fma(T(2), n.r, -n.dw);
  f.sun = ul + n.u;
  f.sut = vl + n.v;
  f.dr = n.dw;
  f.dun = n.u - ul;
  f.dut = n.v - vl;
  f.gt = from_left(n.gy) + n.gy;
  f.dunt = from_left(gyu) + gyu;
  f.dutt = from_left(gyv) + gyv;
  f.lap = from_left(n.lap) + n.lap;
  return f;
}

// y-face between rows y (b) and y+1 (t) of the lane's column: dr = density
// difference, g..u, g..v = undivided velocity differences across the column
template <typename T>
__device__ __forceinline__ FaceSums<T> y_sums(const NodeQ<T>& b, const NodeQ<T>& t, T dr, T gxub,
                                              T gxut, T gxvb, T gxvt, double cth) {
  FaceSums<T> f;
  f.smn = b.my + t.my;
  f.sqn = b.qyy + t.qyy;
  f.sqt = b.qxy + t.qxy;
  f.sh = fma(-cth, t.th - b.th, (double)(b.hv + t.hv));
  f.scp = b.cp + t.cp;
  f.scu = fma(b.cp, b.v, t.cp * t.v);
  f.sr = b.r + t.r;
  f.sun = b.v + t.v;
  f.sut = b.u + t.u;
  f.dr = dr;
  f.dun = t.v - b.v;
  f.dut = t.u - b.u;
  f.gt = b.gx + t.gx;
  f.dunt = gxvb + gxvt;
  f.dutt = gxub + gxut;
  f.lap = b.lap + t.lap;
  return f;
}

// ---- open (Hedstrom) ghost cells ----------------------------------------
// What open_ghost_cell (dim2d_open.cuh) evaluates one cell per thread -- both
// faces of a cell from scratch, some 20 node primitives and a dependent chain
// of divisions and square roots that took 12 us whatever the field's size --
// done by a warp for a run of one layer's cells along an edge: a lane holds
// one position along the edge and the three nodes across it (both ghost
// layers and the first interior one), and neighbours come by shuffle as in the
// strips.  Per RK3 step: 64^2 open 30.7 -> 12.3 us, 301x187 half_wall_S_open
// 59 -> 29 us, 1024^2 open 82 -> 69 us.  Both layers in one warp would halve
// the loads but need more registers than the strips leave (160 bytes of spill
// in the batched kernels).

// Characteristic time derivative (hedstrom_xy_module.f:445-558 with the
// node's own eigenquantities) in the edge's frame: u along the edge, v across
// it, g.. = one-sided derivatives across it; out = (mass, momentum along,
// momentum across, energy).  The speed of sound of sound_speed() with its
// radicands multiplied out: c^2 = 3 (e + (P + 3 rho^2)/cv_r)/(rho (3 - rho)),
// e = P + rho^2 (2 rho - 3); where one of those radicands is negative the
// value is NaN there, and here.
__device__ __forceinline__ void char_term_run(double r, const NodeUV& n, double p, double gr,
                                              double gu, double gv, double gp, bool right,
                                              const DimConst& k, double out[4]) {
  const double u = n.u, v = n.v;
  const double ee = fma(r * r, fma(2.0, r, -3.0), p), pe = fma(3.0 * r, r, p);
  double c2 = fma(3.0, ee, k.c3cv * pe) * n.inv;
  if (!(r >= 0.0 && (3.0 - r) * ee >= 0.0 && pe * ee >= 0.0)) c2 = NAN;
  const double c = sqrt(c2), ic2 = 1.0 / c2;
  const double qc = 0.5 * r * c;
  auto amp = [&](double ev, double lg) {
    return (right ? ev <= 0.0 : ev >= 0.0) ? 0.0 : -ev * lg;  // openbc_operators_module.f:97-136
  };
  const double a0 = amp(v, gu), a1 = amp(v, fma(-ic2, gp, gr));
  const double a2 = amp(v - c, fma(-qc, gv, 0.5 * gp)), a3 = amp(v + c, fma(qc, gv, 0.5 * gp));
  const double tp = a2 + a3, tr = fma(ic2, tp, a1), tv = n.ir * c * ic2 * (a3 - a2);
  // conservative <- primitive Jacobian, ns_vdw2d_prim_module.f:249-320
  const double de = 0.5 * fma(u, u, v * v) - 6.0 * r -
                    1.0 / 3.0 * k.cv_r * fma(9.0 * (r - 2.0), r, p);
  out[0] = tr;
  out[1] = fma(tr, u, a0 * r);
  out[2] = fma(tr, v, tv * r);
  out[3] = fma(tr, de, r * fma(a0, u, tv * v)) + tp * (k.cv_r * (1.0 - r / 3.0));
}

__device__ __forceinline__ double pressure(const NodeUV& n, double r, double mx, double my,
                                           double e, const DimConst& k) {
  const double m3r2 = mul(-3.0 * r, r);
  const double w = fma(-0.5, fma(mx, n.u, my * n.v), e) - m3r2;
  return fma(mul(k.c15cv * r, n.inv), w + w, m3r2);
}

// L(u) (MODE 0) or stage update (MODE 1) of a ghost cell: q its state, L its
// time derivative (in place)
template <int MODE>
__device__ __forceinline__ void update_ghost(const StageArgs& a, const double q[4], double L[4],
                                             const double un[4]) {
  if (a.k.gravity_ac) {  // openbc_operators_module.f:354-372
    L[2] = fma(-q[0], a.k.gravity, L[2]);
    L[3] = fma(-q[2], a.k.gravity, L[3]);
  }
  if (MODE == 1) {
#pragma unroll
    for (int v = 0; v < 4; v++) {
      L[v] = fma(a.dt, L[v], q[v]);
      if (a.stage != 1) L[v] = fma(a.b, un[v], (1.0 - a.b) * L[v]);
    }
  }
}

// The ghost cell at position s along edge `side` (0..3 = S, N, W, E) in the
// inner or outer layer, from the lanes that hold the positions beside it (lane
// l-1 and l+1): its offset, and L(u) or new state in out.  Inner layer: the
// interior operators across the edge; outer layer: the one-sided ones (the
// *_L0 / *_R0 sets, bc_operators_openbc_normal_class.f:563-713), whose second
// derivative across the edge is the inner layer's.  All lanes take part.
template <int MODE>
__device__ __forceinline__ size_t open_edge_cell(const StageArgs& a, int side, int s, bool outer,
                                                 double out[4]) {
  const Field& f = a.f;
  const DimConst& k = a.k;
  const bool ye = side >= 2, hi = side & 1;  // edge along y; N or E
  const size_t along = ye ? f.pitch : 1, across = ye ? 1 : f.pitch;
  const int na = ye ? f.ny : f.nx, nc = ye ? f.nx : f.ny;
  const int c0 = hi ? nc - 3 : 0;  // the three nodes across: c0, c0+1, c0+2
  const size_t o0 = min(max(s, 0), na - 1) * along + c0 * across;
  const size_t V = f.plane, vs = ye ? 2 * V : V, vc = ye ? V : 2 * V;
  double r[3], ms[3], mc[3], e[3], un[4];
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const double* p = a.uin + o0 + j * across;
    r[j] = __ldcg(p);
    ms[j] = __ldcg(p + vs);
    mc[j] = __ldcg(p + vc);
    e[j] = __ldcg(p + 3 * V);
  }
  const int jl = outer ? (hi ? 2 : 0) : 1;  // the layer's node
  const size_t o = o0 + jl * across;
#pragma unroll
  for (int v = 0; v < 4; v++)
    un[v] = MODE == 1 && a.stage != 1 ? __ldcg(a.u0 + o + v * V) : 0.0;

  // coefficients in the edge's frame (x = along it, y = across it)
  const FaceCoef<double>& ca = ye ? a.c.y : a.c.x;
  StripCoef<double> c;
  c.c15cv = a.c.c15cv;
  c.gx = ye ? a.c.gy : a.c.gx;
  c.gy = ye ? a.c.gx : a.c.gy;
  c.lx = ye ? a.c.ly : a.c.lx;
  c.ly = ye ? a.c.lx : a.c.ly;
  const double rda = ye ? a.rdy : a.rdx, rdc = ye ? a.rdx : a.rdy;

  NodeUV n[3];
  double p[3];
#pragma unroll
  for (int j = 0; j < 3; j++) {
    n[j] = node_uv(r[j], ms[j], mc[j]);
    p[j] = pressure(n[j], r[j], ms[j], mc[j], e[j], k);
  }
  auto own = [&](const double* q) { return outer ? (hi ? q[2] : q[0]) : q[1]; };
  // difference across the edge that the layer's one-sided operators take, and
  // twice the undivided derivative of its tangential operators
  auto side_diff = [&](double q0, double q1, double q2) { return hi == outer ? q2 - q1 : q1 - q0; };
  auto twice = [&](double q0, double q1, double q2) {
    return outer ? 2.0 * (hi ? q2 - q1 : q1 - q0) : (q2 - q1) + (q1 - q0);
  };
  const double rl = own(r), msl = own(ms), mcl = own(mc), el = own(e), pl = own(p);
  const NodeUV nl = outer ? (hi ? n[2] : n[0]) : n[1];
  const double dw = rl - from_left(rl), de = from_right(rl) - rl;
  const NodeQ<double> q =
      node<double>(nl, rl, msl, mcl, el, dw, de + dw, de - dw, twice(r[0], r[1], r[2]),
                   (r[2] - r[1]) - (r[1] - r[0]), c);
  const FaceSums<double> fs =
      x_sums(q, from_left(q.u), from_left(q.v), twice(n[0].u, n[1].u, n[2].u),
             twice(n[0].v, n[1].v, n[2].v), ca.th);
  double F[3], F3;
  face2(fs, ca, a.c.s, F, &F3);
  if (ye && a.wall_s && s == BC) {
    // the face under the first interior row carries the wall corner's flux
    // (bc_operators_wall_xy_class.f:702-854)
    wall_face2(fs, ca, q.th, a.dy, wall_heat_flux(a.wall, a.xmap0 + (c0 + jl) * a.dx), k, F, &F3);
  }
  __syncwarp();
  double D[4];
#pragma unroll
  for (int v = 0; v < 3; v++) D[v] = F[v] - from_right(F[v]);
  D[3] = F3 - from_right(F3);
  double ch[4];
  char_term_run(rl, nl, pl, rdc * side_diff(r[0], r[1], r[2]),
                rdc * side_diff(n[0].u, n[1].u, n[2].u),
                rdc * side_diff(n[0].v, n[1].v, n[2].v), rdc * side_diff(p[0], p[1], p[2]), hi, k,
                ch);
  const double h = 0.5 * rda;
  const double qc[4] = {rl, ye ? mcl : msl, ye ? msl : mcl, el};
  out[0] = fma(h, D[0], ch[0]);
  out[1] = ye ? fma(h, D[2], ch[2]) : fma(h, D[1], ch[1]);
  out[2] = ye ? fma(h, D[1], ch[1]) : fma(h, D[2], ch[2]);
  out[3] = fma(h, D[3], ch[3]);
  update_ghost<MODE>(a, qc, out, un);
  return o;
}

// One ghost layer (0 inner, 1 outer) of `count` <= OPEN_RUN cells from position
// `first` along edge `side`.  Lane l holds position first-2+l; cells are lanes
// 2 .. count+1, faces lanes 2 .. count+2.
template <int MODE>
__device__ __forceinline__ void open_edge_run(const StageArgs& a, int side, int layer, int first,
                                              int count) {
  const int lane = threadIdx.x & 31, s = first - 2 + lane;
  double q[4];
  const size_t o = open_edge_cell<MODE>(a, side, s, layer == 1, q);
  if (lane < 2 || lane >= 2 + count) return;
  double* out = a.uout + o;
#pragma unroll
  for (int v = 0; v < 4; v++) out[v * a.f.plane] = q[v];
  // half_wall_S_open's NW corner mirrors the open N ghost rows
  if (MODE == 1 && side == 1 && s < 2 * BC && (a.mirror & NODE_W)) {
    out += 2 * BC - 1 - 2 * s;
#pragma unroll
    for (int v = 0; v < 4; v++) out[v * a.f.plane] = v == 1 ? -q[v] : q[v];
  }
}

// The corner cells of the sections in `mask`, lanes 0..15 (four per corner,
// SW, SE, NW, NE): characteristic terms of both directions.
template <int MODE>
__device__ __forceinline__ void open_corner_cells(const StageArgs& a, int mask) {
  const int lane = threadIdx.x & 31, c = lane >> 2;
  if (lane >= 16 || !(mask >> (4 + c) & 1)) return;
  const Field& f = a.f;
  const DimConst& k = a.k;
  const bool east = c & 1, north = c >> 1;
  const int x = (east ? f.nx - BC : 0) + (lane & 1), y = (north ? f.ny - BC : 0) + (lane >> 1 & 1);
  const size_t o = (size_t)y * f.pitch + x, V = f.plane;
  // the node and its neighbours inwards along x and along y
  const ptrdiff_t d[3] = {0, east ? -1 : 1, north ? -(ptrdiff_t)f.pitch : f.pitch};
  double q[3][4], un[4];
#pragma unroll
  for (int j = 0; j < 3; j++)
#pragma unroll
    for (int v = 0; v < 4; v++) q[j][v] = __ldcg(a.uin + o + d[j] + v * V);
#pragma unroll
  for (int v = 0; v < 4; v++)
    un[v] = MODE == 1 && a.stage != 1 ? __ldcg(a.u0 + o + v * V) : 0.0;
  NodeUV n[3];
  double p[3];
#pragma unroll
  for (int j = 0; j < 3; j++) {
    n[j] = node_uv(q[j][0], q[j][1], q[j][2]);
    p[j] = pressure(n[j], q[j][0], q[j][1], q[j][2], q[j][3], k);
  }
  const double sx = east ? a.rdx : -a.rdx, sy = north ? a.rdy : -a.rdy;
  const NodeUV t{n[0].inv, n[0].ir, n[0].v, n[0].u};  // along y, across x
  double cx[4], cy[4], L[4];
  char_term_run(q[0][0], t, p[0], sx * (q[0][0] - q[1][0]), sx * (n[0].v - n[1].v),
                sx * (n[0].u - n[1].u), sx * (p[0] - p[1]), east, k, cx);
  char_term_run(q[0][0], n[0], p[0], sy * (q[0][0] - q[2][0]), sy * (n[0].u - n[2].u),
                sy * (n[0].v - n[2].v), sy * (p[0] - p[2]), north, k, cy);
  L[0] = cx[0] + cy[0];
  L[1] = cx[2] + cy[1];
  L[2] = cx[1] + cy[2];
  L[3] = cx[3] + cy[3];
  update_ghost<MODE>(a, q[0], L, un);
#pragma unroll
  for (int v = 0; v < 4; v++) a.uout[o + v * V] = L[v];
}

// ghost run number m of a launch: the runs of the open edges S, N, W, E, then
// one for the corners (found before the wait: 64^2 open 12.0 us per step, 11.3)
template <int MODE>
__device__ __forceinline__ void open_run(const StageArgs& a, int m) {
  int side = 0, cells = 0;
  for (; side < 4; side++) {
    if (!(a.open >> side & 1)) continue;
    cells = (side < 2 ? a.f.nx : a.f.ny) - 2 * BC;
    const int runs = BC * ((cells + OPEN_RUN - 1) / OPEN_RUN);
    if (m < runs) break;
    m -= runs;
  }
  wait_for_launch_before();
  if (side == 4) {
    open_corner_cells<MODE>(a, a.open);
    return;
  }
  const int at = m / BC * OPEN_RUN;
  open_edge_run<MODE>(a, side, m % BC, BC + at, min(OPEN_RUN, cells - at));
}

// The strip of one warp: columns c0 .. c0+29 (interior ones), rows y0 ..
// y1-1.
// UN: whether the stage reads u^n (stages 2 and 3), 2: by a.stage (persistent
// kernel: no images of mirrors).  KEEP: the launch has wall runs; with `keep`
// (two rows) nothing is stored, and the new state of row y0 and the new
// density of row y0+1 stay in the lane's places of the ring (KEEP_AT).
template <int MODE, int UN, bool MIX, bool KEEP = false>
__device__ __forceinline__ void strip_warp(const StageArgs& a, int c0, int y0, int y1,
                                           bool keep = false) {
  using T = typename FaceType<MIX>::type;
  const int lane = threadIdx.x & 31;
  const Field f = a.f;
  const StripCoef<double>& cd = a.c;
  const StripCoef<T>& c = coef_of(a, T(0));
  const bool need_un = MODE == 1 && (UN == 2 ? a.stage != 1 : UN == 1);

  if (UN != 2) wait_for_launch_before();

  // the lane's column (columns past the field are not stored); its place in
  // a ring row
  const int x = c0 - 1 + lane;
  const size_t P = f.pitch, V = f.plane;
  double* const ring = g_ring + (threadIdx.x >> 5) * WARP_DOUBLES;
  double* const uring = ring + NS * ST_ROW;
  auto st = [&](int slot) { return ring + slot * ST_ROW + lane + 1; };

  // rows y0-2 .. y0+2 into slots 0 .. 4, all in flight together
  RowCopy copy(a.uin, f, c0, y0 - 2, lane);
  auto copy_state = [&](int row, double* to) {  // rows in order
    if (MODE == 3) copy.narrow_state(f, a.uin, c0, row, to, lane);
    else copy.state(f, to, lane);
  };
#pragma unroll
  for (int i = 0; i < 4; i++) {
    copy_state(y0 - 2 + i, ring + i * ST_ROW);
    copy.src += P;
  }
  cp_async_commit();
  // u^n of the row two below the state row being copied
  const ptrdiff_t un_row = (a.u0 - a.uin) - 2 * (ptrdiff_t)P;
  copy_state(y0 + 2, ring + 4 * ST_ROW);
  if (need_un) copy.un(f, un_row, uring);
  copy.src += P;
  cp_async_commit();
  cp_async_wait<1>();
  __syncwarp();
  const double rm = st(1)[0];
  double r0 = st(2)[0], mx0 = st(2)[RC], my0 = st(2)[2 * RC], e0 = st(2)[3 * RC];
  double r1 = st(3)[0];

  // node quantities of rows y0-1 and y0, bottom face of row y0
  NodeQ<T> n0;
  T um, vm;              // velocity of row y-1
  T ul0, vl0, gxu0, gxv0;  // row y: left velocity, undivided differences across the column
  double dn0 = r1 - r0;  // density difference between rows y and y+1
  double Gb[3];  // in the face frame: mass, m_y, m_x
  double gb3;
  {
    const double dn = r0 - rm;
    const double mxm = st(1)[RC], mym = st(1)[2 * RC];
    const NodeQ<T> nm = node<T>(node_uv(rm, mxm, mym), rm, mxm, mym, st(1)[3 * RC],
                                rm - st(1)[-1], st(1)[1] - rm, rm - st(0)[0], dn, cd);
    n0 = node<T>(node_uv(r0, mx0, my0), r0, mx0, my0, e0, r0 - st(2)[-1], st(2)[1] - r0, dn, dn0,
                 cd);
    um = nm.u;
    vm = nm.v;
    ul0 = from_left(n0.u);
    vl0 = from_left(n0.v);
    gxu0 = from_right(n0.u) - ul0;
    gxv0 = from_right(n0.v) - vl0;
    const FaceSums<T> s = y_sums(nm, n0, (T)dn, (T)(from_right(um) - from_left(um)), gxu0,
                                 (T)(from_right(vm) - from_left(vm)), gxv0, cd.y.th);
    if (a.wall_s && y0 == BC)
      wall_face2(s, cd.y, n0.th, a.dy, wall_heat_flux(a.wall, a.xmap0 + x * a.dx), a.k, Gb, &gb3);
    else {
      T G[3];
      face2(s, c.y, c.s, G, &gb3);
#pragma unroll
      for (int v = 0; v < 3; v++) Gb[v] = (double)G[v];
    }
  }

  const bool active = lane >= 1 && lane <= SW && x <= f.nx - 1 - BC &&
                      (MODE < 2 || (x >= a.box_x0 && x <= a.box_x1));
  // column of the cell's image in a ghost layer of a periodic or mirror side
  const bool images = MODE == 1 && (a.periodic || (UN != 2 && a.mirror));
  int ix2 = -1;
  if (images) {
    if (x < 2 * BC && (a.periodic || (a.mirror & NODE_W)))
      ix2 = a.periodic ? x + f.nx - 2 * BC : 2 * BC - 1 - x;
    else if (x >= f.nx - 2 * BC && (a.periodic || (a.mirror & NODE_E)))
      ix2 = a.periodic ? x - (f.nx - 2 * BC) : 2 * (f.nx - BC) - 1 - x;
  }
  const bool column_images = images && __any_sync(0xffffffffu, ix2 >= 0);
  // stage update: out = b u^n + (1 - b) (u + dt L), L from doubled fluxes
  const double w = MODE == 1 ? (1.0 - a.b) * a.dt : 1.0;
  const double wx = 0.5 * a.rdx * w, wy = 0.5 * a.rdy * w;

  double* __restrict__ out = a.uout + (size_t)y0 * P + x;

  const double* const un = uring + lane + 1;

  // the next row's copies: state row y0+3 into the slot of row y0-2
  __syncwarp();
  if (y0 + 1 < y1) {
    copy_state(y0 + 3, ring);
    if (need_un) copy.un(f, un_row, uring + UN_ROW);
    copy.src += P;
  }
  cp_async_commit();

  // ring slots of state rows y+1, y+2 and (to be written) y+4, of u^n rows y
  // and (to be written) y+2
  int o1 = 3 * ST_ROW, o2 = 4 * ST_ROW, ow = ST_ROW, ou = 0, ouw = 2 * UN_ROW;

  // r0/mx0/my0/e0 = state row y, r1 = density of row y+1
#pragma unroll(UN == 2 ? 1 : 2)  // (persistent kernel: registers)
  for (int y = y0; y < y1; y++) {
    if (y + 2 < y1) {
      copy_state(y + 4, ring + ow);
      if (need_un) copy.un(f, un_row, uring + ouw);
      copy.src += P;
    }
    cp_async_commit();
    cp_async_wait<2>();  // rows up to y+2 and u^n(y) are there
    __syncwarp();
    const double* const s1 = ring + o1 + lane + 1;
    const double mx1 = s1[RC], my1 = s1[2 * RC], e1 = s1[3 * RC];
    const double r2 = ring[o2 + lane + 1];

    // velocity of row y+1
    const NodeUV uv = node_uv(r1, mx1, my1);
    const T gyu = (T)uv.u - um, gyv = (T)uv.v - vm;

    // x-face of row y, and the right one from lane+1
    T Fx[3];
    double fx3;
    face2(x_sums(n0, ul0, vl0, gyu, gyv, cd.x.th), c.x, c.s, Fx, &fx3);
    double D[4];  // 2 (F_left - F_right)
#pragma unroll
    for (int v = 0; v < 3; v++) D[v] = (double)Fx[v] - (double)from_right(Fx[v]);
    D[3] = fx3 - from_right(fx3);

    // node quantities of row y+1
    const double dn1 = r2 - r1;
    const NodeQ<T> n1 =
        node<T>(uv, r1, mx1, my1, e1, r1 - s1[-1], s1[1] - r1, dn0, dn1, cd);

    // the dependent launch may start (on its last row: its warps then find
    // every SM about as empty as the others; let in at the start of this
    // launch, they crowd the SMs that finish first: 1024^2 open 71.7 us per
    // step, 67.7 so)
    if (UN != 2 && y == y1 - 1) let_dependents_start();

    // y-face between rows y and y+1
    const T ul1 = from_left(n1.u), vl1 = from_left(n1.v);
    const T gxu1 = from_right(n1.u) - ul1, gxv1 = from_right(n1.v) - vl1;
    T G[3];
    double Gt[3], gt3;
    face2(y_sums(n0, n1, (T)dn0, gxu0, gxu1, gxv0, gxv1, cd.y.th), c.y, c.s, G, &gt3);
#pragma unroll
    for (int v = 0; v < 3; v++) Gt[v] = (double)G[v];

    // update of cell (x, y)
    const double uc[4] = {r0, mx0, my0, e0};
    double q[4];
#pragma unroll
    for (int v = 0; v < 4; v++) {
      const int g = v == 1 ? 2 : (v == 2 ? 1 : 0);  // frame order of m_x and m_y
      const double dG = v < 3 ? Gb[g] - Gt[g] : gb3 - gt3;
      q[v] = MODE != 1 ? 0.0 : need_un ? fma(a.b, un[ou + v * RC], (1.0 - a.b) * uc[v]) : uc[v];
      q[v] = fma(wx, D[v], fma(wy, dG, q[v]));
    }
    if (a.k.gravity_ac) {  // pmodel_eq_class.f:1889-1904
      q[2] = fma(-w, r0 * a.k.gravity, q[2]);
      q[3] = fma(-w, my0 * a.k.gravity, q[3]);
    }
    if (KEEP && keep) {
      // (slots 1 and 2, of rows y0-1 and y0, are free after the prologue)
#pragma unroll
      for (int v = 0; v < 4; v++) ring[KEEP_AT + (y - y0) * ST_ROW + v * 32 + lane] = q[v];
    }
    // MODE 2 writes the interior_pt points of the layer map only
    else if (active && (MODE < 2 || __ldcg(a.mask + (size_t)y * P + x) == 1)) {
#pragma unroll
      for (int v = 0; v < 4; v++) out[v * V] = q[v];
      // periodic_xy/bc_operators_class.f:156-199; mirrors change the sign of
      // the normal momentum (bc_operators_reflection_{x,y}_class.f:178-296)
      if (images && (column_images || y < 2 * BC || y >= f.ny - 2 * BC)) {
        int iy2 = -1;
        if (y < 2 * BC && (a.periodic || (a.mirror & NODE_S)))
          iy2 = a.periodic ? y + f.ny - 2 * BC : 2 * BC - 1 - y;
        else if (y >= f.ny - 2 * BC && (a.periodic || (a.mirror & NODE_N)))
          iy2 = a.periodic ? y - (f.ny - 2 * BC) : 2 * (f.ny - BC) - 1 - y;
        if (ix2 >= 0 || iy2 >= 0) {
          const double mx = a.periodic ? q[1] : -q[1], my = a.periodic ? q[2] : -q[2];
#pragma unroll
          for (int v = 0; v < 4; v++) {
            double* dst = a.uout + v * V;
            const double qx = v == 1 ? mx : q[v], qy = v == 2 ? my : q[v];
            if (ix2 >= 0) dst[(size_t)y * P + ix2] = qx;
            if (iy2 >= 0) {
              dst[(size_t)iy2 * P + x] = qy;
              if (ix2 >= 0) dst[(size_t)iy2 * P + ix2] = v == 1 ? mx : qy;
            }
          }
        }
      }
    }
    out += P;

    um = n0.u;
    vm = n0.v;
    n0 = n1;
    ul0 = ul1;
    vl0 = vl1;
    gxu0 = gxu1;
    gxv0 = gxv1;
    Gb[0] = Gt[0];
    Gb[1] = Gt[1];
    Gb[2] = Gt[2];
    gb3 = gt3;
    dn0 = dn1;
    r0 = r1;
    mx0 = mx1;
    my0 = my1;
    e0 = e1;
    r1 = r2;
    __syncwarp();  // row y+1 and u^n(y) have been read
    o1 = o2;
    o2 = o2 == (NS - 1) * ST_ROW ? 0 : o2 + ST_ROW;
    ow = ow == (NS - 1) * ST_ROW ? 0 : ow + ST_ROW;
    ou = ou == (NU - 1) * UN_ROW ? 0 : ou + UN_ROW;
    ouw = ouw == (NU - 1) * UN_ROW ? 0 : ouw + UN_ROW;
  }
  cp_async_wait<0>();  // nothing lands after the warp's end or in its next strip
  __syncwarp();
}

// Wall run m of a field with a south wall: the ghost cells of up to 29 wall
// columns (the first of the interior runs) or 28, or of the wall corner at an
// open side: its two ghost columns and the interior column beside them.  The
// warp evaluates the new state of the two rows above the columns as the strips
// do, without storing it (in an open side's ghost columns as the ghost runs
// do), and solves each column's root from its lanes, so that no pass over the
// stage's output has to follow it: before, a launch of its own stood between
// two stages, some 5 us on small fields.  The runs take the first CTAs of the
// grid; their dependent evaluations overlap the strips.
// The rows are evaluated by the strips' own code (strip_warp with `keep`): a
// copy of it for the runs cost the strips of the same kernel 10 % by its
// register allocation (wall_S_reflection 1024^2: 82 us per step, 73.9 so;
// as a called function 73.6, but the runs, which small fields wait for, slower:
// 512^2 32.8 instead of 30.7).
struct WallRun {
  int corner;  // -1 interior run, else the open side (2 = W, 3 = E)
  int m, c0;   // number of the interior run; first interior column of the lanes
               // (even: the rows' 16-byte pairs)
  __device__ __forceinline__ WallRun(const StageArgs& a, int b) : corner(-1), m(b) {
    if (a.open & OPEN_W) {
      if (m == 0) corner = 2;
      m--;
    }
    if (corner < 0 && (a.open & OPEN_E)) {
      if (m == 0) corner = 3;
      m--;
    }
    c0 = corner == 2 ? BC : corner == 3 ? (a.f.nx - 2 * BC) & ~1 : BC + m * OPEN_RUN;
  }
};
__device__ __forceinline__ void wall_columns(const StageArgs& a, const WallRun& run) {
  const int lane = threadIdx.x & 31;
  const Field& f = a.f;
  const size_t V = f.plane, P = f.pitch;
  const bool mw = a.mirror & NODE_W, me = a.mirror & NODE_E;
  const int corner = run.corner, m = run.m;
  int x = run.c0 - 1 + lane;
  if (corner == 2 && lane == 31) x = 0;  // (lane 0 holds x = 1)
  bool mine;
  if (corner == 2) mine = x <= BC;
  else if (corner == 3) mine = x >= f.nx - BC - 1 && x < f.nx;
  else mine = lane >= (m == 0 ? 1 : 2) && lane <= 29 && x >= (mw ? BC : BC + 1) &&
              x <= f.nx - BC - (me ? 1 : 2);
  const double* kept = g_ring + KEEP_AT + lane;
  double keep[5];
#pragma unroll
  for (int v = 0; v < 4; v++) keep[v] = kept[v * 32];
  keep[4] = kept[ST_ROW];
  // u^n around the first interior node
  const int xc = min(x, f.nx - 1);
  const double* u0 = a.u0 + 2 * P + xc;
  WallIn in;
  in.gr = __ldcg(u0);
  in.gmx = __ldcg(u0 + V);
  in.gmy = __ldcg(u0 + 2 * V);
  in.gE = __ldcg(u0 + 3 * V);
  in.grw = __ldcg(u0 - (xc > 0 ? 1 : 0));
  in.gre = __ldcg(u0 + (xc < f.nx - 1 ? 1 : 0));
  in.grs = __ldcg(u0 - P);
  in.grn = __ldcg(u0 + P);
  if (corner >= 0) {
    // ghost cells of rows BC, BC+1: lanes l and 16+l hold row l of the inner
    // and the outer layer
    double g[4];
    open_edge_cell<1>(a, corner, lane & 15, lane >= 16, g);
    const int layer = corner == 2 ? 1 - x : x - (f.nx - BC);  // 0, 1 in the ghost columns
    const int src = (layer == 1 ? 16 : 0) + BC;
    const double g0 = __shfl_sync(0xffffffffu, g[0], src), g1 = __shfl_sync(0xffffffffu, g[1], src);
    const double g2 = __shfl_sync(0xffffffffu, g[2], src), g3 = __shfl_sync(0xffffffffu, g[3], src);
    const double g4 = __shfl_sync(0xffffffffu, g[0], src + 1);
    if (layer == 0 || layer == 1) {
      keep[0] = g0;
      keep[1] = g1;
      keep[2] = g2;
      keep[3] = g3;
      keep[4] = g4;
    }
  }
  in.r1 = keep[0];
  in.mx1 = keep[1];
  in.my1 = keep[2];
  in.E1 = keep[3];
  in.r2 = keep[4];
  in.rw = __shfl_sync(0xffffffffu, keep[0], lane - 1 & 31);  // (x = 0 is lane 31)
  in.re = __shfl_sync(0xffffffffu, keep[0], lane + 1 & 31);
  if (mw && x == BC) in.rw = keep[0];  // mirror image of the column itself
  if (me && x == f.nx - BC - 1) in.re = keep[0];
  if (!mine) return;
  const int gt = x == 0 ? WG_L0 : (x == f.nx - 1 ? WG_R0 : WG_CENTRED);
  unsigned int st = 0;
  const WallOut o =
      wall_column(in, gt, wall_heat_flux(a.wall, a.xmap0 + x * a.dx), a.wc, &st);
  if (st) atomicOr(a.status, st);
  double* u = a.uout + x;
  u[P] = o.r;
  u[0] = o.r0;
  u[V + P] = o.mx;
  u[2 * V + P] = o.my;
  // the corners of a mirror side
  int d = 0;
  if (mw && x < 2 * BC) d = 2 * BC - 1 - 2 * x;
  else if (me && x >= f.nx - 2 * BC) d = 2 * (f.nx - BC) - 1 - 2 * x;
  if (d) {
    u[P + d] = o.r;
    u[d] = o.r0;
    u[V + P + d] = -o.mx;
    u[2 * V + P + d] = o.my;
  }
}

// What a launch does beside its strips, in its first CTAs: nothing, the
// ghost runs of open sections, or wall runs and then ghost runs.
enum StripEdges : int { E_NONE = 0, E_OPEN = 1, E_WALL = 2 };

// CTA number b of one field (one warp per CTA): its edge_ctas edge runs, then
// its strips, sx per band of h rows, x fastest.
template <int MODE, int UN, int EDGES, bool MIX, bool BATCH = false>
__device__ __forceinline__ void strip_cta(const StageArgs& a, int b, int edge_ctas, int sx, int h) {
  constexpr bool WALLS = MODE == 1 && EDGES == E_WALL;
  bool wall = false;
  if (EDGES && b < edge_ctas) {
    if (WALLS) wall = b < a.wall_runs;
    if (!wall) {
      open_run<MODE>(a, b - (WALLS ? a.wall_runs : 0));
      return;
    }
  } else {
    b -= edge_ctas;
  }
  // MODE 2 (buffer-layer grid): strips over the border box, the first one
  // starting at an even column so that the rows' 16-byte pairs stay aligned
  int c0 = (MODE >= 2 ? (a.box_x0 & ~1) : BC) + (b % sx) * SW;
  int y0 = (MODE >= 2 ? a.box_y0 : BC) + (b / sx) * h;
  const int ylast = MODE >= 2 ? a.box_y1 : a.f.ny - BC - 1;
  int y1 = min(y0 + h, ylast + 1);
  // Every strip has a row and a column.  The test makes a warp compute its place
  // before it waits for the launch before; without it that moves behind the wait:
  // 128^2 periodic 8.97 us per step, 8.46 so, 512^2 wall 25.58, 25.36.  (Not in
  // batches, which look their domain up before and have no registers for it.)
  auto some = [&]() { return BATCH || (c0 < a.f.nx && y0 < y1); };
  if (WALLS) {
    const WallRun run(a, b);
    if (wall) {
      c0 = run.c0;
      y0 = BC;
      y1 = BC + 2;
    }
    if (some()) strip_warp<MODE, UN, MIX, true>(a, c0, y0, y1, wall);
    if (wall) wall_columns(a, run);
  } else {
    if (some()) strip_warp<MODE, UN, MIX>(a, c0, y0, y1);
  }
}

template <int MODE, int UN, int EDGES, bool MIX>
__global__ void __launch_bounds__(32, WARPS) k_strip(const __grid_constant__ StageArgs a,
                                                    int edge_ctas, int sx, int h) {
  int b = blockIdx.x;
  if (a.reverse && b >= edge_ctas) b = edge_ctas + (int)gridDim.x - 1 - b;
  strip_cta<MODE, UN, EDGES, MIX>(a, b, edge_ctas, sx, h);
}

// ghost runs alone (launch_stage_work: the corner cells of an untuned open field)
template <int MODE>
__global__ void __launch_bounds__(32) k_open_runs(const __grid_constant__ StageArgs a) {
  let_dependents_start();
  open_run<MODE>(a, blockIdx.x);
}

// stage arguments of domain i of a batched launch
template <bool MIX>
__device__ __forceinline__ StageArgs batch_stage_args(const BatchStageArgs& P, int i) {
  const BatchDomain& d = P.d[i];
  StageArgs a;
  a.uin = d.uin;
  a.u0 = d.u0;
  a.uout = d.uout;
  a.f = d.f;
  a.dx = d.dx;
  a.dy = d.dy;
  a.rdx = d.rdx;
  a.rdy = d.rdy;
  a.dt = d.dt;
  a.b = P.b;
  a.stage = P.stage;
  a.periodic = d.periodic;
  a.wall_s = d.wall_s;
  a.variant = 0;
  a.open = d.open;
  a.mirror = d.mirror;
  a.wall_runs = d.wall_runs;
  a.status = d.status;
  a.wc = d.wc;
  a.reverse = 0;
  a.mixed = 0;
  a.xmap0 = d.xmap0;
  a.wall = P.wall;
  a.k = P.k;
  a.c = d.c;
  if (MIX) a.cf = d.cf;
  return a;
}

// last domain i in [0, n) whose first CTA (edge0 or strip0) is <= b
template <bool EDGES>
__device__ __forceinline__ int batch_domain(const BatchStageArgs& P, int b) {
  int lo = 0, hi = P.ndom - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    const int first = EDGES ? P.d[mid].edge0 : P.d[mid].strip0;
    if (first <= b) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// One RK stage of every domain of a batch (one boundary kind): the edge runs of
// all domains first, then every domain's strips.
template <int UN, int EDGES, bool MIX>
__global__ void __launch_bounds__(32, WARPS)
    k_strip_batch(const __grid_constant__ BatchStageArgs P, int h) {
  int b = blockIdx.x;
  const bool edge = EDGES && b < P.edge_ctas;
  if (!edge) b -= P.edge_ctas;
  const int i = edge ? batch_domain<true>(P, b) : batch_domain<false>(P, b);
  const StageArgs a = batch_stage_args<MIX>(P, i);
  const BatchDomain& d = P.d[i];
  // its edge runs are numbered from 0, its strips from edge_ctas
  strip_cta<1, UN, EDGES, MIX, true>(a, edge ? b - d.edge0 : P.edge_ctas + b - d.strip0,
                                     P.edge_ctas, d.sx, h);
}

// ---- persistent batched kernel -----------------------------------------
// Item it of a launch is item it % items_per_step of the per-step table, in
// step it / items_per_step.  Buffer roles of step k (A = buf[0] holds u^n at
// launch, B = buf[1]): u^n = A on even steps and B on odd steps, the other
// one of the pair takes stages 1 and 3, C takes stage 2 -- the A/B swap of
// rk3_step, step after step.
constexpr int PW = 2;  // warps per CTA of the persistent kernel

__device__ __forceinline__ unsigned long long load_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long load_relaxed(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void fence_acquire() {
  asm volatile("fence.acq_rel.gpu;" ::: "memory");
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// wait until done >= target (every lane loads with acquire semantics);
// false if the launch was stopped or the wait ran out (which stops it)
__device__ bool wait_done(const PersistArgs& P, const unsigned long long* done,
                          unsigned long long target) {
  if (load_acquire(done) >= target) return true;
  const unsigned long long t0 = global_ns();
  unsigned ns = 64;
  // the iteration cap (a few seconds of 2 us sleeps) bounds the wait even
  // if the timer stalled
  for (int it = 0; it < (1 << 21); it++) {
    __nanosleep(ns);
    if (ns < 2048) ns *= 2;
    if (load_acquire(done) >= target) return true;
    if (*(volatile unsigned int*)&P.ctl[0]) return false;
    if (global_ns() - t0 > P.wait_ns) break;
  }
  atomicOr(&P.ctl[1], 1u);
  atomicExch(&P.ctl[0], 1u);
  return false;
}

// Stage arguments of an item, built by the warp in shared memory: strips and
// ghost runs read them from there as they need them.  In registers, and with
// 16 warps per SM, they spilled 500 bytes in the strips' loop (64-domain FP64
// batch 1235 us per step); from shared memory 912 at 16 warps (144 bytes), 651
// at 12 (158 registers, none).
template <bool MIX>
__device__ __forceinline__ void persist_stage_args(const PersistArgs& P, const PDomain& d,
                                                   int step, int st, StageArgs& a) {
  __syncwarp();  // the warp is done with its item before
  const int lane = threadIdx.x & 31;
  constexpr int NC = sizeof(StripCoef<double>) / sizeof(double);
  if (lane < NC) {
    reinterpret_cast<double*>(&a.c)[lane] = reinterpret_cast<const double*>(&d.c)[lane];
    if (MIX) reinterpret_cast<float*>(&a.cf)[lane] = reinterpret_cast<const float*>(&d.cf)[lane];
  }
  const int odd = (P.step0 + step) & 1;
  double* X = odd ? d.buf[1] : d.buf[0];  // u^n
  double* Y = odd ? d.buf[0] : d.buf[1];
  if (lane == 0) {
    a.uin = st == 1 ? X : (st == 2 ? Y : d.buf[2]);
    a.u0 = X;
    a.uout = st == 2 ? d.buf[2] : Y;
    a.f = d.f;
    a.dx = d.dx;
    a.dy = d.dy;
    a.rdx = d.rdx;
    a.rdy = d.rdy;
    a.dt = d.dt * P.dt_scale;
    a.b = st == 2 ? 0.75 : (st == 3 ? 1.0 / 3.0 : 0.0);  // rk3tvd_steps_module.f:225,444
    a.stage = st;
    a.periodic = d.periodic;
    a.wall_s = d.wall_s;
    a.open = d.open;
    a.xmap0 = d.xmap0;
    a.mirror = a.wall_runs = 0;  // its node items
    a.reverse = 0;
    a.wall = P.wall;
    a.k = P.k;
  }
  __syncwarp();
}

__device__ __forceinline__ NodeBcArgs persist_node_args(const PersistArgs& P, const PDomain& d,
                                                        int step, int st) {
  const int odd = (P.step0 + step) & 1;
  double* X = odd ? d.buf[1] : d.buf[0];
  double* Y = odd ? d.buf[0] : d.buf[1];
  NodeBcArgs a;
  a.utmp = X;
  a.u = st == 2 ? d.buf[2] : Y;
  a.f = d.f;
  a.dx = d.dx;
  a.dy = d.dy;
  a.rdx = d.rdx;
  a.rdy = d.rdy;
  a.xmap0 = d.xmap0;
  a.south_wall = d.south_wall;
  a.corners_y = d.corners_y;
  a.open_w = d.open_w;
  a.open_e = d.open_e;
  a.open_n = d.open_n;
  a.status = d.status;
  a.wall = P.wall;
  a.k = P.k;
  return a;
}

// wait until band b of domain d has completed `inst` stage-instances
__device__ __forceinline__ bool wait_band(const PersistArgs& P, const PDomain& d, int b,
                                          unsigned long long inst) {
  return wait_done(P, P.done + d.band0 + b, inst * (unsigned long long)P.sg[d.band0 + b]);
}

template <bool MIX>
__global__ void __launch_bounds__(32 * PW, 6) k_batch_persistent(const __grid_constant__ PersistArgs P) {
  const int lane = threadIdx.x & 31;
  const unsigned long long total = (unsigned long long)P.items_per_step * P.nsteps;
  __shared__ StageArgs args[PW];
  StageArgs& a = args[threadIdx.x >> 5];
  for (;;) {
    unsigned long long it = 0;
    if (lane == 0) it = atomicAdd(P.next, 1ull);
    it = __shfl_sync(0xffffffffu, it, 0);
    if (it >= total || *(volatile unsigned int*)&P.ctl[0]) break;
    const int step = (int)(it / (unsigned long long)P.items_per_step);
    const PItem item = P.items[it % (unsigned long long)P.items_per_step];
    const PDomain& d = P.dom[item.dom];
    // stage-instances (3 per step) that precede this item's stage
    const unsigned long long inst = 3ull * (unsigned long long)step + (unsigned long long)(item.stage - 1);
    // Every lane checks the counters the item depends on: the counters read
    // together with relaxed loads and, if they are all ready (the usual
    // case), one acquire fence (the acquire pattern: strong reads, then
    // fence.acq_rel) -- one round trip; otherwise bounded waits, one counter
    // at a time.  (Lane 0 checking alone and the warp barrier passing the
    // order on measured 1.5x slower: divergent lanes wait on its branch.)
    // Strips that read no ghost cell of the node pass skip its wait
    // (`count` flags those that do).
    bool ok = true;
    if (item.type == PI_NODE) {
      for (int b = 0; b < d.nb && ok; b++) ok = wait_band(P, d, b, inst + 1);
    } else {
      const bool need_node = d.nn && (item.type != PI_STRIP || item.count);
      int bands[3];
      for (int o = -1; o <= 1; o++) {
        int bb = item.band + o;
        if (bb < 0 || bb >= d.nb) bb = d.periodic ? (bb + d.nb) % d.nb : item.band;
        bands[o + 1] = bb;
      }
      const unsigned long long c0 = load_relaxed(P.done + d.band0 + bands[0]);
      const unsigned long long c1 = load_relaxed(P.done + d.band0 + bands[1]);
      const unsigned long long c2 = load_relaxed(P.done + d.band0 + bands[2]);
      const unsigned long long cn = need_node ? load_relaxed(P.ndone + item.dom) : 0ull;
      const bool ready = c0 >= inst * (unsigned long long)P.sg[d.band0 + bands[0]] &&
                         c1 >= inst * (unsigned long long)P.sg[d.band0 + bands[1]] &&
                         c2 >= inst * (unsigned long long)P.sg[d.band0 + bands[2]] &&
                         cn >= (need_node ? inst * (unsigned long long)d.nn : 0ull);
      if (ready) {
        fence_acquire();
      } else {
        for (int o = 0; o < 3 && ok; o++) ok = wait_band(P, d, bands[o], inst);
        if (ok && need_node)
          ok = wait_done(P, P.ndone + item.dom, inst * (unsigned long long)d.nn);
      }
    }
    // a wait that ran out stops the warp (the launch is aborted)
    if (!__all_sync(0xffffffffu, ok)) break;
    if (item.type == PI_STRIP) {
      persist_stage_args<MIX>(P, d, step, item.stage, a);
      const int c0 = BC + (item.index % d.sx) * SW;
      const int y0 = BC + item.band * P.h_rows;
      // the last band runs to the last interior row (it absorbs a remainder
      // of fewer than 2 rows, so that the rows a periodic field images into
      // the opposite ghost rows never span two bands)
      const int y1 = item.band == d.nb - 1 ? d.f.ny - BC : y0 + P.h_rows;
      strip_warp<1, 2, MIX>(a, c0, y0, y1);
    } else if (item.type == PI_GHOST) {
      persist_stage_args<false>(P, d, step, item.stage, a);
      const int side = item.index >> 24;
      if (side < 4)
        open_edge_run<1>(a, side, item.index >> 20 & 1, item.index & 0xfffff, item.count);
      else open_corner_cells<1>(a, item.count);
    } else {
      node_bc_cell(persist_node_args(P, d, step, item.stage), item.index * 32 + lane);
    }
    // release: the warp barrier orders every lane's stores before lane 0,
    // whose fence (cumulative) precedes the counter increment.  The
    // counter's address is looked up again from the item table rather than
    // kept live across the work.
    __syncwarp();
    if (lane == 0 && (long long)it != P.withhold) {
      __threadfence();
      const PItem& done_item = P.items[it % (unsigned long long)P.items_per_step];
      atomicAdd(done_item.type == PI_NODE
                    ? P.ndone + done_item.dom
                    : P.done + P.dom[done_item.dom].band0 + done_item.band,
                1ull);
    }
  }
}

// launch of one-warp CTAs with their rings
inline cudaError_t launch_strips(const void* fn, unsigned blocks, cudaStream_t s, void** args) {
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                       cudaSharedmemCarveoutMaxShared);
  if (e != cudaSuccess) return e;
  return launch_dependent(fn, blocks, 32, WARP_DOUBLES * sizeof(double), s, args);
}

// rows per strip of shape 0..4
constexpr int SHAPE_ROWS[5] = {8, 16, 32, 4, 2};
// Rows per strip by size: as few as still let every strip of the launch be
// resident at once (148 SMs x 16 warps), since a stage then lasts as long as
// one strip; 16 where even those do not fit (more rows leave the last wave
// emptier, fewer repeat the two rows below a strip more often).  us per step:
//   rows                       by size    2      4      8      16
//   64^2 open                   8.5 (1)    8.3   10.1   14.9   24.3
//   128^2 periodic              8.5 (1)   10.0   13.6   21.2   36.3
//   301x187 half_wall_S_open   21.8 (2)   20.7   20.4   22.2   36.6
//   512^2 wall_S_reflection    25.1 (4)   29.8   25.1   27.1   38.8
//   1024^2 open                66.2 (16)  88.4   73.9   68.2   67.2
//   1531x1117 periodic         109 (16)   140    115    108    110
//   2048^2 open                230 (16)   335    272    251    232
template <typename Strips>
int rows_of(int shape, Strips strips) {
  if (shape != SHAPE_BY_SIZE) return SHAPE_ROWS[shape];
  int h = 1;
  while (h < 16 && strips(h) > 148LL * WARPS) h *= 2;
  return h;
}
template <int UN, bool MIX>
const void* stage_fn(int edges) {
  return edges == E_WALL   ? (const void*)k_strip<1, UN, E_WALL, MIX>
         : edges == E_OPEN ? (const void*)k_strip<1, UN, E_OPEN, MIX>
                           : (const void*)k_strip<1, UN, E_NONE, MIX>;
}
template <bool MIX>
const void* strip_fn(int mode, bool un, int edges) {
  if (mode == 0)
    return edges ? (const void*)k_strip<0, 0, E_OPEN, MIX> : (const void*)k_strip<0, 0, E_NONE, MIX>;
  return un ? stage_fn<1, MIX>(edges) : stage_fn<0, MIX>(edges);
}

int strips_across(const Field& f) { return (f.nx - 2 * BC + SW - 1) / SW; }
int strips_up(const Field& f, int h) { return (f.ny - 2 * BC + h - 1) / h; }

template <int UN, bool MIX>
const void* strip_batch_fn(int kind) {
  return kind == BK_WALL   ? (const void*)k_strip_batch<UN, E_WALL, MIX>
         : kind == BK_OPEN ? (const void*)k_strip_batch<UN, E_OPEN, MIX>
                           : (const void*)k_strip_batch<UN, E_NONE, MIX>;
}

}  // namespace

cudaError_t launch_batch_persistent(const PersistArgs& P, bool mixed, cudaStream_t s, int* ctas) {
  const void* fn = mixed ? (const void*)k_batch_persistent<true> : (const void*)k_batch_persistent<false>;
  int dev = 0, sms = 0, per_sm = 0;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                                       cudaSharedmemCarveoutMaxShared);
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const size_t smem = (size_t)PW * WARP_DOUBLES * sizeof(double);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, 32 * PW, smem);
  if (e != cudaSuccess) return e;
  const int n = sms * (per_sm > 0 ? per_sm : 1);
  if (ctas) *ctas = n;
  PersistArgs pa = P;
  void* args[] = {&pa};
  return cudaLaunchKernel(fn, dim3((unsigned)n), dim3(32 * PW), args, smem, s);
}

cudaError_t launch_strip_batch(BatchStageArgs& P, int kind, int shape, bool mixed,
                               cudaStream_t s) {
  if (P.ndom <= 0) return cudaSuccess;
  if (P.ndom > BATCH_MAX || shape < SHAPE_BY_SIZE || shape > 4) return cudaErrorInvalidValue;
  int h = rows_of(shape, [&](int rows) {
    long long n = 0;
    for (int i = 0; i < P.ndom; i++)
      n += (long long)strips_across(P.d[i].f) * strips_up(P.d[i].f, rows);
    return n;
  });
  long long ghost = 0, strips = 0;
  for (int i = 0; i < P.ndom; i++) {
    BatchDomain& d = P.d[i];
    d.sx = strips_across(d.f);
    d.edge0 = (int)ghost;
    d.strip0 = (int)strips;
    if (kind != BK_PLAIN) ghost += d.wall_runs + open_run_count(d.f, d.open);
    strips += (long long)d.sx * strips_up(d.f, h);
  }
  if (ghost + strips > 0x7fffffffLL) return cudaErrorInvalidValue;
  P.edge_ctas = (int)ghost;
  const void* fn = P.stage != 1 ? (mixed ? strip_batch_fn<1, true>(kind) : strip_batch_fn<1, false>(kind))
                                : (mixed ? strip_batch_fn<0, true>(kind) : strip_batch_fn<0, false>(kind));
  void* args[] = {&P, &h};
  return launch_strips(fn, (unsigned)(ghost + strips), s, args);
}

// L(u) of a buffer-layer grid at its interior_pt points (MODE 2) over the
// border box [box_x0, box_x1] x [box_y0, box_y1] (box_x0, box_y0 >= BC, so
// every row and column read lies inside the grid).  MODE 3 where the layout
// does not suit the rows' 16-byte copies (odd nx; 14.4 us on 2047 x 256 and
// 6.2 us on 1001 x 100, where the tile kernel before it took 26.8 and 8.2; the
// 16-byte form takes 12.0 us on 2048 x 256).
cudaError_t launch_strip_masked(const StageArgs& a, cudaStream_t s) {
  int sx = (a.box_x1 - (a.box_x0 & ~1) + SW) / SW;
  const int rows = a.box_y1 - a.box_y0 + 1;
  int h = rows_of(SHAPE_BY_SIZE, [&](int r) { return (long long)sx * ((rows + r - 1) / r); });
  int edge_ctas = 0;
  StageArgs aa = a;
  void* args[] = {&aa, &edge_ctas, &sx, &h};
  const unsigned blocks = (unsigned)sx * (unsigned)((rows + h - 1) / h);
  if (strip_layout_ok(a))
    return launch_strips((const void*)k_strip<2, 0, E_NONE, false>, blocks, s, args);
  return cudaLaunchKernel((const void*)k_strip<3, 0, E_NONE, false>, dim3(blocks), dim3(32), args,
                          WARP_DOUBLES * sizeof(double), s);
}

cudaError_t launch_strip_stage(const StageArgs& a, int mode, int shape, cudaStream_t s) {
  if (shape < SHAPE_BY_SIZE || shape > 4) return cudaErrorInvalidValue;
  int sx = strips_across(a.f);
  int h = rows_of(shape, [&](int rows) { return (long long)sx * strips_up(a.f, rows); });
  const int walls = mode == 1 ? a.wall_runs : 0;
  int edge_ctas = walls + open_run_count(a.f, a.open);
  const int edges = walls ? E_WALL : (edge_ctas ? E_OPEN : E_NONE);
  const void* fn = a.mixed ? strip_fn<true>(mode, a.stage != 1, edges)
                           : strip_fn<false>(mode, a.stage != 1, edges);
  StageArgs aa = a;
  void* args[] = {&aa, &edge_ctas, &sx, &h};
  return launch_strips(fn, (unsigned)edge_ctas + (unsigned)sx * (unsigned)strips_up(a.f, h), s,
                       args);
}

cudaError_t launch_open_runs(const StageArgs& a, int mode, cudaStream_t s) {
  const unsigned n = (unsigned)open_run_count(a.f, a.open);
  StageArgs aa = a;
  void* args[] = {&aa};
  return launch_dependent(mode == 0 ? (const void*)k_open_runs<0> : (const void*)k_open_runs<1>, n,
                          32, 0, s, args);
}

}  // namespace dim2d
