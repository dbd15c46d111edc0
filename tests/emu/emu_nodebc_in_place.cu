// Host emulation of the node boundary kernel in place (nodes_tmp = nodes, as
// after an upload): node_bc_cell() for every thread index in the order the
// program is given (0 ascending, 1 descending).  A read of a value that another
// thread index writes counts as a race, whichever comes first.
// Used by tests/test_nodebc_in_place.py.
#include <cstdio>
#include <cstdlib>
#include <set>
#include <utility>
#include <vector>
static double *g_lo, *g_hi;
static long g_bad = 0, g_cur = 0;
static std::vector<long> g_writer;
static std::set<std::pair<long, long>> g_reads;  // cell, reader
static inline double chk(const double* p) {
  if (p < g_lo || p >= g_hi) {
    g_bad++;
    return 0.0;
  }
  g_reads.insert({p - g_lo, g_cur});
  return *p;
}
static inline void emu_store(double* p, double v) {
  if (p < g_lo || p >= g_hi) {
    g_bad++;
    return;
  }
  if (g_writer[p - g_lo] >= 0 && g_writer[p - g_lo] != g_cur) g_bad++;
  g_writer[p - g_lo] = g_cur;
  *p = v;
}
#define DIM2D_LDG_HOST(p) chk(p)
#define DIM2D_ST_HOST(p, v) emu_store(p, v)
#include "../../dim2d_finite_volume_b200/csrc/dim2d_nodebc.cu"
using namespace dim2d;
int main(int argc, char** argv) {
  FILE* fi = fopen(argv[1], "rb");
  int hdr[8];      // nx, ny, south_wall, corners_y, open_w, open_e, open_n, order
  double par[8];   // dx, dy, re, we, pr, cv_r, cos_angle, xmap0
  if (fread(hdr, 4, 8, fi) != 8 || fread(par, 8, 8, fi) != 8) return 2;
  const size_t plane = (size_t)hdr[0] * hdr[1];
  std::vector<double> u(4 * plane);
  if (fread(u.data(), 8, 4 * plane, fi) != 4 * plane) return 2;
  fclose(fi);
  g_lo = u.data();
  g_hi = g_lo + 4 * plane;
  g_writer.assign(4 * plane, -1);
  NodeBcArgs a{};
  a.utmp = a.u = u.data();
  a.f.nx = a.f.pitch = hdr[0];
  a.f.ny = hdr[1];
  a.f.plane = plane;
  a.dx = par[0];
  a.dy = par[1];
  a.rdx = 1.0 / par[0];
  a.rdy = 1.0 / par[1];
  a.south_wall = hdr[2];
  a.corners_y = hdr[3];
  a.open_w = hdr[4];
  a.open_e = hdr[5];
  a.open_n = hdr[6];
  unsigned int status = 0;
  a.status = &status;
  a.k.re = par[2];
  a.k.we = par[3];
  a.k.pr = par[4];
  a.k.cv_r = par[5];
  a.wall.cos_angle = par[6];
  a.xmap0 = par[7];
  const int total = node_bc_count(a);
  for (int i = 0; i < total; i++) {
    g_cur = hdr[7] ? total - 1 - i : i;
    node_bc_cell(a, g_cur);
  }
  long race = 0;
  for (const auto& r : g_reads) race += g_writer[r.first] >= 0 && g_writer[r.first] != r.second;
  printf("total=%d bad=%ld race=%ld status=%u\n", total, g_bad, race, status);
  FILE* fo = fopen(argv[2], "wb");
  fwrite(u.data(), 8, 4 * plane, fo);
  fclose(fo);
  return 0;
}
