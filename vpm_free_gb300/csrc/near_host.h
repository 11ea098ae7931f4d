// near_host.h -- plan of the near field's tables (near_host.cpp) and the
// weight formula that the tables hold, shared by host and device code.
#pragma once
#include <cmath>
#include <vector>

#ifdef __CUDACC__
#define VPMG_HD __host__ __device__ __forceinline__
#else
#define VPMG_HD inline
#endif

namespace vpmg {

constexpr int kNearLevels = 8;
constexpr int kNearDigits = 7, kNearCols = 64;

struct NearTable {           // one level and kind of face pair
  int s, top, par;           // panels per cell side; coarsest level; parallel (1) or perpendicular (0) faces
  int TB, rows;              // a node block: TB nodes along w times `rows`
  int w0, nkp;               // window along w: first cell (from the block's first), blocks of 16 cells
  int r0, nrow, nchunk;      // cell rows, tiles of 64 nodes
  int dn;                    // parallel: the faces' distance in nodes
  double hw, hr, hn;         // spacings along w, across it in the source face, and along the source normal
  double ds, thr2_own, thr2_out;  // cell area; squared opening radii of the level and of its parents
};
struct NearRow {             // one run of target nodes: where its sources are and its sums go
  long long abase, obase;    // first digit of its component's lines; sum of the block's node (0, 0)
  int row0, rs, nrow, wst, Wp;         // source row of table row 0, step, rows; first window cell; line length
  int ostr_r, ostr_w, rlim, wlim;      // strides of the sums along the block's rows and w; nodes that exist
};
struct NearPlan {
  int cell0[kNearLevels][7], ma[kNearLevels][6], mb[kNearLevels][6], Wp[kNearLevels][2][6];
  long long dbase[kNearLevels][2][6], abase[6];
  long long ndig = 0, nacc = 0;
  int edge = 0;
  std::vector<NearTable> tabs;
  std::vector<std::vector<NearRow>> runs;
};
// false where the cells of some level are not a uniform lattice on every face
bool build_near_plan(const int n3[3], const double d3[3], int L, NearPlan& P);

// Whether the rounded coordinates of nodes and leaf centres are those of the
// lattice closely enough for the lattice's weights to stand for the walk's: a
// leaf centre is h / sqrt 2 or more from a node, so offsets that are off by 4e-11 h
// along each axis change a weight by less than 1e-10 of it.  An origin further
// than some 2e5 spacings from zero fails (unless its nodes are exact).
bool lattice_exact(const double xmin[3], const double d[3], const int n[3]);

// in-plane axes of face f (normal f / 2): the panels' fast and slow axes
VPMG_HD int face_u(int f) { return (f >> 1) == 0 ? 1 : 0; }
VPMG_HD int face_v(int f) { return (f >> 1) == 2 ? 1 : 2; }
VPMG_HD int floor_half(int c) { return (c >= 0 ? c : c - 1) / 2; }
VPMG_HD double near_area(const double d3[3], int l, int fn) {  // of a level-l cell of a face with normal fn
  return (d3[face_u(2 * fn)] * (double)(1 << l)) * (d3[face_v(2 * fn)] * (double)(1 << l));
}
VPMG_HD double near_thr2(const double d3[3], int l, int fn) { return 100.0 * near_area(d3, l, fn); }

// Sums and products rounded one by one (host code is compiled without
// contraction), so that every user decides alike.
VPMG_HD double rn_mul(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dmul_rn(a, b);
#else
  return a * b;
#endif
}
VPMG_HD double rn_add(double a, double b) {
#ifdef __CUDA_ARCH__
  return __dadd_rn(a, b);
#else
  return a + b;
#endif
}
// r^2 of an offset in nodes along the source face's two axes and its normal.
VPMG_HD double lattice_r2(double a, double ha, double b, double hb, double n, double hn) {
  const double x = rn_mul(a, ha), y = rn_mul(b, hb), z = rn_mul(n, hn);
  return rn_add(rn_add(rn_mul(x, x), rn_mul(y, y)), rn_mul(z, z));
}
VPMG_HD double lattice_weight(double ds, double r2) {
#ifdef __CUDA_ARCH__
  return r2 > 0.0 ? __ddiv_rn(ds, __dsqrt_rn(r2)) : 0.0;
#else
  return r2 > 0.0 ? ds / std::sqrt(r2) : 0.0;
#endif
}

// Whether an offset in nodes lies within 1e-5 of length, where the reference
// takes a cell's potential at its own centre (tree_calc_3d, source/pmbound.f90:980-1249).
// The squares are added by size, so that every order of the axes decides alike.
VPMG_HD bool lattice_close(double a, double ha, double b, double hb, double n, double hn) {
  const double x = rn_mul(a, ha), y = rn_mul(b, hb), z = rn_mul(n, hn);
  const double u = rn_mul(x, x), v = rn_mul(y, y), w = rn_mul(z, z);
  const double lo = u < v ? u : v, hi = u < v ? v : u;
  const double mid = w < lo ? lo : (w < hi ? w : hi);
  const double r2 = rn_add(rn_add(w < lo ? w : lo, mid), w < hi ? hi : w);
#ifdef __CUDA_ARCH__
  return !(__dsqrt_rn(r2) > 1e-05);
#else
  return !(std::sqrt(r2) > 1e-05);
#endif
}
// log((sqrt 2 - 1) / (sqrt 2 + 1)): a square panel of area dS has the potential
// -2 sqrt(dS) times it at its centre
constexpr double kPanelLog = -1.7627471740390861;
// Weight of a cell of area ds at an offset: ds / r, within 1e-5 the panel's own
// potential, 0 at the cell's centre (such a cell is always opened).
VPMG_HD double lattice_weight(double ds, double a, double ha, double b, double hb, double n, double hn) {
  const double r2 = lattice_r2(a, ha, b, hb, n, hn);
  if (r2 > 0.0 && r2 < 1.01e-10 && lattice_close(a, ha, b, hb, n, hn)) {
#ifdef __CUDA_ARCH__
    return rn_mul(rn_mul(-2.0, __dsqrt_rn(ds)), kPanelLog);
#else
    return -2.0 * std::sqrt(ds) * kPanelLog;
#endif
  }
  return lattice_weight(ds, r2);
}

// Weight of (column, row, cell) of a table.
VPMG_HD double near_weight(const NearTable& T, int n, int row, int cell) {
  const int tr = n / T.TB, tw = n - tr * T.TB;
  if (tr >= T.rows) return 0.0;
  const double s = (double)T.s;
  const int cw = T.w0 + cell, cr = T.par ? T.r0 + row : row;
  const double ow = s * ((double)cw + 0.5) - (double)tw;
  const double orr = T.par ? s * ((double)cr + 0.5) - (double)tr : s * ((double)cr + 0.5);
  const double on = T.par ? (double)T.dn : (double)tr;
  const double r2 = lattice_r2(ow, T.hw, orr, T.hr, on, T.hn);
  if (T.top) return r2 < T.thr2_own ? -lattice_weight(T.ds, ow, T.hw, orr, T.hr, on, T.hn) : 0.0;
  const double pw = 2.0 * s * ((double)floor_half(cw) + 0.5) - (double)tw;
  const double pc = 2.0 * s * ((double)floor_half(cr) + 0.5);
  const double pr = T.par ? pc - (double)tr : pc;
  if (!(lattice_r2(pw, T.hw, pr, T.hr, on, T.hn) < T.thr2_out)) return 0.0;
  if (T.s > 1 && r2 < T.thr2_own) return 0.0;
  return lattice_weight(T.ds, ow, T.hw, orr, T.hr, on, T.hn);
}

}  // namespace vpmg
