// vpmg_internal.h -- shared declarations of the sm_103a particle-mesh library.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <vector>

#include "../../include/vpmg.h"
#include "near_host.h"

namespace vpmg {

constexpr double kPI = 3.14159265358979323846264338327950288;

// ------------------------------------------------------------ errors ----
struct Error {
  int status;
  std::string msg;
};
#define VPMG_CUDA(x)                                                                      \
  do {                                                                                    \
    cudaError_t e_ = (x);                                                                 \
    if (e_ != cudaSuccess)                                                                \
      throw ::vpmg::Error{VPMG_ERR_CUDA, std::string(#x) + ": " + cudaGetErrorString(e_)}; \
  } while (0)
#define VPMG_CHECK(cond, code, text)                                  \
  do {                                                                \
    if (!(cond)) throw ::vpmg::Error{(code), std::string(text)};      \
  } while (0)

// Kernel launch counter shared by every launch site (instrumentation).
extern thread_local long long* g_launch_counter;
inline void count_launch(int n = 1) {
  if (g_launch_counter) *g_launch_counter += n;
}
#define VPMG_LAUNCHED() ::vpmg::count_launch()

// ---------------------------------------------------- device buffers ----
template <class T>
struct DBuf {
  T* p = nullptr;
  size_t n = 0;
  DBuf() = default;
  DBuf(const DBuf&) = delete;
  DBuf& operator=(const DBuf&) = delete;
  ~DBuf() { release(); }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
  void ensure(size_t count) {
    if (count <= n && p) return;
    release();
    if (count == 0) return;
    cudaError_t e = cudaMalloc(&p, count * sizeof(T));
    if (e != cudaSuccess) {
      cudaGetLastError();
      p = nullptr;
      throw Error{VPMG_ERR_NOMEM, "cudaMalloc of " + std::to_string(count * sizeof(T)) + " bytes failed"};
    }
    n = count;
  }
  size_t bytes() const { return n * sizeof(T); }
};

// A handle's device error word holds the largest of these since the last host
// sync, which turns it into a status (check_particle_errors).
enum { kErrOutside = 1, kErrCapacity = 2, kErrWait = 3 };
// Polls after which a wait inside a kernel gives up; VPMG_WAIT_POLLS sets it
// for the plans and operators made from then on.
int wait_polls();

// ------------------------------------------------------------- grids ----
// A node grid: origin, spacing and node counts (1-based node i sits at
// xmin + (i-1)*d, as everywhere in the reference).
struct Grid {
  double xmin[3], d[3];
  int n[3];
  size_t count() const { return (size_t)n[0] * n[1] * n[2]; }
};

// --------------------------------------------------- Dirichlet solver ----
// FFT plan for a DST-I of n = N-1 points.  N even: real-symmetric form,
// two real lines packed in one complex FFT of length M = N (rs = 1);
// N odd: the odd extension, complex length M = 2N (rs = 0).
struct FFTPlan {
  int n = 0, N = 0, M = 0;
  int rs = 0;
  int pairs = 4;     // line pairs per CTA of the DST kernels (tuned per plan)
  int arith = VPMG_ARITH_FP64;  // arithmetic of the transforms
  int nst = 0;
  int radix[24];
  DBuf<double2> twd; // e^{-2 pi i t / M}, t = 0..M-1, FP64
  DBuf<float4> tw;   // the same as float-float (re.hi, re.lo, im.hi, im.lo)
  DBuf<double> sn;   // sin(pi j / N), j = 0..N-1 (rs only)
};
void make_fft_plan(FFTPlan& p, int n, int arith);

// A Dirichlet box inside a node array of dims dims[3]: nodes box[0..2] to
// box[3..5] (0-based, inclusive).  Interior m[d] = box[d+3]-box[d]-1.
struct DirichletPlan {
  int dims[3] = {0, 0, 0};
  int box[6] = {0, 0, 0, 0, 0, 0};
  int m[3] = {0, 0, 0};
  double h[3] = {0, 0, 0};
  int arith = VPMG_ARITH_FP64;  // arithmetic of the transforms and sweeps
  FFTPlan fx, fy;
  // FP64 lines long and many enough: the passes as products (dst_mma.cu),
  // with the sine matrices (xf: x forward, times the solve's factor) and a
  // second array for 3 components, as those passes are not in place
  bool mma_x = false, mma_y = false;
  DBuf<unsigned char> tx, txf, ty;
  int xf_shift = 0, xf_neg = 0;
  DBuf<double> tmp;
  int polls = 0;          // of those passes' waits (wait_polls),
  int* status = nullptr;  // and the error word that one which runs out sets
  DBuf<float2> rinv;  // float-float plans: reciprocal Thomas pivots, [k][q][p], float-float pairs
  DBuf<double> rinvd; // FP64: rows 0..m2/2-1 of them and the middle's constant (thomas_sweep)
  bool ready = false;
};
void dirichlet_prepare(DirichletPlan& P, const int dims[3], const int box[6], const double h[3], cudaStream_t s,
                       int arith, int* status);
// Interior of sol <- solution of Lap_h u = rhs with the box faces of sol as
// boundary values (zero_bc = false) or zero (true; then the box faces of
// sol are zeroed).  work: >= m0*m1*m2 doubles.
// nc components in one pass: rhs and sol rcs and scs doubles apart, work
// nc * m0*m1*m2 doubles.
void dirichlet_solve(DirichletPlan& P, const double* rhs, double* sol, bool zero_bc, double* work, cudaStream_t s,
                     int nc = 1, size_t rcs = 0, size_t scs = 0);
// The z pass in FP64 (block_solve.cu): per mode (p,q) and component the
// tridiagonal system -u[k-1] + d u[k] - u[k+1] = g[k] (+ face terms), from
// g to out (may be the same array), components cs doubles apart.
struct FaceTerms {
  const double *fxs, *fxd, *fys, *fyd, *fz0, *fzN;  // transforms: [k][q], [k][p], [q][p]
  size_t cs;                                        // doubles between components
  const double *ex1, *ey1;                          // sin(pi (p+1)/(m+1)) along x and y
  double cx, cy, cz;                                // -scale / h^2
};
void thomas_launch(const double* g, double* out, const double* rinv, const int m[3], int nc, size_t cs,
                   const FaceTerms* F, cudaStream_t s);
void thomas_sweep(const double* g, double* out, const double* rinv, const int m[3], int nc, size_t cs,
                  const FaceTerms* F, cudaStream_t s);  // the same, counted
// Pieces of a partially evaluated solve (block_solve.cu).
double dirichlet_scale(const DirichletPlan& P);  // factor applied in the forward x pass
void dst_forward_xy(DirichletPlan& P, const double* rhs, const double* sol, bool zero_bc, double* ghat,
                    cudaStream_t s, int nc = 1, size_t rcs = 0, size_t scs = 0);
// data (overwritten) -> interior of the box of sol
void dst_inverse_xy(DirichletPlan& P, double* data, double* sol, cudaStream_t s, int nc, size_t scs);
// Up to 8 of the above in one launch (each job with its own plan and arrays;
// the plans share one arithmetic).  Results equal the single launches'.
struct DstYLines {
  const FFTPlan* plan;
  double* data;
  int m0, m1, m2;
  size_t cs;  // doubles between the nc components
};
void dst_lines_y_jobs(const DstYLines* jobs, int n, cudaStream_t s, int nc);
struct DstXInvLines {
  const FFTPlan* plan;
  const double* data;
  double* sol;
  int dims[3], o[3], m[3];
  size_t wcs, scs;
};
void dst_x_inv_jobs(const DstXInvLines* jobs, int n, cudaStream_t s, int nc);

// ------------------------------------------------- boundary operator ----
struct TreeGeom;  // host-built quadtree of one grid (tree_host.cpp)
// Frame of one boundary plane for the constant-source panel potential
// (FSOUR_A4): unit vectors E1..E3, corner offsets S/T, side lengths D,
// diagonal and area of one cell of that plane.
struct PanelFrame {
  double E1[3], E2[3], E3[3], S[4], T[4], D[4], diag, area;
};

// The coarsest tree level of an operator on uniform lattices evaluated as
// convolutions on them (farfield.cu).  Every target sums every coarsest cell
// (the opened ones included) by FFTs: between parallel faces a 2-D
// convolution, between perpendicular faces a 1-D convolution along their
// shared axis and a dense sum over the other two; the tables below take the
// cells each target opened back out.
struct FarFieldAxis {    // complex FFT of length P = 2^a 3^b along one axis
  int P = 0, nst = 0, npair = 1;
  int radix[16];
  DBuf<double2> tw;      // e^{-2 pi i t / P}
};
struct FarField {
  bool on = false;
  int istep = 0;                      // panels per coarsest cell side
  int N[3] = {0, 0, 0};               // grid nodes per axis
  double h[3] = {0, 0, 0};            // grid spacing per axis
  double dS[6] = {0, 0, 0, 0, 0, 0};  // area of a coarsest cell of each face
  int cell0[6] = {0, 0, 0, 0, 0, 0};  // first coarsest cell of each face (within the level)
  FarFieldAxis ax[3];
  long long kpar_off[3][2] = {{0, 0}, {0, 0}, {0, 0}};  // [normal axis][same face, opposite face]
  long long kperp_off[24] = {};       // [target face * 4 + perpendicular source slot]
  long long t_off[6][2] = {}, s2_off[6][2] = {}, sw_off[6][2] = {}, z_off[6][2] = {};
  DBuf<double> kpar, kperp;           // kernel spectra (real), the inverse scalings folded in
  DBuf<double2> T, S2, X, Sw, Z;      // transform work arrays
  double flops = 0.0;                 // FP64 flops of one apply (FFTs 5 P log2 P per line, products, sums)
  long long ncorr = 0;                // correction rows: cells the walk and the lattice rule take differently
  DBuf<long long> crow;               // six pointers per boundary node (its rows by source face)
  DBuf<int> ccol;
  DBuf<double> cw;
  long long bytes() const;
};

// The opened cells by weight tables on the tensor cores (nearfield.cu).
struct NearUnit {            // a tile of 128 runs x 64 nodes over stages k0..k1 of a list
  long long table;
  int row0, nrun, klist, k0, k1, col0, TB, q, sh;
};
struct NearField {
  bool on = false;
  int cell0[kNearLevels][7], ma[kNearLevels][6], mb[kNearLevels][6], Wp[kNearLevels][2][6];
  long long dbase[kNearLevels][2][6], abase[6];
  long long nacc = 0, stages = 0;   // sums; K = 16 products of one apply (tiles of 128 x 64, 28 digit pairs)
  int edge = 0, group = 0, uc = 0, nunit = 0, sms = 0, polls = 0;
  DBuf<unsigned char> table;
  DBuf<unsigned short> dig;
  DBuf<unsigned long long> acc;
  DBuf<NearRow> rows;
  DBuf<NearUnit> units;
  DBuf<unsigned> klist;
  long long bytes() const;
};

// A cell of the tree walk, in the walk's order.
struct alignas(16) WalkNode {
  double x, y, z, ds;
  long long open2;  // opened where the bits of d^2 are below this
  int cell;         // flat cell
  int skip;         // the next cell when this one is not opened; sign: a coarsest cell
};

struct BoundaryOp {
  // panels (level 0) and aggregated levels, device copies
  int nbound = 0, levmax = 0, ncell_total = 0, ntarget = 0;
  int ibctyp = 2;     // 2: point sources -dS/(4 pi r); 3: constant-source panels
  int arith = VPMG_ARITH_FP64;  // recorded weights and their products: FP64 or float-float
  bool tree = true;   // Bounds3d_lev (tree) or the untreed Bounds3d
  PanelFrame frame[6];                  // ibctyp 3: one per target plane
  std::vector<int> lev_off;    // flat offset of each level's cells
  std::vector<int> nbound_lev; // cumulative cells per level (all faces)
  DBuf<double> cx, cy, cz, cds, cthr;   // per flat cell: centre, area, 10*sqrt(ds)
  DBuf<int> child;                      // per flat cell: 4 flat child ids (-1 unused)
  DBuf<int> flags;                      // per flat cell: ilev_t(.,.,6)
  DBuf<int> agg_leaf0;                  // per flat cell: first leaf (flat) or -1 (dummy)
  DBuf<int> agg_rowlen;                 // per flat cell: fast-axis leaf count of its face
  DBuf<int> agg_istep;
  DBuf<int> anc;                        // [(lev-1)*nbound + leaf]: flat ancestor cell or -1
  DBuf<double> csrc;                    // 3 * ncell_total aggregated sources
  DBuf<float2> csrc_ff;                 // the same packed [cell][s0 s1 s2 0] in 8-byte words (doubles or float-float pairs)
  DBuf<unsigned> smax;                  // per component: high word of the largest panel source's magnitude
  long long budget = 0;                 // bytes that a recorded operator may take
  bool refused = false;                 // recording did not fit: not tried again (captured transposes walk by now)
  int* status = nullptr;                // the handle's error word
  // panels: face geometry for the normal derivative
  DBuf<int> pan_face, pan_i, pan_j, pan_k;  // lower-corner node (0-based) of each panel
  // targets
  DBuf<int> tgt_node;                   // linear node index of each boundary node
  DBuf<double> tx, ty, tz;
  DBuf<int> tgt_frame;                  // ibctyp 3: frame slot of each target's plane
  // precomputed operator (CSR over targets)
  bool precomputed = false;
  long long nnz = 0;
  DBuf<long long> rowptr;
  DBuf<int> col;
  DBuf<float2> w;                       // weights dS/r, 8-byte words: doubles, or float-float pairs (hi + lo = dS/r to 2^-48)
  // the coarsest level, which every target walks in full, as a dense block:
  // [target / 32][cell][target % 32] weight words (as w), zero where the
  // cell was opened; the rows above then hold only the finer levels
  bool dense = false;
  int ntopd = 0;                        // cells of the coarsest level
  long long ndense_acc = 0;             // accepted interactions in the block
  DBuf<float2> wtop;
  int dseg = 1;                         // segments of the coarsest cells (k_apply_dense grid y)
  DBuf<double> dsum;                    // [segment][3][ntarget] partial sums of the block
  DBuf<unsigned long long> dcount;
  // its transpose (CSR over cells, for the reverse mode), built on first use
  bool transposed = false;
  DBuf<long long> colptr;
  DBuf<int> trow;
  DBuf<float2> tw;                      // weight words of the transposed list
  DBuf<float2> vff;                     // per target: the boundary-value adjoint in the operator's arithmetic
  DBuf<double> dpart;                   // dense transpose: partial sums [chunk group][cell]
  // apply by the walk (not recorded)
  DBuf<WalkNode> wnodes;
  DBuf<int> toppos;
  int walkseg = 1;
  DBuf<double> walkpart;                // [segment][3][ntarget] partial sums
  FarField ff;                          // the coarsest level by FFT (uniform lattices) ...
  NearField near;                       // ... with the opened cells of every level by tables
  long long bytes() const;
};
void boundary_prepare(BoundaryOp& B, const Grid& g, int levmax, long long budget_bytes, cudaStream_t s,
                      int ibctyp, bool tree, int arith, int* status, bool once = false);  // once: applied a single time
// Sets B.ff and B.near up (the operator needs no recorded rows then) when the
// cells of every level form uniform lattices on every face (ibctyp 2,
// tree) and VPMG_FARFIELD is not "0"; set-up time, outside stream capture.
bool farfield_prepare(BoundaryOp& B, const Grid& g, cudaStream_t s);
bool near_prepare(BoundaryOp& B, const Grid& g, long long budget_bytes, cudaStream_t s);
void near_apply(BoundaryOp& B, cudaStream_t s);
void near_release(BoundaryOp& B);
// Records the interaction lists if they fit the budget (B.precomputed).
void boundary_record(BoundaryOp& B, cudaStream_t s);
// sol += the boundary values: every coarsest cell by FFT, the near field's
// sums (near_apply first) and the correction rows.
void farfield_apply(BoundaryOp& B, double* const sol[3], cudaStream_t s);
void farfield_release(BoundaryOp& B);
// Normal-derivative panels of the three components from their zero-BC
// solutions (scs doubles apart); boundary_apply aggregates them and adds the
// boundary values into the faces of sol.
void boundary_panels(BoundaryOp& B, const Grid& g, const double* sol0, size_t scs, cudaStream_t s);
void boundary_apply(BoundaryOp& B, const Grid& g, double* const sol[3], cudaStream_t s);
// Problems that share one recorded operator (same index geometry, weights
// in proportion to the mesh spacing): each problem's sources go to its slot
// of an interleaved buffer [cell][slot][4] (float2, nprob slots per cell),
// then one launch adds
// every problem's boundary values (o[p][c] at the target nodes, times scale[p]).
constexpr int kGroupMax = 16;
struct GroupOut {
  double* o[kGroupMax][3];
  double scale[kGroupMax];
};
// Rows of a follower's operator that are not the leader's times the ratio
// (ties of the opening test broken by each problem's rounding): the
// follower's row minus the scaled leader's row, applied after the group.
struct GroupCorrection {
  int nrows = 0;
  long long nnz = 0;
  DBuf<int> rows;
  DBuf<long long> rowptr;
  DBuf<int> col;
  DBuf<double> w;
};
// true when F can share L's recorded operator: same index geometry and
// tree, weights L's times *ratio except for the cells where the two walks
// decided differently, which C holds (at most max_frac of the interactions)
bool boundary_group_match(const BoundaryOp& L, const Grid& gl, const BoundaryOp& F, const Grid& gf, double max_frac,
                          double* ratio, GroupCorrection& C, cudaStream_t s);
void boundary_group_correct(const BoundaryOp& F, const GroupCorrection& C, double* const sol[3], cudaStream_t s);
// Frees the recorded operator (and its transpose): applies walk the tree again.
void boundary_release_recorded(BoundaryOp& B);
void boundary_group_sources(BoundaryOp& B, float2* gsrc, int slot, int lanes, cudaStream_t s);
// doubles of the dense block's partial sums for a group of nprob problems
size_t boundary_group_partial_count(const BoundaryOp& L, int nprob);
void boundary_group_apply(const BoundaryOp& L, const float2* gsrc, int nprob, double* part, const GroupOut& G,
                          cudaStream_t s);
// Transposes (one component): boundary-value adjoint (grid node array) ->
// cell adjoints -> panel adjoints -> accumulated into the sol0 adjoint.
void boundary_apply_T(BoundaryOp& B, const double* bcbar, size_t bcs, double* cellbar, cudaStream_t s);
// Builds the transposed interaction list when the operator is recorded and
// the copy fits in half of the free device memory (set-up time, outside
// stream capture); boundary_apply_T then gathers per cell instead of
// scattering with atomics.
void boundary_transpose_prepare(BoundaryOp& B, cudaStream_t s);
void boundary_agg_T(BoundaryOp& B, const double* cellbar, double* panelbar, cudaStream_t s);
void boundary_panels_T(BoundaryOp& B, const Grid& g, const double* panelbar, double* sol0bar, size_t scs, cudaStream_t s);

// ---------------------------------------------------- small kernels ----
void fill_zero(double* p, size_t n, cudaStream_t s);
void exclusive_scan_int(const int* in, int* out, size_t n, int* block_sums, cudaStream_t s);
size_t scan_block_sums_needed(size_t n);
double measure_fp64_peak(cudaStream_t s);  // TFLOP/s of a DFMA loop

}  // namespace vpmg
