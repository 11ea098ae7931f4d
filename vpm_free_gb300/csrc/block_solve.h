// block_solve.h -- the padded YAPS block's two infinite-domain solves,
// evaluated only where the step reads them (block_solve.cu).
#pragma once
#include "vpmg_internal.h"

namespace vpmg {

struct BlockSolve {
  bool ready = false;
  int dims[3] = {0, 0, 0};  // block node counts
  int m[3] = {0, 0, 0};     // interior counts
  int nsx = 0, nsy = 0, nsz = 0;
  DBuf<double> ghat;        // 3 * interior: forward transforms of the RHS
  DBuf<double> W;           // 3 * interior: Thomas output
  int arith = VPMG_ARITH_FP64;  // the plan's arithmetic
  // sine rows sin(pi (i+1)(p+1)/N) of the selected interior indices, one
  // 8-byte word each: a double, or a float-float pair (arith)
  DBuf<double> S_fx, S_fy_lo, S_ix, S_iy_lo, S_sx, S_sy;
  DBuf<double> e_x1, e_y1;  // sines of the first interior layer along x and y
  DBuf<int> l_fx, l_ix, l_sx, l_sy, l_sz, l_idy, l_idz;  // node lists for scatters / plane lists
  DBuf<double> X8, Y4, X2, Y1, Ys, XS;  // compact partial results
  DBuf<double> f;           // the faces' values, then their transforms (3 * face_doubles)
  int inner_lo[3] = {0, 0, 0}, inner_hi[3] = {0, 0, 0};  // interior indices of the inner-box faces
  void prepare(const DirichletPlan& P, const int nnbl_bl[6], int ncoarse);
};

// A whole box's Dirichlet solve with its face values entering in DST space
// (as the block's BC solve does): forward x/y transforms of the RHS alone,
// so vorticity-free tiles skip their FFTs; the faces of sol, transformed
// along their own axes, join the Thomas sweep; full inverse transforms into
// sol's interior.  work and out: nc interior-size scratch arrays each.
// Doubles of one component's six faces: the x and y pairs as (sum,
// difference), the z faces as they are.
size_t face_doubles(const DirichletPlan& P);
struct FaceSolve {
  bool ready = false;
  DBuf<double> f;   // the six faces' values, then their transforms (3 components)
  DBuf<double> e;   // sines of the first interior layer along x and y
  void prepare(const DirichletPlan& P);
};
void dirichlet_solve_faces(DirichletPlan& P, FaceSolve& F, const double* rhs, size_t rcs, double* sol, size_t scs,
                           int nc, double* work, double* out, cudaStream_t s);

// nc components at a time (arrays rcs / scs doubles apart):
// the zero-BC solve: forward transforms kept in ghat, u near the six faces
// (4 interior layers) written into sol0;
void block_solve_zero_bc(BlockSolve& B, DirichletPlan& P, const double* rhs, size_t rcs, double* sol0, size_t scs,
                         int nc, cudaStream_t s);
// the solve with the boundary values already on the faces of sol: writes the
// inner-box faces and the every-ncoarse-th interior samples of sol.
void block_solve_bc(BlockSolve& B, DirichletPlan& P, double* sol, size_t scs, int nc, cudaStream_t s);

}  // namespace vpmg
