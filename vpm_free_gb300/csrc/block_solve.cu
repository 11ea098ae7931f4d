// block_solve.cu -- the padded YAPS block's infinite-domain solve, evaluated
// only where the reference's step reads it.
//
// yaps3d (source/yaps3d.f90:52-53 -> pmlib.f90:115-154) solves the padded
// block twice per component with the same right-hand side:
//   1. zero boundary values (solve_eq_0_3d, pmsolve.f90:367-432), of which
//      calc_normalderiv_3d (pinfdomain.f90:294-547) reads only the 4
//      interior layers next to each face;
//   2. the quadtree boundary values (solve_eq_3d, pmsolve.f90:284-365), of
//      which the step reads only the every-nc-th samples
//      (yaps3d.f90:104-138) and the six faces of the inner block box
//      (interp_stencil targets, yaps3d.f90:340-395; final-solve boundary).
// Both share the forward transform ghat = DST_y DST_x RHS: the boundary
// values of solve 2 enter in transform space as rank-structured face terms
// added inside the Thomas sweep.  The inverse transforms are evaluated only
// on the needed layers: dot products with the selected sine rows along one
// axis, then a full inverse DST along the other.  The values produced are
// those of the full discrete solves (same linear algebra, different
// rounding).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "arith.cuh"
#include "block_solve.h"

namespace vpmg {

namespace {

constexpr int kLines = 16;  // lines per CTA of the x dot-product kernel

__device__ __forceinline__ double shfl_xor(double v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }
__device__ __forceinline__ float2 shfl_xor(float2 v, int m) {
  return make_float2(__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m));
}

// The dot products below run in the policy's arithmetic (arith.cuh): the
// sine rows are stored in it (doubles, or float-float pairs), W enters it
// as it is staged, and each result is joined back into a double.

// out[i + nsel*(q + m1*kk)] = sum_p S[i][p] * W[p + m0*(q + m1*k)],  k = klist ? klist[kk] : kk,
// for nc components of W (wcs doubles apart; their outputs follow each other).
//
// pair: the selected rows are nsel layers i and their mirrors m-1-i, whose
// sines are (-1)^p times the layer's: with the sums over the even and the odd
// p apart, E and O, the layer is E + O and its mirror E - O: half the FMAs
// (both partial kernels were bound by them).  The mirrors' outputs follow in
// reverse order, at 2 nsel - 1 - i.
// Persistent CTAs walk tiles of up to kLines lines; the sine rows are
// staged once per CTA.  In FP64 (dbl) the next tile is staged with
// asynchronous copies (cp.async, 8 bytes each) while the current one is
// reduced, so the loads' latency hides behind the FMAs.  Float-float
// staging converts each value as it lands, which cannot run ahead: one
// buffer, and the smaller footprint keeps more CTAs on an SM instead.
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

template <class A>
__device__ __forceinline__ void stage_x_tile(typename A::R* tile, const double* __restrict__ W, int m0, int m1,
                                             int nlines, const int* __restrict__ klist, int tile_id, int ntile1,
                                             size_t wcs, int lines) {
  W += (size_t)(tile_id / ntile1) * wcs;
  const int l0 = (tile_id % ntile1) * lines;
  for (int t = threadIdx.x; t < lines * m0; t += blockDim.x) {
    const int li = t / m0, p = t - li * m0;
    const int l = l0 + li;
    if (l < nlines) {
      const int q = l % m1, kk = l / m1;
      const int k = klist ? klist[kk] : kk;
      const double* src = W + (size_t)p + (size_t)m0 * (q + (size_t)m1 * k);
      if constexpr (A::kFF) tile[t] = A::from(*src);
      else cp_async8(&tile[t], src);
    } else {
      tile[t] = A::zero();
    }
  }
  if constexpr (!A::kFF) cp_async_commit();
}

template <class A>
__global__ void __launch_bounds__(128) k_partial_x(const double* __restrict__ W, int m0, int m1, int nk,
                                                   const int* __restrict__ klist, const typename A::R* __restrict__ S,
                                                   int nsel, double* __restrict__ out, int lines, int dbl, int nc,
                                                   size_t wcs, int pair) {
  using R = typename A::R;
  extern __shared__ double smx[];
  R* Ss = reinterpret_cast<R*>(smx);               // nsel x m0
  R* const buf0 = Ss + (size_t)nsel * m0;           // one or two (dbl) tiles of `lines` x m0 (lines <= kLines)
  R* const buf1 = buf0 + (size_t)lines * m0;
  const int nlines = m1 * nk;
  const int ntile1 = (nlines + lines - 1) / lines, ntiles = ntile1 * nc;
  const int nw = pair ? 2 * nsel : nsel;  // rows written
  const size_t ocs = (size_t)nw * nlines;
  for (int t = threadIdx.x; t < nsel * m0; t += blockDim.x) Ss[t] = S[t];
  int cur = 0;
  if (dbl && (int)blockIdx.x < ntiles)
    stage_x_tile<A>(buf0, W, m0, m1, nlines, klist, blockIdx.x, ntile1, wcs, lines);
  // R adjacent threads share one dot product (R = 128 / outputs, a power of
  // two up to 8, when the CTA has fewer outputs than threads), each summing
  // every R-th term; their partials meet in a fixed shuffle tree.
  const int nout = lines * nsel;
  int Rs = 1;
  while (Rs < 8 && nout * Rs * 2 <= (int)blockDim.x) Rs *= 2;
  const int r = threadIdx.x % Rs;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int next = tile + gridDim.x;
    if (dbl) {
      if (next < ntiles) {
        stage_x_tile<A>(cur ? buf0 : buf1, W, m0, m1, nlines, klist, next, ntile1, wcs, lines);
        if constexpr (!A::kFF) cp_async_wait<1>();  // the current tile's copies are done
      } else {
        if constexpr (!A::kFF) cp_async_wait<0>();
      }
    } else {
      stage_x_tile<A>(buf0, W, m0, m1, nlines, klist, tile, ntile1, wcs, lines);
      if constexpr (!A::kFF) cp_async_wait<0>();
    }
    __syncthreads();
    const R* tl = cur ? buf1 : buf0;
    const int l0 = (tile % ntile1) * lines;
    double* const oc = out + (size_t)(tile / ntile1) * ocs;
    for (int o0 = 0; o0 < nout; o0 += blockDim.x / Rs) {
      const int o = o0 + threadIdx.x / Rs;
      const int li = o % lines, i = o / lines;
      const int l = l0 + li;
      const bool ok = o < nout && l < nlines;
      R a0 = A::zero(), a1 = a0, a2 = a0, a3 = a0;
      if (ok) {
        const R* a = tl + (size_t)li * m0;
        const R* b = Ss + (size_t)i * m0;
        int p = r;
        for (; p + 3 * Rs < m0; p += 4 * Rs) {
          a0 = A::fma(a[p], b[p], a0);
          a1 = A::fma(a[p + Rs], b[p + Rs], a1);
          a2 = A::fma(a[p + 2 * Rs], b[p + 2 * Rs], a2);
          a3 = A::fma(a[p + 3 * Rs], b[p + 3 * Rs], a3);
        }
        for (; p < m0; p += Rs) a0 = A::fma(a[p], b[p], a0);
      }
      R v = A::add(A::add(a0, a1), A::add(a2, a3));
      for (int m = pair ? 2 : 1; m < Rs; m <<= 1) {
        const R w = shfl_xor(v, m);
        v = (r & m) ? A::add(w, v) : A::add(v, w);
      }
      if (pair) {  // Rs is even: threads of even r hold E, of odd r O
        const R w = shfl_xor(v, 1);
        v = (r & 1) ? A::sub(w, v) : A::add(v, w);
      }
      if (ok && (r == 0 || (pair && r == 1))) {
        const int q = l % m1, kk = l / m1;
        oc[(r ? nw - 1 - i : i) + (size_t)nw * (q + (size_t)m1 * kk)] = A::to(v);
      }
    }
    __syncthreads();  // the buffer is refilled next (one buffer) or two tiles on (dbl)
    if (dbl) cur ^= 1;
  }
}

// out[p + m0*(j + nsel*kk)] = sum_q S[j][q] * W[p + m0*(q + m1*k)]
// A CTA stages the m1 x 32 column tile (p0..p0+31, all q) of plane k in
// shared memory with coalesced row loads -- W is read from HBM once -- and
// its threads then form the nsel x 32 dot products from the tile.
constexpr int kColTile = 32;
template <class A>
__device__ __forceinline__ void stage_y_tile(typename A::R* tile, const double* __restrict__ W, int m0, int m1,
                                             const int* __restrict__ klist, int p0, int kk) {
  const int k = klist ? klist[kk] : kk;
  const double* plane = W + (size_t)m0 * m1 * k;
  const int lane = threadIdx.x % kColTile, row = threadIdx.x / kColTile, rows = blockDim.x / kColTile;
  const int p = p0 + lane;
  for (int q = row; q < m1; q += rows) {
    if (p < m0) {
      if constexpr (A::kFF) tile[q * kColTile + lane] = A::from(plane[(size_t)m0 * q + p]);
      else cp_async8(&tile[q * kColTile + lane], plane + (size_t)m0 * q + p);
    } else {
      tile[q * kColTile + lane] = A::zero();
    }
  }
  if constexpr (!A::kFF) cp_async_commit();
}

// Persistent CTAs walk (column tile, plane) pairs; with dbl (FP64, when two
// tiles fit) the next pair's tile is staged asynchronously while the
// current one is reduced.
template <class A>
__global__ void __launch_bounds__(256) k_partial_y(const double* __restrict__ W, int m0, int m1, int nk,
                                                   const int* __restrict__ klist, const typename A::R* __restrict__ S,
                                                   int nsel, double* __restrict__ out, double* __restrict__ out2,
                                                   int dbl, int nc, size_t wcs, int pair) {
  using R = typename A::R;
  extern __shared__ double smy[];
  R* const buf0 = reinterpret_cast<R*>(smy);              // [q][lane], m1 x kColTile
  R* const buf1 = buf0 + (size_t)m1 * kColTile;             // the second tile (dbl)
  R* const partial = (dbl ? buf1 : buf0) + (size_t)m1 * kColTile;  // partial sums [row][lane]
  const int nbx = (m0 + kColTile - 1) / kColTile;
  const int ntile1 = nbx * nk, ntiles = ntile1 * nc;
  // pair: out2 holds the mirrors' rows (nsel of them, in reverse order)
  const size_t ocs = (size_t)m0 * nsel * nk, ocs2 = ocs;
  const int lane = threadIdx.x % kColTile, row = threadIdx.x / kColTile, rows = blockDim.x / kColTile;
  // R rows share one output row set when there are fewer outputs than rows
  // (R a power of two), each summing every R-th q; the partials are added
  // in row order through shared memory.
  const int nout = nsel;
  int Rs = 1;
  while (Rs < rows && nout * Rs * 2 <= rows) Rs *= 2;
  const int r = row % Rs;
  int cur = 0;
  if (dbl && (int)blockIdx.x < ntiles)
    stage_y_tile<A>(buf0, W + (size_t)((int)blockIdx.x / ntile1) * wcs, m0, m1, klist,
                    ((int)blockIdx.x % nbx) * kColTile, ((int)blockIdx.x % ntile1) / nbx);
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int comp = tile / ntile1;
    const int p0 = (tile % nbx) * kColTile, kk = (tile % ntile1) / nbx;  // nbx divides ntile1
    const int next = tile + gridDim.x;
    if (dbl) {
      if (next < ntiles) {
        stage_y_tile<A>(cur ? buf0 : buf1, W + (size_t)(next / ntile1) * wcs, m0, m1, klist, (next % nbx) * kColTile,
                        (next % ntile1) / nbx);
        if constexpr (!A::kFF) cp_async_wait<1>();
      } else {
        if constexpr (!A::kFF) cp_async_wait<0>();
      }
    } else {
      stage_y_tile<A>(buf0, W + (size_t)comp * wcs, m0, m1, klist, p0, kk);
      if constexpr (!A::kFF) cp_async_wait<0>();
    }
    __syncthreads();
    const R* tl = cur ? buf1 : buf0;
    const int p = p0 + lane;
    for (int j0 = 0; j0 < nout; j0 += rows / Rs) {
      const int jj = j0 + row / Rs;
      R a0 = A::zero(), a1 = a0, a2 = a0, a3 = a0;
      if (jj < nout && p < m0) {
        const R* Sj = S + (size_t)jj * m1;
        int q = r;
        for (; q + 3 * Rs < m1; q += 4 * Rs) {
          a0 = A::fma(__ldg(&Sj[q]), tl[q * kColTile + lane], a0);
          a1 = A::fma(__ldg(&Sj[q + Rs]), tl[(q + Rs) * kColTile + lane], a1);
          a2 = A::fma(__ldg(&Sj[q + 2 * Rs]), tl[(q + 2 * Rs) * kColTile + lane], a2);
          a3 = A::fma(__ldg(&Sj[q + 3 * Rs]), tl[(q + 3 * Rs) * kColTile + lane], a3);
        }
        for (; q < m1; q += Rs) a0 = A::fma(__ldg(&Sj[q]), tl[q * kColTile + lane], a0);
      }
      R v = A::add(A::add(a0, a1), A::add(a2, a3));
      if (Rs > 1) {
        partial[row * kColTile + lane] = v;
        __syncthreads();
        if (pair) {  // Rs is even: rows of even r hold parts of E, of odd r of O
          R O = A::zero();
          if (r == 0) {
            O = partial[(row + 1) * kColTile + lane];
            for (int m = 2; m < Rs; m += 2) {
              v = A::add(v, partial[(row + m) * kColTile + lane]);
              O = A::add(O, partial[(row + m + 1) * kColTile + lane]);
            }
            if (jj < nout && p < m0)
              out2[comp * ocs2 + (size_t)p + (size_t)m0 * (nsel - 1 - jj + (size_t)nsel * kk)] = A::to(A::sub(v, O));
            v = A::add(v, O);
          }
        } else if (r == 0) {
          for (int m = 1; m < Rs; ++m) v = A::add(v, partial[(row + m) * kColTile + lane]);
        }
        __syncthreads();
      }
      if (r == 0 && jj < nout && p < m0) {
        out[comp * ocs + (size_t)p + (size_t)m0 * (jj + (size_t)nsel * kk)] = A::to(v);
      }
    }
    __syncthreads();  // the tile's buffer is refilled next
    if (dbl) cur ^= 1;
  }
}

// dst node (ia[a], ib[b], ic[c]) <- src[a + na*(b + nb*c)]; a null list means identity + off.
__global__ void k_scatter3(const double* __restrict__ src, int na, int nb, int nc, const int* __restrict__ ia,
                           const int* __restrict__ ib, const int* __restrict__ ic, int off, double* __restrict__ dst,
                           int dx, int dy, size_t dcs) {
  const size_t n = (size_t)na * nb * nc;
  src += blockIdx.y * n;  // component
  dst += blockIdx.y * dcs;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x) {
    const int a = (int)(t % na), b = (int)((t / na) % nb), c = (int)(t / ((size_t)na * nb));
    const int i = ia ? ia[a] : a + off, j = ib ? ib[b] : b + off, k = ic ? ic[c] : c + off;
    dst[(size_t)i + (size_t)dx * (j + (size_t)dy * k)] = src[t];
  }
}

// The first and last interior layers' sines along an axis of m nodes are
// sin(pi (p+1)/(m+1)) and sin(pi m (p+1)/(m+1)) = (-1)^p sin(pi (p+1)/(m+1)),
// so a pair of opposite faces enters mode p of the sweep as its sum (p
// even) or its difference (p odd) times the first layer's sine.  The face
// extractions below store the x and y pairs that way (the transforms along
// the faces' own axes are linear): one FMA per axis and node in the sweep.
//
// The six faces of the box whose node (0,0,0) sits at (o0,o1,o2) of an
// NX x NY x * array, interior m0 x m1 x m2: x pair (sum, difference) [k][j],
// y pair [k][i], z faces [j][i].
__global__ void k_extract_box_faces(const double* __restrict__ s, int NX, int NY, int o0, int o1, int o2, int m0,
                                    int m1, int m2, double* __restrict__ fxs, double* __restrict__ fxd,
                                    double* __restrict__ fys, double* __restrict__ fyd, double* __restrict__ fz0,
                                    double* __restrict__ fzN, size_t scs, size_t fcs) {
  const size_t sy = NX, sz = (size_t)NX * NY;
  const long nx = (long)m1 * m2, ny = (long)m0 * m2, nz = (long)m0 * m1;
  s += blockIdx.y * scs;  // component
  fxs += blockIdx.y * fcs; fxd += blockIdx.y * fcs; fys += blockIdx.y * fcs;
  fyd += blockIdx.y * fcs; fz0 += blockIdx.y * fcs; fzN += blockIdx.y * fcs;
  auto at = [&](int a, int b, int c) { return s[(size_t)(o0 + a) + sy * (o1 + b) + sz * (o2 + c)]; };
  for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < nx + ny + nz; t += (long)gridDim.x * blockDim.x) {
    if (t < nx) {
      const int j = (int)(t % m1) + 1, k = (int)(t / m1) + 1;
      const double a = at(0, j, k), b = at(m0 + 1, j, k);
      fxs[t] = a + b;
      fxd[t] = a - b;
    } else if (t < nx + ny) {
      const long u = t - nx;
      const int i = (int)(u % m0) + 1, k = (int)(u / m0) + 1;
      const double a = at(i, 0, k), b = at(i, m1 + 1, k);
      fys[u] = a + b;
      fyd[u] = a - b;
    } else {
      const long u = t - nx - ny;
      const int i = (int)(u % m0) + 1, j = (int)(u / m0) + 1;
      fz0[u] = at(i, j, 0);
      fzN[u] = at(i, j, m2 + 1);
    }
  }
}

// The z pass: -u[k-1] + d u[k] - u[k+1] = r[k] per mode, r = g (+ the
// transformed Dirichlet face terms), eliminated from both ends to the middle
// and substituted back outwards ("burn at both ends"), with the reciprocal
// pivots of k_pivots: the matrix is the same read from either end, so both
// chains use one table of half the planes.  A thread owns one mode of NC
// components: 2 NC independent chains of m2 / 2 steps each way, which share
// the table's loads.  The recurrence stays in FP64 in both arithmetics.
// Bound: HBM at large boxes (g read, the forward values written and read, u
// written, half the table read twice: 32 + 8 / NC bytes per node); the
// chains' latency at small ones, hence the U planes loaded ahead.
template <int NC, bool BC>
__global__ void __launch_bounds__(128) k_thomas_ends(const double* g, double* out, const double* __restrict__ rinv,
                                                     int m0, int m1, int m2, size_t cs, FaceTerms F) {
  if (NC == 1) {  // blockIdx.y = component
    g += blockIdx.y * cs;
    out += blockIdx.y * cs;
    if constexpr (BC) {
      const size_t f = blockIdx.y * F.cs;
      F.fxs += f; F.fxd += f; F.fys += f; F.fyd += f; F.fz0 += f; F.fzN += f;
    }
  }
  const int pq = blockIdx.x * blockDim.x + threadIdx.x;
  if (pq >= m0 * m1) return;
  const int p = pq % m0, q = pq / m0;
  const size_t plane = (size_t)m0 * m1;
  constexpr int U = NC == 1 ? 8 : 4;
  double ax = 0.0, ay = 0.0;
  const double *fx = nullptr, *fy = nullptr;
  if constexpr (BC) {
    ax = F.cx * F.ex1[p];
    ay = F.cy * F.ey1[q];
    fx = ((p & 1) ? F.fxd : F.fxs) + q;  // the x pair's sum (p even) or difference
    fy = ((q & 1) ? F.fyd : F.fys) + p;
  }
  auto rhs = [&](int c, int k) -> double {
    double r = g[c * cs + pq + plane * k];
    if constexpr (BC) r = fma(ay, fy[c * F.cs + (size_t)k * m0], fma(ax, fx[c * F.cs + (size_t)k * m1], r));
    return r;
  };
  const int h = m2 >> 1;
  double yt[NC], yb[NC];  // the two chains' values
  if (h > 0) {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      yt[c] = rhs(c, 0);
      yb[c] = rhs(c, m2 - 1);
      if constexpr (BC) {
        yt[c] += F.cz * F.fz0[c * F.cs + pq];
        yb[c] += F.cz * F.fzN[c * F.cs + pq];
      }
      out[c * cs + pq] = yt[c];
      out[c * cs + pq + plane * (m2 - 1)] = yb[c];
    }
  }
  auto fwd = [&](int k, int n) {  // planes k .. k+n-1 from both ends
    double rt[U][NC], rb[U][NC], rv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= n) break;
      rv[u] = rinv[pq + plane * (k + u - 1)];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        rt[u][c] = rhs(c, k + u);
        rb[u][c] = rhs(c, m2 - 1 - (k + u));
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= n) break;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        yt[c] = fma(yt[c], rv[u], rt[u][c]);
        yb[c] = fma(yb[c], rv[u], rb[u][c]);
        out[c * cs + pq + plane * (k + u)] = yt[c];
        out[c * cs + pq + plane * (m2 - 1 - (k + u))] = yb[c];
      }
    }
  };
  int k = 1;
  for (; k + U <= h; k += U) fwd(k, U);
  for (; k < h; ++k) fwd(k, 1);
  const double mid = rinv[pq + plane * h];
  const double rl = h > 0 ? rinv[pq + plane * (h - 1)] : 0.0;
  if (m2 & 1) {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      double r = rhs(c, h);
      if (h > 0) {
        r = fma(rl, yt[c] + yb[c], r);
      } else if constexpr (BC) {
        r += F.cz * F.fz0[c * F.cs + pq];
        r += F.cz * F.fzN[c * F.cs + pq];
      }
      yt[c] = yb[c] = mid * r;
      out[c * cs + pq + plane * h] = yt[c];
    }
    k = h - 1;
  } else {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const double a = yt[c], b = yb[c];
      yt[c] = mid * fma(rl, b, a);
      yb[c] = mid * fma(rl, a, b);
      out[c * cs + pq + plane * (h - 1)] = yt[c];
      out[c * cs + pq + plane * h] = yb[c];
    }
    k = h - 2;
  }
  auto bwd = [&](int kk, int n) {  // planes kk, kk-1, .. kk-n+1 outwards
    double ot[U][NC], ob[U][NC], rv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= n) break;
      rv[u] = rinv[pq + plane * (kk - u)];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        ot[u][c] = out[c * cs + pq + plane * (kk - u)];
        ob[u][c] = out[c * cs + pq + plane * (m2 - 1 - (kk - u))];
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= n) break;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        yt[c] = (ot[u][c] + yt[c]) * rv[u];
        yb[c] = (ob[u][c] + yb[c]) * rv[u];
        out[c * cs + pq + plane * (kk - u)] = yt[c];
        out[c * cs + pq + plane * (m2 - 1 - (kk - u))] = yb[c];
      }
    }
  };
  for (; k - U + 1 >= 0; k -= U) bwd(k, U);
  for (; k >= 0; --k) bwd(k, 1);
}

// sin(pi (i+1)(p+1)/N) of the selected rows, one 8-byte word each: the
// double (FP64) or its float-float pair (hi, lo) in the word's bytes.
std::vector<double> sine_rows(const std::vector<int>& sel, int m, int arith) {
  std::vector<double> S(sel.size() * (size_t)m);
  const double N = m + 1;
  for (size_t i = 0; i < sel.size(); ++i)
    for (int p = 0; p < m; ++p) {
      const double v = std::sin(kPI * (double)(sel[i] + 1) * (double)(p + 1) / N);
      if (arith == VPMG_ARITH_FF48) {
        const float hi = (float)v;
        const float2 f = make_float2(hi, (float)(v - (double)hi));
        std::memcpy(&S[i * m + p], &f, sizeof(double));
      } else {
        S[i * m + p] = v;
      }
    }
  return S;
}

template <class T>
void up(DBuf<T>& b, const std::vector<T>& h) {
  b.ensure(std::max<size_t>(h.size(), 1));
  if (!h.empty()) VPMG_CUDA(cudaMemcpy(b.p, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice));
}

std::vector<int> plus1(const std::vector<int>& v) {
  std::vector<int> r(v);
  for (int& x : r) x += 1;
  return r;
}

// Dynamic shared memory granted to k_partial_x and k_partial_y so far, per
// device: the limit is an attribute of each kernel on each device, and one
// process may hold handles on several devices.  Raised at set-up only
// (outside any stream capture), never lowered.
constexpr int kMaxDev = 64;
size_t g_partial_smem[kMaxDev] = {0};
size_t g_partial_y_smem[kMaxDev] = {0};
size_t& granted(size_t* table) {
  int dev = 0;
  VPMG_CUDA(cudaGetDevice(&dev));
  VPMG_CHECK(dev >= 0 && dev < kMaxDev, VPMG_ERR_UNSUPPORTED, "device index beyond the per-device tables");
  return table[dev];
}

// k_partial_x's shared memory: the sine rows and one or two (dbl) tiles,
// 8 bytes per value in both arithmetics.
size_t partial_x_smem(int m0, int nsel, int lines, bool dbl) {
  return sizeof(double) * ((dbl ? 2 : 1) * (size_t)lines * m0 + (size_t)nsel * m0);
}
// Tile height of k_partial_x: the most lines (up to kLines) whose staged
// tiles and the sine rows fit in a CTA's shared memory.
int partial_x_lines(int m0, int nsel, bool dbl) {
  int lines = kLines;
  while (lines > 1 && partial_x_smem(m0, nsel, lines, dbl) > 227 * 1024) lines /= 2;
  return lines;
}

void partial_x_reserve(int m0, int nsel) {
  const size_t sm = partial_x_smem(m0, nsel, partial_x_lines(m0, nsel, true), true);
  VPMG_CHECK(sm <= 227 * 1024, VPMG_ERR_UNSUPPORTED, "partial transform tile too large");
  // the whole per-CTA maximum: every call's tile height keeps it within
  const size_t cap = 227 * 1024;
  size_t& have = granted(g_partial_smem);
  if (cap > have) {
    VPMG_CUDA(cudaFuncSetAttribute(k_partial_x<F64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap));
    VPMG_CUDA(cudaFuncSetAttribute(k_partial_x<FF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap));
    have = cap;
  }
}

void partial_x(int arith, const double* W, int m0, int m1, int nk, const int* klist, const double* S, int nsel,
               double* out, cudaStream_t s, int nc, size_t wcs, bool pair = false) {
  const int nlines = m1 * nk;
  const bool dbl = arith != VPMG_ARITH_FF48;
  const int lines = partial_x_lines(m0, nsel, dbl);
  const size_t sm = partial_x_smem(m0, nsel, lines, dbl);
  VPMG_CHECK(!pair || lines * nsel <= 64, VPMG_ERR_STATE, "paired rows need two threads per output");
  VPMG_CHECK(sm <= granted(g_partial_smem), VPMG_ERR_STATE, "k_partial_x shared memory not reserved");
  // persistent CTAs: as many as fit on the SMs at this shared-memory size
  const unsigned ntiles = (unsigned)nc * ((nlines + lines - 1) / lines);
  const unsigned per_sm = (unsigned)std::max<size_t>(1, std::min<size_t>(8, (227 * 1024) / (sm + 1024)));
  const unsigned g = std::min(ntiles, 152u * per_sm);
  if (arith == VPMG_ARITH_FF48)
    k_partial_x<FF><<<g, 128, sm, s>>>(W, m0, m1, nk, klist, reinterpret_cast<const float2*>(S), nsel, out, lines, 0,
                                       nc, wcs, pair ? 1 : 0);
  else
    k_partial_x<F64><<<g, 128, sm, s>>>(W, m0, m1, nk, klist, S, nsel, out, lines, 1, nc, wcs,
                                        pair ? 1 : 0);
  VPMG_LAUNCHED();
}

// k_partial_y's shared memory: one or two column tiles and the partial sums
// of 8 rows; two tiles (double buffering) when they fit.
size_t partial_y_smem(int m1, bool dbl) { return sizeof(double) * ((dbl ? 2 : 1) * (size_t)m1 + 8) * kColTile; }
bool partial_y_dbl(int m1) { return partial_y_smem(m1, true) <= 227 * 1024; }

void partial_y_reserve(int m1) {
  const size_t sm = partial_y_smem(m1, partial_y_dbl(m1));
  VPMG_CHECK(sm <= 227 * 1024, VPMG_ERR_UNSUPPORTED, "partial transform tile too large");
  size_t& have = granted(g_partial_y_smem);
  if (sm > have) {
    VPMG_CUDA(cudaFuncSetAttribute(k_partial_y<F64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    VPMG_CUDA(cudaFuncSetAttribute(k_partial_y<FF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    have = sm;
  }
}

void partial_y(int arith, const double* W, int m0, int m1, int nk, const int* klist, const double* S, int nsel,
               double* out, cudaStream_t s, int nc, size_t wcs, double* mirrors = nullptr) {
  VPMG_CHECK(!mirrors || nsel <= 4, VPMG_ERR_STATE, "paired rows need two rows of threads per output");
  const int dbl = (arith != VPMG_ARITH_FF48 && partial_y_dbl(m1)) ? 1 : 0;
  const size_t sm = partial_y_smem(m1, dbl);  // tiles + partial sums of 8 rows
  VPMG_CHECK(sm <= granted(g_partial_y_smem), VPMG_ERR_STATE, "k_partial_y shared memory not reserved");
  // persistent CTAs: as many as fit on the SMs at this shared-memory size
  const unsigned ntiles = (unsigned)nc * (unsigned)(((m0 + kColTile - 1) / kColTile) * nk);
  const unsigned per_sm = (unsigned)std::max<size_t>(1, std::min<size_t>(8, (227 * 1024) / (sm + 1024)));
  const unsigned g = std::min(ntiles, 152u * per_sm);
  if (arith == VPMG_ARITH_FF48)
    k_partial_y<FF><<<g, 256, sm, s>>>(W, m0, m1, nk, klist, reinterpret_cast<const float2*>(S), nsel, out,
                                      mirrors, dbl, nc, wcs, mirrors ? 1 : 0);
  else
    k_partial_y<F64><<<g, 256, sm, s>>>(W, m0, m1, nk, klist, S, nsel, out, mirrors, dbl, nc, wcs,
                                        mirrors ? 1 : 0);
  VPMG_LAUNCHED();
}

void scatter3(const double* src, int na, int nb, int nc, const int* ia, const int* ib, const int* ic, int off,
              double* dst, const int dims[3], cudaStream_t s, int ncomp, size_t dcs) {
  const size_t n = (size_t)na * nb * nc;
  k_scatter3<<<dim3((unsigned)std::min<size_t>((n + 255) / 256, 152 * 16), ncomp), 256, 0, s>>>(
      src, na, nb, nc, ia, ib, ic, off, dst, dims[0], dims[1], dcs);
  VPMG_LAUNCHED();
}

// The six faces of a box of sol as FaceTerms arrays of nc components in
// buf, transformed along their own axes (two launches of job lists).
FaceTerms face_terms(const DirichletPlan& P, double* buf, const double* ex1, const double* ey1, const double* sol,
                     size_t scs, int nc, cudaStream_t s) {
  const int m0 = P.m[0], m1 = P.m[1], m2 = P.m[2];
  FaceTerms F;
  double* fxs = buf;
  double* fxd = fxs + (size_t)m1 * m2;
  double* fys = fxd + (size_t)m1 * m2;
  double* fyd = fys + (size_t)m0 * m2;
  double* fz0 = fyd + (size_t)m0 * m2;
  double* fzN = fz0 + (size_t)m0 * m1;
  F.cs = face_doubles(P);
  F.fxs = fxs; F.fxd = fxd; F.fys = fys; F.fyd = fyd; F.fz0 = fz0; F.fzN = fzN;
  F.ex1 = ex1;
  F.ey1 = ey1;
  const double scale = dirichlet_scale(P);
  F.cx = -scale / (P.h[0] * P.h[0]);
  F.cy = -scale / (P.h[1] * P.h[1]);
  F.cz = -scale / (P.h[2] * P.h[2]);
  k_extract_box_faces<<<dim3(256, nc), 256, 0, s>>>(sol, P.dims[0], P.dims[1], P.box[0], P.box[1], P.box[2], m0, m1, m2,
                                                    fxs, fxd, fys, fyd, fz0, fzN, scs, F.cs);
  VPMG_LAUNCHED();
  // rows over j -> q (x faces), over i -> p (y faces, and the z faces' rows)
  // in one launch; then the z faces' columns over j
  const DstYLines rows[6] = {{&P.fy, fxs, 1, m1, m2, F.cs}, {&P.fy, fxd, 1, m1, m2, F.cs},
                             {&P.fx, fys, 1, m0, m2, F.cs}, {&P.fx, fyd, 1, m0, m2, F.cs},
                             {&P.fx, fz0, 1, m0, m1, F.cs}, {&P.fx, fzN, 1, m0, m1, F.cs}};
  dst_lines_y_jobs(rows, 6, s, nc);
  const DstYLines cols[2] = {{&P.fy, fz0, m0, m1, 1, F.cs}, {&P.fy, fzN, m0, m1, 1, F.cs}};
  dst_lines_y_jobs(cols, 2, s, nc);
  return F;
}

}  // namespace

size_t face_doubles(const DirichletPlan& P) {
  const size_t m0 = P.m[0], m1 = P.m[1], m2 = P.m[2];
  return 2 * (m1 * m2 + m0 * m2 + m0 * m1);
}

void thomas_launch(const double* g, double* out, const double* rinv, const int m[3], int nc, size_t cs,
                   const FaceTerms* F, cudaStream_t s) {
  const size_t modes = (size_t)m[0] * m[1];
  const FaceTerms f = F ? *F : FaceTerms{};
  // Three components per thread where the modes alone fill the GPU (they share
  // the pivot loads); fewer modes as one component per thread in CTAs of one
  // warp, for as many SMs as possible: at 79 x 79 modes 49 CTAs of 128 threads
  // held the sweep with faces to a third of the FP64 units (two sweeps of a
  // 64^3 step 130 -> 65 us, the three without faces 60 -> 40 us; at 255 x 255
  // modes both forms keep the FP64 units busy and the shared pivots win).
  if (nc == 3 && modes >= 152 * 256) {
    const unsigned nb = (unsigned)((modes + 127) / 128);
    if (F) k_thomas_ends<3, true><<<nb, 128, 0, s>>>(g, out, rinv, m[0], m[1], m[2], cs, f);
    else k_thomas_ends<3, false><<<nb, 128, 0, s>>>(g, out, rinv, m[0], m[1], m[2], cs, f);
  } else {
    const int th = modes * nc >= 152 * 256 ? 128 : 32;
    const dim3 nb((unsigned)((modes + th - 1) / th), nc);
    if (F) k_thomas_ends<1, true><<<nb, th, 0, s>>>(g, out, rinv, m[0], m[1], m[2], cs, f);
    else k_thomas_ends<1, false><<<nb, th, 0, s>>>(g, out, rinv, m[0], m[1], m[2], cs, f);
  }
}
void thomas_sweep(const double* g, double* out, const double* rinv, const int m[3], int nc, size_t cs,
                  const FaceTerms* F, cudaStream_t s) {
  thomas_launch(g, out, rinv, m, nc, cs, F, s);
  count_launch();
  VPMG_CUDA(cudaGetLastError());
}

void BlockSolve::prepare(const DirichletPlan& P, const int nnbl_bl[6], int ncoarse) {
  arith = P.arith;
  for (int d = 0; d < 3; ++d) { dims[d] = P.dims[d]; m[d] = P.m[d]; }
  VPMG_CHECK(m[0] >= 8 && m[1] >= 8 && m[2] >= 8, VPMG_ERR_UNSUPPORTED, "block too small for the partial solve");
  const size_t nint = (size_t)m[0] * m[1] * m[2];
  ghat.ensure(3 * nint);
  W.ensure(3 * nint);
  // normal-derivative layers: interior indices 0..3 and m-4..m-1
  std::vector<int> fx = {0, 1, 2, 3, m[0] - 4, m[0] - 3, m[0] - 2, m[0] - 1};
  // the first of each pair of mirrored layers
  up(S_fx, sine_rows({0, 1, 2, 3}, m[0], arith));
  up(S_fy_lo, sine_rows({0, 1, 2, 3}, m[1], arith));
  up(l_fx, plus1(fx));
  // inner-box faces: 1-based node nnbl_bl -> interior index nnbl_bl - 2
  for (int d = 0; d < 3; ++d) {
    inner_lo[d] = nnbl_bl[d] - 2;
    inner_hi[d] = nnbl_bl[d + 3] - 2;
    VPMG_CHECK(inner_lo[d] >= 0 && inner_hi[d] < m[d] && inner_lo[d] < inner_hi[d], VPMG_ERR_ARG,
               "inner block box outside the padded block");
  }
  for (int d = 0; d < 2; ++d)
    VPMG_CHECK(inner_hi[d] == m[d] - 1 - inner_lo[d], VPMG_ERR_UNSUPPORTED, "inner block box not centred in the block");
  std::vector<int> ix = {inner_lo[0], inner_hi[0]};
  up(S_ix, sine_rows({inner_lo[0]}, m[0], arith));
  up(S_iy_lo, sine_rows({inner_lo[1]}, m[1], arith));
  up(l_ix, plus1(ix));
  // samples: 0-based nodes nc*t inside the block interior -> interior index nc*t - 1
  auto samples = [&](int d) {
    std::vector<int> v;
    for (int t = 1; ncoarse * t <= dims[d] - 2; ++t) v.push_back(ncoarse * t - 1);
    return v;
  };
  std::vector<int> sx = samples(0), sy = samples(1), sz = samples(2);
  nsx = (int)sx.size(); nsy = (int)sy.size(); nsz = (int)sz.size();
  up(S_sx, sine_rows(sx, m[0], arith));
  up(S_sy, sine_rows(sy, m[1], arith));
  up(l_sx, plus1(sx));
  up(l_sy, plus1(sy));
  up(l_sz, sz);  // plane list (interior index) for the y dots
  std::vector<int> idz(sz);
  up(l_idz, plus1(idz));  // node list for the scatter
  // first layer sines for the face terms
  auto edge = [&](int mm) {
    std::vector<double> e(mm);
    const double N = mm + 1;
    for (int p = 0; p < mm; ++p) e[p] = std::sin(kPI * (double)(p + 1) / N);
    return e;
  };
  up(e_x1, edge(m[0]));
  up(e_y1, edge(m[1]));
  partial_x_reserve(m[0], std::max(8, nsx));
  partial_y_reserve(m[1]);
  X8.ensure((size_t)3 * 8 * m[1] * m[2]);
  Y4.ensure((size_t)3 * m[0] * 8 * m[2]);  // low and high face rows
  X2.ensure((size_t)3 * 2 * m[1] * m[2]);
  Y1.ensure((size_t)3 * m[0] * 2 * m[2]);
  Ys.ensure((size_t)3 * m[0] * nsy * nsz);
  XS.ensure((size_t)3 * nsx * nsy * nsz);
  f.ensure(3 * face_doubles(P));
  ready = true;
}

void block_solve_zero_bc(BlockSolve& B, DirichletPlan& P, const double* rhs, size_t rcs, double* sol0, size_t scs,
                         int nc, cudaStream_t s) {
  const int m0 = B.m[0], m1 = B.m[1], m2 = B.m[2];
  const size_t nint = (size_t)m0 * m1 * m2, plane = (size_t)m0 * m1;
  dst_forward_xy(P, rhs, nullptr, true, B.ghat.p, s, nc, rcs, 0);
  thomas_sweep(B.ghat.p, B.W.p, P.rinvd.p, B.m, nc, nint, nullptr, s);
  // x faces: 8 layers by dot products along x; y faces: 4 + 4 rows by dot products along y
  partial_x(B.arith, B.W.p, m0, m1, m2, nullptr, B.S_fx.p, 4, B.X8.p, s, nc, nint, true);
  const size_t xcs = (size_t)8 * m1 * m2, ycs = (size_t)m0 * 4 * m2;
  double* Y4b = B.Y4.p + 3 * ycs;
  partial_y(B.arith, B.W.p, m0, m1, m2, nullptr, B.S_fy_lo.p, 4, B.Y4.p, s, nc, nint, Y4b);
  // one launch of inverse y transforms: the x-face layers and the first and
  // last 4 planes (z faces, in place on W after the dots) ...
  double* top = B.W.p + plane * (m2 - 4);
  const DstYLines ys[3] = {{&P.fy, B.X8.p, 8, m1, m2, xcs}, {&P.fy, B.W.p, m0, m1, 4, nint}, {&P.fy, top, m0, m1, 4, nint}};
  dst_lines_y_jobs(ys, 3, s, nc);
  scatter3(B.X8.p, 8, m1, m2, B.l_fx.p, nullptr, nullptr, 1, sol0, B.dims, s, nc, scs);
  // ... then inverse x transforms into sol0: the y-face rows, then the z
  // planes.  Jobs of one launch write disjoint nodes; where the rows and the
  // planes meet (box edges) the planes' launch writes last, every run.
  const DstXInvLines xr[2] = {
      {&P.fx, B.Y4.p, sol0, {B.dims[0], B.dims[1], B.dims[2]}, {1, 1, 1}, {m0, 4, m2}, ycs, scs},
      {&P.fx, Y4b, sol0, {B.dims[0], B.dims[1], B.dims[2]}, {1, 1 + m1 - 4, 1}, {m0, 4, m2}, ycs, scs}};
  dst_x_inv_jobs(xr, 2, s, nc);
  const DstXInvLines xz[2] = {
      {&P.fx, B.W.p, sol0, {B.dims[0], B.dims[1], B.dims[2]}, {1, 1, 1}, {m0, m1, 4}, nint, scs},
      {&P.fx, top, sol0, {B.dims[0], B.dims[1], B.dims[2]}, {1, 1, 1 + m2 - 4}, {m0, m1, 4}, nint, scs}};
  dst_x_inv_jobs(xz, 2, s, nc);
  VPMG_CUDA(cudaGetLastError());
}

void block_solve_bc(BlockSolve& B, DirichletPlan& P, double* sol, size_t scs, int nc, cudaStream_t s) {
  const int m0 = B.m[0], m1 = B.m[1], m2 = B.m[2];
  const size_t nint = (size_t)m0 * m1 * m2, plane = (size_t)m0 * m1;
  // boundary values of the faces, transformed along the face's axes
  const FaceTerms F = face_terms(P, B.f.p, B.e_x1.p, B.e_y1.p, sol, scs, nc, s);
  thomas_sweep(B.ghat.p, B.W.p, P.rinvd.p, B.m, nc, nint, &F, s);
  // dot products: the inner-box x faces along x, its y faces along y, and
  // the interior samples along y then x
  partial_x(B.arith, B.W.p, m0, m1, m2, nullptr, B.S_ix.p, 1, B.X2.p, s, nc, nint, true);
  const size_t xcs = (size_t)2 * m1 * m2, ycs = (size_t)m0 * m2;
  double* Y1b = B.Y1.p + 3 * ycs;
  partial_y(B.arith, B.W.p, m0, m1, m2, nullptr, B.S_iy_lo.p, 1, B.Y1.p, s, nc, nint, Y1b);
  partial_y(B.arith, B.W.p, m0, m1, B.nsz, B.l_sz.p, B.S_sy.p, B.nsy, B.Ys.p, s, nc, nint);
  partial_x(B.arith, B.Ys.p, m0, B.nsy, B.nsz, nullptr, B.S_sx.p, B.nsx, B.XS.p, s, nc, (size_t)m0 * B.nsy * B.nsz);
  scatter3(B.XS.p, B.nsx, B.nsy, B.nsz, B.l_sx.p, B.l_sy.p, B.l_idz.p, 0, sol, B.dims, s, nc, scs);
  // one launch of inverse y transforms: the x-face layers and the inner-box
  // z planes (in place on W, after the dots) ...
  double* pl0 = B.W.p + plane * B.inner_lo[2];
  double* pl1 = B.W.p + plane * B.inner_hi[2];
  const DstYLines ys[3] = {{&P.fy, B.X2.p, 2, m1, m2, xcs}, {&P.fy, pl0, m0, m1, 1, nint}, {&P.fy, pl1, m0, m1, 1, nint}};
  dst_lines_y_jobs(ys, 3, s, nc);
  scatter3(B.X2.p, 2, m1, m2, B.l_ix.p, nullptr, nullptr, 1, sol, B.dims, s, nc, scs);
  // ... then inverse x transforms into sol: the y-face rows, then the z
  // planes (jobs of one launch write disjoint nodes; at the box edges the
  // planes' launch writes last, every run)
  const int dm[3] = {B.dims[0], B.dims[1], B.dims[2]};
  const DstXInvLines xr[2] = {
      {&P.fx, B.Y1.p, sol, {dm[0], dm[1], dm[2]}, {1, B.inner_lo[1] + 1, 1}, {m0, 1, m2}, ycs, scs},
      {&P.fx, Y1b, sol, {dm[0], dm[1], dm[2]}, {1, B.inner_hi[1] + 1, 1}, {m0, 1, m2}, ycs, scs}};
  dst_x_inv_jobs(xr, 2, s, nc);
  const DstXInvLines xz[2] = {
      {&P.fx, pl0, sol, {dm[0], dm[1], dm[2]}, {1, 1, B.inner_lo[2] + 1}, {m0, m1, 1}, nint, scs},
      {&P.fx, pl1, sol, {dm[0], dm[1], dm[2]}, {1, 1, B.inner_hi[2] + 1}, {m0, m1, 1}, nint, scs}};
  dst_x_inv_jobs(xz, 2, s, nc);
  VPMG_CUDA(cudaGetLastError());
}

void FaceSolve::prepare(const DirichletPlan& P) {
  const int m0 = P.m[0], m1 = P.m[1];
  f.ensure(3 * face_doubles(P));
  std::vector<double> e((size_t)m0 + (size_t)m1);
  for (int p = 0; p < m0; ++p) e[p] = std::sin(kPI * (double)(p + 1) / (double)(m0 + 1));
  for (int q = 0; q < m1; ++q) e[m0 + q] = std::sin(kPI * (double)(q + 1) / (double)(m1 + 1));
  this->e.ensure(e.size());
  VPMG_CUDA(cudaMemcpy(this->e.p, e.data(), sizeof(double) * e.size(), cudaMemcpyHostToDevice));
  ready = true;
}

void dirichlet_solve_faces(DirichletPlan& P, FaceSolve& FS, const double* rhs, size_t rcs, double* sol, size_t scs,
                           int nc, double* work, double* out, cudaStream_t s) {
  VPMG_CHECK(FS.ready && nc >= 1 && nc <= 3, VPMG_ERR_STATE, "face solve not prepared");
  const int m0 = P.m[0], m1 = P.m[1], m2 = P.m[2];
  const size_t nint = (size_t)m0 * m1 * m2;
  // forward transforms of the RHS alone (zero tiles skip their FFTs)
  dst_forward_xy(P, rhs, nullptr, true, work, s, nc, rcs, 0);
  // the faces' values, transformed along their own axes; the sweep with
  // them, then the full inverse transforms
  const FaceTerms F = face_terms(P, FS.f.p, FS.e.p, FS.e.p + m0, sol, scs, nc, s);
  thomas_sweep(work, out, P.rinvd.p, P.m, nc, nint, &F, s);
  dst_inverse_xy(P, out, sol, s, nc, scs);
  VPMG_CUDA(cudaGetLastError());
}

}  // namespace vpmg
