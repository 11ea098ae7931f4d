// nearfield.cu -- the opened part of the boundary operator as exact products
// on the tensor cores.
//
// The walk of Bounds3d_lev / tree_calc_3d (source/pmbound.f90:980-1249) opens
// the cells closer than 10 sqrt(dS) to a boundary node.  With uniform cell
// lattices on every face (farfield.cu) the set of cells that a node takes
// from a level, and their weights dS/r, depend only on the node's position
// within the level's period (the parent cells' side) and on the cells'
// offsets: one small weight table per level and kind of face pair serves
// every node.  What the lattice rule and the walk decide differently (cells
// exactly on an opening radius in index units, where the walk's rounding
// decides) is found once at set-up and kept as correction rows.
//
// Tables: a node of face F sees, of face G,
//   * parallel pairs (the same face, or the opposite one where the box is
//     thin): cells in a window around it in both axes of the face;
//   * perpendicular pairs: with w the shared axis, nodes i steps from G's
//     plane and cells c deep from F's plane, in a window along w.
// Levels below the coarsest hold the accepted cells (+dS/r); the coarsest
// level, summed over all its cells by FFT, holds its opened ones (-dS/r).
//
// Product: rows of the A operand are runs of target nodes (a block of TB
// nodes along w, at one row base, for one component, face and side), its K
// the source cells of the window, the columns of the B operand the nodes of
// the block: D[run][node] = sum_cell S[run][cell] W[node][cell].  FP64 is two
// lanes per clock and SM here and tensor cores have no FP64 worth using, so
// both operands are 55-bit integers at a common scale (weights: per table,
// sources: per component), cut into seven balanced base-256 digits held as
// FP16.  Digit products d_i e_j with i + j <= 6 (28 of 49) accumulate in
// seven FP32 accumulators by i + j, exact while below 2^24, which 256 cells
// guarantee (checked against the table's digits); then the seven sums join
// as a 64-bit integer per node.  Of the dropped products the six with i + j = 7
// reach 2^-53.4 of a product's scale at worst; as digits of either sign they are a
// seventh of that (root mean square), below the rounding of an FP64 FMA chain.  Integer sums
// do not depend on the order, so units of work are dealt dynamically and
// added with 64-bit integer atomics, and results stay the same bits.
//
// Tile: M = 128 runs, N = 64 nodes: seven 64-column accumulators fill 448 of
// the 512 tensor-memory columns.  K = 16 per stage (43 KB: 28 KB of source
// digits gathered by 16-byte asynchronous copies, 14 KB of table by one bulk
// copy), five stages.  The products alone take about 53 clocks each at N = 64
// (their operands' shared-memory reads), 1480 a stage; reading the sums every
// 16 stages, when the tensor core waits, 400 more (57 thousand conversions to
// integers at 16 per clock).  One warp each for the products and the tables
// beside the gathering ones took the 81^3 block of a 64^3 step from 358 to
// 283 us and the 273^3 block of a 256^3 step from 1.50 to 1.21 ms; with one
// barrier of all threads per stage the next gather waited for the products.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "near_host.h"
#include "tc05.cuh"
#include "vpmg_internal.h"

namespace vpmg {

namespace {

constexpr int kWorkers = 256;               // threads that gather the sources and read the sums
constexpr int kThreads = kWorkers + 64;     // and a warp each for the tables and the products
constexpr int kStages = 5;
constexpr int kLag = 3;                     // stages whose copies a worker has in flight
constexpr int kDigits = kNearDigits;
constexpr int kRunsM = 128;   // runs per tile
constexpr int kCols = kNearCols;  // nodes per tile
constexpr int kGroup = 16;    // stages between reads of the accumulators (256 cells)
constexpr int kBytesA = kDigits * 2 * kRunsM * 16, kBytesB = kDigits * 2 * kCols * 16;
constexpr int kStageBytes = kBytesA + kBytesB;
constexpr int kSmem = kStages * kStageBytes + 1024;

// flags[(chunk * nrow + row) * nkp + kp]: whether the block of 64 nodes x 16
// cells has a weight; wmax: high word of the largest |weight| (a warp per block).
__global__ void k_near_flags(const __grid_constant__ NearTable T, unsigned char* __restrict__ flags,
                             unsigned* __restrict__ wmax) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (warp >= T.nchunk * T.nrow * T.nkp) return;
  const int kp = warp % T.nkp, row = (warp / T.nkp) % T.nrow, ch = warp / (T.nkp * T.nrow);
  unsigned m = 0;
  for (int n = lane; n < kCols; n += 32)
    for (int k = 0; k < 16; ++k)
      m = max(m, (unsigned)__double2hiint(near_weight(T, ch * kCols + n, row, kp * 16 + k)) & 0x7FFFFFFFu);
  m = __reduce_max_sync(0xffffffffu, m);
  if (lane == 0) {
    flags[warp] = m != 0;
    if (m) atomicMax(wmax, m);
  }
}

// Table blocks [digit][2][64][8] of the listed (row, kp), per node the sum of
// |weight| (wsum), and the largest sum of |digits 0..5| over a group of
// blocks (dmax).  blockIdx.y = tile of 64 nodes (span: its first list entry
// and their number), one CTA per group of kGroup blocks.
__global__ void __launch_bounds__(128) k_near_fill(const __grid_constant__ NearTable T, const int2* __restrict__ span,
                                                   const unsigned* __restrict__ klist, const unsigned* __restrict__ wmax,
                                                   uint4* __restrict__ out, unsigned long long* __restrict__ wsum,
                                                   unsigned* __restrict__ dmax) {
  const int n = threadIdx.x & 63, kg = threadIdx.x >> 6, ch = blockIdx.y;
  const int2 sp = span[ch];
  const int b0 = blockIdx.x * kGroup, b1 = min(sp.y, b0 + kGroup);
  if (b0 >= sp.y) return;  // whole CTA
  const int ew = tc05::scale_exp(*wmax);
  klist += sp.x;
  out += (size_t)sp.x * (kBytesB / 16);
  wsum += (size_t)ch * kCols;
  double ws = 0.0;
  unsigned ds = 0;
  for (int b = b0; b < b1; ++b) {
    const unsigned e = klist[b];
    const int row = (int)(e >> 8), kp = (int)(e & 255u);
    unsigned short d[8][kDigits];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const double w = near_weight(T, ch * kCols + n, row, kp * 16 + kg * 8 + k);
      ws += fabs(w);
      tc05::digits256(tc05::fixed55(w, ew), d[k]);
#pragma unroll
      for (int j = 0; j < 6; ++j) {
        const unsigned short h = d[k][j];
        float f;
        asm("{\n.reg .b16 t;\nmov.b16 t, %1;\ncvt.f32.f16 %0, t;\n}\n" : "=f"(f) : "h"(h));
        ds += (unsigned)fabsf(f);
      }
    }
#pragma unroll
    for (int j = 0; j < kDigits; ++j) {
      uint4 v;
      v.x = d[0][j] | (unsigned)d[1][j] << 16;
      v.y = d[2][j] | (unsigned)d[3][j] << 16;
      v.z = d[4][j] | (unsigned)d[5][j] << 16;
      v.w = d[6][j] | (unsigned)d[7][j] << 16;
      out[(size_t)b * (kBytesB / 16) + (j * 2 + kg) * kCols + n] = v;
    }
  }
  __shared__ double sw[128];
  __shared__ unsigned sd[128];
  sw[threadIdx.x] = ws;
  sd[threadIdx.x] = ds;
  __syncthreads();
  if (kg == 0) {
    atomicMax(dmax, sd[n] + sd[64 + n]);
    // an upper bound of the node's sum over groups: added as integers of 2^-20 of the scale, rounded up
    const double t = scalbn(sw[n] + sw[64 + n], 20 + 1022 - ew);
    atomicAdd(&wsum[n], (unsigned long long)t + 1ull);
  }
}

// Source digits of every level: cell (a, b) of face f into the row-along-u
// array (orient 0) and, near the edges, the row-along-v array (orient 1).
struct DigitsDev {
  int lev[kNearLevels + 1];                        // first cell of each level
  int off[kNearLevels][7], ma[kNearLevels][6], mb[kNearLevels][6];  // per level: cells before face f; lattice sides
  long long base[kNearLevels][2][6];               // FP16 offsets per orientation and face (component 0, digit 0)
  int Wp[kNearLevels][2][6];
  int edge;                                        // orient 1 rows nearer than this to either end are written
};
__global__ void k_near_sources(const __grid_constant__ DigitsDev D, const double* __restrict__ x, int ncell,
                               const unsigned* __restrict__ smax, unsigned short* __restrict__ dig) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ncell) return;
  int l = 0;
  while (t >= D.lev[l + 1]) ++l;
  const int i = t - D.lev[l];
  int f = 0;
  while (i >= D.off[l][f + 1]) ++f;
  const int k = i - D.off[l][f], ma = D.ma[l][f], mb = D.mb[l][f];
  const int a = k % ma, b = k / ma;
  const int c = blockIdx.y;
  unsigned short d[kDigits];
  tc05::digits256(tc05::fixed55(x[(size_t)c * ncell + t], tc05::scale_exp(smax[c])), d);
  const int W0 = D.Wp[l][0][f], W1 = D.Wp[l][1][f];
  const long long d0 = (long long)mb * W0, d1 = (long long)ma * W1;
  unsigned short* o0 = dig + D.base[l][0][f] + c * kDigits * d0 + (long long)b * W0 + a;
  unsigned short* o1 = dig + D.base[l][1][f] + c * kDigits * d1 + (long long)a * W1 + b;
  const bool e1 = a < D.edge || a >= ma - D.edge;
#pragma unroll
  for (int j = 0; j < kDigits; ++j) {
    o0[j * d0] = d[j];
    if (e1) o1[j * d1] = d[j];
  }
}

struct MmaArgs {
  const NearUnit* units;
  int nunit, group;
  const NearRow* rows;
  const unsigned* klist;
  const unsigned char* table;
  const unsigned short* dig;
  unsigned long long* acc;
  int polls;     // limit of every wait
  int* failed;   // set when one runs out (the boundary values are NaN then),
  int* status;   // and the handle's error word
};

// Units are dealt longest first, forth and back over the CTAs.  Warps 0..7
// gather the sources' digits and, at the end of a group of stages, read the
// sums; warp 8 loads the tables, warp 9 issues the products.  They meet in
// mbarriers only, and the gathers run ahead of the products across the ends of
// groups and units.  Every wait has a limit: whoever waited in vain stops, the
// others then wait in vain too, and all meet at the end, where the copies and
// products in flight are waited for before the CTA ends.
__global__ void __launch_bounds__(kThreads, 1) k_near_mma(const __grid_constant__ MmaArgs P) {
  extern __shared__ unsigned char near_sm[];
  __shared__ __align__(8) uint64_t bars[2 * kStages + 3];
  __shared__ uint32_t arrived[kWorkers / 32];  // stages that each gathering warp has filled
  __shared__ uint32_t tslot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t sm = (tc05::smem_u32(near_sm) + 1023u) & ~1023u;
  const uint32_t full = tc05::smem_u32(bars), empty = full + 8 * kStages, done = full + 16 * kStages, unread = done + 8,
                 drained = done + 16;
  if (warp == 0) tc05::tmem_alloc(tc05::smem_u32(&tslot), 512);
  if (tid == 0) {
    for (int i = 0; i < kStages; ++i) {
      tc05::bar_init(full + 8 * i, kWorkers / 32 + 1);  // the gathering warps and the table's copy
      tc05::bar_init(empty + 8 * i, 1);
    }
    tc05::bar_init(done, 1);
    tc05::bar_init(unread, kWorkers / 32);
    tc05::bar_init(drained, 1);
    tc05::bar_init_fence();
  }
  tc05::fence_before();
  __syncthreads();
  tc05::fence_after();
  const uint32_t tb = tslot;
  constexpr uint32_t idesc = tc05::idesc_f16(kRunsM, kCols);
  bool dead = false;
  uint32_t loads = 0;  // tables copied by this thread
  auto unit_of = [&](int i) {  // this CTA's i-th unit
    const long long u = (long long)i * gridDim.x + ((i & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
    return u < P.nunit ? (int)u : -1;
  };
  if (warp == kWorkers / 32) {
    if (lane == 0) {  // the tables
      uint32_t g = 0;
      for (int i = 0, u; !dead && (u = unit_of(i)) >= 0; ++i) {
        const NearUnit U = P.units[u];
        const unsigned char* src = P.table + U.table + (size_t)U.k0 * kBytesB;
        for (int k = U.k0; k < U.k1; ++k, ++g, src += kBytesB) {
          const uint32_t st = g % kStages;
          if (g >= (uint32_t)kStages) tc05::bar_wait(empty + 8 * st, ((g / kStages) - 1) & 1, dead, P.polls);
          if (dead) break;
          tc05::bar_expect(full + 8 * st, kBytesB);
          tc05::bulk_load(sm + st * kStageBytes + kBytesA, src, kBytesB, full + 8 * st);
          ++loads;
        }
      }
    }
    __syncwarp();
  } else if (warp > kWorkers / 32) {
    if (lane == 0) {  // the products
      uint32_t g = 0, groups = 0;
      for (int i = 0, u; !dead && (u = unit_of(i)) >= 0; ++i) {
        const int nst = P.units[u].k1 - P.units[u].k0;
        for (int k = 0; k < nst; ++k, ++g) {
          const uint32_t st = g % kStages;
          const int kin = k % P.group;
          if (kin == 0 && groups > 0) tc05::bar_wait(unread, (groups - 1) & 1, dead, P.polls);
          tc05::bar_wait(full + 8 * st, (g / kStages) & 1, dead, P.polls);
          if (dead) break;
          tc05::fence_after();
          const uint32_t base = sm + st * kStageBytes;
          const uint64_t da = tc05::desc(base, kRunsM * 16), db = tc05::desc(base + kBytesA, kCols * 16);
#pragma unroll
          for (int w = 0; w < kDigits; ++w)
#pragma unroll
            for (int j = 0; j < kDigits - w; ++j)
              tc05::mma(tb + (w + j) * kCols, da + (uint64_t)(j * (2 * kRunsM * 16 >> 4)),
                        db + (uint64_t)(w * (2 * kCols * 16 >> 4)), idesc, (w > 0 || kin > 0) ? 1u : 0u);
          tc05::commit(empty + 8 * st);
          if (kin == P.group - 1 || k == nst - 1) {
            tc05::commit(done);
            ++groups;
          }
        }
      }
    }
    __syncwarp();
  } else {
    // this thread's run and 8-cell group of a stage: eight neighbouring threads write 128 bytes
    const int r = 16 * warp + (lane & 15), kg = lane >> 4;
    const uint32_t adst = (uint32_t)((kg * kRunsM + r) * 16);
    // the gathers' place: unit, its stages, its run
    int ii = 0, iu = unit_of(0), ik = 0, in = 0;
    NearRow R{};
    const unsigned* kl = nullptr;
    unsigned e = 0;
    auto enter = [&] {
      if (iu < 0) return;
      const NearUnit U = P.units[iu];
      ik = 0;
      in = U.k1 - U.k0;
      kl = P.klist + U.klist + U.k0;
      e = __ldg(kl);
      R = NearRow{};
      if (r < U.nrun) R = P.rows[U.row0 + r];  // else no source row (nrow = 0)
    };
    enter();
    // the sums' place
    int ai = 0, au = iu, ak = 0, an = in, q = au >= 0 ? P.units[au].q : 0;
    uint32_t g = 0, ga = 0, groups = 0;
    long long sum[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) sum[i] = 0;
    for (int step = 0; au >= 0; ++step) {
      if (iu >= 0) {
        const uint32_t st = g % kStages;
        const int row = R.row0 + R.rs * (int)(e >> 8), cell = R.wst + 16 * (int)(e & 255u) + 8 * kg;
        const bool ok = row >= 0 && row < R.nrow && cell >= 0 && cell < R.Wp;
        const unsigned short* src = P.dig + (ok ? R.abase + (long long)row * R.Wp + cell : 0);
        const long long ds = ok ? (long long)R.nrow * R.Wp : 0;
        if (ik + 1 < in) e = __ldg(kl + ik + 1);
        if (g >= (uint32_t)kStages) tc05::bar_wait(empty + 8 * st, ((g / kStages) - 1) & 1, dead, P.polls);
        if (__any_sync(0xffffffffu, dead)) {
          dead = true;
          break;
        }
        const uint32_t dst = sm + st * kStageBytes + adst;
#pragma unroll
        for (int j = 0; j < kDigits; ++j) tc05::cp16(dst + j * (2 * kRunsM * 16), src + j * ds, ok);
        ++g;
        if (++ik == in) {
          iu = unit_of(++ii);
          enter();
        }
      }
      tc05::cp_commit();
      if (step < kLag) continue;
      // the copies of kLag steps ago are in
      tc05::cp_wait<kLag>();
      tc05::fence_async();
      __syncwarp();
      if (lane == 0) tc05::bar_arrive(full + 8 * (ga % kStages));
      ++ga;
      ++ak;
      if (ak % P.group != 0 && ak != an) continue;
      // the group's exact sums join the running integers
      tc05::bar_wait(done, groups & 1, dead, P.polls);
      if (__any_sync(0xffffffffu, dead)) {
        dead = true;
        break;
      }
      ++groups;
      tc05::fence_after();
      const uint32_t ta = tb + ((uint32_t)(32 * (warp & 3)) << 16) + 32 * (warp >> 2);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        uint32_t v[kDigits][4];
#pragma unroll
        for (int d = 0; d < kDigits; ++d) tc05::ld4(ta + d * kCols + 4 * c, v[d]);
        tc05::ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          auto n = [&](int d) { return (long long)__float2int_rn(__uint_as_float(v[d][i])); };
          const long long hi = (n(0) << 32) + (n(1) << 24) + (n(2) << 16) + (n(3) << 8) + n(4);
          const long long lo = (n(5) << 8) + n(6);
          sum[4 * c + i] += (hi << (16 - q)) + ((lo + ((1ll << q) >> 1)) >> q);
        }
      }
      tc05::fence_before();
      __syncwarp();
      if (lane == 0) tc05::bar_arrive(unread);  // the next products may overwrite
      if (ak != an) continue;
      // row `run` of the tile, columns 32 (warp / 4) ..
      const NearUnit U = P.units[au];
      const int run = 32 * (warp & 3) + lane;
      if (run < U.nrun) {
        const NearRow O = P.rows[U.row0 + run];
        const long long half = (1ll << U.sh) >> 1;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int n = U.col0 + 32 * (warp >> 2) + i;
          const int tr = n / U.TB, tw = n - tr * U.TB;
          if (tr < O.rlim && tw < O.wlim)
            atomicAdd(&P.acc[O.obase + (long long)tr * O.ostr_r + (long long)tw * O.ostr_w],
                      (unsigned long long)((sum[i] + half) >> U.sh));
        }
      }
#pragma unroll
      for (int i = 0; i < 32; ++i) sum[i] = 0;
      au = unit_of(++ai);
      ak = 0;
      if (au >= 0) {
        an = P.units[au].k1 - P.units[au].k0;
        q = P.units[au].q;
      }
    }
    tc05::cp_wait<0>();
    if (lane == 0) arrived[warp] = ga;
  }
  if (__syncthreads_or(dead)) {
    bool late = false;  // these waits have the full limit
    if (warp == kWorkers / 32 && lane == 0)
      // the last copy into each stage, with the arrivals of the gathering warps
      // that stopped before it (one at most: a stage is loaded again only once
      // all of them have filled it and its products are done)
      for (uint32_t i = 0; i < (uint32_t)kStages && i < loads; ++i) {
        const uint32_t last = (loads - i - 1) / kStages;
        for (int w = 0; w < kWorkers / 32; ++w)
          if (arrived[w] <= i + last * kStages) tc05::bar_arrive(full + 8 * i);
        tc05::bar_wait(full + 8 * i, last & 1, late, tc05::kPolls);
      }
    if (warp == kWorkers / 32 + 1 && lane == 0) {
      tc05::commit(drained);
      tc05::bar_wait(drained, 0, late, tc05::kPolls);
    }
    if (tid == 0) {
      atomicExch(P.failed, 1);
      if (P.status) atomicMax(P.status, kErrWait);
    }
    __syncthreads();
  }
  if (warp == 0) tc05::tmem_free(tb, 512);
}

// ---- the walk against the lattice rule -------------------------------------
struct DiffDev {
  const double *cx, *cy, *cz, *cds, *cthr, *tx, *ty, *tz;
  const int *child, *tgt_node;
  int ntarget, levmax;
  int lev_off[kNearLevels + 1];
  int cell0[kNearLevels][7], ma[kNearLevels][6];
  int N[3];
  double h[3];
  double ds[kNearLevels][3], thr2[kNearLevels][3];  // per level and source normal
};
// Counts (FILL = false) or writes the cells that a node's walk and the
// lattice rule take differently: the walk's with weight dS/r, the rule's
// with -dS/r, and both where only one sees the cell within the 1e-5 of length
// at which the weight changes.  Decisions away from a radius are made in FP32
// (both sides agree there); within 1e-4 of one the walk's own expressions
// decide for the walk and lattice_r2 (lattice_close) for the rule.  FINE: some
// cell can lie that close (looking for them on every mesh doubled the set-up of
// 256^3, 180 to 350 ms).
template <bool FILL, bool FINE>
__global__ void k_near_diff(const __grid_constant__ DiffDev D, int* __restrict__ counts,
                            unsigned long long* __restrict__ accepted, const long long* __restrict__ rowptr,
                            int* __restrict__ col, double* __restrict__ wgt) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x, f = blockIdx.y;  // a node and a source face
  const unsigned valid = __ballot_sync(0xffffffffu, t < D.ntarget);
  if (t >= D.ntarget) return;
  const double X = D.tx[t], Y = D.ty[t], Z = D.tz[t];
  const int node = D.tgt_node[t];
  const int ti[3] = {node % D.N[0], (node / D.N[0]) % D.N[1], node / (D.N[0] * D.N[1])};
  const float hf[3] = {(float)D.h[0], (float)D.h[1], (float)D.h[2]};
  int cnt = 0;
  unsigned na = 0, nd = 0;
  long long out = FILL ? rowptr[6 * (size_t)t + f] : 0;
  auto emit = [&](int c, double w) {
    if (FILL) {
      col[out] = c;
      wgt[out] = w;
      ++out;
    } else {
      ++cnt;
    }
  };
  int pa[kNearLevels], pb[kNearLevels], pc[kNearLevels], pos[kNearLevels], mode[kNearLevels];
  {
    const int fu = face_u(f), fv = face_v(f), fn = f >> 1, L = D.levmax;
    const int n = D.cell0[L][f + 1] - D.cell0[L][f];
    int l = L;
    pos[L] = 0;
    for (;;) {
      int a, b, c, md;
      if (l == L) {
        if (pos[L] >= n) break;
        a = pos[L] % D.ma[L][f];
        b = pos[L] / D.ma[L][f];
        c = D.lev_off[L] + D.cell0[L][f] + pos[L]++;
        md = 3;
      } else {
        if (pos[l] >= 4) {
          ++l;
          continue;
        }
        const int k = pos[l]++;
        // children in the order (0,0), (1,0), (1,1), (0,1)
        a = 2 * pa[l] + ((k == 1 || k == 2) ? 1 : 0);
        b = 2 * pb[l] + (k >= 2 ? 1 : 0);
        c = D.child[4 * (size_t)pc[l] + k];
        md = mode[l];
      }
      const int s = 1 << l;
      int o2[3];  // twice the centre, in nodes
      o2[fn] = 2 * ((f & 1) ? D.N[fn] - 1 : 0);
      o2[fu] = 2 * a * s + s;
      o2[fv] = 2 * b * s + s;
      bool wo = false, ro = false;
      // FP64 only where a decision is close: these run for one pair in thousands
      auto off = [&](int a) { return 0.5 * (double)(2 * ti[a] - o2[a]); };
      auto walk_r = [&] {
        const double XR = __dsub_rn(D.cx[c], X), YR = __dsub_rn(D.cy[c], Y), ZR = __dsub_rn(D.cz[c], Z);
        return __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(XR, XR), __dmul_rn(YR, YR)), __dmul_rn(ZR, ZR)));
      };
      auto walk_weight = [&](double rr) {
        return rr > 1e-05 ? __ddiv_rn(D.cds[c], rr) : -2.0 * __dsqrt_rn(D.cds[c]) * kPanelLog;
      };
      auto rule_weight = [&] {
        return lattice_weight(D.ds[l][fn], off(fu), D.h[fu], off(fv), D.h[fv], off(fn), D.h[fn]);
      };
      float r2 = 0.f;
      if (FINE || l > 0) {
        const float ex = 0.5f * (float)(2 * ti[0] - o2[0]) * hf[0], ey = 0.5f * (float)(2 * ti[1] - o2[1]) * hf[1],
                    ez = 0.5f * (float)(2 * ti[2] - o2[2]) * hf[2];
        r2 = ex * ex + ey * ey + ez * ez;
      }
      if (l > 0) {
        const float th = (float)D.thr2[l][fn];
        if (fabsf(r2 - th) > 1e-4f * th) {
          wo = ro = r2 < th;
        } else {
          wo = walk_r() < D.cthr[c];
          ro = lattice_r2(off(fu), D.h[fu], off(fv), D.h[fv], off(fn), D.h[fn]) < D.thr2[l][fn];
        }
      }
      const bool w = md & 1, g = md & 2;
      const bool wa = w && !wo, ra = g && !ro;
      if (wa) {
        if (l == L) ++nd;
        else ++na;
      }
      if (wa != ra) {
        if (wa) emit(c, walk_weight(walk_r()));
        else emit(c, -rule_weight());
      } else if (FINE && wa && !(fabsf(r2 - 1e-10f) > 1e-14f)) {
        const double rr = walk_r();
        if ((rr > 1e-05) == lattice_close(off(fu), D.h[fu], off(fv), D.h[fv], off(fn), D.h[fn])) {
          emit(c, walk_weight(rr));
          emit(c, -rule_weight());
        }
      }
      const int cm = ((w && wo) ? 1 : 0) | ((g && ro) ? 2 : 0);
      if (cm && l > 0) {
        --l;
        pa[l] = a;
        pb[l] = b;
        pc[l] = c;
        mode[l] = cm;
        pos[l] = 0;
      }
    }
  }
  if (!FILL) {
    counts[6 * (size_t)t + f] = cnt;
    __syncwarp(valid);
    na = __reduce_add_sync(valid, na);
    nd = __reduce_add_sync(valid, nd);
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(&accepted[0], (unsigned long long)na);
      atomicAdd(&accepted[1], (unsigned long long)nd);
    }
  }
}

template <class T>
void up(DBuf<T>& b, const std::vector<T>& h) {
  b.ensure(std::max<size_t>(h.size(), 1));
  if (!h.empty()) VPMG_CUDA(cudaMemcpy(b.p, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice));
}

constexpr int kMaxDev = 64;
bool g_smem_set[kMaxDev] = {false};

}  // namespace

long long NearField::bytes() const {
  return (long long)(table.bytes() + dig.bytes() + acc.bytes() + rows.bytes() + units.bytes() + klist.bytes());
}

void near_release(BoundaryOp& B) {
  NearField& F = B.near;
  F.on = false;
  F.table.release(); F.dig.release(); F.acc.release(); F.rows.release(); F.units.release(); F.klist.release();
}

bool near_prepare(BoundaryOp& B, const Grid& g, long long budget_bytes, cudaStream_t s) {
  near_release(B);
  NearField& F = B.near;
  F.polls = wait_polls();
  const int L = B.levmax;
  NearPlan P;
  if (!build_near_plan(g.n, g.d, L, P)) return false;
  for (int l = 0; l <= L; ++l)
    if (P.cell0[l][6] != B.nbound_lev[l]) return false;
  std::memcpy(F.cell0, P.cell0, sizeof(F.cell0));
  std::memcpy(F.ma, P.ma, sizeof(F.ma));
  std::memcpy(F.mb, P.mb, sizeof(F.mb));
  std::memcpy(F.Wp, P.Wp, sizeof(F.Wp));
  std::memcpy(F.dbase, P.dbase, sizeof(F.dbase));
  std::memcpy(F.abase, P.abase, sizeof(F.abase));
  const long long nd = P.ndig, na = P.nacc;
  F.nacc = na;
  F.edge = P.edge;
  std::vector<NearTable>& tabs = P.tabs;
  std::vector<std::vector<NearRow>>& runs = P.runs;
  // ---- table contents --------------------------------------------------------
  const int nt = (int)tabs.size();
  DBuf<unsigned> wmax;
  wmax.ensure(nt + 1);
  VPMG_CUDA(cudaMemsetAsync(wmax.p, 0, sizeof(unsigned) * (nt + 1), s));
  std::vector<std::vector<unsigned char>> flags(nt);
  size_t fmax = 1;
  for (auto& T : tabs) {
    if (T.nkp > 255 || T.nkp < 1 || T.nrow < 1) return false;
    fmax += (size_t)T.nchunk * T.nrow * T.nkp;
  }
  DBuf<unsigned char> dflags;
  dflags.ensure(fmax);
  size_t fo = 0;
  for (int t = 0; t < nt; ++t) {
    const size_t nb = (size_t)tabs[t].nchunk * tabs[t].nrow * tabs[t].nkp;
    k_near_flags<<<(unsigned)((nb * 32 + 255) / 256), 256, 0, s>>>(tabs[t], dflags.p + fo, wmax.p + t);
    VPMG_LAUNCHED();
    fo += nb;
  }
  VPMG_CUDA(cudaGetLastError());
  std::vector<unsigned char> hf(fo);
  std::vector<unsigned> hw(nt + 1);
  VPMG_CUDA(cudaMemcpyAsync(hf.data(), dflags.p, fo, cudaMemcpyDeviceToHost, s));
  VPMG_CUDA(cudaMemcpyAsync(hw.data(), wmax.p, sizeof(unsigned) * nt, cudaMemcpyDeviceToHost, s));
  VPMG_CUDA(cudaStreamSynchronize(s));
  std::vector<unsigned> kl;
  std::vector<std::vector<std::pair<int, int>>> span(nt);  // per chunk: first list entry, entries
  fo = 0;
  for (int t = 0; t < nt; ++t) {
    const NearTable& T = tabs[t];
    for (int ch = 0; ch < T.nchunk; ++ch) {
      const int k0 = (int)kl.size();
      for (int row = 0; row < T.nrow; ++row)
        for (int kp = 0; kp < T.nkp; ++kp, ++fo)
          if (hf[fo]) kl.push_back((unsigned)row << 8 | (unsigned)kp);
      span[t].push_back({k0, (int)kl.size() - k0});
    }
  }
  const long long tbytes = (long long)kl.size() * kBytesB;
  size_t free_b = 0, total_b = 0;
  VPMG_CUDA(cudaMemGetInfo(&free_b, &total_b));
  if (tbytes + 2 * nd + 8 * na > budget_bytes || tbytes + 2 * nd + 8 * na > (long long)(0.5 * (double)free_b)) return false;
  up(F.klist, kl);
  F.table.ensure(std::max<size_t>((size_t)tbytes, 16));
  F.dig.ensure((size_t)nd + 64);
  VPMG_CUDA(cudaMemsetAsync(F.dig.p, 0, F.dig.bytes(), s));
  F.acc.ensure((size_t)na + 1);  // the sums, then the failure flag (second int)
  std::vector<size_t> col0(nt + 1, 0);  // first node of each table in wsum
  for (int t = 0; t < nt; ++t) col0[t + 1] = col0[t] + (size_t)tabs[t].nchunk * kCols;
  DBuf<unsigned long long> wsum;
  wsum.ensure(col0[nt]);
  VPMG_CUDA(cudaMemsetAsync(wsum.p, 0, wsum.bytes(), s));
  std::vector<int2> hspan;
  for (int t = 0; t < nt; ++t)
    for (auto& c : span[t]) hspan.push_back(make_int2(c.first, c.second));
  DBuf<int2> dspan;
  up(dspan, hspan);
  size_t so = 0;
  for (int t = 0; t < nt; ++t) {
    int most = 0;
    for (auto& c : span[t]) most = std::max(most, c.second);
    if (most) {
      k_near_fill<<<dim3((unsigned)((most + kGroup - 1) / kGroup), (unsigned)tabs[t].nchunk), 128, 0, s>>>(
          tabs[t], dspan.p + so, F.klist.p, wmax.p + t, reinterpret_cast<uint4*>(F.table.p), wsum.p + col0[t],
          wmax.p + nt);
      VPMG_LAUNCHED();
    }
    so += span[t].size();
  }
  VPMG_CUDA(cudaGetLastError());
  std::vector<unsigned long long> hs(col0[nt]);
  unsigned dmax = 0;
  VPMG_CUDA(cudaMemcpyAsync(hs.data(), wsum.p, wsum.bytes(), cudaMemcpyDeviceToHost, s));
  VPMG_CUDA(cudaMemcpyAsync(&dmax, wmax.p + nt, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
  VPMG_CUDA(cudaStreamSynchronize(s));
  // digits of a source are at most 128: the accumulators of a group stay
  // exact while 128 * sum |digits 0..5| <= 2^24 (the last accumulator's
  // rounding is far below the result's)
  F.group = kGroup;
  while (F.group > 1 && 128.0 * (double)dmax * F.group / kGroup > 16777216.0) F.group /= 2;
  // ---- scales ---------------------------------------------------------------
  // A node's weights sum to at most bound; its 64-bit integer then has the
  // unit 2^uc, bound * 2^55 / 2^uc <= 2^62.
  std::vector<double> sumw(nt);
  double bound = 0.0;
  for (int t = 0; t < nt; ++t) {
    const int ew = std::max((int)(hw[t] >> 20), 1);
    unsigned long long m = 0;
    for (size_t n = col0[t]; n < col0[t + 1]; ++n) m = std::max(m, hs[n]);
    sumw[t] = std::ldexp((double)m, ew - 1022 - 20);
    bound += (tabs[t].par ? 1.0 : 4.0) * sumw[t];
  }
  if (!(bound > 0.0)) return false;
  F.uc = (int)std::ceil(std::log2(bound)) - 7 + 1;
  // ---- units of work ----------------------------------------------------------
  long long stages = 0;
  std::vector<NearRow> allrows;
  std::vector<NearUnit> units;
  for (int t = 0; t < nt; ++t)
    for (auto& c : span[t]) stages += (long long)c.second * ((runs[t].size() + kRunsM - 1) / kRunsM);
  int dev = 0, sms = 152;
  VPMG_CUDA(cudaGetDevice(&dev));
  VPMG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  // stages per unit: about six units per SM, at least one group
  long long per = (stages / (6LL * sms) + kGroup) / kGroup * kGroup;
  per = std::max<long long>(per, kGroup);
  for (int t = 0; t < nt; ++t) {
    const NearTable& T = tabs[t];
    if (!hw[t]) continue;  // no weight: a face exactly an opening radius away
    const int ew = std::max((int)(hw[t] >> 20), 1);
    const int q = std::max(0, (int)std::ceil(std::log2(std::max(sumw[t], 1e-300))) - ew + 1022 + 1);
    const int sh = F.uc - 48 - q - ew + 1077;
    if (q > 16 || sh < 0 || sh > 62) { near_release(B); return false; }
    const int row0 = (int)allrows.size();
    allrows.insert(allrows.end(), runs[t].begin(), runs[t].end());
    for (size_t m = 0; m < runs[t].size(); m += kRunsM)
      for (int ch = 0; ch < T.nchunk; ++ch) {
        const auto [k0, nk] = span[t][ch];
        for (long long a = 0; a < nk; a += per) {
          NearUnit U{};
          U.row0 = row0 + (int)m;
          U.nrun = (int)std::min<size_t>(kRunsM, runs[t].size() - m);
          U.klist = k0;
          U.table = (long long)k0 * kBytesB;
          U.k0 = (int)a;
          U.k1 = (int)std::min<long long>(nk, a + per);
          U.col0 = ch * kCols;
          U.TB = T.TB;
          U.q = q;
          U.sh = sh;
          units.push_back(U);
        }
      }
  }
  std::stable_sort(units.begin(), units.end(), [](const NearUnit& a, const NearUnit& b) { return a.k1 - a.k0 > b.k1 - b.k0; });
  up(F.rows, allrows);
  up(F.units, units);
  F.nunit = (int)units.size();
  F.stages = stages;
  F.sms = sms;
  // ---- the walk against the rule ----------------------------------------------
  DiffDev D{};
  D.cx = B.cx.p; D.cy = B.cy.p; D.cz = B.cz.p; D.cds = B.cds.p; D.cthr = B.cthr.p;
  D.tx = B.tx.p; D.ty = B.ty.p; D.tz = B.tz.p; D.child = B.child.p; D.tgt_node = B.tgt_node.p;
  D.ntarget = B.ntarget;
  D.levmax = L;
  for (int l = 0; l <= L; ++l) {
    D.lev_off[l] = B.lev_off[l];
    for (int f = 0; f < 7; ++f) D.cell0[l][f] = F.cell0[l][f];
    for (int f = 0; f < 6; ++f) D.ma[l][f] = F.ma[l][f];
    for (int a = 0; a < 3; ++a) {
      D.ds[l][a] = near_area(g.d, l, a);
      D.thr2[l][a] = near_thr2(g.d, l, a);
    }
  }
  for (int a = 0; a < 3; ++a) { D.N[a] = g.n[a]; D.h[a] = g.d[a]; }
  DBuf<int> counts;
  DBuf<unsigned long long> acc2;
  counts.ensure(6 * (size_t)B.ntarget);
  acc2.ensure(2);
  VPMG_CUDA(cudaMemsetAsync(acc2.p, 0, 2 * sizeof(unsigned long long), s));
  const dim3 blocks((unsigned)((B.ntarget + 127) / 128), 6);
  // leaf centres are at least half a diagonal from every node
  const bool fine = std::min({g.d[0], g.d[1], g.d[2]}) < 2e-5;
  if (fine) k_near_diff<false, true><<<blocks, 128, 0, s>>>(D, counts.p, acc2.p, nullptr, nullptr, nullptr);
  else k_near_diff<false, false><<<blocks, 128, 0, s>>>(D, counts.p, acc2.p, nullptr, nullptr, nullptr);
  VPMG_LAUNCHED();
  const size_t nrow = 6 * (size_t)B.ntarget;  // a node's row: its six faces' in turn
  std::vector<int> hc(nrow);
  unsigned long long ha[2];
  VPMG_CUDA(cudaMemcpyAsync(hc.data(), counts.p, sizeof(int) * nrow, cudaMemcpyDeviceToHost, s));
  VPMG_CUDA(cudaMemcpyAsync(ha, acc2.p, sizeof(ha), cudaMemcpyDeviceToHost, s));
  VPMG_CUDA(cudaStreamSynchronize(s));
  std::vector<long long> rp(nrow + 1, 0);
  for (size_t t = 0; t < nrow; ++t) rp[t + 1] = rp[t] + hc[t];
  FarField& FF = B.ff;
  FF.ncorr = rp[nrow];
  up(FF.crow, rp);
  FF.ccol.ensure((size_t)std::max<long long>(FF.ncorr, 1));
  FF.cw.ensure((size_t)std::max<long long>(FF.ncorr, 1));
  if (FF.ncorr) {
    if (fine) k_near_diff<true, true><<<blocks, 128, 0, s>>>(D, nullptr, nullptr, FF.crow.p, FF.ccol.p, FF.cw.p);
    else k_near_diff<true, false><<<blocks, 128, 0, s>>>(D, nullptr, nullptr, FF.crow.p, FF.ccol.p, FF.cw.p);
    VPMG_LAUNCHED();
  }
  VPMG_CUDA(cudaGetLastError());
  B.nnz = (long long)ha[0];
  B.ndense_acc = (long long)ha[1];
  VPMG_CHECK(dev >= 0 && dev < kMaxDev, VPMG_ERR_UNSUPPORTED, "device index beyond the per-device tables");
  if (!g_smem_set[dev]) {
    VPMG_CUDA(cudaFuncSetAttribute(k_near_mma, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    g_smem_set[dev] = true;
  }
  VPMG_CUDA(cudaStreamSynchronize(s));
  F.on = true;
  return true;
}

// acc[face][component][v][u] = the near field's integers of every face node.
void near_apply(BoundaryOp& B, cudaStream_t s) {
  NearField& F = B.near;
  VPMG_CUDA(cudaMemsetAsync(F.acc.p, 0, F.acc.bytes(), s));  // and the flag behind the sums
  DigitsDev D{};
  for (int l = 0; l <= B.levmax; ++l) {
    D.lev[l] = B.lev_off[l];
    D.lev[l + 1] = B.lev_off[l + 1];
    for (int f = 0; f < 7; ++f) D.off[l][f] = F.cell0[l][f];
    for (int f = 0; f < 6; ++f) {
      D.ma[l][f] = F.ma[l][f];
      D.mb[l][f] = F.mb[l][f];
      for (int o = 0; o < 2; ++o) {
        D.base[l][o][f] = F.dbase[l][o][f];
        D.Wp[l][o][f] = F.Wp[l][o][f];
      }
    }
  }
  D.edge = F.edge;
  k_near_sources<<<dim3((unsigned)((B.ncell_total + 255) / 256), 3), 256, 0, s>>>(D, B.csrc.p, B.ncell_total, B.smax.p,
                                                                                 F.dig.p);
  VPMG_LAUNCHED();
  MmaArgs A{};
  A.units = F.units.p;
  A.nunit = F.nunit;
  A.group = F.group;
  A.rows = F.rows.p;
  A.klist = F.klist.p;
  A.table = F.table.p;
  A.dig = F.dig.p;
  A.acc = F.acc.p;
  A.failed = reinterpret_cast<int*>(F.acc.p + F.nacc) + 1;
  A.polls = F.polls;
  A.status = B.status;
  k_near_mma<<<std::min(F.nunit, F.sms), kThreads, kSmem, s>>>(A);
  VPMG_LAUNCHED();
  VPMG_CUDA(cudaGetLastError());
}

}  // namespace vpmg
