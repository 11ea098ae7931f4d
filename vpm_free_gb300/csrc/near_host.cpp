// near_host.cpp -- which weight tables the near field needs on a grid, and for
// every table the runs of target nodes that use it: where a run's source
// cells lie in the digit arrays and where its sums go (nearfield.cu).
// Compiled with -ffp-contract=off, as the other mesh geometry.
#include <algorithm>
#include <cmath>
#include <map>
#include <tuple>

#include "near_host.h"

namespace vpmg {

bool lattice_exact(const double xmin[3], const double d[3], const int n[3]) {
  for (int a = 0; a < 3; ++a) {
    double node = 0.0, leaf = 0.0;
    for (int i = 0; i < n[a]; ++i) {
      // the tree's coordinates (build_tree_geometry)
      const double x0 = xmin[a] + (double)i * d[a], x1 = xmin[a] + (double)(i + 1) * d[a];
      node = std::max(node, std::fabs((x0 - xmin[a]) - (double)i * d[a]));
      if (i == n[a] - 1) continue;
      for (double c : {0.25 * (((x0 + x0) + x1) + x1), 0.25 * (((x1 + x1) + x0) + x0), 0.25 * (((x0 + x1) + x1) + x0)})
        leaf = std::max(leaf, std::fabs((c - xmin[a]) - ((double)i + 0.5) * d[a]));
    }
    if (!(node + leaf <= 4e-11 * d[a])) return false;
  }
  return true;
}

bool build_near_plan(const int n3[3], const double d3[3], int L, NearPlan& P) {
  if (L < 1 || L >= kNearLevels) return false;
  int M[kNearLevels][3];  // cells per level and axis
  for (int a = 0; a < 3; ++a) {
    if ((n3[a] - 1) % (1 << L) != 0 || n3[a] - 1 <= (1 << L)) return false;
    for (int l = 0; l <= L; ++l) M[l][a] = (n3[a] - 1) >> l;
  }
  for (int l = 0; l <= L; ++l) {
    int n = 0;
    for (int f = 0; f < 6; ++f) {
      P.cell0[l][f] = n;
      P.ma[l][f] = M[l][face_u(f)];
      P.mb[l][f] = M[l][face_v(f)];
      n += M[l][face_u(f)] * M[l][face_v(f)];
    }
    P.cell0[l][6] = n;
  }
  auto area = [&](int l, int fn) { return near_area(d3, l, fn); };
  auto thr2 = [&](int l, int fn) { return near_thr2(d3, l, fn); };
  // ---- source digit arrays and the sums' layout ----------------------------
  long long nd = 0;
  for (int l = 0; l <= L; ++l)
    for (int o = 0; o < 2; ++o)
      for (int f = 0; f < 6; ++f) {
        const int w = o ? face_v(f) : face_u(f), r = o ? face_u(f) : face_v(f);
        P.Wp[l][o][f] = (M[l][w] + 7) & ~7;
        P.dbase[l][o][f] = nd;
        nd += 3LL * kNearDigits * M[l][r] * P.Wp[l][o][f];
      }
  long long na = 0;
  for (int f = 0; f < 6; ++f) {
    P.abase[f] = na;
    na += 3LL * n3[face_u(f)] * n3[face_v(f)];
  }
  P.nacc = na;
  P.ndig = nd;
  // ---- tables and the runs that use them -----------------------------------
  std::vector<NearTable>& tabs = P.tabs;
  std::vector<std::vector<NearRow>>& runs = P.runs;
  std::map<std::tuple<int, int, double, double, double, int, int>, int> seen;
  int edge = 0;
  auto window = [&](int s, int top, double hh, double thr, int span, int* lo, int* hi) {
    // cells whose opening centre lies within thr of some node 0..span-1, along one axis
    const int far = (int)(thr / (hh * s)) + span / s + 4;
    *lo = 1 << 30;
    *hi = -(1 << 30);
    for (int c = -far; c <= far; ++c) {
      const double centre = top ? s * (c + 0.5) : 2.0 * s * (floor_half(c) + 0.5);
      const double d = std::max(0.0, std::max(-centre, centre - (span - 1)));
      if (d * hh < thr) {
        *lo = std::min(*lo, c);
        *hi = std::max(*hi, c);
      }
    }
  };
  for (int l = 0; l <= L; ++l) {
    const int s = 1 << l, top = l == L ? 1 : 0;
    const int TB = 16 * s;
    auto common = [&](NearTable& T, int fn, double thr) {
      T.s = s;
      T.top = top;
      T.TB = TB;
      T.ds = area(l, fn);
      T.thr2_own = l > 0 ? thr2(l, fn) : 0.0;
      T.thr2_out = top ? 0.0 : thr2(l + 1, fn);
      int lo, hi;
      window(s, top, T.hw, thr, TB, &lo, &hi);
      T.w0 = (lo >= 0 ? lo / 8 : -((-lo + 7) / 8)) * 8;
      T.nkp = (hi + 1 - T.w0 + 15) / 16;
      T.nchunk = (T.TB * T.rows + kNearCols - 1) / kNearCols;
    };
    for (int fn = 0; fn < 3; ++fn) {
      // parallel pairs: w = u, rows along v
      const int fu = face_u(2 * fn), fv = face_v(2 * fn);
      // a little more than the radius: the tables decide the ties
      const double thr = (1.0 + 1e-9) * std::sqrt(top ? thr2(l, fn) : thr2(l + 1, fn));
      for (int opp = 0; opp < 2; ++opp) {
        const int dn = opp ? n3[fn] - 1 : 0;
        if (!((double)dn * d3[fn] < thr)) continue;
        const int RB = top ? s : std::max(4, 2 * s);
        const auto key = std::make_tuple(l, 1, d3[fu], d3[fv], d3[fn], dn, 0);
        if (!seen.count(key)) {
          NearTable T{};
          T.par = 1;
          T.rows = RB;
          T.dn = dn;
          T.hw = d3[fu]; T.hr = d3[fv]; T.hn = d3[fn];
          common(T, fn, thr);
          int lo, hi;
          window(s, top, T.hr, thr, RB, &lo, &hi);
          T.r0 = lo;
          T.nrow = hi - lo + 1;
          seen[key] = (int)tabs.size();
          tabs.push_back(T);
          runs.emplace_back();
        }
        const int ti = seen[key];
        const NearTable& T = tabs[ti];
        for (int side = 0; side < 2; ++side) {
          const int ft = 2 * fn + side, G = opp ? ft ^ 1 : ft;
          for (int c = 0; c < 3; ++c)
            for (int rb = 0; rb * RB < n3[fv]; ++rb)
              for (int wb = 0; wb * TB < n3[fu]; ++wb) {
                NearRow R{};
                R.Wp = P.Wp[l][0][G];
                R.nrow = M[l][fv];
                R.abase = P.dbase[l][0][G] + (long long)c * kNearDigits * R.nrow * R.Wp;
                R.rs = 1;
                R.row0 = rb * (RB / s) + T.r0;
                R.wst = wb * 16 + T.w0;
                R.obase = P.abase[ft] + (long long)c * n3[fu] * n3[fv] + (long long)rb * RB * n3[fu] + wb * TB;
                R.ostr_r = n3[fu];
                R.ostr_w = 1;
                R.rlim = std::min(RB, n3[fv] - rb * RB);
                R.wlim = std::min(TB, n3[fu] - wb * TB);
                runs[ti].push_back(R);
              }
        }
      }
      // perpendicular pairs: source normal fn, target normal nf, shared axis w
      for (int nf = 0; nf < 3; ++nf) {
        if (nf == fn) continue;
        const int w = 3 - fn - nf;
        int R = 0;
        while (R < n3[fn] && (double)R * d3[fn] < thr) ++R;
        int lo, hi;
        window(s, top, d3[nf], thr, 1, &lo, &hi);  // cells on either side of the target's plane; the box has c >= 0
        const int depth = std::min(hi + 1, M[l][nf]);
        edge = std::max(edge, depth);
        const auto key = std::make_tuple(l, 0, d3[w], d3[nf], d3[fn], R, depth);
        if (!seen.count(key)) {
          NearTable T{};
          T.par = 0;
          T.rows = R;
          T.hw = d3[w]; T.hr = d3[nf]; T.hn = d3[fn];
          common(T, fn, thr);
          T.r0 = 0;
          T.nrow = depth;
          seen[key] = (int)tabs.size();
          tabs.push_back(T);
          runs.emplace_back();
        }
        const int ti = seen[key];
        const NearTable& T = tabs[ti];
        for (int sf = 0; sf < 2; ++sf)
          for (int sg = 0; sg < 2; ++sg) {
            const int ft = 2 * nf + sf, G = 2 * fn + sg;
            const int o = w == face_u(G) ? 0 : 1;
            const int Nu = n3[face_u(ft)], Nv = n3[face_v(ft)];
            const int str_n = face_u(ft) == fn ? 1 : Nu, str_w = face_u(ft) == w ? 1 : Nu;
            for (int c = 0; c < 3; ++c)
              for (int wb = 0; wb * TB < n3[w]; ++wb) {
                NearRow Q{};
                Q.Wp = P.Wp[l][o][G];
                Q.nrow = M[l][nf];
                Q.abase = P.dbase[l][o][G] + (long long)c * kNearDigits * Q.nrow * Q.Wp;
                Q.rs = sf ? -1 : 1;
                Q.row0 = sf ? Q.nrow - 1 : 0;
                Q.wst = wb * 16 + T.w0;
                Q.obase = P.abase[ft] + (long long)c * Nu * Nv + (sg ? (long long)(n3[fn] - 1) * str_n : 0) +
                          (long long)wb * TB * str_w;
                Q.ostr_r = sg ? -str_n : str_n;
                Q.ostr_w = str_w;
                Q.rlim = R;
                Q.wlim = std::min(TB, n3[w] - wb * TB);
                runs[ti].push_back(Q);
              }
          }
      }
    }
  }
  P.edge = edge;
  return true;
}

}  // namespace vpmg
