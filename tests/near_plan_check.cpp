// CPU restatement of the near field's products from its plan (near_host.cpp)
// against the direct sum over the lattice rule; every index is checked
// against its array.  Usage: near_plan_check nx ny nz hx hy hz levmax
// prints the largest relative difference, or an index that is out of range.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "near_host.h"

using namespace vpmg;

int main(int argc, char** argv) {
  if (argc != 8) return 2;
  const int n[3] = {std::atoi(argv[1]), std::atoi(argv[2]), std::atoi(argv[3])};
  const double h[3] = {std::atof(argv[4]), std::atof(argv[5]), std::atof(argv[6])};
  const int L = std::atoi(argv[7]);
  NearPlan P;
  if (!build_near_plan(n, h, L, P)) {
    std::printf("no plan\n");
    return 0;
  }
  // sources per level and cell (one value for each component), and the arrays as the kernel lays them out
  std::vector<std::vector<double>> src(L + 1);
  std::vector<double> dig(P.ndig, 0.0), acc(P.nacc, 0.0);
  unsigned rnd = 12345;
  for (int l = 0; l <= L; ++l) {
    src[l].resize(3 * (size_t)P.cell0[l][6]);
    for (int f = 0; f < 6; ++f)
      for (int b = 0; b < P.mb[l][f]; ++b)
        for (int a = 0; a < P.ma[l][f]; ++a)
          for (int c = 0; c < 3; ++c) {
            rnd = rnd * 1664525u + 1013904223u;
            const double v = (double)(rnd >> 8) / 8388608.0 - 1.0;
            src[l][3 * (size_t)(P.cell0[l][f] + b * P.ma[l][f] + a) + c] = v;
            dig.at(P.dbase[l][0][f] + (long long)c * kNearDigits * P.mb[l][f] * P.Wp[l][0][f] + (long long)b * P.Wp[l][0][f] + a) = v;
            if (a < P.edge || a >= P.ma[l][f] - P.edge)
              dig.at(P.dbase[l][1][f] + (long long)c * kNearDigits * P.ma[l][f] * P.Wp[l][1][f] + (long long)a * P.Wp[l][1][f] + b) = v;
          }
  }
  for (size_t t = 0; t < P.tabs.size(); ++t) {
    const NearTable& T = P.tabs[t];
    if (T.w0 % 8 || T.nkp < 1 || T.nkp > 255) { std::printf("table %zu: bad window\n", t); return 1; }
    for (const NearRow& R : P.runs[t]) {
      if (R.abase % 8 || R.Wp % 8 || R.wst % 8) { std::printf("table %zu: misaligned run\n", t); return 1; }
      const long long dstr = (long long)R.nrow * R.Wp;
      if (R.abase < 0 || R.abase + kNearDigits * dstr > P.ndig) { std::printf("table %zu: digits out of range\n", t); return 1; }
      for (int col = 0; col < T.nchunk * kNearCols; ++col) {
        const int tr = col / T.TB, tw = col % T.TB;
        if (tr >= R.rlim || tw >= R.wlim) continue;
        const long long o = R.obase + (long long)tr * R.ostr_r + (long long)tw * R.ostr_w;
        if (o < 0 || o >= P.nacc) { std::printf("table %zu: sum out of range\n", t); return 1; }
        double v = 0.0;
        for (int row = 0; row < T.nrow; ++row) {
          const int sr = R.row0 + R.rs * row;
          if (sr < 0 || sr >= R.nrow) continue;
          for (int k = 0; k < 16 * T.nkp; ++k) {
            const int cell = R.wst + k;
            if (cell < 0 || cell >= R.Wp) continue;
            const double w = near_weight(T, col, row, k);
            if (w != 0.0) v += w * dig[R.abase + (long long)sr * R.Wp + cell];
          }
        }
        acc[o] += v;
      }
    }
  }
  double worst = 0.0, big = 0.0;
  for (int F = 0; F < 6; ++F) {
    const int fu = face_u(F), fv = face_v(F), fn = F >> 1;
    for (int v = 0; v < n[fv]; ++v)
      for (int u = 0; u < n[fu]; ++u) {
        int ti[3];
        ti[fn] = (F & 1) ? n[fn] - 1 : 0;
        ti[fu] = u;
        ti[fv] = v;
        double sum[3] = {0, 0, 0};
        for (int l = 0; l <= L; ++l)
          for (int G = 0; G < 6; ++G) {
            const int gu = face_u(G), gv = face_v(G), gn = G >> 1, s = 1 << l;
            auto r2 = [&](int lev, int a, int b) {
              const double S = 1 << lev;
              const double on = (double)(ti[gn] - ((G & 1) ? n[gn] - 1 : 0));
              return lattice_r2(S * (a + 0.5) - ti[gu], h[gu], S * (b + 0.5) - ti[gv], h[gv], on, h[gn]);
            };
            for (int b = 0; b < P.mb[l][G]; ++b)
              for (int a = 0; a < P.ma[l][G]; ++a) {
                const double q = r2(l, a, b);
                double w = 0.0;
                if (l == L) {
                  if (q < near_thr2(h, l, gn)) w = -lattice_weight(near_area(h, l, gn), q);
                } else if (r2(l + 1, a / 2, b / 2) < near_thr2(h, l + 1, gn) && !(l > 0 && q < near_thr2(h, l, gn))) {
                  w = lattice_weight(near_area(h, l, gn), q);
                }
                if (w != 0.0)
                  for (int c = 0; c < 3; ++c) sum[c] += w * src[l][3 * (size_t)(P.cell0[l][G] + b * P.ma[l][G] + a) + c];
              }
          }
        for (int c = 0; c < 3; ++c) {
          const double got = acc[P.abase[F] + ((long long)c * n[fv] + v) * n[fu] + u];
          worst = std::max(worst, std::fabs(got - sum[c]));
          big = std::max(big, std::fabs(sum[c]));
        }
      }
  }
  std::printf("%.3e\n", worst / big);
  return 0;
}
