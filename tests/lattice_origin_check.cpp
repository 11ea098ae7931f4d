// Weights 1 / r of the leaf cells next to a node from the tree's rounded
// coordinates against those from lattice offsets, on an axis of n nodes of
// spacing h whose first node lies at x0 (the same along both axes of a face).
// Usage: lattice_origin_check n h x0
// prints whether lattice_exact accepts it and the largest relative difference.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include "near_host.h"

int main(int argc, char** argv) {
  if (argc != 4) return 2;
  const int m = std::atoi(argv[1]);
  const double h = std::atof(argv[2]), x0 = std::atof(argv[3]);
  const double xmin[3] = {x0, x0, x0}, d[3] = {h, h, h};
  const int n[3] = {m, m, m};
  double worst = 0.0;
  auto node = [&](int i) { return x0 + (double)i * h; };
  auto leaf = [&](int i) { return 0.25 * (((node(i) + node(i)) + node(i + 1)) + node(i + 1)); };
  for (int i = 0; i + 1 < m; ++i)
    for (int j = 0; j + 1 < m; ++j)
      for (int a = 0; a < 2; ++a)
        for (int b = 0; b < 2; ++b) {
          const double x = leaf(i) - node(i + a), y = leaf(j) - node(j + b);
          worst = std::max(worst, std::fabs(h * std::sqrt(0.5) / std::sqrt(x * x + y * y) - 1.0));
        }
  std::printf("%d %.3e\n", vpmg::lattice_exact(xmin, d, n) ? 1 : 0, worst);
  return 0;
}
