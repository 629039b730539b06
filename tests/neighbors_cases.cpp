// Neighbour search on axes too short for a cubic or quadratic interpolation:
// an error status, and no read past an axis (built with the address sanitizer).
#include <cuda_runtime.h>

#include <cstdio>
#include <vector>

#include "../pasta_b200/csrc/common.cuh"

using namespace pb;

struct Axes {
  std::vector<double> t, m, l;
  std::vector<int> lo, hi;
  std::vector<int64_t> cum;
  Axes(int nt, int nm, int nl) {
    for (int i = 0; i < nt; i++) t.push_back(6000.0 + 250.0 * i);
    for (int i = 0; i < nm; i++) m.push_back(-0.5 + 0.25 * i);
    for (int i = 0; i < nl; i++) l.push_back(3.0 + 0.5 * i);
    for (int i = 0; i < nt; i++) {
      lo.push_back(0);
      hi.push_back(nl - 1);
      cum.push_back((int64_t)i * nl);
    }
  }
  GridGeom geom() const {
    return GridGeom{t.data(), m.data(), l.data(), lo.data(), hi.data(), cum.data(), (int)t.size(), (int)m.size(), (int)l.size()};
  }
};

int main() {
  int bad = 0;
  for (int nt = 1; nt <= 5; nt++)
    for (int nm = 1; nm <= 5; nm++)
      for (int nl = 1; nl <= 5; nl++) {
        const Axes A(nt, nm, nl);
        const GridGeom G = A.geom();
        // at every point and halfway to the next
        for (int a = 0; a < 2 * nt - 1; a++)
          for (int b = 0; b < 2 * nm - 1; b++)
            for (int c = 0; c < 2 * nl - 1; c++) {
              int cols[64];
              float w[64];
              const int st = local_grid(G, 6000.0 + 125.0 * a, -0.5 + 0.125 * b, 3.0 + 0.25 * c, cols, w);
              const bool enough = nt >= 3 && nm >= 3 && nl >= 3;
              bool ok = enough ? st == S_OK : st == S_NEIGHBORS;
              if (!st) {
                double sum = 0.0;
                for (int k = 0; k < 64; k++) {
                  ok = ok && cols[k] < nt * nm * nl && (cols[k] >= 0 || w[k] == 0.0f);
                  sum += w[k];
                }
                ok = ok && sum > 0.999 && sum < 1.001;
              }
              if (!ok && bad++ < 5) std::printf("%d x %d x %d points, label %d %d %d: status %d\n", nt, nm, nl, a, b, c, st);
            }
      }
  return bad != 0;
}
