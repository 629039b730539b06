// The layout of the allocation-free chi2's scratch array at its limits.
#include <cstdio>
#include <set>

#include "../pasta_b200/csrc/noalloc_layout.h"

using namespace pb;

int main() {
  int bad = 0;
  for (int npx = 64; npx < 400000; npx += 191) {
    const int64_t stride = (npx + 63) / 64 * 64;
    const int bstr = bnd_stride_for(npx);
    const int64_t most = noalloc_max_labels(stride, bstr);
    // every remainder of a segment at the upper end, and the smallest counts
    for (int64_t L = 1; L <= most; L += L == 70 && most > 210 ? most - 140 : 1) {
      const NoallocLayout o = noalloc_layout(L, stride, bstr);
      const size_t end = o.gcount + sizeof(int) * (size_t)((L + SEG - 1) / SEG);
      if (o.total > NOALLOC_SCRATCH_BYTES || end > o.total) {
        if (bad++ < 5) std::printf("%d pixels, %lld labels: %zu bytes\n", npx, (long long)L, o.total);
      }
    }
  }
  return bad != 0;
}
