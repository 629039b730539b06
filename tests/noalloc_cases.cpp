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
    // no fewer labels than with the 616-byte preparation and 4,656-byte group
    // records that 32 MiB were laid out for
    const size_t fixed = align256(sizeof(DevStar)) + align256(63 * 4656) + 256;
    const size_t per = align256(616) + 2 * align256(1025 * 8) + 3 * 256 + 2 * (size_t)stride * 4 +
                       align256((size_t)bstr * 4) + align256(4656);
    if (most < (int64_t)(((32u << 20) - fixed) / per)) {
      if (bad++ < 5) std::printf("%d pixels: %lld labels\n", npx, (long long)most);
    }
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
