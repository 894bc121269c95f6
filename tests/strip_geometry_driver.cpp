// Test driver (CPU only): the shared memory a block of the alignment and
// final-pass kernels asks for with the strip aligner, against the device's
// limit, at every length the entry points take. Prints the first misfit.
#include "dgpu_common.h"

#include <cstdio>

int main() {
  using namespace dgpu;
  constexpr size_t kLimit = 232448;  // bytes a block may ask for on sm_100
  for (int ncol : {1, 42, 94, 256})
    for (int w : {3, 62, 63, 125, 248})
      for (int lmax = 2; lmax < 9999; ++lmax) {
        NwGeom g{};
        g.lmax = lmax;
        strip_geometry(g, w, ncol);
        const size_t strip = strip_smem_per_warp(g);
        const size_t align = err_smem_bytes(ncol) + kNwWarps * strip;
        const size_t subs = kNwWarps * (strip + align16(size_t(16) * ncol * 4));
        if (align > kLimit || subs > kLimit) {
          std::printf("%d nt, %d diagonals, %d columns: %zu and %zu bytes\n", lmax, w, ncol, align, subs);
          return 1;
        }
        // the lambda indices lie in the two code rows
        if (size_t(lmax) * 2 > 2 * align16(size_t(lmax) + kStripPad)) return 2;
      }
  // a matrix so wide that the words no longer fit beside it: they go to global memory
  for (int ncol = 700; ncol < 860; ++ncol) {
    NwGeom g{};
    g.lmax = 400;
    strip_geometry(g, 33, ncol);
    if (strip_block_bytes(g, ncol) > kBlockSmemMax) return 3;
    if (ncol == 700 && !g.strip_smem) return 4;
    if (ncol == 859 && g.strip_smem) return 5;
  }
  std::printf("ok\n");
  return 0;
}
