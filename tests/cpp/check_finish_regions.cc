// Host check of finish_regions (akb_patch.cuh), no GPU: for interior slices at
// the start of a mesh and past the 4 GB marks of its nodal arrays, every copy
// starts on the 16-byte boundary at or below its slice, ends on the one at or
// above it, and lands the slice's first item where off says. Exits non-zero on
// any failure.
#include <cstdio>

#include "akb_patch.cuh"

using namespace akb;

namespace {

int fails = 0;

template <int d, bool FEXT>
void check(int ib, int nint) {
  uint32_t off[5], bytes[5], at = 0;
  size_t lo[5];
  const uint32_t total = finish_regions<d, FEXT>(ib, nint, off, lo, bytes);
  const unsigned __int128 row[5] = {8 * d, 8 * d, 8, d, 8 * d};
  for (int k = 0; k < (FEXT ? 5 : 4); ++k) {
    const unsigned __int128 s0 = ib * row[k], s1 = ((unsigned __int128)ib + nint) * row[k];
    const bool ok = lo[k] % 16 == 0 && bytes[k] % 16 == 0 && lo[k] <= s0 && s0 - lo[k] < 16 &&
                    lo[k] + (unsigned __int128)bytes[k] >= s1 && lo[k] + (unsigned __int128)bytes[k] - s1 < 16 &&
                    off[k] == at + (uint32_t)(s0 - lo[k]);
    if (!ok && fails++ < 20) printf("FAIL dim %d, ib %d, nint %d, input %d: lo %zu\n", d, ib, nint, k, lo[k]);
    at += bytes[k];
  }
  if (total != at && fails++ < 20) printf("FAIL total, dim %d, ib %d\n", d, ib);
}

}  // namespace

int main() {
  const int begins[] = {0, 1, 3, 1000, 178956969, 178956970, 178956971, 268435455, 268435457, 536870913, 2147480000};
  for (int ib : begins)
    for (int nint : {1, 2, 7, 400}) {
      check<1, true>(ib, nint);
      check<2, false>(ib, nint);
      check<2, true>(ib, nint);
      check<3, false>(ib, nint);
      check<3, true>(ib, nint);
    }
  printf("fails %d\n", fails);
  return fails != 0;
}
