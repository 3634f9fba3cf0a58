// Host check of the fan build on elements that name a node twice or more (no
// GPU; built with the address sanitizer): every element is in the plan once, and
// each such element is a fan of its own. Exits non-zero on any failure.
#include <algorithm>
#include <cstdio>
#include <vector>

#include "akb_patch.cuh"

using namespace akb;

namespace {

int fails = 0;

void check(const char* name, int dim, const std::vector<double>& X, const std::vector<uint32_t>& C) {
  const int n = dim + 1, ne = (int)C.size() / n;
  const PatchHost P = build_patches(X.data(), C.data(), (int64_t)X.size() / dim, ne, dim, n, 64, 100, 8,
                                    nullptr, 8, 128);
  std::vector<int> seen(ne, 0);
  for (uint32_t e : P.elem_order) seen[e]++;
  bool ok = (int)P.elem_order.size() == ne && *std::min_element(seen.begin(), seen.end()) == 1;
  for (int p = 0; p < P.npatch; ++p) {
    const uint16_t* rec = &P.cdata[(size_t)P.chunks[P.chunk_base[p]].off16 * 8];
    const uint16_t* info = rec + rec[4];
    for (int t = 0; t < rec[0]; ++t)
      for (int k = 0; k < (info[2 * t] & 0x7fff); ++k) {
        const uint32_t* c = &C[(size_t)P.elem_order[P.elem_ptr[p] + info[2 * t + 1] + k] * n];
        bool twice = false;
        for (int a = 0; a < n; ++a)
          for (int b = 0; b < a; ++b) twice = twice || c[a] == c[b];
        ok = ok && (!twice || (info[2 * t] & 0x7fff) == 1);
      }
  }
  if (!ok) ++fails;
  printf("%s: %s\n", name, ok ? "ok" : "FAIL");
}

}  // namespace

int main() {
  const std::vector<double> X3{0, 0, 0, 1, 0, 0, 0, 1, 0, 0, 0, 1, 1, 1, 1}, X2{0, 0, 1, 0, 0, 1, 1, 1};
  check("one node twice, first", 3, X3, {0, 0, 1, 2, 0, 1, 2, 3, 1, 2, 3, 4});
  check("one node twice, last", 3, X3, {0, 1, 2, 3, 1, 2, 3, 4, 0, 1, 2, 2});
  check("pairs", 3, X3, {0, 0, 1, 1, 0, 1, 0, 1, 2, 3, 3, 2, 0, 1, 2, 3});
  check("one node only", 3, X3, {0, 0, 0, 0, 1, 1, 1, 2, 4, 4, 4, 4, 0, 1, 2, 4});
  check("triangles", 2, X2, {0, 0, 1, 0, 1, 2, 1, 3, 2, 3, 3, 3, 2, 0, 2});
  printf("fails %d\n", fails);
  return fails != 0;
}
