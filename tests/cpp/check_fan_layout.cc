// Host check of the fan records (akb_patch_build.cu), no GPU: every element
// is in one fan, as an even permutation of its own nodes; every index a record
// yields stays inside its buffer; a node's contribution list is exactly the
// slots of its rows; the interior / shared numbering is a bijection. Also
// prints the mean fan length. Exits non-zero on any failure.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <set>
#include <vector>

#include "akb_patch.cuh"

using namespace akb;

namespace {

struct Mesh {
  std::vector<double> X;
  std::vector<uint32_t> C;
  int dim;
};

Mesh tet_box(int nx, int ny, int nz) {
  Mesh m{{}, {}, 3};
  for (int k = 0; k <= nz; ++k)
    for (int j = 0; j <= ny; ++j)
      for (int i = 0; i <= nx; ++i) m.X.insert(m.X.end(), {double(i), double(j), double(k)});
  const uint32_t off[3] = {1, (uint32_t)(nx + 1), (uint32_t)((nx + 1) * (ny + 1))};
  const int perm[6][3] = {{0, 1, 2}, {0, 2, 1}, {1, 0, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}};
  for (int k = 0; k < nz; ++k)
    for (int j = 0; j < ny; ++j)
      for (int i = 0; i < nx; ++i)
        for (int q = 0; q < 6; ++q) {
          const uint32_t b = i * off[0] + j * off[1] + k * off[2];
          uint32_t a = b + off[perm[q][0]], c = a + off[perm[q][1]], d = c + off[perm[q][2]];
          if (q == 1 || q == 2 || q == 5) std::swap(a, c);
          m.C.insert(m.C.end(), {b, a, c, d});
        }
  return m;
}

Mesh tri_plate(int nx, int ny) {
  Mesh m{{}, {}, 2};
  for (int j = 0; j <= ny; ++j)
    for (int i = 0; i <= nx; ++i) m.X.insert(m.X.end(), {double(i), double(j)});
  auto id = [&](int i, int j) { return (uint32_t)(j * (nx + 1) + i); };
  for (int j = 0; j < ny; ++j)
    for (int i = 0; i < nx; ++i) {
      m.C.insert(m.C.end(), {id(i, j), id(i + 1, j), id(i + 1, j + 1)});
      m.C.insert(m.C.end(), {id(i, j), id(i + 1, j + 1), id(i, j + 1)});
    }
  return m;
}

Mesh tri_star(int k) {  // k triangles around node 0
  Mesh m{{0, 0}, {}, 2};
  for (int i = 0; i < k; ++i) m.X.insert(m.X.end(), {std::cos(6.283185 * i / k), std::sin(6.283185 * i / k)});
  for (int i = 0; i < k; ++i) m.C.insert(m.C.end(), {0u, 1u + i, 1u + (i + 1) % k});
  return m;
}

Mesh tet_star(int k) {  // a chain of tetrahedra sharing node 0
  Mesh m{{0, 0, 0}, {}, 3};
  for (int i = 0; i < k + 2; ++i) m.X.insert(m.X.end(), {std::cos(i * 0.37), std::sin(i * 0.37), i * 0.1});
  for (uint32_t i = 0; i < (uint32_t)k; ++i) m.C.insert(m.C.end(), {0u, i + 1, i + 2, i + 3});
  return m;
}

// node ids and elements scrambled, elements rotated by even permutations
Mesh scrambled(Mesh m, unsigned seed) {
  srand(seed);
  const int d = m.dim, n = d + 1, nn = (int)m.X.size() / d, ne = (int)m.C.size() / n;
  std::vector<uint32_t> to(nn);
  for (int i = 0; i < nn; ++i) to[i] = i;
  for (int i = nn - 1; i > 0; --i) std::swap(to[i], to[rand() % (i + 1)]);
  std::vector<double> X(m.X.size());
  for (int i = 0; i < nn; ++i)
    for (int k = 0; k < d; ++k) X[to[i] * d + k] = m.X[i * d + k] + 0.1 * rand() / RAND_MAX;
  m.X = X;
  for (auto& c : m.C) c = to[c];
  for (int e = ne - 1; e > 0; --e) {
    const int f = rand() % (e + 1);
    for (int a = 0; a < n; ++a) std::swap(m.C[e * n + a], m.C[f * n + a]);
    std::rotate(&m.C[e * n], &m.C[e * n + 1], &m.C[e * n + 3]);  // a 3-cycle: even
  }
  return m;
}

int fails = 0;
#define CHECK(c)                                                                   \
  do {                                                                             \
    if (!(c) && fails++ < 20)                                                      \
      printf("FAIL %s (line %d, case %s, patch %d)\n", #c, __LINE__, name, p);     \
  } while (0)

void check(const char* name, const Mesh& m, int target, int maxn, int cap, int max_fans,
           const std::vector<uint8_t>* force = nullptr) {
  const int d = m.dim, n = d + 1, H = d - 1;
  const int64_t nn = (int64_t)m.X.size() / d, ne = (int64_t)m.C.size() / n;
  const PatchHost P = build_patches(m.X.data(), m.C.data(), nn, ne, d, n, target, maxn, 8,
                                    force ? force->data() : nullptr, cap, max_fans);
  int p = -1;
  CHECK(P.fans && (int64_t)P.elem_order.size() == ne);
  std::vector<int> hit(nn, 0), seen(ne, 0);
  for (int64_t v = 0; v < nn; ++v)
    if (P.perm[v] < (uint64_t)nn) hit[P.perm[v]]++;
  for (int64_t v = 0; v < nn; ++v) CHECK(hit[v] == 1);
  long nfans = 0;
  for (p = 0; p < P.npatch; ++p) {
    const int nint = P.nint[p], s0 = P.sh_ptr[p], L = nint + P.sh_ptr[p + 1] - s0, eb = P.elem_ptr[p];
    const int nep = P.elem_ptr[p + 1] - eb;
    CHECK(P.chunk_base[p + 1] - P.chunk_base[p] == 1 && L <= P.max_nodes && L - nint <= P.max_shared);
    const ChunkDesc cd = P.chunks[P.chunk_base[p]];
    CHECK((int)cd.bytes <= P.chunk_bytes && cd.bytes % 16 == 0);
    CHECK((size_t)cd.off16 * 8 + cd.bytes / 2 <= P.cdata.size());
    const uint16_t* rec = &P.cdata[(size_t)cd.off16 * 8];
    const int end = (int)cd.bytes / 2, nf = rec[0], rows = rec[1], slots = rec[7];
    const uint16_t *ro = rec + rec[2], *node = rec + rec[3], *info = rec + rec[4], *cnt = rec + rec[5],
                   *goff = rec + rec[6];
    const int entries = ro[rows];
    CHECK(rec[2] >= 8 && rec[2] + rows + 1 <= rec[3] && rec[3] + 2 * entries <= rec[4]);
    CHECK(rec[4] + 2 * nf <= rec[5] && rec[5] + L <= rec[6] && rec[6] + (L + 31) / 32 <= end);
    CHECK(slots <= P.contrib_slots && rows <= H + 1 + cap && ro[0] == 0 && entries <= slots);
    CHECK(rec[3] % 2 == 0 && rec[4] % 2 == 0);  // read as 32-bit words
    CHECK(nf <= max_fans || nf == 1);
    nfans += nf;
    std::vector<int> written(slots, -1);  // the position each slot belongs to
    int next = 0;
    for (int t = 0; t < nf; ++t) {
      const int k = info[2 * t] & 0x7fff, closed = info[2 * t] >> 15;
      CHECK(info[2 * t + 1] == next && k >= 1 && k <= cap);
      next += k;
      const int r = H + k + (closed ? 0 : 1);
      CHECK(r <= rows);
      std::vector<int64_t> id(r);
      for (int j = 0; j < r; ++j) {
        CHECK(t < ro[j + 1] - ro[j]);
        const int e = ro[j] + t, at = node[2 * e], s = node[2 * e + 1];
        CHECK(e < entries && s < slots && at < L && written[s] < 0);
        if (s < slots) written[s] = at;
        id[j] = at < nint ? (int64_t)P.ibeg[p] + at : (int64_t)P.sgid[s0 + at - nint];
      }
      for (int s = 0; s < k; ++s) {  // the element: an even permutation of its own nodes
        const uint32_t e = P.elem_order[eb + info[2 * t + 1] + s];
        seen[e]++;
        std::vector<int64_t> got(id.begin(), id.begin() + H);
        got.push_back(id[H + s]);
        got.push_back(closed && s == k - 1 ? id[H] : id[H + s + 1]);
        int at[4], inv = 0;
        for (int a = 0; a < n; ++a) {
          at[a] = -1;
          for (int b = 0; b < n; ++b)
            if ((int64_t)P.perm[m.C[(size_t)e * n + b]] == got[a]) at[a] = b;
          CHECK(at[a] >= 0);
          for (int b = 0; b < a; ++b) {
            CHECK(at[a] != at[b]);
            inv += at[b] > at[a];
          }
        }
        CHECK(inv % 2 == 0);
      }
    }
    CHECK(next == nep);
    std::vector<int> read(slots, 0);
    for (int j = 0; j < L; ++j)
      for (int q = 0; q < cnt[j]; ++q) {
        const int at = goff[j / 32] + 32 * q + j % 32;
        CHECK(at >= rec[6] + (L + 31) / 32 && at < end);
        if (at >= end) continue;
        CHECK(rec[at] < slots);
        if (rec[at] < slots) {
          CHECK(written[rec[at]] == j);
          read[rec[at]]++;
        }
      }
    for (int s = 0; s < slots; ++s) CHECK(read[s] == (written[s] >= 0));
  }
  p = -1;
  for (int64_t e = 0; e < ne; ++e) CHECK(seen[e] == 1);
  printf("%-24s patches %5d max_nodes %4d slots %5d record %6d elements per fan %.2f\n", name, P.npatch,
         P.max_nodes, P.contrib_slots, P.chunk_bytes, nfans ? (double)ne / nfans : 0.0);
}

}  // namespace

int main() {
  check("tet box", tet_box(20, 19, 21), 768, 400, 8, 128);
  check("tet box, scrambled", scrambled(tet_box(12, 13, 11), 1), 768, 400, 8, 128);
  check("tet box, single elements", tet_box(7, 6, 5), 256, 200, 1, 1 << 20);
  check("tet box, tiny caps", tet_box(5, 6, 7), 3, 5, 6, 2);
  check("one tet", tet_box(1, 1, 1), 1, 4, 1, 128);
  check("tet star", tet_star(300), 1024, 400, 8, 128);
  check("tri plate", tri_plate(200, 20), 768, 500, 8, 128);
  check("tri plate, scrambled", scrambled(tri_plate(57, 43), 2), 768, 500, 8, 128);
  check("tri plate, pairs", tri_plate(31, 17), 128, 100, 2, 64);
  check("tri star", tri_star(200), 1024, 600, 8, 128);
  check("one square", tri_plate(1, 1), 1024, 640, 8, 128);
  {
    Mesh c = tet_box(12, 12, 12);  // the interface nodes of a partitioned mesh
    std::vector<uint8_t> force(c.X.size() / 3, 0);
    for (size_t v = 0; v < force.size(); ++v) force[v] = c.X[v * 3] == 6.0;
    check("tet forced interface", c, 768, 400, 8, 128, &force);
  }
  {
    Mesh c = tri_plate(9, 9);  // nodes of no element
    c.X.insert(c.X.end(), {50, 50, 60, 60});
    check("tri with orphan nodes", c, 256, 200, 8, 128);
  }
  {
    Mesh c = tet_box(2, 2, 2);  // an element that names a node twice
    c.C[1] = c.C[0];
    const PatchHost P = build_patches(c.X.data(), c.C.data(), 27, 48, 3, 4, 64, 100, 8, nullptr, 8, 128);
    std::vector<uint32_t> o(P.elem_order);
    std::sort(o.begin(), o.end());
    for (uint32_t e = 0; e < 48; ++e)
      if (o.size() != 48 || o[e] != e) ++fails;
  }
  printf("fails %d\n", fails);
  return fails != 0;
}
