// The rank order of the nonlocal scatter (host code only; links libinqb200 for the table
// builder): every entry has one place, a tile's ranks cover its entries, the entries of
// one rank touch different points, and a point's entries keep their order over the ranks.
#include <cstdio>
#include <cstdlib>
#include <set>
#include <vector>

#include "../../inq-wannier-fork_b200/csrc/inqb_internal.h"
namespace inqb {
int build_proj_tables(const inqb_ctx& ctx, int nproj, int L, int smax, const int* counts, const int* coords,
                      const float* relpos, const double* beta, const double* coeff, ProjTables& t);
}

static int check(int nx, int ny, int nz, int nproj, int smax, unsigned seed) {
  inqb_ctx ctx;
  double lat[9] = {6, 0, 0, 0, 7, 0, 0, 0, 8};
  ctx.nr[0] = nx;
  ctx.nr[1] = ny;
  ctx.nr[2] = nz;
  ctx.N = (long)nx * ny * nz;
  ctx.cell.init(lat);
  ctx.dV = ctx.cell.volume / ctx.N;
  srand(seed);
  // random points, repeated ones within an atom among them (periodic images)
  std::vector<int> counts(nproj), coords((size_t)nproj * smax * 3, -1);
  for (int a = 0; a < nproj; a++) {
    counts[a] = rand() % (smax + 1);
    for (int p = 0; p < counts[a]; p++) {
      int* c = &coords[((size_t)a * smax + p) * 3];
      c[0] = rand() % (rand() % 2 ? nx : 2);
      c[1] = rand() % ny;
      c[2] = rand() % 5;
    }
  }
  std::vector<float> rel((size_t)nproj * smax * 3, 0.f);
  std::vector<double> beta((size_t)nproj * 2 * smax, 1.0), coeff((size_t)nproj * 2, 1.0);
  inqb::ProjTables t;
  if (inqb::build_proj_tables(ctx, nproj, 2, smax, counts.data(), coords.data(), rel.data(), beta.data(), coeff.data(), t))
    return 1;
  int bad = 0, most = 0;
  const int ntile = nx * t.y1;
  std::vector<int> at(t.nent, -1);
  for (int e = 0; e < t.nent; e++) {
    if (t.rk_pos[e] < 0 || t.rk_pos[e] >= t.nent || at[t.rk_pos[e]] >= 0) return 1;
    at[t.rk_pos[e]] = e;
  }
  if ((int)t.rk_ptr.size() != ntile + 1 || t.rk_start.back() != t.nent) return 1;
  for (int tile = 0; tile < ntile; tile++) {
    const int e0 = t.seg_ent[t.seg_ptr[tile]], e1 = t.seg_ent[t.seg_ptr[tile + 1]];
    const int k0 = t.rk_ptr[tile], k1 = t.rk_ptr[tile + 1];
    most = k1 - k0 > most ? k1 - k0 : most;
    if (t.rk_start[k0] != e0 || t.rk_start[k1] != e1) bad++;
    std::vector<int> last(t.tile_pts, -1);
    std::set<int> before;
    for (int k = k0; k < k1; k++) {
      if (t.rk_start[k + 1] <= t.rk_start[k]) bad++;
      std::set<int> seen;
      for (int q = t.rk_start[k]; q < t.rk_start[k + 1]; q++) {
        const int e = at[q], off = t.ent_off[e];
        if (e < e0 || e >= e1) bad++;
        if (!seen.insert(off).second) bad++;
        if (k > k0 && !before.count(off)) bad++;  // a point's entries fill the ranks from the first
        if (e <= last[off]) bad++;
        last[off] = e;
      }
      before = seen;
    }
  }
  printf("%dx%dx%d atoms=%d nent=%d ranks<=%d bad=%d\n", nx, ny, nz, nproj, t.nent, most, bad);
  return bad != 0;
}

int main() {
  return check(16, 16, 16, 5, 60, 1) | check(24, 36, 20, 9, 200, 2) | check(12, 18, 24, 1, 0, 3) |
         check(20, 24, 30, 40, 50, 4);
}
