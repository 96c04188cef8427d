// Host-only check of which residual-window tiles the CTAs of a (request, kv head) fetch (compiled with nvcc, runs on the CPU): every
// tile with rows, and beyond those at most one per CTA, unless the window is no longer than two tiles.
#include <cstdio>

#include "decode.cuh"

using namespace r2k;

int main() {
  long cases = 0;
  for (int nR = 0; nR <= 64; ++nR)
    for (int pools = 0; pools <= 24; pools += 4)
      for (int ctas = 1; ctas <= 9; ++ctas)
        for (int cluster = 0; cluster <= 1; ++cluster) {
          DecodeParams p{};
          p.bh_total = 2; p.n4 = pools; p.nR = nR; p.units = pools + nR;
          if (p.units == 0) continue;
          p.cF = 14; p.c4 = 21; p.c2 = 24; p.cR = 5;
          p.c_bh = p.n4 * p.c4 + p.nR * p.cR;
          p.grid = 2 * ctas;
          const bool whole = window_comes_whole(p, cluster != 0);
          for (int rows = 0; rows <= nR * kTR; rows += rows % 32 == 0 ? 1 : 31) {
            int fetched = 0, with_rows = 0, first_of_ctas = 0;
            for (int cta = 0; cta < ctas; ++cta) {   // those of the first head
              const CostPos c0 = cta_pos(p, cta), c1 = cta_pos(p, cta + 1);
              if (c0.bh > 0) break;   // no range of this head
              const int u0 = units_before(p, c0.r), u1 = units_before(p, c1.bh > 0 ? p.c_bh : c1.r);
              const int first = u0 > p.n4 ? u0 : p.n4;
              for (int u = first; u < u1; ++u) {
                const int row = (u - p.n4) * kTR;
                const bool comes = window_tile_comes(whole, row, rows, u == first);
                if (row < rows && !comes) { std::printf("FAIL: tile with rows left out (%d tiles, %d rows)\n", nR, rows); return 1; }
                fetched += comes;
                with_rows += row < rows;
              }
              first_of_ctas += first < u1;
            }
            if (with_rows != (rows + kTR - 1) / kTR) { std::printf("FAIL: %d of %d rows' tiles\n", with_rows, rows); return 1; }
            if (nR > 2 && fetched > with_rows + first_of_ctas) {
              std::printf("FAIL: %d tiles fetched of a window of %d with %d rows (cluster %d)\n", fetched, nR, rows, cluster);
              return 1;
            }
            ++cases;
          }
        }
  std::printf("OK %ld cases\n", cases);
  return 0;
}
