// The boundary tables as set_fx_tables leaves them against each entry converted
// alone: prints the entries that differ.
#include <cstdio>
#include <cstdlib>

#include "lbm_fused.cuh"

int main() {
  lbm_geometry g;
  std::memset(&g, 0, sizeof(g));
  g.nx = g.ny = 8;
  std::srand(5);
  // sets of numbers, of zeros, of negative zeros, and of one number among zeros
  for (int s = 0; s < LBM_MAX_SETS; ++s)
    for (int i = 0; i < 9; ++i) {
      const double v = (std::rand() % 2001 - 1000) * 1e-4;
      g.kconst[s][i] = s % 4 == 0 ? v : (s % 4 == 1 ? 0.0 : (s % 4 == 2 ? -0.0 : (i == 4 ? v : 0.0)));
      g.cconst[s][i] = s % 4 == 3 ? 0.1 + v : (s % 4 == 2 ? 0.0 : (s % 4 == 1 ? -0.0 : (i == 8 ? v : 0.0)));
    }
  lbm::GeoK q;
  if (!lbm::to_geok(&g, q)) return 1;
  lbm::set_fx_tables(q);
  int bad = 0;
  auto differs = [](double slot, int64_t want) {
    int64_t b;
    std::memcpy(&b, &slot, 8);
    return b != want;
  };
  for (int s = 0; s < LBM_MAX_SETS; ++s)
    for (int i = 0; i < 9; ++i)
      bad += differs(q.kconst[s][i], lbm::fx::round_scaled(g.kconst[s][i], lbm::fx::kS)) +
             differs(q.cconst[s][i], lbm::fx::to_fx(g.cconst[s][i], lbm::wd(i)));
  for (int i = 0; i < 9; ++i) bad += differs(q.edge_in_f[i], lbm::fx::to_fx(0.0, lbm::wd(i)));
  std::printf("%d\n", bad);
  return 0;
}
