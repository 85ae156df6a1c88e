// Host build of the fixed-point pressure rewrite (fx::pressure_q): random nodes
// against the same expression in long double.  Prints the largest error in
// units of 2^-56 over the accepted nodes and their number.  Arguments: seed,
// velocity range, density range.  Test infrastructure for
// tests/test_fx_pressure_host.py; compile with -ffp-contract=off.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../../lattice_boltzmann_parallel_solver_gb300/csrc/lbm_fx.cuh"

using namespace lbm;

int main(int argc, char** argv) {
  if (argc != 4) return 2;
  std::mt19937_64 gen(strtoull(argv[1], nullptr, 10));
  const double um = atof(argv[2]), dr = atof(argv[3]);
  auto uni = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(gen); };
  const int cx[9] = {0, 1, 0, -1, 0, 1, -1, -1, 1}, cy[9] = {0, 0, 1, 0, -1, 1, 1, -1, -1};
  const int w36[9] = {16, 4, 4, 4, 4, 1, 1, 1, 1};
  const long double one = 72057594037927936.0L;  // 2^56
  long double worst = 0;
  long accepted = 0;
  for (int t = 0; t < 20000; ++t) {
    const double rho = 1 + uni(-dr, dr), ux = uni(-um, um), uy = uni(-um, um), target = 1 + uni(-dr, dr);
    int64_t d[9], add[9];
    for (int i = 0; i < 9; ++i) {
      const double w = w36[i] / 36.0, cu = cx[i] * ux + cy[i] * uy;
      d[i] = fx::to_fx(w * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * (ux * ux + uy * uy)) + uni(-1e-3, 1e-3) * w, w);
    }
    const int64_t tq = fx::round_scaled(target - 1.0, fx::kS);
    if (!fx::pressure_q(d, tq, 0x1FFu, add)) continue;
    ++accepted;
    long double D = 0, jx = 0, jy = 0;
    for (int i = 0; i < 9; ++i) {
      D += d[i];
      jx += cx[i] * (long double)d[i];
      jy += cy[i] * (long double)d[i];
    }
    const long double vx = jx / (one + D), vy = jy / (one + D);
    for (int i = 0; i < 9; ++i) {
      const long double cu = cx[i] * vx + cy[i] * vy;
      const long double ref = w36[i] / 36.0L * (1 + 3 * cu + 4.5L * cu * cu - 1.5L * (vx * vx + vy * vy)) * (tq - D);
      worst = fmaxl(worst, fabsl(add[i] - ref));
    }
  }
  printf("%.4f %ld\n", (double)worst, accepted);
  return 0;
}
