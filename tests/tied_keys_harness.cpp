// Compares prefix_rule_signed (stencil.cuh), the fast form of the order rule on a neighbourhood as a brick
// keeps it (sign bit: special key), with prefix_rule on lattice neighbourhoods rich in keys
// (t, d >= 1, t): special ones whose level equals their traveltime, which only the sign tells from ordinary ones.
// Usage: tied_keys_harness cases seed; prints "decided differing tied", tied: neighbourhoods with such a key.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "stencil.cuh"

using namespace eik;

int main(int argc, char** argv) {
  if (argc != 3) return 2;
  constexpr int ND = 3;
  const long long cases = std::atoll(argv[1]);
  std::mt19937_64 gen(std::strtoull(argv[2], nullptr, 10));
  std::uniform_real_distribution<double> U(0.0, 1.0);
  long long decided = 0, differing = 0, tied = 0;
  for (long long q = 0; q < cases; q++) {
    Nbhd nb;
    nb_clear(nb);
    const double h = 1.0;
    for (int a = 0; a < 3; a++) nb.dh[a] = h;
    nb.slow = 1.0 / (1.0 + (int)(3.99 * U(gen)));
    // a lattice of fractions of the node's own step, as rationally related velocities give
    const double step = h * nb.slow, quant = step / (1 << (int)(2.99 * U(gen))), base = quant * (int)(40.0 * U(gen));
    const double rate = U(gen) < 0.5 ? 0.1 : 0.4, equal = U(gen);
    double t1[ND][2], t2[ND][2], L1[ND][2], L2[ND][2], c1[ND], c2[ND];
    int d1[ND][2];
    bool tie = false;
    for (int a = 0; a < ND; a++) {
      c1[a] = 1.0 / (h * h);
      c2[a] = 9.0 / (4.0 * (h * h));
      for (int l = 0; l < 2; l++) {
        t2[a][l] = L2[a][l] = EIK_INF;
        for (int m = 0; m < 2; m++) {
          double t = base + quant * (int)(9.0 * U(gen)) - (m == 1 ? quant * (int)(5.0 * U(gen)) : 0.0);
          if (t < 0.0) t = 0.0;
          if (U(gen) < 0.2) t = EIK_INF;
          double L = t;
          int d = 0;
          if (t < EIK_INF && U(gen) < rate) {
            if (U(gen) < 0.05) {
              L = -EIK_INF;
            } else {
              if (U(gen) >= equal) L = t + quant * (int)(3.0 * U(gen));
              d = 1 + (int)(4.99 * U(gen));
            }
          }
          const bool special = L != t || d > 0;
          const bool there = m == 0 || U(gen) < 0.85;
          tie = tie || (special && L == t && there);
          if (m == 0) {
            nb_put1(nb, a, l, t, L, d);
            t1[a][l] = special ? -t : t;
            L1[a][l] = L;
            d1[a][l] = d;
          } else if (there) {
            nb_put2(nb, a, l, t, L, d);
            t2[a][l] = special ? -t : t;
            L2[a][l] = L;
          }
        }
      }
    }
    tied += tie;
    int8_t cr[3] = {0, 0, 0}, cf[ND];
    Key key;
    bool neg = false;
    double vf, Lf;
    int df;
    const double v = prefix_rule<ND>(nb, cr, &key, &neg);
    if (!prefix_rule_signed<ND>(t1, t2, L1, L2, d1, c1, c2, nb.slow, &vf, &Lf, &df, cf)) continue;
    decided++;
    if (std::memcmp(&v, &vf, 8) || std::memcmp(&key.L, &Lf, 8) || key.d != df || neg || std::memcmp(cr, cf, ND)) differing++;
  }
  std::printf("%lld %lld %lld\n", decided, differing, tied);
  return 0;
}
