// Compares prefix_rule_fast (stencil.cuh) with prefix_rule on random neighbourhoods: the same
// value, codes and key, bit for bit, wherever the fast rule decides.
// Usage: fast_rule_harness nd cases seed specials(0/1); prints "decided differing".
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#include "stencil.cuh"

using namespace eik;

template <int ND>
static void run(long long cases, unsigned long long seed, bool specials) {
  std::mt19937_64 gen(seed);
  std::uniform_real_distribution<double> U(0.0, 1.0);
  long long decided = 0, differing = 0;
  for (long long q = 0; q < cases; q++) {
    Nbhd nb;
    nb_clear(nb);
    const double h = 0.1;
    const bool uniform = U(gen) < 0.5;
    for (int a = 0; a < 3; a++) nb.dh[a] = uniform ? h : h * (0.5 + U(gen));
    nb.slow = 0.2 + 0.3 * U(gen);
    // from beside the source to 10^6 nodes away; one neighbourhood in four on a lattice (ties)
    const double step = h * nb.slow, base = U(gen) < 0.3 ? U(gen) * 0.05 : std::exp(14.0 * U(gen));
    const double quant = U(gen) < 0.25 ? step / 4.0 : 0.0, rate = U(gen) < 0.5 ? 0.06 : 0.35;
    for (int a = 0; a < ND; a++)
      for (int l = 0; l < 2; l++) {
        double t1 = base + 2.0 * step * U(gen), t2 = t1 - step * (0.5 + 0.7 * U(gen)) * (U(gen) < 0.8 ? 1.0 : -1.0);
        for (int m = 0; m < 2; m++) {
          double t = m == 0 ? t1 : (t2 > 0.0 ? t2 : 0.0);
          if (quant > 0.0) t = base + quant * std::floor((t - base) / quant);
          if (t < 0.0) t = 0.0;
          if (U(gen) < 0.2) t = EIK_INF;
          double L = t;
          int d = 0;
          const double r = U(gen);
          if (specials && t < EIK_INF) {
            if (r < 0.03) L = -EIK_INF;
            else if (r < rate) {
              L = t + step * U(gen);
              if (quant > 0.0) L = base + quant * std::ceil((L - base) / quant);
              d = 1 + (int)(4.99 * U(gen));
            }
          }
          if (m == 0) nb_put1(nb, a, l, t, L, d);
          else if (U(gen) < 0.85) nb_put2(nb, a, l, t, L, d);
        }
      }
    double t1[ND][2], t2[ND][2], L1[ND][2], L2[ND][2], c1[ND], c2[ND];
    int d1[ND][2];
    bool special = false;
    for (int a = 0; a < ND; a++) {
      c1[a] = 1.0 / (nb.dh[a] * nb.dh[a]);
      c2[a] = 9.0 / (4.0 * (nb.dh[a] * nb.dh[a]));
      for (int l = 0; l < 2; l++) {
        t1[a][l] = nb.t1[a][l];
        t2[a][l] = nb.t2[a][l];
        d1[a][l] = (int)((nb.d1 >> (4 * slot(a, l))) & 15u);
        L1[a][l] = nb.L1[a][l];
        L2[a][l] = nb.L2[a][l];
        special = special || L1[a][l] != t1[a][l] || L2[a][l] != t2[a][l];
      }
    }
    int8_t cr[3] = {0, 0, 0}, cf[ND];
    Key key;
    bool neg = false;
    double vf, Lf;
    int df;
    const double v = prefix_rule<ND>(nb, cr, &key, &neg);
    const bool ok = special ? prefix_rule_fast<ND, true>(t1, t2, L1, L2, d1, c1, c2, nb.slow, &vf, &Lf, &df, cf)
                            : prefix_rule_fast<ND, false>(t1, t2, t1, t2, d1, c1, c2, nb.slow, &vf, &Lf, &df, cf);
    if (!ok) continue;
    decided++;
    if (std::memcmp(&v, &vf, 8) || std::memcmp(&key.L, &Lf, 8) || key.d != df || neg || std::memcmp(cr, cf, ND)) differing++;
  }
  std::printf("%lld %lld\n", decided, differing);
}

int main(int argc, char** argv) {
  if (argc != 5) return 2;
  const long long cases = std::atoll(argv[2]);
  const unsigned long long seed = std::strtoull(argv[3], nullptr, 10);
  if (std::atoi(argv[1]) == 3) run<3>(cases, seed, std::atoi(argv[4]) != 0);
  else run<2>(cases, seed, std::atoi(argv[4]) != 0);
  return 0;
}
