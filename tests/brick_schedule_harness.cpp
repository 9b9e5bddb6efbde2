// Host emulation of the forward solve by bricks (brick.cuh, coarse.cu) on a Cartesian grid, one visit after
// the other. A round visits one colour of the bricks and bricks of a colour read nothing of one
// another, so the order within a round changes nothing; inside a visit the nodes go in batches of 32 whose reads
// all come before their writes, as on the GPU. Restated here: pending nodes and their fronts, the round
// threshold, the inner window, waiting nodes, the bound on scans, the nodes a change leaves alone. The order
// rule is the product's (stencil.cuh, compiled for the host): the fast form where a visit uses it, the
// general rule for the rest.
//
// Usage: brick_schedule_harness in.bin out.bin
//   in:  int32 nd, n0, n1, n2; double h, gate; int32 small, scans (0 = the product's bound), general (1 = no fast
//        form), rounds (limit); int64 nseed; N doubles slowness; nseed int64 node indices; nseed doubles
//        traveltimes of the fixed source points.
//   out: N doubles traveltime; int64 rounds, evaluations, evaluations left to the general rule, nodes whose
//        rule would still change their value or key, special nodes whose level equals their traveltime.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "stencil.cuh"

using namespace eik;

namespace {

float round_up(double v) {
  if (!(v < EIK_INF)) return INFINITY;
  float f = (float)v;
  if ((double)f < v) f = std::nextafterf(f, INFINITY);
  return std::min(f, 3.402823466e38f);
}
double high_word(double v) {  // the traveltime that a front is made from
  unsigned long long u;
  memcpy(&u, &v, 8);
  u &= 0xffffffff00000000ull;
  memcpy(&v, &u, 8);
  return v;
}

struct Result {
  double v, L;
  int d;
};

template <int ND>
struct Solver {
  int n[3], bs, nb[3], maxscans, maxrounds;
  bool general;
  double h, c1u, c2u, delta, linc;
  float din;
  long long N, st[3];
  std::vector<double> slow, t, L;
  std::vector<uint8_t> d;
  std::vector<float> pf;     // pending front inside a visit, else INFINITY
  std::vector<char> pending;
  std::vector<float> front;  // per brick
  long long evals = 0, slowpath = 0;

  bool special(long long l) const { return L[l] != t[l] || d[l] != 0; }
  void coords(long long l, int* c) const {
    c[0] = (int)(l % n[0]);
    c[1] = (int)((l / n[0]) % n[1]);
    c[2] = (int)(l / st[2]);
  }
  long long brick(const int* c) const {
    return c[0] / bs + (long long)nb[0] * (c[1] / bs + (long long)nb[1] * (ND == 3 ? c[2] / bs : 0));
  }
  bool inside(const int* c, int a, int off) const { return c[a] + off >= 0 && c[a] + off < n[a]; }
  // distance-2 node allowed: the first neighbour is off the border in every coordinate
  bool second(const int* c, int a, int sh) const {
    for (int q = 0; q < ND; q++) {
      const int x = c[q] + (q == a ? sh : 0);
      if (x < 1 || x > n[q] - 2) return false;
    }
    return true;
  }

  Result by_general_rule(long long l, const int* c) const {
    Nbhd nb_;
    nb_clear(nb_);
    for (int a = 0; a < 3; a++) nb_.dh[a] = h;
    nb_.slow = slow[l];
    nb_.c1u = c1u;
    nb_.c2u = c2u;
    for (int a = 0; a < ND; a++)
      for (int s = 0; s < 2; s++) {
        const int sh = s == 0 ? 1 : -1;
        if (!inside(c, a, sh)) continue;
        const long long x = l + sh * st[a];
        nb_put1(nb_, a, s, t[x], L[x], d[x]);
        if (second(c, a, sh)) nb_put2(nb_, a, s, t[x + sh * st[a]], L[x + sh * st[a]], d[x + sh * st[a]]);
      }
    int8_t cd[3];
    bool neg = false;
    Key k;
    Result r;
    r.v = prefix_rule<ND>(nb_, cd, &k, &neg);
    r.L = k.L;
    r.d = k.d;
    return r;
  }
  // the neighbourhood as a visit reads it; returns whether a special key is among it
  bool read(long long l, const int* c, double (&t1)[ND][2], double (&t2)[ND][2], double (&L1)[ND][2], double (&L2)[ND][2],
            int (&d1)[ND][2]) const {
    bool any = false;
    for (int a = 0; a < ND; a++)
      for (int s = 0; s < 2; s++) {
        const int sh = s == 0 ? 1 : -1;
        t1[a][s] = t2[a][s] = L1[a][s] = L2[a][s] = EIK_INF;
        d1[a][s] = 0;
        if (!inside(c, a, sh)) continue;
        const long long x = l + sh * st[a];
        t1[a][s] = special(x) ? -t[x] : t[x];
        L1[a][s] = L[x];
        d1[a][s] = d[x];
        any = any || special(x);
        if (!second(c, a, sh)) continue;
        const long long y = x + sh * st[a];
        t2[a][s] = special(y) ? -t[y] : t[y];
        L2[a][s] = L[y];
        any = any || special(y);
      }
    return any;
  }
  Result evaluate(long long l, const int* c, bool levels) {
    evals++;
    double t1[ND][2], t2[ND][2], L1[ND][2], L2[ND][2], c1[ND], c2[ND];
    int d1[ND][2];
    const bool any = read(l, c, t1, t2, L1, L2, d1);
    for (int a = 0; a < ND; a++) {
      c1[a] = c1u;
      c2[a] = c2u;
    }
    Result r;
    int8_t cd[ND];
    bool done = false;
    if (general) {
    } else if (ND == 2 || !levels) {
      done = prefix_rule_fast<ND, false>(t1, t2, t1, t2, d1, c1, c2, slow[l], &r.v, &r.L, &r.d, cd) && !any;
      r.d = r.L == r.v ? 0 : 1;
    } else if constexpr (ND == 3) {
      done = prefix_rule_signed<ND>(t1, t2, L1, L2, d1, c1, c2, slow[l], &r.v, &r.L, &r.d, cd);
    }
    if (done) return r;
    slowpath++;
    return by_general_rule(l, c);
  }

  // marks node x (of brick b or of one across a face) pending with front f
  void mark(long long x, float f, long long b) {
    int c[3];
    coords(x, c);
    pending[x] = 1;
    const long long bx = brick(c);
    if (bx == b) pf[x] = std::min(pf[x], f);
    else front[bx] = std::min(front[bx], f);
  }
  void changed(long long l, const int* c, double oldL, float f, long long b) {
    const double lim = std::min(oldL, L[l]);
    for (int a = 0; a < ND; a++)
      for (int s = -1; s <= 1; s += 2) {
        if (!inside(c, a, s)) continue;
        const long long x = l + s * st[a];
        if (special(x) || t[x] > lim) mark(x, f, b);
        if (!inside(c, a, 2 * s) || !(t[x] < EIK_INF)) continue;
        const long long y = x + s * st[a];
        if (special(y) || t[y] > lim) mark(y, f, b);
      }
  }

  void visit(long long b, float T) {
    const int bc[3] = {(int)(b % nb[0]), (int)((b / nb[0]) % nb[1]), (int)(b / ((long long)nb[0] * nb[1]))};
    std::vector<long long> node;
    for (int q = 0; q < (ND == 3 ? bs * bs * bs : bs * bs); q++) {
      const int c[3] = {bc[0] * bs + q % bs, bc[1] * bs + (q / bs) % bs, ND == 3 ? bc[2] * bs + q / (bs * bs) : 0};
      if (c[0] < n[0] && c[1] < n[1] && c[2] < n[2]) node.push_back(c[0] + st[1] * c[1] + st[2] * c[2]);
    }
    for (long long l : node) {
      pf[l] = INFINITY;
      if (!pending[l]) continue;
      int c[3];
      coords(l, c);
      double pot = EIK_INF;
      for (int a = 0; a < ND; a++)
        for (int s = -1; s <= 1; s += 2)
          if (inside(c, a, s)) pot = std::min(pot, high_word(t[l + s * st[a]]));
      pf[l] = round_up(pot + linc * slow[l]);
      if (!(pf[l] < INFINITY)) pending[l] = 0;
    }
    for (int scans = 0;;) {  // those in which a node changed
      float mn = INFINITY;
      for (long long l : node) mn = std::min(mn, pf[l]);
      if (!(mn <= T) || scans >= maxscans) {
        front[b] = mn;
        break;
      }
      float Tl = mn + din;
      if ((double)Tl < (double)mn + (double)din) Tl = std::nextafterf(Tl, INFINITY);
      Tl = std::min(T, Tl);
      bool moved = false;
      std::vector<long long> list;
      for (long long l : node)
        if (pf[l] <= Tl && list.size() < 64) list.push_back(l);
      for (size_t k = 0; k < list.size(); k += 32) {
        const size_t e = std::min(list.size(), k + 32);
        bool levels = false;
        std::vector<char> run(e - k);
        for (size_t i = k; i < e; i++) {
          const long long l = list[i];
          pf[l] = INFINITY;
          pending[l] = 0;
          run[i - k] = !(L[l] == -EIK_INF);
          double t1[ND][2], t2[ND][2], L1[ND][2], L2[ND][2];
          int d1[ND][2], c[3];
          coords(l, c);
          levels = levels || (run[i - k] && read(l, c, t1, t2, L1, L2, d1));
        }
        std::vector<Result> res(e - k);
        for (size_t i = k; i < e; i++) {
          int c[3];
          coords(list[i], c);
          if (run[i - k]) res[i - k] = evaluate(list[i], c, levels);
        }
        std::vector<char> ch(e - k);
        std::vector<double> oldL(e - k);
        for (size_t i = k; i < e; i++) {
          if (!run[i - k]) continue;
          const long long l = list[i];
          const Result& r = res[i - k];
          if (r.v == t[l] && r.L == L[l] && r.d == d[l]) continue;
          if (r.v > (double)T && r.v < EIK_INF && T < 3.402823466e38f) {
            pending[l] = 1;
            pf[l] = round_up(r.v);
            continue;
          }
          ch[i - k] = 1;
          moved = true;
          oldL[i - k] = L[l];
          t[l] = r.v;
          L[l] = r.L;
          d[l] = (uint8_t)r.d;
        }
        for (size_t i = k; i < e; i++) {
          if (!ch[i - k]) continue;
          int c[3];
          coords(list[i], c);
          changed(list[i], c, oldL[i - k], round_up(t[list[i]] + linc * slow[list[i]]), b);
        }
      }
      scans += moved;
    }
  }

  long long solve() {
    float T = 0.0f;
    long long r = 0;
    for (; r < maxrounds; r++) {
      float m = INFINITY;
      for (float f : front) m = std::min(m, f);
      if (!(m < INFINITY)) break;
      T = std::max(T, round_up((double)m + delta));
      for (long long b = 0; b < (long long)front.size(); b++) {
        const int colour = (int)(b % nb[0] + (b / nb[0]) % nb[1] + b / ((long long)nb[0] * nb[1])) & 1;
        if (colour == (r & 1) && front[b] <= T && front[b] < INFINITY) visit(b, T);
      }
    }
    return r;
  }
};

template <int ND>
int run(FILE* f, const int32_t* hd, const char* out) {
  Solver<ND> s;
  double dd[2];
  int32_t opt[4];
  int64_t ns;
  if (fread(dd, 8, 2, f) != 2 || fread(opt, 4, 4, f) != 4 || fread(&ns, 8, 1, f) != 1) return 3;
  for (int a = 0; a < 3; a++) s.n[a] = hd[1 + a];
  s.st[0] = 1;
  s.st[1] = s.n[0];
  s.st[2] = (long long)s.n[0] * s.n[1];
  s.N = s.st[2] * s.n[2];
  s.slow.resize(s.N);
  std::vector<int64_t> lin(ns);
  std::vector<double> tt(ns);
  if (fread(s.slow.data(), 8, s.N, f) != (size_t)s.N || fread(lin.data(), 8, ns, f) != (size_t)ns ||
      fread(tt.data(), 8, ns, f) != (size_t)ns)
    return 3;
  fclose(f);
  const bool small = opt[0] != 0;
  s.bs = ND == 3 ? (small ? 4 : 8) : (small ? 8 : 16);
  s.maxscans = opt[1] > 0 ? opt[1] : (ND == 3 ? (small ? 11 : 16) : (small ? 40 : 24));
  s.general = opt[2] != 0;
  s.maxrounds = opt[3];
  s.h = dd[0];
  s.c1u = 1.0 / (s.h * s.h);
  s.c2u = 9.0 / (4.0 * (s.h * s.h));
  const double u = s.h * *std::min_element(s.slow.begin(), s.slow.end());
  s.delta = dd[1] * u;
  s.linc = 0.999 * (2.0 / 3.0) * s.h / std::sqrt((double)ND);
  s.din = (float)((ND == 3 ? (small ? 0.75 : 0.5) : 1.0) * u);
  long long nbr = 1;
  for (int a = 0; a < 3; a++) {
    s.nb[a] = a < ND ? (s.n[a] + s.bs - 1) / s.bs : 1;
    nbr *= s.nb[a];
  }
  s.t.assign(s.N, EIK_INF);
  s.L.assign(s.N, EIK_INF);
  s.d.assign(s.N, 0);
  s.pf.assign(s.N, INFINITY);
  s.pending.assign(s.N, 0);
  s.front.assign(nbr, INFINITY);
  for (int64_t q = 0; q < ns; q++) {
    s.t[lin[q]] = tt[q];
    s.L[lin[q]] = -EIK_INF;
  }
  for (int64_t q = 0; q < ns; q++) {
    int c[3];
    s.coords(lin[q], c);
    for (int a = 0; a < ND; a++)
      for (int off = -2; off <= 2; off++)
        if (off && s.inside(c, a, off)) s.mark(lin[q] + off * s.st[a], round_up(tt[q]), -1);
  }
  const long long rounds = s.solve();
  long long unsettled = 0, tied = 0;
  for (long long l = 0; l < s.N; l++) {
    if (s.L[l] == -EIK_INF) continue;
    int c[3];
    s.coords(l, c);
    const Result r = s.by_general_rule(l, c);
    unsettled += !(r.v == s.t[l] && r.L == s.L[l] && r.d == s.d[l]);
    tied += s.d[l] != 0 && s.L[l] == s.t[l];
  }
  FILE* o = fopen(out, "wb");
  if (!o) return 3;
  const int64_t cnt[5] = {rounds, s.evals, s.slowpath, unsettled, tied};
  fwrite(s.t.data(), 8, s.N, o);
  fwrite(cnt, 8, 5, o);
  fclose(o);
  return 0;
}

}  // namespace

int main(int argc, char** argv) {
  if (argc != 3) return 2;
  FILE* f = fopen(argv[1], "rb");
  int32_t hd[4];
  if (!f || fread(hd, 4, 4, f) != 4) return 3;
  return hd[0] == 3 ? run<3>(f, hd, argv[2]) : run<2>(f, hd, argv[2]);
}
