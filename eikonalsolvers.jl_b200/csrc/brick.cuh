// Bricks of the forward round solver: layout, and the visit that settles one brick.
//
// A problem's grid is cut into bricks of 8x8x8 nodes (3D) or 16x16 (2D). The traveltimes are
// kept brick by brick (a brick's nodes consecutive, x fastest), so a brick and the two layers
// around it that its stencils read come in as 16-byte pieces whatever the grid's size. The
// stencil reaches +-1 and +-2 along each axis: a brick reads only the bricks across its faces.
// Bricks are therefore coloured like a checkerboard, and a round visits bricks of one colour
// only: everything a visit reads outside its brick stands still while it runs, no write of a
// round is read in the same round, and a visit needs no fence, flag or retry.
//
// One warp visits one brick. It copies the brick and its surroundings to shared memory,
// evaluates the pending nodes there in the order of their fronts until none is left below the
// round's threshold, and writes the brick back. A node is pending from the moment something
// its rule may read has changed until it has been evaluated; the pending nodes of a brick are
// a bit mask in global memory between visits. A node that changes makes the nodes whose
// stencil reads it pending, in the warp's own brick (in shared memory) or in the brick across
// a face (its mask, at the end of the visit).
//
// Why this shape: visited one by one from worklists, a node costs ~100 scattered sectors
// (its neighbours, their codes and stamps, the relisting filter) and a round per layer of the
// front. A brick visit reads ~10 KB in full sectors for ~200 evaluations and settles several
// layers, so rounds are fewer (256^3 x 4 sources: 857 instead of 3970) and the evaluation chain
// runs on shared memory. 8^3 nodes with one warp: a front crosses a brick in sheets of about 64
// nodes, two warp-wide evaluations; larger bricks fill the lanes a little better but leave
// fewer warps per SM to hide latency. Forward solve, worklists of nodes -> bricks, B200:
// 256^3 x 4 420 -> 116 ms, 128^3 x 8 123 -> 33 ms, 64^3 x 32 48 -> 14 ms, 128^3 x 1 40 -> 10.4 ms,
// 1024x640 x 64 196 -> 39 ms (small bricks in the middle three). What bounds it: the longest visit of
// a round (256^3 x 4: 98 us, a visit averages 30 us, and 68 % of the warps' time is spent at the
// barrier; 31 % at 256^3 x 32), inside a visit the instructions' latency; DRAM and the FP64 pipe are
// idle (below 1 % and 3 %).
#pragma once

#include "kernels.cuh"
#include "node.cuh"

namespace eik {

constexpr unsigned FULL_WARP = 0xffffffffu;
constexpr unsigned PF_NONE = 0x7f800000u;  // +inf: no pending value

// Brick geometry. Nodes are numbered x + BX*(y + BY*z); the shared-memory cube holds the brick
// and two layers around it, x-pitch PY per row and PZ per plane, node (0,0,0) at ORG. Small
// bricks (4x4x4, 8x8) shorten the chain of steps of a round and are for solves whose rounds have
// fewer large bricks than the GPU has warps (small_bricks in api.cu).
template <int ND, bool SMALL>
struct Brick {
  static constexpr int BX = ND == 3 ? (SMALL ? 4 : 8) : (SMALL ? 8 : 16);
  static constexpr int BY = BX, BZ = ND == 3 ? BX : 1;
  static constexpr int NODES = BX * BY * BZ, WORDS = NODES / 32, FACES = 2 * ND;
  static constexpr int PY = BX + 4, PZ = ND == 3 ? PY * PY : 0;
  static constexpr int ORG = 2 * PZ + 2 * PY + 2, CUBE = ND == 3 ? PY * PY * PY : PY * PY;
  // Runs of the 3D cube that no stencil of the brick reads: two rows of PY before the brick's
  // in the plane z = -2, and four rows between the brick's rows of the planes z = -2, -1 and
  // z = BZ, BZ + 1 (each plane's last two rows and the next one's first two).
  static constexpr int FREE0 = 0, FREE1 = PZ - 2 * PY, FREE2 = (BZ + 3) * PZ - 2 * PY;
};

// Number of bricks along an axis and in a problem, and the brick-ordered index of a node.
template <int ND, bool SMALL>
EIK_HD int bricks_along(const GridDesc& g, int a) {
  typedef Brick<ND, SMALL> B;
  const int b = a == 0 ? B::BX : (a == 1 ? B::BY : B::BZ);
  return (g.n[a] + b - 1) / b;
}
template <int ND, bool SMALL>
EIK_HD long long brick_count(const GridDesc& g) {
  long long c = 1;
  for (int a = 0; a < ND; a++) c *= bricks_along<ND, SMALL>(g, a);
  return c;
}
template <int ND, bool SMALL>
EIK_HD long long brick_node(const GridDesc& g, int i, int j, int k) {
  typedef Brick<ND, SMALL> B;
  const int bi = i / B::BX, bj = j / B::BY, bk = ND == 3 ? k / B::BZ : 0;
  const long long b =
      bi + (long long)bricks_along<ND, SMALL>(g, 0) * (bj + (long long)bricks_along<ND, SMALL>(g, 1) * bk);
  return b * B::NODES + (i - bi * B::BX) + B::BX * ((j - bj * B::BY) + B::BY * (ND == 3 ? k - bk * B::BZ : 0));
}
EIK_HD long long brick_node(const GridDesc& g, bool small, int i, int j, int k) {
  if (g.nd == 3) return small ? brick_node<3, true>(g, i, j, k) : brick_node<3, false>(g, i, j, k);
  return small ? brick_node<2, true>(g, i, j, k) : brick_node<2, false>(g, i, j, k);
}

// Shared memory of one warp. The list of a scan and the spherical coefficients (1/h^2 and
// 9/(4h^2) of axes 1 and 2 per radial index of the brick) take free runs of the cube in 3D:
// 20.9 KB a warp, 11 warps an SM (small bricks: 5.0 KB).
template <int ND, bool SMALL>
struct __align__(16) WarpMem {
  typedef Brick<ND, SMALL> B;
  double cube[B::CUBE];                // traveltimes; sign bit: special key
  double slow[B::NODES];
  unsigned pf[B::NODES];               // pending front (float bits) or PF_NONE
  uint8_t code[B::NODES];
  unsigned face[B::FACES * B::WORDS];  // nodes made pending in the bricks across the faces
  unsigned facemin[8];                 // and their smallest front
  double extra[ND == 3 ? 2 : 48];
  __device__ __forceinline__ uint16_t* list() {
    return reinterpret_cast<uint16_t*>(ND == 3 ? cube + B::FREE0 : extra);  // 64 entries, 16 doubles
  }
  __device__ __forceinline__ double* coef() { return ND == 3 ? cube + B::FREE1 : extra + 16; }  // up to 32
};
static_assert(2 * Brick<3, true>::PY >= 16 && 4 * Brick<3, true>::PY >= 4 * 4 && 4 * Brick<3, false>::PY >= 4 * 8,
              "the free runs hold the list and the coefficients");

__device__ __forceinline__ unsigned front_bits(double v) {
  // smallest float >= v, finite: a pending node is never lost to overflow
  const float f = __double2float_ru(v);
  return v < EIK_INF ? __float_as_uint(fminf(f, 3.402823466e38f)) : PF_NONE;
}

// 16 bytes through L2 only: the brick state is written by other SMs between rounds, and L1
// may hold an older copy. (cp_async8 below goes through L1: for the slowness, which is constant.)
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ bool sign_set(double v) { return __double2hiint(v) < 0; }

// key_le without branches.
__device__ __forceinline__ bool key_le_flat(const Key& a, const Key& b) {
  const bool deep = (a.d < b.d) | ((a.d == b.d) & ((a.L == -EIK_INF) | (a.t <= b.t)));
  return (a.L < b.L) | ((a.L == b.L) & deep);
}

// The order rule by full keys, for the nodes the fast rule leaves out (about one in a thousand,
// but clustered), by the whole warp: prefix_rule (stencil.cuh) goes through the groups of equal
// keys one after the other; here the nodes take 2*ND lanes each, lane j the group of immediate
// neighbour j, and the rule's result is read off the groups' outcomes: the first one, in the
// order of the keys, at which the rule ends, or the one before a depth limit. One lane going
// through the groups took 14 000 cycles, which made the bricks where such nodes cluster the
// longest visits of a round (with the fast rule taking non-causal and mixed nodes: 256^3 x 4 forward
// 238 -> 151 ms).
//
// Called by all lanes; a lane's inputs are those of its node (the same in the node's 2*ND lanes),
// and so is what it returns. t: the node in the cube; ok2: sides (bit slot) where 2nd order is
// allowed; l: column-major node index; i: radial index; active: the lane has a node.
template <int ND, bool SMALL>
__device__ __noinline__ RuleOut rule_slow(const CoarseProblem& P, const double* t, unsigned ok2, long long l, int i,
                                          double slow, bool active, int lane) {
  typedef Brick<ND, SMALL> B;
  constexpr int G = 2 * ND;
  const int j = lane % G, base = lane - j;
  // the keys of immediate neighbour j and of the node beyond it
  const int a0 = j >> 1;
  const long long st = a0 == 0 ? 1LL : (a0 == 1 ? (long long)P.g.n[0] : (long long)P.g.n[0] * P.g.n[1]);
  const int cs = a0 == 0 ? 1 : (a0 == 1 ? B::PY : B::PZ), sh = (j & 1) ? -1 : 1;
  double v1 = active ? t[sh * cs] : EIK_INF, v2 = active && ((ok2 >> j) & 1u) ? t[2 * sh * cs] : EIK_INF;
  const bool s1 = sign_set(v1), s2 = sign_set(v2);
  const double l1 = s1 ? __ldcg(P.kL + l + sh * st) : v1, l2 = s2 ? __ldcg(P.kL + l + 2 * sh * st) : v2;
  const int d1 = s1 ? (int)__ldcg(P.kd + l + sh * st) : 0, d2 = s2 ? (int)__ldcg(P.kd + l + 2 * sh * st) : 0;
  v1 = fabs(v1);
  v2 = fabs(v2);
  const Key kg{l1, d1, v1};
  const bool reached = key_reached(kg);
  NbhdM nb;
  double L[G];
  int d[G];
  unsigned acc = 0u;
  int rank = 0;
#pragma unroll
  for (int k = 0; k < G; k++) {
    const int from = min(base + k, 31);
    const Key kn{__shfl_sync(FULL_WARP, l1, from), __shfl_sync(FULL_WARP, d1, from), __shfl_sync(FULL_WARP, v1, from)};
    const Key km{__shfl_sync(FULL_WARP, l2, from), __shfl_sync(FULL_WARP, d2, from), __shfl_sync(FULL_WARP, v2, from)};
    acc |= (unsigned)key_le_flat(kn, kg) << k | (unsigned)key_le_flat(km, kg) << (6 + k);
    rank += !key_le_flat(kg, kn);
    nb.t1[k >> 1][k & 1] = kn.t;
    nb.t2[k >> 1][k & 1] = km.t;
    L[k] = kn.L;
    d[k] = kn.d;
  }
  node_dh(P.g, i, nb.dh);
  nb.slow = slow;
  nb.c1u = P.c1u;
  nb.c2u = P.c2u;
  int8_t cd[3] = {0, 0, 0};
  bool neg = false;
  double v = EIK_INF;
  if (reached) v = update_at_g<ND>(nb, acc, cd, &neg);
  const bool above = v > kg.L;
  const Key mine = above ? key_normal(v) : Key{kg.L, kg.d + 1, v};
  // the next group: the smallest rank above this one's (equal keys share a rank)
  int next = 7;
  Key kn = key_unreached();
#pragma unroll
  for (int k = 0; k < G; k++) {
    const int rk = __shfl_sync(FULL_WARP, reached ? rank : 7, min(base + k, 31));
    if (rk > rank && rk < next) {
      next = rk;
      kn = Key{L[k], d[k], nb.t1[k >> 1][k & 1]};
    }
  }
  // how the rule leaves this group: 2 at the depth limit, 1 with this group's value, 0 onwards
  const int event = !reached ? 0 : (!above && kg.d >= EIK_MAX_DEPTH && rank > 0) ? 2 : (next == 7 || key_le(mine, kn)) ? 1 : 0;
  int first = 8, pick = -1, before = -1, brank = -1, fev = 0;
#pragma unroll
  for (int k = 0; k < G; k++) {
    const int code = __shfl_sync(FULL_WARP, reached ? rank * 4 + event : 32, min(base + k, 31));
    const int rk = code >> 2, ek = code & 3;
    if (ek && rk < first) {
      first = rk;
      fev = ek;
      pick = k;
    }
  }
#pragma unroll
  for (int k = 0; k < G; k++) {
    const int rk = __shfl_sync(FULL_WARP, reached ? rank : 8, min(base + k, 31));
    if (rk < first && rk > brank) {
      brank = rk;
      before = k;
    }
  }
  if (fev == 2) pick = before;
  const int from = min(base + max(pick, 0), 31);
  const int packed = ((int)(uint8_t)cd[0]) | ((int)(uint8_t)cd[1] << 8) | ((int)(uint8_t)cd[2] << 16);
  RuleOut o;
  o.v = __shfl_sync(FULL_WARP, v, from);
  o.key.L = __shfl_sync(FULL_WARP, mine.L, from);
  o.key.d = __shfl_sync(FULL_WARP, mine.d, from);
  const int pc = __shfl_sync(FULL_WARP, packed, from);
  if (pick < 0) {
    o.v = EIK_INF;
    o.key.L = EIK_INF;
    o.key.d = 0;
  }
  o.key.t = o.v;
#pragma unroll
  for (int a = 0; a < 3; a++) o.cd[a] = pick < 0 ? (int8_t)0 : (int8_t)(pc >> (8 * a));
  return o;
}

// Copies brick b (at brick coordinates bc, bricks nb per axis) of a brick-ordered array and the
// layers around it that exist to a cube; positions across the grid's faces get `outside`.
template <int ND, bool SMALL>
__device__ __forceinline__ void load_cube(double* cube, const double* array, size_t b, const int (&bc)[3],
                                          const int (&nb)[3], double outside, int lane) {
  typedef Brick<ND, SMALL> B;
  const double* own = array + b * B::NODES;
  constexpr int ROWP = B::BX / 2;  // 16-byte pieces of a row
#pragma unroll
  for (int q = 0; q < B::NODES / 2; q += 32) {
    const int e = q + lane, row = e / ROWP, xp = e % ROWP;
    const int y = row % B::BY, z = row / B::BY;
    cp_async16(&cube[B::ORG + z * B::PZ + y * B::PY + 2 * xp], own + 2 * e);
  }
  // layers across the faces: side 0 = +, side 1 = - (as slot())
  const long long bst[3] = {1, nb[0], (long long)nb[0] * nb[1]};
#pragma unroll
  for (int a = 0; a < ND; a++)
#pragma unroll
    for (int s = 0; s < 2; s++) {
      const bool have = s == 0 ? bc[a] + 1 < nb[a] : bc[a] > 0;
      const double* src = s == 0 ? own + bst[a] * B::NODES : own - bst[a] * B::NODES;
      // pairs of the two layers: along x one pair per row, else ROWP pairs per row of 2 rows
      const int pieces = a == 0 ? B::BY * B::BZ : (a == 1 ? 2 * ROWP * B::BZ : 2 * ROWP * B::BY);
#pragma unroll
      for (int q = 0; q < pieces; q += 32) {
        const int e = q + lane;
        if (e < pieces) {
          int ci, si;
          if (a == 0) {
            const int y = e % B::BY, z = e / B::BY;
            ci = B::ORG + z * B::PZ + y * B::PY + (s == 0 ? B::BX : -2);
            si = e * B::BX + (s == 0 ? 0 : B::BX - 2);
          } else if (a == 1) {
            const int z = e / (2 * ROWP), rr = (e / ROWP) & 1, xp = e % ROWP;
            const int y = s == 0 ? rr : B::BY - 2 + rr;
            ci = B::ORG + z * B::PZ + (s == 0 ? B::BY + rr : rr - 2) * B::PY + 2 * xp;
            si = (z * B::BY + y) * B::BX + 2 * xp;
          } else {
            const int rr = e / (B::BY * ROWP), y = (e / ROWP) % B::BY, xp = e % ROWP;
            const int z = s == 0 ? rr : B::BZ - 2 + rr;
            ci = B::ORG + (s == 0 ? B::BZ + rr : rr - 2) * B::PZ + y * B::PY + 2 * xp;
            si = (z * B::BY + y) * B::BX + 2 * xp;
          }
          if (have) {
            cp_async16(&cube[ci], src + si);
          } else {
            cube[ci] = outside;
            cube[ci + 1] = outside;
          }
        }
      }
    }
}

// Visit outcome counters of a warp (lane k < 7 holds outcome k).
struct VisitTally {
  unsigned n = 0;
  __device__ __forceinline__ void add(unsigned oc, int lane) {
    const unsigned b0 = __ballot_sync(FULL_WARP, oc & 1u), b1 = __ballot_sync(FULL_WARP, oc & 2u),
                   b2 = __ballot_sync(FULL_WARP, oc & 4u);
    if (lane < 7) {
      const unsigned mk = ((lane & 1) ? b0 : ~b0) & ((lane & 2) ? b1 : ~b1) & ((lane & 4) ? b2 : ~b2);
      n += (unsigned)__popc(mk);
    }
  }
};

// Scans (steps of up to two warps of nodes) of a visit in which a node changes, before it hands its pending
// nodes back to the next round of its colour. A visit needs about eight; a few need a hundred and would
// hold up the round: 256^3 x 4 at 8 / 12 / 16 / 24 / 192 scans: 140 / 126 / 122 / 129 / 150 ms, 64^3 x
// 32 18.2 / 16.6 / 17.0 / 19.4 / 20.5 ms, 1024x640 x 64 61 / 53 / 49 / 44 / 53 ms. Small 3D bricks have an
// eighth of the nodes to settle: 128^3 x 1 at 8 / 11 / 16 scans 10.2 / 10.4 / 11.9 ms, 128^3 x 8 33.7 / 33.2 /
// 36.0, 64^3 x 32 14.3 / 13.9 / 14.8, spherical 100x90x90 x 12 35.7 / 33.0 / 34.1; small 2D ones, which
// with wide rounds settle in a few long visits, 24 / 28 / 32 / 40 / 56 at the best width of each: 300x220 x 4
// 5.2 / 4.6 / 4.0 / 4.0 / 4.0 ms, 517x323 x 4 8.8 / 7.7 / 6.9 / 6.6 / 6.7, 128x80 x 1 2.0 / 1.6 / 1.5 / 1.4 / 1.4
// (all with every scan counted). It also ends a visit in which values alternate (the rule's depth limit lets some
// transient keys do so). Scans without a change do not count: a visit starts from the nodes' lower
// bounds, so nodes that wait above the front are evaluated anew by each, and where velocities differ by 30 or
// more they lie in more inner windows than the bound has scans; counted, they kept every visit from the nodes
// behind them for good. There are at most as many as nodes (each takes one out of the visit). Times are the
// same (256^3 x 4 gradient 130.5 -> 130.4 ms, 1024x640 x 64 52.4 -> 52.1), a 64^3 layer of 20 times the velocity
// 27 ms.
template <int ND, bool SMALL>
constexpr int VISIT_MAX_SCANS = ND == 3 ? (SMALL ? 11 : 16) : (SMALL ? 40 : 24);

// Which steps -2, -1, +1, +2 along an axis stay within [lo, hi) from position p: bits 0..3 of
// nibble p of the table, for positions 0..15 (low half: 0..7).
__device__ __forceinline__ unsigned long long step_table(int lo, int hi) {
  auto upto = [](int e) { return e <= 0 ? 0ull : (e >= 16 ? ~0ull : (1ull << (4 * e)) - 1ull); };
  const unsigned long long one = 0x1111111111111111ull;
  return (one & ~upto(lo + 2)) | ((one << 1) & ~upto(lo + 1)) | ((one << 2) & upto(hi - 1)) | ((one << 3) & upto(hi - 2));
}

// Settles brick b up to threshold T (a float-valued bound): returns the smallest pending front
// left in it (float bits, PF_NONE if none), its mask written back. The fronts and masks for
// the bricks across its faces are left in w.facemin / w.face for the caller to publish.
template <int ND, bool SMALL>
__device__ __forceinline__ unsigned visit_brick(WarpMem<ND, SMALL>& w, const BrickState& bs, const CoarseProblem& P, size_t b,
                                                const int (&bc)[3], const int (&nb)[3], float T, int lane,
                                                VisitTally& tally) {
  typedef Brick<ND, SMALL> B;
  uint16_t* list = w.list();
  double* coef = w.coef();
  unsigned pend = 0u;
  if (lane < B::WORDS) pend = __ldcg(bs.mask + b * B::WORDS + lane);
  load_cube<ND, SMALL>(w.cube, bs.t, b, bc, nb, EIK_INF, lane);
  if (lane < B::NODES / 16) cp_async16(&w.code[lane * 16], bs.code + b * B::NODES + lane * 16);
  for (int q = lane; q < B::FACES * B::WORDS; q += 32) w.face[q] = 0u;
  if (lane < 8) w.facemin[lane] = PF_NONE;
  // the problem's constants in registers: the visit's barriers would make the compiler read
  // them from memory again at every step
  const int n[3] = {P.g.n[0], P.g.n[1], P.g.n[2]};
  const int x0[3] = {bc[0] * B::BX, bc[1] * B::BY, bc[2] * B::BZ};
#pragma unroll
  for (int q = 0; q < B::NODES; q += 32) {
    const int e = q + lane, x = x0[0] + e % B::BX, y = x0[1] + (e / B::BX) % B::BY, z = x0[2] + e / (B::BX * B::BY);
    if (x < n[0] && y < n[1] && z < n[2])
      cp_async8(&w.slow[e], P.slow + (x + (long long)n[0] * (y + (long long)n[1] * z)));
  }
  double* const kL = P.kL;
  uint8_t* const kd = P.kd;
  const bool cart = P.c1u > 0.0;
  if (!cart && lane < B::BX && x0[0] + lane < n[0]) {
    double dh[3];
    node_dh(P.g, x0[0] + lane, dh);
#pragma unroll
    for (int a = 1; a < ND; a++) {
      coef[(lane * (ND - 1) + a - 1) * 2] = 1.0 / (dh[a] * dh[a]);
      coef[(lane * (ND - 1) + a - 1) * 2 + 1] = 9.0 / (4.0 * (dh[a] * dh[a]));
    }
  }
  const double h0 = P.g.spac[0];
  const double c10 = cart ? P.c1u : 1.0 / (h0 * h0), c20 = cart ? P.c2u : 9.0 / (4.0 * (h0 * h0));
  const double linc = P.linc;
  const float din = P.din;
  // steps that stay in the brick, and in the grid; whether 2nd order is allowed everywhere
  unsigned long long tb[ND], tg[ND];
  bool border = false;
#pragma unroll
  for (int a = 0; a < ND; a++) {
    const int ext = a == 0 ? B::BX : (a == 1 ? B::BY : B::BZ), left = n[a] - x0[a];
    tb[a] = step_table(0, min(ext, left));
    tg[a] = step_table(x0[a] > 0 ? -2 : 0, left);
    border = border || x0[a] == 0 || left < ext + 2;
  }
  cp_async_wait();
  __syncwarp();
  // fronts of the pending nodes: smallest neighbouring traveltime plus the least increment
  // (from the high words, which is exact enough for an order, and for all nodes, which keeps
  // the loads in flight)
  const unsigned* hi = reinterpret_cast<const unsigned*>(w.cube) + 1;
#pragma unroll 4
  for (int k = 0; k < B::WORDS; k++) {
    const unsigned word = __shfl_sync(FULL_WARP, pend, k);
    const int q = 32 * k + lane;
    const int ci = B::ORG + (q / (B::BX * B::BY)) * B::PZ + ((q / B::BX) % B::BY) * B::PY + q % B::BX;
    auto t = [&](int off) { return hi[2 * (ci + off)] & 0x7fffffffu; };
    unsigned pot = min(min(t(1), t(-1)), min(t(B::PY), t(-B::PY)));
    if constexpr (ND == 3) pot = min(pot, min(t(B::PZ), t(-B::PZ)));
    const unsigned f = front_bits(__hiloint2double((int)pot, 0) + linc * w.slow[q]);
    w.pf[q] = ((word >> lane) & 1u) ? f : PF_NONE;
  }
  __syncwarp();
  const unsigned Tb = __float_as_uint(T), below = (1u << lane) - 1u;
  unsigned left = PF_NONE, leftmask = 0u;
  int scans = 0;  // in which a node changed
#pragma unroll 1
  for (;;) {
    unsigned v[B::WORDS];
    unsigned mn = PF_NONE;
#pragma unroll
    for (int k = 0; k < B::WORDS; k++) {
      v[k] = w.pf[32 * k + lane];
      mn = min(mn, v[k]);
    }
    mn = __reduce_min_sync(FULL_WARP, mn);
    if (mn > Tb || mn == PF_NONE || scans >= VISIT_MAX_SCANS<ND, SMALL>) {
      left = mn;
#pragma unroll
      for (int k = 0; k < B::WORDS; k++) {
        const unsigned mm = __ballot_sync(FULL_WARP, v[k] != PF_NONE);
        if (lane == k) leftmask = mm;
      }
      break;
    }
    // the nodes within the inner window above the smallest front, up to two warps of them
    const float Tl = fminf(T, __fadd_ru(__uint_as_float(mn), din));
    const unsigned Tlb = min(__float_as_uint(Tl), PF_NONE - 1u);
    int cnt = 0;
    unsigned sel[B::WORDS];
#pragma unroll
    for (int k = 0; k < B::WORDS; k++) sel[k] = __ballot_sync(FULL_WARP, v[k] <= Tlb);
#pragma unroll
    for (int k = 0; k < B::WORDS; k++) {
      const int pos = cnt + __popc(sel[k] & below);
      if (v[k] <= Tlb && pos < 64) list[pos] = (uint16_t)(32 * k + lane);
      cnt += __popc(sel[k]);
    }
    cnt = min(cnt, 64);
    bool moved = false;
    __syncwarp();
#pragma unroll 1
    for (int c0 = 0; c0 < cnt; c0 += 32) {
      const bool act = c0 + lane < cnt;
      const unsigned uq = act ? (unsigned)list[c0 + lane] : 0u;
      const int q = (int)uq, x = (int)(uq % B::BX), y = (int)((uq / B::BX) % B::BY), z = (int)(uq / (B::BX * B::BY));
      const int ci = B::ORG + z * B::PZ + y * B::PY + x;
      if (act) w.pf[q] = PF_NONE;
      const double traw = w.cube[ci];
      const double told = fabs(traw);
      const double slow = w.slow[q];
      double t1[ND][2], t2[ND][2];
      int sgn = 0;
      unsigned ok2 = 0xffu;
#pragma unroll
      for (int a = 0; a < ND; a++) {
        const int st = a == 0 ? 1 : (a == 1 ? B::PY : B::PZ);
#pragma unroll
        for (int s = 0; s < 2; s++) {
          const int sh = s == 0 ? st : -st;
          t1[a][s] = w.cube[ci + sh];
          t2[a][s] = w.cube[ci + 2 * sh];
        }
      }
      if (border) {
        // 2nd order needs the first neighbour off the border in every coordinate (isonbord)
        const int gx[3] = {x0[0] + x, x0[1] + y, x0[2] + z};
#pragma unroll
        for (int a = 0; a < ND; a++) {
          bool inner = true;
#pragma unroll
          for (int d = 0; d < ND; d++)
            if (d != a) inner = inner && gx[d] >= 1 && gx[d] <= n[d] - 2;
          if (!(inner && gx[a] + 1 <= n[a] - 2)) ok2 &= ~(1u << slot(a, 0));
          if (!(inner && gx[a] - 1 >= 1)) ok2 &= ~(1u << slot(a, 1));
        }
#pragma unroll
        for (int a = 0; a < ND; a++)
#pragma unroll
          for (int s = 0; s < 2; s++)
            if (!((ok2 >> slot(a, s)) & 1u)) t2[a][s] = EIK_INF;
      }
#pragma unroll
      for (int a = 0; a < ND; a++)
#pragma unroll
        for (int s = 0; s < 2; s++) sgn |= __double2hiint(t1[a][s]) | __double2hiint(t2[a][s]);
      double Lold = told;
      int dold = 0;
      unsigned oc = VISIT_NONE;
      if (act && sign_set(traw)) {
        const long long l = (x0[0] + x) + (long long)n[0] * ((x0[1] + y) + (long long)n[1] * (x0[2] + z));
        Lold = __ldcg(kL + l);
        dold = (int)__ldcg(kd + l);
        if (Lold == -EIK_INF) oc = VISIT_SOURCE;  // source points are fixed
      }
      const bool ev = act && oc == VISIT_NONE;
      double nv, nL;
      int nd;
      int8_t cd[3] = {0, 0, 0};
      bool done;
      {
        double c1[ND], c2[ND];
        c1[0] = c10;
        c2[0] = c20;
#pragma unroll
        for (int a = 1; a < ND; a++) {
          c1[a] = c10;
          c2[a] = c20;
        }
        if (!cart) {
#pragma unroll
          for (int a = 1; a < ND; a++) {
            c1[a] = coef[(x * (ND - 1) + a - 1) * 2];
            c2[a] = coef[(x * (ND - 1) + a - 1) * 2 + 1];
          }
        }
        int8_t cf[ND];
        if (ND == 2 || !__any_sync(FULL_WARP, ev && sgn < 0)) {
          const int d1[ND][2] = {};
          done = prefix_rule_fast<ND, false>(t1, t2, t1, t2, d1, c1, c2, slow, &nv, &nL, &nd, cf);
          nd = nL == nv ? 0 : 1;
          if (ND == 2 && sgn < 0) done = false;
        } else if constexpr (ND == 3) {
          // special neighbours of some lane: the same with key levels. In 2D, where that is one
          // batch in 400, the general rule takes those nodes: the second copy of the fast rule
          // costs the others more (300x220 x 4 5.5 -> 5.2 ms without it).
          const long long l = (x0[0] + x) + (long long)n[0] * ((x0[1] + y) + (long long)n[1] * (x0[2] + z));
          double L1[ND][2], L2[ND][2];
          int d1[ND][2];
#pragma unroll
          for (int a = 0; a < ND; a++) {
            const long long st = a == 0 ? 1LL : (a == 1 ? (long long)n[0] : (long long)n[0] * n[1]);
#pragma unroll
            for (int s = 0; s < 2; s++) {
              const long long l1 = s == 0 ? l + st : l - st, l2 = s == 0 ? l1 + st : l1 - st;
              L1[a][s] = sign_set(t1[a][s]) ? __ldcg(kL + l1) : t1[a][s];
              L2[a][s] = sign_set(t2[a][s]) ? __ldcg(kL + l2) : t2[a][s];
              d1[a][s] = sign_set(t1[a][s]) ? (int)__ldcg(kd + l1) : 0;
            }
          }
          done = prefix_rule_signed<ND>(t1, t2, L1, L2, d1, c1, c2, slow, &nv, &nL, &nd, cf);
        }
#pragma unroll
        for (int a = 0; a < ND; a++) cd[a] = cf[a];
      }
      for (unsigned sl = __ballot_sync(FULL_WARP, ev && !done); sl;) {
        // the next 32 / (2*ND) of them, 2*ND lanes each
        constexpr int G = 2 * ND, PAR = 32 / G;
        unsigned mine = sl;
        for (int k = 0; k < lane / G; k++) mine &= mine - 1u;
        const bool has = mine != 0u && lane < PAR * G;
        const int src = has ? __ffs(mine) - 1 : 0;
        const int sq = __shfl_sync(FULL_WARP, q, src), sci = __shfl_sync(FULL_WARP, ci, src);
        const unsigned sok = __shfl_sync(FULL_WARP, ok2, src);
        const double ss = __shfl_sync(FULL_WARP, slow, src);
        const int sx = x0[0] + sq % B::BX;
        const long long l = sx + (long long)n[0] * ((x0[1] + (sq / B::BX) % B::BY) + (long long)n[1] * (x0[2] + sq / (B::BX * B::BY)));
        const RuleOut o = rule_slow<ND, SMALL>(P, &w.cube[sci], sok, l, sx, ss, has, lane);
        // back to the node's own lane
        const int place = __popc(sl & below);
        const bool take = ((sl >> lane) & 1u) && place < PAR;
        const int from = take ? place * G : 0;
        const double rv = __shfl_sync(FULL_WARP, o.v, from), rL = __shfl_sync(FULL_WARP, o.key.L, from);
        const int rd = __shfl_sync(FULL_WARP, o.key.d, from);
        const int rc = __shfl_sync(FULL_WARP, (o.cd[0] + 2) | (o.cd[1] + 2) << 4 | (o.cd[2] + 2) << 8, from);
        if (take) {
          nv = rv;
          nL = rL;
          nd = rd;
#pragma unroll
          for (int a = 0; a < 3; a++) cd[a] = (int8_t)(((rc >> (4 * a)) & 15) - 2);
        }
        for (int k = 0; k < PAR && sl; k++) sl &= sl - 1u;
      }
      __syncwarp();  // every lane has read before any writes
      bool changed = false;
      if (ev) {
        const bool same = nv == told && nL == Lold && nd == dold;  // +inf equals +inf
        const bool wait = !same && nv > (double)T && nv < EIK_INF && T < 3.402823466e38f;
        changed = !same && !wait;
        moved = moved || changed;
        oc = same ? (nv < EIK_INF ? VISIT_SAME : VISIT_UNREACHED) : (wait ? VISIT_WAIT : VISIT_CHANGED);
        if (wait) {
          w.pf[q] = front_bits(nv);  // not final yet: the old value stands until the front is there
        } else {
          const bool spec = !(nL == nv && nd == 0);
          w.cube[ci] = spec ? -nv : nv;
          w.code[q] = pack_codes(cd, ND);
          if (spec && changed) {
            const long long l = (x0[0] + x) + (long long)n[0] * ((x0[1] + y) + (long long)n[1] * (x0[2] + z));
            kL[l] = nL;
            kd[l] = (uint8_t)nd;
          }
        }
      }
      tally.add(oc, lane);
      __syncwarp();
      // The nodes whose stencil reads a changed node become pending, except those whose own key
      // is at most both its old and its new key: their rule never accepts it, so their value
      // cannot change. An ordinary key (t, 0, t) is at most both when t is at most both levels;
      // a special one (sign bit: largest as unsigned) is always taken. The node two steps away
      // reads this one only beyond a reached node.
      unsigned cm = 0u;
      if (changed) {
        const unsigned long long lim = (unsigned long long)__double_as_longlong(fmin(Lold, nL));
#pragma unroll
        for (int a = 0; a < ND; a++) {
          const int st = a == 0 ? 1 : (a == 1 ? B::PY : B::PZ);
          const unsigned long long m2 = __double_as_longlong(w.cube[ci - 2 * st]), m1 = __double_as_longlong(w.cube[ci - st]),
                                   p1 = __double_as_longlong(w.cube[ci + st]), p2 = __double_as_longlong(w.cube[ci + 2 * st]);
          const bool rm = ((unsigned)(m1 >> 32) & 0x7fffffffu) < 0x7ff00000u,
                     rp = ((unsigned)(p1 >> 32) & 0x7fffffffu) < 0x7ff00000u;
          cm |= (rm && m2 > lim ? 1u : 0u) << (4 * a) | (m1 > lim ? 2u : 0u) << (4 * a) |
                (p1 > lim ? 4u : 0u) << (4 * a) | (rp && p2 > lim ? 8u : 0u) << (4 * a);
        }
        unsigned inb = 0u, ing = 0u;
#pragma unroll
        for (int a = 0; a < ND; a++) {
          const int p = a == 0 ? x : (a == 1 ? y : z);
          inb |= ((unsigned)(tb[a] >> (4 * p)) & 15u) << (4 * a);
          ing |= ((unsigned)(tg[a] >> (4 * p)) & 15u) << (4 * a);
        }
        // their front: the least increment over the new value, at this node's slowness (an
        // ordering only: a pending node is evaluated whatever its front was)
        const unsigned fb = front_bits(nv + linc * slow);
        const unsigned in = cm & inb;
        cm &= ing & ~inb;
#pragma unroll
        for (int k = 0; k < 4 * ND; k++) {
          const int a = k >> 2, j = k & 3;
          const int qst = a == 0 ? 1 : (a == 1 ? B::BX : B::BX * B::BY);
          if ((in >> k) & 1u) atomicMin(&w.pf[q + (j < 2 ? j - 2 : j - 1) * qst], fb);
        }
        while (cm) {
          const int k = __ffs(cm) - 1, a = k >> 2, j = k & 3;
          cm &= cm - 1u;
          const int off = j < 2 ? j - 2 : j - 1;
          const int ext = a == 0 ? B::BX : (a == 1 ? B::BY : B::BZ);
          const int qst = a == 0 ? 1 : (a == 1 ? B::BX : B::BX * B::BY);
          const int qj = q + (j < 2 ? off + ext : off - ext) * qst, f = 2 * a + (j < 2 ? 1 : 0);
          atomicOr(&w.face[f * B::WORDS + (qj >> 5)], 1u << (qj & 31));
          atomicMin(&w.facemin[f], fb);
        }
      }
      __syncwarp();
    }
    scans += __any_sync(FULL_WARP, moved);
  }
  // write back
  double* own = bs.t + b * B::NODES;
  constexpr int ROWP = B::BX / 2;
#pragma unroll
  for (int q = 0; q < B::NODES / 2; q += 32) {
    const int e = q + lane, row = e / ROWP, xp = e % ROWP;
    const int y = row % B::BY, z = row / B::BY;
    *reinterpret_cast<double2*>(own + 2 * e) =
        *reinterpret_cast<const double2*>(&w.cube[B::ORG + z * B::PZ + y * B::PY + 2 * xp]);
  }
  if (lane < B::NODES / 16)
    *reinterpret_cast<uint4*>(bs.code + b * B::NODES + lane * 16) = *reinterpret_cast<const uint4*>(&w.code[lane * 16]);
  if (lane < B::WORDS) bs.mask[b * B::WORDS + lane] = leftmask;
  return left;
}

}  // namespace eik
