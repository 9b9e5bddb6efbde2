// Nodes of a grid as the solves address them, and the outcomes of a node's visits.
#pragma once

#include "kernels.cuh"

namespace eik {

// Visit outcomes, in the order of eik_stats.fwd_visits. The forward solve by bricks has no visits
// of the first and the fourth kind: a pending node stays unvisited until its front is reached.
enum : unsigned {
  VISIT_STANDS = 0,  // value cached above the front, nothing it reads changed
  VISIT_SOURCE,      // source point (fixed)
  VISIT_UNREACHED,   // no neighbour reached yet
  VISIT_BOUND,       // lower bound above the front
  VISIT_WAIT,        // evaluated, above the front
  VISIT_SAME,        // evaluated, value and key unchanged
  VISIT_CHANGED,     // evaluated and accepted
  VISIT_NONE
};

// Result of the order rule on one node.
struct RuleOut {
  double v;
  Key key;
  int8_t cd[3];
};

// Neighbour directions of a node: k = 4*axis + {0: -2, 1: -1, 2: +1, 3: +2}.
__device__ __forceinline__ int dir_off(int k) { return (k & 3) < 2 ? (k & 3) - 2 : (k & 3) - 1; }
// Grid coordinates of node l. A problem has fewer than 2^32 nodes (a launch numbers its
// node-sources in 32 bits), so 32-bit division is exact and far cheaper than 64-bit.
__device__ __forceinline__ void node_coords(const GridDesc& g, long long l, int* c) {
  const unsigned ul = (unsigned)l, n0 = (unsigned)g.n[0], n1 = (unsigned)g.n[1];
  const unsigned q = ul / n0;
  c[0] = (int)(ul - q * n0);
  c[1] = (int)(q % n1);
  c[2] = (int)(q / n1);
}
// Linear index of the node in direction k of node l, which the direction must
// keep in the grid: the grid is column-major (lin3), so a step along an axis adds that axis's
// stride. Arithmetic only: an array indexed by the loop's axis would live in local memory.
__device__ __forceinline__ long long dir_lin(const GridDesc& g, long long l, int k) {
  const int ax = k >> 2;
  const long long st = ax == 0 ? 1LL : (ax == 1 ? (long long)g.n[0] : (long long)g.n[0] * g.n[1]);
  return l + dir_off(k) * st;
}

}  // namespace eik
