// Device-side interfaces between the kernels of libeikcuda and its host runtime.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "common.cuh"

namespace eik {

// Refined-grid window of one source (createfinegrid, eikmainfwd.jl:950-1104), 0-based.
struct FineInfo {
  int32_t ds;
  int32_t ijk1[3];    // coarse index of the window origin
  int32_t nf[3];      // fine grid size
  int32_t outmin[3];  // window clipped at the model's lower border on this axis
  int32_t outmax[3];
};

// Per-source results of the start-up stage.
struct SrcOut {
  FineInfo fine;
  int32_t nseeds;       // coarse source points (traveltimes fixed before the coarse solve)
  int32_t nsrcf;        // source-box corners (of the fine grid if refined, else coarse)
  int32_t nacc;         // accepted fine nodes at the stop (refined only)
  uint32_t warn;
  int32_t corn[8][3];   // source-box corners
  double distcorn[8];
  double velcorn[8];
};

struct ForwardBatch {
  GridDesc g;               // coarse grid
  int32_t nsrc;
  int32_t ds, noderadius;
  int32_t seedcap;          // capacity of seed lists per source
  long long nfmax;          // capacity of fine arrays per source
  int32_t heapcap;          // shared-memory heap capacity (fine FMM)
  const double* vel;        // coarse velocity
  const double* slow;       // 1/vel
  const double* coordsrc;   // nsrc x nd
  SrcOut* out;
  int32_t* seed_lin;        // nsrc x seedcap: coarse node index
  double* seed_tt;          // nsrc x seedcap
  double* fine_tt;          // nsrc x nfmax
  uint8_t* fine_status;
  uint8_t* fine_code;
  int32_t* fine_idx;        // heap handle positions
  int32_t* fine_order;      // accepted fine nodes in FMM order
  uint8_t* fine_onh;        // accepted fine node coincides with a coarse node
  uint32_t* err;
};

// One coarse solve: a source on a grid. Several problems share one persistent launch.
struct CoarseProblem {
  GridDesc g;
  const double* slow;
  double* t;       // traveltime
  uint8_t* code;   // packed derivative codes; bit 7: special key (source or non-causal)
  double* kL;      // key level of special nodes (-inf for source points)
  uint8_t* kd;     // key depth of special nodes
  double delta;    // round width of the forward solve (traveltime units)
  double linc;     // least increment of the local update over a neighbour per unit of slowness: (2/3) h / sqrt(nd),
                   // h the smallest spacing
  float din;       // inner window of a brick visit (traveltime units)
  double c1u, c2u; // Cartesian grids: the local solver's coefficients 1/h^2 and 9/(4h^2); 0 otherwise
};

// The coefficients of a grid with the same spacing h on every axis, computed with the
// local solver's own expressions (so they are the values it would compute per call).
EIK_HD void uniform_coeffs(const GridDesc& g, double* c1u, double* c2u) {
  if (is_cart(g)) {
    const double h = g.spac[0];
    *c1u = 1.0 / (h * h);
    *c2u = 9.0 / (4.0 * (h * h));
  } else {
    *c1u = *c2u = 0.0;
  }
}

// Counters of the round-synchronous solves.
struct RoundState {
  unsigned int* bar;           // [2] grid barrier: arrivals, generation
  int32_t* rounds;             // rounds run
  unsigned long long* visits;  // [7] outcomes of the forward's visits
  int32_t max_rounds;
};

// Inner window of a brick visit: the nodes evaluated together lie within this much of the
// brick's smallest pending front. Narrower windows re-evaluate fewer nodes, wider ones fill
// more lanes of a step; u is the least time across one node (smallest spacing x slowness).
// 3D, 0.35 / 0.5 / 0.75 u with small bricks: 64^3 x 32 15.2 / 14.9 / 14.5 ms; large ones 0.5 u.
EIK_HD float inner_window(int nd, bool small, double u) { return (float)((nd == 3 ? (small ? 0.75 : 0.5) : 1.0) * u); }

// State of the forward solve by bricks (brick.cuh): problem p's bricks are p * stride + b.
struct BrickState {
  double* t;            // traveltimes in brick order; sign bit: special key
  uint8_t* code;        // derivative codes in brick order (low 7 bits)
  unsigned* mask;       // pending nodes of each brick, one bit a node
  unsigned* front;      // smallest pending front of each brick (float bits)
  unsigned* listed;     // brick is in a list
  unsigned* lists;      // [colour*2+phase][listcap]: bricks to visit
  size_t listcap;
  unsigned* ctr;        // cnt[colour*2+phase] at 0..3, grab[round % 3] at 4..6
  unsigned* exam;       // [4][nprob] smallest front left by a round's visits (float bits)
  unsigned* marks;      // [4][nprob] smallest front a round's visits put on other bricks
  float* thr;           // [2][nprob] threshold of the previous / current round
  unsigned stride;      // bricks per problem (the call's largest grid)
  int32_t small;        // small bricks
};

struct SolveArgs {
  const CoarseProblem* probs;
  int32_t nprob;
  int32_t nd;
  unsigned long long* activations;  // list entries visited
  unsigned long long* node_evals;
  uint32_t* err;
  int32_t* abort_flag;
  long long timeout_ns;
  RoundState rs;
  BrickState bs;
};


// launchers (defined in the .cu files)
void launch_srcbox(const ForwardBatch& fb, cudaStream_t st);
void launch_fine(const ForwardBatch& fb, cudaStream_t st);
size_t fine_smem_bytes(int heapcap);
// Brick state reset, seeding from per-problem seed lists (fixed values), the solve, and the
// results in the problems' own arrays (column-major traveltimes and codes).
void launch_bricks_init(const SolveArgs& sa, cudaStream_t st);
void launch_bricks_seed(const SolveArgs& sa, const int32_t* seed_lin, const double* seed_tt, const SrcOut* out,
                        bool fine_corners, int seedcap, cudaStream_t st);
cudaError_t launch_bricks_solve(const SolveArgs& sa, int nsm, cudaStream_t st);
// All four in one launch after the counters' (reset, seeds, solve, store), for small solves.
cudaError_t launch_bricks_fused(const SolveArgs& sa, const int32_t* seed_lin, const double* seed_tt, const SrcOut* out,
                                bool fine_corners, int seedcap, int nsm, cudaStream_t st);
void launch_bricks_store(const SolveArgs& sa, cudaStream_t st);
// Nodes of a brick, and bricks of a grid (rounded up to whole ones).
int brick_size(int nd, bool small);
unsigned long long brick_number(const GridDesc& g, bool small);
// Refined start-up as a fixed point: window set-up, the fine problems' arrays, the
// acceptance set at the reference's stop, and the exact heap replay for the sources
// whose stop is decided by a tie (flags in fine_tie, 1 = replay needed, 2 = its warning only).
void launch_fine_setup(const ForwardBatch& fb, CoarseProblem* fprobs, const double* dsmin, double gate, bool small,
                       int32_t* fseed_lin, double* fseed_tt, double* fine_slow, double* fine_kL, uint8_t* fine_kd,
                       cudaStream_t st);
void launch_fine_select(const ForwardBatch& fb, const CoarseProblem* fprobs, uint8_t* fine_tie, cudaStream_t st);
void launch_fine_replay(const ForwardBatch& fb, const CoarseProblem* fprobs, const uint8_t* fine_tie, cudaStream_t st);
void launch_picks(const GridDesc& g, const double* t, long long N, int nsrc, const long long* recoff,
                  const double* rec, double* picks, cudaStream_t st);
// Gaussian smoothing of a gradient field (smoothgradkern = l, odd): weights on the host,
// then one launch from in to out (distinct buffers); d_w holds gaussian_weights(l, nd).
std::vector<double> gaussian_weights(int l, int dim);
cudaError_t launch_smoothgrad(const GridDesc& g, int l, const double* d_w, const double* in, double* out,
                              cudaStream_t st);

}  // namespace eik
