// Coarse-grid forward solve: the reference's heap-ordered FMM main loop
// (ttFMM_core!, src/EikSolv/eikmainfwd.jl:427-823) restated as the fixed point of the
// order rule of stencil.cuh and solved by rounds of brick visits (brick.cuh).
//
// One cooperative persistent launch serves many problems (the sources of a call, or the
// refined windows around them). Rounds alternate between the two colours of bricks and are
// separated by a grid barrier. Round r goes through the list of its colour; a brick whose
// smallest pending front is at most its problem's threshold is visited by one warp, the
// others stay listed. The threshold of problem p is (smallest pending front of p) + a window
// of delta_p, never moving back, so the rounds sweep the grid in traveltime order. Every
// wait is bounded (global timer), the number of rounds is bounded; both report through an
// error word instead of trapping.
#include <algorithm>

#include "brick.cuh"
#include "kernels.cuh"
#include "rounds.cuh"

namespace eik {

// Warps per CTA, one CTA per SM: as many warps as their shared memory allows in 3D (20.9 KB
// each; 12 of small bricks, at 168 registers a thread), 16 in 2D (7 KB each) where a round seldom
// has more bricks per SM.
template <int ND, bool SMALL>
constexpr int BRICK_WARPS = ND == 3 ? (SMALL ? 12 : 11) : 16;

// ----------------------------------------------------------------------- init --
__device__ __forceinline__ void bricks_init(const BrickState& bs, unsigned nprob, int nodes, int words) {
  const size_t nb = (size_t)bs.stride * nprob, t0 = blockIdx.x * (size_t)blockDim.x + threadIdx.x,
               dt = (size_t)gridDim.x * blockDim.x;
  const double2 inf2 = make_double2(EIK_INF, EIK_INF);
  for (size_t q = t0; q < nb * nodes / 2; q += dt) reinterpret_cast<double2*>(bs.t)[q] = inf2;
  const unsigned none = CODE_NONE * 0x01010101u;
  for (size_t q = t0; q < nb * nodes / 16; q += dt)
    reinterpret_cast<uint4*>(bs.code)[q] = make_uint4(none, none, none, none);
  for (size_t q = t0; q < nb * words; q += dt) bs.mask[q] = 0u;
  for (size_t q = t0; q < nb; q += dt) {
    bs.front[q] = PF_NONE;
    bs.listed[q] = 0u;
  }
  for (size_t q = t0; q < 4 * (size_t)nprob; q += dt) {
    bs.exam[q] = PF_NONE;
    bs.marks[q] = PF_NONE;
  }
  for (size_t q = t0; q < 2 * (size_t)nprob; q += dt) bs.thr[q] = 0.0f;
  if (t0 < 8) bs.ctr[t0] = 0u;
}
__global__ void bricks_init_kernel(BrickState bs, unsigned nprob, int nodes, int words) {
  bricks_init(bs, nprob, nodes, words);
}

__global__ void solve_counters_kernel(SolveArgs a) {
  if (threadIdx.x != 0) return;
  a.rs.bar[0] = 0;
  a.rs.bar[1] = 0;
  *a.rs.rounds = 0;
  for (int k = 0; k < 7; k++) a.rs.visits[k] = 0;
  *a.activations = 0;
  *a.node_evals = 0;
  *a.abort_flag = 0;
}

// Seeds: fixed traveltimes of the source points (coarse source box, coarse-coincident
// accepted fine nodes, or the source box of a refined window); the nodes within two steps
// of a seed are pending at the start, with the seed's traveltime as their front.
struct SeedArgs {
  const int32_t* lin;  // nprob x cap
  const double* tt;
  const SrcOut* out;
  int32_t fine_corners, cap;
};
// Problem s by one CTA.
template <int ND, bool SMALL>
__device__ __forceinline__ void seed_problem(const SolveArgs& a, const SeedArgs& sd, int s) {
  typedef Brick<ND, SMALL> B;
  const int32_t* seed_lin = sd.lin;
  const double* seed_tt = sd.tt;
  const int seedcap = sd.cap;
  const CoarseProblem& P = a.probs[s];
  const BrickState& bs = a.bs;
  const int ns = sd.fine_corners ? sd.out[s].nsrcf : sd.out[s].nseeds;
  const size_t base = (size_t)s * bs.stride;
  for (int q = threadIdx.x; q < ns; q += blockDim.x) {
    const long long l = seed_lin[(size_t)s * seedcap + q];
    int c[3];
    node_coords(P.g, l, c);
    bs.t[base * B::NODES + brick_node<ND, SMALL>(P.g, c[0], c[1], c[2])] = -fabs(seed_tt[(size_t)s * seedcap + q]);
    P.kL[l] = -EIK_INF;
    P.kd[l] = 0;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < ns; q += blockDim.x) {
    int c[3];
    node_coords(P.g, seed_lin[(size_t)s * seedcap + q], c);
    const unsigned f = front_bits(fabs(seed_tt[(size_t)s * seedcap + q]));
    if (f == PF_NONE) continue;
    for (int ax = 0; ax < ND; ax++)
      for (int d = -2; d <= 2; d++) {
        if (d == 0) continue;
        int p[3] = {c[0], c[1], c[2]};
        p[ax] += d;
        if (p[ax] < 0 || p[ax] >= P.g.n[ax]) continue;
        const long long bn = brick_node<ND, SMALL>(P.g, p[0], p[1], p[2]);
        const size_t b = base + bn / B::NODES;
        const int qn = (int)(bn % B::NODES);
        atomicOr(bs.mask + b * B::WORDS + (qn >> 5), 1u << (qn & 31));
        atomicMin(bs.front + b, f);
        // pending of both colours: the visits of round 0 and (exam of round -1) of round 1
        atomicMin(bs.marks + 3 * (size_t)a.nprob + s, f);
        atomicMin(bs.exam + 3 * (size_t)a.nprob + s, f);
        if (atomicExch(bs.listed + b, 1u) == 0u) {
          const int col = (p[0] / B::BX + p[1] / B::BY + (ND == 3 ? p[2] / B::BZ : 0)) & 1;
          bs.lists[(size_t)(2 * col) * bs.listcap + atomicAdd(bs.ctr + 2 * col, 1u)] = (unsigned)b;
        }
      }
  }
}

template <int ND, bool SMALL>
__global__ void seed_kernel(SolveArgs a, SeedArgs sd) {
  seed_problem<ND, SMALL>(a, sd, blockIdx.x);
}

// Results in the problems' own arrays: column-major traveltimes, and codes with bit 7 for a
// special key. Problem p by the threads t0, t0 + dt, ...
template <int ND, bool SMALL>
__device__ __forceinline__ void store_problem(const SolveArgs& a, int p, unsigned t0, unsigned dt) {
  typedef Brick<ND, SMALL> B;
  const CoarseProblem& P = a.probs[p];
  const GridDesc& g = P.g;
  const size_t base = (size_t)p * a.bs.stride * B::NODES;
  const unsigned long long N = (unsigned long long)npts(g);
  for (unsigned long long l = t0; l < N; l += dt) {
    int c[3];
    node_coords(g, (long long)l, c);
    const size_t q = base + brick_node<ND, SMALL>(g, c[0], c[1], c[2]);
    const double t = __ldcg(a.bs.t + q);
    P.t[l] = fabs(t);
    P.code[l] = (uint8_t)((__ldcg(a.bs.code + q) & 0x7f) | (sign_set(t) ? CODE_SRC_BIT : 0));
  }
}

// ---------------------------------------------------------------------- solve --
__device__ __forceinline__ unsigned ld_vol(const unsigned* p) { return *(volatile const unsigned*)p; }

// Threshold of problem p in round r: a window above its smallest pending front, which is the
// smallest of what the last round's visits left, what the round before left on the other
// colour, and what the last round put on other bricks. All three are complete when round r
// starts and change again only after it.
__device__ __forceinline__ float round_threshold(const BrickState& bs, int nprob, int p, int r, double delta) {
  const unsigned* e1 = bs.exam + (size_t)((r + 3) & 3) * nprob;
  const unsigned* e2 = bs.exam + (size_t)((r + 2) & 3) * nprob;
  const unsigned* mk = bs.marks + (size_t)((r + 3) & 3) * nprob;
  const float prev = __ldcg(bs.thr + (size_t)((r + 1) & 1) * nprob + p);
  const unsigned m = min(min(__ldcg(e1 + p), __ldcg(e2 + p)), __ldcg(mk + p));
  if (m == PF_NONE) return prev;
  return fmaxf(prev, fminf(__double2float_ru((double)__uint_as_float(m) + delta), 3.402823466e38f));
}

// FUSED: the reset, the seeds and the store are part of the launch (small solves, where each
// launch of its own costs as much as its work).
template <int ND, bool SMALL, bool FUSED>
__global__ void __launch_bounds__(BRICK_WARPS<ND, SMALL> * 32, 1) brick_rounds_kernel(SolveArgs a, SeedArgs sd) {
  typedef Brick<ND, SMALL> B;
  extern __shared__ __align__(16) unsigned char brick_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  WarpMem<ND, SMALL>& w = reinterpret_cast<WarpMem<ND, SMALL>*>(brick_smem)[warp];
  const BrickState bs = a.bs;
  const unsigned nwarps = gridDim.x * BRICK_WARPS<ND, SMALL>;
  // consecutive entries go to different SMs
  const unsigned gwarp = (unsigned)warp * gridDim.x + blockIdx.x;
  VisitTally tally;
  if (FUSED) {
    bricks_init(bs, (unsigned)a.nprob, B::NODES, B::WORDS);
    if (!grid_barrier(a)) return;
    for (int s = blockIdx.x; s < a.nprob; s += gridDim.x) {
      seed_problem<ND, SMALL>(a, sd, s);
      __syncthreads();
    }
    if (!grid_barrier(a)) return;
  }
  int r = 0;
  for (; r < a.rs.max_rounds; r++) {
    const int col = r & 1, ph = (r >> 1) & 1, nph = ph ^ 1, oph = ((r + 1) >> 1) & 1;
    const unsigned n = ld_vol(bs.ctr + 2 * col + ph);
    if (n == 0 && ld_vol(bs.ctr + 2 * (col ^ 1) + oph) == 0) break;  // no entry of either colour
    unsigned* grab = bs.ctr + 4 + r % 3;
    if (blockIdx.x == 0)
      for (int p = threadIdx.x; p < a.nprob; p += blockDim.x)
        bs.thr[(size_t)(r & 1) * a.nprob + p] = round_threshold(bs, a.nprob, p, r, a.probs[p].delta);
    const unsigned* L = bs.lists + (size_t)(2 * col + ph) * bs.listcap;
    unsigned* Lkeep = bs.lists + (size_t)(2 * col + nph) * bs.listcap;
    unsigned* Lother = bs.lists + (size_t)(2 * (col ^ 1) + oph) * bs.listcap;
    // entries a warp takes at a time: one while a round has few, so that every warp gets some
    const unsigned take = max(1u, min(8u, n / (4u * nwarps)));
    unsigned base = gwarp * take;
    while (base < n) {
      unsigned b = 0;
      unsigned f = PF_NONE;
      float T = 0.0f;
      int prob = 0;
      const bool have = lane < take && base + lane < n;
      if (have) {
        b = __ldcg(L + base + lane);
        f = __ldcg(bs.front + b);
        prob = (int)(b / bs.stride);
        T = round_threshold(bs, a.nprob, prob, r, a.probs[prob].delta);
      }
      const bool go = have && f <= __float_as_uint(T);
      unsigned todo = __ballot_sync(FULL_WARP, go);
      unsigned leftf = PF_NONE;  // per entry: smallest front still pending after this round
      if (have && !go) leftf = f;
      while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const unsigned vb = __shfl_sync(FULL_WARP, b, src);
        const int vp = __shfl_sync(FULL_WARP, prob, src);
        const float vT = __shfl_sync(FULL_WARP, T, src);
        const CoarseProblem& P = a.probs[vp];
        const unsigned lb = vb - (unsigned)vp * bs.stride;
        const int nb[3] = {bricks_along<ND, SMALL>(P.g, 0), bricks_along<ND, SMALL>(P.g, 1),
                           ND == 3 ? bricks_along<ND, SMALL>(P.g, 2) : 1};
        const int bc[3] = {(int)(lb % nb[0]), (int)((lb / nb[0]) % nb[1]), (int)(lb / ((unsigned)nb[0] * nb[1]))};
        const unsigned left = visit_brick<ND, SMALL>(w, bs, P, vb, bc, nb, vT, lane, tally);
        if (lane == src) leftf = left;
        if (lane == 0) {
          bs.front[vb] = left;
          if (left == PF_NONE) bs.listed[vb] = 0u;
        }
        // the bricks across the faces: pending bits, front, and a place in the other colour's list
        __syncwarp();
#pragma unroll
        for (int q0 = 0; q0 < B::FACES * B::WORDS; q0 += 32) {
          const int q = q0 + lane;
          const unsigned bits = q < B::FACES * B::WORDS ? w.face[q] : 0u;
          if (bits) {
            const int fc = q / B::WORDS, ax = fc >> 1;
            const int st = ax == 0 ? 1 : (ax == 1 ? nb[0] : nb[0] * nb[1]);
            const unsigned ob = (fc & 1) ? vb - st : vb + st;
            atomicOr(bs.mask + (size_t)ob * B::WORDS + q % B::WORDS, bits);
          }
        }
        if (lane < B::FACES && w.facemin[lane] != PF_NONE) {
          const int ax = lane >> 1;
          const int st = ax == 0 ? 1 : (ax == 1 ? nb[0] : nb[0] * nb[1]);
          const unsigned ob = (lane & 1) ? vb - st : vb + st;
          const unsigned fm = w.facemin[lane];
          atomicMin(bs.front + ob, fm);
          atomicMin(bs.marks + (size_t)(r & 3) * a.nprob + vp, fm);
          if (atomicExch(bs.listed + ob, 1u) == 0u)
            Lother[atomicAdd(bs.ctr + 2 * (col ^ 1) + oph, 1u)] = ob;
        }
        __syncwarp();
      }
      // entries with something pending stay listed for their colour's next round
      const bool keep = have && leftf != PF_NONE;
      const unsigned km = __ballot_sync(FULL_WARP, keep);
      if (km) {
        unsigned at = 0;
        if (lane == __ffs(km) - 1) at = atomicAdd(bs.ctr + 2 * col + nph, (unsigned)__popc(km));
        at = __shfl_sync(FULL_WARP, at, __ffs(km) - 1);
        if (keep) {
          Lkeep[at + __popc(km & ((1u << lane) - 1u))] = b;
          atomicMin(bs.exam + (size_t)(r & 3) * a.nprob + prob, leftf);
        }
      }
      if (lane == 0) base = nwarps * take + atomicAdd(grab, take);
      base = __shfl_sync(FULL_WARP, base, 0);
    }
    // buffers that round r + 1 appends to or accumulates in (last read in round r - 1)
    if (blockIdx.x == 0) {
      if (threadIdx.x == 0) {
        bs.ctr[2 * (col ^ 1) + (oph ^ 1)] = 0u;
        bs.ctr[4 + (r + 2) % 3] = 0u;
      }
      for (int p = threadIdx.x; p < a.nprob; p += blockDim.x) {
        bs.exam[(size_t)((r + 1) & 3) * a.nprob + p] = PF_NONE;
        bs.marks[(size_t)((r + 1) & 3) * a.nprob + p] = PF_NONE;
      }
    }
    if (!grid_barrier(a)) break;
  }
  if (lane < 7 && tally.n) {
    atomicAdd(a.rs.visits + lane, (unsigned long long)tally.n);
    atomicAdd(a.activations, (unsigned long long)tally.n);
  }
  const unsigned evals = __shfl_sync(FULL_WARP, tally.n, VISIT_WAIT) + __shfl_sync(FULL_WARP, tally.n, VISIT_SAME) +
                         __shfl_sync(FULL_WARP, tally.n, VISIT_CHANGED);
  if (lane == 0 && evals) atomicAdd(a.node_evals, (unsigned long long)evals);
  // every visit ended before the barrier that closed the last round
  if (FUSED)
    for (int p = 0; p < a.nprob; p++)
      store_problem<ND, SMALL>(a, p, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *a.rs.rounds = r;
    if (r >= a.rs.max_rounds) {
      atomicOr(a.err, ERRB_NOT_CONVERGED);
      atomicExch(a.abort_flag, 1);
    }
  }
}

template <int ND, bool SMALL>
__global__ void bricks_store_kernel(SolveArgs a) {
  for (int p = blockIdx.y; p < a.nprob; p += gridDim.y)
    store_problem<ND, SMALL>(a, p, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// ------------------------------------------------------------------ picks --
// bilinear_interp / trilinear_interp value mode (eikforward2D.jl:17-87,
// eikforward3D.jl:17-140), corner (i+1,j,k+1) weighted xd*(1-yd)*(1-zd) as the reference.
__global__ void picks_kernel(GridDesc g, const double* t, long long N, int nsrc, const long long* recoff,
                             const double* rec, double* picks) {
  const long long ntot = recoff[nsrc];
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < ntot;
       r += (long long)gridDim.x * blockDim.x) {
    int s = 0;
    while (recoff[s + 1] <= r) s++;
    const double* tt = t + (size_t)s * N;
    const double* p = rec + r * g.nd;
    if (g.nd == 2) {
      const double xh = (p[0] - g.co[0]) / g.spac[0];
      const double yh = (p[1] - g.co[1]) / g.spac[1];
      long long i = (long long)floor(xh + 1), j = (long long)floor(yh + 1);
      if (i == g.n[0]) i -= 1;
      else if (i > g.n[0]) i -= 2;
      if (j == g.n[1]) j -= 1;
      else if (j > g.n[1]) j -= 2;
      const double xd = xh - (double)(i - 1), yd = yh - (double)(j - 1);
      const long long a = lin3(g, (int)i - 1, (int)j - 1, 0);
      const double f00 = tt[a], f10 = tt[a + 1], f01 = tt[a + g.n[0]], f11 = tt[a + g.n[0] + 1];
      picks[r] = f00 * (1.0 - xd) * (1.0 - yd) + f10 * (1.0 - yd) * xd + f01 * (1.0 - xd) * yd + f11 * xd * yd;
    } else {
      const double dx = g.spac[0], dy = g.spac[1], dz = g.spac[2];
      const double xh = (p[0] - g.co[0]) / dx, yh = (p[1] - g.co[1]) / dy, zh = (p[2] - g.co[2]) / dz;
      const double x = p[0] - g.co[0], y = p[1] - g.co[1], z = p[2] - g.co[2];
      long long i = (long long)floor(xh + 1), j = (long long)floor(yh + 1), k = (long long)floor(zh + 1);
      if (i == g.n[0]) i -= 1;
      else if (i > g.n[0]) i -= 2;
      if (j == g.n[1]) j -= 1;
      else if (j > g.n[1]) j -= 2;
      if (k == g.n[2]) k -= 1;
      else if (k > g.n[2]) k -= 2;
      const double x0 = (double)(i - 1) * dx, y0 = (double)(j - 1) * dy, z0 = (double)(k - 1) * dz;
      const double x1 = (double)i * dx, y1 = (double)j * dy, z1 = (double)k * dz;
      const double xd = (x - x0) / (x1 - x0), yd = (y - y0) / (y1 - y0), zd = (z - z0) / (z1 - z0);
      auto T = [&](int a, int b, int c) { return tt[lin3(g, (int)i - 1 + a, (int)j - 1 + b, (int)k - 1 + c)]; };
      picks[r] = T(0, 0, 0) * (1 - xd) * (1 - yd) * (1 - zd) + T(1, 0, 0) * xd * (1 - yd) * (1 - zd) +
                 T(0, 1, 0) * (1 - xd) * yd * (1 - zd) + T(0, 0, 1) * (1 - xd) * (1 - yd) * zd +
                 T(1, 1, 0) * xd * yd * (1 - zd) + T(0, 1, 1) * (1 - xd) * yd * zd +
                 T(1, 0, 1) * xd * (1 - yd) * (1 - zd) + T(1, 1, 1) * xd * yd * zd;
    }
  }
}

// ------------------------------------------------------------------ launchers --
int brick_size(int nd, bool small) {
  return nd == 3 ? (small ? Brick<3, true>::NODES : Brick<3, false>::NODES)
                 : (small ? Brick<2, true>::NODES : Brick<2, false>::NODES);
}
unsigned long long brick_number(const GridDesc& g, bool small) {
  if (g.nd == 3) return (unsigned long long)(small ? brick_count<3, true>(g) : brick_count<3, false>(g));
  return (unsigned long long)(small ? brick_count<2, true>(g) : brick_count<2, false>(g));
}

void launch_bricks_init(const SolveArgs& sa, cudaStream_t st) {
  solve_counters_kernel<<<1, 32, 0, st>>>(sa);
  const int nodes = brick_size(sa.nd, sa.bs.small);
  bricks_init_kernel<<<1184, 256, 0, st>>>(sa.bs, (unsigned)sa.nprob, nodes, nodes / 32);
}

void launch_bricks_seed(const SolveArgs& sa, const int32_t* seed_lin, const double* seed_tt, const SrcOut* out,
                        bool fine_corners, int seedcap, cudaStream_t st) {
  const SeedArgs sd{seed_lin, seed_tt, out, fine_corners ? 1 : 0, seedcap};
  auto go = [&](auto kernel) { kernel<<<sa.nprob, 128, 0, st>>>(sa, sd); };
  if (sa.nd == 3) sa.bs.small ? go(seed_kernel<3, true>) : go(seed_kernel<3, false>);
  else sa.bs.small ? go(seed_kernel<2, true>) : go(seed_kernel<2, false>);
}

template <int ND, bool SMALL, bool FUSED>
static cudaError_t launch_bricks_solve_nd(const SolveArgs& sa, const SeedArgs& sd, int nsm, cudaStream_t st) {
  const void* kernel = (const void*)brick_rounds_kernel<ND, SMALL, FUSED>;
  const size_t sm = sizeof(WarpMem<ND, SMALL>) * BRICK_WARPS<ND, SMALL>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e != cudaSuccess) return e;
  SolveArgs args = sa;
  SeedArgs seeds = sd;
  void* kargs[] = {&args, &seeds};
  // cooperative: every CTA is resident, so the grid barrier between rounds cannot deadlock
  return cudaLaunchCooperativeKernel(kernel, dim3(nsm), dim3(BRICK_WARPS<ND, SMALL> * 32), kargs, sm, st);
}

template <bool FUSED>
static cudaError_t launch_bricks_any(const SolveArgs& sa, const SeedArgs& sd, int nsm, cudaStream_t st) {
  if (sa.nd == 3)
    return sa.bs.small ? launch_bricks_solve_nd<3, true, FUSED>(sa, sd, nsm, st)
                       : launch_bricks_solve_nd<3, false, FUSED>(sa, sd, nsm, st);
  return sa.bs.small ? launch_bricks_solve_nd<2, true, FUSED>(sa, sd, nsm, st)
                     : launch_bricks_solve_nd<2, false, FUSED>(sa, sd, nsm, st);
}

cudaError_t launch_bricks_solve(const SolveArgs& sa, int nsm, cudaStream_t st) {
  return launch_bricks_any<false>(sa, SeedArgs{}, nsm, st);
}

cudaError_t launch_bricks_fused(const SolveArgs& sa, const int32_t* seed_lin, const double* seed_tt, const SrcOut* out,
                                bool fine_corners, int seedcap, int nsm, cudaStream_t st) {
  solve_counters_kernel<<<1, 32, 0, st>>>(sa);
  return launch_bricks_any<true>(sa, SeedArgs{seed_lin, seed_tt, out, fine_corners ? 1 : 0, seedcap}, nsm, st);
}

void launch_bricks_store(const SolveArgs& sa, cudaStream_t st) {
  // blocks per problem: enough in all to fill the GPU, no more than a problem has nodes for
  const unsigned long long nodes = (unsigned long long)sa.bs.stride * brick_size(sa.nd, sa.bs.small);
  const unsigned want = (unsigned)((nodes + 1023) / 1024);
  const unsigned per = std::max(1u, std::min(want, std::max(8u, 2368u / (unsigned)sa.nprob)));
  const dim3 grid(per, std::min(65535u, (unsigned)sa.nprob));
  auto go = [&](auto kernel) { kernel<<<grid, 256, 0, st>>>(sa); };
  if (sa.nd == 3) sa.bs.small ? go(bricks_store_kernel<3, true>) : go(bricks_store_kernel<3, false>);
  else sa.bs.small ? go(bricks_store_kernel<2, true>) : go(bricks_store_kernel<2, false>);
}

void launch_picks(const GridDesc& g, const double* t, long long N, int nsrc, const long long* recoff,
                  const double* rec, double* picks, cudaStream_t st) {
  picks_kernel<<<64, 128, 0, st>>>(g, t, N, nsrc, recoff, rec, picks);
}

}  // namespace eik
