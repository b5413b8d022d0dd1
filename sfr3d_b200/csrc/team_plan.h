// Host side of the batched team launches (team_sync.cuh): their shape, the
// plan batched.cu makes, and the graph that runs the rounds.
#pragma once

#include "internal.h"
#include "team_sync.cuh"

namespace sfr {

// How a team kernel is launched on a device; blocks 0 where it cannot be.
struct TeamShape {
  int per_sm = 0, threads = 0, blocks = 0;  // blocks an SM, threads a block, blocks in all
  size_t smem = 0;                          // dynamic shared memory a block
  int most = 0;                             // slices a block can take
  TeamModel model{};
};

struct TeamPlan {
  TeamShape shape;
  TeamTable table{};
  const int4 *systems = nullptr;  // RoundTable::sys
  int nsys = 0, grid = 0;
  float us = 0.f, us_later = 0.f;  // RoundTable's
};

// The shape of `kern` with `per_sm` blocks of `threads` an SM, of which a
// slice takes slice_bytes at least; far: for unnumbered systems (DevSell::far).
TeamShape team_shape(int device, const void *kern, int threads, int per_sm, int slice_bytes,
                     const TeamModel &model, bool far);

// done_iters: kRoundInts * plan.nsys ints, zero at first; ctl: 16 words.
constexpr int kRoundInts = 3;
inline RoundTable round_table(const TeamPlan &plan, int *done_iters, unsigned *ctl) {
  RoundTable rt{};
  rt.sys = plan.systems;
  rt.done = done_iters;
  rt.iters = done_iters + plan.nsys;
  rt.nsys = plan.nsys;
  rt.most = plan.shape.most;
  rt.model = plan.shape.model;
  rt.us = plan.us;
  rt.us_later = plan.us_later;
  rt.ctl = ctl + 4;
  rt.err = reinterpret_cast<int *>(ctl + 2);
  return rt;
}

// The graph [zero `zero` and the 64 bytes at ctl -> WHILE { kern }]: kern a
// cooperative kernel that clears the condition *more, one of the values
// params point to, when no round is left.
int rounds_graph(const void *kern, const TeamPlan &plan, void **params,
                 cudaGraphConditionalHandle *more, void *zero, size_t zero_bytes, unsigned *ctl,
                 cudaGraph_t *graph);

// FP64 PCG (onchip.cu) and mixed PCG (mixed_team.cu).
TeamShape team_shape_onchip(const sfr_system *s, int per_sm);
size_t team_ws_bytes_onchip(int n, int grid, int nsys);
int graph_team_onchip(sfr_system *s, const double *d_b, double *d_x, double tol, uint32_t maxit,
                      int32_t newx, const TeamPlan &plan, void *ws, SolveOut *d_out,
                      unsigned *ctl, cudaGraph_t *graph);
TeamShape team_shape_mixed(const sfr_system *s, int per_sm);
size_t team_ws_bytes_mixed_team(int n, int grid, int nsys);
int graph_mixed_team(sfr_system *s, const double *d_b, double *d_x, double tol, uint32_t maxit,
                     int32_t newx, const TeamPlan &plan, void *ws, SolveOut *d_out, unsigned *ctl,
                     cudaGraph_t *graph);

}  // namespace sfr
