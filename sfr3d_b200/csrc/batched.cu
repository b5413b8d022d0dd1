// Batched solves: many independent systems of uneven size in one graph launch.
//
// The systems are concatenated into one block-diagonal SELL-32 matrix, each
// system's rows padded to whole slices so that no slice straddles two
// systems.  Each system gets a team of blocks: its own slice range, sums over
// its own blocks and its own bounded waits, so every system iterates at its own
// pace and stops at its own convergence.
//
// PCG runs on the on-chip engine's teams (onchip.cu, mixed_team.cu) where they
// hold the batch, in rounds: the kernel is the body of a graph's WHILE node,
// and each round shares the blocks out anew over the systems left by a model of
// a team's time (team_sync.cuh).  The rest, BiCGSTAB among it, is one persistent
// cooperative launch with a barrier a team (persist.cuh), whose blocks are
// shared out in proportion to each system's work per solve.  The autotuner
// measures the work for both.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <memory>
#include <string>
#include <utility>
#include <vector>

#include "common.cuh"
#include "internal.h"
#include "persist.cuh"
#include "team_plan.h"

struct sfr_batch {
  int32_t device = 0;
  int32_t nsys = 0;
  int32_t storage = 0;
  int32_t unsym = 0;
  std::vector<int32_t> n, row_off, slice_off, nslices, src_off, nsrc;
  sfr_system cat;               // the block-diagonal concatenation
  std::vector<double> weight;   // work per solve: slices x iterations
  std::vector<int> team_blocks; // blocks per team chosen by the autotuner (empty: by weight)
  std::vector<int> blocks_of;   // blocks per team of the installed plan
  std::vector<double> team_ms;  // each team's time in the last solve (ms)
  sfr_batch_tune tune{};        // the last autotune's report
  // launch plan
  int32_t plan_solver = -1, plan_precision = -1, grid = 0;
  int engine = 0;  // of the plan (Engine below)
  sfr::TeamShape shape;  // on chip: how its kernel is launched
  float round_us = 0.f, round_us_later = 0.f;  // on chip: the rounds' times
  sfr::TeamTable table{};
  int4 *d_block = nullptr;
  int2 *d_sys = nullptr;
  int4 *d_systems = nullptr;  // per system {first slice, slices, end row, estimated iterations}
  unsigned *d_bar = nullptr;
  void *ws = nullptr;
  size_t ws_bytes = 0;
  sfr::SolveOut *d_out = nullptr;
  unsigned *d_ctl = nullptr;
  double *d_b = nullptr, *d_x = nullptr;
  // the captured launch and the scalars baked into it
  cudaGraphExec_t exec = nullptr;
  double g_tol = -1.0;
  uint32_t g_maxit = 0;
  int32_t g_newx = -1;
};

namespace sfr {
namespace {

// Blocks per team from the work weights: in proportion, at least one and at
// most one block per slice of the system, all fitting in `gmax`.
std::vector<int> share_by_weight(const sfr_batch *b, int gmax) {
  const int S = b->nsys;
  double wsum = 0.0;
  for (double w : b->weight) wsum += w;
  std::vector<int> nb(S);
  std::vector<double> raw(S);
  int total = 0;
  for (int s = 0; s < S; ++s) {
    raw[s] = gmax * b->weight[s] / wsum;
    nb[s] = std::max(1, std::min(static_cast<int>(raw[s]), b->nslices[s]));
    total += nb[s];
  }
  while (total > gmax) {  // trim the largest teams
    int big = 0;
    for (int s = 1; s < S; ++s)
      if (nb[s] > nb[big]) big = s;
    if (nb[big] <= 1) break;
    --nb[big];
    --total;
  }
  while (total < gmax) {  // hand leftovers to the most under-served teams
    int best = -1;
    double deficit = 0.0;
    for (int s = 0; s < S; ++s) {
      if (nb[s] >= b->nslices[s]) continue;
      const double d = raw[s] - nb[s];
      if (best < 0 || d > deficit) {
        best = s;
        deficit = d;
      }
    }
    if (best < 0 || deficit <= 0.0) break;
    ++nb[best];
    ++total;
  }
  return nb;
}

// The SM's shared memory that a batch of unnumbered systems uses at most: the
// carve-out that leaves 92 KB of L1, where the lines of its scattered gathers
// in flight live.  With all 228 KB, with 196, 164 and 132, ms a solve, mixed and
// FP64: 3 boxes of 90^3 in random order 147, 83, 71, 68 and 130, 76, 68, 65; 8 of
// 48^3 27.9, 17.7, 15.7, 15.4 and 24.8, 14.9, 13.4, 15.7; one of 110^3 80, 60,
// 52, 54 and 88, 58, 54, 52 (the persistent kernels: 112 and 128, 28.1 and 28.6,
// 82 and 96).
constexpr int kFarSmem = 164 << 10;
// ... and the carve-out above, for teams that hold enough in it (plan).
constexpr int kHoldSmem = 196 << 10;

// A block's dynamic shared memory where the SM's is `sm` bytes: less the team
// kernels' static shared memory and the 1 KB the system takes of each block.
size_t team_smem(int sm, int per_sm) {
  constexpr int kStatic = (sizeof(TeamShared) + 255) / 256 * 256;
  return static_cast<size_t>(std::max(0, sm / per_sm - 1024 - kStatic));
}

// What runs a batch: the on-chip teams (PCG: onchip.cu in FP64, mixed_team.cu
// in mixed precision) where every system has room there, else the persistent
// kernels.
enum Engine { kPersistent, kChipFp64, kChipMixed };

// Blocks a system's team needs at least: as many as hold its rows.
std::vector<int> least_blocks(const sfr_batch *b, const TeamShape &sh) {
  std::vector<int> nb(b->nsys, 1);
  if (sh.most > 0)
    for (int s = 0; s < b->nsys; ++s) nb[s] = std::max(1, (b->nslices[s] + sh.most - 1) / sh.most);
  return nb;
}

// Shared memory of a slice with all of its rows' vectors and its slots.
int64_t slice_bytes(const sfr_batch *b, int row, int value) {
  const int64_t slots = b->cat.A.max_width;
  return kWarpHost * (row + slots * (value + (b->cat.A.off ? 2 : 4))) + 4;
}

// Slices of which a block of the mixed teams' has room for `vecs` FP32 vectors
// and the slice pointers.
int mixed_slices(const TeamShape &sh, int vecs) {
  return (static_cast<int>(sh.smem) - 32) / (kWarpHost * 4 * vecs + 4);
}

// Mixed batches too large for the teams to hold q and r in shared memory stay
// with the persistent kernels, whose more warps stream the rest better: 3 boxes
// of 112^3 (131,712 slices) 130 ms and 142 on teams, 4 177 and 195, 6 of 96^3
// 145 and 160, 8 of 62 to 115 cells 170 and 184; 4 of 96^3 (110,592, q and r
// held) 92 and 79.
//
// One block an SM while the systems are at most half as many (96^3 alone:
// 14.6 us an iteration against 17.5 with two blocks an SM; 64 mixed boxes of
// 8 to 96 cells 66 ms against 67), else two: twice the teams, finer shares.
Engine pick_engine(const sfr_batch *b, int32_t solver, int32_t precision, TeamShape *shape) {
  *shape = TeamShape{};
  if (solver != SFR_PCG) return kPersistent;
  const Engine e = precision == SFR_MIXED ? kChipMixed : kChipFp64;
  for (int per_sm : {1, 2}) {
    const TeamShape sh = e == kChipMixed ? team_shape_mixed(&b->cat, per_sm)
                                         : team_shape_onchip(&b->cat, per_sm);
    if (per_sm == 1 && 2 * b->nsys > num_sms(b->device)) continue;
    int64_t total = 0;
    for (int v : least_blocks(b, sh)) total += v;
    if (sh.blocks > 0 && b->nsys <= kMaxTeams && total <= sh.blocks &&
        !(e == kChipMixed && b->cat.A.nslices > sh.blocks * mixed_slices(sh, 2))) {
      *shape = sh;
      return e;
    }
  }
  return kPersistent;
}

int max_grid(const sfr_batch *b, int32_t solver, int32_t precision) {
  TeamShape sh;
  if (pick_engine(b, solver, precision, &sh) != kPersistent) return sh.blocks;
  return precision == SFR_MIXED ? team_max_grid_mixed(solver, b->device)
                                : team_max_grid_fp64(solver, b->device);
}

// Iterations a system is expected to take: its weight a slice, scaled so that
// the largest estimate is the default's for that system (weights are relative).
std::vector<double> estimates(const sfr_batch *b) {
  std::vector<double> it(b->nsys);
  int big = 0;
  for (int s = 0; s < b->nsys; ++s) {
    it[s] = b->weight[s] / b->nslices[s];
    if (it[s] > it[big]) big = s;
  }
  const double scale = 15.0 * std::cbrt(static_cast<double>(b->n[big])) / it[big];
  for (double &v : it) v = std::max(1.0, v * scale);
  return it;
}

// Blocks per team of an on-chip launch's first round: the shares that
// minimise the slowest team's predicted time, as next_teams does on the
// device for the later rounds.
std::vector<int> share_by_model(const sfr_batch *b, const TeamShape &sh) {
  const int S = b->nsys;
  const std::vector<int> least = least_blocks(b, sh);
  const std::vector<double> it = estimates(b);
  auto time = [&](int s, int B) { return it[s] * sh.model.us(b->nslices[s], B); };
  auto need = [&](int s, double T) {  // the fewest blocks within T
    if (time(s, least[s]) <= T) return least[s];
    const double rest = T / it[s] - sh.model.many;
    if (rest <= 0.0) return INT32_MAX;
    const double B = std::max(std::max(least[s], 2) + 0.0,
                              std::ceil(sh.model.slice * b->nslices[s] / rest - 1e-9));
    return B > b->nslices[s] ? INT32_MAX : static_cast<int>(B);
  };
  auto fits = [&](double T) {
    int64_t total = 0;
    for (int s = 0; s < S && total <= sh.blocks; ++s) total += need(s, T);
    return total <= sh.blocks;
  };
  double hi = 0.0, lo = 0.0;
  for (int s = 0; s < S; ++s) hi = std::max(hi, time(s, least[s]));
  for (int i = 0; i < 60; ++i) {
    const double mid = 0.5 * (lo + hi);
    (fits(mid) ? hi : lo) = mid;
  }
  std::vector<int> nb(S);
  int total = 0;
  for (int s = 0; s < S; ++s) total += nb[s] = need(s, hi);
  while (total < sh.blocks) {  // leftovers to the teams predicted slowest
    int worst = -1;
    for (int s = 0; s < S; ++s)
      if (nb[s] < b->nslices[s] && time(s, nb[s] + 1) < time(s, nb[s]) &&
          (worst < 0 || time(s, nb[s]) > time(worst, nb[worst])))
        worst = s;
    if (worst < 0) break;
    ++nb[worst];
    ++total;
  }
  return nb;
}

// The time of an on-chip launch's first round, in us, of teams predicted to
// take t[s] us on nb[s] blocks.  Up to `share` of the slowest team's; less where
// a quarter of the blocks are predicted idle before, a quarter past that time
// (predictions are rough), so that the next round gives those blocks to the
// teams still at work: 112^3 beside 63 boxes of 8^3, which hold 43 % of the
// blocks for 0.3 ms, 31 ms mixed (share alone 44 to 62, the persistent kernels
// 44) and 29 FP64 (50, 99); 200 boxes of 4 to 40 cells 12.3 and 10.3 (16.2 and
// 16.6).  An eighth costs batches of small boxes 4 to 7 %.
double first_round(const std::vector<double> &t, const std::vector<int> &nb, double share) {
  const int S = static_cast<int>(nb.size());
  std::vector<int> order(S);
  int64_t grid = 0, idle = 0;
  double longest = 0.0;
  for (int s = 0; s < S; ++s) {
    order[s] = s;
    grid += nb[s];
    longest = std::max(longest, t[s]);
  }
  std::sort(order.begin(), order.end(), [&](int a, int b) { return t[a] < t[b]; });
  for (int s : order)
    if (4 * (idle += nb[s]) >= grid) return std::min(share * longest, 1.25 * t[s]);
  return share * longest;
}

// Install a launch plan: team s gets nb[s] blocks (b->team_blocks when set
// by the autotuner, else shares of the work weights).
int plan(sfr_batch *b, int32_t solver, int32_t precision) {
  const int gmax = max_grid(b, solver, precision);
  if (gmax <= 0) return SFR_CUDA_ERROR;
  if (b->nsys > gmax) {
    set_last_error("more systems than co-resident blocks in one launch");
    return SFR_UNSUPPORTED;
  }
  const int S = b->nsys;
  TeamShape shape;
  const Engine e = pick_engine(b, solver, precision, &shape);
  b->engine = e;
  auto share = [&] {
    return e == kPersistent ? share_by_weight(b, gmax) : share_by_model(b, shape);
  };
  std::vector<int> nb;
  int total = 0;
  if (static_cast<int>(b->team_blocks.size()) == S) {
    nb = b->team_blocks;
    const std::vector<int> least = least_blocks(b, shape);
    for (int s = 0; s < S; ++s) {
      nb[s] = std::max(least[s], std::min(nb[s], b->nslices[s]));
      total += nb[s];
    }
    if (total > gmax) nb = share();
  } else {
    nb = share();
  }
  total = 0;
  for (int v : nb) total += v;
  b->blocks_of = nb;
  // The carve-out below the largest leaves 60 KB of L1 for 28, where every team
  // holds in it what it holds in all of it, or q, r and xs: 2 boxes of 96^3 42.0
  // -> 39.4 ms (the persistent kernels 37.9), of 80^3 16.8 -> 14.8, 8 of 48^3 9.3
  // -> 8.3.  Teams that lose more lose time: r, 2 boxes of 128^3 144 -> 158; the
  // operator, 148 of 12^3 0.80 -> 1.02, 16 of 32^3 4.5 -> 5.0.
  int widest = 0;  // slices of a block
  for (int s = 0; s < S; ++s) widest = std::max(widest, (b->nslices[s] + nb[s] - 1) / nb[s]);
  if (e == kChipMixed) {
    TeamShape small = shape;
    small.smem = std::min(shape.smem, team_smem(kHoldSmem, shape.per_sm));
    small.most = mixed_slices(small, 1);
    const int64_t whole = slice_bytes(b, 24, 4);
    bool same = widest <= mixed_slices(small, 3);
    for (int s = 0; s < S; ++s) {
      const int64_t need = (b->nslices[s] + nb[s] - 1) / nb[s] * whole + 32;
      same = same && (need <= static_cast<int64_t>(small.smem) ||
                      need > static_cast<int64_t>(shape.smem));
    }
    if (same) shape = small;
  }
  // Unnumbered FP64 teams that hold their operators in the 196 KB carve-out and
  // not in 164: 64 boxes of 12^3 0.51 ms, 0.58 without.
  if (e == kChipFp64 && b->cat.A.far()) {
    const int64_t need = widest * slice_bytes(b, 40, 8) + 32;
    const size_t hold = team_smem(kHoldSmem, shape.per_sm);
    if (need > static_cast<int64_t>(shape.smem) && need <= static_cast<int64_t>(hold))
      shape.smem = hold;
  }
  std::vector<int4> blocks;
  std::vector<int2> sys;
  blocks.reserve(total);
  sys.reserve(total);
  for (int s = 0; s < S; ++s) {
    const int b0 = static_cast<int>(blocks.size());
    const int64_t ns = b->nslices[s];
    for (int j = 0; j < nb[s]; ++j) {
      const int s0 = b->slice_off[s] + static_cast<int>(ns * j / nb[s]);
      const int s1 = b->slice_off[s] + static_cast<int>(ns * (j + 1) / nb[s]);
      blocks.push_back(make_int4(s0, s1, b0, b0 + nb[s]));
      sys.push_back(make_int2(s, b->row_off[s] + b->n[s]));
    }
  }
  const int grid = static_cast<int>(blocks.size());
  const std::vector<double> est = estimates(b);
  std::vector<int4> systems(S);
  std::vector<double> us(S);
  double longest = 0.0;
  for (int s = 0; s < S; ++s) {
    systems[s] = make_int4(b->slice_off[s], b->nslices[s], b->row_off[s] + b->n[s],
                           static_cast<int>(std::min(est[s], 1e9)));
    us[s] = est[s] * shape.model.us(b->nslices[s], nb[s]);
    longest = std::max(longest, us[s]);
  }
  // The first round's time, as a share of what the slowest team is predicted
  // to take, then a quarter a round.  FP64, all of it: 24 small boxes 4.9 ms,
  // half 5.7 (a re-plan costs the small teams more than it gives).  Mixed,
  // half: 64 uneven boxes 72 ms (a quarter 66, all 88, one round 176), small
  // batches 4.5 to 6.5 ms (all 3.5 to 5.6).
  b->round_us = static_cast<float>(first_round(us, nb, e == kChipMixed ? 0.5 : 1.0));
  b->round_us_later = static_cast<float>(0.25 * longest);
  if (cudaMemcpy(b->d_systems, systems.data(), sizeof(int4) * S, cudaMemcpyHostToDevice) !=
      cudaSuccess)
    return SFR_CUDA_ERROR;
  cudaFree(b->d_block);
  cudaFree(b->d_sys);
  b->d_block = nullptr;
  b->d_sys = nullptr;
  if (cudaMalloc(&b->d_block, sizeof(int4) * grid) != cudaSuccess) return SFR_CUDA_ERROR;
  if (cudaMalloc(&b->d_sys, sizeof(int2) * grid) != cudaSuccess) return SFR_CUDA_ERROR;
  if (cudaMemcpy(b->d_block, blocks.data(), sizeof(int4) * grid, cudaMemcpyHostToDevice) !=
          cudaSuccess ||
      cudaMemcpy(b->d_sys, sys.data(), sizeof(int2) * grid, cudaMemcpyHostToDevice) != cudaSuccess)
    return SFR_CUDA_ERROR;
  const size_t need = e == kChipFp64           ? team_ws_bytes_onchip(b->cat.n, grid, S)
                      : e == kChipMixed        ? team_ws_bytes_mixed_team(b->cat.n, grid, S)
                      : precision == SFR_MIXED ? team_ws_bytes_mixed(b->cat.n, grid)
                                               : team_ws_bytes_fp64(b->cat.n, grid);
  if (need > b->ws_bytes) {
    cudaFree(b->ws);
    b->ws = nullptr;
    if (cudaMalloc(&b->ws, need) != cudaSuccess) return SFR_CUDA_ERROR;
    b->ws_bytes = need;
  }
  b->grid = grid;
  b->shape = shape;
  b->table.block = b->d_block;
  b->table.sys = b->d_sys;
  b->table.bar = b->d_bar;
  b->plan_solver = solver;
  b->plan_precision = precision;
  if (b->exec) {
    cudaGraphExecDestroy(b->exec);
    b->exec = nullptr;
  }
  return SFR_OK;
}

// The solve as a graph: [clear the team barriers -> one cooperative launch]
// on the persistent kernels, rounds_graph on chip.
int build(sfr_batch *b, int32_t solver, int32_t precision, double tol, uint32_t maxit,
          int32_t newx) {
  cudaGraph_t g = nullptr;
  int rc = SFR_OK;
  if (b->engine == kPersistent) {
    cudaStream_t cs = nullptr;
    if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) != cudaSuccess)
      return SFR_CUDA_ERROR;
    if (cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
      cudaStreamDestroy(cs);
      return SFR_CUDA_ERROR;
    }
    if (cudaMemsetAsync(b->d_bar, 0, sizeof(unsigned) * 2 * b->nsys, cs) != cudaSuccess)
      rc = SFR_CUDA_ERROR;
    if (rc == SFR_OK)
      rc = precision == SFR_MIXED
               ? enqueue_team_mixed(&b->cat, solver, b->d_b, b->d_x, tol, maxit, newx, b->table,
                                    b->grid, b->ws, b->d_out, b->d_ctl, cs)
               : enqueue_team_fp64(&b->cat, solver, b->d_b, b->d_x, tol, maxit, newx, b->table,
                                   b->grid, b->ws, b->d_out, b->d_ctl, cs);
    const cudaError_t ee = cudaStreamEndCapture(cs, &g);
    if (rc == SFR_OK && ee != cudaSuccess) rc = SFR_CUDA_ERROR;
    cudaStreamDestroy(cs);
  } else {
    TeamPlan plan;
    plan.shape = b->shape;
    plan.table = b->table;
    plan.systems = b->d_systems;
    plan.nsys = b->nsys;
    plan.grid = b->grid;
    plan.us = b->round_us;
    plan.us_later = b->round_us_later;
    rc = (b->engine == kChipFp64 ? graph_team_onchip : graph_mixed_team)(
        &b->cat, b->d_b, b->d_x, tol, maxit, newx, plan, b->ws, b->d_out, b->d_ctl, &g);
  }
  if (rc == SFR_OK && cudaGraphInstantiate(&b->exec, g, 0) != cudaSuccess) rc = SFR_CUDA_ERROR;
  if (g) cudaGraphDestroy(g);
  if (rc == SFR_OK) {
    b->g_tol = tol;
    b->g_maxit = maxit;
    b->g_newx = newx;
  }
  return rc;
}

int run(sfr_batch *b, int32_t solver, double tol, uint32_t maxit, int32_t newx,
        int32_t precision, std::vector<SolveOut> *out, float *ms) {
  int rc;
  if (b->plan_solver != solver || b->plan_precision != precision || !b->d_block) {
    rc = plan(b, solver, precision);
    if (rc != SFR_OK) return rc;
  }
  if (!b->exec || b->g_tol != tol || b->g_maxit != maxit || b->g_newx != newx) {
    if (b->exec) {
      cudaGraphExecDestroy(b->exec);
      b->exec = nullptr;
    }
    rc = build(b, solver, precision, tol, maxit, newx);
    if (rc != SFR_OK) return rc;
  }
  cudaStream_t st = b->cat.stream;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaEventRecord(e0, st);
  cudaError_t err = cudaGraphLaunch(b->exec, st);
  cudaEventRecord(e1, st);
  out->resize(b->nsys);
  unsigned ctl[3] = {0, 0, 0};
  if (err == cudaSuccess)
    err = cudaMemcpyAsync(out->data(), b->d_out, sizeof(SolveOut) * b->nsys,
                          cudaMemcpyDeviceToHost, st);
  if (err == cudaSuccess)
    err = cudaMemcpyAsync(ctl, b->d_ctl, sizeof(ctl), cudaMemcpyDeviceToHost, st);
  if (err == cudaSuccess) err = cudaStreamSynchronize(st);
  if (err == cudaSuccess) cudaEventElapsedTime(ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (err != cudaSuccess) {
    set_last_error(cudaGetErrorString(err));
    return SFR_CUDA_ERROR;
  }
  if (ctl[2] != 0) return static_cast<int>(ctl[2]);
  return SFR_OK;
}

}  // namespace

TeamShape team_shape(int device, const void *kern, int threads, int per_sm, int slice_bytes,
                     const TeamModel &model, bool far) {
  TeamShape sh;
  sh.per_sm = per_sm;
  sh.threads = threads;
  sh.model = model;
  int sm = 0, block = 0, occ = 0;
  if (cudaDeviceGetAttribute(&sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device) !=
          cudaSuccess ||
      cudaDeviceGetAttribute(&block, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) !=
          cudaSuccess)
    return sh;
  const size_t most = std::min(team_smem(sm, per_sm), team_smem(block + 1024, 1));
  const size_t smem = far ? std::min(most, team_smem(kFarSmem, per_sm)) : most;
  // the kernel's limit is one for all batches
  if (smem <= 64 ||
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(most)) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, threads, smem) != cudaSuccess ||
      occ < per_sm) {
    (void)cudaGetLastError();  // the refusal is not a later call's error
    return sh;
  }
  sh.smem = smem;
  sh.most = (static_cast<int>(smem) - 32) / slice_bytes;
  // neighbour_wait watches one block a thread
  sh.blocks = std::min(threads, per_sm * num_sms(device));
  return sh;
}

int rounds_graph(const void *kern, const TeamPlan &plan, void **params,
                 cudaGraphConditionalHandle *more, void *zero, size_t zero_bytes, unsigned *ctl,
                 cudaGraph_t *graph) {
  cudaGraph_t g = nullptr;
  if (cudaGraphCreate(&g, 0) != cudaSuccess) return SFR_CUDA_ERROR;
  *graph = g;
  if (cudaGraphConditionalHandleCreate(more, g, 1, cudaGraphCondAssignDefault) != cudaSuccess)
    return SFR_CUDA_ERROR;
  cudaGraphNode_t prev = nullptr;
  const std::pair<void *, size_t> clear[] = {{zero, zero_bytes}, {ctl, 64}};
  for (const auto &c : clear) {
    cudaMemsetParams mp{};
    mp.dst = c.first;
    mp.elementSize = 4;
    mp.width = c.second / 4;
    mp.height = 1;
    cudaGraphNode_t node = nullptr;
    if (cudaGraphAddMemsetNode(&node, g, prev ? &prev : nullptr, prev ? 1 : 0, &mp) != cudaSuccess)
      return SFR_CUDA_ERROR;
    prev = node;
  }
  cudaGraphNodeParams cp = {cudaGraphNodeTypeConditional};
  cp.conditional.handle = *more;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  cudaGraphNode_t loop = nullptr;
  if (cudaGraphAddNode(&loop, g, &prev, 1, &cp) != cudaSuccess) return SFR_CUDA_ERROR;
  cudaKernelNodeParams kp{};
  kp.func = const_cast<void *>(kern);
  kp.gridDim = dim3(plan.grid);
  kp.blockDim = dim3(plan.shape.threads);
  kp.sharedMemBytes = static_cast<unsigned>(plan.shape.smem);
  kp.kernelParams = params;  // the values are copied
  cudaGraphNode_t kn = nullptr;
  if (cudaGraphAddKernelNode(&kn, cp.conditional.phGraph_out[0], nullptr, 0, &kp) != cudaSuccess)
    return SFR_CUDA_ERROR;
  cudaKernelNodeAttrValue coop{};
  coop.cooperative = 1;
  return cudaGraphKernelNodeSetAttribute(kn, cudaLaunchAttributeCooperative, &coop) == cudaSuccess
             ? SFR_OK
             : SFR_CUDA_ERROR;
}

}  // namespace sfr

extern "C" {

int sfr_gpu_batch_create(int32_t nsys, const int32_t *neq, const int32_t *nad,
                         const int32_t *const *ia, const int32_t *const *ja, int32_t storage,
                         int32_t unsym, int32_t device, sfr_batch **out) {
  if (!out || nsys <= 0 || !neq || !ia) return SFR_BAD_INPUT;
  *out = nullptr;
  auto b = std::make_unique<sfr_batch>();
  b->device = device;
  b->nsys = nsys;
  b->storage = storage;
  b->unsym = unsym;
  sfr::HostSell cat;
  cat.sptr.push_back(0);
  int64_t rows = 0, slices = 0, src = 0;
  for (int s = 0; s < nsys; ++s) {
    sfr::HostSell h;
    std::string why;
    int32_t ns = 0;
    const int rc = sfr::build_sell(neq[s], nad ? nad[s] : 0, ia[s], ja ? ja[s] : nullptr,
                                   storage, unsym, &h, nullptr, &ns, &why);
    if (rc != SFR_OK) {
      sfr::set_last_error(("system " + std::to_string(s) + ": " + why).c_str());
      return rc;
    }
    b->n.push_back(neq[s]);
    b->row_off.push_back(static_cast<int32_t>(rows));
    b->slice_off.push_back(static_cast<int32_t>(slices));
    b->nslices.push_back(h.nslices);
    b->src_off.push_back(static_cast<int32_t>(src));
    b->nsrc.push_back(ns);
    const int32_t slot0 = cat.sptr.back();
    for (int32_t k = 1; k <= h.nslices; ++k) cat.sptr.push_back(slot0 + h.sptr[k]);
    for (size_t e = 0; e < h.col.size(); ++e) {
      cat.col.push_back(h.col[e] + static_cast<int32_t>(rows));
      cat.src.push_back(h.src[e] >= 0 ? h.src[e] + static_cast<int32_t>(src) : -1);
    }
    cat.bandwidth = std::max(cat.bandwidth, h.bandwidth);
    cat.max_width = std::max(cat.max_width, h.max_width);
    cat.far += h.far;
    cat.far_of += h.far_of;
    rows += static_cast<int64_t>(h.nslices) * sfr::kWarpHost;
    slices += h.nslices;
    src += ns;
    if (rows > INT32_MAX || src > INT32_MAX || cat.sptr.back() < 0) return SFR_BAD_INPUT;
    // default work estimate: slices x iterations, about 15 n^(1/3) of them
    b->weight.push_back(15.0 * h.nslices * std::cbrt(static_cast<double>(neq[s])));
  }
  b->team_ms.assign(nsys, 0.0);
  cat.n = static_cast<int32_t>(rows);
  cat.nslices = static_cast<int32_t>(slices);
  sfr_system &c = b->cat;
  c.device = device;
  c.n = cat.n;
  c.storage = storage;
  c.unsym = unsym;
  c.nsrc = static_cast<int32_t>(src);
  if (cudaSetDevice(device) != cudaSuccess) return SFR_CUDA_ERROR;
  if (cudaStreamCreateWithFlags(&c.stream, cudaStreamNonBlocking) != cudaSuccess)
    return SFR_CUDA_ERROR;
  int rc = sfr::upload_sell(cat, &c.A, &c.bytes);
  if (rc != SFR_OK) return rc;
  const size_t nrow = static_cast<size_t>(c.n);
  if (cudaMalloc(&c.d_stage, sizeof(double) * std::max<int64_t>(src, 1)) != cudaSuccess ||
      cudaMalloc(&c.d_diag, sizeof(double) * nrow) != cudaSuccess ||
      cudaMalloc(&c.d_diag32, sizeof(float) * nrow) != cudaSuccess ||
      cudaMalloc(&b->d_b, sizeof(double) * nrow) != cudaSuccess ||
      cudaMalloc(&b->d_x, sizeof(double) * nrow) != cudaSuccess ||
      cudaMalloc(&b->d_bar, sizeof(unsigned) * 2 * nsys) != cudaSuccess ||
      cudaMalloc(&b->d_systems, sizeof(int4) * nsys) != cudaSuccess ||
      cudaMalloc(&b->d_out, sizeof(sfr::SolveOut) * nsys) != cudaSuccess ||
      cudaMalloc(&b->d_ctl, 64) != cudaSuccess)
    return SFR_CUDA_ERROR;
  // padding rows: unit diagonal, zero right-hand side and solution
  std::vector<double> ones(nrow, 1.0);
  if (cudaMemcpy(c.d_diag, ones.data(), sizeof(double) * nrow, cudaMemcpyHostToDevice) !=
          cudaSuccess ||
      cudaMemset(b->d_b, 0, sizeof(double) * nrow) != cudaSuccess ||
      cudaMemset(b->d_x, 0, sizeof(double) * nrow) != cudaSuccess)
    return SFR_CUDA_ERROR;
  *out = b.release();
  return SFR_OK;
}

int sfr_gpu_batch_set_values(sfr_batch *b, const double *const *al, const double *const *ad,
                             const double *const *au) {
  if (!b || !ad || !al) return SFR_BAD_INPUT;
  sfr_system &c = b->cat;
  if (cudaSetDevice(b->device) != cudaSuccess) return SFR_CUDA_ERROR;
  const bool split = b->storage == SFR_CSRC && b->unsym;
  for (int s = 0; s < b->nsys; ++s) {
    if (!ad[s] || (!al[s] && b->nsrc[s] > 0)) return SFR_BAD_INPUT;
    double *dst = c.d_stage + b->src_off[s];
    if (split && au && au[s]) {
      const size_t half = static_cast<size_t>(b->nsrc[s]) / 2;
      if (cudaMemcpyAsync(dst, al[s], sizeof(double) * half, cudaMemcpyHostToDevice, c.stream) !=
              cudaSuccess ||
          cudaMemcpyAsync(dst + half, au[s], sizeof(double) * half, cudaMemcpyHostToDevice,
                          c.stream) != cudaSuccess)
        return SFR_CUDA_ERROR;
    } else if (b->nsrc[s] > 0) {
      if (cudaMemcpyAsync(dst, al[s], sizeof(double) * b->nsrc[s], cudaMemcpyHostToDevice,
                          c.stream) != cudaSuccess)
        return SFR_CUDA_ERROR;
    }
    if (cudaMemcpyAsync(c.d_diag + b->row_off[s], ad[s], sizeof(double) * b->n[s],
                        cudaMemcpyHostToDevice, c.stream) != cudaSuccess)
      return SFR_CUDA_ERROR;
  }
  int rc = sfr::gather_values(&c, &c.A, c.stream);
  if (rc != SFR_OK) return rc;
  rc = sfr::row_compensation(&c, c.A, c.stream);
  if (rc != SFR_OK) return rc;
  if (sfr::convert_diag32(c.d_diag, c.d_diag32, c.n, c.stream) != cudaSuccess ||
      cudaStreamSynchronize(c.stream) != cudaSuccess)
    return SFR_CUDA_ERROR;
  c.values_set = true;
  return SFR_OK;
}

int sfr_gpu_batch_solve(sfr_batch *b, int32_t solver, const double *const *bv, double *const *x,
                        double tol, uint32_t maxit, int32_t newx, int32_t precision,
                        sfr_solve_info *info) {
  if (!b || !bv || !x) return SFR_BAD_INPUT;
  if (solver != SFR_PCG && solver != SFR_PBICGSTAB) return SFR_UNSUPPORTED;
  if (precision != SFR_FP64 && precision != SFR_MIXED) return SFR_UNSUPPORTED;
  if (!b->cat.values_set) return SFR_BAD_INPUT;
  if (maxit == 0) return SFR_BAD_INPUT;
  sfr_system &c = b->cat;
  if (cudaSetDevice(b->device) != cudaSuccess) return SFR_CUDA_ERROR;
  for (int s = 0; s < b->nsys; ++s) {
    if (!bv[s] || !x[s]) return SFR_BAD_INPUT;
    const size_t bytes = sizeof(double) * b->n[s];
    if (cudaMemcpyAsync(b->d_b + b->row_off[s], bv[s], bytes, cudaMemcpyHostToDevice, c.stream) !=
        cudaSuccess)
      return SFR_CUDA_ERROR;
    if (!newx && cudaMemcpyAsync(b->d_x + b->row_off[s], x[s], bytes, cudaMemcpyHostToDevice,
                                 c.stream) != cudaSuccess)
      return SFR_CUDA_ERROR;
  }
  std::vector<sfr::SolveOut> out;
  float ms = 0.f;
  int rc = sfr::run(b, solver, tol, maxit, newx, precision, &out, &ms);
  if (rc != SFR_OK) return rc;
  int worst = SFR_OK;
  for (int s = 0; s < b->nsys; ++s) {
    if (cudaMemcpyAsync(x[s], b->d_x + b->row_off[s], sizeof(double) * b->n[s],
                        cudaMemcpyDeviceToHost, c.stream) != cudaSuccess)
      return SFR_CUDA_ERROR;
    if (info) {
      sfr_solve_info &f = info[s];
      std::memset(&f, 0, sizeof(f));
      f.iters = out[s].iters;
      f.status = out[s].status;
      f.xKx = out[s].xKx;
      f.norm_x = out[s].norm_x;
      f.norm_r = out[s].norm_r;
      f.norm_r_m = out[s].norm_r_m;
      f.conv = out[s].conv;
      f.seconds = ms * 1e-3;
      f.refinements = out[s].refinements;
      f.inner_iters = out[s].inner_iters;
      f.relres = out[s].bnorm > 0 ? out[s].norm_r / out[s].bnorm : std::nan("");
    }
    b->team_ms[s] = out[s].team_ms;
    if (out[s].status != SFR_OK && worst == SFR_OK) worst = out[s].status;
  }
  if (cudaStreamSynchronize(c.stream) != cudaSuccess) return SFR_CUDA_ERROR;
  return worst;
}

int sfr_gpu_batch_set_weights(sfr_batch *b, const double *w) {
  if (!b || !w) return SFR_BAD_INPUT;
  for (int s = 0; s < b->nsys; ++s)
    if (!(w[s] > 0.0)) return SFR_BAD_INPUT;
  b->weight.assign(w, w + b->nsys);
  b->team_blocks.clear();
  b->plan_solver = -1;  // re-plan on the next solve
  return SFR_OK;
}

// Autotuner: the batch's time is its slowest team's, so the blocks are
// shared out to equalise the teams' measured times.
//   1. Measure the default plan (blocks by slices x n^(1/3)) and the plan
//      weighted by slices x measured iterations; every team reports its own
//      time inside the launch (team_ms).
//   2. Fit each team's time to t(B) = f + w / B over the plans measured (f:
//      the barrier- and latency-bound part that more blocks do not shrink,
//      w / B: the part they share).
//   3. Bisect on the target time T for the smallest T whose block counts
//      B_s(T) = ceil(w_s / (T - f_s)) fit in one co-resident launch; hand
//      leftover blocks to the teams predicted slowest.
//   4. Measure that plan, refit, repeat (three model rounds at most); keep
//      the fastest plan measured.  Each plan is timed as the second of two
//      solves (CUDA events), so graph capture is not in the time.
int sfr_gpu_batch_autotune(sfr_batch *b, int32_t solver, const double *const *bv, double tol,
                           uint32_t maxit, int32_t precision, double *ms_out) {
  if (!b || !bv) return SFR_BAD_INPUT;
  const int S = b->nsys;
  std::vector<std::vector<double>> xs(S);
  std::vector<double *> xp(S);
  for (int s = 0; s < S; ++s) {
    xs[s].assign(b->n[s], 0.0);
    xp[s] = xs[s].data();
  }
  const int gmax = sfr::max_grid(b, solver, precision);
  if (gmax <= 0) return SFR_CUDA_ERROR;
  struct Sample {
    std::vector<int> nb;
    std::vector<double> t;
    double total;
  };
  std::vector<Sample> samples;
  std::vector<sfr_solve_info> info(S);
  std::vector<int> iters(S, 1);
  // one plan: install, solve twice, record the second solve's times
  auto measure = [&](const std::vector<int> *nb) -> int {
    if (nb) b->team_blocks = *nb;
    else b->team_blocks.clear();
    b->plan_solver = -1;
    for (int rep = 0; rep < 2; ++rep) {
      const int rc = sfr_gpu_batch_solve(b, solver, bv, xp.data(), tol, maxit, 1, precision,
                                         info.data());
      if (rc < 0) return rc;
    }
    Sample smp;
    smp.nb = b->blocks_of;
    smp.total = info[0].seconds * 1e3;
    smp.t.resize(S);
    for (int s = 0; s < S; ++s) {
      smp.t[s] = b->team_ms[s];
      iters[s] = std::max(1, info[s].inner_iters > 0 ? info[s].inner_iters : info[s].iters);
    }
    samples.push_back(std::move(smp));
    return SFR_OK;
  };
  const std::vector<double> w_default = b->weight;
  int rc = measure(nullptr);  // the default work estimate
  if (rc != SFR_OK) return rc;
  std::vector<double> w1(S);
  for (int s = 0; s < S; ++s) w1[s] = static_cast<double>(b->nslices[s]) * iters[s];
  b->weight = w1;
  rc = measure(nullptr);  // weighted by measured iterations
  if (rc != SFR_OK) return rc;

  for (int round = 0; round < 3; ++round) {
    // fit t = f + w / B per team (least squares over the distinct B seen)
    std::vector<double> f(S), w(S);
    for (int s = 0; s < S; ++s) {
      double su = 0, sv = 0, suu = 0, suv = 0;
      int m = 0;
      for (const Sample &smp : samples) {
        const double u = 1.0 / smp.nb[s];
        su += u;
        sv += smp.t[s];
        suu += u * u;
        suv += u * smp.t[s];
        ++m;
      }
      const double den = m * suu - su * su;
      double ws = 0.0, fs = 0.0;
      if (m >= 2 && den > 1e-18 * m * suu) {
        ws = (m * suv - su * sv) / den;
        fs = (sv - ws * su) / m;
      }
      if (!(ws > 0.0) || !(fs >= 0.0)) {
        // one block count seen, or times that do not shrink with more
        // blocks: split the latest time evenly into the two parts
        const Sample &last = samples.back();
        fs = 0.5 * last.t[s];
        ws = 0.5 * last.t[s] * last.nb[s];
      }
      f[s] = fs;
      w[s] = ws;
    }
    auto need = [&](int s, double T) -> int {  // blocks team s needs for time T
      if (T <= f[s]) return INT32_MAX;
      const double bl = std::ceil(w[s] / (T - f[s]) - 1e-9);
      return bl > INT32_MAX / 2 ? INT32_MAX : std::max(1, static_cast<int>(bl));
    };
    auto fits = [&](double T) {
      int64_t tot = 0;
      for (int s = 0; s < S; ++s) {
        const int bl = need(s, T);
        if (bl > b->nslices[s]) return false;
        tot += bl;
      }
      return tot <= gmax;
    };
    double hi = 0.0;
    for (int s = 0; s < S; ++s) hi = std::max(hi, f[s] + w[s]);  // one block each
    double lo = 0.0;
    if (!fits(hi)) break;  // the model cannot place every team
    for (int it = 0; it < 60; ++it) {
      const double mid = 0.5 * (lo + hi);
      if (fits(mid)) hi = mid;
      else lo = mid;
    }
    std::vector<int> nb(S);
    int total = 0;
    for (int s = 0; s < S; ++s) {
      nb[s] = need(s, hi);
      total += nb[s];
    }
    while (total < gmax) {  // leftovers to the teams predicted slowest
      int worst = -1;
      double tw = -1.0;
      for (int s = 0; s < S; ++s) {
        if (nb[s] >= b->nslices[s]) continue;
        const double t = f[s] + w[s] / nb[s];
        if (t > tw) {
          tw = t;
          worst = s;
        }
      }
      if (worst < 0) break;
      ++nb[worst];
      ++total;
    }
    bool seen = false;
    for (const Sample &smp : samples) seen = seen || smp.nb == nb;
    if (seen) break;  // converged on a plan already measured
    rc = measure(&nb);
    if (rc != SFR_OK) return rc;
  }
  size_t best = 0;
  for (size_t i = 1; i < samples.size(); ++i)
    if (samples[i].total < samples[best].total) best = i;
  // keep the best plan
  if (best == 0) {
    b->weight = w_default;
    b->team_blocks.clear();
  } else if (best == 1) {
    b->team_blocks.clear();
  } else {
    b->team_blocks = samples[best].nb;
  }
  b->plan_solver = -1;
  sfr_batch_tune &r = b->tune;
  r.default_ms = samples[0].total;
  r.weighted_ms = samples[1].total;
  r.tuned_ms = samples[best].total;
  r.plans = static_cast<int32_t>(samples.size());
  r.kept = static_cast<int32_t>(best);
  int g = 0, mx = 0, mn = INT32_MAX;
  for (int v : samples[best].nb) {
    g += v;
    mx = std::max(mx, v);
    mn = std::min(mn, v);
  }
  r.grid = g;
  r.max_team_blocks = mx;
  r.min_team_blocks = mn;
  if (ms_out) *ms_out = samples[best].total;
  return SFR_OK;
}

int sfr_gpu_batch_tune_report(const sfr_batch *b, sfr_batch_tune *out) {
  if (!b || !out) return SFR_BAD_INPUT;
  *out = b->tune;
  return SFR_OK;
}

int sfr_gpu_batch_stats(const sfr_batch *b, int32_t *grid, int64_t *rows, int64_t *bytes) {
  if (!b) return SFR_BAD_INPUT;
  if (grid) *grid = b->grid;
  if (rows) *rows = b->cat.n;
  if (bytes) *bytes = b->cat.bytes + static_cast<int64_t>(b->ws_bytes);
  return SFR_OK;
}

int sfr_gpu_batch_destroy(sfr_batch *b) {
  if (!b) return SFR_OK;
  cudaSetDevice(b->device);
  if (b->exec) cudaGraphExecDestroy(b->exec);
  sfr::free_sell(&b->cat.A);
  cudaFree(b->cat.d_stage);
  cudaFree(b->cat.d_diag);
  cudaFree(b->cat.d_diag32);
  cudaFree(b->cat.d_comp);
  if (b->cat.stream) cudaStreamDestroy(b->cat.stream);
  cudaFree(b->d_block);
  cudaFree(b->d_sys);
  cudaFree(b->d_systems);
  cudaFree(b->d_bar);
  cudaFree(b->ws);
  cudaFree(b->d_out);
  cudaFree(b->d_ctl);
  cudaFree(b->d_b);
  cudaFree(b->d_x);
  delete b;
  return SFR_OK;
}

}  // extern "C"
