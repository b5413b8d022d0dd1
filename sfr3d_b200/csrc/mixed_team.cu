// Mixed-precision PCG for a batch of systems: the iteration of mixed.cu's
// pcg_mixed_kernel (FP32 recurrence, FP64 dot products, FP64 reliable
// updates, one right-hand side) on teams of blocks that exchange their sums
// in one L2 round trip and keep their rows' vectors in shared memory.
//
// Every FP32 number of the recurrence is formed by the same operations from
// the same operands; only the FP64 dot products add their terms in another
// order, and their last places vanish when alpha and beta round to FP32.
//
// What an iteration waits on: the exchanges of (q, p) and of (r, z), the
// publication of p to the blocks that gather it, and the product's two
// dependent L2 round trips.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "common.cuh"
#include "internal.h"
#include "persist.cuh"
#include "team_plan.h"
#include "team_sync.cuh"

namespace sfr {

namespace {

constexpr int kChunk = 6;          // slots of a row loaded before their gathers
constexpr int kSmThreads = 768;    // an SM's, in one block or two: 80 registers each

// Slices (of 6 slots: 1.2 KB of FP32 values and 16-bit columns) of the
// systems left up to which the matrix is kept in L2 between iterations; past
// that it streams, evict-first, and leaves L2 to the vectors.
constexpr int kKeepSlices = 58000;

struct MixedTeamArgs {
  const int *sptr, *col;
  const int16_t *off;
  const float *val32;
  const double *val64, *diag, *comp, *b;
  double *x;
  double *dc;                          // diagonal of the FP32 operator
  float *m32, *r, *p, *xs;             // as mixed.cu names them
  TeamSync sync;
  SolveOut *out;
  double tol, delta;
  unsigned maxit;
  int newx;
};

// Where a system stands between two rounds (r, xs and p are in global memory
// then).
struct MixedState {
  double conv, bnorm, d, rmax;
  unsigned j;
  int refine;
  unsigned long long t0;  // its first round's start (global_ns)
};

// At most `cap` iterations of a system, going on from *st when `resume`; true
// when its solve is over.
template <typename I>
__device__ __forceinline__ bool pcg_mixed_body(const MixedTeamArgs &a, const TeamPart &t,
                                               char *sm_dyn, int smem, TeamShared &sh,
                                               unsigned epoch, unsigned tick, bool stream,
                                               MixedState *st, const RoundTable &rt, bool resume,
                                               unsigned cap) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int s0 = t.s0, s1 = t.s1;
  const int r0 = s0 * kWarp, rows = (s1 - s0) * kWarp;
  const int own = max(0, min(rows, t.row_end - r0));
  const int slot0 = __ldg(a.sptr + s0), nslots = __ldg(a.sptr + s1) - slot0;

  // q and the slice pointers always fit (team_max_slices_mixed_team); what
  // else stays on chip, most traffic saved a byte first
  Carve sm{sm_dyn, smem};
  int *sm_sp = sm.take<int>(s1 - s0 + 1);
  float *vq = sm.take<float>(rows);  // A p, then z = M r
  float *vr = sm.take<float>(rows), *vxs = vr ? sm.take<float>(rows) : nullptr;
  float *vm = vxs ? sm.take<float>(rows) : nullptr;
  double *vdc = vm ? sm.take<double>(rows) : nullptr;
  I *sm_c = vdc ? sm.take<I>(nslots) : nullptr;
  float *sm_v = sm_c ? sm.take<float>(nslots) : nullptr;
  if (!vr) vr = a.r + r0;
  if (!vxs) vxs = a.xs + r0;
  if (!vm) vm = a.m32 + r0;
  if (!vdc) vdc = a.dc + r0;
  const I *cols = cols_of<I>(SlotCols{a.col, a.off});
  for (int i = threadIdx.x; i <= s1 - s0; i += blockDim.x) sm_sp[i] = __ldg(a.sptr + s0 + i);
  if (sm_v)
    for (int i = threadIdx.x; i < nslots; i += blockDim.x) {
      sm_v[i] = __ldcs(a.val32 + slot0 + i);
      sm_c[i] = __ldcs(cols + slot0 + i);
    }
  __syncthreads();
  const bool alone = t.b1 - t.b0 == 1;
  if (!alone) gather_range(t, sm_sp, cols, sh.range);
  uint64_t pol;  // the matrix's L2 policy
  if (stream)
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
  else
    asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(pol));

  auto sum1 = [&](double v, double *out) {
    const double acc[1] = {v};
    double tot[1];
    const bool ok = team_sum<1, false>(a.sync, t, epoch, acc, tot, sh.red, &sh.bad);
    *out = tot[0];
    return ok;
  };
  // the sum also publishes every global write of the team's blocks
  auto sum1_fence = [&](double v, double *out) {
    const double acc[1] = {v};
    double tot[1];
    const bool ok = team_sum<1, true>(a.sync, t, epoch, acc, tot, sh.red, &sh.bad);
    *out = tot[0];
    return ok;
  };
  auto sum2_fence = [&](const double (&acc)[2], double (&tot)[2]) {
    return team_sum<2, true>(a.sync, t, epoch, acc, tot, sh.red, &sh.bad);
  };

  // (A64 x)[row] in FP64 (FMA allowed: the refinement residual)
  auto row64 = [&](int s, int row) {
    const int base = sm_sp[s - s0], w = (sm_sp[s - s0 + 1] - base) >> 5;
    const int *c = a.col + base + lane;
    const double *v = a.val64 + base + lane;
    double y = ld_vec(a.diag + row) * ld_vec(a.x + row);
    for (int e0 = 0; e0 < w; e0 += kChunk) {
      int jj[kChunk];
      double vv[kChunk];
#pragma unroll
      for (int u = 0; u < kChunk; ++u)
        if (e0 + u < w) {
          jj[u] = ld_stream(c + (e0 + u) * kWarp);
          vv[u] = ld_stream(v + (e0 + u) * kWarp);
        }
#pragma unroll
      for (int u = 0; u < kChunk; ++u)
        if (e0 + u < w) y = fma(vv[u], ld_vec(a.x + jj[u]), y);
    }
    return y;
  };
  // reliable update: r = fl32(b - A64 x), z = M r, xs = 0; tot = {(r, M r)
  // of the FP64 residual, (r, z) of the FP32 one}
  auto residual = [&](bool first, double (&tot)[2]) {
    double acc[2] = {0.0, 0.0};
    for (int s = s0 + warp; s < s1; s += nw) {
      const int row = s * kWarp + lane, lr = row - r0;
      if (row >= t.row_end) continue;
      const double rt = ld_vec(a.b + row) - row64(s, row);
      const float rs = __double2float_rn(rt);
      const float zs = vm[lr] * rs;
      vr[lr] = rs;
      vxs[lr] = 0.0f;
      vq[lr] = zs;
      if (first) st_vec(a.p + row, zs);
      acc[0] += rt * (rt / ld_vec(a.diag + row));
      acc[1] += static_cast<double>(rs) * static_cast<double>(zs);
    }
    return sum2_fence(acc, tot);
  };
  // p is written: wait on the blocks whose p this block gathers
  auto publish = [&]() {
    if (alone) {
      __syncthreads();
      return true;
    }
    return neighbour_wait(a.sync.ticks, a.sync.err, a.sync.spin_limit, ++tick, sh.range[0],
                          sh.range[1]);
  };
  auto fold = [&]() {  // x += xs
    for (int lr = threadIdx.x; lr < own; lr += blockDim.x)
      st_vec(a.x + r0 + lr, ld_vec(a.x + r0 + lr) + static_cast<double>(vxs[lr]));
  };

  double conv, bnorm, d, rmax, alpha, beta;
  bool act = true;
  int status = SFR_OK, refine = 0;
  unsigned iters = 0, j = 0;
  if (!resume) {
    double acc[2] = {0.0, 0.0}, tot[2];
    for (int lr = threadIdx.x; lr < own; lr += blockDim.x) {
      const double dk = ld_vec(a.diag + r0 + lr), bk = ld_vec(a.b + r0 + lr);
      vdc[lr] = dk + ld_vec(a.comp + r0 + lr);
      vm[lr] = __double2float_rn(1.0 / dk);
      if (a.newx) st_vec(a.x + r0 + lr, 0.0);
      acc[0] += bk * (bk / dk);
      acc[1] += bk * bk;
    }
    if (!sum2_fence(acc, tot)) return false;
    conv = a.tol * sqrt(fabs(tot[0]));
    bnorm = sqrt(tot[1]);
    if (!residual(true, tot)) return false;
    rmax = sqrt(fabs(tot[0]));
    d = tot[1];
    if (rmax < conv) act = false;
  } else {
    conv = __ldcg(&st->conv);
    bnorm = __ldcg(&st->bnorm);
    d = __ldcg(&st->d);
    rmax = __ldcg(&st->rmax);
    j = __ldcg(&st->j);
    refine = __ldcg(&st->refine);
    for (int lr = threadIdx.x; lr < own; lr += blockDim.x) {
      const double dk = ld_vec(a.diag + r0 + lr);
      vdc[lr] = dk + ld_vec(a.comp + r0 + lr);
      vm[lr] = __double2float_rn(1.0 / dk);
      if (vr != a.r + r0) vr[lr] = ld_vec(a.r + r0 + lr);
      if (vxs != a.xs + r0) vxs[lr] = ld_vec(a.xs + r0 + lr);
    }
    __syncthreads();
  }
  const unsigned stop = j + min(cap, 0xffffffffu - j);
  for (; j < a.maxit && act; ++j) {
    // q = A32 p
    {
      double acc = 0.0, tot;
      for (int s = s0 + warp; s < s1; s += nw) {
        const int base = sm_sp[s - s0], w = (sm_sp[s - s0 + 1] - base) >> 5;
        const int row = s * kWarp + lane, lr = row - r0;
        if (row >= t.row_end) continue;
        const double dcv = vdc[lr];
        const float pk = ld_vec(a.p + row);
        double y = dcv * static_cast<double>(pk);
        if (sm_v) {
          const I *c = sm_c + (base - slot0) + lane;
          const float *v = sm_v + (base - slot0) + lane;
          for (int e0 = 0; e0 < w; e0 += kChunk) {
            float g[kChunk];
#pragma unroll
            for (int u = 0; u < kChunk; ++u)
              if (e0 + u < w) g[u] = ld_vec(a.p + smem_col(c, (e0 + u) * kWarp, row));
#pragma unroll
            for (int u = 0; u < kChunk; ++u)
              if (e0 + u < w)
                y = fma(static_cast<double>(v[(e0 + u) * kWarp]), static_cast<double>(g[u]), y);
          }
        } else {
          const I *c = cols + base + lane;
          const float *v = a.val32 + base + lane;
          int jj[kChunk];
          float vv[kChunk];
          for (int e0 = 0; e0 < w; e0 += kChunk) {
#pragma unroll
            for (int u = 0; u < kChunk; ++u)
              if (e0 + u < w) {
                const int o = ld_mat(c + (e0 + u) * kWarp, pol);
                jj[u] = sizeof(I) == 2 ? row + o : o;
                vv[u] = ld_mat(v + (e0 + u) * kWarp, pol);
              }
#pragma unroll
            for (int u = 0; u < kChunk; ++u)
              if (e0 + u < w)
                y = fma(static_cast<double>(vv[u]), static_cast<double>(ld_vec(a.p + jj[u])), y);
          }
        }
        const float yf = __double2float_rn(y);
        vq[lr] = yf;
        acc += static_cast<double>(yf) * static_cast<double>(pk);
      }
      if (!sum1(acc, &tot)) return false;
      alpha = d / tot;
      if (!isfinite(alpha)) {
        act = false;
        status = SFR_BREAKDOWN;
        iters = j + 1;
        break;
      }
    }
    // xs += alpha p ; r -= alpha q ; z = M r ; (r, z)
    double tot;
    {
      const float af = static_cast<float>(alpha);
      double acc = 0.0;
      for (int lr = threadIdx.x; lr < own; lr += blockDim.x) {
        const float pk = ld_vec(a.p + r0 + lr);
        vxs[lr] = fmaf(af, pk, vxs[lr]);
        const float rk = fmaf(-af, vq[lr], vr[lr]);
        const float zk = vm[lr] * rk;
        vr[lr] = rk;
        vq[lr] = zk;
        acc += static_cast<double>(rk) * static_cast<double>(zk);
      }
      if (!sum1(acc, &tot)) return false;
    }
    if (!isfinite(tot)) {
      act = false;
      status = SFR_BREAKDOWN;
      iters = j + 1;
      break;
    }
    const double est = sqrt(fabs(tot));
    if (est < a.delta * rmax || est < conv) {
      fold();
      double none, rt[2];
      if (!sum1_fence(0.0, &none)) return false;
      if (!residual(false, rt)) return false;
      ++refine;
      const double tr = sqrt(fabs(rt[0]));
      if (tr < conv) {
        act = false;
        iters = j + 1;
        break;
      }
      beta = rt[1] / d;
      d = rt[1];
      rmax = tr;
    } else {
      beta = tot / d;
      d = tot;
    }
    // p = z + beta p
    {
      const float bf = static_cast<float>(beta);
      for (int lr = threadIdx.x; lr < own; lr += blockDim.x)
        st_vec(a.p + r0 + lr, fmaf(bf, ld_vec(a.p + r0 + lr), vq[lr]));
      if (!publish()) return false;
    }
    if (j + 1 == stop && j + 1 < a.maxit) {  // the round is over
      for (int lr = threadIdx.x; lr < own; lr += blockDim.x) {
        if (vr != a.r + r0) st_vec(a.r + r0 + lr, vr[lr]);
        if (vxs != a.xs + r0) st_vec(a.xs + r0 + lr, vxs[lr]);
      }
      if (static_cast<int>(blockIdx.x) == t.b0 && threadIdx.x == 0) {
        rt.put_iters(t.sys, t.round, j + 1);
        *st = MixedState{conv, bnorm, d, rmax, j + 1, refine, resume ? st->t0 : t.t0};
      }
      return false;
    }
  }
  if (act) {  // iteration cap: fold the last correction into x
    status = SFR_MAXIT;
    iters = j + 1;
    fold();
    double none;
    if (!sum1_fence(0.0, &none)) return false;
  }
  // xKx, ||x||, ||b - Ax||_M, ||b - Ax||
  double acc[4] = {0.0, 0.0, 0.0, 0.0}, tot[4];
  for (int s = s0 + warp; s < s1; s += nw) {
    const int row = s * kWarp + lane;
    if (row >= t.row_end) continue;
    const double y = row64(s, row), xk = ld_vec(a.x + row), rk = ld_vec(a.b + row) - y;
    acc[0] += xk * y;
    acc[1] += xk * xk;
    acc[2] += rk * (rk / ld_vec(a.diag + row));
    acc[3] += rk * rk;
  }
  if (!team_sum<4, false>(a.sync, t, epoch, acc, tot, sh.red, &sh.bad)) return false;
  if (static_cast<int>(blockIdx.x) == t.b0 && threadIdx.x == 0) {
    SolveOut o{};
    o.iters = o.inner_iters = static_cast<int>(iters);
    o.status = status;
    o.xKx = tot[0];
    o.norm_x = sqrt(tot[1]);
    o.norm_r_m = sqrt(fabs(tot[2]));
    o.norm_r = sqrt(tot[3]);
    o.conv = conv;
    o.bnorm = bnorm;
    o.refinements = refine;
    o.team_ms = (global_ns() - (resume ? st->t0 : t.t0)) * 1e-6;
    a.out[t.sys] = o;
  }
  return true;
}

template <typename I, int kT>
__global__ void __launch_bounds__(kT, kSmThreads / kT)
    pcg_mixed_team_kernel(const MixedTeamArgs a, const TeamTable tt, const RoundTable rt,
                          MixedState *states, int smem) {
  extern __shared__ double sm_dyn[];
  __shared__ TeamShared sh;
  const unsigned round = __ldcg(rt.ctl);
  {
    const TeamPart mine = team_part(tt, rt, round, sh.scan);
    if (threadIdx.x == 0) sh.part = mine;
    __syncthreads();
  }
  const TeamPart &t = sh.part;
  bool over = false;
  if (t.b1 > t.b0)
    over = pcg_mixed_body<I>(a, t, reinterpret_cast<char *>(sm_dyn), smem, sh, round_base(round),
                             round_base(round), t.slices_left > kKeepSlices, states + t.sys, rt, round > 0, round_cap(rt, t, round));
  __syncthreads();
  end_round(rt, t, over && static_cast<int>(blockIdx.x) == t.b0);
}

const void *team_kernel(const sfr_system *s, int per_sm) {
  if (per_sm == 1)
    return s->A.off ? reinterpret_cast<const void *>(pcg_mixed_team_kernel<int16_t, kSmThreads>)
                    : reinterpret_cast<const void *>(pcg_mixed_team_kernel<int, kSmThreads>);
  return s->A.off
             ? reinterpret_cast<const void *>(pcg_mixed_team_kernel<int16_t, kSmThreads / 2>)
             : reinterpret_cast<const void *>(pcg_mixed_team_kernel<int, kSmThreads / 2>);
}

size_t align256(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }

}  // namespace

// The model: 16 boxes of 16^3 on 9 blocks each (14 slices a block) 8.4 us an
// iteration, 32^3 (111 slices) 13.0, 48^3 (375) 40.7; a block alone with 16
// slices 3.4.
TeamShape team_shape_mixed(const sfr_system *s, int per_sm) {
  return team_shape(s->device, team_kernel(s, per_sm), kSmThreads / per_sm, per_sm, kWarp * 4 + 4,
                    TeamModel{2.5f, 7.5f, 0.12f}, s->A.far());
}

size_t team_ws_bytes_mixed_team(int n, int grid, int nsys) {
  return align256((sizeof(MixedState) + kRoundInts * sizeof(int)) * static_cast<size_t>(nsys)) +
         align256(sizeof(double) * static_cast<size_t>(n)) +
         4 * align256(sizeof(float) * static_cast<size_t>(n)) +
         align256(sizeof(TeamSlot) * 2 * static_cast<size_t>(grid)) +
         align256(64 * static_cast<size_t>(grid));
}

int graph_mixed_team(sfr_system *s, const double *d_b, double *d_x, double tol, uint32_t maxit,
                     int32_t newx, const TeamPlan &plan, void *ws, SolveOut *d_out, unsigned *ctl,
                     cudaGraph_t *graph) {
  const size_t dc_b = align256(sizeof(double) * static_cast<size_t>(s->n));
  const size_t vec = align256(sizeof(float) * static_cast<size_t>(s->n));
  const size_t slot_b = align256(sizeof(TeamSlot) * 2 * static_cast<size_t>(plan.grid));
  const size_t tick_b = align256(64 * static_cast<size_t>(plan.grid));
  const size_t state_b =
      align256((sizeof(MixedState) + kRoundInts * sizeof(int)) * static_cast<size_t>(plan.nsys));
  char *base = static_cast<char *>(ws);
  MixedState *states = reinterpret_cast<MixedState *>(base + slot_b + tick_b);
  RoundTable rt = round_table(plan, reinterpret_cast<int *>(states + plan.nsys), ctl);
  MixedTeamArgs a{};
  a.sptr = s->A.sptr;
  a.col = s->A.col;
  a.off = s->A.off;
  a.val32 = s->A.val32;
  a.val64 = s->A.val;
  a.diag = s->d_diag;
  a.comp = s->d_comp;
  a.b = d_b;
  a.x = d_x;
  a.sync.slots = reinterpret_cast<TeamSlot *>(base);
  a.sync.ticks = reinterpret_cast<unsigned *>(base + slot_b);
  a.sync.err = reinterpret_cast<int *>(ctl + 2);
  a.sync.spin_limit = 1u << 22;
  char *vecs = base + slot_b + tick_b + state_b;
  a.dc = reinterpret_cast<double *>(vecs);
  float **f[] = {&a.m32, &a.r, &a.p, &a.xs};
  for (int i = 0; i < 4; ++i)
    *f[i] = reinterpret_cast<float *>(vecs + dc_b + static_cast<size_t>(i) * vec);
  a.out = d_out;
  a.tol = tol;
  a.delta = reliable_delta(SFR_PCG);
  a.maxit = maxit;
  a.newx = newx;
  int smem = static_cast<int>(plan.shape.smem);
  TeamTable tt = plan.table;
  void *params[] = {&a, &tt, &rt, &states, &smem};
  return rounds_graph(team_kernel(s, plan.shape.per_sm), plan, params, &rt.more, base,
                      slot_b + tick_b + state_b, ctl, graph);
}

}  // namespace sfr
