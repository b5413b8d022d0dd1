// On-chip engine: a whole FP64 Jacobi-PCG solve (Cg.c:47-209, one right-hand
// side) in one launch, with the Krylov state in shared memory and one
// reduction an iteration.
//
// The iteration.  The reference forms two dot products an iteration with a
// dependent vector update between them: alpha needs (q, p), beta needs the
// (r, z) of the updated residual.  Here the SpMV phase forms every product
// at once -- mu = (p, q), delta = (z, q), gamma = (q, M q), nu = (r, z) --
// and beta comes from nu' = nu - 2 alpha delta + alpha^2 gamma, the (r, z)
// the update is about to produce (predict-and-recompute CG: Chen & Carson,
// SIAM J. Matrix Anal. Appl. 2020).  The next SpMV phase recomputes nu from
// the residual it holds, so alpha and the stopping test always use the
// measured product, never the predicted one; nu' only shapes beta, formed as
// 1 - 2 delta / mu + alpha gamma / mu: right to a few eps in absolute terms, so
// that a step which takes (r, z) down by many orders leaves beta few digits or
// none.  p then keeps a few eps of the old direction beside a z many orders
// larger than that, and the solve goes on as the reference's (a right-hand side
// of one eigenvector and 1e-11 of noise: the same count of iterations).  An
// iteration is then SpMV, exchange, update, publication of p: two
// synchronisations instead of three, and no vector but p leaves the chip.
// Every SpMV row keeps the reference's rounding and order (diagonal product,
// then each slot).  A solve runs one SpMV phase beyond its last update, the
// one that measures the residual it stops on.
//
// Two forms, one arithmetic:
//   cluster  one thread-block cluster holds the whole system: matrix, vectors
//            and p in its blocks' shared memory, gathers of p through
//            distributed shared memory, synchronisation by the cluster
//            barrier.
//   grid     one block per SM, the exchange and the publication of p through
//            L2; the matrix streams from L2 or HBM, or sits in shared memory
//            when it fits.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <utility>

#include "common.cuh"
#include "internal.h"
#include "persist.cuh"
#include "team_plan.h"
#include "team_sync.cuh"

namespace sfr {

namespace {

constexpr int kChunk = 6;  // slots of a row loaded before their gathers (a hex cell's faces)

struct ChipArgs {
  int n, nslices;
  const int *sptr, *col;
  const int16_t *off;
  const double *val, *diag, *b;
  double *x;
  double *p;        // grid form: the search direction, nslices * 32 entries
  double *z;        // grid form, level 0: M r, nslices * 32 entries
  TeamSync sync;    // grid form
  SolveOut *out;
  double tol;
  unsigned maxit;
  int newx;
};

// The scalars of iteration j from the exchanged products {mu, delta, gamma,
// nu}: false when the solve stops (status and iters set).  Iteration j - 1's
// tests come first, on the (r, z) of the residual it left (Cg.c:145); the
// square root and the quotient they name are formed only near their
// thresholds, so an ordinary iteration waits on one division's latency.
struct Scalars {
  double conv, conv2, bnorm = 0.0, nu_old = 0.0, alpha = 0.0, beta = 0.0;
  int status = SFR_OK;
  unsigned iters = 0;
  __device__ __forceinline__ explicit Scalars(double c)
      : conv(c), conv2(fma(c, c * (1.0 + 1e-9), 1e-300)) {}
  __device__ __forceinline__ bool next(const double (&t)[4], unsigned j, unsigned maxit) {
    const double nu = t[3], mu = t[0];
    const double inv = 1.0 / mu;
    alpha = nu / mu;
    if (j > 0) {
      if (!(fabs(nu) > conv2) && sqrt(fabs(nu)) < conv) {
        iters = j;
        return false;
      }
      if (!(fabs(nu) < 1e150 && fabs(nu_old) > 1e-150) && !isfinite(nu / nu_old)) {
        iters = j;
        status = SFR_BREAKDOWN;
        return false;
      }
      if (j >= maxit) {
        iters = j + 1;
        status = SFR_MAXIT;
        return false;
      }
    }
    if (!isfinite(alpha)) {
      iters = j + 1;
      status = SFR_BREAKDOWN;
      return false;
    }
    // nu' / nu = 1 - 2 delta / mu + alpha gamma / mu
    beta = fma(fma(alpha, t[2], -2.0 * t[1]), inv, 1.0);
    nu_old = nu;
    return true;
  }
};

// The result record of a finished solve.
__device__ __forceinline__ void put_result(SolveOut *out, const Scalars &sc,
                                           const double (&tot)[4], double ms) {
  SolveOut o{};
  o.iters = static_cast<int>(sc.iters);
  o.status = sc.status;
  o.xKx = tot[0];
  o.norm_x = sqrt(tot[1]);
  o.norm_r_m = sqrt(fabs(tot[2]));
  o.norm_r = sqrt(tot[3]);
  o.conv = sc.conv;
  o.bnorm = sc.bnorm;
  o.inner_iters = static_cast<int>(sc.iters);
  o.team_ms = ms;
  *out = o;
}

// Where a block of the grid form keeps its rows' state, by what fits:
//   level 0  M q in shared memory (8 B a row); z, x, ad and p in L2 or HBM
//   level 1  also z (16 B a row)
//   level 2  also x (24 B a row)
//   level 3  also ad and the block's own p (40 B a row)
// and its slots (values and columns):
//   kHold    in shared memory: they never leave the SM again
//   kKeep    in L2, under its normal policy
//   kStream  from HBM, evict-first
constexpr int kLevels = 4;
__host__ __device__ constexpr int level_bytes(int level) {
  return level == 0 ? 8 : level == 1 ? 16 : level == 2 ? 24 : 40;
}
enum Slots { kHold, kKeep, kStream, kPolicy };  // kPolicy: kKeep or kStream, by the call

// A batch's slices (of 6 slots: 1.9 KB) up to which kPolicy keeps the slots:
// 70 MB, the line kKeepBytes draws for one system.
constexpr int kKeepSlices = 36000;

// Threads a block: 24 warps at 80 registers hold a slice's slots, gathers and
// the four sums without spilling.  An iteration at 96^3 / 128^3: 13.2 / 41.1
// us; 1024 threads (64 registers, 32 bytes spilled) 15.2 / 45.0; 512 threads
// 17.3 / 51.5.
constexpr int kGridThreads = 768;

// Where a system of a batched launch stands between two rounds (z, x and p
// are in a.z, a.x and a.p).
struct ChipState {
  double conv, bnorm, nu_old;
  unsigned j;
  unsigned long long t0;  // its first round's start (global_ns)
};

// The solve, or (st given) at most `cap` of its iterations, going on from
// *st when `resume`; true when it is over.  epoch and tick: what the team's
// exchanges and publications count from.
template <typename I, int kLevel, Slots kSlots>
__device__ __forceinline__ bool pcg_grid_body(const ChipArgs &a, const TeamPart &t,
                                              double *sm_dyn, TeamShared &sh, unsigned epoch,
                                              unsigned tick, ChipState *st,
                                              const RoundTable *rt, bool resume,
                                              unsigned cap) {
  double *const red = sh.red;
  int *const bad = &sh.bad, *const range = sh.range;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int s0 = t.s0, s1 = t.s1;
  const int r0 = s0 * kWarp, rows = (s1 - s0) * kWarp;
  const int own = max(0, min(rows, t.row_end - r0));  // rows that are equations
  const int slot0 = __ldg(a.sptr + s0);
  double *sm_t = sm_dyn;
  double *vz = kLevel >= 1 ? sm_t + rows : a.z + r0;
  double *vx = kLevel >= 2 ? sm_t + 2 * rows : a.x + r0;
  double *sm_d = sm_t + 3 * rows, *sm_p = sm_d + rows;  // level 3
  double *sm_v = sm_t + (level_bytes(kLevel) / 8) * rows;  // kHold
  const I *cols = cols_of<I>(SlotCols{a.col, a.off});
  const int held = kSlots == kHold ? __ldg(a.sptr + s1) - slot0 : 0;  // a multiple of 32
  I *sm_c = reinterpret_cast<I *>(sm_v + held);
  int *sm_sp = reinterpret_cast<int *>(sm_c + held);
  for (int i = threadIdx.x; i <= s1 - s0; i += blockDim.x) sm_sp[i] = __ldg(a.sptr + s0 + i);
  for (int i = threadIdx.x; i < held; i += blockDim.x) {
    sm_v[i] = ld_stream(a.val + slot0 + i);
    sm_c[i] = ld_stream(cols + slot0 + i);
  }
  __syncthreads();
  const bool alone = t.b1 - t.b0 == 1;
  if (!alone) gather_range(t, sm_sp, cols, range);

  uint64_t pol = 0;
  if (kSlots == kPolicy) {
    if (t.slices_left > kKeepSlices)
      asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    else
      asm("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(pol));
  }
  double acc[4], tot[4];

  // y = A v for the block's rows, v in a.p (own rows also in sm_p): post(lr,
  // y, v_row, ad, z).  Each slice's loads go out before its first gather.
  auto matvec = [&](auto post) {
    for (int s = s0 + warp; s < s1; s += nw) {
      const int base = sm_sp[s - s0], w = (sm_sp[s - s0 + 1] - base) >> 5;
      const int row = s * kWarp + lane, lr = row - r0;
      if (row >= t.row_end) continue;
      const double pr = kLevel == 3 ? sm_p[lr] : ld_vec(a.p + row);
      const double dg = kLevel == 3 ? sm_d[lr] : __ldcg(a.diag + row);
      const double zr = vz[lr];
      double y;
      if (kSlots == kHold) {
        const I *c = sm_c + (base - slot0) + lane;
        const double *v = sm_v + (base - slot0) + lane;
        y = xmul(dg, pr);
        for (int e0 = 0; e0 < w; e0 += kChunk) {
          double g[kChunk];
#pragma unroll
          for (int u = 0; u < kChunk; ++u)
            if (e0 + u < w) g[u] = ld_vec(a.p + smem_col(c, (e0 + u) * kWarp, row));
#pragma unroll
          for (int u = 0; u < kChunk; ++u)
            if (e0 + u < w) y = xadd(y, xmul(v[(e0 + u) * kWarp], g[u]));
        }
      } else {
        const I *c = cols + base + lane;
        const double *v = a.val + base + lane;
        int jj[kChunk];
        double vv[kChunk];
        auto load = [&](int e0) {
#pragma unroll
          for (int u = 0; u < kChunk; ++u)
            if (e0 + u < w) {
              const int k = (e0 + u) * kWarp;
              const int o = kSlots == kPolicy   ? ld_mat(c + k, pol)
                            : kSlots == kStream ? __ldcs(c + k)
                                                : __ldcg(c + k);
              jj[u] = sizeof(I) == 2 ? row + o : o;
              vv[u] = kSlots == kPolicy   ? ld_mat(v + k, pol)
                      : kSlots == kStream ? __ldcs(v + k)
                                          : __ldcg(v + k);
            }
        };
        load(0);
        y = xmul(dg, pr);
        for (int e0 = 0; e0 < w; e0 += kChunk) {
          if (e0 > 0) load(e0);
#pragma unroll
          for (int u = 0; u < kChunk; ++u)
            if (e0 + u < w) y = xadd(y, xmul(vv[u], ld_vec(a.p + jj[u])));
        }
      }
      post(lr, y, pr, dg, zr);
    }
  };
  auto put_p = [&](int lr, double v) {
    st_vec(a.p + r0 + lr, v);
    if (kLevel == 3) sm_p[lr] = v;
  };
  // p is complete: wait on the blocks whose p this block gathers (a block has
  // at least as many threads as the grid has blocks, so every range fits)
  auto publish = [&]() {
    if (alone) {
      __syncthreads();
      return true;
    }
    return neighbour_wait(a.sync.ticks, a.sync.err, a.sync.spin_limit, ++tick, range[0], range[1]);
  };

  Scalars sc(0.0);
  unsigned j = 0;
  if (!resume) {
    // x0 and (b, M b); p = z = M b, or p = x0 for the product with the start
    acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
    for (int lr = threadIdx.x; lr < own; lr += blockDim.x) {
      const double d = __ldcg(a.diag + r0 + lr), b = ld_vec(a.b + r0 + lr);
      const double z = xdiv(b, d);
      acc[0] += b * z;
      acc[1] += b * b;
      const double x0 = a.newx ? 0.0 : ld_vec(a.x + r0 + lr);
      if (kLevel >= 2 || a.newx) vx[lr] = x0;
      if (kLevel == 3) sm_d[lr] = d;
      vz[lr] = z;
      put_p(lr, a.newx ? z : x0);
    }
    if (!team_sum<4, true>(a.sync, t, epoch, acc, tot, red, bad)) return false;
    sc = Scalars(a.tol * sqrt(fabs(tot[0])));
    sc.bnorm = sqrt(tot[1]);
    if (!a.newx) {
      matvec([&](int lr, double y, double, double d, double) {
        vz[lr] = xdiv(xsub(ld_vec(a.b + r0 + lr), y), d);
      });
      // every gather of x0 is done
      if (!team_sum<4, false>(a.sync, t, epoch, acc, tot, red, bad)) return false;
      for (int lr = threadIdx.x; lr < own; lr += blockDim.x) put_p(lr, vz[lr]);
      if (!publish()) return false;
    }
  } else {
    sc = Scalars(__ldcg(&st->conv));
    sc.bnorm = __ldcg(&st->bnorm);
    sc.nu_old = __ldcg(&st->nu_old);
    j = __ldcg(&st->j);
    for (int lr = threadIdx.x; lr < own; lr += blockDim.x) {
      if (kLevel >= 1) vz[lr] = ld_vec(a.z + r0 + lr);
      if (kLevel >= 2) vx[lr] = ld_vec(a.x + r0 + lr);
      if (kLevel == 3) {
        sm_d[lr] = __ldcg(a.diag + r0 + lr);
        sm_p[lr] = ld_vec(a.p + r0 + lr);
      }
    }
    __syncthreads();
  }

  const unsigned stop = j + min(cap, 0xffffffffu - j);
  for (;; ++j) {
    acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
    matvec([&](int lr, double y, double p, double d, double z) {
      const double mq = xdiv(y, d);
      sm_t[lr] = mq;
      acc[0] += y * p;
      acc[1] += y * z;
      acc[2] += y * mq;
      acc[3] += (d * z) * z;
    });
    if (!team_sum<4, false>(a.sync, t, epoch, acc, tot, red, bad)) return false;
    if (!sc.next(tot, j, a.maxit)) break;
    const double alpha = sc.alpha, beta = sc.beta;
    for (int lr = threadIdx.x; lr < own; lr += blockDim.x) {
      const double p = kLevel == 3 ? sm_p[lr] : ld_vec(a.p + r0 + lr);
      const double z = xsub(vz[lr], xmul(alpha, sm_t[lr]));
      vz[lr] = z;
      vx[lr] = xadd(vx[lr], xmul(alpha, p));
      put_p(lr, xadd(z, xmul(beta, p)));
    }
    if (!publish()) return false;
    if (st && j + 1 == stop) {  // the round is over: the state goes to global memory
      for (int lr = threadIdx.x; lr < own; lr += blockDim.x) {
        if (kLevel >= 1) st_vec(a.z + r0 + lr, vz[lr]);
        if (kLevel >= 2) st_vec(a.x + r0 + lr, vx[lr]);
      }
      if (static_cast<int>(blockIdx.x) == t.b0 && threadIdx.x == 0) {
        st->conv = sc.conv;
        st->bnorm = sc.bnorm;
        st->nu_old = sc.nu_old;
        st->j = j + 1;
        if (!resume) st->t0 = t.t0;
        rt->put_iters(t.sys, t.round, j + 1);
      }
      return false;
    }
  }

  // xKx, ||x||, ||b - Ax||_M, ||b - Ax||  (Cg.c:155-176), with x in p's place
  for (int lr = threadIdx.x; lr < own; lr += blockDim.x) {
    const double x = vx[lr];
    if (kLevel >= 2) st_vec(a.x + r0 + lr, x);
    put_p(lr, x);
  }
  if (!publish()) return false;
  acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
  matvec([&](int lr, double y, double x, double d, double) {
    const double r = xsub(ld_vec(a.b + r0 + lr), y);
    acc[0] += x * y;
    acc[1] += x * x;
    acc[2] += r * xdiv(r, d);
    acc[3] += r * r;
  });
  if (!team_sum<4, false>(a.sync, t, epoch, acc, tot, red, bad)) return false;
  if (static_cast<int>(blockIdx.x) == t.b0 && threadIdx.x == 0)
    put_result(a.out + t.sys, sc, tot, (global_ns() - (resume ? st->t0 : t.t0)) * 1e-6);
  return true;
}

// One system over the whole grid.
template <typename I, int kLevel, Slots kSlots>
__global__ void __launch_bounds__(kGridThreads, 1) pcg_grid_kernel(const ChipArgs a) {
  extern __shared__ double sm_dyn[];
  __shared__ TeamShared sh;
  TeamPart t{};
  block_slices(a.nslices, &t.s0, &t.s1);
  t.count = a.nslices;
  t.b1 = gridDim.x;
  t.row_end = a.n;
  t.t0 = global_ns();
  (void)pcg_grid_body<I, kLevel, kSlots>(a, t, sm_dyn, sh, 0u, 0u, nullptr, nullptr, false,
                                          0xffffffffu);
}

// Many systems, a team of blocks each, in rounds (team_sync.cuh).  A block
// picks its level by its own rows: blocks of one team need not agree, they
// only exchange sums and p.

template <typename I, int kT>
__global__ void __launch_bounds__(kT, kGridThreads / kT)
    pcg_team_kernel(const ChipArgs a, const TeamTable tt, const RoundTable rt, ChipState *states,
                    int smem) {
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
  if (t.b1 > t.b0) {
    const unsigned base = round_base(round), cap = round_cap(rt, t, round);
    ChipState *st = states + t.sys;
    const int slices = t.s1 - t.s0, rows = slices * kWarp;
    const int left = smem - 4 * (slices + 1);
    const int slots = __ldg(a.sptr + t.s1) - __ldg(a.sptr + t.s0);
    if (block_fits(rows, level_bytes(3), slots, 8 + sizeof(I), left))
      over = pcg_grid_body<I, 3, kHold>(a, t, sm_dyn, sh, base, base, st, &rt,
                                        round > 0, cap);
    else if (block_fits(rows, level_bytes(2), 0, 0, left))
      over = pcg_grid_body<I, 2, kPolicy>(a, t, sm_dyn, sh, base, base, st, &rt,
                                        round > 0, cap);
    else
      over = pcg_grid_body<I, 0, kPolicy>(a, t, sm_dyn, sh, base, base, st, &rt,
                                        round > 0, cap);
  }
  __syncthreads();
  end_round(rt, t, over && static_cast<int>(blockIdx.x) == t.b0);
}

// ---- cluster form --------------------------------------------------------

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ unsigned mapa(unsigned addr, unsigned rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ double ld_cluster(unsigned addr) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}

constexpr int kMaxCluster = 16;
constexpr int kClusterThreads = 512;  // 100 registers a thread

// Totals of four values over the cluster, in every thread, the same bits in
// all blocks: each block's totals go into every block's ex[buf][rank], and
// the cluster barrier publishes them (and, as a barrier, every other shared
// and global write of the cluster before it).  ex: two alternating buffers of
// 16 * 4 doubles, zeroed for the ranks the cluster does not have.
__device__ __forceinline__ void cluster_sum4(double *ex, unsigned &buf, const double (&acc)[4],
                                             double (&tot)[4], double *sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  buf ^= 1u;
  double *cur = ex + buf * (kMaxCluster * 4);
  const double s = block_sum_n<4>(acc, sm);
  if (warp == 0) {
    // lane l holds value l >> 3; it stores it into ranks l & 7 and 8 + (l & 7)
    const unsigned dst = smem_u32(cur + blockIdx.x * 4 + (lane >> 3));
    for (unsigned r = lane & 7; r < gridDim.x; r += 8) st_cluster(mapa(dst, r), s);
  }
  cluster_sync_all();
  // lane l sums value l & 3 over ranks (l >> 2) and 8 + (l >> 2)
  double t = cur[lane] + cur[32 + lane];
  t += __shfl_xor_sync(0xffffffffu, t, 4);
  t += __shfl_xor_sync(0xffffffffu, t, 8);
  t += __shfl_xor_sync(0xffffffffu, t, 16);
#pragma unroll
  for (int i = 0; i < 4; ++i) tot[i] = __shfl_sync(0xffffffffu, t, i);
}

// Bytes of a block: z, M q, M, p and, when `vecs`, x and ad; its slots'
// values and gather addresses; its slice pointers.
size_t cluster_smem(int rows, int64_t slots, int slices, bool vecs) {
  return static_cast<size_t>(rows) * (vecs ? 48 : 32) + static_cast<size_t>(slots) * 12 +
         sizeof(int) * (static_cast<size_t>(slices) + 1);
}

template <bool kVecs>
__global__ void __launch_bounds__(kClusterThreads, 1) pcg_cluster_kernel(const ChipArgs a) {
  extern __shared__ double sm_dyn[];
  __shared__ double red[32 * 4], ex[2 * kMaxCluster * 4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  int s0, s1;
  block_slices(a.nslices, &s0, &s1);
  const int r0 = s0 * kWarp, rows = (s1 - s0) * kWarp;
  const int own = max(0, min(rows, a.n - r0));
  const int slot0 = __ldg(a.sptr + s0), nslots = __ldg(a.sptr + s1) - slot0;
  // every block lays p out at the same offset, so a column's address in its
  // owner follows from the owner's rank alone
  double *sm_p = sm_dyn;
  const int maxrows = ((a.nslices + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x)) * kWarp;
  double *sm_z = sm_p + maxrows, *sm_t = sm_z + rows, *sm_m = sm_t + rows;
  double *sm_x = sm_m + rows, *sm_d = sm_x + rows;
  double *sm_v = kVecs ? sm_d + rows : sm_x;
  unsigned *sm_c = reinterpret_cast<unsigned *>(sm_v + nslots);
  int *sm_sp = reinterpret_cast<int *>(sm_c + nslots);
  const unsigned p_base = smem_u32(sm_p);
  for (int i = threadIdx.x; i < 2 * kMaxCluster * 4; i += blockDim.x) ex[i] = 0.0;
  for (int i = threadIdx.x; i <= s1 - s0; i += blockDim.x) sm_sp[i] = __ldg(a.sptr + s0 + i) - slot0;
  for (int i = threadIdx.x; i < nslots; i += blockDim.x) {
    sm_v[i] = ld_stream(a.val + slot0 + i);
    const int c = ld_stream(a.col + slot0 + i);
    const int o = owner_block(c, a.nslices);
    const int first = static_cast<int>((static_cast<long long>(a.nslices) * o) / gridDim.x);
    sm_c[i] = mapa(p_base + 8u * static_cast<unsigned>(c - first * kWarp),
                   static_cast<unsigned>(o));
  }
  double acc[4], tot[4];
  unsigned buf = 0;
  auto diag_at = [&](int lr) { return kVecs ? sm_d[lr] : __ldg(a.diag + r0 + lr); };
  auto matvec = [&](auto post) {
    for (int s = warp; s < s1 - s0; s += nw) {
      const int base = sm_sp[s], w = (sm_sp[s + 1] - base) >> 5;
      const int lr = s * kWarp + lane;
      if (lr >= own) continue;
      const double pr = sm_p[lr], dg = diag_at(lr);
      const unsigned *c = sm_c + base + lane;
      const double *v = sm_v + base + lane;
      double y = xmul(dg, pr);
      for (int e0 = 0; e0 < w; e0 += kChunk) {
        double g[kChunk];
#pragma unroll
        for (int u = 0; u < kChunk; ++u)
          if (e0 + u < w) g[u] = ld_cluster(c[(e0 + u) * kWarp]);
#pragma unroll
        for (int u = 0; u < kChunk; ++u)
          if (e0 + u < w) y = xadd(y, xmul(v[(e0 + u) * kWarp], g[u]));
      }
      post(lr, y, pr, dg);
    }
  };

  acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
  for (int lr = threadIdx.x; lr < own; lr += blockDim.x) {
    const double d = __ldg(a.diag + r0 + lr), b = ld_vec(a.b + r0 + lr);
    const double m = xdiv(1.0, d), z = xmul(b, m);
    acc[0] += b * z;
    acc[1] += b * b;
    const double x0 = a.newx ? 0.0 : ld_vec(a.x + r0 + lr);
    if (kVecs) {
      sm_x[lr] = x0;
      sm_d[lr] = d;
    } else if (a.newx) {
      a.x[r0 + lr] = 0.0;
    }
    sm_m[lr] = m;
    sm_z[lr] = z;
    sm_p[lr] = a.newx ? z : x0;
  }
  cluster_sync_all();  // ex is zero in every block before the first exchange
  cluster_sum4(ex, buf, acc, tot, red);
  Scalars sc(a.tol * sqrt(fabs(tot[0])));
  sc.bnorm = sqrt(tot[1]);
  if (!a.newx) {
    matvec([&](int lr, double y, double, double) {
      sm_z[lr] = xmul(xsub(ld_vec(a.b + r0 + lr), y), sm_m[lr]);
    });
    cluster_sync_all();  // every gather of x0 is done
    for (int lr = threadIdx.x; lr < own; lr += blockDim.x) sm_p[lr] = sm_z[lr];
    cluster_sync_all();
  }

  for (unsigned j = 0;; ++j) {
    acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
    matvec([&](int lr, double y, double p, double d) {
      const double z = sm_z[lr], t = xmul(y, sm_m[lr]);
      sm_t[lr] = t;
      acc[0] += y * p;
      acc[1] += y * z;
      acc[2] += y * t;
      acc[3] += (d * z) * z;
    });
    cluster_sum4(ex, buf, acc, tot, red);
    if (!sc.next(tot, j, a.maxit)) break;
    const double alpha = sc.alpha, beta = sc.beta;
    for (int lr = threadIdx.x; lr < own; lr += blockDim.x) {
      const double p = sm_p[lr];
      const double z = xsub(sm_z[lr], xmul(alpha, sm_t[lr]));
      sm_z[lr] = z;
      if (kVecs)
        sm_x[lr] = xadd(sm_x[lr], xmul(alpha, p));
      else
        a.x[r0 + lr] = xadd(a.x[r0 + lr], xmul(alpha, p));
      sm_p[lr] = xadd(z, xmul(beta, p));
    }
    cluster_sync_all();
  }

  for (int lr = threadIdx.x; lr < own; lr += blockDim.x) {
    const double x = kVecs ? sm_x[lr] : a.x[r0 + lr];
    if (kVecs) a.x[r0 + lr] = x;
    sm_p[lr] = x;
  }
  cluster_sync_all();
  acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
  matvec([&](int lr, double y, double x, double d) {
    const double r = xsub(ld_vec(a.b + r0 + lr), y);
    acc[0] += x * y;
    acc[1] += x * x;
    acc[2] += r * xdiv(r, d);
    acc[3] += r * r;
  });
  cluster_sum4(ex, buf, acc, tot, red);
  if (blockIdx.x == 0 && threadIdx.x == 0) put_result(a.out, sc, tot, 0.0);
}

// ---- host ------------------------------------------------------------------

int smem_optin(int device) {
  int v = 0;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess)
    return 0;
  return v;
}

// static shared memory of the kernels (reductions, exchange buffers), rounded up
constexpr size_t kGridStatic = 1536, kClusterStatic = 2304;

struct Shape {
  const void *kern = nullptr;
  int grid = 0, threads = 0;
  size_t smem = 0;
  bool cluster = false;
};

cudaLaunchConfig_t cluster_config(const Shape &sh, cudaLaunchAttribute *at, cudaStream_t st) {
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = static_cast<unsigned>(sh.grid);
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(sh.grid);
  cfg.blockDim = dim3(sh.threads);
  cfg.dynamicSmemBytes = sh.smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

// Allows a kernel all the shared memory its form may ask for, and a cluster
// kernel sixteen blocks; false where the device refuses or cannot hold such
// a cluster.  Asked once per kernel and device.
bool ready(const Shape &sh, int device) {
  static std::mutex mu;
  static std::map<std::pair<const void *, int>, bool> known;
  std::lock_guard<std::mutex> lk(mu);
  const auto key = std::make_pair(sh.kern, device);
  const auto it = known.find(key);
  if (it != known.end()) return it->second;
  const int bytes = smem_optin(device) - static_cast<int>(sh.cluster ? kClusterStatic : kGridStatic);
  bool ok = cudaFuncSetAttribute(sh.kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) ==
            cudaSuccess;
  if (ok && sh.cluster) {
    ok = cudaFuncSetAttribute(sh.kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
         cudaSuccess;
    Shape most = sh;
    most.grid = kMaxCluster;
    most.threads = kClusterThreads;
    most.smem = static_cast<size_t>(bytes);
    cudaLaunchAttribute at{};
    const cudaLaunchConfig_t cfg = cluster_config(most, &at, nullptr);
    int n = 0;
    ok = ok && cudaOccupancyMaxActiveClusters(&n, sh.kern, &cfg) == cudaSuccess && n > 0;
  }
  if (!ok) (void)cudaGetLastError();  // the refusal is not a later call's error
  known[key] = ok;
  return ok;
}

// Cluster form: eight SELL slices (256 rows) a block until sixteen blocks
// share the system, then more a block, up to kClusterSlices.  Past that the
// sixteen SMs' arithmetic costs more than the grid form's slower exchange:
// 24^3 (27 slices a block) 3.12 us an iteration against 3.75, 28^3 (43) 3.75
// against 4.08, 32^3 (64) 5.8 against 4.26.
// Without numbering (DevSell::far) most gathers go to other blocks, lane by
// lane: up to eight slices a block only.  16^3 cells in random order 5.3 us an
// iteration in the cluster and 3.9 in the grid form, 20^3 7.6 and 4.7, 24^3 11.0
// and 4.9, 29^3 16.9 and 5.6 (in order 3.9 and 4.4); 10^3 to 14^3 as good.
constexpr int kClusterBlockSlices = 8, kClusterSlices = 48;

bool cluster_shape(const sfr_system *s, Shape *sh) {
  const int ns = s->A.nslices;
  int c = 1;
  while (c < kMaxCluster && (ns + c - 1) / c > kClusterBlockSlices) c *= 2;
  const int slices = (ns + c - 1) / c, rows = slices * kWarp;
  if (slices > (s->A.far() ? kClusterBlockSlices : kClusterSlices)) return false;
  const size_t limit = static_cast<size_t>(smem_optin(s->device)) - kClusterStatic;
  for (bool vecs : {true, false}) {
    const size_t b = cluster_smem(rows, static_cast<int64_t>(rows) * s->A.max_width, slices, vecs);
    if (b > limit) continue;
    *sh = Shape{vecs ? reinterpret_cast<const void *>(pcg_cluster_kernel<true>)
                     : reinterpret_cast<const void *>(pcg_cluster_kernel<false>),
                c, std::min(kClusterThreads, rows), b, true};
    return ready(*sh, s->device);
  }
  return false;
}

// Grid form.  A block an SM, and at least sixteen slices a block: fewer
// blocks make the exchange cheaper than the idle SMs cost (32^3 4.26 us an
// iteration on 64 blocks, 4.69 on 128).
constexpr int kGridBlockSlices = 16;
// Levels 2 and 3 up to this much shared memory a block, level 1 up to the
// second: what they leave is the L1 the gathers of p live in.  108^3: level 2
// with 204 KB 26.6 us an iteration, level 1 with 136 KB 22.4; 88^3: level 3
// with 184 KB 10.75, level 2 11.04; 120^3: level 1 with 187 KB 28.9, level 0
// 33.7; 128^3: level 1 with 227 KB 41.5, level 0 41.1.
constexpr size_t kLevelSmem[kLevels] = {size_t(-1), 216 << 10, 192 << 10, 192 << 10};
// Slots up to this many bytes stay in L2 between iterations (half of its 126
// MB: a line read from both dies lies in both halves).  104^3 (67 MB): 17.8
// us an iteration kept, 18.6 streamed; 108^3 (76 MB): 25.2 and 22.4.
constexpr int64_t kKeepBytes = 70 << 20;

template <typename I>
bool grid_shape(const sfr_system *s, Shape *sh) {
  const int ns = s->A.nslices;
  const size_t limit = static_cast<size_t>(smem_optin(s->device)) - kGridStatic;
  const int g = std::max(1, std::min(num_sms(s->device),
                                     (ns + kGridBlockSlices - 1) / kGridBlockSlices));
  const int slices = (ns + g - 1) / g, rows = slices * kWarp;
  const int threads = std::max((g + kWarp - 1) / kWarp * kWarp, std::min(kGridThreads, rows));
  auto fixed = [&](int level) {
    return static_cast<size_t>(rows) * level_bytes(level) + sizeof(int) * (slices + 1);
  };
  const size_t hold = fixed(3) + static_cast<size_t>(rows) * s->A.max_width * (8 + sizeof(I));
  if (hold <= limit) {
    *sh = Shape{reinterpret_cast<const void *>(pcg_grid_kernel<I, 3, kHold>), g, threads, hold,
                false};
    return true;
  }
  int level = kLevels - 1;
  while (level >= 0 && fixed(level) > std::min(limit, kLevelSmem[level])) --level;
  if (level < 0) return false;
  static const void *const kerns[2][kLevels] = {
      {reinterpret_cast<const void *>(pcg_grid_kernel<I, 0, kKeep>),
       reinterpret_cast<const void *>(pcg_grid_kernel<I, 1, kKeep>),
       reinterpret_cast<const void *>(pcg_grid_kernel<I, 2, kKeep>),
       reinterpret_cast<const void *>(pcg_grid_kernel<I, 3, kKeep>)},
      {reinterpret_cast<const void *>(pcg_grid_kernel<I, 0, kStream>),
       reinterpret_cast<const void *>(pcg_grid_kernel<I, 1, kStream>),
       reinterpret_cast<const void *>(pcg_grid_kernel<I, 2, kStream>),
       reinterpret_cast<const void *>(pcg_grid_kernel<I, 3, kStream>)}};
  const bool keep = s->A.nslots * static_cast<int64_t>(8 + sizeof(I)) <= kKeepBytes;
  *sh = Shape{kerns[keep ? 0 : 1][level], g, threads, fixed(level), false};
  return true;
}

size_t align256(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }

const void *team_kernel(const sfr_system *s, int per_sm) {
  if (per_sm == 1)
    return s->A.off ? reinterpret_cast<const void *>(pcg_team_kernel<int16_t, kGridThreads>)
                    : reinterpret_cast<const void *>(pcg_team_kernel<int, kGridThreads>);
  return s->A.off ? reinterpret_cast<const void *>(pcg_team_kernel<int16_t, kGridThreads / 2>)
                  : reinterpret_cast<const void *>(pcg_team_kernel<int, kGridThreads / 2>);
}

}  // namespace

// The model: 16 boxes of 16^3 on 9 blocks each (14 slices a block) 5.5 us an
// iteration, 32^3 (111 slices) 11.0, 48^3 (375) 36.8; a block alone with 16
// slices 2.4.
TeamShape team_shape_onchip(const sfr_system *s, int per_sm) {
  return team_shape(s->device, team_kernel(s, per_sm), kGridThreads / per_sm, per_sm,
                    kWarp * level_bytes(0) + 4, TeamModel{0.9f, 4.5f, 0.1f}, s->A.far());
}

size_t team_ws_bytes_onchip(int n, int grid, int nsys) {
  return align256((sizeof(ChipState) + kRoundInts * sizeof(int)) * static_cast<size_t>(nsys)) +
         2 * align256(sizeof(double) * static_cast<size_t>(n)) +
         align256(sizeof(TeamSlot) * 2 * static_cast<size_t>(grid)) +
         align256(64 * static_cast<size_t>(grid));
}

int graph_team_onchip(sfr_system *s, const double *d_b, double *d_x, double tol, uint32_t maxit,
                      int32_t newx, const TeamPlan &plan, void *ws, SolveOut *d_out,
                      unsigned *ctl, cudaGraph_t *graph) {
  const size_t vec = align256(sizeof(double) * static_cast<size_t>(s->n));
  const size_t slot_b = align256(sizeof(TeamSlot) * 2 * static_cast<size_t>(plan.grid));
  const size_t tick_b = align256(64 * static_cast<size_t>(plan.grid));
  const size_t state_b =
      align256((sizeof(ChipState) + kRoundInts * sizeof(int)) * static_cast<size_t>(plan.nsys));
  char *base = static_cast<char *>(ws);
  ChipArgs a{};
  a.n = s->n;
  a.nslices = s->A.nslices;
  a.sptr = s->A.sptr;
  a.col = s->A.col;
  a.off = s->A.off;
  a.val = s->A.val;
  a.diag = s->d_diag;
  a.b = d_b;
  a.x = d_x;
  a.sync.slots = reinterpret_cast<TeamSlot *>(base);
  a.sync.ticks = reinterpret_cast<unsigned *>(base + slot_b);
  a.sync.err = reinterpret_cast<int *>(ctl + 2);
  a.sync.spin_limit = 1u << 22;
  ChipState *states = reinterpret_cast<ChipState *>(base + slot_b + tick_b);
  RoundTable rt = round_table(plan, reinterpret_cast<int *>(states + plan.nsys), ctl);
  a.p = reinterpret_cast<double *>(base + slot_b + tick_b + state_b);
  a.z = reinterpret_cast<double *>(base + slot_b + tick_b + state_b + vec);
  a.out = d_out;
  a.tol = tol;
  a.maxit = maxit;
  a.newx = newx;
  int smem = static_cast<int>(plan.shape.smem);
  TeamTable tt = plan.table;
  void *params[] = {&a, &tt, &rt, &states, &smem};
  return rounds_graph(team_kernel(s, plan.shape.per_sm), plan, params, &rt.more, base,
                      slot_b + tick_b + state_b, ctl, graph);
}

int solve_onchip(sfr_system *s, const double *d_diag, const double *d_b, double *d_x, double tol,
                 uint32_t maxit, int32_t newx, cudaStream_t st, sfr_solve_info *info) {
  if (maxit == 0) return SFR_UNSUPPORTED;
  Shape sh;
  if (!cluster_shape(s, &sh) &&
      !(s->A.off ? grid_shape<int16_t>(s, &sh) : grid_shape<int>(s, &sh)))
    return SFR_UNSUPPORTED;
  if (!ready(sh, s->device)) return SFR_UNSUPPORTED;

  auto align = [](size_t v) { return (v + 255) & ~static_cast<size_t>(255); };
  const size_t vec = align(sizeof(double) * static_cast<size_t>(s->A.nslices) * kWarp);
  const size_t slot_b = align(sizeof(TeamSlot) * 2 * static_cast<size_t>(sh.grid));
  const size_t tick_b = align(64 * static_cast<size_t>(sh.grid)) + 256;  // + the error word
  const size_t out_b = align(sizeof(SolveOut));
  // x is written while b and the diagonal are still read: where a caller's x
  // overlaps one of them, it gets a copy
  const size_t nb = sizeof(double) * static_cast<size_t>(s->n);
  const auto under_x = [&](const double *p) {
    const uintptr_t xb = reinterpret_cast<uintptr_t>(d_x), pb = reinterpret_cast<uintptr_t>(p);
    return p && xb < pb + nb && pb < xb + nb;
  };
  const bool overlap = under_x(d_b), overlap_d = under_x(d_diag);
  int rc = ensure_workspace(s, (sh.cluster ? 0 : 2 * vec + slot_b + tick_b) + out_b +
                                   (overlap ? vec : 0) + (overlap_d ? vec : 0));
  if (rc != SFR_OK) return rc;
  char *base = static_cast<char *>(s->ws.base);

  ChipArgs a{};
  a.n = s->n;
  a.nslices = s->A.nslices;
  a.sptr = s->A.sptr;
  a.col = s->A.col;
  a.off = s->A.off;
  a.val = s->A.val;
  a.diag = d_diag ? d_diag : s->d_diag;
  a.b = d_b;
  a.x = d_x;
  a.tol = tol;
  a.maxit = maxit;
  a.newx = newx;
  a.sync.spin_limit = 1u << 22;
  SolveOut *dev_out = reinterpret_cast<SolveOut *>(base);
  base += out_b;
  if (overlap) {
    if (cudaMemcpyAsync(base, d_b, nb, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
      return SFR_CUDA_ERROR;
    a.b = reinterpret_cast<double *>(base);
    base += vec;
  }
  if (overlap_d) {
    if (cudaMemcpyAsync(base, d_diag, nb, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
      return SFR_CUDA_ERROR;
    a.diag = reinterpret_cast<double *>(base);
    base += vec;
  }
  if (!sh.cluster) {
    a.sync.slots = reinterpret_cast<TeamSlot *>(base);
    a.sync.ticks = reinterpret_cast<unsigned *>(base + slot_b);
    a.sync.err = reinterpret_cast<int *>(base + slot_b + tick_b - 256);
    a.p = reinterpret_cast<double *>(base + slot_b + tick_b);
    a.z = reinterpret_cast<double *>(base + slot_b + tick_b + vec);
    if (cudaMemsetAsync(base, 0, slot_b + tick_b, st) != cudaSuccess) return SFR_CUDA_ERROR;
  }
  if (!s->ev0 && cudaEventCreate(&s->ev0) != cudaSuccess) return SFR_CUDA_ERROR;
  if (!s->ev1 && cudaEventCreate(&s->ev1) != cudaSuccess) return SFR_CUDA_ERROR;
  ResultRecord rec;
  a.out = rec.r ? rec.r : dev_out;
  // stays when a wait gave up and the kernel left without a result
  SolveOut out{};
  out.status = SFR_TIMEOUT;
  if (rec.r)
    *rec.r = out;
  else if (cudaMemcpyAsync(dev_out, &out, sizeof(out), cudaMemcpyHostToDevice, st) != cudaSuccess)
    return SFR_CUDA_ERROR;
  void *params[] = {&a};
  cudaError_t ce = cudaEventRecord(s->ev0, st);
  if (ce == cudaSuccess) {
    if (sh.cluster) {
      cudaLaunchAttribute at{};
      const cudaLaunchConfig_t cfg = cluster_config(sh, &at, st);
      ce = cudaLaunchKernelExC(&cfg, sh.kern, params);
    } else {
      ce = cudaLaunchCooperativeKernel(sh.kern, dim3(sh.grid), dim3(sh.threads), params, sh.smem,
                                       st);
    }
  }
  if (ce == cudaSuccess) ce = cudaEventRecord(s->ev1, st);
  if (ce == cudaSuccess && !rec.r)
    ce = cudaMemcpyAsync(&out, dev_out, sizeof(out), cudaMemcpyDeviceToHost, st);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(st);
  float ms = 0.f;
  if (ce == cudaSuccess) cudaEventElapsedTime(&ms, s->ev0, s->ev1);
  if (ce != cudaSuccess) {
    set_last_error(cudaGetErrorString(ce));
    return SFR_CUDA_ERROR;
  }
  if (rec.r) out = *rec.r;
  if (out.status == SFR_TIMEOUT) return SFR_TIMEOUT;
  if (info) {
    std::memset(info, 0, sizeof(*info));
    info->iters = out.iters;
    info->status = out.status;
    info->xKx = out.xKx;
    info->norm_x = out.norm_x;
    info->norm_r = out.norm_r;
    info->norm_r_m = out.norm_r_m;
    info->conv = out.conv;
    info->seconds = ms * 1e-3;
    info->inner_iters = out.inner_iters;
    info->relres = out.bnorm > 0 ? out.norm_r / out.bnorm : 0.0;
  }
  return out.status;
}

}  // namespace sfr
