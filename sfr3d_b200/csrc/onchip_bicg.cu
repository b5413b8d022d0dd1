// On-chip BiCGSTAB: a whole FP64 Jacobi-BiCGSTAB solve (Bicgstab.c:36-230) of
// up to three right-hand sides in one launch, with the blocks' rows of the
// Krylov vectors (and the operator, when it fits) in shared memory and two
// reductions an iteration.
//
// The iteration.  The reference forms its dot products in four places, each
// of which the next vector update waits for.  Here each of the two SpMV
// phases forms every product of the vectors it has at hand:
//   v = A z        (r, r0), (v, r0), (r, r)               [exchange]
//   s = r - alpha v,  z' = M s                            [publish z']
//   t = A z'       (t, s), (t, t), (s, s), (s, r0), (t, r0)  [exchange]
//   r = s - w t,  p = r + beta (p - w v),  z = M p        [publish z]
// The stopping tests on ||s|| and ||r|| and the (r, r0) of alpha use measured
// products, one phase after the reference takes them; only beta's (r', r0) is
// formed ahead of r', as (s, r0) - w (t, r0) (the merged reductions of Yang &
// Brent's improved BiCGSTAB, 2002).  A solve runs one SpMV phase beyond its
// last update.  Every SpMV row and vector update keeps the reference's
// rounding and order.
//
// Device time of a solve (iterations), against the graph engine's five kernels
// an iteration or, below 100,000 rows, the persistent kernel's five barriers:
// 12^3 of 3 systems (3) 47 us, 111 before; 48^3 of 1 (5) 79, 209; 61x47x53 of
// 3 (6) 159, 485; 80^3 of 1 (8) 220, 475; 72^3 of 3 (8) 361, 717.  At 61x47x53
// an iteration is 24 us: two exchanges (16 words a block) of about 3 us, two
// publications of 1 us, the SpMV phases and updates the rest.
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
#include "team_sync.cuh"

namespace sfr {

namespace {

constexpr int kBicgMaxK = 3;
constexpr int kChunk = 3;  // slots of a row loaded before their gathers: six spill 1.3 KB a thread
constexpr int kSumWords = 16;  // words of a block's slot: five products of three systems
// The vectors of a row.  The first four, which the SpMV phases use, are in
// shared memory (kCore); the others join them as far as they fit and are else
// in the block's part of a.vecs.
enum Vec { kVt, kVv, kVr, kVr0, kVp, kVm, kVx, kVecs };
constexpr int kCoreVecs = 4;

template <int K>
struct BicgArgs {
  int n, nslices, npad;
  const int *sptr, *col;
  const int16_t *off;
  const double *val;
  const double *diag[K];
  const double *b;  // [K][n]
  double *x;        // [K][n]
  double *z;        // [K][npad]: what the SpMV phases gather
  double *vecs;     // [npad][kVecs][K], a block's rows together: the vectors not on chip
  int on_chip;      // vectors in shared memory
  ulonglong2 *slots;  // two buffers of kSumWords words a block, zero at launch
  unsigned *ticks;    // 16 words a block, zero at launch (neighbour_wait)
  int *err;
  unsigned spin_limit;
  SolveOut *out[K];
  double tol;
  unsigned maxit;
  int newx;
};

constexpr int bicg_threads(int k) { return k == 1 ? 768 : 512; }

// Totals of NV values over the grid, the same bits in all blocks: each block
// writes its totals with the epoch beside each value, and every block polls
// the words of all, several a thread at a time, so the values arrive with the
// poll (team_sum, with more values than a thread can poll for a block at
// once).  Warp 0 then calls decide(lane) with the totals in fin (shared), and
// what it stores to shared memory is every thread's on return.  Two buffers
// alternate; bounded, and kFence, as team_sum.  sm: NV * 32 doubles.
template <int NV, bool kFence, typename Args, typename F>
__device__ __forceinline__ bool grid_sum(const Args &a, unsigned &epoch, const double (&acc)[NV],
                                         double *fin, double *sm, int *bad, F decide) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int G = gridDim.x;
  ++epoch;
  double s = block_sum_n<NV>(acc, sm);
  if (G > 1) {
    ulonglong2 *cur = a.slots + static_cast<size_t>(epoch & 1u) * G * kSumWords;
    if (warp == 0 && sum_writer<NV>()) {
      if (kFence) cuda::atomic_thread_fence(cuda::memory_order_release, cuda::thread_scope_device);
      st_slot(cur + blockIdx.x * NV + sum_index<NV>(), s, epoch);
    }
    if (threadIdx.x == 0) *bad = 0;
    __syncthreads();  // sm is free again; *bad is 0
    constexpr int kPer = 5;  // words in flight a thread
    const int total = G * NV, step = blockDim.x;  // a multiple of NV: value tid % NV
    double mine = 0.0;
    for (int w0 = threadIdx.x; w0 < total; w0 += kPer * step) {
      double v[kPer];
      cuda::atomic_ref<int, cuda::thread_scope_device> err(*a.err);
      for (unsigned spins = 0;; ++spins) {
        bool all = true;
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
          const int w = w0 + u * step;
          v[u] = 0.0;
          if (w < total) all &= ld_slot(cur + w, &v[u], epoch);
        }
        if (all) break;
        if ((spins & 63u) == 63u && err.load(cuda::memory_order_relaxed) != 0) {
          *bad = 1;
          break;
        }
        if (spins > a.spin_limit) {
          int expected = 0;
          err.compare_exchange_strong(expected, SFR_TIMEOUT, cuda::memory_order_relaxed);
          *bad = 1;
          break;
        }
      }
#pragma unroll
      for (int u = 0; u < kPer; ++u) mine += v[u];
    }
    __syncwarp();
    if (kFence) cuda::atomic_thread_fence(cuda::memory_order_acquire, cuda::thread_scope_device);
#pragma unroll
    for (int o = 16; o >= NV; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
    if (lane < NV) sm[lane * 32 + warp] = mine;
    __syncthreads();
    if (warp == 0) {
      double w[NV];
#pragma unroll
      for (int i = 0; i < NV; ++i) w[i] = lane < nw ? sm[i * 32 + lane] : 0.0;
      s = warp_sum_n<NV>(w);
    }
  }
  if (warp == 0) {
    if (sum_writer<NV>()) fin[sum_index<NV>()] = s;
    __syncwarp();
    decide(lane);
  }
  __syncthreads();
  return G == 1 || *bad == 0;
}

// A system's scalars, in shared memory.
struct BicgScalars {
  double conv, bnorm, alpha, w, rr0, beta;
  int act, status;
  unsigned iters;
  __device__ __forceinline__ void stop(int st, unsigned it) {
    act = 0;
    status = st;
    iters = it;
  }
};

template <int K>
constexpr int kNV1 = K == 1 ? 4 : K == 2 ? 8 : 16;  // three products a system, padded
template <int K>
constexpr int kNV2 = K == 1 ? 8 : 16;               // five

// One block of bicg_threads(K) an SM: 80 registers a thread for one system,
// 128 for three, whose fifteen sums and eighteen gathers in flight need them.
// The scalars live in shared memory: in registers they spilled 2.4 KB.
template <typename I, int K, bool kCore, bool kHold>
__global__ void __launch_bounds__(bicg_threads(K), 1) bicg_grid_kernel(const BicgArgs<K> a) {
  extern __shared__ double sm_dyn[];
  __shared__ double red[kNV2<K> * 32], fin[kNV2<K>];
  __shared__ BicgScalars sc[K];
  __shared__ int bad, range[2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  int s0, s1;
  block_slices(a.nslices, &s0, &s1);
  const int r0 = s0 * kWarp, rows = (s1 - s0) * kWarp;
  const int own = max(0, min(rows, a.n - r0));
  const int slot0 = __ldg(a.sptr + s0);
  const int held = kHold ? __ldg(a.sptr + s1) - slot0 : 0;  // a multiple of 32
  double *sm_v = sm_dyn + static_cast<size_t>(a.on_chip) * K * rows;
  I *sm_c = reinterpret_cast<I *>(sm_v + held);
  int *sm_sp = reinterpret_cast<int *>(sm_c + held);
  double *const gv = a.vecs + static_cast<size_t>(r0) * (kVecs * K);
  auto at = [&](Vec i, int k) -> double * {
    return ((kCore && i < kCoreVecs) || i < a.on_chip ? sm_dyn : gv) + (i * K + k) * rows;
  };
  const I *cols = cols_of<I>(SlotCols{a.col, a.off});
  for (int i = threadIdx.x; i <= s1 - s0; i += blockDim.x) sm_sp[i] = __ldg(a.sptr + s0 + i);
  for (int i = threadIdx.x; i < held; i += blockDim.x) {
    sm_v[i] = ld_stream(a.val + slot0 + i);
    sm_c[i] = ld_stream(cols + slot0 + i);
  }
  __syncthreads();
  const bool alone = gridDim.x == 1;
  if (!alone) {
    TeamPart t{};
    t.s0 = s0;
    t.s1 = s1;
    t.count = a.nslices;
    t.b1 = gridDim.x;
    t.row_end = a.n;
    gather_range(t, sm_sp, cols, range);
  }
  unsigned epoch = 0, tick = 0;

  // y_k = A z_k of the block's rows: post(lr, k, y, z)
  auto matvec = [&](auto post) {
    for (int s = s0 + warp; s < s1; s += nw) {
      const int base = sm_sp[s - s0], w = (sm_sp[s - s0 + 1] - base) >> 5;
      const int row = s * kWarp + lane, lr = row - r0;
      if (row >= a.n) continue;
      const I *c = (kHold ? sm_c + (base - slot0) : cols + base) + lane;
      const double *v = (kHold ? sm_v + (base - slot0) : a.val + base) + lane;
      double y[K], zr[K];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        zr[k] = ld_vec(a.z + static_cast<size_t>(k) * a.npad + row);
        y[k] = xmul(__ldcg(a.diag[k] + row), zr[k]);
      }
      for (int e0 = 0; e0 < w; e0 += kChunk) {
        int jj[kChunk];
        double vv[kChunk], g[K][kChunk];
#pragma unroll
        for (int u = 0; u < kChunk; ++u)
          if (e0 + u < w) {
            const int o = kHold ? c[(e0 + u) * kWarp] : __ldcg(c + (e0 + u) * kWarp);
            jj[u] = sizeof(I) == 2 ? row + o : o;
            vv[u] = kHold ? v[(e0 + u) * kWarp] : __ldcg(v + (e0 + u) * kWarp);
          }
#pragma unroll
        for (int u = 0; u < kChunk; ++u)
          if (e0 + u < w) {
#pragma unroll
            for (int k = 0; k < K; ++k)
              g[k][u] = ld_vec(a.z + static_cast<size_t>(k) * a.npad + jj[u]);
          }
#pragma unroll
        for (int u = 0; u < kChunk; ++u)
          if (e0 + u < w) {
#pragma unroll
            for (int k = 0; k < K; ++k) y[k] = xadd(y[k], xmul(vv[u], g[k][u]));
          }
      }
#pragma unroll
      for (int k = 0; k < K; ++k) post(lr, k, y[k], zr[k]);
    }
  };
  auto put_z = [&](int k, int lr, double v) {
    st_vec(a.z + static_cast<size_t>(k) * a.npad + r0 + lr, v);
  };
  // z is complete: wait on the blocks whose z this block gathers (a block has
  // at least as many threads as the grid has blocks, so every range fits)
  auto publish = [&]() {
    if (alone) {
      __syncthreads();
      return true;
    }
    return neighbour_wait(a.ticks, a.err, a.spin_limit, ++tick, range[0], range[1]);
  };

  auto active = [&]() {
    int any = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) any |= sc[k].act;
    return any != 0;
  };
  // conv = tol ||b|| (Bicgstab.c:72-80); r0 = r = p = b - A x, z = M p
  // (Bicgstab.c:83-99)
  {
    double acc[kNV1<K>] = {};
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll 1
      for (int lr = threadIdx.x; lr < own; lr += blockDim.x) {
        const size_t i = static_cast<size_t>(k) * a.n + r0 + lr;
        const double m = 1.0 / __ldcg(a.diag[k] + r0 + lr), b = ld_vec(a.b + i);
        const double x0 = a.newx ? 0.0 : ld_vec(a.x + i);
        acc[k] += b * b;
        at(kVm, k)[lr] = m;
        at(kVx, k)[lr] = x0;
        if (a.newx) at(kVr0, k)[lr] = at(kVr, k)[lr] = at(kVp, k)[lr] = b;
        put_z(k, lr, a.newx ? xmul(b, m) : x0);
      }
    const auto start = [&](int k) {
      if (k >= K) return;
      sc[k] = BicgScalars{};
      sc[k].bnorm = sqrt(fin[k]);
      sc[k].conv = a.tol * sc[k].bnorm;
      sc[k].act = 1;
    };
    if (!grid_sum<kNV1<K>, true>(a, epoch, acc, fin, red, &bad, start)) return;
    if (!a.newx) {
      matvec([&](int lr, int k, double y, double) {
        const double r = xsub(ld_vec(a.b + static_cast<size_t>(k) * a.n + r0 + lr), y);
        at(kVr0, k)[lr] = at(kVr, k)[lr] = at(kVp, k)[lr] = r;
      });
      // every gather of x0 is done
      if (!grid_sum<kNV1<K>, false>(a, epoch, acc, fin, red, &bad, [](int) {})) return;
#pragma unroll
      for (int k = 0; k < K; ++k)
#pragma unroll 1
        for (int lr = threadIdx.x; lr < own; lr += blockDim.x)
          put_z(k, lr, xmul(at(kVr, k)[lr], at(kVm, k)[lr]));
      if (!publish()) return;
    }
  }
  for (unsigned j = 0;; ++j) {
    // v = A z ; alpha = (r, r0) / (v, r0)  (Bicgstab.c:105-113)
    {
      double acc[kNV1<K>] = {};
      matvec([&](int lr, int k, double y, double) {
        const double r = at(kVr, k)[lr], q = at(kVr0, k)[lr];
        at(kVv, k)[lr] = y;
        acc[3 * k] += r * q;
        acc[3 * k + 1] += y * q;
        acc[3 * k + 2] += r * r;
      });
      const auto decide = [&](int k) {
        if (k >= K || !sc[k].act) return;
        BicgScalars &c = sc[k];
        if (j > 0) {  // iteration j - 1's end (Bicgstab.c:145-165)
          if (sqrt(fin[3 * k + 2]) < c.conv) return c.stop(SFR_OK, j);
          if (!isfinite(c.beta)) return c.stop(SFR_BREAKDOWN, j);
        }
        c.rr0 = fin[3 * k];
        c.alpha = c.rr0 / fin[3 * k + 1];
        if (j >= a.maxit)
          c.stop(SFR_MAXIT, j + 1);
        else if (!isfinite(c.alpha))
          c.stop(SFR_BREAKDOWN, j + 1);
      };
      if (!grid_sum<kNV1<K>, false>(a, epoch, acc, fin, red, &bad, decide)) return;
      if (!active()) break;
    }
    // x += alpha z ; s = r -= alpha v ; z = M s  (Bicgstab.c:116-133)
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (sc[k].act) {
        double *const x = at(kVx, k), *const r = at(kVr, k);
        const double *const v = at(kVv, k), *const m = at(kVm, k);
        const double alpha = sc[k].alpha;
#pragma unroll 1
        for (int lr = threadIdx.x; lr < own; lr += blockDim.x) {
          const double z = ld_vec(a.z + static_cast<size_t>(k) * a.npad + r0 + lr);
          const double s = xsub(r[lr], xmul(alpha, v[lr]));
          x[lr] = xadd(x[lr], xmul(alpha, z));
          r[lr] = s;
          put_z(k, lr, xmul(s, m[lr]));
        }
      }
    if (!publish()) return;
    // t = A z ; ||s|| ; w = (t, s) / (t, t)  (Bicgstab.c:116-142)
    {
      double acc[kNV2<K>] = {};
      matvec([&](int lr, int k, double y, double) {
        const double s = at(kVr, k)[lr], q = at(kVr0, k)[lr];
        at(kVt, k)[lr] = y;
        acc[5 * k] += y * s;
        acc[5 * k + 1] += y * y;
        acc[5 * k + 2] += s * s;
        acc[5 * k + 3] += s * q;
        acc[5 * k + 4] += y * q;
      });
      const auto decide = [&](int k) {
        if (k >= K || !sc[k].act) return;
        BicgScalars &c = sc[k];
        c.w = fin[5 * k] / fin[5 * k + 1];
        c.beta = ((fin[5 * k + 3] - c.w * fin[5 * k + 4]) / c.rr0) * (c.alpha / c.w);
        if (sqrt(fin[5 * k + 2]) < c.conv)
          c.stop(SFR_OK, j + 1);
        else if (!isfinite(c.w))
          c.stop(SFR_BREAKDOWN, j + 1);
      };
      if (!grid_sum<kNV2<K>, false>(a, epoch, acc, fin, red, &bad, decide)) return;
      if (!active()) break;
    }
    // x += w z ; r -= w t ; p = r + beta (p - w v) ; z = M p
    // (Bicgstab.c:145-176)
#pragma unroll
    for (int k = 0; k < K; ++k)
      if (sc[k].act) {
        double *const x = at(kVx, k), *const r = at(kVr, k), *const p = at(kVp, k);
        const double *const v = at(kVv, k), *const t = at(kVt, k), *const m = at(kVm, k);
        const double w = sc[k].w, beta = sc[k].beta;
#pragma unroll 1
        for (int lr = threadIdx.x; lr < own; lr += blockDim.x) {
          const double z = ld_vec(a.z + static_cast<size_t>(k) * a.npad + r0 + lr);
          const double rk = xsub(r[lr], xmul(w, t[lr]));
          const double pk = xadd(rk, xmul(beta, xsub(p[lr], xmul(w, v[lr]))));
          x[lr] = xadd(x[lr], xmul(w, z));
          r[lr] = rk;
          p[lr] = pk;
          put_z(k, lr, xmul(pk, m[lr]));
        }
      }
    if (!publish()) return;
  }

  // xKx, ||x||, ||b - Ax||  (Bicgstab.c:188-204), with x in z's place
#pragma unroll
  for (int k = 0; k < K; ++k)
#pragma unroll 1
    for (int lr = threadIdx.x; lr < own; lr += blockDim.x) put_z(k, lr, at(kVx, k)[lr]);
  if (!publish()) return;
  double acc[kNV1<K>] = {};
  matvec([&](int lr, int k, double y, double x) {
    const size_t i = static_cast<size_t>(k) * a.n + r0 + lr;
    const double r = xsub(ld_vec(a.b + i), y);
    st_vec(a.x + i, x);
    acc[3 * k] += x * y;
    acc[3 * k + 1] += x * x;
    acc[3 * k + 2] += r * r;
  });
  const auto finish = [&](int k) {
    if (k >= K || blockIdx.x != 0 || (gridDim.x > 1 && bad)) return;
    SolveOut o{};
    o.iters = o.inner_iters = static_cast<int>(sc[k].iters);
    o.status = sc[k].status;
    o.xKx = fin[3 * k];
    o.norm_x = sqrt(fin[3 * k + 1]);
    o.norm_r = sqrt(fin[3 * k + 2]);
    o.conv = sc[k].conv;
    o.bnorm = sc[k].bnorm;
    *a.out[k] = o;
  };
  (void)grid_sum<kNV1<K>, false>(a, epoch, acc, fin, red, &bad, finish);
}

// ---- host ------------------------------------------------------------------

// static shared memory of the kernels (reductions, scalars), rounded up
constexpr size_t kStatic = 16 * 33 * 8 + 3 * 64 + 64;
// A block an SM, and at least sixteen slices a block: fewer blocks make the
// exchange cheaper than the idle SMs cost.
constexpr int kBlockSlices = 16;

struct Shape {
  const void *kern = nullptr;
  int grid = 0, threads = 0, on_chip = 0;
  size_t smem = 0;
};

// What an iteration reads past shared memory may be this much of the 126 MB of
// L2, or, from kGraphEngineRows rows on, what live_line says: past it this
// kernel waits on HBM with too few loads in flight, and the streaming engine,
// with four times the warps, hides it better.  (Below, the other choice is the
// persistent kernel, whose five barriers an iteration cost more: 40,000 rows of
// 100 slots, three systems, 38 us and 133.)
constexpr size_t kLiveBytes = 110 << 20;

// us an iteration, this kernel and the streaming engine, FP64, by the live
// bytes in MB and K (m: against the mixed streaming solve):
//   K 1  94^3 cells (76) 43, 73; 96^3 (88) 56, 70; 100^3 (100) 75, 80; 102^3
//        (115) 103, 82; 100,000 rows of 100 slots (102) 68, 74 (m 71); 250,000
//        of 40 (104) 93, 71
//   K 2  80^3 (68) 51, 85; 84^3 (88) 75, 95; 86^3 (94) 87, 94; 88^3 (101) 109,
//        101; 27-point 66^3 (80) 48, 80; 68^3 (93) 100, 96; 100,000 rows of 100
//        slots (102) 152, 84; 600,000 of 8 (101) 100, 86
//   K 3  76^3 (83) 63, 105; 27-point 64^3 (88) 81, 93; 400,000 rows of 12 slots
//        (99) 89, 94; 225,000 of 40 (103) 94, 96; 300,000 of 24 (103) 92, 88;
//        100,000 of 100 (103) 117, 96.  Where the operator is a third at most,
//        what the streaming kernels move of vectors weighs more: 78^3 (101) 97,
//        117; 80^3 (109) 99, 111; 82^3 (117) 114, 122.
// Unnumbered meshes (DevSell::far; with kFarSmem): 72^3 of 3 (75) 87, 124; 80^3
// of 2 (82) 98, 111; 92^3 of 1 (87) 76, 90; 96^3 of 1 (106) 96, 94; 84^3 of 2
// (95) 125, 124; random rows of 20, 250,000 of 2 (96) 165, 148.
size_t live_line(const sfr_system *s, int k, size_t op, size_t live) {
  if (s->n < kGraphEngineRows) return kLiveBytes;
  if (s->A.far()) return 94000000;
  if (k == 3) return 3 * op <= live ? kLiveBytes : 102500000;
  return k == 1 ? 100000000 : 95000000;
}

// Scattered gathers in flight hold a line of L1 each.  Up to this much shared
// memory a block (static and the system's 1 KB included: the 196 KB carve-out)
// leaves 60 KB of L1, the next carve-out 28.  Cells in random order, us an
// iteration with 190 KB at most and with all of it: 52^3 of 3 37 and 54, 60^3 of
// 3 50 and 78, 64^3 of 2 42 and 66, 84^3 of 1 47 and 74, 88^3 of 1 53 and 84
// (the streaming engine: 72, 88, 71, 74 and 80).  Numbered, the vectors that
// leave cost more than the L1 gives: 76^3 of 3 63 with all, 75 without.  So does
// the operator of a system whose z is about as small as that L1 (kFarZ): random
// rows of 20, 2,000 of 2 (32 KB) 23.4 with all, 27.2 without, 4,000 of 2 (64 KB)
// 32.0 and 21.6, 6,000 of 1 (48 KB) 21.1 and 19.4.
constexpr size_t kFarSmem = (196 << 10) - 1024, kFarZ = 40 << 10;

template <typename I, int K>
bool shape_of(const sfr_system *s, bool own_diag, Shape *sh) {
  int optin = 0;
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, s->device) !=
      cudaSuccess)
    return false;
  const size_t most = static_cast<size_t>(optin) - kStatic;
  const bool far = s->A.far() && sizeof(double) * K * static_cast<size_t>(s->n) > kFarZ;
  const size_t limit = far ? std::min(most, kFarSmem - kStatic) : most;
  const int ns = s->A.nslices;
  const int g = std::max(1, std::min(num_sms(s->device), (ns + kBlockSlices - 1) / kBlockSlices));
  const int slices = (ns + g - 1) / g;
  const size_t rows = static_cast<size_t>(slices) * kWarp;
  const size_t slots = rows * s->A.max_width * (8 + sizeof(I)), fixed = sizeof(int) * (slices + 1);
  const size_t vec = rows * K * sizeof(double);
  if (fixed + vec > limit) return false;
  // the operator first, if the vectors of the SpMV phases fit beside it
  const bool hold = fixed + slots + kCoreVecs * vec <= limit;
  const size_t base = fixed + (hold ? slots : 0);
  const bool core = base + kCoreVecs * vec <= limit;
  sh->on_chip = static_cast<int>(std::min<size_t>(kVecs, (limit - base) / vec));
  sh->smem = base + sh->on_chip * vec;
  const size_t op = hold ? 0 : s->A.nslots * (8 + sizeof(I));
  const size_t live = op + sizeof(double) * static_cast<size_t>(s->n) *
                               ((own_diag ? 1 : K) + K * (1 + kVecs - sh->on_chip));
  if (live > live_line(s, K, op, live)) return false;
  sh->grid = g;
  // a thread watches a block in neighbour_wait
  sh->threads = std::max((g + kWarp - 1) / kWarp * kWarp,
                         std::min(bicg_threads(K), slices * kWarp));
  sh->kern = hold   ? reinterpret_cast<const void *>(bicg_grid_kernel<I, K, true, true>)
             : core ? reinterpret_cast<const void *>(bicg_grid_kernel<I, K, true, false>)
                    : reinterpret_cast<const void *>(bicg_grid_kernel<I, K, false, false>);
  // asked once per kernel and device
  static std::mutex mu;
  static std::map<std::pair<const void *, int>, bool> known;
  std::lock_guard<std::mutex> lk(mu);
  const auto key = std::make_pair(sh->kern, s->device);
  const auto it = known.find(key);
  if (it != known.end()) return it->second;
  const bool ok =
      cudaFuncSetAttribute(sh->kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(most)) == cudaSuccess;
  if (!ok) (void)cudaGetLastError();  // the refusal is not a later call's error
  known[key] = ok;
  return ok;
}

template <int K>
bool shape_for(const sfr_system *s, bool own_diag, Shape *sh) {
  return s->A.off ? shape_of<int16_t, K>(s, own_diag, sh) : shape_of<int, K>(s, own_diag, sh);
}

template <int K>
int run(sfr_system *s, const double *d_diag_k, const double *d_b, double *d_x, double tol,
        uint32_t maxit, int32_t newx, cudaStream_t st, SolveOut *out, float *ms) {
  Shape sh;
  if (!shape_for<K>(s, !d_diag_k, &sh)) return SFR_UNSUPPORTED;
  auto align = [](size_t v) { return (v + 255) & ~static_cast<size_t>(255); };
  const size_t npad = static_cast<size_t>(s->A.nslices) * kWarp;
  const size_t slot_b = align(sizeof(ulonglong2) * 2 * kSumWords * sh.grid);
  const size_t tick_b = align(64 * static_cast<size_t>(sh.grid)) + 256;  // + the error word
  const size_t z_b = align(sizeof(double) * K * npad);
  const size_t vec_b = sh.on_chip < kVecs ? align(sizeof(double) * K * kVecs * npad) : 0;
  const size_t out_b = align(sizeof(SolveOut) * K);
  // x is written while b is still read: a caller's x that overlaps b gets a
  // copy of b
  const size_t nb = sizeof(double) * K * static_cast<size_t>(s->n);
  const uintptr_t xb = reinterpret_cast<uintptr_t>(d_x), bb = reinterpret_cast<uintptr_t>(d_b);
  const bool overlap = xb < bb + nb && bb < xb + nb;
  // ... and so do the diagonals, read by every SpMV phase
  const uintptr_t db = reinterpret_cast<uintptr_t>(d_diag_k);
  const bool overlap_d = d_diag_k && xb < db + nb && db < xb + nb;
  const int rc = ensure_workspace(s, slot_b + tick_b + z_b + vec_b + out_b +
                                         (overlap ? align(nb) : 0) + (overlap_d ? align(nb) : 0));
  if (rc != SFR_OK) return rc;
  char *base = static_cast<char *>(s->ws.base);

  BicgArgs<K> a{};
  a.n = s->n;
  a.nslices = s->A.nslices;
  a.npad = static_cast<int>(npad);
  a.sptr = s->A.sptr;
  a.col = s->A.col;
  a.off = s->A.off;
  a.val = s->A.val;
  a.b = d_b;
  a.x = d_x;
  a.tol = tol;
  a.maxit = maxit;
  a.newx = newx;
  a.on_chip = sh.on_chip;
  a.spin_limit = 1u << 22;
  a.slots = reinterpret_cast<ulonglong2 *>(base);
  a.ticks = reinterpret_cast<unsigned *>(base + slot_b);
  a.err = reinterpret_cast<int *>(base + slot_b + tick_b - 256);
  cudaError_t ce = cudaMemsetAsync(base, 0, slot_b + tick_b, st);
  base += slot_b + tick_b;
  a.z = reinterpret_cast<double *>(base);
  base += z_b;
  a.vecs = reinterpret_cast<double *>(base);
  base += vec_b;
  SolveOut *dev_out = reinterpret_cast<SolveOut *>(base);
  base += out_b;
  if (overlap) {
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(base, d_b, nb, cudaMemcpyDeviceToDevice, st);
    a.b = reinterpret_cast<double *>(base);
    base += align(nb);
  }
  const double *dk = d_diag_k;
  if (overlap_d) {
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(base, d_diag_k, nb, cudaMemcpyDeviceToDevice, st);
    dk = reinterpret_cast<double *>(base);
  }
  if (!s->ev0 && cudaEventCreate(&s->ev0) != cudaSuccess) return SFR_CUDA_ERROR;
  if (!s->ev1 && cudaEventCreate(&s->ev1) != cudaSuccess) return SFR_CUDA_ERROR;
  ResultRecord rec[K];
  bool pinned = true;
  for (int k = 0; k < K; ++k) pinned = pinned && rec[k].r;
  for (int k = 0; k < K; ++k) {
    a.diag[k] = dk ? dk + static_cast<size_t>(k) * s->n : s->d_diag;
    a.out[k] = pinned ? rec[k].r : dev_out + k;
    // stays when a wait gave up and the kernel left without a result
    out[k] = SolveOut{};
    out[k].status = SFR_TIMEOUT;
    if (pinned) *rec[k].r = out[k];
  }
  if (ce == cudaSuccess && !pinned)
    ce = cudaMemcpyAsync(dev_out, out, sizeof(SolveOut) * K, cudaMemcpyHostToDevice, st);
  void *params[] = {&a};
  if (ce == cudaSuccess) ce = cudaEventRecord(s->ev0, st);
  if (ce == cudaSuccess)
    ce = cudaLaunchCooperativeKernel(sh.kern, dim3(sh.grid), dim3(sh.threads), params, sh.smem, st);
  if (ce == cudaSuccess) ce = cudaEventRecord(s->ev1, st);
  if (ce == cudaSuccess && !pinned)
    ce = cudaMemcpyAsync(out, dev_out, sizeof(SolveOut) * K, cudaMemcpyDeviceToHost, st);
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(st);
  if (ce == cudaSuccess) cudaEventElapsedTime(ms, s->ev0, s->ev1);
  if (ce != cudaSuccess) {
    set_last_error(cudaGetErrorString(ce));
    return SFR_CUDA_ERROR;
  }
  if (pinned)
    for (int k = 0; k < K; ++k) out[k] = *rec[k].r;
  for (int k = 0; k < K; ++k)
    if (out[k].status == SFR_TIMEOUT) return SFR_TIMEOUT;
  return SFR_OK;
}

}  // namespace

bool onchip_bicg_fits(const sfr_system *s, int32_t k, bool own_diag) {
  Shape sh;
  return k == 1   ? shape_for<1>(s, own_diag, &sh)
         : k == 2 ? shape_for<2>(s, own_diag, &sh)
         : k == 3 && shape_for<3>(s, own_diag, &sh);
}

int solve_onchip_bicg(sfr_system *s, int32_t k, const double *d_diag_k, const double *d_b,
                      double *d_x, double tol, uint32_t maxit, int32_t newx, cudaStream_t st,
                      sfr_solve_info *info) {
  if (maxit == 0 || k > kBicgMaxK) return SFR_UNSUPPORTED;
  SolveOut out[kBicgMaxK];
  float ms = 0.f;
  const int rc = k == 1   ? run<1>(s, d_diag_k, d_b, d_x, tol, maxit, newx, st, out, &ms)
                 : k == 2 ? run<2>(s, d_diag_k, d_b, d_x, tol, maxit, newx, st, out, &ms)
                          : run<3>(s, d_diag_k, d_b, d_x, tol, maxit, newx, st, out, &ms);
  if (rc != SFR_OK) return rc;
  int worst = SFR_OK;
  for (int i = 0; i < k; ++i) {
    if (info) {
      sfr_solve_info &f = info[i];
      std::memset(&f, 0, sizeof(f));
      f.iters = f.inner_iters = out[i].iters;
      f.status = out[i].status;
      f.xKx = out[i].xKx;
      f.norm_x = out[i].norm_x;
      f.norm_r = out[i].norm_r;
      f.conv = out[i].conv;
      f.seconds = ms * 1e-3;
      f.relres = out[i].bnorm > 0 ? out[i].norm_r / out[i].bnorm : 0.0;
    }
    if (out[i].status != SFR_OK && worst == SFR_OK) worst = out[i].status;
  }
  return worst;
}

}  // namespace sfr
