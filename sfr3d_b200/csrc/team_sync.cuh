// Teams of blocks and what they exchange, for kernels that run a whole solve
// in one co-resident launch: sums over a team in one L2 round trip, and the
// range of blocks a block gathers from.
#pragma once

#include "common.cuh"
#include "persist.cuh"

namespace sfr {

// A block's words of an exchange: each value with the epoch it belongs to.
struct alignas(64) TeamSlot {
  ulonglong2 v[4];
};

struct TeamSync {
  TeamSlot *slots;  // two buffers of one slot a block, zero at launch
  unsigned *ticks;  // 16 words a block, zero at launch (neighbour_wait)
  int *err;
  unsigned spin_limit;
};

// The blocks that solve one system together, and this block's part: slices
// [s0, s1) of the system's [first, first + count), which the team's blocks
// [b0, b1) share in order.  A launch for one system is one team.
struct TeamPart {
  int s0, s1, first, count, b0, b1;
  int row_end;  // the system's rows end here
  int sys;
  int slices_left;  // a batched launch: slices of the systems of this round
  unsigned round;   // a batched launch: its round
  unsigned long long t0;  // the block's start (global_ns)
  __device__ __forceinline__ int owner(int row) const {
    const long long B = b1 - b0, ns = count, sl = row / kWarp - first;
    return b0 + static_cast<int>(((sl + 1) * B + ns - 1) / ns - 1);
  }
};

// A batched solve in rounds: the kernel is the body of a graph's WHILE node.
// A round gives every system still iterating a team of blocks, and each team
// as many iterations as the model below fits into the round's time; the next
// round shares the blocks out again over the systems left.  So the blocks of
// a system that converges early do not idle until the slowest one has, which
// the estimates cannot foresee (boxes of one size take 0.3 to 2 times the
// iterations of a cube).  Shares and lengths follow iteration counts alone:
// the same on every run.  (Rounds as a loop inside one launch spilled 2 KB a
// thread.)
constexpr int kMaxTeams = 384;  // systems of a launch: one a thread of a block

// A team's time an iteration, in us: what its exchanges and the publication
// of p cost, which more blocks do not shrink, and a slice's share.
struct TeamModel {
  float alone, many, slice;
  __host__ __device__ float us(int slices, int blocks) const {
    return (blocks > 1 ? many : alone) + slice * slices / blocks;
  }
};

// Blocks make a round's shares each for itself, and one may still be at it
// when a team of the same round stores that it is done.  So what round r
// stores, only the rounds after it read: `done` says in which round, and of
// the two rows of `iters` r reads one and writes the other.  (Every system
// that is not done has a team in each round, which writes its entry.)
struct RoundTable {
  const int4 *sys;   // per system {first slice, slices, end row, estimated iterations}
  int *done;         // per system, 1 + the round that wrote its result; 0: none yet
  int *iters;        // two rows of one entry a system: the iterations of the rounds before
  int nsys;
  int most;          // slices a block can hold
  TeamModel model;
  float us;          // the first round's time
  float us_later;    // a later round's
  unsigned *ctl;     // {round, blocks that finished it, systems done}, zero at first
  int *err;
  cudaGraphConditionalHandle more;  // the WHILE node's condition

  __device__ __forceinline__ bool done_before(int s, unsigned round) const {
    return static_cast<unsigned>(__ldcg(done + s) - 1) < round;
  }
  __device__ __forceinline__ int iters_before(int s, unsigned round) const {
    return __ldcg(iters + (round & 1u) * nsys + s);
  }
  __device__ __forceinline__ void put_done(int s, unsigned round) const {
    done[s] = static_cast<int>(round + 1u);
  }
  __device__ __forceinline__ void put_iters(int s, unsigned round, unsigned n) const {
    iters[((round + 1u) & 1u) * nsys + s] = static_cast<int>(n);
  }
};

// Ends a block's round: the last block to come by counts the round and stops
// the loop when no system is left (or a wait gave up).
__device__ __forceinline__ void end_round(const RoundTable &rt, const TeamPart &t, bool over) {
  if (threadIdx.x != 0) return;
  if (over) {
    rt.put_done(t.sys, t.round);
    atomicAdd(rt.ctl + 2, 1u);
  }
  __threadfence();
  if (atomicAdd(rt.ctl + 1, 1u) != gridDim.x - 1) return;
  __threadfence();
  rt.ctl[1] = 0u;
  rt.ctl[0] += 1u;
  const unsigned finished = atomicAdd(rt.ctl + 2, 0u);
  if (finished >= static_cast<unsigned>(rt.nsys) || *reinterpret_cast<volatile int *>(rt.err) != 0)
    cudaGraphSetConditional(rt.more, 0u);
}

// Shares the grid's blocks over the systems not done before t.round so that
// the slowest team, by the model above and the estimated iterations, takes
// least: from what the rounds before stored, the same in every block.  False
// when none is left; t.b1 == t.b0 for a block without a team.  The block has
// at least nsys threads.  scan: two rows of 32 ints.
__device__ __forceinline__ bool next_teams(const RoundTable &rt, TeamPart &t, int *scan) {
  const int i = threadIdx.x, lane = i & 31, warp = i >> 5, nw = blockDim.x >> 5;
  int4 s = make_int4(0, 0, 0, 1);
  if (i < rt.nsys) {
    s = rt.sys[i];
    if (rt.done_before(i, t.round)) s.y = 0;
    s.w = max(s.w - rt.iters_before(i, t.round), s.w / 4 + 1);  // what it may still need
  }
  // over the block, in every thread
  auto total = [&](int v) {
    v = __reduce_add_sync(0xffffffffu, v);
    if (lane == 0) scan[warp] = v;
    __syncthreads();
    int r = lane < nw ? scan[lane] : 0;
    r = __reduce_add_sync(0xffffffffu, r);
    __syncthreads();
    return r;
  };
  auto most = [&](float v) {  // v >= 0: the order of the bits is the order of the values
    unsigned u = __reduce_max_sync(0xffffffffu, __float_as_uint(v));
    if (lane == 0) scan[warp] = static_cast<int>(u);
    __syncthreads();
    u = lane < nw ? static_cast<unsigned>(scan[lane]) : 0u;
    u = __reduce_max_sync(0xffffffffu, u);
    __syncthreads();
    return __uint_as_float(u);
  };
  t.slices_left = total(s.y);
  if (t.slices_left == 0) return false;
  const int least = (s.y + rt.most - 1) / rt.most;
  const float est = static_cast<float>(s.w), work = rt.model.slice * s.y;
  auto time = [&](int B) { return est * rt.model.us(s.y, B); };
  auto need = [&](float T) {  // blocks for time T; more than the grid when there is no such number
    if (s.y == 0) return 0;
    if (time(least) <= T) return least;
    const float rest = T / est - rt.model.many;
    if (!(rest > 0.0f)) return 1 << 20;
    const float B = ceilf(work / rest);
    return B > s.y ? 1 << 20 : max(static_cast<int>(B), max(least, 2));
  };
  float hi = most(s.y ? time(least) : 0.0f), lo = 0.0f;
  for (int k = 0; k < 24; ++k) {
    const float mid = 0.5f * (lo + hi);
    if (total(min(need(mid), 1 << 20)) <= static_cast<int>(gridDim.x))
      hi = mid;
    else
      lo = mid;
  }
  const int nb = need(hi);
  // blocks before system i
  int pre = nb;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, pre, o);
    if (lane >= o) pre += v;
  }
  if (lane == 31) scan[warp] = pre;
  __syncthreads();
  int before = 0;
  for (int w = 0; w < warp; ++w) before += scan[w];
  pre += before - nb;
  __syncthreads();
  int *mine = scan + 32;
  if (i == 0) mine[0] = -1;
  __syncthreads();
  const int me = static_cast<int>(blockIdx.x);
  if (me >= pre && me < pre + nb) {
    mine[0] = i;
    mine[1] = s.x;
    mine[2] = s.y;
    mine[3] = s.z;
    mine[4] = pre;
    mine[5] = nb;
  }
  __syncthreads();
  t.b0 = t.b1 = 0;
  if (mine[0] >= 0) {
    t.sys = mine[0];
    t.first = mine[1];
    t.count = mine[2];
    t.row_end = mine[3];
    t.b0 = mine[4];
    t.b1 = t.b0 + mine[5];
    const long long ns = t.count, k = me - t.b0, B = mine[5];
    t.s0 = t.first + static_cast<int>(ns * k / B);
    t.s1 = t.first + static_cast<int>(ns * (k + 1) / B);
  }
  __syncthreads();
  return true;
}

// This block's part of the round (t.b1 == t.b0: none).
__device__ __forceinline__ TeamPart team_part(const TeamTable &tt, const RoundTable &rt,
                                              unsigned round, int *scan) {
  TeamPart t;
  t.t0 = global_ns();
  t.round = round;
  if (round > 0) {
    if (!next_teams(rt, t, scan)) t.b0 = t.b1 = 0;
    return t;
  }
  const int4 e = tt.block[blockIdx.x];
  const int2 y = tt.sys[blockIdx.x];
  t.s0 = e.x;
  t.s1 = e.y;
  t.b0 = e.z;
  t.b1 = e.w;
  t.first = tt.block[e.z].x;
  t.count = tt.block[e.w - 1].y - t.first;
  t.sys = y.x;
  t.row_end = y.y;
  t.slices_left = tt.block[gridDim.x - 1].y;
  return t;
}

// Whether a block's rows and slots fit `left` bytes of shared memory.  In 64
// bits: a block of a few hundred rows may have more slots than 2^31 bytes hold.
__host__ __device__ constexpr bool block_fits(int rows, int row_bytes, int slots, int slot_bytes,
                                              int left) {
  return static_cast<long long>(rows) * row_bytes + static_cast<long long>(slots) * slot_bytes <=
         left;
}

// Hands out a block's dynamic shared memory from the front.
struct Carve {
  char *at;
  int left;
  template <typename T>
  __host__ __device__ __forceinline__ T *take(int count) {
    const long long bytes =
        (static_cast<long long>(count) * static_cast<long long>(sizeof(T)) + 7) & ~7ll;
    if (bytes > left) return nullptr;
    T *p = reinterpret_cast<T *>(at);
    at += bytes;
    left -= static_cast<int>(bytes);
    return p;
  }
};

// Matrix loads under an L2 policy.
__device__ __forceinline__ double ld_mat(const double *p, uint64_t pol) {
  double v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ float ld_mat(const float *p, uint64_t pol) {
  float v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ int ld_mat(const int *p, uint64_t pol) {
  int v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.s32 %0, [%1], %2;" : "=r"(v) : "l"(p), "l"(pol));
  return v;
}
__device__ __forceinline__ int ld_mat(const int16_t *p, uint64_t pol) {
  int16_t v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.s16 %0, [%1], %2;" : "=h"(v) : "l"(p), "l"(pol));
  return v;
}

// Exchange epochs and publication counts of a round start here: teams change
// between rounds, so every block counts from the same number.
__device__ __forceinline__ unsigned round_base(unsigned round) { return round << 20; }
// Iterations the round's time holds for this team.  Rounds end before the
// counts above would wrap: the last has no cap.
constexpr unsigned kLastRound = 2000;
__device__ __forceinline__ unsigned round_cap(const RoundTable &rt, const TeamPart &t,
                                              unsigned round) {
  if (round >= kLastRound) return 0xffffffffu;
  const float us = round == 0 ? rt.us : rt.us_later;
  return max(16u, static_cast<unsigned>(fminf(us / rt.model.us(t.count, t.b1 - t.b0), 1e9f)));
}

// NV values (a power of two up to 16) summed over a warp, a butterfly that
// halves the values a lane carries before it halves the lanes (four values:
// six 64-bit shuffles instead of twenty).  Lane l ends with the total of value
// l >> kSumShift<NV>, the same bits in all the lanes that hold it.
template <int NV>
constexpr int kSumShift = NV == 16 ? 1 : NV == 8 ? 2 : NV == 4 ? 3 : NV == 2 ? 4 : 5;

template <int NV, int kLanes = 16>
__device__ __forceinline__ double warp_sum_n(const double (&v)[NV]) {
  static_assert(NV == 1 || NV == 2 || NV == 4 || NV == 8 || NV == 16, "a power of two");
  constexpr unsigned kAll = 0xffffffffu;
  if constexpr (NV == 1) {
    double t = v[0];
#pragma unroll
    for (int o = kLanes; o > 0; o >>= 1) t += __shfl_xor_sync(kAll, t, o);
    return t;
  } else {
    const bool hi = threadIdx.x & kLanes;
    double h[NV / 2];
#pragma unroll
    for (int i = 0; i < NV / 2; ++i)
      h[i] = (hi ? v[i + NV / 2] : v[i]) +
             __shfl_xor_sync(kAll, hi ? v[i] : v[i + NV / 2], kLanes);
    return warp_sum_n<NV / 2, kLanes / 2>(h);
  }
}

// Whether this lane writes the total it holds.
template <int NV>
__device__ __forceinline__ bool sum_writer() {
  return (threadIdx.x & ((1u << kSumShift<NV>) - 1) & 31u) == 0;
}
template <int NV>
__device__ __forceinline__ int sum_index() {
  return static_cast<int>(threadIdx.x & 31) >> kSumShift<NV>;
}

// The block's totals of NV values in the lanes of warp 0, as warp_sum_n
// leaves them (other warps: unspecified).  sm: NV * 32 doubles.
template <int NV>
__device__ __forceinline__ double block_sum_n(const double (&v)[NV], double *sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const double t = warp_sum_n<NV>(v);
  if (sum_writer<NV>()) sm[sum_index<NV>() * 32 + warp] = t;
  __syncthreads();
  double s = 0.0;
  if (warp == 0) {
    double w[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) w[i] = lane < nw ? sm[i * 32 + lane] : 0.0;
    s = warp_sum_n<NV>(w);
  }
  return s;
}

// {value, epoch} in one 16-byte word, stored and loaded whole.
__device__ __forceinline__ void st_slot(ulonglong2 *p, double v, unsigned long long epoch) {
  asm volatile(
      "{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}" ::"l"(p),
      "l"(__double_as_longlong(v)), "l"(epoch)
      : "memory");
}
__device__ __forceinline__ bool ld_slot(const ulonglong2 *p, double *v, unsigned long long epoch) {
  unsigned long long lo, hi;
  asm volatile(
      "{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
      : "=l"(lo), "=l"(hi)
      : "l"(p)
      : "memory");
  *v = __longlong_as_double(static_cast<long long>(lo));
  return hi == epoch;
}

// Totals of NV values over the team, in every thread, the same bits in all
// its blocks.  Each block writes its totals with the epoch beside each value;
// thread b of every block polls block b's slot, so the values arrive with
// the poll: one L2 round trip.  Two buffers alternate: a block writes epoch e
// only after it read every block's epoch e - 1, which each published after it
// had read every epoch e - 2.  kFence: every global write before the call, in
// any block, is visible after it in all.  Bounded: after spin_limit polls a
// block records SFR_TIMEOUT in *err, and a block that sees *err set stops
// waiting.  False on either.  sm: NV * 32 doubles, bad: a shared word.
template <int NV, bool kFence>
__device__ __forceinline__ bool team_sum(const TeamSync &a, const TeamPart &t, unsigned &epoch,
                                         const double (&acc)[NV], double (&tot)[NV], double *sm,
                                         int *bad) {
  const int warp = threadIdx.x >> 5;
  const int G = t.b1 - t.b0;
  ++epoch;
  const double s = block_sum_n<NV>(acc, sm);
  if (G == 1) {  // a team of one block: no other block to tell
    if (warp == 0 && sum_writer<NV>()) sm[sum_index<NV>() * 32] = s;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NV; ++i) tot[i] = sm[i * 32];
    __syncthreads();
    return true;
  }
  TeamSlot *cur = a.slots + static_cast<size_t>(epoch & 1u) * gridDim.x + t.b0;
  if (warp == 0 && sum_writer<NV>()) {
    if (kFence) cuda::atomic_thread_fence(cuda::memory_order_release, cuda::thread_scope_device);
    st_slot(&cur[blockIdx.x - t.b0].v[sum_index<NV>()], s, epoch);
  }
  if (threadIdx.x == 0) *bad = 0;
  __syncthreads();  // sm is free again; *bad is 0
  const int watchers = min(static_cast<int>(blockDim.x), (G + 31) & ~31);
  if (static_cast<int>(threadIdx.x) < watchers) {
    double v[NV] = {};
    cuda::atomic_ref<int, cuda::thread_scope_device> err(*a.err);
    for (int b = threadIdx.x; b < G; b += watchers) {
      double w[NV];
      for (unsigned spins = 0;; ++spins) {
        bool all = true;
#pragma unroll
        for (int i = 0; i < NV; ++i) all &= ld_slot(&cur[b].v[i], &w[i], epoch);
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
      for (int i = 0; i < NV; ++i) v[i] += w[i];
    }
    __syncwarp();
    if (kFence) cuda::atomic_thread_fence(cuda::memory_order_acquire, cuda::thread_scope_device);
    const double q = warp_sum_n<NV>(v);
    if (sum_writer<NV>()) sm[sum_index<NV>() * 32 + warp] = q;
  }
  __syncthreads();
  const int ww = watchers >> 5;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    double q = sm[i * 32];
    for (int w = 1; w < ww; ++w) q += sm[i * 32 + w];
    tot[i] = q;
  }
  const bool ok = *bad == 0;
  __syncthreads();
  return ok;
}

// The blocks [range[0], range[1]] owning the columns this block gathers from.
template <typename I>
__device__ __forceinline__ void gather_range(const TeamPart &t, const int *sm_sp, const I *cols,
                                             int *range) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  int cmin = t.s0 * kWarp, cmax = t.s1 * kWarp - 1;
  for (int s = t.s0 + warp; s < t.s1; s += nw) {
    const int row = s * kWarp + lane;
    if (row >= t.row_end) continue;  // padding: its columns mean nothing
    for (int e = sm_sp[s - t.s0] + lane; e < sm_sp[s - t.s0 + 1]; e += kWarp) {
      const int c = slot_col(cols, e, row);
      cmin = min(cmin, c);
      cmax = max(cmax, c);
    }
  }
  if (threadIdx.x == 0) {
    range[0] = cmin;
    range[1] = cmax;
  }
  __syncthreads();
  atomicMin(range, cmin);
  atomicMax(range + 1, cmax);
  __syncthreads();
  const int lo = t.owner(range[0]), hi = t.owner(range[1]);
  __syncthreads();
  if (threadIdx.x == 0) {
    range[0] = lo;
    range[1] = hi;
  }
  __syncthreads();
}

// A block's static shared memory for the above.
struct TeamShared {
  double red[32 * 4];
  int bad, range[2], scan[64];
  TeamPart part;  // a batched launch's: in registers it spills the solve's
};

}  // namespace sfr
