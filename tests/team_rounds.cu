// Prints the shares that the blocks of a batched launch make of a round's
// systems (team_sync.cuh, next_teams), one line a block: round, block, whether
// any system is left, then its system, its slices and its team's blocks.
// Twice: from what the rounds before stored, and with what teams of the same
// round store when they end before others have read.
#include <cstdio>
#include <vector>

#include "team_sync.cuh"

using namespace sfr;

__global__ void stores(const RoundTable rt, unsigned round) {
  const int i = threadIdx.x;
  if (i >= rt.nsys) return;
  if (i % 3 == round % 3)
    rt.put_done(i, round);
  else if (!rt.done_before(i, round))
    rt.put_iters(i, round, 20u * round * (i % 5));
}

__global__ void shares(const RoundTable rt, unsigned round, int *out) {
  __shared__ int scan[64];
  TeamPart t{};
  t.round = round;
  const bool any = next_teams(rt, t, scan);
  if (threadIdx.x != 0) return;
  int *o = out + blockIdx.x * 6;
  o[0] = any;
  o[1] = t.b1 > t.b0 ? t.sys : -1;
  o[2] = t.s0;
  o[3] = t.s1;
  o[4] = t.b0;
  o[5] = t.b1;
}

int main() {
  constexpr int kSys = 41, kGrid = 96;
  std::vector<int4> sys(kSys);
  int first = 0;
  for (int i = 0; i < kSys; ++i) {
    const int slices = 3 + (i * 37) % 90;
    sys[i] = make_int4(first, slices, (first + slices) * 32, 100 + 40 * i);
    first += slices;
  }
  int4 *d_sys;
  int *d_tab, *d_out;
  if (cudaMalloc(&d_sys, sizeof(int4) * kSys) != cudaSuccess ||
      cudaMalloc(&d_tab, sizeof(int) * 3 * kSys) != cudaSuccess ||
      cudaMalloc(&d_out, sizeof(int) * 6 * kGrid) != cudaSuccess ||
      cudaMemcpy(d_sys, sys.data(), sizeof(int4) * kSys, cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemset(d_tab, 0, sizeof(int) * 3 * kSys) != cudaSuccess)
    return 1;
  RoundTable rt{};
  rt.sys = d_sys;
  rt.done = d_tab;
  rt.iters = d_tab + kSys;
  rt.nsys = kSys;
  rt.most = 120;
  rt.model = TeamModel{0.9f, 4.5f, 0.1f};
  std::vector<int> out(6 * kGrid);
  for (unsigned round = 1; round <= 3; ++round) {
    for (int late = 0; late < 2; ++late) {
      if (late) stores<<<1, kMaxTeams>>>(rt, round);
      shares<<<kGrid, kMaxTeams>>>(rt, round, d_out);
      if (cudaMemcpy(out.data(), d_out, sizeof(int) * 6 * kGrid, cudaMemcpyDeviceToHost) !=
          cudaSuccess)
        return 1;
      for (int b = 0; b < kGrid; ++b)
        std::printf("%u %d %d %d %d %d %d %d %d\n", round, late, b, out[6 * b], out[6 * b + 1],
                    out[6 * b + 2], out[6 * b + 3], out[6 * b + 4], out[6 * b + 5]);
    }
  }
  return 0;
}
