// The sums of the slice-form CG's teams when a CTA has given up on a wait: every
// CTA of the team learns of it at the next sum, whichever CTA it was.  No wait
// runs out here: the mark is set directly, and all CTAs arrive.
//
// Prints one line per team form and marked CTA (-1: none):
//   form late ok   (ok: 1 when all CTAs agree on what is expected)
#include <cstdio>
#include <cstring>

#include "mlsh_cluster_cg.cuh"

using namespace mlsh;

constexpr int kCtas = 4;

struct Out {
  double a[2], b[2], flag[2];
  int any;
};

template <class Team>
__device__ void two_sums(Team &team, CgShared &sh, int late, Out *out) {
  for (int k = 0; k < 2; ++k) {
    if (k == 1 && (int)team.rank == late && threadIdx.x == 0) sh.late = 1;
    __syncthreads();
    double a = threadIdx.x + 1.0, b = 2.0, flag = 0.5;
    team.sums(a, b, flag);
    if (threadIdx.x == 0) {
      out[team.rank].a[k] = a;
      out[team.rank].b[k] = b;
      out[team.rank].flag[k] = flag;
    }
    __syncthreads();
  }
}

__global__ void __cluster_dims__(kCtas, 1, 1) __launch_bounds__(kCgThreads, 1)
    cluster_sums(int late, Out *out) {
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  __shared__ CgShared sh;
  ClusterTeam team{cl, sh, cl.num_blocks(), cl.block_rank(), 0u, 0u};
  cg_init_shared(sh, team.size);
  cl.sync();
  two_sums(team, sh, late, out);
  cl.sync();
  const bool any = team.any_late();
  if (threadIdx.x == 0) out[team.rank].any = any ? 1 : 0;
  cl.sync();
}

__global__ void __launch_bounds__(kCgThreads, 1) grid_sums(int late, GridSpace *space, Out *out) {
  __shared__ CgShared sh;
  cg_init_shared(sh, 1);
  GridTeam team{sh, space, nullptr, gridDim.x, blockIdx.x, 0u, 0u};
  two_sums(team, sh, late, out);
  if (threadIdx.x == 0) out[blockIdx.x].any = late >= 0;
}

int main() {
  Out *d = nullptr, h[kCtas];
  GridSpace *space = nullptr;
  if (cudaMalloc(&d, sizeof(h)) != cudaSuccess ||
      cudaMalloc(&space, sizeof(GridSpace)) != cudaSuccess)
    return 1;
  const double want_a = kCtas * (kCgThreads * (kCgThreads + 1.0) / 2), want_b = kCtas * kCgThreads * 2.0;
  for (int form = 0; form < 2; ++form)
    for (int late = -1; late < kCtas; ++late) {
      cudaMemset(d, 0, sizeof(h));
      cudaMemset(space, 0, sizeof(GridSpace));
      if (form == 0) {
        cluster_sums<<<kCtas, kCgThreads>>>(late, d);
      } else {
        int l = late;
        void *args[] = {&l, &space, &d};
        if (cudaLaunchCooperativeKernel((const void *)grid_sums, dim3(kCtas), dim3(kCgThreads), args, 0,
                                        nullptr) != cudaSuccess)
          return 2;
      }
      if (cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 3;
      int ok = 1;
      for (const Out &o : h) {
        ok &= o.a[0] == want_a && o.b[0] == want_b && o.flag[0] == 0.5;
        if (late < 0) ok &= o.a[1] == want_a && o.b[1] == want_b && o.flag[1] == 0.5;
        else ok &= o.flag[1] == 2.0;
        ok &= o.any == (late >= 0 ? 1 : 0);
      }
      std::printf("%s %d %d\n", form == 0 ? "cluster" : "grid", late, ok);
    }
  return 0;
}
