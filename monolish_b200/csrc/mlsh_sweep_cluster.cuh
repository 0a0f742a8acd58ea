// The triangular sweeps of mlsh_precond.cu on one thread-block cluster: the
// solution distributed over the CTAs' shared memory, a cluster-wide meeting
// between dependency levels.
//
// The multi-CTA sweep passes a result to the blocks that wait for it through
// L2: store, release (the store's way to L2 and back), flag, the waiters'
// polls, their loads -- four trips of 300-700 cycles, 2.3 us a level.  Here a
// level costs one message between CTAs of a cluster (remote mbarrier arrivals)
// and reads from another CTA's shared memory.  What a block needs besides
// solution values depends on the matrix only: one record per block, made once
// and read into registers while the level before is still being waited for,
// holds its entries outside the block (as places in the cluster's shared
// memory instead of columns), the finishing factor, and the affine scan's
// coefficients for each of its five steps, so that a step is one shuffle and
// one multiply-add (the same operations as affine_scan's, in its order).
//
// IC(0)-CG on the 49^3 7-point Laplacian (98 levels a sweep): 19.6 ms per solve
// instead of 27.4.
//
// Takes matrices whose blocks are all resolved by the scan, with at most
// kPre entries of a row outside its block (5- and 7-point stencils), whose
// solution fits the cluster's shared memory.
#pragma once
#include <cooperative_groups.h>

#include <type_traits>

#include "mlsh_internal.cuh"
#include "mlsh_precond.cuh"
#include "mlsh_ptx.cuh"

namespace mlsh {

constexpr int kClSweepThreads = 512;
constexpr int kClSweepWarps = kClSweepThreads / 32;
constexpr int kClSweepMaxCtas = 16;
constexpr size_t kClSweepSmem = 220 * 1024;  // solution and level starts

// One block: [values, places of the entries outside it][finishing factor]
// [scan coefficients].  S: the scan's type.
template <typename T, int MODE>
struct ClusterRec {
  using S = typename std::conditional<MODE == kSorBwd, double, T>::type;
  static constexpr int kVal = 0;
  static constexpr int kPlace = kVal + 4 * 32 * (int)sizeof(T);
  static constexpr int kFin = kPlace + 4 * 32 * 4;
  static constexpr int kBe = kFin + 32 * (int)sizeof(T);
  static constexpr int kBytes = kBe + 5 * 32 * (int)sizeof(S);
};
constexpr unsigned kNoPlace = 0xffffffffu;

// Block number i of the level order is CTA i % ctas' block i / ctas; its row
// base + l sits at element 32 (i / ctas) + l of that CTA's solution.
__device__ __forceinline__ unsigned place_of(int order_index, int within, int ctas) {
  return (unsigned)(order_index % ctas) << 24 | (unsigned)(order_index / ctas * 32 + within);
}

// explicitly rounded (mlsh_precond.cu uses them too)
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }

template <typename T>
struct ClusterSweepArgs {
  const SweepBlock *order;
  const unsigned char *rec;
  const int *level_off;
  int levels;
  int nb;
  const T *rhs;
  T *out;
  const int *done;
  int *err;
  unsigned polls;
};

// What a lane holds of its block.
template <typename T, int MODE>
struct ClusterRow {
  using S = typename ClusterRec<T, MODE>::S;
  T v[4], fin, rhs;
  unsigned place[4];
  S be[5];
};

template <typename T, int MODE>
__device__ __forceinline__ void cluster_row_load(ClusterRow<T, MODE> &r, const unsigned char *rec,
                                                 const SweepBlock &bk, const T *rhs, int lane) {
  using R = ClusterRec<T, MODE>;
  using S = typename R::S;
  const T *v = reinterpret_cast<const T *>(rec + R::kVal) + lane;
  const unsigned *pl = reinterpret_cast<const unsigned *>(rec + R::kPlace) + lane;
  const S *be = reinterpret_cast<const S *>(rec + R::kBe) + lane;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    r.place[u] = __ldg(pl + 32 * u);
    r.v[u] = __ldg(v + 32 * u);
  }
  r.fin = __ldg(reinterpret_cast<const T *>(rec + R::kFin) + lane);
#pragma unroll
  for (int d = 0; d < 5; ++d) r.be[d] = __ldg(be + 32 * d);
  r.rhs = lane < bk.rows ? rhs[bk.base + lane] : T(0);
}

template <typename T>
__device__ __forceinline__ T ld_cluster_at(uint32_t x0, unsigned place) {
  uint32_t at;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(at)
               : "r"(x0 + (place & 0xffffffu) * (unsigned)sizeof(T)), "r"(place >> 24));
  T v;
  if constexpr (sizeof(T) == 8)
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(at) : "memory");
  else
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
  return v;
}

__device__ __forceinline__ bool mbar_test_cluster(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

template <typename S, bool REV>
__device__ __forceinline__ S coefficient_scan(S al, const S (&be)[5]) {
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const S al2 = REV ? __shfl_down_sync(0xffffffffu, al, 1 << k)
                      : __shfl_up_sync(0xffffffffu, al, 1 << k);
    if (be[k] != S(0)) al = al + be[k] * al2;  // 0: nothing from that neighbour
  }
  return al;
}

template <typename T, int MODE>
__device__ __forceinline__ T cluster_row_solve(const ClusterRow<T, MODE> &r, uint32_t x0) {
  constexpr bool REV = MODE == kSorBwd || MODE == kDiagBwd;
  T x[4];
#pragma unroll
  for (int u = 0; u < 4; ++u)
    x[u] = r.place[u] != kNoPlace ? ld_cluster_at<T>(x0, r.place[u]) : T(0);
  if constexpr (MODE == kSorBwd) {
    double sacc = 0.0;  // "auto tmp = 0.0", sor_kernel.hpp:61-66
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (r.place[u] != kNoPlace) sacc = __dadd_rn(sacc, (double)mul_rn(r.v[u], x[u]));
    return (T)coefficient_scan<double, true>((double)r.rhs - sacc * (double)r.fin, r.be);
  } else {
    T acc = r.rhs;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (r.place[u] != kNoPlace) acc = sub_rn(acc, mul_rn(r.v[u], x[u]));
    T al = acc;
    if constexpr (MODE == kSorFwd) al = acc * r.fin;
    if constexpr (MODE == kDiagFwd || MODE == kDiagBwd) al = acc / r.fin;
    return coefficient_scan<T, REV>(al, r.be);
  }
}

template <typename T, int MODE>
__global__ void __launch_bounds__(kClSweepThreads, 1)
    sweep_cluster_kernel(const ClusterSweepArgs<T> a) {
  using R = ClusterRec<T, MODE>;
  namespace cgs = cooperative_groups;
  cgs::cluster_group cl = cgs::this_cluster();
  extern __shared__ __align__(16) unsigned char sweep_cluster_smem[];
  __shared__ uint64_t level_bar[2];  // levels take them in turn (see below)
  __shared__ int s_late;
  if (a.done != nullptr && *(volatile const int *)a.done != 0) return;  // all CTAs alike
  const int ctas = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // [solution of the CTA's blocks][level starts]
  const int mine = a.nb > rank ? (a.nb - rank + ctas - 1) / ctas : 0;  // this CTA's blocks
  const int most = (a.nb + ctas - 1) / ctas;
  T *xs = reinterpret_cast<T *>(sweep_cluster_smem);
  int *s_loff = reinterpret_cast<int *>(sweep_cluster_smem + (size_t)most * 32 * sizeof(T));
  for (int i = threadIdx.x; i <= a.levels; i += kClSweepThreads) s_loff[i] = a.level_off[i];
  const uint32_t bar0 = smem_addr(level_bar);
  if (threadIdx.x == 0) {
    mbar_init(bar0, (uint32_t)ctas);
    mbar_init(bar0 + 8, (uint32_t)ctas);
    s_late = 0;
    fence_mbar_init();
  }
  const uint32_t x0 = smem_addr(xs);
  // the warp's blocks are the CTA's warp-th, (warp + 16)-th, ...; the next
  // one's record is in registers, the one after's schedule entry too
  int k = warp;
  SweepBlock bk{}, bk2{};
  ClusterRow<T, MODE> row;
  auto index = [&](int j) { return j * ctas + rank; };
  if (k < mine) {
    bk = a.order[index(k)];
    cluster_row_load<T, MODE>(row, a.rec + (size_t)index(k) * R::kBytes, bk, a.rhs, lane);
  }
  if (k + kClSweepWarps < mine) bk2 = a.order[index(k + kClSweepWarps)];
  cl.sync();
  for (int lv = 0; lv < a.levels; ++lv) {
    const int end = s_loff[lv + 1];
    while (k < mine && index(k) < end) {
      const T x = cluster_row_solve<T, MODE>(row, x0);
      xs[k * 32 + lane] = x;
      k += kClSweepWarps;
      if (k < mine) {
        bk = bk2;
        cluster_row_load<T, MODE>(row, a.rec + (size_t)index(k) * R::kBytes, bk, a.rhs, lane);
        if (k + kClSweepWarps < mine) bk2 = a.order[index(k + kClSweepWarps)];
      }
    }
    if (lv + 1 == a.levels) break;
    // This CTA's part of the level is written: tell every CTA, wait for all.
    // Arrivals carry no sender and remote ones reach different CTAs in any
    // order, so with one barrier a CTA that has left level lv could fill, with
    // its arrival for lv + 1, the place of one still under way for lv.  With
    // two, the next arrival on this barrier is for lv + 2: its sender has seen
    // everybody arrive for lv + 1, which a CTA does once it has left lv.
    const uint32_t bar = bar0 + 8u * ((uint32_t)lv & 1u);
    const uint32_t phase = ((uint32_t)lv >> 1) & 1u;
    __syncthreads();
    if ((int)threadIdx.x < ctas) {
      uint32_t to;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(bar), "r"(threadIdx.x));
      asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(to)
                   : "memory");
    }
    bool ok = true;
    if (warp == 0) {  // one warp asks, the others wait behind it
      ok = false;
      for (unsigned p = 0; p < a.polls && !ok; ++p) ok = mbar_test_cluster(bar, phase);
      if (!ok) s_late = 1;
    }
    if (__syncthreads_or(ok ? 0 : 1)) break;
  }
  if (s_late && threadIdx.x == 0) atomicCAS(a.err, 0, MLSH_ERR_TIMEOUT);
  cl.sync();  // nobody reads this CTA's shared memory any more
  for (int j = warp; j < mine; j += kClSweepWarps) {
    const SweepBlock o = a.order[index(j)];
    if (lane < o.rows) a.out[o.base + lane] = xs[j * 32 + lane];
  }
}

// Records of a schedule; *bad is set where the form does not apply.
template <typename T, int MODE>
__global__ void __launch_bounds__(256)
    cluster_rec_kernel(const Sweep sw, const int *block_of, const int *order_index, int nb,
                       int ctas, unsigned char *recs, int *bad) {
  using R = ClusterRec<T, MODE>;
  using S = typename R::S;
  constexpr bool BWD = MODE == kSorBwd || MODE == kDiagBwd;
  const int q = (int)(blockIdx.x * 8 + (threadIdx.x >> 5));
  if (q >= nb) return;
  const int lane = threadIdx.x & 31;
  const SweepBlock bk = sw.order[q];
  const int end = bk.base + bk.rows;
  const int row = bk.base + lane;
  const T *val = static_cast<const T *>(sw.val);
  T v[4] = {T(0), T(0), T(0), T(0)}, fin = T(1), a1 = T(0);
  unsigned place[4] = {kNoPlace, kNoPlace, kNoPlace, kNoPlace};
  bool fits = bk.scan != 0;
  if (lane < bk.rows) {
    const int b = BWD ? sw.up_beg[row] : sw.rp[row];
    const int e = BWD ? sw.rp[row + 1] : sw.lo_end[row];
    int k = 0;
    for (int j = b; j < e; ++j) {
      const int c = sw.ci[j];
      if (c >= bk.base && c < end) {
        a1 = val[j];  // the adjacent row (a scan block has no other)
        continue;
      }
      if (k == 4) {
        fits = false;
        break;
      }
      v[k] = val[j];
      // the column's block, where the level order puts it, the row in it
      const int ob = block_of[c];
      place[k++] = place_of(order_index[ob], c - sw.order[order_index[ob]].base, ctas);
    }
    if constexpr (MODE == kSorFwd || MODE == kSorBwd) {
      fin = static_cast<const T *>(sw.scale)[row];
    } else if constexpr (MODE == kDiagFwd || MODE == kDiagBwd) {
      const int d = sw.lo_end[row];
      fin = sw.up_beg[row] > d ? val[d] : T(0);
    }
  }
  if (!__all_sync(0xffffffffu, fits) && lane == 0) *bad = 1;
  S be;
  if constexpr (MODE == kSorFwd) be = -(a1 * fin);
  else if constexpr (MODE == kSorBwd) be = -((double)a1 * (double)fin);
  else if constexpr (MODE == kUnitFwd) be = -a1;
  else be = -(a1 / fin);
  if (lane >= bk.rows) be = S(0);
  unsigned char *rec = recs + (size_t)q * R::kBytes;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    reinterpret_cast<T *>(rec + R::kVal)[u * 32 + lane] = v[u];
    reinterpret_cast<unsigned *>(rec + R::kPlace)[u * 32 + lane] = place[u];
  }
  reinterpret_cast<T *>(rec + R::kFin)[lane] = fin;
  // step k of the scan: be_k as affine_scan composes it; 0 where the lane
  // takes nothing (its coefficient is 0, or there is no lane to take from)
  S *out = reinterpret_cast<S *>(rec + R::kBe) + lane;
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const int d = 1 << k;
    const S be2 = BWD ? __shfl_down_sync(0xffffffffu, be, d) : __shfl_up_sync(0xffffffffu, be, d);
    const bool in = BWD ? lane + d < 32 : lane >= d;
    out[k * 32] = in ? be : S(0);
    if (in && be != S(0)) be = be * be2;
  }
}

}  // namespace mlsh
