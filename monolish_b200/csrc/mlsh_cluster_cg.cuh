// CG on one cluster, or on all SMs at once, for matrices with short rows: the
// matrix in slot-major slices (entry k of 32 consecutive rows side by side),
// in shared memory where it fits and streamed through a small ring where it
// does not, and each thread's own r and q in registers.
//
// What it replaces: the row loop of mlsh_cluster.cuh (still used for matrices
// with a longer row) reads row_ptr, columns and values with one thread per
// CRS row, so a warp's loads stride by the row length and cost two to three
// times the wavefronts of contiguous ones, behind a chain of dependent
// loads; x and 1/diag went through global memory every iteration, every
// thread added the 16 CTA partials of each sum one after another, and the
// cluster barriers waited for the x stores.  Here
//   * at the start of a solve each warp rewrites the rows it owns as slices
//     {values [slots][32], columns [slots][32]}; columns become words that say
//     where p is found (this CTA, another one), so a gather needs no table;
//   * p and x (and 1/diag where it fits) live in shared memory, r and q in
//     registers.  Slices stay in shared memory as far as there is room; the
//     others are streamed from a workspace in L2 by bulk copies into a ring
//     of a few slices per warp, which runs ahead across iterations (the
//     matrix does not change), so no load latency is left in the product;
//   * sums: two values share one reduction's shuffles; a cluster's CTAs send
//     their partials with st.async, which completes on the receivers' mbarrier
//     (one one-way message instead of a store and a cluster barrier); the CTAs
//     of a whole-GPU launch meet at an arrival counter in L2.
// Row sums keep the row's order with separately rounded products; absent
// entries are skipped, not added as zeros.
//
// us per iteration of Jacobi-CG in FP64, row loop -> slices on a cluster /
// slices on all SMs: 16,384 rows (2D) 6.9 -> 3.0 / 6.8; 32,761 rows 13.0 ->
// 3.9 / 7.3; 65,536 rows 24 -> 6.7 / 7.5; 102,400 rows 31 -> 16.0 / 8.1;
// 262,144 rows (3D) kernel engine 22.2, all SMs 15.2; 512,000 rows 29.7, 20.2.
// A cluster is bound by the latency of its two sums and one barrier
// (about 2 us), from 4,096 rows a CTA on by its instructions (about 182 per
// warp, slice and iteration, 110 of them the product's, at 1.6 per cycle on an
// SM); all SMs by the arrival
// counter's round trips through L2 (about 6 us an iteration).
#pragma once
#include <type_traits>

#include "mlsh_cluster.cuh"

namespace mlsh {

// Longest row the slice form takes at all; with many rows a CTA the layout
// below has room for fewer entries: FP64 16 up to 1,024 rows a CTA, 12 at 4,096
// and 7 at 8,192; FP32 16 up to 8,192 and 9 at 16,384.
constexpr int kCgMaxRow = 16;
constexpr int kCgMaxRows = 16384;  // rows per CTA (FP32; 8,192 in FP64)
constexpr int kCgMaxSmem = 227 * 1024 - 6144;  // dynamic; the rest is static
constexpr int kCgRing = 3;         // most ring slices per warp
constexpr int kMaxGridCtas = 256;

// 512 threads: 16 warps fill the schedulers about as well as 32 do (the work
// outside the product -- sums, scalars, barriers -- is per warp), leave 128
// registers for r and q, and halve the rings.  16,384 rows (2D), us per
// iteration: 1,024 threads 6.8 (before the scalars moved to one warp), 512
// threads 3.00, 256 threads 3.21; 32,761 rows: 512 threads 3.85, 256 5.39.
constexpr int kCgThreads = 512;
constexpr int kCgWarps = kCgThreads / 32;

// Dynamic shared memory: [p][x][1/diag, if it fits][resident slices][rings]
// [row lengths, 1 byte].  Warp w owns slices w, w + warps, ...; its first
// `resident` ones stay in shared memory.
struct CgLayout {
  int ok;         // 0: too large for this form
  int resident;   // slices of each warp that stay
  int ring;       // ring slices per warp (0: all are resident)
  int diag;       // 1: 1/diag in shared memory
  unsigned vec, slice, slice_off, ring_off, len_off, bytes;
};
__host__ __device__ inline CgLayout cg_layout(int esz, int rows, int slots) {
  CgLayout l = {};
  const int steps = (rows / 32 + kCgWarps - 1) / kCgWarps;
  l.vec = (unsigned)(rows * esz);
  l.slice = (unsigned)(32 * slots * (esz + 4));
  const unsigned step = l.slice * (unsigned)kCgWarps;
  const unsigned len = ((unsigned)rows + 15u) / 16u * 16u;
  for (int diag = 1; diag >= 0; --diag) {
    const unsigned fixed = (diag ? 3u : 2u) * l.vec + len;
    if (fixed >= (unsigned)kCgMaxSmem) continue;
    const int fit = (int)(((unsigned)kCgMaxSmem - fixed) / step);
    if (fit >= steps) {
      l.resident = steps;
      l.ring = 0;
    } else if (fit >= 2) {
      l.ring = fit < kCgRing ? fit : kCgRing;
      l.resident = fit - l.ring;
    } else {
      continue;
    }
    l.ok = 1;
    l.diag = diag;
    l.slice_off = (diag ? 3u : 2u) * l.vec;
    l.ring_off = l.slice_off + (unsigned)l.resident * step;
    l.len_off = l.ring_off + (unsigned)l.ring * step;
    l.bytes = l.len_off + len;
    return l;
  }
  return l;
}
// Workspace bytes of one CTA: the slices that are not resident, and 1/diag
// where shared memory does not hold it.
inline size_t cg_space_bytes(int esz, int rows, int slots) {
  const CgLayout l = cg_layout(esz, rows, slots);
  const int steps = (rows / 32 + kCgWarps - 1) / kCgWarps;
  const size_t b = (size_t)(steps - l.resident) * kCgWarps * l.slice + (l.diag ? 0 : l.vec);
  return (b + 255) / 256 * 256;
}

// What the CTAs of a whole-GPU launch exchange.
struct GridSpace {
  unsigned count;  // arrivals, zero before the launch
  unsigned late;   // set once a CTA's wait gave up, zero before the launch
  unsigned pad[30];
  double part[2][2][kMaxGridCtas];
  double flag[2];
};

// Shared state of one CTA.
struct __align__(16) CgShared {
  double part[2][2 * kMaxClusterSize];   // [parity][2 rank + value]
  double flag[2];
  double warp[2][kCgWarps];
  double scalar;  // what warp 0 made of a sum: alpha or beta
  int status;
  int late;
  uint64_t sum_bar[2], p_bar;
  uint64_t ring_bar[kCgWarps * kCgRing];
  unsigned long long sys_idx;
};

__device__ __forceinline__ uint32_t map_cluster(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_async(uint32_t addr, double a, double b, uint32_t bar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::
          "r"(addr), "d"(a), "d"(b), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void st_async(uint32_t addr, double a, uint32_t bar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(addr),
      "d"(a), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// An entry's column as the gather reads it: local ones the index within the
// CTA's rows; others bit 31 and, on a cluster, owner << 16 | index, on the
// whole GPU the column itself.
constexpr unsigned kRemote = 0x80000000u;

// Repeats `ready` until it holds, for kWaitLimitNs at most.
template <class F>
__device__ __forceinline__ bool wait_for(F ready) {
  if (ready()) return true;
  const uint64_t t0 = global_timer_ns();
  for (unsigned it = 1;; ++it) {
    if (ready()) return true;
    if ((it & 1023u) == 0 && global_timer_ns() - t0 > kWaitLimitNs) return false;
  }
}

// The CTA's sums of a and b, in warp 0 (all lanes); warp 0 alone goes on to
// the other CTAs' partials and the scalars made of them -- divisions, a square
// root and the trees in every warp were a large part of all instructions --
// while the other warps wait at the CTA barrier behind it.
__device__ __forceinline__ void cta_sum2(CgShared &sh, double &a, double &b) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double s = warp_sum2(a, b, lane);
  if ((lane & 15) == 0) sh.warp[lane >> 4][warp] = s;
  __syncthreads();
  if (warp != 0) return;
  static_assert(kCgWarps == 16, "lane l holds warp l % 16's partial of value l / 16");
  double v = sh.warp[lane >> 4][lane & 15];
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  a = __shfl_sync(0xffffffffu, v, 0);
  b = __shfl_sync(0xffffffffu, v, 16);
}

// What a CTA whose wait gave up sends for its partials: a NaN that no sum
// comes out as.  Whoever reads it among the partials knows that this sum, and
// everything since that wait, holds nothing.
constexpr unsigned long long kLatePartial = 0x7ff81a7e1a7e1a7eull;

// The CTAs of one cluster as the solve sees them.  A wait that gives up sets
// sh.late, which stays set: the CTA sends kLatePartial from then on, so every
// CTA leaves the solve at its next sum, and they meet at the hardware barrier
// that ends it (nobody leaves while messages may arrive).
struct ClusterTeam {
  static constexpr bool kGrid = false;
  cooperative_groups::cluster_group &cl;
  CgShared &sh;
  unsigned size, rank;
  unsigned n_sums, n_bars;  // so far: which barrier and phase comes next
  __device__ void start() { cl.sync(); }
  __device__ void finish() { cl.sync(); }
  // Between two solves: whether a wait gave up in any CTA (the same answer in
  // all of them).  The barriers' phases hold nothing then.
  __device__ bool any_late() {
    int l = 0;
    if (threadIdx.x < size)
      asm volatile("ld.shared::cluster.s32 %0, [%1];"
                   : "=r"(l)
                   : "r"(map_cluster(smem_addr(&sh.late), threadIdx.x))
                   : "memory");
    return __syncthreads_or(l) != 0;
  }
  // Every thread's p is written and everyone may read it.
  __device__ void barrier() {
    __syncthreads();
    const uint32_t bar = smem_addr(&sh.p_bar);
    if (threadIdx.x < size) mbar_arrive_cluster(map_cluster(bar, threadIdx.x));
    const uint32_t ph = n_bars++ & 1u;
    if (!wait_for([&] { return mbar_try_wait_cluster(bar, ph); })) sh.late = 1;
  }
  // Sums of a and b over the team and thread 0 of CTA 0's `flag` (2 after a
  // wait gave up in any CTA), in warp 0.  The partials are added in a fixed
  // tree, so all CTAs hold identical values.
  __device__ void sums(double &a, double &b, double &flag) {
    const int lane = threadIdx.x & 31;
    const unsigned par = n_sums & 1u, ph = (n_sums >> 1) & 1u;
    ++n_sums;
    cta_sum2(sh, a, b);
    if (threadIdx.x >= 32) return;
    const uint32_t bar = smem_addr(&sh.sum_bar[par]);
    const double f = __shfl_sync(0xffffffffu, flag, 0);
    if (lane == 0) mbar_arrive_expect_tx(bar, size * 16u + 8u);
    if (sh.late != 0) a = b = __longlong_as_double((long long)kLatePartial);
    if ((unsigned)lane < size) {
      const uint32_t to = map_cluster(bar, lane);
      st_async(map_cluster(smem_addr(&sh.part[par][2 * rank]), lane), a, b, to);
      if (rank == 0) st_async(map_cluster(smem_addr(&sh.flag[par]), lane), f, to);
    }
    const bool ok = wait_for([&] { return mbar_try_wait_cluster(bar, ph); });
    double v = (unsigned)(lane & 15) < size ? sh.part[par][2 * (lane & 15) + (lane >> 4)] : 0.0;
    const bool lost = !ok || (unsigned long long)__double_as_longlong(v) == kLatePartial;
    if (lost) sh.late = 1;
    __syncwarp();
    flag = sh.late == 0 ? sh.flag[par] : 2.0;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    a = __shfl_sync(0xffffffffu, v, 0);
    b = __shfl_sync(0xffffffffu, v, 16);
  }
  template <typename T>
  __device__ void publish(int, T) {}
  // p at a column word of another CTA (or this one); volatile: the values
  // change between barriers.
  template <typename T>
  __device__ T gather(unsigned word, uint32_t p_addr) const {
    const unsigned owner = (word & kRemote) ? (word >> 16) & 0x7fffu : rank;
    const uint32_t at = map_cluster(p_addr + (word & 0xffffu) * (unsigned)sizeof(T), owner);
    T v;
    if constexpr (sizeof(T) == 8)
      asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(at) : "memory");
    else
      asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
    return v;
  }
};

// All CTAs of a cooperative launch.  p is also kept in global memory, where
// other CTAs read it through L2; sums and barriers go through an arrival
// counter there, which one thread per CTA polls (all threads polling words of
// their own made a sum three times slower).  Waits are bounded as above; a CTA
// whose wait gave up sets space->late before it arrives again.
struct GridTeam {
  static constexpr bool kGrid = true;
  CgShared &sh;
  GridSpace *space;
  void *pg;
  unsigned size, rank;
  unsigned n_sums, n_bars;
  __device__ void start() { barrier(); }
  __device__ void finish() {}
  // One thread: release this CTA's writes (ordered before it by the CTA
  // barrier or the warp), arrive, wait for the others' arrivals.
  __device__ bool meet() {
    if (sh.late != 0) atomicExch(&space->late, 1u);
    __threadfence();
    atomicAdd(&space->count, 1u);
    const unsigned want = n_bars * size;
    return wait_for([&] { return (int)(ld_acquire_gpu(&space->count) - want) >= 0; });
  }
  __device__ void barrier() {
    ++n_bars;
    __syncthreads();
    if (threadIdx.x == 0 && !meet()) sh.late = 1;
    __syncthreads();
  }
  __device__ void sums(double &a, double &b, double &flag) {
    const int lane = threadIdx.x & 31;
    const unsigned par = n_sums++ & 1u;
    ++n_bars;
    cta_sum2(sh, a, b);
    if (threadIdx.x >= 32) return;
    if (lane == 0) {
      space->part[par][0][rank] = a;
      space->part[par][1][rank] = b;
      if (rank == 0) space->flag[par] = flag;
      if (!meet()) sh.late = 1;
    }
    __syncwarp();  // the other lanes' reads come after lane 0's meeting
    const bool lost = sh.late != 0 || __ldcg(&space->late) != 0;
    // CTA c in lane c % 32, then a tree
    double va = 0.0, vb = 0.0;
    for (unsigned c = lane; c < size; c += 32) {
      va += __ldcg(&space->part[par][0][c]);
      vb += __ldcg(&space->part[par][1][c]);
    }
    const double f = __ldcg(&space->flag[par]);
    const double v = warp_sum2(va, vb, lane);
    a = __shfl_sync(0xffffffffu, v, 0);
    b = __shfl_sync(0xffffffffu, v, 16);
    flag = lost ? 2.0 : f;
  }
  template <typename T>
  __device__ void publish(int row, T v) {
    static_cast<T *>(pg)[row] = v;
  }
  template <typename T>
  __device__ T gather(unsigned word, uint32_t p_addr) const {
    if (word & kRemote) return __ldcg(static_cast<const T *>(pg) + (word & 0x7fffffffu));
    T v;
    const uint32_t at = p_addr + word * (unsigned)sizeof(T);
    if constexpr (sizeof(T) == 8)
      asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(at) : "memory");
    else
      asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
    return v;
  }
};

// Slots [k0, k0 + N) of a lane's row added to `sum`; the N loads of each kind
// are in flight together.
template <typename T, int N, bool REMOTE, class Team>
__device__ __forceinline__ T cg_add(const Team &team, const T *val, const unsigned *col, int k0,
                                    int len, const T *p, uint32_t p_addr, T sum) {
  T v[N], g[N];
  unsigned c[N];
#pragma unroll
  for (int u = 0; u < N; ++u) c[u] = col[(k0 + u) * 32];
#pragma unroll
  for (int u = 0; u < N; ++u) v[u] = val[(k0 + u) * 32];
#pragma unroll
  for (int u = 0; u < N; ++u) {
    if constexpr (REMOTE) g[u] = team.template gather<T>(c[u], p_addr);
    else g[u] = p[c[u]];
  }
#pragma unroll
  for (int u = 0; u < N; ++u) {
    const T s = add_rn(sum, mul_rn(v[u], g[u]));
    sum = k0 + u < len ? s : sum;
  }
  return sum;
}

// (A p)_i of a lane's row in a slice of K slots (0: `slots` of them).
template <typename T, int K, bool REMOTE, class Team>
__device__ __forceinline__ T cg_product(const Team &team, const unsigned char *slice, int lane,
                                        int slots, int len, const T *p, uint32_t p_addr) {
  const T *val = reinterpret_cast<const T *>(slice) + lane;
  const unsigned *col = reinterpret_cast<const unsigned *>(
                            slice + 32 * (K > 0 ? K : slots) * sizeof(T)) + lane;
  T sum = T(0);
  if constexpr (K > 0) {
    sum = cg_add<T, K, REMOTE>(team, val, col, 0, len, p, p_addr, sum);
  } else {
    int k = 0;
    for (; k + 3 < slots; k += 4)
      sum = cg_add<T, 4, REMOTE>(team, val, col, k, len, p, p_addr, sum);
    for (; k < slots; ++k) sum = cg_add<T, 1, REMOTE>(team, val, col, k, len, p, p_addr, sum);
  }
  return sum;
}

struct CgArgs {
  ClusterSystem *systems;
  int n_systems;
  unsigned *queue;
  unsigned long long budget_ns;
  int rows;               // rows per CTA (a multiple of 32)
  int jac;                // Jacobi, else no preconditioner
  int slots;              // the launch's longest row
  unsigned char *space;   // per-CTA workspaces of space_bytes
  size_t space_bytes;
  GridSpace *grid;        // whole-GPU form only
  void *pg;
  int *err;
};

// A warp's place in its ring, carried from one system to the next.
struct RingAt {
  unsigned stage, phase;
};

// One solve; RT: rows per thread at most.
template <typename T, int RT, class Team>
__device__ __forceinline__ void cg_solve_slices(Team &team, const CgArgs &a, ClusterSystem &S,
                                                unsigned char *dyn, RingAt &ring_at) {
  constexpr int NT = kCgThreads, NW = kCgWarps;
  CgShared &sh = team.sh;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int rows = Team::kGrid ? a.rows : RT * NT;
  const int slots = a.slots;
  const CgLayout lay = cg_layout(sizeof(T), rows, slots);
  T *p = reinterpret_cast<T *>(dyn);
  T *xs = p + rows;
  unsigned char *lens = dyn + lay.len_off;
  unsigned char *mine = a.space + (size_t)blockIdx.x * a.space_bytes;
  T *ds = lay.diag ? xs + rows : reinterpret_cast<T *>(mine);
  unsigned char *stream = mine + (lay.diag ? 0 : lay.vec);  // slices past the resident ones
  unsigned char *kept = dyn + lay.slice_off + (size_t)warp * lay.resident * lay.slice;
  unsigned char *ring = dyn + lay.ring_off + (size_t)warp * lay.ring * lay.slice;
  const uint32_t ring_bar = smem_addr(&sh.ring_bar[warp * kCgRing]);
  const uint32_t p_addr = smem_addr(p);
  const int rank = (int)team.rank;
  const int row0 = rank * rows;
  const int nloc = max(0, min(rows, S.n - row0));
  const int *rp = S.rp, *ci = S.ci;
  const T *val = static_cast<const T *>(S.val);
  const T *b = static_cast<const T *>(S.b);
  T *x = static_cast<T *>(S.x);
  const double tol = S.tol;
  const long long maxiter = S.maxiter, miniter = S.miniter;
  double *hist = S.hist;
  const long long hist_cap = S.hist_cap;
  const uint64_t t0 = global_timer_ns();

  // rows into slices, 1/diag, x; slice u of warp w holds rows
  // (u NW + w) 32 .. + 31 of the CTA, so a warp reads only what it wrote
  const int live = (nloc + 31) / 32;  // slices with rows
  const int steps = live > warp ? (live - warp + NW - 1) / NW : 0;
  for (int u = 0; u < steps; ++u) {
    const int i = u * NT + t;
    unsigned char *sl = u < lay.resident
                            ? kept + (size_t)u * lay.slice
                            : stream + ((size_t)(u - lay.resident) * NW + warp) * lay.slice;
    T *sv = reinterpret_cast<T *>(sl) + lane;
    unsigned *sc = reinterpret_cast<unsigned *>(sl + 32 * slots * sizeof(T)) + lane;
    int len = 0;
    bool remote = false;
    if (i < nloc) {
      const int row = row0 + i;
      const int j0 = __ldg(rp + row);
      len = min(__ldg(rp + row + 1) - j0, slots);
      T d = T(0);
      for (int k = 0; k < slots; ++k) {
        const int c = k < len ? __ldg(ci + j0 + k) : row;
        const T v = k < len ? __ldg(val + j0 + k) : T(0);
        if (k < len && c == row) d = v;
        const unsigned at = (unsigned)(c - row0);
        unsigned word = at;
        if (at >= (unsigned)rows) {
          remote = true;
          if constexpr (Team::kGrid)
            word = kRemote | (unsigned)c;
          else
            word = kRemote | ((unsigned)c / (RT * NT)) << 16 | ((unsigned)c & (RT * NT - 1));
        }
        sv[k * 32] = v;
        sc[k * 32] = word;
      }
      ds[i] = a.jac ? T(1) / d : T(1);  // 1 r = r: z needs no second form
      const T xi = x[row];
      xs[i] = xi;
      p[i] = xi;
      team.publish(row, xi);
    } else {
      for (int k = 0; k < slots; ++k) {  // rows past the end: read, not used
        sv[k * 32] = T(0);
        sc[k * 32] = 0u;
      }
    }
    // the row's length, and whether any of the slice's rows leaves the CTA
    lens[i] = (unsigned char)(len | (__any_sync(0xffffffffu, remote) ? 0x80 : 0));
  }
  // The ring: a ring slice is refilled as soon as the warp has read it, with
  // the slice needed `ring` streamed steps later (round and round over the
  // warp's streamed slices).
  const int streamed = steps > lay.resident ? steps - lay.resident : 0;
  const unsigned char *src0 = stream + (size_t)warp * lay.slice;
  const unsigned hop = lay.slice * NW;
  const unsigned char *src = src0;  // lane 0: the next slice to copy
  int left = streamed;              // lane 0: slices before src wraps
  auto fill = [&](unsigned st) {
    mbar_arrive_expect_tx(ring_bar + 8 * st, lay.slice);
    bulk_g2s(smem_addr(ring) + st * lay.slice, src, lay.slice, ring_bar + 8 * st);
    src += hop;
    if (--left == 0) {
      src = src0;
      left = streamed;
    }
  };
  if (streamed > 0) {
    asm volatile("fence.proxy.async;" ::: "memory");  // the slices above are read by bulk copies
    __syncwarp();
    if (lane == 0)
      for (int k = 0, st = ring_at.stage; k < lay.ring; ++k) {
        fill((unsigned)st);
        st = st + 1 == lay.ring ? 0 : st + 1;
      }
  }
  unsigned stage = ring_at.stage, phase = ring_at.phase;  // the copy to read next
  team.start();

  T r[RT], q[RT];
#pragma unroll
  for (int u = 0; u < RT; ++u) r[u] = q[u] = T(0);
  // q = A p over the warp's slices; returns the thread's part of (p, q)
  auto product = [&](auto kc) -> double {
    constexpr int K = decltype(kc)::value;
    double pq = 0.0;
#pragma unroll
    for (int u = 0; u < RT; ++u) {
      if (u < steps) {
        const int i = u * NT + t;
        const bool kept_here = u < lay.resident;
        if (!kept_here &&
            !wait_for([&] { return mbar_try_wait(ring_bar + 8 * stage, phase); }))
          sh.late = 1;
        const unsigned char *sl =
            kept_here ? kept + (unsigned)u * lay.slice : ring + stage * lay.slice;
        const int ln = lens[i];
        const T qv =
            (ln & 0x80) ? cg_product<T, K, true>(team, sl, lane, slots, ln & 0x7f, p, p_addr)
                        : cg_product<T, K, false>(team, sl, lane, slots, ln, p, p_addr);
        if (!kept_here) {
          __syncwarp();
          if (lane == 0) fill(stage);
          if (++stage == (unsigned)lay.ring) {
            stage = 0;
            phase ^= 1u;
          }
        }
        if (i < nloc) {
          q[u] = qv;
          pq += (double)p[i] * (double)qv;
        }
      }
    }
    return pq;
  };

  double rz = 0.0, resid = 0.0;
  long long it = 0;
  int status = kRunning;
  bool first = true;
  while (true) {
    // q = A p, (p, q)
    double pq;
    if (slots == 5) pq = product(std::integral_constant<int, 5>{});
    else if (slots == 7) pq = product(std::integral_constant<int, 7>{});
    else pq = product(std::integral_constant<int, 0>{});
    double s0 = 0.0, s1 = 0.0, flag = 0.0;
    if (first) {
      // p = x0 in this pass: r = b - A x0 (cg.cpp:39-40), z = M r, p = z
      // (cg.cpp:43-44)
      first = false;
#pragma unroll
      for (int u = 0; u < RT; ++u) {
        const int i = u * NT + t;
        if (i < nloc) {
          const T ri = b[row0 + i] - q[u];
          r[u] = ri;
          const T zi = ds[i] * ri;
          q[u] = zi;
          s0 += (double)zi * (double)ri;
          s1 += (double)ri * (double)ri;
        }
      }
      team.sums(s0, s1, flag);
      if (warp == 0) {
        rz = s0;
        resid = cl_resid<T>(s1);
        if (flag > 1.0) status = MLSH_ERR_TIMEOUT;
        else if (maxiter <= 0) status = MLSH_SOLVER_MAXITER;
        if (lane == 0) sh.status = status;
      }
      __syncthreads();
      status = sh.status;
      if (status != kRunning) break;
#pragma unroll
      for (int u = 0; u < RT; ++u) {
        const int i = u * NT + t;
        if (i < nloc) {
          p[i] = q[u];
          team.publish(row0 + i, q[u]);
        }
      }
      team.barrier();
      continue;
    }
    double none = 0.0;
    team.sums(pq, none, flag);
    if (warp == 0 && lane == 0) sh.scalar = rz / pq;
    __syncthreads();
    const T alpha = (T)sh.scalar;
    // x += alpha p; r -= alpha q; (z, r), (r, r); time budget.  z takes q's
    // place.
#pragma unroll
    for (int u = 0; u < RT; ++u) {
      const int i = u * NT + t;
      if (i < nloc) {
        xs[i] = alpha * p[i] + xs[i];
        const T ri = -alpha * q[u] + r[u];
        r[u] = ri;
        const T zi = ds[i] * ri;
        q[u] = zi;
        s0 += (double)zi * (double)ri;
        s1 += (double)ri * (double)ri;
      }
    }
    flag = rank == 0 && t == 0 && global_timer_ns() - t0 > a.budget_ns ? 1.0 : 0.0;
    team.sums(s0, s1, flag);
    ++it;
    if (warp == 0) {
      const double beta = s0 / rz;
      rz = s0;
      resid = cl_resid<T>(s1);
      if (rank == 0 && lane == 0 && hist != nullptr && it <= hist_cap) hist[it - 1] = resid;
      if (flag > 1.0) status = MLSH_ERR_TIMEOUT;  // a wait gave up: nothing holds
      else if (resid < tol && miniter <= it) status = MLSH_SUCCESS;
      else if (isnan(resid)) status = MLSH_SOLVER_RESIDUAL_NAN;
      else if (it >= maxiter) status = MLSH_SOLVER_MAXITER;
      else if (flag > 0.0) status = MLSH_ERR_TIMEOUT;
      if (lane == 0) {
        sh.scalar = beta;
        sh.status = status;
      }
    }
    __syncthreads();
    status = sh.status;
    if (status != kRunning) break;
    const T beta = (T)sh.scalar;
    // p = z + beta p (cg.cpp:59)
#pragma unroll
    for (int u = 0; u < RT; ++u) {
      const int i = u * NT + t;
      if (i < nloc) {
        const T pi = q[u] + beta * p[i];
        p[i] = pi;
        team.publish(row0 + i, pi);
      }
    }
    team.barrier();
  }
  // the copies in flight land before their source or place is used again
  if (streamed > 0) {
    for (int k = 0; k < lay.ring; ++k) {
      wait_for([&] { return mbar_try_wait(ring_bar + 8 * stage, phase); });
      if (++stage == (unsigned)lay.ring) {
        stage = 0;
        phase ^= 1u;
      }
    }
    ring_at = RingAt{stage, phase};
  }
  for (int i = t; i < nloc; i += NT) x[row0 + i] = xs[i];
  if (rank == 0 && t == 0) {
    S.status = status;
    S.iters = it;
    S.resid = resid;
    if (a.err != nullptr && status == MLSH_ERR_TIMEOUT) atomicCAS(a.err, 0, MLSH_ERR_TIMEOUT);
  }
  team.finish();
}

__device__ __forceinline__ void cg_init_shared(CgShared &sh, unsigned team_size) {
  if (threadIdx.x == 0) {
    mbar_init(smem_addr(&sh.sum_bar[0]), 1);
    mbar_init(smem_addr(&sh.sum_bar[1]), 1);
    mbar_init(smem_addr(&sh.p_bar), team_size);
    for (int k = 0; k < kCgWarps * kCgRing; ++k) mbar_init(smem_addr(&sh.ring_bar[k]), 1);
    sh.late = 0;
    fence_mbar_init();
  }
  __syncthreads();
}

// Clusters taking systems from a queue (single solves, batches).
template <typename T, int RT>
__global__ void __launch_bounds__(kCgThreads, 1) cluster_cg_kernel(const CgArgs a) {
  cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
  extern __shared__ __align__(128) unsigned char cg_smem[];
  __shared__ CgShared sh;
  ClusterTeam team{cl, sh, cl.num_blocks(), cl.block_rank(), 0u, 0u};
  cg_init_shared(sh, team.size);
  cl.sync();
  RingAt ring_at{0u, 0u};
  while (true) {
    if (team.rank == 0 && threadIdx.x == 0) {
      const unsigned long long idx = atomicAdd(a.queue, 1u);
      for (unsigned q = 0; q < team.size; ++q) *cl.map_shared_rank(&sh.sys_idx, q) = idx;
    }
    cl.sync();
    const unsigned long long idx = sh.sys_idx;
    if (idx >= (unsigned long long)a.n_systems) break;
    cg_solve_slices<T, RT>(team, a, a.systems[idx], cg_smem, ring_at);
    if (team.any_late()) {  // the other clusters take what is left in the queue
      cl.sync();
      break;
    }
  }
}

// One system on all SMs (a cooperative launch, one CTA per SM).
template <typename T, int RT>
__global__ void __launch_bounds__(kCgThreads, 1) grid_cg_kernel(const CgArgs a) {
  extern __shared__ __align__(128) unsigned char cg_smem[];
  __shared__ CgShared sh;
  cg_init_shared(sh, 1);
  GridTeam team{sh, a.grid, a.pg, gridDim.x, blockIdx.x, 0u, 0u};
  RingAt ring_at{0u, 0u};
  cg_solve_slices<T, RT>(team, a, a.systems[0], cg_smem, ring_at);
}

}  // namespace mlsh
