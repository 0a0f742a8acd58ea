// Grouping entries by row (or column) and ordering each group: the kernels
// behind COO sorting and CRS transposition where no row is extremely long.
//
// An entry (key, other, value) goes to its key's group by counting: one pass
// counts the entries of every key, a scan turns the counts into group starts,
// a scatter places 16-byte records {other, input position, value} through an
// atomic cursor per group (in any order), and each group is then put into
// (other, input position) order on its own.  Those pairs are distinct, so the
// result does not depend on the order in which the scatter's atomics ran.
//
// Why not the least-significant-digit radix sort: it moves every (key,
// position) pair once per 8 key bits -- six passes for a 2^21 x 2^21 matrix,
// five launches each -- and gathers the values at random at the end, where
// this takes one random 16-byte store per entry and two streaming reads.
// Measured times of both forms stand at mlsh_coo_sort's dispatch.
#pragma once
#include "mlsh_core.cuh"

namespace mlsh {

template <typename T>
struct __align__(16) SortRec {
  int other;     // the column (COO) or row (transpose)
  unsigned pos;  // input position
  T val;
};
static_assert(sizeof(SortRec<double>) == 16 && sizeof(SortRec<float>) == 16,
              "one 16-byte store per entry");

// Groups up to kSegCap entries are ordered by the warp that owns them, as
// many consecutive groups at a time as fit kSegCap records of shared memory
// (four warps: 24 KB + flags, 8 CTAs per SM): every entry counts the entries
// of its group that precede it, which for the 7-8 entries of a stencil row
// is 8 broadcast reads and no exchange at all.  Longer groups take the CTA
// kernel (bitonic sort in shared memory) up to kLongCap entries.
constexpr int kSegCap = 384;
constexpr int kSegWarps = 4;
constexpr int kLongCap = 16384;
constexpr int kLongThreads = 1024;
constexpr int kLongSmem = kLongCap * (8 + 2);

// Device words of one job.
struct SortFlags {
  int bad;              // an index was out of range
  unsigned longest;     // entries of the largest group
  unsigned n_long;      // groups over kSegCap
  unsigned far;         // sampled warps whose entries' rows lie far apart
};

// Where the ordered entries go (null: not wanted).
template <typename T>
struct SortOut {
  int *key;
  int *other;
  T *val;
  unsigned *pos;
};

template <typename T>
struct GroupArgs {
  const SortRec<T> *rec;
  const unsigned *ends;    // group g holds records [ends[g - 1], ends[g])
  int n_keys;
  unsigned *kept;          // COUNT: entries each group keeps
  const unsigned *starts;  // WRITE: where each group's entries go (null: in place)
  unsigned *long_ids;
  SortFlags *flags;
  int collect;             // this launch lists the groups over kSegCap
  SortOut<T> out;
};

__device__ __forceinline__ unsigned long long sort_key(int other, unsigned pos) {
  return (unsigned long long)(unsigned)other << 32 | pos;
}

// One warp per 32 groups.  MERGE keeps of equal `other`s only the last input
// position.  WRITE = false counts what each group keeps, true writes it.
template <typename T, bool MERGE, bool WRITE>
__global__ void __launch_bounds__(kSegWarps * 32) order_groups(const GroupArgs<T> a) {
  __shared__ SortRec<T> s_rec[kSegWarps][kSegCap];
  __shared__ unsigned char s_group[kSegWarps][kSegCap];
  __shared__ unsigned char s_keep[kSegWarps][MERGE ? kSegCap : 1];
  __shared__ unsigned s_end[kSegWarps][33];  // group ends within the segment, from [1]
  __shared__ unsigned s_cnt[kSegWarps][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long g0 = ((long long)blockIdx.x * kSegWarps + w) * 32;
  if (g0 >= a.n_keys) return;
  const int ng = (int)min(32ll, a.n_keys - g0);
  const unsigned base0 = g0 > 0 ? a.ends[g0 - 1] : 0u;
  const unsigned end = a.ends[g0 + min(lane, ng - 1)];
  unsigned begin = __shfl_up_sync(0xffffffffu, end, 1);
  if (lane == 0) begin = base0;
  if (lane >= ng) begin = end;
  SortRec<T> *rec = s_rec[w];
  int first = 0;
  while (first < ng) {
    const unsigned base = __shfl_sync(0xffffffffu, begin, first);
    // the groups from `first` on that fit the segment together
    const unsigned fit = __ballot_sync(
        0xffffffffu, lane >= first && lane < ng && end - base <= (unsigned)kSegCap);
    const int many = __popc(fit);
    if (many == 0) {  // group `first` alone is larger
      if (lane == 0 && a.collect) a.long_ids[atomicAdd(&a.flags->n_long, 1u)] = (unsigned)(g0 + first);
      ++first;
      continue;
    }
    const int last = first + many;
    const unsigned m = __shfl_sync(0xffffffffu, end, last - 1) - base;
    for (unsigned e = lane; e < m; e += 32) rec[e] = a.rec[base + e];
    if (lane >= first && lane < last) {
      s_end[w][lane - first + 1] = end - base;
      for (unsigned e = begin - base; e < end - base; ++e)
        s_group[w][e] = (unsigned char)(lane - first);
    }
    if (lane == 0) s_end[w][0] = 0u;
    if constexpr (!WRITE) s_cnt[w][lane] = 0u;
    __syncwarp();
    if constexpr (MERGE) {
      for (unsigned e = lane; e < m; e += 32) {
        const int g = s_group[w][e];
        const int c = rec[e].other;
        const unsigned p = rec[e].pos;
        bool keep = true;
        for (unsigned j = s_end[w][g]; j < s_end[w][g + 1]; ++j)
          keep = keep && !(rec[j].other == c && rec[j].pos > p);
        s_keep[w][e] = keep ? 1 : 0;
        if constexpr (!WRITE)
          if (keep) atomicAdd(&s_cnt[w][g], 1u);
      }
      __syncwarp();
    }
    if constexpr (WRITE) {
      for (unsigned e = lane; e < m; e += 32) {
        if constexpr (MERGE)
          if (!s_keep[w][e]) continue;
        const int g = s_group[w][e];
        const SortRec<T> r = rec[e];
        const unsigned long long k = sort_key(r.other, r.pos);
        const unsigned j0 = s_end[w][g];
        unsigned rank = 0;
        for (unsigned j = j0; j < s_end[w][g + 1]; ++j) {
          bool less = sort_key(rec[j].other, rec[j].pos) < k;
          if constexpr (MERGE) less = less && s_keep[w][j];
          rank += less ? 1u : 0u;
        }
        const long long key = g0 + first + g;
        const unsigned q = (a.starts ? a.starts[key] : base + j0) + rank;
        if (a.out.key) a.out.key[q] = (int)key;
        if (a.out.other) a.out.other[q] = r.other;
        if (a.out.val) a.out.val[q] = r.val;
        if (a.out.pos) a.out.pos[q] = r.pos;
      }
    } else {
      if (lane < many) a.kept[g0 + first + lane] = s_cnt[w][lane];
    }
    __syncwarp();
    first = last;
  }
}

// One CTA per listed group of kSegCap < len <= kLongCap entries.
template <typename T, bool MERGE, bool WRITE>
__global__ void __launch_bounds__(kLongThreads, 1) order_long_groups(const GroupArgs<T> a) {
  extern __shared__ __align__(16) unsigned char long_smem[];
  unsigned long long *keys = reinterpret_cast<unsigned long long *>(long_smem);
  unsigned short *at = reinterpret_cast<unsigned short *>(long_smem + kLongCap * 8);
  __shared__ unsigned s_warp[kLongThreads / 32];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const unsigned n_long = a.flags->n_long;
  for (unsigned q = blockIdx.x; q < n_long; q += gridDim.x) {
    const unsigned g = a.long_ids[q];
    const unsigned b = g > 0 ? a.ends[g - 1] : 0u, len = a.ends[g] - b;
    unsigned n2 = 1024;
    while (n2 < len) n2 <<= 1;
    for (unsigned i = t; i < n2; i += kLongThreads) {
      keys[i] = i < len ? sort_key(a.rec[b + i].other, a.rec[b + i].pos) : ~0ull;
      at[i] = (unsigned short)i;
    }
    __syncthreads();
    for (unsigned k = 2; k <= n2; k <<= 1)
      for (unsigned j = k >> 1; j > 0; j >>= 1) {
        for (unsigned i = t; i < n2 / 2; i += kLongThreads) {
          const unsigned lo = 2 * i - (i & (j - 1)), hi = lo + j;
          const unsigned long long x = keys[lo], y = keys[hi];
          if ((x > y) == ((lo & k) == 0)) {
            keys[lo] = y;
            keys[hi] = x;
            const unsigned short s = at[lo];
            at[lo] = at[hi];
            at[hi] = s;
          }
        }
        __syncthreads();
      }
    // consecutive slices of 1,024 in order; a kept entry ends its run
    unsigned done = 0;
    for (unsigned i0 = 0; i0 < len; i0 += kLongThreads) {
      const unsigned i = i0 + t;
      const bool keep = i < len && (!MERGE || i + 1 == len ||
                                    (keys[i] >> 32) != (keys[i + 1] >> 32));
      const unsigned mask = __ballot_sync(0xffffffffu, keep);
      if (lane == 0) s_warp[warp] = __popc(mask);
      __syncthreads();
      unsigned before = 0, all = 0;
      for (int v = 0; v < kLongThreads / 32; ++v) {
        const unsigned c = s_warp[v];
        if (v < warp) before += c;
        all += c;
      }
      if constexpr (WRITE) {
        if (keep) {
          const unsigned o = (a.starts ? a.starts[g] : b) + done + before +
                             __popc(mask & ((1u << lane) - 1u));
          const SortRec<T> r = a.rec[b + at[i]];
          if (a.out.key) a.out.key[o] = (int)g;
          if (a.out.other) a.out.other[o] = r.other;
          if (a.out.val) a.out.val[o] = r.val;
          if (a.out.pos) a.out.pos[o] = r.pos;
        }
      }
      done += all;
      __syncthreads();
    }
    if constexpr (!WRITE)
      if (t == 0) a.kept[g] = done;
  }
}

}  // namespace mlsh
