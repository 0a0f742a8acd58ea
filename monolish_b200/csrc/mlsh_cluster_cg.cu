// Launchers of the slice-form CG kernels (mlsh_cluster_cg.cuh): clusters that
// take systems from a queue, and one system on all SMs.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "mlsh_cluster_cg.cuh"
#include "mlsh_core.cuh"

namespace mlsh {

namespace {

using CgKernelFn = void (*)(const CgArgs);

// The kernel for a number of rows per CTA, or null.
template <typename T, bool GRID, int RT>
constexpr CgKernelFn pick() {
  if constexpr (GRID) return grid_cg_kernel<T, RT>;
  else return cluster_cg_kernel<T, RT>;
}
template <typename T, bool GRID>
CgKernelFn cg_kernel_t(int rows) {
  if (rows <= 2 * kCgThreads) return pick<T, GRID, 2>();
  if (rows <= 4 * kCgThreads) return pick<T, GRID, 4>();
  if (rows <= 8 * kCgThreads) return pick<T, GRID, 8>();
  if constexpr (!GRID || sizeof(T) == 4)
    if (rows <= 16 * kCgThreads) return pick<T, GRID, 16>();
  if constexpr (!GRID && sizeof(T) == 4)
    if (rows <= 32 * kCgThreads) return pick<T, GRID, 32>();
  return nullptr;
}
CgKernelFn cg_kernel(bool grid, int dtype, int rows) {
  if (dtype == MLSH_F64)
    return grid ? cg_kernel_t<double, true>(rows) : cg_kernel_t<double, false>(rows);
  return grid ? cg_kernel_t<float, true>(rows) : cg_kernel_t<float, false>(rows);
}

int set_attributes() {
  static std::once_flag once;
  static int status = MLSH_SUCCESS;
  std::call_once(once, [] {
    for (int rows = 1024; rows <= kCgMaxRows; rows <<= 1)
      for (int dtype : {MLSH_F64, MLSH_F32})
        for (int grid = 0; grid < 2; ++grid) {
          CgKernelFn k = cg_kernel(grid != 0, dtype, rows);
          if (k == nullptr) continue;
          if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kCgMaxSmem) !=
                  cudaSuccess ||
              (!grid && cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed,
                                             1) != cudaSuccess)) {
            cudaGetLastError();
            status = MLSH_ERR_CUDA;
          }
        }
  });
  return status;
}

cudaLaunchConfig_t config(int dtype, int rows, int slots, int ctas, cudaStream_t stream,
                          cudaLaunchAttribute *attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas, 1, 1);
  cfg.blockDim = dim3(kCgThreads, 1, 1);
  cfg.dynamicSmemBytes = cg_layout(dtype_size(dtype), rows, slots).bytes;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

void cluster_attr(cudaLaunchAttribute *attr, int csize) {
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = (unsigned)csize;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
}

size_t round256(size_t b) { return (b + 255) / 256 * 256; }

}  // namespace

int cluster_cg_slots(int kind, int dtype, int rows, int longest_row) {
  if (kind != 0 || rows <= 0 || longest_row < 1 || longest_row > kCgMaxRow) return 0;
  return cg_layout(dtype_size(dtype), rows, longest_row).ok ? longest_row : 0;
}

size_t cluster_cg_workspace(int dtype, int rows, int slots) {
  return slots > 0 ? cg_space_bytes(dtype_size(dtype), rows, slots) : 0;
}

int cluster_cg_max_active(int dtype, int rpc, int csize, int slots) {
  CgKernelFn k = cg_kernel(false, dtype, rpc);
  if (set_attributes() != MLSH_SUCCESS || k == nullptr) return 0;
  cudaLaunchAttribute attr[1];
  cluster_attr(attr, csize);
  cudaLaunchConfig_t cfg = config(dtype, rpc, slots, csize, nullptr, attr);
  int most = 0;
  if (cudaOccupancyMaxActiveClusters(&most, (void *)k, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return most;
}

int cluster_cg_launch(int dtype, bool jac, ClusterSystem *d_systems, int n_systems,
                      unsigned *d_queue, int rpc, int csize, int n_clusters, double budget_s,
                      cudaStream_t stream, int slots, void *space) {
  const int most = cluster_cg_max_active(dtype, rpc, csize, slots);
  if (most < 1) return MLSH_NOT_IMPL;
  CgArgs c = {};
  c.systems = d_systems;
  c.n_systems = n_systems;
  c.queue = d_queue;
  c.budget_ns = (unsigned long long)(budget_s * 1e9);
  c.rows = rpc;
  c.jac = jac ? 1 : 0;
  c.slots = slots;
  c.space = static_cast<unsigned char *>(space);
  c.space_bytes = cluster_cg_workspace(dtype, rpc, slots);
  cudaLaunchAttribute attr[1];
  cluster_attr(attr, csize);
  cudaLaunchConfig_t cfg =
      config(dtype, rpc, slots, csize * std::min(n_clusters, most), stream, attr);
  MLSH_CUDA_TRY(cudaLaunchKernelEx(&cfg, cg_kernel(false, dtype, rpc), c));
  return MLSH_SUCCESS;
}

// Past 4,096 FP64 rows a CTA the kernel engine, which streams from HBM, is the
// faster one: 512,000 rows (3D) 20.2 us per iteration against its 29.7,
// 1,030,301 rows 43.8 against 41.3.
constexpr int kGridMaxBytes = 32768;  // of p per CTA

int grid_cg_rows(int dtype, int64_t n, int num_sms) {
  const int ctas = std::min(num_sms, kMaxGridCtas);
  const int64_t rows = ((n + ctas - 1) / ctas + 31) / 32 * 32;
  return rows * dtype_size(dtype) > kGridMaxBytes ? 0 : (int)rows;
}

size_t grid_cg_space(int dtype, int64_t n, int rows, int slots) {
  const size_t ctas = (size_t)((n + rows - 1) / rows);
  return round256(sizeof(GridSpace)) + round256((size_t)n * dtype_size(dtype)) +
         ctas * cluster_cg_workspace(dtype, rows, slots);
}

int grid_cg_launch(const Handle &h, int dtype, bool jac, ClusterSystem *d_system, int64_t n,
                   int rows, int slots, void *space, double budget_s, cudaStream_t stream) {
  CgKernelFn k = cg_kernel(true, dtype, rows);
  if (set_attributes() != MLSH_SUCCESS || k == nullptr) return MLSH_NOT_IMPL;
  CgArgs c = {};
  c.systems = d_system;
  c.n_systems = 1;
  c.budget_ns = (unsigned long long)(budget_s * 1e9);
  c.rows = rows;
  c.jac = jac ? 1 : 0;
  c.slots = slots;
  unsigned char *p = static_cast<unsigned char *>(space);
  c.grid = reinterpret_cast<GridSpace *>(p);
  p += round256(sizeof(GridSpace));
  c.pg = p;
  p += round256((size_t)n * dtype_size(dtype));
  c.space = p;
  c.space_bytes = cluster_cg_workspace(dtype, rows, slots);
  c.err = h.err_flag;
  MLSH_CUDA_TRY(cudaMemsetAsync(space, 0, 2 * sizeof(unsigned), stream));  // count, late
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cudaLaunchConfig_t cfg =
      config(dtype, rows, slots, (int)((n + rows - 1) / rows), stream, attr);
  if (cudaLaunchKernelEx(&cfg, k, c) != cudaSuccess) {
    cudaGetLastError();  // not resident all at once: the kernel engine takes it
    return MLSH_NOT_IMPL;
  }
  return MLSH_SUCCESS;
}

}  // namespace mlsh
