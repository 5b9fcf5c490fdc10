// Kernel launches: persistent, occupancy-sized grids, and launch helpers that report a refused
// launch to their caller.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <string>
#include <utility>

#include "../../include/ssfft.h"

int ssfft_internal_fail(int code, const std::string &msg);

#define CK(call)                                                                          \
  do {                                                                                    \
    cudaError_t e_ = (call);                                                              \
    if (e_ != cudaSuccess)                                                                \
      return ssfft_internal_fail(SSFFT_E_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

#define CKR(expr)           \
  do {                      \
    int r_ = (expr);        \
    if (r_ != 0) return r_; \
  } while (0)

// ---------------------------------------------------------------------------------------
// persistent grids
// ---------------------------------------------------------------------------------------
// Blocks of a persistent launch: as many as are resident at once on the device (occupancy
// x SMs), but no more than there are items.
struct OccKey {
  const void *f;
  int threads;
  size_t smem;
  int dev;
  int cluster;  // 0: blocks; C: clusters of C blocks
  bool operator<(const OccKey &o) const {
    if (f != o.f) return f < o.f;
    if (threads != o.threads) return threads < o.threads;
    if (smem != o.smem) return smem < o.smem;
    if (dev != o.dev) return dev < o.dev;
    return cluster < o.cluster;
  }
};

static std::mutex g_occ_mutex;
static std::map<OccKey, int> g_occ;

template <typename F> static int resident_blocks(F f, int threads, size_t smem, int dev) {
  const OccKey key{(const void *)f, threads, smem, dev, 0};
  {
    std::lock_guard<std::mutex> lk(g_occ_mutex);
    auto it = g_occ.find(key);
    if (it != g_occ.end()) return it->second;
  }
  int per_sm = 0, sms = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, threads, smem) != cudaSuccess)
    per_sm = 1;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) sms = 148;
  cudaGetLastError();  // of these queries: launches report their own errors
  const int n = std::max(1, per_sm) * std::max(1, sms);
  std::lock_guard<std::mutex> lk(g_occ_mutex);
  g_occ[key] = n;
  return n;
}

template <typename F>
static int persistent_grid(F f, int threads, size_t smem, long long items, int dev) {
  return (int)std::max(1LL, std::min<long long>(items, resident_blocks(f, threads, smem, dev)));
}

// Clusters of C blocks resident at once (a cluster must fit the SMs of one GPC).
template <typename... A>
static int resident_clusters(void (*f)(A...), int C, int threads, size_t smem, int dev) {
  const OccKey key{(const void *)f, threads, smem, dev, C};
  {
    std::lock_guard<std::mutex> lk(g_occ_mutex);
    auto it = g_occ.find(key);
    if (it != g_occ.end()) return it->second;
  }
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, f, &cfg) != cudaSuccess || n < 1) n = 1;
  cudaGetLastError();  // of the query
  std::lock_guard<std::mutex> lk(g_occ_mutex);
  g_occ[key] = n;
  return n;
}

// Status of a launch.  The error is returned at once and taken off the runtime's record: the
// passes of a projection are launched one after the other, and the occupancy queries between
// them clear that record, so a pass refused in the middle would go unnoticed at the end.
static int launch_status(cudaError_t e) {
  if (e == cudaSuccess) return 0;
  cudaGetLastError();
  return ssfft_internal_fail(SSFFT_E_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
}

// Persistent launch of a cluster kernel of `threads` threads a block: as many clusters as
// are resident at once, but no more than there are items.
template <typename... P, typename... A>
static int launch_clustered(void (*f)(P...), int C, int threads, size_t smem, long long items,
                            int dev, cudaStream_t stream, A &&...args) {
  const int ncl = (int)std::max(1LL, std::min<long long>(items, resident_clusters(f, C, threads, smem, dev)));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(ncl * C));
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return launch_status(cudaLaunchKernelEx(&cfg, f, std::forward<A>(args)...));
}

// Launch in stream order.  With `pdl`, a kernel that calls pdl_wait() may start while the kernel
// before it in the stream still runs.
template <typename... P, typename... A>
static int launch_kernel(bool pdl, void (*f)(P...), int grid, int threads, size_t smem,
                         cudaStream_t stream, A &&...args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = at;
  cfg.numAttrs = pdl ? 1 : 0;
  return launch_status(cudaLaunchKernelEx(&cfg, f, std::forward<A>(args)...));
}
