// Helpers of kernels whose CTAs share one output tile over a thread-block cluster (grid z), each with a part of the sum.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"

namespace b200cp {

// ---- sum of a cluster's partial tiles ----------------------------------------------------------------------------------
// Every CTA of the cluster (at most 8) has left its partial tile in shared memory; CTA q adds slice q of all of them in CTA order
// (the result does not depend on scheduling) and hands each sum to `put`.  All CTAs are read at once: a read of another CTA's memory
// takes half a microsecond.
template <typename Put>
__device__ __forceinline__ void cluster_sum(float* tile, int n, int splits, int tid, int nthreads, Put put) {
  namespace cg = cooperative_groups;
  if (splits == 1) {
    __syncthreads();
    for (int i = tid; i < n; i += nthreads) put(i, tile[i]);
    return;
  }
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  const int q = (int)cl.block_rank(), per = (n + splits - 1) / splits;
  const int e = min(n, (q + 1) * per);
  const float* from[8];
#pragma unroll
  for (int p = 0; p < 8; ++p) from[p] = cl.map_shared_rank(tile, p < splits ? p : 0);
  for (int i = q * per + tid; i < e; i += nthreads) {
    float y[8];
#pragma unroll
    for (int p = 0; p < 8; ++p) y[p] = p < splits ? from[p][i] : 0.f;
    float v = y[0];
#pragma unroll
    for (int p = 1; p < 8; ++p)
      if (p < splits) v += y[p];
    put(i, v);
  }
  cl.sync();   // nobody reads this CTA's tile any more
}

template <typename... KArgs, typename... Args>
cudaError_t launch_cluster(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, int cluster_z,
                           bool programmatic, Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  static const bool off = [] {
    const char* e = getenv("B200CP_PDL");
    return e && e[0] == '0';
  }();
  at[0].val.programmaticStreamSerializationAllowed = programmatic && !off ? 1 : 0;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = 1;
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = (unsigned)cluster_z;
  cfg.attrs = at;
  cfg.numAttrs = cluster_z > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

// K units per CTA of a cluster: as many CTAs (at most 8 per cluster) as fill the GPU once, at least `least` units each
inline int pick_cluster(long tiles, int units, int least, int sm_count) {
  int s = 1;
  while (s < 8 && tiles * s * 2 <= sm_count && units / (s * 2) >= least) s *= 2;
  return s;
}

}  // namespace b200cp
