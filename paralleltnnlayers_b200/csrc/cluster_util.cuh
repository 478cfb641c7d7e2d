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

// ---- the same by stores --------------------------------------------------------------------------------------------------
// Every CTA stores its values into the memory of the one that adds them: a store is on its way while the next is issued, and one
// barrier is enough.  4096 -> 64 dense at batch 64 (16 x 32 values of 8 CTAs: 3.2k cycles by reads) 13.2 -> 12.6 us, 96 -> 48 channels 8x20 of
// the reshaped-CP forward 11.4 -> 10.9.  For the large tiles of plane_gemm_kernel, which a thread would store value by value, reads are
// faster (64 x 512 7x7 layer at R = 64, all on FFMA, 72 us by reads, 94 by stores).
struct ClusterSum {
  // this CTA's slice of all CTAs' tiles, [CTA][per], ClusterSum::floats() of memory that nothing else uses, at the same offset in every
  // CTA: a store to another CTA goes to this one's own address there
  float* in;
  int splits, per;
  unsigned rank;
  static __host__ __device__ constexpr int floats(int n) { return n + 8; }   // (at most 8 CTAs)
  // at the start of the kernel, by all threads of the cluster
  __device__ ClusterSum(float* in_, int n, int splits_) : in(in_), splits(splits_), per((n + splits_ - 1) / splits_), rank(0) {
    if (splits == 1) return;
    rank = cooperative_groups::this_cluster().block_rank();
    asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
  }
  // before the first put: the other CTAs have started
  __device__ void ready() const {
    if (splits > 1) asm volatile("barrier.cluster.wait;" ::: "memory");
  }
  __device__ void put(int i, float v) const {
    const int q = i / per;
    cooperative_groups::this_cluster().map_shared_rank(in, q)[rank * per + (i - q * per)] = v;
  }
  // the sums of this CTA's slice of n values
  template <typename Out>
  __device__ void sum(int n, int tid, int nthreads, Out out) const {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    const int first = (int)rank * per, count = min(n - first, per);
    for (int i = tid; i < count; i += nthreads) {
      float y[8];
#pragma unroll
      for (int p = 0; p < 8; ++p) y[p] = p < splits ? in[p * per + i] : 0.f;
      float v = y[0];
#pragma unroll
      for (int p = 1; p < 8; ++p)
        if (p < splits) v += y[p];
      out(first + i, v);
    }
  }
};

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
