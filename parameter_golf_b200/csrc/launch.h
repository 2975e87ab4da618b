// Kernel launch with programmatic dependency on the kernel before it in the stream (`chain_wait` / `chain_next` in common.cuh). Only
// for kernels in which every CTA calls chain_wait, and only up to CHAIN_ROWS token rows: where a launch gap is a visible share of a
// kernel. With every launch chained a step of 4,096 tokens took 4349 us instead of 4783, but one of 98,304 tokens got 3 % slower (CTAs
// of the next kernel settle on the SMs that finish first); at 16,384 it gains 2 %, at 24,576 nothing. The rows are those of the whole
// pass, which a product cannot see from its own sizes (a chunk of the output head has fewer, an optimizer product none): its
// caller hands them over. 0 rows: not a link of a chain. The sharded optimizer's products pass 0: they run beside the next
// forward, and a CTA that waits for its predecessor would hold shared and tensor memory that the forward could use.
#pragma once
#include <cuda_runtime.h>

namespace pgb {

constexpr long long CHAIN_ROWS = 16384;

template <typename... P, typename... A>
inline void launch_chained_clusters(long long rows, int ctas, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (rows > 0 && rows <= CHAIN_ROWS) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (ctas > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = ctas;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = n;
  cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

template <typename... P, typename... A>
inline void launch_chained(long long rows, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  launch_chained_clusters(rows, 1, kern, grid, block, smem, st, static_cast<A&&>(args)...);
}

}  // namespace pgb
