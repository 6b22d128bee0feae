// pg_lin.h -- host launchers of the linear-gap alignment (kernels in pg_lin.cuh,
// compiled per mode in pg_lin_ga.cu and pg_lin_sw.cu).  All launches go to
// stream st; errors surface through cudaGetLastError.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace pg {

struct LinParams;

// lets k_lin_dp take its dynamic shared memory; its resident blocks per SM
template <bool XDROP>
cudaError_t lin_attributes(int *blocks_per_sm);
// class sizes and totals (lp.tot) of the pairs [lp.p0, lp.p1); two launches
template <bool XDROP>
void lin_count(const LinParams &lp, int nsm, cudaStream_t st);
// their list, DP, traceback and results, after lin_count, which found `entries`
// list entries (`wide` regions among them of lin_wide columns) and `jobs`; returns the launches
template <bool XDROP>
int lin_align(const LinParams &lp, uint32_t entries, uint32_t wide, uint32_t jobs, int nsm, int max_blocks,
              cudaStream_t st);

}  // namespace pg
