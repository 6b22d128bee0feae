// pg_dir_sw.cu -- the traceback-form DP and traceback kernels of
// Smith-Waterman (local alignment), in a translation unit of their own.
#include "pg_dir.h"

#include "pg_kernels_dir.cuh"

namespace pg {

cudaError_t dir_set_attributes_sw()
{
    const void *k[16] = {(const void *)k_sw_dir<0, false, false>, (const void *)k_sw_dir<1, false, false>,
                         (const void *)k_sw_dir<2, false, false>, (const void *)k_sw_dir<3, false, false>,
                         (const void *)k_sw_dir<0, true, false>, (const void *)k_sw_dir<1, true, false>,
                         (const void *)k_sw_dir<2, true, false>, (const void *)k_sw_dir<3, true, false>,
                         (const void *)k_sw_dir<0, false, true>, (const void *)k_sw_dir<1, false, true>,
                         (const void *)k_sw_dir<2, false, true>, (const void *)k_sw_dir<3, false, true>,
                         (const void *)k_sw_dir<0, true, true>, (const void *)k_sw_dir<1, true, true>,
                         (const void *)k_sw_dir<2, true, true>, (const void *)k_sw_dir<3, true, true>};
    cudaError_t e = cudaSuccess;
    for (int i = 0; i < 16 && e == cudaSuccess; ++i)
        e = cudaFuncSetAttribute(k[i], cudaFuncAttributeMaxDynamicSharedMemorySize, DIR16_DYN_SMEM);
    return e;
}

template <bool CHK, bool TAG>
static void dp_sw(int tie, const KParams &kp, uint64_t t0, uint64_t t1, const uint64_t *doff,
                   uint8_t *arena, int *dsc, int grid, int dyn, cudaStream_t st)
{
    const dim3 blk(WARPS * 32);
    switch (tie) {
    case 0: k_sw_dir<0, CHK, TAG><<<grid, blk, dyn, st>>>(kp, t0, t1, doff, arena, dsc); break;
    case 1: k_sw_dir<1, CHK, TAG><<<grid, blk, dyn, st>>>(kp, t0, t1, doff, arena, dsc); break;
    case 2: k_sw_dir<2, CHK, TAG><<<grid, blk, dyn, st>>>(kp, t0, t1, doff, arena, dsc); break;
    default: k_sw_dir<3, CHK, TAG><<<grid, blk, dyn, st>>>(kp, t0, t1, doff, arena, dsc); break;
    }
}

int dir_run_sw(int tie, const KParams &kp, uint64_t t0, uint64_t t1, const uint64_t *doff,
               uint8_t *arena, int *dsc, int grid, int dyn, int grid_tb, bool chk, cudaStream_t st)
{
    int launches = 2;
    // with the half-warp pairs
    if (kp.tag) dp_sw<false, true>(tie, kp, t0, t1, doff, arena, dsc, grid, dyn, st);
    else dp_sw<false, false>(tie, kp, t0, t1, doff, arena, dsc, grid, dyn, st);
    if (chk) {
        cudaMemsetAsync(kp.counter, 0, sizeof(unsigned int), st);
        if (kp.tag) dp_sw<true, true>(tie, kp, t0, t1, doff, arena, dsc, grid, dyn, st);
        else dp_sw<true, false>(tie, kp, t0, t1, doff, arena, dsc, grid, dyn, st);
        ++launches;
    }
    if (dir_walk_warps(kp, t1 - t0)) k_tb_sw<true><<<grid_tb, 256, 0, st>>>(kp, t0, t1, doff, arena, dsc);
    else k_tb_sw<false><<<grid_tb, 256, 0, st>>>(kp, t0, t1, doff, arena, dsc);
    return launches;
}

}  // namespace pg
