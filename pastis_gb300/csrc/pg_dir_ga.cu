// pg_dir_ga.cu -- the traceback-form DP and traceback kernels of
// X-drop (global alignment of each seed's region), in a translation unit of their own.
#include "pg_dir.h"

#include "pg_kernels_dir.cuh"

namespace pg {

cudaError_t dir_set_attributes_ga()
{
    const void *k[24] = {(const void *)k_ga_dir<0, false, false>, (const void *)k_ga_dir<1, false, false>,
                         (const void *)k_ga_dir<2, false, false>, (const void *)k_ga_dir<3, false, false>,
                         (const void *)k_ga_dir<0, true, false>, (const void *)k_ga_dir<1, true, false>,
                         (const void *)k_ga_dir<2, true, false>, (const void *)k_ga_dir<3, true, false>,
                         (const void *)k_ga_dir<0, false, true>, (const void *)k_ga_dir<1, false, true>,
                         (const void *)k_ga_dir<2, false, true>, (const void *)k_ga_dir<3, false, true>,
                         (const void *)k_ga_dir<0, true, true>, (const void *)k_ga_dir<1, true, true>,
                         (const void *)k_ga_dir<2, true, true>, (const void *)k_ga_dir<3, true, true>,
                         (const void *)k_ga_pair<0, false>, (const void *)k_ga_pair<1, false>,
                         (const void *)k_ga_pair<2, false>, (const void *)k_ga_pair<3, false>,
                         (const void *)k_ga_pair<0, true>, (const void *)k_ga_pair<1, true>,
                         (const void *)k_ga_pair<2, true>, (const void *)k_ga_pair<3, true>};
    cudaError_t e = cudaSuccess;
    for (int i = 0; i < 24 && e == cudaSuccess; ++i)
        e = cudaFuncSetAttribute(k[i], cudaFuncAttributeMaxDynamicSharedMemorySize, DIR16_DYN_SMEM);
    return e;
}

template <bool CHK, bool TAG>
static void dp_ga(int tie, const KParams &kp, uint64_t t0, uint64_t t1, const uint64_t *doff,
                   uint8_t *arena, int *dsc, int grid, int dyn, cudaStream_t st)
{
    const dim3 blk(WARPS * 32);
    switch (tie) {
    case 0: k_ga_dir<0, CHK, TAG><<<grid, blk, dyn, st>>>(kp, t0, t1, doff, arena, dsc); break;
    case 1: k_ga_dir<1, CHK, TAG><<<grid, blk, dyn, st>>>(kp, t0, t1, doff, arena, dsc); break;
    case 2: k_ga_dir<2, CHK, TAG><<<grid, blk, dyn, st>>>(kp, t0, t1, doff, arena, dsc); break;
    default: k_ga_dir<3, CHK, TAG><<<grid, blk, dyn, st>>>(kp, t0, t1, doff, arena, dsc); break;
    }
}

template <bool TAG>
static void pair_ga(int tie, const KParams &kp, uint64_t t0, uint64_t t1, const uint64_t *doff,
                    uint8_t *arena, int *dsc, int grid, int dyn, cudaStream_t st)
{
    const dim3 blk(WARPS * 32);
    switch (tie) {
    case 0: k_ga_pair<0, TAG><<<grid, blk, dyn, st>>>(kp, t0, t1, doff, arena, dsc); break;
    case 1: k_ga_pair<1, TAG><<<grid, blk, dyn, st>>>(kp, t0, t1, doff, arena, dsc); break;
    case 2: k_ga_pair<2, TAG><<<grid, blk, dyn, st>>>(kp, t0, t1, doff, arena, dsc); break;
    default: k_ga_pair<3, TAG><<<grid, blk, dyn, st>>>(kp, t0, t1, doff, arena, dsc); break;
    }
}

int dir_run_ga(int tie, const KParams &kp, uint64_t t0, uint64_t t1, const uint64_t *doff,
               uint8_t *arena, int *dsc, int grid, int dyn, int grid_tb, bool chk, cudaStream_t st)
{
    int launches = 2;
    if (kp.tag) dp_ga<false, true>(tie, kp, t0, t1, doff, arena, dsc, grid, dyn, st);
    else dp_ga<false, false>(tie, kp, t0, t1, doff, arena, dsc, grid, dyn, st);
    if (kp.dir16_pair) {
        cudaMemsetAsync(kp.counter, 0, sizeof(unsigned int), st);
        if (kp.tag) pair_ga<true>(tie, kp, t0, t1, doff, arena, dsc, grid, dyn, st);
        else pair_ga<false>(tie, kp, t0, t1, doff, arena, dsc, grid, dyn, st);
        ++launches;
    }
    if (chk) {
        cudaMemsetAsync(kp.counter, 0, sizeof(unsigned int), st);
        if (kp.tag) dp_ga<true, true>(tie, kp, t0, t1, doff, arena, dsc, grid, dyn, st);
        else dp_ga<true, false>(tie, kp, t0, t1, doff, arena, dsc, grid, dyn, st);
        ++launches;
    }
    if (dir_walk_warps(kp, t1 - t0)) k_tb_ga<true><<<grid_tb, 256, 0, st>>>(kp, t0, t1, doff, arena, dsc);
    else k_tb_ga<false><<<grid_tb, 256, 0, st>>>(kp, t0, t1, doff, arena, dsc);
    return launches;
}

}  // namespace pg
