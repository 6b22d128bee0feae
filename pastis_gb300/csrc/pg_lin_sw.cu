// pg_lin_sw.cu -- the linear-gap alignment (pg_lin.cuh) of Smith-Waterman, in a
// translation unit of its own.
#define PG_LIN_UNIT
#include "pg_lin.cuh"

namespace pg {
template cudaError_t lin_attributes<false>(int *);
template void lin_count<false>(const LinParams &, int, cudaStream_t);
template int lin_align<false>(const LinParams &, uint32_t, uint32_t, uint32_t, int, int, cudaStream_t);
}  // namespace pg
