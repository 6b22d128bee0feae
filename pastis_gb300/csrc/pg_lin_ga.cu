// pg_lin_ga.cu -- the linear-gap alignment (pg_lin.cuh) of X-drop, in a
// translation unit of its own (it compiles in parallel with the others).
#define PG_LIN_UNIT
#include "pg_lin.cuh"

namespace pg {
template cudaError_t lin_attributes<true>(int *);
template void lin_count<true>(const LinParams &, int, cudaStream_t);
template int lin_align<true>(const LinParams &, uint32_t, uint32_t, uint32_t, int, int, cudaStream_t);
}  // namespace pg
