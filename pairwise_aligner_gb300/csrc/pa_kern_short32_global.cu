// pa_kern_short32_global.cu -- the short-pair kernel in s32 lanes, M_GLOBAL.
#include "pa_kern_short.cuh"

namespace pa {
cudaError_t dp_short32_allow_global() { return allow_profiles<M_GLOBAL>(); }
int dp_short32_occupancy_global(int scoring, int dim) { return occ_short32<M_GLOBAL>(scoring, dim); }
void dp_short32_launch_global(int scoring, int grid, cudaStream_t st, const DpLaunch &L, const DpParams &P)
{
    go_short32<M_GLOBAL>(scoring, grid, st, L, P);
}
}  // namespace pa
