// pa_kern_short32_free.cu -- the short-pair kernel in s32 lanes, M_GLOBAL_FREE.
#include "pa_kern_short.cuh"

namespace pa {
cudaError_t dp_short32_allow_free() { return allow_profiles<M_GLOBAL_FREE>(); }
int dp_short32_occupancy_free(int scoring, int dim) { return occ_short32<M_GLOBAL_FREE>(scoring, dim); }
void dp_short32_launch_free(int scoring, int grid, cudaStream_t st, const DpLaunch &L, const DpParams &P)
{
    go_short32<M_GLOBAL_FREE>(scoring, grid, st, L, P);
}
}  // namespace pa
