// pa_kern_short32_local.cu -- the short-pair kernel in s32 lanes, M_LOCAL.
#include "pa_kern_short.cuh"

namespace pa {
cudaError_t dp_short32_allow_local() { return allow_profiles<M_LOCAL>(); }
int dp_short32_occupancy_local(int scoring, int dim) { return occ_short32<M_LOCAL>(scoring, dim); }
void dp_short32_launch_local(int scoring, int grid, cudaStream_t st, const DpLaunch &L, const DpParams &P)
{
    go_short32<M_LOCAL>(scoring, grid, st, L, P);
}
}  // namespace pa
