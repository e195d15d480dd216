// pa_kern_short_local.cu -- the short-pair kernel in s16x2 lanes, M_LOCAL.
#include "pa_kern_short.cuh"

namespace pa {
int dp_short_occupancy_local(int form) { return occ_short16<M_LOCAL>(form); }
void dp_short_launch_local(int form, int grid, cudaStream_t st, const DpLaunch &L, const DpParams &P)
{
    go_short16<M_LOCAL>(form, grid, st, L, P);
}
}  // namespace pa
