// pa_kern_short_global.cu -- the short-pair kernel in s16x2 lanes, M_GLOBAL.
#include "pa_kern_short.cuh"

namespace pa {
int dp_short_occupancy_global(int form) { return occ_short16<M_GLOBAL>(form); }
void dp_short_launch_global(int form, int grid, cudaStream_t st, const DpLaunch &L, const DpParams &P)
{
    go_short16<M_GLOBAL>(form, grid, st, L, P);
}
}  // namespace pa
