// pa_kern_short_free.cu -- the short-pair kernel in s16x2 lanes, M_GLOBAL_FREE.
#include "pa_kern_short.cuh"

namespace pa {
int dp_short_occupancy_free(int form) { return occ_short16<M_GLOBAL_FREE>(form); }
void dp_short_launch_free(int form, int grid, cudaStream_t st, const DpLaunch &L, const DpParams &P)
{
    go_short16<M_GLOBAL_FREE>(form, grid, st, L, P);
}
}  // namespace pa
