// pa_kern_long_free.cu -- the long-pair kernel, M_GLOBAL_FREE.
#include "pa_kern_long.cuh"

namespace pa {
int dp_long_occupancy_free(bool lanes16) { return occ_long_v<M_GLOBAL_FREE>(lanes16); }
void dp_long_launch_free(bool lanes16, int grid, cudaStream_t st, const DpLaunch &L, const LongQueue &Q,
                       const DpParams &P)
{
    go_long<M_GLOBAL_FREE>(lanes16, grid, st, L, Q, P);
}
}  // namespace pa
