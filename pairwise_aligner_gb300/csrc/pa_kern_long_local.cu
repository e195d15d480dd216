// pa_kern_long_local.cu -- the long-pair kernel, M_LOCAL.
#include "pa_kern_long.cuh"

namespace pa {
int dp_long_occupancy_local(bool lanes16) { return occ_long_v<M_LOCAL>(lanes16); }
void dp_long_launch_local(bool lanes16, int grid, cudaStream_t st, const DpLaunch &L, const LongQueue &Q,
                       const DpParams &P)
{
    go_long<M_LOCAL>(lanes16, grid, st, L, Q, P);
}
}  // namespace pa
