// pa_kern_long_band.cu -- the banded DP of long pairs on the pass queue, M_BAND.  Passes hold
// 512 rows (16 per thread), as the window table does.
#include "pa_kern_long.cuh"

namespace pa {
int dp_long_band_occupancy(bool lanes16)
{
    static int per_sm[2] = {-1, -1};
    int &v = per_sm[lanes16];
    if (v < 0) {
        if (lanes16) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, dp_long<L16, M_BAND, 16>, kBlock, 0);
        else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, dp_long<L32, M_BAND, 16>, kBlock, 0);
        if (v < 1) v = 1;
    }
    return v;
}

void dp_long_band_launch(bool lanes16, int grid, cudaStream_t st, const DpLaunch &L, const LongQueue &Q,
                         const DpParams &P, unsigned long long *epoch)
{
    if (lanes16) {
        k_band_plan<2><<<1, 1024, 0, st>>>(L, Q, epoch);
        dp_long<L16, M_BAND, 16><<<grid, kBlock, 0, st>>>(L, Q, P);
    } else {
        k_band_plan<1><<<1, 1024, 0, st>>>(L, Q, epoch);
        dp_long<L32, M_BAND, 16><<<grid, kBlock, 0, st>>>(L, Q, P);
    }
}
}  // namespace pa
