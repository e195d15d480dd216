// pa_kern_long.cuh -- launcher body of the long-pair kernel, included once per
// pa_kern_long_*.cu (one translation unit per mode).
#include "pa_long.cuh"

namespace pa {
namespace {

template <class V, int MODE>
int occ_long()
{
    static int per_sm = -1;
    if (per_sm < 0) {
        int v = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, dp_long<V, MODE, kLongRows>, kBlock, 0);
        per_sm = v < 1 ? 1 : v;
    }
    return per_sm;
}

template <int MODE>
int occ_long_v(bool lanes16) { return lanes16 ? occ_long<L16, MODE>() : occ_long<L32, MODE>(); }

template <int MODE>
void go_long(bool lanes16, int grid, cudaStream_t st, const DpLaunch &L, const LongQueue &Q, const DpParams &P)
{
    if (lanes16) dp_long<L16, MODE, kLongRows><<<grid, kBlock, 0, st>>>(L, Q, P);
    else dp_long<L32, MODE, kLongRows><<<grid, kBlock, 0, st>>>(L, Q, P);
}

}  // namespace
}  // namespace pa
