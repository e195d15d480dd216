// pa_kern_cta.cu -- instantiations of the CTA-mode DP kernel for long pairs of the
// byte-compare class (the warps of a block pipeline the passes of one pair) and of the team
// kernel for those with few passes (teams of 4 warps, two pairs per block), with the
// branch-free top input.  Long pairs with unitary DNA scores run on dp_long (pa_long.cuh).
#include "pa_dp.cuh"

namespace pa {
namespace {
constexpr int kRowsCta = 16;
constexpr int kTeam = 4;

template <int MODE>
int occ_cta()
{
    static int per_sm = -1;
    if (per_sm < 0) {
        int v = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, dp_kernel_cta<L32, kRowsCta, MODE, true, 36>, kBlock, 0);
        per_sm = v < 1 ? 1 : v;
    }
    return per_sm;
}

template <int MODE>
int occ_team()
{
    static int per_sm = -1;
    if (per_sm < 0) {
        int v = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, dp_kernel_team<L32, kRowsCta, MODE, true, 36, kTeam>, kBlock,
                                                      0);
        per_sm = v < 1 ? 1 : v;
    }
    return per_sm;
}

template <int MODE>
void go_cta(int grid, cudaStream_t st, const DpLaunch &L, const DpParams &P)
{
    dp_kernel_cta<L32, kRowsCta, MODE, true, 36><<<grid, kBlock, 0, st>>>(L, P);
}

template <int MODE>
void go_team(int grid, cudaStream_t st, const DpLaunch &L, const DpParams &P)
{
    dp_kernel_team<L32, kRowsCta, MODE, true, 36, kTeam><<<grid, kBlock, 0, st>>>(L, P);
}
}  // namespace

int dp_cta_occupancy(int mode)
{
    return mode == M_LOCAL ? occ_cta<M_LOCAL>() : mode == M_GLOBAL ? occ_cta<M_GLOBAL>() : occ_cta<M_GLOBAL_FREE>();
}

void dp_cta_launch(int mode, int grid, cudaStream_t st, const DpLaunch &L, const DpParams &P)
{
    if (mode == M_LOCAL) go_cta<M_LOCAL>(grid, st, L, P);
    else if (mode == M_GLOBAL) go_cta<M_GLOBAL>(grid, st, L, P);
    else go_cta<M_GLOBAL_FREE>(grid, st, L, P);
}

int dp_team_occupancy(int mode)
{
    return mode == M_LOCAL ? occ_team<M_LOCAL>() : mode == M_GLOBAL ? occ_team<M_GLOBAL>() : occ_team<M_GLOBAL_FREE>();
}

void dp_team_launch(int mode, int grid, cudaStream_t st, const DpLaunch &L, const DpParams &P)
{
    if (mode == M_LOCAL) go_team<M_LOCAL>(grid, st, L, P);
    else if (mode == M_GLOBAL) go_team<M_GLOBAL>(grid, st, L, P);
    else go_team<M_GLOBAL_FREE>(grid, st, L, P);
}

}  // namespace pa
