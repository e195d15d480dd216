// pa_kern_cluster.cu -- instantiations and launchers of the cluster-mode DP kernel
// (the largest byte-compare pairs: a cluster of kClusterBlocks co-scheduled blocks pipelines
// the row passes of one pair).
#include "pa_dp.cuh"

namespace pa {
namespace {
constexpr int kRowsCl = 16;

template <int MODE>
void *cluster_fn()
{
    return (void *)dp_kernel_cluster<L32, kRowsCl, MODE, true, 36, kClusterBlocks>;
}

void *pick(int mode)
{
    return mode == M_LOCAL ? cluster_fn<M_LOCAL>() : mode == M_GLOBAL ? cluster_fn<M_GLOBAL>() : cluster_fn<M_GLOBAL_FREE>();
}

cudaLaunchConfig_t config_of(int grid, cudaStream_t st, cudaLaunchAttribute *attr)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid, 1, 1);
    cfg.blockDim = dim3(kBlock, 1, 1);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kClusterBlocks;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}
}  // namespace

// Blocks (a multiple of the cluster size) of a cluster-mode launch that are resident at once,
// at most `max_blocks`.
int dp_cluster_grid(int mode, int max_blocks)
{
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = config_of(max_blocks, nullptr, attr);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, pick(mode), &cfg) != cudaSuccess || clusters < 1) {
        cudaGetLastError();
        clusters = 1;
    }
    const int grid = clusters * kClusterBlocks;
    const int cap = (max_blocks / kClusterBlocks) * kClusterBlocks;
    return grid < cap ? grid : (cap > 0 ? cap : kClusterBlocks);
}

cudaError_t dp_cluster_launch(int mode, int grid, cudaStream_t st, const DpLaunch &L, const DpParams &P)
{
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = config_of(grid, st, attr);
    DpLaunch l = L;
    DpParams p = P;
    void *args[2] = {&l, &p};
    return cudaLaunchKernelExC(&cfg, pick(mode), args);
}

}  // namespace pa
