// pa_kern_short.cuh -- launcher body of the short-pair kernel, included by pa_kern_short_*.cu
// (s16x2 lanes) and pa_kern_short32_*.cu (s32 lanes), one translation unit per mode.
#include "pa_short.cuh"
#include "pa_launch.h"

namespace pa {
namespace {

constexpr int kProfileThreads = 128;

// Blocks per SM: the same for every group size (registers and shared memory set it).
template <class V, int SC, int MODE, int R, int NT>
int occ_short(int smem)
{
    int per_sm = 32;
    for (int k = 0; k < 4; ++k) {
        int v = 0;
        const void *f = k == 0   ? (const void *)dp_short<V, SC, MODE, 32, R, NT>
                        : k == 1 ? (const void *)dp_short<V, SC, MODE, 16, R, NT>
                        : k == 2 ? (const void *)dp_short<V, SC, MODE, 8, R, NT>
                                 : (const void *)dp_short<V, SC, MODE, 4, R, NT>;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, f, NT, smem);
        per_sm = v < per_sm ? v : per_sm;
    }
    cudaGetLastError();
    return per_sm < 1 ? 1 : per_sm;
}

template <class V, int SC, int MODE, int R, int NT>
void go_short(int grid, int smem, cudaStream_t st, const DpLaunch &L, const DpParams &P)
{
    if (L.G == 4) dp_short<V, SC, MODE, 4, R, NT><<<grid, NT, smem, st>>>(L, P);
    else if (L.G == 8) dp_short<V, SC, MODE, 8, R, NT><<<grid, NT, smem, st>>>(L, P);
    else if (L.G == 16) dp_short<V, SC, MODE, 16, R, NT><<<grid, NT, smem, st>>>(L, P);
    else dp_short<V, SC, MODE, 32, R, NT><<<grid, NT, smem, st>>>(L, P);
}

// Dynamic shared memory of the profile kernels: a uint4 per thread and symbol.
inline int profile_bytes(int dim) { return ((dim + 3) & ~3) * kProfileThreads * 16; }

// Lanes and scoring of a class; form 0 holds 16 rows per thread, form 1 (s16x2 only) 32.
template <int MODE>
int occ_short16(int form)
{
    return form == 1 ? occ_short<L16, SC_TABLE, MODE, 32, kBlock>(0) : occ_short<L16, SC_TABLE, MODE, 16, kBlock>(0);
}

template <int MODE>
void go_short16(int form, int grid, cudaStream_t st, const DpLaunch &L, const DpParams &P)
{
    if (form == 1) go_short<L16, SC_TABLE, MODE, 32, kBlock>(grid, 0, st, L, P);
    else go_short<L16, SC_TABLE, MODE, 16, kBlock>(grid, 0, st, L, P);
}

// Lets the profile kernels use the shared memory of the largest matrix (32 symbols) on the current
// device.  The attribute belongs to the device, so every context asks for its own.
template <int MODE>
cudaError_t allow_profiles()
{
    constexpr int NT = kProfileThreads, bytes = 32 * NT * 16;
    const void *f[4] = {(const void *)dp_short<L32, SC_PROFILE, MODE, 32, 16, NT>,
                        (const void *)dp_short<L32, SC_PROFILE, MODE, 16, 16, NT>,
                        (const void *)dp_short<L32, SC_PROFILE, MODE, 8, 16, NT>,
                        (const void *)dp_short<L32, SC_PROFILE, MODE, 4, 16, NT>};
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < 4 && e == cudaSuccess; ++k)
        e = cudaFuncSetAttribute(f[k], cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    return e;
}

template <int MODE>
int occ_short32(int scoring, int dim)
{
    if (scoring == SC_TABLE) return occ_short<L32, SC_TABLE, MODE, 16, kBlock>(0);
    if (scoring == SC_BYTES) return occ_short<L32, SC_BYTES, MODE, 16, kBlock>(0);
    return occ_short<L32, SC_PROFILE, MODE, 16, kProfileThreads>(profile_bytes(dim));
}

template <int MODE>
void go_short32(int scoring, int grid, cudaStream_t st, const DpLaunch &L, const DpParams &P)
{
    if (scoring == SC_TABLE) go_short<L32, SC_TABLE, MODE, 16, kBlock>(grid, 0, st, L, P);
    else if (scoring == SC_BYTES) go_short<L32, SC_BYTES, MODE, 16, kBlock>(grid, 0, st, L, P);
    else go_short<L32, SC_PROFILE, MODE, 16, kProfileThreads>(grid, profile_bytes(L.mdim), st, L, P);
}

}  // namespace
}  // namespace pa
