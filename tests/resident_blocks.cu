// Blocks of the FP32 BiCGStab passes that are resident at once where the last
// one forms the sums, and up to how many it does.
#include "k_bicgstab.cu"

extern "C" int resident_blocks(int *resident, int *limit)
{
    using namespace pred;
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, 0) != cudaSuccess) return 1;
    const void *kernels[3] = {(const void *)k_bcg_p<float, true>, (const void *)k_bcg_s<float, true>,
                              (const void *)k_bcg_x<float, true>};
    const int limits[3] = {LAST_MAX<float>, LAST_MAX<float>, LAST_MAX_X};
    for (int q = 0; q < 3; ++q) {
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernels[q], NT, 0) != cudaSuccess) return 2;
        resident[q] = per_sm * prop.multiProcessorCount;
        limit[q] = limits[q];
    }
    return 0;
}
