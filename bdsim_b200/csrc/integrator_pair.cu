// integrator_pair.cu -- the FP64 plain form's pair kernel (--fmad=false; its
// pair products call fma() themselves).
#include "integrator_pair.cuh"

namespace bdcu {

template <int T>
static cudaError_t occupancy_pair_t(size_t smem, int* per_sm) {
    // the occupancy query, made first at plan time, lets the kernel use the
    // device's opt-in shared-memory maximum (no attribute call at launch)
    int dev = 0, v = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(integrate_pair_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, v);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, integrate_pair_kernel<T>, 32 * T, smem);
}

template <int T>
static cudaError_t launch_pair_t(const RunArgs& a, int grid, size_t smem, cudaStream_t s) {
    integrate_pair_kernel<T><<<grid, 32 * T, smem, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_pair(int warps, const RunArgs& a, int grid, size_t smem, cudaStream_t s) {
    switch (warps) {
        case 4: return launch_pair_t<4>(a, grid, smem, s);
        case 8: return launch_pair_t<8>(a, grid, smem, s);
        case 16: return launch_pair_t<16>(a, grid, smem, s);
    }
    return cudaErrorInvalidValue;
}

cudaError_t occupancy_pair(int warps, size_t smem, int* per_sm) {
    switch (warps) {
        case 4: return occupancy_pair_t<4>(smem, per_sm);
        case 8: return occupancy_pair_t<8>(smem, per_sm);
        case 16: return occupancy_pair_t<16>(smem, per_sm);
    }
    return cudaErrorInvalidValue;
}

}  // namespace bdcu
