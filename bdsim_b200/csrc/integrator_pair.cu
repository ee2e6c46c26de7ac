// integrator_pair.cu -- the FP64 plain form's pair kernel (--fmad=false; its
// pair products call fma() themselves).
#include "integrator_pair.cuh"

namespace bdcu {

template <int T, bool H>
static cudaError_t occupancy_pair_t(size_t smem, int* per_sm) {
    // the occupancy query, made first at plan time, lets the kernel use the
    // device's opt-in shared-memory maximum (no attribute call at launch)
    int dev = 0, v = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(integrate_pair_kernel<T, H>, cudaFuncAttributeMaxDynamicSharedMemorySize, v);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, integrate_pair_kernel<T, H>, 32 * T, smem);
}

template <int T, bool H>
static cudaError_t launch_pair_t(const RunArgs& a, int grid, size_t smem, cudaStream_t s) {
    integrate_pair_kernel<T, H><<<grid, 32 * T, smem, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_pair(int warps, bool hi, const RunArgs& a, int grid, size_t smem, cudaStream_t s) {
    switch (warps) {
        case 1: return launch_pair_t<1, true>(a, grid, smem, s);
        case 2: return launch_pair_t<2, true>(a, grid, smem, s);
        case 4: return hi ? launch_pair_t<4, true>(a, grid, smem, s) : launch_pair_t<4, false>(a, grid, smem, s);
        case 8: return launch_pair_t<8, true>(a, grid, smem, s);
        case 16: return launch_pair_t<16, true>(a, grid, smem, s);
    }
    return cudaErrorInvalidValue;
}

cudaError_t occupancy_pair(int warps, bool hi, size_t smem, int* per_sm) {
    switch (warps) {
        case 1: return occupancy_pair_t<1, true>(smem, per_sm);
        case 2: return occupancy_pair_t<2, true>(smem, per_sm);
        case 4: return hi ? occupancy_pair_t<4, true>(smem, per_sm) : occupancy_pair_t<4, false>(smem, per_sm);
        case 8: return occupancy_pair_t<8, true>(smem, per_sm);
        case 16: return occupancy_pair_t<16, true>(smem, per_sm);
    }
    return cudaErrorInvalidValue;
}

}  // namespace bdcu
