// FP64 instantiation of the step kernels (built with -fmad=false so that
// every product and sum is rounded as in the serial reference).
#define GF_FP64_UNIT
#include "gf_kernels_impl.cuh"

template struct GfKernels<double>;

#include <cstdio>

namespace {
namespace gfk {
// Check of the bounded barrier of the thermal sweeps: CTA `absent` of a
// two-CTA co-resident launch never arrives; the other waits at most `limit`
// polls and leaves with therm_sync's give-up value (absent = -1: both arrive
// and pass).
__global__ void k_barrier_probe(unsigned *slot, int absent, int limit, int *passed) {
    if ((int)blockIdx.x == absent) return;
    const int r = therm_sync(slot, false, limit);
    if (threadIdx.x == 0) passed[blockIdx.x] = r >= 0 ? 1 : 0;
}
} // namespace gfk
} // namespace

extern "C" int gf_grid_barrier_selftest(int absent_cta, long long limit, int *passed) {
    if (!passed || absent_cta < -1 || absent_cta > 1 || limit < 1) return GF_ERR_ARG;
    unsigned *bar = nullptr;
    int *d_passed = nullptr;
    cudaError_t e = cudaMalloc(&bar, sizeof(unsigned));
    if (e == cudaSuccess) e = cudaMalloc(&d_passed, 2 * sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(bar, 0, sizeof(unsigned));
    if (e == cudaSuccess) e = cudaMemset(d_passed, 0xff, 2 * sizeof(int));
    if (e == cudaSuccess) {
        cudaLaunchConfig_t lc = {};
        lc.gridDim = dim3(2);
        lc.blockDim = dim3(32);
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        lc.attrs = attr;
        lc.numAttrs = 1;
        e = cudaLaunchKernelEx(&lc, gfk::k_barrier_probe, bar, absent_cta, (int)(limit < (1 << 30) ? limit : (1 << 30)), d_passed);
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpy(passed, d_passed, 2 * sizeof(int), cudaMemcpyDeviceToHost);
    cudaFree(bar);
    cudaFree(d_passed);
    if (e != cudaSuccess) {
        std::fprintf(stderr, "geoflac_gb300: CUDA error in gf_grid_barrier_selftest: %s\n", cudaGetErrorString(e));
        return GF_ERR_CUDA;
    }
    return passed[0] == 0 || passed[1] == 0 ? GF_ERR_TIMEOUT : GF_OK;
}
