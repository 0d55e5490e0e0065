// The RadixSpline's position estimate on its own, from a kernel outside the
// library: est[i], rate[i] of keys[i].
#include <cuda_runtime.h>

#include "gpujoin/device.cuh"

__global__ void k_estimate(gj::rs_view v, const uint64_t* keys, uint64_t m, uint32_t* est, float* rate) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i < m) est[i] = gj::rs_estimate(v, keys[i], rate + i);
}

extern "C" int rs_estimates(const gj_index* index, const uint64_t* d_keys, uint64_t m, uint32_t* d_est, float* d_rate) {
    gj::rs_view v;
    if (gj_index_device_view(index, &v, sizeof(v)) != GJ_OK) return 1;
    k_estimate<<<(unsigned)((m + 255) / 256), 256>>>(v, d_keys, m, d_est, d_rate);
    return cudaDeviceSynchronize() == cudaSuccess ? 0 : 2;
}
