// recip_ge1 against the IEEE division for every float of [1, inf]: out[0] differing bits in [1, 1e37), out[1] the
// largest difference in units of the last place beyond, out[2] NaN for NaN
#include "nsfv1_recip.cuh"

__global__ void k_check(unsigned* out) {
    for (unsigned i = 0x3f800000u + blockIdx.x * blockDim.x + threadIdx.x; i <= 0x7f800000u; i += gridDim.x * blockDim.x) {
        const float x = __uint_as_float(i);
        const int d = abs((int)(__float_as_uint(1.0f / x) - __float_as_uint(nsfv1::recip_ge1(x))));
        if (d == 0) continue;
        if (x < 1.0e37f) atomicAdd(out, 1u);
        else atomicMax(out + 1, (unsigned)d);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) out[2] = isnan(nsfv1::recip_ge1(__uint_as_float(0x7fc00000u)));
}

extern "C" int recip_check(unsigned* host) {
    unsigned* out = nullptr;
    if (cudaMalloc(&out, 12) != cudaSuccess) return 1;
    cudaMemset(out, 0, 12);
    k_check<<<1024, 256>>>(out);
    const bool ok = cudaMemcpy(host, out, 12, cudaMemcpyDeviceToHost) == cudaSuccess;
    cudaFree(out);
    return ok ? 0 : 1;
}
