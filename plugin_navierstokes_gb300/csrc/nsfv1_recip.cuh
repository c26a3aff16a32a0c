// nsfv1_recip.cuh -- the reciprocal of the network's activation.
#pragma once

namespace nsfv1 {

// 1 / x for x >= 1: the hardware estimate and one Newton-Raphson step in fused multiply-adds
// (Markstein, "Computation of elementary functions on the IBM RISC System/6000", 1990).
// Compared with the IEEE division for every float of [1, 1e37): the same bits; beyond, where
// |z / x| < 1e-34, within one unit in the last place (tests/test_gpu_recip.py). Without the
// division's branch, which kept neighbouring elements of the activation from overlapping.
__device__ __forceinline__ float recip_ge1(const float x) {
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    const float e = fmaf(-x, r, 1.0f), q = fmaf(r, e, r);
    return x < 1.0e38f ? q : r;   // x = inf: r = 0
}

}  // namespace nsfv1
