// warp_sums.cuh -- sums of several values over the lanes of a warp.
#pragma once
#include <cuda_runtime.h>

namespace ecg {

// Sum v[0..M) (M a power of two, at most 32) over the warp's lanes: every
// step exchanges half of the values a lane still holds, so M - 1 +
// log2(32 / M) values travel instead of the 5 M of a butterfly per value.  Lane i returns the
// sum of value i / (32 / M).
template <int M>
__device__ __forceinline__ double warp_transpose_sum(double (&v)[M])
{
    const int lane = threadIdx.x & 31;
    int s = 16;
#pragma unroll
    for (int h = M / 2; h >= 1; h /= 2) {
        const bool up = (lane & s) != 0;
#pragma unroll
        for (int i = 0; i < h; i++) {
            const double send = up ? v[i] : v[i + h];
            const double keep = up ? v[i + h] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, s);
        }
        s /= 2;
    }
#pragma unroll
    for (int q = 16 / M; q >= 1; q /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], q);
    return v[0];
}

}  // namespace ecg
