// Transposing warp reduction of FP64 values.
#pragma once
namespace hb {
// sum over the warp of NV values per lane: lane 2 i (NV 16) or i (NV 32) ends with the sum of v[i]; NV - 1
// (+ 1) additions per lane instead of the 5 NV of separate butterflies
template <int NV> __device__ __forceinline__ double warp_sums(double (&v)[NV], int lane) {
    static_assert(NV == 16 || NV == 32, "values per lane");
#pragma unroll
    for (int h = NV / 2, o = 16; h >= 1; h >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const double keep = up ? v[i + h] : v[i], send = up ? v[i] : v[i + h];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    if (NV == 16) v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    return v[0];
}
}  // namespace hb
