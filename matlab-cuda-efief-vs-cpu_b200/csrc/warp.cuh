// Warp reductions of many values at once.
#pragma once

// Sums of n = 32 or 16 values over the warp: lane l is left with the sum of
// value l mod n.  Each step hands half of the values still held to the other
// half of the lanes, so n - 1 exchanges replace 5 n.
template <int n>
__device__ __forceinline__ double warp_sums(double (&d)[n], int lane) {
    if (n == 16)
#pragma unroll
        for (int i = 0; i < n; i++) d[i] += __shfl_xor_sync(0xffffffffu, d[i], 16);
#pragma unroll
    for (int o = n / 2; o > 0; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < n / 2; i++) {
            if (i >= o) break;
            const double keep = up ? d[i + o] : d[i], send = up ? d[i] : d[i + o];
            d[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return d[0];
}
