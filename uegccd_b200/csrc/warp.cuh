// Warp reductions and packed-vector arithmetic shared by the kernels.
#pragma once

#include <cstdint>

namespace uegccd {

// The warp's sums of N values (a power of two), in a fixed order: the lanes halve the values
// between them, then the lanes, 2 N - 2 + log2(32 / N) exchanges for what N separate reductions
// take 5 N.  Returns the index of the sum left in v[0], or -1 for a lane that holds a copy.
template <int N>
__device__ __forceinline__ int warp_sums(double (&v)[N])
{
    const int l = threadIdx.x & 31;
    int at = 0;
#pragma unroll
    for (int o = 16, n = N / 2; o > 0; o >>= 1, n >>= 1) {
        const bool up = l & o;
        if (n > 0) {
#pragma unroll
            for (int k = 0; k < N / 2; k++)
                if (k < n) {
                    const double give = up ? v[k] : v[k + n], keep = up ? v[k + n] : v[k];
                    v[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
            at += up ? n : 0;
        } else {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        }
    }
    return (l & (32 / N - 1)) == 0 ? at : -1;
}

// The warp's maximum of non-negative values (a NaN counts as 0).
__device__ __forceinline__ double warp_max(double x)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(fmax(0.0, x));
    const unsigned hi = (unsigned)(b >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)b : 0u);
    return __longlong_as_double((long long)((unsigned long long)mh << 32 | ml));
}

// Plane-wave vectors packed one component per byte (x | y << 8 | z << 16, two's complement).
// |n_a - n_k|^2 = |n_a|^2 + |n_k|^2 - 2 n_a . n_k is one 4-way byte dot product of neg2(n_a) and n_k
// beside the norms; every component is at most 63 in magnitude (checked when the batch is made), so
// that its double fits a signed byte.
__device__ __forceinline__ int neg2(int p)
{
    const int x = (int8_t)p, y = (int8_t)(p >> 8), z = (int8_t)(p >> 16);
    return ((-2 * x) & 0xff) | (((-2 * y) & 0xff) << 8) | (((-2 * z) & 0xff) << 16);
}

}  // namespace uegccd
