// Warp reductions, packed-vector arithmetic and the PTX of the FP64 tensor-core kernels, shared by them.
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

// One FP64 product of fragments, 8 x 4 by 4 x 8: d += a b (mma.sync; tcgen05 has no f64 kind)
__device__ __forceinline__ void dmma_884(double &d0, double &d1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

}  // namespace uegccd
