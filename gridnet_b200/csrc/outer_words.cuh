// What the persistent kernels of the loop (outer_small.cu, outer_held.cu) exchange between CTAs: 64-bit words that carry the
// number of the step they belong to, so that a reader needs neither flags nor fences.
#pragma once
#include "common.cuh"

namespace gn {

__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ unsigned long long ld_word(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void ld_words(const unsigned long long *p, unsigned long long &a, unsigned long long &b)
{
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ void st_words(unsigned long long *p, unsigned long long a, unsigned long long b)
{
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ unsigned long long cell_word(float v, unsigned step) { return (unsigned long long)step << 32 | __float_as_uint(v); }

// a wait ran out
__device__ __forceinline__ void report_wait(int *error_flag, int *status)
{
    if (error_flag) *error_flag = 1;
    if (status) *status = 1;
}

// One warp: adds up `count` pairs of doubles, a line each, whose low eight bits are `tag`, looking until all are there (or
// gave_up), and returns (mean, rstd). Everything down to the result is done at every look, not only at the last: after
// some thousand cycles without double-precision work the first such instructions take 4500 cycles, which then keeps all blocks
// waiting for each other.
__device__ __forceinline__ float2 watch_sums(const unsigned long long *sums, int count, int line, unsigned long long tag, double per_cell, float eps,
                                             int lane, unsigned limit, bool &gave_up)
{
    for (unsigned spins = 0;;) {
        double sm = 0.0, sq = 0.0;
        bool there = true;
        for (int i = lane; i < count; i += 64) {  // two at a time
            const bool two = i + 32 < count;
            unsigned long long v[4] = {tag, tag, tag, tag};
            ld_words(sums + line * i, v[0], v[1]);
            if (two) ld_words(sums + line * (i + 32), v[2], v[3]);
#pragma unroll
            for (int e = 0; e < 4; ++e) there &= (v[e] & 0xff) == tag;
            sm += __longlong_as_double((long long)(v[0] & ~0xffull));
            sq += __longlong_as_double((long long)(v[1] & ~0xffull));
            if (two) {
                sm += __longlong_as_double((long long)(v[2] & ~0xffull));
                sq += __longlong_as_double((long long)(v[3] & ~0xffull));
            }
        }
        sm = warp_sum(sm);
        sq = warp_sum(sq);
        const double mean = sm * per_cell;
        double var = fma(-mean, mean, sq * per_cell);
        if (var < 0.0) var = 0.0;
        const float2 result = make_float2((float)mean, (float)rsqrt(var + (double)eps));
        if (__all_sync(0xffffffffu, there) || gave_up) return result;
        gave_up = ++spins > limit;
    }
}

}  // namespace gn
