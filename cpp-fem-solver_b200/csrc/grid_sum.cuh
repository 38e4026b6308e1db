// A sum over all CTAs of a cooperative launch, in a fixed order and without
// atomics, for persistent kernels that take a scalar step after every pass.
//
// Each CTA adds its threads' terms (shuffles, then one warp over the warps) and
// publishes the total as two 64-bit words {epoch, 32 value bits} in a 128-byte
// line of its own; thread 32 + b of every CTA polls line b until it carries the
// epoch, and every warp adds the totals in CTA order, so all threads of the grid
// hold the same bits after two block barriers.  It is a grid barrier too, but
// orders no other memory: what the CTAs exchange besides the sum needs its own
// fences.  Two sets of lines alternate: a CTA writes a set again only after a sum
// over the other one, which every CTA took part in after it had read this one.
// A wait ends after kGridSumPolls polls: the CTA records B2S_TIMEOUT and leaves,
// the others give up at their next sum, and the launch ends.
#pragma once
#include "b2s_internal.cuh"

namespace b2s {

constexpr unsigned kGridSumPolls = 1u << 21;  // about a second
constexpr uint32_t kGridSumMaxCtas = 224;  // pollers: threads 32 .. 32 + CTAs - 1 of at least 256
constexpr uint32_t kGridSumStride = 16;    // words between two CTAs' lines

template <int NT>
struct GridSum
{
    static_assert(NT >= 256 && NT % 32 == 0 && NT <= 1024, "block size");
    double warp_part[NT / 32];
    double part[kGridSumMaxCtas];
    int failed;
};

// words a launch of `ctas` CTAs needs, zeroed before the epochs start at 1
inline size_t grid_sum_words(uint32_t ctas) { return 2ull * kGridSumStride * ctas; }

__device__ __forceinline__ double warp_sum_all(double a)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return a;
}

// s.failed must be zero; false (in every thread of the CTA) when a wait gave up
template <int NT>
__device__ __forceinline__ bool grid_sum(GridSum<NT>& s, unsigned long long* lines, uint32_t epoch, double term,
                                         double& sum, int* err)
{
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, ctas = gridDim.x;
    lines += (size_t)(epoch & 1u) * kGridSumStride * ctas;
    const double a = warp_sum_all(term);
    if (lane == 0) s.warp_part[warp] = a;
    __syncthreads();
    if (warp == 0)
    {
        const double t = warp_sum_all(lane < NT / 32 ? s.warp_part[lane] : 0.0);
        if (lane == 0)
        {
            const unsigned long long e = (unsigned long long)epoch << 32, b = (unsigned long long)__double_as_longlong(t);
            asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(lines + (size_t)kGridSumStride * blockIdx.x),
                         "l"(e | (b & 0xffffffffull)), "l"(e | (b >> 32))
                         : "memory");
        }
    }
    else if (tid - 32u < ctas)
    {
        const unsigned long long* w = lines + (size_t)kGridSumStride * (tid - 32u);
        unsigned long long lo = 0, hi = 0;
        bool seen = false;
        for (unsigned polls = 0; polls < kGridSumPolls && !seen; ++polls)
        {
            asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(w) : "memory");
            seen = (uint32_t)(lo >> 32) == epoch && (uint32_t)(hi >> 32) == epoch;
        }
        if (!seen)
        {
            s.failed = 1;
            atomicCAS(err, 0, (int)B2S_TIMEOUT);
        }
        s.part[tid - 32u] = __longlong_as_double((long long)((hi << 32) | (lo & 0xffffffffull)));
    }
    __syncthreads();
    double t = 0.0;
    for (uint32_t b = lane; b < ctas; b += 32) t += s.part[b];
    sum = warp_sum_all(t);
    return s.failed == 0;
}

}  // namespace b2s
