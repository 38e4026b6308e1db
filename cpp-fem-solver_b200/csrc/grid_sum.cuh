// A sum over all CTAs of a cooperative launch, in a fixed order and without
// atomics, for persistent kernels that take a scalar step after every pass.
//
// Each CTA adds its threads' terms (shuffles, then over the warps) and publishes
// the totals as two 64-bit words {epoch, 32 value bits} each in a 128-byte line of
// its own; threads of every CTA poll the lines until they carry the epoch, and
// the totals are added in CTA order, so all threads of the grid hold the same
// bits.  It is a grid barrier too, but orders no other memory: what the CTAs
// exchange besides carries the epoch in its own words.  Two sets of lines
// alternate: a CTA writes a set again only after a sum over the other one, which
// every CTA took part in after it had read this one.  A wait ends after polls_max
// polls (grid_polls: the context's wait limits): the CTA records B2S_TIMEOUT and
// leaves, the others give up at their next sum, and the launch ends.  A kernel
// that sums all the time has an instance of its own for the default bound: one
// that is not a constant cost the tiled PCG 8 % and the one-launch PCG 1 %.
//
// It costs two trips through L2 and their spread over the SMs, about 2 us on 148
// CTAs.  A line for every pair of CTAs instead of one polled by all was no faster
// (5,000 cycles against 4,000); ordering other stores by fences made it 8,200.
#pragma once
#include "b2s_internal.cuh"

namespace b2s {

constexpr uint32_t kGridSumMaxCtas = 160;  // pollers: threads 32 .. 32 + CTAs - 1 of at least 256
constexpr uint32_t kGridSumStride = 16;    // words between two CTAs' lines

// room for sums of up to NV values; one struct serves sum after sum
template <int NT, int NV = 1>
struct GridSum
{
    static_assert(NT >= 256 && NT % 32 == 0 && NT <= 1024 && 2 * NV <= (int)kGridSumStride, "block size, line");
    double warp_part[NV][NT / 32];
    double part[NV][kGridSumMaxCtas];
    int failed;
};

// words a launch of `ctas` CTAs needs, zeroed before the epochs start at 1
__host__ __device__ inline size_t grid_sum_words(uint32_t ctas) { return 2ull * kGridSumStride * ctas; }

__device__ __forceinline__ double warp_sum_all(double a)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return a;
}

// Publishes the CTA's terms (between this and grid_sum_wait a thread may do other
// work; s.failed must be zero at the first).
template <int NT, int ROOM, int NV>
__device__ __forceinline__ void grid_sum_post(GridSum<NT, ROOM>& s, unsigned long long* lines, uint32_t epoch,
                                              const double (&term)[NV])
{
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    lines += ((size_t)(epoch & 1u) * gridDim.x + blockIdx.x) * kGridSumStride;
#pragma unroll
    for (int v = 0; v < NV; ++v)
    {
        const double a = warp_sum_all(term[v]);
        if (lane == 0) s.warp_part[v][warp] = a;
    }
    __syncthreads();
    if (warp != 0) return;
    const unsigned long long e = (unsigned long long)epoch << 32;
#pragma unroll
    for (int v = 0; v < NV; ++v)
    {
        const double t = warp_sum_all(lane < NT / 32 ? s.warp_part[v][lane] : 0.0);
        const unsigned long long b = (unsigned long long)__double_as_longlong(t);
        if (lane == 0)
            asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(lines + 2 * v),
                         "l"(e | (b & 0xffffffffull)), "l"(e | (b >> 32))
                         : "memory");
    }
}

// The sums; false (in every thread of the CTA) when a wait gave up.
template <int NT, int ROOM, int NV>
__device__ __forceinline__ bool grid_sum_wait(GridSum<NT, ROOM>& s, const unsigned long long* lines, uint32_t epoch,
                                              double (&sum)[NV], int* err, unsigned polls_max)
{
    const uint32_t tid = threadIdx.x, lane = tid & 31u, ctas = gridDim.x;
    if (tid - 32u < ctas)  // (the first warp publishes)
    {
        const unsigned long long* w = lines + ((size_t)(epoch & 1u) * ctas + (tid - 32u)) * kGridSumStride;
        unsigned long long lo[NV], hi[NV];
        bool seen = false;
        for (unsigned polls = 0; polls < polls_max && !seen; ++polls)
        {
            seen = true;
#pragma unroll
            for (int v = 0; v < NV; ++v)
                asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                             : "=l"(lo[v]), "=l"(hi[v])
                             : "l"(w + 2 * v)
                             : "memory");
#pragma unroll
            for (int v = 0; v < NV; ++v)
                seen = seen && (uint32_t)(lo[v] >> 32) == epoch && (uint32_t)(hi[v] >> 32) == epoch;
        }
        if (!seen)
        {
            s.failed = 1;
            atomicCAS(err, 0, (int)B2S_TIMEOUT);
        }
#pragma unroll
        for (int v = 0; v < NV; ++v)
            s.part[v][tid - 32u] = __longlong_as_double((long long)((hi[v] << 32) | (lo[v] & 0xffffffffull)));
    }
    __syncthreads();
#pragma unroll
    for (int v = 0; v < NV; ++v)
    {
        double t = 0.0;
        for (uint32_t b = lane; b < ctas; b += 32) t += s.part[v][b];
        sum[v] = warp_sum_all(t);
    }
    return s.failed == 0;
}

// The same exchange with the association of grid_reduce_last (one value) over a
// grid of `blocks` blocks of kThreads threads, so that a persistent kernel's dots
// have the bits of the launch-a-pass kernels'.  Block CTA * vb + 2 s + half is the
// one whose thread t is this CTA's thread half * kThreads + t with term[s]; a CTA
// publishes its vb <= 8 block sums in its line.
constexpr uint32_t kBlockSumMaxBlocks = 8 * 160;
constexpr int kBlockSumThreads = 2 * kThreads;

struct BlockSum
{
    double warp_part[8][kThreads / 32];  // [block of the CTA][warp of the block]
    double part[kBlockSumMaxBlocks];
    double last[kThreads / 32];
    int failed;
};

// lane 0's sum of grid_reduce_last's shuffle tree
__device__ __forceinline__ double warp_sum_down(double a)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    return a;
}

template <int S>
__device__ __forceinline__ bool block_sum(BlockSum& s, unsigned long long* lines, uint32_t epoch, uint32_t blocks,
                                          uint32_t vb, const double (&term)[S], double& sum, int* err,
                                          unsigned polls_max)
{
    static_assert(S <= 4, "at most 8 blocks a CTA");
    constexpr uint32_t W = kThreads / 32;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, half = tid / kThreads;
    lines += (size_t)(epoch & 1u) * kGridSumStride * gridDim.x;
#pragma unroll
    for (int k = 0; k < S; ++k)
    {
        const double a = warp_sum_down(term[k]);
        if (lane == 0) s.warp_part[2 * k + half][warp % W] = a;
    }
    __syncthreads();
    if (warp < (2u * S * W + 31u) / 32u)
    {
        // eight lanes a block: the tree's last three steps (the wider ones add zeros)
        const uint32_t b = warp * (32u / W) + lane / W;
        double a = b < 2u * S ? s.warp_part[b][lane % W] : 0.0;
#pragma unroll
        for (int o = W / 2; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
        if (lane % W == 0 && b < vb && blockIdx.x * vb + b < blocks)
        {
            const unsigned long long e = (unsigned long long)epoch << 32, w = (unsigned long long)__double_as_longlong(a);
            asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(
                             lines + (size_t)kGridSumStride * blockIdx.x + 2 * b),
                         "l"(e | (w & 0xffffffffull)), "l"(e | (w >> 32))
                         : "memory");
        }
    }
    for (uint32_t b = tid; b < blocks; b += kBlockSumThreads)
    {
        const unsigned long long* w = lines + (size_t)kGridSumStride * (b / vb) + 2u * (b % vb);
        unsigned long long lo = 0, hi = 0;
        bool seen = false;
        for (unsigned polls = 0; polls < polls_max && !seen; ++polls)
        {
            asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(w) : "memory");
            seen = (uint32_t)(lo >> 32) == epoch && (uint32_t)(hi >> 32) == epoch;
        }
        if (!seen)
        {
            s.failed = 1;
            atomicCAS(err, 0, (int)B2S_TIMEOUT);
        }
        s.part[b] = __longlong_as_double((long long)((hi << 32) | (lo & 0xffffffffull)));
    }
    __syncthreads();
    if (warp < W)
    {
        double a = 0.0;
        for (uint32_t b = tid; b < blocks; b += kThreads) a += s.part[b];
        a = warp_sum_down(a);
        if (lane == 0) s.last[warp] = a;
    }
    __syncthreads();
    static_assert(W == 8, "the tree below");
    sum = ((s.last[0] + s.last[4]) + (s.last[2] + s.last[6])) + ((s.last[1] + s.last[5]) + (s.last[3] + s.last[7]));
    return s.failed == 0;
}

}  // namespace b2s
