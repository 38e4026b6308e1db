// Exact triangular solves of any pattern in one launch (IC(0) / ILU(0) / block
// ILU(0)): every row of the factor in level order, each waiting for the values
// it reads.
//
// Rows are dealt to lane groups in (level, index) order: GL lanes (4, 8, 16 or 32,
// wave_lanes; longer rows take several passes) own one row, lane q its q-th entry.  A group loads everything that is fixed --
// its entry's column, coefficients, right-hand side, divisor -- and then polls
// the rows it depends on in the exchange array, where a finished row leaves its
// value as 64-bit words {epoch, 32 value bits}: one word per FP32 component, two
// per FP64 one.  A 64-bit access is single-copy atomic, so a reader that sees
// the epoch in a word sees that word's bits: a value crosses to its readers in
// one trip through L2 and no flag, fence or second load lies on the path.  The
// products are formed in the lanes and subtracted in column order by one lane a
// component (through shared memory), so the sums are the reference's.
//
// CTAs take tickets and hold consecutive positions, so a group only waits on
// rows of CTAs that started before its own; each level starts a new warp, so no
// group waits on a row of its own warp.  The waits are bounded: after polls_max
// polls, or once another wait of the launch has given up, a group records
// B2S_TIMEOUT, goes on with what it read and publishes it, so the launch ends.
// The last CTA to leave resets the ticket and advances the epoch; the exchange
// array is never cleared and a captured launch can be replayed.
#pragma once
#include "trsv_grid.cuh"

namespace b2s {

// CTA size by group width.  A CTA holds kWaveThreads / GL consecutive rows;
// narrow rows are bound by the rate at which CTAs come and go (128^3 7-point
// factor in level-order numbering, GL 4: 835 us an apply with 256 threads, 733
// with 512), wide ones by the rows' waits, where a larger CTA holds its slot
// longer (64^3 Q1 elasticity, 3x3 blocks, GL 16: 908 and 937 us).
constexpr int wave_threads(int gl) { return gl <= 8 ? 512 : 256; }
constexpr uint32_t kWaveNone = 0xffffffffu;

// What a row does with its sum: nothing (unit diagonal), divide by d[row] (FP32
// Divide multiplies by the reciprocal, Quotient divides, with one rounding less:
// the triangles no chunk plan could take), or multiply by the inverse diagonal
// block d[row].  BLOCK: the block kernels' products (each block component summed
// from zero, then subtracted).
enum class WaveDiag
{
    Unit,
    Divide,
    Quotient,
    BlockUnit,
    BlockInverse
};

struct WaveArgs
{
    uint32_t npos;
    const uint32_t* order;  // position -> row, kWaveNone where a level's last warp is not full
    const uint32_t *rp, *ci, *level;
    unsigned long long* xch;
    uint32_t* ctl;  // [0] epoch, [1] exit count, [2] ticket
    int* err;
    unsigned polls_max;
};

__device__ __forceinline__ void wave_put(unsigned long long* w, float v, uint32_t epoch)
{
    st_relaxed_u64(w, (unsigned long long)epoch << 32 | __float_as_uint(v));
}
__device__ __forceinline__ void wave_put(unsigned long long* w, double v, uint32_t epoch)
{
    const unsigned long long e = (unsigned long long)epoch << 32, b = (unsigned long long)__double_as_longlong(v);
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(w), "l"(e | (b & 0xffffffffull)), "l"(e | (b >> 32))
                 : "memory");
}
__device__ __forceinline__ bool wave_get(const unsigned long long* w, uint32_t epoch, float& v)
{
    const unsigned long long a = ld_relaxed_u64(w);
    v = __uint_as_float((uint32_t)a);
    return (uint32_t)(a >> 32) == epoch;
}
__device__ __forceinline__ bool wave_get(const unsigned long long* w, uint32_t epoch, double& v)
{
    unsigned long long a, b;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(w) : "memory");
    v = __longlong_as_double((long long)((b << 32) | (a & 0xffffffffull)));
    return (uint32_t)(a >> 32) == epoch && (uint32_t)(b >> 32) == epoch;
}

template <int BS, bool LOWER, WaveDiag DIAG, int GL, typename VT, typename XT, typename RT>
__global__ void __launch_bounds__(wave_threads(GL)) k_trsv_wave(WaveArgs a, const VT* __restrict__ v,
                                                            const VT* __restrict__ d, const RT* __restrict__ rhs,
                                                            XT* __restrict__ x, double* __restrict__ out64,
                                                            const int* done)
{
    if (done && *done) return;
    static_assert(BS <= GL && 32 % GL == 0, "a lane per component");
    constexpr bool BLOCK = DIAG == WaveDiag::BlockUnit || DIAG == WaveDiag::BlockInverse;
    constexpr int WPV = sizeof(XT) == 8 ? 2 : 1;  // exchange words per value
    constexpr int WARPS = wave_threads(GL) / 32, RW = 32 / GL;
    __shared__ uint32_t s_ticket;
    __shared__ XT s_term[WARPS][RW][GL * BS];
    if (threadIdx.x == 0) s_ticket = atomicAdd(&a.ctl[2], 1u);
    __syncthreads();
    const uint32_t epoch = ld_flag(&a.ctl[0]) + 1u;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, g = lane / GL, q = lane % GL;
    const uint32_t pos = (s_ticket * WARPS + warp) * RW + g;
    const uint32_t row = pos < a.npos ? __ldg(&a.order[pos]) : kWaveNone;
    const bool on = row != kWaveNone;
    const uint32_t pa = on ? __ldg(&a.rp[row]) : 0u, pe = on ? __ldg(&a.rp[row + 1]) : 0u;
    XT sum = XT(0), dv[DIAG == WaveDiag::BlockInverse ? BS : 1];
    if (on && q < BS)
    {
        sum = (XT)rhs[(size_t)row * BS + q];
        if constexpr (DIAG == WaveDiag::Divide || DIAG == WaveDiag::Quotient) dv[0] = (XT)__ldg(&d[row]);
        if constexpr (DIAG == WaveDiag::BlockInverse)
#pragma unroll
            for (int c = 0; c < BS; ++c) dv[c] = (XT)__ldg(&d[((size_t)row * BS + q) * BS + c]);
    }
    else
        for (XT& e : dv) e = XT(1);
    // FP32 multiplies by the reciprocal rounded once from FP64, as the chunks do,
    // FP64 forms the quotient from the reciprocal (grid_quotient): both before the
    // wait
    [[maybe_unused]] XT rc = XT(1);
    if constexpr (DIAG == WaveDiag::Divide) rc = (XT)(1.0 / (double)dv[0]);

    for (uint32_t p0 = 0; __any_sync(0xffffffffu, pa + p0 < pe); p0 += GL)
    {
        const uint32_t p = pa + p0 + q;
        uint32_t j = 0, lev = 0;
        bool dep = p < pe;
        if (dep)
        {
            j = __ldg(&a.ci[p]);
            dep = LOWER ? j < row : j > row;  // the diagonal may be stored in the row
            if (dep) lev = __ldg(&a.level[j]);
        }
        XT vv[BS * BS], xj[BS];
        if (dep)
#pragma unroll
            for (int e = 0; e < BS * BS; ++e) vv[e] = (XT)__ldg(&v[(size_t)p * BS * BS + e]);
        bool fresh = !dep;
        const unsigned long long* w = a.xch + (size_t)j * BS * WPV;
        // The first poll asks for every value; after it only the entries of the
        // lowest unfinished level do, since the later ones cannot be ready before
        // them.  (All lanes polling: 1.17 / 1.35 ms FP64 / FP32 on the 64^3 block
        // factor, and up to 2.8 ms at other occupancies, the rows ahead of the
        // wavefront flooding the SM's path to L2; this way 0.91 / 0.83 ms.)
        uint32_t next = 0;
        for (unsigned polls = 0;; ++polls)
        {
            if (!fresh && (polls == 0 || lev == next))
            {
                fresh = true;
#pragma unroll
                for (int c = 0; c < BS; ++c) fresh &= wave_get(w + c * WPV, epoch, xj[c]);
            }
            if (__all_sync(0xffffffffu, fresh)) break;
            // the error word by a vote, so that the warp leaves as one: a lane's own
            // load may come before or after another's
            if (polls + 1 >= a.polls_max || ((polls & 1023u) == 1023u && __any_sync(0xffffffffu, ld_err(a.err) != 0)))
            {
                if (lane == 0) atomicCAS(a.err, 0, (int)B2S_TIMEOUT);
                break;
            }
            next = __reduce_min_sync(0xffffffffu, fresh ? 0xffffffffu : lev);
        }
        XT term[BS];
#pragma unroll
        for (int r = 0; r < BS; ++r)
        {
            if constexpr (BLOCK)
            {
                XT s = XT(0);
#pragma unroll
                for (int c = 0; c < BS; ++c) s += vv[r * BS + c] * xj[c];
                term[r] = dep ? s : XT(0);
            }
            else
                term[r] = dep ? vv[0] * xj[0] : XT(0);
            s_term[warp][g][q * BS + r] = term[r];
        }
        __syncwarp();
        // entries in column order; a lane without one holds +0, which leaves the
        // sum as it is (its sign too)
        if (q < BS)
        {
            const XT* st = &s_term[warp][g][q];
#pragma unroll
            for (uint32_t k = 0; k < (uint32_t)GL; ++k) sum -= st[k * BS];
        }
        __syncwarp();
    }

    XT r = sum;
    if constexpr (DIAG == WaveDiag::Quotient) r = sum / dv[0];
    if constexpr (DIAG == WaveDiag::Divide)
    {
        if constexpr (sizeof(XT) == 4)
            r = sum * rc;
        else
        {
            bool bad = false;
            r = grid_quotient(sum, dv[0], rc, true, bad);
            if (bad) r = sum / dv[0];
        }
    }
    if constexpr (DIAG == WaveDiag::BlockInverse)
    {
        XT s = XT(0);
#pragma unroll
        for (int c = 0; c < BS; ++c) s += dv[c] * __shfl_sync(0xffffffffu, sum, (int)(g * GL) + c);
        r = s;
    }
    if (on && q < BS)
    {
        const size_t i = (size_t)row * BS + q;
        wave_put(a.xch + i * WPV, r, epoch);
        if (out64)
            out64[i] = (double)r;  // given out64, x is scratch and is not written
        else
            x[i] = r;
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        __threadfence();
        if (atomicAdd(&a.ctl[1], 1u) == gridDim.x - 1u)
        {
            a.ctl[1] = 0u;
            a.ctl[2] = 0u;
            a.ctl[0] = epoch;
            __threadfence();
        }
    }
}

// Lanes a row.  More of them take a level's widest row in fewer passes, 0.7 us
// each, but every row has as many, and 20,000 lanes cost as much as a pass (FP64,
// rows of 3 entries, an apply's wider triangle: 262,144 rows at 4 / 8 / 16 / 32
// lanes 41 / 66 / 149 / 283 us).  By the widest row alone, one row of 40 entries in a
// red-black 1,000^2 system had all rows take 32 lanes: 1,248 us an apply, 214 now
// (chunked 369); one of 2,000 in a 512^2 one 364 and 251 (354).
inline uint32_t wave_lanes(uint32_t n, const std::vector<uint32_t>& width)
{
    uint32_t best = 4;
    uint64_t cost = ~0ull;
    for (uint32_t gl = 4; gl <= 32; gl *= 2)
    {
        uint64_t c = (uint64_t)n * gl / 20000;
        for (uint32_t w : width) c += std::max(1u, (w + gl - 1) / gl);
        if (c < cost)
        {
            cost = c;
            best = gl;
        }
    }
    return best;
}

// One triangle's level-order schedule.
struct WaveSchedule
{
    uint32_t n = 0, bs = 1, gl = 32, npos = 0;
    bool quotient = false;  // FP32 divisors: Quotient, not Divide
    DBuf<uint32_t> order, lev, ctl;
    DBuf<unsigned long long> xch;

    // levels: each row's level; rp: the triangle's rows (host)
    void build(b2s_ctx* ctx, const std::vector<uint32_t>& level, const uint32_t* rp, uint32_t block)
    {
        n = (uint32_t)level.size();
        bs = block;
        if (!n) return;
        uint32_t top = 0;
        for (uint32_t l : level) top = std::max(top, l);
        std::vector<uint32_t> width(top + 1, 0);  // each level's widest row
        for (uint32_t i = 0; i < n; ++i) width[level[i]] = std::max(width[level[i]], rp[i + 1] - rp[i]);
        gl = wave_lanes(n, width);
        const uint32_t rw = 32 / gl;
        std::vector<uint32_t> at(top + 2, 0);
        for (uint32_t l : level) ++at[l + 1];
        for (uint32_t l = 0; l <= top; ++l) at[l + 1] = at[l] + (at[l + 1] + rw - 1) / rw * rw;  // whole warps
        npos = at[top + 1];
        std::vector<uint32_t> h(npos, kWaveNone);
        for (uint32_t i = 0; i < n; ++i) h[at[level[i]]++] = i;
        order = upload(ctx, h);
        lev = upload(ctx, level);
        xch.alloc((size_t)n * bs * 2);
        ctl.alloc(3);
        B2S_CUDA(cudaMemsetAsync(xch.p, 0, xch.bytes(), ctx->stream));
        B2S_CUDA(cudaMemsetAsync(ctl.p, 0, ctl.bytes(), ctx->stream));
    }

    template <int BS, bool LOWER, WaveDiag DIAG, typename VT, typename XT, typename RT>
    void run(b2s_ctx* ctx, const uint32_t* rp, const uint32_t* ci, const VT* v, const VT* d, const RT* rhs, XT* x,
             double* out64, const int* done)
    {
        if (!n) return;
        if (gl == 4)
            go<BS, LOWER, DIAG, 4>(ctx, rp, ci, v, d, rhs, x, out64, done);
        else if (gl == 8)
            go<BS, LOWER, DIAG, 8>(ctx, rp, ci, v, d, rhs, x, out64, done);
        else if (gl == 16)
            go<BS, LOWER, DIAG, 16>(ctx, rp, ci, v, d, rhs, x, out64, done);
        else
            go<BS, LOWER, DIAG, 32>(ctx, rp, ci, v, d, rhs, x, out64, done);
    }

    template <int BS, bool LOWER, WaveDiag DIAG, int GL, typename VT, typename XT, typename RT>
    void go(b2s_ctx* ctx, const uint32_t* rp, const uint32_t* ci, const VT* v, const VT* d, const RT* rhs, XT* x,
            double* out64, const int* done)
    {
        constexpr uint32_t T = wave_threads(GL), per_cta = T / GL;
        const WaveArgs a{npos, order.p, rp, ci, lev.p, xch.p, ctl.p, ctx->errword(), grid_polls(ctx)};
        B2S_LAUNCH(ctx, (k_trsv_wave<BS, LOWER, DIAG, GL, VT, XT, RT>), (npos + per_cta - 1) / per_cta, T, 0, a, v, d, rhs, x, out64, done);
    }
};

}  // namespace b2s
