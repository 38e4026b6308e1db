// The whole PCG loop in one persistent kernel over 2-D tiles (tile_plan.hpp),
// for an IC(0)-type preconditioner whose two FP32 triangles are applied by k
// plain Jacobi sweeps (at most two strict entries per row).
//
// A cooperative launch of one CTA per tile (all resident, one per SM).  At
// launch a CTA copies its tile's two blobs into shared memory: the global
// rows of its owned rows and halos, every extended row's two dependencies as
// local indices, the triangles' strict entries and reciprocals, and its
// owned rows of A with local columns.  Nothing static is read from global
// memory again.  Each iteration is three phases:
//   1. p = z + beta p_old for the owned rows and the SpMV's ring; Ap = A p and
//      p.Ap for the owned rows (CSR order);
//   2. r = r - alpha Ap for every row of the tile's lower extended set, and the
//      forward sweeps over it; the owned rows take x += alpha p and r.r;
//   3. the backward sweeps over the upper extended set on y; the owned rows
//      take z and r.z.
// Sweep s computes the rows of layers 0..k-s (a prefix of the local order),
// so the owned rows equal the global sweep definition bit for bit, as the
// banded kernel's do.  The arithmetic of every row is that of k_pcg_band;
// only the association of the two per-iteration dot products differs (the
// tiles are other row sets).
//
// Every tile keeps r over its whole lower set and p over its ring itself, by the
// owners' arithmetic, so what the tiles exchange is Ap (phase 1), z (phase 3; an
// FP32 value) and, unfused, y (phase 2): 64-bit words {epoch, 32 value bits} that
// a reader polls until they carry the iteration, while the phase's sum over the
// grid (grid_sum.cuh) is on its way.  No store needs a fence, and a phase starts
// with its operands in registers.  512^2, 6 sweeps: 20.0 us an iteration with the
// vectors behind fenced all-reduces, about 15 us this way.  Each wait is bounded
// (polls_max polls): a CTA that gives up records B2S_TIMEOUT and leaves, and
// the others give up at their next sum, so the launch always ends.
#pragma once

#include "grid_sum.cuh"
#include "pcg_band.cuh"
#include "tile_plan.hpp"
#include "trsv_chunk.cuh"

namespace b2s {

static_assert(kTileMaxTiles <= (int)kGridSumMaxCtas, "a poller per tile");

struct PcgTileArgs
{
    uint32_t n, ntiles, work, ystride, ring;
    int k;
    const TileDesc* desc;
    const uint4* vals;  // value blobs
    const uint4* idx;   // index blobs
    double* x;
    const double *r, *p, *z;        // the state before the first iteration
    double* rloc;                   // ntiles x ystride: each tile's r over its lower set
    double* ploc;                   // ntiles x ring: p over the rings (past one entry a thread)
    unsigned long long *apw, *zw;   // Ap (two words a row) and z (one), zero at launch
    unsigned long long* yw;         // unfused: the forward sweeps' results (one word a row)
    unsigned long long* lines;      // two regions of grid_sum_words, zero at launch
    KState* st;
    int* err;
    unsigned polls_max;  // of one wait, where the context's bounds are not the default
    int stall_window;
};

__device__ __forceinline__ void tile_put(unsigned long long* w, float v, uint32_t epoch)
{
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(w), "l"((unsigned long long)epoch << 32 | __float_as_uint(v))
                 : "memory");
}
__device__ __forceinline__ void tile_put(unsigned long long* w, double v, uint32_t epoch)
{
    const unsigned long long e = (unsigned long long)epoch << 32, b = (unsigned long long)__double_as_longlong(v);
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(w), "l"(e | (b & 0xffffffffull)), "l"(e | (b >> 32))
                 : "memory");
}
__device__ __forceinline__ bool tile_get(const unsigned long long* w, uint32_t epoch, float& v)
{
    unsigned long long a;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(a) : "l"(w) : "memory");
    v = __uint_as_float((uint32_t)a);
    return (uint32_t)(a >> 32) == epoch;
}
__device__ __forceinline__ bool tile_get(const unsigned long long* w, uint32_t epoch, double& v)
{
    unsigned long long a, b;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(w) : "memory");
    v = __longlong_as_double((long long)((b << 32) | (a & 0xffffffffull)));
    return (uint32_t)(a >> 32) == epoch && (uint32_t)(b >> 32) == epoch;
}
// another tile's value of this iteration
template <typename T>
__device__ __forceinline__ T tile_await(const unsigned long long* w, uint32_t epoch, int* failed, int* err,
                                        unsigned polls_max)
{
    T v;
    for (unsigned polls = 0; polls < polls_max; ++polls)
        if (tile_get(w, epoch, v)) return v;
    *failed = 1;
    atomicCAS(err, 0, (int)B2S_TIMEOUT);
    return v;
}

// k + 1 passes over the extended set; rows of layers 0..k-s at pass s.
// Returns the buffer holding pass k.  Branch-free over the thread's Q rows:
// every row is evaluated at every pass and only rows t < cnt[k - s] are
// stored.  An absent dependency names the spare slot `dummy` past the set,
// which holds +0 in both buffers, with a coefficient of +0, so that
// sum - 0 * 0 leaves sum unchanged (its sign included) and the stored rows
// equal the global sweep definition bit for bit.
template <uint32_t Q>
__device__ __forceinline__ const float* tile_sweeps(int k, const uint16_t* cnt, const uint32_t (&dep)[Q],
                                                    const float2 (&val)[Q], const float (&di)[Q],
                                                    const float (&rr)[Q], float* y0, float* y1, uint32_t dummy)
{
    constexpr uint32_t NT = kTileThreads;
    if (threadIdx.x == 0)
    {
        y0[dummy] = 0.f;
        y1[dummy] = 0.f;
    }
    for (int s = 0; s <= k; ++s)
    {
        const float* yin = (s & 1) ? y0 : y1;
        float* yout = (s & 1) ? y1 : y0;
        const uint32_t t1 = cnt[k - s];
        float out[Q];
        if (s == 0)
        {
#pragma unroll
            for (uint32_t q = 0; q < Q; ++q) out[q] = rr[q] * di[q];
        }
        else
        {
            float a0[Q], a1[Q];
#pragma unroll
            for (uint32_t q = 0; q < Q; ++q)
            {
                a0[q] = yin[dep[q] & 0xFFFFu];
                a1[q] = yin[dep[q] >> 16];
            }
#pragma unroll
            for (uint32_t q = 0; q < Q; ++q)
            {
                float sum = rr[q];
                sum -= val[q].x * a0[q];
                sum -= val[q].y * a1[q];
                out[q] = sum * di[q];
            }
        }
#pragma unroll
        for (uint32_t q = 0; q < Q; ++q)
        {
            const uint32_t t = threadIdx.x + NT * q;
            if (t < t1) yout[t] = out[q];
        }
        __syncthreads();
    }
    return (k & 1) ? y1 : y0;
}

// a row's two dependencies with the absent ones (kTileNoDep) sent to the spare slot
__device__ __forceinline__ uint32_t tile_dep_slots(uint32_t w, uint32_t dummy)
{
    const uint32_t d0 = w & 0xFFFFu, d1 = w >> 16;
    return (d0 == kTileNoDep ? dummy : d0) | ((d1 == kTileNoDep ? dummy : d1) << 16);
}

// LIMITED: waits of a.polls_max polls, not of the default number
template <uint32_t Q, bool FUSED, bool LIMITED>
__global__ void __launch_bounds__(kTileThreads, 1) k_pcg_tile(PcgTileArgs a)
{
    const unsigned polls_max = LIMITED ? a.polls_max : kGridPolls;
    constexpr uint32_t NT = kTileThreads;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ KState sst;
    __shared__ GridSum<NT, 2> gs;
    __shared__ double s_best;
    __shared__ int s_best_at;
    const uint32_t tile = blockIdx.x, ntiles = a.ntiles, tid = threadIdx.x;
    const TileDesc& Dg = a.desc[tile];
    const uint32_t n_own = Dg.n_own, n_el = Dg.n_el, n_eu = Dg.n_eu, n_ae = Dg.n_ae;
    // ---- the tile's blobs -> shared memory (16-byte copies)
    {
        const uint4* vs = a.vals + Dg.vbase / 16;
        const uint4* is = a.idx + Dg.ibase / 16;
        uint4* vd = reinterpret_cast<uint4*>(smem);
        uint4* id = reinterpret_cast<uint4*>(smem + Dg.vbytes);
        for (uint32_t i = tid; i < Dg.vbytes / 16; i += NT) cp_async16(vd + i, vs + i);
        for (uint32_t i = tid; i < Dg.ibytes / 16; i += NT) cp_async16(id + i, is + i);
        cp_async_wait_all();
    }
    __shared__ uint16_t s_lcnt[kTileMaxSweeps + 1], s_ucnt[kTileMaxSweeps + 1];
    if (tid <= (uint32_t)a.k)
    {
        s_lcnt[tid] = Dg.lcnt[tid];
        s_ucnt[tid] = Dg.ucnt[tid];
    }
    if (tid == 0)
    {
        sst = *a.st;
        gs.failed = 0;
        s_best = HUGE_VAL;
        s_best_at = 0;
    }
    __syncthreads();
    const unsigned char* ib = smem + Dg.vbytes;
    const double* aval = reinterpret_cast<const double*>(smem + Dg.o_aval);
    const float2* lvals = reinterpret_cast<const float2*>(smem + Dg.o_lvals);
    const float2* uvals = reinterpret_cast<const float2*>(smem + Dg.o_uvals);
    const float* ldinv = reinterpret_cast<const float*>(smem + Dg.o_ldinv);
    const float* udinv = reinterpret_cast<const float*>(smem + Dg.o_udinv);
    const uint32_t* owned = reinterpret_cast<const uint32_t*>(ib + Dg.o_owned);
    const uint32_t* lhalo = reinterpret_cast<const uint32_t*>(ib + Dg.o_lhalo);
    const uint32_t* ldeps = reinterpret_cast<const uint32_t*>(ib + Dg.o_ldeps);
    const uint32_t* uhalo = reinterpret_cast<const uint32_t*>(ib + Dg.o_uhalo);
    const uint32_t* udeps = reinterpret_cast<const uint32_t*>(ib + Dg.o_udeps);
    const uint32_t* ahalo = reinterpret_cast<const uint32_t*>(ib + Dg.o_ahalo);
    const uint32_t* arp = reinterpret_cast<const uint32_t*>(ib + Dg.o_arp);
    const uint16_t* acol = reinterpret_cast<const uint16_t*>(ib + Dg.o_acol);
    float* const y0 = reinterpret_cast<float*>(smem + a.work);
    float* const y1 = y0 + a.ystride;
    double* const pe = reinterpret_cast<double*>(smem + a.work);  // phase 1 only (aliases y0 / y1)
    const uint32_t lbase = s_lcnt[0];  // the lower set's layer 0: the owned rows, or (fused) the upper set
    const uint32_t dummy = a.ystride - 1;  // the sweeps' spare slot (past every set)

    unsigned long long* const lines1 = a.lines;
    unsigned long long* const lines2 = a.lines + grid_sum_words(ntiles);

    // convergence test on r.r (thread 0), with the learned solve's stall guard
    auto converge = [&](double rr) {
        if (!pcg_check_converged(&sst, rr) && a.stall_window > 0)
        {
            if (sst.relres < 0.5 * s_best)
            {
                s_best = sst.relres;
                s_best_at = sst.it;
            }
            else if (sst.it - s_best_at >= a.stall_window)
            {
                sst.stalled = 1;
                sst.iters = sst.it + 1;
                finish(&sst, B2S_OK);
            }
        }
    };

    // The owned rows' p and x live in registers (thread's rows t = tid + NT q), as
    // does p of the thread's first ring entry; r of its rows of the lower set in
    // its own words of rloc, read back while a sum is awaited.
    double* const rl = a.rloc + (size_t)tile * a.ystride;
    double* const pl = a.ploc + (size_t)tile * a.ring;
    const uint32_t n_ring = n_ae - n_own;
    auto lower_row = [&](uint32_t t) { return t < n_own ? owned[t] : t < lbase ? uhalo[t - n_own] : lhalo[t - lbase]; };
    double pv[Q], xv[Q], ph = 0.0;
    float zv[Q], zh = 0.f;
#pragma unroll
    for (uint32_t q = 0; q < Q; ++q)
    {
        const uint32_t t = tid + NT * q;
        const bool in = t < n_own;
        const uint32_t g = in ? owned[t] : 0u;
        pv[q] = in ? a.p[g] : 0.0;
        xv[q] = in ? a.x[g] : 0.0;
        zv[q] = in ? (float)a.z[g] : 0.f;  // (an FP32 value)
        if (t < n_el) rl[t] = a.r[lower_row(t)];
    }
    for (uint32_t t = tid; t < n_ring; t += NT)
    {
        if (t >= NT) pl[t] = a.p[ahalo[t]];
        if (t < NT)
        {
            ph = a.p[ahalo[t]];
            zh = (float)a.z[ahalo[t]];
        }
    }
    const float* yf = y0;  // the forward sweeps' result (phase 2 -> phase 3)
    uint32_t epoch = 0;
    while (!sst.done)
    {
        // ---- 1. p = z + beta p_old at the SpMV's columns; Ap; p.Ap
        double Apv[Q];
        {
            const double beta = sst.beta;
#pragma unroll
            for (uint32_t q = 0; q < Q; ++q)
            {
                const uint32_t t = tid + NT * q;
                pv[q] = (double)zv[q] + beta * pv[q];
                if (t < n_own) pe[t] = pv[q];
            }
            if (tid < n_ring)
            {
                ph = (double)zh + beta * ph;
                pe[n_own + tid] = ph;
            }
            for (uint32_t t = tid + NT; t < n_ring; t += NT)
            {
                const float zt = epoch ? tile_await<float>(&a.zw[ahalo[t]], epoch, &gs.failed, a.err, polls_max) : (float)a.z[ahalo[t]];
                pe[n_own + t] = pl[t] = (double)zt + beta * pl[t];
            }
            ++epoch;
            __syncthreads();
            double acc[1] = {0.0}, tot[1];
#pragma unroll
            for (uint32_t q = 0; q < Q; ++q)
            {
                const uint32_t t = tid + NT * q;
                Apv[q] = 0.0;
                if (t < n_own)
                {
                    double sum = 0.0;
                    for (uint32_t e = arp[t]; e < arp[t + 1]; ++e) sum += aval[e] * pe[acol[e]];
                    tile_put(&a.apw[2 * (size_t)owned[t]], sum, epoch);
                    acc[0] += pv[q] * sum;
                    Apv[q] = sum;
                }
            }
            grid_sum_post(gs, lines1, epoch, acc);
            // the other tiles' Ap over the lower set, while the sum is on its way
#pragma unroll
            for (uint32_t q = 0; q < Q; ++q)
            {
                const uint32_t t = tid + NT * q;
                if (t >= n_own && t < n_el)
                    Apv[q] = tile_await<double>(&a.apw[2 * (size_t)lower_row(t)], epoch, &gs.failed, a.err, polls_max);
            }
            if (!grid_sum_wait(gs, lines1, epoch, tot, a.err, polls_max)) break;
            if (tid == 0) pcg_alpha(&sst, tot[0]);
            __syncthreads();
            if (sst.done) break;
        }
        // ---- 2. r = r - alpha Ap, forward sweeps on it; x; r.r
        double rr_acc = 0.0;
        {
            const double alpha = sst.alpha;
            uint32_t dep[Q];
            float2 val[Q];
            float di[Q], rr[Q];
#pragma unroll
            for (uint32_t q = 0; q < Q; ++q)
            {
                const uint32_t t = tid + NT * q;
                const bool in = t < n_el;
                dep[q] = tile_dep_slots(in ? ldeps[t] : 0xFFFFFFFFu, dummy);
                val[q] = in ? lvals[t] : make_float2(0.f, 0.f);
                di[q] = in ? ldinv[t] : 0.f;
                const double rv = in ? rl[t] - alpha * Apv[q] : 0.0;
                rr[q] = (float)rv;
                if (in) rl[t] = rv;
                if (t < n_own)  // the owned rows' r.r and x now, before the sweeps
                {
                    rr_acc += rv * rv;
                    xv[q] += alpha * pv[q];
                }
            }
            yf = tile_sweeps<Q>(a.k, s_lcnt, dep, val, di, rr, y0, y1, dummy);
            if constexpr (!FUSED)
#pragma unroll
                for (uint32_t q = 0; q < Q; ++q)
                {
                    const uint32_t t = tid + NT * q;
                    if (t < n_own) tile_put(&a.yw[owned[t]], yf[t], epoch);
                }
        }
        // ---- 3. backward sweeps on y; z; r.r and r.z: the test and beta
        {
            uint32_t dep[Q];
            float2 val[Q];
            float di[Q], rr[Q];
#pragma unroll
            for (uint32_t q = 0; q < Q; ++q)
            {
                const uint32_t t = tid + NT * q;
                const bool in = t < n_eu;
                dep[q] = tile_dep_slots(in ? udeps[t] : 0xFFFFFFFFu, dummy);
                val[q] = in ? uvals[t] : make_float2(0.f, 0.f);
                di[q] = in ? udinv[t] : 0.f;
                // this thread's own forward results (read before its sweeps write):
                // every row of the upper set when fused, else the owned rows
                if constexpr (FUSED)
                    rr[q] = in ? yf[t] : 0.f;
                else
                    rr[q] = t < n_own ? yf[t]
                            : in      ? tile_await<float>(&a.yw[uhalo[t - n_own]], epoch, &gs.failed, a.err, polls_max)
                                      : 0.f;
            }
            const float* yk = tile_sweeps<Q>(a.k, s_ucnt, dep, val, di, rr, y0, y1, dummy);
            double acc[2] = {rr_acc, 0.0}, tot[2];
#pragma unroll
            for (uint32_t q = 0; q < Q; ++q)
            {
                const uint32_t t = tid + NT * q;
                if (t < n_own)
                {
                    zv[q] = yk[t];
                    tile_put(&a.zw[owned[t]], zv[q], epoch);
                    acc[1] += rl[t] * (double)zv[q];  // (this thread's own store of phase 2)
                }
            }
            grid_sum_post(gs, lines2, epoch, acc);
            if (tid < n_ring) zh = tile_await<float>(&a.zw[ahalo[tid]], epoch, &gs.failed, a.err, polls_max);
            if (!grid_sum_wait(gs, lines2, epoch, tot, a.err, polls_max)) break;
            if (tid == 0)
            {
                converge(tot[0]);
                if (!sst.done) pcg_next(&sst, tot[1]);
            }
            __syncthreads();
        }
    }
#pragma unroll
    for (uint32_t q = 0; q < Q; ++q)
    {
        const uint32_t t = tid + NT * q;
        if (t < n_own) a.x[owned[t]] = xv[q];
    }
    if (tile == 0 && tid == 0) *a.st = sst;
}

// Builds the index blobs of a 5-point grid's tiles (tile_plan.hpp,
// grid5_build_elem / grid5_build_dep): block t builds tile t, one thread per
// blob element, then one per extended row for the dependencies once the
// halos are written.  *bad = 1 when an index falls outside its segment.
__global__ void __launch_bounds__(kThreads) k_tile_build_grid5(const TileDesc* __restrict__ desc,
                                                               const TileGeom* __restrict__ geom,
                                                               uint8_t* __restrict__ idx, uint32_t B, uint32_t ny,
                                                               uint32_t K, bool fused, int* bad)
{
    __shared__ TileDesc D;
    __shared__ TileGeom G;
    if (threadIdx.x == 0)
    {
        D = desc[blockIdx.x];
        G = geom[blockIdx.x];
    }
    __syncthreads();
    uint8_t* ib = idx + D.ibase;
    const uint32_t ne = grid5_elements(D, G, B, ny, K, fused);
    for (uint32_t e = threadIdx.x; e < ne; e += blockDim.x)
        if (!grid5_build_elem(D, G, B, ny, K, fused, e, ib)) atomicExch(bad, 1);
    __syncthreads();  // the halos, read back below
    for (uint32_t t = threadIdx.x; t < D.n_el; t += blockDim.x) grid5_build_dep(D, G, B, ny, K, true, fused, t, ib);
    for (uint32_t t = threadIdx.x; t < D.n_eu; t += blockDim.x) grid5_build_dep(D, G, B, ny, K, false, fused, t, ib);
}

// Fills the value blobs after factorisation: A's values for the owned rows
// (checking that A's row holds exactly the planned columns), the triangles'
// strict entries and reciprocals from the banded sweep arrays (slot e of row
// g at e*n + g, checking the planned dependency's offset).  *bad = 1 when A's
// pattern or the factor's differs from the plan.
__global__ void k_tile_pack(const TileDesc* __restrict__ desc, const uint8_t* __restrict__ idx,
                            uint8_t* __restrict__ vals, uint32_t n, int k, const uint32_t* __restrict__ Arp,
                            const uint32_t* __restrict__ Aci, const double* __restrict__ Av,
                            const uint16_t* __restrict__ loff, const float* __restrict__ lval,
                            const float* __restrict__ ldinv, const uint16_t* __restrict__ uoff,
                            const float* __restrict__ uval, const float* __restrict__ udinv, int* bad)
{
    const TileDesc D = desc[blockIdx.x];
    const uint8_t* ib = idx + D.ibase;
    uint8_t* vb = vals + D.vbase;
    const uint32_t* owned = reinterpret_cast<const uint32_t*>(ib + D.o_owned);
    const uint32_t* lhalo = reinterpret_cast<const uint32_t*>(ib + D.o_lhalo);
    const uint32_t* ldeps = reinterpret_cast<const uint32_t*>(ib + D.o_ldeps);
    const uint32_t* uhalo = reinterpret_cast<const uint32_t*>(ib + D.o_uhalo);
    const uint32_t* udeps = reinterpret_cast<const uint32_t*>(ib + D.o_udeps);
    const uint32_t* ahalo = reinterpret_cast<const uint32_t*>(ib + D.o_ahalo);
    const uint32_t* arp = reinterpret_cast<const uint32_t*>(ib + D.o_arp);
    const uint16_t* acol = reinterpret_cast<const uint16_t*>(ib + D.o_acol);
    double* aval = reinterpret_cast<double*>(vb + D.o_aval);
    float2* lv = reinterpret_cast<float2*>(vb + D.o_lvals);
    float2* uv = reinterpret_cast<float2*>(vb + D.o_uvals);
    float* ld = reinterpret_cast<float*>(vb + D.o_ldinv);
    float* ud = reinterpret_cast<float*>(vb + D.o_udinv);
    auto ae_global = [&](uint32_t c) { return c < D.n_own ? owned[c] : ahalo[c - D.n_own]; };
    for (uint32_t q = threadIdx.x; q < D.n_own; q += blockDim.x)
    {
        const uint32_t g = owned[q];
        const uint32_t a0 = Arp[g], cntA = Arp[g + 1] - a0, e0 = arp[q], cntP = arp[q + 1] - e0;
        if (cntA != cntP)
        {
            atomicExch(bad, 1);
            continue;
        }
        for (uint32_t e = 0; e < cntP; ++e)
        {
            if (Aci[a0 + e] != ae_global(acol[e0 + e])) atomicExch(bad, 1);
            aval[e0 + e] = Av[a0 + e];
        }
    }
    // one triangle's extended rows: values and reciprocal from the band slots;
    // rows of layers below k (computed by the sweeps) must have every factor
    // entry planned (a missing entry shows as a planned "none" over a band slot)
    // (a fused plan's lower set: the upper set's rows first, then its own halo from base on)
    auto tri = [&](uint32_t ne, uint32_t below_k, uint32_t base, const uint32_t* halo, const uint32_t* deps,
                   const uint16_t* off, const float* val, const float* dinv, float2* outv, float* outd, bool lower) {
        auto glob = [&](uint32_t t) {
            return t < D.n_own ? owned[t] : t < base ? uhalo[t - D.n_own] : halo[t - base];
        };
        for (uint32_t t = threadIdx.x; t < ne; t += blockDim.x)
        {
            const uint32_t g = glob(t);
            const uint32_t dp[2] = {deps[t] & 0xFFFFu, deps[t] >> 16};
            float v2[2];
            for (int e = 0; e < 2; ++e)
            {
                const uint32_t o = off[(size_t)e * n + g];
                v2[e] = val[(size_t)e * n + g];
                if (dp[e] != kTileNoDep)  // (an entry of a layer-k row may point outside the set: never read)
                {
                    const uint32_t j = glob(dp[e]);
                    if (o != (lower ? g - j : j - g)) atomicExch(bad, 1);
                }
                else
                {
                    if (o != 0 && t < below_k) atomicExch(bad, 1);
                    v2[e] = 0.f;  // (read against the sweeps' +0 spare slot; layer-k rows never read it)
                }
            }
            outv[t] = make_float2(v2[0], v2[1]);
            outd[t] = dinv[g];
        }
    };
    tri(D.n_el, k > 0 ? D.lcnt[k - 1] : 0u, D.lcnt[0], lhalo, ldeps, loff, lval, ldinv, lv, ld, true);
    tri(D.n_eu, k > 0 ? D.ucnt[k - 1] : 0u, D.n_own, uhalo, udeps, uoff, uval, udinv, uv, ud, false);
}

}  // namespace b2s
