// Block matvec kernels (BlockMatrix::matvec, blockMatrix.hpp:208-234) with
// an epilogue, shared by the BAIJ operator (baij.cu) and the AMG V-cycle
// (amg.cu), whose residual and smoothing updates ride on the products.
//
// Block matvec (bs >= 2): a warp owns a contiguous range of block rows and
// streams its blocks, 32 (16 of 4x4) a pass, through a two-stage ring in shared
// memory: cp.async brings the next pass's values and columns while lane b
// gathers x_J of block b of this one and forms the block's bs row dots with the
// reference's association (blk_row_dot).  The dots go to a second ring, and
// whenever the stream has passed the end of a group of 32/bs rows the lane of
// output component (I, r) adds the dots of row I in block order -- the
// reference's order, so y is bit-exact.  No CTA-wide barrier.
//
// Bound by the stream of values once the warp's chain (columns, x, dots, sums)
// is covered: the sums are the serial part, 3 to 6 lanes wide when taken every
// pass and a whole group wide from the ring.  64^3 Q1 elasticity, 3x3 (552 MB,
// a copy of as many bytes takes 84 us): 127 us with register-staged passes
// summed one by one at 32 warps an SM; here 99 us at 24 warps (20: 103, 32 with a
// ring of half the size: 107, 16 with twice: 107; x gathered a pass ahead: 122,
// three stages at 16 warps: 107).  The coarse products of the block hierarchies
// gain more, their few rows now spread over all warps: V-cycle of 48^3 elements
// 466 -> 221 us, of 10^3 172 -> 132.
#pragma once
#include "block_ops.cuh"
#include "spmv_staged.cuh"

namespace b2s {

constexpr int kBaijThreads = 192;
constexpr int kBaijCtasPerSm = 4;
inline uint32_t baij_warps(const b2s_ctx* ctx) { return (uint32_t)ctx->sm_count * kBaijCtasPerSm * (kBaijThreads / 32); }

// Rows are dealt evenly, or, where that gives a warp more than kBaijUneven times
// the mean blocks, by weight, a row kBaijWarpRow besides its blocks (k_baij_split).
// 3x3, 120,000 rows of 9 blocks with 200 adjacent rows of 2,500: 97 us by weight,
// 2,700 evenly.  Up to twice the mean an even deal, which reads no partition, is as
// good: half the rows of 27 blocks, half of 3 (1.8 times): 39 us.
constexpr uint32_t kBaijUneven = 2;
constexpr uint32_t kBaijWarpRow = 2;

template <int BS, typename VT>
struct alignas(16) BaijWarpSmem
{
    static constexpr int NB = BS <= 3 ? 32 : 256 / (BS * BS);  // blocks a pass, one lane each
    static constexpr int RING = 4 * NB;                        // blocks whose dots are kept (a power of two)
    VT val[2][NB * BS * BS];
    uint32_t col[2][NB];
    double dot[RING * BS];
};

// VT: stored value type (double, or float for the FP32 copies of the AMG
// hierarchy); products and sums are FP64 either way.  v is 16-byte aligned.
// per: block rows a warp, or PARTED, part: the warps' first rows (warps + 1 of them).
// An instance each: looking at part cost an even deal 0.1 us of 18.3 (3x3, 32^3 elements).
template <int BS, typename VT, bool PARTED, class Epi>
__global__ void __launch_bounds__(kBaijThreads, kBaijCtasPerSm)
    k_baij_warp(uint32_t nbr, uint32_t per, const uint32_t* __restrict__ part, uint32_t warps,
                const uint32_t* __restrict__ rp, const uint32_t* __restrict__ ci, const VT* __restrict__ v,
                const double* __restrict__ x, Epi epi, const int* done)
{
    if (done && *done) return;
    using Smem = BaijWarpSmem<BS, VT>;
    constexpr int BV = BS * BS, NB = Smem::NB, RING = Smem::RING;
    constexpr uint32_t GR = 32 / BS;                           // block rows a group
    constexpr int CHUNKS = (NB * BV * (int)sizeof(VT) + 511) / 512;  // 16-byte copies a lane and pass
    __shared__ Smem smem[kBaijThreads / 32];
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5, r = lane % BS;
    Smem& s = smem[wid];
    const uint32_t w = blockIdx.x * (kBaijThreads / 32) + wid;
    if (w >= warps) return;
    // the group's first row, and the end of the warp's
    uint32_t I0 = PARTED ? __ldg(&part[w]) : w * per;
    const uint32_t R1 = PARTED ? __ldg(&part[w + 1]) : nbr - I0 < per ? nbr : I0 + per;
    if (PARTED && I0 >= R1) return;
    const uint32_t p0 = __ldg(&rp[I0]), p1 = __ldg(&rp[R1]);
    const uint32_t first = p0 & ~3u;  // four blocks of any size and type are whole 16-byte units
    const uint32_t passes = (p1 - first + NB - 1) / NB;
    auto copy = [&](uint32_t i) {
        if (i < passes)
        {
            const uint32_t base = first + i * NB, nb = p1 - base < NB ? p1 - base : NB;
            const uint32_t bytes = nb * BV * (uint32_t)sizeof(VT);
            const char* src = reinterpret_cast<const char*>(v + (size_t)base * BV);
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s.val[i & 1u]);
#pragma unroll
            for (int k = 0; k < CHUNKS; ++k)
            {
                const uint32_t c = (k * 32 + lane) * 16u;
                if (c < bytes)  // (the last unit may be part of one: the copy reads no further)
                    asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"(dst + c), "l"(src + c),
                                 "r"(bytes - c < 16u ? bytes - c : 16u)
                                 : "memory");
            }
            if (lane < nb)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                                 (uint32_t)__cvta_generic_to_shared(&s.col[i & 1u][lane])),
                             "l"(ci + base + lane)
                             : "memory");
        }
    };
    copy(0);
    // the group: this lane's row [a, b), the group's end, and the next group's row
    uint32_t a = 0, b = 0, gend = 0, na = 0, nb = 0;
    bool out = false;
    double acc = 0.0;
    auto row_of = [&](uint32_t g0, uint32_t& ra, uint32_t& rb) {
        const uint32_t I = g0 + lane / BS;
        const bool on = lane < GR * BS && I < R1;
        ra = on ? __ldg(&rp[I]) : 0u;
        rb = on ? __ldg(&rp[I + 1]) : 0u;
    };
    row_of(I0, na, nb);
    auto group = [&] {
        const uint32_t rows = R1 - I0 < GR ? R1 - I0 : GR;
        out = lane < rows * BS;
        a = na;
        b = nb;
        gend = __shfl_sync(0xffffffffu, b, (rows - 1) * BS);
        acc = 0.0;
        row_of(I0 + GR, na, nb);
    };
    group();
    uint32_t low = p0;  // dots of blocks below are summed
    for (uint32_t i = 0; i < passes; ++i)
    {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        const uint32_t base = first + i * NB, end = p1 - base < NB ? p1 : base + NB, q = base + lane;
        const bool on = lane < NB && q < end && q >= p0;
        double xv[BS];
        if (on)
        {
            const double* xj = x + (size_t)s.col[i & 1u][lane] * BS;
#pragma unroll
            for (int c = 0; c < BS; ++c) xv[c] = __ldg(&xj[c]);
        }
        copy(i + 1);  // into the stage of pass i - 1
        if (on)
        {
            double vv[BV];
#pragma unroll
            for (int e = 0; e < BV; ++e) vv[e] = (double)s.val[i & 1u][lane * BV + e];
#pragma unroll
            for (int c = 0; c < BS; ++c) s.dot[(q % RING) * BS + c] = blk_row_dot<BS>(&vv[c * BS], xv);
        }
        __syncwarp();
        // sum the groups that end here; part of one when the ring has no room for another pass
        while (I0 < R1 && (gend <= end || end - low > RING - NB))
        {
            const uint32_t to = b < end ? b : end;
            if (out)
#pragma unroll 4
                for (uint32_t k = a > low ? a : low; k < to; ++k) acc += s.dot[(k % RING) * BS + r];
            if (gend > end)
            {
                low = end;
                break;
            }
            low = gend;
            epi.template put<BS>(I0 + lane / BS, r, acc, out, lane);
            I0 += GR;
            if (I0 < R1) group();
        }
        __syncwarp();
    }
    while (I0 < R1)  // no blocks at all
    {
        epi.template put<BS>(I0 + lane / BS, r, acc, out, lane);
        I0 += GR;
        if (I0 < R1) group();
    }
}

// y = A x with the stored values v (A's pattern), every output component
// handed to the epilogue: epi.put<BS>(I, r, y_Ir, valid, lane).  For BS >= 2
// all 32 lanes of a warp call put together (valid false on idle lanes), so an
// epilogue may exchange a block row's components with shuffles; the lanes of
// block row I are lanes (lane / BS) * BS .. + BS - 1.  For BS = 1 a thread
// calls put for its own rows only.
//
// 1x1 blocks with long rows (the coarse operators and restrictions of a
// scalar AMG hierarchy, 30 to 100+ entries a row): a CTA takes a contiguous
// range of at most kThreads rows (the partition in A.blk_row).  All its
// threads load entries and gather x, so that the row length does not bound
// the loads in flight, and leave the products in shared memory; then one
// thread a row adds its products in column order.  Bound by the stream of
// values and columns on the large levels and by the chain row pointers,
// entries, x, sum on the small ones.  On the hierarchy of the 128^3 Poisson
// grid, against one thread a row that also gathered its x from staged
// columns: restriction of 7.2M entries 56 -> 33 us, operator of 6.2M entries
// 46 -> 29, of 0.4M 14 -> 7, restriction of 60k entries 27 -> 8.
//
// The partition is cut on the device by a weight that grows with entries and
// rows, so that both are bounded (k_baij_split): greedy blocks needed the row
// pointers on the host, 0.3 to 0.6 ms for each of the three large operators of
// that hierarchy (set-up 9.6 -> 8.6 ms).
constexpr uint32_t kBaijStagedCap = 2048;   // products a pass
constexpr uint32_t kBaijStagedMin = 256;    // entries of the smallest share of a CTA
constexpr uint32_t kBaijStagedRow = 16;     // weight of a row besides its entries
constexpr uint32_t kBaijStagedMinRow = 16;  // mean entries per row from which the staged kernel is used

// The weight of a CTA's rows.  About a full pass of mean rows, and no more rows
// than threads, where the matrix gives every SM several CTAs; less on the small
// levels, whose time is one CTA's chain.
inline uint32_t baij_staged_share(const b2s_ctx* ctx, uint64_t rows, uint64_t nnz)
{
    const uint64_t mean = (nnz + rows - 1) / rows;
    const uint64_t full = mean < kBaijStagedCap / 2 ? kBaijStagedCap - mean : kBaijStagedCap / 2;
    const uint64_t entries = std::min(std::max<uint64_t>(nnz / (4ull * ctx->sm_count), kBaijStagedMin), full);
    return (uint32_t)std::min(entries * (nnz + kBaijStagedRow * rows) / nnz, (uint64_t)kBaijStagedRow * kThreads);
}

template <typename VT, class Epi>
__global__ void __launch_bounds__(kThreads, 6)
    k_baij_staged1(const uint32_t* __restrict__ rp, const uint32_t* __restrict__ ci, const VT* __restrict__ v,
                   const uint32_t* __restrict__ blk_row, const double* __restrict__ x, Epi epi, const int* done)
{
    if (done && *done) return;
    constexpr int U = kBaijStagedCap / kThreads;
    __shared__ double P[kBaijStagedCap];
    const uint32_t r0 = __ldg(&blk_row[blockIdx.x]), r1 = __ldg(&blk_row[blockIdx.x + 1]);
    const uint32_t row = r0 + threadIdx.x;
    const bool own = row < r1;
    const uint32_t p0 = __ldg(&rp[r0]), p1 = __ldg(&rp[r1]);
    const uint32_t a = own ? __ldg(&rp[row]) : 0u, b = own ? __ldg(&rp[row + 1]) : 0u;
    double sum = 0.0;
    // one pass of a CTA whose rows are of about the mean length, more where they are longer
    for (uint32_t base = p0, end; base < p1; base = end)
    {
        end = p1 - base < kBaijStagedCap ? p1 : base + kBaijStagedCap;
        VT vv[U];
        uint32_t cc[U];
#pragma unroll
        for (int k = 0; k < U; ++k)
        {
            const uint32_t q = base + k * kThreads + threadIdx.x;
            vv[k] = q < end ? ld_stream(v + q) : (VT)0;
            cc[k] = q < end ? ld_stream(ci + q) : 0u;
        }
#pragma unroll
        for (int k = 0; k < U; ++k)
        {
            const uint32_t q = base + k * kThreads + threadIdx.x;
            if (q < end) P[k * kThreads + threadIdx.x] = (double)vv[k] * __ldg(&x[cc[k]]);
        }
        __syncthreads();
        const uint32_t lo = a > base ? a : base, hi = b < end ? b : end;
#pragma unroll 8
        for (uint32_t q = lo; q < hi; ++q) sum += P[q - base];
        if (end < p1) __syncthreads();
    }
    if (own) epi.template put<1>(row, 0, sum, true, 0u);
}

// 1x1 blocks with short rows (the fine operator and the prolongation) use
// the CSR SpMV's warp kernel.  Both sum a row from 0 in column order, which
// is blk_row_dot<1>'s order, so every kernel gives the same bits.
template <class Epi>
struct EpiRowsOf
{
    static constexpr int NV = 0;
    Epi e;
    __device__ __forceinline__ void row(uint32_t r, double s, double*) const { e.template put<1>(r, 0, s, true, 0u); }
    __device__ __forceinline__ void last(const double*) const {}
};

template <int BS, typename VT, class Epi>
void baij_mv(b2s_ctx* ctx, const BaijDev& A, const VT* v, const double* x, Epi epi, const int* done)
{
    if (A.nbr == 0) return;
    if constexpr (BS == 1)
    {
        if (A.nblk)
            B2S_LAUNCH(ctx, (k_baij_staged1<VT, Epi>), A.nblk, kThreads, 0, A.rp.p, A.ci.p, v, A.blk_row.p, x, epi,
                       done);
        else
            B2S_LAUNCH(ctx, (k_spmv_warp<EpiRowsOf<Epi>, XDirect, VT>), spmv_warp_grid(ctx, A.nbr), kThreads, 0,
                       A.nbr, A.rp.p, A.ci.p, v, XDirect{x}, done, EpiRowsOf<Epi>{epi}, (double*)nullptr,
                       (unsigned int*)nullptr);
    }
    else
    {
        // one wave of warps
        constexpr uint32_t W = kBaijThreads / 32;
        const uint32_t per = baij_even_rows(ctx, A.nbr);
        const uint32_t warps = A.nblk ? A.nblk : (A.nbr + per - 1) / per;
        const auto kern = A.nblk ? k_baij_warp<BS, VT, true, Epi> : k_baij_warp<BS, VT, false, Epi>;
        B2S_LAUNCH(ctx, kern, (warps + W - 1) / W, kBaijThreads, 0, A.nbr, per,
                   A.nblk ? A.blk_row.p : (const uint32_t*)nullptr, warps, A.rp.p, A.ci.p, v, x, epi, done);
    }
}

// the plain product: y[I * BS + r] = (A x)_Ir
struct EpiStoreY
{
    double* y;
    template <int BS>
    __device__ __forceinline__ void put(uint32_t I, int r, double v, bool valid, uint32_t) const
    {
        if (valid) y[(size_t)I * BS + r] = v;
    }
};

}  // namespace b2s
