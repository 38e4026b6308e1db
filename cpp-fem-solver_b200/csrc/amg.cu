// Smoothed-aggregation AMG on BAIJ operators (make_block_amg_preconditioner,
// blockMatrix.hpp:1051-1179; V-cycle blk_amg_vcycle, 946-1046).  The scalar
// "amg" preconditioner runs the same code on the BS = 1 condensed matrix, as
// test_BlockMatrix_schur3d.cpp:143-146 does with the reference.
//
// Setup, per level, all on the device:
//   diag_inv   Gauss-Jordan inverse of each diagonal block (a failed inverse
//              leaves zeros; the reference ignores the failure too)
//   strength   off-diagonal blocks with Frobenius norm >= 0.25 * row maximum
//   aggregates the reference's greedy rule -- rows in natural order, a row not
//              yet aggregated opens an aggregate and pulls in up to 3 of its
//              unaggregated strong neighbours in list order.  The rule is
//              sequential by definition; one thread walks it with the strong
//              lists streamed from HBM, which makes the aggregates identical
//              to the reference's.
//   P          (I - 2/3 D^-1 A) P_tent, one thread per row, blocks accumulated
//              in the reference's order and emitted with ascending aggregate
//   R = P^T    block transpose (rows sorted afterwards)
//   A_c        R (A P): two-phase block SpGEMM -- candidate columns, segmented
//              sort + unique for the pattern, then each output block summed in
//              the reference's (pa, pb) order: bit-equal Galerkin operators
//   coarsest   at most 50 block rows: dense elimination on one CTA, either the
//              reference's own (amg_ref_coarse = 1: rows swapped in the matrix
//              only, the V-cycle solve then repeats blockMatrix.hpp:958-1000
//              exactly) or a correct partial-pivot LU (default).
// Apply: one V(1,1) cycle with 2/3-damped block Jacobi; the pre-smoothing
// step starts from zero so its residual is the right-hand side itself.
#include <cub/cub.cuh>

#include <algorithm>

#include "baij_mv.cuh"
#include "block_ops.cuh"
#include "trisolve.cuh"

namespace b2s {

namespace {

constexpr double kTheta = 0.25, kOmega = 2.0 / 3.0;

// ------------------------------------------------------------ BAIJ helpers

// dptr: each row's diagonal block; after them the most blocks in a range of
// `per` rows (zero before; per 0: left) and the number of blocks
__global__ void k_find_diag(uint32_t nb, uint32_t per, const uint32_t* __restrict__ rp,
                            const uint32_t* __restrict__ ci, uint32_t* dptr)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += gridDim.x * blockDim.x)
    {
        uint32_t lo = rp[i];
        const uint32_t end = rp[i + 1];
        if (per && i % per == 0)
        {
            const uint32_t blocks = rp[nb - i < per ? nb : i + per] - lo;
            if (blocks > *(volatile uint32_t*)&dptr[nb]) atomicMax(&dptr[nb], blocks);
        }
        if (i + 1 == nb) dptr[nb + 1] = end;
        for (uint32_t hi = end; lo < hi;)  // columns ascend
        {
            const uint32_t mid = lo + (hi - lo) / 2;
            if (ci[mid] < i)
                lo = mid + 1;
            else
                hi = mid;
        }
        dptr[i] = lo < end && ci[lo] == i ? lo : 0xFFFFFFFFu;
    }
}

// finalise a device-built BAIJ: diagonal pointers, the block count, the
// matvec's row partition
void finish_baij(b2s_ctx* ctx, BaijDev& M)
{
    M.diag_ptr.alloc((size_t)M.nbr + 2);
    uint32_t h[2] = {0, 0};
    if (M.nbr)
    {
        if (M.bs > 1) B2S_CUDA(cudaMemsetAsync(M.diag_ptr.p + M.nbr, 0, sizeof(uint32_t), ctx->stream));
        B2S_LAUNCH(ctx, k_find_diag, stream_grid(ctx, M.nbr), kThreads, 0, M.nbr,
                   M.bs > 1 ? baij_even_rows(ctx, M.nbr) : 0u, M.rp.p, M.ci.p, M.diag_ptr.p);
        d2h(ctx, h, M.diag_ptr.p + M.nbr, sizeof(h));
        sync(ctx);
    }
    M.nnzb = h[1];
    baij_partition(ctx, M, h[0]);
}

template <int BS>
__global__ void k_diag_inv(uint32_t nb, const double* __restrict__ v, const uint32_t* __restrict__ dptr,
                           double* __restrict__ dinv)
{
    constexpr int BV = BS * BS;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += gridDim.x * blockDim.x)
    {
        double M[BV], Mi[BV];
        for (int k = 0; k < BV; ++k) Mi[k] = 0.0;
        if (dptr[i] != 0xFFFFFFFFu)
        {
            for (int k = 0; k < BV; ++k) M[k] = v[(size_t)dptr[i] * BV + k];
            double T[BV];
            if (blk_inv<BS>(M, T))
                for (int k = 0; k < BV; ++k) Mi[k] = T[k];
        }
        for (int k = 0; k < BV; ++k) dinv[(size_t)i * BV + k] = Mi[k];
    }
}

// ------------------------------------------------------------ strength

template <int BS>
__device__ __forceinline__ double fro(const double* b)
{
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < BS * BS; ++k) s += b[k] * b[k];
    return sqrt(s);
}

// Strong columns of a row: ||A_ij|| >= theta max_k ||A_ik||, in row order.  GL lanes
// a row: one for the short rows of a fine operator, a warp for the long rows of
// the few that a coarse one has (a thread a row took 0.14 - 0.18 ms a pass at
// 5,520 rows and below).
template <int BS, int GL>
__global__ void k_strength(uint32_t nb, const uint32_t* __restrict__ rp, const uint32_t* __restrict__ ci,
                           const double* __restrict__ v, const uint32_t* __restrict__ sp, uint32_t* __restrict__ cnt,
                           uint32_t* __restrict__ sc)
{
    constexpr int BV = BS * BS;
    const uint32_t l = threadIdx.x % GL, groups = gridDim.x * blockDim.x / GL;
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) / GL; i < nb; i += groups)
    {
        const uint32_t p0 = rp[i], p1 = rp[i + 1];
        double mx = 0.0;
        for (uint32_t p = p0 + l; p < p1; p += GL)
            if (ci[p] != i)
            {
                const double f = fro<BS>(&v[(size_t)p * BV]);
                mx = mx < f ? f : mx;
            }
        if constexpr (GL > 1)
#pragma unroll
            for (int o = GL / 2; o; o >>= 1)
            {
                const double f = __shfl_xor_sync(0xffffffffu, mx, o);
                mx = mx < f ? f : mx;
            }
        const double thr = kTheta * mx;
        uint32_t c = 0;
        const uint32_t w = sp ? sp[i] : 0;
        for (uint32_t q = p0; q < p1; q += GL)
        {
            const uint32_t p = q + l;
            const bool strong = p < p1 && ci[p] != i && fro<BS>(&v[(size_t)p * BV]) >= thr;
            if constexpr (GL > 1)
            {
                const uint32_t m = __ballot_sync(0xffffffffu, strong);
                if (sc && strong) sc[w + c + __popc(m & ((1u << l) - 1u))] = ci[p];
                c += __popc(m);
            }
            else if (strong)
            {
                if (sc) sc[w + c] = ci[p];
                ++c;
            }
        }
        if (cnt && l == 0) cnt[i] = c;
    }
    if (cnt && blockIdx.x == 0 && threadIdx.x == 0) cnt[nb] = 0;
}

// ------------------------------------------------------------ aggregation

// The greedy rule of blockMatrix.hpp:1101-1111, walked by one thread.
__global__ void k_aggregate(uint32_t nb, const uint32_t* __restrict__ sp, const uint32_t* __restrict__ sc,
                            int32_t* __restrict__ agg, uint32_t* __restrict__ nagg_out)
{
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    int32_t nagg = 0;
    for (uint32_t i = 0; i < nb; ++i)
    {
        if (agg[i] != -1) continue;
        agg[i] = nagg;
        int sz = 1;
        const uint32_t a = __ldg(&sp[i]), b = __ldg(&sp[i + 1]);
        for (uint32_t p = a; p < b && sz < 4; ++p)
        {
            const uint32_t j = __ldg(&sc[p]);
            if (agg[j] == -1)
            {
                agg[j] = nagg;
                ++sz;
            }
        }
        ++nagg;
    }
    *nagg_out = (uint32_t)nagg;
}

// Standard three-phase smoothed-aggregation rule (no reference counterpart):
// 1. a row whose strong neighbours are all free becomes a root and takes them
// all; 2. a free row joins the phase-1 aggregate of its first aggregated
// strong neighbour; 3. the remaining rows group with their free strong
// neighbours.  One thread walks the rows in natural order (the phases are
// order-dependent); snap holds the phase-1 aggregates.
__global__ void k_aggregate_std(uint32_t nb, const uint32_t* __restrict__ sp, const uint32_t* __restrict__ sc,
                                int32_t* __restrict__ agg, int32_t* __restrict__ snap, uint32_t* __restrict__ nagg_out)
{
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    int32_t nagg = 0;
    for (uint32_t i = 0; i < nb; ++i)
    {
        if (agg[i] != -1) continue;
        const uint32_t a = __ldg(&sp[i]), b = __ldg(&sp[i + 1]);
        bool free_all = true;
        for (uint32_t p = a; p < b; ++p)
            if (agg[__ldg(&sc[p])] != -1)
            {
                free_all = false;
                break;
            }
        if (!free_all) continue;
        agg[i] = nagg;
        for (uint32_t p = a; p < b; ++p) agg[__ldg(&sc[p])] = nagg;
        ++nagg;
    }
    for (uint32_t i = 0; i < nb; ++i) snap[i] = agg[i];
    for (uint32_t i = 0; i < nb; ++i)
    {
        if (snap[i] != -1) continue;
        for (uint32_t p = __ldg(&sp[i]); p < __ldg(&sp[i + 1]); ++p)
        {
            const int32_t g = snap[__ldg(&sc[p])];
            if (g != -1)
            {
                agg[i] = g;
                break;
            }
        }
    }
    for (uint32_t i = 0; i < nb; ++i)
    {
        if (agg[i] != -1) continue;
        agg[i] = nagg;
        for (uint32_t p = __ldg(&sp[i]); p < __ldg(&sp[i + 1]); ++p)
            if (agg[__ldg(&sc[p])] == -1) agg[__ldg(&sc[p])] = nagg;
        ++nagg;
    }
    *nagg_out = (uint32_t)nagg;
}

// Parallel aggregation (the library default; no reference counterpart).
// Deterministic, with every pass reading only state from the previous pass:
//   roots: a distance-2 independent set of the strength graph, chosen in
//     rounds.  Each row has a fixed key (an integer hash of the row in the
//     high word, the row + 1 in the low word).  In a round, m1(i) is the
//     largest key among the undecided rows of {i} U S(i), and an undecided
//     row whose key equals the largest m1 over {i} U S(i) becomes a root.
//     Undecided rows within two strength edges of a root then leave the set.
//     The undecided row with the largest key always becomes a root, so the
//     rounds end.
//   aggregates: roots are numbered in row order; a row with a root among its
//     strong neighbours joins the one with the largest key; a row still
//     without an aggregate then joins the aggregate of its assigned strong
//     neighbour with the largest key (as assigned after the first phase);
//     the rows left over become singletons, numbered after the roots in row
//     order.
// S(i) are the strong columns of row i (the same strength test as above).

__device__ __host__ __forceinline__ uint64_t agg_key(uint32_t i)
{
    // integer hash (xorshift-multiply mix) of the row, then the row itself
    uint32_t x = i;
    x ^= x >> 16;
    x *= 0x7feb352du;
    x ^= x >> 15;
    x *= 0x846ca68bu;
    x ^= x >> 16;
    return ((uint64_t)x << 32) | (uint64_t)(i + 1u);
}

enum : uint8_t { kAggUndecided = 0, kAggRoot = 1, kAggOut = 2 };

__global__ void k_mis_m1(uint32_t n, const uint32_t* __restrict__ sp, const uint32_t* __restrict__ sc,
                         const uint8_t* __restrict__ st, uint64_t* __restrict__ m1)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        uint64_t m = st[i] == kAggUndecided ? agg_key(i) : 0ull;
        for (uint32_t p = sp[i]; p < sp[i + 1]; ++p)
        {
            const uint32_t j = sc[p];
            if (st[j] == kAggUndecided)
            {
                const uint64_t k = agg_key(j);
                m = k > m ? k : m;
            }
        }
        m1[i] = m;
    }
}

__global__ void k_mis_select(uint32_t n, const uint32_t* __restrict__ sp, const uint32_t* __restrict__ sc,
                             const uint64_t* __restrict__ m1, uint8_t* __restrict__ st)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        if (st[i] != kAggUndecided) continue;
        uint64_t m = m1[i];
        for (uint32_t p = sp[i]; p < sp[i + 1]; ++p)
        {
            const uint64_t k = m1[sc[p]];
            m = k > m ? k : m;
        }
        if (m == agg_key(i)) st[i] = kAggRoot;
    }
}

// c1(i): i is a root or has a strong neighbour that is one
__global__ void k_mis_cover1(uint32_t n, const uint32_t* __restrict__ sp, const uint32_t* __restrict__ sc,
                             const uint8_t* __restrict__ st, uint8_t* __restrict__ c1)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        uint8_t c = st[i] == kAggRoot;
        for (uint32_t p = sp[i]; p < sp[i + 1] && !c; ++p) c = st[sc[p]] == kAggRoot;
        c1[i] = c;
    }
}

// undecided rows with c1 on {i} U S(i) leave; counts the rows still undecided
__global__ void k_mis_cover2(uint32_t n, const uint32_t* __restrict__ sp, const uint32_t* __restrict__ sc,
                             const uint8_t* __restrict__ c1, uint8_t* __restrict__ st, uint32_t* __restrict__ left)
{
    uint32_t cnt = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        if (st[i] != kAggUndecided) continue;
        bool c = c1[i] != 0;
        for (uint32_t p = sp[i]; p < sp[i + 1] && !c; ++p) c = c1[sc[p]] != 0;
        if (c)
            st[i] = kAggOut;
        else
            ++cnt;
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if ((threadIdx.x & 31u) == 0 && cnt) atomicAdd(left, cnt);
}

__global__ void k_agg_flag(uint32_t n, const uint8_t* __restrict__ st, const int32_t* __restrict__ agg, int mode,
                           uint32_t* __restrict__ flag)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        flag[i] = mode == 0 ? (st[i] == kAggRoot) : (agg[i] < 0);
}

// roots take their number; other rows join the root neighbour with the largest key
__global__ void k_agg_roots(uint32_t n, const uint32_t* __restrict__ sp, const uint32_t* __restrict__ sc,
                            const uint8_t* __restrict__ st, const uint32_t* __restrict__ rank, int32_t* __restrict__ agg)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        if (st[i] == kAggRoot)
        {
            agg[i] = (int32_t)rank[i];
            continue;
        }
        uint64_t best = 0;
        int32_t g = -1;
        for (uint32_t p = sp[i]; p < sp[i + 1]; ++p)
        {
            const uint32_t j = sc[p];
            if (st[j] != kAggRoot) continue;
            const uint64_t k = agg_key(j);
            if (k > best)
            {
                best = k;
                g = (int32_t)rank[j];
            }
        }
        agg[i] = g;
    }
}

// rows still without an aggregate join the assigned strong neighbour with the largest key (snapshot)
__global__ void k_agg_extend(uint32_t n, const uint32_t* __restrict__ sp, const uint32_t* __restrict__ sc,
                             const int32_t* __restrict__ snap, int32_t* __restrict__ agg)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        if (snap[i] >= 0) continue;
        uint64_t best = 0;
        int32_t g = -1;
        for (uint32_t p = sp[i]; p < sp[i + 1]; ++p)
        {
            const uint32_t j = sc[p];
            if (snap[j] < 0) continue;
            const uint64_t k = agg_key(j);
            if (k > best)
            {
                best = k;
                g = snap[j];
            }
        }
        agg[i] = g;
    }
}

__global__ void k_agg_single(uint32_t n, uint32_t base, const uint32_t* __restrict__ rank, int32_t* __restrict__ agg)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (agg[i] < 0) agg[i] = (int32_t)(base + rank[i]);
}

// returns the aggregate count
static uint32_t aggregate_parallel(b2s_ctx* ctx, uint32_t n, const uint32_t* sp, const uint32_t* sc, int32_t* agg)
{
    if (!n) return 0;
    const unsigned g = stream_grid(ctx, n);
    DBuf<uint8_t> st(n), c1(n);
    DBuf<uint64_t> m1(n);
    DBuf<uint32_t> left(1), flag(n + 1), rank(n + 1);
    B2S_CUDA(cudaMemsetAsync(st.p, 0, n, ctx->stream));
    for (uint32_t round = 0;; ++round)
    {
        if (round > n) fail(B2S_CUDA_ERROR, "aggregation rounds did not terminate");
        B2S_CUDA(cudaMemsetAsync(left.p, 0, sizeof(uint32_t), ctx->stream));
        B2S_LAUNCH(ctx, k_mis_m1, g, kThreads, 0, n, sp, sc, st.p, m1.p);
        B2S_LAUNCH(ctx, k_mis_select, g, kThreads, 0, n, sp, sc, m1.p, st.p);
        B2S_LAUNCH(ctx, k_mis_cover1, g, kThreads, 0, n, sp, sc, st.p, c1.p);
        B2S_LAUNCH(ctx, k_mis_cover2, g, kThreads, 0, n, sp, sc, c1.p, st.p, left.p);
        uint32_t h = 0;
        d2h(ctx, &h, left.p, sizeof(uint32_t));
        sync(ctx);
        if (!h) break;
    }
    B2S_LAUNCH(ctx, k_agg_flag, g, kThreads, 0, n, st.p, (const int32_t*)nullptr, 0, flag.p);
    const uint32_t nroots = exclusive_scan(ctx, flag.p, rank.p, n);
    B2S_LAUNCH(ctx, k_agg_roots, g, kThreads, 0, n, sp, sc, st.p, rank.p, agg);
    DBuf<int32_t> snap(n);
    d2d(ctx, snap.p, agg, (size_t)n * sizeof(int32_t));
    B2S_LAUNCH(ctx, k_agg_extend, g, kThreads, 0, n, sp, sc, snap.p, agg);
    B2S_LAUNCH(ctx, k_agg_flag, g, kThreads, 0, n, st.p, agg, 1, flag.p);
    const uint32_t nsingle = exclusive_scan(ctx, flag.p, rank.p, n);
    if (nsingle) B2S_LAUNCH(ctx, k_agg_single, g, kThreads, 0, n, nroots, rank.p, agg);
    return nroots + nsingle;
}

// ------------------------------------------------------------ prolongation

// distinct aggregates among {agg[i]} U {agg[k] : k in row i}, ascending; GL lanes
// (a thread, or a whole warp) hold the row, every lane gets the count
template <int GL>
__device__ __forceinline__ uint32_t p_row_cols(uint32_t i, const uint32_t* rp, const uint32_t* ci, const int32_t* agg,
                                               uint32_t* out)
{
    // count distinct; write ascending when out != null
    const uint32_t l = threadIdx.x % GL;
    uint32_t cnt = 0;
    int32_t last = -1;
    for (;;)
    {
        // smallest candidate greater than `last`
        int32_t best = 0x7fffffff;
        const int32_t gi = agg[i];
        if (gi > last && gi < best) best = gi;
        for (uint32_t p = rp[i] + l; p < rp[i + 1]; p += GL)
        {
            const int32_t g = agg[ci[p]];
            if (g > last && g < best) best = g;
        }
        if constexpr (GL > 1) best = __reduce_min_sync(0xffffffffu, best);
        if (best == 0x7fffffff) break;
        if (out && l == 0) out[cnt] = (uint32_t)best;
        ++cnt;
        last = best;
    }
    if constexpr (GL > 1) __syncwarp();  // the columns are read by every lane
    return cnt;
}

template <int GL>
__global__ void k_p_count(uint32_t nb, const uint32_t* __restrict__ rp, const uint32_t* __restrict__ ci,
                          const int32_t* __restrict__ agg, uint32_t* __restrict__ cnt)
{
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) / GL; i < nb; i += gridDim.x * blockDim.x / GL)
    {
        const uint32_t c = p_row_cols<GL>(i, rp, ci, agg, nullptr);
        if (threadIdx.x % GL == 0) cnt[i] = c;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) cnt[nb] = 0;
}

// Row i of P: the tentative prolongation's identity block and the smoothing
// terms, each column's in row order.  With a warp a row, lane l owns every 32nd
// column and adds that column's terms itself, so the order stays the row's.
template <int BS, int GL>
__global__ void k_p_fill(uint32_t nb, const uint32_t* __restrict__ rp, const uint32_t* __restrict__ ci,
                         const double* __restrict__ v, const double* __restrict__ dinv, const int32_t* __restrict__ agg,
                         const uint32_t* __restrict__ prp, uint32_t* pci, double* __restrict__ pv)
{
    constexpr int BV = BS * BS;
    const uint32_t l = threadIdx.x % GL;
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) / GL; i < nb; i += gridDim.x * blockDim.x / GL)
    {
        const uint32_t base = prp[i];
        const uint32_t cnt = p_row_cols<GL>(i, rp, ci, agg, pci + base);
        for (uint32_t s = l; s < cnt; s += GL)
            for (int k = 0; k < BV; ++k) pv[(size_t)(base + s) * BV + k] = 0.0;
        auto slot = [&](uint32_t g) {
            uint32_t lo = 0, hi = cnt;
            while (lo < hi)
            {
                const uint32_t mid = (lo + hi) / 2;
                if (pci[base + mid] < g)
                    lo = mid + 1;
                else
                    hi = mid;
            }
            return lo;
        };
        const uint32_t diag = slot((uint32_t)agg[i]);
        if (diag % GL == l)
        {
            double* I = &pv[(size_t)(base + diag) * BV];
            for (int r = 0; r < BS; ++r) I[r * BS + r] = 1.0;
        }
        const double* Di = &dinv[(size_t)i * BV];
        for (uint32_t q = rp[i]; q < rp[i + 1]; q += GL)
        {
            // GL entries' slots, then each entry by its column's owner
            const uint32_t mine = q + l < rp[i + 1] ? slot((uint32_t)agg[ci[q + l]]) : 0u;
            const uint32_t m = GL > 1 ? min((uint32_t)GL, rp[i + 1] - q) : 1u;
            for (uint32_t t = 0; t < m; ++t)
            {
                const uint32_t at = GL > 1 ? __shfl_sync(0xffffffffu, mine, t) : mine;
                if (at % GL != l) continue;
                const double* ab = &v[(size_t)(q + t) * BV];
                double* dst = &pv[(size_t)(base + at) * BV];
                for (int r = 0; r < BS; ++r)
                    for (int c = 0; c < BS; ++c)
                    {
                        double s = 0.0;
                        for (int k = 0; k < BS; ++k) s += Di[r * BS + k] * ab[k * BS + c];
                        dst[r * BS + c] -= kOmega * s;
                    }
            }
        }
    }
}

// ------------------------------------------------------------ block transpose

__global__ void k_bt_count(uint32_t nb, const uint32_t* __restrict__ rp, const uint32_t* __restrict__ ci,
                           uint32_t* __restrict__ cnt)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += gridDim.x * blockDim.x)
        for (uint32_t p = rp[i]; p < rp[i + 1]; ++p) atomicAdd(&cnt[ci[p]], 1u);
}

// T's entry d = A's entry perm[d], its block transposed; rows ascending by construction
template <int BS>
__global__ void k_bt_gather(uint32_t nnz, const uint32_t* __restrict__ perm, const uint32_t* __restrict__ row_of,
                            const double* __restrict__ v, uint32_t* __restrict__ tci, double* __restrict__ tv)
{
    constexpr int BV = BS * BS;
    for (uint32_t d = blockIdx.x * blockDim.x + threadIdx.x; d < nnz; d += gridDim.x * blockDim.x)
    {
        const uint32_t p = perm[d];
        tci[d] = row_of[p];
#pragma unroll
        for (int r = 0; r < BS; ++r)
#pragma unroll
            for (int c = 0; c < BS; ++c) tv[(size_t)d * BV + r * BS + c] = v[(size_t)p * BV + c * BS + r];
    }
}

template <int BS>
void block_transpose(b2s_ctx* ctx, const BaijDev& A, BaijDev& T)
{
    constexpr int BV = BS * BS;
    T.bs = BS;
    T.nbr = A.nbc;
    T.nbc = A.nbr;
    DBuf<uint32_t> cnt(T.nbr + 1);
    B2S_CUDA(cudaMemsetAsync(cnt.p, 0, cnt.bytes(), ctx->stream));
    if (A.nbr) B2S_LAUNCH(ctx, k_bt_count, stream_grid(ctx, A.nbr), kThreads, 0, A.nbr, A.rp.p, A.ci.p, cnt.p);
    T.rp.alloc(T.nbr + 1);
    const uint32_t nnz = exclusive_scan(ctx, cnt.p, T.rp.p, T.nbr);
    T.ci.alloc(nnz ? nnz : 1);
    T.v.alloc(nnz ? (size_t)nnz * BV : 1);
    DBuf<uint32_t> perm, row_of;
    transpose_order(ctx, A.nbr, A.nbc, A.rp.p, A.ci.p, nnz, perm, row_of);
    if (nnz)
        B2S_LAUNCH(ctx, k_bt_gather<BS>, stream_grid(ctx, nnz), kThreads, 0, nnz, perm.p, row_of.p, A.v.p, T.ci.p,
                   T.v.p);
    finish_baij(ctx, T);
}

// ------------------------------------------------------------ block SpGEMM

__global__ void k_mm_ub(uint32_t nr, const uint32_t* __restrict__ arp, const uint32_t* __restrict__ aci,
                        const uint32_t* __restrict__ brp, uint32_t* __restrict__ cnt)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nr; i += gridDim.x * blockDim.x)
    {
        uint32_t c = 0;
        for (uint32_t p = arp[i]; p < arp[i + 1]; ++p) c += brp[aci[p] + 1] - brp[aci[p]];
        cnt[i] = c;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) cnt[nr] = 0;
}

__global__ void k_mm_cand(uint32_t nr, const uint32_t* __restrict__ arp, const uint32_t* __restrict__ aci,
                          const uint32_t* __restrict__ brp, const uint32_t* __restrict__ bci,
                          const uint32_t* __restrict__ off, uint32_t* __restrict__ cand)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nr; i += gridDim.x * blockDim.x)
    {
        uint32_t w = off[i];
        for (uint32_t p = arp[i]; p < arp[i + 1]; ++p)
            for (uint32_t q = brp[aci[p]]; q < brp[aci[p] + 1]; ++q) cand[w++] = bci[q];
    }
}

__global__ void k_mm_unique_count(uint32_t nr, const uint32_t* __restrict__ off, const uint32_t* __restrict__ cand,
                                  uint32_t* __restrict__ cnt)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nr; i += gridDim.x * blockDim.x)
    {
        uint32_t c = 0;
        for (uint32_t k = off[i]; k < off[i + 1]; ++k) c += (k == off[i] || cand[k] != cand[k - 1]);
        cnt[i] = c;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) cnt[nr] = 0;
}

__global__ void k_mm_unique_fill(uint32_t nr, const uint32_t* __restrict__ off, const uint32_t* __restrict__ cand,
                                 const uint32_t* __restrict__ crp, uint32_t* __restrict__ cci)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nr; i += gridDim.x * blockDim.x)
    {
        uint32_t w = crp[i];
        for (uint32_t k = off[i]; k < off[i + 1]; ++k)
            if (k == off[i] || cand[k] != cand[k - 1]) cci[w++] = cand[k];
    }
}

// One row i of C = A B per group of GL lanes: the row's distinct columns are
// collected in an open-addressing hash table of SL slots in shared memory
// (inserted with atomicCAS), the group taking A's row entries in order and its
// lanes one row of B.  MmMode::Count: cnt[i] = their number; Columns: they are
// written in ascending order (rank sort, the columns being distinct) to
// cci[crp[i]...]; Values (scalars): their sums too, every product added in A's
// entry order -- the entries of one row of B have distinct columns, so no two
// lanes add into one slot between two barriers -- which is the reference's order.
// A row whose columns do not fit the table raises *overflow, and the groups stop
// after the row they are at; the caller takes a larger one.
//
// A row of B is as short as 3 or 4 entries (the prolongation), so a warp a row left
// most lanes idle and cleared and searched a 512-slot table for 8 columns: 128^3,
// A P and R (A P) of the first level 1.14 + 2.64 + 0.60 and 0.53 + 1.01 + 1.34 ms
// (count, columns, values apart), 0.19 + 0.56 and 0.24 + 0.67 this way (values with the
// columns).
enum class MmMode
{
    Count,
    Columns,
    Values
};
constexpr uint32_t kMmEmpty = 0xFFFFFFFFu;

// shared memory of one group
template <int SL, MmMode MODE>
struct MmTable
{
    double val[MODE == MmMode::Values ? SL : 1];
    uint32_t key[SL];
    uint32_t list[MODE == MmMode::Count ? 1 : SL];  // the keys found, and their slots
    uint16_t slot[MODE == MmMode::Count ? 2 : SL];
};

template <int GL, int SL, MmMode MODE>
__global__ void __launch_bounds__(kThreads) k_mm_row(uint32_t nr, const uint32_t* __restrict__ arp,
                                                     const uint32_t* __restrict__ aci, const double* __restrict__ av,
                                                     const uint32_t* __restrict__ brp, const uint32_t* __restrict__ bci,
                                                     const double* __restrict__ bv, uint32_t* __restrict__ cnt,
                                                     const uint32_t* __restrict__ crp, uint32_t* __restrict__ cci,
                                                     double* __restrict__ cv, int* overflow)
{
    static_assert(SL >= GL && SL % GL == 0 && (SL & (SL - 1)) == 0 && 32 % GL == 0, "table");
    constexpr int RPC = kThreads / GL, U = MODE == MmMode::Count ? 2 : 4;
    constexpr int SHIFT = 32 - (SL == 32 ? 5 : SL == 128 ? 7 : SL == 256 ? 8 : 9);
    constexpr bool VALUES = MODE == MmMode::Values;
    extern __shared__ __align__(16) unsigned char mm_sm[];
    const uint32_t g = threadIdx.x / GL, l = threadIdx.x % GL, in_warp = (threadIdx.x & 31u) / GL;
    MmTable<SL, MODE>& T = reinterpret_cast<MmTable<SL, MODE>*>(mm_sm)[g];
    if (MODE == MmMode::Count && blockIdx.x == 0 && threadIdx.x == 0) cnt[nr] = 0;
    for (uint32_t i0 = blockIdx.x * RPC; i0 < nr; i0 += gridDim.x * RPC)
    {
        const uint32_t i = i0 + g;
        int stop = 0;  // looked at when the row is done
        if constexpr (MODE == MmMode::Count) stop = *(volatile int*)overflow;
        for (uint32_t s = l; s < (uint32_t)SL; s += GL)
        {
            T.key[s] = kMmEmpty;
            if constexpr (VALUES) T.val[s] = 0.0;
        }
        __syncwarp();
        const uint32_t a0 = i < nr ? arp[i] : 0u, na = i < nr ? arp[i + 1] - a0 : 0u;
        const uint32_t nmax = __reduce_max_sync(0xffffffffu, na);
        uint32_t added = 0;
        bool full = false;
        // one entry of B into the table (s: the product's term)
        auto take = [&](uint32_t j, double term) {
            if (MODE == MmMode::Count && full) return;
            uint32_t h = (j * 2654435761u) >> SHIFT;
            for (uint32_t probes = 0;; ++probes)
            {
                if (probes == (uint32_t)SL)
                {
                    full = true;
                    return;
                }
                const uint32_t old = atomicCAS(&T.key[h], kMmEmpty, j);
                if (old == kMmEmpty) ++added;
                if (old == kMmEmpty || old == j) break;
                h = (h + 1) & (SL - 1);
            }
            if constexpr (VALUES) T.val[h] += term;
        };
        for (uint32_t c = 0; c < nmax; c += GL)
        {
            // GL entries of A's row, one a lane
            uint32_t b0 = 0, len = 0;
            double a = 0.0;
            if (c + l < na)
            {
                const uint32_t k = aci[a0 + c + l];
                b0 = brp[k];
                len = brp[k + 1] - b0;
                if constexpr (VALUES) a = av[a0 + c + l];
            }
            // U of them at a time, their rows of B in flight together
            for (uint32_t t = 0; t < (uint32_t)GL && c + t < nmax; t += U)
            {
                uint32_t kb[U], ln[U], j[U];
                double v[U], ak[U];
#pragma unroll
                for (int u = 0; u < U; ++u)
                {
                    kb[u] = __shfl_sync(0xffffffffu, b0, t + u, GL);
                    ln[u] = __shfl_sync(0xffffffffu, len, t + u, GL);
                    ak[u] = VALUES ? __shfl_sync(0xffffffffu, a, t + u, GL) : 0.0;
                    j[u] = l < ln[u] ? bci[kb[u] + l] : kMmEmpty;
                    v[u] = VALUES && l < ln[u] ? bv[kb[u] + l] : 0.0;
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                {
                    if (j[u] != kMmEmpty) take(j[u], 0.0 + ak[u] * v[u]);
                    for (uint32_t q = l + GL; q < ln[u]; q += GL)
                        take(bci[kb[u] + q], VALUES ? 0.0 + ak[u] * bv[kb[u] + q] : 0.0);
                    if constexpr (VALUES) __syncwarp();
                }
            }
        }
        __syncwarp();
        if (full) atomicExch(overflow, 1);
        if constexpr (MODE == MmMode::Count)
        {
#pragma unroll
            for (int o = GL / 2; o; o >>= 1) added += __shfl_xor_sync(0xffffffffu, added, o);
            if (l == 0 && i < nr) cnt[i] = added;
            // counts of this table size are of no use once a row has not fitted
            if (__any_sync(0xffffffffu, stop != 0)) return;
        }
        else
        {
            uint32_t found = 0;
            for (uint32_t s0 = 0; s0 < (uint32_t)SL; s0 += GL)
            {
                const uint32_t key = T.key[s0 + l];
                const uint32_t m = (__ballot_sync(0xffffffffu, key != kMmEmpty) >> (in_warp * GL)) & (0xffffffffu >> (32 - GL));
                if (key != kMmEmpty)
                {
                    const uint32_t at = found + __popc(m & ((1u << l) - 1u));
                    T.list[at] = key;
                    T.slot[at] = (uint16_t)(s0 + l);
                }
                found += __popc(m);
            }
            __syncwarp();
            const uint32_t out = i < nr ? crp[i] : 0u;
            for (uint32_t x = l; x < found; x += GL)
            {
                const uint32_t key = T.list[x];
                uint32_t r = 0;
                for (uint32_t y = 0; y < found; ++y) r += T.list[y] < key;
                cci[out + r] = key;
                if constexpr (VALUES) cv[out + r] = T.val[T.slot[x]];
            }
        }
        __syncwarp();  // the table is reused by the next row
    }
}

// C row i: every (pa, pb) product added into its column's block in the
// reference's order (blk_matmul, blockMatrix.hpp:883-932)
template <int BS>
__global__ void k_mm_numeric(uint32_t nr, const uint32_t* __restrict__ arp, const uint32_t* __restrict__ aci,
                             const double* __restrict__ av, const uint32_t* __restrict__ brp,
                             const uint32_t* __restrict__ bci, const double* __restrict__ bv,
                             const uint32_t* __restrict__ crp, const uint32_t* __restrict__ cci, double* __restrict__ cv)
{
    constexpr int BV = BS * BS;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nr; i += gridDim.x * blockDim.x)
    {
        const uint32_t c0 = crp[i], c1 = crp[i + 1];
        for (uint32_t s = c0; s < c1; ++s)
            for (int k = 0; k < BV; ++k) cv[(size_t)s * BV + k] = 0.0;
        for (uint32_t pa = arp[i]; pa < arp[i + 1]; ++pa)
        {
            const uint32_t k = aci[pa];
            const double* ab = &av[(size_t)pa * BV];
            for (uint32_t pb = brp[k]; pb < brp[k + 1]; ++pb)
            {
                const uint32_t j = bci[pb];
                uint32_t lo = c0, hi = c1;
                while (lo < hi)
                {
                    const uint32_t mid = (lo + hi) / 2;
                    if (cci[mid] < j)
                        lo = mid + 1;
                    else
                        hi = mid;
                }
                const double* bb = &bv[(size_t)pb * BV];
                double* cb = &cv[(size_t)lo * BV];
                for (int r = 0; r < BS; ++r)
                    for (int c = 0; c < BS; ++c)
                    {
                        double s = 0.0;
                        for (int m = 0; m < BS; ++m) s += ab[r * BS + m] * bb[m * BS + c];
                        cb[r * BS + c] += s;
                    }
            }
        }
    }
}

// The same product, one warp per C row: the warp walks A's row entries pa in
// order and its lanes take the entries pb of B's row k in parallel.  The
// entries of one B row have distinct columns, so within a pa no two lanes add
// into the same C block, and a __syncwarp between pa keeps every C block's
// additions in pa order -- the order of k_mm_numeric.  Used when B's rows are
// long (R (A P)); for short rows (A P) the thread-per-row kernel is faster.
template <int BS>
__global__ void k_mm_numeric_warp(uint32_t nr, const uint32_t* __restrict__ arp, const uint32_t* __restrict__ aci,
                                  const double* __restrict__ av, const uint32_t* __restrict__ brp,
                                  const uint32_t* __restrict__ bci, const double* __restrict__ bv,
                                  const uint32_t* __restrict__ crp, const uint32_t* __restrict__ cci,
                                  double* __restrict__ cv)
{
    constexpr int BV = BS * BS;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < nr; i += warps)
    {
        const uint32_t c0 = crp[i], c1 = crp[i + 1];
        for (uint32_t s = c0 * BV + lane; s < c1 * BV; s += 32) cv[s] = 0.0;
        __syncwarp();
        for (uint32_t pa = arp[i]; pa < arp[i + 1]; ++pa)
        {
            const uint32_t k = aci[pa];
            double ab[BV];
#pragma unroll
            for (int q = 0; q < BV; ++q) ab[q] = av[(size_t)pa * BV + q];
            for (uint32_t pb = brp[k] + lane; pb < brp[k + 1]; pb += 32)
            {
                const uint32_t j = bci[pb];
                uint32_t lo = c0, hi = c1;
                while (lo < hi)
                {
                    const uint32_t mid = (lo + hi) / 2;
                    if (cci[mid] < j)
                        lo = mid + 1;
                    else
                        hi = mid;
                }
                const double* bb = &bv[(size_t)pb * BV];
                double* cb = &cv[(size_t)lo * BV];
#pragma unroll
                for (int r = 0; r < BS; ++r)
#pragma unroll
                    for (int c = 0; c < BS; ++c)
                    {
                        double sum = 0.0;
#pragma unroll
                        for (int m = 0; m < BS; ++m) sum += ab[r * BS + m] * bb[m * BS + c];
                        cb[r * BS + c] += sum;
                    }
            }
            __syncwarp();
        }
    }
}

template <int GL, int SL, MmMode MODE>
void mm_rows_t(b2s_ctx* ctx, const BaijDev& A, const BaijDev& B, BaijDev& C, uint32_t* cnt, int* overflow)
{
    constexpr uint32_t rpc = kThreads / GL, smem = rpc * sizeof(MmTable<SL, MODE>);
    auto kern = k_mm_row<GL, SL, MODE>;
    B2S_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const unsigned grid = std::min<unsigned>((A.nbr + rpc - 1) / rpc, (unsigned)ctx->sm_count * 8);
    B2S_LAUNCH(ctx, kern, grid, kThreads, smem, A.nbr, A.rp.p, A.ci.p, A.v.p, B.rp.p, B.ci.p, B.v.p, cnt, C.rp.p, C.ci.p,
               C.v.p, overflow);
}

// tier: 32, 128, 256 or 512 slots a row; lanes a row by B's mean row length, so
// that a row of B is about one pass of them.  Whole products, ms, at 4 / 8 / 16
// lanes and 32 slots for rows of B of 3 entries (P of the 64^3 grid) 3.42 / 3.44 /
// 3.64; at 8 / 16 / 32 lanes for 25 (27-point, 128 slots) 17.7 / 17.6 / 18.1, for 51
// (a band, 128) 4.2 / 3.9 / 3.8; at 16 / 32 for 228 (512 slots) 7.8 / 5.7.  Slots
// beyond the columns cost their clearing: 3.42 with 32 at 3 entries, 3.9 with 512.
// A table that is too small costs little, as its counts stop at the first row that
// does not fit: a 64^3 grid whose one long row, and the rows that refer to it, have
// 900 columns 25 ms (66 when the counts of three sizes ran to their end).
template <MmMode MODE>
void mm_rows(b2s_ctx* ctx, int tier, double mean_b, const BaijDev& A, const BaijDev& B, BaijDev& C, uint32_t* cnt,
             int* overflow)
{
    if (tier == 0 && mean_b <= 4.5)
        mm_rows_t<4, 32, MODE>(ctx, A, B, C, cnt, overflow);
    else if (tier == 0)
        mm_rows_t<8, 32, MODE>(ctx, A, B, C, cnt, overflow);
    else if (tier == 1 && mean_b <= 10.0)
        mm_rows_t<8, 128, MODE>(ctx, A, B, C, cnt, overflow);
    else if (tier == 1 && mean_b <= 20.0)
        mm_rows_t<16, 128, MODE>(ctx, A, B, C, cnt, overflow);
    else if (tier == 1)
        mm_rows_t<32, 128, MODE>(ctx, A, B, C, cnt, overflow);
    else if (tier == 2 && mean_b <= 20.0)
        mm_rows_t<16, 256, MODE>(ctx, A, B, C, cnt, overflow);
    else if (tier == 2)
        mm_rows_t<32, 256, MODE>(ctx, A, B, C, cnt, overflow);
    else
        mm_rows_t<32, 512, MODE>(ctx, A, B, C, cnt, overflow);
}

template <int BS>
void block_matmul(b2s_ctx* ctx, const BaijDev& A, const BaijDev& B, BaijDev& C)
{
    constexpr int BV = BS * BS;
    const uint32_t nr = A.nbr;
    C.bs = BS;
    C.nbr = nr;
    C.nbc = B.nbc;
    DBuf<uint32_t> cnt(nr + 1);
    C.rp.alloc(nr + 1);
    // lanes by B's mean row, slots by the candidates of a row of C; a table that
    // overflows is tried again at the next size, and past 512 columns the rows'
    // candidates are sorted
    const double mean_b = B.nbr ? (double)B.nnzb / B.nbr : 0.0, cand = nr ? (double)A.nnzb / nr * mean_b : 0.0;
    int tier = cand <= 32.0 ? 0 : cand <= 1024.0 ? 1 : cand <= 8192.0 ? 2 : 3;
    DBuf<int> overflow(1);
    uint32_t nnz = 0;
    int wide = 0;
    for (; tier < 4; ++tier)
    {
        B2S_CUDA(cudaMemsetAsync(overflow.p, 0, sizeof(int), ctx->stream));
        if (nr) mm_rows<MmMode::Count>(ctx, tier, mean_b, A, B, C, cnt.p, overflow.p);
        nnz = exclusive_scan(ctx, cnt.p, C.rp.p, nr);
        d2h(ctx, &wide, overflow.p, sizeof(int));
        sync(ctx);
        if (!wide) break;
    }
    bool values = false;
    if (!wide)
    {
        C.ci.alloc(nnz ? nnz : 1);
        C.v.alloc(nnz ? (size_t)nnz * BV : 1);
        if (nr && BS == 1)
            mm_rows<MmMode::Values>(ctx, tier, mean_b, A, B, C, nullptr, overflow.p);
        else if (nr)
            mm_rows<MmMode::Columns>(ctx, tier, mean_b, A, B, C, nullptr, overflow.p);
        values = BS == 1;
    }
    else
    {
        DBuf<uint32_t> off(nr + 1);
        if (nr) B2S_LAUNCH(ctx, k_mm_ub, stream_grid(ctx, nr), kThreads, 0, nr, A.rp.p, A.ci.p, B.rp.p, cnt.p);
        const uint32_t total = exclusive_scan(ctx, cnt.p, off.p, nr);
        DBuf<uint32_t> cand(total ? total : 1), sorted(total ? total : 1);
        if (nr)
            B2S_LAUNCH(ctx, k_mm_cand, stream_grid(ctx, nr), kThreads, 0, nr, A.rp.p, A.ci.p, B.rp.p, B.ci.p, off.p,
                       cand.p);
        if (total)
        {
            size_t bytes = 0;
            B2S_CUDA(cub::DeviceSegmentedSort::SortKeys(nullptr, bytes, cand.p, sorted.p, (int64_t)total, (int64_t)nr,
                                                        off.p, off.p + 1, ctx->stream));
            DBuf<uint8_t> tmp(bytes ? bytes : 1);
            B2S_CUDA(cub::DeviceSegmentedSort::SortKeys(tmp.p, bytes, cand.p, sorted.p, (int64_t)total, (int64_t)nr,
                                                        off.p, off.p + 1, ctx->stream));
            ctx->launches += 1;
        }
        if (nr) B2S_LAUNCH(ctx, k_mm_unique_count, stream_grid(ctx, nr), kThreads, 0, nr, off.p, sorted.p, cnt.p);
        nnz = exclusive_scan(ctx, cnt.p, C.rp.p, nr);
        C.ci.alloc(nnz ? nnz : 1);
        if (nr) B2S_LAUNCH(ctx, k_mm_unique_fill, stream_grid(ctx, nr), kThreads, 0, nr, off.p, sorted.p, C.rp.p, C.ci.p);
    }
    if (wide) C.v.alloc(nnz ? (size_t)nnz * BV : 1);
    if (nr && !values)
    {
        // B's mean row length decides: warp per C row for long rows, thread per C row otherwise
        if (B.nbr && B.nnzb >= 8ull * B.nbr)
        {
            const uint64_t warps = nr, ctas = (warps + kThreads / 32 - 1) / (kThreads / 32);
            const unsigned grid = (unsigned)std::min<uint64_t>(ctas, (uint64_t)ctx->sm_count * 8);
            B2S_LAUNCH(ctx, k_mm_numeric_warp<BS>, grid, kThreads, 0, nr, A.rp.p, A.ci.p, A.v.p, B.rp.p, B.ci.p,
                       B.v.p, C.rp.p, C.ci.p, C.v.p);
        }
        else
            B2S_LAUNCH(ctx, k_mm_numeric<BS>, stream_grid(ctx, nr), kThreads, 0, nr, A.rp.p, A.ci.p, A.v.p, B.rp.p,
                       B.ci.p, B.v.p, C.rp.p, C.ci.p, C.v.p);
    }
    finish_baij(ctx, C);
}

// ------------------------------------------------------------ coarsest level

template <int BS>
__global__ void k_dense_from_baij(uint32_t nb, const uint32_t* __restrict__ rp, const uint32_t* __restrict__ ci,
                                  const double* __restrict__ v, double* __restrict__ D, int sz)
{
    constexpr int BV = BS * BS;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += gridDim.x * blockDim.x)
        for (uint32_t p = rp[i]; p < rp[i + 1]; ++p)
            for (int r = 0; r < BS; ++r)
                for (int c = 0; c < BS; ++c)
                    D[(size_t)(i * BS + r) * sz + ci[p] * BS + c] = v[(size_t)p * BV + r * BS + c];
}

// The coarsest operator fits shared memory up to this size (and a thread a row)
constexpr int kDenseSmem = 160;
inline size_t dense_smem(int sz) { return sz <= kDenseSmem ? (size_t)sz * (sz | 1) * sizeof(double) : 0; }

// One CTA.  ref == 1: the reference's elimination (blockMatrix.hpp:962-981):
// rows swapped, pivot clamped to +-1e-14, the multiplier column eliminated
// along with the row (j from k).  ref == 0: LU with partial pivoting,
// multipliers stored below the diagonal and the permutation kept in piv.
// The matrix sits in shared memory (global memory past kDenseSmem), the pivot is
// one warp's search and the update spreads over rows and columns: 47 unknowns
// 0.557 -> 0.031 ms (one thread scanning the CTA's candidates and a thread a row).
__global__ void __launch_bounds__(kThreads) k_dense_factor(double* Dg, int sz, int ref, int* piv)
{
    extern __shared__ __align__(16) double dense_sm[];
    __shared__ int s_pk;
    const bool in_smem = sz <= kDenseSmem;
    double* const D = in_smem ? dense_sm : Dg;
    const int ld = in_smem ? (sz | 1) : sz;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    constexpr int TY = kThreads / 32;
    if (in_smem)
        for (int i = ty; i < sz; i += TY)
            for (int j = tx; j < sz; j += 32) D[i * ld + j] = Dg[(size_t)i * sz + j];
    for (int i = threadIdx.x; i < sz; i += blockDim.x) piv[i] = i;
    __syncthreads();
    for (int k = 0; k < sz; ++k)
    {
        // first row with the largest |D[i][k]|, i >= k (strict > keeps the earliest)
        if (ty == 0)
        {
            double best = -1.0;
            int bi = k;
            for (int i = k + tx; i < sz; i += 32)
            {
                const double a = fabs(D[(size_t)i * ld + k]);
                if (a > best)
                {
                    best = a;
                    bi = i;
                }
            }
#pragma unroll
            for (int o = 16; o; o >>= 1)
            {
                const double b = __shfl_xor_sync(0xffffffffu, best, o);
                const int i = __shfl_xor_sync(0xffffffffu, bi, o);
                if (b > best || (b == best && i < bi))
                {
                    best = b;
                    bi = i;
                }
            }
            if (tx == 0) s_pk = bi;
        }
        __syncthreads();
        const int pk = s_pk;
        if (pk != k)
        {
            for (int j = threadIdx.x; j < sz; j += blockDim.x)
            {
                const double t = D[(size_t)k * ld + j];
                D[(size_t)k * ld + j] = D[(size_t)pk * ld + j];
                D[(size_t)pk * ld + j] = t;
            }
            if (threadIdx.x == 0 && !ref)
            {
                const int t = piv[k];
                piv[k] = piv[pk];
                piv[pk] = t;
            }
        }
        __syncthreads();
        const double raw = D[(size_t)k * ld + k];
        double d = raw;
        if (ref)
        {
            if (fabs(d) < 1e-14) d = (d >= 0 ? 1e-14 : -1e-14);
        }
        else if (fabs(d) < 1e-300)
            d = 1e-300;
        __syncthreads();  // (the pivot is read before it is replaced)
        if (!ref && d != raw && threadIdx.x == 0) D[(size_t)k * ld + k] = d;
        // a warp a row: every lane forms the row's multiplier, then takes its columns
        for (int i = k + 1 + ty; i < sz; i += TY)
        {
            const double f = D[(size_t)i * ld + k] / d;
            __syncwarp();
            if (ref)
            {
                if (tx == 0) D[(size_t)i * ld + k] -= f * raw;
            }
            else if (tx == 0)
                D[(size_t)i * ld + k] = f;
            for (int j = k + 1 + tx; j < sz; j += 32) D[(size_t)i * ld + j] -= f * D[(size_t)k * ld + j];
        }
        __syncthreads();
    }
    if (in_smem)
        for (int i = ty; i < sz; i += TY)
            for (int j = tx; j < sz; j += 32) Dg[(size_t)i * sz + j] = D[i * ld + j];
}

// Coarsest solve, one CTA.  The reference's row sums are sequential: forward, row i
// takes column j's term when x_j is known, so a thread a row works through the
// columns together; backward, row i starts with x_{i+1}'s term, so the row's
// products are formed side by side and subtracted by one thread in order.  47
// unknowns 65 -> 17 us (one thread for all of it).
__global__ void __launch_bounds__(kThreads) k_dense_solve(const double* __restrict__ Dg, int sz, int ref,
                                                          const int* __restrict__ piv, const double* __restrict__ rhs,
                                                          double* __restrict__ x, const int* done)
{
    if (done && *done) return;
    extern __shared__ __align__(16) double dense_sm[];
    __shared__ double s_x[kDenseSmem], s_t[kDenseSmem];
    const int t = threadIdx.x, tx = t & 31;
    if (sz <= kDenseSmem)
    {
        const int ld = sz | 1;
        for (int i = t >> 5; i < sz; i += kThreads / 32)
            for (int j = tx; j < sz; j += 32) dense_sm[i * ld + j] = Dg[(size_t)i * sz + j];
        auto pivot = [&](int i) {
            const double d = dense_sm[i * ld + i];
            return ref && fabs(d) < 1e-14 ? (d >= 0 ? 1e-14 : -1e-14) : d;
        };
        double xi = t < sz ? rhs[ref ? t : piv[t]] : 0.0;
        __syncthreads();
        for (int j = 0; j < sz; ++j)
        {
            if (t == j) s_x[j] = xi;
            __syncthreads();
            if (t > j && t < sz)
            {
                const double f = ref ? dense_sm[t * ld + j] / pivot(j) : dense_sm[t * ld + j];
                xi -= f * s_x[j];
            }
        }
        __syncthreads();
        if (t >= 32) return;
        for (int i = sz - 1; i >= 0; --i)
        {
            for (int j = i + 1 + tx; j < sz; j += 32) s_t[j] = dense_sm[i * ld + j] * s_x[j];
            __syncwarp();
            if (tx == 0)
            {
                double v = s_x[i];
#pragma unroll 4
                for (int j = i + 1; j < sz; ++j) v -= s_t[j];
                s_x[i] = v / pivot(i);
            }
            __syncwarp();
        }
        for (int i = tx; i < sz; i += 32) x[i] = s_x[i];
        return;
    }
    if (t != 0) return;
    // Each row's running value stays in a register while its terms are
    // subtracted in the same order as an in-place x[i] -= ... loop would.
    const double* const D = Dg;
    if (ref)
    {
        for (int i = 0; i < sz; ++i) x[i] = rhs[i];
        for (int k = 0; k < sz; ++k)
        {
            double d = D[(size_t)k * sz + k];
            if (fabs(d) < 1e-14) d = (d >= 0 ? 1e-14 : -1e-14);
            const double xk = x[k];
            for (int i = k + 1; i < sz; ++i) x[i] -= (D[(size_t)i * sz + k] / d) * xk;
        }
        for (int i = sz - 1; i >= 0; --i)
        {
            double xi = x[i];
            for (int j = i + 1; j < sz; ++j) xi -= D[(size_t)i * sz + j] * x[j];
            double d = D[(size_t)i * sz + i];
            if (fabs(d) < 1e-14) d = (d >= 0 ? 1e-14 : -1e-14);
            x[i] = xi / d;
        }
    }
    else
    {
        for (int i = 0; i < sz; ++i)
        {
            double xi = rhs[piv[i]];
            for (int j = 0; j < i; ++j) xi -= D[(size_t)i * sz + j] * x[j];
            x[i] = xi;
        }
        for (int i = sz - 1; i >= 0; --i)
        {
            double xi = x[i];
            for (int j = i + 1; j < sz; ++j) xi -= D[(size_t)i * sz + j] * x[j];
            x[i] = xi / D[(size_t)i * sz + i];
        }
    }
}

// ------------------------------------------------------------ V-cycle kernels

// pre-smoothing from zero: sol = omega * dinv * rhs   (A*0 = 0, so r = rhs)
template <int BS, typename T>
__global__ void k_smooth0(uint32_t nb, const T* __restrict__ dinv, const double* __restrict__ rhs,
                          double* __restrict__ sol, const int* done)
{
    if (done && *done) return;
    constexpr int BV = BS * BS;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nb; i += gridDim.x * blockDim.x)
        for (int c = 0; c < BS; ++c)
        {
            double corr = 0.0;
            for (int rr = 0; rr < BS; ++rr) corr += (double)dinv[(size_t)i * BV + c * BS + rr] * rhs[(size_t)i * BS + rr];
            sol[(size_t)i * BS + c] = 0.0 + kOmega * corr;
        }
}

// Epilogues of the V-cycle's block products (baij_mv.cuh).  Each repeats the
// arithmetic of the separate vector pass it replaces, so the cycle's output is
// unchanged bit for bit.

// res = rhs - A sol
struct EpiResidual
{
    const double* rhs;
    double* res;
    template <int BS>
    __device__ __forceinline__ void put(uint32_t I, int r, double v, bool valid, uint32_t) const
    {
        if (!valid) return;
        const size_t i = (size_t)I * BS + r;
        res[i] = rhs[i] - v;
    }
};

// dst = sol + P e (coarse-grid correction)
struct EpiAddTo
{
    const double* sol;
    double* dst;
    template <int BS>
    __device__ __forceinline__ void put(uint32_t I, int r, double v, bool valid, uint32_t) const
    {
        if (!valid) return;
        const size_t i = (size_t)I * BS + r;
        dst[i] = sol[i] + v;
    }
};

// post-smoothing: sol = mid + omega * dinv * (rhs - A mid).  A block row's
// residual components come from the BS lanes of its row.
template <typename T>
struct EpiJacobi
{
    const T* dinv;
    const double* rhs;
    const double* mid;
    double* sol;
    template <int BS>
    __device__ __forceinline__ void put(uint32_t I, int r, double v, bool valid, uint32_t lane) const
    {
        constexpr int BV = BS * BS;
        const size_t i = (size_t)I * BS + r;
        const double res = valid ? rhs[i] - v : 0.0;
        double rv[BS];
        if constexpr (BS == 1)
            rv[0] = res;
        else
#pragma unroll
            for (int q = 0; q < BS; ++q) rv[q] = __shfl_sync(0xffffffffu, res, (lane / BS) * BS + q);
        if (!valid) return;
        double corr = 0.0;
#pragma unroll
        for (int q = 0; q < BS; ++q) corr += (double)dinv[(size_t)I * BV + r * BS + q] * rv[q];
        sol[i] = mid[i] + kOmega * corr;
    }
};

__global__ void k_zero(uint64_t n, double* __restrict__ x, const int* done)
{
    if (done && *done) return;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        x[i] = 0.0;
}

// ------------------------------------------------------------ hierarchy

struct Level
{
    std::unique_ptr<BaijDev> own;  // operator (null on level 0 when borrowed)
    const BaijDev* A = nullptr;
    BaijDev P, R;
    DBuf<double> dinv;
    DBuf<int32_t> agg;
    uint32_t nrows = 0;
    bool has_p = false;
    DBuf<double> tmp, r, rc, ec, sol;  // V-cycle work (rc / ec sized for the next level)
    DBuf<float> A32, P32, R32, dinv32;  // FP32 copies of the values (precision FP32)
};

__global__ void k_amg_to_f32(const double* __restrict__ a, float* __restrict__ b, uint64_t n)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        b[i] = (float)a[i];
}

static void amg_to_f32(b2s_ctx* ctx, const double* a, DBuf<float>& b, uint64_t n)
{
    b.alloc(n ? n : 1);
    if (n) B2S_LAUNCH(ctx, k_amg_to_f32, stream_grid(ctx, n), kThreads, 0, a, b.p, n);
}

struct PcAMG final : PcImpl
{
    int bs = 1;
    bool ref_coarse = false;
    bool fp32 = false;  // V-cycle reads FP32 copies of A, P, R and D^-1 (FP64 arithmetic and vectors)
    int aggregation = 0;  // b2s_pc_opts::amg_aggregation
    std::vector<std::unique_ptr<Level>> lv;
    std::unique_ptr<BaijDev> fine_copy;  // BS=1 copy of a CSR operator
    DBuf<double> dense;
    DBuf<int> piv;
    int sz = 0;

    template <int BS>
    void vcycle(b2s_ctx* ctx, int l, const double* rhs, double* sol, const int* done)
    {
        Level& L = *lv[l];
        const unsigned g = stream_grid(ctx, L.nrows);
        if (l == (int)lv.size() - 1)
        {
            B2S_LAUNCH(ctx, k_dense_solve, 1, kThreads, dense_smem(sz), dense.p, sz, ref_coarse ? 1 : 0, piv.p, rhs, sol, done);
            return;
        }
        // products on FP64 or FP32 values, each with its epilogue
        auto mv = [&](const BaijDev& M, const DBuf<float>& v32, const double* x, auto epi) {
            if (fp32)
                baij_mv<BS>(ctx, M, v32.p, x, epi, done);
            else
                baij_mv<BS>(ctx, M, M.v.p, x, epi, done);
        };
        // pre-smoothing from zero, residual, restriction
        if (fp32)
            B2S_LAUNCH(ctx, (k_smooth0<BS, float>), g, kThreads, 0, L.nrows, L.dinv32.p, rhs, sol, done);
        else
            B2S_LAUNCH(ctx, (k_smooth0<BS, double>), g, kThreads, 0, L.nrows, L.dinv.p, rhs, sol, done);
        mv(*L.A, L.A32, sol, EpiResidual{rhs, L.r.p});
        mv(L.R, L.R32, L.r.p, EpiStoreY{L.rc.p});
        const uint64_t nc = (uint64_t)L.R.nbr * BS;
        if (l + 1 < (int)lv.size() - 1)
            vcycle<BS>(ctx, l + 1, L.rc.p, L.ec.p, done);
        else
        {
            B2S_LAUNCH(ctx, k_zero, stream_grid(ctx, nc), kThreads, 0, nc, L.ec.p, done);
            vcycle<BS>(ctx, l + 1, L.rc.p, L.ec.p, done);
        }
        // coarse-grid correction into tmp, then post-smoothing back into sol
        mv(L.P, L.P32, L.ec.p, EpiAddTo{sol, L.tmp.p});
        if (fp32)
            mv(*L.A, L.A32, L.tmp.p, EpiJacobi<float>{L.dinv32.p, rhs, L.tmp.p, sol});
        else
            mv(*L.A, L.A32, L.tmp.p, EpiJacobi<double>{L.dinv.p, rhs, L.tmp.p, sol});
    }

    void apply(b2s_ctx* ctx, const double* r, double* z, const int* done) override
    {
        switch (bs)
        {
            case 1: vcycle<1>(ctx, 0, r, z, done); break;
            case 2: vcycle<2>(ctx, 0, r, z, done); break;
            case 3: vcycle<3>(ctx, 0, r, z, done); break;
            case 4: vcycle<4>(ctx, 0, r, z, done); break;
        }
    }

    void export_baij(b2s_ctx* ctx, const BaijDev& M, uint64_t* sizes, uint32_t* rp, uint32_t* ci, double* v)
    {
        const size_t bv = (size_t)M.bs * M.bs;
        sizes[0] = (uint64_t)M.nbr + 1;
        sizes[1] = M.nnzb;
        sizes[2] = (uint64_t)M.nnzb * bv;
        if (rp) d2h(ctx, rp, M.rp.p, (M.nbr + 1) * sizeof(uint32_t));
        if (ci) d2h(ctx, ci, M.ci.p, M.nnzb * sizeof(uint32_t));
        if (v) d2h(ctx, v, M.v.p, M.nnzb * bv * sizeof(double));
        sync(ctx);
    }

    void export_data(b2s_ctx* ctx, const std::string& what, uint64_t* sizes, uint32_t* rp, uint32_t* ci,
                     double* v) override
    {
        if (what == "amg.levels")
        {
            sizes[0] = 0;
            sizes[1] = lv.size();
            sizes[2] = 0;
            if (ci)
                for (size_t k = 0; k < lv.size(); ++k) ci[k] = lv[k]->nrows;
            return;
        }
        unsigned l = 0;
        char tail[32] = {0};
        if (std::sscanf(what.c_str(), "amg.%u.%31s", &l, tail) == 2 && l < lv.size())
        {
            Level& L = *lv[l];
            const std::string t(tail);
            if (t == "A") return export_baij(ctx, *L.A, sizes, rp, ci, v);
            if (t == "P" && L.has_p) return export_baij(ctx, L.P, sizes, rp, ci, v);
            if (t == "dinv")
            {
                sizes[0] = 0;
                sizes[1] = 0;
                sizes[2] = (uint64_t)L.nrows * bs * bs;
                if (v) d2h(ctx, v, L.dinv.p, sizes[2] * sizeof(double));
                sync(ctx);
                return;
            }
            if (t == "agg" && L.has_p)
            {
                sizes[0] = 0;
                sizes[1] = L.nrows;
                sizes[2] = 0;
                if (ci) d2h(ctx, ci, L.agg.p, L.nrows * sizeof(uint32_t));
                sync(ctx);
                return;
            }
        }
        PcImpl::export_data(ctx, what, sizes, rp, ci, v);
    }
};

template <int BS>
void build_hierarchy(b2s_ctx* ctx, PcAMG& pc, const BaijDev& A0, int max_levels, uint32_t coarse_max)
{
    constexpr int BV = BS * BS;
    const BaijDev* cur = &A0;
    std::unique_ptr<BaijDev> cur_own;
    for (int lvl = 0; lvl < max_levels; ++lvl)
    {
        auto L = std::make_unique<Level>();
        const uint32_t n = cur->nbr;
        L->nrows = n;
        L->own = std::move(cur_own);
        L->A = cur;
        L->dinv.alloc((size_t)n * BV + 1);
        if (n) B2S_LAUNCH(ctx, k_diag_inv<BS>, stream_grid(ctx, n), kThreads, 0, n, cur->v.p, cur->diag_ptr.p, L->dinv.p);
        if (n <= coarse_max)
        {
            pc.lv.push_back(std::move(L));
            cur = nullptr;
            break;
        }
        // strength
        DBuf<uint32_t> cnt(n + 1), sp(n + 1);
        // lanes a row of the setup kernels that walk rows: a warp where the rows are long
        const bool long_rows = cur->nnzb >= 16ull * n && n <= 65536u;
        const unsigned rows_grid = stream_grid(ctx, long_rows ? 32ull * n : n);
        const auto strength = long_rows ? k_strength<BS, 32> : k_strength<BS, 1>;
        const auto p_count = long_rows ? k_p_count<32> : k_p_count<1>;
        const auto p_fill = long_rows ? k_p_fill<BS, 32> : k_p_fill<BS, 1>;
        B2S_LAUNCH(ctx, strength, rows_grid, kThreads, 0, n, cur->rp.p, cur->ci.p, cur->v.p, (const uint32_t*)nullptr,
                   cnt.p, (uint32_t*)nullptr);
        const uint32_t ns = exclusive_scan(ctx, cnt.p, sp.p, n);
        DBuf<uint32_t> sc(ns ? ns : 1);
        B2S_LAUNCH(ctx, strength, rows_grid, kThreads, 0, n, cur->rp.p, cur->ci.p, cur->v.p, sp.p, (uint32_t*)nullptr,
                   sc.p);
        // aggregation
        L->agg.alloc(n);
        B2S_CUDA(cudaMemsetAsync(L->agg.p, 0xFF, (size_t)n * sizeof(int32_t), ctx->stream));
        uint32_t nagg = 0;
        if (pc.aggregation == 0)
            nagg = aggregate_parallel(ctx, n, sp.p, sc.p, L->agg.p);
        else
        {
            DBuf<uint32_t> nagg_d(1);
            if (pc.aggregation == 1)
                B2S_LAUNCH(ctx, k_aggregate, 1, 32, 0, n, sp.p, sc.p, L->agg.p, nagg_d.p);
            else
            {
                DBuf<int32_t> snap(n);
                B2S_LAUNCH(ctx, k_aggregate_std, 1, 32, 0, n, sp.p, sc.p, L->agg.p, snap.p, nagg_d.p);
                sync(ctx);
            }
            d2h(ctx, &nagg, nagg_d.p, sizeof(uint32_t));
            sync(ctx);
        }
        // smoothed prolongation
        L->P.bs = BS;
        L->P.nbr = n;
        L->P.nbc = nagg;
        B2S_LAUNCH(ctx, p_count, rows_grid, kThreads, 0, n, cur->rp.p, cur->ci.p, L->agg.p, cnt.p);
        L->P.rp.alloc(n + 1);
        const uint32_t pn = exclusive_scan(ctx, cnt.p, L->P.rp.p, n);
        L->P.ci.alloc(pn ? pn : 1);
        L->P.v.alloc(pn ? (size_t)pn * BV : 1);
        B2S_LAUNCH(ctx, p_fill, rows_grid, kThreads, 0, n, cur->rp.p, cur->ci.p, cur->v.p, L->dinv.p,
                   L->agg.p, L->P.rp.p, L->P.ci.p, L->P.v.p);
        finish_baij(ctx, L->P);
        block_transpose<BS>(ctx, L->P, L->R);
        L->has_p = true;
        // Galerkin
        BaijDev AP;
        block_matmul<BS>(ctx, *cur, L->P, AP);
        cur_own = std::make_unique<BaijDev>();
        block_matmul<BS>(ctx, L->R, AP, *cur_own);
        cur = cur_own.get();
        pc.lv.push_back(std::move(L));
    }
    // work vectors
    for (size_t k = 0; k < pc.lv.size(); ++k)
    {
        Level& L = *pc.lv[k];
        const size_t nd = (size_t)L.nrows * BS + 1;
        L.tmp.alloc(nd);
        L.r.alloc(nd);
        if (L.has_p)
        {
            const size_t nc = (size_t)L.R.nbr * BS + 1;
            L.rc.alloc(nc);
            L.ec.alloc(nc);
        }
    }
    // coarsest dense operator (the last level; if max_levels was reached its P is unused)
    Level& C = *pc.lv.back();
    pc.sz = (int)(C.nrows * BS);
    pc.dense.alloc((size_t)pc.sz * pc.sz + 1);
    pc.piv.alloc(pc.sz + 1);
    B2S_CUDA(cudaMemsetAsync(pc.dense.p, 0, pc.dense.bytes(), ctx->stream));
    if (C.nrows)
        B2S_LAUNCH(ctx, k_dense_from_baij<BS>, stream_grid(ctx, C.nrows), kThreads, 0, C.nrows, C.A->rp.p, C.A->ci.p,
                   C.A->v.p, pc.dense.p, pc.sz);
    for (const void* kern : {(const void*)k_dense_factor, (const void*)k_dense_solve})
        B2S_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dense_smem(kDenseSmem)));
    B2S_LAUNCH(ctx, k_dense_factor, 1, kThreads, dense_smem(pc.sz), pc.dense.p, pc.sz, pc.ref_coarse ? 1 : 0, pc.piv.p);
    // FP32 copies of every operator the V-cycle multiplies by (the coarsest level is the dense LU, kept in FP64)
    if (pc.fp32)
        for (size_t k = 0; k + 1 < pc.lv.size(); ++k)
        {
            Level& L = *pc.lv[k];
            amg_to_f32(ctx, L.A->v.p, L.A32, (uint64_t)L.A->nnzb * BV);
            amg_to_f32(ctx, L.P.v.p, L.P32, (uint64_t)L.P.nnzb * BV);
            amg_to_f32(ctx, L.R.v.p, L.R32, (uint64_t)L.R.nnzb * BV);
            amg_to_f32(ctx, L.dinv.p, L.dinv32, (uint64_t)L.nrows * BV);
        }
    sync(ctx);
}

std::unique_ptr<PcImpl> build_amg(b2s_ctx* ctx, const BaijDev& A, const b2s_pc_opts& o,
                                  std::unique_ptr<BaijDev> owned)
{
    need(A.nbr == A.nbc, B2S_SHAPE, "block AMG needs a square block matrix");
    auto pc = std::make_unique<PcAMG>();
    pc->bs = A.bs;
    pc->ref_coarse = o.amg_ref_coarse != 0;
    pc->fp32 = o.precision != B2S_FP64;
    pc->aggregation = o.amg_aggregation;
    pc->fine_copy = std::move(owned);
    const int max_levels = o.amg_max_levels > 0 ? o.amg_max_levels : 20;
    const uint32_t coarse_max = o.amg_coarse_max > 0 ? (uint32_t)o.amg_coarse_max : 50u;
    switch (A.bs)
    {
        case 1: build_hierarchy<1>(ctx, *pc, A, max_levels, coarse_max); break;
        case 2: build_hierarchy<2>(ctx, *pc, A, max_levels, coarse_max); break;
        case 3: build_hierarchy<3>(ctx, *pc, A, max_levels, coarse_max); break;
        case 4: build_hierarchy<4>(ctx, *pc, A, max_levels, coarse_max); break;
        default: fail(B2S_UNSUPPORTED, "block size must be 1..4");
    }
    return pc;
}

}  // namespace

std::unique_ptr<PcImpl> make_pc_amg_baij(b2s_ctx* ctx, const BaijDev& A, const b2s_pc_opts& o)
{
    return build_amg(ctx, A, o, nullptr);
}

// scalar SA-AMG: BlockMatrix<double,1>::condense of the CSR operator, which
// for a block size of 1 is the same pattern and values
std::unique_ptr<PcImpl> make_pc_amg_csr(b2s_ctx* ctx, const CsrDev& A, const b2s_pc_opts& o)
{
    need(A.n == A.m, B2S_SHAPE, "AMG needs a square matrix");
    auto B = std::make_unique<BaijDev>();
    B->bs = 1;
    B->nbr = A.n;
    B->nbc = A.m;
    B->rp.alloc(A.n + 1);
    B->ci.alloc(A.nnz ? A.nnz : 1);
    B->v.alloc(A.nnz ? A.nnz : 1);
    d2d(ctx, B->rp.p, A.rp.p, (A.n + 1) * sizeof(uint32_t));
    d2d(ctx, B->ci.p, A.ci.p, A.nnz * sizeof(uint32_t));
    d2d(ctx, B->v.p, A.v.p, A.nnz * sizeof(double));
    finish_baij(ctx, *B);
    const BaijDev& ref = *B;
    return build_amg(ctx, ref, o, std::move(B));
}

// scalar (bs = 1) product and transpose for general CSR operators: the
// C ABI's b2s_csr_matmul / b2s_csr_transpose (csr.cu)
void scalar_matmul(b2s_ctx* ctx, const BaijDev& A, const BaijDev& B, BaijDev& C) { block_matmul<1>(ctx, A, B, C); }
void scalar_transpose(b2s_ctx* ctx, const BaijDev& A, BaijDev& T) { block_transpose<1>(ctx, A, T); }

}  // namespace b2s
