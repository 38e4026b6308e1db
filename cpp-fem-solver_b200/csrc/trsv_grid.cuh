// Exact triangular solves of 5- and 7-point grid factors (IC(0) / ILU(0) of a
// natural-order stencil on a B x ny x nz grid; nz = 1 for 5 points).
//
// Row i = (z ny + y) B + x of a lower factor depends on (x, y, z - 1),
// (x, y - 1, z) and (x - 1, y, z), in that column order; an upper one on
// (x + 1, y, z), (x, y + 1, z) and (x, y, z + 1).  In solve order (the upper
// factor walked from the far corner) both have the lower shape.  A compute warp
// owns a TY x TZ tile of lines (TY TZ = 32), lane j = jz TY + jy the line
// (jy, jz) of it, and walks them one point per step, lane j at step s on point
// k = s - jy - jz: the line's previous point is in a register and both
// neighbouring lines' values come from the lanes below by a shuffle, computed
// the step before.  Only the tile's far edges cross warps: TZ lines to the next
// tile in y, TY lines to the next in z, every step's values as epoch-tagged
// words ({epoch, 32 value bits}, single-copy atomic) in rows of the producer's
// steps, which the consumer reads TY - 1 (TZ - 1) rows ahead of its own step.
//
// Bound by latency: B + ny + nz steps plus about 10 for each of the
// nty + ntz - 2 tile hand-overs on the critical path, so what counts is the
// length of a step and the lag of a hand-over.  Everything but the recurrence is
// therefore moved off the compute warp: a stager warp copies the packed
// coefficients of a group of steps with one bulk copy and the right-hand side
// with cp.async into a ring, and writes the finished groups back; poller warps
// read the neighbouring tiles' words until they carry the epoch and leave the
// values in the same ring.  The compute warp meets them at one mbarrier a group,
// reads shared memory, and stores only the words its neighbours wait for.
// 128^3 ILU(0) apply FP64 / FP32 268 / 197 us (one warp doing all of it, in tiles:
// 323 / 247; a plane at a time: 978 / 740), 512^2 238 / 156 (one warp a 32-line
// block, no tiles: 368 / 307).
//
// Warps take tickets in the order of their tiles' start times, so each waits
// only on warps that started before it.  Every wait is bounded: a poller that
// gives up (B2S_TIMEOUT) hands over what it read and goes on without waiting.
//
// The arithmetic is the reference's (column order; FP32 multiplies by the
// reciprocal rounded once from FP64; FP64 forms the correctly rounded
// quotient from the correctly rounded reciprocal, grid_quotient, and redoes a
// group with the division where that is not exact), so the results equal the
// other schedules bit for bit.  The coefficients are packed at set-up in
// consumption order: slot (w, s, j) = {c_z, c_y, c_x[, divisor[, 1 / d]]} (16
// bytes FP32, 48 bytes FP64, 32 with a unit diagonal), padded off the grid with
// zero coefficients and unit divisors.
#pragma once
#include "trsv_chunk.cuh"

namespace b2s {

constexpr uint32_t kGrid5MaxLines = 4096;      // 5-point grids with more lines keep the other schedules
constexpr uint32_t kGrid7MaxWarps = 1u << 16;  // 7-point: ny / 32 * nz
// Steps of a group, groups in the ring, and poller warps, for 5- (Z3 false) and
// 7-point grids.  A group costs the compute warp about 300 cycles besides its
// steps (the barrier, the reads, the end of the recurrence), but a hand-over
// waits for a whole one: 5-point grids cross few and take 8, 7-point grids many
// and take 4 (ILU(0) apply FP64 / FP32, 4 against 8: 512^2 253 / 186 and 238 / 156
// us, 16 261 / 169; 128^3 287 / 217 and 334 / 232).  A poller asks for one group a trip
// through L2 (~450 ns) and takes every P-th group; one poller would set the pace
// (512^2 FP32: 1: 265, 2: 186, 3: 188; 128^3 FP64: 1: 288, 2: 287, 4: 268).
constexpr int grid_group(bool z3) { return z3 ? 4 : 8; }
constexpr uint32_t grid_stages(bool z3) { return z3 ? 8u : 4u; }
constexpr uint32_t grid_pollers(bool z3) { return z3 ? 4u : 2u; }
constexpr uint32_t grid_threads(bool z3) { return 64u + 32u * grid_pollers(z3); }  // compute, stager, pollers
constexpr uint32_t kGridHandover = 10;  // steps a tile hand-over adds (the shape's cost model)
// two CTAs an SM: one leaves large grids short of warps (200^3 FP64 679 us
// against 513) and is no faster elsewhere (64^3, 512^2 the same)
constexpr uint32_t kGridSmem = 100u << 10;
constexpr uint32_t kGridMbarPolls = 1u << 27;  // the other warps of a CTA always make progress: a backstop

// The tiling of a B x ny x nz grid's lines.
struct GridTiles
{
    uint32_t B = 0, ny = 0, nz = 0;
    uint32_t ly = 0;            // TY = 1 << ly, TZ = 32 >> ly
    uint32_t nty = 0, ntz = 0;  // tiles in y and z
    __host__ __device__ uint32_t ty() const { return 1u << ly; }
    __host__ __device__ uint32_t tz() const { return 32u >> ly; }
    __host__ __device__ uint32_t tiles() const { return nty * ntz; }
    // B + TY + TZ - 2 steps a tile, rounded up to whole groups: its packed slots and exchange rows
    __host__ __device__ uint32_t rows() const
    {
        const uint32_t g = (uint32_t)grid_group(nz > 1);
        return (B + ty() + tz() - 2u + g - 1u) / g * g;
    }
};

// The shape with the shortest estimated time: the critical path (padded lines
// and hand-overs) or the tiles' steps dealt over the SMs, whichever is longer;
// on a tie the fewer tiles.
inline GridTiles grid_tiles(uint32_t B, uint32_t ny, uint32_t nz, uint32_t sm_count)
{
    GridTiles best;
    uint64_t cost = ~0ull;
    for (uint32_t ly = 0; ly <= 5; ++ly)
    {
        GridTiles s{B, ny, nz, ly};
        s.nty = (ny + s.ty() - 1) / s.ty();
        s.ntz = (nz + s.tz() - 1) / s.tz();
        const uint64_t path = (uint64_t)B + s.nty * s.ty() + s.ntz * s.tz() + kGridHandover * (s.nty + s.ntz - 2);
        const uint64_t work = (uint64_t)s.tiles() * s.rows() / sm_count;
        const uint64_t c = (std::max(path, work) << 24) + std::min(s.tiles(), (1u << 24) - 1);
        if (c < cost)
        {
            cost = c;
            best = s;
        }
    }
    return best;
}

template <typename VT, bool UNIT>
struct GridSlot;
template <bool UNIT>
struct alignas(16) GridSlot<float, UNIT>
{
    float cz, cy, cx, dv;
};
template <>
struct alignas(16) GridSlot<double, true>
{
    double cz, cy, cx, pad;
};
template <>
struct alignas(16) GridSlot<double, false>
{
    double cz, cy, cx, dv, rc, pad;
};

// sum / d rounded to nearest from the correctly rounded reciprocal y = 1 / d:
// q0 = sum * y is within 1.5 ulp of the quotient; one correction
// q1 = q0 + (sum - d q0) y (residual by FMA) is faithful, and a second
// correction from the exact residual of q1 is the correctly rounded quotient
// (P. Markstein, IBM J. Res. Develop. 34(1), 1990: a quotient within one ulp
// and a reciprocal within half an ulp give the correctly rounded result after
// one such step).  A zero dividend gives q0, whose sign is the quotient's.
// `bad` is set where a residual could underflow or a product overflow; the
// caller then divides instead.
__device__ __forceinline__ double grid_quotient(double sum, double d, double y, bool active, bool& bad)
{
    const double q0 = sum * y;
    const double q1 = fma(fma(-q0, d, sum), y, q0);
    const double q = fma(fma(-q1, d, sum), y, q1);
    const double as = fabs(sum), aq = fabs(q0);
    const bool zero = sum == 0.0;
    bad |= active && !(zero || (as >= 0x1p-900 && as <= 0x1p+900 && aq >= 0x1p-900 && aq <= 0x1p+900));
    return zero ? q0 : q;
}

__device__ __forceinline__ void grid_st_if(bool p, unsigned long long* a, unsigned long long v)
{
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.relaxed.gpu.global.u64 [%0], %1;\n\t}" ::"l"(a), "l"(v),
        "r"((unsigned)p));
}
__device__ __forceinline__ void grid_stx_if(bool p, float* a, float v)
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.global.f32 [%0], %1;\n\t}" ::"l"(a), "f"(v),
                 "r"((unsigned)p));
}
__device__ __forceinline__ void grid_stx_if(bool p, double* a, double v)
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.global.f64 [%0], %1;\n\t}" ::"l"(a), "d"(v),
                 "r"((unsigned)p));
}
__device__ __forceinline__ void grid_st2_if(bool q, unsigned long long* p, unsigned long long a, unsigned long long b)
{
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\t@q st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};\n\t}" ::"l"(p),
        "l"(a), "l"(b), "r"((unsigned)q));
}
// one exchange value's words; `none` in each where q is false
__device__ __forceinline__ void grid_ld_if(bool q, const unsigned long long* p, unsigned long long none,
                                         unsigned long long (&w)[1])
{
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.u64 %0, %3;\n\t@q ld.relaxed.gpu.global.u64 %0, [%1];\n\t}"
        : "=&l"(w[0])
        : "l"(p), "r"((unsigned)q), "l"(none));
}
__device__ __forceinline__ void grid_ld_if(bool q, const unsigned long long* p, unsigned long long none,
                                         unsigned long long (&w)[2])
{
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\tmov.u64 %0, %4;\n\tmov.u64 %1, %4;\n\t"
        "@q ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];\n\t}"
        : "=&l"(w[0]), "=&l"(w[1])
        : "l"(p), "r"((unsigned)q), "l"(none));
}
// BYTES (4 or 8) of src, zero-filled where src_bytes is 0
template <int BYTES>
__device__ __forceinline__ void grid_cp_small(uint32_t dst, const void* src, uint32_t src_bytes)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(BYTES), "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void grid_mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void grid_mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void grid_mbar_expect(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// one arrival when this thread's earlier cp.async copies have landed
__device__ __forceinline__ void grid_mbar_cp_arrive(uint32_t bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool grid_mbar_wait(uint32_t bar, uint32_t parity)
{
    for (uint32_t i = 0; i < kGridMbarPolls; ++i)
    {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
// global -> shared, completion counted in bytes on `bar`
__device__ __forceinline__ void grid_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

template <typename VT, bool UNIT>
__global__ void __launch_bounds__(kThreads) k_grid_pack(GridTiles sh, bool lower, const uint32_t* __restrict__ rp,
                                                        const uint32_t* __restrict__ ci, const VT* __restrict__ v,
                                                        const VT* __restrict__ d, GridSlot<VT, UNIT>* __restrict__ slot)
{
    const uint32_t B = sh.B, P = B * sh.ny, n = P * sh.nz, TY = sh.ty(), rows = sh.rows();
    const size_t total = (size_t)sh.tiles() * rows * 32u;
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (size_t)gridDim.x * blockDim.x)
    {
        const uint32_t j = (uint32_t)(q % 32u), jy = j & (TY - 1u), jz = j >> sh.ly;
        const size_t ws = q / 32u;
        const uint32_t s = (uint32_t)(ws % rows), w = (uint32_t)(ws / rows);
        // solve order; k wraps before the line
        const uint32_t y = w % sh.nty * TY + jy, z = w / sh.nty * sh.tz() + jz, k = s - jy - jz;
        GridSlot<VT, UNIT> c{};
        if constexpr (!UNIT) c.dv = VT(1);
        if constexpr (!UNIT && sizeof(VT) == 8) c.rc = 1.0;
        if (y < sh.ny && z < sh.nz && k < B)
        {
            const uint32_t ii = (z * sh.ny + y) * B + k, i = lower ? ii : n - 1u - ii;
            for (uint32_t e = rp[i]; e < rp[i + 1]; ++e)
            {
                const uint32_t j2 = ci[e];
                if (sh.nz > 1 && (lower ? j2 + P == i : j2 == i + P)) c.cz = v[e];
                if (lower ? j2 + B == i : j2 == i + B) c.cy = v[e];
                if (lower ? j2 + 1 == i : j2 == i + 1) c.cx = v[e];
            }
            if constexpr (!UNIT)
            {
                if constexpr (sizeof(VT) == 4)
                    c.dv = (VT)(1.0 / (double)d[i]);
                else
                {
                    c.dv = d[i];
                    c.rc = 1.0 / d[i];
                }
            }
        }
        slot[q] = c;
    }
}

// One ring stage: a group's operands, its neighbour values and its results.
template <bool UNIT, bool Z3, typename VT, typename XT, typename RT>
struct GridStage
{
    GridSlot<VT, UNIT> c[grid_group(Z3)][32];
    XT nb[grid_group(Z3)][32], res[grid_group(Z3)][32], zb[Z3 ? grid_group(Z3) : 1][32];
    RT rhs[grid_group(Z3)][32];
};

// ctl: [0] epoch, [1] exit count, [2] ticket (the last CTA to leave resets
// [1], [2] and advances [0], so the launch can be replayed).  order: ticket ->
// tile.  words: each tile's exchange rows, one a step: TZ values of its last
// lines in y, then TY of its last lines in z (one word per FP32 value, two per
// FP64 one).  Z3: the grid has planes (7 points).
template <bool LOWER, bool UNIT, bool Z3, typename VT, typename XT, typename RT>
__global__ void __launch_bounds__(grid_threads(Z3), 2) k_trsv_grid(GridTiles sh, const uint32_t* __restrict__ order,
                                                            const GridSlot<VT, UNIT>* __restrict__ slot,
                                                            const RT* __restrict__ rhs, XT* __restrict__ x,
                                                            double* __restrict__ out64, const int* done,
                                                            unsigned long long* words, uint32_t* ctl, int* err,
                                                            unsigned polls_max)
{
    if (done && *done) return;
    using Slot = GridSlot<VT, UNIT>;
    using Stage = GridStage<UNIT, Z3, VT, XT, RT>;
    constexpr int G = grid_group(Z3);
    constexpr uint32_t NS = grid_stages(Z3), NP = grid_pollers(Z3);
    constexpr int WPV = sizeof(XT) == 8 ? 2 : 1;  // exchange words per value
    constexpr bool MARK = sizeof(XT) == 8 && !UNIT;
    extern __shared__ __align__(128) unsigned char grid_sm[];
    Stage* const ring = reinterpret_cast<Stage*>(grid_sm);
    __shared__ uint32_t s_tile;
    __shared__ __align__(8) unsigned long long s_full[NS], s_done[NS];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0)
    {
        s_tile = __ldg(&order[atomicAdd(&ctl[2], 1u)]);
        for (uint32_t s = 0; s < NS; ++s)
        {
            grid_mbar_init(smem_u32(&s_full[s]), 34u);  // the stager's 32 copies and its bulk copy, the poller
            grid_mbar_init(smem_u32(&s_done[s]), 1u);   // the compute warp
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const uint32_t w = s_tile, epoch = ld_flag(&ctl[0]) + 1u;
    const uint32_t B = sh.B, ny = sh.ny, TY = sh.ty(), TZ = sh.tz(), groups = sh.rows() / G;
    const uint32_t ty = w % sh.nty, tz = w / sh.nty, jy = lane & (TY - 1u), jz = lane >> sh.ly;
    const uint32_t y = ty * TY + jy, z = tz * TZ + jz, L = z * ny + y;  // this lane's line in solve order
    const uint32_t n = B * ny * sh.nz;
    const uint32_t k0 = y < ny && z < sh.nz ? 0u - jy - jz : B;  // point of step 0 (wraps before the line)
    const bool edge_y = jy == 0u, edge_z = jz == 0u;             // neighbours in another tile (or off the grid)
    const uint32_t RW = (TY + TZ) * WPV;                         // words of an exchange row
    const size_t tile_words = (size_t)sh.rows() * RW;
    const unsigned long long etag = (unsigned long long)epoch << 32;
    auto bar = [](unsigned long long* b, uint32_t g) { return smem_u32(&b[g % NS]); };
    bool ok = true;

    if (warp >= 2)
    {
        // ---- poller: the neighbouring tiles' values of each group; a lane that
        // needs none, and a step off its line, gets a zero
        const bool rd_y = edge_y && ty > 0u, rd_z = Z3 && edge_z && tz > 0u;
        const unsigned long long* iy =
            words + (ty > 0u ? w - 1u : w) * tile_words + (size_t)(TY - 1u) * RW + jz * WPV;
        const unsigned long long* iz =
            words + (tz > 0u ? w - sh.nty : w) * tile_words + (size_t)(TZ - 1u) * RW + (TZ + jy) * WPV;
        bool gave_up = false;
        auto ask = [&](uint32_t g, unsigned long long (&yw)[G][WPV], unsigned long long (&zw)[G][WPV]) {
#pragma unroll
            for (int u = 0; u < G; ++u)
            {
                const bool on = k0 + g * G + (uint32_t)u < B;
                grid_ld_if(rd_y && on, iy + (size_t)(g * G + u) * RW, etag, yw[u]);
                if constexpr (Z3) grid_ld_if(rd_z && on, iz + (size_t)(g * G + u) * RW, etag, zw[u]);
            }
        };
        for (uint32_t g = warp - 2u; g < groups && ok; g += NP)
        {
            if (g >= NS) ok = grid_mbar_wait(bar(s_done, g), (g / NS - 1u) & 1u);
            unsigned long long yw[G][WPV], zw[G][WPV];
            for (unsigned polls = 0;; ++polls)
            {
                bool fresh = true;
                ask(g, yw, zw);
#pragma unroll
                for (int u = 0; u < G; ++u)
#pragma unroll
                    for (int c = 0; c < WPV; ++c)
                    {
                        fresh &= (uint32_t)(yw[u][c] >> 32) == epoch;
                        if constexpr (Z3) fresh &= (uint32_t)(zw[u][c] >> 32) == epoch;
                    }
                if (gave_up || __all_sync(0xffffffffu, fresh)) break;
                if (__any_sync(0xffffffffu, polls + 1u >= polls_max || ((polls & 63u) == 63u && ld_err(err) != 0)))
                {
                    if (lane == 0) atomicCAS(err, 0, (int)B2S_TIMEOUT);
                    gave_up = true;
                }
            }
            auto value = [](const unsigned long long (&wd)[WPV]) -> XT {
                if constexpr (WPV == 1)
                    return (XT)__uint_as_float((uint32_t)wd[0]);
                else
                    return (XT)__longlong_as_double((long long)((wd[WPV - 1] << 32) | (wd[0] & 0xffffffffull)));
            };
            Stage& S = ring[g % NS];
#pragma unroll
            for (int u = 0; u < G; ++u)
            {
                S.nb[u][lane] = value(yw[u]);
                if constexpr (Z3) S.zb[u][lane] = value(zw[u]);
            }
            __syncwarp();
            if (lane == 0) grid_mbar_arrive(bar(s_full, g));
        }
    }
    else if (warp == 1)
    {
        // ---- stager: writes group i - NS back, then refills its stage with group i
        double* const o64 = out64 ? out64 : reinterpret_cast<double*>(x);
        const bool w64 = out64 != nullptr;
        for (uint32_t i = 0; i < groups + NS && ok; ++i)
        {
            Stage& S = ring[i % NS];
            if (i >= NS && i - NS < groups)
            {
                ok = grid_mbar_wait(bar(s_done, i), (i / NS - 1u) & 1u);
                // runs of G consecutive points of 32 / G lines at a time
#pragma unroll
                for (uint32_t pass = 0; pass < (uint32_t)G; ++pass)
                {
                    const uint32_t l = pass * (32u / G) + lane / G, u = lane % G;
                    const uint32_t ly = l & (TY - 1u), lz = l >> sh.ly, yl = ty * TY + ly, zl = tz * TZ + lz;
                    const uint32_t k = (i - NS) * G + u - ly - lz;
                    const bool p = ok && yl < ny && zl < sh.nz && k < B;
                    const uint32_t q = (zl * ny + yl) * B + k, row = LOWER ? q : n - 1u - q;
                    const XT r = S.res[u][l];
                    grid_stx_if(p && !w64, x + row, r);  // given out64, the FP64 copy is the result and x is not written
                    grid_stx_if(p && w64, o64 + row, (double)r);
                }
                __syncwarp();
            }
            if (i < groups && ok)
            {
                const uint32_t b = bar(s_full, i);
                if (lane == 0)
                {
                    grid_mbar_expect(b, (uint32_t)sizeof(S.c));
                    grid_bulk(smem_u32(S.c), slot + ((size_t)w * groups + i) * (G * 32u), (uint32_t)sizeof(S.c), b);
                }
#pragma unroll
                for (uint32_t u = 0; u < (uint32_t)G; ++u)
                {
                    const uint32_t k = k0 + i * G + u, q = L * B + k;
                    const bool on = k < B;
                    grid_cp_small<sizeof(RT)>(smem_u32(&S.rhs[u][lane]), on ? &rhs[LOWER ? q : n - 1u - q] : rhs,
                                            on ? (uint32_t)sizeof(RT) : 0u);
                }
                grid_mbar_cp_arrive(b);
            }
        }
    }
    else
    {
        // ---- compute
        const bool pub_y = jy == TY - 1u && ty + 1u < sh.nty, pub_z = Z3 && jz == TZ - 1u && tz + 1u < sh.ntz;
        unsigned long long* oy = words + w * tile_words + jz * WPV;
        unsigned long long* oz = words + w * tile_words + (TZ + jy) * WPV;
        // the row's entries in column order: lower (z-1), (y-1), (x-1); upper
        // (x+1), (y+1), (z+1); absent ones have +0 coefficients and +0 values
        auto row_sum = [&](RT r, const Slot& c, XT zb, XT nb, XT pv) -> XT {
            XT sum = (XT)r;
            if constexpr (LOWER)
            {
                if constexpr (Z3) sum -= (XT)c.cz * zb;
                sum -= (XT)c.cy * nb;
                sum -= (XT)c.cx * pv;
            }
            else
            {
                sum -= (XT)c.cx * pv;
                sum -= (XT)c.cy * nb;
                if constexpr (Z3) sum -= (XT)c.cz * zb;
            }
            return sum;
        };
        // a step's value to the next tiles
        auto publish = [&](bool on, int u, XT r) {
            const size_t o = (size_t)u * RW;
            if constexpr (WPV == 1)
            {
                const unsigned long long b = etag | __float_as_uint((float)r);
                grid_st_if(on && pub_y, oy + o, b);
                if constexpr (Z3) grid_st_if(on && pub_z, oz + o, b);
            }
            else
            {
                const unsigned long long bits = (unsigned long long)__double_as_longlong((double)r);
                const unsigned long long lo = etag | (bits & 0xffffffffull), hi = etag | (bits >> 32);
                grid_st2_if(on && pub_y, oy + o, lo, hi);
                if constexpr (Z3) grid_st2_if(on && pub_z, oz + o, lo, hi);
            }
        };
        XT prev = XT(0);
        for (uint32_t g = 0; g < groups; ++g)
        {
            Stage& S = ring[g % NS];
            ok = grid_mbar_wait(bar(s_full, g), (g / NS) & 1u);
            if (!ok) break;
            const uint32_t kg = k0 + g * G;
            Slot c[G];
            RT rr[G];
            XT nbv[G], zbv[G];
#pragma unroll
            for (int u = 0; u < G; ++u)
            {
                c[u] = S.c[u][lane];
                rr[u] = S.rhs[u][lane];
                nbv[u] = S.nb[u][lane];
                zbv[u] = Z3 ? S.zb[u][lane] : XT(0);
            }
            const XT prev0 = prev;
            bool bad = false;
#pragma unroll
            for (int u = 0; u < G; ++u)
            {
                const bool active = kg + (uint32_t)u < B;
                XT nb = __shfl_up_sync(0xffffffffu, prev, 1), zb = XT(0);
                if (edge_y) nb = nbv[u];
                if constexpr (Z3)
                {
                    zb = __shfl_up_sync(0xffffffffu, prev, TY);
                    if (edge_z) zb = zbv[u];
                }
                const XT sum = row_sum(rr[u], c[u], zb, nb, prev);
                XT r;
                if constexpr (UNIT)
                    r = sum;
                else if constexpr (sizeof(XT) == 4)
                    r = sum * (XT)c[u].dv;
                else
                    r = grid_quotient(sum, c[u].dv, c[u].rc, active, bad);
                prev = active ? r : prev;
                S.res[u][lane] = r;
                // with the FP64 quotient only while no lane of the group has needed the
                // division yet (a redo keeps the earlier steps' values: both roundings
                // are correct), the rest after the group
                bool on = true;
                if constexpr (MARK) on = !__any_sync(0xffffffffu, bad);
                publish(on, u, r);
            }
            if constexpr (MARK)
            {
                if (__any_sync(0xffffffffu, bad))
                {
                    prev = prev0;
#pragma unroll 1
                    for (int u = 0; u < G; ++u)
                    {
                        const bool active = kg + (uint32_t)u < B;
                        XT nb = __shfl_up_sync(0xffffffffu, prev, 1), zb = XT(0);
                        if (edge_y) nb = S.nb[u][lane];
                        if constexpr (Z3)
                        {
                            zb = __shfl_up_sync(0xffffffffu, prev, TY);
                            if (edge_z) zb = S.zb[u][lane];
                        }
                        const Slot cu = S.c[u][lane];
                        const XT r = row_sum(S.rhs[u][lane], cu, zb, nb, prev) / cu.dv;
                        prev = active ? r : prev;
                        S.res[u][lane] = r;
                        publish(true, u, r);  // steps already handed over get the same value again
                    }
                }
            }
            oy += (size_t)G * RW;
            oz += (size_t)G * RW;
            __syncwarp();
            if (lane == 0) grid_mbar_arrive(bar(s_done, g));
        }
    }
    if (!ok && lane == 0) atomicCAS(err, 0, (int)B2S_TIMEOUT);
    __syncthreads();
    if (threadIdx.x == 0)
    {
        __threadfence();
        if (atomicAdd(&ctl[1], 1u) == gridDim.x - 1u)
        {
            ctl[1] = 0u;
            ctl[2] = 0u;
            ctl[0] = epoch;
            __threadfence();
        }
    }
}

// One triangle's grid schedule: packed slots, the exchange words and the launch.
struct GridTri
{
    bool on = false;
    GridTiles sh;
    DBuf<uint4> slots;
    const void* packed_v = nullptr;
    uint32_t packed_vs = 0;
    DBuf<unsigned long long> words;
    DBuf<uint32_t> ctl, order;

    static bool fits5(uint32_t b, uint32_t lines) { return b && lines && lines <= kGrid5MaxLines; }
    static bool fits7(uint32_t b, uint32_t y, uint32_t z)
    {
        return b >= 2 && y >= 2 && z >= 2 && (uint64_t)(y + 31) / 32 * z <= kGrid7MaxWarps;
    }
    // a grid that fits5 (z = 1) or fits7
    void enable(b2s_ctx* ctx, uint32_t b, uint32_t y, uint32_t z)
    {
        on = true;
        sh = grid_tiles(b, y, z, (uint32_t)ctx->sm_count);
    }
    template <typename VT, typename XT>
    bool usable() const
    {
        return on && packed_v && packed_vs == sizeof(VT) && ctl.p;
    }
    template <typename VT, bool UNIT>
    void pack_t(b2s_ctx* ctx, const uint32_t* rp, const uint32_t* ci, const VT* v, const VT* d, bool lower)
    {
        using Slot = GridSlot<VT, UNIT>;
        const size_t count = (size_t)sh.tiles() * sh.rows() * 32, units = count * sizeof(Slot) / 16;
        if (slots.n < units) slots.alloc(units);
        B2S_LAUNCH(ctx, (k_grid_pack<VT, UNIT>), stream_grid(ctx, count), kThreads, 0, sh, lower, rp, ci, v, d,
                   reinterpret_cast<Slot*>(slots.p));
    }
    template <typename VT>
    void pack(b2s_ctx* ctx, const uint32_t* rp, const uint32_t* ci, const VT* v, const VT* d, bool lower, bool unit)
    {
        if (!on) return;
        if (!ctl.p)
        {
            words.alloc((size_t)sh.tiles() * sh.rows() * (sh.ty() + sh.tz()) * 2);
            ctl.alloc(3);
            B2S_CUDA(cudaMemsetAsync(words.p, 0, words.bytes(), ctx->stream));
            B2S_CUDA(cudaMemsetAsync(ctl.p, 0, ctl.bytes(), ctx->stream));
            // tiles by start time, which puts every tile after the two it waits on
            std::vector<uint32_t> h(sh.tiles());
            for (uint32_t t = 0; t < sh.tiles(); ++t) h[t] = t;
            const uint32_t cy = sh.ty() + kGridHandover, cz = sh.tz() + kGridHandover;
            std::stable_sort(h.begin(), h.end(), [&](uint32_t a, uint32_t b) {
                return a % sh.nty * cy + a / sh.nty * cz < b % sh.nty * cy + b / sh.nty * cz;
            });
            order = upload(ctx, h);
        }
        if (unit)
            pack_t<VT, true>(ctx, rp, ci, v, d, lower);
        else
            pack_t<VT, false>(ctx, rp, ci, v, d, lower);
        packed_v = v;
        packed_vs = sizeof(VT);
    }
    template <bool LOWER, bool UNIT, typename VT, typename XT, typename RT>
    void run(b2s_ctx* ctx, const RT* rhs, XT* x, double* out64, const int* done)
    {
        if (sh.nz > 1)
            go<LOWER, UNIT, true, VT>(ctx, rhs, x, out64, done);
        else
            go<LOWER, UNIT, false, VT>(ctx, rhs, x, out64, done);
    }
    template <bool LOWER, bool UNIT, bool Z3, typename VT, typename XT, typename RT>
    void go(b2s_ctx* ctx, const RT* rhs, XT* x, double* out64, const int* done)
    {
        static_assert(grid_stages(Z3) * sizeof(GridStage<UNIT, Z3, VT, XT, RT>) <= kGridSmem, "the ring fits");
        auto kern = k_trsv_grid<LOWER, UNIT, Z3, VT, XT, RT>;
        B2S_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGridSmem));
        B2S_LAUNCH(ctx, kern, sh.tiles(), grid_threads(Z3), kGridSmem, sh, order.p,
                   reinterpret_cast<const GridSlot<VT, UNIT>*>(slots.p), rhs, x, out64, done, words.p, ctl.p,
                   ctx->errword(), grid_polls(ctx));
    }
};

// Host checks of the patterns: a lower triangle whose strict entries are
// {i - B if y > 0, i - 1 if x > 0} (column order), and an upper one whose are
// {i + 1 if x + 1 < B, i + B if y + 1 < ny}; the diagonal may be stored anywhere.
inline bool grid5_triangle(uint32_t n, const uint32_t* rp, const uint32_t* ci, uint32_t B, bool lower)
{
    if (!B || n % B) return false;
    const uint32_t ny = n / B;
    for (uint32_t i = 0; i < n; ++i)
    {
        const uint32_t x = i % B, y = i / B;
        uint32_t want[2], nw = 0;
        if (lower)
        {
            if (y > 0) want[nw++] = i - B;
            if (x > 0) want[nw++] = i - 1;
        }
        else
        {
            if (x + 1 < B) want[nw++] = i + 1;
            if (y + 1 < ny) want[nw++] = i + B;
        }
        uint32_t got = 0;
        for (uint32_t e = rp[i]; e < rp[i + 1]; ++e)
        {
            const uint32_t j = ci[e];
            if (j == i) continue;
            if (got >= nw || j != want[got]) return false;
            ++got;
        }
        if (got != nw) return false;
    }
    return true;
}

// Host checks: the dimensions of a lower triangle that is a natural-order
// 7-point grid's (B >= 2, ny >= 2, nz >= 2; strict entries {i - B ny if
// z > 0, i - B if y > 0, i - 1 if x > 0} in column order), and the same test
// for either triangle at given dimensions (the diagonal may be stored anywhere).
inline bool grid7_triangle(uint32_t n, const uint32_t* rp, const uint32_t* ci, uint32_t B, uint32_t ny, bool lower)
{
    if (B < 2 || ny < 2 || n % (B * ny) || n / (B * ny) < 2) return false;
    const uint32_t P = B * ny, nz = n / P;
    for (uint32_t i = 0; i < n; ++i)
    {
        const uint32_t x = i % B, y = (i / B) % ny, z = i / P;
        uint32_t want[3], nwant = 0;
        if (lower)
        {
            if (z > 0) want[nwant++] = i - P;
            if (y > 0) want[nwant++] = i - B;
            if (x > 0) want[nwant++] = i - 1;
        }
        else
        {
            if (x + 1 < B) want[nwant++] = i + 1;
            if (y + 1 < ny) want[nwant++] = i + B;
            if (z + 1 < nz) want[nwant++] = i + P;
        }
        uint32_t got = 0;
        for (uint32_t e = rp[i]; e < rp[i + 1]; ++e)
        {
            const uint32_t j = ci[e];
            if (j == i) continue;
            if (got >= nwant || j != want[got]) return false;
            ++got;
        }
        if (got != nwant) return false;
    }
    return true;
}

// {B, ny, nz} of a lower triangle with the 7-point grid pattern, else zeros:
// B is the first row with an entry farther than one column back, B ny the
// first with an entry farther than B back.
inline void grid7_dims(uint32_t n, const uint32_t* rp, const uint32_t* ci, uint32_t* dims)
{
    dims[0] = dims[1] = dims[2] = 0;
    uint32_t B = 0, P = 0;
    for (uint32_t i = 0; i < n && !P; ++i)
        for (uint32_t e = rp[i]; e < rp[i + 1]; ++e)
        {
            const uint32_t j = ci[e];
            if (j >= i) continue;
            if (!B && i - j > 1) B = i - j;
            else if (B && i - j > B) P = i - j;
        }
    if (!B || !P || P % B || n % P) return;
    if (!grid7_triangle(n, rp, ci, B, P / B, true)) return;
    dims[0] = B;
    dims[1] = P / B;
    dims[2] = n / P;
}

}  // namespace b2s
