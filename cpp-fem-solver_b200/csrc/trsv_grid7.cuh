// Exact triangular solves of 7-point grid factors (IC(0) / ILU(0) of a
// natural-order 7-point stencil on a B x ny x nz grid), the 3-D form of the
// 5-point grid schedule in trsv_grid5.cuh.
//
// Row i = (z ny + y) B + x of a lower factor depends on (x, y, z - 1),
// (x, y - 1, z) and (x - 1, y, z), in that column order; an upper one on
// (x + 1, y, z), (x, y + 1, z) and (x, y, z + 1).  In solve order (the upper
// factor walked from the far corner) both have the lower shape.  A warp owns a
// TY x TZ tile of lines (TY TZ = 32), lane j = jz TY + jy the line (jy, jz) of
// it, and walks them one point per step, lane j at step s on point
// k = s - jy - jz: the line's previous point is in a register and both
// neighbouring lines' values come from the lanes below by a shuffle, computed
// the step before.  Only the tile's far edges cross warps: TZ lines to the next
// tile in y, TY lines to the next in z, every step's values as epoch-tagged
// words in rows of the producer's steps, which the consumer reads TY - 1 (TZ - 1)
// rows ahead of its own step, a group of kGrid7Group steps at a time, one group
// ahead, and checks with warp-uniform branches.
//
// Bound by latency: the critical path is B + ny + nz steps plus about 10 for
// each of the nty + ntz - 2 tile hand-overs on it (two groups and a trip through
// L2).  A plane at a time (TZ = 1) that was nz + ny / 32 hand-overs, 130 on
// 128^3; the squarest tile has 46, and a step stores 12 words where it stored
// one a lane.  128^3 ILU(0) apply FP64 / FP32 978 / 740 -> 323 / 247 us.
//
// Warps take tickets in the order of their tiles' start times, so each waits
// only on warps that started before it.
//
// The arithmetic is the reference's (column order; FP32 multiplies by the
// reciprocal rounded once from FP64; FP64 forms the correctly rounded
// quotient from the correctly rounded reciprocal, g5_quotient, and redoes a
// group with the division where that is not exact), so the results equal the
// other schedules bit for bit.  The coefficients are packed at set-up in
// consumption order: slot (w, s, j) = {c_z, c_y, c_x[, divisor[, 1 / d]]} (16
// bytes FP32, 48 bytes FP64, 32 with a unit diagonal), padded off the grid with
// zero coefficients and unit divisors.
#pragma once
#include "trsv_grid5.cuh"

namespace b2s {

constexpr uint32_t kGrid7MaxWarps = 1u << 16;  // ny / 32 * nz
constexpr uint32_t kGrid7Ring = 16;            // steps of operands in flight (shared-memory ring); 32: the same
// Steps between a warp's checks.  ILU(0) apply, FP64 / FP32, 128^3 and 64^3 (us):
// 2: 388 / 341 and 122 / 98; 4: 342 / 262 and 147 / 104; 8: 516 / 339 and 238 / 157
// (a plane at a time with 8: 978 / 740 on 128^3).
constexpr int kGrid7Group = 4;
constexpr uint32_t kGrid7Handover = 10;        // steps a tile hand-over adds (the shape's cost model)
// two warps an SM: one leaves the SMs short of warps on large grids (200^3 FP64
// 863 us, two 581, four 627; 128^3 338, 323, 344; 64^3 the same)
constexpr uint32_t kGrid7Smem = 100u << 10;

// The tiling of a B x ny x nz grid's lines.
struct Grid7Shape
{
    uint32_t B = 0, ny = 0, nz = 0;
    uint32_t ly = 0;            // TY = 1 << ly, TZ = 32 >> ly
    uint32_t nty = 0, ntz = 0;  // tiles in y and z
    uint32_t SP = 0;            // packed steps per warp: whole groups, plus the ring's copies ahead
    __host__ __device__ uint32_t ty() const { return 1u << ly; }
    __host__ __device__ uint32_t tz() const { return 32u >> ly; }
    __host__ __device__ uint32_t tiles() const { return nty * ntz; }
    __host__ __device__ uint32_t steps() const { return B + ty() + tz() - 2u; }
    __host__ __device__ uint32_t rows() const  // exchange rows per warp
    {
        return (steps() + kGrid7Group - 1u) / kGrid7Group * kGrid7Group;
    }
};

// The shape with the shortest estimated time: the critical path (padded lines
// and hand-overs) or the tiles' steps dealt over the SMs, whichever is longer;
// on a tie the fewer tiles.
inline Grid7Shape grid7_shape(uint32_t B, uint32_t ny, uint32_t nz, uint32_t sm_count)
{
    Grid7Shape best;
    uint64_t cost = ~0ull;
    for (uint32_t ly = 0; ly <= 5; ++ly)
    {
        Grid7Shape s{B, ny, nz, ly};
        s.nty = (ny + s.ty() - 1) / s.ty();
        s.ntz = (nz + s.tz() - 1) / s.tz();
        s.SP = s.rows() + kGrid7Ring;
        const uint64_t path = (uint64_t)B + s.nty * s.ty() + s.ntz * s.tz() + kGrid7Handover * (s.nty + s.ntz - 2);
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
struct G7Slot;
template <bool UNIT>
struct alignas(16) G7Slot<float, UNIT>
{
    float cz, cy, cx, dv;
};
template <>
struct alignas(16) G7Slot<double, true>
{
    double cz, cy, cx, pad;
};
template <>
struct alignas(16) G7Slot<double, false>
{
    double cz, cy, cx, dv, rc, pad;
};

template <bool UNIT>
__device__ __forceinline__ G7Slot<float, UNIT> g7_slot(const G7Slot<float, UNIT>* p)
{
    const float4 q = __ldg(reinterpret_cast<const float4*>(p));
    return {q.x, q.y, q.z, q.w};
}
__device__ __forceinline__ G7Slot<double, true> g7_slot(const G7Slot<double, true>* p)
{
    const double2* q = reinterpret_cast<const double2*>(p);
    const double2 a = __ldg(q), b = __ldg(q + 1);
    return {a.x, a.y, b.x, b.y};
}
__device__ __forceinline__ G7Slot<double, false> g7_slot(const G7Slot<double, false>* p)
{
    const double2* q = reinterpret_cast<const double2*>(p);
    const double2 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
    return {a.x, a.y, b.x, b.y, c.x, 0.0};
}
__device__ __forceinline__ void g7_st2_if(bool q, unsigned long long* p, unsigned long long a, unsigned long long b)
{
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\t@q st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};\n\t}" ::"l"(p),
        "l"(a), "l"(b), "r"((unsigned)q));
}
// one exchange value's words; `none` in each where q is false
__device__ __forceinline__ void g7_ld_if(bool q, const unsigned long long* p, unsigned long long none,
                                         unsigned long long (&w)[1])
{
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\tmov.u64 %0, %3;\n\t@q ld.relaxed.gpu.global.u64 %0, [%1];\n\t}"
        : "=&l"(w[0])
        : "l"(p), "r"((unsigned)q), "l"(none));
}
__device__ __forceinline__ void g7_ld_if(bool q, const unsigned long long* p, unsigned long long none,
                                         unsigned long long (&w)[2])
{
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %3, 0;\n\tmov.u64 %0, %4;\n\tmov.u64 %1, %4;\n\t"
        "@q ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];\n\t}"
        : "=&l"(w[0]), "=&l"(w[1])
        : "l"(p), "r"((unsigned)q), "l"(none));
}
__device__ __forceinline__ void g7_cp16(uint32_t dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// BYTES (4 or 8) of src, zero-filled where src_bytes is 0
template <int BYTES>
__device__ __forceinline__ void g7_cp_small(uint32_t dst, const void* src, uint32_t src_bytes)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(BYTES), "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void g7_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void g7_cp_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <typename VT, bool UNIT>
__global__ void __launch_bounds__(kThreads) k_grid7_pack(Grid7Shape sh, bool lower, const uint32_t* __restrict__ rp,
                                                         const uint32_t* __restrict__ ci, const VT* __restrict__ v,
                                                         const VT* __restrict__ d, G7Slot<VT, UNIT>* __restrict__ slot)
{
    const uint32_t B = sh.B, P = B * sh.ny, n = P * sh.nz, TY = sh.ty();
    const size_t total = (size_t)sh.tiles() * sh.SP * 32u;
    for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (size_t)gridDim.x * blockDim.x)
    {
        const uint32_t j = (uint32_t)(q % 32u), jy = j & (TY - 1u), jz = j >> sh.ly;
        const size_t ws = q / 32u;
        const uint32_t s = (uint32_t)(ws % sh.SP), w = (uint32_t)(ws / sh.SP);
        // solve order; k wraps before the line
        const uint32_t y = w % sh.nty * TY + jy, z = w / sh.nty * sh.tz() + jz, k = s - jy - jz;
        G7Slot<VT, UNIT> P7{};
        if constexpr (!UNIT) P7.dv = VT(1);
        if constexpr (!UNIT && sizeof(VT) == 8) P7.rc = 1.0;
        if (y < sh.ny && z < sh.nz && k < B)
        {
            const uint32_t ii = (z * sh.ny + y) * B + k, i = lower ? ii : n - 1u - ii;
            for (uint32_t e = rp[i]; e < rp[i + 1]; ++e)
            {
                const uint32_t c = ci[e];
                if (lower ? c + P == i : c == i + P) P7.cz = v[e];
                if (lower ? c + B == i : c == i + B) P7.cy = v[e];
                if (lower ? c + 1 == i : c == i + 1) P7.cx = v[e];
            }
            if constexpr (!UNIT)
            {
                if constexpr (sizeof(VT) == 4)
                    P7.dv = (VT)(1.0 / (double)d[i]);
                else
                {
                    P7.dv = d[i];
                    P7.rc = 1.0 / d[i];
                }
            }
        }
        slot[q] = P7;
    }
}

// ctl: [0] epoch, [1] exit count, [2] ticket (the last CTA to leave resets
// [1], [2] and advances [0], so the launch can be replayed).  order: ticket ->
// tile.  words: each tile's exchange rows, one a step: TZ values of its last
// lines in y, then TY of its last lines in z (one word per FP32 value, two per
// FP64 one).
template <bool LOWER, bool UNIT, typename VT, typename XT, typename RT>
__global__ void __launch_bounds__(32, 1) k_trsv_grid7(Grid7Shape sh, const uint32_t* __restrict__ order,
                                                      const G7Slot<VT, UNIT>* __restrict__ slot,
                                                      const RT* __restrict__ rhs, XT* __restrict__ x,
                                                      double* __restrict__ out64, const int* done,
                                                      unsigned long long* words, uint32_t* ctl, int* err,
                                                      unsigned polls_max)
{
    if (done && *done) return;
    using Slot = G7Slot<VT, UNIT>;
    constexpr int G = kGrid7Group;
    constexpr int WPV = sizeof(XT) == 8 ? 2 : 1;  // exchange words per value
    constexpr bool MARK = sizeof(XT) == 8 && !UNIT;
    extern __shared__ __align__(16) unsigned long long g7_sm[];  // two groups of results (4 KB), the operand ring
    XT* const stg = reinterpret_cast<XT*>(g7_sm);
    const uint32_t lane = threadIdx.x, nw = gridDim.x;
    uint32_t w = 0;
    if (lane == 0) w = __ldg(&order[atomicAdd(&ctl[2], 1u)]);
    w = __shfl_sync(0xffffffffu, w, 0);
    const uint32_t epoch = ld_flag(&ctl[0]) + 1u;
    const uint32_t B = sh.B, ny = sh.ny, TY = sh.ty(), TZ = sh.tz(), SP = sh.SP, S = sh.steps();
    const uint32_t ty = w % sh.nty, tz = w / sh.nty, jy = lane & (TY - 1u), jz = lane >> sh.ly;
    const uint32_t y = ty * TY + jy, z = tz * TZ + jz, L = z * ny + y;  // this lane's line in solve order
    const bool valid = y < ny && z < sh.nz;
    const uint32_t n = B * ny * sh.nz;
    const uint32_t k0 = valid ? 0u - jy - jz : B;
    const bool edge_y = jy == 0u, edge_z = jz == 0u;  // neighbours in another tile (or off the grid)
    const bool rd_y = edge_y && ty > 0u, rd_z = edge_z && tz > 0u;
    const bool pub_y = jy == TY - 1u && ty + 1u < sh.nty, pub_z = jz == TZ - 1u && tz + 1u < sh.ntz;
    const uint32_t RW = (TY + TZ) * WPV;  // words of an exchange row
    const size_t tile_words = (size_t)sh.rows() * RW;
    unsigned long long* const oy = words + w * tile_words + jz * WPV;
    unsigned long long* const oz = words + w * tile_words + (TZ + jy) * WPV;
    const unsigned long long* const iy = words + (ty > 0u ? w - 1u : w) * tile_words + (size_t)(TY - 1u) * RW + jz * WPV;
    const unsigned long long* const iz =
        words + (tz > 0u ? w - sh.nty : w) * tile_words + (size_t)(TZ - 1u) * RW + (TZ + jy) * WPV;
    const unsigned long long etag = (unsigned long long)epoch << 32;
    const Slot* ps = slot + (size_t)w * SP * 32u + lane;
    uint32_t lk = k0, li = L * B - jy - jz, lq = 0;  // k, solve-order index and ring entry of the step being fetched
    // a shared-memory ring of kGrid7Ring steps copied asynchronously
    // kGrid7Ring - 1 steps ahead (a step takes 120 - 190 ns, so that covers what
    // DRAM takes to answer): step s reads entry s % kGrid7Ring, and its copy for
    // step s + kGrid7Ring - 1 refills the entry that step s - 1 read
    constexpr uint32_t D = kGrid7Ring;
    const uint32_t ring_c = (uint32_t)__cvta_generic_to_shared(g7_sm) + 4096u;
    const uint32_t ring_r = ring_c + D * 32u * (uint32_t)sizeof(Slot);
    const Slot* ring_cp = reinterpret_cast<const Slot*>(reinterpret_cast<const unsigned char*>(g7_sm) + 4096);
    const RT* ring_rp = reinterpret_cast<const RT*>(ring_cp + D * 32u);
    auto copy_next = [&]() {
        const uint32_t e = lq * 32u + lane;
#pragma unroll
        for (uint32_t c = 0; c < sizeof(Slot) / 16; ++c)
            g7_cp16(ring_c + e * (uint32_t)sizeof(Slot) + 16u * c, reinterpret_cast<const unsigned char*>(ps) + 16u * c);
        const bool on = lk < B;
        g7_cp_small<sizeof(RT)>(ring_r + e * (uint32_t)sizeof(RT), on ? &rhs[LOWER ? li : n - 1u - li] : rhs,
                                on ? (uint32_t)sizeof(RT) : 0u);
        g7_cp_commit();
        ps += 32;
        ++lk;
        ++li;
        lq = lq + 1u == D ? 0u : lq + 1u;
    };
    // the neighbouring tiles' words of this lane for the group starting at s0: a
    // lane that needs none, and a step off its line, holds an epoch-tagged zero
    unsigned long long yw[G][WPV], zw[G][WPV];
    auto load_nb = [&](uint32_t s0) {
#pragma unroll
        for (int u = 0; u < G; ++u)
        {
            const bool on = k0 + s0 + (uint32_t)u < B;
            g7_ld_if(rd_y && on, iy + (size_t)(s0 + u) * RW, etag, yw[u]);
            g7_ld_if(rd_z && on, iz + (size_t)(s0 + u) * RW, etag, zw[u]);
        }
    };
    double* o64 = out64 ? out64 : reinterpret_cast<double*>(x);
    const bool w64 = out64 != nullptr;
    auto write_back = [&](int pass, uint32_t sg, const XT* buf) {
        const uint32_t l = (uint32_t)pass * (32u / G) + lane / G, u = lane % G;
        const uint32_t ly = l & (TY - 1u), lz = l >> sh.ly, yl = ty * TY + ly, zl = tz * TZ + lz;
        const uint32_t k = sg + u - ly - lz;
        const bool p = yl < ny && zl < sh.nz && k < B;
        const uint32_t i = (zl * ny + yl) * B + k, ii = LOWER ? i : n - 1u - i;
        const XT r = buf[u * 32u + l];
        g5_stx_if(p && !w64, x + ii, r);  // given out64, the FP64 copy is the result and x is not written
        g5_stx_if(p && w64, o64 + ii, (double)r);
    };
    // the row's entries in column order: lower (z-1), (y-1), (x-1); upper
    // (x+1), (y+1), (z+1); absent ones have +0 coefficients and +0 values
    auto row_sum = [&](RT r, const Slot& c, XT zb, XT nb, XT pv) -> XT {
        XT sum = (XT)r;
        if (LOWER)
        {
            sum -= (XT)c.cz * zb;
            sum -= (XT)c.cy * nb;
            sum -= (XT)c.cx * pv;
        }
        else
        {
            sum -= (XT)c.cx * pv;
            sum -= (XT)c.cy * nb;
            sum -= (XT)c.cz * zb;
        }
        return sum;
    };
    auto word_value = [](const unsigned long long (&wd)[WPV]) -> XT {
        if constexpr (WPV == 1)
            return (XT)__uint_as_float((uint32_t)wd[0]);
        else
            return (XT)__longlong_as_double((long long)((wd[WPV - 1] << 32) | (wd[0] & 0xffffffffull)));
    };
    // the value of step s to the next tiles
    auto publish = [&](bool on, uint32_t s, XT r) {
        const size_t o = (size_t)s * RW;
        if constexpr (WPV == 1)
        {
            const unsigned long long b = etag | __float_as_uint((float)r);
            g5_st_if(on && pub_y, oy + o, b);
            g5_st_if(on && pub_z, oz + o, b);
        }
        else
        {
            const unsigned long long bits = (unsigned long long)__double_as_longlong((double)r);
            const unsigned long long lo = etag | (bits & 0xffffffffull), hi = etag | (bits >> 32);
            g7_st2_if(on && pub_y, oy + o, lo, hi);
            g7_st2_if(on && pub_z, oz + o, lo, hi);
        }
    };
    for (uint32_t q = 0; q + 1 < D; ++q) copy_next();
    load_nb(0);
    XT prev = XT(0);
    uint32_t s0 = 0, g = 0;
    // the group's words must carry the epoch; stale ones are read again
    // (warp-uniform branches)
    auto fresh = [&]() {
        bool all = true;
#pragma unroll
        for (int u = 0; u < G; ++u)
#pragma unroll
            for (int c = 0; c < WPV; ++c)
                all &= (uint32_t)(yw[u][c] >> 32) == epoch && (uint32_t)(zw[u][c] >> 32) == epoch;
        return all;
    };
    bool failed = false;
    for (; s0 < S; s0 += G, ++g)
    {
        if (!__all_sync(0xffffffffu, fresh()))
            for (unsigned polls = 0;; ++polls)
            {
#pragma unroll
                for (int u = 0; u < G; ++u)
                {
                    const bool on = k0 + s0 + (uint32_t)u < B;
                    g7_ld_if(rd_y && on, iy + (size_t)(s0 + u) * RW, etag, yw[u]);
                    g7_ld_if(rd_z && on, iz + (size_t)(s0 + u) * RW, etag, zw[u]);
                }
                if (__all_sync(0xffffffffu, fresh())) break;
                if (__any_sync(0xffffffffu, polls >= polls_max || ld_err(err) != 0))
                {
                    if (lane == 0) atomicCAS(err, 0, (int)B2S_TIMEOUT);
                    failed = true;
                    break;
                }
            }
        if (failed) break;
        XT nbv[G], zbv[G];
#pragma unroll
        for (int u = 0; u < G; ++u)
        {
            nbv[u] = word_value(yw[u]);
            zbv[u] = word_value(zw[u]);
        }
        load_nb(s0 + G);  // the next group's words, checked when it starts
        __syncwarp();     // the previous group's results are in stg for every lane
        XT* cur = stg + (g & 1u) * (G * 32);
        const XT* old = stg + ((g & 1u) ^ 1u) * (G * 32);
        const uint32_t kg = k0 + s0;
        const XT prev0 = prev;
        bool bad = false;
#pragma unroll
        for (int u = 0; u < G; ++u)
        {
            const bool active = kg + (uint32_t)u < B;
            XT nb = __shfl_up_sync(0xffffffffu, prev, 1), zb = __shfl_up_sync(0xffffffffu, prev, TY);
            if (edge_y) nb = nbv[u];
            if (edge_z) zb = zbv[u];
            g7_cp_wait<D - 2>();  // this step's copies have landed
            const uint32_t e = ((s0 % D) + (uint32_t)u) * 32u + lane;
            const Slot c = ring_cp[e];
            const RT rr = ring_rp[e];
            copy_next();
            const XT sum = row_sum(rr, c, zb, nb, prev);
            XT r;
            if constexpr (UNIT)
                r = sum;
            else if constexpr (sizeof(XT) == 4)
                r = sum * (XT)c.dv;
            else
                r = g5_quotient(sum, c.dv, c.rc, active, bad);
            prev = active ? r : prev;
            cur[u * 32 + lane] = r;
            write_back(u, s0 - G, old);
            // with the FP64 quotient only while no lane of the group has needed the
            // division yet (a redo keeps the earlier steps' values: both roundings
            // are correct), the rest after the group
            bool on = true;
            if constexpr (MARK) on = !__any_sync(0xffffffffu, bad);
            publish(on, s0 + u, r);
        }
        if constexpr (MARK)
        {
            if (__any_sync(0xffffffffu, bad))
            {
                prev = prev0;
#pragma unroll
                for (int u = 0; u < G; ++u)
                {
                    const uint32_t k = kg + (uint32_t)u;
                    const bool active = k < B;
                    XT nb = __shfl_up_sync(0xffffffffu, prev, 1), zb = __shfl_up_sync(0xffffffffu, prev, TY);
                    if (edge_y) nb = nbv[u];
                    if (edge_z) zb = zbv[u];
                    const Slot c = g7_slot(slot + ((size_t)w * SP + s0 + u) * 32u + lane);
                    const uint32_t i = L * B + k;
                    const RT rr = active ? rhs[LOWER ? i : n - 1u - i] : RT(0);
                    const XT r = row_sum(rr, c, zb, nb, prev) / c.dv;
                    prev = active ? r : prev;
                    cur[u * 32 + lane] = r;
                    publish(true, s0 + u, r);  // steps already handed over get the same value again
                }
            }
        }
    }
    if (!failed && g)
    {
        __syncwarp();
#pragma unroll
        for (int pass = 0; pass < G; ++pass) write_back(pass, s0 - G, stg + ((g - 1u) & 1u) * (G * 32));
    }
    g7_cp_wait<0>();  // no copy into shared memory outlives the CTA
    if (lane == 0)
    {
        __threadfence();
        if (atomicAdd(&ctl[1], 1u) == nw - 1u)
        {
            ctl[1] = 0u;
            ctl[2] = 0u;
            ctl[0] = epoch;
            __threadfence();
        }
    }
}

// One triangle's 7-point grid schedule: packed slots, the exchange words and
// the launch.
struct Grid7Tri
{
    bool on = false;
    Grid7Shape sh;
    DBuf<uint4> slots;
    const void* packed_v = nullptr;
    uint32_t packed_vs = 0;
    DBuf<unsigned long long> words;
    DBuf<uint32_t> ctl, order;

    static bool fits(uint32_t b, uint32_t y, uint32_t z)
    {
        return b >= 2 && y >= 2 && z >= 2 && (uint64_t)(y + 31) / 32 * z <= kGrid7MaxWarps;
    }
    void enable(b2s_ctx* ctx, uint32_t b, uint32_t y, uint32_t z)
    {
        on = fits(b, y, z);
        if (on) sh = grid7_shape(b, y, z, (uint32_t)ctx->sm_count);
    }
    template <typename VT, typename XT>
    bool usable() const
    {
        return on && packed_v && packed_vs == sizeof(VT) && ctl.p;
    }
    template <typename VT, bool UNIT>
    void pack_t(b2s_ctx* ctx, const uint32_t* rp, const uint32_t* ci, const VT* v, const VT* d, bool lower)
    {
        using Slot = G7Slot<VT, UNIT>;
        const size_t count = (size_t)sh.tiles() * sh.SP * 32, units = count * sizeof(Slot) / 16;
        if (slots.n < units) slots.alloc(units);
        B2S_LAUNCH(ctx, (k_grid7_pack<VT, UNIT>), stream_grid(ctx, count), kThreads, 0, sh, lower, rp, ci, v, d,
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
            const uint32_t cy = sh.ty() + kGrid7Handover, cz = sh.tz() + kGrid7Handover;
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
        auto kern = k_trsv_grid7<LOWER, UNIT, VT, XT, RT>;
        B2S_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGrid7Smem));
        B2S_LAUNCH(ctx, kern, sh.tiles(), 32, kGrid7Smem, sh, order.p,
                   reinterpret_cast<const G7Slot<VT, UNIT>*>(slots.p), rhs, x, out64, done, words.p, ctl.p,
                   ctx->errword(), grid_polls(ctx));
    }
};

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
