// The rules of csrc/trsv_plan.hpp that say which schedule takes an exact
// triangular solve: rows_fit_chunks against the planner itself on both sides of
// the longest row, and wave_pays on patterns whose two schedules were measured.
#include <cstdio>
#include <random>
#include <vector>

#include "../../cpp-fem-solver_b200/csrc/trsv_plan.hpp"

using namespace b2s;

struct Pattern
{
    std::vector<uint32_t> rp{0}, ci;
};

// strict lower rows; mirrored for an upper triangle
static Pattern rows(const std::vector<std::vector<uint32_t>>& r, bool lower)
{
    const uint32_t n = (uint32_t)r.size();
    Pattern P;
    for (uint32_t i = 0; i < n; ++i)
    {
        const std::vector<uint32_t>& row = r[lower ? i : n - 1 - i];
        if (lower)
            P.ci.insert(P.ci.end(), row.begin(), row.end());
        else
            for (auto it = row.rbegin(); it != row.rend(); ++it) P.ci.push_back(n - 1 - *it);
        P.rp.push_back((uint32_t)P.ci.size());
    }
    return P;
}

static std::vector<std::vector<uint32_t>> band(uint32_t n, uint32_t w)
{
    std::vector<std::vector<uint32_t>> r(n);
    for (uint32_t i = 0; i < n; ++i)
        for (uint32_t k = std::min(i, w); k > 0; --k) r[i].push_back(i - k);
    return r;
}

static int bad = 0;

static void expect(const char* name, const std::vector<std::vector<uint32_t>>& r, bool want, uint32_t bs = 1)
{
    for (bool lower : {true, false})
    {
        const Pattern P = rows(r, lower);
        std::vector<uint32_t> lev;
        compute_levels((uint32_t)r.size(), P.rp.data(), P.ci.data(), lower, lev);
        const bool got = wave_pays(lev, P.rp.data(), P.ci.data(), lower, bs);
        if (got != want) ++bad, std::printf("%s bs %u %s: %d\n", name, bs, lower ? "lower" : "upper", got);
    }
}

int main()
{
    for (uint32_t vs : {4u, 8u})
        for (uint32_t dv : {0u, 1u})
        {
            // n / a / b: a band of one with one row of w entries, w about the longest a chunk takes
            const uint32_t per = 2 * vs + 6, fixed = 160 + vs * dv + 10 + vs + 8, most = (kChunkSmemBudget - fixed) / per;
            for (uint32_t w : {most - 1, most, most + 1, most + 500})
                for (bool lower : {true, false})
                {
                    std::vector<std::vector<uint32_t>> r = band(w + 50, 1);
                    std::vector<uint32_t>& row = r[w + 20];
                    row.clear();
                    for (uint32_t j = 0; j < w; ++j) row.push_back(j);
                    const Pattern P = rows(r, lower);
                    const uint32_t n = (uint32_t)r.size();
                    const bool fits = rows_fit_chunks(n, P.rp.data(), P.ci.data(), lower, dv, vs, vs, 8);
                    const bool ok = plan_chunks(n, P.rp.data(), P.ci.data(), lower, dv, vs, vs, 8).ok;
                    if (fits != ok || fits != (w <= most))
                        ++bad, std::printf("vs %u dv %u w %u lower %d: fits %d plan %d\n", vs, dv, w, lower, fits, ok);
                }
        }

    const uint32_t n = 4000;
    for (uint32_t w = 1; w <= 4; ++w)
        for (uint32_t bs : {1u, 2u, 3u}) expect("short rows", band(n, w), false, bs);
    for (uint32_t w : {5u, 9u, 16u, 33u, 100u})
        for (uint32_t bs : {1u, 2u, 3u}) expect("wide rows", band(n, w), true, bs);
    std::mt19937 rng(1);
    // one row in `every` has `extra` more entries than its band
    auto mixed = [&](uint32_t w, uint32_t every, uint32_t extra) {
        std::vector<std::vector<uint32_t>> r = band(n, w);
        for (uint32_t i = 200; i < n; i += every)
        {
            std::vector<uint32_t> more;
            for (uint32_t k = 0; k < extra; ++k) more.push_back(rng() % (i - w));
            std::sort(more.begin(), more.end());
            more.erase(std::unique(more.begin(), more.end()), more.end());
            r[i].insert(r[i].begin(), more.begin(), more.end());
        }
        return r;
    };
    expect("one long row", mixed(1, n, 500), false);
    expect("one long row", mixed(1, n, 500), false, 3);
    expect("few wide rows", mixed(3, 40, 3), false);
    expect("a quarter wide", mixed(3, 4, 3), false);
    expect("most wide", mixed(4, 1, 4), true);
    expect("few wide blocks", mixed(1, 40, 5), false, 2);
    expect("wide blocks by the half", mixed(4, 2, 4), true, 2);
    // many rows a level
    std::vector<std::vector<uint32_t>> flat(n);
    for (uint32_t i = 0; i < n; ++i)
        if (i >= 600) flat[i].push_back(i - 600);
    expect("600 rows a level", flat, true);
    std::printf(bad ? "%d wrong\n" : "OK\n", bad);
    return bad != 0;
}
