// Host-only checks (no GPU) of the 256 x 256 tiles of the CTA-pair kernels:
//  * sb200::build_tiles and sb200::band_tiles -- every pair i <= j < n in one
//    tile; the banded order is a permutation, bands of A blocks in order and
//    within a band column by column;
//  * sb200::host_plan, host_arrivals and arrival_of, as panels_to_host follows
//    them -- panels partition the list from its end, whole A blocks where they
//    are made of blocks; every row is uploaded once, last rows first; a panel's
//    tiles read only rows of the part they wait for or of earlier ones; the
//    copies tile the packed triangle from its end and follow their tiles.
// Built and run by test_pair_tiles_cpu.py.
#include <algorithm>
#include <cstdio>
#include <vector>

#include "dense.cuh"

using namespace sb200;

static int g_fail = 0;
#define CHECK(c, n)                                                                    \
    do {                                                                               \
        if (!(c)) {                                                                    \
            std::printf("line %d n %llu: %s\n", __LINE__, (unsigned long long)(n), #c); \
            ++g_fail;                                                                  \
            return;                                                                    \
        }                                                                              \
    } while (0)

static void check_cover(int kind, uint64_t n) {
    std::vector<uint2> t, b;
    build_tiles(t, n, kind);
    const uint64_t nb = (n + 255) / 256;
    CHECK(t.size() == nb * (nb + 1) / 2, n);
    std::vector<uint8_t> seen(nb * nb, 0);
    for (const uint2& q : t) {
        CHECK(q.x <= q.y && q.y < nb, n);
        ++seen[q.x * nb + q.y];
    }
    for (uint64_t i = 0; i < nb; ++i)
        for (uint64_t j = i; j < nb; ++j) CHECK(seen[i * nb + j] == 1, n);
    CHECK(std::is_sorted(t.begin(), t.end(), [](uint2 p, uint2 q) { return p.x != q.x ? p.x < q.x : p.y < q.y; }), n);
    b = t;
    band_tiles(b);
    for (const uint2& q : b) ++seen[q.x * nb + q.y];
    for (uint64_t i = 0; i < nb; ++i)
        for (uint64_t j = i; j < nb; ++j) CHECK(seen[i * nb + j] == 2, n);
    for (size_t k = 1; k < b.size(); ++k) {
        const uint2 p = b[k - 1], q = b[k];
        CHECK(p.x / 8 < q.x / 8 || (p.x / 8 == q.x / 8 && (p.y < q.y || (p.y == q.y && p.x < q.x))), n);
    }
}

static void check_plan(int kind, uint64_t n, int sms, uint64_t bus_bytes, bool pinned) {
    std::vector<uint2> t;
    build_tiles(t, n, kind);
    const uint64_t bm = tile_rows_a(kind), bn = tile_rows_b(kind);
    const auto panels = host_plan(kind, n, (uint32_t)t.size(), sms, bus_bytes, pinned);
    // pageable memory: no panels where they would be whole A blocks for the copies' sake
    CHECK(pinned || kind != KIND_F4 || t.size() > 24u * std::max(1, sms / 2) || panels.size() == 1, n);
    const auto arrive = host_arrivals(kind, n, t, panels, sms);
    CHECK(!panels.empty() && !arrive.empty() && arrive.back() == 0 && arrive[0] < n, n);
    for (size_t c = 1; c < arrive.size(); ++c) CHECK(arrive[c] < arrive[c - 1], n);   // each row once, in one part
    std::vector<uint32_t> first_tile(t.back().x + 1, 0);
    for (uint32_t k = (uint32_t)t.size(); k-- > 0;) first_tile[t[k].x] = k;
    uint64_t hi = t.size(), copied_from = n;
    for (const auto& p : panels) {
        CHECK(p.second == hi && p.first < p.second, n);
        hi = p.first;
        uint64_t need = n;
        for (uint32_t k = p.first; k < p.second; ++k) need = std::min<uint64_t>(need, std::min(t[k].x * bm, t[k].y * bn));
        const size_t c = arrival_of(arrive, need);
        for (uint32_t k = p.first; k < p.second; ++k)
            CHECK(t[k].x * bm >= arrive[c] && t[k].y * bn >= arrive[c], n);
        uint64_t b = t[p.first].x;
        if (first_tile[b] != p.first) ++b;
        const uint64_t r = std::min<uint64_t>(n, b * bm);
        if (r < copied_from) {
            for (uint64_t k = 0; k < p.first; ++k) CHECK(t[k].x < b, n);
            copied_from = r;
        }
    }
    CHECK(hi == 0 && copied_from == 0, n);
}

int main() {
    for (int kind : {KIND_F4, (int)STORM_B200_KERNEL_MMA_2CTA})
        for (uint64_t n : {1ull, 255ull, 256ull, 257ull, 512ull, 2047ull, 2049ull, 4096ull, 5000ull, 9000ull})
            check_cover(kind, n);
    for (int kind : {KIND_F4, (int)STORM_B200_KERNEL_MMA_2CTA, (int)STORM_B200_KERNEL_MMA, (int)STORM_B200_KERNEL_MMA_DB,
                     (int)STORM_B200_KERNEL_POPC})
        for (uint64_t n : {1ull, 256ull, 257ull, 700ull, 2000ull, 4097ull, 9000ull, 15000ull, 15104ull, 15105ull, 16000ull,
                           30000ull})
            for (int sms : {1, 2, 147, 148})
                for (uint64_t mib : {0ull, 1ull, 5ull, 1000ull})
                    for (bool pinned : {true, false}) check_plan(kind, n, sms, mib << 20, pinned);
    std::printf(g_fail ? "FAIL (%d)\n" : "ok\n", g_fail);
    return g_fail ? 1 : 0;
}
