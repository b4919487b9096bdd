// Host-only check of RowsByCard (chunk_engine.cuh): nothing is made before the
// order is asked for, it is the stable one by value count, largest first, and it
// is made again after the rows changed. And of rows_join_panel: a panel that is
// asked for by name needs its memory as one that is chosen. Built and run by
// test_walk_cpu.py.
#include <algorithm>
#include <cstdio>
#include <numeric>
#include <random>

#include "chunk_engine.cuh"

using sb200::ChunkRowFacts;

static std::vector<ChunkRowFacts> rows(uint64_t n, uint64_t most, uint64_t seed) {
    std::mt19937_64 g(seed);
    std::vector<ChunkRowFacts> f(n);
    for (auto& x : f) x.card = most ? g() % (most + 1) >> (g() % 40) : 0;
    return f;
}

static bool same(const std::vector<uint32_t>& got, const std::vector<ChunkRowFacts>& f) {
    std::vector<uint32_t> want(f.size());
    std::iota(want.begin(), want.end(), 0u);
    std::stable_sort(want.begin(), want.end(), [&](uint32_t a, uint32_t b) { return f[a].card > f[b].card; });
    return got == want;
}

int main() {
    int fail = 0;
    sb200::ChunkDev d;
    for (uint64_t n : {0ull, 1ull, 2ull, 100ull, 5000ull})
        for (uint64_t most : {0ull, 1ull, 2047ull, 2048ull, 1ull << 27, ~0ull - 1}) {
            d.facts = rows(n, most, n + most);
            d.by_card.rows_changed();
            fail += d.by_card.is_made();
            fail += !same(d.by_card.of(d.facts), d.facts);
            fail += !d.by_card.is_made() || !same(d.by_card.of(d.facts), d.facts);
        }
    // the sums' walk of all plain rows, the same way
    for (uint32_t n : {3u, 5000u}) {
        std::vector<uint32_t> plain(n);
        std::iota(plain.begin(), plain.end(), 0u);
        d.facts.assign(n, ChunkRowFacts{});
        for (auto& f : d.facts) f.chunks = 40, f.list_entries = n;
        d.rows_changed();
        fail += d.plain_walk.is_made() || d.by_card.is_made();
        sb200::WalkShape want;
        want.of(n, [&](uint64_t k) -> const ChunkRowFacts& { return d.facts[k]; });
        for (int call = 0; call < 2; ++call) {
            const sb200::WalkShape& got = d.plain_walk.of(plain, d.facts);
            fail += got.group != want.group || got.groups != want.groups || got.lanes != want.lanes;
            fail += !d.plain_walk.is_made();
        }
    }
    int asked = 0;
    auto fits = [&asked](bool answer) {
        return [&asked, answer] {
            ++asked;
            return answer;
        };
    };
    fail += sb200::rows_join_panel(true, 2.0, 1.0, fits(false));
    fail += sb200::rows_join_panel(false, 1.0, 2.0, fits(false));
    fail += !sb200::rows_join_panel(true, 2.0, 1.0, fits(true));
    fail += !sb200::rows_join_panel(false, 1.0, 2.0, fits(true));
    fail += asked != 4;
    fail += sb200::rows_join_panel(false, 2.0, 1.0, fits(true)) || asked != 4;
    std::printf(fail ? "FAIL (%d)\n" : "ok\n", fail);
    return fail ? 1 : 0;
}
