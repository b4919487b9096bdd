// Host-only check of walk_shape.cuh: the items of a walk take every chunk of
// every row once, in the row's order within an item; its entries in coalesced
// steps; and there are no more than
// one per group of chunks and row and a constant beside them, whatever the longest row.
// Built and run by test_walk_cpu.py.
#include <cstdio>
#include <vector>

#include "chunk_engine.cuh"

static int g_fail = 0;

static void check(const char* name, const std::vector<sb200::ChunkRowFacts>& rows) {
    using namespace sb200;
    const uint64_t n = rows.size();
    WalkShape s;
    s.of(n, [&](uint64_t k) -> const ChunkRowFacts& { return rows[k]; });
    const WalkShape::Dims w = s.dims(n);
    std::vector<std::vector<uint8_t>> seen(n);
    uint64_t groups = 0;
    for (uint64_t r = 0; r < n; ++r) {
        seen[r].assign(rows[r].chunks, 0);
        groups += (rows[r].chunks + s.group - 1) / s.group;
    }
    if (w.items() > groups + n + (1u << 18) || s.lanes > s.groups) {
        std::printf("%s: %llu items for %llu groups of %llu rows\n", name, (unsigned long long)w.items(),
                    (unsigned long long)groups, (unsigned long long)n);
        ++g_fail;
    }
    for (uint64_t it = 0; it < w.items(); ++it) {
        const uint32_t r = w.row(it);
        for (uint64_t cg = w.first_chunk(it); cg < rows[r].chunks; cg += w.step())
            for (uint64_t c = cg; c < cg + s.group && c < rows[r].chunks; ++c) ++seen[r][c];
    }
    for (uint64_t r = 0; r < n; ++r)
        for (uint64_t c = 0; c < rows[r].chunks; ++c)
            if (seen[r][c] != 1) {
                std::printf("%s: chunk %llu of row %llu walked %d times\n", name, (unsigned long long)c,
                            (unsigned long long)r, seen[r][c]);
                ++g_fail;
                return;
            }
}

static sb200::ChunkRowFacts row(uint32_t chunks, uint64_t per_chunk, uint32_t bitmaps = 0) {
    sb200::ChunkRowFacts f;
    f.chunks = chunks;
    f.bitmap_chunks = bitmaps;
    f.list_entries = (chunks - bitmaps) * per_chunk;
    return f;
}

// A step takes 256 entries once, and 32 in a row at a time: a run's values then
// lie in the fewest sectors (eight counters each) at every update.
static void check_step() {
    std::vector<int> seen(sb200::WALK_STEP, 0);
    for (uint32_t q = 0; q < sb200::WALK_STEP / 32; ++q) {
        std::vector<uint8_t> sector(sb200::WALK_STEP / 8, 0);
        int sectors = 0;
        for (uint32_t lane = 0; lane < 32; ++lane) {
            const uint32_t e = sb200::walk_entry(q, lane);
            if (e < sb200::WALK_STEP) ++seen[e];
            if (e < sb200::WALK_STEP && !sector[e / 8]++) ++sectors;
        }
        if (sectors != 4) {
            std::printf("update %u of a step touches %d sectors\n", q, sectors);
            ++g_fail;
        }
    }
    for (int s : seen) g_fail += s != 1;
}

int main() {
    check_step();
    // the run postings gallop where runs are long, and where lists are short whatever the runs
    for (uint32_t wlog = 4; wlog <= 15; ++wlog) {
        g_fail += sb200::run_walk_gallops(wlog, 480000.0, 10000.0) != (wlog >= 6);
        g_fail += !sb200::run_walk_gallops(wlog, 479999.0, 10000.0) || !sb200::run_walk_gallops(wlog, 12000.0, 10000.0);
    }
    using Rows = std::vector<sb200::ChunkRowFacts>;
    check("no rows", {});
    check("empty rows", Rows(5));
    for (uint32_t chunks : {1u, 3u, 4u, 31u, 32u, 33u, 256u, 2048u})
        for (uint64_t per : {3ull, 47ull, 48ull, 4000ull}) {
            check("equal rows", Rows(200, row(chunks, per)));
            for (uint64_t n : {1ull, 1000ull, 100000ull}) {
                Rows r(n, row(1, 3));
                r.push_back(row(chunks, per));
                check("one long row", r);
                r.back() = row(chunks, per, 1);          // groups of one chunk for all
                check("one long row with a bitmap", r);
                r.insert(r.begin(), row(0, 0));
                check("and an empty row", r);
            }
        }
    Rows mixed;
    for (uint32_t k = 0; k < 3000; ++k) mixed.push_back(row(1 + k * k % 700, k % 9 ? 5 : 900));
    check("mixed rows", mixed);
    std::printf(g_fail ? "FAIL (%d)\n" : "ok\n", g_fail);
    return g_fail ? 1 : 0;
}
