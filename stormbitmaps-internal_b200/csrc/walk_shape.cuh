// walk_shape.cuh -- how a set of rows is dealt to warps chunk by chunk (the
// histogram and list passes of the postings, chunk_engine.cu).
//
// Every row group by group: all rows' first groups of consecutive chunks, then
// all rows' second ones, so that the warps at work meet in one part of the
// universe and what they update -- 4 bytes per value somewhere in it -- stays in
// L2. With a warp (or CTA) per row, 200 mixed rows left the GPU idle, and the
// places of 20000 rows' values (67 MB of cursors, 134 of postings) were written
// from DRAM.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>

namespace sb200 {

constexpr uint32_t ROW_WALK_THREADS = 256, ROW_WALK_BLOCKS = 8;   // and blocks per SM
// Rows of few entries a chunk among which most entries lie in chunks of many
// take groups of four: 32 such chunks are a long serial item for one warp
// (3072 Zipf rows over 2^24, histogram to lists: 0.79 ms by 32, 0.59 by 8,
// 0.58 by 4; 1094 over 2^23 0.32, 0.21, 0.20).
constexpr uint32_t WALK_SKEW_GROUP = 4;
// A step of a warp through a list: the lanes on consecutive entries, so that the
// entries of a run meet in the sectors of what is updated per value. Eight
// consecutive entries per lane made each of a warp's updates another sector: the
// sum of 2000 rows of 100 runs over 2^20 took 379 us instead of 208, over 2^24 394
// instead of 184; rows without runs the same either way.
constexpr uint32_t WALK_STEP = 256;
__host__ __device__ inline uint32_t walk_entry(uint32_t q, uint32_t lane) { return 32 * q + lane; }

// How the run postings go through rows' lists: a lane per chunk that gallops from
// run to run, from a mean run length of 2^6 on (wlog) and for short lists, where a
// warp looking at 256 entries at a time has a few to look at (run form forced, ms,
// 256 entries / galloping: 20000 rows of 168 values over 2^24 3.45 / 2.01, 4000 of
// 839 over 2^22 0.94 / 0.78, 300 of 671 over 2^26 0.30 / 0.15).
inline bool run_walk_gallops(uint32_t wlog, double entries, double chunks) {
    return wlog >= 6 || entries < 48.0 * chunks;
}

// Items of a walk beside one per row and one per group that there is: some find
// no chunk, more leave less of a long row to one warp.
constexpr uint64_t WALK_SPARE_ITEMS = 1ull << 18;

// group: chunks per group (one from 48 entries a chunk on, or with bitmap
// chunks). Item k of n x lanes items is row k % n's groups k / n, k / n + lanes,
// and so on: one group each (lanes = those of the longest row) unless most rows
// end long before the longest one does, when nearly all items would find
// nothing.
struct WalkShape {
    uint32_t group = 1, groups = 0, lanes = 0;
    template <class Facts>
    void of(uint64_t n, Facts facts) {
        uint64_t chunks = 0, entries = 0;
        double spread = 0.0;                              // entries x (their row's entries per chunk)
        uint32_t most = 0;
        bool bitmaps = false;
        for (uint64_t k = 0; k < n; ++k) {
            const auto& f = facts(k);                     // ChunkRowFacts (chunk_engine.cuh)
            chunks += f.chunks;
            entries += f.list_entries;
            bitmaps |= f.bitmap_chunks != 0;
            most = std::max(most, f.chunks);
            if (f.chunks) spread += (double)f.list_entries * (double)f.list_entries / (double)f.chunks;
        }
        group = bitmaps || entries >= 48 * chunks ? 1u : spread >= 48.0 * (double)entries ? WALK_SKEW_GROUP : 32u;
        groups = (most + group - 1) / group;
        lanes = (uint32_t)std::min<uint64_t>(groups, n ? (chunks / group + n + WALK_SPARE_ITEMS) / n : 0);
    }
    uint32_t grid(uint64_t n, int sms) const {
        return (uint32_t)std::max<uint64_t>(
            1, std::min<uint64_t>((n * lanes + ROW_WALK_THREADS / 32 - 1) / (ROW_WALK_THREADS / 32), (uint64_t)sms * ROW_WALK_BLOCKS));
    }
    // The same for the kernels: item `it` of n x lanes.
    struct Dims {
        uint32_t n, group, lanes;
        __host__ __device__ uint64_t items() const { return (uint64_t)n * lanes; }
        __host__ __device__ uint32_t row(uint64_t it) const { return (uint32_t)(it % n); }
        // (rows have at most 2048 chunks: universe <= 2^27)
        __host__ __device__ uint32_t first_chunk(uint64_t it) const { return (uint32_t)(it / n) * group; }
        __host__ __device__ uint32_t step() const { return lanes * group; }
    };
    Dims dims(uint64_t n) const { return Dims{(uint32_t)n, group, lanes}; }
};

}  // namespace sb200
