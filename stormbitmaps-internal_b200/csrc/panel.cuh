// panel.cuh -- sparse rows against a transposed dense panel: the bit-slice
// engine of the STORM_t all-pairs planner.
//
// The tensor cores pay for a pair in proportion to the universe, whatever
// the rows hold; a pair of a sparse row x and a dense row p costs only
// |x| bits of p.  For a block of up to 2048 panel rows the engine stores the
// panel TRANSPOSED: DT[v] = 2048 bits, bit r set when panel row r holds
// value v (32 u64 words per value, U x 256 bytes in HBM).  A query row x is
// then one warp: lane w owns panel rows 64w .. 64w + 63, and for every value
// v of x it adds the 64 bits of DT[v][w] (one coalesced 256-byte line per value
// for the warp) into 64 per-row counters held bit-sliced: a tree of carry-save
// adders, and a carry that ripples into vertical counter planes.  Every 2016
// words and after the row, each lane adds its planes' 64 counts to the warp's
// 2048 in shared memory, which go into the packed triangle at the end.  Work per
// pair is |x| / 64 word additions and |x| / 8 bytes of panel traffic, against
// the universe's bits on the tensor cores.
//
// A query row is one work item, or -- when it holds many values -- several:
// items cover ranges of the row's chunks, so that no warp walks millions of
// values alone while the others wait (a warp has 64 values' lines on their
// way at most).  The items of a split row
// write their counts into scratch slots, and panel_reduce_kernel adds the
// slots of each split row into the triangle.
//
// Bound: HBM (the DT lines: 256 bytes per value of a query row per block).
#pragma once
#include "chunk_engine.cuh"
#include "tc_ptx.cuh"

namespace sb200 {

constexpr uint32_t PANEL_ROWS = 2048;                  // panel rows per block
constexpr uint32_t PANEL_WORDS = PANEL_ROWS / 64;      // DT words per value of a whole block
constexpr uint32_t PANEL_X_SLOTS = 32;                 // chunk slots expanded at a time (541 MB)
constexpr uint32_t PANEL_T_WORDS = 4;                  // row words per transpose CTA (256 values)
constexpr uint32_t PANEL_NO_VALUE = 0xFFFFFFFFu;
constexpr uint64_t PANEL_MAX_UNIVERSE = 1ull << 26;    // 16 GiB of transposed block
constexpr uint64_t PANEL_MIN_SEG = 2048;               // values per work item of a split row, at least (8192: the last
                                                       // items kept a query of 183 rows 0.2 ms longer)
constexpr uint32_t PANEL_MAX_SLOTS = 8192;             // scratch slots of split rows (64 MiB)

// X: PANEL_ROWS expanded rows (rows past the block's end are zero),
// block-major, so that the 2048 rows' words a CTA reads lie within 17 MB and
// not on 2048 pages (row-major rows of 2^24 bits took 5.3 ms, these 1.9).
// DT[v * PANEL_WORDS + w] bit r = bit v of row 64 w + r.  CTA: 32 warps, warp w
// transposes rows 64w .. 64w + 63 for PANEL_T_WORDS words: each
// 32 x 32 bit block (32 rows' 32-bit half-word, one per lane) is transposed
// in registers by five butterfly stages (shfl_xor over lanes 16, 8, 4, 2, 1),
// after which lane l holds bit l of that half-word across the 32 rows.  The
// CTA stages the 256 x 32 result (PANEL_T_SMEM bytes of dynamic shared
// memory, each value's 32 words rotated by the value so that a warp's 32
// stores hit distinct banks) and writes it out in order.
constexpr uint32_t panel_t_smem(uint32_t pw) { return 64 * PANEL_T_WORDS * pw * 8; }   // 64 KiB of a whole block

// DT words per value of a block of `rows` panel rows: the last block, often
// the only one, is stored 2048, 1024 or 512 rows wide. What a block costs is
// in proportion to its width: the transposed block is written whole (2^24
// values, expanded and transposed: 3.0 ms 2048 wide, 1.6 ms 1024 wide), and a
// query value reads its whole line (measured 32, 20 and 15 ps a value). The
// planner can then leave rows of medium weight to the postings instead of
// filling a block of 2048 with them: 4096 Zipf rows over 2^24 7.5 -> 6.1 ms.
constexpr double PANEL_HALF_COST = 0.64, PANEL_QUARTER_COST = 0.48;   // a query value against them, of a whole block
inline uint32_t panel_block_words(uint64_t rows) { return rows > PANEL_ROWS / 2 ? 32u : rows > PANEL_ROWS / 4 ? 16u : 8u; }

// 32 x 32 bit transpose across a warp: on entry lane r holds row r (bit c =
// column c); on return lane c holds column c (bit r = row r).  At stage j the
// lanes with bit j clear trade their high j-bit groups for the low groups of
// lane ^ j: a byte permute at 16 and 8, a rotation and a merge at 4, 2 and 1,
// whose selector, amount and mask depend on the lane alone (shifting both ways
// and selecting took 35 instructions for the five stages; these take 13).
struct LaneTranspose {
    uint32_t sel16, sel8, rot4, rot2, rot1, keep4, keep2, keep1;
    __device__ __forceinline__ explicit LaneTranspose(uint32_t lane) {
        sel16 = lane & 16 ? 0x3276u : 0x5410u;
        sel8 = lane & 8 ? 0x3715u : 0x6240u;
        rot4 = lane & 4 ? 28 : 4;
        rot2 = lane & 2 ? 30 : 2;
        rot1 = lane & 1 ? 31 : 1;
        keep4 = lane & 4 ? 0xF0F0F0F0u : 0x0F0F0F0Fu;
        keep2 = lane & 2 ? 0xCCCCCCCCu : 0x33333333u;
        keep1 = lane & 1 ? 0xAAAAAAAAu : 0x55555555u;
    }
    __device__ __forceinline__ uint32_t operator()(uint32_t x) const {
        x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 16), sel16);
        x = __byte_perm(x, __shfl_xor_sync(0xffffffffu, x, 8), sel8);
        uint32_t y = __shfl_xor_sync(0xffffffffu, x, 4);
        x = (x & keep4) | (__funnelshift_l(y, y, rot4) & ~keep4);
        y = __shfl_xor_sync(0xffffffffu, x, 2);
        x = (x & keep2) | (__funnelshift_l(y, y, rot2) & ~keep2);
        y = __shfl_xor_sync(0xffffffffu, x, 1);
        return (x & keep1) | (__funnelshift_l(y, y, rot1) & ~keep1);
    }
};

template <uint32_t PW>
__global__ void __launch_bounds__(PW * 32)
panel_transpose_kernel(const uint64_t* __restrict__ X, RowLayout lay, uint32_t prows, uint64_t* __restrict__ DT) {
    extern __shared__ unsigned long long stage[];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t k0 = (uint64_t)blockIdx.x * PANEL_T_WORDS;   // within X
    const uint64_t at = k0 / CHUNK_WORDS * lay.kstride + k0 % CHUNK_WORDS;
    const uint32_t ra = 64 * warp + lane, rb = ra + 32;
    const LaneTranspose transpose(lane);
    static_assert(PANEL_T_WORDS == 4, "one 32-byte load per row");
    Row32 va{}, vb{};                       // rows past the block's end are zero
    if (ra < prows) va = ldg_row32(X + (uint64_t)ra * lay.pitch + at);
    if (rb < prows) vb = ldg_row32(X + (uint64_t)rb * lay.pitch + at);
    const uint64_t (&xa)[4] = va.w, (&xb)[4] = vb.w;
    // a value's PW words are rotated so that the 16 lanes of a store phase hit distinct bank pairs
    auto turn = [](uint32_t v) { return PW >= 16 ? v : v * PW / 16; };
#pragma unroll
    for (uint32_t q = 0; q < PANEL_T_WORDS; ++q) {
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
            const uint32_t lo = transpose((uint32_t)(xa[q] >> (32 * h)));
            const uint32_t hi = transpose((uint32_t)(xb[q] >> (32 * h)));
            const uint32_t v = 64 * q + 32 * h + lane;     // value within the CTA's 256
            stage[v * PW + ((warp + turn(v)) & (PW - 1))] = ((uint64_t)hi << 32) | lo;
        }
    }
    __syncthreads();
    uint64_t* dst = DT + k0 * 64 * PW;
    for (uint32_t t = threadIdx.x; t < 64 * PANEL_T_WORDS * PW; t += blockDim.x) {
        const uint32_t v = t / PW, w = t % PW;
        __stcs(dst + t, (uint64_t)stage[v * PW + ((w + turn(v)) & (PW - 1))]);
    }
}

__device__ __forceinline__ void panel_csa(uint64_t& h, uint64_t& l, uint64_t a, uint64_t b, uint64_t c) {
    const uint64_t u = a ^ b;
    h = (a & b) | (u & c);
    l = u ^ c;
}

// Bit-sliced counters of a lane, per bit position: sum_k 2^k s[k] + sum_k
// 2^(L + k) planes[k], below 2048.  The 2^L words of a batch go through a tree
// of carry-save adders (s[k] holds what is left at weight 2^k) and one carry of
// weight 2^L ripples into the planes.  More planes, so that no row outgrew
// them, took half the warps' registers and twice the ripple.
constexpr uint32_t PANEL_FLUSH_WORDS = 2016;               // words added between flushes (63 x 32), at most 2047

template <int L, class Load>
__device__ __forceinline__ uint64_t panel_tree(uint32_t at, uint64_t* s, Load load) {
    uint64_t h;
    if constexpr (L == 1) panel_csa(h, s[0], s[0], load(at), load(at + 1));
    else {
        const uint64_t a = panel_tree<L - 1>(at, s, load);
        const uint64_t b = panel_tree<L - 1>(at + (1u << (L - 1)), s, load);
        panel_csa(h, s[L - 1], s[L - 1], a, b);
    }
    return h;
}

// One warp per (work item, block): items[k] (heaviest first), taken from a
// shared counter; the block holds the panel rows at walk positions
// [pw0, pw0 + prows).  Pairs with a panel row at a walk position after the
// query row's are written: out[(i, j)] with i, j the rows' stored indices
// (perm) -- or, for an item of a split row, scratch[slot][t] for panel row t
// -- and the sum over them added into flags.
//
// A row's chunks are walked 32 at a time: one lane reads each chunk's head, and
// the values of the group's lists are read as one sequence (the chunk of entry
// t found in the lanes' prefix sums), the next 32 on their way while the ones
// before them are counted -- chunk by chunk, a row of short lists waited for
// three reads in turn per chunk.
// The lines of 32 values are one batch, copied to shared memory by cp.async,
// PANEL_Q_STAGES batches at a time: what bounds the kernel is how many lines
// are on their way (random 64 PW / 8 byte reads), and lines held in registers
// (16 a warp, 126 registers a thread) left 44 KB of them per SM: 4.9 TB/s. Every
// row in the panel, registers / 1 / 2 / 3 / 4 batches: 4096 Zipf rows over 2^24
// 59 / 55 / 50 / 53 / 55 ms, 9000 over 2^21 36.5 / 29.7 / 27.5 / 30.9 / 34.0 (more
// batches leave fewer warps), batches of 16 values 51 and 28.8 at best.
// With narrow lines a warp adds 32 / PW values at once: lane l holds word
// l % PW of every (l / PW)-th of them.
// Shared memory: the batches, 64 PW counts, 64 staged values.
constexpr uint32_t PANEL_Q_STAGES = 2;
constexpr uint32_t PANEL_Q_SMEM_SM = 228 << 10;           // shared memory of an SM; a CTA takes 1 KiB more than it asks for
constexpr uint32_t panel_q_smem(uint32_t pw) { return PANEL_Q_STAGES * 32 * pw * 8 + 64 * pw * 4 + 64 * 4; }

template <uint32_t PW>
__global__ void __launch_bounds__(32)
panel_query_kernel(ChunkView v, const uint32_t* __restrict__ perm, const PanelItem* __restrict__ items, uint32_t n_items,
                   uint64_t pw0, uint32_t prows, const uint64_t* __restrict__ DT, uint64_t n,
                   uint32_t* __restrict__ out, uint32_t* __restrict__ scratch, DeviceFlags* __restrict__ flags,
                   unsigned long long* __restrict__ counter) {
    constexpr int L = PW == 32 ? 5 : PW == 16 ? 4 : 3, PLANES = 11 - L;
    constexpr uint32_t PARTS = PW / 2, BATCH = 32 * PW;    // 16-byte parts of a line; words of a batch
    extern __shared__ __align__(16) uint64_t ring[];
    uint32_t* const cs = reinterpret_cast<uint32_t*>(ring + PANEL_Q_STAGES * BATCH);
    uint32_t* const vb = cs + 64 * PW;
    const uint32_t lane = threadIdx.x & 31;
    unsigned long long local = 0;
    for (;;) {
        unsigned long long item = 0;
        if (lane == 0) item = atomicAdd(counter, 1ull);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= n_items) break;
        const PanelItem it = items[item];
        const uint64_t xw = it.xw;
        if (xw + 1 >= pw0 + prows) continue;              // no panel row after it in this block
        const uint32_t sx = perm[xw];
        const uint64_t c0 = v.row_off[sx];
        uint64_t cnt[L] = {}, planes[PLANES] = {};
        uint32_t added = 0;                               // words added since the last flush
        bool flushed = false;
        // 64 counts of this lane's panel rows 64 (lane % PW) + r (narrow lines:
        // the sum over the lanes of that word), staged so that the write-out
        // below reads consecutive rows (XOR swizzle by word)
        auto flush = [&]() {
            const uint32_t word = lane % PW;
#pragma unroll 4
            for (uint32_t r = 0; r < 64; ++r) {
                uint32_t x = 0;
#pragma unroll
                for (int k = 0; k < L; ++k) x += (uint32_t)((cnt[k] >> r) & 1u) << k;
#pragma unroll
                for (int k = 0; k < PLANES; ++k) x += (uint32_t)((planes[k] >> r) & 1u) << (k + L);
#pragma unroll
                for (uint32_t o = PW; o < 32; o <<= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
                uint32_t& c = cs[64 * word + (r ^ word)];
                if (PW == 32 || lane < PW) c = flushed ? c + x : x;
            }
#pragma unroll
            for (int k = 0; k < L; ++k) cnt[k] = 0;
#pragma unroll
            for (int k = 0; k < PLANES; ++k) planes[k] = 0;
            flushed = true;
            added = 0;
        };
        uint32_t head = 0, flying = 0;                    // next batch's place in the ring; batches on their way
        auto count = [&]() {                              // the oldest batch, arrived
            if (added == PANEL_FLUSH_WORDS) flush();
            const uint64_t* w = ring + (head >= flying ? head - flying : head + PANEL_Q_STAGES - flying) * BATCH + lane;
            uint64_t c = panel_tree<L>(0u, cnt, [&](uint32_t t) { return w[32 * t]; });
#pragma unroll
            for (int k = 0; k < PLANES; ++k) {
                const uint64_t nc = planes[k] & c;
                planes[k] ^= c;
                c = nc;
            }
            added += PW;
            --flying;
            __syncwarp();                                 // read by every lane: its place may be filled again
        };
        auto batch = [&](uint32_t myv) {                  // 32 values, one per lane (PANEL_NO_VALUE: none)
            const uint32_t dst = smem_u32(ring + head * BATCH);
#pragma unroll
            for (uint32_t t = 0; t < PARTS; ++t) {
                const uint32_t part = 32 * t + lane;
                const uint32_t val = __shfl_sync(0xffffffffu, myv, part / PARTS);
                const bool has = val != PANEL_NO_VALUE;
                const uint64_t* src = DT + (has ? (uint64_t)val * PW + part % PARTS * 2 : 0);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + 16 * part), "l"(src),
                             "r"(has ? 16 : 0)
                             : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            head = head + 1 == PANEL_Q_STAGES ? 0 : head + 1;
            if (++flying == PANEL_Q_STAGES) {
                asm volatile("cp.async.wait_group %0;" ::"n"(PANEL_Q_STAGES - 1) : "memory");
                __syncwarp();                             // every lane's parts are there
                count();
            }
        };
        uint32_t fill = 0;                                // staged values (warp-uniform)
        auto push = [&](bool valid, uint32_t val) {
            const uint32_t m = __ballot_sync(0xffffffffu, valid);
            if (valid) vb[fill + __popc(m & ((1u << lane) - 1u))] = val;
            fill += __popc(m);
            __syncwarp();
            if (fill >= 32) {
                batch(vb[lane]);
                const uint32_t rest = fill - 32;
                const uint32_t carry = lane < rest ? vb[32 + lane] : 0u;
                __syncwarp();
                if (lane < rest) vb[lane] = carry;
                fill = rest;
                __syncwarp();
            }
        };
        for (uint32_t g0 = it.c_lo; g0 < it.c_hi; g0 += 32) {
            uint32_t k = 0, base = 0, len = 0;
            uint64_t off = 0;
            if (g0 + lane < it.c_hi) {
                const uint64_t c = c0 + g0 + lane;
                k = v.ckl[c];
                base = v.cid[c] << 16;
                off = v.coff[c];
                len = k & CK_BITMAP ? 0u : k & CK_LEN;
            }
            uint32_t incl = len;                          // list entries of the group's chunks up to this lane's
#pragma unroll
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
            const uint64_t origin = off - (incl - len);   // entry t of the group lies at origin + t
            auto fetch = [&](uint32_t t) -> uint32_t {
                uint32_t q = 0;                           // the first lane whose prefix is past t
#pragma unroll
                for (uint32_t o = 16; o; o >>= 1)
                    if (__shfl_sync(0xffffffffu, incl, q + o - 1) <= t) q += o;
                const uint32_t b = __shfl_sync(0xffffffffu, base, q);
                const uint64_t at = __shfl_sync(0xffffffffu, origin, q) + t;
                return t < total ? b | v.lst[at] : PANEL_NO_VALUE;
            };
            uint32_t next = fetch(lane);
            for (uint32_t t0 = 0; t0 < total; t0 += 32) {
                const uint32_t val = next;
                next = fetch(t0 + 32 + lane);
                push(val != PANEL_NO_VALUE, val);
            }
            for (uint32_t bm = __ballot_sync(0xffffffffu, (k & CK_BITMAP) != 0); bm; bm &= bm - 1) {
                const int src = __ffs(bm) - 1;
                const uint32_t b = __shfl_sync(0xffffffffu, base, src);
                const uint64_t* wd = v.bm + __shfl_sync(0xffffffffu, off, src);
                for (uint32_t q0 = 0; q0 < CHUNK_WORDS; q0 += 32) {
                    uint64_t w = wd[q0 + lane];
                    while (__any_sync(0xffffffffu, w != 0)) {
                        const bool has = w != 0;
                        const uint32_t val = has ? b | ((q0 + lane) << 6) | (uint32_t)(__ffsll((long long)w) - 1) : 0u;
                        w &= w - 1;
                        push(has, val);
                    }
                }
            }
        }
        if (fill) batch(lane < fill ? vb[lane] : PANEL_NO_VALUE);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncwarp();
        while (flying) count();
        flush();
        __syncwarp();
        uint32_t* slot = it.slot != PANEL_NO_VALUE && out ? scratch + (uint64_t)it.slot * PANEL_ROWS : nullptr;
        for (uint32_t t = lane; t < prows; t += 32) {
            const uint64_t pw = pw0 + t;
            if (pw <= xw) continue;
            const uint32_t x = cs[(t & ~63u) + ((t & 63u) ^ (t >> 6))];
            if (slot) {
                slot[t] = x;
            } else if (out) {
                const uint32_t sp = perm[pw];
                const uint64_t i = sx < sp ? sx : sp, j = sx < sp ? sp : sx;
                out[tri_index(n, i, j)] = x;
            }
            local += x;
        }
        __syncwarp();
    }
    local = warp_sum_u64(local);
    if (lane == 0 && local) atomicAdd(&flags->sum, local);
}

// The counts of every split row against the block: the sum of its items'
// slots, written into the triangle (the sum over pairs was added by the
// items).  CTA per split row, threads over the block's panel rows.
__global__ void __launch_bounds__(256)
panel_reduce_kernel(const uint32_t* __restrict__ perm, const PanelSplit* __restrict__ splits, uint32_t n_splits,
                    uint64_t pw0, uint32_t prows, const uint32_t* __restrict__ scratch, uint64_t n,
                    uint32_t* __restrict__ out) {
    for (uint32_t r = blockIdx.x; r < n_splits; r += gridDim.x) {
        const PanelSplit sp = splits[r];
        const uint64_t xw = sp.xw;
        if (xw + 1 >= pw0 + prows) continue;
        const uint32_t sx = perm[xw];
        for (uint32_t t = threadIdx.x; t < prows; t += blockDim.x) {
            const uint64_t pw = pw0 + t;
            if (pw <= xw) continue;
            uint32_t x = 0;
            for (uint32_t k = 0; k < sp.nslots; ++k) x += scratch[(uint64_t)(sp.slot0 + k) * PANEL_ROWS + t];
            const uint32_t sq = perm[pw];
            const uint64_t i = sx < sq ? sx : sq, j = sx < sq ? sq : sx;
            out[tri_index(n, i, j)] = x;
        }
    }
}

}  // namespace sb200
