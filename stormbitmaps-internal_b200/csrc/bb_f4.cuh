// bb_f4.cuh -- B x B on the 4-bit tensor pipe: tcgen05 kind::mxf4 on CTA
// pairs, operands expanded from bits TMA brought into shared memory.
//
// Arithmetic.  Bits become e2m1 values whose products are 0 or exactly 1, and
// the fp32 accumulator counts them: exact while a count is at most 2^24.  A
// nibble with one bit set is 0.5, 1 or 2 (bit 0, 1, 2), so a 32-bit word w of
// a row needs no shuffling, only masks: its expansion is four words,
//     A:  w & 1..,  w & 2..,  w & 4..,  (w >> 3) & 1..        0.5  1  2   0.5
//     B: (w << 2) & 4..,  w & 2..,  (w >> 2) & 1..,  (w >> 1) & 4..  2  1  0.5  2
// (masks repeated in every nibble), the same permutation of K on both sides.
// All scale factors are 1.  Five and seven integer operations expand 32 bits
// (an 8-bit expansion takes sixteen), into half the bytes.
//
// Shape and what bounds it.  kind::mxf4 multiplies twice as many elements per
// clock as kind::i8: a 256 x 256 tile of a CTA pair takes 1024 clocks per 512
// bits.  In that time each SM must write and read its operands in shared
// memory: raw bits in (TMA, 16 KiB) and out (16 KiB), expanded B in (32 KiB)
// and out to the tensor core (32 KiB), 768 clocks of 128 bytes.  One CTA with
// 128 x 256 tiles would need 1408, so the pair (each CTA holds half of B) is
// what lets the tensor pipe set the pace; A goes to tensor memory, which has
// its own write port.
//
// Per CTA (832 threads): warps 0-7 expand its 128 A rows into TMEM and warps
// 8-15 its 128 B rows into the swizzled ring, in two groups that take every
// other stage (one group alone needs about 1600 clocks a stage, most of it
// waiting for its own stores and fences); warp 16 loads raw bits (boxes of 512
// bits x 128 rows, one per operand), warp 17 owns TMEM and, in the even CTA of
// the pair, issues the MMAs, warps 18-25 drain the accumulator.  TMEM:
// accumulator [0, 256), three A stages of 64 columns, scale factors at 480.
// The drain warps put their counts into shared memory as 16-bit numbers, free
// the accumulator, and store them while the next tile computes; a block that
// holds a count past 65535 is read again and stored from tensor memory (its
// tile lasts long enough).  Every wait is bounded (2 s), as in the other
// tensor-core kernels.
//
// tiles[t] = (bi, bj): rows [256 bi, +256) x rows [256 bj, +256); CTA r of the
// pair takes A rows 256 bi + 128 r .. and expands B rows 256 bj + 128 r ...
#pragma once
#include <cuda.h>
#include "bb_mma_2cta.cuh"

namespace sb200 {

constexpr int F4_BM = 256;
constexpr int F4_BN = 256;
constexpr int F4_STAGE_WORDS = 8;                          // row words per stage (512 bits)
constexpr int F4_SLOTS = 4;                                // raw stages in flight
constexpr int F4_STAGES = 3;                               // expanded stages
constexpr uint32_t F4_RAW_BYTES = 128 * 64;                // 128 rows x 512 bits of one operand
constexpr uint32_t F4_ATOM_BYTES = 128 * 128;              // 128 B rows x one 128-byte K atom (256 bits)
constexpr uint32_t F4_B_STAGE_BYTES = 2 * F4_ATOM_BYTES;
constexpr uint32_t F4_EPI_WARPS = 8;
constexpr uint32_t F4_EPI_WARP_BYTES = 32 * 128 * 2;       // a warp's 32 x 128 counts of 16 bits
constexpr uint32_t F4_EPI_BYTES = F4_EPI_WARPS * F4_EPI_WARP_BYTES;
constexpr uint32_t F4_OFF_B = F4_SLOTS * 2 * F4_RAW_BYTES;
constexpr uint32_t F4_OFF_EPI = F4_OFF_B + F4_STAGES * F4_B_STAGE_BYTES;
constexpr uint32_t F4_OFF_CTL = F4_OFF_EPI + F4_EPI_BYTES;
constexpr uint32_t F4_SMEM_BYTES = F4_OFF_CTL + 256 + 1024;
constexpr int F4_B_WARP0 = 8, F4_TMA_WARP = 16, F4_MMA_WARP = 17, F4_EPI_WARP0 = 18;
constexpr int F4_THREADS = (F4_EPI_WARP0 + (int)F4_EPI_WARPS) * 32;   // 832
constexpr uint32_t F4_A_COL0 = 256, F4_SF_COL = 480;
// Longest K range one accumulator counts exactly (fp32 integers).
constexpr uint64_t F4_MAX_BITS = 1ull << 24;
static_assert(F4_SMEM_BYTES <= 232448, "shared memory of one CTA");
static_assert(F4_A_COL0 + 64 * F4_STAGES <= F4_SF_COL && F4_SF_COL + 16 <= 512, "tensor memory");

enum : uint32_t {
    ERR_F4_TMA_EMPTY = 0x501, ERR_F4_RAW_FULL = 0x502, ERR_F4_EMPTY = 0x503, ERR_F4_FULL = 0x504,
    ERR_F4_ACCFULL = 0x505, ERR_F4_ACCEMPTY = 0x506, ERR_F4_DRAIN = 0x507, ERR_F4_TMA_DRAIN = 0x508,
};

struct F4Ctl {
    uint64_t raw_full[F4_SLOTS];    // this CTA's TMA
    uint64_t raw_empty[F4_SLOTS];   // the 8 warps that expand the stage
    uint64_t full[F4_STAGES];       // leader: both CTAs' expanding warps
    uint64_t empty[F4_STAGES];      // both: the leader's commit
    uint64_t acc_full, acc_empty, drain;
    uint32_t tmem_base;
    volatile uint32_t abort;
};

// Instruction descriptor of kind::mxf4: A / B e2m1 (1) in [7,10) / [10,12),
// both K-major, N >> 3 in [17,23), scale type ue8m0 in bit 23, M >> 7 in
// [27,29), scale factor ids 0.
__host__ __device__ constexpr uint32_t f4_idesc(uint32_t m, uint32_t n) {
    return (1u << 7) | (1u << 10) | ((n >> 3) << 17) | (1u << 23) | ((m >> 7) << 27);
}

#ifdef __CUDACC__
__device__ __forceinline__ void mma_f4_pair(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                            uint32_t sf_tmem, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::mxf4.block_scale.scale_vec::2X [%0], [%1], %2, %3, [%4], [%4], p;\n\t}" ::"r"(
            d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(sf_tmem), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t x, uint32_t y, uint32_t z,
                                            uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
        : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Arrive on a barrier of either CTA of the pair.  What the arriving warp wrote
// is in this SM's shared memory (behind fence.proxy.async) or tensor memory
// (behind tcgen05.wait / fence) already and is read by the tensor core alone,
// so the default CTA scope serves: a cluster-scope release here costs a
// producer warp 1100 clocks per stage (half its time) against 60.
__device__ __forceinline__ void mbar_arrive_pair(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                 : "memory");
}

// 32 bits of an A row -> 4 words of e2m1 weights 0.5, 1, 2, 0.5.
__device__ __forceinline__ uint4 f4_expand_a(uint32_t w) {
    return make_uint4(w & 0x11111111u, w & 0x22222222u, w & 0x44444444u, (w >> 3) & 0x11111111u);
}
// ... of a B row, weights 2, 1, 0.5, 2.
__device__ __forceinline__ uint4 f4_expand_b(uint32_t w) {
    return make_uint4((w << 2) & 0x44444444u, w & 0x22222222u, (w >> 2) & 0x11111111u, (w >> 1) & 0x44444444u);
}

// CTA scope, as the arrivals (an acquire at cluster scope costs the MMA thread
// 290 clocks a stage).
__device__ __forceinline__ bool f4_wait(uint32_t bar, uint32_t parity, F4Ctl* ctl, DeviceFlags* flags, uint32_t site,
                                        bool drain = false) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = globaltimer_ns();
    for (;;) {
        if (mbar_try_wait(bar, parity)) return true;
        if (!drain && ctl->abort) return false;
        if (globaltimer_ns() - t0 > WAIT_LIMIT_NS) {
            atomicCAS(&flags->error, 0u, site);
            ctl->abort = 1;
            return false;
        }
    }
}

// Where a drain warp's counts go.
struct F4Out {
    uint32_t* out;                  // packed triangle, or null (sum only)
    uint64_t n, n_out;
    const uint32_t* row_map;
    bool partial;                   // one K segment's share: added
};

// One count to its place: stored (how 1), added (how 2), or not at all (how 0
// or !want).  Predicated, since the wanted lanes differ from row to row at the
// diagonal and a branch per count costs more than the count.
__device__ __forceinline__ void f4_put(uint32_t* dst, uint32_t v, bool want, uint32_t how) {
    asm volatile(
        "{\n\t.reg .pred st, ad;\n\t"
        "setp.eq.u32 st, %2, 1;\n\t"
        "setp.eq.u32 ad, %2, 2;\n\t"
        "@st st.global.cs.u32 [%0], %1;\n\t"
        "@ad red.global.add.u32 [%0], %1;\n\t}" ::"l"(dst),
        "r"(v), "r"(want ? how : 0u)
        : "memory");
}

// Stores a block of 32 rows x 32 NC columns from (i0, j0) on, 32 consecutive
// counts of a row per instruction: at(rr, c) is this lane's count of row rr,
// column 32 c + lane.  Returns its share of the sum over i < j.  The diagonal,
// the last rows and row maps take a branch-free loop: the drain of a launch's
// last tile is hidden by nothing, and with an index and a branch per count it
// took 12 us (100 x 1000 bits: 23 -> 15 us of kernel).
template <bool kRowMap, uint32_t NC, class At>
__device__ __forceinline__ unsigned long long f4_emit(const F4Out& o, int lane, uint64_t i0, uint64_t j0, At at) {
    if (i0 >= o.n || j0 >= o.n || i0 >= j0 + 32 * NC) return 0;
    constexpr uint32_t RB = 8 / NC;                        // rows per batch: their counts are read before any store
    const uint32_t rows = o.n - i0 < 32 ? (uint32_t)(o.n - i0) : 32u;
    const uint32_t how = !o.out ? 0u : o.partial ? 2u : 1u;
    // column col of row rr is wanted from the diagonal (lo) to the last row (cols)
    const int32_t cols = o.n - j0 < 32 * NC ? (int32_t)(o.n - j0) : (int32_t)(32 * NC);
    int32_t lo = (int64_t)i0 - (int64_t)j0 < -32 ? -32 : (int32_t)((int64_t)i0 - (int64_t)j0);
    uint32_t s = 0;                                        // at most 128 counts of at most 2^24
    // row maps: entry (a, b), a < b, is at base(a) + b, base(a) = tri_index(n, a, a) - a
    auto base = [&](uint32_t a) { return tri_index(o.n_out, a, a) - a; };
    uint32_t cm[NC], rm_l = ~0u;
    uint64_t cb[NC], rb_l = 0;
    // else: row i + 1 starts n - i entries after row i, one column later
    uint64_t step = o.n - i0 - 1;
    uint32_t* p = o.out + (tri_index(o.n, i0, i0) - i0 + j0 + lane);
    if (!kRowMap && lo + 31 < 0 && cols == (int32_t)(32 * NC) && rows == 32 && how) {   // an inner block: no tests
        if (how == 1) {
#pragma unroll 4
            for (uint32_t rr = 0; rr < 32; ++rr) {
#pragma unroll
                for (uint32_t c = 0; c < NC; ++c) {
                    const uint32_t v = at(rr, c);
                    __stcs(p + 32 * c, v);
                    s += v;
                }
                p += step--;
            }
        } else {
#pragma unroll 4
            for (uint32_t rr = 0; rr < 32; ++rr) {
#pragma unroll
                for (uint32_t c = 0; c < NC; ++c) {
                    const uint32_t v = at(rr, c);
                    atomicAdd(p + 32 * c, v);
                    s += v;
                }
                p += step--;
            }
        }
        return s;
    }
    if (kRowMap) {
#pragma unroll
        for (uint32_t c = 0; c < NC; ++c) {
            const int32_t col = (int32_t)(32 * c) + lane;
            cm[c] = col < cols ? o.row_map[j0 + col] : ~0u;
            cb[c] = cm[c] != ~0u ? base(cm[c]) : 0;
        }
        if (lane < (int)rows) rm_l = o.row_map[i0 + lane];
        if (rm_l != ~0u) rb_l = base(rm_l);
    }
#pragma unroll 1
    for (uint32_t r0 = 0; r0 < rows; r0 += RB) {
        uint32_t v[RB][NC];
#pragma unroll
        for (uint32_t q = 0; q < RB; ++q)
#pragma unroll
            for (uint32_t c = 0; c < NC; ++c) v[q][c] = at(r0 + q, c);
#pragma unroll
        for (uint32_t q = 0; q < RB; ++q, ++lo) {
            uint32_t rm = 0;
            uint64_t rb = 0;
            if (kRowMap) {
                rm = __shfl_sync(0xffffffffu, rm_l, r0 + q);
                rb = __shfl_sync(0xffffffffu, rb_l, r0 + q);
            }
            const bool row_ok = r0 + q < rows && (!kRowMap || rm != ~0u);
#pragma unroll
            for (uint32_t c = 0; c < NC; ++c) {
                const int32_t col = (int32_t)(32 * c) + lane;
                const bool want = row_ok && col >= lo && col < cols && (!kRowMap || cm[c] != ~0u);
                uint32_t* dst = kRowMap ? o.out + (rm < cm[c] ? rb + cm[c] : cb[c] + rm) : p + 32 * c;
                f4_put(dst, v[q][c], want, how);
                s += want && col > lo ? v[q][c] : 0u;
            }
            p += step--;
        }
    }
    return s;
}

// A 32 x 32 block of counts held lane = row i0 + lane, r[c] = column j0 + c:
// through the warp's shared-memory block (16-byte chunks XOR-swizzled by row).
template <bool kRowMap>
__device__ __forceinline__ unsigned long long f4_store_block(const F4Out& o, uint32_t* buf, int lane, uint64_t i0,
                                                             uint64_t j0, const uint32_t (&r)[32]) {
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k)
        *reinterpret_cast<uint4*>(buf + lane * 32 + ((k ^ (lane & 7)) << 2)) =
            make_uint4(r[4 * k], r[4 * k + 1], r[4 * k + 2], r[4 * k + 3]);
    __syncwarp();
    const unsigned long long local = f4_emit<kRowMap, 1>(o, lane, i0, j0, [&](uint32_t rr, uint32_t) {
        return buf[rr * 32 + ((((uint32_t)lane >> 2) ^ (rr & 7)) << 2) + (lane & 3)];
    });
    __syncwarp();
    return local;
}

// Columns 32 c .. of a warp's 32 x 128 counts (fp32 whole numbers, lane = row)
// as 16-bit numbers, 256 bytes per row, 16-byte chunks XOR-swizzled by row.
// x + 2^23 holds x in its low bits.  Returns the largest count.
__device__ __forceinline__ float f4_pack_block(uint32_t* buf, int lane, uint32_t c, const uint32_t (&r)[32]) {
    uint32_t pk[16];
#pragma unroll
    for (uint32_t k = 0; k < 16; ++k)
        pk[k] = __byte_perm(__float_as_uint(__uint_as_float(r[2 * k]) + 8388608.0f),
                            __float_as_uint(__uint_as_float(r[2 * k + 1]) + 8388608.0f), 0x5410);
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k)
        *reinterpret_cast<uint4*>(buf + lane * 64 + (((4 * c + k) ^ ((uint32_t)lane & 7u)) << 2)) =
            make_uint4(pk[4 * k], pk[4 * k + 1], pk[4 * k + 2], pk[4 * k + 3]);
    float most = 0.0f;
#pragma unroll
    for (uint32_t k = 0; k < 32; ++k) most = fmaxf(most, __uint_as_float(r[k]));
    return most;
}

// The packed 32 x 128 block to its places.
template <bool kRowMap>
__device__ __forceinline__ unsigned long long f4_store_packed(const F4Out& o, const uint32_t* buf, int lane,
                                                              uint64_t i0, uint64_t j0) {
    __syncwarp();
    const uint16_t* h = reinterpret_cast<const uint16_t*>(buf);
    const unsigned long long local = f4_emit<kRowMap, 4>(o, lane, i0, j0, [&](uint32_t rr, uint32_t c) {
        const uint32_t col = 32u * c + (uint32_t)lane;
        return (uint32_t)h[rr * 128 + (((col >> 3) ^ (rr & 7)) << 3) + (col & 7)];
    });
    __syncwarp();
    return local;
}

template <bool kRowMap, bool kThresh>
__device__ __forceinline__ void f4_body(const CUtensorMap& map, uint32_t blk_words, uint32_t n, uint32_t w_pad,
                                        const uint2* __restrict__ tiles, uint32_t n_tiles,
                                        uint32_t* __restrict__ out, DeviceFlags* __restrict__ flags,
                                        const uint32_t* __restrict__ row_map, uint64_t n_out, uint32_t k_splits,
                                        TsThresh th = TsThresh{}) {
    extern __shared__ __align__(1024) unsigned char f4_smem[];
    const uint32_t raw_addr = smem_u32(f4_smem);
    const uint32_t pad = ((raw_addr + 1023u) & ~1023u) - raw_addr;   // the same in both CTAs
    const uint32_t base = raw_addr + pad;
    F4Ctl* ctl = reinterpret_cast<F4Ctl*>(f4_smem + pad + F4_OFF_CTL);
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_ctarank();
    const uint32_t cid = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
    const uint32_t nk = w_pad / F4_STAGE_WORDS;               // stages of a whole row (w_pad % 8 == 0)

    if (tid == 0) {
        for (int s = 0; s < F4_SLOTS; ++s) {
            mbar_init(smem_u32(&ctl->raw_full[s]), 1);
            mbar_init(smem_u32(&ctl->raw_empty[s]), 8);
        }
        for (int s = 0; s < F4_STAGES; ++s) {
            mbar_init(smem_u32(&ctl->full[s]), 16);
            mbar_init(smem_u32(&ctl->empty[s]), 1);
        }
        mbar_init(smem_u32(&ctl->acc_full), 1);
        mbar_init(smem_u32(&ctl->acc_empty), 2 * F4_EPI_WARPS);
        mbar_init(smem_u32(&ctl->drain), 1);
        ctl->abort = 0;
        fence_barrier_init();
    }
    if (warp == F4_MMA_WARP) {
        tmem_alloc_pair(smem_u32(&ctl->tmem_base), 512);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    cluster_sync_all();            // barriers initialised in both CTAs before any remote arrival
    tc_fence_after();
    const uint32_t tmem_base = ctl->tmem_base;
    TsSched sched(nk, n_tiles, k_splits, cid, n_clusters);
    uint32_t t, kb0, kb1;
    bool partial;

    if (warp < F4_TMA_WARP) {
        // ---- expand A rows into TMEM, B rows into the ring; every other stage
        const bool is_a = warp < F4_B_WARP0;
        const uint32_t grp = (uint32_t)(warp >> 2) & 1u;
        const uint32_t row = (uint32_t)(tid & 127);
        const uint32_t lane_base = tmem_base + ((uint32_t)(warp & 3) * 32u << 16);
        const uint32_t lead_full0 = mapa_shared(smem_u32(&ctl->full[0]), 0);
        const uint32_t src0 = base + (is_a ? 0u : F4_RAW_BYTES) + row * 64u;
        const uint32_t dst0 = base + F4_OFF_B + (row >> 3) * 1024u + (row & 7u) * 128u;
        if (warp < 4) {            // scale factors: ue8m0 1.0 everywhere
            uint32_t one[16];
#pragma unroll
            for (int k = 0; k < 16; ++k) one[k] = 0x7F7F7F7Fu;
            tmem_st_32x32b_x16(lane_base + F4_SF_COL, one);
            tmem_st_wait();
        }
        uint32_t g = 0;            // stages before this segment
        bool ok = true;
        while (ok && sched.next(t, kb0, kb1, partial)) {
            const uint32_t g1 = g + (kb1 - kb0);
            for (uint32_t gs = g + ((g ^ grp) & 1u); gs < g1; gs += 2) {
                const uint32_t slot = gs % F4_SLOTS, s = gs % F4_STAGES;
                if (!f4_wait(smem_u32(&ctl->raw_full[slot]), (gs / F4_SLOTS) & 1, ctl, flags, ERR_F4_RAW_FULL)) {
                    ok = false;
                    break;
                }
                const uint32_t src = src0 + slot * (2 * F4_RAW_BYTES);
                uint4 v[4];        // 64-byte swizzle: chunk q of row r lies at q ^ ((r / 2) % 4)
#pragma unroll
                for (uint32_t q = 0; q < 4; ++q) v[q] = lds128(src + ((q ^ ((row >> 1) & 3u)) << 4));
                if (!f4_wait(smem_u32(&ctl->empty[s]), ((gs / F4_STAGES) & 1) ^ 1, ctl, flags, ERR_F4_EMPTY)) {
                    ok = false;
                    break;
                }
                if (is_a) {
                    tc_fence_after();
                    const uint32_t taddr = lane_base + F4_A_COL0 + 64u * s;
#pragma unroll
                    for (uint32_t q = 0; q < 4; q += 2) {
                        uint32_t r[32];
#pragma unroll
                        for (uint32_t e = 0; e < 2; ++e) {
                            const uint32_t w[4] = {v[q + e].x, v[q + e].y, v[q + e].z, v[q + e].w};
#pragma unroll
                            for (uint32_t k = 0; k < 4; ++k) {
                                const uint4 x = f4_expand_a(w[k]);
                                uint32_t* o = r + 16 * e + 4 * k;
                                o[0] = x.x;
                                o[1] = x.y;
                                o[2] = x.z;
                                o[3] = x.w;
                            }
                        }
                        tmem_st_32x32b_x32(taddr + 16u * q, r);
                    }
                    tmem_st_wait();
                    tc_fence_before();
                } else {
                    const uint32_t dst = dst0 + s * F4_B_STAGE_BYTES;
#pragma unroll
                    for (uint32_t q = 0; q < 4; ++q) {
                        const uint32_t w[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
#pragma unroll
                        for (uint32_t k = 0; k < 4; ++k) {
                            const uint32_t c = 4 * (q & 1) + k;          // 16-byte chunk within the atom
                            sts128(dst + (q >> 1) * F4_ATOM_BYTES + ((c ^ (row & 7u)) << 4), f4_expand_b(w[k]));
                        }
                    }
                    fence_proxy_async_smem();
                }
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive_pair(lead_full0 + 8u * s);
                    mbar_arrive(smem_u32(&ctl->raw_empty[slot]));
                }
            }
            g = g1;
        }
    } else if (warp == F4_TMA_WARP) {
        if (lane == 0) {
            uint32_t u = 0;
            bool ok = true;
            while (ok && sched.next(t, kb0, kb1, partial)) {
                const uint32_t ra = tiles[t].x * F4_BM + 128u * rank, rb = tiles[t].y * F4_BN + 128u * rank;
                for (uint32_t kb = kb0; kb < kb1; ++kb, ++u) {
                    const uint32_t slot = u % F4_SLOTS;
                    if (!f4_wait(smem_u32(&ctl->raw_empty[slot]), ((u / F4_SLOTS) & 1) ^ 1, ctl, flags,
                                        ERR_F4_TMA_EMPTY)) {
                        ok = false;
                        break;
                    }
                    const uint32_t bar = smem_u32(&ctl->raw_full[slot]);
                    const uint32_t dst = base + slot * (2 * F4_RAW_BYTES);
                    const uint32_t word = kb * F4_STAGE_WORDS;
                    const uint32_t z = blk_words ? word / blk_words : 0u;
                    const uint32_t x = 2u * (word - z * blk_words);
                    mbar_expect_tx(bar, 2 * F4_RAW_BYTES);
                    tma_load_3d(dst, &map, x, ra, z, bar);
                    tma_load_3d(dst + F4_RAW_BYTES, &map, x, rb, z, bar);
                }
            }
            // No copy may still be in flight when the CTA ends, on an abort too.
            for (uint32_t k = u > F4_SLOTS ? u - F4_SLOTS : 0; k < u; ++k)
                f4_wait(smem_u32(&ctl->raw_full[k % F4_SLOTS]), (k / F4_SLOTS) & 1, ctl, flags,
                               ERR_F4_TMA_DRAIN, true);
        }
        __syncwarp();
    } else if (warp == F4_MMA_WARP) {
        if (lane == 0) {
            uint32_t g = 0, tc = 0;
            bool issued = false;
            if (rank == 0) {
                const uint32_t idesc = f4_idesc(F4_BM, F4_BN);
                bool ok = true;
                for (; ok && sched.next(t, kb0, kb1, partial); ++tc) {
                    if (!f4_wait(smem_u32(&ctl->acc_empty), (tc & 1) ^ 1, ctl, flags, ERR_F4_ACCEMPTY)) break;
                    tc_fence_after();
                    for (uint32_t kb = kb0; kb < kb1; ++kb, ++g) {
                        const uint32_t s = g % F4_STAGES;
                        if (!f4_wait(smem_u32(&ctl->full[s]), (g / F4_STAGES) & 1, ctl, flags, ERR_F4_FULL)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        const uint32_t b_addr = base + F4_OFF_B + s * F4_B_STAGE_BYTES;
                        const uint32_t a_col = tmem_base + F4_A_COL0 + 64u * s;
#pragma unroll
                        for (uint32_t kk = 0; kk < 8; ++kk)
                            mma_f4_pair(tmem_base, a_col + 8u * kk,
                                        umma_desc_sw128(b_addr + (kk >> 2) * F4_ATOM_BYTES + (kk & 3) * 32u, 1024),
                                        idesc, tmem_base + F4_SF_COL, (kb != kb0 || kk != 0) ? 1u : 0u);
                        issued = true;
                        tc_commit_pair(smem_u32(&ctl->empty[s]), 0x3);
                    }
                    if (ok) tc_commit_pair(smem_u32(&ctl->acc_full), 0x3);
                }
                if (issued) tc_commit_pair(smem_u32(&ctl->drain), 0x3);
            } else {
                issued = sched.next(t, kb0, kb1, partial);
            }
            // Both CTAs: the pair's MMAs have completed before tensor memory is freed.
            if (issued) f4_wait(smem_u32(&ctl->drain), 0, ctl, flags, ERR_F4_DRAIN, true);
        }
        __syncwarp();
    } else {
        // ---- drain: TMEM lanes 32 (warp % 4) .., 128 columns
        const uint32_t e = (uint32_t)warp - F4_EPI_WARP0;
        uint32_t* buf = reinterpret_cast<uint32_t*>(f4_smem + pad + F4_OFF_EPI + e * F4_EPI_WARP_BYTES);
        const uint32_t lane_grp = (uint32_t)(warp & 3) * 32u, col0 = (e >> 2) * 128u;
        const uint32_t tacc = tmem_base + (lane_grp << 16) + col0;
        const uint32_t lead_acc_empty = mapa_shared(smem_u32(&ctl->acc_empty), 0);
        F4Out o{out, n, n_out, row_map, false};
        unsigned long long total = 0;
        for (uint32_t tc = 0; sched.next(t, kb0, kb1, partial); ++tc) {
            if (!f4_wait(smem_u32(&ctl->acc_full), tc & 1, ctl, flags, ERR_F4_ACCFULL)) break;
            tc_fence_after();
            const uint64_t i0 = (uint64_t)tiles[t].x * F4_BM + 128u * rank + lane_grp;
            const uint64_t j0 = (uint64_t)tiles[t].y * F4_BN + col0;
            o.partial = partial;
            bool packed = !kThresh;
            if (packed) {
                float most = 0.0f;
#pragma unroll 1
                for (uint32_t c = 0; c < 4; ++c) {
                    uint32_t r[32];
                    tmem_ld_32x32b_x32(tacc + 32u * c, r);
                    tmem_ld_wait();
                    most = fmaxf(most, f4_pack_block(buf, lane, c, r));
                }
                packed = !__any_sync(0xffffffffu, most >= 65536.0f);
            }
            if (packed) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_pair(lead_acc_empty);
                total += f4_store_packed<kRowMap>(o, buf, lane, i0, j0);
            } else {
                // The packed rows lie 64 words apart and f4_store_block's 32, so a
                // lane's 32-bit counts go where another lane just put packed ones:
                // those stores are ordered before them (a vote orders no memory).
                __syncwarp();
#pragma unroll 1
                for (uint32_t c = 0; c < 4; ++c) {
                    uint32_t r[32];
                    tmem_ld_32x32b_x32(tacc + 32u * c, r);
                    tmem_ld_wait();
#pragma unroll
                    for (uint32_t k = 0; k < 32; ++k) r[k] = __float2uint_rz(__uint_as_float(r[k]));
                    if constexpr (kThresh) {
                        // whole tiles only (no partial segments).  v / (ci + cj - v) >= t
                        // needs v (1 + t) >= t (ci + cj): an fp32 test with 2^-16 to
                        // spare picks the candidates, the exact one in double
                        // precision decides them (nearly every pair fails the first).
                        const uint64_t i = i0 + lane, jb = j0 + 32u * c;
                        const bool row_ok = i < n;
                        const uint32_t card_i = row_ok ? th.card[i] : 0u;
                        const uint32_t card_j = jb + lane < n ? th.card[jb + lane] : 0u;
                        const float tt = (float)th.t;
                        const float ti = tt * (float)card_i, tj_own = tt * (float)card_j;
                        const float scale = (1.0f + tt) * 1.0000153f;
                        const int64_t q0 = (int64_t)i - (int64_t)jb, q1 = (int64_t)n - (int64_t)jb;   // i < j < n
                        uint32_t cand = 0;
#pragma unroll
                        for (int q = 0; q < 32; ++q) {
                            const float tj = __shfl_sync(0xffffffffu, tj_own, q);
                            const bool in = row_ok && q > q0 && q < q1 && r[q] != 0;
                            if (in) total += r[q];
                            if (in && (!(th.t > 0.0) || !((float)r[q] * scale < ti + tj))) cand |= 1u << q;
                        }
                        const uint32_t some = __reduce_or_sync(0xffffffffu, cand);
                        if (some) {
#pragma unroll
                            for (int q = 0; q < 32; ++q) {
                                if (!(some >> q & 1u)) continue;
                                const uint32_t cj = __shfl_sync(0xffffffffu, card_j, q);
                                bool pass = false;
                                if (cand >> q & 1u) {
                                    const double un = (double)card_i + (double)cj - (double)r[q];
                                    pass = un > 0.0 && (double)r[q] / un >= th.t;
                                }
                                const uint32_t m = __ballot_sync(0xffffffffu, pass);
                                if (!m) continue;
                                const int first = __ffs(m) - 1;
                                unsigned long long b0 = 0;
                                if (lane == first) b0 = atomicAdd(th.found, (unsigned long long)__popc(m));
                                b0 = __shfl_sync(0xffffffffu, b0, first);
                                if (pass) {
                                    const unsigned long long k = b0 + __popc(m & ((1u << lane) - 1u));
                                    if (k < th.cap) {
                                        th.pairs[k] = make_uint2((uint32_t)i, (uint32_t)(jb + q));
                                        th.cnts[k] = r[q];
                                    }
                                }
                            }
                        }
                    } else {
                        total += f4_store_block<kRowMap>(o, buf, lane, i0, j0 + 32u * c, r);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_pair(lead_acc_empty);
            }
        }
        total = warp_sum_u64(total);
        if (lane == 0 && total) atomicAdd(&flags->sum, total);
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();            // neither CTA leaves while the other can still signal it
    if (warp == F4_MMA_WARP) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

// k_splits: the work schedule over the pairs of CTAs (TsSched; its units are
// stages of 512 bits). For any value but 1 partial counts are added into
// out (zeroed beforehand).
__global__ void __launch_bounds__(F4_THREADS, 1)
bb_f4_kernel(const __grid_constant__ CUtensorMap map, uint32_t blk_words, uint32_t n, uint32_t w_pad,
             const uint2* __restrict__ tiles, uint32_t n_tiles, uint32_t* __restrict__ out,
             DeviceFlags* __restrict__ flags, uint32_t k_splits) {
    f4_body<false, false>(map, blk_words, n, w_pad, tiles, n_tiles, out, flags, nullptr, 0, k_splits);
}

// Over a gathered subset of rows, writing into the triangle of the full row
// set through row_map.
__global__ void __launch_bounds__(F4_THREADS, 1)
bb_f4_rows_kernel(const __grid_constant__ CUtensorMap map, uint32_t blk_words, uint32_t n, uint32_t w_pad,
                  const uint2* __restrict__ tiles, uint32_t n_tiles, uint32_t* __restrict__ out,
                  DeviceFlags* __restrict__ flags, uint32_t k_splits, const uint32_t* __restrict__ row_map,
                  uint64_t n_out) {
    f4_body<true, false>(map, blk_words, n, w_pad, tiles, n_tiles, out, flags, row_map, n_out, k_splits);
}

// Thresholded form (whole tiles round robin).
__global__ void __launch_bounds__(F4_THREADS, 1)
bb_f4_thresh_kernel(const __grid_constant__ CUtensorMap map, uint32_t blk_words, uint32_t n, uint32_t w_pad,
                    const uint2* __restrict__ tiles, uint32_t n_tiles, DeviceFlags* __restrict__ flags, TsThresh th) {
    f4_body<false, true>(map, blk_words, n, w_pad, tiles, n_tiles, nullptr, flags, nullptr, 0, 1u, th);
}
#endif

}  // namespace sb200
