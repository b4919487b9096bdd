// dense.cu -- launchers for the B x B kernels (POPC and tcgen05).
#include "dense.cuh"
#include "bb_popc.cuh"
#include "bb_mma.cuh"
#include "bb_mma_ts.cuh"
#include "bb_mma_ts2.cuh"
#include "bb_mma_2cta.cuh"
#include "bb_f4.cuh"
#include "colsum.cuh"

#include <algorithm>
#include <mutex>

namespace sb200 {

// Work schedule of the 8-bit tensor-core kernels (TsSched in bb_mma_ts.cuh),
// rows of more than 2^24 bits: whole tiles round robin when the last wave is
// nearly full (>= 98.5 %), else the first floor(tiles / grid) waves as whole
// tiles and stream-K over the (tile, K stage) space of the rest, at least 32
// stages per CTA. The line was measured at 2^18-bit rows (B200, stream-K over
// every tile): 136 tiles 1.9x faster, 272 8 %, 1088 (92 % fill) 7 %, 4160 (97 %)
// 3 %; longer rows only make a segment's fixed cost smaller. Returns the kernel's
// k_splits argument (1 or 0) and sets the grid.
static uint32_t ts_schedule(uint32_t n_tiles, int sms, uint32_t w_pad, uint32_t& grid,
                            int pref = STORM_B200_SCHED_AUTO) {
    const uint64_t nk = w_pad / (TS_KBITS / 64);
    const uint64_t waves = ((uint64_t)n_tiles + sms - 1) / sms;
    const double fill = waves ? (double)n_tiles / (double)(waves * (uint64_t)sms) : 1.0;
    const bool tiles = pref == STORM_B200_SCHED_TILES || (pref == STORM_B200_SCHED_AUTO && fill >= 0.985);
    if (tiles) {
        grid = n_tiles < (uint32_t)sms ? n_tiles : (uint32_t)sms;
        return 1;
    }
    grid = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)sms, (uint64_t)n_tiles * nk / 32));
    return 0;
}

// The tensor-core kernel a row length runs on: up to 2^24 bits the 4-bit one
// (its fp32 accumulator counts exactly that far), longer rows the 8-bit ones.
// Measured on B200, 8-bit -> 4-bit (ms): 65536 x 2^18 bits 346 -> 177, 50000 x
// 20000 18.5 -> 8.2, 4096 x 65536 0.45 -> 0.20, 100 x 1000 the same.
static int exec_kind(int kind, uint64_t row_bits) {
    return (kind == STORM_B200_KERNEL_MMA || kind == STORM_B200_KERNEL_MMA_DB) && row_bits <= F4_MAX_BITS ? KIND_F4
                                                                                                           : kind;
}

bool same_kernel(int a, int b, uint64_t row_bits) { return exec_kind(a, row_bits) == exec_kind(b, row_bits); }

constexpr uint32_t F4_MIN_SEG = 8;   // stages of a K segment at least

// Schedule of the 4-bit kernel over `pairs` pairs of CTAs, as ts_schedule:
// stream-K when the last wave would be under 98.5 % full and a tile has 64
// stages (32768 bits), and whenever less than half of the pairs have a tile.
// Measured on B200, whole tiles / stream-K (us of kernel): 78 tiles of 65536
// bits 177 / 111, 136 tiles 175 / 175, 528 tiles 654 / 592, 136 tiles of
// 20000 bits 71 / 77, 10 tiles of 20000 bits 47 / 26.  Segments of at least 8
// stages: 3 tiles of 40 stages take 25 us so, 33 with 16 and 40 with 32; with
// 4, 10 such tiles take 36 against 28.
static uint32_t f4_schedule(uint32_t n_tiles, int sms, uint32_t w_pad, uint32_t& pairs,
                            int pref = STORM_B200_SCHED_AUTO) {
    const uint32_t np = std::max(1, sms / 2);
    const uint64_t nk = w_pad / F4_STAGE_WORDS;
    const uint64_t waves = ((uint64_t)n_tiles + np - 1) / np;
    const double fill = waves ? (double)n_tiles / (double)(waves * np) : 1.0;
    const bool tiles = pref == STORM_B200_SCHED_TILES ||
                       (pref == STORM_B200_SCHED_AUTO && (fill >= 0.985 || nk < 64) && n_tiles * 2 > np);
    if (tiles) {
        pairs = std::min(n_tiles, np);
        return 1;
    }
    pairs = (uint32_t)std::min<uint64_t>(np, std::max<uint64_t>(n_tiles, (uint64_t)n_tiles * nk / F4_MIN_SEG));
    return 0;
}

// Tensor map of device rows for the 4-bit kernel: 32-bit elements, boxes of
// 512 bits x 128 rows with a 64-byte swizzle; row-major rows in two
// dimensions (what lies past the row's words reads as zero), block-major
// panels with the 1024-word block as the third.  blk_words: words per block,
// 0 for row-major rows.
static CUtensorMap f4_row_map(const uint64_t* X, uint64_t n, uint32_t w_pad, RowLayout lay, uint32_t* blk_words) {
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                               const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                               CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return (Encode)f;
    }();
    if (!encode) fail(STORM_B200_ECUDA, "cuTensorMapEncodeTiled is not available");
    const bool blocked = lay.kstride != 1024;
    *blk_words = blocked ? 1024u : 0u;
    const cuuint64_t dims[3] = {blocked ? 2048u : 2ull * w_pad, n, blocked ? (w_pad + 1023u) / 1024u : 1u};
    const cuuint64_t strides[2] = {lay.pitch * 8, blocked ? lay.kstride * 8 : lay.pitch * 8};
    const cuuint32_t box[3] = {16, 128, 1}, one[3] = {1, 1, 1};
    CUtensorMap m;
    if (encode(&m, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, (void*)X, dims, strides, box, one,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        fail(STORM_B200_ECUDA, "tensor map of the rows");
    return m;
}

// Launch of a kernel on `pairs` clusters of two CTAs.
template <class... P, class... A>
static cudaError_t launch_pairs(void (*kernel)(P...), uint32_t pairs, uint32_t threads, uint32_t smem, cudaStream_t st,
                                A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs, 1, 1);
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Rows per A block and per B block of a kernel's tiles.
uint64_t tile_rows_a(int kind) {
    return kind == STORM_B200_KERNEL_POPC       ? POPC_BM
           : kind == KIND_F4                    ? F4_BM
           : kind == STORM_B200_KERNEL_MMA_2CTA ? C2_BM
                                                : MMA_BM;
}
uint64_t tile_rows_b(int kind) {
    return kind == STORM_B200_KERNEL_POPC     ? POPC_BM
           : kind == STORM_B200_KERNEL_MMA_DB ? T2_BN
           : kind == KIND_F4                  ? F4_BN
           : kind == STORM_B200_KERNEL_MMA_2CTA ? C2_BN
                                                : MMA_BN;
}

void build_tiles(std::vector<uint2>& t, uint64_t n, int kind) {
    t.clear();
    // tile indices and counts are 32-bit (the kernels' work lists); bound the
    // count by the full block grid before building anything
    const uint64_t bm = tile_rows_a(kind), bn = tile_rows_b(kind);
    if (((n + bm - 1) / bm) * ((n + bn - 1) / bn) > 0xFFFFFFFFull)
        fail(STORM_B200_ELIMIT, "more than 2^32 tiles: split the rows into several containers");
    static_assert(F4_BM == C2_BM && F4_BN == C2_BN, "both pair kernels use 256 x 256 tiles");
    if (kind == STORM_B200_KERNEL_MMA_2CTA || kind == KIND_F4) {
        const uint64_t nb = (n + C2_BM - 1) / C2_BM;
        for (uint64_t bi = 0; bi < nb; ++bi)
            for (uint64_t bj = bi; bj < nb; ++bj) t.push_back(make_uint2((uint32_t)bi, (uint32_t)bj));
    } else if (kind == STORM_B200_KERNEL_MMA || kind == STORM_B200_KERNEL_MMA_SS) {
        const uint64_t nbi = (n + MMA_BM - 1) / MMA_BM, nbj = (n + MMA_BN - 1) / MMA_BN;
        // Tile (bi, bj) holds a pair with i <= j iff 128 bi <= 256 bj + 255,
        // i.e. bj >= floor(bi / 2).
        for (uint64_t bi = 0; bi < nbi; ++bi)
            for (uint64_t bj = bi / 2; bj < nbj; ++bj) t.push_back(make_uint2((uint32_t)bi, (uint32_t)bj));
    } else if (kind == STORM_B200_KERNEL_MMA_DB) {
        const uint64_t nbi = (n + T2_BM - 1) / T2_BM, nbj = (n + T2_BN - 1) / T2_BN;
        // 128 bi <= 192 bj + 191  <=>  bj >= floor(128 bi / 192)
        for (uint64_t bi = 0; bi < nbi; ++bi)
            for (uint64_t bj = (128 * bi) / 192; bj < nbj; ++bj) t.push_back(make_uint2((uint32_t)bi, (uint32_t)bj));
    } else {
        const uint64_t nb = (n + POPC_BM - 1) / POPC_BM;
        for (uint64_t bi = 0; bi < nb; ++bi)
            for (uint64_t bj = bi; bj < nb; ++bj) t.push_back(make_uint2((uint32_t)bi, (uint32_t)bj));
    }
}

// Automatic choice: tensor cores up to 2^27-bit rows, CUDA-core POPC beyond. Both
// tensor-core names run the 4-bit kernel up to 2^24 bits; which of them a call
// reports there changes at 2^17.
constexpr uint64_t DB_AUTO_MAX_BITS = 1ull << 17;

static int auto_kind(uint64_t row_bits) {
    return row_bits <= DB_AUTO_MAX_BITS   ? STORM_B200_KERNEL_MMA_DB
           : row_bits <= MMA_MAX_BITS_W4 ? STORM_B200_KERNEL_MMA
                                         : STORM_B200_KERNEL_POPC;
}

// A 256 x 256 tile list in bands of F4_BAND A blocks, down each band's columns:
// the tiles that run at one time then read about as many A blocks as B blocks
// (8 + 9 for the 74 CTA pairs) instead of one A block and 74 B blocks, and the
// rows they share come from L2.
constexpr uint32_t F4_BAND = 8;

void band_tiles(std::vector<uint2>& t) {
    std::stable_sort(t.begin(), t.end(), [](const uint2& a, const uint2& b) {
        const uint32_t ba = a.x / F4_BAND, bb = b.x / F4_BAND;
        return ba != bb ? ba < bb : a.y != b.y ? a.y < b.y : a.x < b.x;
    });
}

int DenseEngine::prepare(uint64_t n, uint64_t row_bits, int kernel_pref, bool rows_in_order, cudaStream_t st) {
    if (n > 0xFFFFFFFFull) fail(STORM_B200_ELIMIT, "more than 2^32 rows");
    int kind = kernel_pref;
    if (kind == STORM_B200_KERNEL_AUTO) kind = auto_kind(row_bits);
    if ((kind == STORM_B200_KERNEL_MMA || kind == STORM_B200_KERNEL_MMA_DB || kind == STORM_B200_KERNEL_MMA_2CTA) &&
        row_bits > MMA_MAX_BITS_W4)
        fail(STORM_B200_ELIMIT, "tensor-core kernel is exact only for rows of at most 2^27 bits");
    if (kind == STORM_B200_KERNEL_MMA_SS && row_bits > MMA_MAX_BITS)
        fail(STORM_B200_ELIMIT, "shared-memory tensor-core kernel is exact only for rows of at most 2^23 bits");
    reported = kind;
    kind = exec_kind(kind, row_bits);
    const bool banded = kind == KIND_F4 && !rows_in_order;
    if (tiles_n != n || tiles_kind != kind || tiles_banded != banded) {
        build_tiles(h_tiles, n, kind);
        if (banded) band_tiles(h_tiles);
        d_tiles.reserve(h_tiles.size());
        SB_CUDA(cudaMemcpyAsync(d_tiles.p, h_tiles.data(), h_tiles.size() * sizeof(uint2), cudaMemcpyHostToDevice,
                                st));
        n_tiles = (uint32_t)h_tiles.size();
        tiles_n = n;
        tiles_kind = kind;
        tiles_banded = banded;
    }
    d_flags.reserve(1);
    SB_CUDA(cudaMemsetAsync(d_flags.p, 0, sizeof(DeviceFlags), st));
    log.ensure();
    return kind;
}

// Stream-K over tiles [t0, t1) of the cached list, which hold every tile of
// their A blocks (TsSched, k_splits 0): tiles from W = t0 + floor(tiles / grid)
// x grid on add into the output: the triangle is zeroed from the first row of
// the lowest A block among them to the last row of the highest.
void DenseEngine::zero_stream_k_rows(uint32_t* d_out, uint32_t n, uint32_t t0, uint32_t t1, uint32_t grid,
                                     cudaStream_t st) {
    const uint32_t whole = t0 + (t1 - t0) / grid * grid;
    if (whole >= t1) return;
    uint32_t lowest = h_tiles[whole].x, highest = lowest;
    for (uint32_t t = whole; t < t1; ++t) {
        lowest = std::min(lowest, h_tiles[t].x);
        highest = std::max(highest, h_tiles[t].x);
    }
    const uint64_t bm = tile_rows_a(tiles_kind);
    const uint64_t r0 = lowest * bm, r1 = std::min<uint64_t>(n, (highest + 1) * bm);
    auto start = [n](uint64_t r) { return r * n - r * (r - (r > 0)) / 2; };   // tri_index(n, r, r)
    SB_CUDA(cudaMemsetAsync(d_out + start(r0), 0, (start(r1) - start(r0)) * sizeof(uint32_t), st));
}

// Tiles [t0, t0 + count) of the cached list.
void DenseEngine::launch(int kind, const uint64_t* dX, uint32_t n, uint32_t w_pad, uint32_t t0, uint32_t count,
                         uint32_t* d_out, cudaStream_t st) {
    const int sms = require_device();
    if (count == 0) return;
    const RowLayout lay = row_major(dense_pitch(w_pad));
    // stream-K only for a launch that holds every tile of its A blocks: its rows
    // of the triangle can be zeroed first for the partial-count atomics
    const bool whole_list = t0 == 0 && count == n_tiles;
    const bool whole_blocks = (t0 == 0 || h_tiles[t0 - 1].x != h_tiles[t0].x) &&
                              (t0 + count == n_tiles || h_tiles[t0 + count].x != h_tiles[t0 + count - 1].x);
    if (kind == KIND_F4) {
        static std::atomic<uint64_t> done{0};
        smem_attr_once(bb_f4_kernel, (int)F4_SMEM_BYTES, done);
        uint32_t pairs = std::min<uint32_t>(count, (uint32_t)std::max(1, sms / 2));
        const uint32_t ks =
            whole_list || (whole_blocks && !tiles_banded) ? f4_schedule(count, sms, w_pad, pairs, schedule) : 1;
        if (ks != 1 && d_out) zero_stream_k_rows(d_out, n, t0, t0 + count, pairs, st);
        uint32_t blk_words = 0;
        const CUtensorMap map = f4_row_map(dX, n, w_pad, lay, &blk_words);
        SB_CUDA(launch_pairs(bb_f4_kernel, pairs, F4_THREADS, F4_SMEM_BYTES, st, map, blk_words, n, w_pad,
                             (const uint2*)(d_tiles.p + t0), count, d_out, d_flags.p, ks));
    } else if (kind == STORM_B200_KERNEL_MMA) {
        static std::atomic<uint64_t> done{0};
        smem_attr_once(bb_mma_ts_long_kernel, (int)TS_SMEM_BYTES, done);
        uint32_t grid = count < (uint32_t)sms ? count : (uint32_t)sms;
        const uint32_t ks = whole_list ? ts_schedule(count, sms, w_pad, grid, schedule) : 1;
        if (ks != 1 && d_out) zero_stream_k_rows(d_out, n, t0, t0 + count, grid, st);
        bb_mma_ts_long_kernel<<<grid, TS_THREADS, TS_SMEM_BYTES, st>>>(dX, n, w_pad, lay, d_tiles.p + t0, count,
                                                                            d_out, d_flags.p, ks);
    } else if (kind == STORM_B200_KERNEL_MMA_DB) {
        static std::atomic<uint64_t> done{0};
        smem_attr_once(bb_mma_ts2_long_kernel, (int)T2_SMEM_BYTES, done);
        uint32_t grid = count < (uint32_t)sms ? count : (uint32_t)sms;
        const uint32_t ks = whole_list ? ts_schedule(count, sms, w_pad, grid, schedule) : 1;
        if (ks != 1 && d_out) zero_stream_k_rows(d_out, n, t0, t0 + count, grid, st);
        bb_mma_ts2_long_kernel<<<grid, T2_THREADS, T2_SMEM_BYTES, st>>>(dX, n, w_pad, lay, d_tiles.p + t0, count,
                                                                       d_out, d_flags.p, ks);
    } else if (kind == STORM_B200_KERNEL_MMA_2CTA) {
        // CTA pairs (clusters of 2), one per two SMs, whole tiles round robin
        static std::atomic<uint64_t> done_a{0}, done_b{0};
        smem_attr_once(bb_mma_2cta_kernel, (int)C2_SMEM_BYTES, done_a);
        smem_attr_once(bb_mma_2cta_long_kernel, (int)C2_SMEM_BYTES, done_b);
        const uint32_t pairs = std::max<uint32_t>(1u, std::min<uint32_t>(count, (uint32_t)sms / 2));
        const uint32_t smem = (uint64_t)w_pad * 64 <= C2_COALESCE_MAX_BITS ? C2_SMEM_BYTES
                                                                          : C2_SMEM_BYTES - C2_EPI_BYTES;
        const uint2* tl = d_tiles.p + t0;
        SB_CUDA(launch_pairs((uint64_t)w_pad * 64 <= MMA_MAX_BITS ? bb_mma_2cta_kernel : bb_mma_2cta_long_kernel, pairs,
                             C2_THREADS, smem, st, dX, n, w_pad, lay, tl, count, d_out, d_flags.p));
    } else if (kind == STORM_B200_KERNEL_MMA_SS) {
        static std::atomic<uint64_t> done{0};
        smem_attr_once(bb_mma_kernel, (int)MMA_SMEM_BYTES, done);
        const uint32_t grid = count < (uint32_t)sms ? count : (uint32_t)sms;
        bb_mma_kernel<<<grid, MMA_THREADS, MMA_SMEM_BYTES, st>>>(dX, n, w_pad, lay.pitch, d_tiles.p + t0, count, d_out,
                                                                  d_flags.p);
    } else {
        const size_t smem = sizeof(PopcSmem);
        static std::atomic<uint64_t> done{0};
        smem_attr_once(bb_popc_kernel, (int)smem, done);
        const uint32_t cap = (uint32_t)sms * 2;
        const uint32_t grid = count < cap ? count : cap;
        bb_popc_kernel<<<grid, POPC_THREADS, smem, st>>>(dX, n, w_pad, lay.pitch, d_tiles.p + t0, count, d_out, d_flags.p);
    }
    SB_CUDA(cudaGetLastError());
}

uint64_t DenseEngine::run(const uint64_t* dX, uint64_t n, uint32_t w_pad, uint64_t row_bits,
                          uint32_t* d_out, int kernel_pref, cudaStream_t st) {
    if (n == 0) {
        log.launches = 0;
        log.last_ms = 0.f;
        return 0;
    }
    // The sum alone, no kernel asked for: from the columns' counts.
    if (!d_out && kernel_pref == STORM_B200_KERNEL_AUTO && colsum_room(d_hist, n, w_pad))
        return run_sum(dX, n, w_pad, row_bits, st);
    const int kind = prepare(n, row_bits, kernel_pref, false, st);
    SB_CUDA(cudaEventRecord(log.ev0, st));
    launch(kind, dX, (uint32_t)n, w_pad, 0, n_tiles, d_out, st);
    SB_CUDA(cudaEventRecord(log.ev1, st));
    const DeviceFlags f = read_flags(d_flags.p, st);
    SB_CUDA(cudaEventElapsedTime(&log.last_ms, log.ev0, log.ev1));
    log.launches = 1;
    log.kernel = reported;
    if (f.error) fail(STORM_B200_ETIMEOUT, "bitmap x bitmap kernel: bounded wait expired");
    return f.sum;
}

uint64_t DenseEngine::run_sum(const uint64_t* dX, uint64_t n, uint32_t w_pad, uint64_t row_bits, cudaStream_t st) {
    const int sms = require_device();
    const uint32_t strip = std::min<uint32_t>(w_pad, COLSUM_STRIP);
    d_flags.reserve(1);
    log.ensure();
    SB_CUDA(cudaMemsetAsync(d_flags.p, 0, sizeof(DeviceFlags), st));
    SB_CUDA(cudaEventRecord(log.ev0, st));
    log.launches = 0;
    for (uint32_t w0 = 0; w0 < w_pad; w0 += strip) {
        const uint32_t words = std::min(strip, w_pad - w0);
        const uint32_t gx = (words + COLSUM_WORDS - 1) / COLSUM_WORDS;
        // about four blocks per SM: enough loads in flight, while a block's
        // fixed cost (the planes of 2048 columns into counts) stays below its rows'
        const uint64_t splits = std::max<uint64_t>(1, (uint64_t)sms * 4 / gx);
        const uint64_t per = std::min<uint64_t>(COLSUM_WARPS * COLSUM_WARP_ROWS,
                                                round_up((n + splits - 1) / splits, 8 * COLSUM_WARPS));
        SB_CUDA(cudaMemsetAsync(d_hist.p, 0, 64ull * words * sizeof(uint32_t), st));
        column_counts_kernel<<<dim3(gx, (uint32_t)((n + per - 1) / per)), COLSUM_WARPS * 32, 0, st>>>(
            dX, n, dense_pitch(w_pad), w0, words, per, d_hist.p);
        pairs_of_counts_kernel<<<(uint32_t)std::min<uint64_t>((64ull * words + 255) / 256, (uint64_t)sms * 4), 256, 0,
                                 st>>>(d_hist.p, 64ull * words, &d_flags.p->sum);
        SB_CUDA(cudaGetLastError());
        log.launches += 2;
    }
    SB_CUDA(cudaEventRecord(log.ev1, st));
    const DeviceFlags f = read_flags(d_flags.p, st);
    SB_CUDA(cudaEventElapsedTime(&log.last_ms, log.ev0, log.ev1));
    log.kernel = auto_kind(row_bits);
    return f.sum;
}

// Panels of the host-output forms, in processing order (the bottom of the
// triangle first): [t0, t1) ranges of the tile list. Sizes are whole waves of
// the launch's grid (no SM idles at a launch's end), growing from one wave at
// both ends -- the first panel reads only the last rows, the last panel's
// rows are the only copy still running when the tiles end -- to about 1/24
// of the tiles. Small lists run as one launch.
std::vector<std::pair<uint32_t, uint32_t>> host_panels(uint32_t n_tiles, uint32_t wave) {
    std::vector<std::pair<uint32_t, uint32_t>> p;
    if (n_tiles <= 4ull * wave) {
        p.emplace_back(0u, n_tiles);
        return p;
    }
    const uint64_t total_w = n_tiles / wave;   // the remainder (< 1 wave) joins the last panel
    const uint64_t cap = std::max<uint64_t>(1, total_w / 24);
    std::vector<uint64_t> head;
    uint64_t used = 0;
    for (uint64_t s = 1; s < cap && used + 2 * s <= total_w / 2; s *= 2) {
        head.push_back(s);
        used += s;
    }
    std::vector<uint64_t> sizes(head);
    for (uint64_t mid = total_w - 2 * used; mid > 0;) {
        const uint64_t s = std::min(cap, mid);
        sizes.push_back(s);
        mid -= s;
    }
    sizes.insert(sizes.end(), head.rbegin(), head.rend());
    uint64_t hi = n_tiles;
    for (size_t k = 0; k < sizes.size(); ++k) {
        const uint64_t lo = (k + 1 == sizes.size()) ? 0 : hi - sizes[k] * wave;
        p.emplace_back((uint32_t)lo, (uint32_t)hi);
        hi = lo;
    }
    return p;
}

// Rows of `wpr` words one after another to rows of w_pad words `pitch` apart,
// the words past wpr zeroed. A warp per row; bound by HBM.
__global__ void __launch_bounds__(256)
repitch_rows_kernel(const uint64_t* __restrict__ src, uint32_t wpr, uint64_t* __restrict__ dst, uint64_t pitch,
                    uint32_t w_pad, uint64_t rows) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += nw) {
        const uint64_t* s = src + r * wpr;
        uint64_t* d = dst + r * pitch;
        for (uint32_t w = lane; w < w_pad; w += 32) d[w] = w < wpr ? __ldcs(s + w) : 0;
    }
}

// Host rows into device rows `pitch` words apart (dense.cuh says which way they
// take): `stage` holds as many words as the host rows, or is null.
void rows_to_device(uint64_t* dst, uint64_t pitch, uint32_t w_pad, const uint64_t* host, uint32_t wpr, uint64_t rows,
                    uint64_t* stage, cudaStream_t st) {
    if (rows == 0) return;
    if (stage) {
        SB_CUDA(cudaMemcpyAsync(stage, host, rows * wpr * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
        repitch_rows_kernel<<<(uint32_t)std::min<uint64_t>((rows + 7) / 8, 1184), 256, 0, st>>>(stage, wpr, dst, pitch,
                                                                                              w_pad, rows);
        SB_CUDA(cudaGetLastError());
        return;
    }
    if (wpr == pitch) {
        SB_CUDA(cudaMemcpyAsync(dst, host, rows * wpr * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
        return;
    }
    if (wpr != w_pad)
        SB_CUDA(cudaMemset2DAsync(dst + wpr, pitch * sizeof(uint64_t), 0, (w_pad - wpr) * sizeof(uint64_t), rows, st));
    SB_CUDA(cudaMemcpy2DAsync(dst, pitch * sizeof(uint64_t), host, (size_t)wpr * sizeof(uint64_t),
                              (size_t)wpr * sizeof(uint64_t), rows, cudaMemcpyHostToDevice, st));
}

// Panels of a host-output call. Where the tiles take long beside the copies
// (more than 24 waves), host_panels: whole waves. Below, the copies do, and what
// counts is that the copy back starts early and never waits: up to eight panels
// of whole A blocks, equal in rows -- a fifth of the triangle is copied while the
// second-last panel's rows come in -- of which each spreads over all SMs
// (stream-K), and no more than one per 2 MiB that crosses the bus.
static bool panels_of_blocks(int kind, uint32_t n_tiles, int sms) {
    return kind == KIND_F4 && n_tiles <= 24u * (uint32_t)std::max(1, sms / 2);
}

// A copy into pageable memory blocks the host until it is done, so that panels
// would run one after the other with nothing beside them: there one panel (3000 x
// 20032 bits into pageable memory, eight panels / one: 1.47 / 1.10 ms, rows from
// the host too 2.00 / 1.55; 8000 rows 7.5 / 7.1 and 8.4 / 8.1).
std::vector<std::pair<uint32_t, uint32_t>> host_plan(int kind, uint64_t n, uint32_t n_tiles, int sms,
                                                     uint64_t bus_bytes, bool pinned_out) {
    const uint32_t wave = kind == STORM_B200_KERNEL_POPC        ? 2u * (uint32_t)sms
                          : kind == STORM_B200_KERNEL_MMA_2CTA || kind == KIND_F4 ? (uint32_t)std::max(1, sms / 2)
                                                               : (uint32_t)sms;
    if (!panels_of_blocks(kind, n_tiles, sms)) return host_panels(n_tiles, wave);
    const uint32_t nb = (uint32_t)((n + F4_BM - 1) / F4_BM);
    const uint32_t k = pinned_out ? (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>({8, nb, bus_bytes >> 21})) : 1u;
    auto first = [nb](uint32_t b) { return (uint32_t)((uint64_t)b * nb - (uint64_t)b * (b - (b > 0)) / 2); };   // tile of block b
    std::vector<std::pair<uint32_t, uint32_t>> p;
    for (uint32_t q = k; q-- > 0;) p.emplace_back(first(nb * q / k), first(nb * (q + 1) / k));
    return p;
}

std::vector<uint64_t> host_arrivals(int kind, uint64_t n, const std::vector<uint2>& tiles,
                                    const std::vector<std::pair<uint32_t, uint32_t>>& panels, int sms) {
    std::vector<uint64_t> arrive;
    if (panels.size() == 1) {
        arrive.push_back(0);
    } else if (panels_of_blocks(kind, (uint32_t)tiles.size(), sms)) {
        for (const auto& q : panels) arrive.push_back((uint64_t)tiles[q.first].x * F4_BM);
    } else {
        const uint64_t chunk_rows = round_up(std::max<uint64_t>(1, (n + 31) / 32), 128);
        for (uint64_t c = (n + chunk_rows - 1) / chunk_rows; c-- > 0;) arrive.push_back(c * chunk_rows);
    }
    return arrive;
}

size_t arrival_of(const std::vector<uint64_t>& arrive, uint64_t row) {
    size_t c = 0;
    while (c + 1 < arrive.size() && arrive[c] > row) ++c;
    return c;
}

// Whether copies to this host memory run beside the host (asked where a call may
// take more than one panel: from 4 MiB on the bus).
static bool pinned(const void* p) {
    cudaPointerAttributes a{};
    const bool known = cudaPointerGetAttributes(&a, p) == cudaSuccess && a.type != cudaMemoryTypeUnregistered;
    cudaGetLastError();
    return known;
}

uint64_t DenseEngine::run_to_host(const uint64_t* dX, uint64_t n, uint32_t w_pad, uint64_t row_bits,
                                  uint32_t* d_out, uint32_t* host_out, int kernel_pref, cudaStream_t st,
                                  cudaStream_t copy_st) {
    if (n == 0) {
        log.launches = 0;
        log.last_ms = 0.f;
        return 0;
    }
    const int kind = prepare(n, row_bits, kernel_pref, true, st);
    const uint64_t bus_bytes = tri_size(n) * sizeof(uint32_t);
    const auto panels = host_plan(kind, n, n_tiles, require_device(), bus_bytes, bus_bytes < (2u << 21) || pinned(host_out));
    return panels_to_host(dX, n, w_pad, kind, panels, {}, d_out, host_out, st, copy_st);
}

uint64_t DenseEngine::run_host_to_host(uint64_t* dX, uint64_t n, uint32_t w_pad, uint64_t row_bits,
                                       const uint64_t* host_rows, uint32_t host_wpr, uint32_t* d_out,
                                       uint32_t* host_out, int kernel_pref, cudaStream_t st, cudaStream_t copy_st,
                                       cudaStream_t h2d_st) {
    if (n == 0) {
        log.launches = 0;
        log.last_ms = 0.f;
        return 0;
    }
    const int kind = prepare(n, row_bits, kernel_pref, true, st);
    const int sms = require_device();
    const uint64_t bus_bytes = tri_size(n) * sizeof(uint32_t) + n * host_wpr * sizeof(uint64_t);
    const auto panels = host_plan(kind, n, n_tiles, sms, bus_bytes, bus_bytes < (2u << 21) || pinned(host_out));
    const bool one = panels.size() == 1;             // everything on one stream
    cudaStream_t in = one ? st : h2d_st;
    // Rows [n, n_pad) read as zero: whole tiles read them.
    const uint64_t n_pad = round_up(n, 256), pitch = dense_pitch(w_pad);
    if (n_pad > n) SB_CUDA(cudaMemsetAsync(dX + n * pitch, 0, (n_pad - n) * pitch * sizeof(uint64_t), in));
    uint64_t* const stage = row_stage(d_stage, n, host_wpr);
    const std::vector<uint64_t> arrive = host_arrivals(kind, n, h_tiles, panels, sms);
    while (h2d_ev.size() < arrive.size()) {
        cudaEvent_t e;
        SB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        h2d_ev.push_back(e);
    }
    uint64_t s = 0;
    try {
        uint64_t r1 = n;
        for (size_t c = 0; c < arrive.size(); ++c) {
            const uint64_t r0 = arrive[c];
            rows_to_device(dX + r0 * pitch, pitch, w_pad, host_rows + r0 * host_wpr, host_wpr, r1 - r0,
                           stage ? stage + r0 * host_wpr : nullptr, in);
            if (!one) SB_CUDA(cudaEventRecord(h2d_ev[c], in));
            r1 = r0;
        }
        s = panels_to_host(dX, n, w_pad, kind, panels, one ? std::vector<uint64_t>{} : arrive, d_out, host_out, st,
                           copy_st);
    } catch (...) {
        cudaStreamSynchronize(in);   // no copy may still read the caller's rows after the return
        throw;
    }
    SB_CUDA(cudaStreamSynchronize(in));
    return s;
}

// arrive: rows [arrive[c], n) are resident once event h2d_ev[c] has passed
// (descending; empty: all are); each panel waits for the lowest row its tiles
// read.
uint64_t DenseEngine::panels_to_host(const uint64_t* dX, uint64_t n, uint32_t w_pad, int kind,
                                     const std::vector<std::pair<uint32_t, uint32_t>>& panels,
                                     const std::vector<uint64_t>& arrive, uint32_t* d_out, uint32_t* host_out,
                                     cudaStream_t st, cudaStream_t copy_st) {
    const uint64_t bm = tile_rows_a(kind), bn = tile_rows_b(kind);
    // first tile of each A block (the list is ordered by A block)
    std::vector<uint32_t> first_tile((size_t)h_tiles.back().x + 1, 0);
    for (uint32_t t = n_tiles; t-- > 0;) first_tile[h_tiles[t].x] = t;
    while (panel_ev.size() < panels.size()) {
        cudaEvent_t e;
        SB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        panel_ev.push_back(e);
    }
    SB_CUDA(cudaEventRecord(log.ev0, st));
    cudaStream_t back = panels.size() == 1 ? st : copy_st;   // one launch: its copy follows on the same stream
    uint64_t copied_from = n;   // rows [copied_from, n) are on their way to the host
    DeviceFlags f;
    try {
        for (size_t p = 0; p < panels.size(); ++p) {
            const uint32_t t0 = panels[p].first, t1 = panels[p].second;
            if (!arrive.empty()) {
                uint64_t need = n;
                for (uint32_t t = t0; t < t1; ++t)
                    need = std::min(need, std::min<uint64_t>(h_tiles[t].x * bm, h_tiles[t].y * bn));
                SB_CUDA(cudaStreamWaitEvent(st, h2d_ev[arrival_of(arrive, need)], 0));
            }
            launch(kind, dX, (uint32_t)n, w_pad, t0, t1 - t0, d_out, st);
            if (p + 1 == panels.size()) SB_CUDA(cudaEventRecord(log.ev1, st));
            if (back != st) SB_CUDA(cudaEventRecord(panel_ev[p], st));
            // Every tile from t0 on is done: the A blocks whose first tile is at
            // or past t0 are complete, and their rows are contiguous in the
            // packed triangle.
            uint64_t b = h_tiles[t0].x;
            if (first_tile[b] != t0) ++b;
            const uint64_t r = std::min<uint64_t>(n, b * bm);
            if (r < copied_from) {
                const uint64_t e0 = r * n - (r * (r - 1)) / 2;   // tri_index(n, r, r)
                const uint64_t e1 = copied_from * n - (copied_from * (copied_from - 1)) / 2;
                if (back != st) SB_CUDA(cudaStreamWaitEvent(back, panel_ev[p], 0));
                SB_CUDA(cudaMemcpyAsync(host_out + e0, d_out + e0, (e1 - e0) * sizeof(uint32_t),
                                        cudaMemcpyDeviceToHost, back));
                copied_from = r;
            }
        }
        f = read_flags(d_flags.p, st);
    } catch (...) {
        // no copy may still write the caller's buffer after the return
        cudaStreamSynchronize(st);
        cudaStreamSynchronize(copy_st);
        throw;
    }
    if (back != st) SB_CUDA(cudaStreamSynchronize(back));
    SB_CUDA(cudaEventElapsedTime(&log.last_ms, log.ev0, log.ev1));
    log.launches = (uint32_t)panels.size();
    log.kernel = reported;
    if (f.error) fail(STORM_B200_ETIMEOUT, "bitmap x bitmap kernel: bounded wait expired");
    if (copied_from != 0) fail(STORM_B200_ECUDA, "panel schedule left rows uncopied");
    return f.sum;
}
}  // namespace sb200

// ===================================================================
// Allocation-free entry point.
//
// Some callers cannot allocate device memory at the time they need the
// counts: a service that reserves all of HBM for its own pool at start-up
// and forbids cudaMalloc afterwards (a cudaMalloc on a busy device can
// stall other work and can fail mid-request), or a host framework that owns
// every device buffer through its own allocator.  They hand in the rows and
// the output buffer; this path adds nothing to them.  The tensor-core
// kernel's scratch -- the status / sum words and the tile list -- lives in
// the file-scope array below, sized for at most NOALLOC_MAX_TILES tiles,
// which every GPU that loads the library keeps until the process exits.
// ===================================================================
namespace sb200 {

constexpr uint64_t NOALLOC_MAX_ROWS = 46080;
constexpr uint32_t NOALLOC_MAX_TILES = (NOALLOC_MAX_ROWS / F4_BM) * (NOALLOC_MAX_ROWS / F4_BM + 1) / 2;

struct NoAllocScratch {
    DeviceFlags flags;
    uint2 tiles[NOALLOC_MAX_TILES];
};

static __device__ __align__(256) NoAllocScratch g_noalloc_scratch;

// One thread per A block row bi writes its tiles (bi, bj), bj >= bi, at
// offset bi * nb - bi (bi - 1) / 2.
__global__ void noalloc_tiles_kernel(NoAllocScratch* s, uint32_t nb) {
    const uint32_t bi = blockIdx.x * blockDim.x + threadIdx.x;
    if (bi >= nb) return;
    uint64_t t = (uint64_t)bi * nb - (uint64_t)bi * (bi - (bi > 0)) / 2;
    for (uint32_t bj = bi; bj < nb; ++bj, ++t) s->tiles[t] = make_uint2(bi, bj);
}

}  // namespace sb200

extern "C" int STORM_contig_pairw_intersect_matrix_noalloc(const uint64_t* d_rows, uint64_t n_rows,
                                                           uint32_t row_pitch_words, uint64_t row_bits,
                                                           uint32_t* d_out, uint64_t out_len, uint64_t* sum,
                                                           void* stream) {
    using namespace sb200;
    if (d_rows == NULL) return STORM_B200_EVALUES;
    if (n_rows == 0 || n_rows > 0xFFFFFFFFull) return STORM_B200_EARG;
    if ((uintptr_t)d_rows % 32 != 0) return STORM_B200_EARG;   // the call's contract; TMA itself wants 16
    if (row_pitch_words == 0 || row_pitch_words % 8 != 0 || (uint64_t)row_pitch_words * 64 < row_bits)
        return STORM_B200_EARG;
    if (row_bits > MMA_MAX_BITS) return STORM_B200_ELIMIT;
    const uint64_t need = n_rows * (n_rows + 1) / 2;
    if (d_out != NULL && out_len < need) return STORM_B200_ESIZE;
    if (n_rows > NOALLOC_MAX_ROWS) return STORM_B200_ELIMIT;

    // Once per device, with that device current: the device address of the
    // scratch array, and the kernel's shared-memory opt-in.
    static std::mutex mu;
    static void* scratch_of[64] = {nullptr};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return STORM_B200_ECUDA;
    NoAllocScratch* scratch = nullptr;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (scratch_of[dev] == nullptr) {
            int major = 0;
            if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess || major != 10)
                return STORM_B200_ECUDA;
            void* p = nullptr;
            if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || p == nullptr) return STORM_B200_ECUDA;
            if (cudaFuncSetAttribute(bb_f4_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)F4_SMEM_BYTES) != cudaSuccess)
                return STORM_B200_ECUDA;
            scratch_of[dev] = p;
        }
        scratch = static_cast<NoAllocScratch*>(scratch_of[dev]);
    }
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return STORM_B200_ECUDA;
    // A CUDA error still pending from earlier work is reported before
    // anything is queued, so that it cannot be taken for a failed launch here.
    if (cudaPeekAtLastError() != cudaSuccess) return STORM_B200_ECUDA;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(&scratch->flags, 0, sizeof(DeviceFlags), st) != cudaSuccess) return STORM_B200_ECUDA;
    const uint32_t nb = (uint32_t)((n_rows + F4_BM - 1) / F4_BM), n_pair_tiles = nb * (nb + 1) / 2;
    noalloc_tiles_kernel<<<(nb + 127) / 128, 128, 0, st>>>(scratch, nb);
    const uint32_t pairs = std::min<uint32_t>(n_pair_tiles, (uint32_t)std::max(1, sms / 2));
    uint32_t blk_words = 0;
    CUtensorMap map;
    try {
        map = f4_row_map(d_rows, n_rows, row_pitch_words, row_major(row_pitch_words), &blk_words);
    } catch (const Status&) {
        cudaStreamSynchronize(st);
        return STORM_B200_ECUDA;
    }
    launch_pairs(bb_f4_kernel, pairs, F4_THREADS, F4_SMEM_BYTES, st, map, blk_words, (uint32_t)n_rows, row_pitch_words,
                 (const uint2*)scratch->tiles, n_pair_tiles, d_out, &scratch->flags, 1u);
    if (cudaGetLastError() != cudaSuccess) {
        cudaStreamSynchronize(st);   // nothing already queued may still write d_out after the return
        return STORM_B200_ECUDA;
    }
    DeviceFlags f;
    if (cudaMemcpyAsync(&f, &scratch->flags, sizeof(f), cudaMemcpyDeviceToHost, st) != cudaSuccess)
        return STORM_B200_ECUDA;
    if (cudaStreamSynchronize(st) != cudaSuccess) return STORM_B200_ECUDA;
    if (f.error) return STORM_B200_ETIMEOUT;
    if (sum) *sum = f.sum;
    return 0;
}

// ===================================================================
// Bounded-wait self-test
//
// The tensor-core kernels bound every mbarrier wait (ts_wait): when a wait
// gives up, the kernel records the site in the status word, stops its other
// roles, frees its tensor memory and returns, and the host call returns
// STORM_B200_ETIMEOUT with the context still usable.  This kernel runs that
// path on purpose, on a barrier nothing ever arrives on, with a short limit:
// warp 1 holds tensor memory as the real kernels do, warp 0's lane 0 waits.
// ===================================================================
namespace sb200 {

constexpr uint32_t ERR_SELFTEST = 0x301;

__global__ void __launch_bounds__(64) wait_selftest_kernel(DeviceFlags* flags, uint64_t limit_ns) {
    __shared__ TsCtl ctl;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&ctl.full[0]), 1);
        ctl.abort = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&ctl.tmem_base), 32);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0 && lane == 0) ts_wait(smem_u32(&ctl.full[0]), 0, &ctl, flags, ERR_SELFTEST, false, limit_ns);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(ctl.tmem_base, 32);
    }
}

}  // namespace sb200

extern "C" int STORM_b200_wait_selftest(uint32_t limit_us) {
    using namespace sb200;
    if (limit_us == 0 || limit_us > 10000000u) return STORM_B200_EARG;
    return guard([&]() -> int {
        require_device();
        cudaStream_t st = nullptr;
        SB_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
        DevBuf<DeviceFlags> f;
        f.reserve(1);
        DeviceFlags h{};
        cudaError_t e = cudaMemsetAsync(f.p, 0, sizeof(DeviceFlags), st);
        if (e == cudaSuccess) {
            wait_selftest_kernel<<<1, 64, 0, st>>>(f.p, (uint64_t)limit_us * 1000ull);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaMemcpyAsync(&h, f.p, sizeof(h), cudaMemcpyDeviceToHost, st);
        const cudaError_t es = cudaStreamSynchronize(st);
        cudaStreamDestroy(st);
        SB_CUDA(e);
        SB_CUDA(es);
        return h.error == ERR_SELFTEST ? STORM_B200_ETIMEOUT : 0;
    });
}

// ===================================================================
// Thresholded output
// ===================================================================
namespace sb200 {

// |Xi| of each row: warp per row.
__global__ void row_popcount_kernel(const uint64_t* __restrict__ X, uint64_t n, uint32_t w_pad, uint64_t pitch,
                                    uint32_t* __restrict__ card) {
    const int lane = threadIdx.x & 31;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n; r += nw) {
        uint32_t c = 0;
        for (uint32_t w = lane; w < w_pad; w += 32) c += __popcll(X[r * pitch + w]);
        c = warp_sum_u32(c);
        if (lane == 0) card[r] = c;
    }
}

__global__ void diag_card_kernel(const uint32_t* __restrict__ tri, uint64_t n, uint32_t* __restrict__ card) {
    for (uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; r < n; r += (uint64_t)gridDim.x * blockDim.x)
        card[r] = tri[tri_index(n, r, r)];
}

// Warp per row i, lanes over j > i; warp-aggregated appends.
__global__ void tri_threshold_kernel(const uint32_t* __restrict__ tri, uint64_t n, const uint32_t* __restrict__ card,
                                     double t, uint2* __restrict__ pairs, uint32_t* __restrict__ cnts,
                                     unsigned long long cap, unsigned long long* __restrict__ found) {
    const int lane = threadIdx.x & 31;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += nw) {
        const uint64_t base = tri_index(n, i, i) - i;
        const double ci = (double)card[i];
        for (uint64_t j0 = i + 1; j0 < n; j0 += 32) {
            const uint64_t j = j0 + lane;
            bool pass = false;
            uint32_t cnt = 0;
            if (j < n) {
                cnt = tri[base + j];
                if (cnt) {
                    const double u = ci + (double)card[j] - (double)cnt;
                    pass = u > 0.0 && (double)cnt / u >= t;
                }
            }
            const uint32_t m = __ballot_sync(0xffffffffu, pass);
            if (!m) continue;
            const int leader = __ffs(m) - 1;
            unsigned long long b0 = 0;
            if (lane == leader) b0 = atomicAdd(found, (unsigned long long)__popc(m));
            b0 = __shfl_sync(0xffffffffu, b0, leader);
            if (pass) {
                const unsigned long long k = b0 + __popc(m & ((1u << lane) - 1u));
                if (k < cap) {
                    pairs[k] = make_uint2((uint32_t)i, (uint32_t)j);
                    cnts[k] = cnt;
                }
            }
        }
    }
}

uint64_t threshold_from_triangle(const uint32_t* d_tri, uint64_t n, double t, uint32_t* card,
                                 unsigned long long* found, uint2* d_pairs, uint32_t* d_cnts, uint64_t cap,
                                 cudaStream_t st) {
    const int sms = require_device();
    SB_CUDA(cudaMemsetAsync(found, 0, sizeof(unsigned long long), st));
    if (n) {
        diag_card_kernel<<<(uint32_t)std::min<uint64_t>((n + 255) / 256, (uint64_t)sms * 8), 256, 0, st>>>(d_tri, n,
                                                                                                          card);
        tri_threshold_kernel<<<(uint32_t)std::min<uint64_t>((n + 7) / 8, (uint64_t)sms * 16), 256, 0, st>>>(
            d_tri, n, card, t, d_pairs, d_cnts, cap, found);
        SB_CUDA(cudaGetLastError());
    }
    unsigned long long h = 0;
    SB_CUDA(cudaMemcpyAsync(&h, found, sizeof(h), cudaMemcpyDeviceToHost, st));
    SB_CUDA(cudaStreamSynchronize(st));
    return h;
}

int threshold_to_host(const uint2* d_pairs, const uint32_t* d_cnts, uint64_t found, uint64_t cap, uint32_t* out_i,
                      uint32_t* out_j, uint32_t* out_count, cudaStream_t st) {
    const uint64_t m = std::min<uint64_t>(found, cap);
    std::vector<uint2> pr(m);
    std::vector<uint32_t> ct(m);
    if (m) {
        SB_CUDA(cudaMemcpyAsync(pr.data(), d_pairs, m * sizeof(uint2), cudaMemcpyDeviceToHost, st));
        SB_CUDA(cudaMemcpyAsync(ct.data(), d_cnts, m * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
        SB_CUDA(cudaStreamSynchronize(st));
    }
    // Ordered by (i, j): dealt to their rows, then each row's few sorted by j
    // (a sort of all of them through an index took most of such a call).
    uint32_t rows = 0;
    for (uint64_t k = 0; k < m; ++k) rows = std::max(rows, pr[k].x + 1);
    std::vector<uint64_t> at((uint64_t)rows + 1, 0);
    for (uint64_t k = 0; k < m; ++k) ++at[pr[k].x + 1];
    for (uint64_t r = 0; r < rows; ++r) at[r + 1] += at[r];
    std::vector<uint64_t> hit(m);   // j << 32 | count
    for (uint64_t k = 0; k < m; ++k) hit[at[pr[k].x]++] = (uint64_t)pr[k].y << 32 | ct[k];
    for (uint64_t r = 0, k = 0; r < rows; ++r) {
        std::sort(hit.begin() + k, hit.begin() + at[r]);   // at[r] is now the row's end
        for (; k < at[r]; ++k) {
            if (out_i) out_i[k] = (uint32_t)r;
            if (out_j) out_j[k] = (uint32_t)(hit[k] >> 32);
            if (out_count) out_count[k] = (uint32_t)hit[k];
        }
    }
    return found > cap ? STORM_B200_ESIZE : 0;
}

uint64_t DenseEngine::run_threshold(const uint64_t* dX, uint64_t n, uint32_t w_pad, uint64_t row_bits,
                                    int kernel_pref, double t, uint2* d_pairs, uint32_t* d_cnts, uint64_t cap,
                                    uint64_t* sum, cudaStream_t st) {
    const int sms = require_device();
    d_found.reserve(1);
    d_card.reserve(n ? n : 1);
    if (n == 0) {
        log.launches = 0;
        log.last_ms = 0.f;
        if (sum) *sum = 0;
        return 0;
    }
    // The filter is fused into the drain of the 4-bit kernel and, past 2^24 bits,
    // of MMA's 8-bit one; MMA_DB's has none, so rows it would take go to MMA's.
    if ((kernel_pref == STORM_B200_KERNEL_AUTO || kernel_pref == STORM_B200_KERNEL_MMA_DB) &&
        row_bits <= MMA_MAX_BITS_W4)
        kernel_pref = STORM_B200_KERNEL_MMA;
    const int kind = prepare(n, row_bits, kernel_pref, false, st);
    SB_CUDA(cudaEventRecord(log.ev0, st));
    uint64_t found = 0;
    if (kind == STORM_B200_KERNEL_MMA || kind == KIND_F4) {
        SB_CUDA(cudaMemsetAsync(d_found.p, 0, sizeof(unsigned long long), st));
        row_popcount_kernel<<<(uint32_t)std::min<uint64_t>((n + 7) / 8, (uint64_t)sms * 16), 256, 0, st>>>(
            dX, n, w_pad, dense_pitch(w_pad), d_card.p);
        const TsThresh th{d_card.p, t, d_pairs, d_cnts, (unsigned long long)cap, d_found.p};
        const RowLayout lay = row_major(dense_pitch(w_pad));
        if (kind == KIND_F4) {
            static std::atomic<uint64_t> done{0};
            smem_attr_once(bb_f4_thresh_kernel, (int)F4_SMEM_BYTES, done);
            const uint32_t pairs = std::min<uint32_t>(n_tiles, (uint32_t)std::max(1, sms / 2));
            uint32_t blk_words = 0;
            const CUtensorMap map = f4_row_map(dX, n, w_pad, lay, &blk_words);
            SB_CUDA(launch_pairs(bb_f4_thresh_kernel, pairs, F4_THREADS, F4_SMEM_BYTES, st, map, blk_words, (uint32_t)n,
                                 w_pad, (const uint2*)d_tiles.p, n_tiles, d_flags.p, th));
        } else {
            static std::atomic<uint64_t> done{0};
            smem_attr_once(bb_mma_ts_thresh_long_kernel, (int)TS_SMEM_BYTES, done);
            const uint32_t grid = n_tiles < (uint32_t)sms ? n_tiles : (uint32_t)sms;
            bb_mma_ts_thresh_long_kernel<<<grid, TS_THREADS, TS_SMEM_BYTES, st>>>(
                dX, (uint32_t)n, w_pad, lay, d_tiles.p, n_tiles, d_flags.p, th);
        }
        SB_CUDA(cudaGetLastError());
        unsigned long long h = 0;
        SB_CUDA(cudaMemcpyAsync(&h, d_found.p, sizeof(h), cudaMemcpyDeviceToHost, st));
        SB_CUDA(cudaStreamSynchronize(st));
        found = h;
        log.launches = 2;
    } else {
        d_scratch_tri.reserve(tri_size(n));
        launch(kind, dX, (uint32_t)n, w_pad, 0, n_tiles, d_scratch_tri.p, st);
        found = threshold_from_triangle(d_scratch_tri.p, n, t, d_card.p, d_found.p, d_pairs, d_cnts, cap, st);
        log.launches = 3;
    }
    SB_CUDA(cudaEventRecord(log.ev1, st));
    const DeviceFlags f = read_flags(d_flags.p, st);
    SB_CUDA(cudaEventElapsedTime(&log.last_ms, log.ev0, log.ev1));
    log.kernel = reported;
    if (f.error) fail(STORM_B200_ETIMEOUT, "bitmap x bitmap kernel: bounded wait expired");
    if (sum) *sum = f.sum;
    return found;
}

}  // namespace sb200

// ===================================================================
// Kernel-layer dense block: the tensor-core kernel over a gathered subset of
// rows, counts scattered into the full row set's triangle.
// ===================================================================
namespace sb200 {

// Gathered rows of more than 2^24 bits: the 8-bit kernel.
static bool rows_f4(uint32_t w_pad) { return (uint64_t)w_pad * 64 <= F4_MAX_BITS; }

uint32_t rows_block_a(uint32_t w_pad) { return rows_f4(w_pad) ? F4_BM : MMA_BM; }

void build_rows_tiles(std::vector<uint2>& t, uint64_t n, uint32_t w_pad) {
    build_tiles(t, n, rows_f4(w_pad) ? KIND_F4 : STORM_B200_KERNEL_MMA);
}

void launch_ts_rows(const uint64_t* X, uint32_t n, uint32_t w_pad, RowLayout lay, const uint2* tiles,
                    uint32_t n_tiles, uint32_t* out, DeviceFlags* flags, const uint32_t* row_map, uint64_t n_out, cudaStream_t st,
                    bool out_zeroed) {
    const int sms = require_device();
    if (n_tiles == 0) return;
    if ((uint64_t)w_pad * 64 > MMA_MAX_BITS_W4) fail(STORM_B200_ELIMIT, "dense block rows longer than 2^27 bits");
    // With stream-K the partial counts are added into out, so the whole
    // triangle is zeroed first; the other phases write their own pairs after.
    const bool f4 = rows_f4(w_pad);
    uint32_t grid = 0;
    const uint32_t ks = f4 ? f4_schedule(n_tiles, sms, w_pad, grid) : ts_schedule(n_tiles, sms, w_pad, grid);
    if (ks != 1 && out && !out_zeroed) SB_CUDA(cudaMemsetAsync(out, 0, tri_size(n_out) * sizeof(uint32_t), st));
    if (f4) {
        static std::atomic<uint64_t> done{0};
        smem_attr_once(bb_f4_rows_kernel, (int)F4_SMEM_BYTES, done);
        uint32_t blk_words = 0;
        const CUtensorMap map = f4_row_map(X, n, w_pad, lay, &blk_words);
        SB_CUDA(launch_pairs(bb_f4_rows_kernel, grid, F4_THREADS, F4_SMEM_BYTES, st, map, blk_words, n, w_pad, tiles,
                             n_tiles, out, flags, ks, row_map, n_out));
    } else {
        static std::atomic<uint64_t> done{0};
        smem_attr_once(bb_mma_ts_rows_long_kernel, (int)TS_SMEM_BYTES, done);
        bb_mma_ts_rows_long_kernel<<<grid, TS_THREADS, TS_SMEM_BYTES, st>>>(X, n, w_pad, lay, tiles, n_tiles, out,
                                                                                flags, row_map, n_out, ks);
    }
    SB_CUDA(cudaGetLastError());
}

}  // namespace sb200
