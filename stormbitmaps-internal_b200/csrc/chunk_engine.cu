// chunk_engine.cu -- packing and the warp-per-pair kernel over 65536-bit
// chunks (layout and cell rules: chunk_engine.cuh).
#include <cmath>
#include <cstring>
#include <algorithm>
#include <exception>
#include <mutex>
#include <thread>
#include "chunk_engine.cuh"
#include "dense.cuh"
#include "list16_ref.cuh"
#include "panel.cuh"
#include "run_pieces.cuh"

namespace sb200 {

// Maximal runs of set bits of a bitmap chunk (its words as stored).
static uint64_t bitmap_runs(const STORM_bitmap_t& b) {
    if (!b.data) return 0;
    const uint32_t nw = b.n_bitmap < CHUNK_WORDS ? b.n_bitmap : CHUNK_WORDS;
    uint64_t runs = 0, carry = 0;
    for (uint32_t w = 0; w < nw; ++w) {
        const uint64_t x = b.data[w];
        runs += (uint64_t)__builtin_popcountll(x & ~((x << 1) | carry));
        carry = x >> 63;
    }
    return runs;
}

void ChunkPack::add_chunk(uint32_t id, const STORM_bitmap_t& b) {
    cid.push_back(id);
    if (b.n_bitmap) {
        const uint32_t nw = b.n_bitmap < CHUNK_WORDS ? b.n_bitmap : CHUNK_WORDS;
        coff.push_back(bm.size());
        ckl.push_back(CK_BITMAP | nw);
        const size_t off = bm.size();
        bm.resize(off + CHUNK_WORDS, 0);
        if (b.data) std::copy(b.data, b.data + nw, bm.begin() + off);
    } else {
        const uint32_t ns = b.scalar ? b.n_scalar : 0;
        // Lists start on a 16-byte boundary.
        while (lst.size() % 8) lst.push_back(0);
        coff.push_back(lst.size());
        uint32_t flags = ns & CK_LEN;
        for (uint32_t e = 1; e < ns; ++e)
            if (b.scalar[e] <= b.scalar[e - 1]) { flags |= CK_DUP; break; }
        ckl.push_back(flags);
        lst.insert(lst.end(), b.scalar, b.scalar + ns);
    }
}

void ChunkPack::add_row(const STORM_bitmap_cont_t* c) {
    ChunkRowFacts f;
    if (c && c->bitmaps && c->block_ids) {
        for (uint32_t k = 0; k < c->n_bitmaps; ++k) {
            const STORM_bitmap_t& b = c->bitmaps[k];
            const uint32_t id = c->block_ids[k];
            add_chunk(id, b);
            ++f.chunks;
            if (k > 0 && id <= c->block_ids[k - 1]) f.plain = false;
            if (b.n_bitmap) {
                if (b.n_bitmap != CHUNK_WORDS || b.data == NULL) f.plain = false;
                f.card += b.n_bits_set;
                ++f.bitmap_chunks;
                f.runs += bitmap_runs(b);
            } else {
                if (ckl.back() & CK_DUP) f.plain = false;
                const uint32_t ns = b.scalar ? b.n_scalar : 0;
                f.card += ns;
                f.list_entries += ns;
                for (uint32_t e = 0; e < ns; ++e) f.runs += e == 0 || b.scalar[e] != b.scalar[e - 1] + 1;
            }
            if (id > max_cid) max_cid = id;
        }
    }
    facts.push_back(f);
    end_row();
}

void ChunkPack::add_rows(const STORM_bitmap_cont_t* rows, uint64_t n) {
    if (n == 0) return;
    auto live = [&](uint64_t r) { return rows[r].bitmaps && rows[r].block_ids ? rows[r].n_bitmaps : 0u; };
    // Pass 1: every row's chunk count, bitmap chunks and list slots (each
    // list starts on a multiple of 8 entries, as add_chunk places them).
    std::vector<uint64_t> c_base(n + 1), b_base(n + 1), l_base(n + 1);
    std::vector<uint64_t> l_used(n);
    std::vector<uint8_t> has_list(n);
    for (uint64_t r = 0; r < n; ++r) {
        const uint32_t k_n = live(r);
        uint64_t nb = 0, pos = 0;
        bool lists = false;
        for (uint32_t k = 0; k < k_n; ++k) {
            const STORM_bitmap_t& b = rows[r].bitmaps[k];
            if (b.n_bitmap) {
                ++nb;
            } else {
                pos = (pos + 7) / 8 * 8 + (b.scalar ? b.n_scalar : 0);
                lists = true;
            }
        }
        c_base[r + 1] = c_base[r] + k_n;
        b_base[r + 1] = b_base[r] + nb * CHUNK_WORDS;
        l_used[r] = pos;
        has_list[r] = lists;
        l_base[r + 1] = l_base[r] + (pos + 7) / 8 * 8;
    }
    // Global placement: appended after what the pack already holds.
    const uint64_t c0 = cid.size(), b0 = bm.size();
    uint64_t last_list_row = n;
    for (uint64_t r = n; r-- > 0;)
        if (has_list[r]) {
            last_list_row = r;
            break;
        }
    const uint64_t l0 = last_list_row < n ? (lst.size() + 7) / 8 * 8 : lst.size();
    const uint64_t l_end = last_list_row < n ? l0 + l_base[last_list_row] + l_used[last_list_row] : lst.size();
    cid.resize(c0 + c_base[n]);
    ckl.resize(c0 + c_base[n]);
    coff.resize(c0 + c_base[n]);
    bm.resize(b0 + b_base[n]);
    lst.resize(l_end, 0);   // padding between lists stays zero
    std::vector<ChunkRowFacts> fr(n);
    std::vector<uint32_t> row_max(n, 0);
    // Pass 2: fill, rows split over threads by the bytes they copy.
    auto fill = [&](uint64_t r0, uint64_t r1) {
        for (uint64_t r = r0; r < r1; ++r) {
            ChunkRowFacts f;
            uint32_t mx = 0;
            uint64_t c = c0 + c_base[r], w = b0 + b_base[r], pos = 0;
            const uint64_t lb = l0 + l_base[r];
            const uint32_t k_n = live(r);
            for (uint32_t k = 0; k < k_n; ++k, ++c) {
                const STORM_bitmap_t& b = rows[r].bitmaps[k];
                const uint32_t id = rows[r].block_ids[k];
                cid[c] = id;
                ++f.chunks;
                if (k > 0 && id <= rows[r].block_ids[k - 1]) f.plain = false;
                if (b.n_bitmap) {
                    const uint32_t nw = b.n_bitmap < CHUNK_WORDS ? b.n_bitmap : CHUNK_WORDS;
                    coff[c] = w;
                    ckl[c] = CK_BITMAP | nw;
                    uint64_t* dst = bm.data() + w;
                    const uint32_t copied = b.data ? nw : 0;
                    if (copied) std::memcpy(dst, b.data, copied * sizeof(uint64_t));
                    std::memset(dst + copied, 0, (CHUNK_WORDS - copied) * sizeof(uint64_t));
                    w += CHUNK_WORDS;
                    if (b.n_bitmap != CHUNK_WORDS || b.data == NULL) f.plain = false;
                    f.card += b.n_bits_set;
                    ++f.bitmap_chunks;
                    f.runs += bitmap_runs(b);
                } else {
                    const uint32_t ns = b.scalar ? b.n_scalar : 0;
                    pos = (pos + 7) / 8 * 8;
                    coff[c] = lb + pos;
                    uint32_t flags = ns & CK_LEN;
                    for (uint32_t e = 0; e < ns; ++e) {
                        if (e && b.scalar[e] <= b.scalar[e - 1]) flags |= CK_DUP;
                        f.runs += e == 0 || b.scalar[e] != b.scalar[e - 1] + 1;
                    }
                    ckl[c] = flags;
                    if (ns) std::memcpy(lst.data() + lb + pos, b.scalar, ns * sizeof(uint16_t));
                    pos += ns;
                    if (flags & CK_DUP) f.plain = false;
                    f.card += ns;
                    f.list_entries += ns;
                }
                if (id > mx) mx = id;
            }
            fr[r] = f;
            row_max[r] = mx;
        }
    };
    const uint64_t work = b_base[n] * 8 + l_base[n] * 2 + c_base[n] * 16;
    const unsigned hw = host_threads();
    const uint64_t n_thr = std::min<uint64_t>({(uint64_t)std::min(hw, 32u), n, 1 + work / (8u << 20)});
    if (n_thr <= 1) {
        fill(0, n);
    } else {
        // contiguous row ranges of about equal bytes
        std::vector<uint64_t> cut{0};
        uint64_t acc = 0;
        for (uint64_t r = 0; r < n && cut.size() < n_thr; ++r) {
            acc += (b_base[r + 1] - b_base[r]) * 8 + (l_base[r + 1] - l_base[r]) * 2 +
                   (c_base[r + 1] - c_base[r]) * 16;
            if (acc * n_thr >= work * cut.size()) cut.push_back(r + 1);
        }
        if (cut.back() != n) cut.push_back(n);
        std::vector<std::thread> th;
        for (size_t t = 0; t + 1 < cut.size(); ++t)
            if (cut[t] < cut[t + 1]) th.emplace_back(fill, cut[t], cut[t + 1]);
        for (auto& t : th) t.join();
    }
    for (uint64_t r = 0; r < n; ++r) {
        facts.push_back(fr[r]);
        row_off.push_back(c0 + c_base[r + 1]);
        if (row_max[r] > max_cid) max_cid = row_max[r];
    }
}

double chunk_self_pair_ns(const ChunkCostModel& m, const ChunkRowFacts& f, uint64_t slots) {
    if (f.chunks == 0 || slots == 0) return 0.0;
    const uint32_t lists = f.chunks - f.bitmap_chunks;
    double iters = 32.0 * f.bitmap_chunks;
    if (lists) {
        const double e = std::max(1.0, (double)f.list_entries / lists);
        iters += lists * std::ceil(e / 32.0) * (std::log2(e) + 1.0);
    }
    const double shared = (double)f.chunks * f.chunks / (double)slots;
    return shared * (m.ns_per_shared_chunk + m.ns_per_lane_iteration * iters / f.chunks);
}

double tensor_pair_ns(const ChunkCostModel& m, uint64_t slots) { return m.ns_per_tensor_bit * 65536.0 * slots; }

template <class T, class A>
static void put(DevBuf<T>& d, const std::vector<T, A>& h, cudaStream_t st) {
    d.reserve(h.size() ? h.size() : 1);
    if (!h.empty()) SB_CUDA(cudaMemcpyAsync(d.p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, st));
}

void ChunkDev::upload(const ChunkPack& p, cudaStream_t st) {
    put(row_off, p.row_off, st);
    put(cid, p.cid, st);
    put(ckl, p.ckl, st);
    put(coff, p.coff, st);
    put(bm, p.bm, st);
    put(lst, p.lst, st);
    n_rows = p.rows();
    facts = p.facts;
    rows_changed();
    max_cid = p.max_cid;
    SB_CUDA(cudaStreamSynchronize(st));
}

// A radix sort: 20000 rows in 0.1 ms, a comparison sort 1.1.
const std::vector<uint32_t>& RowsByCard::of(const std::vector<ChunkRowFacts>& facts) {
    if (made) return order;
    const uint64_t n = facts.size();
    order.resize(n);
    uint64_t most = 0;
    for (uint64_t r = 0; r < n; ++r) {
        order[r] = (uint32_t)r;
        most = std::max(most, facts[r].card);
    }
    std::vector<uint32_t> other(n);
    std::vector<uint64_t> at(2049);
    for (int shift = 0; shift < 64 && most >> shift; shift += 11) {
        std::fill(at.begin(), at.end(), 0);
        auto digit = [&](uint32_t r) { return 2047 - (facts[r].card >> shift & 2047); };   // largest first
        for (uint32_t r : order) ++at[digit(r) + 1];
        for (uint64_t k = 0; k < 2048; ++k) at[k + 1] += at[k];
        for (uint32_t r : order) other[at[digit(r)]++] = r;
        order.swap(other);
    }
    made = true;
    return order;
}

PinnedStage::~PinnedStage() {
    for (Lane& l : lanes) {
        if (l.st) {
            cudaStreamSynchronize(l.st);
            cudaStreamDestroy(l.st);
        }
        for (cudaEvent_t e : l.done)
            if (e) cudaEventDestroy(e);
    }
    if (ready) cudaEventDestroy(ready);
    if (pool) cudaFreeHost(pool);
}

void PinnedStage::ensure() {
    if (pool) return;
    const unsigned w = std::max(1u, std::min(64u, host_threads()));
    SB_CUDA(cudaHostAlloc((void**)&pool, TOTAL, cudaHostAllocDefault));
    lane_bytes = TOTAL / (2 * w) / 4096 * 4096;   // >= 1 MiB: any chunk's payload fits
    lanes.resize(w);
    for (unsigned t = 0; t < w; ++t) {
        Lane& l = lanes[t];
        l.buf[0] = pool + (2 * (uint64_t)t) * lane_bytes;
        l.buf[1] = l.buf[0] + lane_bytes;
        SB_CUDA(cudaStreamCreateWithFlags(&l.st, cudaStreamNonBlocking));
        for (cudaEvent_t& e : l.done) SB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    SB_CUDA(cudaEventCreateWithFlags(&ready, cudaEventDisableTiming));
}

// Waits for a lane's stream when a worker leaves, also by an exception, so
// that no copy of a failed call still reads or writes the lane's buffers
// when the next call fills them.
struct LaneSync {
    cudaStream_t st;
    ~LaneSync() { cudaStreamSynchronize(st); }
};

// Runs fn(t) for t in [0, workers) on that many host threads (t = 0 on the
// calling thread) and rethrows the first failure after all have ended.
template <class F>
static void run_workers(unsigned workers, F fn) {
    std::mutex mu;
    std::exception_ptr first;
    auto body = [&](unsigned t) {
        try {
            fn(t);
        } catch (...) {
            std::lock_guard<std::mutex> lock(mu);
            if (!first) first = std::current_exception();
        }
    };
    std::vector<std::thread> th;
    for (unsigned t = 1; t < workers; ++t) th.emplace_back(body, t);
    body(0);
    for (auto& t : th) t.join();
    if (first) std::rethrow_exception(first);
}

// Splits [0, n) into at most `parts` contiguous ranges of about equal weight
// (prefix[r] = weight of rows before r) and runs fn(r0, r1) on each, one
// host thread per range.
template <class F>
static void parallel_rows(uint64_t n, const std::vector<uint64_t>& prefix, unsigned parts, F fn) {
    if (n == 0) return;
    const uint64_t total = prefix[n];
    const uint64_t k = std::max<uint64_t>(1, std::min<uint64_t>({(uint64_t)parts, n, 1 + total / (4u << 20)}));
    if (k <= 1) {
        fn((uint64_t)0, n);
        return;
    }
    std::vector<uint64_t> cut{0};
    for (uint64_t r = 0; r < n && cut.size() < k; ++r)
        if (prefix[r + 1] * k >= total * cut.size()) cut.push_back(r + 1);
    if (cut.back() != n) cut.push_back(n);
    run_workers((unsigned)(cut.size() - 1), [&](unsigned t) { fn(cut[t], cut[t + 1]); });
}

// Lists are not necessarily strictly increasing in the public layout (a
// repeated value, or values added out of order): one warp per chunk tests a
// list's entries, flags the chunk CK_DUP and marks its row; and counts the
// chunk's maximal runs of consecutive values into its row.
__global__ void list_order_kernel(const uint64_t* __restrict__ row_off, uint64_t n_rows, uint32_t* __restrict__ ckl,
                                  const uint64_t* __restrict__ coff, const uint16_t* __restrict__ lst,
                                  const uint64_t* __restrict__ bm, uint64_t nc, uint8_t* __restrict__ row_dup,
                                  uint32_t* __restrict__ row_runs) {
    const int lane = threadIdx.x & 31;
    const uint64_t warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t c = (uint64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < nc; c += warps) {
        const uint32_t k = ckl[c];
        const uint32_t len = k & CK_LEN;
        if (len == 0) continue;
        bool bad = false;
        uint32_t runs = 0;   // maximal runs of consecutive values (the run sweep's pieces)
        if (k & CK_BITMAP) {
            // run starts: set bits whose lower neighbour is clear
            const uint64_t* wd = bm + coff[c];
            uint64_t carry = 0;
            for (uint32_t w0 = 0; w0 < len; w0 += 32) {
                const uint32_t wi = w0 + lane;
                const uint64_t x = wi < len ? wd[wi] : 0ull;
                const uint64_t prev = __shfl_up_sync(0xffffffffu, x, 1);
                const uint64_t cin = lane ? prev >> 63 : carry;
                carry = __shfl_sync(0xffffffffu, x, 31) >> 63;
                runs += warp_sum_u32((uint32_t)__popcll(x & ~((x << 1) | cin)));
            }
        } else {
            const uint16_t* l = lst + coff[c];
            for (uint32_t e0 = 0; e0 < len; e0 += 32) {
                const uint32_t e = e0 + lane;
                const bool in = e < len;
                bad |= __any_sync(0xffffffffu, in && e > 0 && l[e] <= l[e - 1]);
                runs += __popc(__ballot_sync(0xffffffffu, in && (e == 0 || l[e] != l[e - 1] + 1)));
            }
        }
        if (lane == 0) {
            uint64_t lo = 0, hi = n_rows;   // the row r with row_off[r] <= c < row_off[r + 1]
            while (lo + 1 < hi) {
                const uint64_t mid = (lo + hi) >> 1;
                if (row_off[mid] <= c) lo = mid;
                else hi = mid;
            }
            if (bad) {
                ckl[c] = k | CK_DUP;
                row_dup[lo] = 1;
            }
            atomicAdd(&row_runs[lo], runs);
        }
    }
}

void ChunkDev::upload_rows(const STORM_bitmap_cont_t* rows, uint64_t n, cudaStream_t st, PinnedStage& stage) {
    const unsigned hw = std::max(1u, std::min(64u, host_threads()));
    auto live = [&](uint64_t r) { return rows[r].bitmaps && rows[r].block_ids ? rows[r].n_bitmaps : 0u; };
    // Pass 1: per row its chunk count, bitmap words, list slots (each list on
    // a multiple of 8 entries, as ChunkPack places them) and facts; the
    // lists' order is tested on the device below.
    std::vector<uint64_t> c_base(n + 1, 0), b_base(n + 1, 0), l_base(n + 1, 0), w1(n + 1, 0);
    std::vector<uint32_t> row_max(n, 0);
    facts.assign(n, ChunkRowFacts{});
    rows_changed();
    for (uint64_t r = 0; r < n; ++r) w1[r + 1] = w1[r] + 1 + live(r);
    parallel_rows(n, w1, hw, [&](uint64_t r0, uint64_t r1) {
        for (uint64_t r = r0; r < r1; ++r) {
            ChunkRowFacts f;
            uint64_t nb = 0, pos = 0;
            uint32_t mx = 0;
            const uint32_t k_n = live(r);
            for (uint32_t k = 0; k < k_n; ++k) {
                const STORM_bitmap_t& b = rows[r].bitmaps[k];
                const uint32_t id = rows[r].block_ids[k];
                ++f.chunks;
                if (k > 0 && id <= rows[r].block_ids[k - 1]) f.plain = false;
                if (b.n_bitmap) {
                    ++nb;
                    if (b.n_bitmap != CHUNK_WORDS || b.data == NULL) f.plain = false;
                    f.card += b.n_bits_set;
                    ++f.bitmap_chunks;
                } else {
                    const uint32_t ns = b.scalar ? b.n_scalar : 0;
                    pos = (pos + 7) / 8 * 8 + ns;
                    f.card += ns;
                    f.list_entries += ns;
                }
                if (id > mx) mx = id;
            }
            facts[r] = f;
            row_max[r] = mx;
            c_base[r + 1] = k_n;
            b_base[r + 1] = nb * CHUNK_WORDS;
            l_base[r + 1] = (pos + 7) / 8 * 8;
        }
    });
    max_cid = 0;
    for (uint64_t r = 0; r < n; ++r) {
        c_base[r + 1] += c_base[r];
        b_base[r + 1] += b_base[r];
        l_base[r + 1] += l_base[r];
        max_cid = std::max(max_cid, row_max[r]);
    }
    n_rows = n;
    const uint64_t nc = c_base[n], nbw = b_base[n], nl = l_base[n];
    payload_bytes = nbw * 8 + nl * 2;
    // Pass 2: chunk metadata on host threads, then to the device.
    std::vector<uint64_t> h_row_off(n + 1);
    std::vector<uint32_t, NoInitAlloc<uint32_t>> h_cid(nc), h_ckl(nc);
    std::vector<uint64_t, NoInitAlloc<uint64_t>> h_coff(nc);
    for (uint64_t r = 0; r <= n; ++r) h_row_off[r] = c_base[r];
    parallel_rows(n, w1, hw, [&](uint64_t r0, uint64_t r1) {
        for (uint64_t r = r0; r < r1; ++r) {
            uint64_t c = c_base[r], w = b_base[r], pos = 0;
            const uint32_t k_n = live(r);
            for (uint32_t k = 0; k < k_n; ++k, ++c) {
                const STORM_bitmap_t& b = rows[r].bitmaps[k];
                h_cid[c] = rows[r].block_ids[k];
                if (b.n_bitmap) {
                    h_coff[c] = w;
                    h_ckl[c] = CK_BITMAP | (b.n_bitmap < CHUNK_WORDS ? b.n_bitmap : CHUNK_WORDS);
                    w += CHUNK_WORDS;
                } else {
                    const uint32_t ns = b.scalar ? b.n_scalar : 0;
                    pos = (pos + 7) / 8 * 8;
                    h_coff[c] = l_base[r] + pos;
                    h_ckl[c] = ns & CK_LEN;
                    pos += ns;
                }
            }
        }
    });
    row_off.reserve(n + 1);
    cid.reserve(nc ? nc : 1);
    ckl.reserve(nc ? nc : 1);
    coff.reserve(nc ? nc : 1);
    bm.reserve(nbw ? nbw : 1);
    lst.reserve(nl ? nl : 1);
    SB_CUDA(cudaMemcpyAsync(row_off.p, h_row_off.data(), (n + 1) * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
    if (nc) {
        SB_CUDA(cudaMemcpyAsync(cid.p, h_cid.data(), nc * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
        SB_CUDA(cudaMemcpyAsync(ckl.p, h_ckl.data(), nc * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
        SB_CUDA(cudaMemcpyAsync(coff.p, h_coff.data(), nc * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
    }
    // Pass 3: the payload. Each worker takes a range of rows of about equal
    // bytes and moves it in slices of whole chunks: bitmaps (1024 words,
    // short ones zero-filled) at the front of its buffer, list slots (the
    // list, zero padding to a multiple of 8 entries) behind them, two copies
    // per slice on the worker's stream while it fills its other buffer.
    stage.ensure();
    std::vector<uint64_t> pb(n + 1, 0);   // payload bytes of rows before r
    for (uint64_t r = 0; r < n; ++r)
        pb[r + 1] = pb[r] + (b_base[r + 1] - b_base[r]) * 8 + (l_base[r + 1] - l_base[r]) * 2;
    const unsigned workers =
        (unsigned)std::max<uint64_t>(1, std::min<uint64_t>({(uint64_t)stage.lanes.size(), n, 1 + pb[n] / (4u << 20)}));
    std::vector<uint64_t> cut{0};
    for (uint64_t r = 0; r < n && cut.size() < workers; ++r)
        if (pb[r + 1] * workers >= pb[n] * cut.size()) cut.push_back(r + 1);
    while (cut.size() <= workers) cut.push_back(n);
    SB_CUDA(cudaEventRecord(stage.ready, st));   // the metadata copies and earlier work on st
    const uint64_t cap = stage.lane_bytes;
    run_workers(workers, [&](unsigned t) {
        PinnedStage::Lane& L = stage.lanes[t];
        const LaneSync lane_sync{L.st};
        SB_CUDA(cudaStreamWaitEvent(L.st, stage.ready, 0));
        uint64_t r = cut[t], k = 0;
        const uint64_t r_end = cut[t + 1];
        bool used[2] = {false, false};
        int which = 0;
        auto advance = [&]() {
            ++k;
            while (r < r_end && k >= live(r)) {
                ++r;
                k = 0;
            }
        };
        while (r < r_end && k >= live(r)) {
            ++r;
            k = 0;
        }
        while (r < r_end) {
            // the slice: whole chunks from (r, k) while they fit
            uint64_t sr = r, sk = k, bw = 0, ls = 0;
            uint64_t b0 = ~0ull, l0 = ~0ull;
            while (r < r_end) {
                const STORM_bitmap_t& b = rows[r].bitmaps[k];
                const uint64_t c = c_base[r] + k;
                uint64_t nb = 0, nls = 0;
                if (b.n_bitmap) nb = CHUNK_WORDS;
                else nls = ((uint64_t)(h_ckl[c] & CK_LEN) + 7) / 8 * 8;
                if ((bw + nb) * 8 + (ls + nls) * 2 > cap) {
                    if (bw || ls) break;
                    // a list longer than a buffer (the public layout allows
                    // any length): straight from its own memory
                    const uint64_t ns = h_ckl[c] & CK_LEN;
                    if (ns) SB_CUDA(cudaMemcpyAsync(lst.p + h_coff[c], b.scalar, ns * 2, cudaMemcpyHostToDevice, L.st));
                    if (nls > ns) SB_CUDA(cudaMemsetAsync(lst.p + h_coff[c] + ns, 0, (nls - ns) * 2, L.st));
                    advance();
                    sr = r;
                    sk = k;
                    continue;
                }
                if (nb && b0 == ~0ull) b0 = h_coff[c];
                if (nls && l0 == ~0ull) l0 = h_coff[c];
                bw += nb;
                ls += nls;
                advance();
            }
            if (used[which]) SB_CUDA(cudaEventSynchronize(L.done[which]));
            uint64_t* sbm = reinterpret_cast<uint64_t*>(L.buf[which]);
            uint16_t* slst = reinterpret_cast<uint16_t*>(L.buf[which] + bw * 8);
            uint64_t w = 0, p = 0;
            for (uint64_t q = sr, qk = sk; q < r || (q == r && qk < k);) {
                const STORM_bitmap_t& b = rows[q].bitmaps[qk];
                if (b.n_bitmap) {
                    const uint32_t nw = b.n_bitmap < CHUNK_WORDS ? b.n_bitmap : CHUNK_WORDS;
                    const uint32_t copied = b.data ? nw : 0;
                    if (copied) std::memcpy(sbm + w, b.data, copied * sizeof(uint64_t));
                    std::memset(sbm + w + copied, 0, (CHUNK_WORDS - copied) * sizeof(uint64_t));
                    w += CHUNK_WORDS;
                } else {
                    const uint32_t ns = b.scalar ? b.n_scalar : 0;
                    const uint64_t slot = ((uint64_t)ns + 7) / 8 * 8;
                    if (ns) std::memcpy(slst + p, b.scalar, ns * sizeof(uint16_t));
                    std::memset(slst + p + ns, 0, (slot - ns) * sizeof(uint16_t));
                    p += slot;
                }
                ++qk;
                while (q < r_end && qk >= live(q)) {
                    ++q;
                    qk = 0;
                }
            }
            if (bw) SB_CUDA(cudaMemcpyAsync(bm.p + b0, sbm, bw * 8, cudaMemcpyHostToDevice, L.st));
            if (ls) SB_CUDA(cudaMemcpyAsync(lst.p + l0, slst, ls * 2, cudaMemcpyHostToDevice, L.st));
            SB_CUDA(cudaEventRecord(L.done[which], L.st));
            used[which] = true;
            which ^= 1;
        }
        SB_CUDA(cudaStreamSynchronize(L.st));
    });
    // The lists' order and runs, on the device.
    d_row_dup.reserve(n ? n : 1);
    d_row_runs.reserve(n ? n : 1);
    SB_CUDA(cudaMemsetAsync(d_row_dup.p, 0, n ? n : 1, st));
    SB_CUDA(cudaMemsetAsync(d_row_runs.p, 0, (n ? n : 1) * sizeof(uint32_t), st));
    if (nc) {
        const uint64_t blocks = std::min<uint64_t>((nc + 7) / 8, 148ull * 16);
        list_order_kernel<<<(unsigned)blocks, 256, 0, st>>>(row_off.p, n, ckl.p, coff.p, lst.p, bm.p, nc,
                                                            d_row_dup.p, d_row_runs.p);
        SB_CUDA(cudaGetLastError());
    }
    std::vector<uint8_t> dup(n ? n : 1);
    std::vector<uint32_t> runs(n ? n : 1);
    SB_CUDA(cudaMemcpyAsync(dup.data(), d_row_dup.p, n ? n : 1, cudaMemcpyDeviceToHost, st));
    SB_CUDA(cudaMemcpyAsync(runs.data(), d_row_runs.p, (n ? n : 1) * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    SB_CUDA(cudaStreamSynchronize(st));
    for (uint64_t r = 0; r < n; ++r) {
        if (dup[r]) facts[r].plain = false;
        facts[r].runs = runs[r];
    }
}

void copy_to_host(uint32_t* out, const uint32_t* d_src, uint64_t count, cudaStream_t st, PinnedStage& stage) {
    const uint64_t bytes = count * sizeof(uint32_t);
    if (bytes == 0) return;
    cudaPointerAttributes a{};
    const bool known = cudaPointerGetAttributes(&a, out) == cudaSuccess;
    cudaGetLastError();   // an attribute query of plain host memory may leave an error behind
    if (known && a.type == cudaMemoryTypeDevice) fail(STORM_B200_EARG, "the host output buffer is device memory");
    const bool pinned = known && a.type == cudaMemoryTypeHost;
    if (pinned || bytes < (32u << 20)) {
        SB_CUDA(cudaMemcpyAsync(out, d_src, bytes, cudaMemcpyDeviceToHost, st));
        SB_CUDA(cudaStreamSynchronize(st));
        return;
    }
    stage.ensure();
    const uint64_t cap = stage.lane_bytes / sizeof(uint32_t);
    const unsigned workers =
        (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(stage.lanes.size(), bytes / (8u << 20)));
    SB_CUDA(cudaEventRecord(stage.ready, st));
    run_workers(workers, [&](unsigned t) {
        PinnedStage::Lane& L = stage.lanes[t];
        const LaneSync lane_sync{L.st};
        SB_CUDA(cudaStreamWaitEvent(L.st, stage.ready, 0));
        const uint64_t lo = count * t / workers, hi = count * (t + 1) / workers;
        auto issue = [&](uint64_t x, int b) {
            const uint64_t len = std::min(cap, hi - x);
            SB_CUDA(cudaMemcpyAsync(L.buf[b], d_src + x, len * sizeof(uint32_t), cudaMemcpyDeviceToHost, L.st));
            SB_CUDA(cudaEventRecord(L.done[b], L.st));
        };
        if (lo < hi) issue(lo, 0);
        int b = 0;
        for (uint64_t x = lo; x < hi; x += cap, b ^= 1) {
            if (x + cap < hi) issue(x + cap, b ^ 1);   // its buffer was drained in the last round
            SB_CUDA(cudaEventSynchronize(L.done[b]));
            std::memcpy(out + x, L.buf[b], std::min(cap, hi - x) * sizeof(uint32_t));
        }
    });
}

template <class T>
__device__ __forceinline__ uint32_t lower_bound_dev(const T* a, uint32_t n, T x) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (a[mid] < x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// This lane's share of |chunk ca & chunk cb| (warp-cooperative; every lane
// must call it with the same ca, cb).
__device__ __forceinline__ uint32_t chunk_cell_lane(const ChunkView& v, uint64_t ca, uint64_t cb, int lane) {
    const uint32_t ka = v.ckl[ca], kb = v.ckl[cb];
    const bool ba = (ka & CK_BITMAP) != 0, bb = (kb & CK_BITMAP) != 0;
    uint32_t cnt = 0;
    if (ba && bb) {
        const uint64_t* wa = v.bm + v.coff[ca];
        const uint64_t* wb = v.bm + v.coff[cb];
        const uint32_t nw = ka & CK_LEN;   // the reference counts bitmap1->n_bitmap words
        for (uint32_t w = lane; w < nw; w += 32) cnt += __popcll(wa[w] & wb[w]);
    } else if (ba || bb) {
        const uint64_t* w = v.bm + v.coff[ba ? ca : cb];
        const uint32_t kl = ba ? kb : ka;
        const uint16_t* l = v.lst + v.coff[ba ? cb : ca];
        const uint32_t nl = kl & CK_LEN;
        for (uint32_t e = lane; e < nl; e += 32) {
            const uint32_t x = l[e];
            cnt += (uint32_t)(w[x >> 6] >> (x & 63)) & 1u;
        }
    } else if ((ka | kb) & CK_DUP) {
        // A list with a repeated or out-of-order entry: the reference's
        // blocked SSE4.2 count, which then differs from the set size, on
        // one lane (ca is row i's chunk: the reference's first list).
        if (lane == 0)
            cnt = (uint32_t)list16_blocked_count(v.lst + v.coff[ca], v.lst + v.coff[cb], ka & CK_LEN, kb & CK_LEN);
    } else {
        // Strictly increasing lists: each entry of the shorter one is
        // searched in the longer one.
        const uint32_t la = ka & CK_LEN, lb = kb & CK_LEN;
        const bool a_short = la <= lb;
        const uint16_t* s = v.lst + v.coff[a_short ? ca : cb];
        const uint16_t* g = v.lst + v.coff[a_short ? cb : ca];
        const uint32_t ns = a_short ? la : lb, ng = a_short ? lb : la;
        for (uint32_t e = lane; e < ns; e += 32) {
            const uint16_t x = s[e];
            const uint32_t p = lower_bound_dev<uint16_t>(g, ng, x);
            cnt += (p < ng && g[p] == x) ? 1u : 0u;
        }
    }
    return cnt;
}

// Row start S(i) = i*n - i(i-1)/2 of the packed triangle; p -> (i, j).
__device__ __forceinline__ void tri_decode(uint64_t n, uint64_t p, uint64_t& i, uint64_t& j) {
    const double b = 2.0 * (double)n + 1.0;
    double x = (b - sqrt(b * b - 8.0 * (double)p)) * 0.5;
    int64_t ii = (int64_t)x;
    if (ii < 0) ii = 0;
    if ((uint64_t)ii >= n) ii = (int64_t)n - 1;
    auto S = [n](uint64_t r) { return r * n - (r * (r - 1)) / 2; };
    while (ii > 0 && S((uint64_t)ii) > p) --ii;
    while ((uint64_t)ii + 1 < n && S((uint64_t)ii + 1) <= p) ++ii;
    i = (uint64_t)ii;
    j = p - S(i) + i;
}

// Expands chunk slots [s0, s0 + ns) of plain rows (`slots` in all) into
// contiguous bitmaps: local row r of X (in layout `lay`: chunk slot s0 + s of
// row r -- one 1024-word block -- at X + r x pitch + s x kstride) is row rows[r]. A warp
// per (row, chunk slot): absent chunks and padding rows (~0) become zeros,
// bitmap chunks are copied, list chunks are set bit by bit in a shared-memory
// copy of the chunk and written out. Bound: the 8 KiB written per item. A warp
// finds its chunk by a 32-way search of the row's ids, with no chunk before it
// in its way: with a CTA per row walking its slots one after another, 2048
// rows of 2^24 values took 5.9 ms on B200.
constexpr int EXPAND_WARPS = 4;

// Expanded rows for the tensor cores are stored block-major: chunk slot s of
// all the panel's rows together, rows PANEL_PITCH words (8 KiB + 64 bytes)
// apart within it.  A tile's 512 rows at one K stage then lie in about 4 MiB
// instead of on 512 pages of 2 MiB (rows of 2^24 bits row-major), and no two
// rows share a pitch that is a power of two.
constexpr uint64_t PANEL_PITCH = CHUNK_WORDS + 8;
inline uint64_t panel_row_words(uint64_t W) { return W / CHUNK_WORDS * PANEL_PITCH; }

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t x, int lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    return x;
}

// Index of the first of n ascending ids that is >= x (warp-cooperative: 32
// probes at a time).
__device__ __forceinline__ uint32_t warp_lower_bound(const uint32_t* __restrict__ ids, uint32_t n, uint32_t x, int lane) {
    uint32_t lo = 0, len = n;              // the answer lies in [lo, lo + len]
    while (len > 32) {
        const uint32_t step = (len + 31) / 32;
        const uint32_t at = lo + lane * step;
        const uint32_t below = __popc(__ballot_sync(0xffffffffu, lane * step < len && ids[at] < x));
        if (below == 0) return lo;
        const uint32_t left = len - (below - 1) * step;
        lo += (below - 1) * step;          // ids[lo] < x
        len = left < step ? left : step;
    }
    return lo + __popc(__ballot_sync(0xffffffffu, lane < (int)len && ids[lo + lane] < x));
}

// Calls f(first entry, count) with up to eight consecutive entries of a list
// (16-byte aligned) per lane, 256 per step of the warp.
template <class F>
__device__ __forceinline__ void warp_list8(const uint16_t* __restrict__ l, uint32_t nl, int lane, F f) {
    for (uint32_t e0 = 0; e0 < nl; e0 += 256) {
        const uint32_t e = e0 + 8 * lane;
        uint16_t x[8];
        if (e + 8 <= nl) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(l + e));
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k = 0; k < 8; ++k) x[k] = (uint16_t)(w[k / 2] >> (16 * (k & 1)));
        } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) x[k] = e + k < nl ? l[e + k] : (uint16_t)0;
        }
        f(x, e >= nl ? 0u : nl - e < 8 ? nl - e : 8u);
    }
}

__global__ void __launch_bounds__(EXPAND_WARPS * 32)
expand_rows_kernel(ChunkView v, const uint32_t* __restrict__ rows, uint32_t m, uint32_t s0, uint32_t ns, uint32_t slots,
                   RowLayout lay, uint64_t* __restrict__ X) {
    __shared__ __align__(16) uint32_t chunk[EXPAND_WARPS][2 * CHUNK_WORDS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t items = (uint64_t)m * ns, nw = (uint64_t)gridDim.x * EXPAND_WARPS;
    for (uint64_t it = (uint64_t)blockIdx.x * EXPAND_WARPS + warp; it < items; it += nw) {
        const uint32_t r = (uint32_t)(it % m), sl = (uint32_t)(it / m), s = s0 + sl;
        const uint32_t row = rows[r];
        uint4* dst = reinterpret_cast<uint4*>(X + (uint64_t)r * lay.pitch + (uint64_t)sl * lay.kstride);
        uint64_t pos = 0;
        bool have = false;
        if (row != ~0u) {
            const uint64_t c0 = v.row_off[row];
            const uint32_t nc = (uint32_t)(v.row_off[row + 1] - c0);
            const uint32_t q = nc == slots ? s : warp_lower_bound(v.cid + c0, nc, s, lane);
            pos = c0 + q;
            have = q < nc && v.cid[pos] == s;
        }
        if (!have) {
            for (uint32_t q = lane; q < CHUNK_WORDS / 2; q += 32) dst[q] = make_uint4(0, 0, 0, 0);
            continue;
        }
        const uint32_t k = v.ckl[pos];
        if (k & CK_BITMAP) {
            const uint4* src = reinterpret_cast<const uint4*>(v.bm + v.coff[pos]);
            for (uint32_t q = lane; q < CHUNK_WORDS / 2; q += 32) dst[q] = __ldg(src + q);
        } else {
            uint32_t* cw = chunk[warp];
            uint4* c4 = reinterpret_cast<uint4*>(cw);
            for (uint32_t q = lane; q < CHUNK_WORDS / 2; q += 32) c4[q] = make_uint4(0, 0, 0, 0);
            __syncwarp();
            warp_list8(v.lst + v.coff[pos], k & CK_LEN, lane, [&](const uint16_t (&x)[8], uint32_t cnt) {
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q)
                    if (q < cnt) atomicOr(&cw[x[q] >> 5], 1u << (x[q] & 31));
            });
            __syncwarp();
            for (uint32_t q = lane; q < CHUNK_WORDS / 2; q += 32) dst[q] = c4[q];
            __syncwarp();
        }
    }
}

// Pair p of the walk -> rows (i, j), i < j or i == j, as stored:
//   PAIRS_TRIANGLE  p-th entry of the packed triangle of n1 walk rows (a
//                   prefix of it when n_pairs < n1 (n1 + 1) / 2);
//   PAIRS_RECT      walk rows ib + p / n2 and jb + p % n2.
// perm (optional) maps walk rows to stored rows. Counts land at the packed
// index of (i, j) in the triangle of n_out rows when out is given; the sum
// over i != j accumulates into flags->sum.
__global__ void __launch_bounds__(256)
chunk_pairs_kernel(ChunkView v, uint32_t mode, uint64_t n1, uint64_t n2, uint64_t n_pairs,
                   const uint32_t* __restrict__ perm, uint64_t ib, uint64_t jb, uint64_t n_out,
                   uint32_t* __restrict__ out, DeviceFlags* __restrict__ flags) {
    const int lane = threadIdx.x & 31;
    const uint64_t wid = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    unsigned long long local = 0;
    for (uint64_t p = wid; p < n_pairs; p += nwarps) {
        uint64_t i, j;
        if (mode == PAIRS_TRIANGLE) {
            tri_decode(n1, p, i, j);
        } else {
            i = ib + p / n2;
            j = jb + p % n2;
        }
        if (perm) {
            const uint64_t a = perm[i], b = perm[j];
            i = a < b ? a : b;
            j = a < b ? b : a;
        }
        const uint64_t a0 = v.row_off[i], b0 = v.row_off[j];
        const uint32_t na = (uint32_t)(v.row_off[i + 1] - a0), nb = (uint32_t)(v.row_off[j + 1] - b0);
        const bool a_short = na <= nb;
        const uint64_t s0 = a_short ? a0 : b0, l0 = a_short ? b0 : a0;
        const uint32_t ns = a_short ? na : nb, nl = a_short ? nb : na;
        uint32_t cnt = 0;
        for (uint32_t base = 0; base < ns; base += 32) {
            const uint32_t e = base + lane;
            int32_t match = -1;
            if (e < ns) {
                const uint32_t id = v.cid[s0 + e];
                uint32_t r = 0;
                if (e > 0 && v.cid[s0 + e - 1] == id) r = e - lower_bound_dev<uint32_t>(v.cid + s0, e, id);
                const uint32_t q = lower_bound_dev<uint32_t>(v.cid + l0, nl, id) + r;
                if (q < nl && v.cid[l0 + q] == id) match = (int32_t)q;
            }
            uint32_t mask = __ballot_sync(0xffffffffu, match >= 0);
            while (mask) {
                const int src = __ffs(mask) - 1;
                mask &= mask - 1;
                const uint32_t q = (uint32_t)__shfl_sync(0xffffffffu, match, src);
                const uint64_t cs = s0 + base + (uint32_t)src, cl = l0 + q;
                // Row i's chunk is the first argument, as in the reference.
                cnt += a_short ? chunk_cell_lane(v, cs, cl, lane) : chunk_cell_lane(v, cl, cs, lane);
            }
        }
        cnt = warp_sum_u32(cnt);
        if (lane == 0) {
            if (out) out[tri_index(n_out, i, j)] = cnt;
            if (j != i) local += cnt;
        }
    }
    if (lane == 0 && local) atomicAdd(&flags->sum, local);
}

// ---- postings: pairs of plain rows without bitmap chunks ----------------
// value of entry e of list chunk c: cid << 16 | entry (universe <= 2^27)

// Group `g0` .. of `group` (1 .. 32) consecutive chunks [cg, c1) of a row, one
// warp: f(value, its place in the list pool) for every list entry, h(chunk) -- warp-cooperative -- for
// every bitmap chunk. Long lists are walked one chunk at a time (group 1), eight
// entries of each lane read together (walk_entry); of short ones (a chunk of a very sparse row holds a
// handful of values) the warp walks the concatenated entries of 32 chunks,
// whose kinds and places it reads side by side.
template <class F, class H>
__device__ __forceinline__ void walk_group_chunks(const ChunkView& v, uint64_t cg, uint64_t c1, uint32_t group, int lane,
                                                  F f, H h) {
    if (group == 1) {
        const uint32_t k = v.ckl[cg], base = v.cid[cg] << 16;
        if (k & CK_BITMAP) {
            h(cg);
            return;
        }
        const uint64_t off = v.coff[cg];
        const uint32_t nl = k & CK_LEN;
        for (uint32_t e0 = 0; e0 < nl; e0 += WALK_STEP) {
            uint16_t x[WALK_STEP / 32];
#pragma unroll
            for (uint32_t q = 0; q < WALK_STEP / 32; ++q) {
                const uint32_t e = e0 + walk_entry(q, lane);
                x[q] = e < nl ? v.lst[off + e] : (uint16_t)0;
            }
#pragma unroll
            for (uint32_t q = 0; q < WALK_STEP / 32; ++q) {
                const uint32_t e = e0 + walk_entry(q, lane);
                if (e < nl) f(base | x[q], off + e);
            }
        }
        return;
    }
    const uint64_t c = cg + lane;
    const bool in = lane < (int)group && c < c1;
    const uint32_t k = in ? v.ckl[c] : 0u;
    const uint32_t base = in ? v.cid[c] << 16 : 0u;
    const uint64_t off = in ? v.coff[c] : 0ull;
    for (uint32_t bm = __ballot_sync(0xffffffffu, (k & CK_BITMAP) != 0); bm; bm &= bm - 1)
        h(cg + (uint32_t)(__ffs(bm) - 1));
    const uint32_t len = k & CK_BITMAP ? 0u : k & CK_LEN;
    const uint32_t incl = warp_incl_scan(len, lane), excl = incl - len;
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    for (uint32_t t0 = 0; t0 < total; t0 += 32) {
        const uint32_t t = t0 + lane;
        uint32_t o = 0;                    // the last chunk of the group whose entries start at or before t
#pragma unroll
        for (uint32_t step = 16; step; step >>= 1)
            if (__shfl_sync(0xffffffffu, excl, o + step) <= t) o += step;
        const uint32_t e = t - __shfl_sync(0xffffffffu, excl, o), b = __shfl_sync(0xffffffffu, base, o);
        const uint64_t at = __shfl_sync(0xffffffffu, off, o);
        if (t < total) f(b | v.lst[at + e], at + e);
    }
}

// One row by a CTA: its warps take every eighth group of the row's chunks.
template <class F, class H>
__device__ __forceinline__ void row_walk(const ChunkView& v, uint32_t row, uint32_t group, F f, H h) {
    const uint64_t c0 = v.row_off[row], c1 = v.row_off[row + 1];
    for (uint64_t cg = c0 + (uint64_t)(threadIdx.x >> 5) * group; cg < c1; cg += (uint64_t)(blockDim.x >> 5) * group)
        walk_group_chunks(v, cg, c1, group, threadIdx.x & 31, f, h);
}

// Rows (all of the first w.n when `rows` is null) dealt to the grid's warps as
// walk_shape.cuh says: f(index of the row, value, place), h(chunk).
template <class F, class H>
__device__ __forceinline__ void rows_walk(const ChunkView& v, const uint32_t* __restrict__ rows, WalkShape::Dims w,
                                          F f, H h) {
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5, items = w.items();
    for (uint64_t it = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; it < items; it += nw) {
        const uint32_t r = w.row(it);
        const uint32_t row = rows ? rows[r] : r;
        const uint64_t c0 = v.row_off[row], c1 = v.row_off[row + 1];
        for (uint32_t k = w.first_chunk(it); k < (uint32_t)(c1 - c0); k += w.step())
            walk_group_chunks(v, c0 + k, c1, w.group, threadIdx.x & 31, [&](uint32_t x, uint64_t at) { f(r, x, at); }, h);
    }
}

// rows == nullptr: rows [0, w.n). Bitmap chunks count every set bit (only the
// sums over pairs send rows that have them).
__global__ void __launch_bounds__(ROW_WALK_THREADS, ROW_WALK_BLOCKS)
postings_hist_kernel(ChunkView v, const uint32_t* __restrict__ rows, WalkShape::Dims w, uint32_t* __restrict__ counts) {
    const int lane = threadIdx.x & 31;
    rows_walk(
        v, rows, w, [&](uint32_t, uint32_t x, uint64_t) { atomicAdd(&counts[x], 1u); },
        [&](uint64_t c) {
            const uint64_t* wd = v.bm + v.coff[c];
            const uint32_t base = v.cid[c] << 16;
            for (uint32_t q = lane; q < CHUNK_WORDS; q += 32)
                for (uint64_t x = wd[q]; x; x &= x - 1)
                    atomicAdd(&counts[base | (q << 6) | (uint32_t)__ffsll((long long)x) - 1u], 1u);
        });
}

// sum over values of a[x] * b[x] into flags->sum: the rectangle sum of two
// sets of plain rows.
__global__ void counts_dot_kernel(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, uint64_t U,
                                  DeviceFlags* __restrict__ flags) {
    unsigned long long acc = 0;
    for (uint64_t x = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; x < U; x += (uint64_t)gridDim.x * blockDim.x)
        acc += (unsigned long long)a[x] * b[x];
    acc = warp_sum_u64(acc);
    if ((threadIdx.x & 31) == 0 && acc) atomicAdd(&flags->sum, acc);
}

struct PostingsStats {
    unsigned long long pairs;     // sum over values of C(rows holding it, 2)
    unsigned long long lists;     // values held by >= 2 rows
    unsigned long long entries;   // their rows, summed
    unsigned long long cursor[2]; // allocation cursors (entries, lists)
};

__global__ void postings_stats_kernel(const uint32_t* __restrict__ counts, uint64_t U, PostingsStats* st) {
    unsigned long long p = 0, l = 0, e = 0;
    for (uint64_t x = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; x < U; x += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t c = counts[x];
        if (c >= 2) {
            p += (unsigned long long)c * (c - 1) / 2;
            l += 1;
            e += c;
        }
    }
    p = warp_sum_u64(p);
    l = warp_sum_u64(l);
    e = warp_sum_u64(e);
    if ((threadIdx.x & 31) == 0 && l) {
        atomicAdd(&st->pairs, p);
        atomicAdd(&st->lists, l);
        atomicAdd(&st->entries, e);
    }
}

// Gives every value held by >= 2 rows a slot range in the postings array
// (start) and, when `lists` is given, a list record; other values get
// start = ~0. With `heads` (16-bit lists) a list's length stands in front of
// it. A block takes 4096 values at a time and the two allocation
// cursors once for all of them: one atomic per warp on the same two words took
// 0.64 ms for 2^24 values (the counts and starts, 134 MB, cost 0.03). (The run
// postings use it for bins.)
constexpr uint32_t ALLOC_THREADS = 256, ALLOC_PER_THREAD = 16;

__global__ void __launch_bounds__(ALLOC_THREADS)
postings_alloc_kernel(const uint32_t* __restrict__ counts, uint64_t U, uint32_t* __restrict__ start,
                      uint2* __restrict__ lists, uint16_t* __restrict__ heads, PostingsStats* st) {
    const uint32_t head = heads ? 1u : 0u;
    __shared__ uint32_t we[ALLOC_THREADS / 32], wl[ALLOC_THREADS / 32];
    __shared__ unsigned long long e0s, l0s;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr uint32_t TILE = ALLOC_THREADS * ALLOC_PER_THREAD;
    for (uint64_t x0 = (uint64_t)blockIdx.x * TILE; x0 < U; x0 += (uint64_t)gridDim.x * TILE) {
        // value x0 + 512 warp + 32 k + lane: a warp's 16 groups of 32 in order
        uint32_t c[ALLOC_PER_THREAD];
        uint32_t e = 0, l = 0;
        const uint64_t xw = x0 + (uint64_t)warp * 32 * ALLOC_PER_THREAD + lane;
#pragma unroll
        for (uint32_t k = 0; k < ALLOC_PER_THREAD; ++k) {
            const uint64_t x = xw + 32 * k;
            c[k] = x < U ? counts[x] : 0u;
            e += c[k] >= 2 ? c[k] + head : 0u;
            l += c[k] >= 2 ? 1u : 0u;
        }
        const uint32_t ei = warp_incl_scan(e, lane), li = warp_incl_scan(l, lane);
        if (lane == 31) {
            we[warp] = ei;
            wl[warp] = li;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t te = 0, tl = 0;
            for (uint32_t k = 0; k < ALLOC_THREADS / 32; ++k) {
                const uint32_t a = we[k], b = wl[k];
                we[k] = te;
                wl[k] = tl;
                te += a;
                tl += b;
            }
            e0s = tl ? atomicAdd(&st->cursor[0], (unsigned long long)te) : 0ull;
            l0s = tl ? atomicAdd(&st->cursor[1], (unsigned long long)tl) : 0ull;
        }
        __syncthreads();
        uint32_t s = (uint32_t)e0s + we[warp] + ei - e;      // list places of this thread's values
        uint64_t q = l0s + wl[warp] + li - l;
#pragma unroll
        for (uint32_t k = 0; k < ALLOC_PER_THREAD; ++k) {
            const uint64_t x = xw + 32 * k;
            if (x >= U) continue;
            if (c[k] >= 2) {
                if (heads) heads[s] = (uint16_t)c[k];
                start[x] = s + head;
                if (lists) lists[q] = make_uint2(s, c[k]);
                s += c[k] + head;
                ++q;
            } else {
                start[x] = ~0u;
            }
        }
        __syncthreads();   // we, wl and the bases are read before the next tile's
    }
}

// Writes each Q row's position in the Q list (its local index) into the
// lists of its values; start[x] advances to the end of x's list.
__global__ void __launch_bounds__(ROW_WALK_THREADS, ROW_WALK_BLOCKS)
postings_scatter_kernel(ChunkView v, const uint32_t* __restrict__ rows, WalkShape::Dims w,
                        uint32_t* __restrict__ start, uint32_t* __restrict__ post) {
    rows_walk(
        v, rows, w,
        [&](uint32_t r, uint32_t x, uint64_t) {
            // a value of one row has start ~0, and its one row adds to it once
            const uint32_t at = atomicAdd(&start[x], 1u);
            if (at != ~0u) post[at] = r;
        },
        [](uint64_t) {});
}

// One increment per (pair of rows, shared value): thread per list for lists
// of up to POST_THREAD_MAX rows, warp per list beyond.
constexpr uint32_t POST_THREAD_MAX = 64;

__global__ void postings_pairs_kernel(const uint2* __restrict__ lists, uint64_t n_lists,
                                      const uint32_t* __restrict__ post, const uint32_t* __restrict__ qrows,
                                      uint64_t n, uint32_t* __restrict__ out) {
    const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const uint64_t nt = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t li = tid; li < n_lists; li += nt) {
        const uint2 L = lists[li];
        if (L.y > POST_THREAD_MAX) continue;
        for (uint32_t a = 0; a + 1 < L.y; ++a) {
            const uint32_t ra = qrows[post[L.x + a]];
            for (uint32_t b = a + 1; b < L.y; ++b) {
                const uint32_t rb = qrows[post[L.x + b]];
                atomicAdd(&out[ra < rb ? tri_index(n, ra, rb) : tri_index(n, rb, ra)], 1u);
            }
        }
    }
    const int lane = threadIdx.x & 31;
    for (uint64_t li = tid >> 5; li < n_lists; li += nt >> 5) {
        const uint2 L = lists[li];
        if (L.y <= POST_THREAD_MAX) continue;
        for (uint32_t a = 0; a + 1 < L.y; ++a) {
            const uint32_t ra = qrows[post[L.x + a]];
            for (uint32_t b = a + 1 + lane; b < L.y; b += 32) {
                const uint32_t rb = qrows[post[L.x + b]];
                atomicAdd(&out[ra < rb ? tri_index(n, ra, rb) : tri_index(n, rb, ra)], 1u);
            }
        }
    }
}

// The lists of the 16-bit row sweep, each behind its length (heads of
// postings_alloc_kernel): the rows' positions are written into them, counts[x]
// counting down to the places, and place[p] becomes the list of the pool's
// entry p (of its own value), so that the sweep finds a row's lists without
// looking its values up.
__global__ void __launch_bounds__(ROW_WALK_THREADS, ROW_WALK_BLOCKS)
postings_scatter16_kernel(ChunkView v, const uint32_t* __restrict__ rows, WalkShape::Dims w,
                          uint32_t* __restrict__ counts, const uint32_t* __restrict__ start,
                          uint16_t* __restrict__ post, uint32_t* __restrict__ place) {
    rows_walk(
        v, rows, w,
        [&](uint32_t r, uint32_t x, uint64_t at) {
            const uint32_t s = start[x];
            place[at] = s;
            if (s != ~0u) post[s + atomicSub(&counts[x], 1u) - 1u] = (uint16_t)r;
        },
        [](uint64_t) {});
}

// Row sweep over 16-bit lists: CTA per Q row a. A row's entries lie together in
// the list pool, so its lists' places are read in order, and a list -- its
// length and members, two bytes each -- is one sector mostly: one random read
// per value instead of three (count, end, members), from a third of the bytes.
// Every list member b > a gets a shared-memory increment; then the row's slice
// of the triangle is written once. At most 65535 rows of at most 65535 values:
// members, lengths and counts fit 16 bits.
constexpr uint32_t POST_ROWS_THREADS = 512;
constexpr uint32_t POST16_MAX = 0xFFFF;

__global__ void __launch_bounds__(POST_ROWS_THREADS)
postings_rows16_kernel(ChunkView v, const uint32_t* __restrict__ qrows, uint32_t nq, bool all_rows,
                       const uint32_t* __restrict__ place, const uint16_t* __restrict__ post, uint64_t n,
                       uint32_t* __restrict__ out) {
    extern __shared__ uint32_t cnt[];
    __shared__ uint32_t card;
    const uint32_t words = (nq + 1) / 2;
    for (uint32_t a = blockIdx.x; a < nq; a += gridDim.x) {
        const uint32_t row = qrows[a];
        const uint64_t c0 = v.row_off[row], c1 = v.row_off[row + 1];
        for (uint32_t b = (a + 1) / 2 + threadIdx.x; b < words; b += blockDim.x) cnt[b] = 0;
        if (threadIdx.x == 0) card = 0;
        __syncthreads();
        uint32_t mine = 0;
        for (uint64_t c = c0 + threadIdx.x; c < c1; c += blockDim.x) mine += v.ckl[c] & CK_LEN;
        if (mine) atomicAdd(&card, mine);
        if (c1 > c0) {
            const uint64_t p1 = v.coff[c1 - 1] + (v.ckl[c1 - 1] & CK_LEN);
            for (uint64_t p = v.coff[c0] + threadIdx.x; p < p1; p += blockDim.x) {
                const uint32_t s = place[p];
                if (s == ~0u) continue;            // a value of this row alone, or between two lists
                const uint32_t len = post[s - 1];
                for (uint32_t k = 0; k < len; k += 4) {
                    uint32_t b[4];                 // read together (the list is followed by at least 4 places)
#pragma unroll
                    for (uint32_t q = 0; q < 4; ++q) b[q] = post[s + k + q];
#pragma unroll
                    for (uint32_t q = 0; q < 4; ++q)
                        if (k + q < len && b[q] > a) atomicAdd(&cnt[b[q] >> 1], b[q] & 1u ? 0x10000u : 1u);
                }
            }
        }
        __syncthreads();
        const uint64_t base = tri_index(n, row, row) - row;   // out index of (row, j) is base + j
#pragma unroll 4
        for (uint32_t b = a + 1 + threadIdx.x; b < nq; b += blockDim.x) {
            const uint32_t gb = all_rows ? b : qrows[b];      // ascending: gb > row (the other order kept exact too)
            __stcs(out + (gb > row ? base + gb : tri_index(n, gb, row)), (cnt[b >> 1] >> (16 * (b & 1u))) & 0xFFFFu);
        }
        if (threadIdx.x == 0) out[base + row] = card;
        __syncthreads();
    }
}

// Row sweep of more rows, or longer ones: CTA per Q row a; for every value of
// a, the rows b > a on that
// value's list get one shared-memory increment; then a's slice of the
// triangle (its Q partners b > a and its diagonal) is written once, in
// ascending order. Bound: the random reads of a value's count, end and list
// (three sectors, from L2 in part), hidden by full SMs: counts of 16 bits
// (kSmall, no row of more than 65535 values) let four CTAs share an SM.
// Partners are counted for one block of local indices [pb0, pb0 + pbn) per
// launch (at most POST_SWEEP_MAX_ROWS, the counters shared memory holds):
// more postings rows take one launch per block, each reading a row's lists
// again; the launch of block 0 writes the diagonal.
// Lists hold local indices, list x is [end[x] - counts[x], end[x]).
constexpr uint32_t POST_SWEEP_THREADS = 256;      // run sweep
constexpr uint32_t POST_SWEEP_MAX_ROWS = 51200;   // 200 KiB of counters

template <bool kSmall>
__global__ void __launch_bounds__(POST_ROWS_THREADS)
postings_rows_kernel(ChunkView v, const uint32_t* __restrict__ qrows, uint32_t nq, bool all_rows, uint32_t group,
                     const uint32_t* __restrict__ counts, const uint32_t* __restrict__ end,
                     const uint32_t* __restrict__ post, uint64_t n, uint32_t* __restrict__ out, uint32_t pb0,
                     uint32_t pbn) {
    extern __shared__ uint32_t cnt[];
    __shared__ uint32_t card;
    const uint32_t pb1 = pb0 + pbn;
    const uint32_t words = kSmall ? (pbn + 1) / 2 : pbn;
    for (uint32_t a = blockIdx.x; a < nq; a += gridDim.x) {
        if (a + 1 >= pb1 && pb0 > 0) continue;     // no partner after a in this block, diagonal not here
        const uint32_t row = qrows[a];
        const uint32_t w0 = a + 1 <= pb0 ? 0u : kSmall ? (a + 1 - pb0) / 2 : a + 1 - pb0;
        for (uint32_t b = w0 + threadIdx.x; b < words; b += blockDim.x) cnt[b] = 0;
        if (threadIdx.x == 0) card = 0;
        __syncthreads();
        uint32_t mine = 0;
        row_walk(
            v, row, group,
            [&](uint32_t x, uint64_t) {
                ++mine;
                const uint32_t len = counts[x], e1 = end[x];
                if (len < 2) return;
                for (uint32_t k = e1 - len; k < e1; k += 4) {
                    uint32_t b[4];                 // read together: the increments between them would part the reads
#pragma unroll
                    for (uint32_t q = 0; q < 4; ++q) b[q] = k + q < e1 ? __ldg(post + k + q) : 0u;
#pragma unroll
                    for (uint32_t q = 0; q < 4; ++q) {
                        if (b[q] <= a || b[q] < pb0 || b[q] >= pb1) continue;
                        const uint32_t at = b[q] - pb0;
                        if (kSmall) atomicAdd(&cnt[at >> 1], at & 1u ? 0x10000u : 1u);
                        else atomicAdd(&cnt[at], 1u);
                    }
                }
            },
            [](uint64_t) {});
        mine = warp_sum_u32(mine);
        if ((threadIdx.x & 31) == 0 && mine) atomicAdd(&card, mine);
        __syncthreads();
        const uint64_t base = tri_index(n, row, row) - row;   // out index of (row, j) is base + j
#pragma unroll 4
        for (uint32_t b = (a + 1 > pb0 ? a + 1 : pb0) + threadIdx.x; b < pb1; b += blockDim.x) {
            const uint32_t gb = all_rows ? b : qrows[b];   // ascending: gb > row (the other order kept exact too)
            const uint32_t q = b - pb0;
            const uint32_t c = kSmall ? (cnt[q >> 1] >> (16 * (q & 1u))) & 0xFFFFu : cnt[q];
            __stcs(out + (gb > row ? base + gb : tri_index(n, gb, row)), c);
        }
        if (threadIdx.x == 0 && pb0 == 0) out[base + row] = card;
        __syncthreads();
    }
}

// ---- run postings: L x L by overlaps of runs, bin by bin ----------------
// The universe is cut into bins of 2^wlog values (16 .. 32768, so that no
// bin straddles a chunk); a piece is a maximal run of a row's values inside
// one bin. A row's pieces are disjoint, so |Xa & Xb| is the sum over bins of
// the overlaps of a's pieces with b's pieces there: rows made of long runs
// cost per piece instead of per value. Each bin held by >= 2 pieces gets a
// list of (row, start, end) entries (offsets inside the bin), built like the
// value postings (histogram, allocation, scatter); then a row sweep: a CTA
// per row, for each of its pieces the entries of the piece's bin, overlaps
// with rows after it added in shared memory, its triangle slice written once.
// The piece rules: run_pieces.cuh.
constexpr uint32_t RUN_SWEEP_BATCH = 2048;   // pieces prefixed in shared memory at once

// Word wi of a bitmap chunk held by this lane (a warp walks the chunk 32
// words at a time, `carry` = bit 63 of the word before the warp's first):
// the bits that start a piece and the bits that end one.
__device__ __forceinline__ void run_bitmap_word(const uint64_t* wd, uint32_t nwc, uint32_t w0, int lane,
                                                uint32_t wlog, uint64_t& carry, uint64_t& starts, uint64_t& lasts) {
    const uint32_t wi = w0 + lane;
    const uint64_t x = wi < nwc ? wd[wi] : 0ull;
    const uint64_t prev = __shfl_up_sync(0xffffffffu, x, 1);
    const uint64_t next = __shfl_down_sync(0xffffffffu, x, 1);
    const uint64_t cin = lane ? prev >> 63 : carry;
    const uint64_t nin = lane < 31 ? next & 1ull : (w0 + 32 < nwc ? wd[w0 + 32] & 1ull : 0ull);
    carry = __shfl_sync(0xffffffffu, x, 31) >> 63;
    run_word_masks(x, cin, nin, wi, wlog, starts, lasts);
}

// Eight consecutive entries of a strictly increasing list, two per word, with
// the entry before them: bit k of the result says that entry k starts a piece
// (run_pieces.cuh: after a gap, or at a bin's first value). Pairs of 16-bit
// entries at a time.
__device__ __forceinline__ uint32_t run_starts8(const uint32_t (&w)[4], uint32_t before, uint32_t wmask) {
    uint32_t st = 0;
    uint32_t prev = before << 16;          // entry -1 in the upper half
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
        const uint32_t pw = __byte_perm(prev, w[q], 0x5432);          // the entries before these two
        const uint32_t gap = __vcmpne2(__vsub2(w[q], pw), 0x00010001u);
        const uint32_t bin = __vcmpeq2(w[q] & (wmask | wmask << 16), 0u);
        const uint32_t m = gap | bin;
        st |= ((m & 1u) | (m >> 15 & 2u)) << (2 * q);
        prev = w[q];
    }
    return st;
}

// Entry k of eight packed ones.
__device__ __forceinline__ uint32_t entry8(const uint32_t (&w)[4], uint32_t k) {
    const uint32_t lo = k & 2u ? w[1] : w[0], hi = k & 2u ? w[3] : w[2];
    return (k & 4u ? hi : lo) >> (16 * (k & 1u)) & 0xFFFFu;
}

// Eight entries of a list from e on (fewer at its end: zeros follow).
__device__ __forceinline__ void list_load8(const uint16_t* __restrict__ l, uint32_t nl, uint32_t e, uint32_t (&w)[4]) {
    if (e + 8 <= nl) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(l + e));
        w[0] = v.x;
        w[1] = v.y;
        w[2] = v.z;
        w[3] = v.w;
    } else {
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            const uint32_t a = e + 2 * q < nl ? l[e + 2 * q] : 0u, b = e + 2 * q + 1 < nl ? l[e + 2 * q + 1] : 0u;
            w[q] = a | b << 16;
        }
    }
}

// The list and bitmap chunks [c0, c1) of a row by one warp, in order: list
// chunks in steps of 256 entries as f(chunk, its first value, step's entries w,
// starts, lasts) with bits per entry, then done(chunk); bitmap chunks as
// h(chunk). The kinds and places of 32 chunks are read side by side, and the
// next step's entries -- of this chunk or the next one -- are on their way while
// this one's are worked on (a chunk of a row of runs is a few hundred entries:
// one or two steps, which their loads would make wait).
template <class F, class D, class H>
__device__ __forceinline__ void run_chunks(const ChunkView& v, uint64_t c0, uint64_t c1, uint32_t wmask, int lane, F f,
                                           D done, H h) {
    for (uint64_t cg = c0; cg < c1; cg += 32) {
        const bool in = cg + lane < c1;
        const uint32_t kk = in ? v.ckl[cg + lane] : 0u, bb = in ? v.cid[cg + lane] << 16 : 0u;
        const uint64_t off = in ? v.coff[cg + lane] : 0ull;
        const uint32_t m = (uint32_t)(c1 - cg < 32 ? c1 - cg : 32);
        uint32_t nw[4] = {0, 0, 0, 0};
        uint32_t k = __shfl_sync(0xffffffffu, kk, 0);
        const uint16_t* l = v.lst + __shfl_sync(0xffffffffu, off, 0);
        if (!(k & CK_BITMAP)) list_load8(l, k & CK_LEN, 8 * lane, nw);
        for (uint32_t j = 0; j < m; ++j) {
            const uint32_t base = __shfl_sync(0xffffffffu, bb, j);
            // the chunk after this one
            const uint32_t k2 = j + 1 < m ? __shfl_sync(0xffffffffu, kk, j + 1) : CK_BITMAP;
            const uint16_t* l2 = v.lst + __shfl_sync(0xffffffffu, off, (j + 1) & 31);
            const uint32_t nl = k & CK_BITMAP ? 0u : k & CK_LEN;
            if (nl == 0 && !(k2 & CK_BITMAP)) list_load8(l2, k2 & CK_LEN, 8 * lane, nw);
            if (k & CK_BITMAP) {
                h(cg + j);
            } else {
                uint32_t carry = 0;
                for (uint32_t e0 = 0; e0 < nl; e0 += 256) {
                    const uint32_t e = e0 + 8 * lane;
                    const uint32_t w[4] = {nw[0], nw[1], nw[2], nw[3]};
                    if (e0 + 256 < nl) list_load8(l, nl, e + 256, nw);
                    else if (!(k2 & CK_BITMAP)) list_load8(l2, k2 & CK_LEN, 8 * lane, nw);
                    const uint32_t last = w[3] >> 16;
                    const uint32_t up = __shfl_up_sync(0xffffffffu, last, 1);
                    uint32_t st = run_starts8(w, lane ? up : carry, wmask);
                    if (e == 0) st |= 1u;
                    const uint32_t cnt = e >= nl ? 0u : nl - e < 8 ? nl - e : 8u;
                    st &= (1u << cnt) - 1u;
                    // an entry ends a piece where the next one starts one, or is not there
                    uint32_t next = __shfl_down_sync(0xffffffffu, st, 1) & 1u;
                    const uint32_t nx = __shfl_sync(0xffffffffu, nw[0], 0) & 0xFFFFu;   // the next step's first
                    if (lane == 31) next = nx != last + 1 || (nx & wmask) == 0;
                    uint32_t la = (st >> 1 | next << 7) & ((1u << cnt) - 1u);
                    if (cnt && e + cnt == nl) la |= 1u << (cnt - 1);
                    f(cg + j, base, w, st, la);
                    carry = __shfl_sync(0xffffffffu, last, 31);
                }
                done(cg + j);
            }
            k = k2;
            l = l2;
        }
    }
}

// The same chunks a lane per list chunk, for rows made of long runs: in a
// strictly increasing list entry e + 1 follows entry e exactly where value minus
// index stays the same, so a run's last entry is found by halving -- at once,
// when the rest of the list is one run -- and the entries in between are never
// read. g(lane's chunk index within the share's 32, chunk, base, first, last)
// per run, by the lane that found it; list_done(chunk) once per lane and list
// chunk; bitmap chunks as h(chunk), warp-cooperative. (256 entries per step of
// a warp are 250 instructions to look at them all: 4000 rows of 51000 values in
// runs of 256 took 323 us to count and 458 to fill.)
template <class G, class D, class H>
__device__ __forceinline__ void gallop_chunks(const ChunkView& v, uint64_t c0, uint64_t c1, int lane, G g, D list_done,
                                              H h) {
    for (uint64_t cg = c0; cg < c1; cg += 32) {
        const uint64_t c = cg + lane;
        const uint32_t k = c < c1 ? v.ckl[c] : 0u;
        if (c < c1 && !(k & CK_BITMAP)) {
            const uint16_t* l = v.lst + v.coff[c];
            const uint32_t base = v.cid[c] << 16, nl = k & CK_LEN;
            uint32_t e = 0;
            const uint32_t end = nl ? l[nl - 1] : 0u;
            while (e < nl) {
                const uint32_t x = l[e];
                uint32_t lo = e, last = x;                 // l[lo] = last is in x's run
                if (end - x == nl - 1 - e) {
                    lo = nl - 1;
                    last = end;
                } else {
                    uint32_t hi = nl - 1;                  // l[hi] is not
                    while (hi - lo > 1) {
                        const uint32_t mid = (lo + hi) >> 1, y = l[mid];
                        if (y - x == mid - e) {
                            lo = mid;
                            last = y;
                        } else {
                            hi = mid;
                        }
                    }
                }
                g(c, base, x, last);
                e = lo + 1;
            }
            list_done(c);
        }
        __syncwarp();
        for (uint32_t bm = __ballot_sync(0xffffffffu, (k & CK_BITMAP) != 0); bm; bm &= bm - 1)
            h(cg + (uint32_t)(__ffs(bm) - 1));
    }
}

// A row's chunks dealt to the warps of its CTA in consecutive shares.
__device__ __forceinline__ void warp_share(uint64_t c0, uint64_t c1, uint64_t& lo, uint64_t& hi) {
    constexpr uint32_t WARPS = ROW_WALK_THREADS / 32;
    const uint32_t warp = threadIdx.x >> 5;
    lo = c0 + (c1 - c0) * warp / WARPS;
    hi = c0 + (c1 - c0) * (warp + 1) / WARPS;
}

// Pieces per row, per chunk and per bin; CTA per row.
template <bool kGallop>
__global__ void __launch_bounds__(ROW_WALK_THREADS)
run_count_kernel(ChunkView v, const uint32_t* __restrict__ rows, uint32_t nq, uint32_t wlog,
                 uint32_t* __restrict__ pieces, uint32_t* __restrict__ chunk_pieces, uint32_t* __restrict__ bins) {
    __shared__ uint32_t total;
    const int lane = threadIdx.x & 31;
    for (uint32_t r = blockIdx.x; r < nq; r += gridDim.x) {
        if (threadIdx.x == 0) total = 0;
        __syncthreads();
        const uint32_t row = rows[r];
        uint64_t lo, hi;
        warp_share(v.row_off[row], v.row_off[row + 1], lo, hi);
        uint32_t cnt = 0, mine = 0;
        auto warp_done = [&](uint64_t c) {     // the warp's chunk
            const uint32_t t = warp_sum_u32(cnt);
            if (lane == 0) {
                chunk_pieces[c] = t;
                mine += t;
            }
            cnt = 0;
        };
        auto bitmap = [&](uint64_t c) {
            const uint64_t* wd = v.bm + v.coff[c];
            const uint32_t nwc = v.ckl[c] & CK_LEN, base = v.cid[c] << 16;
            uint64_t carry = 0, starts, lasts;
            for (uint32_t w0 = 0; w0 < nwc; w0 += 32) {
                run_bitmap_word(wd, nwc, w0, lane, wlog, carry, starts, lasts);
                cnt += __popcll(starts);
                for (uint64_t x = starts; x; x &= x - 1)
                    atomicAdd(&bins[(base + ((w0 + lane) << 6) + (uint32_t)(__ffsll((long long)x) - 1)) >> wlog], 1u);
            }
            warp_done(c);
        };
        if constexpr (kGallop) {
            gallop_chunks(
                v, lo, hi, lane,
                [&](uint64_t, uint32_t base, uint32_t first, uint32_t last) {
                    const uint32_t b1 = (base | last) >> wlog;
                    for (uint32_t b = (base | first) >> wlog; b <= b1; ++b, ++cnt) atomicAdd(&bins[b], 1u);
                },
                [&](uint64_t c) {              // the lane's own chunk
                    chunk_pieces[c] = cnt;
                    mine += cnt;
                    cnt = 0;
                },
                bitmap);
        } else {
            run_chunks(
                v, lo, hi, (1u << wlog) - 1u, lane,
                [&](uint64_t, uint32_t base, const uint32_t (&w)[4], uint32_t st, uint32_t) {
                    cnt += __popc(st);
                    for (uint32_t m = st; m; m &= m - 1) atomicAdd(&bins[(base | entry8(w, __ffs(m) - 1)) >> wlog], 1u);
                },
                warp_done, bitmap);
        }
        mine = warp_sum_u32(mine);
        if (lane == 0 && mine) atomicAdd(&total, mine);
        __syncthreads();
        if (threadIdx.x == 0) pieces[r] = total;
        __syncthreads();
    }
}

// Over the bins held by >= 2 pieces: st[0] += their pieces (list entries),
// st[1] += pieces^2 (the sweep's entry reads).
__global__ void run_stats_kernel(const uint32_t* __restrict__ bins, uint64_t nb, unsigned long long* __restrict__ st) {
    unsigned long long e = 0, q = 0;
    for (uint64_t x = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; x < nb; x += (uint64_t)gridDim.x * blockDim.x) {
        const unsigned long long c = bins[x];
        if (c >= 2) {
            e += c;
            q += c * c;
        }
    }
    e = warp_sum_u64(e);
    q = warp_sum_u64(q);
    if ((threadIdx.x & 31) == 0 && e) {
        atomicAdd(&st[0], e);
        atomicAdd(&st[1], q);
    }
}

// The rows' pieces in row order: pieces[poff[r] + k] = (first value, end),
// the k-th start and the k-th last value of the row paired by rank (list
// entries, or set bits of bitmap chunks). A piece lies in one chunk, so the
// pieces counted per chunk place every chunk's (a prefix over the row's at
// most 2048 chunks), and a CTA's warps take the chunks side by side: with a
// warp per row, 4000 rows of 51000 values took 1.24 ms, and counting 0.85.
constexpr uint32_t RUN_MAX_CHUNKS = 2048;    // universe <= 2^27

template <bool kGallop>
__global__ void __launch_bounds__(ROW_WALK_THREADS)
run_fill_kernel(ChunkView v, const uint32_t* __restrict__ rows, uint32_t nq, uint32_t wlog,
                const uint64_t* __restrict__ poff, const uint32_t* __restrict__ chunk_pieces,
                uint2* __restrict__ pieces) {
    __shared__ uint32_t first[RUN_MAX_CHUNKS];
    __shared__ uint32_t wsum[ROW_WALK_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t wmask = (1u << wlog) - 1u;
    for (uint32_t r = blockIdx.x; r < nq; r += gridDim.x) {
        const uint32_t row = rows[r];
        const uint64_t c0 = v.row_off[row];
        const uint32_t nc = (uint32_t)(v.row_off[row + 1] - c0);
        // first[k]: pieces of the chunks before chunk k
        constexpr uint32_t PER = RUN_MAX_CHUNKS / ROW_WALK_THREADS;
        uint32_t own[PER], sum = 0;
#pragma unroll
        for (uint32_t q = 0; q < PER; ++q) {
            const uint32_t k = threadIdx.x * PER + q;
            own[q] = sum;
            sum += k < nc ? chunk_pieces[c0 + k] : 0u;
        }
        const uint32_t incl = warp_incl_scan(sum, lane);
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        uint32_t before = incl - sum;
        for (int w = 0; w < warp; ++w) before += wsum[w];
#pragma unroll
        for (uint32_t q = 0; q < PER; ++q) {
            const uint32_t k = threadIdx.x * PER + q;
            if (k < nc) first[k] = before + own[q];
        }
        __syncthreads();
        uint64_t lo, hi;
        warp_share(c0, c0 + nc, lo, hi);
        uint2* const out0 = pieces + poff[r];
        auto bitmap = [&](uint64_t c) {
            uint2* out = out0 + first[c - c0];
            const uint64_t* wd = v.bm + v.coff[c];
            const uint32_t nwc = v.ckl[c] & CK_LEN, base = v.cid[c] << 16;
            uint64_t carry = 0, starts, lasts;
            uint32_t ks = 0, kl = 0;
            for (uint32_t w0 = 0; w0 < nwc; w0 += 32) {
                run_bitmap_word(wd, nwc, w0, lane, wlog, carry, starts, lasts);
                const uint32_t ns = (uint32_t)__popcll(starts), nls = (uint32_t)__popcll(lasts);
                const uint32_t xs = warp_incl_scan(ns, lane), xl = warp_incl_scan(nls, lane);
                const uint32_t word0 = base + ((w0 + lane) << 6);
                uint32_t j = ks + xs - ns;
                for (uint64_t x = starts; x; x &= x - 1) out[j++].x = word0 + (uint32_t)(__ffsll((long long)x) - 1);
                j = kl + xl - nls;
                for (uint64_t x = lasts; x; x &= x - 1) out[j++].y = word0 + (uint32_t)__ffsll((long long)x);
                ks += __shfl_sync(0xffffffffu, xs, 31);
                kl += __shfl_sync(0xffffffffu, xl, 31);
            }
        };
        if constexpr (kGallop) {
            uint32_t j = 0;                // pieces of the lane's chunk so far
            gallop_chunks(
                v, lo, hi, lane,
                [&](uint64_t c, uint32_t base, uint32_t from, uint32_t last) {
                    uint2* out = out0 + first[c - c0];
                    const uint32_t end = (base | last) + 1u;
                    for (uint32_t s = base | from; s < end;) {
                        const uint32_t next = (s | wmask) + 1u;        // the next bin
                        out[j++] = make_uint2(s, next < end ? next : end);
                        s = next;
                    }
                },
                [&](uint64_t) { j = 0; }, bitmap);
        } else {
            uint64_t at = ~0ull;           // the chunk being walked
            uint32_t ks = 0, kl = 0;       // its starts and lasts so far
            run_chunks(
                v, lo, hi, wmask, lane,
                [&](uint64_t c, uint32_t base, const uint32_t (&w)[4], uint32_t st, uint32_t la) {
                    if (c != at) ks = kl = 0;
                    at = c;
                    uint2* out = out0 + first[c - c0];
                    // ranks of the lane's starts and lasts, 16 bits each (a step holds 256 entries)
                    const uint32_t both = __popc(st) | (uint32_t)__popc(la) << 16;
                    const uint32_t inc = warp_incl_scan(both, lane), exc = inc - both;
                    uint32_t j = ks + (exc & 0xFFFFu);
                    for (uint32_t m = st; m; m &= m - 1) out[j++].x = base | entry8(w, __ffs(m) - 1);
                    j = kl + (exc >> 16);
                    for (uint32_t m = la; m; m &= m - 1) out[j++].y = (base | entry8(w, __ffs(m) - 1)) + 1u;
                    const uint32_t tot = __shfl_sync(0xffffffffu, inc, 31);
                    ks += tot & 0xFFFFu;
                    kl += tot >> 16;
                },
                [](uint64_t) {}, bitmap);
        }
        __syncthreads();   // first is read before the next row's
    }
}

// Each piece of a bin held by >= 2 pieces into the bin's list: (row, start
// | end << 16), offsets inside the bin; start[b] advances to the list's end.
__global__ void run_scatter_kernel(uint32_t nq, uint32_t wlog, const uint64_t* __restrict__ poff,
                                   const uint2* __restrict__ pieces, uint32_t* __restrict__ start,
                                   uint2* __restrict__ list) {
    const int lane = threadIdx.x & 31;
    const uint32_t wmask = (1u << wlog) - 1u;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nq; r += nw)
        for (uint64_t p = poff[r] + lane; p < poff[r + 1]; p += 32) {
            const uint2 pc = pieces[p];
            const uint32_t bin = pc.x >> wlog;
            if (start[bin] == ~0u) continue;
            list[atomicAdd(&start[bin], 1u)] = make_uint2(r, (pc.x & wmask) | ((pc.y - (bin << wlog)) << 16));
        }
}

// The row sweep over pieces: CTA per row a; the (piece, bin entry) pairs of
// a batch of a's pieces are split evenly over the threads (a shared-memory
// prefix of the pieces' bin lengths maps work index -> piece). Partners in
// one block of local indices [pb0, pb0 + pbn) per launch, as in
// postings_rows_kernel. Shared memory: pbn counters, then RUN_SWEEP_BATCH + 1
// prefix words. Bin b's list is [end[b] - bins[b], end[b]). Adds the sum
// over a's partners after it (in the block) to flags->sum.
__global__ void __launch_bounds__(POST_SWEEP_THREADS)
run_sweep_kernel(const uint32_t* __restrict__ qrows, uint32_t nq, const uint64_t* __restrict__ poff,
                 const uint2* __restrict__ pieces, uint32_t wlog, const uint32_t* __restrict__ bins,
                 const uint32_t* __restrict__ end, const uint2* __restrict__ list, uint64_t n,
                 uint32_t* __restrict__ out, DeviceFlags* __restrict__ flags, uint32_t pb0, uint32_t pbn) {
    extern __shared__ uint32_t cnt[];
    uint32_t* pref = cnt + pbn;
    const uint32_t pb1 = pb0 + pbn;
    __shared__ uint32_t warp_tot[POST_SWEEP_THREADS / 32];
    __shared__ unsigned long long row_card;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (uint32_t a = blockIdx.x; a < nq; a += gridDim.x) {
        if (a + 1 >= pb1 && pb0 > 0) continue;     // no partner after a in this block, diagonal not here
        const uint32_t row = qrows[a];
        for (uint32_t b = threadIdx.x; b < pbn; b += blockDim.x) cnt[b] = 0;
        if (threadIdx.x == 0) row_card = 0;
        const uint64_t p0 = poff[a], np = poff[a + 1] - p0;
        unsigned long long card = 0;
        for (uint64_t pb = 0; pb < np; pb += RUN_SWEEP_BATCH) {
            const uint32_t m = (uint32_t)(np - pb < RUN_SWEEP_BATCH ? np - pb : RUN_SWEEP_BATCH);
            // pref[k] = entries of the bins of pieces pb .. pb + k - 1: each
            // thread sums a contiguous segment, then a block scan of the sums
            const uint32_t seg = (m + POST_SWEEP_THREADS - 1) / POST_SWEEP_THREADS;
            const uint32_t k0 = threadIdx.x * seg, k1 = k0 + seg < m ? k0 + seg : m;
            uint32_t mine = 0;
            for (uint32_t k = k0; k < k1; ++k) {
                const uint2 pc = pieces[p0 + pb + k];
                card += pc.y - pc.x;
                const uint32_t c = bins[pc.x >> wlog];
                mine += c >= 2 ? c : 0u;
            }
            uint32_t inc = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += y;
            }
            __syncthreads();   // the previous batch is done with pref and warp_tot
            if (lane == 31) warp_tot[wid] = inc;
            __syncthreads();
            uint32_t before = 0, total = 0;
            for (int w = 0; w < POST_SWEEP_THREADS / 32; ++w) {
                if (w < wid) before += warp_tot[w];
                total += warp_tot[w];
            }
            uint32_t acc = before + inc - mine;
            for (uint32_t k = k0; k < k1; ++k) {
                pref[k] = acc;
                const uint32_t c = bins[pieces[p0 + pb + k].x >> wlog];
                acc += c >= 2 ? c : 0u;
            }
            if (threadIdx.x == 0) pref[m] = total;
            __syncthreads();
            const uint32_t work = a + 1 < pb1 ? total : 0u;   // no partner in the block: the diagonal only
            for (uint32_t t = threadIdx.x; t < work; t += blockDim.x) {
                uint32_t lo = 0, hi = m;           // last piece k with pref[k] <= t
                while (hi - lo > 1) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (pref[mid] <= t) lo = mid;
                    else hi = mid;
                }
                const uint2 pc = pieces[p0 + pb + lo];
                const uint32_t bin = pc.x >> wlog;
                const uint2 E = list[end[bin] - bins[bin] + (t - pref[lo])];
                if (E.x > a && E.x >= pb0 && E.x < pb1) {
                    const uint32_t b0 = bin << wlog;
                    const uint32_t s2 = b0 + (E.y & 0xFFFFu), e2 = b0 + (E.y >> 16);
                    const uint32_t s = pc.x > s2 ? pc.x : s2, e = pc.y < e2 ? pc.y : e2;
                    if (e > s) atomicAdd(&cnt[E.x - pb0], e - s);
                }
            }
        }
        card = warp_sum_u64(card);
        if (lane == 0 && card) atomicAdd(&row_card, card);
        __syncthreads();
        const uint64_t base = tri_index(n, row, row) - row;   // out index of (row, j) is base + j
        unsigned long long sum = 0;
        for (uint32_t b = (a + 1 > pb0 ? a + 1 : pb0) + threadIdx.x; b < pb1; b += blockDim.x) {
            const uint32_t gb = qrows[b];
            out[gb > row ? base + gb : tri_index(n, gb, row)] = cnt[b - pb0];
            sum += cnt[b - pb0];
        }
        sum = warp_sum_u64(sum);
        if (lane == 0 && sum) atomicAdd(&flags->sum, sum);
        if (threadIdx.x == 0 && pb0 == 0) out[base + row] = (uint32_t)row_card;
        __syncthreads();
    }
}

// Diagonal of rows with bitmap chunks too (warp per row): each row's value
// count, set bits of its bitmap chunks plus its list entries.
__global__ void row_card_diag_kernel(ChunkView v, const uint32_t* __restrict__ rows, uint32_t m, uint64_t n,
                                     uint32_t* __restrict__ out) {
    const int lane = threadIdx.x & 31;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < m; r += nw) {
        const uint32_t row = rows[r];
        uint32_t card = 0;
        for (uint64_t c = v.row_off[row]; c < v.row_off[row + 1]; ++c) {
            const uint32_t k = v.ckl[c];
            if (k & CK_BITMAP) {
                const uint64_t* wd = v.bm + v.coff[c];
                for (uint32_t w = lane; w < (k & CK_LEN); w += 32) card += __popcll(wd[w]);
            } else if (lane == 0) {
                card += k & CK_LEN;
            }
        }
        card = warp_sum_u32(card);
        if (lane == 0) out[tri_index(n, row, row)] = card;
    }
}

// Diagonal of the postings rows: their value count.
__global__ void postings_diag_kernel(ChunkView v, const uint32_t* __restrict__ rows, uint32_t nq, uint64_t n,
                                     uint32_t* __restrict__ out) {
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < nq; r += gridDim.x * blockDim.x) {
        const uint32_t row = rows[r];
        uint32_t card = 0;
        for (uint64_t c = v.row_off[row]; c < v.row_off[row + 1]; ++c) card += v.ckl[c] & CK_LEN;
        out[tri_index(n, row, row)] = card;
    }
}

uint64_t ChunkEngine::run(const ChunkDev& d, PairMode mode, uint64_t n1, uint64_t n2, uint32_t* d_out,
                          cudaStream_t st) {
    const int sms = require_device();
    const uint64_t n_pairs_all = mode == PAIRS_TRIANGLE ? tri_size(n1) : n1 * n2;
    log.launches = 0;
    log.last_ms = 0.f;
    last_dense_rows = last_dense_panels = last_postings_rows = 0;
    last_panel_rows = last_panel_queries = 0;
    last_postings_form = -1;
    for (int k = 0; k < 4; ++k) last_engine_ms[k] = last_engine_pred_ms[k] = last_engine_work[k] = 0.0;
    if (n_pairs_all == 0) return 0;
    d_flags.reserve(1);
    SB_CUDA(cudaMemsetAsync(d_flags.p, 0, sizeof(DeviceFlags), st));
    log.ensure();
    uint32_t launches = 0;
    auto chunk_launch = [&](uint32_t m, uint64_t np, const uint32_t* perm, uint64_t ib, uint64_t jb, uint64_t nn1,
                            uint64_t nn2) {
        if (np == 0) return;
        const uint64_t want_blocks = (np + 7) / 8;
        const uint32_t grid = (uint32_t)(want_blocks < (uint64_t)sms * 16 ? want_blocks : (uint64_t)sms * 16);
        chunk_pairs_kernel<<<grid, 256, 0, st>>>(d.view(), m, nn1, nn2, np, perm, ib, jb, n1, d_out, d_flags.p);
        SB_CUDA(cudaGetLastError());
        ++launches;
    };
    if (mode == PAIRS_RECT) {   // the rectangle of rows [0, n1) x [n1, n1 + n2): sums only
        SB_CUDA(cudaEventRecord(log.ev0, st));
        // All rows plain: sum over values of (rows of the first set holding
        // it) x (rows of the second set holding it), from two histograms.
        const uint64_t U = ((uint64_t)d.max_cid + 1) * 65536;
        bool plain = postings_mode != 0 && U <= POSTINGS_MAX_UNIVERSE && d.facts.size() == n1 + n2 &&
                     n_pairs_all >= 1024;
        for (uint64_t r = 0; plain && r < n1 + n2; ++r) plain = d.facts[r].plain;
        if (plain) {
            d_counts.reserve(U);
            d_start.reserve(U);
            SB_CUDA(cudaMemsetAsync(d_counts.p, 0, U * sizeof(uint32_t), st));
            SB_CUDA(cudaMemsetAsync(d_start.p, 0, U * sizeof(uint32_t), st));
            d_qrows.reserve(n2);
            std::vector<uint32_t> second(n2);
            for (uint64_t r = 0; r < n2; ++r) second[r] = (uint32_t)(n1 + r);
            SB_CUDA(cudaMemcpyAsync(d_qrows.p, second.data(), n2 * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
            WalkShape ws;
            ws.of(n1 + n2, [&](uint64_t r) -> const ChunkRowFacts& { return d.facts[r]; });
            postings_hist_kernel<<<ws.grid(n1, sms), ROW_WALK_THREADS, 0, st>>>(d.view(), nullptr, ws.dims(n1), d_counts.p);
            postings_hist_kernel<<<ws.grid(n2, sms), ROW_WALK_THREADS, 0, st>>>(d.view(), d_qrows.p, ws.dims(n2),
                                                                              d_start.p);
            counts_dot_kernel<<<sms * 8, 256, 0, st>>>(d_counts.p, d_start.p, U, d_flags.p);
            SB_CUDA(cudaGetLastError());
            launches += 3;
            last_postings_rows = n1 + n2;
        } else {
            uint32_t* keep = d_out;
            d_out = nullptr;
            chunk_launch(PAIRS_RECT, n_pairs_all, nullptr, 0, n1, n1, n2);
            d_out = keep;
        }
        SB_CUDA(cudaEventRecord(log.ev1, st));
        const DeviceFlags f = read_flags(d_flags.p, st);
        SB_CUDA(cudaEventElapsedTime(&log.last_ms, log.ev0, log.ev1));
        log.launches = launches;
        return f.sum;
    }

    // ---- row classes, in walk order [C | L | M | H]:
    //   C  chunk kernel: every pair with a C row (rows with a repeated list
    //      value, or anything the other engines cannot take);
    //   L  postings rows (plain, no bitmap chunk): L x L by value postings;
    //   M  panel rows queried and stored: (L u M) x (M u H) pairs by the
    //      transposed-panel engine (panel.cuh), each pair once;
    //   H  tensor rows: H x H on the tensor cores -- and, in the plan without
    //      a panel, H x L too (the L rows expanded behind the H rows).
    const uint64_t n = n1;
    const uint64_t slots = (uint64_t)d.max_cid + 1;
    const uint64_t U = slots * 65536;                      // universe of the rows' values
    const uint64_t W = slots * CHUNK_WORDS;                // words per expanded row
    const bool facts_ok = d.facts.size() == n;
    const bool tc_ok = dense_min_density != 0.0 && U <= TC_MAX_ROW_BITS && facts_ok;
    const bool post_ok = postings_mode != 0 && U <= POSTINGS_MAX_UNIVERSE && facts_ok;
    const double tc_ns = tensor_pair_ns(cost, slots);
    std::vector<uint8_t> cls(n, 0);                        // 0 C, 1 L, 2 M, 3 H
    if (!ev_hist) SB_CUDA(cudaEventCreate(&ev_hist));
    if (!ev_hist0) SB_CUDA(cudaEventCreate(&ev_hist0));
    bool hist_ran = false;
    last_panel_rows = last_panel_queries = 0;

    SB_CUDA(cudaEventRecord(log.ev0, st));
    PostingsStats ps{};
    WalkShape q_walk;                                      // of the postings rows
    auto walk_of = [&](const std::vector<uint32_t>& rows) {
        WalkShape w;
        w.of(rows.size(), [&](uint64_t k) -> const ChunkRowFacts& { return d.facts[rows[k]]; });
        return w;
    };
    auto histogram = [&](const std::vector<uint32_t>& rows, const WalkShape& shape) {
        d_qrows.reserve(rows.size());
        SB_CUDA(cudaEventRecord(ev_hist0, st));
        SB_CUDA(cudaMemcpyAsync(d_qrows.p, rows.data(), rows.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
        d_counts.reserve(U);
        d_pstats.reserve(1);
        SB_CUDA(cudaMemsetAsync(d_counts.p, 0, U * sizeof(uint32_t), st));
        SB_CUDA(cudaMemsetAsync(d_pstats.p, 0, sizeof(PostingsStats), st));
        q_walk = shape;
        postings_hist_kernel<<<q_walk.grid(rows.size(), sms), ROW_WALK_THREADS, 0, st>>>(
            d.view(), d_qrows.p, q_walk.dims(rows.size()), d_counts.p);
        postings_stats_kernel<<<sms * 8, 256, 0, st>>>(d_counts.p, U, d_pstats.p);
        SB_CUDA(cudaGetLastError());
        SB_CUDA(cudaEventRecord(ev_hist, st));
        hist_ran = true;
        launches += 2;
        PostingsStats h{};
        SB_CUDA(cudaMemcpyAsync(&h, d_pstats.p, sizeof(h), cudaMemcpyDeviceToHost, st));
        SB_CUDA(cudaStreamSynchronize(st));
        return h;
    };
    // Run postings (run_sweep_kernel): bins of 2^rwlog values, the mean run
    // length of the plain list rows rounded to a power of two in [16, 32768]
    // (a run of length l spans about 1 + l / bin bins; the sweep's entry
    // reads, pieces^2 x bin / U for uniform rows, are least at bin = l).
    uint32_t rwlog = 4, most_chunks = 0;
    bool run_gallop = false;
    if (facts_ok) {
        double sc = 0.0, sr = 0.0;
        uint64_t chunks = 0;
        for (uint64_t r = 0; r < n; ++r) {
            const ChunkRowFacts& f = d.facts[r];
            if (f.plain && f.bitmap_chunks == 0) {
                sc += (double)f.card;
                sr += (double)f.runs;
                most_chunks = std::max(most_chunks, f.chunks);
                chunks += f.chunks;
            }
        }
        const double ml = sr > 0.0 ? sc / sr : 1.0;
        rwlog = (uint32_t)std::min(15.0, std::max(4.0, std::round(std::log2(std::max(ml, 1.0)))));
        run_gallop = run_walk_gallops(rwlog, sc, (double)chunks);
    }
    const double RW = (double)(1u << rwlog);
    const uint64_t n_bins = U >> rwlog;
    auto pieces_est = [&](const ChunkRowFacts& f) { return (double)f.runs + (double)f.card / RW; };
    unsigned long long run_entries = 0, run_checks = 0;   // exact, from the piece histogram
    std::vector<uint32_t> h_rpieces;
    bool use_run = false;
    auto run_histogram = [&](const std::vector<uint32_t>& rows) {
        const uint64_t q = rows.size();
        d_qrows.reserve(q);
        SB_CUDA(cudaEventRecord(ev_hist0, st));
        SB_CUDA(cudaMemcpyAsync(d_qrows.p, rows.data(), q * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
        d_rbins.reserve(n_bins);
        d_rpieces.reserve(q);
        d_rstats.reserve(2);
        SB_CUDA(cudaMemsetAsync(d_rbins.p, 0, n_bins * sizeof(uint32_t), st));
        SB_CUDA(cudaMemsetAsync(d_rstats.p, 0, 2 * sizeof(unsigned long long), st));
        d_cpieces.reserve(d.cid.n);
        const uint32_t gq = (uint32_t)std::min<uint64_t>(q, (uint64_t)sms * 64);
        auto count = run_gallop ? run_count_kernel<true> : run_count_kernel<false>;
        count<<<gq, ROW_WALK_THREADS, 0, st>>>(d.view(), d_qrows.p, (uint32_t)q, rwlog, d_rpieces.p,
                                                         d_cpieces.p, d_rbins.p);
        run_stats_kernel<<<sms * 8, 256, 0, st>>>(d_rbins.p, n_bins, d_rstats.p);
        SB_CUDA(cudaGetLastError());
        SB_CUDA(cudaEventRecord(ev_hist, st));
        hist_ran = true;
        launches += 2;
        unsigned long long h[2] = {0, 0};
        h_rpieces.resize(q);
        SB_CUDA(cudaMemcpyAsync(h, d_rstats.p, sizeof(h), cudaMemcpyDeviceToHost, st));
        SB_CUDA(cudaMemcpyAsync(h_rpieces.data(), d_rpieces.p, q * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
        SB_CUDA(cudaStreamSynchronize(st));
        run_entries = h[0];
        run_checks = h[1];
    };
    auto finish = [&](uint64_t extra_sum) {
        SB_CUDA(cudaEventRecord(log.ev1, st));
        const DeviceFlags f = read_flags(d_flags.p, st);
        if (f.error) fail(STORM_B200_ETIMEOUT, "tensor-core dense block: a pipeline wait timed out");
        SB_CUDA(cudaEventElapsedTime(&log.last_ms, log.ev0, log.ev1));
        log.launches = launches;
        return f.sum + extra_sum;
    };

    // Sum-only calls: over every pair of plain rows the sum is
    // sum_v C(rows holding v, 2) -- one value histogram, no pair touched
    // (bitmap chunks count every set bit); pairs with another row run on the
    // chunk kernel.
    if (!d_out && post_ok) {
        std::vector<uint32_t> plain;
        for (uint32_t r = 0; r < n; ++r)
            if (d.facts[r].plain) plain.push_back(r);
        uint64_t q_sum = 0;
        if (plain.size() >= 2) {
            q_sum = histogram(plain, d.plain_walk.of(plain, d.facts)).pairs;
            last_postings_rows = plain.size();
        }
        const uint64_t nc = n - plain.size();
        if (nc) {
            for (uint32_t r : plain) cls[r] = 1;
            std::vector<uint32_t> h_perm;
            h_perm.reserve(n);
            for (int k = 0; k < 2; ++k)
                for (uint32_t r = 0; r < n; ++r)
                    if (cls[r] == k) h_perm.push_back(r);
            d_perm.reserve(n);
            SB_CUDA(cudaMemcpyAsync(d_perm.p, h_perm.data(), n * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
            chunk_launch(PAIRS_TRIANGLE, nc * n - (nc * (nc - 1)) / 2, d_perm.p, 0, 0, n, 0);
        }
        return finish(q_sum);
    }

    // Per-pair form of the postings: increments list by list into the output,
    // or the row sweep (partners counted in shared memory, each output written
    // once), whichever the constants say. Measured on B200, list by list / row
    // sweep (ms, histogram and lists included): 4000 rows of 16777 values over
    // 2^24 3.0 / 3.2, 6000 of 4194 over 2^22 1.2 / 1.3, 8000 of 16777 12.2 / 7.5,
    // 20000 of 1678 2.8 / 1.8, 20000 of 5033 17.2 / 5.7, 20000 of 168 0.27 / 0.56.
    const bool big_out = tri_size(n) * sizeof(uint32_t) > POST_L2_BYTES;
    const double c_list = big_out ? cost.ns_per_posting_pair_hbm : cost.ns_per_posting_pair;
    // The row sweeps count partners in blocks of POST_SWEEP_MAX_ROWS rows,
    // reading each row's lists (or bins) once per block; up to POST16_MAX rows
    // of value postings take one block.
    auto sweep_blocks = [&](uint64_t q) { return (double)((q + POST_SWEEP_MAX_ROWS - 1) / POST_SWEEP_MAX_ROWS); };
    auto sweep_ns = [&](double incr, uint64_t q, double entries) {
        const double reads = entries * cost.ns_per_sweep_entry + incr * cost.ns_per_posting_sweep;
        return (double)q * (double)q * cost.ns_per_sweep_count + (q <= POST16_MAX ? reads : 3.0 * reads * sweep_blocks(q));
    };
    auto sweep_form = [&](double incr, uint64_t q, double entries) {
        if (postings_mode == 2) return false;
        return postings_mode == 3 || sweep_ns(incr, q, entries) < incr * c_list;
    };
    // ns of the postings for a set of q rows of `entries` values with incr
    // increments (sums need only the histogram)
    auto post_ns = [&](double incr, uint64_t q, double entries) {
        const double per_pair = sweep_form(incr, q, entries) ? sweep_ns(incr, q, entries) : incr * c_list;
        return (d_out ? per_pair : 0.0) + entries * cost.ns_per_posting_entry + (double)U * cost.ns_per_universe_value;
    };
    // ns of the tensor cores for h rows among themselves and against m more:
    // whole 256 x 256 tiles, and the rows' expansion
    auto tensor_ns = [&](double h, double m) {
        const double nb = std::ceil(h / 256.0), mb = std::ceil(m / 256.0);
        return h <= 0.0 ? 0.0
                        : tc_ns * 65536.0 * (nb * (nb + 1.0) / 2.0 + nb * mb) +
                              (h + m) * (double)W * 8.0 * cost.ns_per_expand_byte;
    };
    // ns of the run sweep with `checks` entry reads for q rows of `pieces`
    // pieces (per pair only)
    auto run_ns = [&](double checks, uint64_t q, double pieces) {
        return (double)q * (double)q * cost.ns_per_sweep_row_pair + checks * cost.ns_per_run_check * sweep_blocks(q) +
               pieces * cost.ns_per_run_piece + (double)most_chunks * cost.ns_per_run_row_chunk +
               (double)n_bins * cost.ns_per_universe_value;
    };
    auto run_ok = [&](uint64_t q) {
        return d_out != nullptr && q >= 2 && postings_mode != 2 && postings_mode != 3;
    };
    std::vector<uint32_t> qrows, dense, mrows;             // L, H, M
    // L x L for `rest` (plain rows without bitmap chunks) by postings when
    // predicted faster than `alt` ns (or when forced): the run sweep when its
    // estimate beats the value postings' and its exact count (the piece
    // histogram) beats `alt`, else the value postings on their exact count
    // (the value histogram).
    auto values_of = [&](const std::vector<uint32_t>& rows) {
        uint64_t c = 0;
        for (uint32_t r : rows) c += d.facts[r].card;
        return c;
    };
    auto decide = [&](const std::vector<uint32_t>& rest, double alt) -> bool {
        const uint64_t q = rest.size();
        if (q < 2) return false;
        bool lists_only = true;   // the value postings index list chunks only
        for (uint32_t r : rest) lists_only = lists_only && d.facts[r].bitmap_chunks == 0;
        if (run_ok(q)) {
            double P = 0.0, C1 = 0.0, C2 = 0.0;
            for (uint32_t r : rest) {
                const ChunkRowFacts& f = d.facts[r];
                P += pieces_est(f);
                C1 += (double)f.card;
                C2 += (double)f.card * (double)f.card;
            }
            const double run_e = run_ns(P * P * RW / (double)U, q, P);
            const double val_e = post_ns((C1 * C1 - C2) / (2.0 * (double)U), q, C1);
            if (postings_mode == 4 || run_e < val_e || !lists_only) {
                run_histogram(rest);
                if (postings_mode == 4 || postings_mode == 1 || run_ns((double)run_checks, q, P) < alt) {
                    use_run = true;
                    qrows = rest;
                    return true;
                }
            }
        }
        if (!lists_only) return false;
        ps = histogram(rest, walk_of(rest));
        if (ps.entries < (1ull << 32) && (postings_mode > 0 || post_ns((double)ps.pairs, q, (double)values_of(rest)) < alt)) {
            qrows = rest;
            return true;
        }
        return false;
    };
    bool panel_plan = false;
    // The panel's blocks of `rows` panel rows: the bytes that expansion (written,
    // read again) and transposed lines take, and what one query value costs
    // against all of them, in units of a whole block (ns_per_panel_value): a
    // narrow line reads in proportion to its width, the staging of the value
    // does not shrink.
    auto panel_last = [](uint64_t rows) { return rows ? (rows - 1) % PANEL_ROWS + 1 : 0; };
    auto panel_bytes = [&](uint64_t rows) {
        const double lines = (double)(rows - panel_last(rows)) + 64.0 * (rows ? panel_block_words(panel_last(rows)) : 0);
        return (2.0 * (double)rows + lines) * (double)W * 8.0;
    };
    auto panel_blocks = [&](uint64_t rows) {
        if (!rows) return 0.0;
        const uint32_t pw = panel_block_words(panel_last(rows));
        return (double)((rows - 1) / PANEL_ROWS) + (pw == 32 ? 1.0 : pw == 16 ? PANEL_HALF_COST : PANEL_QUARTER_COST);
    };
    // The panel needs a transposed block and some of its rows expanded in HBM.
    const uint64_t px_words = PANEL_ROWS * PANEL_PITCH * std::min<uint64_t>(slots, PANEL_X_SLOTS);
    auto dt_words = [&](uint64_t rows) { return U * panel_block_words(rows); };   // of its widest block
    auto panel_fits = [&](uint64_t rows) {
        if (!facts_ok || panel_mode == 0 || U > PANEL_MAX_UNIVERSE) return false;
        if (d_DT.n >= dt_words(rows) && d_pX.n >= px_words) return true;   // it is there already
        size_t fr = 0, tot = 0;
        SB_CUDA(cudaMemGetInfo(&fr, &tot));
        return (double)((dt_words(rows) + px_words) * sizeof(uint64_t)) < 0.5 * ((double)fr + (double)(d_pX.n + d_DT.n) * sizeof(uint64_t));
    };

    if (panel_mode == 2 && facts_ok && U <= PANEL_MAX_UNIVERSE) {
        // Every plain row in the panel: all their pairs by the transposed
        // panel, rows queried against the blocks after them.
        for (uint32_t r = 0; r < n; ++r)
            if (d.facts[r].plain) mrows.push_back(r);
        panel_plan = true;
    } else if (tc_ok && dense_min_density > 0.0) {
        // Explicit threshold: plain rows with value count >= min_density x U.
        const double min_card = dense_min_density * (double)U;
        std::vector<uint32_t> rest;
        double chunk_rest = 0.0;
        for (uint32_t r = 0; r < n; ++r) {
            const ChunkRowFacts& f = d.facts[r];
            if (!f.plain) continue;
            if ((double)f.card >= min_card) {
                dense.push_back(r);
            } else if (post_ok && f.bitmap_chunks == 0) {
                rest.push_back(r);
                chunk_rest += chunk_self_pair_ns(cost, f, slots);
            }
        }
        if (rest.size() >= 2) decide(rest, 0.5 * ((double)rest.size() - 1.0) * chunk_rest);
    } else if (tc_ok && post_ok) {
        // Plain rows, heaviest first.  Plan A (no panel): rows with bitmap
        // chunks go to H, list rows join H while that lowers tensor time (H x
        // everything) + postings time (increments estimated as for
        // independent uniform rows, sum_{i<j} c_i c_j / U).  Plan B (panel):
        // the top h rows H, the next m rows M, the rest L; every row with a
        // bitmap chunk in H u M.  The cheaper predicted plan runs.
        std::vector<uint32_t> pl;
        pl.reserve(n);
        for (uint32_t r : d.by_card.of(d.facts))
            if (d.facts[r].plain) pl.push_back(r);
        const uint64_t np = pl.size();
        std::vector<double> S1(np + 1, 0.0), S2(np + 1, 0.0), S3(np + 1, 0.0);
        uint64_t lb = 0;                                   // rows [0, lb) hold every bitmap-chunk row
        for (uint64_t t = 0; t < np; ++t) {
            const double c = (double)d.facts[pl[t]].card;
            S1[t + 1] = S1[t] + c;
            S2[t + 1] = S2[t] + c * c;
            S3[t + 1] = S3[t] + pieces_est(d.facts[pl[t]]);
            if (d.facts[pl[t]].bitmap_chunks) lb = t + 1;
        }
        // postings ns of the rows [from, np): the value form (rows without
        // bitmap chunks: from >= lb) or the run form (any plain rows)
        auto post_est = [&](uint64_t from) {
            const uint64_t q = np - from;
            if (q < 2) return 0.0;
            const double r1 = S1[np] - S1[from], r2 = S2[np] - S2[from];
            double v = from >= lb ? post_ns((r1 * r1 - r2) / (2.0 * (double)U), q, r1) : HUGE_VAL;
            if (run_ok(q)) {
                const double P = S3[np] - S3[from];
                v = std::min(v, run_ns(P * P * RW / (double)U, q, P));
            }
            return v;
        };
        // Plan A: H = [0, k); the rows below k by postings.
        uint64_t best_k = lb;
        double best_a = -1.0;
        // H fills whole tiles: every 256th row, and the two ends
        for (uint64_t k = 0; k <= np; k = k == np ? np + 1 : std::min(np, (k < lb && k + 256 > lb) ? lb : k / 256 * 256 + 256)) {
            const double v = tensor_ns((double)k, (double)(np - k)) + post_est(k);
            if (best_a < 0 || v < best_a) {
                best_a = v;
                best_k = k;
            }
        }
        if (postings_mode == 4) best_k = 0;                // forced: every plain row to the run sweep
        else if (postings_mode > 0) best_k = lb;           // forced: every list row to the postings
        // ns of the panel over the rows [0, e) (H the first h of them), queried by
        // M among themselves and by all that follow
        auto panel_ns = [&](uint64_t h, uint64_t e) {
            const double m = (double)(e - h), hh = (double)h, nl = (double)(np - e), nb = panel_blocks(e);
            const double sl = S1[np] - S1[e], sm = S1[e] - S1[h];
            return cost.ns_per_panel_value * (sl * nb + sm * std::min(nb, (hh + 0.5 * m) / PANEL_ROWS + 0.5)) +
                   cost.ns_per_panel_pair * (nl * (double)e + m * (m - 1.0) / 2.0 + m * hh) +
                   cost.ns_per_panel_byte * panel_bytes(e) + cost.ns_panel_fixed;
        };
        // Plan B over candidate cuts (h, m).
        uint64_t best_h = 0, best_m = 0;
        double best_b = -1.0;
        if (postings_mode < 0 && panel_mode != 0 && facts_ok && U <= PANEL_MAX_UNIVERSE) {
            // cuts: every 12 %, and where the tensor tiles and the narrow blocks end
            std::vector<uint64_t> cand{0, lb, np};
            for (double x = 1.0; x < (double)np; x *= 1.12) cand.push_back((uint64_t)x);
            for (uint64_t x = 256; x < np && x <= 2 * PANEL_ROWS; x += 256) cand.push_back(x);
            std::sort(cand.begin(), cand.end());
            cand.erase(std::unique(cand.begin(), cand.end()), cand.end());
            for (uint64_t e : cand) {                      // e = h + m; rows past e: postings (value or run form)
                if (e == 0 || e > np) continue;
                const double rest_ns = post_est(e);
                for (uint64_t h : cand) {
                    if (h > e) break;
                    if (panel_mode > 0 && e == h) break;   // forced: some rows in M
                    const double v = tensor_ns((double)h, 0.0) + panel_ns(h, e) + rest_ns;
                    if (best_b < 0 || v < best_b) {
                        best_b = v;
                        best_h = h;
                        best_m = e - h;
                    }
                }
            }
        }
        // The estimates are within 10 % of the times where the plans are close.
        // The free memory is asked for last: the query takes up to milliseconds.
        panel_plan = best_b >= 0 && (panel_mode > 0 || best_b < 0.9 * best_a) && panel_fits(best_h + best_m);
        std::vector<uint32_t> rest;
        if (panel_plan) {
            dense.assign(pl.begin(), pl.begin() + best_h);
            mrows.assign(pl.begin() + best_h, pl.begin() + best_h + best_m);
        } else {
            dense.assign(pl.begin(), pl.begin() + best_k);
        }
        {                                                  // stored order: ascending output writes
            std::vector<uint8_t> is_rest(n, 0);
            for (uint64_t t = panel_plan ? best_h + best_m : best_k; t < np; ++t) is_rest[pl[t]] = 1;
            for (uint32_t r = 0; r < n; ++r)
                if (is_rest[r]) rest.push_back(r);
        }
        if (rest.size() >= 2) {
            // The estimate assumes independent rows; correlated rows share
            // more. With the exact count, keep the postings only if they beat
            // the alternative on these pairs: the panel with these rows in it
            // too (more lines, a wider block) or the tensor cores.
            const double alt = panel_plan ? panel_ns(best_h, np) - panel_ns(best_h, best_h + best_m)
                                          : tensor_ns((double)rest.size(), 0.0);
            if (decide(rest, alt)) rest.clear();
        }
        if (panel_plan && !rest.empty()) {                 // they join the panel, or all go to the tensor cores
            panel_plan = rows_join_panel(panel_mode > 0, tensor_ns((double)best_h, 0.0) + panel_ns(best_h, np),
                                         tensor_ns((double)np, 0.0), [&] { return panel_fits(np); });
            mrows.insert(mrows.end(), rest.begin(), rest.end());
            if (!panel_plan) {
                dense.insert(dense.end(), mrows.begin(), mrows.end());
                mrows.clear();
            }
        } else {
            dense.insert(dense.end(), rest.begin(), rest.end());
        }
    } else if (tc_ok) {
        // Per-row rule: plain rows whose chunk-kernel cost against a row
        // like themselves exceeds a tensor-core pair.
        for (uint32_t r = 0; r < n; ++r) {
            const ChunkRowFacts& f = d.facts[r];
            if (f.plain && chunk_self_pair_ns(cost, f, slots) >= tc_ns) dense.push_back(r);
        }
    } else if (post_ok) {
        std::vector<uint32_t> rest;
        double chunk_rest = 0.0;
        for (uint32_t r = 0; r < n; ++r) {
            const ChunkRowFacts& f = d.facts[r];
            if (f.plain && f.bitmap_chunks == 0) {
                rest.push_back(r);
                chunk_rest += chunk_self_pair_ns(cost, f, slots);
            }
        }
        if (rest.size() >= 2) decide(rest, 0.5 * ((double)rest.size() - 1.0) * chunk_rest);
    }
    if (panel_plan && mrows.empty() && dense.empty()) panel_plan = false;
    // Rows the tensor cores expand behind the H rows: the L rows in the plan
    // without a panel (H x L on the tensor cores), none with it.
    const std::vector<uint32_t> none;
    const std::vector<uint32_t>& tq = panel_plan ? none : qrows;
    // The tensor cores take H x H (and H x tq): expanded rows in the order
    // [H | padding to a multiple of 256 | tq], so that every 128-row and
    // 256-row block is all H or all tq and the tq x tq blocks can be left out.
    // Panels of P rows when they do not all fit the budget.
    if (panel_plan) {
        d_pX.reserve(px_words);
        d_DT.reserve(dt_words(mrows.size() + dense.size()));
    }
    const uint64_t nd0 = dense.size();
    const uint64_t nd_pad = round_up(nd0, 256);
    const uint64_t ne = nd0 ? nd_pad + tq.size() : 0;
    uint64_t P = 0;
    if (ne) {
        uint64_t budget = dense_budget_bytes;
        if (!budget && d_panel.n >= round_up(ne, 256) * panel_row_words(W)) {
            budget = d_panel.n * sizeof(uint64_t);   // they fit the buffer of an earlier call
        } else if (!budget) {
            size_t fr = 0, tot = 0;
            SB_CUDA(cudaMemGetInfo(&fr, &tot));
            budget = (uint64_t)(0.6 * (double)(fr + d_panel.n * sizeof(uint64_t)));
        }
        const uint64_t cap_rows = budget / (panel_row_words(W) * sizeof(uint64_t));
        P = round_up(ne, 256) <= cap_rows ? round_up(ne, 256) : cap_rows / 2 / 256 * 256;
        if (P == 0) {   // not even two panels fit: the H rows go to the chunk kernel (or the panel)
            if (panel_plan) mrows.insert(mrows.end(), dense.begin(), dense.end());
            dense.clear();
        }
    }
    for (uint32_t r : qrows) cls[r] = 1;
    for (uint32_t r : mrows) cls[r] = 2;
    for (uint32_t r : dense) cls[r] = 3;
    // Walk order: C, L, M, H rows.
    std::vector<uint32_t> h_perm;
    h_perm.reserve(n);
    for (int k = 0; k < 4; ++k)
        for (uint32_t r = 0; r < n; ++r)
            if (cls[r] == k) h_perm.push_back(r);
    const uint64_t nd = dense.size(), nq = qrows.size(), nm = mrows.size(), nc = n - nd - nq - nm;
    const uint32_t* perm = nullptr;
    if (nd || nq || nm) {
        d_perm.reserve(n);
        SB_CUDA(cudaMemcpyAsync(d_perm.p, h_perm.data(), n * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
        perm = d_perm.p;
        // The tensor cores (stream-K) and the list form add into the triangle;
        // a row sweep over every row writes all of it.
        const bool swept = nq == n && (use_run || sweep_form((double)ps.pairs, nq, (double)values_of(qrows)));
        if (d_out && !swept) SB_CUDA(cudaMemsetAsync(d_out, 0, tri_size(n) * sizeof(uint32_t), st));
    }

    // ---- predicted device time of each engine for this plan
    for (int k = 0; k < 4; ++k) last_engine_ms[k] = last_engine_pred_ms[k] = last_engine_work[k] = 0.0;
    for (cudaEvent_t& e : ev_eng)
        if (!e) SB_CUDA(cudaEventCreate(&e));
    {
        const double dd = (double)nd, tqn = (double)tq.size();
        last_engine_pred_ms[0] = 1e-6 * tensor_ns(dd, tqn);
        last_engine_work[0] = 2.0 * (dd * (dd + 1.0) / 2.0 + dd * tqn) * (double)U;
        last_engine_work[1] = (double)(nc * n - (nc * (nc - 1)) / 2 * (nc ? 1 : 0));
        if (panel_plan && (nm || nd) && (nq + nm)) {
            const uint64_t npw = nm + nd;
            double vb = 0.0, lines = 0.0, pairs = 0.0;
            for (uint64_t w = nc; w < nc + nq + nm; ++w) {
                const uint64_t after = std::min<uint64_t>(n - 1 - w, npw);   // panel rows after it
                const uint64_t skip = (npw - after) / PANEL_ROWS * PANEL_ROWS;   // in blocks it is not queried against
                const double c = (double)d.facts[h_perm[w]].card;
                vb += c * panel_blocks(npw - skip);
                lines += c * 8.0 * (double)((npw - skip - panel_last(npw)) / 64 + panel_block_words(panel_last(npw)));
                pairs += (double)after;
            }
            last_engine_pred_ms[2] = 1e-6 * (cost.ns_per_panel_value * vb + cost.ns_per_panel_pair * pairs +
                                             panel_bytes(npw) * cost.ns_per_panel_byte);
            last_engine_work[2] = lines + 4.0 * pairs + panel_bytes(npw);
        }
        if (nq && use_run) {
            // run sweep: the pieces (8 B each, written and read), the bin
            // entries each piece reads (8 B), 4 B per count of the slice
            double pcs = 0.0;
            for (uint32_t k : h_rpieces) pcs += (double)k;
            last_engine_pred_ms[3] = 1e-6 * run_ns((double)run_checks, nq, pcs);
            last_engine_work[3] = 16.0 * pcs + 8.0 * (double)run_entries + 8.0 * (double)run_checks +
                                  4.0 * (double)nq * ((double)nq + 1.0) / 2.0 + 4.0 * (double)n_bins;
        } else if (nq) {
            last_engine_pred_ms[3] = 1e-6 * post_ns((double)ps.pairs, nq, (double)values_of(qrows));
            double vals = 0.0;
            for (uint32_t r : qrows) vals += (double)d.facts[r].card;
            last_engine_work[3] = 8.0 * vals + 8.0 * (double)ps.entries + 8.0 * (double)ps.pairs + 8.0 * (double)U;
        }
    }
    SB_CUDA(cudaEventRecord(ev_eng[0], st));   // the postings' histogram and the set-up precede it

    // ---- tensor cores: H x H and H x tq, panel by panel
    if (nd) {
        std::vector<uint32_t> emap(nd_pad + tq.size(), ~0u);   // expanded row -> stored row (~0: padding)
        std::copy(dense.begin(), dense.end(), emap.begin());
        std::copy(tq.begin(), tq.end(), emap.begin() + nd_pad);
        const uint64_t ne2 = emap.size();
        const bool single = P >= round_up(ne2, 256);
        const uint64_t rows_alloc = single ? P : 2 * P;
        // Block-major panels: chunk slot s of every expanded row together,
        // rows PANEL_PITCH words apart within it (see panel_row_words).
        const RowLayout lay{PANEL_PITCH, rows_alloc * PANEL_PITCH};
        d_panel.reserve(rows_alloc * panel_row_words(W));
        d_map.reserve(rows_alloc);
        const uint32_t bm = rows_block_a((uint32_t)W);
        d_tiles.reserve((P / 128) * (2 * P / 256 + 1));
        const uint64_t npan = single ? 1 : (ne2 + P - 1) / P;
        auto is_q = [&](uint64_t global_row) { return global_row >= nd_pad; };
        std::vector<uint2> tl;
        auto expand = [&](uint64_t first, uint64_t m, uint64_t slot) {
            SB_CUDA(cudaMemcpyAsync(d_map.p + slot, emap.data() + first, m * sizeof(uint32_t),
                                    cudaMemcpyHostToDevice, st));
            const uint32_t grid = (uint32_t)std::min<uint64_t>((m * slots + EXPAND_WARPS - 1) / EXPAND_WARPS,
                                                               (uint64_t)sms * 64);
            expand_rows_kernel<<<grid, EXPAND_WARPS * 32, 0, st>>>(d.view(), d_map.p + slot, (uint32_t)m, 0u,
                                                                   (uint32_t)slots, (uint32_t)slots, lay,
                                                                   d_panel.p + slot * lay.pitch);
            SB_CUDA(cudaGetLastError());
            ++launches;
        };
        auto tensor = [&](uint64_t n_local) {
            if (tl.empty()) return;
            SB_CUDA(cudaMemcpyAsync(d_tiles.p, tl.data(), tl.size() * sizeof(uint2), cudaMemcpyHostToDevice, st));
            launch_ts_rows(d_panel.p, (uint32_t)n_local, (uint32_t)W, lay, d_tiles.p, (uint32_t)tl.size(), d_out,
                           d_flags.p, d_map.p, n, st, /*out_zeroed=*/true);
            ++launches;
        };
        for (uint64_t I = 0; I < npan; ++I) {
            const uint64_t gI = I * P, mI = std::min<uint64_t>(P, ne2 - gI);
            if (is_q(gI)) break;                          // this and later panels are all tq
            expand(gI, mI, 0);
            std::vector<uint2> tri;
            build_rows_tiles(tri, mI, (uint32_t)W);        // I x I triangle, tq x tq blocks left out
            tl.clear();
            for (const uint2& t : tri)
                if (!(is_q(gI + (uint64_t)t.x * bm) && is_q(gI + (uint64_t)t.y * 256))) tl.push_back(t);
            tensor(mI);
            for (uint64_t J = I + 1; J < npan; ++J) {      // I x J rectangle (I is a full panel)
                const uint64_t gJ = J * P, mJ = std::min<uint64_t>(P, ne2 - gJ);
                expand(gJ, mJ, P);
                tl.clear();
                for (uint32_t bi = 0; bi < P / bm; ++bi) {
                    if (is_q(gI + (uint64_t)bi * bm) && is_q(gJ)) continue;
                    for (uint32_t bj = (uint32_t)(P / 256); bj < (uint32_t)((P + mJ + 255) / 256); ++bj)
                        if (!(is_q(gI + (uint64_t)bi * bm) && is_q(gJ + (uint64_t)bj * 256 - P)))
                            tl.push_back(make_uint2(bi, bj));
                }
                tensor(P + mJ);
            }
        }
        last_dense_rows = nd;
        last_dense_panels = npan;
    }
    SB_CUDA(cudaEventRecord(ev_eng[1], st));
    // ---- chunk kernel: every pair with a C row (the walk's triangle prefix)
    chunk_launch(PAIRS_TRIANGLE, nc * n - (nc * (nc - 1)) / 2 * (nc ? 1 : 0), perm, 0, 0, n, 0);
    SB_CUDA(cudaEventRecord(ev_eng[2], st));
    // ---- transposed panel: (L u M) x (M u H), blocks of PANEL_ROWS panel rows
    if (panel_plan && (nm || nd) && (nq + nm)) {
        const uint64_t pw0 = nc + nq;                      // walk position of the first panel row
        const uint64_t npw = nm + nd;
        // Work items over the query rows (walk positions of L and M),
        // heaviest first: a row with more than `seg` values is split into
        // ranges of its chunks (about seg values each), so that the warps
        // finish together; seg is sized for ~64 items per SM and at least
        // PANEL_MIN_SEG values (the per-item epilogue costs about as much as
        // a few hundred values), and doubled until the split rows' scratch
        // slots fit PANEL_MAX_SLOTS.
        double total = 0.0;
        for (uint64_t w = nc; w < nc + nq + nm; ++w) total += (double)d.facts[h_perm[w]].card;
        std::vector<PanelItem> items;
        std::vector<PanelSplit> splits;
        std::vector<double> weight;
        uint32_t nslots = 0;
        for (uint64_t seg = std::max<uint64_t>(PANEL_MIN_SEG, (uint64_t)(total / (64.0 * sms)));; seg *= 2) {
            items.clear();
            splits.clear();
            weight.clear();
            nslots = 0;
            for (uint64_t w = nc; w < nc + nq + nm; ++w) {
                const ChunkRowFacts& f = d.facts[h_perm[w]];
                const uint32_t ns =
                    f.card > seg && f.chunks > 1 ? (uint32_t)std::min<uint64_t>(f.chunks, (f.card + seg - 1) / seg) : 1u;
                if (ns == 1) {
                    items.push_back(PanelItem{(uint32_t)w, 0u, f.chunks, PANEL_NO_VALUE});
                    weight.push_back((double)f.card);
                    continue;
                }
                splits.push_back(PanelSplit{(uint32_t)w, nslots, ns, 0u});
                for (uint32_t k = 0; k < ns; ++k) {
                    const uint32_t lo = (uint32_t)((uint64_t)f.chunks * k / ns);
                    const uint32_t hi = (uint32_t)((uint64_t)f.chunks * (k + 1) / ns);
                    items.push_back(PanelItem{(uint32_t)w, lo, hi, nslots + k});
                    weight.push_back((double)f.card * (double)(hi - lo) / (double)f.chunks);
                }
                nslots += ns;
            }
            if (nslots <= PANEL_MAX_SLOTS) break;
        }
        {
            std::vector<uint32_t> ord(items.size());
            for (uint32_t k = 0; k < ord.size(); ++k) ord[k] = k;
            std::stable_sort(ord.begin(), ord.end(), [&](uint32_t x, uint32_t y) { return weight[x] > weight[y]; });
            std::vector<PanelItem> sorted(items.size());
            for (uint32_t k = 0; k < ord.size(); ++k) sorted[k] = items[ord[k]];
            items.swap(sorted);
        }
        d_items.reserve(items.size());
        d_ctr.reserve(1);
        d_pmap.reserve(PANEL_ROWS);
        SB_CUDA(cudaMemcpyAsync(d_items.p, items.data(), items.size() * sizeof(PanelItem), cudaMemcpyHostToDevice, st));
        if (!splits.empty()) {
            d_splits.reserve(splits.size());
            d_pscratch.reserve((uint64_t)nslots * PANEL_ROWS);
            SB_CUDA(cudaMemcpyAsync(d_splits.p, splits.data(), splits.size() * sizeof(PanelSplit),
                                    cudaMemcpyHostToDevice, st));
        }
        static std::atomic<uint64_t> t_done{0};
        smem_attr_once(panel_transpose_kernel<32>, (int)panel_t_smem(32), t_done);
        for (uint64_t b0 = 0; b0 < npw; b0 += PANEL_ROWS) {
            const uint32_t prows = (uint32_t)std::min<uint64_t>(PANEL_ROWS, npw - b0);
            const uint32_t pw = panel_block_words(prows);
            SB_CUDA(cudaMemcpyAsync(d_pmap.p, h_perm.data() + pw0 + b0, prows * sizeof(uint32_t), cudaMemcpyHostToDevice,
                                    st));
            // PANEL_X_SLOTS chunk slots at a time, block-major as the tensor
            // panels: the expanded rows of a whole block would take as much
            // memory as the block itself, and its allocation 20 ms of a
            // container's first call.
            const RowLayout play{PANEL_PITCH, PANEL_ROWS * PANEL_PITCH};
            for (uint32_t s0 = 0; s0 < slots; s0 += PANEL_X_SLOTS) {
                const uint32_t ns = (uint32_t)std::min<uint64_t>(PANEL_X_SLOTS, slots - s0);
                const uint32_t items = (prows * ns + EXPAND_WARPS - 1) / EXPAND_WARPS;
                expand_rows_kernel<<<std::min(items, (uint32_t)sms * 64), EXPAND_WARPS * 32, 0, st>>>(
                    d.view(), d_pmap.p, prows, s0, ns, (uint32_t)slots, play, d_pX.p);
                auto transpose = pw == 32 ? panel_transpose_kernel<32> : pw == 16 ? panel_transpose_kernel<16>
                                                                                  : panel_transpose_kernel<8>;
                transpose<<<ns * CHUNK_WORDS / PANEL_T_WORDS, pw * 32, panel_t_smem(pw), st>>>(
                    d_pX.p, play, prows, d_DT.p + (uint64_t)s0 * CHUNK_WORDS * 64 * pw);
                launches += 2;
            }
            SB_CUDA(cudaMemsetAsync(d_ctr.p, 0, sizeof(unsigned long long), st));
            const uint32_t ni = (uint32_t)items.size();
            uint32_t* scr = splits.empty() ? nullptr : d_pscratch.p;
            auto query = [&](auto kernel) {
                kernel<<<(uint32_t)sms * (PANEL_Q_SMEM_SM / (panel_q_smem(pw) + 1024)), 32, panel_q_smem(pw), st>>>(d.view(), perm, d_items.p, ni, pw0 + b0, prows, d_DT.p, n,
                                                             d_out, scr, d_flags.p, d_ctr.p);
            };
            if (pw == 32) query(panel_query_kernel<32>);
            else if (pw == 16) query(panel_query_kernel<16>);
            else query(panel_query_kernel<8>);
            launches += 1;
            if (scr && d_out) {
                panel_reduce_kernel<<<(uint32_t)std::min<uint64_t>(splits.size(), (uint64_t)sms * 8), 256, 0, st>>>(
                    perm, d_splits.p, (uint32_t)splits.size(), pw0 + b0, prows, scr, n, d_out);
                ++launches;
            }
            SB_CUDA(cudaGetLastError());
        }
        last_panel_rows = npw;
        last_panel_queries = nq + nm;
    }
    SB_CUDA(cudaEventRecord(ev_eng[3], st));
    // ---- L x L by postings
    uint64_t q_sum = 0;
    last_postings_form = -1;
    if (nq && use_run) {
        // run sweep (the sum over these pairs is added by the kernel)
        last_postings_form = 2;
        std::vector<uint64_t> poff(nq + 1, 0);
        for (uint64_t k = 0; k < nq; ++k) poff[k + 1] = poff[k] + h_rpieces[k];
        d_rpoff.reserve(nq + 1);
        SB_CUDA(cudaMemcpyAsync(d_rpoff.p, poff.data(), (nq + 1) * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
        d_pieces.reserve(poff[nq] ? poff[nq] : 1);
        d_rstart.reserve(n_bins);
        d_rlist.reserve(run_entries ? run_entries : 1);
        d_pstats.reserve(1);
        SB_CUDA(cudaMemsetAsync(d_pstats.p, 0, sizeof(PostingsStats), st));
        const uint32_t gq = (uint32_t)std::min<uint64_t>((nq + 7) / 8, (uint64_t)sms * 16);
        auto fill = run_gallop ? run_fill_kernel<true> : run_fill_kernel<false>;
        fill<<<(uint32_t)std::min<uint64_t>(nq, (uint64_t)sms * 64), ROW_WALK_THREADS, 0, st>>>(
            d.view(), d_qrows.p, (uint32_t)nq, rwlog, d_rpoff.p, d_cpieces.p, d_pieces.p);
        postings_alloc_kernel<<<sms * 8, ALLOC_THREADS, 0, st>>>(d_rbins.p, n_bins, d_rstart.p, nullptr, nullptr, d_pstats.p);
        run_scatter_kernel<<<gq, 256, 0, st>>>((uint32_t)nq, rwlog, d_rpoff.p, d_pieces.p, d_rstart.p, d_rlist.p);
        static std::atomic<uint64_t> done{0};
        smem_attr_once(run_sweep_kernel, (int)((POST_SWEEP_MAX_ROWS + RUN_SWEEP_BATCH + 1) * sizeof(uint32_t)), done);
        const uint32_t gr = (uint32_t)std::min<uint64_t>(nq, (uint64_t)sms * 8);
        for (uint64_t pb0 = 0; pb0 < nq; pb0 += POST_SWEEP_MAX_ROWS) {
            const uint32_t pbn = (uint32_t)std::min<uint64_t>(POST_SWEEP_MAX_ROWS, nq - pb0);
            const uint32_t smem = (uint32_t)((pbn + RUN_SWEEP_BATCH + 1) * sizeof(uint32_t));
            run_sweep_kernel<<<gr, POST_SWEEP_THREADS, smem, st>>>(d_qrows.p, (uint32_t)nq, d_rpoff.p, d_pieces.p,
                                                                   rwlog, d_rbins.p, d_rstart.p, d_rlist.p, n, d_out,
                                                                   d_flags.p, (uint32_t)pb0, pbn);
            ++launches;
        }
        SB_CUDA(cudaGetLastError());
        launches += 3;
        last_postings_rows = nq;
    } else if (nq) {
        q_sum = ps.pairs;
        const bool sweep = sweep_form((double)ps.pairs, nq, (double)values_of(qrows));
        last_postings_form = sweep ? 1 : 0;
        if (d_out) {
            d_start.reserve(U);
            uint64_t most = 0;
            for (uint32_t r : qrows) most = std::max(most, d.facts[r].card);
            // without room for the entries' lists: the sweep that looks them up
            const bool sweep16 = sweep && nq <= POST16_MAX && most <= POST16_MAX &&
                                 ps.entries + ps.lists < 0xFFFFFFFFull &&
                                 reserve_both(d_post16, ps.entries + ps.lists + 8, d_place, d.lst.n);
            if (!sweep16) {
                if (!sweep) d_lists.reserve(ps.lists ? ps.lists : 1);
                d_post.reserve(ps.entries ? ps.entries : 1);
            }
            postings_alloc_kernel<<<sms * 8, ALLOC_THREADS, 0, st>>>(d_counts.p, U, d_start.p, sweep ? nullptr : d_lists.p,
                                                                    sweep16 ? d_post16.p : nullptr, d_pstats.p);
            if (sweep16) {
                SB_CUDA(cudaMemsetAsync(d_place.p, 0xFF, d.lst.n * sizeof(uint32_t), st));
                postings_scatter16_kernel<<<q_walk.grid(nq, sms), ROW_WALK_THREADS, 0, st>>>(
                    d.view(), d_qrows.p, q_walk.dims(nq), d_counts.p, d_start.p, d_post16.p, d_place.p);
                static std::atomic<uint64_t> done16{0};
                smem_attr_once(postings_rows16_kernel, (int)((POST16_MAX + 1) * sizeof(uint16_t)), done16);
                postings_rows16_kernel<<<(uint32_t)std::min<uint64_t>(nq, (uint64_t)sms * 16), POST_ROWS_THREADS,
                                         (nq + 1) / 2 * sizeof(uint32_t), st>>>(
                    d.view(), d_qrows.p, (uint32_t)nq, nq == n, d_place.p, d_post16.p, n, d_out);
                SB_CUDA(cudaGetLastError());
                launches += 3;
            } else {
                postings_scatter_kernel<<<q_walk.grid(nq, sms), ROW_WALK_THREADS, 0, st>>>(
                    d.view(), d_qrows.p, q_walk.dims(nq), d_start.p, d_post.p);
                if (sweep) {
                    const bool small = most <= 0xFFFF;   // a count is at most its row's values
                    static std::atomic<uint64_t> done_s{0}, done_l{0};
                    const int smem_max = (int)(POST_SWEEP_MAX_ROWS * sizeof(uint32_t));
                    smem_attr_once(postings_rows_kernel<true>, smem_max / 2, done_s);
                    smem_attr_once(postings_rows_kernel<false>, smem_max, done_l);
                    const uint32_t gr = (uint32_t)std::min<uint64_t>(nq, (uint64_t)sms * 16);
                    // a row's groups over all the warps of its CTA
                    const uint32_t warps = POST_ROWS_THREADS / 32, chunks = q_walk.group * q_walk.groups;
                    const uint32_t group =
                        q_walk.group == 1 ? 1u : std::max(2u, std::min(32u, (chunks + warps - 1) / warps));
                    for (uint64_t pb0 = 0; pb0 < nq; pb0 += POST_SWEEP_MAX_ROWS) {
                        const uint32_t pbn = (uint32_t)std::min<uint64_t>(POST_SWEEP_MAX_ROWS, nq - pb0);
                        const uint32_t smem = (uint32_t)(small ? (pbn + 1) / 2 : pbn) * sizeof(uint32_t);
                        auto kernel = small ? postings_rows_kernel<true> : postings_rows_kernel<false>;
                        kernel<<<gr, POST_ROWS_THREADS, smem, st>>>(d.view(), d_qrows.p, (uint32_t)nq, nq == n, group,
                                                                   d_counts.p, d_start.p, d_post.p, n, d_out, (uint32_t)pb0,
                                                                   pbn);
                        ++launches;
                    }
                    launches += 2;
                } else {
                    const uint32_t gp = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((ps.lists + 255) / 256,
                                                                                           (uint64_t)sms * 16));
                    postings_pairs_kernel<<<gp, 256, 0, st>>>(d_lists.p, ps.lists, d_post.p, d_qrows.p, n, d_out);
                    postings_diag_kernel<<<(uint32_t)std::min<uint64_t>((nq + 255) / 256, (uint64_t)sms * 4), 256, 0,
                                           st>>>(d.view(), d_qrows.p, (uint32_t)nq, n, d_out);
                    launches += 4;
                }
            }
            SB_CUDA(cudaGetLastError());
        }
        last_postings_rows = nq;
    }
    // ---- diagonal of the M rows (no other engine pairs them with themselves)
    if (nm && d_out) {
        d_mrows.reserve(nm);
        SB_CUDA(cudaMemcpyAsync(d_mrows.p, h_perm.data() + nc + nq, nm * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
        row_card_diag_kernel<<<(uint32_t)std::min<uint64_t>((nm + 7) / 8, (uint64_t)sms * 16), 256, 0, st>>>(
            d.view(), d_mrows.p, (uint32_t)nm, n, d_out);
        SB_CUDA(cudaGetLastError());
        ++launches;
    }
    const uint64_t total = finish(q_sum);
    float t_pre = 0, t_hist = 0, t_tc = 0, t_ch = 0, t_pa = 0, t_po = 0;
    SB_CUDA(cudaEventElapsedTime(&t_pre, log.ev0, ev_eng[0]));
    if (hist_ran) SB_CUDA(cudaEventElapsedTime(&t_hist, ev_hist0, ev_hist));
    SB_CUDA(cudaEventElapsedTime(&t_tc, ev_eng[0], ev_eng[1]));
    SB_CUDA(cudaEventElapsedTime(&t_ch, ev_eng[1], ev_eng[2]));
    SB_CUDA(cudaEventElapsedTime(&t_pa, ev_eng[2], ev_eng[3]));
    SB_CUDA(cudaEventElapsedTime(&t_po, ev_eng[3], log.ev1));
    last_engine_ms[0] = t_tc;
    last_engine_ms[1] = t_ch;
    last_engine_ms[2] = t_pa;
    last_engine_ms[3] = t_po + (nq ? t_hist : 0.f);
    // the rest of the time before the engines: planning on the host while
    // the GPU waits (before the histogram and after its statistics are read
    // back), the row order's upload and the output's clearing
    last_plan_ms = nq ? t_pre - t_hist : t_pre;
    return total;
}

}  // namespace sb200
