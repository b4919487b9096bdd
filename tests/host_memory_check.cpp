// Host-only check of what the library does when device memory runs out, on a
// fake of the CUDA calls that hand memory out (no GPU, no CUDA runtime): a
// budget of bytes, and a record of what is held. Built and run by
// test_host_memory_cpu.py.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <thread>

#include "colsum.cuh"
#include "dense.cuh"

static int g_fail = 0;
#define CHECK(c)                                             \
    do {                                                     \
        if (!(c)) {                                          \
            std::printf("line %d: %s\n", __LINE__, #c);      \
            ++g_fail;                                        \
        }                                                    \
    } while (0)

static std::map<void*, size_t> g_held;
static std::set<void*> g_registered;
static size_t g_used = 0, g_budget = 0;
static cudaError_t g_error = cudaSuccess, g_refusal = cudaErrorMemoryAllocation;

extern "C" {
cudaError_t cudaMalloc(void** p, size_t bytes) {
    if (g_used + bytes > g_budget) return g_error = g_refusal;
    *p = std::malloc(bytes ? bytes : 1);
    g_held[*p] = bytes;
    g_used += bytes;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    CHECK(g_held.count(p));
    g_used -= g_held[p];
    g_held.erase(p);
    std::free(p);
    return cudaSuccess;
}
// CUDA's own pinned memory goes with the device; registered memory is the caller's.
cudaError_t cudaMallocHost(void** p, size_t bytes) { return cudaMalloc(p, bytes); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaHostRegister(void* p, size_t, unsigned int) {
    if (g_budget == 0) return g_error = cudaErrorNotSupported;
    g_registered.insert(p);
    return cudaSuccess;
}
cudaError_t cudaHostUnregister(void* p) {
    if (!g_registered.erase(p)) return g_error = cudaErrorHostMemoryNotRegistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t bytes, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(dst, src, bytes);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = g_error;
    g_error = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}

namespace sb200 {
DeviceFlags* flags_slot() {                                      // as runtime.cu keeps it
    static thread_local RegisteredPage page;
    return static_cast<DeviceFlags*>(page.p);
}
}  // namespace sb200

using namespace sb200;

static void buffers_a_call_can_do_without() {
    DevBuf<uint32_t> b;
    g_budget = 400;
    CHECK(b.try_reserve(100) && b.n == 100 && g_used == 400);
    CHECK(b.try_reserve(50) && b.n == 100);                      // large enough as it is
    CHECK(!b.try_reserve(101) && b.p == nullptr && b.n == 0 && g_used == 0);
    CHECK(g_error == cudaSuccess);                               // nothing left for the next launch's check
    g_refusal = cudaErrorUnknown;
    bool threw = false;
    try {
        b.try_reserve(101);
    } catch (const Status& e) {
        threw = e.code == STORM_B200_ECUDA;
    }
    CHECK(threw);                                                // any other failure is one
    g_refusal = cudaErrorMemoryAllocation;
    g_error = cudaSuccess;
}

// The 16-bit row sweep's buffers (2 bytes per list place, 4 per list entry) and
// then the look-up sweep's (4 per place), in memory that holds the first or the
// third of them but not the first two.
static void sweep_buffers() {
    const size_t places = 1000, entries = 3000;
    DevBuf<uint16_t> post16;
    DevBuf<uint32_t> place, post;
    g_budget = 5000;
    CHECK(!reserve_both(post16, places, place, entries));
    CHECK(g_used == 0 && post16.p == nullptr && place.p == nullptr);
    post.reserve(places);                                        // would throw beside a kept post16
    CHECK(post.n == places);
    post.release();
    g_budget = 14000;
    CHECK(reserve_both(post16, places, place, entries) && g_used == 14000);
}

// Host rows cross the bus by way of a staging buffer, or without one.
static void staged_rows() {
    DevBuf<uint64_t> stage;
    g_budget = 300 * 313 * 8 - 1;
    CHECK(row_stage(stage, 300, 313) == nullptr && g_used == 0);
    g_budget = 300 * 313 * 8;
    CHECK(row_stage(stage, 300, 313) == stage.p && stage.p);
    CHECK(row_stage(stage, 1, ROW_STAGE_WORDS + 1) == nullptr);  // long rows: straight to their places
    for (uint32_t wpr : {8u, 64u, 312u, 400u, 512u, 632u})       // and rows of whole 64 bytes, whatever their length
        CHECK(row_stage(stage, 1, wpr) == nullptr);
    CHECK(row_stage(stage, ROW_STAGE_BYTES / 8 / 313 + 1, 313) == nullptr);
}

// The sum from the columns' counts, or (false) from every pair.
static void column_counts() {
    DevBuf<uint32_t> hist;
    g_budget = 64 * 8 * 4;
    CHECK(colsum_room(hist, 100, 8) && g_used == g_budget);
    CHECK(!colsum_room(hist, 100, 16) && g_used == 0);
    g_budget = 64ull * COLSUM_STRIP * 4;
    CHECK(colsum_room(hist, COLSUM_MAX_ROWS, 1u << 20));         // longer rows take several strips
    CHECK(!colsum_room(hist, COLSUM_MAX_ROWS + 1, 8));           // more blocks than a grid has
}

// A thread's place for the flags is the library's own memory: it holds through
// a reset of the device, after which CUDA knows nothing of it and has handed its
// own pinned memory to others, and goes with the thread.
static void flags() {
    for (size_t budget : {size_t(1) << 20, size_t(0)}) {         // registered, and where nothing can be
        g_budget = budget;
        std::thread([&] {
            DeviceFlags on_device{0, 0, 42};
            CHECK(read_flags(&on_device, nullptr).sum == 42);
            CHECK(g_held.empty());                               // none of CUDA's memory is kept
            CHECK(g_registered.size() == (budget ? 1u : 0u) && g_error == cudaSuccess);
            g_registered.clear();                                // cudaDeviceReset
            on_device.sum = 43;
            CHECK(read_flags(&on_device, nullptr).sum == 43);
        }).join();
        g_budget = 1 << 20;
        std::thread([] {
            DeviceFlags on_device{0, 0, 44};
            CHECK(read_flags(&on_device, nullptr).sum == 44 && g_registered.size() == 1);
        }).join();
        CHECK(g_registered.empty());
    }
}

int main() {
    buffers_a_call_can_do_without();
    sweep_buffers();
    staged_rows();
    column_counts();
    flags();
    CHECK(g_held.empty());
    std::printf(g_fail ? "FAIL (%d)\n" : "ok\n", g_fail);
    return g_fail ? 1 : 0;
}
