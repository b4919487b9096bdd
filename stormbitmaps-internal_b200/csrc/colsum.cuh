// colsum.cuh -- the sum over all pairs of dense rows without a pair.
//
// sum_{i<j} |Xi & Xj| = sum_v C(n_v, 2), n_v = the rows holding column v, so a
// call that wants only the sum reads the rows once.  What it cannot do without is
// that read; what bounds it is the chain of each warp's few steps (eight loads,
// then their adders) and the unpacking of its planes, at a third of HBM's rate.
// A warp reads 32 consecutive words of a row (256 bytes); each thread counts
// its 64 columns over the warp's rows in bit-sliced planes: eight rows go
// through carry-save adders into ones / twos / fours and a carry of weight 8
// that ripples up, about 6 integer operations per word.  A block's eight
// warps take every eighth group of its rows and meet in shared memory, and a
// block adds its 2048 counts to the histogram once.  10007 rows x 100003 bits
// on B200, the whole call: 1.31 ms on the tensor cores (every pair), 0.091 ms
// so (both kernels 0.060 ms, 2.1 TB/s).
#pragma once
#include "common.cuh"

namespace sb200 {

constexpr uint32_t COLSUM_WARPS = 8;
constexpr uint32_t COLSUM_WORDS = 32;          // row words per block (a warp's lanes)
constexpr uint32_t COLSUM_PLANES = 9;          // planes of weight 8 .. 2048: a warp counts at most 4095 rows
constexpr uint64_t COLSUM_WARP_ROWS = 4088;
constexpr uint32_t COLSUM_STRIP = 1u << 16;    // row words per histogram (2^22 columns, 16 MiB)
constexpr uint64_t COLSUM_MAX_ROWS = 65535ull * COLSUM_WARPS * COLSUM_WARP_ROWS;   // a grid's blocks along the rows

// Whether the sum over n rows can come from the columns' counts: `hist` then
// holds a strip of them. Without room for it every pair is counted.
inline bool colsum_room(DevBuf<uint32_t>& hist, uint64_t n, uint32_t w_pad) {
    return n <= COLSUM_MAX_ROWS && hist.try_reserve(64ull * (w_pad < COLSUM_STRIP ? w_pad : COLSUM_STRIP));
}

#ifdef __CUDACC__
__device__ __forceinline__ void csa(uint64_t& sum, uint64_t& carry, uint64_t a, uint64_t b, uint64_t c) {
    sum = a ^ b ^ c;
    carry = (a & b) | (c & (a ^ b));
}

// Words [w0, w0 + words) of rows [rows_per_block x blockIdx.y, ..) into
// hist[64 x word + bit], words <= COLSUM_STRIP.
__global__ void __launch_bounds__(COLSUM_WARPS * 32)
column_counts_kernel(const uint64_t* __restrict__ X, uint64_t n, uint64_t pitch, uint32_t w0, uint32_t words,
                     uint64_t rows_per_block, uint32_t* __restrict__ hist) {
    __shared__ uint32_t cnt[64 * COLSUM_WORDS];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint32_t k = threadIdx.x; k < 64 * COLSUM_WORDS; k += blockDim.x) cnt[k] = 0;
    __syncthreads();
    const uint32_t w = blockIdx.x * COLSUM_WORDS + lane;
    const uint64_t r0 = blockIdx.y * rows_per_block;
    const uint64_t r1 = r0 + rows_per_block < n ? r0 + rows_per_block : n;
    if (w < words) {
        const uint64_t* src = X + w0 + w;
        uint64_t ones = 0, twos = 0, fours = 0, up[COLSUM_PLANES] = {};
        for (uint64_t r = r0 + 8 * warp; r < r1; r += 8 * COLSUM_WARPS) {
            uint64_t x[8];
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) x[k] = r + k < r1 ? __ldcs(src + (r + k) * pitch) : 0;
            uint64_t ta, tb, fa, fb, e;
            csa(ones, ta, ones, x[0], x[1]);
            csa(ones, tb, ones, x[2], x[3]);
            csa(twos, fa, twos, ta, tb);
            csa(ones, ta, ones, x[4], x[5]);
            csa(ones, tb, ones, x[6], x[7]);
            csa(twos, fb, twos, ta, tb);
            csa(fours, e, fours, fa, fb);
#pragma unroll
            for (uint32_t k = 0; k < COLSUM_PLANES; ++k) {
                const uint64_t t = up[k] & e;
                up[k] ^= e;
                e = t;
            }
        }
#pragma unroll 4
        for (uint32_t b = 0; b < 64; ++b) {
            uint32_t c = (uint32_t)(ones >> b) & 1u;
            c |= ((uint32_t)(twos >> b) & 1u) << 1;
            c |= ((uint32_t)(fours >> b) & 1u) << 2;
#pragma unroll
            for (uint32_t k = 0; k < COLSUM_PLANES; ++k) c |= ((uint32_t)(up[k] >> b) & 1u) << (3 + k);
            if (c) atomicAdd(&cnt[b * COLSUM_WORDS + lane], c);
        }
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < 64 * COLSUM_WORDS; k += blockDim.x) {
        const uint32_t ww = blockIdx.x * COLSUM_WORDS + k / 64, c = cnt[(k % 64) * COLSUM_WORDS + k / 64];
        if (ww < words && c) atomicAdd(hist + 64ull * ww + k % 64, c);
    }
}

// sum += sum_v C(hist[v], 2).
__global__ void __launch_bounds__(256)
pairs_of_counts_kernel(const uint32_t* __restrict__ hist, uint64_t columns, unsigned long long* __restrict__ sum) {
    unsigned long long s = 0;
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < columns; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t c = hist[v];
        s += c * (c - (c > 0)) / 2;
    }
    s = warp_sum_u64(s);
    if ((threadIdx.x & 31) == 0 && s) atomicAdd(sum, s);
}
#endif

}  // namespace sb200
