// drawsort.cu -- the resampling draws of a frame, generated and sorted.
//
// Draws are 24-bit keys of 1 - u: sorting the keys ascending orders the draws u * joint_max ascending
// for any joint_max >= 0, so the draws can be sorted before the weights exist
// (resamplingGenerateRandomNumbersKernel + thrust::sort, resampling.cu:38-53,
// src/common/dom.cu:277-285). The keys follow from (seed, frame, particle) and have no payload, and
// they are uniform, so they are sorted by their value instead of in digit passes over memory:
//   k_draw_count    generates the keys and counts them per bucket (the 12 high bits, per scene);
//   k_draw_scatter  generates them again and writes each into its bucket's range;
//   k_draw_buckets  orders each bucket, a warp each.
// Generating costs a quarter of a Philox block per key, so the keys move through memory three times
// (write, read, write) instead of eight in a histogram and three radix passes. None is bound by DRAM
// (5 % of its rate at most): counting and scattering wait for their atomics (a third and a fifth of the
// issue slots used), the buckets' warps issue in 70 % of the cycles with 14 of 32 lanes (the writing
// out of equal values and of ranks diverges). 4,194,304 draws alone on the
// GPU, cold cache: 208 us in digit passes, 95 in buckets (1,000,000: 91 and 56; 16,384: 54 and 30).
// Any distribution of keys sorts correctly (counters, not capacities).
#include <cuda_runtime.h>

#include "common.cuh"
#include "internal.h"
#include "scan.cuh"

namespace k3dom {

using namespace k3dom_draws;

constexpr int kDrawThreads = 1024;
constexpr int kDrawHi = 12, kDrawLo = 24 - kDrawHi;  // bucket bits, bits within a bucket
constexpr int kDrawBuckets = 1 << kDrawHi;
constexpr uint32_t kDrawRankMax = 64;                // keys a warp orders by ranks
constexpr int kDrawSortThreads = 256;

int draw_blocks(int P) { return div_up(P, kDrawPerBlock); }
long draw_row_words(int blocks) { return (long)blocks * kDrawBuckets; }
long draw_bucket_words(int S) { return (long)S * kDrawBuckets; }

// The block's scene and its draws [i0, i1) of the scene's P, four per Philox block.
struct DrawBlock {
    int sc, i0, i1;
};
__device__ __forceinline__ DrawBlock draw_block(const Batch& bt) {
    DrawBlock d;
    d.sc = scene_of(bt.off->draw, bt.S, blockIdx.x);
    d.i0 = (blockIdx.x - bt.off->draw[d.sc]) * kDrawPerBlock;
    d.i1 = min(d.i0 + kDrawPerBlock, bt.off->part[d.sc + 1] - bt.off->part[d.sc]);
    return d;
}
template <typename F>
__device__ __forceinline__ void for_each_draw(const Batch& bt, const DrawBlock& d, F f) {
    const FrameParams& fp = bt.fp[d.sc];
    const uint64_t seed = fp.seed;
    const uint32_t frame = fp.frame;
    for (int i = d.i0 + 4 * (int)threadIdx.x; i < d.i1; i += 4 * kDrawThreads) {
        const U4 w = block(seed, frame, kResample, (uint64_t)(i >> 2), 0);  // resample_word of i .. i + 3
        f(one_minus_u01_key(w.x));
        if (i + 1 < d.i1) f(one_minus_u01_key(w.y));
        if (i + 2 < d.i1) f(one_minus_u01_key(w.z));
        if (i + 3 < d.i1) f(one_minus_u01_key(w.w));
    }
}

// rows[block][bucket]: the block's first slot in the bucket, relative to the bucket's start (rows of
// buckets that the block does not reach keep stale values that are never used). totals: zero between
// frames (k_draw_buckets clears them).
__global__ void __launch_bounds__(kDrawThreads) k_draw_count(Batch bt, uint32_t* __restrict__ totals,
                                                             uint32_t* __restrict__ rows) {
    __shared__ uint32_t cnt[kDrawBuckets];
    for (int b = threadIdx.x; b < kDrawBuckets; b += kDrawThreads) cnt[b] = 0u;
    __syncthreads();
    const DrawBlock d = draw_block(bt);
    for_each_draw(bt, d, [&](uint32_t key) { atomicAdd(&cnt[key >> kDrawLo], 1u); });
    __syncthreads();
    uint32_t* tot = totals + (long)d.sc * kDrawBuckets;
    uint32_t* row = rows + (long)blockIdx.x * kDrawBuckets;
    for (int b = threadIdx.x; b < kDrawBuckets; b += kDrawThreads)
        if (cnt[b]) row[b] = atomicAdd(&tot[b], cnt[b]);
}

// starts[scene][bucket]: first slot of the bucket in the scene's range (written by its first block).
__global__ void __launch_bounds__(kDrawThreads)
    k_draw_scatter(Batch bt, const uint32_t* __restrict__ totals, const uint32_t* __restrict__ rows,
                   uint32_t* __restrict__ starts, uint32_t* __restrict__ out) {
    __shared__ uint32_t pos[kDrawBuckets];
    __shared__ uint32_t sm[kDrawThreads / 32 + 1];
    const DrawBlock d = draw_block(bt);
    constexpr int kPer = kDrawBuckets / kDrawThreads;
    static_assert(kPer == 4, "one 16-byte load of totals per thread");
    const uint4 t = reinterpret_cast<const uint4*>(totals + (long)d.sc * kDrawBuckets)[threadIdx.x];
    const uint32_t n[kPer] = {t.x, t.y, t.z, t.w};
    uint32_t total;
    uint32_t at = block_exclusive_scan<uint32_t, kDrawThreads>(t.x + t.y + t.z + t.w, sm, &total);
    const uint32_t* row = rows + (long)blockIdx.x * kDrawBuckets;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int b = threadIdx.x * kPer + k;
        if (d.i0 == 0) starts[(long)d.sc * kDrawBuckets + b] = at;
        pos[b] = at + row[b];
        at += n[k];
    }
    __syncthreads();
    uint32_t* dst = out + bt.off->part[d.sc];
    const uint32_t P = (uint32_t)(bt.off->part[d.sc + 1] - bt.off->part[d.sc]);
    for_each_draw(bt, d, [&](uint32_t key) {
        const uint32_t p = atomicAdd(&pos[key >> kDrawLo], 1u);
        if (p < P) dst[p] = key;  // always, with rows and totals of the same frame
    });
}

// One bucket per warp. Up to kDrawRankMax keys: each lane ranks its own among all of them. More: the
// bucket's 4,096 possible values are counted in bytes of shared memory and written out in order, 128
// values a step, so that the warp's writes are contiguous; a byte that overflowed shows as a wrong
// sum (never with uniform keys: 255 equal ones), and the values are counted again in 32-bit words,
// 1,024 at a time.
__global__ void __launch_bounds__(kDrawSortThreads)
    k_draw_buckets(Batch bt, uint32_t* __restrict__ totals, const uint32_t* __restrict__ starts,
                   const uint32_t* __restrict__ keys, uint32_t* __restrict__ sorted) {
    constexpr int kW = kDrawSortThreads / 32;
    constexpr int kWords = (1 << kDrawLo) / 4;  // byte counters of a bucket
    __shared__ uint32_t s_cnt[kW][kWords];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const long g = (long)blockIdx.x * kW + wid;
    const int sc = (int)(g >> kDrawHi);
    const uint32_t n = totals[g];
    if (n == 0u) return;
    const long at = (long)bt.off->part[sc] + starts[g];
    const uint32_t* a = keys + at;
    uint32_t* out = sorted + at;
    uint32_t* cnt = s_cnt[wid];
    __syncwarp();
    if (lane == 0) totals[g] = 0u;
    if (n <= kDrawRankMax) {
        uint32_t key[2], rank[2] = {0u, 0u};
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const uint32_t i = k * 32 + lane;
            key[k] = i < n ? a[i] : 0xFFFFFFFFu;
            cnt[i] = key[k];
        }
        __syncwarp();
        for (uint32_t j = 0; j < n; ++j) {
            const uint32_t o = cnt[j];
#pragma unroll
            for (int k = 0; k < 2; ++k) rank[k] += o < key[k] || (o == key[k] && j < (uint32_t)(k * 32 + lane));
        }
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if ((uint32_t)(k * 32 + lane) < n) out[rank[k]] = key[k];
        return;
    }
    const uint32_t hi = (uint32_t)(g & (kDrawBuckets - 1)) << kDrawLo;
    for (int w = lane; w < kWords; w += 32) cnt[w] = 0u;
    __syncwarp();
    for (uint32_t i = lane; i < n; i += 32) {
        const uint32_t v = a[i] & ((1u << kDrawLo) - 1u);
        atomicAdd(&cnt[v >> 2], 1u << (8 * (v & 3u)));
    }
    __syncwarp();
    uint32_t sum = 0;
    for (int w = lane; w < kWords; w += 32) sum = __dp4a(cnt[w], 0x01010101u, sum);
    uint32_t p = 0;
    if (__reduce_add_sync(0xffffffffu, sum) == n) {
        for (int w0 = 0; w0 < kWords; w0 += 32) {
            const uint32_t c = cnt[w0 + lane], m = __dp4a(c, 0x01010101u, 0u);
            const uint32_t inc = warp_inclusive_scan<uint32_t>(m);
            uint32_t q = p + inc - m;
            const uint32_t v = hi | (uint32_t)(w0 + lane) << 2;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                for (uint32_t r = (c >> (8 * k)) & 0xFFu; r > 0u; --r) out[q++] = v + k;
            p += __shfl_sync(0xffffffffu, inc, 31);
        }
        return;
    }
    for (uint32_t part = 0; part < 4u; ++part) {
        __syncwarp();
        for (int w = lane; w < kWords; w += 32) cnt[w] = 0u;
        __syncwarp();
        for (uint32_t i = lane; i < n; i += 32) {
            const uint32_t v = a[i] & ((1u << kDrawLo) - 1u);
            if (v / kWords == part) atomicAdd(&cnt[v % kWords], 1u);
        }
        __syncwarp();
        for (int w0 = 0; w0 < kWords; w0 += 32) {
            const uint32_t m = cnt[w0 + lane];
            const uint32_t inc = warp_inclusive_scan<uint32_t>(m);
            uint32_t q = p + inc - m;
            for (uint32_t r = m; r > 0u; --r) out[q++] = hi | (part * kWords + (uint32_t)(w0 + lane));
            p += __shfl_sync(0xffffffffu, inc, 31);
        }
    }
}

void launch_sorted_draws(const Batch& bt, int blocks, const DrawScratch& d, uint32_t* sorted, cudaStream_t st) {
    if (bt.P <= 0) return;
    g_launches += 3;
    k_draw_count<<<blocks, kDrawThreads, 0, st>>>(bt, d.totals, d.rows);
    k_draw_scatter<<<blocks, kDrawThreads, 0, st>>>(bt, d.totals, d.rows, d.starts, d.keys);
    k_draw_buckets<<<bt.S * (kDrawBuckets / (kDrawSortThreads / 32)), kDrawSortThreads, 0, st>>>(
        bt, d.totals, d.starts, d.keys, sorted);
}

}  // namespace k3dom
