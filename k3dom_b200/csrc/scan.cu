// scan.cu -- exclusive scan of u32 values: tile sums, one block over them, apply. No block waits on
// another.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "internal.h"
#include "scan.cuh"

namespace k3dom {

long g_launches = 0;

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;  // 2048
constexpr int kGridCap = 148 * 8;

__global__ void scan_u32_tile_sums(const uint32_t* __restrict__ in, long n, uint32_t* __restrict__ tile_sums) {
    __shared__ uint32_t sm[kScanThreads / 32 + 1];
    const long nt = (n + kScanTile - 1) / kScanTile;
    for (long tile = blockIdx.x; tile < nt; tile += gridDim.x) {
        const long base = tile * kScanTile;
        uint32_t s = 0;
#pragma unroll
        for (int j = 0; j < kScanItems; ++j) {
            long i = base + (long)j * kScanThreads + threadIdx.x;
            if (i < n) s += in[i];
        }
        uint32_t tot;
        block_exclusive_scan<uint32_t, kScanThreads>(s, sm, &tot);
        if (threadIdx.x == 0) tile_sums[tile] = tot;
    }
}

// One block scans the tile sums in place (exclusive) and writes the grand total.
__global__ void scan_u32_tile_offsets(uint32_t* __restrict__ tile_sums, long n, uint32_t* __restrict__ total) {
    __shared__ uint32_t sm[kScanThreads / 32 + 1];
    const long nt = (n + kScanTile - 1) / kScanTile;
    uint32_t carry = 0;
    for (long b = 0; b < nt; b += kScanThreads) {
        long i = b + threadIdx.x;
        uint32_t v = (i < nt) ? tile_sums[i] : 0u;
        uint32_t tot;
        uint32_t ex = block_exclusive_scan<uint32_t, kScanThreads>(v, sm, &tot);
        if (i < nt) tile_sums[i] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0 && total) *total = carry;
}

__global__ void scan_u32_apply(const uint32_t* __restrict__ in, long n, const uint32_t* __restrict__ tile_offsets,
                               uint32_t* __restrict__ out) {
    __shared__ uint32_t sm[kScanThreads / 32 + 1];
    const long nt = (n + kScanTile - 1) / kScanTile;
    for (long tile = blockIdx.x; tile < nt; tile += gridDim.x) {
        const long base = tile * kScanTile + (long)threadIdx.x * kScanItems;
        uint32_t v[kScanItems];
        uint32_t s = 0;
#pragma unroll
        for (int j = 0; j < kScanItems; ++j) {
            long i = base + j;
            v[j] = (i < n) ? in[i] : 0u;
            s += v[j];
        }
        uint32_t tot;
        uint32_t ex = block_exclusive_scan<uint32_t, kScanThreads>(s, sm, &tot);
        uint32_t run = tile_offsets[tile] + ex;
#pragma unroll
        for (int j = 0; j < kScanItems; ++j) {
            long i = base + j;
            if (i < n) out[i] = run;
            run += v[j];
        }
    }
}

int scan_u32_tiles(long n) { return div_up(n, kScanTile); }

static int tile_grid(long tiles) { return (int)std::max(1L, std::min(tiles, (long)kGridCap)); }

// Exclusive scan of n u32 values (in may alias out). tmp needs scan_u32_tiles(n) words. total
// (optional, device) receives the sum.
cudaError_t scan_u32_exclusive(const uint32_t* in, uint32_t* out, long n, uint32_t* tmp, uint32_t* total,
                               cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const int nt = scan_u32_tiles(n);
    g_launches += 3;
    scan_u32_tile_sums<<<tile_grid(nt), kScanThreads, 0, st>>>(in, n, tmp);
    scan_u32_tile_offsets<<<1, kScanThreads, 0, st>>>(tmp, n, total);
    scan_u32_apply<<<tile_grid(nt), kScanThreads, 0, st>>>(in, n, tmp, out);
    return cudaGetLastError();
}

}  // namespace k3dom
