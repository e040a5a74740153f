// evidence.cu -- measurement evidence and the per-cell mass update, for every scene of a batch
// in one launch per kernel.
//
// K3DOM: Bayesian kernel inference (BGKI, src/k3dom/kernel/mass_update.cu:32-77) followed by
// predict_mass / update_mass / separate_newborn_part (:79-150), with the per-cell parts of
// updatePersistentParticlesKernel2 (update_persistent_particles.cu:28-44) and
// statisticalMomentsKernel2 (statistical_moments.cu:36-63) fused into the same pass.
// DS-PHD/MIB: calcMeasurementGridKernel (src/dsphdmib/kernel/measurement_grid.cu:64-162)
// followed by gridCellPredictionUpdateKernel (src/dsphdmib/kernel/mass_update.cu:46-87).
//
// The reference evaluates every (cell, point) pair: C x N (2.5e11 at 2.1M cells / 120k
// points). Both evidence models have compact support -- the sparse kernel is zero beyond
// ls, the DS window is 0.866 res wide -- so each ray is binned to the tiles of cells its
// support can reach (segment sensor->point with radius ls for K3DOM, the half-line through
// the point with the window radius for DS). Tiles of all scenes share one global numbering
// (scene tile offset + local tile), so one pass builds every scene's lists. K3DOM places each
// ray into its tiles' ranges through per-block tallies of each tile (its exact sums make the order
// within a tile immaterial); DS keeps a tile's rays in input order, as its first-100 rule needs (bit
// masks per block of rays, k_ds_mark); with too many tiles for either, a stable sort by tile. One CTA
// takes one (tile, chunk of rays) work item from a device work counter and stages the chunk's rays in
// shared memory; its warps pull the tile's 4x4x2-cell sub-blocks from a block-local counter and cull
// 32 rays at a time with one ballot, collect the surviving rays into batches of 32, resolve them in
// FP64 and evaluate two rays at a time for four cells per lane. DS walks each ray's cells (see
// k_ds_rays).
//
// K3DOM evidence is summed in fixed point: each kernel value is rounded once to an integer
// number of units of 2^-k sigma (the table carries the scale), summed exactly in 64-bit
// integers (per lane, then atomics across sub-blocks and chunks), so a cell's evidence is the
// same for any tiling, chunking, ray order or scheduling. The
// last CTA to finish a tile's chunks runs the cell update for the whole tile. No block ever
// waits on another.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <cmath>
#include <cstddef>

#include "common.cuh"
#include "internal.h"
#include "scan.cuh"

namespace k3dom {

constexpr int kChunk = 1024;      // largest number of rays per work item
constexpr int kKernelTab = 512;  // intervals of the sparse-kernel table over u = d^2 / ls^2
constexpr int kKernelTabEntries = kKernelTab + 1;  // + a zero entry at u = 1
static_assert(kKernelTabEntries == kKernelTableSize, "kernel table size");
constexpr int kEvThreads = 256;
constexpr int kEvWarps = kEvThreads / 32;
constexpr int kEvCtas = 4;  // K3DOM evidence CTAs per SM: 64 registers a thread
constexpr uint32_t kDsMaxNeighbors = 100;  // measurement_grid.cu:87
constexpr int kFxShift = 40;  // fixed-point units of the K3DOM and calibration sums: 2^-40 of the scaled kernel

// ================================================================ binning
struct BinGeom {
    float ax, ay, az;  // sensor in cell-index space (cell centre ix sits at u = ix)
    float R;           // support radius in cells
    float R_far;       // DS: the radius for rays of ds_extreme
    int G, Gz, tx, ty, tz, ntx, nty, ntz;
};

// Whether the segment a + t d, t in [t0, t1], meets the box [l, h]; inv[k] = 1 / d[k] (unused
// where d[k] = 0).
__device__ __forceinline__ bool seg_box(const float a[3], const float d[3], const float inv[3], const float l[3],
                                        const float h[3], float t0, float t1) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (d[k] == 0.0f) {
            if (a[k] < l[k] || a[k] > h[k]) return false;
        } else {
            const float e0 = (l[k] - a[k]) * inv[k], e1 = (h[k] - a[k]) * inv[k];
            t0 = fmaxf(t0, fminf(e0, e1));
            t1 = fminf(t1, fmaxf(e0, e1));
        }
    }
    return t0 <= t1;
}

// v[k] for k in {0, 1, 2} by selects (a run-time index into a local array would go through
// local memory).
template <typename T>
__device__ __forceinline__ T sel3(T v0, T v1, T v2, int k) { return k == 0 ? v0 : (k == 1 ? v1 : v2); }

// Visit every tile whose cell-centre box, grown by R, meets the segment a -> b; only the slabs
// (layers of tiles across the ray's dominant axis) first, first + step, ... of them, so that
// `step` threads can share one ray. The reciprocals 1 / d are formed once per ray.
template <typename F>
__device__ __forceinline__ void for_each_tile(const BinGeom& g, float bx, float by, float bz, F f, int first = 0,
                                              int step = 1) {
    const float a[3] = {g.ax, g.ay, g.az};
    const float d[3] = {bx - g.ax, by - g.ay, bz - g.az};
    float inv[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) inv[k] = d[k] != 0.0f ? 1.0f / d[k] : 0.0f;
    const float glo[3] = {-g.R, -g.R, -g.R};
    const float ghi[3] = {(float)(g.G - 1) + g.R, (float)(g.G - 1) + g.R, (float)(g.Gz - 1) + g.R};
    float t0 = 0.0f, t1 = 1.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (d[k] == 0.0f) {
            if (a[k] < glo[k] || a[k] > ghi[k]) return;
        } else {
            const float e0 = (glo[k] - a[k]) * inv[k], e1 = (ghi[k] - a[k]) * inv[k];
            t0 = fmaxf(t0, fminf(e0, e1));
            t1 = fminf(t1, fmaxf(e0, e1));
        }
    }
    if (t0 > t1) return;
    int A = 0;
    float dmax = fabsf(d[0]);
    if (fabsf(d[1]) > dmax) {
        A = 1;
        dmax = fabsf(d[1]);
    }
    if (fabsf(d[2]) > dmax) A = 2;
    const int Bx = (A + 1) % 3, Cx = (A + 2) % 3;
    // the dominant axis A and the two others, B and C
    const float aA = sel3(a[0], a[1], a[2], A), dA = sel3(d[0], d[1], d[2], A), invA = sel3(inv[0], inv[1], inv[2], A);
    const float aB = sel3(a[0], a[1], a[2], Bx), dB = sel3(d[0], d[1], d[2], Bx);
    const float aC = sel3(a[0], a[1], a[2], Cx), dC = sel3(d[0], d[1], d[2], Cx);
    const int tsA = sel3(g.tx, g.ty, g.tz, A), tsB = sel3(g.tx, g.ty, g.tz, Bx), tsC = sel3(g.tx, g.ty, g.tz, Cx);
    const int ntA = sel3(g.ntx, g.nty, g.ntz, A), ntB = sel3(g.ntx, g.nty, g.ntz, Bx);
    const int ntC = sel3(g.ntx, g.nty, g.ntz, Cx);
    const float pa0 = aA + dA * t0, pa1 = aA + dA * t1;
    int ta0 = (int)floorf((fminf(pa0, pa1) - g.R) / (float)tsA);
    int ta1 = (int)floorf((fmaxf(pa0, pa1) + g.R) / (float)tsA);
    ta0 = max(ta0, 0);
    ta1 = min(ta1, ntA - 1);
    for (int ta = ta0 + first; ta <= ta1; ta += step) {
        const float slo = (float)(ta * tsA) - g.R, shi = (float)(ta * tsA + tsA - 1) + g.R;
        float s0 = t0, s1 = t1;
        if (dA != 0.0f) {
            const float e0 = (slo - aA) * invA, e1 = (shi - aA) * invA;
            s0 = fmaxf(s0, fminf(e0, e1));
            s1 = fminf(s1, fmaxf(e0, e1));
        } else if (aA < slo || aA > shi) {
            continue;
        }
        if (s0 > s1) continue;
        const float b0 = aB + dB * s0, b1 = aB + dB * s1;
        const float c0 = aC + dC * s0, c1 = aC + dC * s1;
        int tb0 = max((int)floorf((fminf(b0, b1) - g.R) / (float)tsB), 0);
        int tb1 = min((int)floorf((fmaxf(b0, b1) + g.R) / (float)tsB), ntB - 1);
        int tc0 = max((int)floorf((fminf(c0, c1) - g.R) / (float)tsC), 0);
        int tc1 = min((int)floorf((fmaxf(c0, c1) + g.R) / (float)tsC), ntC - 1);
        for (int tb = tb0; tb <= tb1; ++tb) {
            for (int tc = tc0; tc <= tc1; ++tc) {
                // the tile's (x, y, z) index: ta along A, tb along B, tc along C
                const int tx = A == 0 ? ta : (Bx == 0 ? tb : tc);
                const int ty = A == 1 ? ta : (Bx == 1 ? tb : tc);
                const int tz = A == 2 ? ta : (Bx == 2 ? tb : tc);
                const float l[3] = {(float)(tx * g.tx) - g.R, (float)(ty * g.ty) - g.R, (float)(tz * g.tz) - g.R};
                const float h[3] = {(float)(tx * g.tx + g.tx - 1) + g.R, (float)(ty * g.ty + g.ty - 1) + g.R,
                                    (float)(tz * g.tz + g.tz - 1) + g.R};
                if (seg_box(a, d, inv, l, h, t0, t1)) f(tx + g.ntx * (ty + g.nty * tz));
            }
        }
    }
}

// The sensor's place in cell-index space comes from the frame scalars in device memory, so a
// captured graph stays valid while the sensor moves.
__device__ __forceinline__ void place_sensor(BinGeom& g, const DevParams& p, const FrameParams& f) {
    const float hg = (float)p.G / 2.0f, hz = (float)p.Gz / 2.0f;
    // a point q (metres, sensor frame) sits at u = (q + s)/res + G/2 - 0.5
    g.ax = f.sensor_x / p.res + hg - 0.5f;
    g.ay = f.sensor_y / p.res + hg - 0.5f;
    g.az = f.sensor_z / p.res + hz - 0.5f;
}

struct RayPrep {
    bool ok;
    float bx, by, bz;  // far end of the binned segment (cell-index space)
};

// DS rays whose |m|^2 leaves [2^-80, 2^80] (points beyond 1e12 m, or within 1e-12 m of the sensor). The
// reference's FP32 test overflows or underflows for them: with |m|^2 infinite it accepts the cells
// around the sensor whatever the ray's direction, and with (c.m)^2 infinite cells beside the line. So
// a window around the half-line does not hold their neighbours; they take every cell of the
// sub-blocks near it (ds_reaches_sub_block), in lists of the widest radius.
__device__ __forceinline__ bool ds_extreme(float sq) { return !(sq >= 8.2718061e-25f && sq <= 1.2089258e24f); }

// Per-ray constants. K3DOM: (m, d_m) and (m/d_m, margin), d_m and margin as the reference
// forms them (mass_update.cu:29-31,55). DS: (m, |m|^2) as measurement_grid.cu:90.
// consts = false: only ok and the segment's far end (K3DOM), for a second thread of the ray.
// A ray of ds_extreme widens g.R.
__device__ __forceinline__ RayPrep prep_ray(const DevParams& p, BinGeom& g, float mx, float my, float mz,
                                           bool ds, float4* ra, double4* rc, bool consts = true) {
    RayPrep r;
    r.ok = isfinite(mx) && isfinite(my) && isfinite(mz);
    r.bx = r.by = r.bz = 0.0f;
    *ra = make_float4(0.f, 0.f, 0.f, 0.f);
    *rc = make_double4(0.0, 0.0, 0.0, 0.0);
    if (!r.ok) return r;
    const float sq = __fadd_rn(__fadd_rn(__fmul_rn(mx, mx), __fmul_rn(my, my)), __fmul_rn(mz, mz));
    if (!ds && !consts) {
        r.bx = g.ax + mx / p.res;
        r.by = g.ay + my / p.res;
        r.bz = g.az + mz / p.res;
    } else if (!ds) {
        // d_m and the margin point (mass_update.cu:29-31,55) in FP64; a zero-length ray gets
        // 1/d_m = 0, which turns its free evidence off as the reference's NaN comparisons do
        const double dmd = sqrt((double)mx * mx + (double)my * my + (double)mz * mz);
        const double margd = fmax(0.9 * dmd, dmd - 2.0 * (double)p.res);
        const double inv = dmd > 0.0 ? 1.0 / dmd : 0.0;
        const float dm = (float)dmd;
        *ra = make_float4(mx, my, mz, dm);
        *rc = make_double4(dmd, margd, inv, 0.0);
        r.bx = g.ax + mx / p.res;
        r.by = g.ay + my / p.res;
        r.bz = g.az + mz / p.res;
    } else {
        *ra = make_float4(mx, my, mz, sq);
        const float len = sqrtf(sq);
        if (!(len > 0.0f)) {
            r.ok = false;  // |m| = 0: inner product 0, never a neighbour (measurement_grid.cu:92)
            return r;
        }
        if (ds_extreme(sq)) g.R = g.R_far;
        // length of the binned half-line in cells: past the grid's far corner, also from a sensor
        // outside the grid
        const float diag = sqrtf((float)(2 * g.G * g.G + g.Gz * g.Gz));
        const float cx = g.ax - 0.5f * (float)(g.G - 1), cy = g.ay - 0.5f * (float)(g.G - 1);
        const float cz = g.az - 0.5f * (float)(g.Gz - 1);
        const float L = fmaxf(diag, 0.5f * diag + sqrtf(cx * cx + cy * cy + cz * cz)) + 2.0f * g.R + 4.0f;
        const float sc = L / (len / p.res);
        r.bx = g.ax + mx / p.res * sc;
        r.by = g.ay + my / p.res * sc;
        r.bz = g.az + mz / p.res * sc;
    }
    return r;
}


// The distance from a ray's half-line within which a cell can pass the DS neighbour test, in cells, for
// cells at most `dist` metres from the sensor. The test compares |c|^2 - (c.m)^2 / |m|^2 with the
// window in FP32: the two terms carry at most 3 and 11 roundings of |c|^2, 8.4e-7 of it together.
__device__ __forceinline__ float ds_window(float wr2, float dist2, float res) {
    return sqrtf(wr2 + 1e-6f * dist2) / res + 1e-3f;
}
// (A slack for cells up to twice the grid's extent away made the window 2.05 cells at 256 cells of
// 0.1 m instead of 0.9: 120,000 rays, lists 158 -> 139 us, k_ds_rays 0.62 -> 0.18 ms.)

__device__ __forceinline__ BinGeom scene_geom(const SceneDev& sd, const FrameParams& f) {
    BinGeom g;
    g.R = g.R_far = sd.bin_R;
    if (sd.p.variant != 0) {  // DS: from the farthest cell
        const float ext = sqrtf(f.sensor_x * f.sensor_x + f.sensor_y * f.sensor_y + f.sensor_z * f.sensor_z) +
                          0.5f * sd.p.res * sqrtf((float)(2 * sd.p.G * sd.p.G + sd.p.Gz * sd.p.Gz));
        g.R = fminf(g.R, ds_window(sd.wr2, ext * ext, sd.p.res) + 0.02f);  // 0.02: the tile walk's arithmetic
    }
    g.G = sd.p.G;
    g.Gz = sd.p.Gz;
    g.tx = sd.ts.tx; g.ty = sd.ts.ty; g.tz = sd.ts.tz;
    g.ntx = sd.ts.ntx; g.nty = sd.ts.nty; g.ntz = sd.ts.ntz;
    place_sensor(g, sd.p, f);
    return g;
}

// Pass 1 over every point slot of every scene: per-ray constants and the number of tiles the
// ray's support reaches (0 for slots past the scene's point count). TALLY (placed lists): each
// reached tile's ray count is also added to tile_tally, through a block histogram of the T tiles
// in shared memory (the tiles around a sensor are reached by nearly every ray: one global atomic
// per block and tile instead of one per ray); the value that atomic returns is the block's first
// slot in the tile's range (relative to its start), kept in block_base for k_ray_place. TALLY
// also gives each ray two threads (the ray's even and odd slabs of tiles, counts per thread):
// the walk is latency bound, and 120,000 rays make only 25 warps per SM.
template <bool TALLY>
__global__ void k_ray_count(Batch bt, const float* __restrict__ xs, const float* __restrict__ ys,
                            const float* __restrict__ zs, int ds, float4* __restrict__ ra,
                            double4* __restrict__ rc, uint32_t* __restrict__ counts,
                            uint32_t* __restrict__ tile_tally, uint32_t* __restrict__ block_base,
                            DevStatus* status) {
    extern __shared__ uint32_t s_tally[];  // [T] (TALLY)
    if (blockIdx.x == 0 && threadIdx.x == 0) status->overflow = 0u;  // per-frame flag (set by k_ray_emit / k_tile_ranges)
    if (TALLY) {
        for (int t = threadIdx.x; t < bt.T; t += blockDim.x) s_tally[t] = 0u;
        __syncthreads();
    }
    constexpr int kPer = TALLY ? kRayThreads : 1;  // threads per ray
    const long nt = (long)bt.N * kPer;
    for (long tid = (long)blockIdx.x * blockDim.x + threadIdx.x; tid < nt; tid += (long)gridDim.x * blockDim.x) {
        const int i = (int)(tid / kPer), half = (int)(tid % kPer);
        const int sc = scene_of(bt.off->point, bt.S, i);
        const FrameParams f = bt.fp[sc];
        if (i - bt.off->point[sc] >= f.n_points) {
            counts[tid] = 0;
            continue;
        }
        const SceneDev& sd = bt.sc[sc];
        BinGeom g = scene_geom(sd, f);
        float mx = xs[i], my = ys[i], mz = zs[i];
        if (f.has_transform) apply_transform(f, &mx, &my, &mz);
        float4 a;
        double4 cc;
        const RayPrep r = prep_ray(sd.p, g, mx, my, mz, ds != 0, &a, &cc, half == 0);
        if (half == 0) {
            ra[i] = a;
            if (!ds) rc[i] = cc;
        }
        uint32_t c = 0;
        if (r.ok) {
            const uint32_t toff = (uint32_t)bt.off->tile[sc];
            for_each_tile(
                g, r.bx, r.by, r.bz,
                [&](int t) {
                    ++c;
                    if (TALLY) atomicAdd(&s_tally[toff + (uint32_t)t], 1u);
                },
                half, kPer);
        } else if (half == 0 && !(isfinite(mx) && isfinite(my) && isfinite(mz))) {
            atomicAdd(&status->nonfinite_points, 1ull);
        }
        counts[tid] = c;
    }
    if (TALLY) {
        __syncthreads();
        uint32_t* row = block_base + (size_t)blockIdx.x * bt.T;
        for (int t = threadIdx.x; t < bt.T; t += blockDim.x) {
            const uint32_t v = s_tally[t];
            if (v) row[t] = atomicAdd(&tile_tally[t], v);
        }
    }
}

// Pass 2: (global tile, ray) entries at the ray's scanned offset.
__global__ void k_ray_emit(Batch bt, const float* __restrict__ xs, const float* __restrict__ ys,
                           const float* __restrict__ zs, int ds, const uint32_t* __restrict__ offsets,
                           uint32_t* __restrict__ total, long capacity, uint32_t* __restrict__ ekeys,
                           uint32_t* __restrict__ evals, DevStatus* status) {
    const bool over = (long)total[0] > capacity;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        total[2] = over ? 0u : total[0];  // live entry count for the sort
        if (over) atomicOr(&status->overflow, 1u);
    }
    if (over) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < bt.N; i += gridDim.x * blockDim.x) {
        const int sc = scene_of(bt.off->point, bt.S, i);
        const FrameParams f = bt.fp[sc];
        if (i - bt.off->point[sc] >= f.n_points) continue;
        const SceneDev& sd = bt.sc[sc];
        BinGeom g = scene_geom(sd, f);
        float mx = xs[i], my = ys[i], mz = zs[i];
        if (f.has_transform) apply_transform(f, &mx, &my, &mz);
        float4 a;
        double4 c;
        const RayPrep r = prep_ray(sd.p, g, mx, my, mz, ds != 0, &a, &c);
        if (!r.ok) continue;
        // never write more entries than were counted: the count pass sized this ray's range
        const uint32_t o0 = offsets[i];
        const uint32_t cnt = (i + 1 < bt.N) ? offsets[i + 1] - o0 : total[0] - o0;
        const uint32_t toff = (uint32_t)bt.off->tile[sc];
        uint32_t o = o0;
        for_each_tile(g, r.bx, r.by, r.bz, [&](int t) {
            if (o - o0 < cnt) {
                ekeys[o] = toff + (uint32_t)t;
                evals[o] = (uint32_t)i;
                ++o;
            }
        });
        for (; o - o0 < cnt; ++o) {  // pad with a key past the last tile (sorted last, ignored)
            ekeys[o] = (uint32_t)bt.T;
            evals[o] = (uint32_t)i;
        }
    }
}

// tile_start[t] = first sorted entry of tile t, for t in [0, T].
__global__ void k_tile_start(const uint32_t* __restrict__ skeys, const uint32_t* __restrict__ total, int T,
                             uint32_t* __restrict__ tile_start) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t > T) return;
    const long n = (long)total[2];
    long lo = 0, hi = n;
    while (lo < hi) {
        const long mid = (lo + hi) >> 1;
        if (skeys[mid] < (uint32_t)t) lo = mid + 1; else hi = mid;
    }
    tile_start[t] = (uint32_t)lo;
}

// Rays per work item of a frame with `entries` (tile, ray) entries: at most chunk, and so few that
// every CTA slot of the evidence launch gets about kItemsPerSlot items (a multiple of 32 rays, kItemMin
// at least: two full batches for a sub-block that all of them reach). slots = 0: always chunk. The
// sums are exact, so the size changes no bit. With 1,024-ray items a small scan leaves most of the
// GPU idle while a few CTAs walk long lists: 2,000 rays in 32x32x8 voxels, evidence 98 -> 27 us;
// 30,000 rays in 64x64x16, 139 -> 106 us; 60,000 in 100x100x12, 158 -> 130 us. From about 1.2
// million entries on nothing changes. Four or eight items per slot cost more staging than they
// balance (30,000 rays: 111 and 128 us); 32 or 128 rays at least measured the same.
constexpr int kItemsPerSlot = 2;
constexpr int kItemMin = 64;
//
// DS (spare > 0): chunk rays, or as many as keep the items beyond one per tile within `spare`, which
// the per-(item, cell) summaries are sized for (ds_spare_items). The first-100 rule holds for any size.
__device__ __forceinline__ int item_rays(uint32_t entries, int chunk, int slots, int spare) {
    if (spare > 0) {
        const int n = (int)(entries / (uint32_t)spare) + 1;
        return n <= chunk ? chunk : (n + 31) & ~31;
    }
    if (slots <= 0) return chunk;
    const uint32_t n = entries / (uint32_t)(slots * kItemsPerSlot);
    return min(chunk, max(kItemMin, (int)((n + 31u) & ~31u)));
}

__global__ void k_tile_items(const uint32_t* __restrict__ tile_start, const uint32_t* __restrict__ total, int T,
                             int max_chunk, int slots, int spare, uint32_t* __restrict__ items) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    const int chunk = item_rays(total[2], max_chunk, slots, spare);
    const uint32_t len = tile_start[t + 1] - tile_start[t];
    items[t] = len == 0 ? 1u : (len + chunk - 1) / chunk;
}

__global__ void k_finish_lists(const uint32_t* __restrict__ item_off, int T, DevStatus* status,
                               const uint32_t* __restrict__ total) {
    status->work_items = item_off[T];
    status->ray_entries = total[0];
    // k_ray_count has finished counting this frame's non-finite points: keep the frame's count
    status->nonfinite_frame = (unsigned int)status->nonfinite_points;
    status->nonfinite_points = 0;
    status->work_counter = 0;
    status->work_counter2 = 0;
    status->kernel_evals = 0;
}

// K3DOM lists without a sort. The evidence sums are exact integers, so the order of a tile's
// rays changes no result; k_ray_count<true> has tallied each tile's rays, this pass turns the
// tallies into ranges (tile_start) and clears them for the
// next frame, counts the work items per tile and their offsets, and ends the frame's list
// counters as k_finish_lists does. One block: a batch holds at most a few tens of thousands of
// tiles. On overflow (more entries than the list holds) every range is empty.
constexpr int kRangeThreads = 1024;
__global__ void __launch_bounds__(kRangeThreads)
    k_tile_ranges(uint32_t* __restrict__ tile_tally, int T, int max_chunk, int slots, int spare, long capacity,
                  uint32_t* __restrict__ tile_start,
                  uint32_t* __restrict__ item_off, uint32_t* __restrict__ total, DevStatus* status) {
    __shared__ unsigned long long sm[kRangeThreads / 32 + 1];
    const int per = (T + kRangeThreads - 1) / kRangeThreads;
    const int t0 = min(T, (int)threadIdx.x * per), t1 = min(T, t0 + per);
    unsigned long long n = 0;
    for (int t = t0; t < t1; ++t) n += tile_tally[t];
    unsigned long long entries;
    const unsigned long long base = block_exclusive_scan<unsigned long long, kRangeThreads>(n, sm, &entries);
    const bool over = entries > (unsigned long long)capacity;
    const int chunk = item_rays(over ? 0u : (uint32_t)entries, max_chunk, slots, spare);
    unsigned long long o = over ? 0ull : base;
    unsigned long long ni = 0;
    for (int t = t0; t < t1; ++t) {
        const uint32_t c = over ? 0u : tile_tally[t];
        tile_start[t] = (uint32_t)o;
        o += c;
        ni += c == 0 ? 1u : (c + chunk - 1) / chunk;
    }
    unsigned long long items;
    const unsigned long long ibase = block_exclusive_scan<unsigned long long, kRangeThreads>(ni, sm, &items);
    unsigned long long io = ibase;
    for (int t = t0; t < t1; ++t) {
        const uint32_t c = over ? 0u : tile_tally[t];
        item_off[t] = (uint32_t)io;
        io += c == 0 ? 1u : (c + chunk - 1) / chunk;
        tile_tally[t] = 0u;
    }
    if (threadIdx.x == 0) {
        const uint32_t e32 = (uint32_t)min(entries, 0xFFFFFFFFull);
        tile_start[T] = over ? 0u : e32;
        item_off[T] = (uint32_t)items;
        total[0] = e32;
        total[2] = over ? 0u : e32;
        if (over) atomicOr(&status->overflow, 1u);
        status->work_items = (uint32_t)items;
        status->ray_entries = e32;
        // k_ray_count has finished counting this frame's non-finite points: keep the frame's count
        status->nonfinite_frame = (unsigned int)status->nonfinite_points;
        status->nonfinite_points = 0;
        status->work_counter = 0;
        status->work_counter2 = 0;
        status->kernel_evals = 0;
    }
}

// Pass 2 of the placed lists, on the grid of the tally (the same rays in each block): each ray
// takes one slot in the range of each tile it reaches, at most as many tiles as it tallied (the
// same enumeration as the tally's, on the same values), from the block's own share of the range,
// and never a slot past the list. The segment's far end is formed from the staged ray constants
// as prep_ray forms it.
template <typename F>
__device__ __forceinline__ void for_each_placed_tile(const Batch& bt, const float4* __restrict__ ra,
                                                     const uint32_t* __restrict__ counts, F f) {
    const long nt = (long)bt.N * kRayThreads;
    for (long tid = (long)blockIdx.x * blockDim.x + threadIdx.x; tid < nt; tid += (long)gridDim.x * blockDim.x) {
        const int i = (int)(tid / kRayThreads), half = (int)(tid % kRayThreads);
        const uint32_t cnt = counts[tid];
        if (cnt == 0u) continue;
        const int sc = scene_of(bt.off->point, bt.S, i);
        const SceneDev& sd = bt.sc[sc];
        const BinGeom g = scene_geom(sd, bt.fp[sc]);
        const float4 a = ra[i];
        const float bx = g.ax + a.x / sd.p.res, by = g.ay + a.y / sd.p.res, bz = g.az + a.z / sd.p.res;
        const uint32_t toff = (uint32_t)bt.off->tile[sc];
        uint32_t k = 0;
        for_each_tile(
            g, bx, by, bz,
            [&](int t) {
                if (k < cnt) {
                    f(i, toff + (uint32_t)t);
                    ++k;
                }
            },
            half, kRayThreads);
    }
}

__global__ void k_ray_place(Batch bt, const float4* __restrict__ ra, const uint32_t* __restrict__ counts,
                            const uint32_t* __restrict__ tile_start, const uint32_t* __restrict__ block_base,
                            const uint32_t* __restrict__ total, uint32_t* __restrict__ evals) {
    extern __shared__ uint32_t s_slot[];  // [T]: the block's next slot in each tile's range
    const uint32_t n = total[2];
    if (n == 0u) return;  // overflow, or no entries (the same for every thread)
    const uint32_t* row = block_base + (size_t)blockIdx.x * bt.T;
    // rows of tiles this block does not reach hold stale values that are never used
    for (int t = threadIdx.x; t < bt.T; t += blockDim.x) s_slot[t] = tile_start[t] + row[t];
    __syncthreads();
    for_each_placed_tile(bt, ra, counts, [&](int i, uint32_t gt) {
        const uint32_t pos = atomicAdd(&s_slot[gt], 1u);
        if (pos < n) evals[pos] = (uint32_t)i;
    });
}

// ---------------------------------------------------------------- DS lists in ray order
// The DS half of the placed lists: each tile keeps its rays in input order (the first-100 rule
// depends on it), so a slot cannot come from an atomic. A block of kMarkRays consecutive rays marks
// the tiles they reach in a bit mask per tile in shared memory; the number of a tile's rays in the
// block, and a ray's place among them, are population counts. k_ds_mark<false> keeps the counts, one
// row of T per block, and adds them up per group of kMarkGroup blocks; k_mark_groups turns the group
// sums into prefixes; k_tile_ranges places the tiles; k_ds_mark<true> marks again (the walk costs
// less than keeping the masks: 16 bytes per block and tile) and writes each tile's rays in order.
// Two round trips through the counts replace emitting (tile, ray) pairs, their histogram and two
// sort passes: 200x200x25 voxels, 60,000 rays 123 -> 58 us, 256x256x32 voxels, 120,000 rays 145 -> 76.
// (Thread per tile in the last loop instead of lane per ray: 115 us.)
constexpr int kMarkWords = kMarkRays / 32;

template <bool PLACE>
__global__ void __launch_bounds__(kMarkRays * kRayThreads)
k_ds_mark(Batch bt, const float* __restrict__ xs, const float* __restrict__ ys, const float* __restrict__ zs,
          float4* __restrict__ ra, uint32_t* __restrict__ rows, uint32_t* __restrict__ groups,
          const uint32_t* __restrict__ tile_start, const uint32_t* __restrict__ total,
          uint32_t* __restrict__ evals, DevStatus* status) {
    extern __shared__ uint4 s_mark[];  // [T]: the block's rays that reach the tile
    static_assert(kMarkWords == 4, "one uint4 per tile");
    const uint32_t n = PLACE ? total[2] : 0u;
    if (PLACE && n == 0u) return;  // overflow, or no entries (the same for every thread)
    if (!PLACE && blockIdx.x == 0 && threadIdx.x == 0) status->overflow = 0u;
    for (int t = threadIdx.x; t < bt.T; t += blockDim.x) s_mark[t] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    const int r = (int)threadIdx.x / kRayThreads, half = (int)threadIdx.x % kRayThreads;
    const int first = blockIdx.x * kMarkRays, i = first + r;
    const int sc = i < bt.N ? scene_of(bt.off->point, bt.S, i) : 0;
    if (i < bt.N && i - bt.off->point[sc] < bt.fp[sc].n_points) {
        const FrameParams f = bt.fp[sc];
        const SceneDev& sd = bt.sc[sc];
        BinGeom g = scene_geom(sd, f);
        float mx = xs[i], my = ys[i], mz = zs[i];
        if (f.has_transform) apply_transform(f, &mx, &my, &mz);
        float4 a;
        double4 c;
        const RayPrep p = prep_ray(sd.p, g, mx, my, mz, true, &a, &c);
        if (!PLACE && half == 0) ra[i] = a;
        if (p.ok) {
            uint32_t* word = reinterpret_cast<uint32_t*>(s_mark + bt.off->tile[sc]) + (r >> 5);
            const uint32_t bit = 1u << (r & 31);
            for_each_tile(g, p.bx, p.by, p.bz, [&](int t) { atomicOr(word + kMarkWords * t, bit); }, half, kRayThreads);
        } else if (!PLACE && half == 0 && !(isfinite(mx) && isfinite(my) && isfinite(mz))) {
            atomicAdd(&status->nonfinite_points, 1ull);
        }
    }
    __syncthreads();
    const int b = blockIdx.x, g0 = b / kMarkGroup;
    uint32_t* row = rows + (size_t)b * bt.T;
    if (!PLACE) {
        for (int t = threadIdx.x; t < bt.T; t += blockDim.x) {
            const uint4 m = s_mark[t];
            const uint32_t v = __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
            row[t] = v;
            if (v) atomicAdd(&groups[(size_t)g0 * bt.T + t], v);
        }
        return;
    }
    // a lane finds the block's first slot in its tile, then the warp writes the 32 tiles' rays one tile
    // at a time, a lane per ray
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    for (int t0 = (int)(threadIdx.x & ~31u); t0 < bt.T; t0 += blockDim.x) {
        const int t = t0 + lane;
        uint4 m = make_uint4(0u, 0u, 0u, 0u);
        if (t < bt.T) m = s_mark[t];
        const bool any = (m.x | m.y | m.z | m.w) != 0u;
        uint32_t pos = 0;
        if (any) {
            pos = tile_start[t] + groups[(size_t)g0 * bt.T + t];
#pragma unroll 8
            for (int q = g0 * kMarkGroup; q < b; ++q) pos += rows[(size_t)q * bt.T + t];
        }
        for (unsigned left = __ballot_sync(0xffffffffu, any); left; left &= left - 1u) {
            const int src = __ffs(left) - 1;
            uint32_t at = __shfl_sync(0xffffffffu, pos, src);
            const uint32_t w[kMarkWords] = {__shfl_sync(0xffffffffu, m.x, src), __shfl_sync(0xffffffffu, m.y, src),
                                            __shfl_sync(0xffffffffu, m.z, src), __shfl_sync(0xffffffffu, m.w, src)};
#pragma unroll
            for (int k = 0; k < kMarkWords; ++k) {
                const uint32_t o = at + __popc(w[k] & below);
                if ((w[k] >> lane & 1u) && o < n) evals[o] = (uint32_t)(first + 32 * k + lane);
                at += __popc(w[k]);
            }
        }
    }
}

// Per tile: group sums -> exclusive prefixes over the groups, and the tile's count.
__global__ void k_mark_groups(uint32_t* __restrict__ groups, int ngroups, int T, uint32_t* __restrict__ tile_tally) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T) return;
    uint32_t run = 0;
#pragma unroll 16
    for (int g = 0; g < ngroups; ++g) {
        uint32_t* p = groups + (size_t)g * T + t;
        const uint32_t v = *p;
        *p = run;
        run += v;
    }
    tile_tally[t] = run;
}

long ds_spare_items(long capacity, int chunk, int stride) {
    const long full = capacity / chunk + 1, kept = std::max(full / kDsSpareDiv, kDsSpareBytes / (5L * stride));
    return std::min({full, kept, 0x7FFFFFFFL});
}

int mark_blocks(int N) { return std::max(1, div_up(N, kMarkRays)); }
int mark_groups(int N) { return div_up(mark_blocks(N), kMarkGroup); }

// Blocks of the two placed-list passes (the same grid for both): at most kBinBlocksMax rows of
// block_base.
int bin_blocks(long n) { return (int)std::max(1L, std::min((n + kBlock - 1) / kBlock, (long)kBinBlocksMax)); }

// Largest |c| of a cell centre seen from a sensor inside or near the grid [m].
static float max_extent(const DevParams& p) { return 2.0f * ((float)p.G * p.res * 1.7320508f + p.size_z); }

void fill_scene_evidence(SceneDev& sd, bool ds, float4* ktab) {
    const DevParams& p = sd.p;
    if (!ds) {
        sd.bin_R = p.ls / p.res * (1.0f + 1e-4f) + 1e-3f;
    } else {
        // an upper bound of ds_window's radius, for the capacity of the ray lists
        const float ext = max_extent(p);
        const float slack = 64.0f * 5.96e-8f * ext * ext;
        sd.bin_R = sqrtf(p.window_radius * p.window_radius + slack) / p.res + 1e-3f;
    }
    sd.wr2 = p.window_radius * p.window_radius;
    // box culls (box_reaches): the support radius with a margin; DS (rays of ds_extreme): bin_R in metres
    const float rls = ds ? sd.bin_R * p.res : p.ls * (1.0f + 1e-4f) + 1e-3f * p.res;
    sd.cull_ls2 = rls * rls;
    // fixed point: the table is scaled by a power of two so that a kernel value is at most 1, and
    // one unit is 2^-40 of that: at most 2^40 units a value, leaving 2^23 terms of headroom in a
    // signed 64-bit sum
    const double sig = std::max((double)p.sigma, 1e-30);
    const int sh = kFxShift - (int)std::ceil(std::log2(sig));
    sd.fx_inv = std::ldexp(1.0, -sh);
    if (ktab) build_kernel_table(p.sigma, std::ldexp(1.0, sh - kFxShift), ktab);
}

// Worst case of tiles one ray can reach: for each slab of tiles along the ray's dominant axis A,
// the segment clipped to the slab grown by R spans at most ts[A] - 1 + 2R cells along every
// axis (|d_o| <= |d_A|), and the tiles within R of it along axis o number at most
// ceil((ts[A] + 4R) / ts[o]) + 1. Times the slabs, for the worst axis.
long ray_entries_bound(const DevParams& p, const TileShape& ts, int max_points, float bin_R) {
    const double R = (double)bin_R + 0.01;
    const int tsz[3] = {ts.tx, ts.ty, ts.tz}, nt[3] = {ts.ntx, ts.nty, ts.ntz};
    long worst = 0;
    for (int A = 0; A < 3; ++A) {
        long per_slab = 1;
        for (int k = 1; k <= 2; ++k) {
            const int o = (A + k) % 3;
            const long n = (long)std::ceil((tsz[A] + 4.0 * R) / tsz[o]) + 1;
            per_slab *= std::min<long>(n, nt[o]);
        }
        worst = std::max(worst, per_slab * nt[A]);
    }
    worst = std::min<long>(worst, (long)ts.ntx * ts.nty * ts.ntz);
    return worst * (long)max_points;
}

cudaError_t build_ray_lists(const Batch& bt, const float* xs, const float* ys, const float* zs, RayBuffers& rb,
                            bool ds, DevStatus* status, const SortWait& wait, cudaStream_t st) {
    const int N = bt.N;
    const int T = bt.T;
    if (ds && placed_lists(true, T, N)) {
        const size_t marks = sizeof(uint4) * (size_t)T;
        const int blocks = mark_blocks(N), groups = mark_groups(N);
        cudaError_t e = cudaMemsetAsync(rb.mark_groups, 0, sizeof(uint32_t) * (size_t)groups * T, st);
        if (e != cudaSuccess) return e;
        g_launches += 4;
        k_ds_mark<false><<<blocks, kMarkRays * kRayThreads, marks, st>>>(
            bt, xs, ys, zs, rb.ray_a, rb.block_base, rb.mark_groups, nullptr, nullptr, nullptr, status);
        k_mark_groups<<<div_up(T, 64), 64, 0, st>>>(rb.mark_groups, groups, T, rb.tile_tally);
        k_tile_ranges<<<1, kRangeThreads, 0, st>>>(rb.tile_tally, T, rb.chunk, rb.item_slots, rb.ds_spare, rb.capacity,
                                                   rb.tile_start, rb.item_off, rb.total, status);
        k_ds_mark<true><<<blocks, kMarkRays * kRayThreads, marks, st>>>(
            bt, xs, ys, zs, rb.ray_a, rb.block_base, rb.mark_groups, rb.tile_start, rb.total, rb.evals2, status);
        return cudaGetLastError();
    }
    if (placed_lists(ds, T, N)) {  // K3DOM: tally, ranges, place
        const size_t hist = sizeof(uint32_t) * (size_t)T;
        const int blocks = bin_blocks((long)N * kRayThreads);
        ++g_launches;
        k_ray_count<true><<<blocks, kBlock, hist, st>>>(bt, xs, ys, zs, 0, rb.ray_a, rb.ray_c, rb.counts,
                                                         rb.tile_tally, rb.block_base, status);
        ++g_launches;
        k_tile_ranges<<<1, kRangeThreads, 0, st>>>(rb.tile_tally, T, rb.chunk, rb.item_slots, rb.ds_spare, rb.capacity,
                                                   rb.tile_start, rb.item_off, rb.total, status);
        ++g_launches;
        k_ray_place<<<blocks, kBlock, hist, st>>>(bt, rb.ray_a, rb.counts, rb.tile_start, rb.block_base, rb.total,
                                                   rb.evals2);
        return cudaGetLastError();
    }
    // more tiles than a block holds in shared memory (or more DS counts than kMarkMaxCounts): entries
    // in ray order, then a stable sort by tile
    ++g_launches;
    k_ray_count<false><<<grid_for(N), kBlock, 0, st>>>(bt, xs, ys, zs, ds ? 1 : 0, rb.ray_a, rb.ray_c, rb.counts,
                                                        nullptr, nullptr, status);
    cudaError_t e = scan_u32_exclusive(rb.counts, rb.offsets, N, rb.scan_tmp, rb.total, st);
    if (e != cudaSuccess) return e;
    ++g_launches;
    k_ray_emit<<<grid_for(N), kBlock, 0, st>>>(bt, xs, ys, zs, ds ? 1 : 0, rb.offsets, rb.total, rb.capacity,
                                               rb.ekeys, rb.evals, status);
    int bits = 1;
    while ((1 << bits) < T + 1) ++bits;
    // stable: each tile keeps its rays in input order (the DS first-100 rule depends on it)
    SortWait w = wait;
    w.skip_tile = -1;
    e = onesweep_sort_pairs_dn(rb.ekeys, rb.evals, rb.ekeys2, rb.evals2, rb.ekeys_alt, rb.evals_alt, rb.capacity,
                               rb.total + 2, bits, rb.os_scratch, rb.os_words, status, w, st);
    if (e != cudaSuccess) return e;
    ++g_launches;
    k_tile_start<<<div_up(T + 1, kBlock), kBlock, 0, st>>>(rb.ekeys2, rb.total, T, rb.tile_start);
    ++g_launches;
    k_tile_items<<<div_up(T, kBlock), kBlock, 0, st>>>(rb.tile_start, rb.total, T, rb.chunk, rb.item_slots, rb.ds_spare,
                                                        rb.tile_items);
    e = scan_u32_exclusive(rb.tile_items, rb.item_off, T, rb.scan_tmp, rb.item_off + T, st);
    if (e != cudaSuccess) return e;
    ++g_launches;
    k_finish_lists<<<1, 1, 0, st>>>(rb.item_off, T, status, rb.total);
    return cudaGetLastError();
}

// ================================================================ shared kernel machinery
// Cell centre of index triple (ix, iy, iz), the expression of mass_update.cu:92-99 /
// measurement_grid.cu:77-84 evaluated in FP32 in the reference's order.
__device__ __forceinline__ void centre_xyz(int ix, int iy, int iz, const DevParams& p, float sx, float sy, float sz,
                                           float* x, float* y, float* z) {
    const float hg = __fdiv_rn((float)p.G, 2.0f), hz = __fdiv_rn((float)p.Gz, 2.0f);
    *x = __fsub_rn(__fmul_rn(__fsub_rn(__fadd_rn((float)ix, 0.5f), hg), p.res), sx);
    *y = __fsub_rn(__fmul_rn(__fsub_rn(__fadd_rn((float)iy, 0.5f), hg), p.res), sy);
    *z = __fsub_rn(__fmul_rn(__fsub_rn(__fadd_rn((float)iz, 0.5f), hz), p.res), sz);
}

// First cell (of the lowest indices) of sub-block sb in tile t.
struct SbCell {
    int x, y, z;
};
__device__ __forceinline__ SbCell sb_cell(const TileShape& ts, int t, int sb) {
    const int tx = t % ts.ntx, ty = (t / ts.ntx) % ts.nty, tz = t / (ts.ntx * ts.nty);
    const int sbx = sb % ts.nsbx, sby = (sb / ts.nsbx) % ts.nsby, sbz = sb / (ts.nsbx * ts.nsby);
    return SbCell{tx * ts.tx + sbx * 4, ty * ts.ty + sby * 4, tz * ts.tz + sbz * 2};
}

// Sub-blocks go to the warps nearest to the sensor first. A sub-block's work grows with the rays
// that pass it, which is largest on the tile's sensor side (rays that end inside the tile never
// reach its far side, and near the sensor every ray passes close), so the costly sub-blocks start
// first and the cheap ones fill the end of the work item, where warps that run out of sub-blocks
// wait at the item's barrier. The sums are exact, so the order changes no result.
constexpr int kMaxOrderedSb = 64;  // the largest tiling (16x16x8) has 64 sub-blocks

struct SbOrder {
    float key[kMaxOrderedSb];
    uint8_t idx[kMaxOrderedSb];
};

// Phase 1 (thread i < nsb): squared distance of sub-block i's anchor from the sensor.
__device__ __forceinline__ void sb_order_keys(SbOrder& o, const DevParams& p, const TileShape& ts, int t, int nsb,
                                              float sx, float sy, float sz) {
    const int i = threadIdx.x;
    if (nsb > kMaxOrderedSb || i >= nsb) return;
    const SbCell b = sb_cell(ts, t, i);
    float x, y, z;
    centre_xyz(b.x + 2, b.y + 2, b.z + 1, p, sx, sy, sz, &x, &y, &z);
    o.key[i] = x * x + y * y + z * z;
}

// Phase 2, after a barrier: sub-block i's place in the order (ties by index).
__device__ __forceinline__ void sb_order_rank(SbOrder& o, int nsb) {
    const int i = threadIdx.x;
    if (nsb > kMaxOrderedSb || i >= nsb) return;
    const float k = o.key[i];
    int r = 0;
    for (int j = 0; j < nsb; ++j) {
        const float kj = o.key[j];
        r += (kj < k) || (kj == k && j < i);
    }
    o.idx[r] = (uint8_t)i;
}

__device__ __forceinline__ int sb_at(const SbOrder& o, int n, int nsb) { return nsb > kMaxOrderedSb ? n : o.idx[n]; }

struct EvArgs {
    Batch bt;
    const uint32_t* item_off;
    const uint32_t* tile_start;
    const uint32_t* evals;
    const float4* ray_a;
    const double4* ray_c;
    const uint32_t* total;  // [2]: entries in the lists
    int item_slots, ds_spare;  // see item_rays
    uint32_t* tile_done;
    unsigned long long* acc;
    uint32_t* ds_r2;
    uint8_t* ds_counts;
    long ds_capacity;
    int ds_stride;
    CellState cs;
    CellWork cw;
    DevStatus* status;
    int first_frame;
    int chunk;  // rays per work item (<= kChunk)
    int fuse_update;  // K3DOM: the last CTA of a tile updates its cells (else k_k3dom_update_cells)
    cudaTextureObject_t ktex;  // the scenes' kernel tables (K3DOM), f's table (calibration)
};

// ================================================================ K3DOM
// The sparse kernel of mass_update.cu:24-26,
//   k(d) = max(0, sigma ((2 + cos(2 pi x)) (1 - x) / 3 + sin(2 pi x) / (2 * 3.141592))),  x = d / ls,
// (the reference's truncated pi in the sine term is kept) is tabulated as a function of
// u = d^2 / ls^2 (no square root in the hot loop): kKernelTab intervals, on each a cubic in the
// local coordinate through four FP64 samples (f = 0, 1/3, 2/3, 1). Evaluated in FP32 by Horner,
// it is within 1.2e-7 relative of the FP64 kernel wherever k > 1e-3 sigma and within 8e-8 sigma
// absolute everywhere; the direct FP32 formula loses up to ~1e-5 to cancellation between its two
// terms over the outer half of the support.
static double kernel_ref(double u, double sigma) {
    const double x = std::sqrt(u);
    const double v = sigma * ((2.0 + std::cos(M_PI * 2.0 * x)) * (1.0 - x) / 3.0 +
                              std::sin(M_PI * 2.0 * x) / (2.0 * 3.141592));
    return v > 0.0 ? v : 0.0;
}

void build_kernel_table(float sigma, double scale, float4* out) {
    for (int i = 0; i < kKernelTab; ++i) {
        double y[4];
        for (int j = 0; j < 4; ++j) y[j] = scale * kernel_ref(std::min(1.0, (i + j / 3.0) / kKernelTab), sigma);
        // inverse Vandermonde of the nodes 0, 1/3, 2/3, 1
        const double c0 = y[0];
        const double c1 = -5.5 * y[0] + 9.0 * y[1] - 4.5 * y[2] + y[3];
        const double c2 = 9.0 * y[0] - 22.5 * y[1] + 18.0 * y[2] - 4.5 * y[3];
        const double c3 = -4.5 * y[0] + 13.5 * y[1] - 13.5 * y[2] + 4.5 * y[3];
        out[i] = make_float4((float)c0, (float)c1, (float)c2, (float)c3);
    }
    out[kKernelTab] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

// Table position t = d^2 * (kKernelTab / ls^2) = u * kKernelTab (the factor kKernelTab is a power
// of two, so folding it into 1 / ls^2 changes no bit): interval i = floor(t), offset f = t - i.
// Inside the support (d^2 < ls^2) t <= kKernelTab, and entry kKernelTab is zero, so no clamp is
// needed. The floor is taken without conversion instructions: t + 2^23 rounded down is
// 2^23 + floor(t) exactly for 0 <= t < 2^23, whose low mantissa bits are floor(t).
struct TabPos {
    int i;
    float f;
};

// mass_update.cu:12-14, 1 - 2 / (1 + exp(2 mass / mass_scale)), with k2 = 2 / mass_scale
__device__ __forceinline__ double calc_credit(double mass, double k2) {
    return 1.0 - 2.0 / (1.0 + exp(mass * k2));
}
__device__ __forceinline__ double positive_diff(double a, double b) { return fmax(0.0, a - b); }
// mass_update.cu:16-19, 1 / (1 + rest / numerator), written numerator / (numerator + rest)
__device__ __forceinline__ double calc_ratio(double numerator, double rest) {
    return (numerator <= 0.0 || rest < 0.0) ? 0.0 : numerator / (numerator + rest);
}
__device__ __forceinline__ float calc_norm(float weight_sum, float rho_p) {
    return weight_sum > 0.0f ? rho_p / weight_sum : 0.0f;
}

// gridCellPredictionUpdateKernel's per-cell body (mass_update.cu:163-181) plus the per-cell
// updates of the persistent-particle and moment stages. Masses are stored in FP32; the update
// is evaluated in FP64 (it has several cancelling differences) and rounded once.
// g = gamma^dt of the frame.
// A cell's inputs to the update, loaded together so that their reads overlap (the particle sums
// are read whether or not the cell holds particles; they are used only when it does).
struct CellIn {
    float m_f, m_s, m_d, sum_w, wvx, wvy, wvz;
    int start;
};
__device__ __forceinline__ CellIn load_cell_in(const CellState& cs, const CellWork& cw, int c, bool first_frame) {
    CellIn in;
    in.m_f = cs.free_m[c];
    in.m_s = cs.static_m[c];
    in.m_d = cs.dyn_m[c];
    in.start = first_frame ? -1 : cw.start[c];
    in.sum_w = cw.sum_w[c];
    in.wvx = cw.sum_wvx[c];
    in.wvy = cw.sum_wvy[c];
    in.wvz = cw.sum_wvz[c];
    return in;
}

// The update of cell c from its inputs `in` (outputs written to cs, cw).
__device__ void k3dom_cell_update_in(const DevParams& p, double g, int c, double del_occ, double del_free,
                                     const CellIn& in, CellState cs, CellWork cw, bool first_frame) {
    double m_f = in.m_f, m_s = in.m_s, m_d = in.m_d;
    const int start = in.start;
    const bool has = start >= 0;
    const double dyn_pred = has ? (double)in.sum_w : 0.0;
    const double k2 = 2.0 / (double)p.mass_scale;
    const double pred_total = (m_f + m_d) * g;
    // predict_mass (:79-84)
    m_s *= g;
    m_d = fmin(dyn_pred, fmax(0.0, pred_total - m_s));
    m_f = pred_total - m_d;
    // update_mass (:86-139)
    if (del_free > 0.0 || del_occ > 0.0) {
        const double del_sigma = del_free + del_occ;
        const double prime_sigma = m_f + m_s + m_d;
        double l_DtoF = 0.0, l_StoFD = 0.0, l_FtoD = 0.0;
        if (prime_sigma > 0.0) {
            // base_f m / prime_sigma with base_f = credit (del_free - del_occ)+ / del_sigma:
            // one reciprocal of z = del_sigma prime_sigma serves the three fractions
            const double z = del_sigma * prime_sigma;
            const double w = calc_credit(sqrt(z), k2) / z;
            const double wf = w * positive_diff(del_free, del_occ);
            const double wo = w * positive_diff(del_occ, del_free);
            l_DtoF = wf * m_d;
            l_StoFD = wf * positive_diff(m_s + m_d, m_f);
            l_FtoD = wo * positive_diff(m_f, m_s + m_d);
        }
        const double diff_f = l_StoFD / 2.0 * m_s + l_DtoF * m_d - l_FtoD * m_f;
        const double diff_s = -l_StoFD * m_s;
        const double diff_d = l_FtoD * m_f + l_StoFD / 2.0 * m_s - l_DtoF * m_d;
        m_f += diff_f;
        m_s += diff_s;
        m_d += diff_d;
        const double credit2 = calc_credit(m_s + m_d, k2);
        const double beta = (1.0 - credit2) + credit2 * calc_ratio(m_s, m_d);
        m_s = m_s + beta * del_occ;
        m_d = m_d + (1.0 - beta) * del_occ;
        m_f = m_f + del_free;
    }
    // separate_newborn_part (:141-150)
    double born;
    if (dyn_pred <= 0.0) born = m_d;
    else if (pred_total <= dyn_pred) born = 0.0;
    else born = (m_d * p.p_B * (pred_total - dyn_pred)) / (dyn_pred + p.p_B * (pred_total - dyn_pred));
    const double pers = m_d - born;
    cs.free_m[c] = (float)m_f;
    cs.static_m[c] = (float)m_s;
    cs.dyn_m[c] = (float)m_d;
    cs.born_m[c] = (float)born;
    cs.pers_m[c] = (float)pers;
    cs.pred_m[c] = (float)dyn_pred;
    cw.del_occ[c] = (float)del_occ;
    cw.del_free[c] = (float)del_free;
    if (first_frame) return;
    // updatePersistentParticlesKernel2: mu_UA = pers / pred (p_A = 0 -> the only factor)
    const double mu_UA = (has && dyn_pred > 0.0) ? pers / dyn_pred : 0.0;
    cw.factor[c] = (float)mu_UA;
    // statisticalMomentsKernel2 with sum(w' v) = mu_UA * sum(w v)
    double vx = 0.0, vy = 0.0, vz = 0.0;
    if (has && pers > 0.0) {
        const double q = mu_UA / pers;
        vx = q * (double)in.wvx;
        vy = q * (double)in.wvy;
        vz = q * (double)in.wvz;
    }
    cs.mvx[c] = (float)vx;
    cs.mvy[c] = (float)vy;
    cs.mvz[c] = (float)vz;
}

__device__ __forceinline__ void k3dom_cell_update(const DevParams& p, double g, int c, double del_occ,
                                                  double del_free, CellState cs, CellWork cw, bool first_frame) {
    k3dom_cell_update_in(p, g, c, del_occ, del_free, load_cell_in(cs, cw, c, first_frame), cs, cw, first_frame);
}

// Shared memory of the evidence kernels: one chunk of rays (the cull's constants; the FP64 ones are
// read from global memory for the candidates only), the per-warp candidate rings and pair records.
// Dynamic, sized by the largest work item's ray count.
struct BgkiSmem {
    float* stage;    // [warps][kStageWarpFloats] pair records of the candidate rays
    uint16_t* ring;  // [warps][2][kRing] candidate rays waiting for a full batch: interior, general
    float4* u;       // [chunk] m / d_m, d_m
    uint32_t* rid;   // [chunk] point slot
    uint16_t* reg;   // [kRegions][chunk] rays per region of a 16x16 tile
};

// A 16x16-cell tile splits into kRegions columns of 8x8 cells (full tile height); a ray's region
// list holds it when its segment meets the column's cell-centre box grown by the binning radius
// (plus a quarter cell), the test that put it in the tile's list, so every ray that can reach a
// cell of the column is in the column's list. Sub-blocks then cull only their column's rays.
constexpr int kRegions = 4;

// A pair record holds the staged constants of two rays a, b interleaved per component, so that one
// 8-byte register pair feeds a packed instruction:
//   float4 0: (perp0.x, perp0.y) of a, b     1: (perp0.z, u.x)     2: (u.y, u.z)
// and, in the records of near and edge rays,
//   float4 3: (par0, par0 - margin)          4: (occ0.x, occ0.y)   5: (occ0.z, par0 - d_m)
// each float4 as (a, b, a, b); the larger records are padded by a seventh float4 so that the four
// records a step reads lie in different banks (12 floats do without).
constexpr int kRecInterior = 12, kRecGeneral = 28;
constexpr int kStageWarpFloats = 16 * kRecGeneral;
constexpr int kRing = 64;  // candidates kept per warp and class: up to 31 waiting and 32 new ones

constexpr size_t kBgkiFixedBytes = (size_t)kEvWarps * (sizeof(float) * kStageWarpFloats + 2 * sizeof(uint16_t) * kRing);
static_assert(kBgkiFixedBytes % 32 == 0, "alignment of what follows");

inline size_t bgki_smem_bytes(int chunk) {
    return kBgkiFixedBytes +
           (size_t)chunk * (sizeof(float4) + sizeof(uint32_t) + kRegions * sizeof(uint16_t));
}

__device__ __forceinline__ BgkiSmem bgki_smem(unsigned char* base, int chunk) {
    BgkiSmem S;
    S.stage = reinterpret_cast<float*>(base);
    S.ring = reinterpret_cast<uint16_t*>(base + sizeof(float) * (size_t)kEvWarps * kStageWarpFloats);
    S.u = reinterpret_cast<float4*>(base + kBgkiFixedBytes);
    S.rid = reinterpret_cast<uint32_t*>(S.u + chunk);
    S.reg = reinterpret_cast<uint16_t*>(S.rid + chunk);
    return S;
}

// Parameter interval [t0, t1] of a + t d inside the slab lo <= u <= hi (empty when t0 > t1).
__device__ __forceinline__ void slab(float a, float d, float lo, float hi, float* t0, float* t1) {
    if (d == 0.0f) {
        const bool in = a >= lo && a <= hi;
        *t0 = in ? -INFINITY : INFINITY;
        *t1 = in ? INFINITY : -INFINITY;
        return;
    }
    const float inv = 1.0f / d;
    const float e0 = (lo - a) * inv, e1 = (hi - a) * inv;
    *t0 = fminf(e0, e1);
    *t1 = fmaxf(e0, e1);
}

// Bit q (q = qx + 2 qy) set when the ray's binned segment a -> a + d (cell-index space) meets
// region q's box [x0 + 8 qx, x0 + 8 qx + 7] x [y0 + 8 qy, +7] x [z0, z0 + tz - 1] grown by R.
__device__ __forceinline__ unsigned region_mask(float ax, float ay, float az, float dx, float dy, float dz, float x0,
                                                float y0, float z0, int tz, float R) {
    float zl, zh;
    slab(az, dz, z0 - R, z0 + (float)(tz - 1) + R, &zl, &zh);
    zl = fmaxf(zl, 0.0f);
    zh = fminf(zh, 1.0f);
    float xl[2], xh[2], yl[2], yh[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        slab(ax, dx, x0 + 8.0f * h - R, x0 + 8.0f * h + 7.0f + R, &xl[h], &xh[h]);
        slab(ay, dy, y0 + 8.0f * h - R, y0 + 8.0f * h + 7.0f + R, &yl[h], &yh[h]);
    }
    unsigned q = 0;
#pragma unroll
    for (int qy = 0; qy < 2; ++qy)
#pragma unroll
        for (int qx = 0; qx < 2; ++qx)
            if (fmaxf(zl, fmaxf(xl[qx], yl[qy])) <= fminf(zh, fminf(xh[qx], yh[qy]))) q |= 1u << (qx + 2 * qy);
    return q;
}

// What the warps of a CTA need of the work item they hold, in shared memory: kept in registers it
// would crowd out the evaluation loops' own values at 64 registers a thread.
struct ItemConst {
    int live;  // 0: no item left
    int t, lt, nr, nsb, regions, coff, tbase;
    uint32_t item, e0, n_items;
    TileShape ts;
    int sc, G, Gz;
    float res, sx, sy, sz;
    float bin_R, ls2, tscale, rls2, rls;
};

// The tile of a work item: last t in [0, T) with item_off[t] <= item, 32 probes a step (the calling
// warp, item the same in every lane).
__device__ __forceinline__ int warp_find_tile(const uint32_t* __restrict__ item_off, int T, uint32_t item) {
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = T;
    while (hi - lo > 1) {
        const int span = hi - lo;
        const int pos = span <= 33 ? min(lo + 1 + lane, hi) : lo + (int)((long)(lane + 1) * span / 33);
        const unsigned m = __ballot_sync(0xffffffffu, pos < hi && item_off[pos] <= item);
        const int n = __popc(m);  // a prefix of the lanes
        const int at = __shfl_sync(0xffffffffu, pos, n > 0 ? n - 1 : 0);
        const int up = __shfl_sync(0xffffffffu, pos, n < 32 ? n : 31);
        if (n > 0) lo = at;
        if (n < 32) hi = min(hi, up);
    }
    return lo;
}

// Takes the next work item (the calling warp only).
__device__ __forceinline__ void fetch_item(const EvArgs& A, uint32_t total_items, int chunk, ItemConst* I) {
    const Batch& bt = A.bt;
    const int lane = threadIdx.x & 31;
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(&A.status->work_counter, 1u);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= total_items) {
        if (lane == 0) I->live = 0;
        return;
    }
    const int lo = warp_find_tile(A.item_off, bt.T, item);
    if (lane != 0) return;
    I->live = 1;
    I->item = item;
    I->t = lo;
    I->sc = scene_of(bt.off->tile, bt.S, lo);
    I->lt = lo - bt.off->tile[I->sc];
    const uint32_t first = A.item_off[lo];
    I->n_items = A.item_off[lo + 1] - first;
    I->e0 = A.tile_start[lo] + (item - first) * (uint32_t)chunk;
    const uint32_t e1 = min(A.tile_start[lo + 1], I->e0 + (uint32_t)chunk);
    I->nr = (int)(e1 > I->e0 ? e1 - I->e0 : 0);
    const SceneDev& sd = bt.sc[I->sc];
    const FrameParams& fp = bt.fp[I->sc];
    const TileShape ts = sd.ts;
    I->ts = ts;
    I->nsb = ts.nsbx * ts.nsby * (ts.tz / 2);
    I->regions = ts.tx == 16 && ts.ty == 16;
    I->coff = bt.off->cell[I->sc];
    I->tbase = I->sc * kKernelTabEntries;
    I->G = sd.p.G;
    I->Gz = sd.p.Gz;
    I->res = sd.p.res;
    I->sx = fp.sensor_x;
    I->sy = fp.sensor_y;
    I->sz = fp.sensor_z;
    I->bin_R = sd.bin_R;
    const float ls2 = sd.p.ls * sd.p.ls;
    I->ls2 = ls2;
    I->tscale = (1.0f / ls2) * (float)kKernelTab;  // d^2 -> table position
    I->rls2 = sd.cull_ls2;
    I->rls = sqrtf(sd.cull_ls2);
}

// Stages the item's rays in shared memory and, for a 16x16 tile, appends each ray to the lists of
// the regions it reaches (rcnt zeroed before the call; list order is arbitrary, the sums are
// exact). Every thread of the block calls it.
__device__ __forceinline__ void stage_item_rays(const EvArgs& A, const ItemConst& I, const BgkiSmem& S, int* rcnt) {
    const int lane = threadIdx.x & 31;
    const unsigned lanes_below = (1u << lane) - 1u;
    const TileShape ts = I.ts;
    const bool regions = I.regions != 0;
    const int nr = I.nr;
    // the sensor in cell-index space (place_sensor)
    const float hg = (float)I.G / 2.0f, hz = (float)I.Gz / 2.0f, ir = 1.0f / I.res;
    const float ax = I.sx / I.res + hg - 0.5f, ay = I.sy / I.res + hg - 0.5f, az = I.sz / I.res + hz - 0.5f;
    const float x0 = (float)(I.lt % ts.ntx * 16), y0 = (float)((I.lt / ts.ntx) % ts.nty * 16);
    const float z0 = (float)(I.lt / (ts.ntx * ts.nty) * ts.tz);
    for (int r0 = 0; r0 < nr; r0 += kEvThreads) {  // uniform trip count: the ballots below
        const int r = r0 + (int)threadIdx.x;
        unsigned qm = 0;
        if (r < nr) {
            uint32_t rid = A.evals[I.e0 + r];
            if (rid >= (uint32_t)A.bt.N) rid = 0;  // defensive: never read past the ray arrays
            const float4 a4 = A.ray_a[rid];
            const double inv = A.ray_c[rid].z;
            S.rid[r] = rid;
            S.u[r] = make_float4((float)(a4.x * inv), (float)(a4.y * inv), (float)(a4.z * inv), a4.w);
            if (regions)  // K3DOM binning segment: sensor -> point
                qm = region_mask(ax, ay, az, a4.x * ir, a4.y * ir, a4.z * ir, x0, y0, z0, ts.tz, I.bin_R + 0.25f);
        }
        if (regions) {
#pragma unroll
            for (int q = 0; q < kRegions; ++q) {
                const unsigned b = __ballot_sync(0xffffffffu, (qm >> q) & 1u);
                if (!b) continue;
                int base = 0;
                if (lane == 0) base = atomicAdd(&rcnt[q], __popc(b));
                base = __shfl_sync(0xffffffffu, base, 0);
                if ((qm >> q) & 1u) S.reg[q * A.chunk + base + __popc(b & lanes_below)] = (uint16_t)r;
            }
        }
    }
}

// Region of sub-block sb in a 16x16 tile (4x4 sub-blocks per layer).
__device__ __forceinline__ int sb_region(const TileShape& ts, int sb) {
    return ((sb % ts.nsbx) >> 1) + 2 * (((sb / ts.nsbx) % ts.nsby) >> 1);
}

// Pair geometry. For the anchor o of a sub-block and a ray m (FP64, once per lane-ray):
//   par0 = o.u, perp0 = o - par0 u, occ0 = o - m, and par0 - margin, par0 - d_m.
// For a cell c = o + delta (delta small and exact), with dpar = delta.u:
//   projection d_proj = par0 + dpar; perpendicular offset perp0 + delta - dpar u;
//   distance to the free segment [0, margin u] (the three branches of mass_update.cu:57-65)
//   = |perp|^2 + (min(d_proj, 0) + max(d_proj - margin, 0))^2, valid while d_proj < d_m;
//   distance to the point = |occ0 + delta|.
// Every FP32 quantity is O(ls), so the FP32 evaluation keeps ~1e-7 relative accuracy at any
// distance from the sensor (the direct |c|^2 - d_proj^2 form of :60 loses ~1e-5 at 20 m).
//
// The cull (cull_hits, FP32, one listed ray per lane) bounds the distance from a convex set K (the
// segment [0, d_m u], or the point) to the
// sub-block's cell centres x = c + h, |h_i| <= e_i, e = (1.5, 1.5, 0.5) res around the centroid c.
// dist(K, .) is convex with gradient D / |D| at c (D = c minus the closest point of K), so
// dist(K, x) >= |D| - (e . |D|) / |D| for every cell centre, where |D| is taken componentwise in
// e . |D|. No cell is within rls = ls (1 + 1e-4) + 1e-3 res of K unless |D|^2 - e . |D| < rls |D|
// (box_reaches). This is tighter than a sphere around c for the flat 4x4x2 sub-block, above all
// for the near-horizontal rays of a LiDAR scan. D is formed in FP32 from the sensor-relative
// centroid, so rls grows by 1e-6 of the centroid's distance (about four times the rounding of the
// products); a ray let through in excess adds nothing.
//
// The candidates are collected over the listed rays in two warp-private rings until 32 of a class
// are there, and only then resolved in FP64, one per lane, into pair records:
//   interior  every cell of the sub-block projects inside [0, margin] and is farther than ls from
//             the point: the occupied term and the along-ray term are exactly zero and are left
//             out, as is the d_m test;
//   general   the others: near rays (the point's sphere can reach a cell) and edge rays (a cell may
//             project before the sensor or beyond the margin).
// The class is decided from the cull's FP32 geometry with the same rounding slack (3 res is the most
// a cell's own offset can add to a projection), so a ray near a limit is taken as general, which is
// always right. Within a general batch the near rays are told apart exactly (box_reaches on the
// point): for the others no cell with d_proj >= d_m is within ls of the free segment either (margin
// <= d_m, so such a cell is at least as far from the segment's end as from the point, and the bound
// above keeps 1e-4 ls + 1e-3 res of slack), so their free term needs no d_m test.
__device__ __forceinline__ bool box_reaches(float Dx, float Dy, float Dz, float D2, float hres, float rls2) {
    const float s = fmaf(3.0f * hres, fabsf(Dx) + fabsf(Dy), hres * fabsf(Dz));
    const float t = D2 - s;
    return t <= 0.0f || t * t < rls2 * D2;
}

enum RayClass { kRayNone, kRayInterior, kRayGeneral };

// The cull of one ray (unit direction u.xyz, length u.w) on the sub-block with centroid (cx, cy,
// cz); rls: support radius with the rounding slack eps.
__device__ __forceinline__ RayClass cull_ray(const float4& u, float cx, float cy, float cz, float hres, float rls,
                                             float eps) {
    const float proj = fmaf(cz, u.z, fmaf(cy, u.y, cx * u.x));
    const float t = fminf(fmaxf(proj, 0.0f), u.w);
    const float Dx = fmaf(-t, u.x, cx), Dy = fmaf(-t, u.y, cy), Dz = fmaf(-t, u.z, cz);
    const float D2 = fmaf(Dz, Dz, fmaf(Dy, Dy, Dx * Dx));
    if (!box_reaches(Dx, Dy, Dz, D2, hres, rls * rls)) return kRayNone;
    // interior: proj is the centroid's projection, the anchor's lies within sqrt(3)/2 res of it, a
    // cell's within 3 res of that
    const float reach = 8.0f * hres + eps;
    const float margin = fmaxf(0.9f * u.w, u.w - 4.0f * hres);
    const float e = u.w - t, far2 = rls + 4.4f * hres;  // 4.36 hres: half diagonal of the cell centres
    return proj > reach && margin - proj > reach && fmaf(e, e, D2) > far2 * far2 ? kRayInterior : kRayGeneral;
}

// The constants of a candidate, in the order of the pair record.
struct RayStage {
    float v[12];
};

__device__ __forceinline__ void stage_interior(const float4& a, double inv, const float4& u, float oxf, float oyf,
                                               float ozf, RayStage* st) {
    const double ox = oxf, oy = oyf, oz = ozf;
    const double par0 = (ox * a.x + oy * a.y + oz * a.z) * inv;
    const double sc = par0 * inv;
    const double px = ox - sc * a.x, py = oy - sc * a.y, pz = oz - sc * a.z;
    st->v[0] = (float)px; st->v[1] = (float)py; st->v[2] = (float)pz;
    st->v[3] = u.x; st->v[4] = u.y; st->v[5] = u.z;
}

// Also true when the ray is near.
__device__ __forceinline__ bool stage_general(const float4& a, const double4& cd, const float4& u, float oxf,
                                              float oyf, float ozf, float hres, float rls2, RayStage* st) {
    const double ox = oxf, oy = oyf, oz = ozf;
    const double par0 = (ox * a.x + oy * a.y + oz * a.z) * cd.z;
    const double sc = par0 * cd.z;
    const double px = ox - sc * a.x, py = oy - sc * a.y, pz = oz - sc * a.z;
    const float ex = __fsub_rn(oxf, a.x), ey = __fsub_rn(oyf, a.y), ez = __fsub_rn(ozf, a.z);
    st->v[0] = (float)px; st->v[1] = (float)py; st->v[2] = (float)pz;
    st->v[3] = u.x; st->v[4] = u.y; st->v[5] = u.z;
    st->v[6] = (float)par0; st->v[7] = (float)(par0 - cd.y);
    st->v[8] = ex; st->v[9] = ey; st->v[10] = ez;
    st->v[11] = (float)(par0 - cd.x);
    const float cx = ex - hres, cy = ey - hres, cz = ez - hres;
    return box_reaches(cx, cy, cz, cx * cx + cy * cy + cz * cz, hres, rls2);
}

// Two FP32 values in one 8-byte register pair for the packed f32x2 instructions of sm_100a: one
// instruction applies the same IEEE operation (round to nearest unless stated) to both halves, so
// each half equals the scalar operation on it.
struct F2 {
    unsigned long long v;
    static __device__ __forceinline__ F2 of(float a, float b) {
        F2 r;
        asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
        return r;
    }
    __device__ __forceinline__ void split(float& a, float& b) const {
        asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    }
};
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    F2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
    return d;
}
__device__ __forceinline__ F2 add2_rd(F2 a, F2 b) {  // rounded toward -infinity
    F2 d;
    asm("add.rm.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
    return d;
}
__device__ __forceinline__ F2 sub2(F2 a, F2 b) {
    F2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
    return d;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d.v) : "l"(a.v), "l"(b.v));
    return d;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return d;
}

// A lane evaluates four cells of the sub-block, x = lane & 3, y = 2 * ((lane >> 2) & 1) + {0, 1} at
// both heights, for one of the four pair records of a step (its quarter-warp's): a record's 8-byte
// operands are loaded for 8 lanes x 4 cells instead of 32 lanes x 1, which divides the shared-memory
// traffic per evaluation by four, and the parts of the arithmetic that depend on x, y or z alone are
// done once per column. The anchor is a cell centre of the upper layer, so the upper cells' own z
// offset is exactly 0.
//
// What bounds k_bgki: with one cell per lane the record loads (512 bytes returned to registers per
// 16-byte broadcast) and the table's gathers filled half of the L1 data path each while instruction
// issue sat at 72 %, so cutting instructions alone changed little. 256x256x32 voxels at 0.1 m,
// 120,000 rays, 3.0e8 evaluations, evidence stage: one cell per lane, a conversion instruction per
// value and a batch per 32 listed rays 1.51 ms; the units' sums by additions, the interior class and
// full batches 1.38 ms; two cells per lane 1.24 ms; four 1.20 ms (200x200x25 voxels at 0.2 m, 60,000
// rays, ls 0.5 m: 0.54 -> 0.42 ms). The warp instructions per evaluation went from 4.2 to 3.2; what
// is left is the table's gathers (half of the L1 data path) and the waits on them. Two registers
// fewer for the tests (two limits and NaN columns instead of four limits) end the spills: evidence
// 1.19 -> 1.14 ms, the frame 1.745 -> 1.672. Slower here: the
// table in shared memory (1.38 ms), predicated fetches for all cells at once (spills at 64 registers,
// and 1.36 ms at 128 registers with 2 CTAs per SM), 3 CTAs per SM at 80 registers (1.21 ms).
struct Cols {
    F2 EX, EY[2], EZ;  // anchor minus the cell centres: x, both y, z of the lower cells
    F2 TS;             // table scale
    float ls2[2];      // ls^2 of the lower and the upper cells; -1 outside the grid (a column
                       // outside it has NaN offsets, so no test on it is true)
};

// Squared perpendicular distances of the four cells to the lines of the two rays of a pair record
// (float4 0-2); nd = -delta.u: q = p + delta - dp u = (p - E) + nd u, squares summed in x, y, z
// order.
struct Perp {
    F2 nd[4], d2[4];
};
__device__ __forceinline__ Perp perp_d2(const float4* __restrict__ R, const Cols& C) {
    const float4 b0 = R[0], b1 = R[1], b2 = R[2];
    const F2 ux = F2::of(b1.z, b1.w), uy = F2::of(b2.x, b2.y), uz = F2::of(b2.z, b2.w);
    const F2 sx = mul2(C.EX, ux);
    const F2 ax = sub2(F2::of(b0.x, b0.y), C.EX), py = F2::of(b0.z, b0.w), pz = F2::of(b1.x, b1.y);
    const F2 azl = sub2(pz, C.EZ);
    Perp r;
#pragma unroll
    for (int y = 0; y < 2; ++y) {
        const F2 up = fma2(C.EY[y], uy, sx), lo = fma2(C.EZ, uz, up);
        const F2 ay = sub2(py, C.EY[y]);
        r.nd[y] = lo;
        r.nd[2 + y] = up;
        {
            const F2 qx = fma2(lo, ux, ax), qy = fma2(lo, uy, ay), qz = fma2(lo, uz, azl);
            r.d2[y] = fma2(qz, qz, fma2(qy, qy, mul2(qx, qx)));
        }
        {
            const F2 qx = fma2(up, ux, ax), qy = fma2(up, uy, ay), qz = fma2(up, uz, pz);
            r.d2[2 + y] = fma2(qz, qz, fma2(qy, qy, mul2(qx, qx)));
        }
    }
    return r;
}

// The along-ray part added to it: al = min(par0 + dp, 0) + max(par0 - margin + dp, 0).
__device__ __forceinline__ F2 along_d2(F2 perp2, const float4& b3, F2 nd) {
    float a0, a1, e0, e1;
    sub2(F2::of(b3.x, b3.y), nd).split(a0, a1);  // d_proj
    sub2(F2::of(b3.z, b3.w), nd).split(e0, e1);  // d_proj - margin
    const F2 al = add2(F2::of(fminf(a0, 0.0f), fminf(a1, 0.0f)), F2::of(fmaxf(e0, 0.0f), fmaxf(e1, 0.0f)));
    return fma2(al, al, perp2);
}

// tab_pos for two squared distances: t = d^2 * tscale, then the floor without conversions.
struct TabPos2 {
    TabPos a, b;
};
__device__ __forceinline__ TabPos2 tab_pos2(F2 d2, F2 tscale) {
    const F2 c23 = F2::of(8388608.0f, 8388608.0f);
    const F2 t = mul2(d2, tscale);
    const F2 tr = add2_rd(t, c23);
    const F2 f = sub2(t, sub2(tr, c23));
    float ra, rb;
    tr.split(ra, rb);
    TabPos2 q;
    q.a.i = __float_as_int(ra) - 0x4B000000;
    q.b.i = __float_as_int(rb) - 0x4B000000;
    f.split(q.a.f, q.b.f);
    return q;
}

// Exact sums of values in [-1, 2) in units of 2^-kFxShift, without conversion instructions. A value
// v is split as h + l, h the nearest multiple of 2^-21 (v + 6 has that ulp) and l the exact rest;
// l + 1.5 * 2^-17 has an ulp of one unit, so it rounds l (and with it v, since h is a multiple of
// two units) to the nearest integer number of units, ties to even: the integer __float2ll_rn gives
// for v * 2^40. The mantissas of the two sums are those integers plus a constant, so their bit
// patterns are added as 32-bit integers and the constants leave once, by the number of values n.
// Two values cost four packed additions and two three-operand integer adds; the conversion
// instruction they replace issues at a quarter of that rate or less.
constexpr float kFxHi = 6.0f;                    // [4, 8): ulp 2^-21
constexpr float kFxLo = 1.5f / (1 << 17);        // [2^-17, 2^-16): ulp 2^-40
constexpr uint32_t kFxHiBits = 0x40C00000u, kFxLoBits = 0x37400000u;
constexpr int kFxMost = 2047, kFxMostSigned = 1023;
// Values a sub-block adds per cell: the item's rays, and up to 7 pads in the last batch of each class.
constexpr int kFxPads = 14;
static_assert(kChunk + kFxPads <= kFxMost, "K3DOM sums");
static_assert(kCalibChunk + kFxPads <= kFxMostSigned, "calibration sums: the derivative's are signed");

struct FxSum {
    uint32_t hi, lo;
    __device__ __forceinline__ void add(F2 v) {
        const F2 H = F2::of(kFxHi, kFxHi), L = F2::of(kFxLo, kFxLo);
        const F2 t = add2(v, H);
        const F2 q = add2(sub2(v, sub2(t, H)), L);
        float ta, tb, qa, qb;
        t.split(ta, tb);
        q.split(qa, qb);
        hi += __float_as_uint(ta) + __float_as_uint(tb);
        lo += __float_as_uint(qa) + __float_as_uint(qb);
    }
    // The sum of n added values, in units; at most kFxMost values in [0, 1] (total), or kFxMostSigned in
    // [-1, 1] (total_signed): the high parts, at most 2^21 each, add up in 32 bits.
    __device__ __forceinline__ long long total(uint32_t n) const {
        return ((long long)(uint32_t)(hi - n * kFxHiBits) << 19) + (int32_t)(lo - n * kFxLoBits);
    }
    __device__ __forceinline__ long long total_signed(uint32_t n) const {
        return ((long long)(int32_t)(hi - n * kFxHiBits) << 19) + (int32_t)(lo - n * kFxLoBits);
    }
};

// Writes the first N staged constants of a candidate into half (slot & 1) of pair record slot / 2.
template <int REC, int N>
__device__ __forceinline__ void stage_put(float* stg, int slot, const RayStage& st) {
    float* d = stg + (slot >> 1) * REC + (slot & 1);
#pragma unroll
    for (int i = 0; i < N; ++i) d[2 * i] = st.v[i];
}

// A pad ray: perpendicular and point offsets of 1e15 put every cell at a squared distance near 3e30
// (finite in FP32, far beyond ls^2), and d_proj - d_m = d_proj = 0 fails the d_proj < d_m test, so
// the pad adds nothing.
__device__ __forceinline__ RayStage pad_ray() {
    RayStage st;
#pragma unroll
    for (int i = 0; i < 12; ++i) st.v[i] = (i < 3 || (i >= 8 && i < 11)) ? 1e15f : 0.0f;
    return st;
}

// Batches of up to 32 candidate rays (r of each lane; the first n lanes hold one) against the
// sub-block with anchor (ox, oy, oz): FP64 resolution, pair records (padded to a multiple of four
// records by rays that reach no cell), evaluation. V evaluates: occ(i, pos, a, b) and free(...) take
// the table positions of a pair and whether each ray's value counts for the lane's cell i.
template <class V>
__device__ __forceinline__ void interior_batch(const EvArgs& A, const BgkiSmem& S, const Cols& C, float ox, float oy,
                                               float oz, float* stg, int r, int n, V& ev) {
    const int lane = threadIdx.x & 31;
    {
        RayStage st = pad_ray();
        if (lane < n) {
            const uint32_t rid = S.rid[r];
            stage_interior(__ldg(A.ray_a + rid), __ldg(&A.ray_c[rid].z), S.u[r], ox, oy, oz, &st);
        }
        stage_put<kRecInterior, 6>(stg, lane, st);
        __syncwarp();
    }
    const int steps = (n + 7) >> 3;
    const float* rec = stg + (lane >> 3) * kRecInterior;  // the quarter-warp's record of each step
#pragma unroll 1
    for (int k = 0; k < steps; ++k, rec += 4 * kRecInterior) {
        const Perp p = perp_d2(reinterpret_cast<const float4*>(rec), C);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float da, db;
            p.d2[i].split(da, db);
            ev.free(i, tab_pos2(p.d2[i], C.TS), da < C.ls2[i >> 1], db < C.ls2[i >> 1]);
        }
    }
    ev.n_free += steps;
    __syncwarp();
}

template <class V>
__device__ __forceinline__ void general_batch(const EvArgs& A, const BgkiSmem& S, const ItemConst& I, const Cols& C,
                                              float ox, float oy, float oz, float* stg, int r, int n, V& ev) {
    const int lane = threadIdx.x & 31;
    int near_steps;
    {
        RayStage st = pad_ray();
        bool near = false;
        if (lane < n) {
            const uint32_t rid = S.rid[r];
            const double2* c = reinterpret_cast<const double2*>(A.ray_c + rid);
            const double2 c0 = __ldg(c), c1 = __ldg(c + 1);
            near = stage_general(__ldg(A.ray_a + rid), make_double4(c0.x, c0.y, c1.x, 0.0), S.u[r], ox, oy, oz,
                                 0.5f * I.res, I.rls2, &st);
        }
        // near rays first; a step that holds one evaluates all its rays as near, which adds nothing
        // for the others
        const unsigned m = __ballot_sync(0xffffffffu, near);
        const int nn = __popc(m), below = __popc(m & ((1u << lane) - 1u));
        stage_put<kRecGeneral, 12>(stg, near ? below : nn + lane - below, st);
        near_steps = (nn + 7) >> 3;
        __syncwarp();
    }
    const int steps = (n + 7) >> 3;
    const float* rec = stg + (lane >> 3) * kRecGeneral;
    int k = 0;
    // steps holding a near ray: occupied (mass_update.cu:48-52) and free (:54-71) evidence
    ev.begin_occ();
#pragma unroll 1
    for (; k < near_steps; ++k, rec += 4 * kRecGeneral) {
        const float4* R = reinterpret_cast<const float4*>(rec);
        float da, db;
        {
            const float4 b4 = R[4], b5 = R[5];
            const F2 vx = sub2(F2::of(b4.x, b4.y), C.EX), vz = F2::of(b5.x, b5.y), vl = sub2(vz, C.EZ);
            const F2 xx = mul2(vx, vx);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const F2 vy = sub2(F2::of(b4.z, b4.w), C.EY[i & 1]);
                const F2 w = i < 2 ? vl : vz;
                const F2 d2 = fma2(w, w, fma2(vy, vy, xx));
                d2.split(da, db);
                ev.occ(i, tab_pos2(d2, C.TS), da < C.ls2[i >> 1], db < C.ls2[i >> 1]);
            }
        }
        const Perp p = perp_d2(R, C);
        const float4 b3 = R[3], b5 = R[5];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const F2 d2 = along_d2(p.d2[i], b3, p.nd[i]);
            float ea, eb;
            d2.split(da, db);
            sub2(F2::of(b5.z, b5.w), p.nd[i]).split(ea, eb);  // d_proj - d_m
            ev.free(i, tab_pos2(d2, C.TS), ea < 0.0f && da < C.ls2[i >> 1], eb < 0.0f && db < C.ls2[i >> 1]);
        }
    }
    if (near_steps) ev.end_occ(near_steps);
    // the other steps: free evidence only
#pragma unroll 1
    for (; k < steps; ++k, rec += 4 * kRecGeneral) {
        const float4* R = reinterpret_cast<const float4*>(rec);
        const Perp p = perp_d2(R, C);
        const float4 b3 = R[3];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const F2 d2 = along_d2(p.d2[i], b3, p.nd[i]);
            float da, db;
            d2.split(da, db);
            ev.free(i, tab_pos2(d2, C.TS), da < C.ls2[i >> 1], db < C.ls2[i >> 1]);
        }
    }
    ev.n_free += steps;
    __syncwarp();
}

// The evidence of sub-block sb of the item: the cull of its listed rays (its region's, or all of
// the item's), their batches, and the cells' sums.
template <class V>
__device__ __forceinline__ void eval_sub_block(const EvArgs& A, const BgkiSmem& S, const ItemConst& I, int sb,
                                               const int* rcnt, float* stg, uint16_t* ring, V& ev) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const uint16_t* list = nullptr;
    int nlist = I.nr;
    if (I.regions) {
        const int q = sb_region(I.ts, sb);
        list = S.reg + q * A.chunk;
        nlist = rcnt[q];
    }
    if (nlist == 0) return;
    Cols C;
    float ox, oy, oz;
    {
        DevParams p;  // the fields centre_xyz reads
        p.G = I.G; p.Gz = I.Gz; p.res = I.res;
        const SbCell b = sb_cell(I.ts, I.lt, sb);
        const int ix = b.x + (lane & 3), iy = b.y + 2 * ((lane >> 2) & 1);
        float x, y0, y1, z, t;
        centre_xyz(ix, iy, b.z, p, I.sx, I.sy, I.sz, &x, &y0, &z);
        centre_xyz(ix, iy + 1, b.z, p, I.sx, I.sy, I.sz, &t, &y1, &t);
        centre_xyz(b.x + 2, b.y + 2, b.z + 1, p, I.sx, I.sy, I.sz, &ox, &oy, &oz);
        // exact (nearby floats)
        const float nan = __int_as_float(0x7fffffff);
        const float ex = ix < I.G ? ox - x : nan, ey0 = iy < I.G ? oy - y0 : nan, ey1 = iy + 1 < I.G ? oy - y1 : nan;
        const float ez = oz - z, ts = I.tscale;
        C.EX = F2::of(ex, ex); C.EY[0] = F2::of(ey0, ey0); C.EY[1] = F2::of(ey1, ey1); C.EZ = F2::of(ez, ez);
        C.TS = F2::of(ts, ts);
        C.ls2[0] = b.z < I.Gz ? I.ls2 : -1.0f;
        C.ls2[1] = b.z + 1 < I.Gz ? I.ls2 : -1.0f;
    }
    ev.begin(I);
    uint16_t* gring = ring + kRing;
    int head = 0, n = 0, ghead = 0, gn = 0;  // interior and general candidates
    for (int g0 = 0; g0 < nlist; g0 += 32) {
        const int j = g0 + lane;
        int r = j;
        RayClass cls = kRayNone;
        if (j < nlist) {
            if (list) r = list[j];
            const float hres = 0.5f * I.res;
            const float cx = ox - hres, cy = oy - hres, cz = oz - hres;
            const float eps = 1e-6f * (fabsf(cx) + fabsf(cy) + fabsf(cz));
            cls = cull_ray(S.u[r], cx, cy, cz, hres, I.rls + eps, eps);
        }
        const unsigned mi = __ballot_sync(0xffffffffu, cls == kRayInterior);
        const unsigned mg = __ballot_sync(0xffffffffu, cls == kRayGeneral);
        if (cls == kRayInterior) ring[(head + n + __popc(mi & below)) & (kRing - 1)] = (uint16_t)r;
        if (cls == kRayGeneral) gring[(ghead + gn + __popc(mg & below)) & (kRing - 1)] = (uint16_t)r;
        n += __popc(mi);
        gn += __popc(mg);
        const bool last = g0 + 32 >= nlist;
        if (n < 32 && gn < 32 && !last) continue;
        __syncwarp();
        // full batches, and what is left after the last group
#pragma unroll 1
        for (; n >= 32 || (last && n > 0); n -= 32, head += 32)
            interior_batch(A, S, C, ox, oy, oz, stg, ring[(head + lane) & (kRing - 1)], min(n, 32), ev);
#pragma unroll 1
        for (; gn >= 32 || (last && gn > 0); gn -= 32, ghead += 32)
            general_batch(A, S, I, C, ox, oy, oz, stg, gring[(ghead + lane) & (kRing - 1)], min(gn, 32), ev);
    }
    // lane's output cell: column (lane & 7) of its four cells, the one of its quarter-warp
    const SbCell b = sb_cell(I.ts, I.lt, sb);
    const int q = lane >> 3;
    const int ix = b.x + (lane & 3), iy = b.y + 2 * ((lane >> 2) & 1) + (q & 1), iz = b.z + (q >> 1);
    const bool in = ix < I.G && iy < I.G && iz < I.Gz;
    ev.end(A, (long)I.coff + ix + I.G * iy + I.G * I.G * iz, in);
}

// The four quarter-warps' sums of the lane's four cells, added up: quarter q keeps cell q.
__device__ __forceinline__ FxSum quarter_merge(const FxSum s[4]) {
    const bool odd = (threadIdx.x & 8) != 0, up = (threadIdx.x & 16) != 0;
    FxSum k[2];  // cells (odd, z = 0, 1) of two quarters
#pragma unroll
    for (int z = 0; z < 2; ++z) {
        const FxSum mine = odd ? s[2 * z + 1] : s[2 * z], other = odd ? s[2 * z] : s[2 * z + 1];
        k[z].hi = mine.hi + __shfl_xor_sync(0xffffffffu, other.hi, 8);
        k[z].lo = mine.lo + __shfl_xor_sync(0xffffffffu, other.lo, 8);
    }
    const FxSum mine = up ? k[1] : k[0], other = up ? k[0] : k[1];
    return FxSum{mine.hi + __shfl_xor_sync(0xffffffffu, other.hi, 16),
                 mine.lo + __shfl_xor_sync(0xffffffffu, other.lo, 16)};
}

// K3DOM values: the scene's table through the texture path. FMA.SAT turns a negative table value
// (the kernel's max(0, .)) into 0; values are at most 1. The free sums are kept for the lane's four
// cells, the occupied ones (few rays are near) are merged after every run of near steps.
struct K3domEval {
    cudaTextureObject_t tex;
    int base;                   // the scene's table in the texture
    FxSum so[4], sf[4], occ_sum;
    int n_occ, n_free;          // steps added (two values per quarter-warp and step)
    unsigned nev;               // in-support evaluations of this lane (the roofline's work count)
    __device__ __forceinline__ void begin(const ItemConst& I) {
        base = I.tbase;
#pragma unroll
        for (int i = 0; i < 4; ++i) sf[i] = FxSum{0u, 0u};
        occ_sum = FxSum{0u, 0u};
        n_occ = n_free = 0;
    }
    __device__ __forceinline__ void begin_occ() {
#pragma unroll
        for (int i = 0; i < 4; ++i) so[i] = FxSum{0u, 0u};
    }
    __device__ __forceinline__ void end_occ(int steps) {
        const FxSum o = quarter_merge(so);
        occ_sum.hi += o.hi;
        occ_sum.lo += o.lo;
        n_occ += steps;
    }
    __device__ __forceinline__ float value(const TabPos& q) {
        const float4 c = tex1Dfetch<float4>(tex, base + q.i);
        return __saturatef(fmaf(q.f, fmaf(q.f, fmaf(q.f, c.w, c.z), c.y), c.x));
    }
    __device__ __forceinline__ F2 pair(const TabPos2& q, bool a, bool b) {
        float va = 0.0f, vb = 0.0f;
        if (a) { va = value(q.a); ++nev; }
        if (b) { vb = value(q.b); ++nev; }
        return F2::of(va, vb);
    }
    __device__ __forceinline__ void occ(int i, const TabPos2& q, bool a, bool b) { so[i].add(pair(q, a, b)); }
    __device__ __forceinline__ void free(int i, const TabPos2& q, bool a, bool b) { sf[i].add(pair(q, a, b)); }
    __device__ __forceinline__ void end(const EvArgs& A, long c, bool in) {
        const FxSum f = quarter_merge(sf);
        if (!in) return;
        unsigned long long* ac = A.acc + 2 * c;
        const long long vo = occ_sum.total(8u * n_occ), vf = f.total(8u * n_free);
        if (vo) atomicAdd(ac, (unsigned long long)vo);
        if (vf) atomicAdd(ac + 1, (unsigned long long)vf);
    }
};

// The work loop of a persistent CTA: items from the device counter, each staged by the whole CTA,
// its sub-blocks pulled by the warps; done(I) runs on every thread after an item's last sub-block
// (between barriers).
template <class V, class D>
__device__ __forceinline__ void run_items(const EvArgs& A, unsigned char* smem, V& ev, D done) {
    __shared__ ItemConst I;
    __shared__ int s_next_sb;
    __shared__ SbOrder s_order;
    __shared__ int s_rcnt[kRegions];
    const BgkiSmem S = bgki_smem(smem, A.chunk);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t total_items = A.item_off[A.bt.T];
    const int chunk = item_rays(A.total[2], A.chunk, A.item_slots, 0);
    for (;;) {
        if (wid == 0) fetch_item(A, total_items, chunk, &I);
        if (threadIdx.x < kRegions) s_rcnt[threadIdx.x] = 0;
        if (threadIdx.x == kEvThreads - 1) s_next_sb = 0;
        __syncthreads();
        if (!I.live) break;
        stage_item_rays(A, I, S, s_rcnt);
        {
            DevParams p;
            p.G = I.G; p.Gz = I.Gz; p.res = I.res;
            sb_order_keys(s_order, p, I.ts, I.lt, I.nsb, I.sx, I.sy, I.sz);
        }
        __syncthreads();
        sb_order_rank(s_order, I.nsb);
        __syncthreads();
        for (;;) {
            int sb = 0;
            if (lane == 0) sb = atomicAdd(&s_next_sb, 1);
            sb = __shfl_sync(0xffffffffu, sb, 0);
            if (sb >= I.nsb) break;
            eval_sub_block(A, S, I, sb_at(s_order, sb, I.nsb), s_rcnt, S.stage + wid * kStageWarpFloats,
                           S.ring + 2 * wid * kRing, ev);
        }
        done(I);
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kEvThreads, kEvCtas) k_bgki(EvArgs A) {
    extern __shared__ __align__(32) unsigned char smem_raw[];
    __shared__ int s_last;
    K3domEval ev;
    ev.tex = A.ktex;
    ev.nev = 0;
    run_items(A, smem_raw, ev, [&](const ItemConst& I) {
        if (!A.fuse_update) return;  // the cells are updated by k_k3dom_update_cells after this kernel
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) s_last = (atomicAdd(&A.tile_done[I.t], 1u) == I.n_items - 1) ? 1 : 0;
        __syncthreads();
        if (!s_last) return;
        __threadfence();
        const SceneDev& sd = A.bt.sc[I.sc];
        const DevParams& p = sd.p;
        const TileShape ts = I.ts;
        const double gdt = A.bt.fp[I.sc].gamma_dt;
        const int tx = I.lt % ts.ntx, ty = (I.lt / ts.ntx) % ts.nty, tz = I.lt / (ts.ntx * ts.nty);
        const int tile_cells = ts.tx * ts.ty * ts.tz;
        for (int li = threadIdx.x; li < tile_cells; li += kEvThreads) {
            const int lx = li % ts.tx, ly = (li / ts.tx) % ts.ty, lz = li / (ts.tx * ts.ty);
            const int ix = tx * ts.tx + lx, iy = ty * ts.ty + ly, iz = tz * ts.tz + lz;
            if (ix >= p.G || iy >= p.G || iz >= p.Gz) continue;
            const int c = I.coff + ix + p.G * iy + p.G * p.G * iz;
            // every chunk of the tile has added its share (fence + tile counter above); read
            // the totals from L2 and clear only what was written
            unsigned long long* ac = A.acc + 2 * (long)c;
            const long long fo = (long long)__ldcg(ac);
            const long long ff = (long long)__ldcg(ac + 1);
            if (fo) __stcg(ac, 0ull);
            if (ff) __stcg(ac + 1, 0ull);
            k3dom_cell_update(p, gdt, c, (double)fo * sd.fx_inv, (double)ff * sd.fx_inv, A.cs, A.cw,
                              A.first_frame != 0);
        }
        if (threadIdx.x == 0) A.tile_done[I.t] = 0;
    });
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ev.nev += __shfl_xor_sync(0xffffffffu, ev.nev, o);
    if (lane == 0 && ev.nev) atomicAdd(&A.status->kernel_evals, (unsigned long long)ev.nev);
}

// ================================================================ DS-PHD/MIB
struct DsMeas {
    float occ, free_m;
};

// The measurement masses of measurement_grid.cu:98-157 from the neighbour summary.
__device__ __forceinline__ DsMeas ds_meas_from(const DevParams& p, float acs, int nb, bool all_farther,
                                               float max_occ) {
    DsMeas m;
    if (nb == 0) {
        m.occ = 0.0f;
        m.free_m = 0.0f;
        return m;
    }
    float mo, mf;
    if (all_farther) {
        // pFree (:41-50): p_min + r / max_range * (p_max - p_min)
        const float r = sqrtf(acs);
        const float unc = __fadd_rn(0.15f, __fmul_rn(__fdiv_rn(r, p.max_range), __fsub_rn(1.0f, 0.15f)));
        if (max_occ > unc) {
            mo = max_occ;
            mf = 0.0f;
        } else {
            mo = 0.0f;
            mf = __fsub_rn(1.0f, unc);
        }
    } else {
        mo = max_occ > 0.5f ? max_occ : 0.0f;
        mf = 0.0f;
    }
    const float eps = 0.00001f;
    m.occ = fmaxf(eps, fminf(__fsub_rn(1.0f, eps), mo));
    m.free_m = fmaxf(eps, fminf(__fsub_rn(1.0f, eps), mf));
    return m;
}

// update_masses (src/dsphdmib/kernel/mass_update.cu:17-30) keeping its double promotions.
__device__ __forceinline__ void ds_update_masses(float mop, float mfp, DsMeas mc, float* occ, float* fr) {
    const float unknown_pred = (float)(1.0 - (double)mop - (double)mfp);
    const float meas_unknown = (float)(1.0 - (double)mc.free_m - (double)mc.occ);
    const float K = __fadd_rn(__fmul_rn(mfp, mc.occ), __fmul_rn(mop, mc.free_m));
    const float no = __fadd_rn(__fadd_rn(__fmul_rn(mop, meas_unknown), __fmul_rn(unknown_pred, mc.occ)),
                               __fmul_rn(mop, mc.occ));
    const float nf = __fadd_rn(__fadd_rn(__fmul_rn(mfp, meas_unknown), __fmul_rn(unknown_pred, mc.free_m)),
                               __fmul_rn(mfp, mc.free_m));
    const double den = 1.0 - (double)K;
    *occ = (float)((double)no / den);
    *fr = (float)((double)nf / den);
}

__device__ void ds_cell_update(const DevParams& p, int c, DsMeas mc, CellState cs, CellWork cw, bool first_frame) {
    cw.meas_occ[c] = mc.occ;
    cw.meas_free[c] = mc.free_m;
    if (first_frame) {
        cs.born_m[c] = mc.occ;  // copyMassesKernel (measurement_grid.cu:55-62)
        return;
    }
    const int start = cw.start[c];
    const bool has = start >= 0;
    const float free0 = cs.free_m[c];
    float occ_up, free_up, rho_b = 0.0f, mop = 0.0f, divisor = 0.0f;
    if (has) {
        mop = cw.sum_w[c];
        if (mop > 1.0f) {
            divisor = mop;  // normalize_weights (:37-44), applied in the reweight kernel
            mop = 1.0f;
        }
        const float mfp = fminf(__fmul_rn(0.9f, free0), __fsub_rn(1.0f, mop));
        ds_update_masses(mop, mfp, mc, &occ_up, &free_up);
        // separate_newborn_part (:32-35) with its double promotions
        const double om = 1.0 - (double)mop;
        rho_b = (float)(((double)__fmul_rn(occ_up, p.p_B) * om) / ((double)mop + (double)p.p_B * om));
    } else {
        const float m_occ = cs.occ_m[c];
        const float m_free = fminf(__fmul_rn(0.9f, free0), __fsub_rn(1.0f, m_occ));
        ds_update_masses(m_occ, m_free, mc, &occ_up, &free_up);
    }
    const float pers = __fsub_rn(occ_up, rho_b);
    cs.born_m[c] = rho_b;
    cs.pers_m[c] = pers;
    cs.free_m[c] = free_up;
    cs.occ_m[c] = occ_up;
    cs.pred_m[c] = mop;
    const float mu_UA = has ? calc_norm(mop, pers) : 0.0f;
    cw.factor[c] = mu_UA;
    cw.divisor[c] = divisor;
    float vx = 0.0f, vy = 0.0f, vz = 0.0f;
    if (has && pers > 0.0f) {
        float sx = cw.sum_wvx[c], sy = cw.sum_wvy[c], sz = cw.sum_wvz[c];
        if (divisor > 0.0f) {
            sx /= divisor;
            sy /= divisor;
            sz /= divisor;
        }
        vx = (mu_UA * sx) / pers;
        vy = (mu_UA * sy) / pers;
        vz = (mu_UA * sz) / pers;
    }
    cs.mvx[c] = vx;
    cs.mvy[c] = vy;
    cs.mvz[c] = vz;
}

// Neighbour test of measurement_grid.cu:88-99 in the reference's FP32 operation order.
__device__ __forceinline__ bool ds_is_neighbor(float x, float y, float z, float acs, float4 m, float wr2) {
    const float ip = __fadd_rn(__fadd_rn(__fmul_rn(x, m.x), __fmul_rn(y, m.y)), __fmul_rn(z, m.z));
    return ip > 0.0f && __fsub_rn(acs, __fdiv_rn(__fmul_rn(ip, ip), m.w)) < wr2;
}

// pOcc (measurement_grid.cu:28-39) from the squared distance between cell centre and point.
__device__ __forceinline__ float ds_r_sqr(float x, float y, float z, float4 m) {
    const float dx = __fsub_rn(x, m.x), dy = __fsub_rn(y, m.y), dz = __fsub_rn(z, m.z);
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}
__device__ __forceinline__ float ds_pocc(float r_sqr, float delta) {
    const float delta_sqr = __fmul_rn(delta, delta);
    return __fmul_rn(0.95f, expf(__fdiv_rn(__fmul_rn(-0.5f, r_sqr), delta_sqr)));
}

// The measurement grid by rays. A ray's half-line meets about 300 cells of a 256x256x32 grid, 4 of
// the 32 in a sub-block that it passes, so one lane per cell leaves most lanes idle; here one lane
// takes one ray of a work item and walks the cells around the half-line inside the item's tile,
// applies the reference's FP32 neighbour test to each and adds an accepted one to the cell's summary
// in shared memory with two atomics. The summary is order-free: pOcc falls with the distance (every
// operation of ds_pocc is monotone; expf was checked over all floats of [-110, 0]), so its maximum
// over the neighbours is pOcc of the smallest squared distance, kept as float bits (>= 0) by an
// integer minimum; beside it the number of neighbours and of those closer to the sensor than the
// cell. Only the reference's first-100 rule (measurement_grid.cu:86-97) depends on the input order,
// and only for cells with more than 100 neighbours. A tile's items hold its rays in input order, so
// the items before the hundredth neighbour count in full, and the one that holds it is walked again
// in order, by a warp, for that cell alone (k_ds_partial).
//   k_ds_rays     per item: summaries; a tile with one item writes its cells' totals, the others
//                 write per (item, cell) summaries; cells past 100 go to the worklist
//   k_ds_combine  cells of tiles with several items: the items in order up to the hundredth neighbour
//   k_ds_partial  the worklist
//   k_ds_update   the measurement-to-mass step and the Dempster update of every cell
// 256x256x32 voxels at 0.1 m, 120,000 rays: the lane-per-cell passes took 0.65 + 1.10 ms, these 0.18 +
// 0.04 + 0.07 + 0.05 ms; 200x200x25 at 0.2 m, 60,000 rays: 0.69 -> 0.20 ms. k_ds_rays is bound by
// instruction issue and by its waits at the items' ends. With the window of the lists at 2.05 cells
// (see ds_window): one ray per lane with the layers as a loop ran at 6 of 32 lanes (1.52 ms), one
// (ray, layer) per lane with plain loops over its cells 0.86 ms, with unrolled blocks 0.62 ms; CTAs of
// 128 or 64 threads wait less but leave longer tails (1.01x and 1.27x the time).
constexpr int kMaxTileCells = 16 * 16 * 8;
constexpr uint32_t kDsNone = 0xFFFFFFFFu;
constexpr uint32_t kDsCloser = 0x10000u;  // in a cell's counter: neighbours | closer ones << 16
static_assert(kDsSpareDiv * kChunk + 64 < 0x10000, "an item's count fits 16 bits");

// Per-cell results in the evidence accumulators' memory (4 words per cell).
struct DsCells {
    uint32_t *r2, *flags, *work_cell, *work_item;  // flags: 1 any neighbour, 2 one closer than the cell
    __device__ __forceinline__ DsCells(const EvArgs& A) {
        r2 = reinterpret_cast<uint32_t*>(A.acc);
        flags = r2 + A.bt.C;
        work_cell = flags + A.bt.C;
        work_item = work_cell + A.bt.C;
    }
};

struct DsTile {
    float2 c[3][16];  // cell-centre coordinate and its square, per axis
    int o[3], n[3];   // first cell and number of cells inside the grid
    uint32_t cf[kMaxTileCells], r2[kMaxTileCells];
};

// A ray's line through a tile, in layers along its axis A (x or y, whichever is larger; z for rays
// steeper than that): at layer i (cells from the tile's first one) it crosses the layer at
// B = pb + sb i, C = pc + sc i, and the cells of the layer within the window of the line form an
// ellipse with half-extents eb = R sqrt(1 + sb^2) and ec along B and C. (B, C) is (y, z), (x, z) or
// (x, y), so that the reference's sums over x, y, z are (A + B) + C, or (B + C) + A for axis z.
struct DsRay {
    float4 line;  // pb, sb, pc, sc
    float4 ext;   // eb, ec, 1 / |m|^2, axis
    float4 m;     // m, |m|^2
};
struct DsWarp {
    DsRay ray[32];
    uint16_t layer[32 * 16];  // lane of the ray | layer << 5
};

// Lays out the line of ray m and returns its range of layers (none: hi < lo). Distances are formed in
// cell-index space; R carries the slack of the reference's FP32 test and of this arithmetic. A
// neighbour needs a positive projection, which lies within 1.3 cells of its layer's crossing.
__device__ __forceinline__ int2 ds_line(const DsTile& S, const float a[3], float4 m, float R, DsRay* out) {
    const float il = rsqrtf(m.w);
    const float ux = m.x * il, uy = m.y * il, uz = m.z * il;
    const float hx = fabsf(ux), hy = fabsf(uy);
    const int ax = fabsf(uz) > fmaxf(hx, hy) ? 2 : (hx >= hy ? 0 : 1);
    const float uA = ax == 0 ? ux : (ax == 1 ? uy : uz), uB = ax == 0 ? uy : ux, uC = ax == 2 ? uy : uz;
    const int B = ax == 0 ? 1 : 0, C = ax == 2 ? 1 : 2;
    const float aA = sel3(a[0], a[1], a[2], ax), aB = sel3(a[0], a[1], a[2], B), aC = sel3(a[0], a[1], a[2], C);
    const float iu = 1.0f / uA, sb = uB * iu, sc = uC * iu;
    const float eb = R * sqrtf(fmaf(sb, sb, 1.0f)), ec = R * sqrtf(fmaf(sc, sc, 1.0f));
    const float a0 = (float)S.o[ax] - aA;
    const float pb = aB - (float)S.o[B] + sb * a0, pc = aC - (float)S.o[C] + sc * a0;
    float lo = 0.0f, hi = (float)(S.n[ax] - 1);
    if (uA > 0.0f) lo = fmaxf(lo, -a0 - 2.0f); else hi = fminf(hi, -a0 + 2.0f);
    // layers where the line is inside the tile's B and C ranges
    if (fabsf(sb) > 1e-3f) {
        const float is = 1.0f / sb, t0 = (-eb - pb) * is, t1 = ((float)(S.n[B] - 1) + eb - pb) * is;
        lo = fmaxf(lo, fminf(t0, t1) - 0.05f);
        hi = fminf(hi, fmaxf(t0, t1) + 0.05f);
    }
    if (fabsf(sc) > 1e-3f) {
        const float is = 1.0f / sc, t0 = (-ec - pc) * is, t1 = ((float)(S.n[C] - 1) + ec - pc) * is;
        lo = fmaxf(lo, fminf(t0, t1) - 0.05f);
        hi = fminf(hi, fmaxf(t0, t1) + 0.05f);
    }
    out->line = make_float4(pb, sb, pc, sc);
    out->ext = make_float4(eb, ec, 1.0f / m.w, __int_as_float(ax));
    out->m = m;
    return make_int2((int)ceilf(lo), (int)floorf(hi));
}

// The candidate cells of one layer of one ray. STEEP: axis z.
template <bool STEEP>
__device__ __forceinline__ void ds_layer(DsTile& S, const TileShape& ts, const DsRay& r, int ax, int i, float wr2) {
    const float4 ln = r.line, ex = r.ext, m = r.m;
    const int B = STEEP ? 0 : 1 - ax, C = STEEP ? 1 : 2;
    const float qb = fmaf(ln.y, (float)i, ln.x), qc = fmaf(ln.w, (float)i, ln.z);
    const int b0 = max((int)ceilf(qb - ex.x), 0), b1 = min((int)floorf(qb + ex.x), S.n[B] - 1);
    const int c0 = max((int)ceilf(qc - ex.y), 0), c1 = min((int)floorf(qc + ex.y), S.n[C] - 1);
    const int stA = STEEP ? ts.tx * ts.ty : (ax == 0 ? 1 : ts.tx), stB = STEEP ? 1 : (ax == 0 ? ts.tx : 1);
    const int stC = STEEP ? ts.tx : ts.tx * ts.ty;
    const float mA = STEEP ? m.z : (ax == 0 ? m.x : m.y), mB = STEEP ? m.x : (ax == 0 ? m.y : m.x);
    const float mC = STEEP ? m.y : m.z;
    const float2 va = S.c[STEEP ? 2 : ax][i];
    const float pa = __fmul_rn(va.x, mA), da = __fsub_rn(va.x, mA), dda = __fmul_rn(da, da);
    // the layer's cells in blocks of 3 x 2 (nearly always one: the window is 1.73 cells wide across the
    // ray and C slopes little for LiDAR rays), unrolled so that the six tests overlap
    for (int cb = c0; cb <= c1; cb += 2) {
        float2 vc[2];
        float pc[2], ddc[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            vc[k] = S.c[C][min(cb + k, 15)];
            pc[k] = __fmul_rn(vc[k].x, mC);
            const float d = __fsub_rn(vc[k].x, mC);
            ddc[k] = __fmul_rn(d, d);
        }
        for (int bb = b0; bb <= b1; bb += 3) {
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                if (bb + j > b1) continue;
                const float2 vb = S.c[B][bb + j];
                const float pb = __fmul_rn(vb.x, mB), db = __fsub_rn(vb.x, mB), ddb = __fmul_rn(db, db);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    // the test of measurement_grid.cu:88-99 (ds_is_neighbor), sums in x, y, z order; its
                    // IEEE division is taken only where the reciprocal's result is within the rounding
                    // of the limit
                    const float ip = STEEP ? __fadd_rn(__fadd_rn(pb, pc[k]), pa) : __fadd_rn(__fadd_rn(pa, pb), pc[k]);
                    const float acs = STEEP ? __fadd_rn(__fadd_rn(vb.y, vc[k].y), va.y)
                                            : __fadd_rn(__fadd_rn(va.y, vb.y), vc[k].y);
                    const float q = __fmul_rn(ip, ip);
                    const float over = fmaf(-q, ex.z, acs) - wr2;
                    bool in = over < 0.0f;
                    if (fabsf(over) <= 3e-7f * acs) in = __fsub_rn(acs, __fdiv_rn(q, m.w)) < wr2;
                    if (in && ip > 0.0f && cb + k <= c1) {
                        const float r2 = STEEP ? __fadd_rn(__fadd_rn(ddb, ddc[k]), dda)  // ds_r_sqr
                                               : __fadd_rn(__fadd_rn(dda, ddb), ddc[k]);
                        const int li = i * stA + (bb + j) * stB + (cb + k) * stC;
                        atomicAdd(&S.cf[li], acs > m.w ? 1u + kDsCloser : 1u);
                        atomicMin(&S.r2[li], __float_as_uint(r2));
                    }
                }
            }
        }
    }
}

// Whether a ray of ds_extreme takes the cells of the sub-block with centroid (qx, qy, qz): the box
// bound (box_reaches) on the distance from its half-line, in the FP32 arithmetic whose direction is
// zero for an infinite |m|^2 (then the half-line is the sensor). It does not depend on the tiling.
__device__ __forceinline__ bool ds_reaches_sub_block(float qx, float qy, float qz, const float4& m, float hres,
                                                     float rls2) {
    const float len = sqrtf(m.w), inv = len > 0.0f ? 1.0f / len : 0.0f;
    const float ux = m.x * inv, uy = m.y * inv, uz = m.z * inv;
    const float t = fmaxf(qx * ux + qy * uy + qz * uz, 0.0f);
    const float Dx = qx - t * ux, Dy = qy - t * uy, Dz = qz - t * uz;
    return box_reaches(Dx, Dy, Dz, Dx * Dx + Dy * Dy + Dz * Dz, hres, rls2);
}

// A ray of ds_extreme in the tile, by a warp: the reference's test on every cell of the sub-blocks near
// its half-line. Such rays are too rare to be worth more (a sensor's far-away marker for no return).
__device__ __noinline__ void ds_extreme_ray(DsTile& S, const ItemConst& I, const float4& mr, float wr2) {
    const TileShape& ts = I.ts;
    const float4 m = mr;
    const float hres = 0.5f * I.res, rls2 = I.rls2;
    const int lane = threadIdx.x & 31;
    for (int s0 = 0; s0 < I.nsb; s0 += 32) {
        const int sb = s0 + lane;
        bool hit = false;
        if (sb < I.nsb) {
            const SbCell b = sb_cell(ts, 0, sb);
            hit = ds_reaches_sub_block(S.c[0][b.x + 2].x - hres, S.c[1][b.y + 2].x - hres, S.c[2][b.z + 1].x - hres, m,
                                       hres, rls2);
        }
        for (unsigned left = __ballot_sync(0xffffffffu, hit); left; left &= left - 1u) {
            const SbCell b = sb_cell(ts, 0, s0 + __ffs(left) - 1);
            const int x = b.x + (lane & 3), y = b.y + ((lane >> 2) & 3), z = b.z + (lane >> 4);
            if (x >= S.n[0] || y >= S.n[1] || z >= S.n[2]) continue;
            const float2 cx = S.c[0][x], cy = S.c[1][y], cz = S.c[2][z];
            const float acs = __fadd_rn(__fadd_rn(cx.y, cy.y), cz.y);
            if (!ds_is_neighbor(cx.x, cy.x, cz.x, acs, m, wr2)) continue;
            const int li = x + ts.tx * (y + ts.ty * z);
            atomicAdd(&S.cf[li], acs > m.w ? 1u + kDsCloser : 1u);
            atomicMin(&S.r2[li], __float_as_uint(ds_r_sqr(cx.x, cy.x, cz.x, m)));
        }
    }
}

__global__ void __launch_bounds__(kEvThreads) k_ds_rays(EvArgs A) {
    __shared__ ItemConst I;
    __shared__ DsTile S;
    __shared__ DsWarp s_warp[kEvWarps];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const Batch& bt = A.bt;
    const DsCells D(A);
    const uint32_t total_items = A.item_off[bt.T];
    const int chunk = item_rays(A.total[2], A.chunk, 0, A.ds_spare);
    unsigned nev = 0;  // neighbours accepted in the cells this thread finished (the roofline's work count)
    for (;;) {
        if (wid == 0) fetch_item(A, total_items, chunk, &I);
        __syncthreads();
        if (!I.live) break;
        const TileShape ts = I.ts;
        const int tc[3] = {I.lt % ts.ntx, (I.lt / ts.ntx) % ts.nty, I.lt / (ts.ntx * ts.nty)};
        const int tile_cells = ts.tx * ts.ty * ts.tz;
        for (int i = threadIdx.x; i < tile_cells; i += kEvThreads) {
            S.cf[i] = 0u;
            S.r2[i] = kDsNone;
        }
        if (threadIdx.x < 16) {
            DevParams p;  // the fields centre_xyz reads
            p.G = I.G; p.Gz = I.Gz; p.res = I.res;
            const int k = threadIdx.x;
            float x, y, z;
            centre_xyz(tc[0] * ts.tx + k, tc[1] * ts.ty + k, tc[2] * ts.tz + k, p, I.sx, I.sy, I.sz, &x, &y, &z);
            S.c[0][k] = make_float2(x, __fmul_rn(x, x));
            S.c[1][k] = make_float2(y, __fmul_rn(y, y));
            S.c[2][k] = make_float2(z, __fmul_rn(z, z));
            if (k == 0) {
                S.o[0] = tc[0] * ts.tx; S.o[1] = tc[1] * ts.ty; S.o[2] = tc[2] * ts.tz;
                S.n[0] = min(ts.tx, I.G - S.o[0]); S.n[1] = min(ts.ty, I.G - S.o[1]);
                S.n[2] = min(ts.tz, I.Gz - S.o[2]);
            }
        }
        __syncthreads();
        {
            const float wr2 = bt.sc[I.sc].wr2;
            // the window at the tile's farthest cell, and 0.01 cells for the walk's own arithmetic
            float far2 = 0.0f;
#pragma unroll
            for (int k = 0; k < 3; ++k) far2 += fmaxf(S.c[k][0].y, S.c[k][S.n[k] - 1].y);
            const float R = ds_window(wr2, far2, I.res) + 0.01f;
            const float hg = (float)I.G / 2.0f, hz = (float)I.Gz / 2.0f;
            const float a[3] = {I.sx / I.res + hg - 0.5f, I.sy / I.res + hg - 0.5f, I.sz / I.res + hz - 0.5f};
            DsWarp& W = s_warp[wid];
            for (int g = wid * 32; g < I.nr; g += kEvThreads) {
                // one ray per lane: its line and layers; then one (ray, layer) per lane
                int2 ly = make_int2(0, -1);
                bool extreme = false;
                if (g + lane < I.nr) {
                    uint32_t rid = A.evals[I.e0 + g + lane];
                    if (rid >= (uint32_t)bt.N) rid = 0;  // defensive: never read past the ray arrays
                    const float4 m = A.ray_a[rid];
                    extreme = m.w > 0.0f && ds_extreme(m.w);
                    if (extreme) W.ray[lane].m = m;
                    else if (m.w > 0.0f) ly = ds_line(S, a, m, R, &W.ray[lane]);
                }
                const int n = max(ly.y - ly.x + 1, 0);
                int end = n;  // inclusive prefix over the lanes
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, end, o);
                    if (lane >= o) end += v;
                }
                const int total = __shfl_sync(0xffffffffu, end, 31);
                for (int i = 0; i < n; ++i) W.layer[end - n + i] = (uint16_t)(lane | (ly.x + i) << 5);
                __syncwarp();
                for (int k = lane; k < total; k += 32) {
                    const int e = W.layer[k];
                    const DsRay& r = W.ray[e & 31];
                    const int ax = __float_as_int(r.ext.w);
                    if (ax == 2) ds_layer<true>(S, ts, r, 2, e >> 5, wr2);
                    else ds_layer<false>(S, ts, r, ax, e >> 5, wr2);
                }
                for (unsigned left = __ballot_sync(0xffffffffu, extreme); left; left &= left - 1u)
                    ds_extreme_ray(S, I, W.ray[__ffs(left) - 1].m, wr2);
                __syncwarp();
            }
        }
        __syncthreads();
        const bool single = I.n_items == 1;
        const long base = (long)I.item * A.ds_stride;
        for (int i = threadIdx.x; i < tile_cells; i += kEvThreads) {
            const uint32_t cf = S.cf[i], cnt = cf & 0xFFFFu;
            if (!single) {
                if (base + i < A.ds_capacity) {
                    A.ds_counts[base + i] = (uint8_t)(min(cnt, kDsMaxNeighbors + 1u) | (cf >= kDsCloser ? 0x80u : 0u));
                    if (cnt) A.ds_r2[base + i] = S.r2[i];
                }
                continue;
            }
            if (!cnt) continue;
            const int lx = i % ts.tx, ly = (i / ts.tx) % ts.ty, lz = i / (ts.tx * ts.ty);
            const int c = I.coff + (S.o[0] + lx) + I.G * (S.o[1] + ly) + I.G * I.G * (S.o[2] + lz);
            nev += min(cnt, kDsMaxNeighbors);
            if (cnt <= kDsMaxNeighbors) {
                D.r2[c] = S.r2[i];
                D.flags[c] = 1u | (cf >= kDsCloser ? 2u : 0u);
            } else {
                const uint32_t w = atomicAdd(&A.status->work_counter2, 1u);
                D.work_cell[w] = (uint32_t)c;
                D.work_item[w] = I.item;
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nev += __shfl_xor_sync(0xffffffffu, nev, o);
    if (lane == 0 && nev) atomicAdd(&A.status->kernel_evals, (unsigned long long)nev);
}

// The tiles with several items, a cell per thread and kEvThreads cells per CTA.
__global__ void __launch_bounds__(kEvThreads) k_ds_combine(EvArgs A, int ctas_per_tile) {
    const Batch& bt = A.bt;
    const DsCells D(A);
    const int t = blockIdx.x / ctas_per_tile, i = (blockIdx.x % ctas_per_tile) * kEvThreads + threadIdx.x;
    const uint32_t first = A.item_off[t], n_items = A.item_off[t + 1] - first;
    if (n_items <= 1) return;
    const int sc = scene_of(bt.off->tile, bt.S, t);
    const SceneDev& sd = bt.sc[sc];
    const TileShape ts = sd.ts;
    const int lt = t - bt.off->tile[sc], G = sd.p.G, Gz = sd.p.Gz;
    const int ix = lt % ts.ntx * ts.tx + i % ts.tx, iy = (lt / ts.ntx) % ts.nty * ts.ty + (i / ts.tx) % ts.ty;
    const int iz = lt / (ts.ntx * ts.nty) * ts.tz + i / (ts.tx * ts.ty);
    unsigned nev = 0;
    if (i < ts.tx * ts.ty * ts.tz && ix < G && iy < G && iz < Gz) {
        const int c = bt.off->cell[sc] + ix + G * iy + G * G * iz;
        uint32_t pre = 0, r2 = kDsNone, closer = 0;
        constexpr uint32_t kAhead = 8;  // counts read at once: a tile next to the sensor has many items
        bool open = true;
        for (uint32_t k0 = 0; k0 < n_items && open; k0 += kAhead) {
            uint32_t cf[kAhead];
#pragma unroll
            for (uint32_t j = 0; j < kAhead; ++j) {
                const long e = (long)(first + k0 + j) * A.ds_stride + i;
                cf[j] = k0 + j < n_items && e < A.ds_capacity ? A.ds_counts[e] : 0u;
            }
#pragma unroll
            for (uint32_t j = 0; j < kAhead; ++j) {
                const uint32_t cnt = cf[j] & 0x7Fu;
                if (!cnt || !open) continue;
                if (pre + cnt > kDsMaxNeighbors) {
                    open = false;
                    if (pre < kDsMaxNeighbors) {  // the item that holds the hundredth neighbour
                        const uint32_t w = atomicAdd(&A.status->work_counter2, 1u);
                        D.work_cell[w] = (uint32_t)c;
                        D.work_item[w] = first + k0 + j;
                        nev += kDsMaxNeighbors - pre;
                    }
                    continue;
                }
                pre += cnt;
                closer |= cf[j] & 0x80u;
                r2 = min(r2, A.ds_r2[(long)(first + k0 + j) * A.ds_stride + i]);
            }
        }
        if (pre) {
            nev += pre;
            D.r2[c] = r2;
            D.flags[c] = 1u | (closer ? 2u : 0u);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nev += __shfl_xor_sync(0xffffffffu, nev, o);
    if ((threadIdx.x & 31) == 0 && nev) atomicAdd(&A.status->kernel_evals, (unsigned long long)nev);
}

// A warp per worklist entry: the first (100 - neighbours of the tile's earlier items) neighbours of
// the cell among the item's rays, in list order, added to the cell's result.
__global__ void __launch_bounds__(kEvThreads) k_ds_partial(EvArgs A) {
    const Batch& bt = A.bt;
    const DsCells D(A);
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const uint32_t n = A.status->work_counter2;
    const uint32_t chunk = (uint32_t)item_rays(A.total[2], A.chunk, 0, A.ds_spare);
    for (uint32_t w = blockIdx.x * kEvWarps + (threadIdx.x >> 5); w < n; w += gridDim.x * kEvWarps) {
        const int c = (int)D.work_cell[w];
        const uint32_t item = D.work_item[w];
        const int t = warp_find_tile(A.item_off, bt.T, item);
        const int sc = scene_of(bt.off->cell, bt.S, c);
        const SceneDev& sd = bt.sc[sc];
        const FrameParams& fp = bt.fp[sc];
        const TileShape ts = sd.ts;
        int ix, iy, iz;
        cell_xyz(c - bt.off->cell[sc], sd.p.G, &ix, &iy, &iz);
        const int li = ix % ts.tx + ts.tx * (iy % ts.ty + ts.ty * (iz % ts.tz));
        const uint32_t first = A.item_off[t];
        int quota = (int)kDsMaxNeighbors;
        for (uint32_t k = first; k < item; k += 32) {
            const long e = (long)(k + lane) * A.ds_stride + li;
            const int cnt = k + lane < item && e < A.ds_capacity ? A.ds_counts[e] & 0x7F : 0;
            quota -= (int)__reduce_add_sync(0xffffffffu, (unsigned)cnt);
        }
        float x, y, z;
        centre_xyz(ix, iy, iz, sd.p, fp.sensor_x, fp.sensor_y, fp.sensor_z, &x, &y, &z);
        const float acs = __fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z));
        const uint32_t e0 = A.tile_start[t] + (item - first) * chunk;
        const uint32_t e1 = min(A.tile_start[t + 1], e0 + chunk);
        const float hres = 0.5f * sd.p.res;
        float qx, qy, qz;  // centroid of the cell's sub-block
        centre_xyz((ix & ~3) + 2, (iy & ~3) + 2, (iz & ~1) + 1, sd.p, fp.sensor_x, fp.sensor_y, fp.sensor_z, &qx, &qy,
                   &qz);
        qx -= hres; qy -= hres; qz -= hres;
        uint32_t r2 = kDsNone, closer = 0;
        for (uint32_t e = e0; e < e1 && quota > 0; e += 32) {
            bool in = false;
            float4 m = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (e + lane < e1) {
                uint32_t rid = A.evals[e + lane];
                if (rid >= (uint32_t)bt.N) rid = 0;
                m = A.ray_a[rid];
                in = ds_is_neighbor(x, y, z, acs, m, sd.wr2) &&
                     (!ds_extreme(m.w) || ds_reaches_sub_block(qx, qy, qz, m, hres, sd.cull_ls2));
            }
            const unsigned mask = __ballot_sync(0xffffffffu, in);
            if (in && __popc(mask & below) < quota) {
                r2 = min(r2, __float_as_uint(ds_r_sqr(x, y, z, m)));
                if (acs > m.w) closer = 2u;
            }
            quota -= __popc(mask);
        }
        r2 = __reduce_min_sync(0xffffffffu, r2);
        closer = __reduce_or_sync(0xffffffffu, closer);
        if (lane == 0) {
            const uint32_t f = D.flags[c];
            D.r2[c] = (f & 1u) ? min(D.r2[c], r2) : r2;
            D.flags[c] = f | 1u | closer;
        }
    }
}

__global__ void __launch_bounds__(kBlock) k_ds_update(EvArgs A) {
    const Batch& bt = A.bt;
    const DsCells D(A);
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < bt.C; c += gridDim.x * blockDim.x) {
        const int sc = scene_of(bt.off->cell, bt.S, c);
        const SceneDev& sd = bt.sc[sc];
        const FrameParams& fp = bt.fp[sc];
        const uint32_t f = D.flags[c];
        float acs = 0.0f, occ = 0.0f;
        if (f) {
            D.flags[c] = 0u;
            int ix, iy, iz;
            cell_xyz(c - bt.off->cell[sc], sd.p.G, &ix, &iy, &iz);
            float x, y, z;
            centre_xyz(ix, iy, iz, sd.p, fp.sensor_x, fp.sensor_y, fp.sensor_z, &x, &y, &z);
            acs = __fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z));
            occ = ds_pocc(__uint_as_float(D.r2[c]), sd.p.meas_occ_stddev);
        }
        const DsMeas mc = ds_meas_from(sd.p, acs, (f & 1u) ? 1 : 0, (f & 2u) == 0, occ);
        ds_cell_update(sd.p, c, mc, A.cs, A.cw, A.first_frame != 0);
    }
}

// ================================================================ launchers
static EvArgs make_args(const Batch& bt, RayBuffers& rb, CellState cs, CellWork cw, bool first_frame,
                        DevStatus* status) {
    EvArgs A;
    A.bt = bt;
    A.item_off = rb.item_off;
    A.tile_start = rb.tile_start;
    A.evals = rb.evals2;
    A.ray_a = rb.ray_a;
    A.ray_c = rb.ray_c;
    A.total = rb.total;
    A.item_slots = rb.item_slots;
    A.ds_spare = rb.ds_spare;
    A.tile_done = rb.tile_done;
    A.acc = rb.acc;
    A.ds_r2 = rb.ds_r2;
    A.ds_counts = rb.ds_counts;
    A.ds_capacity = rb.ds_capacity;
    A.ds_stride = rb.ds_stride;
    A.cs = cs;
    A.cw = cw;
    A.status = status;
    A.first_frame = first_frame ? 1 : 0;
    A.chunk = rb.chunk;
    A.fuse_update = 1;
    A.ktex = rb.ktex;
    return A;
}

// ================================================================ calibration sums
// For the differentiable update: per cell and frame, the sums of the unit-amplitude sparse
// kernel f(d/ls) over the occupied and free pairs, and of d f(d/ls) / d ls (times ls, i.e.
// -x f'(x)), from the same tiles, culls and pair geometry as k_bgki. Both are summed exactly
// in fixed point (units of 2^-40), so the loss and its gradient are deterministic. No per-pair
// value is stored: the derivative is formed in the same pass as the value.
//
// f(x) = max(0, (2 + cos 2 pi x)(1 - x) / 3 + sin(2 pi x) / (2 * 3.141592)), mass_update.cu:24-26.
static double unit_kernel(double x) {
    const double v = (2.0 + std::cos(M_PI * 2.0 * x)) * (1.0 - x) / 3.0 + std::sin(M_PI * 2.0 * x) / (2.0 * 3.141592);
    return v > 0.0 ? v : 0.0;
}
// -x f'(x) where f > 0 (0 where the clamp is active)
static double unit_kernel_dls(double x) {
    const double v = (2.0 + std::cos(M_PI * 2.0 * x)) * (1.0 - x) / 3.0 + std::sin(M_PI * 2.0 * x) / (2.0 * 3.141592);
    if (!(v > 0.0)) return 0.0;
    const double fp = (-2.0 * M_PI * std::sin(M_PI * 2.0 * x) * (1.0 - x) - (2.0 + std::cos(M_PI * 2.0 * x))) / 3.0 +
                      2.0 * M_PI * std::cos(M_PI * 2.0 * x) / (2.0 * 3.141592);
    return -x * fp;
}

static void build_table(double (*fn)(double), double scale, float4* out) {
    for (int i = 0; i < kKernelTab; ++i) {
        double y[4];
        for (int j = 0; j < 4; ++j) y[j] = scale * fn(std::sqrt(std::min(1.0, (i + j / 3.0) / kKernelTab)));
        const double c0 = y[0];
        const double c1 = -5.5 * y[0] + 9.0 * y[1] - 4.5 * y[2] + y[3];
        const double c2 = 9.0 * y[0] - 22.5 * y[1] + 18.0 * y[2] - 4.5 * y[3];
        const double c3 = -4.5 * y[0] + 13.5 * y[1] - 13.5 * y[2] + 4.5 * y[3];
        out[i] = make_float4((float)c0, (float)c1, (float)c2, (float)c3);
    }
    out[kKernelTab] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

void build_calib_tables(float4* f_tab, float4* dls_tab) {
    build_table(unit_kernel, 1.0, f_tab);
    build_table(unit_kernel_dls, 1.0, dls_tab);
}

// The calibration's values: f from its table through the texture path, -x f' from one in shared
// memory, two sums per evidence kind. f is clamped at 0 by FMA.SAT, -x f' lies in [-3e-7, 0.78].
// The kernel is bound by these gathers, and the two paths run side by side: gradient step at
// 256x256x32 voxels with two 120,000-ray frames, 3.75 ms with both tables in shared memory, 3.96 ms
// with both through the texture path, 3.50 ms with one in each.
static_assert(kCalibShift == kFxShift, "units of the calibration sums");

struct CalibEval {
    cudaTextureObject_t tex;  // f
    const float4* htab;       // [kKernelTabEntries] -x f'
    unsigned long long* acc4;
    FxSum fo[4], ff[4], ho[4], hf[4], occ_f, occ_h;
    int n_occ, n_free;
    __device__ __forceinline__ void begin(const ItemConst&) {
#pragma unroll
        for (int i = 0; i < 4; ++i) ff[i] = hf[i] = FxSum{0u, 0u};
        occ_f = occ_h = FxSum{0u, 0u};
        n_occ = n_free = 0;
    }
    __device__ __forceinline__ void begin_occ() {
#pragma unroll
        for (int i = 0; i < 4; ++i) fo[i] = ho[i] = FxSum{0u, 0u};
    }
    __device__ __forceinline__ void end_occ(int steps) {
        const FxSum f = quarter_merge(fo), h = quarter_merge(ho);
        occ_f.hi += f.hi;
        occ_f.lo += f.lo;
        occ_h.hi += h.hi;
        occ_h.lo += h.lo;
        n_occ += steps;
    }
    __device__ __forceinline__ void value(const TabPos& q, float* f, float* h) {
        const float4 c = tex1Dfetch<float4>(tex, q.i), d = htab[q.i];
        *f = __saturatef(fmaf(q.f, fmaf(q.f, fmaf(q.f, c.w, c.z), c.y), c.x));
        *h = fmaf(q.f, fmaf(q.f, fmaf(q.f, d.w, d.z), d.y), d.x);
    }
    __device__ __forceinline__ void pair(const TabPos2& q, bool a, bool b, FxSum& f, FxSum& h) {
        float fa = 0.0f, fb = 0.0f, ha = 0.0f, hb = 0.0f;
        if (a) value(q.a, &fa, &ha);
        if (b) value(q.b, &fb, &hb);
        f.add(F2::of(fa, fb));
        h.add(F2::of(ha, hb));
    }
    __device__ __forceinline__ void occ(int i, const TabPos2& q, bool a, bool b) { pair(q, a, b, fo[i], ho[i]); }
    __device__ __forceinline__ void free(int i, const TabPos2& q, bool a, bool b) { pair(q, a, b, ff[i], hf[i]); }
    __device__ __forceinline__ void end(const EvArgs&, long c, bool in) {
        const FxSum sff = quarter_merge(ff), shf = quarter_merge(hf);
        if (!in) return;
        unsigned long long* ac = acc4 + 4 * c;
        const uint32_t no = 8u * n_occ, nf = 8u * n_free;
        const long long v[4] = {occ_f.total(no), sff.total(nf), occ_h.total_signed(no), shf.total_signed(nf)};
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (v[i]) atomicAdd(ac + i, (unsigned long long)v[i]);
    }
};

constexpr size_t kCalibTabBytes = (sizeof(float4) * kKernelTabEntries + 31) & ~(size_t)31;

inline size_t calib_smem_bytes(int chunk) { return kCalibTabBytes + bgki_smem_bytes(chunk); }

// acc4: 4 signed 64-bit sums per cell (f occ, f free, -x f' occ, -x f' free), in units. Same
// tiles, culls and pair geometry as k_bgki; each value is rounded once to an integer number of
// units (round to nearest even).
__global__ void __launch_bounds__(kEvThreads, kEvCtas) k_bgki_sums(EvArgs A, const float4* __restrict__ htab,
                                                               unsigned long long* __restrict__ acc4) {
    extern __shared__ __align__(32) unsigned char smem_raw[];
    float4* tab = reinterpret_cast<float4*>(smem_raw);  // used after run_items' first barrier
    for (int i = threadIdx.x; i < kKernelTabEntries; i += kEvThreads) tab[i] = htab[i];
    CalibEval ev;
    ev.tex = A.ktex;
    ev.htab = tab;
    ev.acc4 = acc4;
    run_items(A, smem_raw + kCalibTabBytes, ev, [](const ItemConst&) {});
}

cudaError_t launch_bgki_sums(const Batch& bt, RayBuffers& rb, const float4* dls_tab, unsigned long long* acc4,
                             DevStatus* status, int num_sms, cudaStream_t st) {
    if (rb.chunk < 32 || rb.chunk > kCalibChunk) return cudaErrorInvalidValue;
    EvArgs A = make_args(bt, rb, CellState{}, CellWork{}, false, status);
    const size_t sm = calib_smem_bytes(rb.chunk);
    int per_sm = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bgki_sums, kEvThreads, sm);
    ++g_launches;
    k_bgki_sums<<<num_sms * std::max(1, per_sm), kEvThreads, sm, st>>>(A, dls_tab, acc4);
    return cudaGetLastError();
}

// The K3DOM evidence launch is persistent: one CTA per resident slot.
struct BgkiLaunch {
    int blocks;
    size_t smem;
};

static BgkiLaunch bgki_launch(int chunk) {
    int dev = 0, sms = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    BgkiLaunch L;
    L.smem = bgki_smem_bytes(chunk);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_bgki, kEvThreads, L.smem);
    L.blocks = sms * std::max(1, per_sm);
    return L;
}

int evidence_slots(int num_sms) { return num_sms * kEvCtas; }

int k3dom_evidence_blocks(int chunk) { return bgki_launch(chunk).blocks; }

cudaError_t launch_k3dom_evidence(const Batch& bt, RayBuffers& rb, CellState cs, CellWork cw, bool first_frame,
                                  DevStatus* status, cudaStream_t st, bool fuse_update) {
    if (rb.chunk < 32 || rb.chunk > kChunk) return cudaErrorInvalidValue;
    EvArgs A = make_args(bt, rb, cs, cw, first_frame, status);
    A.fuse_update = fuse_update ? 1 : 0;
    const BgkiLaunch L = bgki_launch(rb.chunk);
    ++g_launches;
    k_bgki<<<L.blocks, kEvThreads, L.smem, st>>>(A);
    return cudaGetLastError();
}

// The cell update of k_bgki's tile tails as a pass of its own over every cell: a steady frame
// accumulates the evidence beside prediction and assignment (the evidence needs only the ray
// lists) and updates the cells once the particles' per-cell sums are in. Each cell's two
// fixed-point sums are read and cleared, then k3dom_cell_update runs as in the tail: same inputs,
// same bits.
__global__ void __launch_bounds__(kBlock) k_k3dom_update_cells(EvArgs A) {
    const Batch& bt = A.bt;
    ulonglong2* acc = reinterpret_cast<ulonglong2*>(A.acc);  // (occupied, free) per cell
    for (long c = (long)blockIdx.x * blockDim.x + threadIdx.x; c < bt.C; c += (long)gridDim.x * blockDim.x) {
        const int sc = scene_of(bt.off->cell, bt.S, (int)c);
        const SceneDev& sd = bt.sc[sc];
        const ulonglong2 v = acc[c];
        if (v.x || v.y) acc[c] = make_ulonglong2(0ull, 0ull);
        k3dom_cell_update(sd.p, bt.fp[sc].gamma_dt, (int)c, (double)(long long)v.x * sd.fx_inv,
                          (double)(long long)v.y * sd.fx_inv, A.cs, A.cw, A.first_frame != 0);
    }
}

// The same pass with each CTA's inputs brought into shared memory by bulk copies: the pass is
// latency bound on its per-cell reads, and one cp.async.bulk per input array (8 arrays of 1,024
// cells and the fixed-point sums, 48 KB per CTA, completed on one mbarrier) puts all of a CTA's
// bytes in flight at once without holding them in registers. Each copy is a plain one-CTA copy of
// this GPU's own memory. Every array base is 16-byte aligned (checked by the
// launcher) and a full tile starts at a multiple of 4 KB, as the copies require; the last, partial
// tile reads its cells directly. The wait is bounded: when it runs out the CTA records
// copy_timeout, waits (bounded again) for its copies to land, and skips its cells.
// Maps below kUcBulk cells take the plain kernel: a CTA per 1,024 cells leaves too few of them to
// hide the copies' latency (8k cells 10.1 -> 4.0 us, 120k 11.3 -> 6.1, 1.2M 30.0 -> 23.7, 1M equal;
// 2.1M cells are 65 us that way and 56 by copies).
constexpr int kUcCells = 1024;
constexpr int kUcThreads = 256;
constexpr int kUcBulk = 1500000;
constexpr uint32_t kUcMaxPolls = 1u << 22;
constexpr size_t kUcSmem = 8 * sizeof(float) * kUcCells + sizeof(ulonglong2) * kUcCells;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :
                 : "r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}

// Polls the barrier's phase 0 at most max_polls times; true once it has completed.
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t max_polls) {
    for (uint32_t it = 0; it < max_polls; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(smem_addr(bar))
            : "memory");
        if (done) return true;
    }
    return false;
}

__global__ void __launch_bounds__(kUcThreads) k_k3dom_update_cells_bulk(EvArgs A) {
    extern __shared__ __align__(16) unsigned char uc_smem[];
    __shared__ __align__(8) uint64_t bar;
    const Batch& bt = A.bt;
    ulonglong2* acc = reinterpret_cast<ulonglong2*>(A.acc);
    const long c0 = (long)blockIdx.x * kUcCells;
    const int n = (int)min((long)kUcCells, (long)bt.C - c0);
    const bool first = A.first_frame != 0;
    if (n < kUcCells) {  // the partial last tile: direct reads (the same update)
        for (int i = threadIdx.x; i < n; i += kUcThreads) {
            const int c = (int)(c0 + i);
            const int sc = scene_of(bt.off->cell, bt.S, c);
            const SceneDev& sd = bt.sc[sc];
            const ulonglong2 v = acc[c];
            if (v.x || v.y) acc[c] = make_ulonglong2(0ull, 0ull);
            k3dom_cell_update(sd.p, bt.fp[sc].gamma_dt, c, (double)(long long)v.x * sd.fx_inv,
                              (double)(long long)v.y * sd.fx_inv, A.cs, A.cw, first);
        }
        return;
    }
    float* s_f = reinterpret_cast<float*>(uc_smem);
    float* s_s = s_f + kUcCells;
    float* s_d = s_s + kUcCells;
    int* s_start = reinterpret_cast<int*>(s_d + kUcCells);
    float* s_w = reinterpret_cast<float*>(s_start + kUcCells);
    float* s_vx = s_w + kUcCells;
    float* s_vy = s_vx + kUcCells;
    float* s_vz = s_vy + kUcCells;
    ulonglong2* s_acc = reinterpret_cast<ulonglong2*>(s_vz + kUcCells);
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        constexpr uint32_t fb = sizeof(float) * kUcCells;
        constexpr uint32_t total = 8 * fb + sizeof(ulonglong2) * kUcCells;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&bar)), "r"(total)
                     : "memory");
        bulk_load(s_f, A.cs.free_m + c0, fb, &bar);
        bulk_load(s_s, A.cs.static_m + c0, fb, &bar);
        bulk_load(s_d, A.cs.dyn_m + c0, fb, &bar);
        bulk_load(s_start, A.cw.start + c0, fb, &bar);
        bulk_load(s_w, A.cw.sum_w + c0, fb, &bar);
        bulk_load(s_vx, A.cw.sum_wvx + c0, fb, &bar);
        bulk_load(s_vy, A.cw.sum_wvy + c0, fb, &bar);
        bulk_load(s_vz, A.cw.sum_wvz + c0, fb, &bar);
        bulk_load(s_acc, acc + c0, sizeof(ulonglong2) * kUcCells, &bar);
    }
    if (!bar_wait(&bar, kUcMaxPolls)) {
        if (threadIdx.x == 0) atomicOr(&A.status->copy_timeout, 1u);
        bar_wait(&bar, kUcMaxPolls);  // the copies still write this CTA's shared memory
        return;
    }
    for (int i = threadIdx.x; i < kUcCells; i += kUcThreads) {
        const int c = (int)(c0 + i);
        const int sc = scene_of(bt.off->cell, bt.S, c);
        const SceneDev& sd = bt.sc[sc];
        const ulonglong2 v = s_acc[i];
        if (v.x || v.y) acc[c] = make_ulonglong2(0ull, 0ull);
        CellIn in;
        in.m_f = s_f[i];
        in.m_s = s_s[i];
        in.m_d = s_d[i];
        in.start = first ? -1 : s_start[i];
        in.sum_w = s_w[i];
        in.wvx = s_vx[i];
        in.wvy = s_vy[i];
        in.wvz = s_vz[i];
        k3dom_cell_update_in(sd.p, bt.fp[sc].gamma_dt, c, (double)(long long)v.x * sd.fx_inv,
                             (double)(long long)v.y * sd.fx_inv, in, A.cs, A.cw, first);
    }
}

cudaError_t make_kernel_table_texture(RayBuffers& rb, int S) {
    rb.ktex = 0;
    cudaResourceDesc rd = {};
    rd.resType = cudaResourceTypeLinear;
    rd.res.linear.devPtr = rb.ktab;
    rd.res.linear.desc = cudaCreateChannelDesc<float4>();
    rd.res.linear.sizeInBytes = sizeof(float4) * (size_t)kKernelTabEntries * (size_t)S;
    cudaTextureDesc td = {};
    td.readMode = cudaReadModeElementType;  // the stored FP32 values, no filtering
    td.filterMode = cudaFilterModePoint;
    td.addressMode[0] = cudaAddressModeClamp;
    return cudaCreateTextureObject(&rb.ktex, &rd, &td, nullptr);
}

cudaError_t launch_k3dom_update_cells(const Batch& bt, RayBuffers& rb, CellState cs, CellWork cw, DevStatus* status,
                                      cudaStream_t st) {
    const EvArgs A = make_args(bt, rb, cs, cw, false, status);
    ++g_launches;
    const uintptr_t bases = reinterpret_cast<uintptr_t>(cs.free_m) | reinterpret_cast<uintptr_t>(cs.static_m) |
                            reinterpret_cast<uintptr_t>(cs.dyn_m) | reinterpret_cast<uintptr_t>(cw.start) |
                            reinterpret_cast<uintptr_t>(cw.sum_w) | reinterpret_cast<uintptr_t>(cw.sum_wvx) |
                            reinterpret_cast<uintptr_t>(cw.sum_wvy) | reinterpret_cast<uintptr_t>(cw.sum_wvz) |
                            reinterpret_cast<uintptr_t>(rb.acc);
    if (bt.C >= kUcBulk && (bases & 15u) == 0) {  // the bulk copies' alignment (cudaMalloc gives 256 bytes)
        k_k3dom_update_cells_bulk<<<div_up(bt.C, kUcCells), kUcThreads, kUcSmem, st>>>(A);
        return cudaGetLastError();
    }
    // one thread per cell: the update is latency bound, so every cell's reads are in flight at once
    k_k3dom_update_cells<<<div_up(bt.C, kBlock), kBlock, 0, st>>>(A);
    return cudaGetLastError();
}

// The DS passes: k_ds_rays is persistent, one CTA per resident slot; k_ds_partial gets as many.
static int ds_blocks(const void* kern) {
    int dev = 0, sms = 148, per = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, kEvThreads, 0);
    return sms * std::max(1, per);
}

void k3dom_ds_evidence_blocks(int* ray_blocks, int* partial_blocks) {
    *ray_blocks = ds_blocks((const void*)k_ds_rays);
    *partial_blocks = ds_blocks((const void*)k_ds_partial);
}

cudaError_t launch_ds_measure(const Batch& bt, RayBuffers& rb, DevStatus* status, cudaStream_t st) {
    if (rb.chunk < 32 || rb.chunk > kChunk) return cudaErrorInvalidValue;
    const EvArgs A = make_args(bt, rb, CellState{}, CellWork{}, false, status);
    g_launches += 3;
    k_ds_rays<<<ds_blocks((const void*)k_ds_rays), kEvThreads, 0, st>>>(A);
    const int per_tile = div_up(rb.ds_stride, kEvThreads);
    k_ds_combine<<<bt.T * per_tile, kEvThreads, 0, st>>>(A, per_tile);
    k_ds_partial<<<ds_blocks((const void*)k_ds_partial), kEvThreads, 0, st>>>(A);
    return cudaGetLastError();
}

cudaError_t launch_ds_update(const Batch& bt, RayBuffers& rb, CellState cs, CellWork cw, bool first_frame,
                             DevStatus* status, cudaStream_t st) {
    const EvArgs A = make_args(bt, rb, cs, cw, first_frame, status);
    ++g_launches;
    k_ds_update<<<div_up(bt.C, kBlock), kBlock, 0, st>>>(A);
    return cudaGetLastError();
}

cudaError_t evidence_init() {
    const int marks = (int)(sizeof(uint4) * kMarkMaxTiles);
    cudaError_t m = cudaFuncSetAttribute(k_ds_mark<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, marks);
    if (m == cudaSuccess) m = cudaFuncSetAttribute(k_ds_mark<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, marks);
    const int hist = (int)(sizeof(uint32_t) * kPlacedMaxTiles);
    if (m == cudaSuccess) m = cudaFuncSetAttribute(k_ray_count<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, hist);
    if (m == cudaSuccess) m = cudaFuncSetAttribute(k_ray_place, cudaFuncAttributeMaxDynamicSharedMemorySize, hist);
    if (m != cudaSuccess) return m;
    cudaError_t e = cudaFuncSetAttribute(k_bgki, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)bgki_smem_bytes(kChunk));
    if (e != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(k_bgki_sums, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)calib_smem_bytes(kCalibChunk))))
        return e;
    // 48 KB of copies plus the static barrier: above the default per-CTA limit
    return cudaFuncSetAttribute(k_k3dom_update_cells_bulk, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)kUcSmem);
}

}  // namespace k3dom
