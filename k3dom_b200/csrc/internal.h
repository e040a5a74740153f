// internal.h -- launch wrappers shared between the .cu files of the library.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "common.cuh"

namespace k3dom {

// Kernel launches enqueued by this library (host counter; a frame's count is the difference
// across it). Handles are single-threaded, as the reference's DOM is.
extern long g_launches;

// scan.cu
int scan_u32_tiles(long n);
cudaError_t scan_u32_exclusive(const uint32_t* in, uint32_t* out, long n, uint32_t* tmp, uint32_t* total,
                               cudaStream_t st);

// onesweep.cu: the particle sort (one histogram read, then one read and write per 7-bit digit
// with decoupled look-back). A look-back poll loop gives up after max_polls polls and sets
// DevStatus::sort_timeout; skip_tile >= 0 keeps that tile of the first pass from publishing its
// counts (a test hook: every later tile's wait then runs out).
struct SortWait {
    uint32_t max_polls = 1u << 20;
    int skip_tile = -1;
    bool cleared = false;  // the caller has cleared the scratch (onesweep_clear)
};
int onesweep_plan(int key_bits, int* pass_bits);
long onesweep_scratch_words(long n, int key_bits);
cudaError_t onesweep_clear(uint32_t* scratch, long n, int key_bits, cudaStream_t st);
cudaError_t onesweep_init();
cudaError_t onesweep_sort_pairs(const uint32_t* keys, const uint32_t* vals, uint32_t* keys_out, uint32_t* vals_out,
                                uint32_t* alt_k, uint32_t* alt_v, long n, int key_bits, uint32_t* scratch,
                                long scratch_words, DevStatus* ds, const SortWait& wait, cudaStream_t st);
// The same with the element count min(*dn, nmax) read on the device (dn may be nullptr).
cudaError_t onesweep_sort_pairs_dn(const uint32_t* keys, const uint32_t* vals, uint32_t* keys_out, uint32_t* vals_out,
                                   uint32_t* alt_k, uint32_t* alt_v, long nmax, const uint32_t* dn, int key_bits,
                                   uint32_t* scratch, long scratch_words, DevStatus* ds, const SortWait& wait,
                                   cudaStream_t st);

// exactscan.cu: inclusive prefix sums of non-negative floats, exact in 128-bit fixed
// point and rounded once to float.
int exact_scan_tiles(long n);
// Scratch bytes for exact_scan of n elements.
size_t exact_scan_scratch_bytes(long n);
cudaError_t exact_scan_float(const float* in, float* out, long n, void* scratch, cudaStream_t st);
// Same over the concatenation a[0..na) ++ b[0..nb).
cudaError_t exact_scan_float2(const float* a, long na, const float* b, long nb, float* out,
                              void* scratch, cudaStream_t st);

// Segmented exact scan driven by a plan of tiles (each <= 2048 elements, one contiguous input
// and output range, and the index of its segment's first tile).
struct ExactTile {
    float* in;  // writable: a scan may clear its sign-bit inputs in place
    float* out;
    int n;
    int seg_first;
};
// Appends one segment made of `pieces` input ranges, written contiguously from `out`.
void exact_plan_add(std::vector<ExactTile>& plan, float* const* in, const long* n, int pieces, float* out);
size_t exact_plan_scratch_bytes(int ntiles);
// clear_signed: every input with its sign bit set (counted as 0 by the scan) is also set to +0 in
// place, the penalty step of resampling.cu:13-36 folded into the joint weights' scan.
cudaError_t exact_scan_plan(const ExactTile* tiles, int nt, void* scratch, cudaStream_t st, bool clear_signed = false);

// particles.cu
// Prediction reads the structure-of-arrays set a and writes each particle as a 32-byte record
// (x[2i] = px py pz vx, x[2i+1] = vy vz w assoc) plus its cell index a.cell.
void launch_predict(const Batch& bt, Particles a, float4* x, cudaStream_t st);
void launch_pack_records(int n, Particles a, float4* x, cudaStream_t st);
void launch_unpack_records(int n, const float4* x, Particles a, cudaStream_t st);
void launch_shift_particles(int n, Particles a, int mx, int my, int mz, cudaStream_t st);
// Piece sums of one 128-slot range of the sorted particles (gather + segmented sums): the
// range's first piece when its cell began in an earlier range, and its last piece when its cell
// continues into the next range.
struct SegRec {
    double lead[4];   // sum w, w vx, w vy, w vz of the first piece
    double trail[4];  // the same of the last piece
    int lead_end;     // position of the first piece's last particle; -1: it reaches the range's end
    int trail_head;   // position of the last piece's cell head; -1: no such piece
};
long seg_rec_count(long P);
void launch_gather_segsum(const Batch& bt, const float4* x, Particles s, const uint32_t* sorted_keys,
                          const uint32_t* perm, CellWork cw, SegRec* rec, cudaStream_t st);
void launch_reweight(const Batch& bt, Particles s, const uint32_t* sorted_keys, CellWork cw, cudaStream_t st);
void launch_births(const Batch& bt, const float* born, const float* born_cum, Particles b, cudaStream_t st);
void launch_init_particles(const Batch& bt, const float* born_cum, Particles a, cudaStream_t st);
long res_bracket_count(long P);
void launch_resample(const Batch& bt, const float* joint_cum, const uint32_t* sorted_draws, Particles s,
                     Particles b, Particles out, int* ancestors, float* joint_max_out, int2* brackets,
                     cudaStream_t st);
void launch_debug_draws(uint64_t seed, int frame, int stage, long first, long count, float* dst,
                        cudaStream_t st);

// drawsort.cu: the frame's resampling draws as 24-bit keys of 1 - u, sorted within each scene's
// particle range.
constexpr int kDrawPerBlock = 16384;
int draw_blocks(int P);              // blocks of a scene of P particles
long draw_row_words(int blocks);     // words of DrawScratch::rows
long draw_bucket_words(int S);       // words of totals and of starts
struct DrawScratch {
    uint32_t *totals, *starts, *rows, *keys;  // totals: zero between calls; keys: one per particle
};
void launch_sorted_draws(const Batch& bt, int blocks, const DrawScratch& d, uint32_t* sorted, cudaStream_t st);

// cells.cu
void launch_cells_init(const Batch& bt, CellState cs, CellWork cw, cudaStream_t st);
void launch_map_shift_full(const DevParams& p, CellState src, CellState dst, const int* s_start,
                           const int* s_end, int* d_start, int* d_end, int mx, int my, int mz,
                           cudaStream_t st);
// Exports take the scene's own ranges (pointers offset by its cell range); range_base is the
// scene's first sorted particle.
void launch_export_field(const DevParams& p, int field, CellState cs, CellWork cw,
                         const float* born_cum, int range_base, float* dst, cudaStream_t st);
void launch_export_gridcell(const DevParams& p, CellState cs, CellWork cw, const float* born_cum,
                            int range_base, void* dst, cudaStream_t st);
void launch_export_mappoints(const DevParams& p, float cx, float cy, float cz, CellState cs,
                             CellWork cw, float* dst, cudaStream_t st);

// evidence.cu
struct RayBuffers {
    float4* ray_a;         // m.x, m.y, m.z, d_m (K3DOM) | |m|^2 (DS)
    double4* ray_c;        // d_m, margin, 1/d_m, 0 in FP64 (K3DOM)
    float4* ktab;          // per scene: sparse-kernel table with the fixed-point scale folded in
    cudaTextureObject_t ktex;  // the kernel table through the texture path (k_bgki: ktab; k_bgki_sums: f), 0 when not made
    uint32_t* counts;      // [kRayThreads * N] tiles touched per point slot (sorted lists) or per thread of a slot
                           // (placed K3DOM lists)
    uint32_t* offsets;     // exclusive scan of counts (sorted lists)
    uint32_t* ekeys;       // entries: global tile id (sorted lists)
    uint32_t* evals;       // entries: point slot (sorted lists)
    uint32_t* ekeys2;      // sorted lists
    uint32_t* evals2;      // the lists: point slots grouped by tile (placed or sorted)
    uint32_t* tile_tally;  // T: rays per tile, zero between K3DOM frames
    uint32_t* mark_groups;  // DS: [mark_groups(N)][T], counts per group of blocks, then their prefixes
    uint32_t* block_base;  // DS: [mark_blocks(N)][T], rays per block and tile; K3DOM:
                           // [bin_blocks(kRayThreads N)][T], each binning block's first slot in each
                           // tile's range, relative to the range's start
    uint32_t* ekeys_alt;
    uint32_t* evals_alt;
    uint32_t* tile_start;  // T+1
    uint32_t* tile_items;  // T: work items per tile
    uint32_t* item_off;    // T+1 work-item offsets per tile
    uint32_t* tile_done;   // T
    unsigned long long* acc;  // 2*C fixed-point accumulators (K3DOM) / DS partials
    uint32_t* ds_r2;       // DS: per (item, cell) smallest squared point distance (float bits)
    uint8_t* ds_counts;    // DS: per (item, cell) neighbours (101 = more than 100), bit 7: one closer than the cell
    uint32_t* scan_tmp;
    long scan_words;
    uint32_t* os_scratch;  // onesweep sort of the entries by tile
    long os_words;
    uint32_t* total;       // [0] = entries, [2] = entries kept (0 on overflow)
    long capacity;         // entries
    long ds_capacity;      // DS: (item, cell) summaries
    int ds_stride;         // DS: cells of the largest tile
    int ds_spare;          // DS: items beyond one per tile that the summaries are sized for (0: K3DOM)
    int chunk;             // largest number of rays per work item
    int item_slots;        // CTA slots the work items are spread over (0: items of chunk rays whatever the scene)
};
// Rays per work item for a tuned chunk: K3DOM takes kItemLeast at least (fewer leave its batches of 32
// candidates per class part empty, and every sub-block's set-up is paid per item). A frame of
// 256x256x32 voxels, 120,000 rays, 16x16x8 tiles, by chunk: 32 rays 5,725 us, 64 3,523, 128 2,406, 256
// 1,778 (one cell a lane without batches: 3,829, 2,921, 2,487, 2,294); 64x64x16, 30,000 rays, 8x8x4
// tiles: 358, 273, 229, 214 (269, 237, 218, 220).
constexpr int kItemLeast = 256;
inline int evidence_chunk(bool ds, int chunk) { return ds || chunk > kItemLeast ? chunk : kItemLeast; }
long ray_entries_bound(const DevParams& p, const TileShape& ts, int max_points, float bin_R);
// Ray lists are placed per tile through block histograms (K3DOM: 4 bytes a tile) or bit masks (DS: 16
// bytes) of all T tiles in shared memory; otherwise the entries are sorted by tile. Both take what
// lets two blocks share an SM. K3DOM, 1 to 4 scenes of 256x256x32 voxels at 0.1 m and 120,000 rays in
// 8x8x4 tiles, lists placed and sorted: 8,192 tiles 177 and 400 us, 16,384 344 and 655, 24,576 638 and
// 894, 32,768 (one block per SM) 1,439 and 1,154. DS, one such scene: 1,024 tiles 76 and 145 us, 2,048
// 94 and 156, 8,192 (one block) 271 and 229. DS keeps up to kMarkMaxCounts counts (128 MB).
constexpr int kPlacedMaxTiles = 28416;
constexpr int kMarkMaxTiles = 6144;
constexpr int kMarkRays = 128;   // rays per block of the DS passes
constexpr int kMarkGroup = 32;   // blocks whose counts are added up together
constexpr long kMarkMaxCounts = 32L << 20;
int mark_blocks(int N);
int mark_groups(int N);
inline bool placed_lists(bool ds, int T, int N) {
    return ds ? T <= kMarkMaxTiles && (long)mark_blocks(N) * T <= kMarkMaxCounts : T <= kPlacedMaxTiles;
}
// DS summaries take 5 bytes per (item, cell), and the items of chunk rays that lists at their capacity
// would make need far more of them than frames do (256x256x32 voxels, 120,000 rays: capacity 23.0M
// entries, 2.3M held). A tenth of those items is allowed for, 64 MB at least; a frame with more entries
// than that makes larger items (item_rays), up to kDsSpareDiv times the chunk. The handle there takes
// 520 MB instead of 912 (items of 512 rays) and 1.2 GB instead of 7.8 (32 rays), at the same frame time
// (837 and 838 us).
constexpr int kDsSpareDiv = 10;
constexpr long kDsSpareBytes = 64L << 20;
long ds_spare_items(long capacity, int chunk, int stride);
constexpr int kBinBlocksMax = 1024;
int bin_blocks(long n);  // blocks of the placed-list passes over n threads
constexpr int kRayThreads = 2;  // threads per ray in the placed-list passes
// Texture object over the S kernel tables (point sampling, FP32 as stored), for k_bgki.
cudaError_t make_kernel_table_texture(RayBuffers& rb, int S);
// Per-scene evidence constants (binning radius, cull radius, fixed-point scale); writes the
// scene's kernel table when ktab is not null.
void fill_scene_evidence(SceneDev& sd, bool ds, float4* ktab);
cudaError_t build_ray_lists(const Batch& bt, const float* xs, const float* ys, const float* zs, RayBuffers& rb,
                            bool ds, DevStatus* status, const SortWait& wait, cudaStream_t st);
cudaError_t launch_k3dom_evidence(const Batch& bt, RayBuffers& rb, CellState cs, CellWork cw, bool first_frame,
                                  DevStatus* status, cudaStream_t st, bool fuse_update = true);
// The cell update of a K3DOM frame whose evidence ran with fuse_update = false.
cudaError_t launch_k3dom_update_cells(const Batch& bt, RayBuffers& rb, CellState cs, CellWork cw, DevStatus* status,
                                      cudaStream_t st);
// DS: the measurement grid from the ray lists, then the masses of every cell.
cudaError_t launch_ds_measure(const Batch& bt, RayBuffers& rb, DevStatus* status, cudaStream_t st);
cudaError_t launch_ds_update(const Batch& bt, RayBuffers& rb, CellState cs, CellWork cw, bool first_frame,
                             DevStatus* status, cudaStream_t st);
// CTA slots of the K3DOM and calibration evidence kernels, for RayBuffers::item_slots.
int evidence_slots(int num_sms);
// CTAs of the K3DOM evidence launch for a chunk size (persistent grid).
int k3dom_evidence_blocks(int chunk);
// CTAs of the DS pass over the rays and of the pass over the cells past 100 neighbours.
void k3dom_ds_evidence_blocks(int* ray_blocks, int* partial_blocks);
cudaError_t evidence_init();
// Host: the sparse-kernel table for sigma, every value multiplied by scale: 512 intervals and a
// zero entry at u = 1 (513 float4), so an index taken at the support's edge needs no clamp.
void build_kernel_table(float sigma, double scale, float4* out);
constexpr int kKernelTableSize = 513;
// Rays per calibration work item at most: 4 CTAs per SM still fit beside the derivative's table
// (gradient step at 256x256x32 voxels: 448 rays 3.90 ms, 768 rays 3.75 ms).
constexpr int kCalibChunk = 768;
// Calibration: unit-amplitude kernel and -x f'(x) tables scaled to units of 2^-kCalibShift.
constexpr int kCalibShift = 40;
void build_calib_tables(float4* f_tab, float4* dls_tab);
// rb.ktex: f's table; dls_tab: the table of -x f'.
cudaError_t launch_bgki_sums(const Batch& bt, RayBuffers& rb, const float4* dls_tab, unsigned long long* acc4,
                             DevStatus* status, int num_sms, cudaStream_t st);

}  // namespace k3dom
