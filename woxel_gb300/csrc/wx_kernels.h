// wx_kernels.h — host-side view of the kernels in kernels.cu (internal).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "sdf_steps.h"
#include "woxel_gb300.h"

namespace wxk {

// Device node pools of one grid (see api.cpp for the layout).
struct DevGrid {
    const int4 *root;        // root block: header, N5 origins, dense root-key table (api.cpp)
    const uint32_t *slot5;   // N5 slot words
    const uint32_t *slot4;   // N4 slot words
    const uint8_t *leaf;     // N3: one byte per voxel, 0 hit, 1..254 distance, 255 = see ovf
    const uint2 *ovf;        // (voxel key = leaf << 9 | offset, distance), sorted by key
    const float *values;     // level-set value per leaf voxel (zero-crossing mode), or null
    uint32_t n5, n_ovf;
    float band;              // value of voxels outside leaves (+band; -band in active tiles)
    uint32_t inside;         // bit 0: every N5 lies in [-4096, 4096)^3 (origins -4096 or 0 on each axis);
                             // bit 1: some tile distance is 2^24 or more
    uint32_t n4, n3;         // node counts of the N4 and N3 pools (checked in bounds-checked builds)
};

// The N5 slot words of the box [-4096, 4096)^3 as one dense table of 64^3 words, which lies just
// before slot5: word x << 12 | y << 6 | z for the N4-sized cell (x, y, z) of the box.
constexpr uint32_t kTopWords = 64u * 64u * 64u;

// One frame of one grid: the unit the persistent kernels draw ray tiles from.
struct Job {
    DevGrid g;
    uint32_t width, height;
    uint16_t tile_w, tile_h;       // pixel tile of one warp (tile_w * tile_h = 32)
    uint32_t order;                // bit 0, tile rows: 0 top to bottom, 1 middle row first, then outwards;
                                   // from bit 8: the grid's place in the launch's GridTable
    uint32_t tiles_x, tiles;       // tiles per row / per frame over the dispatched region
    uint32_t tile_begin;           // first global (queue) tile id of this job
    uint32_t tile_off;             // first frame tile of this job (a job may cover part of a frame)
    uint32_t *rgba;
    wx_hit *hits;
    wx_state_uniform s;
    // Cancellation (batched launches given a cancel table): the job's tiles are
    // skipped once cancel[cancel_slot] == cancel_id (nonzero). 0 = never.
    uint32_t cancel_slot, cancel_id;
};

// The distinct grids of a batched launch, a kernel parameter; n = kTableGrids + 1 when there are more than kTableGrids
// (the jobs' own copies are then used).
constexpr uint32_t kTableGrids = 64;
struct GridTable {
    DevGrid g[kTableGrids];
    uint32_t n;
};

struct Tuning {
    int kernel = 1;            // 1 one warp per tile (k_pixel), 0 persistent warps on a tile queue
    int warps_per_block = 4;   // 1..16
    int blocks_per_sm = 0;     // 0 = as many as fit
    int tile_w = 8;            // 4, 8, 16 or 32 pixels wide (x 32/tile_w high)
    int order = 1;             // Job::order
    int rays = 1;              // k_pixel: 1 pixel per lane; 2, 4 or 8 tiles per warp with lanes that refill (k_wave)
};

cudaError_t init_device_tables();
// Fills the dense table before g.slot5 from the root block and slot5.
cudaError_t build_top_table(const DevGrid &g, cudaStream_t st);
int max_blocks_per_sm(int kernel, bool batched, int warps_per_block);
// disjoint: the job's outputs do not overlap those of the previous kernel on st,
// a k_pixel launch (see k_pixel); false is always safe. split: 2^split warps share a tile (not in k_wave).
cudaError_t launch_pixel(const Job &job, const Tuning &t, bool disjoint, uint32_t split, cudaStream_t st);
cudaError_t launch_persistent(const Job &job, uint32_t *ctr, const Tuning &t, int num_sms, cudaStream_t st);
// all: some job renders mode 4 or 5 (the kernels compiled for every mode).
// cancel (may be NULL): the table the jobs' cancel_slot index; skipped (may be
// NULL) counts the tiles skipped for a cancelled job (the caller clears it).
// tab: index_grid of every job, which must be done before the jobs are copied to jobs_dev.
cudaError_t launch_batched(const Job *jobs_dev, uint32_t njobs, const GridTable &tab, uint32_t total_tiles, uint32_t *ctr,
                           const Tuning &t, int num_sms, bool all, cudaStream_t st,
                           const uint32_t *cancel = nullptr, uint32_t *skipped = nullptr);
// Enters a launch of `tiles` into the process's ring of launches (launch_ring.h); returns the tiles of the other streams of its
// device, or a number above `enough`.
uint64_t enter_launch(int device, cudaStream_t st, uint64_t tiles, uint64_t enough = 0);
// Enters the job's grid into the table (unless it has overflowed: n = kTableGrids + 1) and its place into job.order.
void index_grid(Job &job, GridTable &tab);
// Modes 4 (glossy) and 5 (zero crossing) need the kernels compiled for every mode.
bool all_modes(const wx_state_uniform &s);
bool all_modes(const Job *jobs, size_t n);
// Device pools and device of a grid handle (defined in api.cpp); false for NULL.
bool grid_device_view(const wx_grid *grid, DevGrid *out, int *device);
// Device index and SM count of a context (defined in api.cpp).
void ctx_device_info(const wx_ctx *ctx, int *device, int *num_sms);

// GPU SDF build (sdf.cu). The tree structure that neighbours are looked up in:
// the root block of the grid layout (header, origins, root-key table) and the
// child-index tables (slot -> child DFS index or 0xFFFFFFFF).
struct SdfTree {
    const int4 *root;
    uint32_t n5;
    const uint32_t *c5, *c4;
};
// pre: a word per mask word, filled here.
cudaError_t sdf_child_table(const uint64_t *kid, uint32_t *pre, const uint32_t *first, uint64_t nodes,
                            int slots_log2, uint32_t *cidx, cudaStream_t st);
cudaError_t sdf_child_origins(const uint32_t *cidx, const int4 *org, uint64_t nodes, int log2d, int child_span_log2,
                              int4 *org_child, cudaStream_t st);
cudaError_t sdf_neighbours(int level, const int4 *org, uint32_t nc, const SdfTree &t, uint32_t *nb, cudaStream_t st);
// *count += the clear bits of `words` mask words.
cudaError_t sdf_count_clear(const uint64_t *w, uint64_t words, unsigned long long *count, cudaStream_t st);
// Steps whose W sets are kept until sdf_expand. Level sets are done after about this many.
constexpr uint32_t kSdfWindow = 8u;
// One level of the tree in the distance computation (sdf.cu). Masks are those of the grid (bit = cell, D^3 a node).
struct SdfLevel {
    // kSdfWindow + 3 sets of (n + 1) nodes, `stride` words each. 0: z, the cells that start at distance 0 (children,
    // active voxels), which is F(0) and W(0); 1..kSdfWindow: W(k), then, for larger k, W(k) in the last of them or the
    // one before by parity; the two after them: F(k) by parity. Node n, the missing neighbour, is all ones in z and
    // the W sets.
    uint64_t *sets;
    uint32_t stride;
    const uint64_t *val;     // N5/N4: active tiles
    const uint32_t *nb;      // 27 neighbours of each node (n where there is none)
    uint32_t *act;           // n + 1 words: last k at which the node or a neighbour changed; starts at 0
    uint32_t *slot;          // N5/N4: slot words
    uint32_t n;              // nodes
};
struct SdfWork {
    SdfLevel lv[3];          // N5, N4, leaves
    uint8_t *leaf;           // leaf bytes
    uint2 *ovf;              // (cell, distance) of distances >= 255
    uint32_t ovf_cap;
    SdfCtl *ctl;
};
// Steps k0..k1 (fewer when no cell is left). ctl->error is set when a wait hit its bound.
// spin_limit: polls (256 ns apart) a CTA makes at the barrier between two steps before it sets
// the error flag and every CTA returns.
constexpr uint32_t kSdfSpinLimit = 1u << 23;  // about 2 s
constexpr uint32_t kSdfMaxLevel = 4095u;      // no grid reaches it
cudaError_t sdf_levels(const SdfWork &w, uint32_t k0, uint32_t k1, int num_sms, uint32_t spin_limit, cudaStream_t st);
// Slot words and leaf bytes from the W sets of steps 0..kSdfWindow: after sdf_levels(1, kSdfWindow), before larger k.
cudaError_t sdf_expand(const SdfWork &w, const uint32_t *cidx5, const uint32_t *cidx4, cudaStream_t st);

// Packing of the flattened view (pack.cu): a piece of an atlas in device memory, whole layers of d * d nodes or some
// block rows (d nodes) of one layer, with the masks of its nodes. The texel of node idx's slot (x, y, z) is at ((idx' / d^2 * D + z) * h + (idx' / d % d * D + y)) * w + idx' % d * D + x
// with idx' = idx - first.
struct ViewSlab {
    const uint32_t *texels;
    uint32_t w, h;       // width of the texture, height of the piece
    uint32_t d;          // nodes per row and rows per layer, as the shader derives them
    uint64_t first, count;  // nodes of the piece; first is a multiple of d
};
cudaError_t pack_view_nodes(int level, const ViewSlab &s, const uint32_t *kids, const uint32_t *vals, uint32_t nchild,
                            uint32_t *slot, uint32_t *flags, cudaStream_t st);
cudaError_t pack_view_leaves(const ViewSlab &s, const uint32_t *vals, uint8_t *leaf, uint2 *ovf, uint32_t cap,
                             unsigned long long *n_ovf, cudaStream_t st);

// Exhaustive check of the fast floor-division path against IEEE division:
// every divisor m < max_m and every significand of [1,2) and [-2,-1).
// out[0] = mismatch count, out[1] = first mismatching m, out[2] = its x bits.
cudaError_t check_division(uint32_t max_m, unsigned long long *out_dev, cudaStream_t st);
// Bounds-checked builds: reads and zeroes the device's count of out-of-range indices.
cudaError_t take_bounds_violations(unsigned long long *count);

}  // namespace wxk
