// Launchers of the tile-list stage (sort.cu).
#pragma once

#include "common.cuh"

namespace lfs {

// Lists of one camera. The per-Gaussian stage has counted the instances of every tile into the counters (cleared before it).
struct TileListArgs {
    bool count;          // the instances have not been counted yet (see count_tiles_apart)
    int N, tw, th, tile_size;
    const float* means2d;
    const int32_t* radii;
    const float* depths;
    const int32_t* tiles;  // [N] tiles per Gaussian
    int32_t* n_isects_dev; // device int32: total number of instances
    int64_t capacity;      // room in entries and flatten_ids
    uint64_t* entries;     // [capacity] scratch
    int32_t* flatten_ids;  // [capacity]
    int32_t* overflow;     // device flag set when an instance does not fit: no list is built, all offsets are 0
    int32_t* tile_offsets; // [tw*th + 1]
    int32_t* state;        // [tile_list_state_words(tw*th, capacity)], 16-byte aligned
    // EWA path: when set, a Gaussian's instances are the tiles of its bounds rectangle that pass the exact
    // ellipse test (`tiles` holds that count); means2d / radii / depths are unused
    const ushort4* ewa_bounds = nullptr;        // [N] (x_min, x_max, y_min, y_max) in tiles
    const float4* ewa_records = nullptr;        // [N*3], see ewa_common.cuh
    const uint64_t* ewa_masks = nullptr;        // [N] which tiles of a rectangle of up to 64 pass, in row-major order
    const uint32_t* ewa_depth_bits = nullptr;   // [N]
};

int build_tile_lists(const TileListArgs& a, cudaStream_t st);
// whether a kernel of its own counts the instances of N Gaussians in `bins` tiles, instead of the per-Gaussian stage
bool count_tiles_apart(int64_t N, int64_t bins);
size_t tile_list_state_words(int64_t bins, int64_t capacity);
TileCounters tile_list_counters(int32_t* state, int64_t bins);
int clear_tile_counters(const TileCounters& t, cudaStream_t st);
const int32_t* tile_list_order(const int32_t* state, int64_t bins);   // [bins]: tile indices, longest lists first

// Operator level: C cameras with N Gaussians each (flattened index = cid * N + gid), 64-bit keys (camera | tile | depth bits).
struct IsectBuffers {
    int32_t* state;
    SortScratch scratch;
    uint64_t* entries;   // [n_isects]
    int32_t* prefix;     // [C*N], unsorted lists only; shares the memory of entries
};
size_t isect_lists_bytes(int64_t total, int64_t n_isects, IsectBuffers* b, void* base);
// sort = 0: emission order, 1: (camera, tile, depth, index) order
int build_isect_lists(int C, int N, int tw, int th, int tile_size, int sort, const float* means2d, const int32_t* radii, const float* depths,
                      const int32_t* tiles, int64_t n_isects, const IsectBuffers& b, int64_t* isect_ids, int32_t* flatten_ids, cudaStream_t st);
int launch_isect_offset(int64_t n, const int64_t* isect_ids, int C, int tw, int th, int32_t* offsets, cudaStream_t st);
int launch_sum_i32(int64_t n, const int32_t* src, int64_t* out_dev, cudaStream_t st);

}  // namespace lfs
