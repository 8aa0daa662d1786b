// Tile-list construction: the depth-sorted list of Gaussians of every tile, and prefix sums.
//
// Replaces gsplat/IntersectTile.cu:24 (second pass), the at::cumsum + CUB DeviceRadixSort::SortPairs
// call of gsplat/Intersect.cpp:75 / gsplat/IntersectTile.cu:290-328, and gsplat/IntersectTile.cu:206.
//
// The reference sorts n_isects 12-byte (int64 key, int32 value) pairs over 32 + tile_bits + cam_bits bits. The order that comes out
// (camera, tile, depth bits, ties by ascending flattened Gaussian index) is a total one inside each tile, so nothing has to be stable:
// the per-Gaussian stage counts the instances of every tile (one reduction to memory per instance), one cluster turns the counts into
// offsets, the instances drop into their tile's range in any order (8 bytes each, one returning atomic), and every range is sorted by
// (depth bits, index) where it fits into shared memory. Against two global radix sorts (depth of N, then tile of the instances) the
// instances are written twice instead of six times and there are three launches instead of eleven. All of the list build, projection's
// extra counting included, in us, before and now: 16 k Gaussians at 256x256 90 and 36, 150 k at 640x360 126 and 53, 1 M at 1296x840
// 253 and 131, 3 M at 1600x1064 632 and 420, 6 M at 3840x2160 743 and 320.
#include "gsmath.cuh"
#include "sort.cuh"
#include "ewa_common.cuh"

#include <cooperative_groups.h>

namespace lfs {

namespace {

constexpr int kThreads = 256;
constexpr int kTile = 2048;

// Exclusive scan over the block (any multiple of 32 threads up to 1024); returns the block total.
__device__ __forceinline__ int block_excl_scan(int v, int& total, int* smem /*[33]*/) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int incl = warp_incl_scan(v);
    if (lane == 31) smem[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int s = lane < nw ? smem[lane] : 0;
        const int si = warp_incl_scan(s);
        smem[lane] = si - s;
        if (lane == 31) smem[32] = si;
    }
    __syncthreads();
    const int base = smem[warp];
    total = smem[32];
    __syncthreads();
    return base + incl - v;
}

// ---- prefix sum -----------------------------------------------------------------------------
__global__ void __launch_bounds__(kThreads) scan_reduce_kernel(const int32_t* __restrict__ src, int64_t n, int64_t chunk, uint32_t* __restrict__ block_sums) {
    __shared__ int sm[33];
    const int64_t lo = (int64_t)blockIdx.x * chunk, hi = min(n, lo + chunk);
    int s = 0;
    for (int64_t i = lo + threadIdx.x; i < hi; i += kThreads) s += src[i];
    int total;
    block_excl_scan(s, total, sm);
    if (threadIdx.x == 0) block_sums[blockIdx.x] = (uint32_t)total;
}

__global__ void __launch_bounds__(1024) scan_block_sums_kernel(uint32_t* __restrict__ sums, int n, int32_t* __restrict__ total_dev) {
    __shared__ int sm[33];
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < n; base += 1024) {
        const int i = base + threadIdx.x;
        const int v = i < n ? (int)sums[i] : 0;
        int total;
        const int ex = block_excl_scan(v, total, sm);
        if (i < n) sums[i] = (uint32_t)(carry + ex);
        __syncthreads();
        if (threadIdx.x == 0) carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0 && total_dev) *total_dev = carry;
}

__global__ void __launch_bounds__(kThreads) scan_apply_kernel(const int32_t* __restrict__ src, int64_t n, int64_t chunk, const uint32_t* __restrict__ block_sums,
                                                              int32_t* __restrict__ out) {
    __shared__ int sm[33];
    const int64_t lo = (int64_t)blockIdx.x * chunk, hi = min(n, lo + chunk);
    int carry = (int)block_sums[blockIdx.x];
    for (int64_t base = lo; base < hi; base += kThreads) {
        const int64_t i = base + threadIdx.x;
        const int v = i < hi ? src[i] : 0;
        int total;
        const int ex = block_excl_scan(v, total, sm);
        if (i < hi) out[i] = carry + ex;
        carry += total;
    }
}

// ---- scatter ------------------------------------------------------------------------------------
// One entry per instance, (depth bits, flattened Gaussian index), to the next free place of its tile's range. Bound by the latency of the
// returning atomics, so a lane has kInFlight of them under way (8.3 M instances of 6 M Gaussians at 3840x2160: 195 us with one, 171 with two, 152
// with four, 269 with eight; 1 M at 1296x840 no difference).
constexpr int kInFlight = 4;
__global__ void __launch_bounds__(kThreads) tile_scatter_kernel(int64_t total, int N, int tw, int th, float tile_size, const int32_t* __restrict__ tiles,
                                                                const float* __restrict__ means2d, const int32_t* __restrict__ radii,
                                                                const float* __restrict__ depths, int64_t first_bin, int64_t n_bins, int64_t capacity,
                                                                const int32_t* __restrict__ overflow, TileCounters t, uint64_t* __restrict__ entries, int parts) {
    if (overflow && *overflow) return;
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32), chunks = (total + 31) / 32;
    for (int64_t w = (int64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; w < chunks * parts; w += warps) {
        const int64_t base = w % chunks * 32;
        const int part = (int)(w / chunks);
        const int64_t i = base + lane;
        int32_t* cursors = t.cursors + t.replica(base);
        const int nt = i < total ? max(tiles[i], 0) : 0;
        uint32_t x0 = 0, y0 = 0, x1 = 0, y1 = 0, key = 0;
        if (nt > 0) {
            tile_rect(means2d[i * 2], means2d[i * 2 + 1], radii[i * 2], radii[i * 2 + 1], tile_size, tw, th, x0, y0, x1, y1);
            key = __float_as_uint(depths[i]);
        }
        for_each_tile<kInFlight>(nt, x0, y0, x1 - x0, part, parts, [&](bool on, int owner, uint32_t tx, uint32_t ty, uint32_t) {
            const int64_t bin = (N == total ? 0 : (base + owner) / N * ((int64_t)tw * th)) + (int64_t)ty * tw + tx - first_bin;
            return on && bin >= 0 && bin < n_bins ? atomicAdd(cursors + bin, 1) : -1;
        }, [&](int owner, int pos) {
            const uint32_t d = __shfl_sync(0xffffffffu, key, owner);
            if ((uint32_t)pos < (uint32_t)capacity) entries[pos] = ((uint64_t)d << 32) | (uint64_t)(base + owner);
        });
    }
}

// EWA: the tiles of the bounds rectangle that the ellipse reaches (create_instances_cu,
// src/training/fastgs/rasterization/include/kernels_forward.cuh:205-309). Rectangles of up to 64 tiles carry the answers of the
// per-Gaussian stage as a mask, larger ones are tested again.
__global__ void __launch_bounds__(kThreads) ewa_scatter_kernel(int N, int tw, const int32_t* __restrict__ n_touched, const ushort4* __restrict__ bounds,
                                                               const uint64_t* __restrict__ masks, const float4* __restrict__ records,
                                                               const uint32_t* __restrict__ depth_bits, int64_t n_bins, int64_t capacity,
                                                               const int32_t* __restrict__ overflow, TileCounters t, uint64_t* __restrict__ entries, int parts) {
    if (*overflow) return;
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32), chunks = (N + 31) / 32;
    for (int64_t w = (int64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; w < chunks * parts; w += warps) {
        const int64_t base = w % chunks * 32;
        const int part = (int)(w / chunks);
        const int64_t i = base + lane;
        int32_t* cursors = t.cursors + t.replica(base);
        const bool on_screen = i < N && n_touched[i] > 0;
        ushort4 b = make_ushort4(0, 0, 0, 0);
        uint64_t mask = 0;
        uint32_t key = 0;
        if (on_screen) { b = bounds[i]; mask = masks[i]; key = depth_bits[i]; }
        const int width = b.y - b.x, area = width * (b.w - b.z);
        for_each_tile<kInFlight>(area, b.x, b.z, width, part, parts, [&](bool on, int owner, uint32_t tx, uint32_t ty, uint32_t local) {
            const uint64_t m = __shfl_sync(0xffffffffu, mask, owner);
            const int owner_area = __shfl_sync(0xffffffffu, area, owner);
            const int64_t g = base + owner, bin = (int64_t)ty * tw + tx;
            bool hit = on && bin < n_bins;
            if (owner_area <= 64) {
                hit = hit && ((m >> local) & 1u);
            } else if (hit) {
                const float4 c0 = records[g * 3], c1 = records[g * 3 + 1], c2 = records[g * 3 + 2];
                hit = ewa_tile_contributes(c0.x - 0.5f, c0.y - 0.5f, c0.z, c0.w, c1.x, tx, ty, c2.z);
            }
            return hit ? atomicAdd(cursors + bin, 1) : -1;
        }, [&](int owner, int pos) {
            const uint32_t d = __shfl_sync(0xffffffffu, key, owner);
            if ((uint32_t)pos < (uint32_t)capacity) entries[pos] = ((uint64_t)d << 32) | (uint64_t)(base + owner);
        });
    }
}

// Operator level: instances per tile.
__global__ void __launch_bounds__(kThreads) tile_histogram_kernel(int64_t total, int N, int tw, int th, float tile_size, const int32_t* __restrict__ tiles,
                                                                  const float* __restrict__ means2d, const int32_t* __restrict__ radii, int64_t first_bin,
                                                                  int64_t n_bins, TileCounters t, int parts) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32), chunks = (total + 31) / 32;
    for (int64_t w = (int64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; w < chunks * parts; w += warps) {
        const int64_t base = w % chunks * 32;
        const int part = (int)(w / chunks);
        const int64_t i = base + lane;
        int32_t* counts = t.counts + t.replica(base);
        const int nt = i < total ? max(tiles[i], 0) : 0;
        uint32_t x0 = 0, y0 = 0, x1 = 0, y1 = 0;
        if (nt > 0) tile_rect(means2d[i * 2], means2d[i * 2 + 1], radii[i * 2], radii[i * 2 + 1], tile_size, tw, th, x0, y0, x1, y1);
        for_each_tile<1>(nt, x0, y0, x1 - x0, part, parts, [&](bool on, int owner, uint32_t tx, uint32_t ty, uint32_t) {
            const int64_t bin = (N == total ? 0 : (base + owner) / N * ((int64_t)tw * th)) + (int64_t)ty * tw + tx - first_bin;
            if (on && bin >= 0 && bin < n_bins) atomicAdd(counts + bin, 1);
            return 0;
        }, [](int, int) {});
    }
}

// Operator level, unsorted: instances in the order of the Gaussians, each Gaussian's tiles in row-major order. offs: exclusive prefix
// of `tiles`.
__global__ void __launch_bounds__(kThreads) emit_unsorted_kernel(int64_t total, int N, int tw, int th, float tile_size, uint32_t tile_n_bits,
                                                                 const int32_t* __restrict__ tiles, const int32_t* __restrict__ offs,
                                                                 const float* __restrict__ means2d, const int32_t* __restrict__ radii,
                                                                 const float* __restrict__ depths, int64_t capacity, int64_t* __restrict__ isect_ids,
                                                                 int32_t* __restrict__ flatten_ids) {
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x + threadIdx.x - lane; base < total; base += stride) {
        const int64_t i = base + lane;
        const int nt = i < total ? max(tiles[i], 0) : 0;
        uint32_t x0 = 0, y0 = 0, x1 = 0, y1 = 0, key = 0;
        int off = 0;
        if (nt > 0) {
            tile_rect(means2d[i * 2], means2d[i * 2 + 1], radii[i * 2], radii[i * 2 + 1], tile_size, tw, th, x0, y0, x1, y1);
            key = __float_as_uint(depths[i]);
            off = offs[i];
        }
        for_each_tile(nt, x0, y0, x1 - x0, [&](bool on, int owner, uint32_t tx, uint32_t ty, uint32_t local) {
            const uint32_t d = __shfl_sync(0xffffffffu, key, owner);
            const int64_t pos = (int64_t)__shfl_sync(0xffffffffu, off, owner) + local, g = base + owner;
            if (on && pos < capacity) {
                isect_ids[pos] = (((g / N) << tile_n_bits | ((int64_t)ty * tw + tx)) << 32) | d;
                flatten_ids[pos] = (int32_t)g;
            }
        });
    }
}

// ---- offsets, overflow, launch order ---------------------------------------------------------------
// Launch order of the tile CTAs: tiles with the longest lists first, so that the last wave of a rasterizer launch is made of short tiles.
// 132 buckets by the leading one and the next two bits of the list length (a floating-point-like key with a 2-bit mantissa); the order
// inside a bucket is arbitrary.
__device__ __forceinline__ int tile_order_bucket(int c) {
    if (c <= 0) return 131;
    const int lz = __clz(c);                              // 0 .. 31, small = long list
    const int shift = max(0, 29 - lz);                    // bring the two bits below the leading one down
    const int mant = (c >> shift) & 3;
    return lz * 4 + (3 - mant);
}
// first bucket of the lists shorter than 2^K
template <int K>
constexpr int kBucketBelow = (32 - K) * 4;
static_assert(kBucketBelow<8> == kBucketBelow<10> + 8, "");

// Words of the list state in front of the per-bin arrays.
// lists of at least 2^10 and 2^8 entries, and of any; of at least 2^kFarLog
constexpr int kMetaLists = 0, kMetaFar = 3, kMetaParts = 8, kMetaWords = 16, kKinds = 3;
// Lists longer than kRoomCta are sorted in parts of some kPart entries, by as many CTAs. Each part reads the whole list, so lists of 2^kFarLog and
// more are cut into bins first, where there may be such lists (tile_far_kernel).
constexpr int kRoomCta = 8192, kPart = 3072, kFarLog = 16;

// One cluster: counts -> offsets [n_bins + 1] and cursors, the total and the overflow flag (with it all offsets are 0: the list is not
// built), the launch order, and how many lists each kind of sorting group has. Every CTA takes a run of bins, 1024 at a time; the CTAs
// exchange their totals and their bucket counts through each other's shared memory. carry: instances of earlier bins (operator
// level with more bins than the arrays hold), updated.
// One CTA alone took 52 us for the 32,400 bins of a 4K image.
constexpr int kScanCluster = 8;
__global__ void __cluster_dims__(kScanCluster, 1, 1) __launch_bounds__(1024) tile_scan_kernel(
    int n_bins, TileCounters t, int64_t capacity, int64_t* carry, int32_t* __restrict__ n_out, int32_t* overflow, int32_t* __restrict__ offsets,
    int32_t* __restrict__ order, int2* __restrict__ ranges, int4* __restrict__ parts, int32_t* __restrict__ meta, bool far_lists) {
    __shared__ int64_t warp_sums[32], block_sum;
    __shared__ int hist[132], cursor[132], sm[33];
    const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rank = blockIdx.x;
    const uint32_t lt_mask = (1u << lane) - 1u;
    if (threadIdx.x < 132) hist[threadIdx.x] = 0;
    __syncthreads();
    const int run = (n_bins + kScanCluster - 1) / kScanCluster;
    const int first = min(rank * run, n_bins), last = min(first + run, n_bins);
    // the replicas of a bin, eight loads in flight
    auto count = [&](int i) {
        int c = 0;
        for (int r0 = 0; r0 < t.replicas; r0 += 8) {
            int v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = r0 + k < t.replicas ? t.counts[(size_t)(r0 + k) * t.stride + i] : 0;
#pragma unroll
            for (int k = 0; k < 8; ++k) c += v[k];
        }
        return c;
    };
    int64_t sum = 0;
    int kept = 0;   // the count of the first round
    for (int base = first; base < last; base += 1024) {
        const int i = base + threadIdx.x;
        const int c = i < last ? count(i) : 0;
        if (base == first) kept = c;
        sum += c;
        const int bucket = i < last ? tile_order_bucket(c) : -1;
        const uint32_t peers = __match_any_sync(0xffffffffu, bucket);
        if (bucket >= 0 && (peers & lt_mask) == 0) atomicAdd(&hist[bucket], __popc(peers));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) warp_sums[warp] = sum;
    __syncthreads();
    if (warp == 0) {
        int64_t v = warp_sums[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) block_sum = v;
    }
    cluster.sync();
    int64_t at = carry ? *carry : 0, total = at;
    {
        // everybody's totals; one thread per bucket: its count in all CTAs and in the earlier ones
        int64_t v[kScanCluster];
        int h[kScanCluster], all = 0, earlier = 0;
#pragma unroll
        for (int r = 0; r < kScanCluster; ++r) {
            v[r] = *cluster.map_shared_rank(&block_sum, r);
            h[r] = threadIdx.x < 132 ? cluster.map_shared_rank(hist, r)[threadIdx.x] : 0;
        }
#pragma unroll
        for (int r = 0; r < kScanCluster; ++r) {
            total += v[r];
            all += h[r];
            if (r < rank) { at += v[r]; earlier += h[r]; }
        }
        int sum_all;
        const int before = block_excl_scan(all, sum_all, sm);
        if (threadIdx.x < 132) cursor[threadIdx.x] = before + earlier;
    }
    __syncthreads();
    if (rank == 0 && threadIdx.x < kMetaWords) {
        // the first CTA's share of a bucket starts where the bucket does
        const int k = threadIdx.x;
        meta[k] = k == kKinds - 1 ? cursor[131] : k < kKinds - 1 ? cursor[kBucketBelow<10> + 8 * k] : k == kMetaFar && far_lists ? cursor[kBucketBelow<kFarLog>] : 0;
    }
    cluster.sync();   // nobody reads another CTA's memory, or the carry, from here on; meta is set
    const bool dropped = overflow && total > capacity;
    const int32_t total32 = (int32_t)min(total, (int64_t)0x7fffffff);
    if (rank == 0) {
        if (threadIdx.x == 0) {
            if (n_out) *n_out = total32;
            if (dropped) *overflow = 1;
            if (carry) *carry = total;
            offsets[n_bins] = dropped ? 0 : total32;
        }
    }
    __syncthreads();
    for (int base = first; base < last; base += 1024) {
        const int i = base + threadIdx.x;
        const int c = base == first ? kept : i < last ? count(i) : 0;
        int round;
        const int ex = block_excl_scan(c, round, sm);
        const int bucket = i < last ? tile_order_bucket(c) : -1;
        const uint32_t peers = __match_any_sync(0xffffffffu, bucket);
        int slot = 0;
        if (bucket >= 0 && (peers & lt_mask) == 0) slot = atomicAdd(&cursor[bucket], __popc(peers));
        slot = __shfl_sync(0xffffffffu, slot, __ffs(peers) - 1) + __popc(peers & lt_mask);
        if (i < last) {
            order[slot] = i;
            int64_t pos = at + ex;
            const int from = (int)min(pos, capacity), n = (int)min(pos + c, capacity) - from;
            ranges[slot] = make_int2(from, n);
            if (n > kRoomCta && !dropped && !(far_lists && c >> kFarLog)) {
                const int k = (n + kPart - 1) / kPart, base = atomicAdd(meta + kMetaParts, k);
                for (int q = 0; q < k; ++q) parts[base + q] = make_int4(from, n, i, q);
            }
            offsets[i] = dropped ? 0 : (int32_t)min(pos, (int64_t)0x7fffffff);
            for (int r0 = 0; r0 < t.replicas; r0 += 8) {
                int v[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] = r0 + k < t.replicas ? t.counts[(size_t)(r0 + k) * t.stride + i] : 0;
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    if (r0 + k < t.replicas) {
                        t.cursors[(size_t)(r0 + k) * t.stride + i] = (int32_t)min(pos, (int64_t)0x7fffffff);
                        pos += v[k];
                    }
            }
        }
        at += round;
    }
}

// ---- sorting a tile's range --------------------------------------------------------------------------
// A group of G threads sorts n <= K G entries: the range between the smallest and the largest depth is cut into about n buckets of equal
// width in the bits of the depth, the entries are counted into them (the count's return value is an entry's place inside its bucket),
// a prefix over the buckets places them bucket by bucket in shared memory, and an entry's final place is the start of its bucket plus the
// number of smaller entries in it: a handful of compares where depths are spread, which they are except in constructed scenes. Where some
// bucket holds more than kHeavy entries, a bitonic network sorts the list instead. Issue slots (27 M warp instructions for 4.1 M entries, 59 %) and the
// barriers between the passes bound it: 45 us for 1 M Gaussians at 1296x840 (lists of 967), 157 for 3 M at 1600x1064 (lists of 2,136).
// Up to eight entries per thread stay in registers between the passes; with sixteen (RELOAD) they are read again.
constexpr int kSortThreads = 512, kHeavy = 96, kLongLog = 11;
constexpr int kRoomGroup = 1024, kRoomWarp = 256;
static_assert(kRoomCta == 16 * kSortThreads, "");
struct SortShared {
    uint64_t entry[kRoomCta];
    uint32_t start[kRoomCta / 32 * 33 + 64];      // every group has its own run and four more words (bucket_slot)
    uint32_t cum[(1 << kLongLog) + 1];            // long lists: prefix over the bins
    uint32_t red[2][kSortThreads / 32][2];
    uint64_t red64[2][kSortThreads / 32];
    uint32_t cursor;
};

template <int G>
__device__ __forceinline__ void group_sync(int group) {
    if (G == 32) __syncwarp();
    else if (G == kSortThreads) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(G) : "memory");
}

// Where a bucket's word lies: one word is left out after every 32, so that threads that own runs of 2 to 16 buckets read different banks.
__device__ __forceinline__ uint32_t bucket_slot(uint32_t b) { return b + (b >> 5); }

template <int G, int K, bool RELOAD, class Red, class Load, class Out>
__device__ __forceinline__ void sort_group_k(int tid, int group, int n, uint64_t* entry, uint32_t* __restrict__ start, Red red, Load load, Out out) {
    constexpr int kWarps = G / 32;
    const int lane = tid & 31, warp = tid >> 5;
    uint64_t key[RELOAD ? 1 : K];
    uint32_t rank[K];
    uint32_t lo = 0xFFFFFFFFu, hi = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int i = tid + k * G;
        if (!RELOAD) key[k] = 0;
        if (i < n) {
            const uint64_t x = load(i);
            if (!RELOAD) key[k] = x;
            const uint32_t d = (uint32_t)(x >> 32);
            lo = min(lo, d); hi = max(hi, d);
        }
    }
    // as many buckets as entries, a power of two, at least one per thread
    const int log_b = max(32 - __clz(n - 1), 31 - __clz(G)), buckets = 1 << log_b, per = buckets / G;
    for (int i = tid; i < buckets + buckets / 32; i += G) start[i] = 0;
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (kWarps > 1) {
        if (lane == 0) { red[0][warp][0] = lo; red[0][warp][1] = hi; }
        group_sync<G>(group);
        lo = __reduce_min_sync(0xffffffffu, red[0][lane & (kWarps - 1)][0]);
        hi = __reduce_max_sync(0xffffffffu, red[0][lane & (kWarps - 1)][1]);
    } else {
        __syncwarp();
    }
    const int shift = max(0, 32 - __clz(hi - lo) - log_b);
    auto bucket = [&](uint64_t k) { return ((uint32_t)(k >> 32) - lo) >> shift; };
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int i = tid + k * G;
        rank[k] = 0;
        if (i < n) rank[k] = atomicAdd(&start[bucket_slot(bucket(RELOAD ? load(i) : key[RELOAD ? 0 : k]))], 1u);
    }
    group_sync<G>(group);
    uint32_t sum = 0, most = 0;
#pragma unroll
    for (int j = 0; j < K; ++j)
        if (j < per) {
            const uint32_t c = start[bucket_slot(tid * per + j)];
            sum += c;
            most = max(most, c);
        }
    uint32_t at = (uint32_t)warp_incl_scan((int)sum);
    most = __reduce_max_sync(0xffffffffu, most);
    if (kWarps > 1) {
        if (lane == 31) { red[1][warp][0] = at; red[1][warp][1] = most; }
        group_sync<G>(group);
        const uint32_t v = red[1][lane & (kWarps - 1)][0];
        most = __reduce_max_sync(0xffffffffu, red[1][lane & (kWarps - 1)][1]);
        at += __reduce_add_sync(0xffffffffu, lane < warp ? v : 0u);   // warp < kWarps <= 32 lanes
    }
    at -= sum;
#pragma unroll
    for (int j = 0; j < K; ++j)
        if (j < per) {
            const uint32_t c = start[bucket_slot(tid * per + j)];
            start[bucket_slot(tid * per + j)] = at;
            at += c;
        }
    if (tid == G - 1) start[bucket_slot(buckets)] = (uint32_t)n;
    group_sync<G>(group);
    if (most > (uint32_t)kHeavy) {
        const int width = 1 << (32 - __clz(n - 1));   // n > kHeavy > 1
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int i = tid + k * G;
            if (i < width) entry[i] = i < n ? (RELOAD ? load(i) : key[RELOAD ? 0 : k]) : ~0ull;
        }
        for (int size = 2; size <= width; size <<= 1)
            for (int step = size >> 1; step > 0; step >>= 1) {
                group_sync<G>(group);
                for (int q = tid; q < width / 2; q += G) {
                    const int i = 2 * q - (q & (step - 1)), j = i + step;   // q with a zero bit inserted at `step`
                    const uint64_t a = entry[i], b = entry[j];
                    if ((a > b) == ((i & size) == 0)) { entry[i] = b; entry[j] = a; }
                }
            }
        group_sync<G>(group);
        for (int i = tid; i < n; i += G) out(i, entry[i]);
    } else {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int i = tid + k * G;
            if (i < n) {
                const uint64_t x = RELOAD ? load(i) : key[RELOAD ? 0 : k];
                entry[start[bucket_slot(bucket(x))] + rank[k]] = x;
            }
        }
        group_sync<G>(group);
        for (int i = tid; i < n; i += G) {
            const uint64_t mine = entry[i];
            const uint32_t b = bucket(mine), from = start[bucket_slot(b)], to = start[bucket_slot(b + 1)];
            uint32_t pos = from;
            if (to - from > 1)
                for (uint32_t j = from; j < to; ++j) pos += entry[j] < mine ? 1u : 0u;
            out((int)pos, mine);
        }
    }
    group_sync<G>(group);
}
// n <= 8 G, or 16 G where the entries can be read again. `load` may read `entry` itself unless LONG: every entry is in a register before the first is written.
template <int G, bool LONG, class Load, class Out>
__device__ __forceinline__ void sort_group(int tid, int group, int n, uint64_t* entry, uint32_t* __restrict__ start,
                                           uint32_t (*red)[kSortThreads / 32][2], Load load, Out out) {
    if (n <= 4 * G) sort_group_k<G, 4, false>(tid, group, n, entry, start, red, load, out);
    else if (!LONG || n <= 8 * G) sort_group_k<G, 8, false>(tid, group, n, entry, start, red, load, out);
    else sort_group_k<G, 16, true>(tid, group, n, entry, start, red, load, out);
}

// visit(k) for the entries k of a list, by the whole CTA, eight loads in flight.
template <class List, class Visit>
__device__ __forceinline__ void visit_list(int n, List list, Visit visit) {
    int i = (int)threadIdx.x;
    for (; i + 7 * kSortThreads < n; i += 8 * kSortThreads) {
        uint64_t k[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) k[u] = list(i + u * kSortThreads);
#pragma unroll
        for (int u = 0; u < 8; ++u) visit(k[u]);
    }
    for (; i < n; i += kSortThreads) visit(list(i));
}
constexpr int kLongBins = 1 << kLongLog;
// counts of the keys in [next, top] by (key - next) >> shift, as an exclusive prefix in sm.cum [kLongBins + 1]
template <class List>
__device__ __forceinline__ void long_histogram(int n, List list, SortShared& sm, uint64_t next, uint64_t top, int shift) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int kOwn = kLongBins / kSortThreads;
    __syncthreads();
    for (int i = tid; i < kLongBins; i += kSortThreads) sm.cum[i] = 0;
    __syncthreads();
    visit_list(n, list, [&](uint64_t k) {
        if (k >= next && k <= top) atomicAdd(&sm.cum[(k - next) >> shift], 1u);
    });
    __syncthreads();
    uint32_t c[kOwn], sum = 0;
#pragma unroll
    for (int j = 0; j < kOwn; ++j) { c[j] = sm.cum[tid * kOwn + j]; sum += c[j]; }
    uint32_t at = (uint32_t)warp_incl_scan((int)sum);
    if (lane == 31) sm.red[1][warp][0] = at;
    __syncthreads();
    {
        const uint32_t v = sm.red[1][lane & (kSortThreads / 32 - 1)][0];
        at += __reduce_add_sync(0xffffffffu, lane < warp ? v : 0u) - sum;
    }
#pragma unroll
    for (int j = 0; j < kOwn; ++j) { sm.cum[tid * kOwn + j] = at; at += c[j]; }
    if (tid == kSortThreads - 1) sm.cum[kLongBins] = at;
    __syncthreads();
}
__device__ __forceinline__ int long_shift(uint64_t range) { return max(0, 64 - __clzll((long long)range) - kLongLog); }

// The keys of a list between lo and hi (both included; `count` of them), sorted by the whole CTA: a histogram over 2048 bins of the keys from `next` on (64
// bits, which are all different), then runs of bins that hold up to 4096 entries are gathered into shared memory and sorted. A bin that holds more by
// itself is cut into 2048 again.
template <class List, class Out>
__device__ void sort_long(int n, List list, uint64_t lo, uint64_t hi, int count, SortShared& sm, Out out) {
    constexpr int kRoom = 8 * kSortThreads;
    const int tid = threadIdx.x;
    uint64_t next = lo;   // every smaller key is out
    int done = 0;
    while (done < count) {
        uint64_t top = hi;
        int shift;
        for (;;) {
            shift = long_shift(top - next);
            long_histogram(n, list, sm, next, top, shift);
            // the first bin that holds anything: the last one that starts at 0
            int b = 0;
            for (int step = kLongBins / 2; step > 0; step >>= 1)
                if (sm.cum[b + step] == 0) b += step;
            if (shift == 0 || sm.cum[b + 1] <= (uint32_t)kRoom) break;
            next += (uint64_t)b << shift;
            top = min(top, next + (((uint64_t)1 << shift) - 1));
        }
        int s = 0;
        while (s < kLongBins && done < count) {
            const uint32_t have = sm.cum[s];
            int e = s;   // the last bin boundary within reach
            for (int step = kLongBins; step > 0; step >>= 1)
                if (e + step <= kLongBins && sm.cum[e + step] - have <= (uint32_t)kRoom) e += step;
            if (e == s) {
                if (shift > 0) break;
                // more than 4096 equal keys: not from this file's callers, but the loop has to end
                const int m = (int)(sm.cum[s + 1] - have);
                for (int i = tid; i < m; i += kSortThreads) out(done + i, next + (uint64_t)s);
                done += m;
                ++s;
                continue;
            }
            const int m = (int)(sm.cum[e] - have);
            if (m > 0) {
                if (tid == 0) sm.cursor = 0;
                __syncthreads();
                visit_list(n, list, [&](uint64_t k) {
                    if (k >= next && k <= top) {
                        const int b = (int)((k - next) >> shift);
                        if (b >= s && b < e) sm.entry[min(atomicAdd(&sm.cursor, 1u), (uint32_t)kRoom - 1u)] = k;
                    }
                });
                __syncthreads();
                sort_group<kSortThreads, false>(tid, 0, m, sm.entry, sm.start, sm.red, [&](int i) { return sm.entry[i]; },
                                                [&](int i, uint64_t k) { out(done + i, k); });
                done += m;
            }
            s = e;
        }
        if (s == kLongBins || (uint64_t)s > ((top - next) >> shift)) next = top + 1;   // top == hi: done == count
        else next += (uint64_t)s << shift;
    }
    __syncthreads();
}

// smallest and largest key of a list, to all threads of the CTA
template <class List>
__device__ __forceinline__ void list_bounds(int n, List list, SortShared& sm, uint64_t& lo, uint64_t& hi) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    lo = ~0ull;
    hi = 0;
    visit_list(n, list, [&](uint64_t k) { lo = min(lo, k); hi = max(hi, k); });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (lane == 0) { sm.red64[0][warp] = lo; sm.red64[1][warp] = hi; }
    __syncthreads();
    for (int w = 0; w < kSortThreads / 32; ++w) { lo = min(lo, sm.red64[0][w]); hi = max(hi, sm.red64[1][w]); }
}

// Part q of a list of n entries, by the whole CTA. Every part counts the list's keys into the same bins and takes those that start in its own share of the
// ranks, so the parts need nothing from one another. A call, as sort_far_part: long lists are rare, and inlined they cost the others registers.
template <class List, class Out>
__device__ __noinline__ void sort_part(int q, int n, List list, Out out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SortShared& sm = *reinterpret_cast<SortShared*>(smem_raw);
    const int parts = (n + kPart - 1) / kPart;
    uint64_t lo, hi;
    list_bounds(n, list, sm, lo, hi);
    const int shift = long_shift(hi - lo);
    long_histogram(n, list, sm, lo, hi, shift);
    // first bin that starts at or after the share's first rank
    auto bound = [&](uint32_t rank) {
        int b = 0;   // bins that start before it
        for (int step = kLongBins; step > 0; step >>= 1)
            if (b + step <= kLongBins && sm.cum[b + step - 1] < rank) b += step;
        return b;
    };
    const int from = bound((uint32_t)((int64_t)n * q / parts)), to = q + 1 == parts ? kLongBins : bound((uint32_t)((int64_t)n * (q + 1) / parts));
    const uint32_t first = sm.cum[from], count = sm.cum[to] - first;
    __syncthreads();   // sm.cum is counted anew
    if (count == 0) return;
    const uint64_t key_lo = lo + ((uint64_t)from << shift), key_hi = to == kLongBins ? hi : lo + ((uint64_t)to << shift) - 1;
    sort_long(n, list, key_lo, key_hi, (int)count, sm, [&](int i, uint64_t k) { out((int)first + i, k); });
}

// ---- far lists ------------------------------------------------------------------------------------------
// A list of 65,536 entries and more: 8,192 keys drawn from it and sorted give the limits of 4,096 bins. A cluster counts the list into them, an eighth by
// every CTA, and with the counts of all eight drops the Gaussians into their bins in flatten_ids. Where there are fewer lists than clusters, several share a list:
// each reads all of it, counts what lies below its own share of the bins and places what lies in it. A cluster with a list to itself leaves the bins of the
// keys in the list, so that it searches once. The parts that follow are runs of bins: a sort CTA
// reads its own part only, with the depths fetched by index. Drawn limits, since a key range cut evenly puts most of a distant object between two of them as
// soon as one Gaussian floats near the camera. A bin holds n / 4096 entries, some five times that at the worst.
// Bound by the shared-memory pipe: the search for a key's bin (12 conflicting loads) and the atomics. Sorting, this kernel included, in us, with lists of every
// length read four times by each of their parts and now: 1 M Gaussians, two lists of 632 k 1102 and 338; 1 M at 64x64, four lists of 419 k 4669 and 632; 4 M,
// two of 2.5 M 14654 and 1198; 4 M at 64x64 63446 and 2257. Two lists of 190 k (300 k Gaussians) 183 and 179, which is where the line lies.
constexpr int kFarThreads = 1024, kFarCluster = 8, kFarClusters = 16, kFarBins = 4096;
struct FarShared {
    uint64_t entry[2 * kFarBins];
    uint32_t start[2 * kFarBins / 32 * 33 + 64];
    uint32_t red[2][kFarThreads / 32][2];
    uint64_t limit[kFarBins];        // the first key of bin b + 1
    uint32_t count[kFarBins];        // read by the other CTAs of the cluster
    uint32_t cursor[kFarBins];
    uint32_t first[kFarBins + 1];    // of every bin, from the start of the list
    int scan[33];
    int below;                       // keys before the share, in this CTA's eighth of the list
    int part0;
};
__global__ void __cluster_dims__(kFarCluster, 1, 1) __launch_bounds__(kFarThreads) tile_far_kernel(
    const int32_t* __restrict__ order, const int2* __restrict__ ranges, int4* __restrict__ parts, int32_t* meta,
    uint64_t* entries, const int32_t* __restrict__ overflow, int32_t* __restrict__ flatten_ids) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FarShared& sm = *reinterpret_cast<FarShared*>(smem_raw);
    if (overflow && *overflow) return;
    const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const int tid = threadIdx.x, rank = (int)cluster.block_rank();
    constexpr int kOwn = kFarBins / kFarThreads, kDrawn = 2 * kFarBins, kAhead = 8;
    const int n_far = meta[kMetaFar], clusters = gridDim.x / kFarCluster, shares = max(1, clusters / max(n_far, 1));
    for (int job = blockIdx.x / kFarCluster; job < n_far * shares; job += clusters) {
        const int idx = job / shares, from = ranges[idx].x, n = ranges[idx].y;
        if (n <= kRoomCta) continue;   // cut off by the capacity: sorted like any short list
        uint64_t* list = entries + from;
        // every CTA draws the same keys: one from each of as many stretches of the list
        sort_group_k<kFarThreads, kDrawn / kFarThreads, false>(tid, 0, kDrawn, sm.entry, sm.start, sm.red, [&](int i) {
            const int64_t a = (int64_t)n * i / kDrawn, b = (int64_t)n * (i + 1) / kDrawn;
            return list[a + (int64_t)(((uint64_t)((uint32_t)i * 2654435769u) * (uint64_t)(b - a)) >> 32)];
        }, [&](int i, uint64_t k) { if (i & 1) sm.limit[i >> 1] = k; });
        for (int b = tid; b < kFarBins; b += kFarThreads) sm.count[b] = 0;
        if (tid == 0) sm.below = 0;
        cluster.sync();   // nobody overwrites a key that another CTA still draws
        const int bin0 = kFarBins * (job % shares) / shares, bin1 = kFarBins * (job % shares + 1) / shares;
        const uint64_t key0 = bin0 ? sm.limit[bin0 - 1] : 0, key1 = bin1 < kFarBins ? sm.limit[bin1 - 1] : ~0ull;   // no key has all bits set
        const int lo = (int)((int64_t)n * rank / kFarCluster), hi = (int)((int64_t)n * (rank + 1) / kFarCluster);
        auto bins = [&](int i0, uint64_t (&k)[kAhead], int (&b)[kAhead]) {
#pragma unroll
            for (int u = 0; u < kAhead; ++u) { k[u] = i0 + u * kFarThreads < hi ? list[i0 + u * kFarThreads] : ~0ull; b[u] = 0; }
#pragma unroll
            for (int step = kFarBins / 2; step > 0; step >>= 1)
#pragma unroll
                for (int u = 0; u < kAhead; ++u)
                    if (k[u] >= key0 && k[u] < key1 && sm.limit[b[u] + step - 1] <= k[u]) b[u] += step;
        };
        int below = 0;
        for (int i0 = lo + tid; i0 < hi; i0 += kAhead * kFarThreads) {
            uint64_t k[kAhead];
            int b[kAhead];
            bins(i0, k, b);
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                below += k[u] < key0 ? 1 : 0;
                if (k[u] >= key0 && k[u] < key1) {
                    atomicAdd(&sm.count[b[u]], 1u);
                    if (shares == 1) list[i0 + u * kFarThreads] = (uint64_t)b[u] << 32 | (uint32_t)k[u];   // for this thread, below
                }
            }
        }
        below = __reduce_add_sync(0xffffffffu, below);
        if ((tid & 31) == 0) atomicAdd(&sm.below, below);
        cluster.sync();
        uint32_t all[kOwn], earlier[kOwn], sum = 0;
#pragma unroll
        for (int j = 0; j < kOwn; ++j) {
            all[j] = earlier[j] = 0;
#pragma unroll
            for (int r = 0; r < kFarCluster; ++r) {
                const uint32_t c = cluster.map_shared_rank(sm.count, r)[tid * kOwn + j];
                all[j] += c;
                if (r < rank) earlier[j] += c;
            }
            sum += all[j];
        }
        int base = 0;
#pragma unroll
        for (int r = 0; r < kFarCluster; ++r) base += *cluster.map_shared_rank(&sm.below, r);
        int total;
        uint32_t at = (uint32_t)(base + block_excl_scan((int)sum, total, sm.scan));
#pragma unroll
        for (int j = 0; j < kOwn; ++j) {
            sm.first[tid * kOwn + j] = at;
            sm.cursor[tid * kOwn + j] = at + earlier[j];
            at += all[j];
        }
        const int n_parts = (total + kPart - 1) / kPart;
        if (tid == 0) {
            sm.first[kFarBins] = (uint32_t)(base + total);
            if (rank == 0) sm.part0 = atomicAdd(meta + kMetaParts, n_parts);
        }
        cluster.sync();   // the counts of the other CTAs have been read
        for (int i0 = lo + tid; i0 < hi; i0 += kAhead * kFarThreads) {
            uint64_t k[kAhead];
            int b[kAhead];
            if (shares == 1) {
#pragma unroll
                for (int u = 0; u < kAhead; ++u) { k[u] = i0 + u * kFarThreads < hi ? list[i0 + u * kFarThreads] : ~0ull; b[u] = (int)(k[u] >> 32); }
            } else {
                bins(i0, k, b);
            }
#pragma unroll
            for (int u = 0; u < kAhead; ++u)
                if (k[u] >= key0 && k[u] < key1) flatten_ids[from + (int)atomicAdd(&sm.cursor[b[u]], 1u)] = (int32_t)(uint32_t)k[u];
        }
        if (rank == 0) {
            // first bin that starts at or after a rank of the share
            auto bound = [&](int64_t r) {
                int b = 0;
                for (int step = kFarBins; step > 0; step >>= 1)
                    if (b + step <= kFarBins && (int64_t)sm.first[b + step - 1] - base < r) b += step;
                return b;
            };
            for (int q = tid; q < n_parts; q += kFarThreads) {
                const int b0 = bound((int64_t)total * q / n_parts), b1 = q + 1 == n_parts ? kFarBins : bound((int64_t)total * (q + 1) / n_parts);
                parts[sm.part0 + q] = make_int4(from + (int)sm.first[b0], (int)(sm.first[b1] - sm.first[b0]), order[idx], -1);
            }
        }
        __syncthreads();
    }
}

// n Gaussians of a far list, by the whole CTA, sorted where they lie. `room`: n entries that nobody needs any more.
template <class Out>
__device__ __noinline__ void sort_far_part(int n, const int32_t* ids, const uint32_t* __restrict__ keys, uint64_t* room, Out out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SortShared& sm = *reinterpret_cast<SortShared*>(smem_raw);
    auto load = [&](int i) {
        const uint32_t id = (uint32_t)ids[i];
        return (uint64_t)keys[id] << 32 | id;
    };
    if (n <= kRoomCta) {
        if (n > 0) sort_group<kSortThreads, true>(threadIdx.x, 0, n, sm.entry, sm.start, sm.red, load, out);
        return;
    }
    // bins of a list of ten million and more
    for (int i = threadIdx.x; i < n; i += kSortThreads) __stcg(reinterpret_cast<unsigned long long*>(room + i), (unsigned long long)load(i));
    __syncthreads();
    auto list = [&](int i) { return (uint64_t)__ldcg(reinterpret_cast<const unsigned long long*>(room + i)); };
    uint64_t lo, hi;
    list_bounds(n, list, sm, lo, hi);
    sort_long(n, list, lo, hi, n, sm, out);
}

// Groups of G threads share lists first .. last - 1 of the launch order: a round gives one list to every group, the longest to the first group of every
// CTA, then to the second ones, and every other round runs backwards. (By ticket, thousands of groups queue for one counter: 30 us instead of 15 on
// the smallest scenes.) The range of the next list is on its way while one is sorted.
template <int G, class Body>
__device__ __forceinline__ void share_lists(int tid, int group, int first, int last, const int2* __restrict__ ranges, Body body) {
    const int groups = (int)gridDim.x * (kSortThreads / G), mine = group * (int)gridDim.x + (int)blockIdx.x;
    auto list = [&](int round) { return first + round * groups + (round & 1 ? groups - 1 - mine : mine); };
    int2 r = make_int2(0, 0);
    if (list(0) < last) r = ranges[list(0)];
    for (int round = 0; first + round * groups < last; ++round) {
        const int idx = list(round), after = list(round + 1);
        const int2 now = r;
        if (after < last) r = ranges[after];
        if (idx < last && now.y > 0) body(idx, now.x, now.y);
    }
}

// OP: operator level, with the 64-bit keys. keys: depth bits by flattened Gaussian index.
template <bool OP>
__global__ void __launch_bounds__(kSortThreads, 2) tile_sort_kernel(const int32_t* __restrict__ order, const int2* __restrict__ ranges, const int4* __restrict__ parts,
                                                                    const int32_t* __restrict__ meta, const uint32_t* __restrict__ keys,
                                                                    uint64_t* entries, const int32_t* __restrict__ overflow,
                                                                    int64_t first_bin, uint32_t n_tiles, uint32_t tile_n_bits,
                                                                    int32_t* __restrict__ flatten_ids, int64_t* __restrict__ isect_ids) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SortShared& sm = *reinterpret_cast<SortShared*>(smem_raw);
    if (overflow && *overflow) return;
    const int tid = threadIdx.x;
    auto writer = [&](int bin, int from) {
        const int64_t id = OP ? first_bin + bin : 0;
        const int64_t tile_key = OP ? (id / n_tiles << tile_n_bits | id % n_tiles) << 32 : 0;
        return [=](int i, uint64_t k) {
            flatten_ids[from + i] = (int32_t)(uint32_t)k;
            if (OP) isect_ids[from + i] = tile_key | (int64_t)(k >> 32);
        };
    };
    const int n_cta = meta[kMetaLists], n_group = meta[kMetaLists + 1], n_warp = meta[kMetaLists + 2];
    for (int u = blockIdx.x, n_parts = meta[kMetaParts]; u < n_parts; u += gridDim.x) {
        const int4 part = parts[u];
        if (part.w < 0) sort_far_part(part.y, flatten_ids + part.x, keys, entries + part.x, writer(part.z, part.x));
        else sort_part(part.w, part.y, [list = entries + part.x](int i) { return list[i]; }, writer(part.z, part.x));
        __syncthreads();
    }
    share_lists<kSortThreads>(tid, 0, 0, n_cta, ranges, [&](int idx, int from, int n) {
        if (n <= kRoomCta)
            sort_group<kSortThreads, true>(tid, 0, n, sm.entry, sm.start, sm.red, [&](int i) { return entries[from + i]; }, writer(OP ? order[idx] : 0, from));
    });
    __syncthreads();
    {
        const int group = tid / 128, t = tid % 128;
        uint32_t (*red)[kSortThreads / 32][2] = reinterpret_cast<uint32_t (*)[kSortThreads / 32][2]>(&sm.red[0][group * 4][0]);
        share_lists<128>(t, group, n_cta, n_group, ranges, [&](int idx, int from, int n) {
            sort_group<128, false>(t, group, n, sm.entry + group * kRoomGroup, sm.start + group * (kRoomGroup / 32 * 33 + 4), red,
                                   [&](int i) { return entries[from + i]; }, writer(OP ? order[idx] : 0, from));
        });
    }
    __syncthreads();
    {
        const int group = tid / 32, t = tid % 32;
        share_lists<32>(t, group, n_group, n_warp, ranges, [&](int idx, int from, int n) {
            sort_group<32, false>(t, group, n, sm.entry + group * kRoomWarp, sm.start + group * (kRoomWarp / 32 * 33 + 4), sm.red,
                                  [&](int i) { return entries[from + i]; }, writer(OP ? order[idx] : 0, from));
        });
    }
}

// Operator-level intersect_offset on 64-bit keys.
__global__ void __launch_bounds__(kThreads) isect_offset_kernel(int64_t n, const int64_t* __restrict__ isect_ids, int64_t n_ids,
                                                                uint32_t n_tiles, uint32_t tile_n_bits,
                                                                int32_t* __restrict__ offsets) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n == 0) {
        for (int64_t i = tid; i < n_ids; i += stride) offsets[i] = 0;
        return;
    }
    const int64_t tmask = ((int64_t)1 << tile_n_bits) - 1;
    for (int64_t i = tid; i < n; i += stride) {
        const int64_t cur = isect_ids[i] >> 32;
        const int64_t id_curr = (cur >> tile_n_bits) * n_tiles + (cur & tmask);
        if (i == 0)
            for (int64_t t = 0; t <= id_curr && t < n_ids; ++t) offsets[t] = 0;
        if (i == n - 1)
            for (int64_t t = id_curr + 1; t < n_ids; ++t) offsets[t] = (int32_t)n;
        if (i > 0) {
            const int64_t prev = isect_ids[i - 1] >> 32;
            if (prev != cur) {
                const int64_t id_prev = (prev >> tile_n_bits) * n_tiles + (prev & tmask);
                for (int64_t t = id_prev + 1; t <= id_curr && t < n_ids; ++t) offsets[t] = (int32_t)i;
            }
        }
    }
}

__global__ void __launch_bounds__(kThreads) sum_i32_kernel(int64_t n, const int32_t* __restrict__ src, unsigned long long* out) {
    long long s = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) s += src[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0 && s) atomicAdd(out, (unsigned long long)s);
}

}  // namespace

int exclusive_scan(const int32_t* src, int64_t n, int32_t* out, int32_t* total_dev, const SortScratch& s, cudaStream_t st) {
    if (n <= 0) {
        if (total_dev) cudaMemsetAsync(total_dev, 0, sizeof(int32_t), st);
        return LFS_OK;
    }
    int nb = (int)((n + kTile - 1) / kTile);
    nb = min(nb, min(4 * num_sms(), kScanBlocks));
    const int64_t chunk = (n + nb - 1) / nb;
    LFS_TIMED("exclusive_scan", st);
    scan_reduce_kernel<<<nb, kThreads, 0, st>>>(src, n, chunk, s.block_sums);
    scan_block_sums_kernel<<<1, 1024, 0, st>>>(s.block_sums, nb, total_dev);
    scan_apply_kernel<<<nb, kThreads, 0, st>>>(src, n, chunk, s.block_sums, out);
    return check_launch("exclusive_scan");
}

static uint32_t bit_width_u32(uint32_t v) {
    uint32_t b = 0;
    while (v) { ++b; v >>= 1; }
    return b;
}

// ---- list state: kMetaWords | carry (int64) | counts [replicas][stride] | cursors [replicas][stride] | order [bins] | ranges [bins] | offsets [bins + 1] | parts --------
namespace {
int64_t pad8(int64_t n) { return (n + 7) / 8 * 8; }
// Counters of neighbouring tiles share a 32-byte sector, and the memory system applies one request to a sector at a time: some 12 cycles each.
// On small images, where a tile has thousands of instances, that is a queue, so the counters exist several times and Gaussians take them
// in turn, 32 at a time; up to 16 sets and 65,536 counters (more cost the scan what they save, and tear a tile's entries apart). Scatter in us with one set of counters and now: 150 k Gaussians at
// 640x360 47 and 15, 1 M at 1296x840 116 and 58, 6 M 180 degree fisheye at 1920x1920 322 and 174; counting them inside the projection 33 and 3, 20 and 15.
int list_replicas(int64_t bins) {
    int r = 1;
    while (r < 16 && bins * r * 2 <= 65536) r *= 2;
    return r;
}
struct ListState {
    int32_t *meta, *order, *offsets;
    int64_t* carry;
    int2* ranges;
    int4* parts;   // [capacity / kPart + capacity / kRoomCta + 1 + kFarClusters]
    TileCounters t;
};
ListState list_state(int32_t* base, int64_t bins) {
    ListState s;
    s.meta = base;
    s.carry = reinterpret_cast<int64_t*>(base + kMetaWords);
    s.t.replicas = list_replicas(bins);
    s.t.stride = (int32_t)pad8(bins);
    s.t.counts = base + kMetaWords + 16;
    s.t.cursors = s.t.counts + (size_t)s.t.replicas * s.t.stride;
    s.order = s.t.cursors + (size_t)s.t.replicas * s.t.stride;
    s.ranges = reinterpret_cast<int2*>(s.order + pad8(bins));
    s.offsets = s.order + 3 * pad8(bins);
    s.parts = reinterpret_cast<int4*>(s.offsets + pad8(bins + 1));
    return s;
}
// a list of n > kRoomCta entries has at most n / kPart + 1 parts, one more for every further cluster that shares it, and there are at most capacity / kRoomCta such
// lists
size_t list_words(int64_t bins, int64_t counters, int64_t capacity) {
    return (size_t)(kMetaWords + 16 + 2 * counters + 3 * pad8(bins) + pad8(bins + 1) + 4 * (capacity / kPart + capacity / kRoomCta + 1 + kFarClusters));
}
}  // namespace

size_t tile_list_state_words(int64_t bins, int64_t capacity) { return list_words(bins, list_replicas(bins) * pad8(bins), capacity); }
TileCounters tile_list_counters(int32_t* state, int64_t bins) { return list_state(state, bins).t; }
const int32_t* tile_list_order(const int32_t* state, int64_t bins) { return list_state(const_cast<int32_t*>(state), bins).order; }
int clear_tile_counters(const TileCounters& t, cudaStream_t st) {
    return cudaMemsetAsync(t.counts, 0, (size_t)t.replicas * t.stride * sizeof(int32_t), st) == cudaSuccess ? LFS_OK : LFS_ECUDA;
}

static int launch_tile_scan(int bins, const ListState& s, int64_t capacity, int64_t* carry, int32_t* n_out, int32_t* overflow, int32_t* offsets, bool far_lists,
                            cudaStream_t st) {
    LFS_TIMED("tile_scan", st);
    tile_scan_kernel<<<kScanCluster, 1024, 0, st>>>(bins, s.t, capacity, carry, n_out, overflow, offsets, s.order, s.ranges, s.parts, s.meta, far_lists);
    return check_launch("tile_scan");
}

// A list holds a Gaussian once, so only many Gaussians make a list long enough for tile_far_kernel to pay; where there is none it costs a launch of 2 us.
static bool far_lists_possible(int64_t N) { return N > 262144; }

template <bool OP>
static int launch_tile_sort(int bins, const ListState& s, const uint32_t* keys, uint64_t* entries, const int32_t* overflow, int64_t first_bin, uint32_t n_tiles,
                            uint32_t tile_n_bits, int32_t* flatten_ids, int64_t* isect_ids, bool far_lists, cudaStream_t st) {
    if (far_lists) {
        LFS_TIMED("tile_far", st);
        cudaFuncSetAttribute(tile_far_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FarShared));
        tile_far_kernel<<<kFarClusters * kFarCluster, kFarThreads, sizeof(FarShared), st>>>(s.order, s.ranges, s.parts, s.meta, entries, overflow, flatten_ids);
    }
    LFS_TIMED("tile_sort", st);
    cudaFuncSetAttribute(tile_sort_kernel<OP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SortShared));
    tile_sort_kernel<OP><<<min(bins, 2 * num_sms()), kSortThreads, sizeof(SortShared), st>>>(s.order, s.ranges, s.parts, s.meta, keys, entries, overflow, first_bin,
                                                                                             n_tiles, tile_n_bits, flatten_ids, isect_ids);
    return check_launch("tile_sort");
}

// Warps per 32 Gaussians, where four or more of them still fit the GPU with eight CTAs per SM: of few Gaussians on a large image each has hundreds of tiles
// (11 k at 2790x1646, 160 each: scatter 102 -> 24 us; 60 k, EWA, 777x519: 16.8 -> 12.9).
static int scatter_parts(int64_t total) {
    const int64_t parts = (int64_t)64 * num_sms() / max((total + 31) / 32, (int64_t)1);
    return parts < 4 ? 1 : (int)min(parts, (int64_t)8);
}
// The per-Gaussian stage has one warp per 32 Gaussians, so where scatter_parts takes more and the image is large beside the Gaussians' number the
// counting gets a launch of its own (the same scene: projection 77 us, of which 61 went into the counting; 77 -> 16 and 17 for the launch). Render of 3 k, 10 k and 60 k
// Gaussians, counted in the projection and apart, us: 4,293 tiles, 10 and 40 tiles a Gaussian: 84 and 86, 110 and 112, 199 and 205; 244 and 190, 288 and 234, 535 and 503;
// 18,025 tiles: 180 and 173, 267 and 259, 556 and 554; 824 and 565, 1002 and 746, 428 and 264. It costs 7 us at most and saves up to 260.
bool count_tiles_apart(int64_t N, int64_t bins) { return scatter_parts(N) > 1 && 8 * bins >= N; }

int build_tile_lists(const TileListArgs& a, cudaStream_t st) {
    const int parts = scatter_parts(a.N);
    const int bins = a.tw * a.th;
    const ListState s = list_state(a.state, bins);
    if (a.count && a.N > 0) {
        LFS_TIMED("tile_histogram", st);
        tile_histogram_kernel<<<grid_for((int64_t)a.N * parts, kThreads), kThreads, 0, st>>>(a.N, a.N, a.tw, a.th, (float)a.tile_size, a.tiles, a.means2d,
                                                                                            a.radii, 0, bins, s.t, parts);
    }
    const bool far_lists = far_lists_possible(a.N);
    int rc = launch_tile_scan(bins, s, a.capacity, nullptr, a.n_isects_dev, a.overflow, a.tile_offsets, far_lists, st);
    if (rc != LFS_OK) return rc;
    if (a.N > 0 && a.capacity > 0 && bins > 0) {
        {
            LFS_TIMED("tile_scatter", st);
            if (a.ewa_bounds)
                ewa_scatter_kernel<<<grid_for((int64_t)a.N * parts, kThreads), kThreads, 0, st>>>(a.N, a.tw, a.tiles, a.ewa_bounds, a.ewa_masks, a.ewa_records, a.ewa_depth_bits,
                                                                                 bins, a.capacity, a.overflow, s.t, a.entries, parts);
            else
                tile_scatter_kernel<<<grid_for((int64_t)a.N * parts, kThreads), kThreads, 0, st>>>(a.N, a.N, a.tw, a.th, (float)a.tile_size, a.tiles, a.means2d, a.radii,
                                                                                  a.depths, 0, bins, a.capacity, a.overflow, s.t, a.entries, parts);
        }
        const uint32_t* keys = a.ewa_bounds ? a.ewa_depth_bits : reinterpret_cast<const uint32_t*>(a.depths);
        rc = launch_tile_sort<false>(bins, s, keys, a.entries, a.overflow, 0, 1, 0, a.flatten_ids, nullptr, far_lists, st);
        if (rc != LFS_OK) return rc;
    }
    return check_launch("build_tile_lists");
}

// Operator level. The grid is not known to the workspace query, so the per-bin arrays hold kOperatorBins bins and larger grids take
// several rounds.
constexpr int64_t kOperatorBins = 1 << 17;

size_t isect_lists_bytes(int64_t total, int64_t n_isects, IsectBuffers* b, void* base) {
    size_t off = 0;
    auto take = [&](size_t bytes) {
        off = (off + 255) & ~(size_t)255;
        void* p = base ? reinterpret_cast<char*>(base) + off : nullptr;
        off += bytes;
        return p;
    };
    IsectBuffers x;
    // any number of bins up to kOperatorBins, each with its replicas: 65,536 counters and the padding of 16 sets, or one set
    x.state = (int32_t*)take(list_words(kOperatorBins, kOperatorBins + 8 * 16, n_isects) * sizeof(int32_t));
    x.scratch.block_sums = (uint32_t*)take((kScanBlocks + 1) * sizeof(uint32_t));
    // sorted: the entries; unsorted: the prefix over the Gaussians
    const size_t entries = (size_t)n_isects * sizeof(uint64_t), prefix = (size_t)total * sizeof(int32_t);
    void* p = take(entries > prefix ? entries : prefix);
    x.entries = (uint64_t*)p;
    x.prefix = (int32_t*)p;
    if (b) *b = x;
    return (off + 255) & ~(size_t)255;
}

int build_isect_lists(int C, int N, int tw, int th, int tile_size, int sort, const float* means2d, const int32_t* radii, const float* depths,
                      const int32_t* tiles, int64_t n_isects, const IsectBuffers& b, int64_t* isect_ids, int32_t* flatten_ids, cudaStream_t st) {
    const int64_t total = (int64_t)C * N, n_ids = (int64_t)C * tw * th;
    const uint32_t n_tiles = (uint32_t)tw * th, tile_n_bits = bit_width_u32(n_tiles);
    if (tile_n_bits + bit_width_u32((uint32_t)C) > 32) {
        set_error("build_isect_lists: tile and camera ids need more than 32 bits");
        return LFS_EINVAL;
    }
    const int parts = scatter_parts(total), grid = grid_for(total * parts, kThreads);
    if (!sort) {
        const int rc = exclusive_scan(tiles, total, b.prefix, nullptr, b.scratch, st);
        if (rc != LFS_OK) return rc;
        LFS_TIMED("emit_unsorted", st);
        emit_unsorted_kernel<<<grid, kThreads, 0, st>>>(total, N, tw, th, (float)tile_size, tile_n_bits, tiles, b.prefix, means2d, radii, depths, n_isects,
                                                        isect_ids, flatten_ids);
        return check_launch("emit_unsorted");
    }
    const bool far_lists = far_lists_possible(N);
    cudaMemsetAsync(list_state(b.state, 1).carry, 0, sizeof(int64_t), st);
    for (int64_t first = 0; first < n_ids; first += kOperatorBins) {
        const int bins = (int)min(kOperatorBins, n_ids - first);
        const ListState s = list_state(b.state, bins);
        if (clear_tile_counters(s.t, st) != LFS_OK) { set_error("build_isect_lists: memset failed"); return LFS_ECUDA; }
        {
            LFS_TIMED("tile_histogram", st);
            tile_histogram_kernel<<<grid, kThreads, 0, st>>>(total, N, tw, th, (float)tile_size, tiles, means2d, radii, first, bins, s.t, parts);
        }
        int rc = launch_tile_scan(bins, s, n_isects, s.carry, nullptr, nullptr, s.offsets, far_lists, st);
        if (rc != LFS_OK) return rc;
        {
            LFS_TIMED("tile_scatter", st);
            tile_scatter_kernel<<<grid, kThreads, 0, st>>>(total, N, tw, th, (float)tile_size, tiles, means2d, radii, depths, first, bins, n_isects, nullptr,
                                                           s.t, b.entries, parts);
        }
        rc = launch_tile_sort<true>(bins, s, reinterpret_cast<const uint32_t*>(depths), b.entries, nullptr, first, n_tiles, tile_n_bits, flatten_ids, isect_ids,
                                    far_lists, st);
        if (rc != LFS_OK) return rc;
    }
    return check_launch("build_isect_lists");
}

int launch_isect_offset(int64_t n, const int64_t* isect_ids, int C, int tw, int th, int32_t* offsets, cudaStream_t st) {
    const uint32_t n_tiles = (uint32_t)tw * th;
    const int64_t n_ids = (int64_t)C * n_tiles;
    isect_offset_kernel<<<grid_for(n > 0 ? n : n_ids, 256), 256, 0, st>>>(n, isect_ids, n_ids, n_tiles,
                                                                          bit_width_u32(n_tiles), offsets);
    return check_launch("isect_offset");
}

int launch_sum_i32(int64_t n, const int32_t* src, int64_t* out_dev, cudaStream_t st) {
    cudaMemsetAsync(out_dev, 0, sizeof(int64_t), st);
    if (n > 0) sum_i32_kernel<<<grid_for(n, 256), 256, 0, st>>>(n, src, reinterpret_cast<unsigned long long*>(out_dev));
    return check_launch("sum_i32");
}

}  // namespace lfs
