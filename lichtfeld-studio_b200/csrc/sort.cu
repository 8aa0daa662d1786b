// Tile-list construction: prefix sums, a stable LSD radix sort on (uint32 key, uint32 value) pairs,
// instance emission and per-tile offsets.
//
// Replaces gsplat/IntersectTile.cu:24 (second pass), the at::cumsum + CUB DeviceRadixSort::SortPairs
// call of gsplat/Intersect.cpp:75 / gsplat/IntersectTile.cu:290-328, and gsplat/IntersectTile.cu:206.
//
// The reference sorts n_isects 12-byte (int64 key, int32 value) pairs over 32 + tile_bits + cam_bits
// bits. The same order (camera, tile, depth bits, ties by ascending flattened Gaussian index) is
// produced here with far less traffic: the Gaussians are sorted once by their 32 depth bits, the
// instances are emitted in that order, and a stable sort on the (camera, tile) key alone finishes.
// All passes are HBM-bound integer work; nothing here is shaped for tensor cores. Prefixes over the tiles of a list travel by
// decoupled look-back (Merrill and Garland) inside the kernel that uses them, so a short sort is one histogram kernel and one
// kernel per digit, and the prefix over the Gaussians' tile counts and the emission of their instances are one kernel: 9 launches
// where separate histogram, scan and scatter kernels took 22.
#include "gsmath.cuh"
#include "sort.cuh"
#include "ewa_common.cuh"

namespace lfs {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 8;
constexpr int kTile = kThreads * kItems;

__device__ __forceinline__ int warp_incl_scan(int v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) >= o) v += t;
    }
    return v;
}

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

__device__ __forceinline__ int64_t device_count(const int32_t* n_dev, int64_t n_max) {
    if (n_dev == nullptr) return n_max;
    int64_t n = *n_dev;
    if (n > n_max) n = n_max;
    if (n < 0) n = 0;
    return n;
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

// ---- decoupled look-back ------------------------------------------------------------------------
// One word per list tile (and digit): 0 = nothing yet, top bit clear = the tile's own count + 1, top bit set = the count of this
// and all earlier tiles. Value and flag share the word, so relaxed accesses are enough. Tiles are numbered by a ticket, so every
// predecessor of a tile belongs to a CTA that is already running and publishes its own count without waiting for anybody:
// each wait ends. The poll limit only bounds the damage of a defect: it raises a flag, after which nobody reads the list, and every
// store below checks its position.
constexpr uint32_t kInclusive = 0x80000000u;
constexpr int kPollLimit = 1 << 21;

__device__ __forceinline__ uint32_t ld_state(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_state(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// ---- radix sort -------------------------------------------------------------------------------
// Digit counts of all passes in one read of the keys; zeroes the look-back words of the passes that follow.
__global__ void __launch_bounds__(kThreads) radix_hist_kernel(const uint32_t* __restrict__ keys, const int32_t* n_dev,
                                                              int64_t n_max, int bits, int passes,
                                                              uint32_t* __restrict__ hist, uint4* __restrict__ state,
                                                              int64_t pass_stride4) {
    __shared__ uint32_t h[4][256];
    const int64_t n = device_count(n_dev, n_max);
    const int64_t tid = (int64_t)blockIdx.x * kThreads + threadIdx.x, stride = (int64_t)gridDim.x * kThreads;
    const int64_t n_words4 = (n + kTile - 1) / kTile * 64;
    for (int p = 0; p < passes; ++p)
        for (int64_t i = tid; i < n_words4; i += stride) state[p * pass_stride4 + i] = make_uint4(0u, 0u, 0u, 0u);
    for (int p = 0; p < 4; ++p) h[p][threadIdx.x] = 0;
    __syncthreads();
    const uint32_t mask = (1u << bits) - 1u;
    for (int64_t i = tid; i < n; i += stride) {
        const uint32_t k = keys[i];
        for (int p = 0; p < passes; ++p) atomicAdd(&h[p][(k >> (p * bits)) & mask], 1u);
    }
    __syncthreads();
    for (int p = 0; p < passes; ++p)
        if (h[p][threadIdx.x]) atomicAdd(&hist[p * 256 + threadIdx.x], h[p][threadIdx.x]);
}

// Long lists: one digit count per CTA and pass over its chunk of the list (row d of a digit-major table), ...
__global__ void __launch_bounds__(kThreads) radix_count_kernel(const uint32_t* __restrict__ keys, const int32_t* n_dev,
                                                               int64_t n_max, int shift, uint32_t mask, int nb,
                                                               uint32_t* __restrict__ table) {
    __shared__ uint32_t h[256];
    const int64_t n = device_count(n_dev, n_max);
    const int64_t chunk = (n + nb - 1) / nb;
    const int64_t lo = (int64_t)blockIdx.x * chunk, hi = min(n, lo + chunk);
    h[threadIdx.x] = 0;
    __syncthreads();
    for (int64_t i = lo + threadIdx.x; i < hi; i += kThreads) atomicAdd(&h[(keys[i] >> shift) & mask], 1u);
    __syncthreads();
    table[(size_t)threadIdx.x * nb + blockIdx.x] = h[threadIdx.x];
}

// ... and one CTA per digit: exclusive scan of that digit's counts and the digit total.
__global__ void __launch_bounds__(kThreads) radix_scan_kernel(uint32_t* __restrict__ table, int nb, uint32_t* __restrict__ digit_totals) {
    __shared__ int sm[33];
    uint32_t* row = table + (size_t)blockIdx.x * nb;
    int carry = 0;
    for (int base = 0; base < nb; base += kThreads) {
        const int i = base + threadIdx.x;
        const int v = i < nb ? (int)row[i] : 0;
        int total;
        const int ex = block_excl_scan(v, total, sm);
        if (i < nb) row[i] = (uint32_t)(carry + ex);
        carry += total;
    }
    if (threadIdx.x == 0) digit_totals[blockIdx.x] = (uint32_t)carry;
}

// Scatter of the chunked pass: the CTA walks its chunk in tiles of 2048 pairs. Every item gets its rank among the equal digits
// of the tile (warp match + per-warp counters), the tile is reordered by digit in shared memory, and consecutive threads write
// consecutive addresses of each digit's output run, so the global stores are contiguous runs instead of 4-byte scatters.
__global__ void __launch_bounds__(kThreads) radix_scatter_chunk_kernel(
    const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in, uint32_t* __restrict__ keys_out,
    uint32_t* __restrict__ vals_out, const int32_t* n_dev, int64_t n_max, int shift, uint32_t mask, int nb,
    const uint32_t* __restrict__ table, const uint32_t* __restrict__ digit_totals) {
    __shared__ uint32_t cnt[kWarps][256];   // per-warp digit counts, then per-warp start inside the tile
    __shared__ uint32_t gbase[256];         // where the next item of digit d from this CTA goes
    __shared__ uint32_t tstart[256];        // start of digit d inside the reordered tile
    __shared__ uint32_t skeys[kTile], svals[kTile];
    __shared__ int sm[33];
    const int64_t n = device_count(n_dev, n_max);
    const int64_t chunk = (n + nb - 1) / nb;
    const int64_t lo = (int64_t)blockIdx.x * chunk, hi = min(n, lo + chunk);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt_mask = (1u << lane) - 1u;
    {
        // start of digit d = totals of the smaller digits + this digit's counts in the earlier blocks
        int total;
        const int digit_base = block_excl_scan((int)digit_totals[threadIdx.x], total, sm);
        gbase[threadIdx.x] = (uint32_t)digit_base + table[(size_t)threadIdx.x * nb + blockIdx.x];
    }
    for (int64_t tile_lo = lo; tile_lo < hi; tile_lo += kTile) {
        const int tile_n = (int)min((int64_t)kTile, hi - tile_lo);
#pragma unroll
        for (int w = 0; w < kWarps; ++w) cnt[w][threadIdx.x] = 0;
        __syncthreads();
        uint32_t key[kItems], val[kItems], rank[kItems];
        const int64_t wbase = tile_lo + (int64_t)warp * (32 * kItems);
#pragma unroll
        for (int r = 0; r < kItems; ++r) {
            const int64_t i = wbase + r * 32 + lane;
            const bool ok = i < hi;
            key[r] = ok ? keys_in[i] : 0u;
            val[r] = ok ? vals_in[i] : 0u;
        }
#pragma unroll
        for (int r = 0; r < kItems; ++r) {
            const int64_t i = wbase + r * 32 + lane;
            const bool ok = i < hi;
            const uint32_t d = ok ? ((key[r] >> shift) & mask) : 0xFFFFFFFFu;
            const uint32_t peers = __match_any_sync(0xffffffffu, d);
            uint32_t prev = 0;
            if (ok) prev = cnt[warp][d];
            __syncwarp();
            if (ok && (peers & lt_mask) == 0) cnt[warp][d] = prev + __popc(peers);
            __syncwarp();
            rank[r] = prev + __popc(peers & lt_mask);
        }
        __syncthreads();
        {
            // digit threadIdx.x: exclusive prefix over the warps and the digit's total in this tile
            uint32_t run = 0;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                const uint32_t c = cnt[w][threadIdx.x];
                cnt[w][threadIdx.x] = run;
                run += c;
            }
            int total;
            const int start = block_excl_scan((int)run, total, sm);  // start of this digit inside the tile
            tstart[threadIdx.x] = (uint32_t)start;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) cnt[w][threadIdx.x] += (uint32_t)start;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kItems; ++r) {
            const int64_t i = wbase + r * 32 + lane;
            if (i < hi) {
                const uint32_t d = (key[r] >> shift) & mask;
                const uint32_t pos = cnt[warp][d] + rank[r];
                skeys[pos] = key[r];
                svals[pos] = val[r];
            }
        }
        __syncthreads();
        // write out: item j of the reordered tile belongs to digit d = digit(skeys[j]) and goes to
        // gbase[d] + (j - tstart[d]); neighbouring j of one digit are neighbouring addresses
#pragma unroll
        for (int r = 0; r < kItems; ++r) {
            const int j = r * kThreads + threadIdx.x;
            if (j < tile_n) {
                const uint32_t k = skeys[j];
                const uint32_t d = (k >> shift) & mask;
                const uint32_t pos = gbase[d] + ((uint32_t)j - tstart[d]);
                keys_out[pos] = k;
                vals_out[pos] = svals[j];
            }
        }
        __syncthreads();
        {
            // advance the global bases by this tile's digit totals
            const uint32_t next = threadIdx.x + 1 < 256 ? tstart[threadIdx.x + 1] : (uint32_t)tile_n;
            gbase[threadIdx.x] += next - tstart[threadIdx.x];
        }
        __syncthreads();
    }
}

// Stable scatter of one radix pass. A CTA takes tiles of 2048 pairs by ticket: every item gets its rank among the equal
// digits of the tile (warp match + per-warp counters), the tile's digit counts are published, the tile is reordered by
// digit in shared memory, the counts of the earlier tiles are looked up (one thread per digit, four tiles at a time), and then
// consecutive threads write consecutive addresses of each digit's output run.
__global__ void __launch_bounds__(kThreads) radix_scatter_kernel(
    const uint32_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in, uint32_t* __restrict__ keys_out,
    uint32_t* __restrict__ vals_out, const int32_t* n_dev, int64_t n_max, int shift, uint32_t mask,
    const uint32_t* __restrict__ hist, uint32_t* ticket, uint32_t* state, int32_t* gave_up) {
    __shared__ uint32_t cnt[kWarps][256];   // per-warp digit counts, then per-warp start inside the tile
    __shared__ uint32_t gbase[256];         // where the items of digit d of this tile go
    __shared__ uint32_t tstart[256];        // start of digit d inside the reordered tile
    __shared__ uint32_t skeys[kTile], svals[kTile];
    __shared__ int sm[33];
    __shared__ uint32_t s_tile;
    const int64_t n = device_count(n_dev, n_max);
    const uint32_t n_list_tiles = (uint32_t)((n + kTile - 1) / kTile);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint32_t digit_base;   // start of digit threadIdx.x in the output: totals of the smaller digits
    {
        int total;
        digit_base = (uint32_t)block_excl_scan((int)hist[threadIdx.x], total, sm);
    }
    for (;;) {
        if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
#pragma unroll
        for (int w = 0; w < kWarps; ++w) cnt[w][threadIdx.x] = 0;
        __syncthreads();
        const uint32_t tile = s_tile;
        if (tile >= n_list_tiles) break;
        const int64_t tile_lo = (int64_t)tile * kTile;
        const int tile_n = (int)min((int64_t)kTile, n - tile_lo);
        uint32_t key[kItems], val[kItems], rank[kItems];
        const int wbase = warp * (32 * kItems);
#pragma unroll
        for (int r = 0; r < kItems; ++r) {
            const int i = wbase + r * 32 + lane;
            const bool ok = i < tile_n;
            key[r] = ok ? keys_in[tile_lo + i] : 0u;
            val[r] = ok ? vals_in[tile_lo + i] : 0u;
        }
#pragma unroll
        for (int r = 0; r < kItems; ++r) {
            const bool ok = wbase + r * 32 + lane < tile_n;
            const uint32_t d = (key[r] >> shift) & mask;
            // lanes with the same digit: one ballot per digit bit. The warp's match instruction works through the distinct values
            // one by one, which a tile that its successors wait for feels (60 k keys 48 us with it, 42 with ballots).
            uint32_t peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
            for (int bit = 0; bit < 8; ++bit) {
                if (mask >> bit) {
                    const bool one = (d >> bit) & 1u;
                    const uint32_t b = __ballot_sync(0xffffffffu, one);
                    peers &= one ? b : ~b;
                }
            }
            uint32_t prev = 0;
            if (ok) prev = cnt[warp][d];
            __syncwarp();
            if (ok && (peers & lt_mask) == 0) cnt[warp][d] = prev + __popc(peers);
            __syncwarp();
            rank[r] = prev + __popc(peers & lt_mask);
        }
        __syncthreads();
        uint32_t* my_state = state + (size_t)tile * 256 + threadIdx.x;
        uint32_t run = 0;   // items of digit threadIdx.x in this tile
        {
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                const uint32_t c = cnt[w][threadIdx.x];
                cnt[w][threadIdx.x] = run;
                run += c;
            }
            st_state(my_state, tile == 0 ? (kInclusive | run) : run + 1u);
            int total;
            const int start = block_excl_scan((int)run, total, sm);  // start of this digit inside the tile
            tstart[threadIdx.x] = (uint32_t)start;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) cnt[w][threadIdx.x] += (uint32_t)start;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kItems; ++r) {
            if (wbase + r * 32 + lane < tile_n) {
                const uint32_t d = (key[r] >> shift) & mask;
                const uint32_t pos = cnt[warp][d] + rank[r];
                skeys[pos] = key[r];
                svals[pos] = val[r];
            }
        }
        uint32_t prefix = 0;
        if (tile > 0) {
            int polls = 0;
            const uint32_t* p = my_state - 256;
            int64_t left = tile;   // predecessors not yet counted
            bool found = false;
            while (!found && left > 0) {
                uint32_t v[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) v[q] = q < left ? ld_state(p - q * 256) : 0u;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (found || v[q] == 0u) break;
                    prefix += (v[q] & kInclusive) ? (v[q] & ~kInclusive) : v[q] - 1u;
                    found = (v[q] & kInclusive) != 0u;
                    p -= 256;
                    --left;
                }
                if (++polls > kPollLimit) {
                    atomicExch(gave_up, 1);
                    break;
                }
            }
            st_state(my_state, kInclusive | (prefix + run));
        }
        gbase[threadIdx.x] = digit_base + prefix;
        __syncthreads();
        // write out: item j of the reordered tile belongs to digit d = digit(skeys[j]) and goes to
        // gbase[d] + (j - tstart[d]); neighbouring j of one digit are neighbouring addresses
#pragma unroll
        for (int r = 0; r < kItems; ++r) {
            const int j = r * kThreads + threadIdx.x;
            if (j < tile_n) {
                const uint32_t k = skeys[j];
                const uint32_t d = (k >> shift) & mask;
                const uint32_t pos = gbase[d] + ((uint32_t)j - tstart[d]);
                if (pos < (uint32_t)n) {
                    keys_out[pos] = k;
                    vals_out[pos] = svals[j];
                }
            }
        }
        __syncthreads();
    }
}

// ---- instance emission ----------------------------------------------------------------------
// Prefix over the Gaussians' tile counts (in emission order) and their instances, in one kernel. A CTA takes 256 or
// 1024 Gaussians by ticket, scans their counts, finds the instances of the earlier tiles by look-back (one warp, 32 tiles at a time)
// and writes its instances as one contiguous run: thread k of a round finds the owner of instance k by bisection, so the stores
// are coalesced and a Gaussian that covers the whole image does not hold up one thread.
// EWA: a Gaussian's instances are the tiles of the bounds rectangle that the ellipse reaches (create_instances_cu,
// src/training/fastgs/rasterization/include/kernels_forward.cuh:205-309), in row-major tile order: no closed form for the k-th,
// so eight lanes walk a rectangle together.
constexpr int kEmitItems = 4;
template <bool EWA, int ITEMS>
__global__ void __launch_bounds__(kThreads) emit_instances_kernel(
    int64_t total, int N, const uint32_t* __restrict__ order, const int32_t* __restrict__ tiles,
    const float* __restrict__ means2d, const int32_t* __restrict__ radii, const ushort4* __restrict__ ewa_bounds,
    const float4* __restrict__ rec, float tile_size, uint32_t tw, uint32_t th, uint32_t tile_n_bits, int64_t capacity,
    uint32_t* __restrict__ tkeys, uint32_t* __restrict__ tvals, int32_t* overflow, int32_t* gave_up, int32_t* __restrict__ n_out,
    uint32_t* ticket, uint32_t* state) {
    constexpr int kList = kThreads * ITEMS;
    __shared__ int sm[33];
    __shared__ uint32_t s_tile, s_prefix;
    __shared__ int s_off[kList + 1];
    __shared__ uint32_t s_idx[kList], s_w[EWA ? 1 : kList];
    __shared__ uint2 s_xy[EWA ? 1 : kList];
    const uint32_t n_list_tiles = (uint32_t)((total + kList - 1) / kList);
    const int lane = threadIdx.x & 31;
    for (;;) {
        if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
        __syncthreads();
        const uint32_t tile = s_tile;
        if (tile >= n_list_tiles) break;
        const int64_t r0 = (int64_t)tile * kList + threadIdx.x * ITEMS;
        uint32_t idx[ITEMS];
        int nt[ITEMS], sum = 0;
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const int64_t r = r0 + k;
            idx[k] = r < total ? (order ? order[r] : (uint32_t)r) : 0u;
            nt[k] = r < total && idx[k] < (uint64_t)total ? max(tiles[idx[k]], 0) : 0;
        }
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) sum += nt[k];
        int block_total;
        int off = block_excl_scan(sum, block_total, sm);
        if (threadIdx.x == 0) st_state(state + tile, tile == 0 ? (kInclusive | (uint32_t)block_total) : (uint32_t)block_total + 1u);
        if (threadIdx.x == 0) s_off[kList] = block_total;
        {
            int o = off;
#pragma unroll
            for (int k = 0; k < ITEMS; ++k) {
                const int e = threadIdx.x * ITEMS + k;
                s_off[e] = o;
                s_idx[e] = idx[k];
                if (!EWA && nt[k] > 0) {
                    const size_t g = (size_t)idx[k] * 2;
                    uint32_t x0, y0, x1, y1;
                    tile_rect(means2d[g], means2d[g + 1], radii[g], radii[g + 1], tile_size, tw, th, x0, y0, x1, y1);
                    s_xy[e] = make_uint2(x0, y0);
                    s_w[e] = max(x1 - x0, 1u);
                }
                o += nt[k];
            }
        }
        if (threadIdx.x < 32) {
            uint32_t prefix = 0;
            int64_t j = (int64_t)tile - 1;
            int polls = 0;
            while (j >= 0) {
                const uint32_t v = j - lane >= 0 ? ld_state(state + (j - lane)) : kInclusive;
                const uint32_t incl = __ballot_sync(0xffffffffu, (v & kInclusive) != 0u), empty = __ballot_sync(0xffffffffu, v == 0u);
                const int last = incl ? __ffs(incl) - 1 : 31;   // nearest predecessor whose total covers everything before it
                if (empty & (last == 31 ? 0xffffffffu : (2u << last) - 1u)) {
                    if (++polls > kPollLimit) {
                        if (lane == 0) atomicExch(gave_up, 1);
                        break;
                    }
                    continue;
                }
                const uint32_t c = lane > last ? 0u : (v & kInclusive) ? (v & ~kInclusive) : v - 1u;
                prefix = min(prefix + __reduce_add_sync(0xffffffffu, c), 0x7fffffffu);
                if (incl) break;
                j -= 32;
            }
            if (lane == 0) {
                const uint32_t upto = min(prefix + (uint32_t)block_total, 0x7fffffffu);
                if (tile > 0) st_state(state + tile, kInclusive | upto);
                s_prefix = prefix;
                if (tile == n_list_tiles - 1) *n_out = (int32_t)upto;
                if ((int64_t)prefix + block_total > capacity && overflow) atomicExch(overflow, 1);
            }
        }
        __syncthreads();
        const int64_t base = s_prefix;
        if (!EWA) {
            for (int k = threadIdx.x; k < block_total; k += kThreads) {
                int lo = 0;   // last entry whose first instance is at or before k
#pragma unroll
                for (int step = kList / 2; step > 0; step >>= 1)
                    if (s_off[lo + step] <= k) lo += step;
                const uint32_t local = (uint32_t)(k - s_off[lo]), w = s_w[lo], g = s_idx[lo];
                const uint32_t y = local / w, x = local - y * w;
                const uint2 xy = s_xy[lo];
                if (base + k < capacity) {
                    tkeys[base + k] = ((g / (uint32_t)N) << tile_n_bits) | ((xy.y + y) * tw + xy.x + x);
                    tvals[base + k] = g;
                }
            }
        } else {
            // eight lanes test eight tiles of one rectangle at a time; the ballot gives each reached tile its place
            const int sub = lane & 7, group = lane >> 3;
            for (int q0 = (threadIdx.x >> 5) * 4; q0 < kList; q0 += kWarps * 4) {
                const int q = q0 + group;
                int64_t at = base + s_off[q];
                const int64_t end = base + s_off[q + 1];
                const uint32_t g = s_idx[q];
                ushort4 b = make_ushort4(0, 0, 0, 0);
                float4 c0 = make_float4(0.f, 0.f, 0.f, 0.f), c1 = c0, c2 = c0;
                if (at < end && end <= capacity) {
                    b = ewa_bounds[g];
                    c0 = rec[(size_t)g * 3]; c1 = rec[(size_t)g * 3 + 1]; c2 = rec[(size_t)g * 3 + 2];
                }
                const uint32_t width = b.y - b.x, area = width * (b.w - b.z);
                for (uint32_t k = sub; __any_sync(0xffffffffu, k - sub < area); k += 8) {
                    const uint32_t row = k < area ? k / width : 0u, ty = b.z + row, tx = b.x + (k - row * width);
                    const bool hit = k < area && ewa_tile_contributes(c0.x - 0.5f, c0.y - 0.5f, c0.z, c0.w, c1.x, tx, ty, c2.z);
                    const uint32_t hits = (__ballot_sync(0xffffffffu, hit) >> (8 * group)) & 0xffu;
                    const int64_t pos = at + __popc(hits & ((1u << sub) - 1u));
                    if (hit && pos < end) {
                        tkeys[pos] = ty * tw + tx;
                        tvals[pos] = g;
                    }
                    at += __popc(hits);
                }
            }
        }
        __syncthreads();
    }
}

// offsets[t] = first sorted instance whose (camera, tile) id >= t, for t in [0, n_ids]; entry n_ids
// (one past the last tile) holds the instance count. Keys hold (cid << tile_n_bits) | tile.
// When the overflow flag is set the instance list is incomplete (some slots were never written), so
// the keys cannot be trusted: all offsets are zeroed and the rasterizer draws nothing. Ids are clamped to
// n_ids in any case so that no key value can direct a store outside the offsets array.
__global__ void __launch_bounds__(kThreads) tile_offsets_kernel(const uint32_t* __restrict__ tkeys, const int32_t* n_dev,
                                                                int64_t n_max, uint32_t n_tiles, uint32_t tile_n_bits,
                                                                int64_t n_ids, const int32_t* __restrict__ overflow,
                                                                int32_t* __restrict__ offsets) {
    const int64_t n = (overflow && *overflow) ? 0 : device_count(n_dev, n_max);
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (n == 0) {
        for (int64_t i = tid; i <= n_ids; i += stride) offsets[i] = 0;
        return;
    }
    const uint32_t tmask = (1u << tile_n_bits) - 1u;
    for (int64_t i = tid; i < n; i += stride) {
        const uint32_t k = tkeys[i];
        const int64_t id_curr = min((int64_t)(k >> tile_n_bits) * n_tiles + (k & tmask), n_ids - 1);
        if (i == 0)
            for (int64_t t = 0; t <= id_curr; ++t) offsets[t] = 0;
        if (i == n - 1)
            for (int64_t t = id_curr + 1; t <= n_ids; ++t) offsets[t] = (int32_t)n;
        if (i > 0) {
            const uint32_t kp = tkeys[i - 1];
            if (kp != k) {
                const int64_t id_prev = min((int64_t)(kp >> tile_n_bits) * n_tiles + (kp & tmask), n_ids - 1);
                for (int64_t t = id_prev + 1; t <= id_curr; ++t) offsets[t] = (int32_t)i;
            }
        }
    }
}

// Operator-level output: 64-bit keys (camera | tile | depth bits) and int32 flattened ids. A list that was given up (some of its
// slots were never written) comes out as the largest key and id 0 throughout, beyond every tile.
__global__ void __launch_bounds__(kThreads) compose_isect_ids_kernel(int64_t n, const uint32_t* __restrict__ tkeys,
                                                                     const uint32_t* __restrict__ tvals,
                                                                     const float* __restrict__ depths,
                                                                     const int32_t* __restrict__ gave_up,
                                                                     int64_t* __restrict__ isect_ids,
                                                                     int32_t* __restrict__ flatten_ids) {
    const bool failed = *gave_up != 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t v = failed ? 0u : tvals[i];
        isect_ids[i] = failed ? INT64_MAX : ((int64_t)tkeys[i] << 32) | (int64_t)__float_as_uint(depths[v]);
        flatten_ids[i] = (int32_t)v;
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

__global__ void depth_keys_kernel(int64_t total, const float* __restrict__ depths, const int32_t* __restrict__ tiles,
                                  uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        keys[i] = tiles[i] > 0 ? __float_as_uint(depths[i]) : 0xFFFFFFFFu;
        vals[i] = (uint32_t)i;
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

// Words of the list state: tickets [64] | digit counts [2 sorts][4 passes][256] | emission look-back | sort look-back. The first three
// are zeroed by one memset per list build, the last by the histogram kernel of each sort, which knows the count.
namespace {
constexpr size_t kTicketWords = 64, kHistWords = 2 * 4 * 256;   // tickets: nine, and at 32 the word of list_gave_up
int32_t* list_gave_up(uint32_t* state) { return reinterpret_cast<int32_t*>(state) + 32; }
size_t emit_state_words(int64_t total) { return ((size_t)((total + kThreads - 1) / kThreads) + 63) / 64 * 64; }
// Look-back serves short lists, where a sort is mostly launches (16 k keys, four passes: 42 us against 66 with separate counting
// kernels; 250 k 51 against 68; 1 M 79 against 94); on long lists its waves of tiles queue behind one another's words and the
// three-kernel pass with one chunk per CTA is the faster one (6 M keys: 217 us against 279; 7 M instances, two passes: 291
// against 360). A device-side count is bounded by the list's capacity, which users leave a few times larger than the list.
int64_t lookback_limit(bool count_on_device) { return count_on_device ? (int64_t)6 << 20 : (int64_t)2 << 20; }
constexpr int64_t kMaxChunks = 1024;   // the size query must not depend on a device
int chunk_blocks(int64_t n_max) { return (int)min((n_max + kTile - 1) / kTile, min((int64_t)4 * num_sms(), kMaxChunks)); }
// Never less for a longer list, although a chunked sort needs less than the longest look-back: a workspace made for a capacity
// serves every list up to it.
size_t sort_state_words(bool count_on_device, int64_t n, int passes) {
    const int64_t limit = lookback_limit(count_on_device);
    const size_t lookback = (size_t)((min(n, limit) + kTile - 1) / kTile) * 256 * passes;
    const size_t chunked = n > limit ? (size_t)256 * (min((n + kTile - 1) / kTile, kMaxChunks) + 1) : 0;
    return lookback > chunked ? lookback : chunked;
}
int tile_sort_passes(int key_bits) { return (key_bits + 7) / 8; }
}  // namespace

size_t tile_list_state_words(int64_t total, int64_t capacity, int key_bits) {
    // the instance count is read on the device, the number of Gaussians is not
    const size_t depth = sort_state_words(false, total, 4);
    const size_t tile = sort_state_words(true, capacity, tile_sort_passes(key_bits));
    return kTicketWords + kHistWords + emit_state_words(total) + (depth > tile ? depth : tile);
}

// Stable LSD radix sort of (key, value) uint32 pairs over key bits [0, key_bits). n is read from *n_dev when n_dev != nullptr
// (device-side count, bounded by n_max), else n_max is the count. Returns the index (0 or 1) of the pair holding the result.
// tickets [4], hist [4 * 256]: zero on entry. state: sort_state_words.
static int radix_sort_pairs(uint32_t* keys[2], uint32_t* vals[2], const int32_t* n_dev, int64_t n_max, int key_bits,
                            uint32_t* tickets, uint32_t* hist, uint32_t* state, int32_t* gave_up, cudaStream_t st) {
    if (n_max <= 0 || key_bits <= 0) return 0;
    const int passes = tile_sort_passes(key_bits);
    const int bits = (key_bits + passes - 1) / passes;
    const uint32_t mask = (1u << bits) - 1u;
    int cur = 0;
    LFS_TIMED(n_dev ? "radix_sort_tile" : "radix_sort_depth", st);
    if (n_max <= lookback_limit(n_dev != nullptr)) {
        const int64_t max_tiles = (n_max + kTile - 1) / kTile;
        // six CTAs per SM (27 KB of shared memory each) keep enough keys in flight; more only queue for tickets
        const int nb = (int)min(max_tiles, (int64_t)6 * num_sms());
        radix_hist_kernel<<<(int)min(max_tiles, (int64_t)4 * num_sms()), kThreads, 0, st>>>(
            keys[0], n_dev, n_max, bits, passes, hist, reinterpret_cast<uint4*>(state), max_tiles * 64);
        for (int p = 0; p < passes; ++p) {
            radix_scatter_kernel<<<nb, kThreads, 0, st>>>(keys[cur], vals[cur], keys[cur ^ 1], vals[cur ^ 1], n_dev, n_max,
                                                                 p * bits, mask, hist + p * 256, tickets + p,
                                                                 state + (size_t)p * max_tiles * 256, gave_up);
            cur ^= 1;
        }
    } else {
        const int nb = chunk_blocks(n_max);
        uint32_t *table = state, *totals = state + (size_t)256 * nb;
        for (int p = 0; p < passes; ++p) {
            radix_count_kernel<<<nb, kThreads, 0, st>>>(keys[cur], n_dev, n_max, p * bits, mask, nb, table);
            radix_scan_kernel<<<256, kThreads, 0, st>>>(table, nb, totals);
            radix_scatter_chunk_kernel<<<nb, kThreads, 0, st>>>(keys[cur], vals[cur], keys[cur ^ 1], vals[cur ^ 1], n_dev, n_max, p * bits,
                                                                mask, nb, table, totals);
            cur ^= 1;
        }
    }
    if (check_launch("radix_sort") != LFS_OK) return -1;
    return cur;
}

static uint32_t bit_width_u32(uint32_t v) {
    uint32_t b = 0;
    while (v) { ++b; v >>= 1; }
    return b;
}

int build_tile_lists(const TileListArgs& a, cudaStream_t st) {
    const int64_t total = (int64_t)a.C * a.N;
    const uint32_t n_tiles = (uint32_t)a.tw * a.th;
    const uint32_t tile_n_bits = bit_width_u32(n_tiles);
    const uint32_t cam_n_bits = bit_width_u32((uint32_t)a.C);
    if (tile_n_bits + cam_n_bits > 32) {
        set_error("build_tile_lists: tile and camera ids need more than 32 bits");
        return LFS_EINVAL;
    }
    const int key_bits = (int)(tile_n_bits + cam_n_bits);
    uint32_t *tickets = a.state, *hist = tickets + kTicketWords, *emit_state = hist + kHistWords;
    uint32_t* sort_state = emit_state + emit_state_words(total);
    // raised by a look-back that ran out of polls; without an overflow flag of the caller's a word behind the tickets, read by
    // compose_isect_ids_kernel
    int32_t* gave_up = a.overflow ? a.overflow : list_gave_up(a.state);
    cudaMemsetAsync(a.state, 0, (kTicketWords + kHistWords + emit_state_words(total)) * sizeof(uint32_t), st);
    const uint32_t* order = nullptr;
    if (a.sort) {
        if (!a.keys_ready) {
            depth_keys_kernel<<<grid_for(total, 256), 256, 0, st>>>(total, a.depths, a.tiles, a.gkeys[0], a.gvals[0]);
        }
        uint32_t* k[2] = {a.gkeys[0], a.gkeys[1]};
        uint32_t* v[2] = {a.gvals[0], a.gvals[1]};
        const int sel = radix_sort_pairs(k, v, nullptr, total, 32, tickets, hist, sort_state, gave_up, st);
        if (sel < 0) return LFS_ECUDA;
        order = v[sel];
    }
    if (total > 0) {
        LFS_TIMED("emit_instances", st);
        // Four Gaussians per thread make fewer tickets and a shorter look-back, one makes more CTAs in flight. us with one and with four,
        // 1296x840 (in thousands of Gaussians): 450: 33 / 57, 1000: 54 / 71, 1500: 69 / 66, 2000: 93 / 76, 3000: 137 / 118. EWA, whose
        // rectangle walk is longer than the scan: 300: 58 / 133, 450: 67 / 111, 700: 99 / 124, 1000: 123 / 107, 2000: 259 / 185.
        const bool four = total > (a.ewa_bounds ? (int64_t)850000 : (int64_t)2 << 20);
        const int64_t list = four ? kThreads * kEmitItems : kThreads;
        const int nb = (int)min((total + list - 1) / list, (int64_t)8 * num_sms());
#define LFS_EMIT(EWA, ITEMS)                                                                                                                 \
    emit_instances_kernel<EWA, ITEMS><<<nb, kThreads, 0, st>>>(total, a.N, order, a.tiles, a.means2d, a.radii, a.ewa_bounds, a.ewa_records,    \
                                                        (float)a.tile_size, (uint32_t)a.tw, (uint32_t)a.th, tile_n_bits, a.capacity,   \
                                                        a.tkeys[0], a.tvals[0], a.overflow, gave_up, a.n_isects_dev, tickets + 8, emit_state)
        if (a.ewa_bounds) { if (four) LFS_EMIT(true, kEmitItems); else LFS_EMIT(true, 1); }
        else { if (four) LFS_EMIT(false, kEmitItems); else LFS_EMIT(false, 1); }
#undef LFS_EMIT
    } else {
        cudaMemsetAsync(a.n_isects_dev, 0, sizeof(int32_t), st);
    }
    int sel = 0;
    if (a.sort && a.capacity > 0) {
        uint32_t* k[2] = {a.tkeys[0], a.tkeys[1]};
        uint32_t* v[2] = {a.tvals[0], a.tvals[1]};
        sel = radix_sort_pairs(k, v, a.n_isects_dev, a.capacity, key_bits, tickets + 4, hist + 4 * 256, sort_state, gave_up, st);
        if (sel < 0) return LFS_ECUDA;
    }
    if (a.sel_out) *a.sel_out = sel;
    if (a.tile_offsets) {
        const int64_t n_ids = (int64_t)a.C * n_tiles;
        LFS_TIMED("tile_offsets", st);
        tile_offsets_kernel<<<grid_for(a.capacity > 0 ? a.capacity : 1, 256), 256, 0, st>>>(
            a.tkeys[sel], a.n_isects_dev, a.capacity, n_tiles, tile_n_bits, n_ids, a.overflow, a.tile_offsets);
    }
    return check_launch("build_tile_lists");
}

// Launch order of the tile CTAs: tiles with the longest lists first, so that the last wave of a rasterizer launch
// is made of short tiles. 132 buckets by the leading one and the next two bits of the list length (a
// floating-point-like key with a 2-bit mantissa); the order inside a bucket is arbitrary. offsets has n_tiles + 1
// entries.
__device__ __forceinline__ int tile_order_bucket(int c) {
    if (c <= 0) return 131;
    const int lz = __clz(c);                              // 0 .. 31, small = long list
    const int shift = max(0, 29 - lz);                    // bring the two bits below the leading one down
    const int mant = (c >> shift) & 3;
    return lz * 4 + (3 - mant);
}

__global__ void __launch_bounds__(1024) tile_order_kernel(int n_tiles, const int32_t* __restrict__ offsets,
                                                          int32_t* __restrict__ order) {
    __shared__ int hist[132], cursor[132];
    if (threadIdx.x < 132) hist[threadIdx.x] = 0;
    __syncthreads();
    for (int t = threadIdx.x; t < n_tiles; t += blockDim.x) atomicAdd(&hist[tile_order_bucket(offsets[t + 1] - offsets[t])], 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int b = 0; b < 132; ++b) { cursor[b] = run; run += hist[b]; }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < n_tiles; t += blockDim.x)
        order[atomicAdd(&cursor[tile_order_bucket(offsets[t + 1] - offsets[t])], 1)] = t;
}

int launch_tile_order(int n_tiles, const int32_t* offsets, int32_t* order, cudaStream_t st) {
    if (n_tiles <= 0) return LFS_OK;
    LFS_TIMED("tile_order", st);
    tile_order_kernel<<<1, 1024, 0, st>>>(n_tiles, offsets, order);
    return check_launch("tile_order");
}

int launch_compose_isect_ids(int64_t n, const uint32_t* tkeys, const uint32_t* tvals, const float* depths, const uint32_t* list_state,
                             int64_t* isect_ids, int32_t* flatten_ids, cudaStream_t st) {
    if (n <= 0) return LFS_OK;
    compose_isect_ids_kernel<<<grid_for(n, 256), 256, 0, st>>>(n, tkeys, tvals, depths, list_gave_up(const_cast<uint32_t*>(list_state)), isect_ids,
                                                                flatten_ids);
    return check_launch("compose_isect_ids");
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
