// Deterministic scan and stable LSD radix sort with device-resident counts.
//
// Every launch is sized from a host-known capacity and reads the live element
// count from device memory, so the index build needs no host synchronisation
// and can be captured in a CUDA graph.  The sort is stable (equal keys keep
// their input order), which is what the reference's cub::DeviceRadixSort
// calls rely on (libs/star/common/algorithm_types.cuh:37-83).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

namespace ws {

constexpr int kSortThreads = 256;
// Keys per thread of a tile: 8, or 16 from a capacity of 4 M keys.  A frame's keys fill few tiles (500 k in all; two
// passes' scatter of 500 nodes 12.9 / 15.4 us, 8000 nodes 25.5 / 31.5), a batch's tables of tiles are read and
// written for all digits (64 scenes, all three kernels 859 / 627 us).
constexpr int kSortRoundsSmall = 8, kSortRoundsLarge = 16;
inline int sort_rounds(uint32_t cap) { return cap <= (4u << 20) ? kSortRoundsSmall : kSortRoundsLarge; }
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;    // 2048 elements per tile

__device__ __forceinline__ uint32_t warp_incl_scan_u32(uint32_t v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t n = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += n;
    }
    return v;
}

// Block-wide exclusive scan of one value per thread (blockDim.x <= 1024, multiple of 32).
__device__ __forceinline__ uint32_t block_excl_scan_u32(uint32_t v, uint32_t *total, uint32_t *smem32) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint32_t inc = warp_incl_scan_u32(v);
    __syncthreads();
    if (lane == 31) smem32[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < nw ? smem32[lane] : 0u;
        w = warp_incl_scan_u32(w);
        if (lane < nw) smem32[lane] = w;
    }
    __syncthreads();
    const uint32_t warp_off = warp > 0 ? smem32[warp - 1] : 0u;
    if (total) *total = smem32[nw - 1];
    return warp_off + inc - v;
}

// ---------------------------------------------------------------------------
// Exclusive scan: out[i] = sum_{j<i} in[i]; out[n] = total.  Up to kScanSmall elements in one launch of one
// block, beyond in three: tile sums, scan of tile sums (one block), tile scans.  A launch costs some 2 us beside
// its work: with one to three of them a scan, a frame's five scans of 300 to 8000 elements took 30 us, now 8.
// ---------------------------------------------------------------------------
constexpr uint32_t kScanSmall = 16384;   // four passes of the block, as long as three launches

struct ScanArrays {
    const uint32_t *in[2];
    uint32_t *out[2];
};

// Block b scans array b; in and out may alias.
static __global__ void __launch_bounds__(1024) k_scan_small(ScanArrays a, uint32_t n) {
    __shared__ uint32_t sm[32];
    const uint32_t *in = a.in[blockIdx.x];
    uint32_t *out = a.out[blockIdx.x];
    uint32_t carry = 0;
    for (uint32_t base = 0; base < n; base += 4096) {
        const uint32_t i0 = base + 4 * threadIdx.x;
        uint32_t v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = i0 + k < n ? in[i0 + k] : 0u;
        uint32_t total;
        uint32_t run = carry + block_excl_scan_u32(v[0] + v[1] + v[2] + v[3], &total, sm);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (i0 + k < n) out[i0 + k] = run;
            run += v[k];
        }
        carry += total;
        __syncthreads();   // sm is reused by the next pass's scan
    }
    if (threadIdx.x == 0) out[n] = carry;
}

static __global__ void k_scan_tile_sums(const uint32_t *in, uint32_t n, uint32_t *tile_sums) {
    __shared__ uint32_t sm[32];
    const uint32_t base = blockIdx.x * kScanTile;
    uint32_t s = 0;
    if (base < n) {
#pragma unroll
        for (int i = 0; i < kScanItems; ++i) {
            const uint32_t idx = base + threadIdx.x * kScanItems + i;
            if (idx < n) s += in[idx];
        }
    }
    uint32_t total;
    block_excl_scan_u32(s, &total, sm);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// The total goes to tile_sums[num_tiles].
static __global__ void k_scan_tile_offsets(uint32_t *tile_sums, int num_tiles) {
    __shared__ uint32_t sm[32];
    __shared__ uint32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < num_tiles; base += blockDim.x) {
        const int i = base + threadIdx.x;
        const uint32_t v = i < num_tiles ? tile_sums[i] : 0u;
        uint32_t total;
        const uint32_t ex = block_excl_scan_u32(v, &total, sm);
        if (i < num_tiles) tile_sums[i] = carry + ex;
        __syncthreads();
        if (threadIdx.x == 0) carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) tile_sums[num_tiles] = carry;
}

static __global__ void k_scan_apply(const uint32_t *in, uint32_t n, const uint32_t *tile_offsets, int num_tiles,
                                    uint32_t *out) {
    __shared__ uint32_t sm[32];
    const uint32_t base = blockIdx.x * kScanTile;
    uint32_t v[kScanItems];
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const uint32_t idx = base + threadIdx.x * kScanItems + i;
        v[i] = idx < n ? in[idx] : 0u;
        s += v[i];
    }
    uint32_t ex = block_excl_scan_u32(s, nullptr, sm) + tile_offsets[blockIdx.x];
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        const uint32_t idx = base + threadIdx.x * kScanItems + i;
        if (idx < n) out[idx] = ex;
        ex += v[i];
    }
    if (base <= n && n < base + kScanTile && threadIdx.x == 0) out[n] = tile_offsets[num_tiles];
}

// Host drivers; return the launches.  `in` and `out` may alias; out has n + 1 entries, tile_sums n / 2048 + 2.
inline int exclusive_scan(const uint32_t *in, uint32_t *out, uint32_t n, uint32_t *tile_sums, cudaStream_t st) {
    if (n <= kScanSmall) {
        k_scan_small<<<1, 1024, 0, st>>>({{in, nullptr}, {out, nullptr}}, n);
        return 1;
    }
    const int tiles = (int)(n / kScanTile) + 1;
    k_scan_tile_sums<<<tiles, kScanThreads, 0, st>>>(in, n, tile_sums);
    k_scan_tile_offsets<<<1, 1024, 0, st>>>(tile_sums, tiles);
    k_scan_apply<<<tiles, kScanThreads, 0, st>>>(in, n, tile_sums, tiles, out);
    return 3;
}

// Two arrays of n elements.
inline int exclusive_scan2(const uint32_t *in0, uint32_t *out0, const uint32_t *in1, uint32_t *out1, uint32_t n,
                           uint32_t *tile_sums, cudaStream_t st) {
    if (n <= kScanSmall) {
        k_scan_small<<<2, 1024, 0, st>>>({{in0, in1}, {out0, out1}}, n);
        return 1;
    }
    return exclusive_scan(in0, out0, n, tile_sums, st) + exclusive_scan(in1, out1, n, tile_sums, st);
}

// ---------------------------------------------------------------------------
// Stable LSD radix sort of (key, u32 value), D = 8 or 9 bits per pass (256 or 512 digits; each
// thread of a 256-thread block looks after one or two of them).  A tile has R keys per thread.
// hist layout: hist[digit * max_tiles + tile].
// ---------------------------------------------------------------------------
// Counts a tile's digits: all keys of a thread are read before the first is counted (64 scenes, all passes 258 -> 182
// us).  Shared atomics merge equal digits of a warp well enough: merging them by matching takes 226 us.
// A warp has R * 32 consecutive keys of the tile, lane l the keys 32 r + l.
template <class K, int D, int R>
__global__ void __launch_bounds__(kSortThreads) k_radix_upsweep(const K *keys, const uint32_t *n_dev, uint32_t n_static,
                                                                int shift, uint32_t *hist, int max_tiles) {
    constexpr uint32_t kDigits = 1u << D;
    __shared__ uint32_t h[kDigits];
    const uint32_t n = n_dev ? *n_dev : n_static;
    const uint32_t base = blockIdx.x * (uint32_t)(kSortThreads * R);
    for (uint32_t d = threadIdx.x; d < kDigits; d += kSortThreads) h[d] = 0;
    const int lane = threadIdx.x & 31;
    const uint32_t first = base + (threadIdx.x >> 5) * (32u * R) + (uint32_t)lane;
    K key[R];
#pragma unroll
    for (int r = 0; r < R; ++r) key[r] = first + 32u * r < n ? keys[first + 32u * r] : K(0);
    __syncthreads();
    if (base < n) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const bool valid = first + 32u * r < n;
            const uint32_t d = (uint32_t)(key[r] >> shift) & (kDigits - 1u);
            if (valid) atomicAdd(&h[d], 1u);
        }
    }
    __syncthreads();
    for (uint32_t d = threadIdx.x; d < kDigits; d += kSortThreads) hist[(size_t)d * max_tiles + blockIdx.x] = h[d];
}

// Exclusive scan of one digit's tile counts (one block per digit) over the tiles in use,
// 1024 consecutive counts per pass (4 per thread), with the running total carried along.
static __global__ void k_radix_scan(uint32_t *hist, int max_tiles, uint32_t tile, const uint32_t *n_dev, uint32_t n_static,
                                    uint32_t *digit_total) {
    __shared__ uint32_t sm[32];
    const uint32_t n = n_dev ? *n_dev : n_static;
    const int used = min(max_tiles, (int)((n + tile - 1) / tile));
    uint32_t *row = hist + (size_t)blockIdx.x * max_tiles;
    uint32_t carry = 0;
    for (int base = 0; base < used; base += 4 * (int)blockDim.x) {
        const int i0 = base + 4 * (int)threadIdx.x;
        uint32_t v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = (i0 + k < used) ? row[i0 + k] : 0u;
        const uint32_t local = v[0] + v[1] + v[2] + v[3];
        uint32_t total;
        uint32_t run = block_excl_scan_u32(local, &total, sm) + carry;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (i0 + k < used) row[i0 + k] = run;
            run += v[k];
        }
        carry += total;
        __syncthreads();   // sm is reused by the next pass's scan
    }
    if (threadIdx.x == 0) digit_total[blockIdx.x] = carry;
}

// Places a tile's keys and values, all of them read at once.  What bounds it is the ranking (every key's place among
// its digit's) and the writes: a warp ranks its own run of keys against counters of its own, with nothing shared
// until all are ranked, and the tile goes through shared memory in digit order, so that a digit's keys are written
// side by side.  Ranking by rounds of the whole block, four barriers a round, and writing each key where it belongs
// took, for all passes of 64 scenes' lists 613 us, now 412; 8000 nodes' 58, now 26; 200 k voxels 52, now 18.
// Ranking by ballots of the digit's bits instead of matching: 585 us for 64 scenes.
template <class K, int D, int R>
__global__ void __launch_bounds__(kSortThreads)
k_radix_scatter(const K *keys_in, const uint32_t *vals_in, K *keys_out, uint32_t *vals_out,
                const uint32_t *n_dev, uint32_t n_static, int shift,
                const uint32_t *hist, int max_tiles, const uint32_t *digit_total) {
    constexpr uint32_t kDigits = 1u << D;
    constexpr int kPer = (int)kDigits / kSortThreads;   // digits per thread
    constexpr int kWarps = kSortThreads / 32;
    static_assert(kPer == 1 || kPer == 2, "8- or 9-bit digits");
    __shared__ uint32_t delta[kDigits];                 // digit -> its first place in the output less that in the tile
    __shared__ uint16_t wcount[kWarps][kDigits];
    __shared__ K s_key[kSortThreads * R];
    __shared__ uint32_t s_val[kSortThreads * R];
    __shared__ uint32_t sm[32];
    const uint32_t n = n_dev ? *n_dev : n_static;
    const uint32_t base = blockIdx.x * (uint32_t)(kSortThreads * R);
    if (base >= n) return;                      // uniform for the whole block
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t first = base + (uint32_t)warp * (32u * R) + (uint32_t)lane;
    K key[R];
    uint32_t val[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t idx = first + 32u * r;
        key[r] = idx < n ? keys_in[idx] : K(0);
        val[r] = idx < n ? vals_in[idx] : 0u;
    }
    // thread t owns digits kPer t .. kPer t + kPer - 1
    uint32_t global[kPer];
    {
        uint32_t tot[kPer], sum = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            tot[k] = digit_total[kPer * t + k];
            sum += tot[k];
        }
        uint32_t ex = block_excl_scan_u32(sum, nullptr, sm);
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            global[k] = ex + hist[(size_t)(kPer * t + k) * max_tiles + blockIdx.x];
            ex += tot[k];
        }
    }
    for (uint32_t d = (uint32_t)lane; d < kDigits; d += 32) wcount[warp][d] = 0;
    __syncwarp();
    uint16_t rank[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const bool valid = first + 32u * r < n;
        const uint32_t d = (uint32_t)(key[r] >> shift) & (kDigits - 1u);
        const unsigned peers = __match_any_sync(0xffffffffu, valid ? d : kDigits);
        const uint32_t before = wcount[warp][d];
        const uint32_t lower = (uint32_t)__popc(peers & ((1u << lane) - 1u));
        rank[r] = (uint16_t)(before + lower);
        __syncwarp();
        if (valid && lower == 0) wcount[warp][d] = (uint16_t)(before + (uint32_t)__popc(peers));
        __syncwarp();
    }
    __syncthreads();
    {
        uint32_t tot[kPer], sum = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            tot[k] = 0;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) tot[k] += wcount[w][kPer * t + k];
            sum += tot[k];
        }
        uint32_t at = block_excl_scan_u32(sum, nullptr, sm);
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            delta[kPer * t + k] = global[k] - at;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                const uint32_t c = wcount[w][kPer * t + k];
                wcount[w][kPer * t + k] = (uint16_t)at;
                at += c;
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (first + 32u * r < n) {
            const uint32_t d = (uint32_t)(key[r] >> shift) & (kDigits - 1u);
            const uint32_t at = (uint32_t)wcount[warp][d] + rank[r];
            s_key[at] = key[r];
            s_val[at] = val[r];
        }
    }
    __syncthreads();
    const uint32_t count = min((uint32_t)(kSortThreads * R), n - base);
#pragma unroll 4
    for (uint32_t i = (uint32_t)t; i < count; i += kSortThreads) {
        const K k = s_key[i];
        const uint32_t at = delta[(uint32_t)(k >> shift) & (kDigits - 1u)] + i;
        keys_out[at] = k;
        vals_out[at] = s_val[i];
    }
}

inline int sort_max_tiles(uint32_t cap) {
    const uint32_t tile = (uint32_t)(kSortThreads * sort_rounds(cap));
    return (int)((cap + tile - 1) / tile) + 1;
}
constexpr int kSortMaxDigits = 512;

template <class K, int D, int R>
inline void radix_pass(const K *ki, const uint32_t *vi, K *ko, uint32_t *vo, const uint32_t *n_dev, uint32_t n_static,
                       int shift, uint32_t *hist, int max_tiles, uint32_t *digit_total, cudaStream_t st) {
    k_radix_upsweep<K, D, R><<<max_tiles, kSortThreads, 0, st>>>(ki, n_dev, n_static, shift, hist, max_tiles);
    k_radix_scan<<<1 << D, 256, 0, st>>>(hist, max_tiles, (uint32_t)(kSortThreads * R), n_dev, n_static, digit_total);
    k_radix_scatter<K, D, R><<<max_tiles, kSortThreads, 0, st>>>(ki, vi, ko, vo, n_dev, n_static, shift, hist, max_tiles,
                                                                  digit_total);
}

// Sorts `bits` low bits of the keys, 9 bits per pass when that saves a pass over 8 bits.
// Buffers a/b ping-pong; returns true when the result ended in the `alt` buffers.  hist needs
// kSortMaxDigits * sort_max_tiles(cap) entries, digit_total kSortMaxDigits.
template <class K>
inline bool radix_sort(K *keys, uint32_t *vals, K *keys_alt, uint32_t *vals_alt,
                       const uint32_t *n_dev, uint32_t n_static, uint32_t cap, int bits,
                       uint32_t *hist, uint32_t *digit_total, cudaStream_t st) {
    const int max_tiles = sort_max_tiles(cap);
    const int step = ((bits + 8) / 9 < (bits + 7) / 8) ? 9 : 8;
    const bool small = sort_rounds(cap) == kSortRoundsSmall;
    bool in_alt = false;
    for (int shift = 0; shift < bits; shift += step) {
        K *ki = in_alt ? keys_alt : keys;
        uint32_t *vi = in_alt ? vals_alt : vals;
        K *ko = in_alt ? keys : keys_alt;
        uint32_t *vo = in_alt ? vals : vals_alt;
        auto pass = step == 9 ? (small ? radix_pass<K, 9, kSortRoundsSmall> : radix_pass<K, 9, kSortRoundsLarge>)
                              : (small ? radix_pass<K, 8, kSortRoundsSmall> : radix_pass<K, 8, kSortRoundsLarge>);
        pass(ki, vi, ko, vo, n_dev, n_static, shift, hist, max_tiles, digit_total, st);
        in_alt = !in_alt;
    }
    return in_alt;
}

// Radix passes of radix_sort for `bits` key bits.
inline int radix_passes(int bits) { return std::min((bits + 8) / 9, (bits + 7) / 8); }

inline int bits_for(uint64_t max_value) {
    int b = 1;
    while (b < 64 && (max_value >> b) != 0) ++b;
    return b;
}

}  // namespace ws
