// Index build of the B200 warp-field solver: pixel-term compaction,
// node->term and node-pair->term maps, and the block-CSR sparsity pattern.
//
// All scenes of a batch are processed by the same launches; per-scene counts
// live in device memory (Plan), so nothing here waits on the host.
#include <cuda_runtime.h>

#include <algorithm>

#include "ws_common.cuh"
#include "ws_prims.cuh"
#include "ws_workspace.h"

namespace ws {

constexpr int kPixTileThreads = 256;
constexpr int kPixPerThread = 4;
constexpr int kPixTile = kPixTileThreads * kPixPerThread;   // 1024 pixels per tile

__device__ __forceinline__ void set_error(int *flag, int code) { atomicCAS(flag, 0, code); }

// markPotentialValidImageTermPixelKernel (examples/mono_star/opt/ImageTermKNNFetcher.cu:9-29):
// a pixel is a potential term iff its index map holds a surfel id.
// A pixel counts only when its surfel id is in range (out-of-range ids are treated as empty,
// which keeps every later gather inside the caller's arrays).
__device__ __forceinline__ bool valid_surfel(uint32_t id, const Scene &sc) {
    return id != kInvalidIndex && id < (uint32_t)sc.num_surfels;
}

__global__ void k_pixel_count(const Scene *scenes, const uint32_t *tile_scene, int num_tiles, uint32_t *tile_count) {
    __shared__ uint32_t sm[32];
    const int t = blockIdx.x;
    if (t >= num_tiles) return;
    const Scene &sc = scenes[tile_scene[t]];
    const uint32_t npix = (uint32_t)sc.width * (uint32_t)sc.height;
    const uint32_t p0 = (uint32_t)(t - sc.tile_base) * kPixTile + threadIdx.x * kPixPerThread;
    uint32_t c = 0;
#pragma unroll
    for (int i = 0; i < kPixPerThread; ++i) {
        const uint32_t p = p0 + i;
        if (p < npix) {
            const uint32_t y = p / (uint32_t)sc.width, x = p - y * (uint32_t)sc.width;
            c += valid_surfel(sc.index_map[(size_t)y * sc.pitch + x], sc) ? 1u : 0u;
        }
    }
    uint32_t total;
    block_excl_scan_u32(c, &total, sm);
    if (threadIdx.x == 0) tile_count[t] = total;
}

// compactPontentialImageTermPixelsKernel (ImageTermKNNFetcher.cu:56-88) fused with
// queryPixelKNNKernel (WarpSolver.cu:7-47): raster-order compaction of
// (x, y, x + flow_x, y + flow_y) and the surfel's 4-NN and weights.
__global__ void k_pixel_compact(const Scene *scenes, const uint32_t *tile_scene, int num_tiles,
                                const uint32_t *tile_offset, ushort4 *pixels, ushort4 *knn,
                                float4 *sw, float4 *cw, uint32_t *term_scene, uint32_t cap, int *err) {
    __shared__ uint32_t sm[32];
    const int t = blockIdx.x;
    if (t >= num_tiles) return;
    const uint32_t s = tile_scene[t];
    const Scene &sc = scenes[s];
    const uint32_t npix = (uint32_t)sc.width * (uint32_t)sc.height;
    const uint32_t p0 = (uint32_t)(t - sc.tile_base) * kPixTile + threadIdx.x * kPixPerThread;
    uint32_t ids[kPixPerThread];
    uint32_t c = 0;
#pragma unroll
    for (int i = 0; i < kPixPerThread; ++i) {
        const uint32_t p = p0 + i;
        ids[i] = kInvalidIndex;
        if (p < npix) {
            const uint32_t y = p / (uint32_t)sc.width, x = p - y * (uint32_t)sc.width;
            ids[i] = sc.index_map[(size_t)y * sc.pitch + x];
            if (!valid_surfel(ids[i], sc)) ids[i] = kInvalidIndex;
            c += (ids[i] != kInvalidIndex) ? 1u : 0u;
        }
    }
    uint32_t pos = tile_offset[t] + block_excl_scan_u32(c, nullptr, sm);
#pragma unroll
    for (int i = 0; i < kPixPerThread; ++i) {
        if (ids[i] == kInvalidIndex) continue;
        const uint32_t p = p0 + i;
        const uint32_t y = p / (uint32_t)sc.width, x = p - y * (uint32_t)sc.width;
        float2 fl = make_float2(0.f, 0.f);
        if (sc.flow) fl = sc.flow[(size_t)y * sc.pitch + x];
        const unsigned tx = __float2uint_rn(fl.x + float(x));
        const unsigned ty = __float2uint_rn(fl.y + float(y));
        if (pos < cap) {
            pixels[pos] = make_ushort4((unsigned short)x, (unsigned short)y, (unsigned short)tx, (unsigned short)ty);
            ushort4 k4 = sc.surfel_knn[ids[i]];
            const unsigned nn = (unsigned)sc.num_nodes;
            if (k4.x >= nn || k4.y >= nn || k4.z >= nn || k4.w >= nn) {   // node id out of range
                set_error(err, WS_ERR_INVALID_ARGUMENT);
                k4 = make_ushort4(0, 0, 0, 0);
            }
            knn[pos] = k4;
            sw[pos] = sc.surfel_sw[ids[i]];
            cw[pos] = sc.surfel_cw[ids[i]];
            term_scene[pos] = s;
        }
        ++pos;
    }
}

// Per-scene counts and key/value ranges (term_offset_types.h:62-82 size2offset),
// computed after the compaction scan.
__global__ void k_plan(const Scene *scenes, int num_scenes, const uint32_t *tile_offset, int total_tiles,
                       Plan *plan, uint32_t *counts, uint32_t *pcg_vec, uint32_t cap_n2t, uint32_t cap_pair, int *err) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    uint32_t n2t = 0, pair = 0;
    for (int s = 0; s < num_scenes; ++s) {
        const Scene &sc = scenes[s];
        Plan p;
        p.dense_begin = tile_offset[sc.tile_base];
        p.dense_count = tile_offset[sc.tile_base + sc.num_tiles] - p.dense_begin;
        p.n2t_base = n2t;
        p.n2t_count = 4u * p.dense_count + 2u * sc.num_edges + sc.num_nodes + 4u * sc.num_features;
        p.pair_base = pair;
        p.pair_count = 6u * p.dense_count + sc.num_edges + 6u * sc.num_features;
        p.pad[0] = p.pad[1] = 0;
        n2t += p.n2t_count;
        pair += p.pair_count;
        plan[s] = p;
        pcg_vec[s] = 0;   // raised by k_pcg_plan
    }
    if (n2t > cap_n2t || pair > cap_pair) {
        set_error(err, WS_ERR_CAPACITY);
        n2t = min(n2t, cap_n2t);
        pair = min(pair, cap_pair);
    }
    counts[kCntDense] = tile_offset[total_tiles];
    counts[kCntN2T] = n2t;
    counts[kCntPairKV] = pair;
    counts[kCntPcgCost] = counts[kCntPcgCost + 1] = 0;   // raised by k_pcg_plan
}

// Node-graph edge endpoints clamped into the scene (an out-of-range id flags WS_ERR_INVALID_ARGUMENT).
__device__ __forceinline__ void edge_ends(const Scene &sc, uint32_t e, uint16_t &x, uint16_t &y, int *err) {
    x = sc.edges[3 * e];
    y = sc.edges[3 * e + 1];
    const uint16_t last = (uint16_t)(sc.num_nodes - 1);
    if (x > last || y > last) {
        set_error(err, WS_ERR_INVALID_ARGUMENT);
        x = min(x, last);
        y = min(y, last);
    }
}

__device__ __forceinline__ ushort4 clamp_knn(ushort4 k, const Scene &sc, int *err) {
    const uint16_t last = (uint16_t)(sc.num_nodes - 1);
    if (k.x > last || k.y > last || k.z > last || k.w > last) {
        set_error(err, WS_ERR_INVALID_ARGUMENT);
        k = make_ushort4(min(k.x, last), min(k.y, last), min(k.z, last), min(k.w, last));
    }
    return k;
}


// Node->term keys and values (buildTermKeyValueKernel, examples/mono_star/opt/Node2TermsIndex.cu:6-76):
// keys are global node ids, values are the scene-local term ids of the reference's term space
// [dense | reg | node-motion | feature]; self edges get the invalid key.  Per scene the entries
// sit at plan.n2t_base as [4 per dense term | 2 per edge | 1 per node | 4 per feature].  One
// thread per dense term writes that term's 4 entries (its scene from the compaction), and
// one block row per scene writes the scene's other entries, so no entry searches for its scene.
constexpr uint32_t kTailBlocks = 16;
__device__ __forceinline__ void n2t_kv_dense(uint32_t block, uint32_t blocks, const Scene *scenes, const Plan *plan,
                                             const uint32_t *counts, const uint32_t *term_scene,
                                             const ushort4 *dense_knn, uint32_t *keys, uint32_t *vals) {
    const uint32_t n = counts[kCntDense];
    for (uint32_t t = block * blockDim.x + threadIdx.x; t < n; t += blocks * blockDim.x) {
        const uint32_t s = term_scene[t];
        const Plan &p = plan[s];
        const uint32_t lt = t - p.dense_begin, base = p.n2t_base + 4u * lt, nb = scenes[s].node_base;
        const ushort4 k4 = dense_knn[t];
        keys[base] = nb + k4.x;
        keys[base + 1] = nb + k4.y;
        keys[base + 2] = nb + k4.z;
        keys[base + 3] = nb + k4.w;
        vals[base] = vals[base + 1] = vals[base + 2] = vals[base + 3] = lt;
    }
}

__device__ __forceinline__ void n2t_kv_tail(uint32_t s, uint32_t block, const Scene *scenes, const Plan *plan,
                                            uint32_t *keys, uint32_t *vals, uint32_t invalid_key, int *err) {
    const Scene &sc = scenes[s];
    const Plan &p = plan[s];
    const uint32_t nd = p.dense_count, ne = sc.num_edges, nn = sc.num_nodes, nf = sc.num_features;
    const uint32_t len = 2u * ne + nn + 4u * nf, base = p.n2t_base + 4u * nd;
    for (uint32_t j0 = block * blockDim.x + threadIdx.x; j0 < len; j0 += kTailBlocks * blockDim.x) {
        uint32_t j = j0, key, val;
        if (j < 2u * ne) {
            const uint32_t e = j >> 1;
            uint16_t x, y;
            edge_ends(sc, e, x, y, err);
            key = (x != y) ? sc.node_base + ((j & 1u) ? y : x) : invalid_key;
            val = nd + e;
        } else if ((j -= 2u * ne) < nn) {
            key = sc.node_base + j;
            val = nd + ne + j;
        } else {
            j -= nn;
            const uint32_t f = j >> 2;
            const ushort4 k4 = clamp_knn(sc.feature_knn[f], sc, err);
            const uint32_t slot = j & 3u;
            const uint16_t id = slot == 0 ? k4.x : slot == 1 ? k4.y : slot == 2 ? k4.z : k4.w;
            key = sc.node_base + id;
            val = nd + ne + nn + f;
        }
        keys[base + j0] = key;
        vals[base + j0] = val;
    }
}

// The first kTailBlocks blocks of every scene write its edge, node and feature entries, the others the dense ones.
__global__ void __launch_bounds__(256) k_n2t_kv(const Scene *scenes, int num_scenes, const Plan *plan,
                                                const uint32_t *counts, const uint32_t *term_scene,
                                                const ushort4 *dense_knn, uint32_t *keys, uint32_t *vals,
                                                uint32_t invalid_key, int *err) {
    const uint32_t tails = kTailBlocks * (uint32_t)num_scenes;
    if (blockIdx.x < tails)
        n2t_kv_tail(blockIdx.x / kTailBlocks, blockIdx.x % kTailBlocks, scenes, plan, keys, vals, invalid_key, err);
    else
        n2t_kv_dense(blockIdx.x - tails, gridDim.x - tails, scenes, plan, counts, term_scene, dense_knn, keys, vals);
}

// computeTermOffsetKernel (Node2TermsIndex.cu:78-121) as a lower bound per node.
// Also clears the pairs' counts below the diagonal for the pair map.
__global__ void k_n2t_offsets(const uint32_t *sorted_keys, const uint32_t *counts, uint32_t total_nodes,
                              uint32_t *offsets, uint32_t *row_cnt_lo) {
    const uint32_t n = counts[kCntN2T];
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g <= total_nodes; g += gridDim.x * blockDim.x) {
        if (g < total_nodes) row_cnt_lo[g] = 0;
        uint32_t lo = 0, hi = n;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (sorted_keys[mid] < g) lo = mid + 1; else hi = mid;
        }
        offsets[g] = lo;
    }
}

// ---------------------------------------------------------------------------
// Node pair -> term map (computeKVNodePairKNN + sort + segmentNodePairKernel +
// compactNodePairKeyKernel, NodePair2TermsIndex.cu:11-169), built row by row from the sorted
// node -> term map instead of by sorting one key per (pair, term).
// The reference's sorted list holds, for a pair i < j, one entry of term t for every way t
// touches both nodes: for a dense or feature term, each knn slot holding i times each slot holding
// j (slot pairs with id_a < id_b); for a non-self edge (i, j) or (j, i), one entry; in term order.
// Row i's node -> term list holds t once per slot of i, in term order, so emitting, for each entry
// of the list, the term's nodes above i (every knn slot above i; the other end of an edge) yields
// exactly row i's entries, each pair's in term order.  The pairs are sorted by (row, column), so
// row i's pairs and entries are one contiguous range after those of the rows before it.
// Pass 1 counts each column's entries in a small hash table in shared memory and keeps the row's
// columns sorted; two scans give every row its first pair and first entry; pass 2 writes the pairs
// and places every entry at its pair's next free position.
// What bounds them: the latency of a list's words and of its terms' nodes while rows are few, the
// instructions per entry when there are many.  Hence W warps to a row where rows are few and long
// (each takes a run of whole chunks and counts it apart, so that pass 2 knows where its entries of a
// pair begin), the loads of the next two chunks in flight, and a table whose first probe nearly
// always finds the column.  Both passes together, a warp a row without the pipeline / now: 500
// nodes, lists of some 2000 entries 219 -> 35 us; 3000 nodes with 720p images 339 -> 84; 1800 nodes
// 101 -> 30; 8000 nodes 78 -> 44; 64 scenes of 500 to 8000 nodes 1308 -> 909.
// ---------------------------------------------------------------------------
constexpr int kRowHash = 128;        // hash slots per row (twice kRowPairsMax)
constexpr int kRowWarps = 4;         // warps per block when a warp has a row to itself
constexpr int kRowBlocks = 10;       // such blocks per SM: 64 scenes 909 us; 8 blocks 941, 12 blocks 995
constexpr int kRowLanesEntries = 2;  // list entries per lane and pass (loads in flight)
constexpr int kRowChunk = 32 * kRowLanesEntries;   // list entries per pass
constexpr int kRowStage = 3 * kRowChunk;           // their candidates (at most 3 each)

constexpr uint32_t kNoCol = 0xFFFFFFFFu;

// List entry `t`'s (scene-local term id) nodes, local to the scene: a dense or feature term's four,
// an edge's other end.  What adds no pair to the row (nothing there, a node-motion term, the
// absent slots of an edge) is the row's own node, which is not above itself.
__device__ __forceinline__ ushort4 row_entry_nodes(const Scene &sc, const Plan &p, const ushort4 *dense_knn,
                                                   uint32_t local, uint32_t t, int *err) {
    const uint32_t nd = p.dense_count, ne = (uint32_t)sc.num_edges, nn = (uint32_t)sc.num_nodes;
    const uint16_t l = (uint16_t)local;
    ushort4 k = make_ushort4(l, l, l, l);
    if (t == kNoCol) return k;
    if (t < nd) {
        k = dense_knn[p.dense_begin + t];
    } else if (t >= nd + ne + nn) {
        k = clamp_knn(sc.feature_knn[t - nd - ne - nn], sc, err);
    } else if (t < nd + ne) {
        uint16_t x, y;
        edge_ends(sc, t - nd, x, y, err);
        k.x = x == l ? y : x;   // a self edge is in no list
    }
    return k;
}

// A warp's share of a row's list, kRowChunk entries at a time: lane l has entries base + 32 q + l, so
// every load instruction is coalesced and a lane has kRowLanesEntries gathers in flight.  The words
// of the chunk after next and the nodes of the next one are on the way while a chunk is worked on:
// both loads' latencies, some 1500 cycles together, otherwise stand before every chunk.
__device__ __forceinline__ void row_words(uint32_t (&t)[kRowLanesEntries], const uint32_t *n2t_val, uint32_t base,
                                          uint32_t end, int lane) {
#pragma unroll
    for (int q = 0; q < kRowLanesEntries; ++q) {
        const uint32_t e = base + 32u * q + (uint32_t)lane;
        t[q] = e < end ? n2t_val[e] : kNoCol;
    }
}

// Calls use(t, k) for every chunk of entries beg .. end - 1, in order.
template <class F>
__device__ __forceinline__ void row_walk(const Scene &sc, const Plan &p, const ushort4 *dense_knn,
                                         const uint32_t *n2t_val, uint32_t local, uint32_t beg, uint32_t end, int lane,
                                         int *err, F &&use) {
    if (beg >= end) return;
    uint32_t t[kRowLanesEntries], t_next[kRowLanesEntries], t_after[kRowLanesEntries];
    ushort4 k[kRowLanesEntries], k_next[kRowLanesEntries];
    row_words(t, n2t_val, beg, end, lane);
    const bool longer = beg + kRowChunk < end;
    if (longer) row_words(t_next, n2t_val, beg + kRowChunk, end, lane);
#pragma unroll
    for (int q = 0; q < kRowLanesEntries; ++q) k[q] = row_entry_nodes(sc, p, dense_knn, local, t[q], err);
    for (uint32_t base = beg;;) {
        const bool more = base + kRowChunk < end;
        if (more) {
            row_words(t_after, n2t_val, base + 2 * kRowChunk, end, lane);
#pragma unroll
            for (int q = 0; q < kRowLanesEntries; ++q)
                k_next[q] = row_entry_nodes(sc, p, dense_knn, local, t_next[q], err);
        }
        use(t, k);
        if (!more) return;
        base += kRowChunk;
#pragma unroll
        for (int q = 0; q < kRowLanesEntries; ++q) {
            t[q] = t_next[q];
            t_next[q] = t_after[q];
            k[q] = k_next[q];
        }
    }
}

// Entries beg .. end - 1 of a row's list that warp w of W walks: whole chunks, the same in both passes.
template <int W>
__device__ __forceinline__ void row_share(uint32_t &beg, uint32_t &end, int w) {
    if (W == 1) return;
    const uint32_t chunks = (end - beg + kRowChunk - 1) / kRowChunk, share = (chunks + W - 1) / W * kRowChunk;
    const uint32_t b = beg + (uint32_t)w * share;
    beg = min(b, end);
    end = min(beg + share, end);
}

template <int W>
__device__ __forceinline__ void row_sync() {
    if (W == 1) __syncwarp();
    else __syncthreads();
}

__device__ __forceinline__ uint32_t col_hash(uint32_t c) { return (c * 2654435761u) >> (32 - 7); }

template <int W>
__global__ void __launch_bounds__(32 * (W == 1 ? kRowWarps : W), (W == 1 ? kRowBlocks : 1)) k_pair_rows_count(
    const Scene *scenes, const Plan *plan, const uint32_t *node_scene, uint32_t total_nodes,
    const uint32_t *n2t_offset, const uint32_t *n2t_val, uint32_t cap_n2t, const ushort4 *dense_knn, uint32_t *row_cols,
    uint32_t *row_cnts, uint32_t *row_pairs, uint32_t *row_entries, int *err) {
    static_assert(kRowHash == 128, "col_hash gives 7 bits");
    constexpr int kRows = W == 1 ? kRowWarps : 1;   // rows a block has in hand
    __shared__ uint32_t hkey[kRows][kRowHash], hcnt[kRows][W][kRowHash];
    __shared__ uint32_t lcol[kRows][kRowHash], lslot[kRows][kRowHash];
    __shared__ int hfull[kRows];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int r = W == 1 ? wib : 0, w = W == 1 ? 0 : wib;
    volatile uint32_t *keys = hkey[r];
    uint32_t *cnts = hcnt[r][w];
    const unsigned lower = (1u << lane) - 1u;
    for (uint32_t row = blockIdx.x * kRows + r; row < total_nodes; row += gridDim.x * kRows) {
        for (int k = lane; k < kRowHash; k += 32) {
            if (w == 0) keys[k] = kNoCol;
            cnts[k] = 0;
        }
        if (w == 0 && lane == 0) hfull[r] = 0;
        row_sync<W>();
        const uint32_t s = node_scene[row];
        const Scene &sc = scenes[s];
        const Plan &p = plan[s];
        const uint32_t nb = (uint32_t)sc.node_base, local = row - nb;
        uint32_t beg = n2t_offset[row], end = n2t_offset[row + 1];
        row_share<W>(beg, end, w);
        if (lane == 0 && end > beg + kRowChunk) l2_prefetch_list(n2t_val, beg + kRowChunk, end, cap_n2t);
        // almost every candidate finds its column at the first place it looks
        auto count = [&](uint32_t node) {
            uint32_t slot = col_hash(node);
            uint32_t key = keys[slot];
            const bool above = node > local;
            if (above && key != node) {
                int probe = 0;
                for (; probe < kRowHash; ++probe) {
                    if (key == kNoCol) key = atomicCAS(&hkey[r][slot], kNoCol, node);
                    if (key == kNoCol || key == node) break;
                    slot = (slot + 1) & (kRowHash - 1);
                    key = keys[slot];
                }
                if (probe == kRowHash) hfull[r] = 1;
            }
            if (above) atomicAdd(&cnts[slot], 1u);
        };
        row_walk(sc, p, dense_knn, n2t_val, local, beg, end, lane, err,
                 [&](const uint32_t (&)[kRowLanesEntries], const ushort4 (&k)[kRowLanesEntries]) {
#pragma unroll
                     for (int q = 0; q < kRowLanesEntries; ++q) {
                         count(k[q].x);
                         count(k[q].y);
                         count(k[q].z);
                         count(k[q].w);
                     }
                 });
        row_sync<W>();
        // the table's columns, compacted in slot order, then ranked by column
        if (w == 0) {
            uint32_t n_cols = 0;
            for (int q = 0; q < kRowHash / 32; ++q) {
                const uint32_t c = keys[32 * q + lane];
                const unsigned occ = __ballot_sync(0xffffffffu, c != kNoCol);
                if (c != kNoCol) {
                    const uint32_t idx = n_cols + (uint32_t)__popc(occ & lower);
                    lcol[r][idx] = c;
                    lslot[r][idx] = (uint32_t)(32 * q + lane);
                }
                n_cols += (uint32_t)__popc(occ);
            }
            __syncwarp();
            const bool full = hfull[r] != 0 || n_cols > (uint32_t)kRowPairsMax;
            if (full) {
                if (lane == 0) set_error(err, WS_ERR_CAPACITY);
                n_cols = 0;
            }
            uint32_t entries = 0;
            for (uint32_t x = (uint32_t)lane; x < n_cols; x += 32) {
                const uint32_t c = lcol[r][x];
                uint32_t rank = 0;
                for (uint32_t y = 0; y < n_cols; ++y) rank += lcol[r][y] < c ? 1u : 0u;
                row_cols[(size_t)kRowPairsMax * row + rank] = nb + c;
#pragma unroll
                for (int v = 0; v < W; ++v) {
                    const uint32_t n = hcnt[r][v][lslot[r][x]];
                    row_cnts[((size_t)W * row + v) * kRowPairsMax + rank] = n;
                    entries += n;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) entries += __shfl_xor_sync(0xffffffffu, entries, o);
            if (lane == 0) {
                row_pairs[row] = n_cols;
                row_entries[row] = entries;
            }
        }
        row_sync<W>();
    }
}

template <int W>
__global__ void __launch_bounds__(32 * (W == 1 ? kRowWarps : W), (W == 1 ? kRowBlocks : 1)) k_pair_rows_fill(
    const Scene *scenes, const Plan *plan, const uint32_t *node_scene, uint32_t total_nodes,
    const uint32_t *n2t_offset, const uint32_t *n2t_val, uint32_t cap_n2t, const ushort4 *dense_knn, const uint32_t *row_cols,
    const uint32_t *row_cnts, const uint32_t *pair_first, const uint32_t *entry_first, uint32_t cap_half,
    uint32_t cap_kv, uint32_t *half_row, uint32_t *half_col, uint32_t *half_begin, uint32_t *half_end,
    uint32_t *half_scene, uint32_t *row_cnt_lo, uint32_t *pair_val, uint32_t *counts, int *err) {
    constexpr int kWarps = W == 1 ? kRowWarps : W, kRows = W == 1 ? kRowWarps : 1;
    __shared__ uint32_t hkey[kRows][kRowHash];   // place among the row's columns << 16 | node
    __shared__ uint32_t s_next[kWarps][kRowPairsMax];
    __shared__ uint32_t st_term[kWarps][kRowStage];
    __shared__ uint16_t st_node[kWarps][kRowStage];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int r = W == 1 ? wib : 0, w = W == 1 ? 0 : wib;
    uint32_t *next = s_next[wib], *term = st_term[wib];
    uint16_t *node = st_node[wib];
    const unsigned lower = (1u << lane) - 1u;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        counts[kCntHalf] = min(pair_first[total_nodes], cap_half);
        if (pair_first[total_nodes] > cap_half) set_error(err, WS_ERR_CAPACITY);
    }
    for (uint32_t row = blockIdx.x * kRows + r; row < total_nodes; row += gridDim.x * kRows) {
        const uint32_t h0 = pair_first[row], n_cols = pair_first[row + 1] - h0;
        if (n_cols == 0) continue;
        const uint32_t s = node_scene[row];
        const Scene &sc = scenes[s];
        const Plan &p = plan[s];
        const uint32_t nb = (uint32_t)sc.node_base, local = row - nb;
        if (w == 0)
            for (int k = lane; k < kRowHash; k += 32) hkey[r][k] = kNoCol;
        row_sync<W>();
        // the row's pairs: columns ascending, entry ranges one after another from the row's first; in a
        // pair's range the warps' shares one after another
        uint32_t carry = entry_first[row];
        for (uint32_t k0 = 0; k0 < n_cols; k0 += 32) {
            const uint32_t k = k0 + (uint32_t)lane;
            const uint32_t c = k < n_cols ? row_cols[(size_t)kRowPairsMax * row + k] : kNoCol;
            uint32_t n = 0, before = 0;
#pragma unroll
            for (int v = 0; v < W; ++v) {
                const uint32_t m = k < n_cols ? row_cnts[((size_t)W * row + v) * kRowPairsMax + k] : 0u;
                before += v < w ? m : 0u;
                n += m;
            }
            const uint32_t incl = warp_incl_scan_u32(n);
            const uint32_t begin = carry + incl - n;
            carry += __shfl_sync(0xffffffffu, incl, 31);
            if (k < n_cols) {
                next[k] = begin + before;
                if (w == 0) {
                    uint32_t slot = col_hash(c - nb);
                    for (int probe = 0; probe < kRowHash; ++probe) {
                        if (atomicCAS(&hkey[r][slot], kNoCol, k << 16 | (c - nb)) == kNoCol) break;
                        slot = (slot + 1) & (kRowHash - 1);
                    }
                    const uint32_t h = h0 + k;
                    if (h < cap_half) {
                        half_row[h] = row;
                        half_col[h] = c;
                        half_begin[h] = begin;
                        half_end[h] = begin + n;
                        half_scene[h] = s;
                        atomicAdd(&row_cnt_lo[c], 1u);
                    }
                }
            }
        }
        row_sync<W>();
        uint32_t beg = n2t_offset[row], end = n2t_offset[row + 1];
        row_share<W>(beg, end, w);
        if (lane == 0 && end > beg + kRowChunk) l2_prefetch_list(n2t_val, beg + kRowChunk, end, cap_n2t);
        row_walk(sc, p, dense_knn, n2t_val, local, beg, end, lane, err,
                 [&](const uint32_t (&t)[kRowLanesEntries], const ushort4 (&k)[kRowLanesEntries]) {
            // the chunk's candidates, staged in list order as (node, term)
            uint32_t total = 0;
#pragma unroll
            for (int q = 0; q < kRowLanesEntries; ++q) {
                const uint32_t n = min((uint32_t)(k[q].x > local) + (uint32_t)(k[q].y > local) +
                                           (uint32_t)(k[q].z > local) + (uint32_t)(k[q].w > local), 3u);
                const uint32_t incl = warp_incl_scan_u32(n), stop = total + incl;
                uint32_t at = stop - n;
                auto stage = [&](uint32_t v) {
                    if (v > local && at < stop) {
                        node[at] = (uint16_t)v;
                        term[at] = t[q];
                        ++at;
                    }
                };
                stage(k[q].x);
                stage(k[q].y);
                stage(k[q].z);
                stage(k[q].w);
                total += __shfl_sync(0xffffffffu, incl, 31);
            }
            __syncwarp();
            for (uint32_t v0 = 0; v0 < total; v0 += 32) {
                const uint32_t v = v0 + (uint32_t)lane;
                const uint32_t c = v < total ? (uint32_t)node[v] : kNoCol;
                const unsigned peers = __match_any_sync(0xffffffffu, c);
                uint32_t slot = col_hash(c), kk = kNoCol;
                if (v < total) {
                    uint32_t key = hkey[r][slot];
                    for (int probe = 0; probe < kRowHash && (key & 0xFFFFu) != c && key != kNoCol; ++probe) {
                        slot = (slot + 1) & (kRowHash - 1);
                        key = hkey[r][slot];
                    }
                    kk = (key & 0xFFFFu) == c ? key >> 16 : kNoCol;
                }
                if (kk < n_cols) {
                    const uint32_t pos = next[kk] + (uint32_t)__popc(peers & lower);
                    if (pos < cap_kv) pair_val[pos] = term[v];
                }
                __syncwarp();
                if (kk < n_cols && (peers & lower) == 0) next[kk] += (uint32_t)__popc(peers);
                __syncwarp();
            }
        });
        row_sync<W>();
    }
}

// For the block CSR: every row's first pair and lengths, and the pairs keyed by column for their sort.
__global__ void k_csr_rows(const uint32_t *half_row, const uint32_t *half_col, const uint32_t *counts, const uint32_t *up,
                           const uint32_t *lo, uint32_t total_nodes, uint32_t *row_first, uint32_t *len, uint32_t *items,
                           uint32_t *keys, uint32_t *vals) {
    const uint32_t n = counts[kCntHalf], first = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    for (uint32_t g = first; g < total_nodes; g += stride) {
        len[g] = 1u + up[g] + lo[g];
        items[g] = 1u + up[g];   // stored blocks of the row: the diagonal and the upper pairs
    }
    for (uint32_t h = first; h < n; h += stride) {
        const uint32_t row = half_row[h];
        if (h == 0 || half_row[h - 1] != row) row_first[row] = h;
        keys[h] = half_col[h];
        vals[h] = h;
    }
}

// Block-CSR slots: every row is [diagonal, columns < row ascending, columns > row ascending],
// which is the sorted symmetric pair order of computeSymmetricNodePairKernel + sort
// (NodePair2TermsIndex.cu:171-192, 656-675) with the diagonal block placed first as in the
// Bin-Blocked CSR (NodePairRowColumnIndex.cu:110-124).  Also the item record of every pair
// h = (row, col) of the symmetric store (item h + row + 1): its lower entry is its position
// k among the pairs sorted by column (then row).
// Then the diagonal slot of every row, and the item records of the row's diagonal item (the row, marked
// as a row start, and its scene).
__global__ void k_slots(const uint32_t *sorted_col, const uint32_t *sorted_h, const uint32_t *counts,
                        const uint32_t *half_row, const uint32_t *half_col, const uint32_t *row_first,
                        const uint32_t *row_cnt_lo, const uint32_t *rowptr, uint32_t cap_blocks,
                        uint32_t *slot_up, uint32_t *slot_lo, uint32_t *colidx, uint2 *item_info,
                        uint32_t *item_col, const uint32_t *item_ptr, const uint32_t *node_scene, uint32_t total_nodes,
                        int *err) {
    const uint32_t n = counts[kCntHalf];
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const uint32_t col = sorted_col[k];
        uint32_t lo = 0, hi = k;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (sorted_col[mid] < col) lo = mid + 1; else hi = mid;
        }
        const uint32_t rank_lo = k - lo;
        const uint32_t h = sorted_h[k];
        const uint32_t row = half_row[h];
        const uint32_t s_lo = rowptr[col] + 1u + rank_lo;
        const uint32_t s_up = rowptr[row] + 1u + row_cnt_lo[row] + (h - row_first[row]);
        if (s_lo >= cap_blocks || s_up >= cap_blocks) {
            set_error(err, WS_ERR_CAPACITY);
            slot_lo[h] = slot_up[h] = kInvalidIndex;
            continue;
        }
        slot_lo[h] = s_lo;
        slot_up[h] = s_up;
        colidx[s_lo] = row;
        colidx[s_up] = half_col[h];
        item_info[h + row + 1u] = make_uint2(half_col[h], k);
        item_col[h + row + 1u] = half_col[h];
    }
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < total_nodes; g += gridDim.x * blockDim.x) {
        const uint32_t s = rowptr[g];
        if (s < cap_blocks) colidx[s] = g;
        // the row's first item is its diagonal block
        item_info[item_ptr[g]] = make_uint2(g | kItemRowStart, node_scene[g]);
        item_col[item_ptr[g]] = g | kItemRowStart;
        if (g + 1 == total_nodes && rowptr[total_nodes] > cap_blocks) set_error(err, WS_ERR_CAPACITY);
    }
}

// First row group of every PCG phase-A work unit (kPcgUnitsPerWarp per warp), chosen so that the
// units' stored blocks (items) are about equal.  The groups before `split` (the first half of the
// scenes) and the groups from `split` on get separate units, their numbers in proportion to
// their items (at least one each when both halves have groups): unit w of a half starts at the
// first group of the half whose first item is at or past w / units of the half's items.
// warp_groups[units] is the group count and warp_groups[units + 1] the first half's units.
// unit_info[2w], [2w + 1] describe unit w for the PCG: its groups, rows and items (first, end)
// and the scenes of its first and last group, so that a unit starts from one load.
struct UnitSplit {
    uint32_t split, mid, total, ux, units, groups;
};
__device__ uint32_t unit_first_group(const UnitSplit &U, uint32_t w, const uint32_t *item_ptr,
                                     const uint32_t *group_row, uint32_t total_nodes) {
    if (w >= U.units) return U.groups;
    uint32_t lo, hi, target;
    if (w < U.ux) {
        lo = 0;
        hi = U.split;
        target = (uint32_t)(((unsigned long long)U.mid * w) / U.ux);
    } else {
        lo = U.split;
        hi = U.groups;
        target = U.mid + (uint32_t)(((unsigned long long)(U.total - U.mid) * (w - U.ux)) / (U.units - U.ux));
    }
    while (lo < hi) {
        const uint32_t m = (lo + hi) >> 1;
        if (item_ptr[min(group_row[m], total_nodes)] < target) lo = m + 1;
        else hi = m;
    }
    return lo;
}

__global__ void k_pcg_ranges(const uint32_t *item_ptr, const uint32_t *group_row, const uint32_t *group_scene,
                             uint32_t groups, uint32_t split, uint32_t total_nodes, uint32_t cap_items, uint32_t units,
                             uint32_t *warp_groups, uint4 *unit_info) {
    UnitSplit U;
    U.units = units;
    U.groups = groups;
    U.total = min(item_ptr[total_nodes], cap_items);
    U.split = min(split, groups);
    U.mid = U.split < groups ? min(item_ptr[min(group_row[U.split], total_nodes)], U.total) : U.total;
    U.ux = units;
    if (U.split > 0 && U.split < groups && units > 1) {
        U.ux = (uint32_t)(((unsigned long long)units * U.mid + U.total / 2) / max(U.total, 1u));
        U.ux = min(max(U.ux, 1u), units - 1);
    }
    for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w <= units + 1; w += gridDim.x * blockDim.x) {
        if (w >= units) {
            warp_groups[w] = (w == units) ? groups : U.ux;
            continue;
        }
        const uint32_t g0 = unit_first_group(U, w, item_ptr, group_row, total_nodes);
        const uint32_t g1 = max(g0, unit_first_group(U, w + 1, item_ptr, group_row, total_nodes));
        warp_groups[w] = g0;
        const uint32_t r0 = g0 < groups ? min(group_row[g0], total_nodes) : total_nodes;
        const uint32_t r1 = g1 < groups ? min(group_row[g1], total_nodes) : total_nodes;
        const uint32_t s0 = g0 < g1 ? group_scene[g0] : 0u, s1 = g0 < g1 ? group_scene[g1 - 1] : 0u;
        unit_info[2 * w] = make_uint4(g0, g1, r0, r1);
        unit_info[2 * w + 1] = make_uint4(min(item_ptr[r0], cap_items), min(item_ptr[r1], cap_items), s0, s1);
    }
}

static inline int grid_for(uint32_t n, int threads, int num_sms, uint32_t per_sm = 8u) {
    const uint32_t want = (n + threads - 1) / threads;
    const uint32_t cap = (uint32_t)num_sms * per_sm;
    return (int)std::max<uint32_t>(1u, std::min<uint32_t>(want, cap));
}

// Warps to a row of the pair map.  Several pay while rows are few and their lists long (pixels a node
// say how long), one where rows fill the chip.  The whole index, 1 / 4 / 8 warps to a row, us:
//   500 nodes, 614 px a node 372 / 263 / 239; 1000, 307 px 376 / 296 / 282; 1800, 171 px 341 / 292 / 296;
//   3000, 102 px 341 / 304 / 318; 3000, 307 px 458 / 365 / 371; 5000, 184 px 429 / 382 / 410;
//   8000, 38 px 334 / 360 / 407; 8000, 115 px 401 / 410 / 449; 8 x 500 nodes 538 / 464 / 470;
//   20 x 500 nodes 879 / 812 / 867; 8 x 1800 nodes 521 / 540 / 620.
static int pair_row_warps(const Workspace &w) {
    const uint64_t pixels = scene_pixels(w), n = w.total_nodes;
    if (n <= kRowWide8 && pixels >= 250 * n) return 8;
    if ((n <= 6000 && pixels >= 75 * n) || (n <= kRowWide4 && pixels >= 300 * n)) return 4;
    return 1;
}

// Node pair -> term map, row by row from the node -> term map (see k_pair_rows_count).
template <int W>
static void pair_index_rows(Workspace &w, cudaStream_t st) {
    const uint32_t N = w.total_nodes;
    const int threads = 32 * (W == 1 ? kRowWarps : W);
    const int grid = grid_for(N * 32u * W, threads, w.num_sms, 16);
    k_pair_rows_count<W><<<grid, threads, 0, st>>>(w.scenes, w.plan, w.node_scene, N, w.n2t_offset, w.n2t_sorted_val,
                                                   w.cap_n2t, w.d_knn, w.row_pair_cols, w.row_pair_cnts, w.row_cnt_up,
                                                   w.row_entry_first, w.error_flag);
    count_launch(w, exclusive_scan2(w.row_cnt_up, w.row_pair_first, w.row_entry_first, w.row_entry_first, N, w.scan_tmp, st));
    k_pair_rows_fill<W><<<grid, threads, 0, st>>>(w.scenes, w.plan, w.node_scene, N, w.n2t_offset, w.n2t_sorted_val,
                                                  w.cap_n2t, w.d_knn, w.row_pair_cols, w.row_pair_cnts,
                                                  w.row_pair_first, w.row_entry_first, w.cap_half, w.cap_pair_kv,
                                                  w.half_row, w.half_col, w.half_begin, w.half_end, w.half_scene,
                                                  w.row_cnt_lo, w.pair_val, w.counts, w.error_flag);
    count_launch(w, 1 + 1);
}

static void pair_index(Workspace &w, cudaStream_t st) {
    switch (pair_row_warps(w)) {
        case 8: pair_index_rows<8>(w, st); break;
        case 4: pair_index_rows<4>(w, st); break;
        default: pair_index_rows<1>(w, st);
    }
    w.pair_sorted_val = w.pair_val;
}

cudaError_t index_build(Workspace &w, cudaStream_t st) {
    const int S = w.num_scenes;
    const int T = (int)w.total_tiles;
    const uint32_t N = w.total_nodes;
    // 1. compaction of potential pixels
    k_pixel_count<<<T, kPixTileThreads, 0, st>>>(w.scenes, w.tile_scene, T, w.tile_count);
    count_launch(w, 1 + exclusive_scan(w.tile_count, w.tile_count, (uint32_t)T, w.scan_tmp, st));
    k_plan<<<1, 32, 0, st>>>(w.scenes, S, w.tile_count, T, w.plan, w.counts, w.pcg_vec, w.cap_n2t, w.cap_pair_kv, w.error_flag);
    k_pixel_compact<<<T, kPixTileThreads, 0, st>>>(w.scenes, w.tile_scene, T, w.tile_count, w.d_pixels, w.d_knn,
                                                   w.d_sw, w.d_cw, w.d_scene, w.cap_pixels, w.error_flag);
    count_launch(w, 2);
    // 2. node -> term
    const uint32_t n2t_invalid = (1u << w.node_bits) - 1u;
    k_n2t_kv<<<kTailBlocks * S + grid_for(w.cap_pixels, 256, w.num_sms), 256, 0, st>>>(
        w.scenes, S, w.plan, w.counts, w.d_scene, w.d_knn, w.n2t_key, w.n2t_val, n2t_invalid, w.error_flag);
    count_launch(w);
    const bool n2t_alt = radix_sort<uint32_t>(w.n2t_key, w.n2t_val, w.n2t_key_alt, w.n2t_val_alt, w.counts + kCntN2T, 0,
                                              w.cap_n2t, w.node_bits, w.sort_hist, w.sort_digit, st);
    count_launch(w, 3 * radix_passes(w.node_bits));
    w.n2t_sorted_key = n2t_alt ? w.n2t_key_alt : w.n2t_key;
    w.n2t_sorted_val = n2t_alt ? w.n2t_val_alt : w.n2t_val;
    k_n2t_offsets<<<grid_for(N + 1, 256, w.num_sms), 256, 0, st>>>(w.n2t_sorted_key, w.counts, N, w.n2t_offset,
                                                                  w.row_cnt_lo);
    count_launch(w);
    // 3. node pair -> term
    pair_index(w, st);
    // 4. block CSR
    k_csr_rows<<<grid_for(w.cap_half, 256, w.num_sms), 256, 0, st>>>(w.half_row, w.half_col, w.counts, w.row_cnt_up,
                                                                     w.row_cnt_lo, N, w.row_first, w.rowptr, w.item_ptr,
                                                                     w.col_key, w.col_val);
    count_launch(w, exclusive_scan2(w.rowptr, w.rowptr, w.item_ptr, w.item_ptr, N, w.scan_tmp, st));
    const bool col_alt = radix_sort<uint32_t>(w.col_key, w.col_val, w.col_key_alt, w.col_val_alt, w.counts + kCntHalf,
                                              0, w.cap_half, w.node_bits, w.sort_hist, w.sort_digit, st);
    count_launch(w, 1 + 3 * radix_passes(w.node_bits));
    const uint32_t *scol = col_alt ? w.col_key_alt : w.col_key;
    const uint32_t *sh = col_alt ? w.col_val_alt : w.col_val;
    k_slots<<<grid_for(w.cap_half, 256, w.num_sms), 256, 0, st>>>(
        scol, sh, w.counts, w.half_row, w.half_col, w.row_first, w.row_cnt_lo, w.rowptr, w.cap_blocks, w.half_slot_up,
        w.half_slot_lo, w.colidx, w.item_info, w.item_col, w.item_ptr, w.node_scene, N, w.error_flag);
    count_launch(w);
    pcg_ranges(w, st);
    return pcg_plan(w, st);
}

void pcg_ranges(Workspace &w, cudaStream_t st) {
    const uint32_t units = (uint32_t)(kPcgUnitsPerWarp * pcg_launch_blocks(w) * pcg_warps_per_block());
    k_pcg_ranges<<<grid_for(units + 2, 256, w.num_sms), 256, 0, st>>>(
        w.item_ptr, w.chunk_row, w.chunk_scene, w.total_chunks, pcg_split_group(w), w.total_nodes, w.cap_items, units,
        w.pcg_warp_groups, w.pcg_unit_info);
    count_launch(w);
}

}  // namespace ws
