// Node graph construction and growth, skinning, forward warp and the solver-map splat.
//
// Integer outputs (node candidates, node and surfel k-NN ids) follow the
// reference bit for bit: the same float expressions with the fused
// multiply-adds spelled out, the same strict-inequality heap, and the same
// Lomuto quicksort.  Weights use __expf as the reference does.
#include <cuda_runtime.h>
#include <cuda_fp16.h>

#include <mutex>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "../../include/warpsolve.h"
#include "ws_common.cuh"
#include "ws_obs_point.cuh"
#include "ws_prims.cuh"

namespace ws {

// Squared length as nvcc contracts `x*x + y*y + z*z` under its default -fmad=true.
__device__ __forceinline__ float sq3_fused(float x, float y, float z) {
    return __fmaf_rn(z, z, __fmaf_rn(y, y, __fmul_rn(x, x)));
}

// KnnHeapExpandDevice (libs/star/geometry/node_graph/brute_force_knn.cuh:52-135).
template <int CAP>
struct Heap {
    float d[CAP];
    uint16_t id[CAP];
    int max_id;
    float max_d;
    __device__ __forceinline__ void init(float v) {
#pragma unroll
        for (int i = 0; i < CAP; ++i) { d[i] = v; id[i] = 0; }
        refresh();
    }
    __device__ __forceinline__ void refresh() {
        max_id = 0;
        max_d = d[0];
#pragma unroll
        for (int i = 1; i < CAP; ++i)
            if (d[i] > max_d) { max_d = d[i]; max_id = i; }
    }
    __device__ __forceinline__ void update(uint16_t idx, float dist) {
        if (dist < max_d) {
#pragma unroll
            for (int i = 0; i < CAP; ++i)
                if (i == max_id) { d[i] = dist; id[i] = idx; }
            refresh();
        }
    }
    // Ascending order.  Distinct distances have one: a sorting network in registers.  With ties the
    // order is that of the reference's quicksort.
    __device__ __forceinline__ void sort() {
        float s[CAP];
        uint16_t k[CAP];
#pragma unroll
        for (int i = 0; i < CAP; ++i) { s[i] = d[i]; k[i] = id[i]; }
#pragma unroll
        for (int round = 0; round < CAP; ++round)   // odd-even transposition
#pragma unroll
            for (int i = round & 1; i + 1 < CAP; i += 2) {
                const bool swap = s[i + 1] < s[i];
                const float a = s[i], b = s[i + 1];
                const uint16_t ka = k[i], kb = k[i + 1];
                s[i] = swap ? b : a;
                s[i + 1] = swap ? a : b;
                k[i] = swap ? kb : ka;
                k[i + 1] = swap ? ka : kb;
            }
        bool strict = true;
#pragma unroll
        for (int i = 0; i + 1 < CAP; ++i) strict = strict && s[i] < s[i + 1];
        if (strict) {
#pragma unroll
            for (int i = 0; i < CAP; ++i) { d[i] = s[i]; id[i] = k[i]; }
        } else {
            quicksort(d, id);
        }
    }
    // Lomuto quicksort on strict <, iterative form of the reference's recursion
    // (same partitions in the same order), on copies, since its run-time indices put the arrays in local memory
    // (as a call it cost the loops around it their registers: 300k surfels on 2000 new nodes 615 -> 660 us; inlined,
    // and with the maximum sought again only when a node has entered, 402).
    static __device__ __forceinline__ void quicksort_arrays(float *d, uint16_t *id) {
        int lo_stack[2 * CAP + 2], hi_stack[2 * CAP + 2];
        int top = 0;
        lo_stack[0] = 0;
        hi_stack[0] = CAP - 1;
        top = 1;
        while (top > 0) {
            --top;
            const int low = lo_stack[top], high = hi_stack[top];
            if (low >= high) continue;
            const float pivot = d[high];
            int i = low - 1;
            for (int j = low; j <= high - 1; ++j) {
                if (d[j] < pivot) {
                    ++i;
                    const float td = d[i]; d[i] = d[j]; d[j] = td;
                    const uint16_t ti = id[i]; id[i] = id[j]; id[j] = ti;
                }
            }
            { const float td = d[i + 1]; d[i + 1] = d[high]; d[high] = td; }
            { const uint16_t ti = id[i + 1]; id[i + 1] = id[high]; id[high] = ti; }
            const int pi = i + 1;
            // recursion order: left part first, then right part
            lo_stack[top] = pi + 1; hi_stack[top] = high; ++top;
            lo_stack[top] = low; hi_stack[top] = pi - 1; ++top;
        }
    }
    static __device__ __forceinline__ void quicksort(float (&d)[CAP], uint16_t (&id)[CAP]) {
        float ld[CAP];
        uint16_t li[CAP];
#pragma unroll
        for (int i = 0; i < CAP; ++i) { ld[i] = d[i]; li[i] = id[i]; }
        quicksort_arrays(ld, li);
#pragma unroll
        for (int i = 0; i < CAP; ++i) { d[i] = ld[i]; id[i] = li[i]; }
    }
};

// createVoxelKeyKernel (libs/star/geometry/sampling/VoxelSubsamplerSorting.cu:8-21) with
// encodeVoxel (libs/star/common/encode_utils.h:138-141).  The reference sorts the encoded keys
// as signed ints; a voxel below -512 in z gives a negative key, which sorts first.  The keys here
// go through an unsigned radix sort, so they carry the sign bit flipped (kVoxelKeyBias), which
// orders them as signed ints; the sampler flips it back before decoding.
constexpr uint32_t kVoxelKeyBias = 0x80000000u;
__global__ void k_voxel_key(const float4 *pts, uint32_t n, float voxel, uint32_t *keys, uint32_t *vals) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 p = pts[i];
        const int vx = __float2int_rd(p.x / voxel), vy = __float2int_rd(p.y / voxel), vz = __float2int_rd(p.z / voxel);
        const int enc = (int)((unsigned)(vx + 512) + (unsigned)(vy + 512) * 1024u + (unsigned)(vz + 512) * 1048576u);
        keys[i] = (uint32_t)enc ^ kVoxelKeyBias;
        vals[i] = i;
    }
}

__global__ void k_voxel_marks(const uint32_t *keys, uint32_t n, uint32_t *marks) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        marks[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1u : 0u;
}

// samplingPointsKernel (VoxelSubsamplerSorting.cu:60-96): per voxel the point nearest the
// voxel centre, first wins on ties.  The centre is a rounded float3 computed before the loop
// over the voxel's points, as the source writes it; the intrinsics keep nvcc from fusing its
// product into the subtraction, which moves squared distances by about 1e-10 m^2 and flips
// near-ties between points (about 2 voxels in 89k on a 1M-point torus).
__global__ void k_voxel_sample(const uint32_t *keys, const uint32_t *perm, const uint32_t *head_off, uint32_t n,
                               const float4 *pts, float voxel, float4 *out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (i != 0 && keys[i] == keys[i - 1]) continue;   // not the first point of its voxel
        uint32_t e = i + 1;
        while (e < n && keys[e] == keys[i]) ++e;
        const int enc = (int)(keys[i] ^ kVoxelKeyBias);
        int z = enc / (1024 * 1024);
        int x = enc % 1024;
        int y = (enc - z * 1024 * 1024) / 1024;
        x -= 512; y -= 512; z -= 512;
        const float cx = __fmul_rn(float(x + 0.5), voxel), cy = __fmul_rn(float(y + 0.5), voxel),
                    cz = __fmul_rn(float(z + 0.5), voxel);
        float best = 1e5f;
        uint32_t bi = i;
        for (uint32_t k = i; k < e; ++k) {
            const float4 p = pts[perm[k]];
            const float dd = sq3_fused(__fsub_rn(p.x, cx), __fsub_rn(p.y, cy), __fsub_rn(p.z, cz));
            if (dd < best) { best = dd; bi = k; }
        }
        out[head_off[i]] = pts[perm[bi]];
    }
}

// ---- Overlap check of the node candidates on the device ----
//
// AppendNodeFromVertexHost (libs/star/geometry/node_graph/NodeGraph.cu:652-704) walks the
// candidates in order and keeps one when no candidate kept before it lies within 0.85 R
// (squared distance <= (0.85 R)^2, summed as ((dx*dx + dy*dy) + dz*dz) + dw*dw with dw = 0).
// That is the lexicographically first maximal independent set of the graph that joins
// candidates within 0.85 R: a candidate is rejected once one of its earlier neighbours is kept, and
// kept once all of them are rejected.  Every decision is final and equals the sequential loop's (by
// induction on the index), and the lowest undecided candidate can always be decided.

// Dedup grid: cells of 1.125 x the overlap radius.  Two candidates that pass the distance test
// differ by at most r (1 + 2^-22) per axis, i.e. 0.889 cells; the scaled coordinates are
// clamped to +-2^18 cells, where a float resolves 1/32 of a cell, so their rounding adds at most
// 1/32 and such candidates lie in the same or adjacent cells.  Cell coordinates wrap at
// `cells` per axis, a power of two, which only adds far candidates that the distance test turns away.  The
// candidates are put in cell order by counting (a table of all cells, counts, a scan, placement): their
// order within a cell is left open, since no decision depends on it.  Sorting them by a 30-bit cell key
// and searching it took 13 launches and 18 binary searches a candidate.
constexpr float kDedupCellScale = 1.125f;
// Cells per axis: 64, and 128 from as many candidates as that table has cells (988k candidates spread over 12 m, R =
// 0.025: 3044 / 2758 us in all, 2.9M 12569 / 7869; the table is cleared and scanned, which few candidates would not pay).
constexpr int kDedupCellsMost = 128;
constexpr int dedup_cells(uint32_t nv) { return nv <= (1u << 18) ? 64 : kDedupCellsMost; }
constexpr uint32_t dedup_table(int cells) { return (uint32_t)cells * cells * cells; }

__device__ __forceinline__ int dedup_cell(float v, float inv_cell) {
    return __float2int_rd(fminf(fmaxf(__fmul_rn(v, inv_cell), -262144.f), 262144.f));
}

__device__ __forceinline__ uint32_t dedup_key(int x, int y, int z, int cells) {
    const int m = cells - 1;
    return (uint32_t)(x & m) + (uint32_t)cells * ((uint32_t)(y & m) + (uint32_t)cells * (uint32_t)(z & m));
}
__device__ __forceinline__ uint32_t dedup_key_of(float4 p, float inv_cell, int cells) {
    return dedup_key(dedup_cell(p.x, inv_cell), dedup_cell(p.y, inv_cell), dedup_cell(p.z, inv_cell), cells);
}

__global__ void k_dedup_count(const float4 *cand, uint32_t nv, float inv_cell, int cells, uint32_t *table, int *err) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += gridDim.x * blockDim.x) {
        const float4 p = cand[i];
        if (isnan(p.x) || isnan(p.y) || isnan(p.z)) atomicOr(err, 1);
        atomicAdd(table + dedup_key_of(p, inv_cell, cells), 1u);
    }
}

// table: first position of every cell; on return the end of every cell (the next one's first).
__global__ void k_dedup_place(const float4 *cand, uint32_t nv, float inv_cell, int cells, uint32_t *table, float4 *placed) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += gridDim.x * blockDim.x) {
        const float4 p = cand[i];
        placed[atomicAdd(table + dedup_key_of(p, inv_cell, cells), 1u)] = make_float4(p.x, p.y, p.z, __uint_as_float(i));
    }
}

// Earlier candidates that overlap candidate i, found in the 3 x 3 rows of three cells around
// it (a row is one range unless its x wraps).  kFill = false counts them into `cnt`;
// kFill = true writes their indices from offset `cnt[i]` of `nbr`.
template <bool kFill>
__global__ void k_dedup_neighbours(const float4 *cand, const uint32_t *cell_end, const float4 *placed, uint32_t nv,
                                   float inv_cell, int cells, float thr, uint32_t *cnt, uint32_t *nbr, uint32_t cap,
                                   int *err) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += gridDim.x * blockDim.x) {
        const float4 p = cand[i];
        const int cx = dedup_cell(p.x, inv_cell), cy = dedup_cell(p.y, inv_cell), cz = dedup_cell(p.z, inv_cell);
        const uint32_t x0 = (uint32_t)((cx - 1) & (cells - 1)), x1 = (uint32_t)((cx + 1) & (cells - 1));
        const int ranges = x0 < x1 ? 1 : 2;
        uint32_t c = 0, out = kFill ? cnt[i] : 0u;
        for (int row = 0; row < 9; ++row) {
            const uint32_t c0 = dedup_key(0, cy + row % 3 - 1, cz + row / 3 - 1, cells);
            for (int q = 0; q < ranges; ++q) {
                const uint32_t lo = c0 + (ranges == 1 || q == 0 ? x0 : 0u);
                const uint32_t hi = c0 + (ranges == 1 || q == 1 ? x1 : (uint32_t)(cells - 1));
                const uint32_t e = __ldg(cell_end + hi);
                for (uint32_t b = lo > 0 ? __ldg(cell_end + lo - 1) : 0u; b < e; ++b) {
                    const float4 o = placed[b];
                    const uint32_t j = __float_as_uint(o.w);
                    if (j >= i) continue;
                    const float ex = o.x - p.x, ey = o.y - p.y, ez = o.z - p.z;
                    const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(ex, ex), __fmul_rn(ey, ey)), __fmul_rn(ez, ez));
                    if (d2 <= thr) {
                        if (!kFill) ++c;
                        else if (out < cap) nbr[out++] = j;
                        else atomicOr(err, 8);
                    }
                }
            }
        }
        if (!kFill) cnt[i] = c;
    }
}
// Overlapping pairs kept per candidate.  A candidate is the only one of its voxel (0.7 R), so a ball of 0.85 R around
// one holds about 7.5 (a volume filled at random; eight voxels' candidates in a common corner see 7 each), half of them
// earlier.  (Where there are more, `err` gets 8 and the lists are made again as long as they need to be; a candidate
// has at most 63 neighbours.)  32 a candidate went past the scratch that the pool keeps: 988k candidates 2758 / 1923
// us, 2.9M 7869 / 5691.
constexpr uint32_t kDedupPairsPerCandidate = 8;

// The decisions, without rounds: thread t takes candidates t, t + T, ... (T threads in all) in turn and
// re-reads a candidate's open earlier neighbours until one is kept (rejected) or none is open (kept).
// Decisions (0 open, 1 kept, 2 rejected; zeroed before the launch) are final and read volatile from L2.
// All blocks are resident (a cooperative launch) and a thread's earlier candidates are settled, so the
// lowest open candidate is always being polled and can be decided.  What bounds it is the longest chain
// of candidates that wait for one another, at an L2 round trip each; a round behind a grid barrier cost
// about 15 us each (89k candidates, 361 rounds: 5429 -> 179 us; 5k candidates, in one block: 470 -> 50 us).
// A candidate's wait is bounded: after kDedupFreePolls polls it sleeps between polls, and gives up after
// about two seconds of requested sleep, or when another has: `err` gets 4 and the thread leaves.
constexpr int kDedupThreads = 128;
constexpr int kDedupFreePolls = 4096;
constexpr unsigned kDedupSleepNs = 256;
constexpr unsigned long long kDedupTimeoutNs = 2000000000ull;

__device__ void dedup_decide(const uint32_t *nbr_ptr, const uint32_t *nbr, uint32_t cap, uint32_t first, uint32_t nv,
                             uint32_t step, volatile uint8_t *dec, int *err) {
    constexpr int kBatch = 8;   // neighbours polled side by side; few candidates have more
    uint32_t i = first, b = 0, e = 0;
    uint32_t id[kBatch];
    auto load = [&]() {
        if (i >= nv) return;
        b = __ldg(nbr_ptr + i);
        e = min(__ldg(nbr_ptr + i + 1), cap);
#pragma unroll
        for (int k = 0; k < kBatch; ++k) id[k] = b + k < e ? __ldg(nbr + b + k) : 0u;
    };
    load();
    int polls = 0;
    unsigned long long waited_ns = 0;
    while (i < nv) {
        uint8_t t[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) t[k] = b + k < e ? dec[id[k]] : (uint8_t)2;
        bool kept = false, open = false;
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            kept = kept || t[k] == 1;
            open = open || t[k] == 0;
        }
        for (uint32_t k = b + kBatch; k < e && !kept; ++k) {
            const uint8_t u = dec[__ldg(nbr + k)];
            kept = u == 1;
            open = open || u == 0;
        }
        if (kept || !open) {
            dec[i] = kept ? 2 : 1;
            i += step;
            load();
            polls = 0;
            waited_ns = 0;
        } else if (++polls > kDedupFreePolls) {
            if (waited_ns > kDedupTimeoutNs || (*reinterpret_cast<volatile int *>(err) & 4) != 0) {
                atomicOr(err, 4);
                return;
            }
            __nanosleep(kDedupSleepNs);
            waited_ns += kDedupSleepNs;
        }
    }
}

__global__ void __launch_bounds__(kDedupThreads) k_dedup_decide(const uint32_t *nbr_ptr, const uint32_t *nbr, uint32_t cap,
                                                                uint32_t nv, uint8_t *decision, int *err) {
    dedup_decide(nbr_ptr, nbr, cap, blockIdx.x * kDedupThreads + threadIdx.x, nv, gridDim.x * kDedupThreads, decision,
                 err);
}

// Failure-detection self-test of the wait above: one thread takes candidate 1, whose earlier neighbour 0
// nobody decides, and must give up after about two seconds of requested sleep with bit 2 of err set.
__global__ void k_dedup_wait_selftest(const uint32_t *nbr_ptr, const uint32_t *nbr, uint8_t *decision, int *err) {
    dedup_decide(nbr_ptr, nbr, 1, 1, 2, 2, decision, err);
}

cudaError_t dedup_wait_selftest(int *flags, cudaStream_t st) {
    const uint32_t host[8] = {0, 0, 1, 0, 0, 0, 0, 0};   // nbr_ptr[0..2], nbr[0], decisions, err
    uint32_t *words = nullptr;
    cudaError_t e = cudaMallocAsync(reinterpret_cast<void **>(&words), sizeof(host), st);
    if (e != cudaSuccess) return e;
    e = cudaMemcpyAsync(words, host, sizeof(host), cudaMemcpyHostToDevice, st);
    int *err = reinterpret_cast<int *>(words + 5);
    int flag = 0;
    if (e == cudaSuccess) {
        k_dedup_wait_selftest<<<1, 1, 0, st>>>(words, words + 3, reinterpret_cast<uint8_t *>(words + 4), err);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&flag, err, sizeof(int), cudaMemcpyDeviceToHost, st);
    const cudaError_t f = cudaFreeAsync(words, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = f;
    *flags = flag;
    return e;
}

__global__ void k_dedup_flags(const uint8_t *decision, uint32_t nv, uint32_t *flags) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += gridDim.x * blockDim.x)
        flags[i] = decision[i] == 1 ? 1u : 0u;
}

// Kept candidates in candidate order, w = 1 (the host loop appends make_float4(x, y, z, 1)).
__global__ void k_dedup_emit(const float4 *cand, const uint8_t *decision, const uint32_t *pos, uint32_t nv, float4 *out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nv; i += gridDim.x * blockDim.x)
        if (decision[i] == 1) {
            const float4 c = cand[i];
            out[pos[i]] = make_float4(c.x, c.y, c.z, 1.0f);
        }
}

__global__ void k_fill_u32(uint32_t *a, uint32_t n, uint32_t v) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) a[i] = v;
}

// UpdateNodeDistanceKernel + BuildNodeGraphKernel (libs/star/geometry/node_graph/NodeGraph.cu:10-101):
// half-precision squared distances, k nearest including the node itself, __expf weights normalized.
//
// The reference fills an n x n table of half distances and scans a row of it in column order.
// With node_status, a pair with a deleted node (status .y == kDeletedNodeStatus, NodeGraph.h:18)
// gets the half of 1e6, which is infinite (NodeGraph.cu:20-35), so it never enters a heap; a
// deleted node's own row keeps the heap's initial entries.  `normalize` divides the weights
// by their sum (USE_INTERPOLATE_WEIGHT_NORMALIZATION, NodeGraph.cu:87-99); without it they are the
// raw __expf values, as the reference's geometry library compiles them.
constexpr uint32_t kDeletedNodeStatus = 0xffffffffu;
__device__ __forceinline__ bool node_deleted(const uint2 *status, int i) {
    return status != nullptr && status[i].y == kDeletedNodeStatus;
}

__device__ __forceinline__ float graph_half_distance(float4 a, float4 b) {
    const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;   // the squares do not see the sign
    return __half2float(__float2half_rn(__fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)))));
}

// Row `a` of the node graph from its K neighbours in order (BuildNodeGraphPairKernel, NodeGraph.cu:103-118).
template <int K>
__device__ __forceinline__ void graph_store(int a, const float *d, const uint16_t *id, float r2, int normalize, uint16_t *knn,
                                            float *w, uint16_t *edges) {
    float wv[K], sum = 0.f;
#pragma unroll
    for (int q = 0; q < K; ++q) wv[q] = __expf(-d[q] / (2 * r2));
#pragma unroll
    for (int q = 0; q < K; ++q) sum += wv[q];
    const float inv = 1.0f / sum;
#pragma unroll
    for (int q = 0; q < K; ++q) {
        knn[(size_t)a * K + q] = id[q];
        w[(size_t)a * K + q] = normalize ? wv[q] * inv : wv[q];
        edges[3 * ((size_t)a * K + q)] = (uint16_t)a;
        edges[3 * ((size_t)a * K + q) + 1] = id[q];
        edges[3 * ((size_t)a * K + q) + 2] = (uint16_t)q;
    }
}

// The scan in column order, one warp per node: 32 nodes at a time, the heap in K lanes, its updates in node
// order (a register maximum and two votes each).  Nodes
// list[0 .. *count) (graphs of many nodes: those that k_node_graph_cells leaves open), or all n.  With a list, boxes
// holds the bounds of every 32 nodes that are not deleted: the half of the squared distance to a box, rounded as
// theirs are, bounds theirs, and a box that is not below the heap's maximum is passed over (the whole graph, K = 4,
// without boxes / with: 30k nodes in voxel order 311 / 207 us, all tied in a plane 3154 / 2646, all in one place 1851 /
// 357; 8000 nodes 107 / 95, in random order 124 / 131).
constexpr int kGraphThreads = 128;
template <int K, bool kList>
__global__ void __launch_bounds__(kGraphThreads) k_node_graph_ordered(const float4 *nodes, const uint2 *status, int n,
                                                                      const uint32_t *list, const uint32_t *count,
                                                                      const float4 *boxes, float r2, int normalize,
                                                                      uint16_t *knn, float *w, uint16_t *edges) {
    const int lane = threadIdx.x & 31;
    const uint32_t rows = kList ? min(*count, (uint32_t)n) : (uint32_t)n;
    const uint32_t warps = gridDim.x * (kGraphThreads / 32);
    for (uint32_t row = blockIdx.x * (kGraphThreads / 32) + (threadIdx.x >> 5); row < rows; row += warps) {
        const int a = kList ? (int)list[row] : (int)row;
        const float4 va = nodes[a];
        // slot q of the heap in lane q; half distances are not negative, so their bits order like their values
        uint32_t slot_d = lane < K ? __float_as_uint(1e3f) : 0u, top = __float_as_uint(1e3f);
        int slot_id = 0;
        auto distance = [&](int b) {
            float v = INFINITY;   // deleted nodes, NaN and the end: enter no heap
            if (b < n && !node_deleted(status, b)) v = graph_half_distance(va, nodes[b]);
            return v < 1e3f ? __float_as_uint(v) : __float_as_uint(INFINITY);
        };
        auto enter = [&](uint32_t d, int b0) {   // nodes b0 + lane at d
            unsigned m = __ballot_sync(0xffffffffu, d < top);
            while (m) {   // in node order; an entry replaces the first slot that holds the maximum
                const int l = __ffs(m) - 1;
                const uint32_t v = __shfl_sync(0xffffffffu, d, l);
                const unsigned full = __ballot_sync(0xffffffffu, lane < K && slot_d == top);
                if (lane == __ffs(full) - 1) {
                    slot_d = v;
                    slot_id = b0 + l;
                }
                top = __reduce_max_sync(0xffffffffu, slot_d);
                m &= __ballot_sync(0xffffffffu, d < top) & (0xfffffffeu << l);
            }
        };
        if (node_deleted(status, a)) {
        } else if constexpr (kList) {
            const int blocks = (n + 31) / 32;
            float4 next_lo = __ldg(boxes + 2 * min(lane, blocks - 1)), next_hi = __ldg(boxes + 2 * min(lane, blocks - 1) + 1);
            for (int c0 = 0; c0 < blocks; c0 += 32) {
                const float4 lo = next_lo, hi = next_hi;
                const int ahead = min(c0 + 32 + lane, blocks - 1);
                next_lo = __ldg(boxes + 2 * ahead);
                next_hi = __ldg(boxes + 2 * ahead + 1);
                uint32_t bound = __float_as_uint(INFINITY);
                if (c0 + lane < blocks) {
                    const float x = fmaxf(fmaxf(lo.x - va.x, va.x - hi.x), 0.f), y = fmaxf(fmaxf(lo.y - va.y, va.y - hi.y), 0.f),
                                z = fmaxf(fmaxf(lo.z - va.z, va.z - hi.z), 0.f);
                    bound = __float_as_uint(__half2float(__float2half_rn(__fmaf_rn(z, z, __fmaf_rn(y, y, __fmul_rn(x, x))))));
                }
                unsigned m = __ballot_sync(0xffffffffu, bound < top);
                if (m == 0xffffffffu) {   // nodes in no spatial order: all of them, as without a list
                    for (int b0 = 32 * c0; b0 < 32 * c0 + 1024; b0 += 128) {
                        uint32_t d[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) d[q] = distance(b0 + 32 * q + lane);
#pragma unroll
                        for (int q = 0; q < 4; ++q) enter(d[q], b0 + 32 * q);
                    }
                    continue;
                }
                while (m) {   // in order; four boxes' nodes are loaded at a time
                    int c[4];
                    uint32_t d[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        c[q] = m ? c0 + __ffs(m) - 1 : blocks;
                        m &= m - 1;
                        d[q] = distance(32 * c[q] + lane);
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) enter(d[q], 32 * c[q]);
                    m &= __ballot_sync(0xffffffffu, bound < top);
                }
            }
        } else {
            for (int b0 = 0; b0 < n; b0 += 128) {
                uint32_t d[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) d[q] = distance(b0 + 32 * q + lane);
#pragma unroll
                for (int q = 0; q < 4; ++q) enter(d[q], b0 + 32 * q);
            }
        }
        Heap<K> h;
#pragma unroll
        for (int q = 0; q < K; ++q) {
            h.d[q] = __uint_as_float(__shfl_sync(0xffffffffu, slot_d, q));
            h.id[q] = (uint16_t)__shfl_sync(0xffffffffu, slot_id, q);
        }
        h.sort();
        if (lane == 0) graph_store<K>(a, h.d, h.id, r2, normalize, knn, w, edges);
    }
}

// SkinnerKernel (libs/star/geometry/node_graph/Skinner.cu:10-94) and IncSkinnerKernel (:211-302);
// nodes staged in shared memory.  A deleted node (status .y == kDeletedNodeStatus) enters the
// heap at distance 1e6 (Skinner.cu:39-48).  Full skinning (first_vert = 0, prev_nodes = 0) starts
// every heap at 1e6; the incremental form re-skins surfels first_vert .. n_verts - 1: the heap
// starts from the surfel's current neighbours at their distances and takes the nodes
// prev_nodes .. n_nodes - 1.  `normalize` divides the weights by their sum
// (USE_INTERPOLATE_WEIGHT_NORMALIZATION, Skinner.cu:70-74, 278-282).
__global__ void __launch_bounds__(256) k_skinning(const float4 *nodes, const uint2 *status, int n_nodes,
                                                   int prev_nodes, const float4 *verts, int first_vert, int n_verts,
                                                   float r2, int normalize, ushort4 *knn, float4 *sw, float4 *cw) {
    __shared__ float4 tile[1024];
    __shared__ unsigned char gone[1024];
    const int v = first_vert + (int)(blockIdx.x * blockDim.x + threadIdx.x);
    const bool live = v < n_verts;
    const float4 p = live ? verts[v] : make_float4(0.f, 0.f, 0.f, 0.f);
    Heap<4> h;
    if (prev_nodes > 0 && live) {
        const ushort4 k4 = knn[v];
        const uint16_t ids[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 q = nodes[min((int)ids[i], n_nodes - 1)];
            h.d[i] = sq3_fused(p.x - q.x, p.y - q.y, p.z - q.z);
            h.id[i] = ids[i];
        }
        h.refresh();
    } else {
        h.init(1e6f);
    }
    for (int base = prev_nodes; base < n_nodes; base += 1024) {
        const int cnt = min(1024, n_nodes - base);
        __syncthreads();
        for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
            tile[i] = nodes[base + i];
            gone[i] = node_deleted(status, base + i) ? 1 : 0;
        }
        __syncthreads();
        for (int i = 0; i < cnt; ++i) {
            const float4 q = tile[i];
            h.update((uint16_t)(base + i), gone[i] ? 1e6f : sq3_fused(p.x - q.x, p.y - q.y, p.z - q.z));
        }
    }
    if (!live) return;
    h.sort();
    float wv[4], sum = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 q = nodes[min((int)h.id[i], n_nodes - 1)];
        const float dd = sq3_fused(p.x - q.x, p.y - q.y, p.z - q.z);
        wv[i] = __expf(-dd / (2.f * r2));
        sum += wv[i];
    }
    const float inv = 1.f / sum;
    knn[v] = make_ushort4(h.id[0], h.id[1], h.id[2], h.id[3]);
    sw[v] = normalize ? make_float4(inv * wv[0], inv * wv[1], inv * wv[2], inv * wv[3])
                      : make_float4(wv[0], wv[1], wv[2], wv[3]);
    cw[v] = make_float4(1.f, 1.f, 1.f, 1.f);
}

// Full skinning over a grid of the nodes.  k_skinning tests every node for every surfel; here a surfel tests
// the nodes of the 3 x 3 x 3 cells around it, about 40.  1.2M surfels: 8.4k nodes 13422 -> 361 us, 31k
// nodes 46298 -> 2814 us, 525 nodes 1078 -> 236 us; 3000 surfels on 8.4k nodes 934 -> 45 us.  What bounds it now is shared memory: 16
// random bytes a lane and candidate, and warps that wait for their longest row of cells.
//
// Every block builds the same grid in its shared memory: kSkinCells cells (coordinates wrap, which only
// adds far candidates) and the nodes in cell order.  The cell size starts at 1.75 node radii and is
// halved or doubled until a node shares its cell with a few others, whatever the radius says.  More than
// kSkinGridNodes nodes go through in chunks, a surfel's five nearest kept from one to the next.
// Result: exactly k_skinning's.  When the four nearest found are strictly below the fifth and below
// every node outside the cells (by the distance to their faces, with a margin of a hundredth of a cell
// for the rounding of the scaled coordinates, |cell| <= 4096), and differ from one another, the ordered
// scan ends with the same four in the same order.  Otherwise (ties, far or few nodes, NaN) the surfel is
// open: its warp repeats the ordered scan for it, 32 nodes at a time with the heap updates in node order,
// or, where it has many of them, every lane for its own (skin_open).
constexpr int kSkinThreads = 1024;
constexpr int kSkinCellsX = 32, kSkinCellsY = 32, kSkinCellsZ = 16;
constexpr int kSkinCells = kSkinCellsX * kSkinCellsY * kSkinCellsZ;
constexpr int kSkinGridNodes = 10240;   // 16 bytes a node and 4 a cell fill a block's shared memory
static_assert(kSkinCells % kSkinThreads == 0, "whole cells per thread");

__device__ __forceinline__ float skin_scaled(float v, float inv_h) {
    return fminf(fmaxf(__fmul_rn(v, inv_h), -262144.f), 262144.f);
}
__device__ __forceinline__ int skin_cell(int x, int y, int z) {
    return (x & (kSkinCellsX - 1)) | ((y & (kSkinCellsY - 1)) * kSkinCellsX) |
           ((z & (kSkinCellsZ - 1)) * (kSkinCellsX * kSkinCellsY));
}
__device__ __forceinline__ int skin_cell_of(float4 q, float inv_h) {
    return skin_cell(__float2int_rd(skin_scaled(q.x, inv_h)), __float2int_rd(skin_scaled(q.y, inv_h)),
                     __float2int_rd(skin_scaled(q.z, inv_h)));
}

// Grid of nodes n0 .. n1 - 1 in the block's shared memory; returns the cell size.
__device__ float skin_grid_build(const float4 *nodes, const uint2 *status, int n0, int n1, float h, float4 *cell_nodes,
                                 uint32_t *cell_end) {
    __shared__ unsigned long long sm64[kSkinThreads / 32];
    __shared__ uint32_t sm32[32];
    const int tid = threadIdx.x, n = n1 - n0;
    constexpr int kPer = kSkinCells / kSkinThreads;
    int dir = 0;
    for (int trial = 0;; ++trial) {   // uniform: every thread sees the same sums
        const float inv_h = 1.0f / h;
        __syncthreads();
        for (int c = tid; c < kSkinCells; c += kSkinThreads) cell_end[c] = 0;
        __syncthreads();
        for (int i = n0 + tid; i < n1; i += kSkinThreads)
            // a deleted node enters no heap: its distance is the heap's initial 1e6
            if (!node_deleted(status, i)) atomicAdd(&cell_end[skin_cell_of(nodes[i], inv_h)], 1u);
        __syncthreads();
        unsigned long long sq = 0;
        for (int c = tid; c < kSkinCells; c += kSkinThreads) sq += (unsigned long long)cell_end[c] * cell_end[c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if ((tid & 31) == 0) sm64[tid >> 5] = sq;
        __syncthreads();
        sq = 0;
        for (int i = 0; i < kSkinThreads / 32; ++i) sq += sm64[i];
        // nodes that share a node's cell, itself among them: 1.5 to 16 on average
        const int want = sq > 16ull * n ? -1 : (2ull * sq < 3ull * n ? 1 : 0);
        const float next = want < 0 ? 0.5f * h : 2.0f * h;
        if (want == 0 || trial == 12 || (dir != 0 && want != dir) || !(next > 1e-12f && next < 1e12f)) break;
        dir = want;
        h = next;
    }
    {   // counts -> first positions (thread t owns cells kPer t ..); placing the nodes moves them to the ends
        uint32_t v[kPer], sum = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k) { v[k] = cell_end[kPer * tid + k]; sum += v[k]; }
        uint32_t at = block_excl_scan_u32(sum, nullptr, sm32);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kPer; ++k) { cell_end[kPer * tid + k] = at; at += v[k]; }
    }
    __syncthreads();
    const float inv_h = 1.0f / h;
    for (int i = n0 + tid; i < n1; i += kSkinThreads) {
        if (node_deleted(status, i)) continue;
        const float4 q = nodes[i];
        cell_nodes[atomicAdd(&cell_end[skin_cell_of(q, inv_h)], 1u)] = make_float4(q.x, q.y, q.z, __int_as_float(i));
    }
    __syncthreads();
    return h;
}

// Node graph over a grid of the nodes, for many nodes.  The scan in column order (k_node_graph_ordered) is
// O(n^2) and, in voxel order, updates its heap all the way to the node (1673 us for 27k nodes, K = 8).  One
// block puts the nodes into the cells of the skinning grid (k_graph_grid, 29 us); four lanes a node then keep
// the K + 1 smallest half distances of the 3 x 3 x 3 cells around it (37 us at 23k).  Where they rise strictly and lie below the half distance of every node outside
// (the rounding to half is monotone, so that of the squared distance to the cells' faces bounds theirs), the
// ordered scan ends with the same K in the same order; the others (ties in half precision, 2-5% of the
// nodes, deleted and far ones) go to a list for the ordered scan, which passes over 32 nodes at a time by the boxes
// that the cells' kernel leaves.
__global__ void __launch_bounds__(kSkinThreads, 1) k_graph_grid(const float4 *nodes, const uint2 *status, int n, float h0,
                                                                float4 *cell_nodes, uint32_t *cell_end, float *h_out,
                                                                uint32_t *count) {
    extern __shared__ __align__(16) unsigned char skin_smem[];
    uint32_t *ends = reinterpret_cast<uint32_t *>(skin_smem);
    const float h = skin_grid_build(nodes, status, 0, n, h0, cell_nodes, ends);
    for (int c = threadIdx.x; c < kSkinCells; c += kSkinThreads) cell_end[c] = ends[c];
    if (threadIdx.x == 0) {
        *h_out = h;
        *count = 0;
    }
}

template <int K>
__global__ void __launch_bounds__(kGraphThreads) k_node_graph_cells(const float4 *nodes, const uint2 *status, int n,
                                                                    const float4 *cell_nodes, const uint32_t *cell_end,
                                                                    const float *h_in, float r2, int normalize,
                                                                    uint16_t *knn, float *w, uint16_t *edges,
                                                                    uint32_t *list, uint32_t *count, float4 *boxes) {
    static_assert(kGraphThreads == 4 * 32, "a block has 32 nodes");
    if (threadIdx.x < 32) {   // their box, for the ordered scan
        const int b = 32 * (int)blockIdx.x + (int)threadIdx.x;
        const bool in = b < n && !node_deleted(status, b);
        const float4 q = nodes[min(b, n - 1)];
        float lo[3] = {in ? q.x : INFINITY, in ? q.y : INFINITY, in ? q.z : INFINITY};
        float hi[3] = {in ? q.x : -INFINITY, in ? q.y : -INFINITY, in ? q.z : -INFINITY};
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
                hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
            }
        if (threadIdx.x == 0) {
            boxes[2 * blockIdx.x] = make_float4(lo[0], lo[1], lo[2], 0.f);
            boxes[2 * blockIdx.x + 1] = make_float4(hi[0], hi[1], hi[2], 0.f);
        }
    }
    // four lanes a node: lane q of them takes the rows q, q + 4, q + 8
    const int a = min((int)(blockIdx.x * kGraphThreads + threadIdx.x) >> 2, n - 1), part_lane = threadIdx.x & 3;
    const bool mine = (int)(blockIdx.x * kGraphThreads + threadIdx.x) >> 2 < n;
    const float4 p = nodes[a];
    const float h = *h_in, inv_h = 1.0f / h;
    float ld[K + 1];
    uint16_t lid[K + 1];
#pragma unroll
    for (int q = 0; q <= K; ++q) { ld[q] = 1e3f; lid[q] = 0; }
    const float sx = skin_scaled(p.x, inv_h), sy = skin_scaled(p.y, inv_h), sz = skin_scaled(p.z, inv_h);
    const int cx = __float2int_rd(sx), cy = __float2int_rd(sy), cz = __float2int_rd(sz);
    const int x0 = (cx - 1) & (kSkinCellsX - 1), x1 = (cx + 1) & (kSkinCellsX - 1);
    for (int row = part_lane; row < 9; row += 4) {
        const int c0 = skin_cell(0, cy + row % 3 - 1, cz + row / 3 - 1);
        for (int part = 0; part < (x0 <= x1 ? 1 : 2); ++part) {
            const int lo = c0 + (x0 <= x1 || part == 0 ? x0 : 0);
            const int hi = c0 + (x0 <= x1 || part == 1 ? x1 : kSkinCellsX - 1);
            const uint32_t e = __ldg(cell_end + hi);
            for (uint32_t k = lo > 0 ? __ldg(cell_end + lo - 1) : 0u; k < e; ++k) {
                const float4 v = __ldg(cell_nodes + k);
                const float dist = graph_half_distance(p, v);
                if (dist < ld[K]) {
                    const uint16_t b = (uint16_t)__float_as_int(v.w);
#pragma unroll
                    for (int q = K; q >= 0; --q) {   // shift the larger ones up
                        const bool here = dist < ld[q], below = q > 0 && dist < ld[q > 0 ? q - 1 : 0];
                        ld[q] = below ? ld[q > 0 ? q - 1 : 0] : (here ? dist : ld[q]);
                        lid[q] = below ? lid[q > 0 ? q - 1 : 0] : (here ? b : lid[q]);
                    }
                }
            }
        }
    }
    // the four ascending lists into one: K + 1 times the smallest head (of equal ones the lowest lane's; ties
    // go to the ordered scan anyway)
    float d[K + 1];
    uint16_t id[K + 1];
#pragma unroll
    for (int q = 0; q <= K; ++q) {
        float m = ld[0];
        m = fminf(m, __shfl_xor_sync(0xffffffffu, m, 1));
        m = fminf(m, __shfl_xor_sync(0xffffffffu, m, 2));
        const unsigned has = (__ballot_sync(0xffffffffu, ld[0] == m) >> (threadIdx.x & 28)) & 15u;
        const int from = __ffs(has) - 1;
        d[q] = m;
        id[q] = (uint16_t)__shfl_sync(0xffffffffu, (int)lid[0], from, 4);
        if (part_lane == from) {
#pragma unroll
            for (int k = 0; k < K; ++k) { ld[k] = ld[k + 1]; lid[k] = lid[k + 1]; }
            ld[K] = 1e3f;
        }
    }
    if (!mine || part_lane != 0) return;
    const float fx = sx - floorf(sx), fy = sy - floorf(sy), fz = sz - floorf(sz);
    const float inside = fminf(fminf(fminf(fx, 1.f - fx), fminf(fy, 1.f - fy)), fminf(fz, 1.f - fz));
    const float reach = (0.99f + inside) * h;
    bool sure = fmaxf(fmaxf(fabsf(sx), fabsf(sy)), fabsf(sz)) <= 4096.f && !node_deleted(status, a) &&
                d[K - 1] < __half2float(__float2half_rn(reach * reach));
#pragma unroll
    for (int q = 0; q < K; ++q) sure = sure && d[q] < d[q + 1];
    if (sure) graph_store<K>(a, d, id, r2, normalize, knn, w, edges);
    else list[atomicAdd(count, 1u)] = (uint32_t)a;
}

// One surfel's search: its five nearest so far, ascending, with the ids of four, and the distance up to
// which every node has been seen.
struct SkinNearest {
    float d[5] = {1e6f, 1e6f, 1e6f, 1e6f, 1e6f};
    int id[4] = {0, 0, 0, 0};
    float reach = 1e30f;
    __device__ __forceinline__ void insert(float dist, int node) {   // dist < d[4]
        const bool b0 = dist < d[0], b1 = dist < d[1], b2 = dist < d[2], b3 = dist < d[3];
        d[4] = b3 ? d[3] : dist;
        d[3] = b2 ? d[2] : (b3 ? dist : d[3]);
        id[3] = b2 ? id[2] : (b3 ? node : id[3]);
        d[2] = b1 ? d[1] : (b2 ? dist : d[2]);
        id[2] = b1 ? id[1] : (b2 ? node : id[2]);
        d[1] = b0 ? d[0] : (b1 ? dist : d[1]);
        id[1] = b0 ? id[0] : (b1 ? node : id[1]);
        d[0] = b0 ? dist : d[0];
        id[0] = b0 ? node : id[0];
    }
    // the nearest four are distinct, nearer than the fifth and than every node outside the cells: any order of the
    // nodes gives them
    __device__ __forceinline__ bool sure() const {
        return d[0] < d[1] && d[1] < d[2] && d[2] < d[3] && d[3] < d[4] && reach > 0.f && d[3] < reach * reach;
    }
};

__device__ __forceinline__ void skin_grid_search(float4 p, float h, const float4 *cell_nodes, const uint32_t *cell_end,
                                                 SkinNearest &b) {
    const float inv_h = 1.0f / h;
    const float sx = skin_scaled(p.x, inv_h), sy = skin_scaled(p.y, inv_h), sz = skin_scaled(p.z, inv_h);
    const int cx = __float2int_rd(sx), cy = __float2int_rd(sy), cz = __float2int_rd(sz);
    const int x0 = (cx - 1) & (kSkinCellsX - 1), x1 = (cx + 1) & (kSkinCellsX - 1);
    for (int row = 0; row < 9; ++row) {
        // the row's three cells: one range, or two where x wraps
        const int c0 = skin_cell(0, cy + row % 3 - 1, cz + row / 3 - 1);
        for (int part = 0; part < (x0 <= x1 ? 1 : 2); ++part) {
            const int lo = c0 + (x0 <= x1 || part == 0 ? x0 : 0);
            const int hi = c0 + (x0 <= x1 || part == 1 ? x1 : kSkinCellsX - 1);
            const uint32_t e = cell_end[hi];
            for (uint32_t k = lo > 0 ? cell_end[lo - 1] : 0u; k < e; ++k) {
                const float4 q = cell_nodes[k];
                const float dist = sq3_fused(p.x - q.x, p.y - q.y, p.z - q.z);
                if (dist < b.d[4]) b.insert(dist, __float_as_int(q.w));
            }
        }
    }
    // distance to the nearest face of the 3 x 3 x 3 cells, less the margin
    const float fx = sx - floorf(sx), fy = sy - floorf(sy), fz = sz - floorf(sz);
    const float inside = fminf(fminf(fminf(fx, 1.f - fx), fminf(fy, 1.f - fy)), fminf(fz, 1.f - fz));
    const bool near = fmaxf(fmaxf(fabsf(sx), fabsf(sy)), fabsf(sz)) <= 4096.f;
    b.reach = near ? fminf(b.reach, (0.99f + inside) * h) : -1.f;
}

constexpr float kSkinOpen = -1.f;   // a connect weight, until the surfel's turn comes
constexpr int kSkinMany = 6;   // open surfels of a warp from which on every lane looks at all nodes for its own (skin_open)

struct SkinOut {
    float r2;
    int normalize;
    ushort4 *knn;
    float4 *sw, *cw;
};
__device__ __forceinline__ void skin_store(const SkinOut &o, int v, const float (&d)[4], const int (&id)[4]) {
    float wv[4], sum = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        wv[i] = __expf(-d[i] / (2.f * o.r2));
        sum += wv[i];
    }
    const float inv = 1.f / sum;
    o.knn[v] = make_ushort4((uint16_t)id[0], (uint16_t)id[1], (uint16_t)id[2], (uint16_t)id[3]);
    o.sw[v] = o.normalize ? make_float4(inv * wv[0], inv * wv[1], inv * wv[2], inv * wv[3])
                          : make_float4(wv[0], wv[1], wv[2], wv[3]);
    o.cw[v] = make_float4(1.f, 1.f, 1.f, 1.f);
}

// The ordered scan for the surfel at p of lane `who`, by the whole warp, 32 nodes at a time.
__device__ __forceinline__ void skin_scan_one(const float4 *nodes, const uint2 *status, int n_nodes, float4 p, int who,
                                              Heap<4> &heap) {
    const int lane = threadIdx.x & 31;
    const float px = __shfl_sync(0xffffffffu, p.x, who), py = __shfl_sync(0xffffffffu, p.y, who),
                pz = __shfl_sync(0xffffffffu, p.z, who);
    heap.init(1e6f);
    for (int i0 = 0; i0 < n_nodes; i0 += 32) {
        const int i = i0 + lane;
        float dist = 1e6f;
        if (i < n_nodes && !node_deleted(status, i)) {
            const float4 q = nodes[i];
            dist = sq3_fused(px - q.x, py - q.y, pz - q.z);
        }
        for (unsigned m = __ballot_sync(0xffffffffu, dist < heap.max_d); m; m &= m - 1) {
            const int l = __ffs(m) - 1;
            heap.update((uint16_t)(i0 + l), __shfl_sync(0xffffffffu, dist, l));
        }
    }
    heap.sort();
}

// Many open surfels of a warp: the ordered scan by every lane for its own, 32 nodes at a time from global memory, the
// next 32 on their way.  us, one surfel after another / this / k_skinning, which the grid is not to lose to: surfels far
// from all nodes, 200k on 8000 nodes 5569 / 1376 / 1787, 300 on 8000 2328 / 511 / 622; all tied, 195k on 8000 10445 /
// 1303 / 2072, on 1000 3625 / 350 / 325.
__device__ __forceinline__ void skin_open(const float4 *nodes, const uint2 *status, int n_nodes, float4 p, int v, unsigned open,
                                          const SkinOut &o) {
    const int lane = threadIdx.x & 31;
    const bool mine = (open >> lane) & 1u;
    Heap<4> heap;
    heap.init(1e6f);
    float4 q = nodes[min(lane, n_nodes - 1)];
    bool here = lane < n_nodes && !node_deleted(status, lane);
    for (int i0 = 0; i0 < n_nodes; i0 += 32) {
        const float4 now = q;
        const unsigned alive = __ballot_sync(0xffffffffu, here);
        const int next = i0 + 32 + lane;
        q = nodes[min(next, n_nodes - 1)];
        here = next < n_nodes && !node_deleted(status, next);
        // the distance to the 32 nodes' box, rounded as theirs are, bounds them: what lies beyond enters no heap
        const bool in = (alive >> lane) & 1u;
        float lo[3] = {in ? now.x : INFINITY, in ? now.y : INFINITY, in ? now.z : INFINITY};
        float hi[3] = {in ? now.x : -INFINITY, in ? now.y : -INFINITY, in ? now.z : -INFINITY};
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], o));
                hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], o));
            }
        const float box = sq3_fused(fmaxf(fmaxf(lo[0] - p.x, p.x - hi[0]), 0.f), fmaxf(fmaxf(lo[1] - p.y, p.y - hi[1]), 0.f),
                                    fmaxf(fmaxf(lo[2] - p.z, p.z - hi[2]), 0.f));
        if (!__any_sync(0xffffffffu, mine && box < heap.max_d)) continue;
#pragma unroll 4
        for (int l = 0; l < 32; ++l) {
            const float x = __shfl_sync(0xffffffffu, now.x, l), y = __shfl_sync(0xffffffffu, now.y, l),
                        z = __shfl_sync(0xffffffffu, now.z, l);
            const float dist = (alive >> l) & 1u ? sq3_fused(p.x - x, p.y - y, p.z - z) : 1e6f;
            if (__any_sync(0xffffffffu, mine && dist < heap.max_d)) heap.update((uint16_t)(i0 + l), dist);
        }
    }
    heap.sort();
    if (mine) {
        float d[4];
        int ids[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            ids[i] = heap.id[i];
            const float4 q = nodes[min(ids[i], n_nodes - 1)];
            d[i] = sq3_fused(p.x - q.x, p.y - q.y, p.z - q.z);
        }
        skin_store(o, v, d, ids);
    }
}

// A warp's rounds of 32 surfels: whole rounds of the launch by blocks (neighbouring memory), the last one, or few
// surfels, over all blocks (200k surfels 66 -> 59 us, 3000 on 8000 nodes 110 -> 82).
struct SkinRounds {
    int base, full, stride, shift;
    uint32_t bit = 1;   // of the round, modulo 32
    __device__ __forceinline__ SkinRounds(int first_vert, int n_verts) {
        const int by_block = (int)(blockIdx.x * (kSkinThreads / 32) + (threadIdx.x >> 5)),
                  spread = (int)((threadIdx.x >> 5) * gridDim.x + blockIdx.x);
        stride = 32 * (int)(gridDim.x * (kSkinThreads / 32));
        full = (n_verts - first_vert) / stride;
        shift = 32 * (spread - by_block);
        base = first_vert + 32 * by_block + (full == 0 ? shift : 0);
    }
    __device__ __forceinline__ void next() {
        base += stride;
        if (--full == 0) base += shift;
        bit = __funnelshift_l(bit, bit, 1);
    }
};

// The rounds (modulo 32) of a warp that left many surfels open.  Last: in the loop its code costs the usual case 2 %.
__device__ __forceinline__ void skin_later(const float4 *nodes, const uint2 *status, int n_nodes, const float4 *verts, int first_vert,
                                           int n_verts, uint32_t rounds, const SkinOut &out) {
    const int lane = threadIdx.x & 31;
    for (SkinRounds r(first_vert, n_verts); r.base < n_verts; r.next()) {
        if ((rounds & r.bit) == 0) continue;
        const int v = r.base + lane;
        const unsigned open = __ballot_sync(0xffffffffu, v < n_verts && out.cw[v].x == kSkinOpen);
        if (open) skin_open(nodes, status, n_nodes, verts[min(v, n_verts - 1)], v, open, out);
    }
}

// The surfels of a warp (lane's surfel v at p): the ordered scan where the search does not settle the
// result, then ids and weights.
// Many open surfels are left out and returned; until skin_open's turn their connect weight says so.
__device__ __forceinline__ unsigned skin_grid_finish(const float4 *nodes, const uint2 *status, int n_nodes, float4 p, int v,
                                                     bool live, SkinNearest &b, const SkinOut &o) {
    const int lane = threadIdx.x & 31;
    unsigned open = __ballot_sync(0xffffffffu, live && !b.sure());
    const unsigned many = __popc(open) >= kSkinMany ? open : 0u;
    open &= ~many;
    while (open) {
        const int who = __ffs(open) - 1;
        open &= open - 1;
        Heap<4> heap;
        skin_scan_one(nodes, status, n_nodes, p, who, heap);
        if (lane == who) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                b.id[i] = heap.id[i];
                const float4 q = nodes[min(b.id[i], n_nodes - 1)];
                b.d[i] = sq3_fused(p.x - q.x, p.y - q.y, p.z - q.z);
            }
        }
    }
    if (live && ((many >> lane) & 1u) == 0) {
        const float d[4] = {b.d[0], b.d[1], b.d[2], b.d[3]};
        skin_store(o, v, d, b.id);
    } else if (live) {
        o.cw[v].x = kSkinOpen;
    }
    return many;
}

// kChunked: more than kSkinGridNodes nodes; a launch then covers at most 32 surfels a warp.
template <bool kChunked>
__global__ void __launch_bounds__(kSkinThreads, 1) k_skinning_grid(const float4 *nodes, const uint2 *status, int n_nodes,
                                                                   const float4 *verts, int first_vert, int n_verts,
                                                                   float radius, const SkinOut out) {
    extern __shared__ __align__(16) unsigned char skin_smem[];
    float4 *cell_nodes = reinterpret_cast<float4 *>(skin_smem);                                    // one chunk's
    uint32_t *cell_end = reinterpret_cast<uint32_t *>(skin_smem + 16 * (size_t)min(n_nodes, kSkinGridNodes));
    const int lane = threadIdx.x & 31;
    SkinRounds r(first_vert, n_verts);
    if constexpr (kChunked) {
        const int v = r.base + lane;
        const bool live = v < n_verts;
        const float4 p = live ? verts[v] : make_float4(0.f, 0.f, 0.f, 0.f);
        SkinNearest b;
        for (int n0 = 0; n0 < n_nodes; n0 += kSkinGridNodes) {
            const float h = skin_grid_build(nodes, status, n0, min(n_nodes, n0 + kSkinGridNodes), 1.75f * radius,
                                            cell_nodes, cell_end);
            if (live) skin_grid_search(p, h, cell_nodes, cell_end, b);
        }
        const unsigned many = skin_grid_finish(nodes, status, n_nodes, p, v, live, b, out);
        if (many) skin_open(nodes, status, n_nodes, p, v, many, out);
    } else {
        const float h = skin_grid_build(nodes, status, 0, n_nodes, 1.75f * radius, cell_nodes, cell_end);
        __shared__ uint32_t s_later[kSkinThreads / 32];
        uint32_t &later = s_later[threadIdx.x >> 5];
        if (lane == 0) later = 0;
        for (; r.base < n_verts; r.next()) {
            const int v = r.base + lane;
            const bool live = v < n_verts;
            const float4 p = live ? verts[v] : make_float4(0.f, 0.f, 0.f, 0.f);
            SkinNearest b;
            if (live) skin_grid_search(p, h, cell_nodes, cell_end, b);
            if (skin_grid_finish(nodes, status, n_nodes, p, v, live, b, out) && lane == 0) later |= r.bit;
        }
        __syncwarp();
        if (later != 0)
            skin_later(nodes, status, n_nodes, verts, first_vert, n_verts, later, out);
    }
}

// ForwardWarpVertexAndNodeKernel (libs/star/geometry/surfel/SurfelNodeDeformer.cu:13-79) with
// averageDualQuaternion<4> (libs/star/math/DualQuaternion.hpp:288-306).
__global__ void k_forward_warp(const float *se3, int num_nodes, const float4 *verts, const float4 *normals, int n,
                               const ushort4 *knn, const float4 *sw, const float4 *cw, float4 *out_v, float4 *out_n) {
    const uint16_t last = (uint16_t)(num_nodes - 1);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const ushort4 k4 = knn[i];
        const float4 s4 = sw[i], c4 = cw[i];
        const uint16_t ids[4] = {(uint16_t)min(k4.x, last), (uint16_t)min(k4.y, last), (uint16_t)min(k4.z, last),
                                 (uint16_t)min(k4.w, last)};
        const float wv[4] = {s4.x * c4.x, s4.y * c4.y, s4.z * c4.z, s4.w * c4.w};
        DQf avg;
        avg.q0 = make_float4(0.f, 0.f, 0.f, 0.f);
        avg.q1 = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            DQf d = load_dq(se3 + 8ull * ids[k]);
            dq_normalize(d);
            avg.q0 = make_float4(avg.q0.x + wv[k] * d.q0.x, avg.q0.y + wv[k] * d.q0.y, avg.q0.z + wv[k] * d.q0.z,
                                 avg.q0.w + wv[k] * d.q0.w);
            avg.q1 = make_float4(avg.q1.x + wv[k] * d.q1.x, avg.q1.y + wv[k] * d.q1.y, avg.q1.z + wv[k] * d.q1.z,
                                 avg.q1.w + wv[k] * d.q1.w);
        }
        const SE3f T = dq_se3(avg);
        const float4 v = verts[i];
        const float3 o = mul(T.rot, f3(v.x, v.y, v.z)) + T.t;
        out_v[i] = make_float4(o.x, o.y, o.z, v.w);
        if (normals && out_n) {
            const float4 nn = normals[i];
            const float3 on = mul(T.rot, f3(nn.x, nn.y, nn.z));
            out_n[i] = make_float4(on.x, on.y, on.z, nn.w);
        }
    }
}

// Solver-map splat: projection as shaders/solver_map.vert:21-27 (pixel = floor(f x / z + c + 0.5)),
// nearest depth wins, ties to the lower surfel id.
__global__ void k_splat(const float4 *verts, int n, int W, int H, float fx, float fy, float cx, float cy, int fp,
                        unsigned long long *zbuf) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 v = verts[i];
        if (!(v.z > 0.f)) continue;
        const int px = (int)floorf(fx * v.x / v.z + cx + 0.5f);
        const int py = (int)floorf(fy * v.y / v.z + cy + 0.5f);
        const unsigned long long key = ((unsigned long long)__float_as_uint(v.z) << 32) | (unsigned)i;
        for (int dy = -fp; dy <= fp; ++dy)
            for (int dx = -fp; dx <= fp; ++dx) {
                const int x = px + dx, y = py + dy;
                if (x < 0 || y < 0 || x >= W || y >= H) continue;
                atomicMin(zbuf + (size_t)y * W + x, key);
            }
    }
}

__global__ void k_splat_resolve(const unsigned long long *zbuf, int npix, const float4 *av, const float4 *an,
                                uint32_t *index, float4 *vmap, float4 *nmap) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += gridDim.x * blockDim.x) {
        const unsigned long long k = zbuf[p];
        if (k == ~0ull) {
            index[p] = kInvalidIndex;
            if (vmap) vmap[p] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (nmap) nmap[p] = make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
            const uint32_t id = (uint32_t)(k & 0xffffffffu);
            index[p] = id;
            if (vmap) { const float4 v = av[id]; vmap[p] = make_float4(v.x, v.y, v.z, 1.f); }
            if (nmap) { const float4 nn = an[id]; nmap[p] = make_float4(nn.x, nn.y, nn.z, 0.f); }
        }
    }
}

// ---- Solver maps as the reference's solver-map pass draws them --------------------------------
// Renderer::DrawSolverMaps (libs/star/geometry/render/RendererDraw.cu:105-160) draws every surfel as
// a point with shaders/solver_map.vert:21-53 and solver_map.frag:10-17.  Restated per surfel:
//   * v_cam = world2camera (v, 1), summed ((m0 x + m1 y) + m2 z) + m3 per row;
//   * culled when v_cam.z > max depth, v_cam.z <= 0, or the surfel is unstable and not recent:
//     confidence (vertex_confid.w) < threshold.x and |time (color_time.z) - current time| >= threshold.y
//     (threshold.y = -1 culls every unstable surfel, DrawSolverMaps without recent observation);
//   * pixel floor(fx x / z + cx + 0.5), floor(fy y / z + cy + 0.5) (the shader's 0.5 shift: the point
//     lands in the pixel that holds its window position), and `footprint` pixels around it;
//   * the depth test keeps the nearest z (the depth buffer clears to the far plane, so z = max depth
//     never passes it); equal depths keep the lower surfel id (the first one drawn);
//   * outputs: reference vertex (xyz, 1), reference normal (xyz, 0), surfel id, and the normalized
//     rgbd (colour bytes of color_time.x / 127.5 - 1, 1 / z); untouched pixels keep the clear values
//     (zeros, id 0xFFFFFFFF), GLClearValues.h:21-34.
// The depth compare runs on the float camera z, where the GL depth buffer holds a quantised window
// depth; two surfels closer than that quantum can resolve differently there.
struct RenderArgs {
    int W, H, fp;
    float fx, fy, cx, cy, max_depth, current_time, conf_threshold, time_threshold;
    float m[12];   // world2camera rows 0..2, row-major
};

__device__ __forceinline__ float row_dot(const float *m, float4 v) {
    return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(m[0], v.x), __fmul_rn(m[1], v.y)), __fmul_rn(m[2], v.z)), m[3]);
}

__global__ void k_render_keys(const float4 *vc, const float4 *ct, int n, RenderArgs a, unsigned long long *zbuf) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 v = vc[i];
        const float z = row_dot(a.m + 8, v);
        if (!(z > 0.f) || !(z < a.max_depth)) continue;
        const float t = ct ? ct[i].z : a.current_time;
        if (v.w < a.conf_threshold && fabsf(__fsub_rn(t, a.current_time)) >= a.time_threshold) continue;
        const float x = row_dot(a.m, v), y = row_dot(a.m + 4, v);
        const float fpx = floorf(__fadd_rn(__fadd_rn(__fdiv_rn(__fmul_rn(a.fx, x), z), a.cx), 0.5f));
        const float fpy = floorf(__fadd_rn(__fadd_rn(__fdiv_rn(__fmul_rn(a.fy, y), z), a.cy), 0.5f));
        // a point more than the footprint outside the image covers no pixel (this also keeps the
        // conversion to int in range)
        if (!(fpx >= (float)(-a.fp) && fpx < (float)(a.W + a.fp) && fpy >= (float)(-a.fp) && fpy < (float)(a.H + a.fp)))
            continue;
        const int px = (int)fpx, py = (int)fpy;
        const unsigned long long key = ((unsigned long long)__float_as_uint(z) << 32) | (unsigned)i;
        for (int dy = -a.fp; dy <= a.fp; ++dy)
            for (int dx = -a.fp; dx <= a.fp; ++dx) {
                const int qx = px + dx, qy = py + dy;
                if (qx < 0 || qy < 0 || qx >= a.W || qy >= a.H) continue;
                atomicMin(zbuf + (size_t)qy * a.W + qx, key);
            }
    }
}

__global__ void k_render_resolve(const unsigned long long *zbuf, int npix, const float4 *vc, const float4 *nr,
                                 const float4 *ct, uint32_t *index, float4 *vmap, float4 *nmap, float4 *rgbd) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += gridDim.x * blockDim.x) {
        const unsigned long long k = zbuf[p];
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k == ~0ull) {
            index[p] = kInvalidIndex;
            if (vmap) vmap[p] = zero;
            if (nmap) nmap[p] = zero;
            if (rgbd) rgbd[p] = zero;
            continue;
        }
        const uint32_t id = (uint32_t)(k & 0xffffffffu);
        index[p] = id;
        if (vmap) { const float4 v = vc[id]; vmap[p] = make_float4(v.x, v.y, v.z, 1.f); }
        if (nmap) { const float4 nn = nr[id]; nmap[p] = make_float4(nn.x, nn.y, nn.z, 0.f); }
        if (rgbd) {
            const int enc = ct ? __float_as_int(ct[id].x) : 0;
            const float z = __uint_as_float((uint32_t)(k >> 32));
            rgbd[p] = make_float4(__fsub_rn(__fdiv_rn((float)((enc & 0x00FF0000) >> 16), 127.5f), 1.f),
                                  __fsub_rn(__fdiv_rn((float)((enc & 0x0000FF00) >> 8), 127.5f), 1.f),
                                  __fsub_rn(__fdiv_rn((float)(enc & 0x000000FF), 127.5f), 1.f), __fdiv_rn(1.f, z));
        }
    }
}

// ---- Observation maps as the reference's observation-map pass draws them ----------------------
// Renderer::DrawObservationMaps (libs/star/geometry/render/RendererDraw.cu:353-394) with
// shaders/geometry.vert:40-86 and observation_map.frag:13-17: the same transform, culls and depth
// rule as the solver-map pass, but each surfel is a GL point as wide as its disk's image
// (obs_point in ws_obs_point.cuh, shared with the host check of the tests).  One thread per
// surfel offers its (z bits, id) key to every pixel of its clipped rectangle; the smallest key
// wins, so the nearest z wins and equal depths keep the lower id (GL_LESS in draw order).
__global__ void k_obs_keys(const float4 *vc, const float4 *nr, const float4 *ct, int n, RenderArgs a,
                           unsigned long long *zbuf) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 v4 = vc[i], n4 = nr[i];
        const float v[4] = {v4.x, v4.y, v4.z, v4.w}, nw[4] = {n4.x, n4.y, n4.z, n4.w};
        const float t = ct ? ct[i].z : a.current_time;
        const ObsCover c = obs_point(v, nw, t, a.m, a.fx, a.fy, a.cx, a.cy, a.W, a.H, a.max_depth, a.current_time,
                                     a.conf_threshold, a.time_threshold);
        if (!c.drawn) continue;
        // z > 0 here, so its bits order like its value
        const unsigned long long key = ((unsigned long long)__float_as_uint(c.z) << 32) | (unsigned)i;
        for (int qy = c.y0; qy <= c.y1; ++qy)   // inside the image: obs_point clips the rectangle
            for (int qx = c.x0; qx <= c.x1; ++qx) atomicMin(zbuf + (size_t)qy * a.W + qx, key);
    }
}

__global__ void k_obs_resolve(const unsigned long long *zbuf, int npix, const float4 *ct, uint32_t *index,
                              float4 *rgbd) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += gridDim.x * blockDim.x) {
        const unsigned long long k = zbuf[p];
        if (k == ~0ull) {   // the clear values (GLClearValues.h:26-33)
            index[p] = kInvalidIndex;
            if (rgbd) rgbd[p] = make_float4(0.f, 0.f, 0.f, 0.f);
            continue;
        }
        const uint32_t id = (uint32_t)(k & 0xffffffffu);
        index[p] = id;
        if (rgbd) {
            float o[4];
            obs_rgbd(ct ? __float_as_int(ct[id].x) : 0, __uint_as_float((uint32_t)(k >> 32)), o);
            rgbd[p] = make_float4(o[0], o[1], o[2], o[3]);
        }
    }
}

// Scratch of ws_splat_maps_noalloc: one depth/id key per pixel of the largest supported
// image, in the module's static device memory (no allocation at call time).
static __device__ __align__(256) unsigned long long g_noalloc_zbuf[WS_NOALLOC_MAX_PIXELS];

static int grid_of(long long n, int threads) {
    long long g = (n + threads - 1) / threads;
    return (int)std::max(1LL, std::min(g, 148LL * 32));
}

}  // namespace ws

namespace {

// Device address of g_noalloc_zbuf per device, looked up once with that device current.
// Fixed-size table: the lookup path allocates nothing.
constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mutex;
unsigned long long *g_noalloc_ptr[kMaxDevices] = {};

int noalloc_scratch(unsigned long long **out) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return WS_ERR_CUDA;
    if (dev < 0 || dev >= kMaxDevices) return WS_ERR_NO_DEVICE;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, ws::g_noalloc_zbuf) != cudaSuccess || !p) {
            cudaGetLastError();
            return WS_ERR_CUDA;
        }
        g_noalloc_ptr[dev] = static_cast<unsigned long long *>(p);
    }
    *out = g_noalloc_ptr[dev];
    return WS_OK;
}

// Scratch of the geometry calls, taken and given back in stream order from a pool of the library's own per
// device.  The device's default pool returns its idle memory to the driver at every synchronisation, so the
// first call after one mapped its scratch again: the solver-map pass of a frame took 479 us instead of 35,
// and node construction, which synchronises itself, paid for it within each call.  This pool keeps up to
// kScratchKeep idle bytes (node construction of 1M surfels holds about 50 MB); what is above goes back at the
// next synchronisation, and all of it when the device's last solver is destroyed or the program asks for it
// (ws_trim_scratch: a program may use the geometry calls without a solver).  In a
// capture the allocation is the graph's own, as before.
constexpr unsigned long long kScratchKeep = 64ull << 20;
std::mutex g_scratch_mutex;
cudaMemPool_t g_scratch_pool[kMaxDevices] = {};

cudaMemPool_t scratch_pool() {   // null: none for this device
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_pool[dev]) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        unsigned long long keep = kScratchKeep;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess ||
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
            cudaGetLastError();
            if (pool) cudaMemPoolDestroy(pool);
            return nullptr;
        }
        g_scratch_pool[dev] = pool;
    }
    return g_scratch_pool[dev];
}

cudaError_t scratch_alloc(void **p, size_t bytes, cudaStream_t st) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (st && cudaStreamIsCapturing(st, &capture) != cudaSuccess) {
        cudaGetLastError();
        capture = cudaStreamCaptureStatusNone;
    }
    cudaMemPool_t pool = capture == cudaStreamCaptureStatusNone ? scratch_pool() : nullptr;
    return pool ? cudaMallocFromPoolAsync(p, bytes, pool, st) : cudaMallocAsync(p, bytes, st);
}

// Device temporaries of a node-growth call.
struct DeviceBlocks {
    explicit DeviceBlocks(cudaStream_t s) : st(s) {}
    DeviceBlocks(const DeviceBlocks &) = delete;
    DeviceBlocks &operator=(const DeviceBlocks &) = delete;
    cudaStream_t st;
    std::vector<void *> ptrs;
    cudaError_t err = cudaSuccess;
    template <class T>
    T *get(size_t bytes) {
        void *p = nullptr;
        if (err == cudaSuccess) err = scratch_alloc(&p, std::max<size_t>(bytes, 16), st);
        if (err != cudaSuccess) return nullptr;
        ptrs.push_back(p);
        return static_cast<T *>(p);
    }
    ~DeviceBlocks() {
        for (void *p : ptrs) cudaFreeAsync(p, st);
    }
};

// Node candidates of a point set and the overlap check, all on the device:
// VoxelSubsamplerSorting::PerformSubsample (libs/star/geometry/sampling/VoxelSubsamplerSorting.cu:8-96)
// on a 0.7 R grid, then the greedy check of AppendNodeFromVertexHost (NodeGraph.cu:652-704).
// On WS_OK, (*nodes)[0 .. *kept) holds the kept candidates in candidate order (w = 1).
// Synchronises `st` (the counts return to the host).
int grow_nodes(const float4 *pts, uint32_t n, float node_radius, DeviceBlocks &mem, cudaStream_t st, float4 **nodes,
               uint32_t *kept) {
    const float voxel = 0.7f * node_radius;
    // n + 1 entries: a spare value buffer later takes the scan of the kept flags and its total.
    uint32_t *keys = mem.get<uint32_t>(4ull * (n + 1)), *vals = mem.get<uint32_t>(4ull * (n + 1));
    uint32_t *keys2 = mem.get<uint32_t>(4ull * (n + 1)), *vals2 = mem.get<uint32_t>(4ull * (n + 1));
    uint32_t *heads = mem.get<uint32_t>(4ull * (n + 1));
    uint32_t *tmp = mem.get<uint32_t>(4ull * (std::max(n, ws::dedup_table(ws::kDedupCellsMost)) / ws::kScanTile + 4));
    uint32_t *hist = mem.get<uint32_t>(4ull * 256 * ws::sort_max_tiles(n));
    uint32_t *digit = mem.get<uint32_t>(4ull * 256);
    float4 *cand = mem.get<float4>(16ull * n);
    int *err = mem.get<int>(4);
    if (mem.err != cudaSuccess) return WS_ERR_CUDA;
    uint32_t nv = 0;
    {
        ws::k_voxel_key<<<ws::grid_of(n, 256), 256, 0, st>>>(pts, n, voxel, keys, vals);
        const bool alt = ws::radix_sort<uint32_t>(keys, vals, keys2, vals2, nullptr, n, n, 30, hist, digit, st);
        const uint32_t *sk = alt ? keys2 : keys, *sv = alt ? vals2 : vals;
        ws::k_voxel_marks<<<ws::grid_of(n, 256), 256, 0, st>>>(sk, n, heads);
        ws::exclusive_scan(heads, heads, n, tmp, st);
        ws::k_voxel_sample<<<ws::grid_of(n, 256), 256, 0, st>>>(sk, sv, heads, n, pts, voxel, cand);
        if (cudaMemcpyAsync(&nv, heads + n, 4, cudaMemcpyDeviceToHost, st) != cudaSuccess) return WS_ERR_CUDA;
        if (cudaStreamSynchronize(st) != cudaSuccess) return WS_ERR_CUDA;
    }
    *nodes = mem.get<float4>(16ull * nv);
    if (mem.err != cudaSuccess) return WS_ERR_CUDA;
    *kept = 0;
    if (nv == 0) return WS_OK;
    // The host loop's constants, in the same float arithmetic.
    const float r = 0.85f * node_radius;
    const float thr = r * r;
    const float inv_cell = 1.0f / (ws::kDedupCellScale * r);
    uint32_t *cnt = heads, *pos = vals2;   // free again: the candidates are written
    uint32_t pairs = (uint32_t)std::min<uint64_t>((uint64_t)ws::kDedupPairsPerCandidate * nv, 0xFFFFFFF0ull);
    const int cells = ws::dedup_cells(nv);
    const uint32_t table_cells = ws::dedup_table(cells);
    uint32_t *table = mem.get<uint32_t>(4ull * (table_cells + 1));
    float4 *placed = mem.get<float4>(16ull * nv);
    uint32_t *nbr = mem.get<uint32_t>(4ull * pairs);
    uint8_t *decision = mem.get<uint8_t>(nv);
    int dev = 0, sms = 0, per_sm = 0, coop = 0, flag = 0;
    if (mem.err != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ws::k_dedup_decide, ws::kDedupThreads, 0) != cudaSuccess ||
        per_sm < 1)
        return WS_ERR_CUDA;
    if (cudaMemsetAsync(err, 0, 4, st) != cudaSuccess || cudaMemsetAsync(decision, 0, nv, st) != cudaSuccess ||
        cudaMemsetAsync(table, 0, 4ull * table_cells, st) != cudaSuccess)
        return WS_ERR_CUDA;
    ws::k_dedup_count<<<ws::grid_of(nv, 256), 256, 0, st>>>(cand, nv, inv_cell, cells, table, err);
    ws::exclusive_scan(table, table, table_cells, tmp, st);
    ws::k_dedup_place<<<ws::grid_of(nv, 256), 256, 0, st>>>(cand, nv, inv_cell, cells, table, placed);
    ws::k_dedup_neighbours<false><<<ws::grid_of(nv, 128), 128, 0, st>>>(cand, table, placed, nv, inv_cell, cells, thr, cnt,
                                                                       nullptr, 0, err);
    ws::exclusive_scan(cnt, cnt, nv, tmp, st);
    uint32_t count = 0;
    for (int attempt = 0;; ++attempt) {
        ws::k_dedup_neighbours<true><<<ws::grid_of(nv, 128), 128, 0, st>>>(cand, table, placed, nv, inv_cell, cells, thr, cnt,
                                                                          nbr, pairs, err);
        const long long want = ((long long)nv + ws::kDedupThreads - 1) / ws::kDedupThreads;
        const int grid = (int)std::min<long long>(want, (long long)per_sm * sms);
        const uint32_t *nbr_ptr = cnt;
        uint32_t nv_arg = nv;
        void *args[] = {(void *)&nbr_ptr, (void *)&nbr, (void *)&pairs, (void *)&nv_arg, (void *)&decision, (void *)&err};
        if (cudaLaunchCooperativeKernel((const void *)ws::k_dedup_decide, dim3(grid), dim3(ws::kDedupThreads), args, 0,
                                        st) != cudaSuccess) {
            cudaGetLastError();   // a refused launch leaves no sticky error for later checks
            return WS_ERR_CUDA;
        }
        ws::k_dedup_flags<<<ws::grid_of(nv, 256), 256, 0, st>>>(decision, nv, pos);
        ws::exclusive_scan(pos, pos, nv, tmp, st);
        ws::k_dedup_emit<<<ws::grid_of(nv, 256), 256, 0, st>>>(cand, decision, pos, nv, *nodes);
        if (cudaGetLastError() != cudaSuccess) return WS_ERR_CUDA;
        uint32_t total = 0;
        if (cudaMemcpyAsync(&count, pos + nv, 4, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaMemcpyAsync(&total, cnt + nv, 4, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaMemcpyAsync(&flag, err, 4, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess)
            return WS_ERR_CUDA;
        // AppendNodeFromVertexHost stops on a NaN candidate (LOG(FATAL)).
        if (flag & 1) return WS_ERR_INVALID_ARGUMENT;
        if (!(flag & 8)) break;
        if (attempt > 0) return WS_ERR_CUDA;
        pairs = total;
        nbr = mem.get<uint32_t>(4ull * pairs);
        if (mem.err != cudaSuccess || cudaMemsetAsync(err, 0, 4, st) != cudaSuccess ||
            cudaMemsetAsync(decision, 0, nv, st) != cudaSuccess)
            return WS_ERR_CUDA;
    }
    if (flag & 4) return WS_ERR_TIMEOUT;
    *kept = count;
    return WS_OK;
}

}  // namespace

namespace ws {

// Gives the idle scratch of `device` back to the driver; false when the device refuses.
bool scratch_trim(int device) {
    if (device < 0 || device >= kMaxDevices) return true;   // such devices have no pool
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (!g_scratch_pool[device] || cudaMemPoolTrimTo(g_scratch_pool[device], 0) == cudaSuccess) return true;
    cudaGetLastError();
    return false;
}

}  // namespace ws

extern "C" {

int ws_trim_scratch(int device) {
    int devices = 0;
    if (cudaGetDeviceCount(&devices) != cudaSuccess) {
        cudaGetLastError();
        return WS_ERR_NO_DEVICE;
    }
    if (device < 0 || device >= devices) return WS_ERR_INVALID_ARGUMENT;
    // scratch is given back to the pool in stream order: it is idle once the device has come that far
    int here = 0;
    if (cudaGetDevice(&here) != cudaSuccess || cudaSetDevice(device) != cudaSuccess) return WS_ERR_CUDA;
    const bool done = cudaDeviceSynchronize() == cudaSuccess && ws::scratch_trim(device);
    return cudaSetDevice(here) == cudaSuccess && done ? WS_OK : WS_ERR_CUDA;
}

int ws_init_nodes(const float *surfels, int n, float node_radius, float *nodes_host, int cap, int *num_nodes,
                  void *stream) {
    if (!surfels || n <= 0 || !nodes_host || !num_nodes || cap < 2 || !(node_radius > 0.f))
        return WS_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    DeviceBlocks mem(st);
    float4 *nodes = nullptr;
    uint32_t kept = 0;
    const int rc = grow_nodes(reinterpret_cast<const float4 *>(surfels), (uint32_t)n, node_radius, mem, st, &nodes, &kept);
    if (rc != WS_OK) return rc;
    // InitializeNodeGraphFromVertex (NodeGraph.cu:479-486): two anchors at the origin come first.
    const float anchors[8] = {0.f, 0.f, 0.f, 1.f, 0.f, 0.f, 0.f, 1.f};
    const long long total = (long long)kept + 2;
    *num_nodes = (int)std::min<long long>(total, INT_MAX);
    if (total > cap) return WS_ERR_CAPACITY;
    std::memcpy(nodes_host, anchors, sizeof(anchors));
    if (kept && cudaMemcpyAsync(nodes_host + 8, nodes, 16ull * kept, cudaMemcpyDeviceToHost, st) != cudaSuccess)
        return WS_ERR_CUDA;
    return cudaStreamSynchronize(st) == cudaSuccess ? WS_OK : WS_ERR_CUDA;
}

int ws_expand_nodes(const float *vertices, int num_vertices, float node_radius, float *reference_nodes,
                    float *live_nodes, unsigned *node_time, unsigned current_time, int cap, int *num_nodes,
                    void *stream) {
    if (!num_nodes || !reference_nodes || num_vertices < 0 || !(node_radius > 0.f) || *num_nodes < 0 ||
        cap < *num_nodes)
        return WS_ERR_INVALID_ARGUMENT;
    // NaiveExpandNodeGraphFromVertexUnsupported (NodeGraph.cu:500-510): nothing to add.
    if (num_vertices == 0) return WS_OK;
    if (!vertices) return WS_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    DeviceBlocks mem(st);
    float4 *nodes = nullptr;
    uint32_t kept = 0;
    const int rc =
        grow_nodes(reinterpret_cast<const float4 *>(vertices), (uint32_t)num_vertices, node_radius, mem, st, &nodes, &kept);
    if (rc != WS_OK) return rc;
    const long long before = *num_nodes, total = before + kept;
    if (total > cap) {
        *num_nodes = (int)std::min<long long>(total, INT_MAX);
        return WS_ERR_CAPACITY;
    }
    if (kept) {
        const size_t bytes = 16ull * kept;
        if (cudaMemcpyAsync(reference_nodes + 4 * before, nodes, bytes, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
            return WS_ERR_CUDA;
        if (live_nodes && live_nodes != reference_nodes &&
            cudaMemcpyAsync(live_nodes + 4 * before, nodes, bytes, cudaMemcpyDeviceToDevice, st) != cudaSuccess)
            return WS_ERR_CUDA;
        // updateAppendNodeInitialTime (NodeGraph.cu:316-337)
        if (node_time) {
            ws::k_fill_u32<<<ws::grid_of(kept, 256), 256, 0, st>>>(node_time + before, kept, current_time);
            if (cudaGetLastError() != cudaSuccess) return WS_ERR_CUDA;
        }
    }
    if (cudaStreamSynchronize(st) != cudaSuccess) return WS_ERR_CUDA;
    *num_nodes = (int)total;
    return WS_OK;
}

// Nodes from which the node graph goes over the grid (us, ordered scan of every node / grid; K = 4 and 8): 1843
// nodes 40 / 65 and 50 / 76, 4117 72 / 91 and 91 / 109, 8247 170 / 134 and 240 / 151, 26865 1266 / 317 and
// 1673 / 380.  With one thread a node and box-skipped runs these were 384 us at 1.7k nodes (K = 8) and 2961 at 23k.
constexpr int kGraphGridFrom = 5000;

int ws_build_node_graph_ex(const float *nodes, const uint32_t *node_status, int n, int k, float node_radius,
                           int normalize_weights, uint16_t *knn, float *w, uint16_t *edges, void *stream) {
    if (!nodes || n <= 0 || n > 65535 || !knn || !w || !edges || (k != 4 && k != 8)) return WS_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const float r2 = node_radius * node_radius;
    const float4 *nd = reinterpret_cast<const float4 *>(nodes);
    const uint2 *status = reinterpret_cast<const uint2 *>(node_status);
    const int norm = normalize_weights ? 1 : 0;
    if (n < kGraphGridFrom || !(node_radius > 1e-6f && node_radius < 1e6f)) {
        const int grid = std::min((n + 3) / 4, 148 * 16);
        if (k == 4)
            ws::k_node_graph_ordered<4, false><<<grid, ws::kGraphThreads, 0, st>>>(nd, status, n, nullptr, nullptr, nullptr, r2, norm, knn,
                                                                           w, edges);
        else
            ws::k_node_graph_ordered<8, false><<<grid, ws::kGraphThreads, 0, st>>>(nd, status, n, nullptr, nullptr, nullptr, r2, norm, knn,
                                                                           w, edges);
        return cudaGetLastError() == cudaSuccess ? WS_OK : WS_ERR_CUDA;
    }
    // the grid and the list of open nodes from the stream-ordered pool: the call stays asynchronous
    const size_t table = 4ull * ws::kSkinCells, placed = 16ull * n;
    unsigned char *scratch = nullptr;
    const size_t bounds = 32ull * ((n + 31) / 32);
    if (scratch_alloc(reinterpret_cast<void **>(&scratch), placed + bounds + table + 4ull * n + 16, st) != cudaSuccess)
        return WS_ERR_CUDA;
    float4 *cell_nodes = reinterpret_cast<float4 *>(scratch), *boxes = cell_nodes + n;
    uint32_t *cell_end = reinterpret_cast<uint32_t *>(scratch + placed + bounds);
    uint32_t *list = reinterpret_cast<uint32_t *>(scratch + placed + bounds + table), *count = list + n;
    float *h = reinterpret_cast<float *>(count + 1);
    cudaError_t e = cudaFuncSetAttribute(ws::k_graph_grid, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)table);
    if (e == cudaSuccess) {
        // the K-th of 8 neighbours (itself among them) lies in the second ring around a node
        const float h0 = (k == 4 ? 1.75f : 2.2f) * node_radius;
        ws::k_graph_grid<<<1, ws::kSkinThreads, table, st>>>(nd, status, n, h0, cell_nodes, cell_end, h, count);
        const int grid = (4 * n + ws::kGraphThreads - 1) / ws::kGraphThreads, open_grid = std::min((n + 3) / 4, 148 * 8);
        if (k == 4) {
            ws::k_node_graph_cells<4><<<grid, ws::kGraphThreads, 0, st>>>(nd, status, n, cell_nodes, cell_end, h, r2, norm,
                                                                         knn, w, edges, list, count, boxes);
            ws::k_node_graph_ordered<4, true><<<open_grid, ws::kGraphThreads, 0, st>>>(nd, status, n, list, count, boxes, r2, norm, knn,
                                                                                w, edges);
        } else {
            ws::k_node_graph_cells<8><<<grid, ws::kGraphThreads, 0, st>>>(nd, status, n, cell_nodes, cell_end, h, r2, norm,
                                                                         knn, w, edges, list, count, boxes);
            ws::k_node_graph_ordered<8, true><<<open_grid, ws::kGraphThreads, 0, st>>>(nd, status, n, list, count, boxes, r2, norm, knn,
                                                                                w, edges);
        }
        e = cudaGetLastError();
    }
    const cudaError_t freed = cudaFreeAsync(scratch, st);
    return e == cudaSuccess && freed == cudaSuccess ? WS_OK : WS_ERR_CUDA;
}

int ws_build_node_graph(const float *nodes, int n, int k, float node_radius, uint16_t *knn, float *w, uint16_t *edges,
                        void *stream) {
    return ws_build_node_graph_ex(nodes, nullptr, n, k, node_radius, 1, knn, w, edges, stream);
}

// Nodes from which a full skinning goes over the grid (building it takes about 20 us; both sides measured as replayed
// kernels, k_skinning / grid, at 3000 and 260k surfels of a torus, us: 302 nodes 33 / 28 and 146 / 65, 366 nodes 38 / 28
// and 171 / 65, 535 nodes 54 / 26 and 237 / 63; below, k_skinning takes 13 and 56 at 97 nodes, 27 and 127 at 258).
constexpr int kSkinGridFrom = 300;

int ws_skinning_incremental(const float *nodes, const uint32_t *node_status, int num_nodes, int num_prev_nodes,
                            const float *verts, int num_verts, int num_remaining_surfels, float node_radius,
                            int normalize_weights, uint16_t *knn, float *sw, float *cw, void *stream) {
    if (!nodes || num_nodes <= 0 || num_nodes > 65535 || !verts || num_verts < 0 || !knn || !sw || !cw ||
        num_prev_nodes < 0 || num_prev_nodes > num_nodes || num_remaining_surfels < 0 ||
        num_remaining_surfels > num_verts)
        return WS_ERR_INVALID_ARGUMENT;
    const int count = num_verts - num_remaining_surfels;
    if (count == 0) return WS_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const float r2 = node_radius * node_radius;
    if (num_prev_nodes == 0 && num_nodes >= kSkinGridFrom && node_radius > 1e-6f && node_radius < 1e6f) {
        const bool chunked = num_nodes > ws::kSkinGridNodes;
        const size_t smem = 16 * (size_t)std::min(num_nodes, ws::kSkinGridNodes) + 4 * (size_t)ws::kSkinCells;
        constexpr int kMaxSmem = 16 * ws::kSkinGridNodes + 4 * ws::kSkinCells;   // one value, whichever thread calls
        auto kernel = chunked ? ws::k_skinning_grid<true> : ws::k_skinning_grid<false>;
        int dev = 0, sms = 0;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem) != cudaSuccess ||
            cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            return WS_ERR_CUDA;
        const int slab = chunked ? sms * ws::kSkinThreads : count;   // surfels of a launch
        for (long long v0 = num_remaining_surfels; v0 < num_verts; v0 += slab) {
            const int v1 = (int)std::min<long long>(num_verts, v0 + slab);
            const int grid = (int)std::min<long long>(sms, (v1 - v0 + 31) / 32);
            kernel<<<grid, ws::kSkinThreads, smem, st>>>(
                reinterpret_cast<const float4 *>(nodes), reinterpret_cast<const uint2 *>(node_status), num_nodes,
                reinterpret_cast<const float4 *>(verts), (int)v0, v1, node_radius,
                ws::SkinOut{r2, normalize_weights ? 1 : 0, reinterpret_cast<ushort4 *>(knn), reinterpret_cast<float4 *>(sw),
                            reinterpret_cast<float4 *>(cw)});
        }
        return cudaGetLastError() == cudaSuccess ? WS_OK : WS_ERR_CUDA;
    }
    // small sets in small blocks: 3001 new surfels are 12 blocks of 256 threads, 47 of 64
    const int threads = count <= 148 * 256 ? 64 : 256;
    ws::k_skinning<<<(count + threads - 1) / threads, threads, 0, st>>>(
        reinterpret_cast<const float4 *>(nodes), reinterpret_cast<const uint2 *>(node_status), num_nodes,
        num_prev_nodes, reinterpret_cast<const float4 *>(verts), num_remaining_surfels, num_verts, r2,
        normalize_weights ? 1 : 0, reinterpret_cast<ushort4 *>(knn), reinterpret_cast<float4 *>(sw),
        reinterpret_cast<float4 *>(cw));
    return cudaGetLastError() == cudaSuccess ? WS_OK : WS_ERR_CUDA;
}

int ws_skinning_ex(const float *nodes, const uint32_t *node_status, int num_nodes, const float *verts, int num_verts,
                   float node_radius, int normalize_weights, uint16_t *knn, float *sw, float *cw, void *stream) {
    return ws_skinning_incremental(nodes, node_status, num_nodes, 0, verts, num_verts, 0, node_radius,
                                   normalize_weights, knn, sw, cw, stream);
}

int ws_skinning(const float *nodes, int n_nodes, const float *verts, int n_verts, float node_radius, uint16_t *knn,
                float *sw, float *cw, void *stream) {
    return ws_skinning_ex(nodes, nullptr, n_nodes, verts, n_verts, node_radius, 1, knn, sw, cw, stream);
}

int ws_forward_warp(const float *se3, int num_nodes, const float *verts, const float *normals, int n,
                    const uint16_t *knn, const float *sw, const float *cw, float *out_v, float *out_n, void *stream) {
    if (!se3 || num_nodes <= 0 || num_nodes > 65535 || !verts || n < 0 || !knn || !sw || !cw || !out_v)
        return WS_ERR_INVALID_ARGUMENT;
    if (n == 0) return WS_OK;
    ws::k_forward_warp<<<ws::grid_of(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        se3, num_nodes, reinterpret_cast<const float4 *>(verts), reinterpret_cast<const float4 *>(normals), n,
        reinterpret_cast<const ushort4 *>(knn), reinterpret_cast<const float4 *>(sw),
        reinterpret_cast<const float4 *>(cw), reinterpret_cast<float4 *>(out_v), reinterpret_cast<float4 *>(out_n));
    return cudaGetLastError() == cudaSuccess ? WS_OK : WS_ERR_CUDA;
}

int ws_splat_maps(const float *verts, const float *attr_verts, const float *attr_normals, int n, int W, int H, float fx,
                  float fy, float cx, float cy, int footprint, uint32_t *index_map, float *vertex_map,
                  float *normal_map, void *stream) {
    if (!verts || n < 0 || W <= 0 || H <= 0 || !index_map || footprint < 0 || footprint > 8)
        return WS_ERR_INVALID_ARGUMENT;
    if ((vertex_map && !attr_verts) || (normal_map && !attr_normals)) return WS_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    unsigned long long *zbuf = nullptr;
    const size_t npix = (size_t)W * H;
    if (scratch_alloc(reinterpret_cast<void **>(&zbuf), 8 * npix, st) != cudaSuccess) return WS_ERR_CUDA;
    if (cudaMemsetAsync(zbuf, 0xff, 8 * npix, st) != cudaSuccess) {
        cudaFreeAsync(zbuf, st);
        return WS_ERR_CUDA;
    }
    if (n > 0)
        ws::k_splat<<<ws::grid_of(n, 256), 256, 0, st>>>(reinterpret_cast<const float4 *>(verts), n, W, H, fx, fy, cx,
                                                         cy, footprint, zbuf);
    ws::k_splat_resolve<<<ws::grid_of((long long)npix, 256), 256, 0, st>>>(
        zbuf, (int)npix, reinterpret_cast<const float4 *>(attr_verts), reinterpret_cast<const float4 *>(attr_normals),
        index_map, reinterpret_cast<float4 *>(vertex_map), reinterpret_cast<float4 *>(normal_map));
    cudaFreeAsync(zbuf, st);
    return cudaGetLastError() == cudaSuccess ? WS_OK : WS_ERR_CUDA;
}

int ws_splat_maps_noalloc(const float *verts, const float *attr_verts, const float *attr_normals, int n, int W,
                          int H, float fx, float fy, float cx, float cy, int footprint, uint32_t *index_map,
                          float *vertex_map, float *normal_map, void *stream) {
    if (!verts || n < 0 || W <= 0 || H <= 0 || !index_map || footprint < 0 || footprint > 8)
        return WS_ERR_INVALID_ARGUMENT;
    if ((vertex_map && !attr_verts) || (normal_map && !attr_normals)) return WS_ERR_INVALID_ARGUMENT;
    if ((long long)W * H > WS_NOALLOC_MAX_PIXELS) return WS_ERR_CAPACITY;
    unsigned long long *zbuf = nullptr;
    const int st_scratch = noalloc_scratch(&zbuf);
    if (st_scratch != WS_OK) return st_scratch;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t npix = (size_t)W * H;
    // the array keeps the previous call's keys: clear the part this call uses
    if (cudaMemsetAsync(zbuf, 0xff, 8 * npix, st) != cudaSuccess) return WS_ERR_CUDA;
    if (n > 0)
        ws::k_splat<<<ws::grid_of(n, 256), 256, 0, st>>>(reinterpret_cast<const float4 *>(verts), n, W, H, fx, fy, cx,
                                                         cy, footprint, zbuf);
    ws::k_splat_resolve<<<ws::grid_of((long long)npix, 256), 256, 0, st>>>(
        zbuf, (int)npix, reinterpret_cast<const float4 *>(attr_verts), reinterpret_cast<const float4 *>(attr_normals),
        index_map, reinterpret_cast<float4 *>(vertex_map), reinterpret_cast<float4 *>(normal_map));
    return cudaGetLastError() == cudaSuccess ? WS_OK : WS_ERR_CUDA;
}

int ws_render_solver_maps(const float *vertex_confid, const float *normal_radius, const float *color_time,
                          int num_surfels, const ws_render_params *params, uint32_t *index_map, float *vertex_map,
                          float *normal_map, float *rgbd_map, void *stream) {
    if (!params || !vertex_confid || num_surfels < 0 || !index_map) return WS_ERR_INVALID_ARGUMENT;
    const ws_render_params &p = *params;
    if (p.width <= 0 || p.height <= 0 || p.footprint < 0 || p.footprint > 8 || !(p.max_depth > 0.f))
        return WS_ERR_INVALID_ARGUMENT;
    if (normal_map && !normal_radius) return WS_ERR_INVALID_ARGUMENT;
    ws::RenderArgs a;
    a.W = p.width; a.H = p.height; a.fp = p.footprint;
    a.fx = p.fx; a.fy = p.fy; a.cx = p.cx; a.cy = p.cy;
    a.max_depth = p.max_depth; a.current_time = p.current_time;
    a.conf_threshold = p.confidence_threshold; a.time_threshold = p.time_threshold;
    for (int q = 0; q < 12; ++q) a.m[q] = p.world2camera[q];
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t npix = (size_t)p.width * p.height;
    unsigned long long *zbuf = nullptr;
    if (scratch_alloc(reinterpret_cast<void **>(&zbuf), 8 * npix, st) != cudaSuccess) return WS_ERR_CUDA;
    if (cudaMemsetAsync(zbuf, 0xff, 8 * npix, st) != cudaSuccess) {
        cudaFreeAsync(zbuf, st);
        return WS_ERR_CUDA;
    }
    const float4 *vc = reinterpret_cast<const float4 *>(vertex_confid);
    const float4 *ct = reinterpret_cast<const float4 *>(color_time);
    if (num_surfels > 0) ws::k_render_keys<<<ws::grid_of(num_surfels, 256), 256, 0, st>>>(vc, ct, num_surfels, a, zbuf);
    ws::k_render_resolve<<<ws::grid_of((long long)npix, 256), 256, 0, st>>>(
        zbuf, (int)npix, vc, reinterpret_cast<const float4 *>(normal_radius), ct, index_map,
        reinterpret_cast<float4 *>(vertex_map), reinterpret_cast<float4 *>(normal_map), reinterpret_cast<float4 *>(rgbd_map));
    cudaFreeAsync(zbuf, st);
    return cudaGetLastError() == cudaSuccess ? WS_OK : WS_ERR_CUDA;
}


int ws_render_observation_maps(const float *vertex_confid, const float *normal_radius, const float *color_time,
                               int num_surfels, const ws_render_params *params, uint32_t *index_map, float *rgbd_map,
                               void *stream) {
    if (!params || !vertex_confid || !normal_radius || num_surfels < 0 || !index_map) return WS_ERR_INVALID_ARGUMENT;
    const ws_render_params &p = *params;
    if (p.width <= 0 || p.height <= 0 || !(p.max_depth > 0.f)) return WS_ERR_INVALID_ARGUMENT;
    ws::RenderArgs a;
    a.W = p.width; a.H = p.height; a.fp = 0;
    a.fx = p.fx; a.fy = p.fy; a.cx = p.cx; a.cy = p.cy;
    a.max_depth = p.max_depth; a.current_time = p.current_time;
    a.conf_threshold = p.confidence_threshold; a.time_threshold = p.time_threshold;
    for (int q = 0; q < 12; ++q) a.m[q] = p.world2camera[q];
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t npix = (size_t)p.width * p.height;
    unsigned long long *zbuf = nullptr;
    if (scratch_alloc(reinterpret_cast<void **>(&zbuf), 8 * npix, st) != cudaSuccess) return WS_ERR_CUDA;
    if (cudaMemsetAsync(zbuf, 0xff, 8 * npix, st) != cudaSuccess) {
        cudaFreeAsync(zbuf, st);
        return WS_ERR_CUDA;
    }
    const float4 *ct = reinterpret_cast<const float4 *>(color_time);
    if (num_surfels > 0)
        ws::k_obs_keys<<<ws::grid_of(num_surfels, 256), 256, 0, st>>>(
            reinterpret_cast<const float4 *>(vertex_confid), reinterpret_cast<const float4 *>(normal_radius), ct,
            num_surfels, a, zbuf);
    ws::k_obs_resolve<<<ws::grid_of((long long)npix, 256), 256, 0, st>>>(zbuf, (int)npix, ct, index_map,
                                                                          reinterpret_cast<float4 *>(rgbd_map));
    cudaFreeAsync(zbuf, st);
    return cudaGetLastError() == cudaSuccess ? WS_OK : WS_ERR_CUDA;
}

}  // extern "C"
