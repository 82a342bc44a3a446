// Block PCG that keeps a scene in the shared memory of its blocks, included by ws_solve.cu after the helpers
// it shares with k_pcg (PcgArgs, matvec6, node_dot_group, twist_update_row, the bulk-copy helpers).
//
// What bounds a lone frame's PCG is not the matrix (1.6 MB at 1800 nodes, 7 MB at 8000) but the two
// scene-wide reductions an iteration and the dependent trips to L2 around them: k_pcg takes 22.8 us an
// iteration at 1800 nodes and 27.8 at 8000.  Here a scene's rows are split over blocks of one SM each.  A
// block keeps its rows' part of the symmetric store, the inverse diagonal and the vectors in its shared memory
// for all iterations (what does not fit streams through a ring of bulk copies, or is read from L2), and holds
// s and d of the rows that its items touch elsewhere (its halo).
//   * kGrid = false: the scene is one thread-block cluster (up to 16 SMs).  New s goes into the other blocks'
//     halos and transposed products to the owning block through distributed shared memory, and the
//     reductions are two hardware cluster barriers an iteration: 5.3 us an iteration at 500 nodes, 7.1 at
//     1800 (launches of 20, their load phase included).  What is left is latency and, with more rows a block,
//     shared-memory traffic (192 KB a block and iteration at 1800 nodes).  A batch's scenes are independent
//     clusters, the largest first.
//   * kGrid = true: the scene has a share of all SMs.  Halos, transposed products and partials go through L2,
//     and the blocks meet at a counter there: 9.6 us at 3000 nodes, 10.7 at 8000.  What is left are the two
//     meetings (fence, atomic, poll: 1.3 us each with 148 blocks) and the dependent trips to L2 after them.
//
// The arithmetic is k_pcg's, operation by operation (products per item, row sums in item order,
// contributions in column order, group partials over 16 rows, scene sums over groups in lane-strided
// order), so all forms give the same bits and a scene's result does not depend on which one ran, nor on what
// found room in shared memory.
//
// Waits: the cluster barriers are hardware barriers that every block of the scene reaches; a wait for a
// bulk copy is bounded, sets WS_ERR_TIMEOUT and goes on, so that no block leaves the others waiting.  A
// meeting of the grid is bounded too; a block whose wait gives up sets WS_ERR_TIMEOUT and leaves.
#pragma once

namespace ws {

constexpr int kResMaxCluster = 16;
constexpr int kResThreads = 512;
constexpr int kResRows = kResThreads;   // rows of a block at most: one per thread
constexpr uint32_t kResSmemBytes = 228864;   // beside 3 KB of static shared memory
constexpr uint32_t kResSmemMin = 49152;      // a cluster's partials (8 KB at most), product records and a ring of four
constexpr int kResMaxPolls = 1 << 22;   // polls of a meeting before it gives up (a second or more)
constexpr uint32_t kResNodes = kResRows * kResMaxCluster;   // nodes of a scene at most
constexpr int kPlanThreads = 512;
static_assert(kResNodes <= 8192, "13-bit column numbers in an item word");

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;\n" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory"); }
// Address of block `rank`'s copy of the shared-memory location `local` of this block.
__device__ __forceinline__ uint32_t peer_addr(uint32_t local, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(a) : "r"(local), "r"(rank));
    return a;
}
__device__ __forceinline__ uint32_t ld_peer_u32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];\n" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void st_peer2(uint32_t a, float x, float y) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};\n" ::"r"(a), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ void st_peer_f64(uint32_t a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;\n" ::"r"(a), "d"(v) : "memory");
}

// Item word of a block (built once per solve by k_pcg_plan): bits 0..8 the item's row in the block,
// 9..21 its column as an index into the block's vectors (its own rows, then its halo: the other blocks'
// rows that its items touch, in row order), 22..29 the rank of the block that owns the column, bit 31 a
// diagonal item; the second word is the lower entry the transposed product goes to, counted from the
// owning block's first (kInvalidIndex for none).
constexpr uint32_t kResDiag = 0x80000000u;

struct ResPlan {
    uint2 *words;          // [cap_items] item words
    // clusters: [cap_half] per row, from its first lower entry: (rank << 16) | halo index of the row there;
    // grid: [cap_items] per block, from its first item: the scene rows of its halo
    uint32_t *send;
    // [cap_nodes] clusters: blocks that hold the row in their halo; grid: lower entries from other blocks
    uint32_t *send_count;
    uint32_t *halo;        // halo rows of each block of the launch
    uint32_t *vec;         // grid: most own and halo rows of a block, per scene (zero before the plan)
    // where the device chooses the form (resident_pays; else null): ns an iteration of the launch's slowest block in
    // phase A and in phase B
    uint32_t *cost;
    uint32_t smem;         // bytes that a block of k_pcg_cluster will have
};
constexpr int kResMaxBlocks = 160;   // blocks of a scene at most

// The blocks' ranges of a scene: group, row, first item and first lower entry of every rank.
struct ResRanges {
    uint32_t group[kResMaxBlocks + 1], row[kResMaxBlocks + 1], item[kResMaxBlocks + 1], low[kResMaxBlocks + 1];
};

// Whole groups, balanced by items and rows (a row's own work is about four items').  Called by all
// threads of a block (at least kResMaxBlocks + 1); ends with a block barrier.
__device__ __forceinline__ void res_ranges(const PcgArgs &A, uint32_t nb, uint32_t nn, uint32_t groups, uint32_t size,
                                           ResRanges &R) {
    const uint32_t t = threadIdx.x;
    if (t <= size) {
        const uint32_t i0 = min(A.item_ptr[nb], A.cap_items), i1 = min(A.item_ptr[nb + nn], A.cap_items);
        const uint32_t total = (i1 - i0) + 4u * nn;
        const uint32_t target = (uint32_t)((unsigned long long)total * t / size);
        uint32_t lo = 0, hi = groups;
        while (lo < hi) {
            const uint32_t m = (lo + hi) >> 1, r = min(kRowsPerGroup * m, nn);
            if (min(A.item_ptr[nb + r], A.cap_items) - i0 + 4u * r < target) lo = m + 1;
            else hi = m;
        }
        R.group[t] = t == size ? groups : lo;
    }
    __syncthreads();
    bool even = false;   // a block would get more rows than it can hold: equal numbers of groups instead
    for (uint32_t k = 0; k < size; ++k) even |= (R.group[k + 1] - R.group[k]) * kRowsPerGroup > (uint32_t)kResRows;
    __syncthreads();
    if (t <= size) {
        if (even) R.group[t] = groups * t / size;
        const uint32_t r = nb + min(kRowsPerGroup * R.group[t], nn);
        R.row[t] = r;
        R.item[t] = min(A.item_ptr[r], A.cap_items);
        R.low[t] = min(A.rowptr[r] - A.item_ptr[r], A.cap_half);
    }
    __syncthreads();
}

__device__ __forceinline__ uint32_t res_rank_of(const ResRanges &R, uint32_t size, uint32_t row) {
    uint32_t lo = 0, hi = size - 1;   // the last block that starts at or before the row
    while (lo < hi) {
        const uint32_t m = (lo + hi + 1) >> 1;
        if (R.row[m] <= row) lo = m;
        else hi = m - 1;
    }
    return lo;
}

// Where a block of the launch belongs: its scene, and its rank among the scene's blocks.
struct ResPlace {
    uint32_t scene, rank, size;
};
template <bool kGrid>
__device__ __forceinline__ ResPlace res_place(const PcgArgs &A) {
    ResPlace p;
    if constexpr (kGrid) {
        uint32_t s = 0;   // the scenes' blocks follow one another in scene order
        while (s + 1 < A.num_scenes && blockIdx.x >= (uint32_t)A.scenes[s + 1].pcg_block0) ++s;
        p.scene = s;
        p.rank = blockIdx.x - (uint32_t)A.scenes[s].pcg_block0;
        p.size = (uint32_t)A.scenes[s].pcg_blocks;
    } else {
        p.rank = cluster_rank();
        p.size = cluster_size();
        p.scene = (uint32_t)A.scenes[blockIdx.x / p.size].pcg_order;
    }
    return p;
}

// What bounds a block, in ns an iteration: least squares over launches of 1 to 30 scenes of 500 to 8000 nodes with 5 to
// 30 upper pairs a row, within 15 % of what was measured (5.3 to 180 us).  Phase A: the block's items, on the grid
// twice beyond some 4600 of them, in a cluster also the products sent to other blocks.
// Phase B: the contributions that rows read from L2.
template <bool kGrid>
__device__ __forceinline__ void res_cost(const ResPlan &P, uint32_t vec_rows, uint32_t items, uint32_t lows,
                                         uint32_t crossing, uint32_t outside, uint32_t groups) {
    if (P.cost == nullptr) return;
    const uint32_t vec = 48u * vec_rows + 35000u + (kGrid ? 0u : 16u * groups);   // beside records and a small ring
    const bool vec_fits = vec <= P.smem, low_fits = vec + 24u * lows <= P.smem;
    const float i = (float)items;
    float a, b;
    if (kGrid) {
        a = 7.f * i + 7.2f * fmaxf(i - 4600.f, 0.f) + (vec_fits ? 0.f : 6.f * i);
        b = 4.8f * (float)outside + (low_fits ? 0.f : 0.6f * (float)lows);
    } else {
        a = 3.5f * i + 6.5f * (float)crossing + (vec + 24u * lows + 144u * items > P.smem ? 2500.f : 0.f);
        b = low_fits ? 0.f : 4.6f * (float)lows;
    }
    atomicMax(P.cost, (uint32_t)a);
    atomicMax(P.cost + 1, (uint32_t)b);
}

// Item words, halos and send lists of every block, once per solve (the structure is the same in every
// Gauss-Newton iteration).  One cluster per scene, ranks as in k_pcg_cluster.  A block's halo is a bit
// per scene row; a row's index in it is the number of set bits before it.  A row's lower entries name
// the blocks whose items touch it, and so those its new s has to reach.
template <bool kGrid>
__global__ void __launch_bounds__(kPlanThreads) k_pcg_plan(PcgArgs A, const uint32_t *colidx, ResPlan P) {
    __shared__ ResRanges R;
    __shared__ uint32_t bits[kResNodes / 32], before[kResNodes / 32], first_item[kResRows], warp_sums[kPlanThreads / 32];
    __shared__ uint32_t s_crossing, s_outside;   // items with a column in another block, contributions from other blocks
    static_assert(kResNodes / 32 <= kPlanThreads, "a thread per bitmap word");
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    const ResPlace place = res_place<kGrid>(A);
    const uint32_t rank = place.rank, size = place.size;
    const Scene &sc = A.scenes[place.scene];
    const uint32_t nb = (uint32_t)sc.node_base, nn = (uint32_t)sc.num_nodes;
    res_ranges(A, nb, nn, (uint32_t)sc.num_chunks, size, R);
    const uint32_t row0 = R.row[rank], row1 = R.row[rank + 1], rows = row1 - row0;
    const uint32_t item0 = R.item[rank], items = R.item[rank + 1] - item0;
    if (tid == 0) s_crossing = s_outside = 0;
    if (tid < kResNodes / 32) bits[tid] = 0;
    for (uint32_t r = tid; r < rows; r += kPlanThreads) first_item[r] = min(A.item_ptr[row0 + r], A.cap_items) - item0;
    __syncthreads();
    auto column = [&](uint32_t word) { return min(max(word & ~kItemRowStart, nb), nb + nn - 1); };
    for (uint32_t k = tid; k < items; k += kPlanThreads) {
        const uint32_t col = column(__ldg(A.item_col + item0 + k));
        const bool crosses = col < row0 || col >= row1;
        if (crosses) atomicOr(&bits[(col - nb) >> 5], 1u << ((col - nb) & 31u));
        const unsigned active = __activemask(), crossing = __ballot_sync(active, crosses);
        if (P.cost != nullptr && lane == (uint32_t)__ffs(active) - 1u) atomicAdd(&s_crossing, (uint32_t)__popc(crossing));
    }
    __syncthreads();
    {   // halo rows before each bitmap word
        const uint32_t n = tid < kResNodes / 32 ? (uint32_t)__popc(bits[tid]) : 0u;
        uint32_t inc = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= (uint32_t)o) inc += v;
        }
        if (lane == 31) warp_sums[tid >> 5] = inc;
        __syncthreads();
        uint32_t base = 0;
        for (uint32_t w = 0; w < (tid >> 5); ++w) base += warp_sums[w];
        if (tid < kResNodes / 32) before[tid] = base + inc - n;
        if (tid == kPlanThreads - 1) {
            P.halo[blockIdx.x] = base + inc;
            if constexpr (kGrid) atomicMax(P.vec + place.scene, rows + base + inc);
        }
    }
    __syncthreads();
    for (uint32_t k = tid; k < items; k += kPlanThreads) {
        const uint2 it = __ldg(A.item_info + item0 + k);
        uint32_t lo = 0, hi = rows - 1;   // the last row that starts at or before item k
        while (lo < hi) {
            const uint32_t m = (lo + hi + 1) >> 1;
            if (first_item[m] <= k) lo = m;
            else hi = m - 1;
        }
        const bool diag = (it.x & kItemRowStart) != 0;
        const uint32_t col = column(it.x), c = col - nb, cr = res_rank_of(R, size, col);
        const uint32_t at = cr == rank ? col - row0
                                       : rows + before[c >> 5] + (uint32_t)__popc(bits[c >> 5] & ((1u << (c & 31u)) - 1u));
        uint32_t slot = kInvalidIndex;
        if (!diag && it.y >= R.low[cr] && it.y < R.low[cr + 1]) slot = it.y - R.low[cr];
        P.words[item0 + k] = make_uint2(lo | (at << 9) | (cr << 22) | (diag ? kResDiag : 0u), slot);
    }
    if constexpr (kGrid) {
        for (uint32_t c = tid; c < kResNodes; c += kPlanThreads)
            if ((bits[c >> 5] >> (c & 31u)) & 1u)   // at most one halo row per item
                P.send[item0 + before[c >> 5] + (uint32_t)__popc(bits[c >> 5] & ((1u << (c & 31u)) - 1u))] = nb + c;
        for (uint32_t r = tid; r < rows; r += kPlanThreads) {
            const uint32_t q0 = A.rowptr[row0 + r], p0 = A.item_ptr[row0 + r];
            const uint32_t n = (A.rowptr[row0 + r + 1] - q0) - (A.item_ptr[row0 + r + 1] - p0);
            uint32_t outside = 0;   // columns ascend, so those of other blocks come first
            while (outside < n && q0 + 1u + outside < A.cap_blocks && __ldg(colidx + q0 + 1u + outside) < row0) ++outside;
            P.send_count[row0 + r] = outside;
            if (P.cost != nullptr) atomicAdd(&s_outside, outside);
        }
        __syncthreads();
        if (tid == 0) res_cost<kGrid>(P, rows + P.halo[blockIdx.x], items, R.low[rank + 1] - R.low[rank], s_crossing, s_outside,
                                      (uint32_t)sc.num_chunks);
        return;
    }
    cluster_arrive();
    cluster_wait();   // every block's bitmap is complete
    if (tid == 0) {   // a cluster lays its blocks out alike: by its most vector rows and contributions
        uint32_t most = 0, lows = 0;
        for (uint32_t k = 0; k < size; ++k) {
            most = max(most, R.row[k + 1] - R.row[k] + __ldcg(P.halo + (blockIdx.x - rank + k)));
            lows = max(lows, R.low[k + 1] - R.low[k]);
        }
        res_cost<kGrid>(P, most, items, lows, s_crossing, 0, (uint32_t)sc.num_chunks);
    }
    for (uint32_t r = tid; r < rows; r += kPlanThreads) {
        const uint32_t row = row0 + r, c = row - nb;
        const uint32_t q0 = A.rowptr[row], p0 = A.item_ptr[row];
        const uint32_t l0 = min(q0 - p0, A.cap_half);
        const uint32_t n = min((A.rowptr[row + 1] - q0) - (A.item_ptr[row + 1] - p0), A.cap_half - l0);
        uint32_t sent = 0, last = rank;
        for (uint32_t k = 0; k < n && q0 + 1u + k < A.cap_blocks; ++k) {   // columns ascend, so ranks do
            const uint32_t q = res_rank_of(R, size, min(max(__ldg(colidx + q0 + 1u + k), nb), nb + nn - 1));
            if (q == rank || q == last) continue;
            last = q;
            const uint32_t word = ld_peer_u32(peer_addr(smem_addr(&bits[c >> 5]), q));
            if (((word >> (c & 31u)) & 1u) == 0) continue;
            const uint32_t at = (R.row[q + 1] - R.row[q]) + ld_peer_u32(peer_addr(smem_addr(&before[c >> 5]), q)) +
                                (uint32_t)__popc(word & ((1u << (c & 31u)) - 1u));
            P.send[l0 + sent++] = (q << 16) | at;
        }
        P.send_count[row] = sent;
    }
    cluster_arrive();
    cluster_wait();   // no block leaves while another reads its bitmap
}

// One thread's bounded wait for phase `parity` of `bar`; false when the polls ran out.
__device__ __forceinline__ bool bulk_wait_one(unsigned long long *bar, unsigned parity, int polls = kBulkMaxPolls) {
    unsigned done = 0;
    for (int i = 0; i < polls && done == 0; ++i)
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                     " selp.u32 %0, 1, 0, p;\n}\n"
                     : "=r"(done)
                     : "r"(smem_addr(bar)), "r"(parity)
                     : "memory");
    return done != 0;
}

// Self-test: a wait for a copy that nobody has started runs out.
__global__ void k_bulk_wait_selftest(int *err) {
    __shared__ __align__(8) unsigned long long bar;
    if (threadIdx.x == 0) {
        bulk_init(&bar, 1);
        if (!bulk_wait_one(&bar, 0, 256)) set_err(err, WS_ERR_TIMEOUT);
    }
}

// Sum of a scene's group partials in the order of reduce_scene, eight of a lane's loads at a time.
template <bool kGrid>
__device__ __forceinline__ double res_reduce(const PcgArgs &A, const double *part, int groups, int lane) {
    double v = 0.0;
    for (int c0 = lane; c0 < groups; c0 += 256) {
        double x[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int c = min(c0 + 32 * k, groups - 1);
            x[k] = kGrid ? __ldcg(part + c) : part[c];
        }
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (c0 + 32 * k < groups) v += x[k];
    }
    v = warp_sum(v);
    return A.fp64 ? v : (double)(float)v;
}

constexpr uint32_t kResChunkBytes = 32u * 144u;   // matrix blocks of 32 items
constexpr uint32_t kResMaxRing = 24;
constexpr uint32_t kResMinLocal = 32u * kResThreads + 4u * kResChunkBytes + 64u;   // product records and a small ring

struct ResShared {
    ResRanges R;
    __align__(8) unsigned long long bar, ring[kResMaxRing];
    volatile uint32_t armed[kResMaxRing];   // copies armed on each ring buffer so far
    float scalar[2];                        // alpha and beta
    int left;                               // grid: a wait gave up
};

// kGrid: a scene's blocks are blocks of a cooperative launch; they meet at a counter in L2 and exchange
// halos, contributions and partials through L2.
// kVec: s and d are in shared memory (1) or in A.sd0 / A.sd1 (0) for all of the scene's blocks, since blocks that
// have them in shared memory publish s by another way than blocks that have not; -1: a cluster, which sees by its
// largest block.  (As a run-time answer on the grid it costs registers the kernel has not: frames of 8000 nodes 1780 -> 1820 us.)
template <bool kGrid, int kVec>
__device__ __forceinline__ void pcg_resident(const PcgArgs &A, const ResPlan &P, uint32_t smem_bytes, ResShared &S) {
    constexpr uint32_t kThreads = kResThreads, kWarps = kResThreads / 32;
    constexpr uint32_t kChunkBytes = kResChunkBytes, kMaxRing = kResMaxRing, kMinLocal = kResMinLocal;
    extern __shared__ __align__(128) unsigned char res_smem[];
    ResRanges &R = S.R;
    const uint32_t tid = threadIdx.x;
    const int lane = tid & 31;
    const uint32_t warp = tid >> 5;
    if constexpr (!kGrid) cluster_arrive();   // every block of the cluster has started once the matching wait returns
    const ResPlace place = res_place<kGrid>(A);
    const uint32_t rank = place.rank, size = place.size;
    const Scene &sc = A.scenes[place.scene];
    const uint32_t nb = (uint32_t)sc.node_base, nn = (uint32_t)sc.num_nodes, groups = (uint32_t)sc.num_chunks;
    res_ranges(A, nb, nn, groups, size, R);
    // most vector rows (own and halo) and lower entries of a block: what peers write lies at the same offsets
    const uint32_t halo = __ldg(P.halo + blockIdx.x);
    uint32_t vmax = R.row[rank + 1] - R.row[rank] + halo, lmax = R.low[rank + 1] - R.low[rank];
    if constexpr (!kGrid)
        for (uint32_t k = 0; k < size; ++k) {
            vmax = max(vmax, R.row[k + 1] - R.row[k] + __ldg(P.halo + (blockIdx.x - rank + k)));
            lmax = max(lmax, R.low[k + 1] - R.low[k]);
        }
    const uint32_t row0 = R.row[rank], rows = R.row[rank + 1] - row0;
    const uint32_t item0 = R.item[rank], items = R.item[rank + 1] - item0;
    const uint32_t low0 = R.low[rank], lows = R.low[rank + 1] - low0;
    const uint32_t group0 = R.group[rank], own_groups = R.group[rank + 1] - group0;
    const uint32_t chunks = (items + 31u) / 32u;

    // ---- shared memory: first what peers write (the same offsets in every block), then this block's ----
    const uint32_t off_pa = 0, off_pb = 8u * groups;   // clusters: the partials of phases A and B
    uint32_t off = kGrid ? 0u : (16u * groups + 15u) & ~15u;
    const uint32_t off_s = off, off_d = off + 24u * vmax;
    const bool vec_shared = kVec >= 0 ? kVec != 0 : off + 48u * vmax + kMinLocal <= smem_bytes;
    if (vec_shared) off = (off + 48u * vmax + 15u) & ~15u;
    const uint32_t off_contrib = off;
    const bool contrib_shared = off + 24u * lmax + kMinLocal <= smem_bytes;   // else through A.contrib
    if (contrib_shared) off = (off + 24u * lmax + 15u) & ~15u;
    const bool words_shared = off + 8u * items + kMinLocal <= smem_bytes;
    uint2 *words = words_shared ? reinterpret_cast<uint2 *>(res_smem + off) : P.words + item0;
    if (words_shared) off = (off + 8u * items + 15u) & ~15u;
    // clusters: where the rows' s goes; grid: the rows of the halo
    const uint32_t send_n = kGrid ? halo : lows;
    uint32_t *send_from = P.send + (kGrid ? item0 : low0);
    const bool send_shared = off + 4u * send_n + kMinLocal <= smem_bytes;
    uint32_t *send = send_shared ? reinterpret_cast<uint32_t *>(res_smem + off) : send_from;
    if (send_shared) off = (off + 4u * send_n + 15u) & ~15u;
    // product records: of every item when everything fits, else of one item a thread
    const bool stage_all = off + 32u * items + 144u * rows + kChunkBytes * chunks <= smem_bytes;
    const uint32_t stage_items = stage_all ? max(32u * chunks, (uint32_t)kThreads) : (uint32_t)kThreads;
    float *stage = reinterpret_cast<float *>(res_smem + off);
    off += 32u * (stage_all ? items : (uint32_t)kThreads);
    const bool inv_shared = off + 144u * rows + 4u * kChunkBytes <= smem_bytes;
    float *inv_s = reinterpret_cast<float *>(res_smem + off);
    if (inv_shared) off += 144u * rows;
    // block buffers of 32 items: all chunks when they fit, else the first `resident` chunks and a ring
    // that the others stream through, from one iteration into the next
    const uint32_t bufs = (smem_bytes - off) / kChunkBytes;
    const uint32_t ring = bufs >= chunks ? 0u : min(bufs, min(kMaxRing, kWarps));
    const uint32_t resident = bufs >= chunks ? chunks : bufs - ring, streamed = chunks - resident;
    float *blk_s = reinterpret_cast<float *>(res_smem + off);
    const uint32_t smem_base = smem_addr(res_smem);
    const uint32_t stream_total = streamed * (uint32_t)max(A.pcg_iters, 0);
    // chunk `resident + n % streamed` into ring buffer n % ring
    auto stream_chunk = [&](uint32_t n) {
        const uint32_t first = 32u * (resident + n % streamed), bytes = 144u * min(32u, items - first), b = n % ring;
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(&S.ring[b])), "r"(bytes)
                     : "memory");
        S.armed[b] = n / ring + 1u;
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                         smem_addr(blk_s) + kChunkBytes * (resident + b)),
                     "l"(A.sym_blocks + 36ull * (item0 + first)), "r"(bytes), "r"(smem_addr(&S.ring[b]))
                     : "memory");
    };

    // ---- load: blocks and inverse diagonals by bulk copies, words and send lists by plain loads ----
    if (tid == 0) {
        bulk_init(&S.bar, 1);
        if (ring > 0) bulk_init(S.ring, (int)ring);
        for (uint32_t b = 0; b < kMaxRing; ++b) S.armed[b] = 0;
        const uint32_t block_bytes = 144u * min(32u * resident, items), bytes = block_bytes + (inv_shared ? 144u * rows : 0u);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(&S.bar)), "r"(bytes)
                     : "memory");
        auto copy = [&](const float *src, float *dst, uint32_t n) {   // n bytes, a multiple of 16
            for (uint32_t at = 0; at < n; at += 18432u)
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                        smem_addr(dst) + at),
                    "l"(reinterpret_cast<const char *>(src) + at), "r"(min(18432u, n - at)), "r"(smem_addr(&S.bar))
                    : "memory");
        };
        if (inv_shared) copy(A.inv_diag + 36ull * row0, inv_s, 144u * rows);
        copy(A.sym_blocks + 36ull * item0, blk_s, block_bytes);
        for (uint32_t n = 0; n < min(ring, stream_total); ++n) stream_chunk(n);
    }
    if (words_shared)
        for (uint32_t k = tid; k < items; k += kThreads) words[k] = __ldg(P.words + item0 + k);
    if (send_shared)
        for (uint32_t k = tid; k < send_n; k += kThreads) send[k] = __ldg(send_from + k);
    // the thread's row: sixteen rows (a group) a warp while there are warps enough, so that the row loops of
    // a warp are as long as its longest of sixteen
    const bool sparse = rows <= kResRows / 2;
    const uint32_t r = sparse ? (lane < kRowsPerGroup ? warp * kRowsPerGroup + (uint32_t)lane : (uint32_t)kResRows) : tid;
    const uint32_t row = row0 + r;
    const bool has_row = r < rows;
    const bool row_warp = sparse ? warp * kRowsPerGroup < rows : warp * 32u < rows;
    uint32_t u_begin = 0, u_end = 0, l_begin = 0, l_count = 0, sends = 0;
    float xv[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, rv[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    float dv[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (has_row) {
        const uint32_t p0 = A.item_ptr[row], p1 = A.item_ptr[row + 1], q0 = A.rowptr[row], q1 = A.rowptr[row + 1];
        u_begin = min(p0, A.cap_items) - item0;
        u_end = min(p1, A.cap_items) - item0;
        l_begin = min(min(q0 - p0, A.cap_half) - low0, lows);
        l_count = min((q1 - q0) - (p1 - p0), lows - l_begin);
        sends = min(P.send_count[row], l_count);
        load6(A.jtr + 8ull * row, rv);
    }
    __syncthreads();   // the mbarriers are initialised, the words and send lists written
    if (!bulk_wait(&S.bar, 0) && lane == 0) set_err(A.err, WS_ERR_TIMEOUT);

    // y = M^-1 x of the thread's row
    auto precondition = [&](const float *x, float *y) {
        if (inv_shared) {
            const float4 *M = reinterpret_cast<const float4 *>(inv_s + 36u * r);
#pragma unroll
            for (int i = 0; i < 6; ++i) y[i] = 0.f;
#pragma unroll
            for (int e9 = 0; e9 < 9; ++e9) {
                const float4 v = M[e9];
                const float e4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int e = 4 * e9 + k;
                    y[e / 6] += e4[k] * x[e % 6];
                }
            }
        } else {
            matvec6(A.inv_diag + 36ull * row, x, y);
        }
    };
    // a group's partial to every block of the cluster: lane k of the group writes block k's copy (grid: to L2)
    auto publish = [&](uint32_t off_part, double part) {
        const uint32_t g = r / kRowsPerGroup, k = r % kRowsPerGroup;
        static_assert(kRowsPerGroup >= kResMaxCluster, "a lane per block");
        if constexpr (kGrid) {
            if (g < own_groups && k == 0)
                __stcg(A.group_partial + (off_part == off_pa ? 0u : A.total_groups) + sc.chunk_base + group0 + g, part);
        } else {
            if (g < own_groups && k < size) st_peer_f64(peer_addr(smem_base + off_part + 8u * (group0 + g), k), part);
        }
    };
    // Every block of the scene has reached this point, and what it wrote before is visible; false when the
    // wait gave up (grid only: WS_ERR_TIMEOUT is set, and the block leaves).
    uint32_t meetings = 0;
    auto meet = [&]() -> bool {
        if constexpr (kGrid) {
            ++meetings;
            __syncthreads();
            if (tid == 0) {
                uint32_t *counter = A.scene_counter + (size_t)kSceneSync * place.scene;
                __threadfence();
                atomicAdd(counter, 1u);
                bool ok = false;
                for (int i = 0; i < kResMaxPolls && !ok; ++i) {
                    ok = ld_acquire(counter) >= size * meetings;
                    if (!ok && (i & 1023) == 1023 && *reinterpret_cast<volatile int *>(A.err) == WS_ERR_TIMEOUT) break;
                }
                if (!ok) set_err(A.err, WS_ERR_TIMEOUT);
                S.left = ok ? 0 : 1;
            }
            __syncthreads();
            return S.left == 0;
        } else {
            cluster_arrive();
            cluster_wait();
            return true;
        }
    };
    // the scene's sum of group partials, in the block's first warp
    auto reduce = [&](uint32_t off_part) -> double {
        const double *part = kGrid ? A.group_partial + (off_part == off_pa ? 0u : A.total_groups) + sc.chunk_base
                                   : reinterpret_cast<const double *>(res_smem + off_part);
        return res_reduce<kGrid>(A, part, (int)groups, lane);
    };
    // s of the row into the block's vectors and into the halos that hold the row
    auto store_s = [&](const float *s, float *sd) {
        if (vec_shared) {
            float2 *p = reinterpret_cast<float2 *>(res_smem + off_s + 24u * r);
            p[0] = make_float2(s[0], s[1]);
            p[1] = make_float2(s[2], s[3]);
            p[2] = make_float2(s[4], s[5]);
            if constexpr (kGrid) {   // for the halos (A.r is free here)
                __stcg(reinterpret_cast<float4 *>(A.r + 8ull * row), make_float4(s[0], s[1], s[2], s[3]));
                __stcg(reinterpret_cast<float2 *>(A.r + 8ull * row + 4), make_float2(s[4], s[5]));
            }
            for (uint32_t k = 0; !kGrid && k < sends; ++k) {
                const uint32_t to = send[l_begin + k];
                const uint32_t a = peer_addr(smem_base + off_s + 24u * (to & 0xFFFFu), to >> 16);
                st_peer2(a, s[0], s[1]);
                st_peer2(a + 8u, s[2], s[3]);
                st_peer2(a + 16u, s[4], s[5]);
            }
        } else {
            store6(sd + (size_t)kSdStride * row, s);
        }
    };

    // ---- init: r = b, s = M^-1 b, x = 0, d = 0, delta = <r, s> ----
    if (vec_shared)
        for (uint32_t k = tid; k < 3u * (rows + halo); k += kThreads)
            reinterpret_cast<float2 *>(res_smem + off_d)[k] = make_float2(0.f, 0.f);
    if constexpr (!kGrid) cluster_wait();
    if (row_warp) {
        float s[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (has_row) {
            precondition(rv, s);
            store_s(s, A.sd0);
            if (!vec_shared) store6_f2(A.sd0 + (size_t)kSdStride * row + 6, dv);
        }
        publish(off_pb, node_dot_group(A, rv, s, has_row));
    }
    bool here = meet();
    // the scene's scalars: every block's last warp, the first to have no rows, takes the sums (all blocks see
    // the same partials)
    constexpr uint32_t kScalarWarp = kWarps - 1;
    double delta = 0.0;
    if (here && warp == kScalarWarp) delta = reduce(off_pb);
    // grid: s of the thread's halo row, requested before beta is known
    float halo_s[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (kGrid && here && vec_shared && tid < halo) load6(A.r + 8ull * send[tid], halo_s);
    float beta = 0.f;

    for (int it = 0; here && it < A.pcg_iters; ++it) {
        const float *sd_old = (it & 1) ? A.sd1 : A.sd0;
        float *sd_new = (it & 1) ? A.sd0 : A.sd1;
        // ---- phase A: d = s + beta d (own rows and halo), q = A d, <d, q> ----
        if (vec_shared) {
            const float2 *ps = reinterpret_cast<const float2 *>(res_smem + off_s);
            float2 *pd = reinterpret_cast<float2 *>(res_smem + off_d);
            if constexpr (kGrid)
                for (uint32_t k = tid; k < halo; k += kThreads) {
                    float s[6];
                    if (k == tid) {
#pragma unroll
                        for (int e = 0; e < 6; ++e) s[e] = halo_s[e];
                    } else {
                        load6(A.r + 8ull * send[k], s);
                    }
                    float2 *d = pd + 3u * (rows + k);
#pragma unroll
                    for (int e = 0; e < 3; ++e)
                        d[e] = make_float2(s[2 * e] + beta * d[e].x, s[2 * e + 1] + beta * d[e].y);
                }
            for (uint32_t k = tid; k < 3u * (kGrid ? rows : rows + halo); k += kThreads) {
                const float2 s = ps[k], d = pd[k];
                pd[k] = make_float2(s.x + beta * d.x, s.y + beta * d.y);
            }
            __syncthreads();
        }
        float q[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        double dsum = 0.0;
        for (uint32_t base = 0; base < items; base += stage_items) {
            const uint32_t cnt = min(stage_items, items - base);
            for (uint32_t c0 = warp; 32u * c0 < cnt; c0 += kWarps) {
                const uint32_t k = 32u * c0 + (uint32_t)lane, u = base + k, chunk = u >> 5;
                const bool valid = k < cnt;
                const uint2 w = valid ? words[u] : make_uint2(0u, kInvalidIndex);
                float4 blk[9];
                uint32_t buf = chunk;
                uint32_t n = 0;
                if (chunk >= resident) {
                    n = (uint32_t)it * streamed + (chunk - resident);
                    buf = resident + n % ring;
                    // the copy is armed by the warp that used the buffer before; a parity wait is only
                    // meaningful once it is
                    bool armed = false;
                    for (int i = 0; i < kBulkMaxPolls && !armed; ++i) armed = S.armed[n % ring] > n / ring;
                    armed = __all_sync(0xffffffffu, armed);
                    __syncwarp();
                    if ((!armed || !bulk_wait(&S.ring[n % ring], (n / ring) & 1u)) && lane == 0)
                        set_err(A.err, WS_ERR_TIMEOUT);
                }
                if (valid) {
                    const float4 *b = reinterpret_cast<const float4 *>(blk_s + (kChunkBytes / 4u) * buf + 36u * lane);
#pragma unroll
                    for (int e = 0; e < 9; ++e) blk[e] = b[e];
                }
                if (chunk >= resident) {   // the buffer is free: it takes the chunk `ring` ahead
                    __syncwarp();
                    if (lane == 0 && n + ring < stream_total) stream_chunk(n + ring);
                }
                if (!valid) continue;
                float vr[6], vc[6];
                const uint32_t cr = (w.x >> 22) & 255u;
                if (vec_shared) {
                    const float2 *pr = reinterpret_cast<const float2 *>(res_smem + off_d) + 3u * (w.x & 511u);
                    const float2 *pc = reinterpret_cast<const float2 *>(res_smem + off_d) + 3u * ((w.x >> 9) & 8191u);
#pragma unroll
                    for (int e = 0; e < 3; ++e) {
                        const float2 a = pr[e], b = pc[e];
                        vr[2 * e] = a.x;
                        vr[2 * e + 1] = a.y;
                        vc[2 * e] = b.x;
                        vc[2 * e + 1] = b.y;
                    }
                } else {
                    const uint32_t col = min(max(__ldg(A.item_col + item0 + u) & ~kItemRowStart, nb), nb + nn - 1);
                    float sr[6], dr[6], s2[6], d2[6];
                    const float *pr = sd_old + (size_t)kSdStride * (row0 + (w.x & 511u)), *pc = sd_old + (size_t)kSdStride * col;
                    load6(pr, sr);
                    load6_f2(pr + 6, dr);
                    load6(pc, s2);
                    load6_f2(pc + 6, d2);
#pragma unroll
                    for (int e = 0; e < 6; ++e) {
                        vr[e] = sr[e] + beta * dr[e];
                        vc[e] = s2[e] + beta * d2[e];
                    }
                }
                float a[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, t[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int e9 = 0; e9 < 9; ++e9) {
                    const float e4[4] = {blk[e9].x, blk[e9].y, blk[e9].z, blk[e9].w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int e = 4 * e9 + j, r = e / 6, c = e % 6;
                        a[r] += e4[j] * vc[c];
                        t[c] += e4[j] * vr[r];
                    }
                }
                const bool diag = (w.x & kResDiag) != 0;
                if (w.y != kInvalidIndex) {
                    if (!contrib_shared || (kGrid && cr != rank)) {
                        store6_f2(A.contrib + 6ull * (R.low[cr] + w.y), t);
                    } else if (cr == rank) {
                        store6_f2(reinterpret_cast<float *>(res_smem + off_contrib + 24u * w.y), t);
                    } else if constexpr (!kGrid) {
                        const uint32_t ta = peer_addr(smem_base + off_contrib + 24u * w.y, cr);
                        st_peer2(ta, t[0], t[1]);
                        st_peer2(ta + 8u, t[2], t[3]);
                        st_peer2(ta + 16u, t[4], t[5]);
                    }
                }
                double dot = 0.0;
                if (A.fp64) {
#pragma unroll
                    for (int i = 0; i < 6; ++i) dot += (double)vr[i] * (double)a[i];
                    if (!diag) dot *= 2.0;
                } else {
                    float f = 0.f;
#pragma unroll
                    for (int i = 0; i < 6; ++i) f += vr[i] * a[i];
                    dot = (double)(diag ? f : 2.f * f);
                }
                float4 *o = reinterpret_cast<float4 *>(stage + 8u * k);
                o[0] = make_float4(a[0], a[1], a[2], a[3]);
                o[1] = make_float4(a[4], a[5], __int_as_float(__double2loint(dot)), __int_as_float(__double2hiint(dot)));
            }
            __syncthreads();
            // the row's products in item order, <d, A d> likewise: four records loaded at a time
            const uint32_t k1 = min(u_end, base + cnt);
            for (uint32_t k = max(u_begin, base); k < k1; k += 4) {
                float4 p0[4], p1[4];
#pragma unroll
                for (uint32_t e = 0; e < 4; ++e) {
                    const float4 *p = reinterpret_cast<const float4 *>(stage + 8u * (min(k + e, k1 - 1u) - base));
                    p0[e] = p[0];
                    p1[e] = p[1];
                }
#pragma unroll
                for (uint32_t e = 0; e < 4; ++e)
                    if (k + e < k1) {
                        q[0] += p0[e].x;
                        q[1] += p0[e].y;
                        q[2] += p0[e].z;
                        q[3] += p0[e].w;
                        q[4] += p1[e].x;
                        q[5] += p1[e].y;
                        dsum += __hiloint2double(__float_as_int(p1[e].w), __float_as_int(p1[e].z));
                    }
            }
            if (base + stage_items < items) __syncthreads();
        }
        if (row_warp) {
            if (has_row) {
                if (vec_shared) {
                    const float2 *pd = reinterpret_cast<const float2 *>(res_smem + off_d) + 3u * r;
#pragma unroll
                    for (int e = 0; e < 3; ++e) {
                        dv[2 * e] = pd[e].x;
                        dv[2 * e + 1] = pd[e].y;
                    }
                } else {
                    float s[6];
                    load6(sd_old + (size_t)kSdStride * row, s);
#pragma unroll
                    for (int c = 0; c < 6; ++c) dv[c] = s[c] + beta * dv[c];
                    store6_f2(sd_new + (size_t)kSdStride * row + 6, dv);
                }
            }
            publish(off_pa, A.fp64 ? group_sum(dsum) : (double)group_sum((float)dsum));
        }
        here = meet();
        if (!here) break;
        // ---- phase B: alpha; x += alpha d; r -= alpha q; s = M^-1 r; <r, s> ----
        if (warp == kScalarWarp) {
            const double dq = reduce(off_pa);
            double alpha64 = dq != 0.0 ? delta / dq : 0.0;
            if (!A.fp64 && dq != 0.0) alpha64 = (double)((float)delta / (float)dq);
            if (lane == 0) S.scalar[0] = (float)alpha64;
        }
        // the contributions do not need alpha: summed while the last warp takes it
        if (has_row) {
            if (contrib_shared) {
                const float2 *c = reinterpret_cast<const float2 *>(res_smem + off_contrib) + 3u * l_begin;
                uint32_t k0 = 0;
                if constexpr (kGrid) {   // the first `sends` entries come from other blocks, through L2
                    const float2 *g = reinterpret_cast<const float2 *>(A.contrib) + 3ull * (low0 + l_begin);
                    for (; k0 < sends; k0 += 4) {
                        float2 v[4][3];
#pragma unroll
                        for (uint32_t e = 0; e < 4; ++e)
#pragma unroll
                            for (uint32_t h = 0; h < 3; ++h) v[e][h] = __ldcg(g + 3u * min(k0 + e, sends - 1u) + h);
#pragma unroll
                        for (uint32_t e = 0; e < 4; ++e)
                            if (k0 + e < sends) {
#pragma unroll
                                for (uint32_t h = 0; h < 3; ++h) {
                                    q[2 * h] += v[e][h].x;
                                    q[2 * h + 1] += v[e][h].y;
                                }
                            }
                    }
                    k0 = sends;
                }
                for (uint32_t k = k0; k < l_count; k += 4) {
                    float2 v[4][3];
#pragma unroll
                    for (uint32_t e = 0; e < 4; ++e)
#pragma unroll
                        for (uint32_t h = 0; h < 3; ++h) v[e][h] = c[3u * min(k + e, l_count - 1u) + h];
#pragma unroll
                    for (uint32_t e = 0; e < 4; ++e)
                        if (k + e < l_count) {
#pragma unroll
                            for (uint32_t h = 0; h < 3; ++h) {
                                q[2 * h] += v[e][h].x;
                                q[2 * h + 1] += v[e][h].y;
                            }
                        }
                }
            } else {
                add_lower(A, row, q);
            }
        }
        __syncthreads();
        const bool more = it + 1 < A.pcg_iters;
        if (row_warp) {
            const float alpha = S.scalar[0];
            float s[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (has_row) {
#pragma unroll
                for (int c = 0; c < 6; ++c) {
                    xv[c] += alpha * dv[c];
                    rv[c] -= alpha * q[c];
                }
                if (more) {
                    precondition(rv, s);
                    store_s(s, sd_new);
                }
            }
            if (more) publish(off_pb, node_dot_group(A, rv, s, has_row));
        }
        if (more) {
            here = meet();
            if (!here) break;
            if (kGrid && vec_shared && tid < halo) load6(A.r + 8ull * send[tid], halo_s);
            if (warp == kScalarWarp) {
                const double v = reduce(off_pb);
                double beta64 = delta != 0.0 ? v / delta : 0.0;
                if (!A.fp64 && delta != 0.0) beta64 = (double)((float)v / (float)delta);
                delta = v;
                if (lane == 0) S.scalar[1] = (float)beta64;
            }
            __syncthreads();
            beta = S.scalar[1];
        }
    }
    if (!here) {   // no block leaves with copies on their way into its shared memory
        if (ring > 0 && tid == 0)
            for (uint32_t b = 0; b < ring; ++b)
                if (S.armed[b] > 0) bulk_wait_one(&S.ring[b], (S.armed[b] - 1u) & 1u);
        __syncthreads();
        return;
    }
    if (has_row) {
        store6(A.x + 8ull * row, xv);
        twist_update_row(A, row, xv);
    }
}

template <bool kGrid>
__global__ void __launch_bounds__(kResThreads, 1) k_pcg_cluster(PcgArgs A, ResPlan P, uint32_t smem_bytes) {
    __shared__ ResShared S;
    if (A.cost != nullptr && !resident_pays(A)) return;   // k_pcg runs
    if constexpr (kGrid) {
        // the widest of the scene's blocks decides for all of them
        if (48u * __ldg(P.vec + res_place<true>(A).scene) + kResMinLocal <= smem_bytes)
            pcg_resident<true, 1>(A, P, smem_bytes, S);
        else
            pcg_resident<true, 0>(A, P, smem_bytes, S);
    } else {
        pcg_resident<false, -1>(A, P, smem_bytes, S);
    }
}

}  // namespace ws
