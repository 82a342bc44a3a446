// C ABI of the B200 warp-field solver (include/warpsolve.h).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <vector>

#include "../../include/warpsolve.h"
#include "ws_common.cuh"
#include "ws_prims.cuh"
#include "ws_workspace.h"

struct ws_solver {
    ws::Workspace w;
};

namespace {

constexpr int kPixTile = 1024;

template <class T>
cudaError_t dalloc(T **p, size_t n) {
    *p = nullptr;
    if (n == 0) n = 1;
    return cudaMalloc(reinterpret_cast<void **>(p), n * sizeof(T));
}

// Solvers alive on a device (devices past the table share its last entry).
std::atomic<int> &live_solvers(int device) {
    static std::atomic<int> count[65];
    return count[device >= 0 && device < 64 ? device : 64];
}

void free_all(ws::Workspace &w) {
    void *ptrs[] = {w.scenes, w.plan, w.counts, w.tile_scene, w.tile_count, w.node_scene, w.edge_scene,
                    w.chunk_scene, w.chunk_row, w.scan_tmp, w.sort_hist, w.sort_digit, w.d_pixels, w.d_knn,
                    w.d_sw, w.d_cw, w.d_scene, w.d_record, w.r_record, w.n2t_key, w.n2t_val, w.n2t_key_alt,
                    w.n2t_val_alt, w.n2t_offset, w.row_pair_cols, w.row_pair_cnts, w.row_pair_first,
                    w.row_entry_first, w.pair_val, w.half_row, w.half_col, w.half_begin, w.half_end, w.half_scene, w.half_slot_up,
                    w.half_slot_lo, w.row_cnt_up, w.row_cnt_lo, w.row_first, w.rowptr, w.col_key, w.col_val,
                    w.col_key_alt, w.col_val_alt, w.colidx, w.item_ptr, w.item_info, w.item_col, w.sym_blocks, w.contrib, w.pcg_warp_groups, w.pcg_unit_info, w.pcg_words, w.pcg_send,
                    w.pcg_send_count, w.pcg_halo, w.pcg_vec, w.pcg_sync, w.mf_ux, w.inv_diag, w.diag64, w.jtr, w.x, w.r, w.q,
                    w.sd0, w.sd1, w.se3, w.centers, w.chunk_partial, w.scene_scalars,
                    w.error_flag};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    if (w.graph_exec) cudaGraphExecDestroy(w.graph_exec);
    if (w.h_tables) cudaFreeHost(w.h_tables);
    for (cudaEvent_t e : w.prof_events) cudaEventDestroy(e);
    if (w.tables_free) cudaEventDestroy(w.tables_free);
}

// Rigid inverse of a row-major 4x4 camera-to-world transform.  The reference
// inverts with Eigen's general 4x4 inverse (WarpSolver.cu:151-154); for a rigid
// transform both give [R^T | -R^T t] up to rounding.
void world_from_cam(const float *c2w, float *w2c) {
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) w2c[4 * i + j] = c2w[4 * j + i];
    for (int i = 0; i < 3; ++i)
        w2c[4 * i + 3] = -(w2c[4 * i] * c2w[3] + w2c[4 * i + 1] * c2w[7] + w2c[4 * i + 2] * c2w[11]);
}

int validate(const ws_inputs &in) {
    if (in.width <= 0 || in.height <= 0 || in.width > 65535 || in.height > 65535) return WS_ERR_INVALID_ARGUMENT;
    if (in.pitch != 0 && in.pitch < in.width) return WS_ERR_INVALID_ARGUMENT;
    if (!in.measure_vertex_confid || !in.measure_normal_radius || !in.reference_vertex || !in.reference_normal ||
        !in.index_map)
        return WS_ERR_INVALID_ARGUMENT;
    if (in.num_nodes <= 0 || in.num_nodes > 65535 || !in.reference_node_coords) return WS_ERR_INVALID_ARGUMENT;
    if (in.num_surfels < 0 || (in.num_surfels > 0 && (!in.surfel_knn || !in.surfel_knn_spatial_weight ||
                                                      !in.surfel_knn_connect_weight)))
        return WS_ERR_INVALID_ARGUMENT;
    if (in.num_edges < 0 || (in.num_edges > 0 && (!in.node_graph || !in.node_knn_connect_weight)))
        return WS_ERR_INVALID_ARGUMENT;
    if (in.num_edges > 0 && in.graph_k <= 0) return WS_ERR_INVALID_ARGUMENT;
    if (in.num_features < 0 || (in.num_features > 0 && !in.feature_knn)) return WS_ERR_INVALID_ARGUMENT;
    for (float v : {in.fx, in.fy, in.cx, in.cy, in.lambda_depth, in.lambda_optical_flow, in.lambda_reg,
                    in.lambda_node_translation, in.lambda_feature, in.node_radius_square})
        if (!std::isfinite(v)) return WS_ERR_INVALID_ARGUMENT;
    return WS_OK;
}

}  // namespace

extern "C" {

int ws_version(void) { return 1; }

const char *ws_error_string(int s) {
    switch (s) {
        case WS_OK: return "ok";
        case WS_ERR_INVALID_ARGUMENT: return "invalid argument";
        case WS_ERR_CAPACITY: return "input exceeds solver capacity";
        case WS_ERR_CUDA: return "CUDA runtime error";
        case WS_ERR_NAN: return "NaN in the right-hand side";
        case WS_ERR_TIMEOUT: return "bounded device wait timed out";
        case WS_ERR_NOT_READY: return "no inputs or no solution";
        case WS_ERR_NO_DEVICE: return "no CUDA device";
        default: return "unknown status";
    }
}

void ws_default_penalties(ws_inputs *in) {
    if (!in) return;
    in->lambda_depth = 0.1f;
    in->lambda_optical_flow = 0.0f;
    in->lambda_reg = 1.0f;
    in->lambda_node_translation = 0.0f;
    in->lambda_feature = 1.0f;
}

int ws_create(const ws_config *cfg, ws_solver **out) {
    if (!cfg || !out) return WS_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    if (cfg->max_scenes <= 0 || cfg->max_total_nodes <= 0 || cfg->max_total_pixels <= 0 || cfg->max_total_edges < 0 ||
        cfg->max_total_features < 0)
        return WS_ERR_INVALID_ARGUMENT;
    if (cfg->precision != WS_PREC_MIXED && cfg->precision != WS_PREC_FP32) return WS_ERR_INVALID_ARGUMENT;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= cfg->device || cfg->device < 0) {
        cudaGetLastError();
        return WS_ERR_NO_DEVICE;
    }
    if (cudaSetDevice(cfg->device) != cudaSuccess) return WS_ERR_CUDA;
    ws_solver *h = new (std::nothrow) ws_solver();
    if (!h) return WS_ERR_CAPACITY;
    ws::Workspace &w = h->w;
    w.device = cfg->device;
    w.precision = cfg->precision;
    cudaDeviceGetAttribute(&w.num_sms, cudaDevAttrMultiProcessorCount, w.device);
    w.cap_scenes = cfg->max_scenes;
    w.cap_nodes = (uint32_t)cfg->max_total_nodes;
    w.cap_pixels = (uint32_t)cfg->max_total_pixels;
    w.cap_edges = (uint32_t)cfg->max_total_edges;
    w.cap_features = (uint32_t)cfg->max_total_features;
    w.cap_tiles = w.cap_pixels / kPixTile + (uint32_t)w.cap_scenes + 1;
    w.cap_chunks = w.cap_nodes / ws::kRowsPerGroup + (uint32_t)w.cap_scenes + 1;
    w.cap_n2t = 4u * w.cap_pixels + 2u * w.cap_edges + w.cap_nodes + 4u * w.cap_features;
    w.cap_pair_kv = 6u * w.cap_pixels + w.cap_edges + 6u * w.cap_features;
    w.cap_half = std::min<uint32_t>(w.cap_pair_kv, 64u * w.cap_nodes);
    w.cap_half = std::min<uint32_t>(w.cap_half, (0xFFFFFFF0u - w.cap_nodes) / 2u);
    w.cap_blocks = w.cap_nodes + 2u * w.cap_half;
    w.cap_items = w.cap_nodes + w.cap_half;
    const int sort_tiles = std::max(ws::sort_max_tiles(w.cap_n2t), ws::sort_max_tiles(w.cap_half));
    const uint32_t scan_cap = std::max(w.cap_nodes, w.cap_tiles) + 1;
    cudaError_t e = cudaSuccess;
    auto A = [&](cudaError_t r) { if (e == cudaSuccess) e = r; };
    A(dalloc(&w.scenes, w.cap_scenes));
    A(dalloc(&w.plan, w.cap_scenes));
    A(dalloc(&w.counts, ws::kCounts));
    A(dalloc(&w.tile_scene, w.cap_tiles));
    A(dalloc(&w.tile_count, w.cap_tiles + 1));
    A(dalloc(&w.node_scene, w.cap_nodes));
    A(dalloc(&w.edge_scene, w.cap_edges));
    A(dalloc(&w.chunk_scene, w.cap_chunks));
    A(dalloc(&w.chunk_row, w.cap_chunks));
    A(dalloc(&w.scan_tmp, scan_cap / ws::kScanTile + 4));
    A(dalloc(&w.sort_hist, (size_t)ws::kSortMaxDigits * sort_tiles));
    A(dalloc(&w.sort_digit, ws::kSortMaxDigits));
    A(dalloc(&w.d_pixels, w.cap_pixels));
    A(dalloc(&w.d_knn, w.cap_pixels));
    A(dalloc(&w.d_sw, w.cap_pixels));
    A(dalloc(&w.d_cw, w.cap_pixels));
    A(dalloc(&w.d_scene, w.cap_pixels));
    A(dalloc(&w.d_record, (size_t)w.cap_pixels * ws::kDenseRecord));
    A(dalloc(&w.r_record, (size_t)std::max(1u, w.cap_edges) * ws::kRegRecord));
    A(dalloc(&w.n2t_key, w.cap_n2t));
    A(dalloc(&w.n2t_val, w.cap_n2t));
    A(dalloc(&w.n2t_key_alt, w.cap_n2t));
    A(dalloc(&w.n2t_val_alt, w.cap_n2t));
    A(dalloc(&w.n2t_offset, w.cap_nodes + 1));
    A(dalloc(&w.row_pair_cols, (size_t)w.cap_nodes * ws::kRowPairsMax));
    {   // counts of a row's warps: up to 8 or 4 a row where the rows are few (pair_row_warps)
        const uint32_t shares = std::max({w.cap_nodes, 4u * std::min(w.cap_nodes, ws::kRowWide4),
                                          8u * std::min(w.cap_nodes, ws::kRowWide8)});
        A(dalloc(&w.row_pair_cnts, (size_t)shares * ws::kRowPairsMax));
    }
    A(dalloc(&w.row_pair_first, w.cap_nodes + 1));
    A(dalloc(&w.row_entry_first, w.cap_nodes + 1));
    A(dalloc(&w.pair_val, w.cap_pair_kv));
    A(dalloc(&w.half_row, w.cap_half));
    A(dalloc(&w.half_col, w.cap_half));
    A(dalloc(&w.half_begin, w.cap_half));
    A(dalloc(&w.half_end, w.cap_half));
    A(dalloc(&w.half_scene, w.cap_half));
    A(dalloc(&w.half_slot_up, w.cap_half));
    A(dalloc(&w.half_slot_lo, w.cap_half));
    A(dalloc(&w.row_cnt_up, w.cap_nodes));
    A(dalloc(&w.row_cnt_lo, w.cap_nodes));
    A(dalloc(&w.row_first, w.cap_nodes));
    A(dalloc(&w.rowptr, w.cap_nodes + 1));
    A(dalloc(&w.col_key, w.cap_half));
    A(dalloc(&w.col_val, w.cap_half));
    A(dalloc(&w.col_key_alt, w.cap_half));
    A(dalloc(&w.col_val_alt, w.cap_half));
    A(dalloc(&w.colidx, w.cap_blocks));
    A(dalloc(&w.item_ptr, (size_t)w.cap_nodes + 1));
    A(dalloc(&w.item_info, w.cap_items));
    A(dalloc(&w.item_col, w.cap_items));
    A(dalloc(&w.sym_blocks, (size_t)w.cap_items * 36));
    A(dalloc(&w.contrib, (size_t)std::max<uint32_t>(1u, w.cap_half) * 6));
    A(dalloc(&w.inv_diag, (size_t)w.cap_nodes * 36));
    A(dalloc(&w.diag64, (size_t)w.cap_nodes * 21));
    for (float **v : {&w.jtr, &w.x, &w.r, &w.q}) A(dalloc(v, (size_t)w.cap_nodes * ws::kVecStride));
    for (float **v : {&w.sd0, &w.sd1}) A(dalloc(v, (size_t)w.cap_nodes * ws::kSdStride));
    A(dalloc(&w.se3, (size_t)w.cap_nodes * 8));
    A(dalloc(&w.centers, w.cap_nodes));
    A(dalloc(&w.chunk_partial, 2 * (size_t)w.cap_chunks));
    A(dalloc(&w.scene_scalars, 8ull * w.cap_scenes));
    A(dalloc(&w.pcg_sync, 64ull * (1 + w.cap_scenes)));
    w.pcg_tickets = w.pcg_sync;
    w.scene_counter = w.pcg_sync ? w.pcg_sync + 64 : nullptr;
    A(dalloc(&w.error_flag, 4));
    w.h_tables_bytes = sizeof(ws::Scene) * w.cap_scenes + 4ull * (w.cap_tiles + w.cap_nodes + w.cap_edges + 2ull * w.cap_chunks);
    A(cudaMallocHost(&w.h_tables, w.h_tables_bytes));
    A(cudaEventCreateWithFlags(&w.tables_free, cudaEventDisableTiming));
    if (e == cudaSuccess) {
        A(cudaMemset(w.error_flag, 0, 4 * sizeof(int)));
        A(cudaMemset(w.counts, 0, ws::kCounts * sizeof(uint32_t)));
        A(cudaMemset(w.pcg_sync, 0, 64ull * (1 + w.cap_scenes) * sizeof(uint32_t)));
        A(cudaMemset(w.se3, 0, (size_t)w.cap_nodes * 8 * sizeof(float)));
    }
    if (e == cudaSuccess) {
        w.pcg_grid = ws::pcg_max_blocks(w.device);
        A(dalloc(&w.pcg_warp_groups, (size_t)ws::kPcgUnitsPerWarp * w.pcg_grid * ws::pcg_warps_per_block() + 2));
        A(dalloc(&w.pcg_unit_info, 2 * (size_t)ws::kPcgUnitsPerWarp * w.pcg_grid * ws::pcg_warps_per_block()));
        w.pcg_cluster = ws::pcg_cluster_max(&w.pcg_clusters_active);
        A(dalloc(&w.pcg_words, w.cap_items));
        A(dalloc(&w.pcg_send, w.cap_items));
        A(dalloc(&w.pcg_send_count, w.cap_nodes));
        A(dalloc(&w.pcg_halo, 16ull * w.cap_scenes + 160));   // kResMaxCluster a scene, or kResMaxBlocks
        A(dalloc(&w.pcg_vec, w.cap_scenes));
        w.pcg_grid_most = ws::pcg_grid_max(w.device);
        w.pcg_smem = ws::pcg_smem_max();
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        free_all(w);
        delete h;
        return e == cudaErrorMemoryAllocation ? WS_ERR_CAPACITY : WS_ERR_CUDA;
    }
    live_solvers(w.device).fetch_add(1);
    *out = h;
    return WS_OK;
}

int ws_destroy(ws_solver *h) {
    if (!h) return WS_ERR_INVALID_ARGUMENT;
    const int device = h->w.device;
    cudaSetDevice(device);
    if (h->w.last_stream) cudaStreamSynchronize(h->w.last_stream);
    free_all(h->w);
    delete h;
    if (live_solvers(device).fetch_sub(1) == 1) ws::scratch_trim(device);
    return WS_OK;
}

int ws_set_batch(ws_solver *h, const ws_inputs *scenes, int num_scenes) {
    if (!h || !scenes || num_scenes <= 0) return WS_ERR_INVALID_ARGUMENT;
    ws::Workspace &w = h->w;
    if (num_scenes > w.cap_scenes) return WS_ERR_CAPACITY;
    uint64_t nodes = 0, edges = 0, pixels = 0, feats = 0, tiles = 0, chunks = 0;
    for (int s = 0; s < num_scenes; ++s) {
        const int st = validate(scenes[s]);
        if (st != WS_OK) return st;
        nodes += (uint64_t)scenes[s].num_nodes;
        edges += (uint64_t)scenes[s].num_edges;
        feats += (uint64_t)scenes[s].num_features;
        pixels += (uint64_t)scenes[s].width * scenes[s].height;
        tiles += ((uint64_t)scenes[s].width * scenes[s].height + kPixTile - 1) / kPixTile;
        chunks += ((uint64_t)scenes[s].num_nodes + ws::kRowsPerGroup - 1) / ws::kRowsPerGroup;
    }
    if (nodes > w.cap_nodes || edges > w.cap_edges || pixels > w.cap_pixels || feats > w.cap_features ||
        tiles > w.cap_tiles || chunks > w.cap_chunks)
        return WS_ERR_CAPACITY;
    // host tables, uploaded by the next solve from pinned memory
    // the previous solve may still be copying these pinned tables to the device
    if (w.tables_in_flight) {
        cudaSetDevice(w.device);
        if (cudaEventSynchronize(w.tables_free) != cudaSuccess) return WS_ERR_CUDA;
        w.tables_in_flight = false;
    }
    ws::Scene *hs = reinterpret_cast<ws::Scene *>(w.h_tables);
    uint32_t *tile_scene = reinterpret_cast<uint32_t *>(hs + w.cap_scenes);
    uint32_t *node_scene = tile_scene + w.cap_tiles;
    uint32_t *edge_scene = node_scene + w.cap_nodes;
    uint32_t *chunk_scene = edge_scene + w.cap_edges;
    uint32_t *chunk_row = chunk_scene + w.cap_chunks;
    w.init_ptrs.assign(num_scenes, nullptr);
    uint32_t nb = 0, eb = 0, fb = 0, tb = 0, cb = 0;
    for (int s = 0; s < num_scenes; ++s) {
        const ws_inputs &in = scenes[s];
        ws::Scene sc;
        std::memset(&sc, 0, sizeof(sc));
        sc.width = in.width;
        sc.height = in.height;
        sc.pitch = in.pitch ? in.pitch : in.width;
        sc.fx = in.fx; sc.fy = in.fy; sc.cx = in.cx; sc.cy = in.cy;
        world_from_cam(in.cam2world, sc.w2c);
        sc.mvert = static_cast<const float4 *>(in.measure_vertex_confid);
        sc.mnorm = static_cast<const float4 *>(in.measure_normal_radius);
        sc.rvert = static_cast<const float4 *>(in.reference_vertex);
        sc.rnorm = static_cast<const float4 *>(in.reference_normal);
        sc.index_map = in.index_map;
        sc.flow = static_cast<const float2 *>(in.opticalflow);
        sc.surfel_knn = reinterpret_cast<const ushort4 *>(in.surfel_knn);
        sc.surfel_sw = reinterpret_cast<const float4 *>(in.surfel_knn_spatial_weight);
        sc.surfel_cw = reinterpret_cast<const float4 *>(in.surfel_knn_connect_weight);
        sc.num_surfels = in.num_surfels;
        sc.num_nodes = in.num_nodes;
        sc.node_base = (int)nb;
        sc.num_edges = in.num_edges;
        sc.edge_base = (int)eb;
        sc.edges = in.node_graph;
        sc.node_cw = in.node_knn_connect_weight;
        sc.graph_k = in.graph_k;
        sc.node_r2 = in.node_radius_square;
        sc.node_coords = reinterpret_cast<const float4 *>(in.reference_node_coords);
        sc.node_motion = reinterpret_cast<const float4 *>(in.node_motion_pred);
        sc.num_features = in.num_features;
        sc.feature_base = (int)fb;
        sc.feature_knn = reinterpret_cast<const ushort4 *>(in.feature_knn);
        sc.lam_depth = in.lambda_depth;
        sc.lam_of = in.lambda_optical_flow;
        sc.lam_reg = in.lambda_reg;
        sc.lam_node = in.lambda_node_translation;
        sc.lam_feat = in.lambda_feature;
        const uint32_t nt = (uint32_t)(((uint64_t)in.width * in.height + kPixTile - 1) / kPixTile);
        sc.tile_base = (int)tb;
        sc.num_tiles = (int)nt;
        const uint32_t nc = ((uint32_t)in.num_nodes + ws::kRowsPerGroup - 1) / ws::kRowsPerGroup;
        sc.chunk_base = (int)cb;
        sc.num_chunks = (int)nc;
        for (uint32_t t = 0; t < nt; ++t) tile_scene[tb + t] = (uint32_t)s;
        for (int n = 0; n < in.num_nodes; ++n) node_scene[nb + n] = (uint32_t)s;
        for (int e = 0; e < in.num_edges; ++e) edge_scene[eb + e] = (uint32_t)s;
        for (uint32_t c = 0; c < nc; ++c) {
            chunk_scene[cb + c] = (uint32_t)s;
            chunk_row[cb + c] = nb + (uint32_t)ws::kRowsPerGroup * c;
        }
        hs[s] = sc;
        w.init_ptrs[s] = in.init_node_se3;
        nb += in.num_nodes;
        eb += in.num_edges;
        fb += in.num_features;
        tb += nt;
        cb += nc;
    }
    {
        // k_pcg_cluster starts the batch's largest scenes first
        std::vector<int> order(num_scenes);
        for (int s = 0; s < num_scenes; ++s) order[s] = s;
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return hs[a].num_nodes > hs[b].num_nodes; });
        for (int s = 0; s < num_scenes; ++s) hs[s].pcg_order = order[s];
    }
    w.pcg_grid_blocks = ws::pcg_grid_blocks(hs, num_scenes, w.pcg_grid_most);
    w.h_scenes.assign(hs, hs + num_scenes);
    w.num_scenes = num_scenes;
    w.dense_channels = 1;
    for (int s = 0; s < num_scenes; ++s)
        if (hs[s].lam_of != 0.0f) w.dense_channels = 3;
    w.total_nodes = nb;
    w.total_edges = eb;
    w.total_features = fb;
    w.total_tiles = tb;
    w.total_chunks = cb;
    w.node_bits = ws::bits_for(nb);
    w.have_inputs = true;
    w.have_solution = false;
    return WS_OK;
}

int ws_set_inputs(ws_solver *h, const ws_inputs *in) { return ws_set_batch(h, in, 1); }

}  // extern "C"

namespace {

bool capturing(cudaStream_t st) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (st && cudaStreamIsCapturing(st, &cs) == cudaSuccess) return cs != cudaStreamCaptureStatusNone;
    return false;
}

// Uploads the scene tables, initialises the warp, builds the index and runs the GN loop.
cudaError_t enqueue_solve(ws::Workspace &w, int gn, int pcg, cudaStream_t st) {
    const ws::Scene *hs = reinterpret_cast<const ws::Scene *>(w.h_tables);
    const uint32_t *tile_scene = reinterpret_cast<const uint32_t *>(hs + w.cap_scenes);
    const uint32_t *node_scene = tile_scene + w.cap_tiles;
    const uint32_t *edge_scene = node_scene + w.cap_nodes;
    const uint32_t *chunk_scene = edge_scene + w.cap_edges;
    const uint32_t *chunk_row = chunk_scene + w.cap_chunks;
    cudaError_t e = cudaSuccess;
    auto A = [&](cudaError_t r) { if (e == cudaSuccess) e = r; };
    A(cudaMemcpyAsync(w.scenes, hs, sizeof(ws::Scene) * w.num_scenes, cudaMemcpyHostToDevice, st));
    A(cudaMemcpyAsync(w.tile_scene, tile_scene, 4ull * w.total_tiles, cudaMemcpyHostToDevice, st));
    A(cudaMemcpyAsync(w.node_scene, node_scene, 4ull * w.total_nodes, cudaMemcpyHostToDevice, st));
    if (w.total_edges) A(cudaMemcpyAsync(w.edge_scene, edge_scene, 4ull * w.total_edges, cudaMemcpyHostToDevice, st));
    A(cudaMemcpyAsync(w.chunk_scene, chunk_scene, 4ull * w.total_chunks, cudaMemcpyHostToDevice, st));
    A(cudaMemcpyAsync(w.chunk_row, chunk_row, 4ull * w.total_chunks, cudaMemcpyHostToDevice, st));
    if (e != cudaSuccess) return e;
    if (!capturing(st)) {
        A(cudaEventRecord(w.tables_free, st));
        w.tables_in_flight = true;
    }
    const bool prof = w.profiling && !capturing(st);
    size_t ev = 0;
    auto mark = [&](int phase) {
        if (!prof) return;
        if (ev >= w.prof_events.size()) {
            cudaEvent_t x;
            cudaEventCreate(&x);
            w.prof_events.push_back(x);
        }
        cudaEventRecord(w.prof_events[ev], st);
        if (ev >= w.prof_phase.size()) {
            w.prof_phase.push_back(phase);
            w.prof_launches.push_back(w.launches);
        } else {
            w.prof_phase[ev] = phase;
            w.prof_launches[ev] = w.launches;
        }
        ++ev;
        w.launches = 0;
    };
    w.launches = 0;
    mark(-1);
    ws::init_warp(w, st);
    for (int s = 0; s < w.num_scenes; ++s)
        if (w.init_ptrs[s])
            A(cudaMemcpyAsync(w.se3 + 8ull * w.h_scenes[s].node_base, w.init_ptrs[s],
                              32ull * w.h_scenes[s].num_nodes, cudaMemcpyDeviceToDevice, st));
    A(ws::index_build(w, st));
    mark(0);
    for (int it = 0; it < gn && e == cudaSuccess; ++it) {
        ws::gn_eval(w, st);
        mark(1);
        ws::gn_assemble_node(w, st);
        mark(2);
        ws::gn_assemble_pair(w, st);
        mark(3);
        A(ws::gn_pcg(w, pcg, st));
        mark(4);
    }
    w.prof_count = prof ? (int)ev : 0;
    A(cudaGetLastError());
    return e;
}

}  // namespace

extern "C" {

int ws_solve(ws_solver *h, int gn_iters, int pcg_iters, void *stream) {
    if (!h || gn_iters < 0 || pcg_iters < 0) return WS_ERR_INVALID_ARGUMENT;
    ws::Workspace &w = h->w;
    if (!w.have_inputs) return WS_ERR_NOT_READY;
    cudaSetDevice(w.device);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    w.last_stream = st;
    const cudaError_t e = enqueue_solve(w, gn_iters, pcg_iters, st);
    if (e != cudaSuccess) return WS_ERR_CUDA;
    w.have_solution = true;
    return WS_OK;
}

int ws_solve_graph(ws_solver *h, int gn_iters, int pcg_iters, void *stream) {
    if (!h || gn_iters < 0 || pcg_iters < 0) return WS_ERR_INVALID_ARGUMENT;
    ws::Workspace &w = h->w;
    if (!w.have_inputs) return WS_ERR_NOT_READY;
    cudaSetDevice(w.device);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (!st) return WS_ERR_INVALID_ARGUMENT;   // the legacy stream cannot be captured
    w.last_stream = st;
    const ws::PcgChoice choice = ws::pcg_choice(w);
    const uint64_t key[] = {(uint64_t)gn_iters, (uint64_t)pcg_iters, (uint64_t)w.num_scenes, w.total_nodes,
                            w.total_edges, w.total_tiles, w.total_chunks, (uint64_t)w.node_bits,
                            (uint64_t)w.dense_channels, (uint64_t)ws::pcg_split_group(w),
                            (uint64_t)choice.mode, (uint64_t)choice.sure, (uint64_t)choice.rounds,
                            (uint64_t)w.pcg_grid_blocks, w.pcg_smem};
    constexpr size_t kKey = sizeof(key) / sizeof(key[0]);
    bool same = w.graph_exec && w.graph_key.size() == kKey && std::equal(key, key + kKey, w.graph_key.begin());
    if (same) {
        // device pointers of the inputs live in the uploaded tables, so a replay picks up new inputs;
        // the initial-warp copies are graph nodes with fixed sources, so they must match too
        same = (w.graph_init == w.init_ptrs);
    }
    if (!same) {
        if (w.graph_exec) {
            cudaGraphExecDestroy(w.graph_exec);
            w.graph_exec = nullptr;
        }
        cudaGraph_t g = nullptr;
        if (cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) != cudaSuccess) return WS_ERR_CUDA;
        const cudaError_t e1 = enqueue_solve(w, gn_iters, pcg_iters, st);
        const cudaError_t e2 = cudaStreamEndCapture(st, &g);
        if (e1 != cudaSuccess || e2 != cudaSuccess || !g) {
            if (g) cudaGraphDestroy(g);
            cudaGetLastError();
            return WS_ERR_CUDA;
        }
        size_t nn = 0;
        cudaGraphGetNodes(g, nullptr, &nn);
        std::vector<cudaGraphNode_t> nodes(nn);
        if (nn) cudaGraphGetNodes(g, nodes.data(), &nn);
        int kernels = 0;
        for (auto nd : nodes) {
            cudaGraphNodeType t;
            if (cudaGraphNodeGetType(nd, &t) == cudaSuccess && t == cudaGraphNodeTypeKernel) ++kernels;
        }
        w.graph_kernels = kernels;
        const cudaError_t e3 = cudaGraphInstantiate(&w.graph_exec, g, 0);
        cudaGraphDestroy(g);
        if (e3 != cudaSuccess) {
            w.graph_exec = nullptr;
            cudaGetLastError();
            return WS_ERR_CUDA;
        }
        w.graph_key.assign(key, key + kKey);
        w.graph_init = w.init_ptrs;
    }
    if (cudaGraphLaunch(w.graph_exec, st) != cudaSuccess) return WS_ERR_CUDA;
    // the replay's first nodes copy the pinned tables; the tables are free once the replay ends
    if (cudaEventRecord(w.tables_free, st) != cudaSuccess) return WS_ERR_CUDA;
    w.tables_in_flight = true;
    w.have_solution = true;
    return WS_OK;
}

int ws_set_profiling(ws_solver *h, int enable) {
    if (!h) return WS_ERR_INVALID_ARGUMENT;
    h->w.profiling = enable != 0;
    return WS_OK;
}

int ws_get_phase_times(ws_solver *h, float *ms, int *launches, int cap, int *count) {
    if (!h || !count) return WS_ERR_INVALID_ARGUMENT;
    ws::Workspace &w = h->w;
    *count = ws::Workspace::kPhases;
    if (w.prof_count < 2) return WS_ERR_NOT_READY;
    if (cap < ws::Workspace::kPhases) return WS_ERR_CAPACITY;
    cudaSetDevice(w.device);
    if (cudaEventSynchronize(w.prof_events[w.prof_count - 1]) != cudaSuccess) return WS_ERR_CUDA;
    for (int p = 0; p < ws::Workspace::kPhases; ++p) {
        if (ms) ms[p] = 0.f;
        if (launches) launches[p] = 0;
    }
    for (int i = 1; i < w.prof_count; ++i) {
        float t = 0.f;
        if (cudaEventElapsedTime(&t, w.prof_events[i - 1], w.prof_events[i]) != cudaSuccess) return WS_ERR_CUDA;
        const int p = w.prof_phase[i];
        if (p >= 0 && p < ws::Workspace::kPhases) {
            if (ms) ms[p] += t;
            if (launches) launches[p] += w.prof_launches[i];
        }
    }
    return WS_OK;
}

int ws_graph_kernel_count(ws_solver *h, int *count) {
    if (!h || !count) return WS_ERR_INVALID_ARGUMENT;
    *count = h->w.graph_kernels;
    return h->w.graph_exec ? WS_OK : WS_ERR_NOT_READY;
}

int ws_sync_status(ws_solver *h) {
    if (!h) return WS_ERR_INVALID_ARGUMENT;
    ws::Workspace &w = h->w;
    cudaSetDevice(w.device);
    if (cudaStreamSynchronize(w.last_stream) != cudaSuccess) {
        cudaGetLastError();
        return WS_ERR_CUDA;
    }
    int flag = 0;
    if (cudaMemcpy(&flag, w.error_flag, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return WS_ERR_CUDA;
    if (flag != 0) cudaMemset(w.error_flag, 0, sizeof(int));
    return flag;
}

int ws_spmv(ws_solver *h, const float *x, float *y, void *stream) {
    if (!h || !x || !y) return WS_ERR_INVALID_ARGUMENT;
    ws::Workspace &w = h->w;
    if (!w.have_solution) return WS_ERR_NOT_READY;
    cudaSetDevice(w.device);
    return ws::gn_spmv(w, x, y, (cudaStream_t)stream) == cudaSuccess ? WS_OK : WS_ERR_CUDA;
}

int ws_selftest_wait_timeout(void *stream) {
    int status = 0;
    if (ws::pcg_wait_selftest(&status, (cudaStream_t)stream) != cudaSuccess) return WS_ERR_CUDA;
    return status == 0 ? WS_OK : status;
}

int ws_selftest_resident_timeout(ws_solver *h, void *stream) {
    if (!h) return WS_ERR_INVALID_ARGUMENT;
    ws::Workspace &w = h->w;
    if (!w.have_solution) return WS_ERR_NOT_READY;
    cudaSetDevice(w.device);
    int status = 0;
    if (w.last_stream) cudaStreamSynchronize(w.last_stream);
    if (ws::pcg_resident_selftest(w, &status, (cudaStream_t)stream) != cudaSuccess) {
        cudaGetLastError();
        return WS_ERR_CUDA;
    }
    if (status != WS_ERR_NOT_READY) w.have_solution = false;   // some scenes' warps were updated, others not
    return status;
}

int ws_selftest_grid_barrier_timeout(void *stream) {
    int flags = 0;
    if (ws::dedup_wait_selftest(&flags, (cudaStream_t)stream) != cudaSuccess) return WS_ERR_CUDA;
    return (flags & 4) ? WS_ERR_TIMEOUT : WS_OK;
}

int ws_spmv_matrix_free(ws_solver *h, const float *x, float *y, void *stream) {
    if (!h || !x || !y) return WS_ERR_INVALID_ARGUMENT;
    ws::Workspace &w = h->w;
    if (!w.have_solution) return WS_ERR_NOT_READY;
    cudaSetDevice(w.device);
    const size_t n4 = (size_t)w.cap_pixels + (size_t)w.cap_edges;
    if (!w.mf_ux && cudaMalloc(&w.mf_ux, 16 * std::max<size_t>(1, n4)) != cudaSuccess) {
        cudaGetLastError();
        w.mf_ux = nullptr;
        return WS_ERR_CAPACITY;
    }
    return ws::gn_spmv_matrix_free(w, x, y, w.mf_ux, w.mf_ux + 4ull * w.cap_pixels, (cudaStream_t)stream) ==
                   cudaSuccess
               ? WS_OK
               : WS_ERR_CUDA;
}

static void drop_graph(ws::Workspace &w) {
    if (w.graph_exec) cudaGraphExecDestroy(w.graph_exec);
    w.graph_exec = nullptr;
}

int ws_set_tuning(ws_solver *h, const ws_tuning *t) {
    if (!h || !t) return WS_ERR_INVALID_ARGUMENT;
    auto ok_nt = [](int v) { return v == 64 || v == 128 || v == 256; };
    if (!ok_nt(t->node_threads) || !ok_nt(t->pair_threads) || t->pcg_blocks_per_sm < 1) return WS_ERR_INVALID_ARGUMENT;
    ws::Workspace &w = h->w;
    w.tune.node_threads = t->node_threads;
    w.tune.pair_threads = t->pair_threads;
    w.tune.pcg_blocks_per_sm = t->pcg_blocks_per_sm;
    w.tune.tuned = true;
    drop_graph(w);
    return WS_OK;
}

int ws_set_pcg_form(ws_solver *h, int form, int shared_bytes) {
    if (!h || form < WS_PCG_AUTO || form > WS_PCG_GRID) return WS_ERR_INVALID_ARGUMENT;
    if (shared_bytes != 0 && (shared_bytes < (int)ws::pcg_smem_min() || shared_bytes > (int)ws::pcg_smem_max()))
        return WS_ERR_INVALID_ARGUMENT;
    h->w.pcg_form = form;
    h->w.pcg_smem = shared_bytes == 0 ? ws::pcg_smem_max() : (uint32_t)shared_bytes & ~127u;
    return WS_OK;
}

int ws_get_pcg_form(ws_solver *h, int *form) {
    if (!h || !form) return WS_ERR_INVALID_ARGUMENT;
    if (!h->w.have_inputs) return WS_ERR_NOT_READY;
    *form = (int)(h->w.have_solution ? ws::pcg_ran(h->w) : ws::pcg_choice(h->w).mode);
    return WS_OK;
}

int ws_autotune(ws_solver *h, int pcg_iters, void *stream, ws_tuning *out) {
    if (!h || !out || pcg_iters < 1) return WS_ERR_INVALID_ARGUMENT;
    ws::Workspace &w = h->w;
    if (w.num_scenes <= 0) return WS_ERR_NOT_READY;
    cudaSetDevice(w.device);
    cudaStream_t st = (cudaStream_t)stream;
    std::memset(out, 0, sizeof(*out));
    for (float &x : out->node_ms) x = -1.f;
    for (float &x : out->pair_ms) x = -1.f;
    for (float &x : out->pcg_ms) x = -1.f;
    if (w.tables_in_flight) cudaEventSynchronize(w.tables_free);
    // one Gauss-Newton iteration gives real records and a real matrix to time on
    if (enqueue_solve(w, 1, pcg_iters, st) != cudaSuccess) return WS_ERR_CUDA;
    ws::gn_eval(w, st);
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    auto time_ms = [&](auto &&run) {
        run();   // warm-up
        float best = 1e30f;
        for (int rep = 0; rep < 3; ++rep) {
            cudaEventRecord(e0, st);
            run();
            cudaEventRecord(e1, st);
            cudaEventSynchronize(e1);
            float ms = 0.f;
            cudaEventElapsedTime(&ms, e0, e1);
            best = std::min(best, ms);
        }
        return best;
    };
    const int nts[3] = {64, 128, 256};
    const bool fp64 = w.precision == WS_PREC_MIXED;
    int best_node = 128, best_pair = 128;
    float bn = 1e30f, bp = 1e30f;
    for (int i = 0; i < 3; ++i) {
        if (!(fp64 && nts[i] == 256)) {
            w.tune.node_threads = nts[i];
            out->node_ms[i] = time_ms([&] { ws::gn_assemble_node(w, st); });
            if (out->node_ms[i] < bn) { bn = out->node_ms[i]; best_node = nts[i]; }
        }
        w.tune.pair_threads = nts[i];
        out->pair_ms[i] = time_ms([&] { ws::gn_assemble_pair(w, st); });
        if (out->pair_ms[i] < bp) { bp = out->pair_ms[i]; best_pair = nts[i]; }
    }
    w.tune.node_threads = best_node;
    w.tune.pair_threads = best_pair;
    ws::gn_assemble_node(w, st);
    ws::gn_assemble_pair(w, st);
    const int max_per_sm = std::max(1, std::min(8, w.pcg_grid / std::max(1, w.num_sms)));
    int best_b = max_per_sm;
    float bb = 1e30f;
    // blocks per SM of k_pcg, also where these inputs run resident: later inputs may not
    const int form = w.pcg_form;
    w.pcg_form = WS_PCG_STREAMED;
    for (int b = 1; b <= max_per_sm; ++b) {
        w.tune.pcg_blocks_per_sm = b;
        ws::pcg_ranges(w, st);
        out->pcg_ms[b - 1] = time_ms([&] { ws::gn_pcg(w, pcg_iters, st); });
        if (out->pcg_ms[b - 1] < bb) { bb = out->pcg_ms[b - 1]; best_b = b; }
    }
    w.pcg_form = form;
    w.tune.pcg_blocks_per_sm = best_b;
    w.tune.tuned = true;
    ws::pcg_ranges(w, st);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    drop_graph(w);
    out->node_threads = best_node;
    out->pair_threads = best_pair;
    out->pcg_blocks_per_sm = best_b;
    const int status = ws_sync_status(h);
    return status != WS_OK ? status : (cudaGetLastError() == cudaSuccess ? WS_OK : WS_ERR_CUDA);
}

int ws_get_solution(ws_solver *h, int scene, const float **dev, int *num_nodes) {
    if (!h || !dev || !num_nodes) return WS_ERR_INVALID_ARGUMENT;
    ws::Workspace &w = h->w;
    if (!w.have_solution) return WS_ERR_NOT_READY;
    if (scene < 0 || scene >= w.num_scenes) return WS_ERR_INVALID_ARGUMENT;
    *dev = w.se3 + 8ull * w.h_scenes[scene].node_base;
    *num_nodes = w.h_scenes[scene].num_nodes;
    return WS_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Host copies of the index structures and the assembled system (parity tests).
// ---------------------------------------------------------------------------
namespace {

template <class T>
std::vector<T> download(const T *p, size_t n) {
    std::vector<T> v(n);
    if (n) cudaMemcpy(v.data(), p, n * sizeof(T), cudaMemcpyDeviceToHost);
    return v;
}

int sync_for_debug(ws::Workspace &w, int scene) {
    if (!w.have_solution) return WS_ERR_NOT_READY;
    if (scene < 0 || scene >= w.num_scenes) return WS_ERR_INVALID_ARGUMENT;
    cudaSetDevice(w.device);
    if (cudaStreamSynchronize(w.last_stream) != cudaSuccess) return WS_ERR_CUDA;
    return WS_OK;
}

void plan_of(ws::Workspace &w, int scene, ws::Plan &p) {
    cudaMemcpy(&p, w.plan + scene, sizeof(p), cudaMemcpyDeviceToHost);
}

// Range [first, last) of unique pairs whose row lies in `scene`.
void half_range(ws::Workspace &w, int scene, uint32_t &first, uint32_t &last, std::vector<uint32_t> &rows) {
    uint32_t counts[8];
    cudaMemcpy(counts, w.counts, sizeof(counts), cudaMemcpyDeviceToHost);
    rows = download(w.half_row, counts[ws::kCntHalf]);
    const uint32_t b = (uint32_t)w.h_scenes[scene].node_base, e = b + (uint32_t)w.h_scenes[scene].num_nodes;
    first = (uint32_t)(std::lower_bound(rows.begin(), rows.end(), b) - rows.begin());
    last = (uint32_t)(std::lower_bound(rows.begin(), rows.end(), e) - rows.begin());
}

}  // namespace

extern "C" {

int ws_get_counts(ws_solver *h, int scene, int *nd, int *nhalf, int *nkv) {
    if (!h) return WS_ERR_INVALID_ARGUMENT;
    ws::Workspace &w = h->w;
    const int st = sync_for_debug(w, scene);
    if (st != WS_OK) return st;
    ws::Plan p;
    plan_of(w, scene, p);
    if (nd) *nd = (int)p.dense_count;
    if (nkv) *nkv = (int)p.n2t_count;
    if (nhalf) {
        uint32_t f, l;
        std::vector<uint32_t> rows;
        half_range(w, scene, f, l, rows);
        *nhalf = (int)(l - f);
    }
    return WS_OK;
}

int ws_get_dense_terms(ws_solver *h, int scene, uint16_t *pixels, uint16_t *knn, float *sw, float *cw, int cap,
                       int *count) {
    if (!h || !count) return WS_ERR_INVALID_ARGUMENT;
    ws::Workspace &w = h->w;
    const int st = sync_for_debug(w, scene);
    if (st != WS_OK) return st;
    ws::Plan p;
    plan_of(w, scene, p);
    *count = (int)p.dense_count;
    if ((int)p.dense_count > cap) return WS_ERR_CAPACITY;
    if (pixels) cudaMemcpy(pixels, w.d_pixels + p.dense_begin, 8ull * p.dense_count, cudaMemcpyDeviceToHost);
    if (knn) cudaMemcpy(knn, w.d_knn + p.dense_begin, 8ull * p.dense_count, cudaMemcpyDeviceToHost);
    if (sw) cudaMemcpy(sw, w.d_sw + p.dense_begin, 16ull * p.dense_count, cudaMemcpyDeviceToHost);
    if (cw) cudaMemcpy(cw, w.d_cw + p.dense_begin, 16ull * p.dense_count, cudaMemcpyDeviceToHost);
    return cudaGetLastError() == cudaSuccess ? WS_OK : WS_ERR_CUDA;
}

int ws_get_dense_jacobian(ws_solver *h, int scene, float *residual, float *gradient, int cap, int *count) {
    if (!h || !count) return WS_ERR_INVALID_ARGUMENT;
    ws::Workspace &w = h->w;
    const int st = sync_for_debug(w, scene);
    if (st != WS_OK) return st;
    ws::Plan p;
    plan_of(w, scene, p);
    *count = (int)p.dense_count;
    if ((int)p.dense_count > cap) return WS_ERR_CAPACITY;
    // records of a batch without the flow term hold the depth channel only; the flow
    // channels read back as zero
    const int ch = w.dense_channels;
    const size_t stride = ch == 3 ? ws::DenseLayout<3>::kFloats : ws::DenseLayout<1>::kFloats;
    const auto rec = download(w.d_record + stride * p.dense_begin, stride * p.dense_count);
    for (uint32_t t = 0; t < p.dense_count; ++t) {
        const float *r = rec.data() + stride * t;
        if (gradient) {
            std::memset(gradient + 18ull * t, 0, 18 * sizeof(float));
            std::memcpy(gradient + 18ull * t, r, 6ull * ch * sizeof(float));
        }
        if (residual) {
            std::memset(residual + 3ull * t, 0, 3 * sizeof(float));
            std::memcpy(residual + 3ull * t, r + 6 * ch, (size_t)ch * sizeof(float));
        }
    }
    return WS_OK;
}

int ws_get_node2term(ws_solver *h, int scene, uint32_t *offsets, uint32_t *term_index, int cap, int *count) {
    if (!h || !count) return WS_ERR_INVALID_ARGUMENT;
    ws::Workspace &w = h->w;
    const int st = sync_for_debug(w, scene);
    if (st != WS_OK) return st;
    const ws::Scene &sc = w.h_scenes[scene];
    const auto off = download(w.n2t_offset + sc.node_base, (size_t)sc.num_nodes + 1);
    const uint32_t b = off.front(), e = off.back();
    *count = (int)(e - b);
    if ((int)(e - b) > cap) return WS_ERR_CAPACITY;
    if (offsets)
        for (int n = 0; n <= sc.num_nodes; ++n) offsets[n] = off[n] - b;
    if (term_index && e > b) cudaMemcpy(term_index, w.n2t_sorted_val + b, 4ull * (e - b), cudaMemcpyDeviceToHost);
    return WS_OK;
}

int ws_get_node_pairs(ws_solver *h, int scene, uint32_t *rows, uint32_t *cols, uint32_t *begin, uint32_t *end, int cap,
                      int *count, uint32_t *term_index, int term_cap, int *term_count) {
    if (!h || !count) return WS_ERR_INVALID_ARGUMENT;
    ws::Workspace &w = h->w;
    const int st = sync_for_debug(w, scene);
    if (st != WS_OK) return st;
    uint32_t f, l;
    std::vector<uint32_t> all_rows;
    half_range(w, scene, f, l, all_rows);
    const uint32_t n = l - f;
    *count = (int)n;
    if ((int)n > cap) return WS_ERR_CAPACITY;
    const uint32_t nb = (uint32_t)w.h_scenes[scene].node_base;
    const auto c = download(w.half_col + f, n);
    const auto b = download(w.half_begin + f, n);
    const auto e = download(w.half_end + f, n);
    const uint32_t t0 = n ? b.front() : 0u, t1 = n ? e.back() : 0u;
    for (uint32_t i = 0; i < n; ++i) {
        if (rows) rows[i] = all_rows[f + i] - nb;
        if (cols) cols[i] = c[i] - nb;
        if (begin) begin[i] = b[i] - t0;
        if (end) end[i] = e[i] - t0;
    }
    if (term_count) *term_count = (int)(t1 - t0);
    if (term_index) {
        if ((int)(t1 - t0) > term_cap) return WS_ERR_CAPACITY;
        if (t1 > t0) cudaMemcpy(term_index, w.pair_sorted_val + t0, 4ull * (t1 - t0), cudaMemcpyDeviceToHost);
    }
    return WS_OK;
}

int ws_get_system(ws_solver *h, int scene, uint32_t *rowptr, uint32_t *cols, float *blocks, int block_cap,
                  int *num_blocks, float *inv_diag, float *jtr, float *step) {
    if (!h || !num_blocks) return WS_ERR_INVALID_ARGUMENT;
    ws::Workspace &w = h->w;
    const int st = sync_for_debug(w, scene);
    if (st != WS_OK) return st;
    const ws::Scene &sc = w.h_scenes[scene];
    const auto rp = download(w.rowptr + sc.node_base, (size_t)sc.num_nodes + 1);
    const uint32_t b = rp.front(), e = rp.back();
    *num_blocks = (int)(e - b);
    if ((int)(e - b) > block_cap) return WS_ERR_CAPACITY;
    if (rowptr)
        for (int i = 0; i <= sc.num_nodes; ++i) rowptr[i] = rp[i] - b;
    if (cols) {
        const auto ci = download(w.colidx + b, e - b);
        for (uint32_t i = 0; i < e - b; ++i) cols[i] = ci[i] - (uint32_t)sc.node_base;
    }
    if (blocks) {
        // expand the symmetric store (per row: the diagonal, then the upper pairs in column
        // order) into full block-CSR rows; a lower slot is the transpose of an upper item
        const auto ci = download(w.colidx + b, e - b);
        const auto ip = download(w.item_ptr + sc.node_base, (size_t)sc.num_nodes + 1);
        const uint32_t ub = ip.front(), ue = ip.back();
        const auto sb = download(w.sym_blocks + 36ull * ub, 36ull * (ue - ub));
        const auto cols = download(w.item_col + ub, (size_t)(ue - ub));   // upper items carry no row mark
        const uint32_t nb = (uint32_t)sc.node_base;
        auto upper = [&](uint32_t i, uint32_t col) -> const float * {   // local row i, global column
            uint32_t lo = ip[i] + 1, hi = ip[i + 1];
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (cols[mid - ub] < col) lo = mid + 1; else hi = mid;
            }
            if (lo >= ip[i + 1] || cols[lo - ub] != col) return nullptr;
            return sb.data() + 36ull * (lo - ub);
        };
        for (int i = 0; i < sc.num_nodes; ++i)
            for (uint32_t k = rp[i]; k < rp[i + 1]; ++k) {
                float *out = blocks + 36ull * (k - b);
                const uint32_t col = ci[k - b];
                const bool tr = col < nb + (uint32_t)i;
                const float *src = k == rp[i] ? sb.data() + 36ull * (ip[i] - ub)
                                   : tr       ? upper(col - nb, nb + (uint32_t)i)
                                              : upper((uint32_t)i, col);
                if (!src) return WS_ERR_CAPACITY;
                for (int a = 0; a < 6; ++a)
                    for (int c = 0; c < 6; ++c) out[6 * a + c] = tr ? src[6 * c + a] : src[6 * a + c];
            }
    }
    if (inv_diag) cudaMemcpy(inv_diag, w.inv_diag + 36ull * sc.node_base, 144ull * sc.num_nodes, cudaMemcpyDeviceToHost);
    auto vec6 = [&](const float *src, float *dst) {
        const auto v = download(src + 8ull * sc.node_base, 8ull * sc.num_nodes);
        for (int n = 0; n < sc.num_nodes; ++n)
            for (int q = 0; q < 6; ++q) dst[6 * n + q] = v[8ull * n + q];
    };
    if (jtr) vec6(w.jtr, jtr);
    if (step) vec6(w.x, step);
    return cudaGetLastError() == cudaSuccess ? WS_OK : WS_ERR_CUDA;
}

}  // extern "C"
