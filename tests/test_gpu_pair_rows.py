"""The node pair map with several warps to a row against one warp to a row: a scene alone (few rows, long
lists) and beside enough others (many rows) must give the same bits, and the same rows must be refused."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cut(scene, nodes, pixels_of=None):
    """The scene on `nodes` nodes with a band graph; all pixels' surfels skinned near each other's nodes."""
    near = (scene.surfel_knn.astype(int)[:, 0] * nodes) // scene.num_nodes
    if pixels_of is not None:   # every list but those of four nodes is short
        near[:] = pixels_of
    k = min(4, (nodes - 1) // 2)
    i = np.arange(nodes)[:, None]
    edges = np.stack(np.broadcast_arrays(i, (i + np.arange(k)) % nodes, np.arange(k)), -1)
    return dataclasses.replace(scene, nodes=scene.nodes[:nodes], graph_k=k, node_cw=np.ones((nodes, k), np.float32),
                               surfel_knn=((near[:, None] + np.arange(4)) % nodes).astype(np.uint16),
                               edges=edges.reshape(-1, 3).astype(np.uint16))


def _solve(items, gn=2, pcg=4):
    import torch
    from starhub_b200.solver import WarpSolver
    s = WarpSolver(max_nodes=sum(d.num_nodes for d in items), max_pixels=sum(d.num_pixels for d in items),
                   max_edges=sum(d.num_edges for d in items), max_scenes=len(items))
    s.SetBatchInputs(items)
    s.SolveStreamed(gn, pcg, stream=torch.cuda.Stream())
    s.Sync()
    return [s.SolvedNodeSE3(i).cpu().numpy().copy() for i in (0, len(items) - 1)]


# nodes of a scene of 320x240 pixels: eight warps to a row (up to 307), four (308 to 1024), one in the batch;
# pixels_of: all dense terms on four nodes, whose lists are the longest there are, others nearly empty
@pytest.mark.parametrize("nodes,pixels_of,lambda_of", [(5, None, 0.0), (40, None, 0.1), (40, 0, 0.0), (40, 38, 0.0),
                                                       (307, 70, 0.1), (308, None, 0.0), (900, None, 0.1), (900, 3, 0.0)])
def test_wide_rows_equal_narrow(ws, small_scene_k8, nodes, pixels_of, lambda_of):
    from starhub_b200.solver import DeviceScene
    sc = dataclasses.replace(_cut(small_scene_k8, nodes, pixels_of), lambda_of=lambda_of)
    a, b = DeviceScene.from_scene(sc), DeviceScene.from_scene(small_scene_k8)
    assert (a.num_pixels >= 250 * nodes) == (nodes <= 307) and a.num_pixels >= 75 * nodes
    filler = [b] * (6001 // b.num_nodes + 1)
    total = a.num_nodes + len(filler) * b.num_nodes
    assert total > 6000 and a.num_pixels + len(filler) * b.num_pixels < 300 * total
    alone = _solve([a])[0]
    assert np.isfinite(alone).all()
    np.testing.assert_array_equal(alone, _solve([a] + filler)[0])
    np.testing.assert_array_equal(alone, _solve(filler + [a])[1])


@pytest.mark.parametrize("wide", [True, False])
@pytest.mark.parametrize("pairs", [64, 65])
def test_row_of_64_pairs(ws, small_scene_k8, pairs, wide):
    """A row holds 64 upper pairs; one more is refused, however many warps look at it."""
    from starhub_b200._lib import WarpSolveError
    from starhub_b200.solver import DeviceScene
    sc = _cut(small_scene_k8, 70, pixels_of=60)   # dense terms only between nodes 60 .. 63
    i = np.arange(70)
    to = np.where((i >= 1) & (i <= pairs), 0, i)   # node i to node 0, the others to themselves
    sc = dataclasses.replace(sc, graph_k=1, node_cw=np.ones((70, 1), np.float32),
                             edges=np.stack([i, to, 0 * i], -1).astype(np.uint16))
    a, b = DeviceScene.from_scene(sc), DeviceScene.from_scene(small_scene_k8)
    items = [a] if wide else [a] + [b] * (6001 // b.num_nodes + 1)
    if pairs == 64:
        assert np.isfinite(_solve(items, 1, 1)[0]).all()
    else:
        with pytest.raises(WarpSolveError):
            _solve(items, 1, 1)


@pytest.mark.parametrize("precision,lambda_of", [(0, 0.0), (1, 0.1)])
def test_pairs_drawn_in_runs(ws, small_scene_k8, precision, lambda_of):
    """Past 16 pairs a warp the pair kernel's warps draw runs of four; launch after launch, and whatever the
    blocks' size, every copy's result is the scene's own."""
    import torch
    from starhub_b200.solver import DeviceScene, WarpSolver
    a = DeviceScene.from_scene(dataclasses.replace(_cut(small_scene_k8, 1500), lambda_of=lambda_of))
    copies = 73
    out = []
    for n in (1, copies):
        s = WarpSolver(max_nodes=n * a.num_nodes, max_pixels=n * a.num_pixels, max_edges=n * a.num_edges, max_scenes=n,
                       precision=precision)
        for threads in (64, 128, 256, 64):
            s.set_tuning(threads, threads, 2)
            s.SetBatchInputs([a] * n)
            s.SolveStreamed(2, 3, stream=torch.cuda.Stream())
            s.Sync()
            out += [s.SolvedNodeSE3(i).cpu().numpy().copy() for i in sorted({0, n // 3, n - 1})]
    assert copies * len(s.node_pairs(0)["rows"]) > 16 * 32 * torch.cuda.get_device_properties(0).multi_processor_count
    for x in out[1:]:
        np.testing.assert_array_equal(out[0], x)
