"""The cluster PCG against the persistent one: a lone small scene runs on a cluster, the same scene in a
batch of many on k_pcg, and both must give the same bits (the kernels do the same arithmetic)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cut(scene, nodes, seed):
    """The scene on `nodes` of its nodes (anchors included): surfels skinned to four distinct ones near their
    own, the graph a band (a pair then has at most one smoothness term per direction)."""
    import dataclasses
    keep = np.sort(np.random.default_rng(seed).permutation(scene.num_nodes)[:nodes])
    near = np.searchsorted(keep, scene.surfel_knn.astype(int)[:, 0]).clip(0, nodes - 1)
    k = min(8, (nodes - 1) // 2)
    i = np.arange(nodes)[:, None]
    edges = np.stack(np.broadcast_arrays(i, (i + np.arange(k)) % nodes, np.arange(k)), -1)
    return dataclasses.replace(scene, nodes=scene.nodes[keep], graph_k=k, node_cw=np.ones((nodes, k), np.float32),
                               surfel_knn=((near[:, None] + np.arange(4)) % nodes).astype(np.uint16),
                               edges=edges.reshape(-1, 3).astype(np.uint16))


# nodes: one group, a partial group, fewer groups than blocks, one more than a block each, a whole scene
@pytest.mark.parametrize("nodes,gn,pcg,precision", [(5, 2, 3, 0), (16, 1, 1, 0), (17, 2, 4, 0), (255, 2, 5, 0),
                                                    (257, 2, 5, 1), (900, 1, 0, 0), (900, 2, 2, 0), (1500, 3, 10, 0)])
def test_cluster_equals_persistent(ws, small_scene_k8, nodes, gn, pcg, precision):
    import torch
    from starhub_b200.solver import DeviceScene, WarpSolver
    nodes = min(nodes, small_scene_k8.num_nodes)
    sc = small_scene_k8 if nodes == small_scene_k8.num_nodes else _cut(small_scene_k8, nodes, 3)
    ds = DeviceScene.from_scene(sc)
    copies = 72   # far past the batch size where k_pcg takes over
    out = []
    for n in (1, copies):
        s = WarpSolver(max_nodes=n * ds.num_nodes, max_pixels=n * ds.num_pixels, max_edges=n * ds.num_edges, max_scenes=n,
                       precision=precision)
        s.SetBatchInputs([ds] * n)
        s.SolveStreamed(gn, pcg, stream=torch.cuda.Stream())
        s.Sync()
        out.append([s.SolvedNodeSE3(i).cpu().numpy().copy() for i in {0, n // 2, n - 1}])
    assert np.isfinite(out[0][0]).all()
    for b in out[1]:
        np.testing.assert_array_equal(out[0][0], b)


def test_scattered_node_order(ws, small_scene_k8):
    """Node ids in random order: every block's halo is most of the scene."""
    import dataclasses
    import torch
    from starhub_b200.solver import DeviceScene, WarpSolver
    n = small_scene_k8.num_nodes
    order = np.random.default_rng(9).permutation(n)
    new_id = np.empty(n, int)
    new_id[order] = np.arange(n)
    e = small_scene_k8.edges.astype(int).reshape(n, 8, 3)[order]
    e = np.stack([new_id[e[..., 0]], new_id[e[..., 1]], e[..., 2]], -1).reshape(-1, 3)
    sc = dataclasses.replace(small_scene_k8, nodes=small_scene_k8.nodes[order], node_cw=small_scene_k8.node_cw[order],
                             surfel_knn=new_id[small_scene_k8.surfel_knn.astype(int)].astype(np.uint16),
                             edges=e.astype(np.uint16))
    ds = DeviceScene.from_scene(sc)
    out = []
    for c in (1, 72):
        s = WarpSolver(max_nodes=c * n, max_pixels=c * ds.num_pixels, max_edges=c * ds.num_edges, max_scenes=c)
        s.SetBatchInputs([ds] * c)
        s.SolveStreamed(2, 10, stream=torch.cuda.Stream())
        s.Sync()
        out.append(s.SolvedNodeSE3(c - 1).cpu().numpy().copy())
    np.testing.assert_array_equal(out[0], out[1])


@pytest.mark.parametrize("nodes,lambda_of,precision", [(40, 0.0, 0), (255, 0.0, 1), (255, 0.1, 0), (500, 0.1, 1)])
def test_long_and_short_list_assembly(ws, small_scene_k8, nodes, lambda_of, precision):
    """Alone, the scene's lists are long (many pixels a node) and its pairs' records go through two buffers;
    beside a scene with few pixels a node they go through one.  The sums run in the same order."""
    import dataclasses
    import torch
    from starhub_b200.solver import DeviceScene, WarpSolver
    sc = dataclasses.replace(_cut(small_scene_k8, nodes, 7), lambda_of=lambda_of)
    a, b = DeviceScene.from_scene(sc), DeviceScene.from_scene(small_scene_k8)
    assert a.num_pixels >= 150 * a.num_nodes and a.num_pixels + b.num_pixels < 150 * (a.num_nodes + b.num_nodes)
    out = []
    for items in ([a], [a, b], [b, a]):
        s = WarpSolver(max_nodes=sum(d.num_nodes for d in items), max_pixels=sum(d.num_pixels for d in items),
                       max_edges=sum(d.num_edges for d in items), max_scenes=len(items), precision=precision)
        for threads in (64, 128, 256):
            s.set_tuning(threads, threads, 2)
            s.SetBatchInputs(items)
            s.SolveStreamed(2, 4, stream=torch.cuda.Stream())
            s.Sync()
            at = next(i for i, d in enumerate(items) if d is a)
            out.append(s.SolvedNodeSE3(at).cpu().numpy().copy())
    for x in out[1:]:
        np.testing.assert_array_equal(out[0], x)


@pytest.fixture(scope="module")
def large_scene(orc):
    """About 4500 nodes at 160x120: alone, its PCG runs on the whole grid."""
    from starhub_b200 import scenes
    spec = scenes.spec_for_nodes(5000, scenes.config_spec(0, width=160, height=120, focal=142.5), surfels_per_node=30)
    return scenes.make_scene(spec, orc.OracleGeometry(), seed=21)


@pytest.mark.parametrize("pcg,precision,scattered", [(0, 0, False), (1, 0, False), (12, 0, False), (7, 1, False),
                                                     (6, 0, True)])
def test_grid_equals_persistent(ws, large_scene, small_scene_k8, pcg, precision, scattered):
    """The large scene alone and beside others (the whole grid), and in a batch that only k_pcg takes."""
    import dataclasses
    import torch
    from starhub_b200.solver import DeviceScene, WarpSolver
    sc = large_scene
    n = sc.num_nodes
    if scattered:   # node ids in random order: halos of most of the scene
        order = np.random.default_rng(9).permutation(n)
        new_id = np.empty(n, int)
        new_id[order] = np.arange(n)
        e = sc.edges.astype(int).reshape(n, 8, 3)[order]
        e = np.stack([new_id[e[..., 0]], new_id[e[..., 1]], e[..., 2]], -1).reshape(-1, 3)
        sc = dataclasses.replace(sc, nodes=sc.nodes[order], node_cw=sc.node_cw[order], edges=e.astype(np.uint16),
                                 surfel_knn=new_id[sc.surfel_knn.astype(int)].astype(np.uint16))
    a = DeviceScene.from_scene(sc)
    b, c = DeviceScene.from_scene(_cut(small_scene_k8, 17, 3)), DeviceScene.from_scene(small_scene_k8)
    out = {}
    for key, items in (("alone", [a]), ("few", [b, a, c]), ("other order", [c, a, b]), ("small alone", [c]),
                       ("tiny alone", [b]), ("many", [a] * 40 + [b, c])):
        s = WarpSolver(max_nodes=sum(d.num_nodes for d in items), max_pixels=sum(d.num_pixels for d in items),
                       max_edges=sum(d.num_edges for d in items), max_scenes=len(items), precision=precision)
        s.SetBatchInputs(items)
        s.SolveStreamed(2, pcg, stream=torch.cuda.Stream())
        s.Sync()
        for i, d in enumerate(items):
            name = "a" if d is a else "b" if d is b else "c"
            got = s.SolvedNodeSE3(i).cpu().numpy()
            np.testing.assert_array_equal(out.setdefault(name, got.copy()), got, err_msg=f"{name} in {key}")
