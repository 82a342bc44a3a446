"""Node assembly with a block to a node against a warp to a node: a scene alone (few nodes, long lists) and in a
batch past the size where blocks are used must give the same bits, for every kind of term and batch remainder."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(scene, nodes, pixels_of, lambda_of, motion):
    near = (scene.surfel_knn.astype(int)[:, 0] * nodes) // scene.num_nodes
    if pixels_of is not None:   # all dense terms on four nodes; the other lists hold smoothness terms only
        near[:] = pixels_of
    k = min(4, (nodes - 1) // 2)
    i = np.arange(nodes)[:, None]
    edges = np.stack(np.broadcast_arrays(i, (i + np.arange(k)) % nodes, np.arange(k)), -1)
    rng = np.random.default_rng(3)
    pred = None
    if motion:
        pred = np.concatenate([rng.normal(0, 2e-3, (nodes, 3)), rng.uniform(0.5, 1.0, (nodes, 1))], 1).astype(np.float32)
    return dataclasses.replace(scene, nodes=scene.nodes[:nodes], graph_k=k, node_cw=np.ones((nodes, k), np.float32),
                               surfel_knn=((near[:, None] + np.arange(4)) % nodes).astype(np.uint16),
                               edges=edges.reshape(-1, 3).astype(np.uint16), lambda_of=lambda_of,
                               node_motion_pred=pred, lambda_node=0.3 if motion else 0.0)


# 320x240 pixels: up to 384 nodes a block to a node
@pytest.mark.parametrize("nodes,pixels_of,lambda_of,motion,precision",
                         [(5, None, 0.0, False, 0), (33, None, 0.0, True, 1), (33, 31, 0.1, True, 0),
                          (150, None, 0.1, False, 1), (384, None, 0.0, False, 0), (384, 7, 0.0, False, 1),
                          (384, None, 0.1, True, 0)])
def test_block_equals_warp(ws, small_scene_k8, nodes, pixels_of, lambda_of, motion, precision):
    import torch
    from starhub_b200.solver import DeviceScene, WarpSolver
    a = DeviceScene.from_scene(_scene(small_scene_k8, nodes, pixels_of, lambda_of, motion))
    b = DeviceScene.from_scene(small_scene_k8)
    assert a.num_pixels >= 200 * nodes
    filler = [b] * (3201 // b.num_nodes + 1)
    out = []
    for items in ([a], [a] + filler, filler + [a]):
        s = WarpSolver(max_nodes=sum(d.num_nodes for d in items), max_pixels=sum(d.num_pixels for d in items),
                       max_edges=sum(d.num_edges for d in items), max_scenes=len(items), precision=precision)
        s.SetBatchInputs(items)
        s.SolveStreamed(2, 4, stream=torch.cuda.Stream())
        s.Sync()
        at = next(i for i, d in enumerate(items) if d is a)
        sys_ = s.system(at)
        out.append([s.SolvedNodeSE3(at).cpu().numpy().copy()] + [np.asarray(sys_[k]) for k in ("inv_diag", "jtr")])
    assert all(np.isfinite(x).all() for x in out[0])
    for o in out[1:]:
        for x, y in zip(out[0], o):
            np.testing.assert_array_equal(x, y)
