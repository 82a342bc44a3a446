"""The radix sort of the index build at the edges of its tiles (2048 keys up to a capacity of 4 M, 4096 beyond),
through the node -> term map, whose order is the reference's stable sort."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("capacity", ["small", "large"])
@pytest.mark.parametrize("over", [-4, 0, 4, 2044])
def test_lists_at_tile_edges(ws, orc, small_scene, capacity, over):
    """The number of keys is made 4096 k + over (to 3 more) with feature terms, four keys each."""
    import torch
    from starhub_b200.solver import DeviceScene, WarpSolver
    _, knn, _, _ = orc.compact_pixels(small_scene)
    keys = 4 * len(knn) + 2 * len(small_scene.edges) + small_scene.num_nodes
    features = ((over - keys) % 4096 + 3) // 4
    pick = np.random.default_rng(7).integers(0, len(small_scene.surfel_knn), features + 1)[:features]
    sc = dataclasses.replace(small_scene, feature_knn=small_scene.surfel_knn[pick].copy()) if features else small_scene
    total = keys + 4 * features
    assert abs((total - over) % 4096) < 4
    ds = DeviceScene.from_scene(sc)
    pixels = ds.num_pixels if capacity == "small" else (5 << 20) // 4
    assert (4 * pixels + 2 * ds.num_edges + ds.num_nodes + 4 * features <= 4 << 20) == (capacity == "small")
    s = WarpSolver(max_nodes=ds.num_nodes, max_pixels=pixels, max_edges=ds.num_edges, max_features=features)
    s.SetSolverInputs(ds)
    s.SolveStreamed(1, 1, stream=torch.cuda.Stream())
    s.Sync()
    off, ti = s.node2term()
    ooff, oti = orc.node2term(knn, sc.edges, sc.num_nodes, feat_knn=sc.feature_knn)
    np.testing.assert_array_equal(off, ooff)
    np.testing.assert_array_equal(ti, oti[: ooff[-1]])
    p = s.node_pairs()
    m = orc.nodepair2term(knn, sc.edges, sc.num_nodes, feat_knn=sc.feature_knn)
    np.testing.assert_array_equal(p["rows"], m["half_rows"])
    np.testing.assert_array_equal(p["term_index"], m["term_index"][: m["half_end"][-1]])
