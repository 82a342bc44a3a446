"""The streamed PCG (k_pcg) on its own: the autotuner times it whatever form the inputs run in, its launch shapes give
the same bits, and the benchmark's batch is held to the FP64 oracle in it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(ds, precision=0):
    from starhub_b200.solver import WarpSolver
    s = WarpSolver(max_nodes=sum(d.num_nodes for d in ds), max_pixels=sum(d.num_pixels for d in ds),
                   max_edges=sum(d.num_edges for d in ds), max_scenes=len(ds), precision=precision)
    s.SetBatchInputs(ds)
    return s


@pytest.mark.parametrize("copies", [1, 72])
def test_autotune_times_every_block_count(ws, small_scene, tiny_scene, copies):
    """A batch that runs resident (1) and one that runs streamed (72): each candidate is timed, the fastest is kept,
    and the form stays the caller's."""
    import torch
    from starhub_b200 import _lib
    from starhub_b200.solver import DeviceScene
    s = _solver([DeviceScene.from_scene(small_scene), DeviceScene.from_scene(tiny_scene)] * copies)
    form = s.pcg_form()
    assert (form == _lib.WS_PCG_STREAMED) == (copies == 72)
    t = s.autotune(pcg_iters=5, stream=torch.cuda.Stream())
    offered = [m for m in t["pcg_ms"] if m >= 0]
    assert len(offered) > 1 and offered == t["pcg_ms"][: len(offered)]
    assert t["pcg_ms"][t["pcg_blocks_per_sm"] - 1] == min(offered)
    assert s.pcg_form() == form


@pytest.mark.parametrize("precision", [0, 1])
def test_launch_shapes_give_the_same_bits(ws, small_scene, tiny_scene, small_scene_k8, precision):
    import torch
    from starhub_b200 import _lib
    from starhub_b200.solver import DeviceScene
    ds = [DeviceScene.from_scene(s) for s in (small_scene, tiny_scene, small_scene_k8)]
    s = _solver(ds, precision)
    s.set_pcg_form(_lib.WS_PCG_STREAMED)
    stream, want = torch.cuda.Stream(), None
    for shape in ((64, 64, 64), (64, 64, 1), (128, 128, 2), (128, 256, 3), (256, 64, 1)):
        s.set_tuning(*shape)
        s.SolveStreamed(3, 10, stream=stream, graph=True)
        s.Sync()
        got = [s.SolvedNodeSE3(i).cpu().numpy().copy() for i in range(3)]
        want = want or got
        for a, b in zip(want, got):
            np.testing.assert_array_equal(a, b, err_msg=str(shape))


def test_benchmark_batch_meets_the_bar(ws, orc):
    """Scenes of the 64-scene batch family (8-NN graph, 640x480, 130 surfels per node, 5 Gauss-Newton x 20 PCG) at its
    smallest, median and largest node counts, through the CUDA-graph replay, in the form that the whole batch runs in:
    each within 1e-4 relative twist error and 1e-5 m warped-position error of the FP64 oracle."""
    import torch
    from starhub_b200 import _lib, scenes
    from starhub_b200.scenes import position_error, twist_error
    from starhub_b200.solver import DeviceScene, GpuGeometry
    targets = scenes.batch_node_targets(64, 2)
    order = np.argsort(targets, kind="stable")
    geo = GpuGeometry()
    host = [scenes.batch_scene(int(targets[i]), geo, int(i)) for i in (order[0], order[32], order[-1])]
    b = _solver([DeviceScene.from_scene(sc) for sc in host])
    b.set_pcg_form(_lib.WS_PCG_STREAMED)
    st = torch.cuda.Stream()
    for _ in range(2):                      # capture, then a replay
        b.SolveStreamed(5, 20, stream=st, graph=True)
    b.Sync()
    for i, sc in enumerate(host):
        dq = b.SolvedNodeSE3(i).cpu().numpy().copy()
        ref = orc.solve(sc, gn_iters=5, pcg_iters=20)
        te, pe = twist_error(dq, ref, sc.nodes), position_error(sc, dq, ref)
        assert te <= 1e-4 and pe <= 1e-5, (sc.num_nodes, te, pe)
