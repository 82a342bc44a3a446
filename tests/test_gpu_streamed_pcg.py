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
