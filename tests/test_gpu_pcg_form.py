"""ws_set_pcg_form: a program whose solvers share a device can keep a solver's PCG on the streamed form, and every
form gives the same bits."""
import ctypes as C

import numpy as np
import pytest


def test_arguments():
    from starhub_b200 import _lib, build
    build.build()
    lib = _lib.load()
    form = C.c_int()
    assert lib.ws_set_pcg_form(None, 0, 0) == _lib.WS_ERR_INVALID_ARGUMENT
    assert lib.ws_get_pcg_form(None, C.byref(form)) == _lib.WS_ERR_INVALID_ARGUMENT


@pytest.mark.gpu
@pytest.mark.parametrize("graph", [False, True])
def test_streamed_on_request(ws, small_scene, tiny_scene, graph):
    import torch
    from starhub_b200 import _lib
    from starhub_b200._lib import WarpSolveError
    from starhub_b200.solver import DeviceScene, WarpSolver
    ds = [DeviceScene.from_scene(s) for s in (small_scene, tiny_scene)]
    s = WarpSolver(max_nodes=sum(d.num_nodes for d in ds), max_pixels=sum(d.num_pixels for d in ds),
                   max_edges=sum(d.num_edges for d in ds), max_scenes=2)
    with pytest.raises(WarpSolveError):
        s.pcg_form()   # no inputs yet
    for bad in ((-1, 0), (4, 0), (0, 49151), (0, 228865), (0, -1)):
        with pytest.raises(WarpSolveError):
            s.set_pcg_form(*bad)
    s.SetBatchInputs(ds)
    out, stream = {}, torch.cuda.Stream()
    for form in (_lib.WS_PCG_AUTO, _lib.WS_PCG_STREAMED, _lib.WS_PCG_CLUSTERS, _lib.WS_PCG_GRID, _lib.WS_PCG_AUTO):
        s.set_pcg_form(form)
        ran = s.pcg_form()
        assert ran == form if form != _lib.WS_PCG_AUTO else ran != _lib.WS_PCG_STREAMED
        for _ in range(2):
            s.SolveStreamed(2, 7, stream=stream, graph=graph)
        s.Sync()
        for i in range(2):
            got = s.SolvedNodeSE3(i).cpu().numpy()
            np.testing.assert_array_equal(out.setdefault(i, got.copy()), got, err_msg=f"form {form}")


@pytest.mark.gpu
@pytest.mark.parametrize("scenes,nodes,form", [(1, 500, 2), (1, 1800, 2), (7, 3000, 2), (1, 8000, 3), (8, 1000, 3),
                                               (8, 4000, 3), (8, 8000, 3), (40, 4000, 1)])
def test_form_by_size(ws, scenes, nodes, form):
    """Scenes that do not fit beside one another run in rounds: eight clusters on a device that holds seven take
    twice a cluster's time (8 x 8000 nodes: 60.8 us an iteration, 27.8 over the whole grid, 38.4 streamed)."""
    from starhub_b200.solver import WarpSolver
    from test_gpu_pcg_layouts import random_scene
    a = random_scene(nodes, 1)
    s = WarpSolver(max_nodes=scenes * nodes, max_pixels=scenes * a.num_pixels, max_edges=scenes * a.num_edges,
                   max_scenes=scenes)
    s.SetBatchInputs([a] * scenes)
    assert s.pcg_form() == form


# touches: 1 gives about 4.5 upper pairs a row, 8 about 15, anywhere in the scene
@pytest.mark.gpu
@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("sizes,sparse,dense", [([4000] * 8, 3, 1), ([8000, 3000] * 3, 3, 1), ([3000] * 4, 2, 1)])
def test_form_by_pairs(ws, sizes, sparse, dense, graph):
    """Where the size does not settle it, the device takes the streamed form for rows with many pairs (16 x 4500 nodes
    with 15 pairs a row: 238 us an iteration over the whole grid, 83 streamed); one solver meets both."""
    import torch
    from starhub_b200 import _lib
    from starhub_b200.solver import WarpSolver
    from test_gpu_pcg_layouts import random_scene
    by_size = {(n, t): random_scene(n, t) for n in set(sizes) for t in (1, 10)}
    most = [by_size[n, 10] for n in sizes]
    stream = torch.cuda.Stream()
    s = WarpSolver(max_nodes=sum(sizes), max_pixels=sum(a.num_pixels for a in most),
                   max_edges=sum(a.num_edges for a in most), max_scenes=len(sizes))
    for touches, form in ((10, dense), (1, sparse), (10, dense)):
        items = [by_size[n, touches] for n in sizes]
        out = []
        for ask in (_lib.WS_PCG_AUTO, _lib.WS_PCG_STREAMED):
            s.set_pcg_form(ask)
            s.SetBatchInputs(items)
            for _ in range(2):
                s.SolveStreamed(2, 3, stream=stream, graph=graph)
            s.Sync()
            if ask == _lib.WS_PCG_AUTO:
                assert s.pcg_form() == form, touches
            out.append([s.SolvedNodeSE3(i).cpu().numpy().copy() for i in range(len(items))])
        for a, b in zip(*out):
            assert np.isfinite(a).all()
            np.testing.assert_array_equal(a, b)


@pytest.mark.gpu
@pytest.mark.parametrize("budget", [0, 49152])   # without and with a ring whose copies are on their way
def test_resident_waits_give_up_and_the_device_stays_usable(ws, small_scene_k8, budget):
    """The waits of the PCG over the whole grid are bounded: for a copy that nobody starts, and at a meeting that one
    block never reaches, where the others leave with WS_ERR_TIMEOUT.  A solve afterwards equals one before."""
    import time
    import torch
    from starhub_b200 import _lib
    from starhub_b200.solver import DeviceScene, WarpSolver
    ds = DeviceScene.from_scene(small_scene_k8)
    s = WarpSolver(max_nodes=ds.num_nodes, max_pixels=ds.num_pixels, max_edges=ds.num_edges)
    s.set_pcg_form(_lib.WS_PCG_GRID, budget)
    s.SetSolverInputs(ds)
    lib, stream = _lib.load(), torch.cuda.Stream()
    assert lib.ws_selftest_resident_timeout(s._h, None) == _lib.WS_ERR_NOT_READY
    out = []
    for _ in range(2):
        s.SolveStreamed(2, 6, stream=stream)
        s.Sync()
        out.append(s.SolvedNodeSE3(0).cpu().numpy().copy())
        if len(out) == 1:
            t0 = time.perf_counter()
            assert lib.ws_selftest_resident_timeout(s._h, C.c_void_p(stream.cuda_stream)) == _lib.WS_ERR_TIMEOUT
            assert 0.05 < time.perf_counter() - t0 < 60.0
    np.testing.assert_array_equal(*out)
