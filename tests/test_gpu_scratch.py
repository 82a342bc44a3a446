"""The geometry calls' scratch can be given back by a program that has no solver."""
import pytest

pytestmark = pytest.mark.gpu


def test_trim_gives_the_scratch_back(ws):
    import numpy as np
    import torch
    from starhub_b200 import _lib
    from starhub_b200.solver import GpuGeometry
    lib = _lib.load()
    pts = np.random.default_rng(3).uniform(-0.5, 0.5, (400_000, 4)).astype(np.float32)
    geo = GpuGeometry()
    first = geo.init_nodes(pts, 0.025)   # modules loaded, the pool made
    assert lib.ws_trim_scratch(0) == _lib.WS_OK

    def free():
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        return torch.cuda.mem_get_info()[0]

    before = free()
    again = geo.init_nodes(pts, 0.025)
    kept = before - free()
    assert kept > 0   # 400k surfels take some 20 MB
    assert lib.ws_trim_scratch(0) == _lib.WS_OK
    assert before - free() <= kept - (8 << 20)
    np.testing.assert_array_equal(first, again)
    assert lib.ws_trim_scratch(-1) == _lib.WS_ERR_INVALID_ARGUMENT
    assert lib.ws_trim_scratch(torch.cuda.device_count()) == _lib.WS_ERR_INVALID_ARGUMENT
