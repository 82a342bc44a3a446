"""Node construction with more overlapping pairs than the first lists hold, and with the overlap check's larger table:
candidates crowd around every third voxel's centre, where each has 9.5 earlier neighbours on average.  Bit-exact
against the oracle's sequential check."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
R = 0.025


# candidates: 27 000 (the smaller table), 274 625 (beyond 2^18)
@pytest.mark.parametrize("side", [30, 65])
def test_crowded_candidates(ws, orc, side):
    from starhub_b200.solver import GpuGeometry
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    inside = np.clip((1.5 - (g % 3) - 0.5) + 0.5, 0.02, 0.98)   # towards the middle one of three voxels
    jitter = np.random.default_rng(side).uniform(-0.01, 0.01, g.shape)
    p = np.ones((len(g), 4), np.float32)
    p[:, :3] = (g - side // 2 + inside + jitter) * np.float32(0.7 * R)
    np.testing.assert_array_equal(GpuGeometry().init_nodes(p, R), orc.OracleGeometry().init_nodes(p, R))
