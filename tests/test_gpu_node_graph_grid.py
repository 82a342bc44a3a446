"""The node graph over the node grid against the oracle's ordered scan: the node counts at which the path
changes, many ties in half precision, radii that do not fit the node spacing, deleted and coincident nodes.
Ids and edges bit-exact; weights within 2e-5 relative (__expf on the device, expf in the oracle)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(n, seed, extent=1.0):
    p = np.ones((n, 4), np.float32)
    p[:, :3] = np.random.default_rng(seed).uniform(-extent, extent, (n, 3))
    return p


def _check(orc, nodes, k, radius, status=None, normalize=True):
    from starhub_b200.solver import GpuGeometry
    gk, gw, ge = GpuGeometry().node_graph_ex(nodes, k, radius, status=status, normalize=normalize)
    ok, ow, oe = orc.OracleGeometry().node_graph_ex(nodes, k, radius, status=status, normalize=normalize)
    np.testing.assert_array_equal(gk, ok)
    np.testing.assert_array_equal(ge, oe)
    np.testing.assert_allclose(gw, ow, rtol=2e-5, atol=1e-7)


@pytest.mark.parametrize("k", [4, 8])
@pytest.mark.parametrize("n", [8, 33, 4999, 5000, 30000])
def test_node_counts(ws, orc, n, k):
    _check(orc, _points(n, n), k, 0.6 * max(n, 64) ** (-1 / 3))


@pytest.mark.parametrize("k", [4, 8])
@pytest.mark.parametrize("scale", [0.02, 1.0, 30.0])
def test_radius_far_from_the_spacing(ws, orc, scale, k):
    _check(orc, _points(6000, 3), k, 0.05 * scale, normalize=False)


@pytest.mark.parametrize("k", [4, 8])
def test_lattice_with_deleted_and_coincident_nodes(ws, orc, k):
    g = np.stack(np.meshgrid(*[np.arange(18, dtype=np.float32) * 0.0125] * 3, indexing="ij"), -1).reshape(-1, 3)
    nodes = np.concatenate([g, np.ones((len(g), 1), np.float32)], 1)
    nodes = np.concatenate([nodes, nodes[::29], _points(40, 6, 60.0)]).astype(np.float32)   # some far outside
    status = np.zeros((len(nodes), 2), np.uint32)
    status[np.random.default_rng(4).uniform(size=len(nodes)) < 0.05, 1] = 0xFFFFFFFF
    _check(orc, nodes, k, 0.025)
    _check(orc, nodes, k, 0.025, status=status, normalize=False)
