"""Skinning over the node grid against the oracle's ordered scan, where the grid's answer is not settled by
itself: ties, far or too few nodes, radii that do not fit the node spacing, deleted and NaN nodes, and the
node counts at which the path or its chunks change.  Ids bit-exact; weights within 2e-5 relative (__expf on
the device, expf in the oracle)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
R = 0.025


def _points(n, seed, extent=1.0):
    p = np.ones((n, 4), np.float32)
    p[:, :3] = np.random.default_rng(seed).uniform(-extent, extent, (n, 3))
    return p


def _check(orc, nodes, verts, radius, status=None, normalize=True):
    from starhub_b200.solver import GpuGeometry
    gk, gs, gc = GpuGeometry().skinning_ex(nodes, verts, radius, status=status, normalize=normalize)
    ok, osw, oc = orc.OracleGeometry().skinning_ex(nodes, verts, radius, status=status, normalize=normalize)
    np.testing.assert_array_equal(gk, ok)
    np.testing.assert_allclose(gs, osw, rtol=2e-5, atol=1e-7)
    np.testing.assert_array_equal(gc, oc)


# below and at the grid's first count, a whole chunk, one more, several chunks
@pytest.mark.parametrize("n", [4, 299, 300, 301, 1024, 10240, 10241, 25000])
def test_node_counts(ws, orc, n):
    _check(orc, _points(n, n), _points(1500, 1, 1.2), R * (2000 / max(n, 50)) ** (1 / 3))


@pytest.mark.parametrize("scale", [0.01, 0.1, 1.0, 10.0, 1000.0])
def test_radius_far_from_the_spacing(ws, orc, scale):
    _check(orc, _points(2000, 3), _points(1000, 4, 1.1), 0.1 * scale, normalize=False)


def test_lattice_ties(ws, orc):
    g = np.stack(np.meshgrid(*[np.arange(10, dtype=np.float32) * 0.03125] * 3, indexing="ij"), -1).reshape(-1, 3)
    nodes = np.concatenate([g, np.ones((len(g), 1), np.float32)], 1).astype(np.float32)
    half = nodes.copy()
    half[:, :3] += 0.015625
    _check(orc, nodes, np.concatenate([nodes, half]), R)


def test_doubled_nodes_far_surfels_and_few_live_nodes(ws, orc):
    nodes = np.concatenate([_points(400, 5), _points(400, 5)])
    verts = np.concatenate([_points(300, 6), _points(100, 7, 50.0), _points(40, 8, 3000.0)])
    _check(orc, nodes, verts, R)
    status = np.zeros((len(nodes), 2), np.uint32)
    status[3:, 1] = 0xFFFFFFFF   # three nodes left
    _check(orc, nodes, verts, 0.5, status=status, normalize=False)


def test_wrapped_cells(ws, orc):
    """Clusters whose cells coincide modulo the grid's size."""
    base = _points(200, 9, 0.2)
    nodes = np.concatenate([base + np.float32([k * 32 * 1.75 * R, 0, 0, 0]) for k in range(4)])
    nodes[:, 3] = 1
    _check(orc, nodes, nodes[::3] + np.float32([0.003, 0.002, 0.001, 0]), R)


def test_nan_node_and_surfel(ws, orc):
    from starhub_b200.solver import GpuGeometry
    nodes, verts = _points(800, 10), _points(300, 11)
    clean = GpuGeometry().skinning(nodes, verts, R)
    nodes[77, 1] = np.nan
    got = GpuGeometry().skinning(nodes, verts, R)
    away = ~(clean[0] == 77).any(1)
    np.testing.assert_array_equal(got[0][away], clean[0][away])   # a NaN node enters no heap
    assert not (got[0] == 77).any()
    verts[5, 0] = np.nan
    got = GpuGeometry().skinning(nodes, verts, R)
    np.testing.assert_array_equal(got[0][5], [0, 0, 0, 0])        # the heap's initial entries
