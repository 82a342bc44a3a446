"""The node graph's scan of tied nodes passes over 32 nodes at a time by their box: coincident nodes, a plane lattice in
scan order and out of it, and deleted runs, against the oracle's ordered scan.  Ids and edges bit-exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _nodes(kind, n):
    rng = np.random.default_rng(n)
    p = np.ones((n, 4), np.float32)
    if kind == "coincident":
        p[:, :3] = rng.uniform(0, 1e-4, (n, 3))
    else:
        m = int(np.ceil(np.sqrt(n)))
        i = np.arange(n)
        p[:, :3] = np.stack([i // m, i % m, 0 * i], 1) * np.float32(0.025)
        if kind == "shuffled plane":
            p = p[rng.permutation(n)]
    return p


@pytest.mark.parametrize("k", [4, 8])
@pytest.mark.parametrize("kind", ["coincident", "plane", "shuffled plane"])
@pytest.mark.parametrize("n,deleted", [(5001, False), (5001, True), (9000, False)])
def test_tied_nodes(ws, orc, kind, n, deleted, k):
    from starhub_b200.solver import GpuGeometry
    nodes = _nodes(kind, n)
    status = np.zeros((n, 2), np.uint32)
    if deleted:
        status[64:192, 1] = status[-5:, 1] = 0xFFFFFFFF   # whole boxes, and the end
    gk, gw, ge = GpuGeometry().node_graph_ex(nodes, k, 0.025, status=status, normalize=True)
    ok, ow, oe = orc.OracleGeometry().node_graph_ex(nodes, k, 0.025, status=status, normalize=True)
    np.testing.assert_array_equal(gk, ok)
    np.testing.assert_array_equal(ge, oe)
    np.testing.assert_allclose(gw, ow, rtol=2e-5, atol=1e-7)
