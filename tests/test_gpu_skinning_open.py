"""Skinning where the node grid leaves many of a warp's surfels open (ties, far from all nodes): ids against the scan of
every node, which a radius beyond the grid's range takes, at the counts where a launch's rounds change."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# surfels: less than a warp, spread over the SMs, one more than a whole round of the launch, more than 32 rounds a warp;
# nodes: one chunk, two
@pytest.mark.parametrize("surfels,nodes", [(5, 320), (3001, 320), (148 * 1024 + 1, 320), (5_000_017, 320), (40_003, 10_300)])
@pytest.mark.parametrize("deleted", [False, True])
def test_open_surfels(ws, surfels, nodes, deleted):
    import torch
    from starhub_b200.solver import GpuGeometry
    g = torch.Generator(device="cuda").manual_seed(surfels + nodes)
    m = round(nodes ** (1 / 3)) + 1
    at = torch.arange(m, device="cuda") / 32.0
    lattice = torch.stack(torch.meshgrid(at, at, at, indexing="ij"), -1).reshape(-1, 3)[:nodes]
    def four(x):
        return torch.cat([x, torch.ones(len(x), 1, device="cuda")], 1).contiguous()
    pick = lattice[torch.randint(len(lattice), (surfels,), generator=g, device="cuda")]
    kind = (torch.arange(surfels, device="cuda") // 48) % 3   # warps with one kind of surfel and with two
    far = torch.rand((surfels, 3), generator=g, device="cuda") + 20.0
    verts = torch.where(kind[:, None] == 0, pick + 1 / 64, torch.where(kind[:, None] == 1, far, pick + 0.003 * far))
    status = None
    if deleted:
        status = np.zeros((nodes, 2), np.uint32)
        status[::3, 1] = 0xFFFFFFFF
    geo = GpuGeometry()
    ids, _, cw = geo.skinning_ex(four(lattice), four(verts), 0.025, status=status)
    want, _, _ = geo.skinning_ex(four(lattice), four(verts), 2e6, status=status)
    np.testing.assert_array_equal(ids, want)
    assert (cw == 1).all()
