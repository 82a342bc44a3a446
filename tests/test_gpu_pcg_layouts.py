"""Resident PCG (k_pcg_cluster) on scenes whose blocks do not all hold the same data in shared memory.  Every form of
the PCG gives the same bits, so a batch that a resident form takes is compared with the same scenes in a batch that
only k_pcg takes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def random_scene(nodes, touches, seed=0):
    """A flat patch whose pixels are each skinned to four nodes anywhere in the scene, every node by `touches` pixels:
    about 1.5 touches + 3 upper node pairs a row (3 touches + 6 at most), in scattered order, so that the first rows
    have nearly all of theirs above them and the last rows few."""
    from starhub_b200.solver import DeviceScene, _dev
    rng = np.random.default_rng(seed)
    knn = np.concatenate([rng.permutation(nodes)[: nodes // 4 * 4].reshape(-1, 4) for _ in range(touches)])
    surfels, width = len(knn), 160
    height = -(-surfels // width)
    n = width * height
    f = 0.9 * width
    y, x = np.divmod(np.arange(n), width)
    z = 1.0 + 0.01 * np.sin(0.1 * x) * np.cos(0.13 * y)
    ref = np.stack([(x - width / 2) / f * z, (y - height / 2) / f * z, z, np.ones(n)], 1).astype(np.float32)
    normal = np.tile(np.float32([0.0, 0.0, -1.0, 0.002]), (n, 1))
    meas = ref.copy()
    meas[:, :3] *= (1.0 + 0.002 * rng.standard_normal((n, 1))).astype(np.float32)
    sw = rng.uniform(0.2, 1.0, (surfels, 4))
    index = np.where(np.arange(n) < surfels, np.arange(n), -1)
    i = np.arange(nodes)[:, None]
    edges = np.stack(np.broadcast_arrays(i, (i + np.arange(4)) % nodes, np.arange(4)), -1).reshape(-1, 3)
    pos = np.concatenate([rng.uniform(-0.4, 0.4, (nodes, 2)), rng.uniform(0.95, 1.05, (nodes, 1)), np.ones((nodes, 1))], 1)
    d = lambda a, t: _dev(np.ascontiguousarray(a.astype(t) if t != np.uint16 else a.astype(t).view(np.int16)), "cuda")
    shape = (height, width, 4)
    return DeviceScene(
        width=width, height=height, fx=f, fy=f, cx=width / 2, cy=height / 2, cam2world=np.eye(4, dtype=np.float32),
        measure_vertex=d(meas.reshape(shape), np.float32), measure_normal=d(normal.reshape(shape), np.float32),
        reference_vertex=d(ref.reshape(shape), np.float32), reference_normal=d(normal.reshape(shape), np.float32),
        index_map=d(index.reshape(height, width), np.int32), flow=None, surfel_knn=d(knn, np.uint16),
        surfel_sw=d(sw / sw.sum(1, keepdims=True), np.float32), surfel_cw=d(np.ones((surfels, 4)), np.float32),
        nodes=d(pos, np.float32), edges=d(edges, np.uint16), graph_k=4, node_cw=d(np.ones((nodes, 4)), np.float32),
        node_radius_square=0.025 ** 2)


def host_pairs(scene):
    """The scene's upper node pairs (row, column), rows ascending."""
    knn = np.sort(scene.surfel_knn.cpu().numpy().view(np.uint16).astype(np.int64), 1)
    e = np.sort(scene.edges.cpu().numpy().view(np.uint16).astype(np.int64)[:, :2], 1)
    p = np.concatenate([knn[:, [a, b]] for a in range(4) for b in range(a + 1, 4)] + [e[e[:, 0] != e[:, 1]]])
    p = np.unique(p[p[:, 0] != p[:, 1]], axis=0)
    return p[:, 0], p[:, 1]


def vector_rows(scene, blocks):
    """Own and halo rows of each of the scene's blocks: res_ranges and k_pcg_plan restated."""
    n = scene.num_nodes
    rows, cols = host_pairs(scene)
    item_ptr = np.concatenate([[0], np.cumsum(1 + np.bincount(rows, minlength=n))])
    starts = np.minimum(16 * np.arange(-(-n // 16) + 1), n)
    cost = item_ptr[starts] + 4 * starts
    first = np.searchsorted(cost, (int(item_ptr[n]) + 4 * n) * np.arange(blocks + 1) // blocks)
    first[blocks] = len(starts) - 1
    if (np.diff(first) > 32).any():
        first = (len(starts) - 1) * np.arange(blocks + 1) // blocks
    r = starts[first]
    out = []
    for a, b in zip(r[:-1], r[1:]):
        c = cols[(rows >= a) & (rows < b)]
        out.append(b - a + len(np.unique(c[c >= b])))
    return np.array(out)


FITS = (228864 - (32 * 512 + 4 * 4608 + 64)) // 48   # vector rows that fit beside the product records and the ring


def solve(items, gn, pcg, form):
    import torch
    from starhub_b200.solver import WarpSolver
    s = WarpSolver(max_nodes=sum(d.num_nodes for d in items), max_pixels=sum(d.num_pixels for d in items),
                   max_edges=sum(d.num_edges for d in items), max_scenes=len(items))
    s.set_pcg_form(form)
    s.SetBatchInputs(items)
    s.SolveStreamed(gn, pcg, stream=torch.cuda.Stream())
    s.Sync()
    assert s.pcg_form() == form
    return s


# scenes x nodes, pixels a node: on the grid a few blocks of each scene have more vector rows than fit; `many` is past
# the batch size where k_pcg takes over
@pytest.mark.parametrize("scenes,nodes,touches,many", [(16, 4500, 8, 36), (4, 8000, 11, 22)])
def test_grid_blocks_that_do_not_all_fit(ws, scenes, nodes, touches, many):
    a = random_scene(nodes, touches)
    blocks = (148 - scenes) // scenes + 1
    v = vector_rows(a, blocks)
    assert (v > FITS).any() and (v <= FITS).any(), (v.max(), v.min())
    few, k_pcg = solve([a] * scenes, 2, 8, 3), solve([a] * many, 2, 8, 1)
    want = k_pcg.SolvedNodeSE3(0).cpu().numpy()
    assert np.isfinite(want).all() and np.abs(want - np.float32([0, 0, 0, 1, 0, 0, 0, 0])).max() > 1e-6
    for i in range(scenes):
        np.testing.assert_array_equal(few.SolvedNodeSE3(i).cpu().numpy(), want)


# What a block keeps in shared memory and what it leaves outside, by its budget: at 49152 bytes next to nothing fits
# (products one item a thread, a ring of four or five buffers, vectors, contributions, words, send lists and
# inverses in L2), at 228864 everything of the small scenes.
BUDGETS = (49152, 65536, 100000, 160000, 0)


def compare_forms(items, gn, pcg, precision, forms):
    """Every form and budget against k_pcg, scene by scene."""
    import torch
    from starhub_b200 import _lib
    from starhub_b200.solver import WarpSolver
    s = WarpSolver(max_nodes=sum(d.num_nodes for d in items), max_pixels=sum(d.num_pixels for d in items),
                   max_edges=sum(d.num_edges for d in items), max_scenes=len(items), precision=precision)
    s.SetBatchInputs(items)
    want = None
    for form, budget in [(_lib.WS_PCG_STREAMED, 0)] + [(f, b) for f in forms for b in BUDGETS]:
        s.set_pcg_form(form, budget)
        assert s.pcg_form() == form
        s.SolveStreamed(gn, pcg, stream=torch.cuda.Stream())
        s.Sync()
        got = [s.SolvedNodeSE3(i).cpu().numpy().copy() for i in range(len(items))]
        if want is None:
            want = got
            assert all(np.isfinite(g).all() for g in got)
        for i, (a, b) in enumerate(zip(want, got)):
            np.testing.assert_array_equal(a, b, err_msg=f"form {form}, {budget} bytes, scene {i}")


# one group; a partial group; more than 256 rows a cluster block (a thread a row); 512 rows a block; random and band
@pytest.mark.parametrize("nodes,touches,pcg,precision", [
    (16, 3, 3, 0), (37, 2, 4, 1), (900, 8, 1, 0), (900, 8, 0, 0), (2500, 3, 6, 0), (2500, 12, 5, 1), (4200, 6, 4, 0),
    (8192, 2, 3, 0)])
def test_one_scene_in_every_layout(ws, nodes, touches, pcg, precision):
    compare_forms([random_scene(nodes, touches, seed=nodes)], 2, pcg, precision, (2, 3))


# on the grid: many rows a block (up to 512), blocks of very different lengths, the equal split of the groups; as
# clusters: more scenes than run at once
@pytest.mark.parametrize("sizes,touches,pcg,precision", [
    ([4500] * 9 + [300, 17, 4500], 5, 5, 0), ([8000, 1200, 8000, 40], 9, 4, 1), ([3000, 2000] * 5, 10, 7, 0)])
def test_batches_in_every_layout(ws, sizes, touches, pcg, precision):
    by_size = {n: random_scene(n, touches, seed=n) for n in set(sizes)}
    compare_forms([by_size[n] for n in sizes], 2, pcg, precision, (2, 3))
