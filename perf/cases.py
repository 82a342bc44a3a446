"""What a program built on this library has it do, as cases that can be timed and checked.

A depth-camera reconstruction runs, per frame: the measurement maps of the depth image, the render maps
of the model's surfels, the warp-field solve, and the forward warp of the surfels; when the model grows,
it adds nodes, rebuilds the node graph and skins the surfels.  A server solves many such frames as one
batch.  The cases cover each of these through the public entry points (the solver class, and the C ABI
on device pointers), from a lone small frame to a batch of 64 scenes.

Scenes are the synthetic ones of the benchmark: a torus (or the union of torus, sphere and bumpy plane)
in front of a pinhole camera at the origin, sampled into surfels, deformed by a smooth warp, with depth
noise and, for the union, optical flow with outliers.  They are made on the GPU from the seed.
"""
import ctypes as C
import math

import numpy as np
import torch

from starhub_b200 import _lib, scenes
from starhub_b200.solver import DeviceScene, WarpSolver

DEV = "cuda"
R_NODE = scenes.NODE_RADIUS


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest frame: few nodes, the reference's own graph and iteration counts (launches count)
        dict(name="frame_500", kind="solve", scene="torus", nodes=500, width=640, height=480, graph_k=4, gn=6, pcg=10),
        # the plain configuration: 200k surfels, about 1.8k nodes, 8-NN graph
        dict(name="frame_1800", kind="solve", scene="torus", nodes=1800, width=640, height=480, graph_k=8, gn=5, pcg=20),
        # a large model in one lone frame, at an odd image size
        dict(name="frame_8000", kind="solve", scene="torus", nodes=8000, width=847, height=479, graph_k=8, gn=5, pcg=20),
        # 1280x720 with the optical-flow term (the three-channel records)
        dict(name="frame_flow_720p", kind="solve", scene="union", nodes=3000, width=1280, height=720, graph_k=4, gn=5,
             pcg=30),
        # a server's batch: 64 scenes, nodes spread over [500, 8000], one graph replay
        dict(name="batch_64", kind="batch", scenes=64, lo=500, hi=8000, width=640, height=480, graph_k=8, gn=5, pcg=20),
        # a depth frame into vertex and normal maps
        dict(name="measure_480p", kind="measure", width=640, height=480),
        # render tail of a frame: warp every surfel, then draw the solver maps
        dict(name="warp_render_300k", kind="warp_render", surfels=300_001, nodes=1800, width=640, height=480),
        # skinning of a whole model: the plain one, and a large one
        dict(name="skin_200k", kind="skin", surfels=200_000, nodes=1800),
        dict(name="skin_1200k", kind="skin", surfels=1_200_000, nodes=8000),
        # surfels and nodes appended in a frame: only the new rows are skinned (the smallest call)
        dict(name="skin_appended", kind="skin_inc", surfels=3001, nodes=1800, appended=40),
        # node construction and the node graph of a plain model, and of a large fine one
        dict(name="nodes_200k", kind="nodes", surfels=200_000, nodes=1800, graph_k=8),
        dict(name="nodes_1m", kind="nodes", surfels=1_000_000, nodes=26_000, graph_k=8),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solve", "solve", "solve", "batch", "measure", "warp_render", "skin", "skin_inc", "nodes"])
    k = rng.choice([4, 8])
    if kind == "solve":
        flow = rng.random() < 0.3
        width = rng.randint(960, 1280) if flow else rng.randint(480, 960)
        return dict(kind=kind, scene="union" if flow else "torus", nodes=log_int(1500, 5000) if flow else log_int(500, 8000),
                    width=width, height=rng.randint(int(0.55 * width), int(0.76 * width)), graph_k=k,
                    gn=rng.randint(3, 6), pcg=rng.randint(10, 30 if flow else 20))
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(3, 40), lo=log_int(500, 1000), hi=log_int(2000, 8000), width=640,
                    height=480, graph_k=k, gn=5, pcg=rng.randint(10, 20))
    if kind == "measure":
        width = rng.randint(320, 1280)
        return dict(kind=kind, width=width, height=rng.randint(int(0.55 * width), int(0.76 * width)))
    if kind == "warp_render":
        width = rng.randint(480, 1280)
        return dict(kind=kind, surfels=log_int(50_000, 1_200_000), nodes=log_int(500, 8000), width=width,
                    height=rng.randint(int(0.55 * width), int(0.76 * width)))
    if kind == "skin":
        n = log_int(500, 8000)
        return dict(kind=kind, surfels=n * rng.randint(80, 150), nodes=n)
    if kind == "skin_inc":
        return dict(kind=kind, surfels=log_int(300, 30_000), nodes=log_int(500, 8000), appended=rng.randint(8, 200))
    n = log_int(500, 26_000)
    return dict(kind=kind, surfels=min(1_000_000, n * rng.randint(60, 130)), nodes=n, graph_k=k)


# ---------------------------------------------------------------------------
# scenes on the GPU
# ---------------------------------------------------------------------------
def _ptr(t):
    return None if t is None else C.c_void_p(t.data_ptr())


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _call(name, *args):
    _lib.check(getattr(_lib.load(), name)(*args), name)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 13)


def _rand(g, n, lo=0.0, hi=1.0):
    return torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * (hi - lo) + lo


def _rot_x(p, deg):
    return p @ torch.tensor(scenes.rot_x(deg).T, device=DEV)


def _torus(g, n, R, r):
    """Area-uniform samples: points and outward normals."""
    u, v = _rand(g, 2 * n + 64, 0, 2 * math.pi), _rand(g, 2 * n + 64, 0, 2 * math.pi)
    keep = _rand(g, 2 * n + 64) < (R + r * torch.cos(v)) / (R + r)
    u, v = u[keep][:n], v[keep][:n]
    p = torch.stack([(R + r * v.cos()) * u.cos(), (R + r * v.cos()) * u.sin(), r * v.sin()], 1)
    return p, torch.stack([v.cos() * u.cos(), v.cos() * u.sin(), v.sin()], 1)


def _surface(g, kind, nodes, surfels):
    """Surfels of a scene whose node construction yields about 1.04 x `nodes` nodes: (positions, normals), (S, 4)."""
    if kind == "torus":
        s = math.sqrt(nodes / 1550.0)
        p, n = _torus(g, surfels, 0.30 * s, 0.10 * s)
        p, n = _rot_x(p, 30.0), _rot_x(n, 30.0)
        p[:, 2] += s
    else:   # torus, sphere and bumpy plane side by side
        s = math.sqrt(nodes / 2730.0)
        a, b = int(0.45 * surfels), int(0.30 * surfels)
        c = surfels - a - b
        pt, nt = _torus(g, a, 0.30, 0.10)
        pt, nt = _rot_x(pt, 30.0), _rot_x(nt, 30.0)
        ns = torch.randn(b, 3, generator=g, device=DEV, dtype=torch.float64)
        ns = ns / ns.norm(dim=1, keepdim=True)
        kx, ky = (torch.randn(48, generator=g, device=DEV, dtype=torch.float64) / 0.05 for _ in range(2))
        ph, amp = _rand(g, 48, 0, 2 * math.pi), 0.005 / math.sqrt(24.0)
        x, y = _rand(g, c, -0.3, 0.3), _rand(g, c, -0.3, 0.3)
        arg = x[:, None] * kx + y[:, None] * ky + ph
        pp = torch.stack([x, y, amp * arg.sin().sum(1)], 1)
        npl = torch.stack([amp * (arg.cos() * kx).sum(1), amp * (arg.cos() * ky).sum(1), -torch.ones_like(x)], 1)
        pp, npl = _rot_x(pp, -20.0), _rot_x(npl / npl.norm(dim=1, keepdim=True), -20.0)
        at = torch.tensor([[-0.32, -0.05, 1.1], [0.35, 0.05, 0.95], [0.0, 0.1, 1.45]], device=DEV, dtype=torch.float64)
        p = s * torch.cat([pt + at[0], 0.2 * ns + at[1], pp + at[2]])
        n = torch.cat([nt, ns, npl])
    one = torch.ones(len(p), 1, device=DEV, dtype=torch.float64)
    return torch.cat([p, one], 1).float().contiguous(), torch.cat([n, 0.002 * one], 1).float().contiguous()


def _init_nodes(surfels, radius, out=None):
    """The nodes, in the first rows of `out` (host memory)."""
    if out is None:
        out = np.empty((len(surfels) + 2, 4), np.float32)
    n = C.c_int()
    _call("ws_init_nodes", _ptr(surfels), len(surfels), radius, out.ctypes.data, len(out), C.byref(n), _stream())
    return out[: n.value]


def _graph_buffers(n, k):
    return (torch.zeros((n, k), dtype=torch.int16, device=DEV), torch.zeros((n, k), dtype=torch.float32, device=DEV),
            torch.zeros((n * k, 3), dtype=torch.int16, device=DEV))


def _node_graph(nodes, k, radius, out):
    _call("ws_build_node_graph", _ptr(nodes), len(nodes), k, radius, *map(_ptr, out), _stream())


def _skin_buffers(n):
    return (torch.zeros((n, 4), dtype=torch.int16, device=DEV), torch.zeros((n, 4), dtype=torch.float32, device=DEV),
            torch.zeros((n, 4), dtype=torch.float32, device=DEV))


def _skin(nodes, verts, out):
    _call("ws_skinning", _ptr(nodes), len(nodes), _ptr(verts), len(verts), R_NODE, *map(_ptr, out), _stream())


def _warp(dq, verts, normals, skin, out_v, out_n):
    _call("ws_forward_warp", _ptr(dq), len(dq), _ptr(verts), _ptr(normals), len(verts), *map(_ptr, skin), _ptr(out_v),
          _ptr(out_n), _stream())


def _splat(verts, normals, width, height, focal):
    """Index, vertex and normal maps of camera-frame points, 3x3 pixels a point."""
    idx = torch.empty((height, width), dtype=torch.int32, device=DEV)
    vm, nm = (torch.empty((height, width, 4), dtype=torch.float32, device=DEV) for _ in range(2))
    _call("ws_splat_maps", _ptr(verts), _ptr(verts), _ptr(normals), len(verts), width, height, focal, focal, width / 2.0,
          height / 2.0, 1, _ptr(idx), _ptr(vm), _ptr(nm), _stream())
    return idx, vm, nm


def _model(g, seed, kind, nodes, surfels, max_rot=5.0, max_trans=0.01):
    """A skinned model of `nodes` nodes: surfels, normals, nodes, skinning and a smooth warp of the nodes."""
    sv, sn = _surface(g, kind, nodes, surfels)
    nd = _init_nodes(sv, R_NODE)
    keep = np.sort(np.random.default_rng(seed + 1).permutation(np.arange(2, len(nd)))[: nodes - 2])
    nd = torch.from_numpy(np.concatenate([nd[:2], nd[keep]])).to(DEV)
    skin = _skin_buffers(len(sv))
    _skin(nd, sv, skin)
    pick = sv[torch.randint(len(sv), (64,), generator=g, device=DEV)].cpu().numpy()
    dq = scenes.smooth_warp(np.random.default_rng(seed), nd.cpu().numpy(), pick, max_rot, max_trans)
    return sv, sn, nd, skin, torch.from_numpy(dq).to(DEV)


def _scene(seed, kind, nodes, width, height, graph_k):
    """One frame's solver inputs."""
    g = _gen(seed)
    focal = (570.0 if kind == "torus" else 460.0) * width / 640.0
    surfels = 130 * nodes if kind == "torus" else 400 * nodes
    sv, sn, nd, skin, dq = _model(g, seed, kind, nodes, surfels)
    graph = _graph_buffers(nodes, graph_k)
    _node_graph(nd, graph_k, R_NODE, graph)
    index, ref_v, ref_n = _splat(sv, sn, width, height, focal)
    wv, wn = torch.empty_like(sv), torch.empty_like(sn)
    _warp(dq, sv, sn, skin, wv, wn)
    _, mv, mn = _splat(wv, wn, width, height, focal)
    seen = mv[..., 2] != 0
    noise = 0.001 * torch.randn((height, width), generator=g, device=DEV)
    mv[..., :3] *= torch.where(seen, 1 + noise / mv[..., 2].clamp(min=0.1), 0.0)[..., None]
    mn[..., 3] = torch.where(seen, 0.002, 0.0)
    flow = None
    if kind != "torus":   # correspondences on a 4-pixel grid, half a pixel of noise, one in ten wrong
        flow = torch.zeros((height, width, 2), device=DEV)
        ys, xs = torch.meshgrid(torch.arange(0, height, 4, device=DEV), torch.arange(0, width, 4, device=DEV), indexing="ij")
        ok = index[ys, xs] >= 0
        ys, xs = ys[ok], xs[ok]
        wp = wv[index[ys, xs].long()]
        at = torch.stack([focal * wp[:, 0] / wp[:, 2] + width / 2.0 - xs, focal * wp[:, 1] / wp[:, 2] + height / 2.0 - ys], 1)
        at += 0.5 * torch.randn(at.shape, generator=g, device=DEV)
        wrong = torch.rand(len(xs), generator=g, device=DEV) < 0.1
        far = torch.rand((len(xs), 2), generator=g, device=DEV) * torch.tensor([width, height], device=DEV)
        flow[ys, xs] = torch.where(wrong[:, None], far - torch.stack([xs, ys], 1), at)
    n = len(nd)
    return DeviceScene(
        width=width, height=height, fx=focal, fy=focal, cx=width / 2.0, cy=height / 2.0,
        cam2world=np.eye(4, dtype=np.float32), measure_vertex=mv, measure_normal=mn, reference_vertex=ref_v,
        reference_normal=ref_n, index_map=index, flow=flow, surfel_knn=skin[0], surfel_sw=skin[1], surfel_cw=skin[2],
        nodes=nd, edges=graph[2], graph_k=graph_k, node_cw=torch.ones((n, graph_k), device=DEV),
        node_radius_square=float(np.float32(R_NODE) * np.float32(R_NODE)), lambda_of=0.0 if flow is None else 0.1)


def _batch_scenes(case, seed):
    n, lo, hi = case["scenes"], case["lo"], case["hi"]
    return [_scene(1000 * seed + i, "torus", int(lo * (hi / lo) ** ((i + 0.5) / n)), case["width"], case["height"],
                   case["graph_k"]) for i in range(n)]


# ---------------------------------------------------------------------------
# what a program has in hand, and one pass
# ---------------------------------------------------------------------------
def _solver(items):
    return WarpSolver(max_nodes=sum(s.num_nodes for s in items), max_pixels=sum(s.num_pixels for s in items),
                      max_edges=sum(s.num_edges for s in items), max_scenes=len(items))


def _depth_image(g, width, height):
    """A depth frame in millimetres: a sphere before a slanted wall, sensor noise, dropouts."""
    y, x = torch.meshgrid((torch.arange(height, device=DEV) - height / 2) / width,
                          (torch.arange(width, device=DEV) - width / 2) / width, indexing="ij")
    cx, cy, rad = (float(v) for v in _rand(g, 3, -0.1, 0.1).cpu())
    wall = 1600 + 500 * x + 200 * y + 6 * torch.sin(60 * x) * torch.cos(45 * y)
    d2 = (0.3 + 0.1 * rad) ** 2 - (x - cx) ** 2 - (y - cy) ** 2
    z = torch.where(d2 > 0, 1200 - 800 * d2.clamp(min=0).sqrt(), wall)
    z = z + 1.5 * torch.randn(z.shape, generator=g, device=DEV)
    z[torch.rand(z.shape, generator=g, device=DEV) < 0.03] = 0
    return z.round().to(torch.int16).contiguous()


def prepare(case, seed):
    g, kind = _gen(seed), case["kind"]
    if kind in ("solve", "batch"):
        items = _batch_scenes(case, seed) if kind == "batch" else [
            _scene(seed, case["scene"], case["nodes"], case["width"], case["height"], case["graph_k"])]
        return dict(case=case, items=items, solver=_solver(items), stream=torch.cuda.Stream() if kind == "batch" else None)
    if kind == "measure":
        w, h = case["width"], case["height"]
        return dict(case=case, depth=_depth_image(g, w, h), vertex=torch.empty((h, w, 4), device=DEV),
                    normal=torch.empty((h, w, 4), device=DEV))
    if kind == "warp_render":
        w, h = case["width"], case["height"]
        sv, sn, nd, skin, dq = _model(g, seed, "torus", case["nodes"], case["surfels"])
        sv[:, 3] = torch.rand(len(sv), generator=g, device=DEV) * 3   # confidence: a third is unstable
        ct = torch.zeros_like(sv)
        ct[:, 0] = torch.randint(1 << 24, (len(sv),), generator=g, device=DEV, dtype=torch.int32).view(torch.float32)
        ct[:, 2] = torch.randint(90, 101, (len(sv),), generator=g, device=DEV).float()   # last seen, of frame 100
        p = _lib.WsRenderParams()
        p.width, p.height, p.fx, p.fy, p.cx, p.cy = w, h, 570.0 * w / 640, 570.0 * w / 640, w / 2.0, h / 2.0
        p.world2camera[:] = [float(v) for v in np.eye(4).reshape(-1)]
        p.max_depth, p.current_time, p.confidence_threshold, p.time_threshold, p.footprint = 8.0, 100.0, 1.0, 3.0, 0
        return dict(case=case, verts=sv, normals=sn, skin=skin, dq=dq, color_time=ct, params=p,
                    live=(torch.empty_like(sv), torch.empty_like(sn)),
                    index=torch.empty((h, w), dtype=torch.int32, device=DEV),
                    maps=[torch.empty((h, w, 4), device=DEV) for _ in range(3)])
    if kind == "nodes":
        radius = R_NODE * math.sqrt(1800.0 / case["nodes"])   # the plain torus at a finer grid
        cap = case["nodes"] + case["nodes"] // 4 + 64         # the program's node capacity
        return dict(case=case, radius=radius, surfels=_surface(g, "torus", 1800, case["surfels"])[0],
                    host=np.zeros((cap, 4), np.float32), graph=_graph_buffers(cap, case["graph_k"]))
    if kind == "skin":
        sv, _ = _surface(g, "torus", case["nodes"], case["surfels"])
        return dict(case=case, nodes=torch.from_numpy(_init_nodes(sv, R_NODE).copy()).to(DEV), verts=sv,
                    out=_skin_buffers(len(sv)))
    # skin_inc: surfels appended in a frame, near the surface the nodes grew on; the appended nodes come last
    sv, _ = _surface(g, "torus", case["nodes"], 130 * case["nodes"])
    nd = torch.from_numpy(_init_nodes(sv, R_NODE).copy()).to(DEV)
    order = torch.cat([torch.arange(2, device=DEV), 2 + torch.randperm(len(nd) - 2, generator=g, device=DEV)])
    nd = torch.cat([nd[order[: len(nd) - case["appended"]].sort().values], nd[order[len(nd) - case["appended"]:]]]).contiguous()
    prev = len(nd) - case["appended"]
    verts = sv[: case["surfels"]].contiguous()
    out = _skin_buffers(len(verts))
    _skin(nd[:prev], verts, out)
    return dict(case=case, nodes=nd, prev=prev, verts=verts, before=out[0].clone(), out=out)


def _solved(solver, i):
    t = solver.SolvedNodeSE3(i)
    t.owner = solver   # a view of the solver's memory: whoever holds it holds the solver
    return t


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "solve":      # a frame: new inputs, the solve, its warp
        s["solver"].SetSolverInputs(s["items"][0])
        s["solver"].SolveStreamed(case["gn"], case["pcg"])
        return _solved(s["solver"], 0)
    if kind == "batch":
        here = torch.cuda.current_stream()
        s["stream"].wait_stream(here)
        s["solver"].SetBatchInputs(s["items"])
        s["solver"].SolveStreamed(case["gn"], case["pcg"], stream=s["stream"], graph=True)
        here.wait_stream(s["stream"])
        return [_solved(s["solver"], i) for i in range(len(s["items"]))]
    if kind == "measure":
        w, h = case["width"], case["height"]
        f = 570.0 * w / 640
        _call("ws_measure_maps", _ptr(s["depth"]), w, h, w, f, f, w / 2.0, h / 2.0, 0.1, 3.0, 1.0, _ptr(s["vertex"]),
              _ptr(s["normal"]), _stream())
        return dict(vertex=s["vertex"], normal=s["normal"])
    if kind == "warp_render":
        _warp(s["dq"], s["verts"], s["normals"], s["skin"], *s["live"])
        _call("ws_render_solver_maps", _ptr(s["live"][0]), _ptr(s["live"][1]), _ptr(s["color_time"]), len(s["verts"]),
              C.byref(s["params"]), _ptr(s["index"]), *map(_ptr, s["maps"]), _stream())
        return dict(live_vertex=s["live"][0], live_normal=s["live"][1], index=s["index"], vertex=s["maps"][0],
                    normal=s["maps"][1], rgbd=s["maps"][2])
    if kind == "nodes":
        nodes = _init_nodes(s["surfels"], s["radius"], s["host"])
        _node_graph(torch.from_numpy(nodes).to(DEV), case["graph_k"], s["radius"], s["graph"])
        return dict(count=len(nodes), nodes=s["host"], knn=s["graph"][0], weights=s["graph"][1], edges=s["graph"][2])
    if kind == "skin":
        _skin(s["nodes"], s["verts"], s["out"])
        return dict(knn=s["out"][0], weights=s["out"][1], connect=s["out"][2])
    s["out"][0].copy_(s["before"])   # the neighbours among the earlier nodes, as the frame has them
    _call("ws_skinning_incremental", _ptr(s["nodes"]), None, len(s["nodes"]), s["prev"], _ptr(s["verts"]),
          len(s["verts"]), 0, R_NODE, 1, *map(_ptr, s["out"]), _stream())
    return dict(knn=s["out"][0], weights=s["out"][1], connect=s["out"][2])


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------
def _solve_work(kind, nodes, width, height, k, gn, pcg):
    terms = (0.42 if kind == "torus" else 0.40) * width * height   # pixels that show a surfel
    channels, blocks = (1, 6.3 * nodes) if kind == "torus" else (3, 6.0 * nodes)   # stored 6x6 blocks
    bytes_ = 4 * width * height + terms * (64 + 40 + (0 if kind == "torus" else 8)) + nodes * (16 + 32 + 10 * k)
    per_term = 250 + channels * (21 * 2 + 10 * 2 * 21 + 4 * 12)
    flops = gn * (terms * per_term + nodes * k * 3 * 150 + pcg * (2 * 72 * blocks + 150 * nodes))
    return bytes_, flops


def work(case):
    kind = case["kind"]
    if kind == "solve":
        b, f = _solve_work(case["scene"], case["nodes"], case["width"], case["height"], case["graph_k"], case["gn"], case["pcg"])
    elif kind == "batch":
        n, lo, hi = case["scenes"], case["lo"], case["hi"]
        per = [_solve_work("torus", lo * (hi / lo) ** ((i + 0.5) / n), case["width"], case["height"], case["graph_k"],
                           case["gn"], case["pcg"]) for i in range(n)]
        b, f = sum(p[0] for p in per), sum(p[1] for p in per)
    elif kind == "measure":
        b, f = case["width"] * case["height"] * (2 + 32), case["width"] * case["height"] * 1100
    elif kind == "warp_render":
        b = case["surfels"] * (40 + 32 + 32 + 16) + case["width"] * case["height"] * (4 + 48)
        f = case["surfels"] * 300
    elif kind == "nodes":
        b, f = case["surfels"] * 16 + case["nodes"] * (32 + 12 * case["graph_k"]), case["surfels"] * 30 + case["nodes"] * 1000
    elif kind == "skin":
        b, f = case["surfels"] * (16 + 40) + case["nodes"] * 16, case["surfels"] * 300
    else:
        b, f = case["surfels"] * (16 + 8 + 40) + case["nodes"] * 16, case["surfels"] * case["appended"] * 8
    return {"bytes": int(b), "flops": int(f)}


# ---------------------------------------------------------------------------
# the same values in 64 bits, by plain torch
# ---------------------------------------------------------------------------
def _qmul(a, b):
    ax, ay, az, aw = a.unbind(-1)
    bx, by, bz, bw = b.unbind(-1)
    return torch.stack([aw * bx + ax * bw + ay * bz - az * by, aw * by - ax * bz + ay * bw + az * bx,
                        aw * bz + ax * by - ay * bx + az * bw, aw * bw - ax * bx - ay * by - az * bz], -1)


def _dq_normalized(dq):
    q0, q1 = dq[..., :4], dq[..., 4:]
    n = q0.norm(dim=-1, keepdim=True)
    q0, q1 = q0 / n, q1 / n
    return q0, q1 - (q0 * q1).sum(-1, keepdim=True) * q0


def _dq_rt(dq):
    """Rotation matrices and translations of dual quaternions."""
    q0, q1 = _dq_normalized(dq)
    x, y, z, w = q0.unbind(-1)
    R = torch.stack([1 - 2 * y * y - 2 * z * z, 2 * x * y - 2 * z * w, 2 * x * z + 2 * y * w,
                     2 * x * y + 2 * z * w, 1 - 2 * x * x - 2 * z * z, 2 * y * z - 2 * x * w,
                     2 * x * z - 2 * y * w, 2 * y * z + 2 * x * w, 1 - 2 * x * x - 2 * y * y], -1)
    t = _qmul(2 * q1, q0 * torch.tensor([-1.0, -1, -1, 1], device=q0.device, dtype=q0.dtype))[..., :3]
    return R.reshape(*R.shape[:-1], 3, 3), t


def _ids(knn):
    return knn.long() & 0xFFFF


def _apply(R, v):
    return (R @ v[..., None])[..., 0]


def _axis_angle(w):
    """Rotation matrices of rotation vectors; the identity where they are tiny, as the solver has it."""
    a = w.norm(dim=-1).clamp(min=1e-30)
    k = w / a[..., None]
    c, s = a.cos()[..., None, None], a.sin()[..., None, None]
    zero = torch.zeros_like(a)
    K = torch.stack([zero, -k[..., 2], k[..., 1], k[..., 2], zero, -k[..., 0], -k[..., 1], k[..., 0], zero], -1)
    eye = torch.eye(3, device=w.device, dtype=w.dtype)
    R = eye * c + s * K.reshape(*a.shape, 3, 3) + (1 - c) * k[..., :, None] * k[..., None, :]
    return torch.where((w.abs().sum(-1) < 1e-4)[..., None, None], eye, R)


def _rt_dq(R, t):
    s = torch.sqrt(R[:, 0, 0] + R[:, 1, 1] + R[:, 2, 2] + 1) * 2   # rotations well below a half turn
    q0 = torch.stack([(R[:, 2, 1] - R[:, 1, 2]) / s, (R[:, 0, 2] - R[:, 2, 0]) / s, (R[:, 1, 0] - R[:, 0, 1]) / s, s / 4], 1)
    return torch.cat([q0, _qmul(torch.cat([0.5 * t, torch.zeros_like(t[:, :1])], 1), q0)], 1)


def _exact_solve(s, gn, pcg):
    """Gauss-Newton with block-Jacobi PCG on the scene, matrix-free, twists about the origin."""
    f8, N = torch.float64, s.num_nodes
    index = s.index_map.long()
    ys, xs = torch.nonzero((index >= 0) & (index < len(s.surfel_knn)), as_tuple=True)
    sid = index[ys, xs]
    knn, wk = _ids(s.surfel_knn)[sid], s.surfel_sw[sid].to(f8) * s.surfel_cw[sid].to(f8)
    cv, cn = s.reference_vertex[ys, xs, :3].to(f8), s.reference_normal[ys, xs, :3].to(f8)
    tx, ty = xs, ys
    if s.flow is not None:
        to = (s.flow[ys, xs] + torch.stack([xs, ys], 1).float()).round().clamp(min=0).long()
        tx, ty = to[:, 0], to[:, 1]
    inside = (tx < s.width) & (ty < s.height)
    tx, ty = tx.clamp(max=s.width - 1), ty.clamp(max=s.height - 1)
    tv, tn = s.measure_vertex[ty, tx, :3].to(f8), s.measure_normal[ty, tx, :3].to(f8)
    inside &= ~(tv.abs() < 1e-3).all(1)
    lam = [s.lambda_depth] + ([s.lambda_of] * 2 if s.lambda_of != 0 else [])
    lam2 = torch.tensor(np.float32(lam).astype(np.float64) ** 2, device=DEV)
    ei, ej, ek = _ids(s.edges).unbind(1)
    far = ((s.nodes[ei, :3] - s.nodes[ej, :3]) ** 2).sum(1) > 64 * s.node_radius_square
    use = (ei != ej) & ~far
    ei, ej, ek = ei[use], ej[use], ek[use]
    er = float(np.float32(s.lambda_reg)) * s.node_cw[ei, ek].to(f8)
    xj = s.nodes[ej, :3].to(f8)
    dq = torch.zeros((N, 8), device=DEV, dtype=f8)
    dq[:, 3] = 1
    eye6, eye3 = torch.eye(6, device=DEV, dtype=f8), torch.eye(3, device=DEV, dtype=f8)

    def reg_rows(p):   # d(T x)/d(twist) = [-[p]x, I]
        z = torch.zeros_like(p[:, 0])
        m = torch.stack([z, p[:, 2], -p[:, 1], -p[:, 2], z, p[:, 0], p[:, 1], -p[:, 0], z], -1).reshape(-1, 3, 3)
        return torch.cat([m, eye3.expand_as(m)], 2)

    for _ in range(gn):
        R, t = _dq_rt((wk[..., None] * dq[knn]).sum(1))
        vw, nw = _apply(R, cv) + t, _apply(R, cn)
        ok = inside & ((tn * nw).sum(1) >= 0.7) & ((tv[:, 2] - vw[:, 2]).abs() <= 0.03)
        diff = vw - tv
        dirs, res = [tn], [(tn * diff).sum(1)]
        if len(lam) == 3:
            moved = (diff[:, 0] ** 2 + diff[:, 1] ** 2).sqrt() >= 1e-6
            for c in range(2):
                dirs.append(torch.where(moved[:, None], eye3[c], 0.0))
                res.append(torch.where(moved, diff[:, c], 0.0))
        G = torch.stack([torch.cat([torch.linalg.cross(vw, d), d], 1) for d in dirs], 1) * ok[:, None, None]   # (T, C, 6)
        r = torch.stack(res, 1) * ok[:, None]
        Rn, tn_ = _dq_rt(dq)
        a, b = _apply(Rn[ei], xj) + tn_[ei], _apply(Rn[ej], xj) + tn_[ej]
        Ji, Jj, e_res = er[:, None, None] * reg_rows(a), -er[:, None, None] * reg_rows(b), er[:, None] * (a - b)

        rhs = torch.zeros((N, 6), device=DEV, dtype=f8)
        D = 1e-3 * eye6.repeat(N, 1, 1)
        gg = torch.einsum("c,tca,tcb->tab", lam2, G, G)
        gr = torch.einsum("c,tc,tca->ta", lam2, r, G)
        for k in range(4):
            rhs.index_add_(0, knn[:, k], -wk[:, k, None] ** 2 * gr)
            D.index_add_(0, knn[:, k], wk[:, k, None, None] ** 2 * gg)
        for node, J in ((ei, Ji), (ej, Jj)):
            rhs.index_add_(0, node, -(J * e_res[..., None]).sum(1))
            D.index_add_(0, node, J.transpose(1, 2) @ J)
        M = torch.linalg.inv(D)

        def product(v):
            u = torch.einsum("tca,ta,c->tc", G, (wk[..., None] * v[knn]).sum(1), lam2)
            y, out = torch.einsum("tc,tca->ta", u, G), 1e-3 * v
            for k in range(4):
                out.index_add_(0, knn[:, k], wk[:, k, None] * y)
            e = _apply(Ji, v[ei]) + _apply(Jj, v[ej])
            out.index_add_(0, ei, (Ji * e[..., None]).sum(1))
            out.index_add_(0, ej, (Jj * e[..., None]).sum(1))
            return out

        x, rr = torch.zeros_like(rhs), rhs
        z = _apply(M, rr)
        d, delta = z, (rr * z).sum()
        for _ in range(pcg):
            q = product(d)
            alpha = delta / (d * q).sum()
            x, rr = x + alpha * d, rr - alpha * q
            z = _apply(M, rr)
            new = (rr * z).sum()
            d, delta = z + (new / delta) * d, new
        Ri = _axis_angle(x[:, :3])
        dq = _rt_dq(Ri @ Rn, _apply(Ri, tn_) + x[:, 3:])
    return dq


def _exact_measure(depth, width, height):
    f = 570.0 * width / 640
    z = depth.double() / 1000
    keep = (z >= 0.1) & (z <= 3.0)
    y, x = torch.meshgrid(torch.arange(height, device=DEV).double(), torch.arange(width, device=DEV).double(), indexing="ij")
    p = torch.where(keep[..., None], torch.stack([(x - width / 2.0) / f * z, (y - height / 2.0) / f * z, z], -1), 0.0)
    vertex = torch.cat([p, keep[..., None].double()], -1)
    pad = torch.zeros((height + 6, width + 6, 4), device=DEV, dtype=torch.float64)
    pad[3:-3, 3:-3, :3], pad[3:-3, 3:-3, 3] = p, keep.double()   # every kept depth is at least 0.1 m
    win = [(dy, dx) for dy in range(7) for dx in range(7)]
    s = sum(pad[dy:dy + height, dx:dx + width] for dy, dx in win)
    use = keep & (s[..., 3] > 24)
    mean = s[..., :3] / s[..., 3:].clamp(min=1)
    cov = torch.zeros((height, width, 3, 3), device=DEV, dtype=torch.float64)
    for dy, dx in win:
        if dy < 6 and dx < 6:   # the reference's covariance window leaves out the last row and column
            q = pad[dy:dy + height, dx:dx + width]
            e = (q[..., :3] - mean) * q[..., 3:]
            cov += e[..., :, None] * e[..., None, :]
    flat = cov[use].cpu()
    n = torch.linalg.eigh(flat)[1][:, :, 0].to(DEV)
    n = torch.where(((n * p[use]).sum(1) >= 0)[:, None], -n, n)
    rad = p[use][:, 2] * (1000 * 1.414 / 570.0)
    nz = n[:, 2].abs()
    rad = torch.where(nz > 0.5, rad / nz, 2 * rad)
    normal = torch.zeros((height, width, 4), device=DEV, dtype=torch.float64)
    normal[use] = torch.cat([n, rad[:, None]], 1)
    return dict(vertex=vertex, normal=normal)


def _nearest(verts, nodes, k, half=False):
    """Squared distances of each point's k nearest nodes, ascending (rounded to half precision first if asked)."""
    out = []
    for p in verts[:, :3].double().split(max(1, (1 << 27) // len(nodes))):
        d = sum((p[:, None, c] - nodes[None, :, c].double()) ** 2 for c in range(3))
        out.append((d.half().double() if half else d).topk(k, dim=1, largest=False, sorted=True)[0])
    return torch.cat(out)


def _weights(d2, radius):
    w = torch.exp(-d2 / (2 * float(np.float32(radius) * np.float32(radius))))
    return w / w.sum(1, keepdim=True)


def exact(case, seed):
    kind = case["kind"]
    s = prepare(case, seed)
    if kind == "solve":
        return _exact_solve(s["items"][0], case["gn"], case["pcg"])
    if kind == "batch":
        return [_exact_solve(x, case["gn"], case["pcg"]) for x in s["items"]]
    if kind == "measure":
        return _exact_measure(s["depth"], case["width"], case["height"])
    if kind == "warp_render":
        q0, q1 = _dq_normalized(s["dq"].double()[_ids(s["skin"][0])])
        w = (s["skin"][1].double() * s["skin"][2].double())[..., None]
        R, t = _dq_rt(torch.cat([(w * q0).sum(1), (w * q1).sum(1)], 1))
        v, n = s["verts"].double(), s["normals"].double()
        # the maps are copies of the drawn surfel's values: which surfel that is, is no rounded number
        return dict(live_vertex=torch.cat([_apply(R, v[:, :3]) + t, v[:, 3:]], 1),
                    live_normal=torch.cat([_apply(R, n[:, :3]), n[:, 3:]], 1), index=None, vertex=None, normal=None,
                    rgbd=None)
    if kind == "nodes":
        nodes = torch.from_numpy(_init_nodes(s["surfels"], s["radius"], s["host"])).to(DEV)   # a selection of the inputs
        w = torch.zeros(s["graph"][1].shape, device=DEV, dtype=torch.float64)
        w[: len(nodes)] = _weights(_nearest(nodes, nodes, case["graph_k"], half=True), s["radius"])
        return dict(count=None, nodes=None, knn=None, weights=w, edges=None)
    w = _weights(_nearest(s["verts"], s["nodes"], 4), R_NODE)
    return dict(knn=None, weights=w, connect=torch.ones_like(w))
