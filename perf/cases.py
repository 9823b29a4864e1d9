"""Workloads of the graph-cut framework, through its public entry points.

Every case is a dict of plain values; ``prepare`` makes its inputs (seeded, on
the GPU), ``run`` makes one call or one short chain of calls the way a user's
program does.  The cell graphs are jittered Kuhn lattices in Morton order (the
benchmark's own stand-in for a spatially sorted Delaunay tetrahedralization)
around the meshes the framework's workloads use: a holed sphere, a holed
torus, an open rounded box and a defective (3,5) torus-knot tube.  Tets whose
centroid lies within 0.8 lattice spacings of the surface are labelled 0.

Operations ("op"):
  cut      one graph cut; "host": vertices and labels come and go as host
           arrays through the drop-in module, else all arrays are in HBM
  batch    many graphs cut in one call, arrays in HBM
  raw      an integer-capacity graph given as rows (no reduction)
  surface  the oriented cut surface, drop-in module (host labels and vertices)
  audit    edge-degree watertight audit of a mesh in HBM
  labels   tet-centroid labels from a sparse distance grid, arrays in HBM
  upload   host topology matrix to the int32 device layout
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parents[1] / "wtivo-watertightvoxel_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import gpupr_capi as capi  # noqa: E402
import wtivo_gpupr  # noqa: E402

DEV = torch.device("cuda" if torch.cuda.is_available() else "cpu")
# tet p of a cube walks the axes PERM[p] from the cube's low to its high corner
PERM = [(0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)]
MESHES = ("sphere", "torus", "box", "knot")
# local vertices of face slot k, the vertex opposite to it is 3 - k
FACES = [(0, 1, 2), (0, 1, 3), (0, 2, 3), (1, 2, 3)]


def listed():
    return [
        # one small part remeshed interactively: latency, host arrays in and out
        {"name": "cut_host_60k", "op": "cut", "mesh": "torus", "tets": 60_000, "fill": 10.0, "host": True},
        # an ordinary mid-size part through the drop-in module
        {"name": "cut_host_900k", "op": "cut", "mesh": "box", "tets": 900_000, "fill": 10.0, "host": True},
        # the size of a 500k-point proxy, the pipeline's usual single cut
        {"name": "cut_host_3m", "op": "cut", "mesh": "sphere", "tets": 3_200_000, "fill": 10.0, "host": True},
        # a large open part, arrays already in HBM
        {"name": "cut_dev_8m", "op": "cut", "mesh": "box", "tets": 8_000_000, "fill": 10.0, "host": False},
        # the benchmark: the cell graph of a 12M-point proxy
        {"name": "cut_dev_80m", "op": "cut", "mesh": "knot", "tets": 80_000_000, "fill": 10.0, "host": False},
        # offline processing of a parts library: 64 uneven graphs in one call
        {"name": "batch_64", "op": "batch", "count": 64, "lo": 50_000, "hi": 4_000_000, "fill": 10.0},
        # integer graphs that do not come from the reduction, small and large
        {"name": "raw_200k", "op": "raw", "tets": 200_000, "nlink": 30.0},
        {"name": "raw_12m", "op": "raw", "tets": 11_700_000, "nlink": 10_000.0},
        # the mesh of a finished cut
        {"name": "surface_8m", "op": "surface", "mesh": "knot", "tets": 8_000_000},
        # the audit of a large finished mesh
        {"name": "audit_5m", "op": "audit", "faces": 5_240_000},
        # the initial labels of a large graph
        {"name": "labels_24m", "op": "labels", "mesh": "knot", "tets": 24_000_000},
        # a tetrahedralizer's topology (column-major 64-bit) onto the GPU
        {"name": "upload_3m", "op": "upload", "tets": 3_200_000, "bits": 64, "order": "F"},
    ]


def _between(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    op = rng.choice(("cut", "cut", "cut", "cut", "batch", "raw", "surface", "audit", "labels", "upload"))
    if op == "cut":
        host = rng.random() < 0.5
        return {"op": op, "mesh": rng.choice(MESHES), "tets": _between(rng, 4e4, 8e6 if host else 6e7),
                "fill": rng.choice((5.0, 10.0, 10.0, 20.0)), "host": host}
    if op == "batch":
        return {"op": op, "count": rng.randint(3, 60), "lo": 50_000, "hi": _between(rng, 2e5, 4e6), "fill": 10.0}
    if op == "raw":
        return {"op": op, "tets": _between(rng, 5e4, 1.1e7), "nlink": rng.choice((30.0, 300.0, 10_000.0))}
    if op == "audit":
        return {"op": op, "faces": _between(rng, 2e4, 5.2e6)}
    if op == "upload":
        return {"op": op, "tets": _between(rng, 1e5, 8e6), "bits": rng.choice((32, 64)),
                "order": rng.choice(("C", "F"))}
    top = 8e6 if op == "surface" else 3e7
    return {"op": op, "mesh": rng.choice(MESHES), "tets": _between(rng, 1e5, top)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _spread3(v):
    v = v.to(torch.int64)
    for s, m in ((32, 0x1F00000000FFFF), (16, 0x1F0000FF0000FF), (8, 0x100F00F00F00F00F),
                 (4, 0x10C30C30C30C30C3), (2, 0x1249249249249249)):
        v = (v | (v << s)) & m
    return v


def _lattice(shape, lo, hi, gen, jitter=0.15):
    """Jittered Kuhn lattice: vertices f64 [nv,3], tets and neighbors int32
    [6*cubes,4], cubes in Morton order, neighbor slot k across face FACES[k]."""
    nx, ny, nz = shape
    vx, vy, vz = nx + 1, ny + 1, nz + 1
    h = [(hi[k] - lo[k]) / shape[k] for k in range(3)]
    grid = torch.meshgrid(*(torch.arange(n, device=DEV, dtype=torch.float64) for n in (vz, vy, vx)), indexing="ij")
    V = torch.empty((vz, vy, vx, 3), dtype=torch.float64, device=DEV)
    for k, n in enumerate((vx, vy, vz)):
        g = grid[2 - k]
        j = (torch.rand((vz, vy, vx), generator=gen, device=DEV, dtype=torch.float64) - 0.5) * (2.0 * jitter)
        V[..., k] = lo[k] + (g + j * ((g > 0) & (g < n - 1))) * h[k]   # hull vertices stay on their faces
    C = nx * ny * nz
    c = torch.arange(C, device=DEV, dtype=torch.int32)
    x, y, z = c % nx, (c // nx) % ny, c // (nx * ny)
    code = _spread3(x) | (_spread3(y) << 1) | (_spread3(z) << 2)
    order = torch.argsort(code)
    rank = torch.empty(C, dtype=torch.int32, device=DEV)
    rank[order] = c
    pos = [t[order] for t in (x, y, z)]
    del code, x, y, z
    stride, cube_step = (1, vx, vx * vy), (1, nx, nx * ny)
    v0 = pos[0] + vx * (pos[1] + vy * pos[2])
    minus, plus = [], []
    for k, n in enumerate(shape):
        lo_ok, hi_ok = pos[k] > 0, pos[k] < n - 1
        minus.append(torch.where(lo_ok, rank[(order - cube_step[k]).clamp_(min=0)] * 6, -8))
        plus.append(torch.where(hi_ok, rank[(order + cube_step[k]).clamp_(max=C - 1)] * 6, -8))
    tets = torch.empty((C, 6, 4), dtype=torch.int32, device=DEV)
    nbrs = torch.empty((C, 6, 4), dtype=torch.int32, device=DEV)
    own = c * 6
    for p, (a, b, d) in enumerate(PERM):
        step = 0
        tets[:, p, 0] = v0
        for k, axis in enumerate((a, b, d)):
            step += stride[axis]
            tets[:, p, k + 1] = v0 + step
        nbrs[:, p, 0] = (minus[d] + PERM.index((d, a, b))).clamp_(min=-1)
        nbrs[:, p, 1] = own + PERM.index((a, d, b))
        nbrs[:, p, 2] = own + PERM.index((b, a, d))
        nbrs[:, p, 3] = (plus[a] + PERM.index((b, d, a))).clamp_(min=-1)
    return V.view(-1, 3), tets.view(-1, 4), nbrs.view(-1, 4)


def _centroids(V, tets):
    out = torch.zeros((tets.shape[0], 3), dtype=torch.float32, device=DEV)
    v = V.to(torch.float32)
    for k in range(4):
        out += v[tets[:, k].long()]
    return out.mul_(0.25)


def _knot_curve(n=2048):
    t = torch.arange(n, device=DEV, dtype=torch.float64) * (2 * math.pi / n)
    r = 0.3 + 0.12 * torch.cos(5 * t)
    return torch.stack([r * torch.cos(3 * t), r * torch.sin(3 * t), 0.12 * torch.sin(5 * t)], 1).float()


# half extents of each surface's bounding box, and the radius and area
# share of its holes
BOUNDS = {"sphere": (0.4, 0.4, 0.4), "torus": (0.4, 0.4, 0.1), "box": (0.3, 0.25, 0.2), "knot": (0.47, 0.47, 0.17)}
HOLES = {"sphere": (0.012, 0.05), "torus": (0.0157, 0.03), "box": (0.0, 0.0), "knot": (0.0067, 0.02)}


def _signed_distance(mesh, X):
    """Distance of points to the closed surface (negative inside)."""
    if mesh == "sphere":
        return X.norm(dim=1) - 0.4
    if mesh == "torus":
        return torch.hypot(torch.hypot(X[:, 0], X[:, 1]) - 0.3, X[:, 2]) - 0.1
    if mesh == "box":
        q = X.abs() - torch.tensor([0.25, 0.20, 0.15], device=DEV)
        return q.clamp(min=0).norm(dim=1) + q.amax(dim=1).clamp(max=0) - 0.05
    # knot: distance to the curve from a coarse grid, interpolated
    half = torch.tensor([0.56, 0.56, 0.26], device=DEV)
    dims = (192, 192, 90)
    axes = [torch.linspace(-float(half[k]), float(half[k]), dims[k], device=DEV) for k in range(3)]
    P = torch.stack(torch.meshgrid(axes[2], axes[1], axes[0], indexing="ij"), -1).flip(-1).reshape(-1, 3)
    curve = _knot_curve()
    D = torch.cat([torch.cdist(p, curve, compute_mode="use_mm_for_euclid_dist").amin(1) for p in P.split(1 << 18)])
    D = D.view(1, 1, dims[2], dims[1], dims[0])
    out = [torch.nn.functional.grid_sample(D, (x / half).view(1, 1, 1, -1, 3), align_corners=True).view(-1)
           for x in X.split(1 << 24)]
    return torch.cat(out) - 0.05


def _shape(mesh, tets):
    half = BOUNDS[mesh]
    pad = 0.06 * 2 * max(half)
    ext = [2 * (x + pad) for x in half]
    h = (math.prod(ext) * 6.0 / tets) ** (1.0 / 3.0)
    shape = [max(2, round(e / h)) for e in ext]
    return shape, [-x - pad for x in half], [x + pad for x in half], sum(e / s for e, s in zip(ext, shape)) / 3


def _graph(mesh, tets, seed, solid=False):
    """Cell graph and labels of a mesh; ``solid``: the inside is labelled too
    (the labels of a finished cut)."""
    gen = _gen(seed)
    shape, lo, hi, h = _shape(mesh, tets)
    V, T, Nb = _lattice(shape, lo, hi, gen)
    # a finished cut's labels follow the shape, not this seed's vertices
    X = _centroids(_lattice(shape, lo, hi, gen, 0.0)[0] if solid else V, T)
    d = _signed_distance(mesh, X)
    if solid:
        return V, T, Nb, (d > 0.8 * h).to(torch.uint8)
    near = d.abs() <= 0.8 * h
    if mesh == "knot":   # a duplicated inner shell and vertex noise
        d += 1e-4 * torch.randn(d.shape, generator=gen, device=DEV)
        near = torch.minimum(d.abs(), (d + 0.002).abs()) <= 0.8 * h
    band = torch.nonzero(near).view(-1)
    if mesh == "box":    # one side missing
        side = int(torch.randint(6, (1,), generator=gen, device=DEV))
        q = X[band] / torch.tensor(BOUNDS["box"], device=DEV)
        axis, sign = side // 2, 1.0 if side % 2 else -1.0
        gone = (q.abs().argmax(1) == axis) & (q[:, axis] * sign > 0)
    else:
        r, share = HOLES[mesh]
        cell = math.prod((hi[k] - lo[k]) / shape[k] for k in range(3)) / 6
        count = max(1, int(share * band.numel() * cell / (1.6 * h) / (math.pi * r * r)))
        pick = torch.randint(max(1, band.numel()), (count,), generator=gen, device=DEV)
        centers = X[band[pick]]
        gone = torch.cat([torch.cdist(x, centers, compute_mode="use_mm_for_euclid_dist").amin(1) <= r
                          for x in X[band].split(1 << 20)])
    near[band[gone]] = False
    return V, T, Nb, (~near).to(torch.uint8)


def _raw(tets, nlink, seed):
    """Integer graph on a lattice of the unit cube: n-links by face area, equal
    both ways, t-links from a noisy sphere distance."""
    gen = _gen(seed)
    m = max(2, round((tets / 6) ** (1.0 / 3.0)))
    V, T, Nb = _lattice((m, m, m), (0, 0, 0), (1, 1, 1), gen)
    cap = torch.empty(T.shape, dtype=torch.float32, device=DEV)
    for k, (a, b, c) in enumerate(FACES):
        p = V[T[:, a].long()]
        cap[:, k] = torch.linalg.cross(V[T[:, b].long()] - p, V[T[:, c].long()] - p).norm(dim=1).float()
    cap = torch.where(Nb >= 0, cap, 0.0)
    mean = cap.sum(dtype=torch.float64) / (Nb >= 0).sum()
    cap = torch.round(cap * (nlink / mean).float()).to(torch.int32)
    d = (_centroids(V, T) - 0.5).norm(dim=1) - 0.3
    d += 0.02 * torch.randn(d.shape, generator=gen, device=DEV)
    src = torch.round(100 * (-d).clamp(min=0)).to(torch.int32)
    snk = torch.round(100 * d.clamp(min=0)).to(torch.int32)
    return Nb, cap, src, snk


def _mesh_faces(count, seed):
    """A closed torus grid of about ``count`` faces with a few faces missing."""
    nu = max(8, round(math.sqrt(count)))
    nv = max(4, round(count / (2 * nu)))
    i = torch.arange(nu, device=DEV, dtype=torch.int32).view(-1, 1)
    j = torch.arange(nv, device=DEV, dtype=torch.int32).view(1, -1)
    a, b = i * nv + j, (i + 1) % nu * nv + j
    c, d = (i + 1) % nu * nv + (j + 1) % nv, i * nv + (j + 1) % nv
    F = torch.stack([torch.stack([a, b, c], -1), torch.stack([a, c, d], -1)], 2).view(-1, 3)
    keep = torch.rand(F.shape[0], generator=_gen(seed), device=DEV) > 2e-4
    return F[keep].contiguous()


def _bricks(mesh, h, seed):
    """Narrow-band distance grid of a mesh: 8^3-voxel bricks within three
    voxels of the surface, voxel size h, origin at the low corner's brick."""
    lo = [math.floor((-x - 4 * h) / h / 8) * 8 for x in BOUNDS[mesh]]
    dims = [math.ceil(((x + 4 * h) / h - o) / 8) + 1 for x, o in zip(BOUNDS[mesh], lo)]
    mid = torch.stack(torch.meshgrid(*(torch.arange(n, device=DEV) for n in dims), indexing="ij"), -1).view(-1, 3)
    org = torch.tensor(lo, device=DEV)
    center = ((mid * 8 + org + 3.5) * h).float()
    active = torch.nonzero(_signed_distance(mesh, center).abs() <= (4 * math.sqrt(3) + 4) * h).view(-1)
    table = torch.full((mid.shape[0],), -1, dtype=torch.int32, device=DEV)
    table[active] = torch.arange(active.numel(), dtype=torch.int32, device=DEV)
    w = torch.stack(torch.meshgrid(*(torch.arange(8, device=DEV),) * 3, indexing="ij"), -1).view(1, 512, 3)
    X = ((mid[active].view(-1, 1, 3) * 8 + org + w) * h).float().view(-1, 3)
    d = _signed_distance(mesh, X).abs()
    d += 0.02 * h * torch.randn(d.shape, generator=_gen(seed), device=DEV)
    return {"voxel_size": h, "origin": lo, "dims": dims, "background": 3 * h, "table": table.view(dims),
            "values": d.abs().clamp(max=3 * h).view(-1, 8, 8, 8)}


def _batch_sizes(case, seed):
    rng = np.random.default_rng(seed)
    return np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["count"])).astype(int)


def prepare(case, seed):
    op = case["op"]
    state = {"case": case}
    if op == "cut":
        V, T, Nb, L = _graph(case["mesh"], case["tets"], seed)
        if case["host"]:
            V, L = V.cpu().numpy(), L.cpu().numpy()
        state.update(V=V, T=T, N=Nb, L=L)
    elif op == "batch":
        # the sizes belong to the case, the graphs to the seed
        sizes = _batch_sizes(case, case["count"])
        gs = [_graph(MESHES[k % 3], int(n), seed * 1000 + k) for k, n in enumerate(sizes)]
        for name, k in (("voff", 0), ("toff", 1)):
            state[name] = np.concatenate([[0], np.cumsum([g[k].shape[0] for g in gs])]).astype(np.uint64)
        state.update(zip("VTNL", (torch.cat([g[k] for g in gs]) for k in range(4))))
    elif op == "raw":
        state.update(zip(("nbr", "cap", "src", "snk"), _raw(case["tets"], case["nlink"], seed)))
    elif op == "surface":
        V, T, Nb, L = _graph(case["mesh"], case["tets"], seed, solid=True)
        state.update(V=V.cpu().numpy(), T=T, N=Nb, L=L.cpu().numpy())
    elif op == "audit":
        state["F"] = _mesh_faces(case["faces"], seed)
    elif op == "labels":
        shape, lo, hi, h = _shape(case["mesh"], case["tets"])
        V, T, _ = _lattice(shape, lo, hi, _gen(seed))
        state.update(V=V, T=T, grid=_bricks(case["mesh"], h, seed + 1), lo=np.zeros(3), hi=np.ones(3),
                     threshold=0.8 * h)
    else:
        T = _lattice([max(2, round((case["tets"] / 6) ** (1 / 3)))] * 3, (0, 0, 0), (1, 1, 1), _gen(seed))[2]
        T = torch.where(torch.rand(T.shape[0], 1, generator=_gen(seed), device=DEV) < 0.5, T, T.flip(1))
        a = T.cpu().numpy().astype(np.int64 if case["bits"] == 64 else np.int32)
        state["host"] = np.asfortranarray(a) if case["order"] == "F" else np.ascontiguousarray(a)
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    op = case["op"]
    if op == "cut" and case["host"]:
        r = wtivo_gpupr.graph_cut_fast(state["V"], state["T"], state["N"], state["L"], case["fill"])
        # labels, flows, edge and terminal counts (the other entries are times and work counters)
        return {"labels": r[0], "counts": [int(r[k]) for k in (1, 2, 5, 6, 7, 8, 9)]}
    if op == "cut":
        labels, st = capi.graph_cut(state["V"], state["T"], state["N"], state["L"], case["fill"])
        return {"labels": labels, "counts": [st["adjusted_flow"], st["raw_flow"], st["free_n"], st["free_E"]]}
    if op == "batch":
        labels, items, _ = capi.graph_cut_batch(state["toff"], state["voff"], state["V"], state["T"], state["N"],
                                                state["L"], case["fill"])
        return {"labels": labels, "flows": np.array([i["adjusted_flow"] for i in items])}
    if op == "raw":
        flow, part, _ = capi.solve_ell(state["nbr"], state["cap"], state["src"], state["snk"])
        return {"partition": part, "flow": flow}
    if op == "surface":
        V, F = wtivo_gpupr.surface_extraction_topology_cuda(state["L"], state["V"], state["T"], state["N"])
        return {"vertices": V, "faces": F}
    if op == "audit":
        return {"bad": capi.edge_audit(state["F"])[0]}
    if op == "labels":
        labels, samples = capi.sample_tet_labels(state["grid"], state["V"], state["T"], state["lo"], state["hi"], 0.0,
                                                 state["threshold"], device_out=True)
        return {"labels": labels, "samples": samples}
    return {"topology": wtivo_gpupr.topology_to_cuda_chunked(state["host"])}


def work(case):
    """Inputs read once and outputs written once; no floating-point work counts."""
    op = case["op"]
    if op == "audit":
        n = case["faces"] * 12
    elif op == "raw":
        n = case["tets"] * (16 + 16 + 4 + 4 + 1)
    elif op == "upload":
        n = case["tets"] * (4 * case["bits"] // 8 + 16)
    elif op == "labels":
        n = case["tets"] * (16 + 4 + 1 + 4)
    elif op == "batch":
        n = int(_batch_sizes(case, case["count"]).sum()) * (16 + 16 + 1 + 4 + 1)
    else:
        n = case["tets"] * (16 + 16 + 1 + 4 + (1 if op == "cut" else 0))
    return {"bytes": n, "flops": 0}


# ---------------------------------------------------------------------------
# the floating-point outputs in 64 bits (integer outputs are equal or wrong)
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["op"] == "surface":
        V, T, Nb, L = _graph(case["mesh"], case["tets"], seed, solid=True)
        used = torch.zeros(V.shape[0], dtype=torch.bool, device=DEV)
        for k, f in enumerate(FACES):
            other = torch.where(Nb[:, k] < 0, 1, L[Nb[:, k].clamp(min=0).long()])
            for q in f:
                used[T[(L == 0) & (other != 0), q].long()] = True
        return {"vertices": V[used], "faces": None}
    if case["op"] == "labels":
        s = prepare(case, seed)
        g, vals = s["grid"], s["grid"]["values"].double()
        x = torch.zeros((s["T"].shape[0], 3), dtype=torch.float64, device=DEV)
        for k in range(4):
            x += s["V"][s["T"][:, k].long()]
        x = x * 0.25 / g["voxel_size"]
        f = x.floor()
        w = x - f
        f = f.long() - torch.tensor(g["origin"], device=DEV)
        dims = torch.tensor(g["dims"], device=DEV)
        out = torch.zeros(x.shape[0], dtype=torch.float64, device=DEV)
        for corner in range(8):
            o = [(corner >> 2) & 1, (corner >> 1) & 1, corner & 1]
            q = f + torch.tensor(o, device=DEV)
            b = q >> 3
            ok = ((q >= 0) & (b < dims)).all(1)
            brick = g["table"][tuple(torch.where(ok[:, None], b, 0).T)].long()
            v = vals[(brick.clamp(min=0),) + tuple((q & 7).T)]
            v = torch.where(ok & (brick >= 0), v, float(np.float32(g["background"])))
            for k in range(3):
                v = v * (w[:, k] if o[k] else 1 - w[:, k])
            out += v
        return {"labels": None, "samples": out}
    return None
