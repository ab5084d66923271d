"""What a user of the framework has it do, as measurable cases: field builds (a small part, a drilled
assembly, a milled part at 1024^3, a batch of recipes), exact distance transforms, point queries, the
consumers of the transform (clearance, route mask, resistor network), the packed tree, the exported
mesh and the mesh -> field stage.  Every case is seeded synthetic data with the sizes and the value
distributions of the benchmark, the tests and the reference's published runs.

listed() are the fixed cases, draw(rng) gives further ones over the same ranges, prepare(case, seed)
makes what a program holds before the call, run(state) is one pass through the public entry points,
work(case) the bytes and operations a pass cannot do without, exact(case, seed) the outputs in 64 bits
from plain torch (None where an output is whole numbers, or has no cheap 64-bit value).

A case's outputs have the same shapes for every seed: builds run into buffers of a fixed capacity, and
the seeded obstacles and balls that decide how many nodes, edges or triangles there are stand apart
from one another, the same pieces in other places.
"""
import math

import numpy as np
import torch

import field_b200.batch as BT
import field_b200.build as B
import field_b200.clearance as CL
import field_b200.edt as E
import field_b200.export as EX
import field_b200.expr as X
import field_b200.mesh as MS
import field_b200.query as Q
import field_b200.tree as TR
from field_b200.grid import GridMeta

DEV = "cuda:0"
F64 = dict(dtype=torch.float64, device=DEV)
EXACT_EVALS = 4e10  # primitive evaluations in 64 bits that exact() spends on one field


def listed():
    return [
        # the reference's own test field (a plate with a bore) at its published size M: the smallest
        # build a program makes, where launches and host reads are the time
        dict(name="build_plate", path="build", scene="plate", nx=169, ny=129, nz=89, pitch=0.25, block=8, parts=1, tools=1),
        # an assembly of drilled parts: a tree that is no chain and runs as a general program
        dict(name="build_assembly", path="build", scene="assembly", nx=192, ny=160, nz=121, pitch=1 / 160, block=8, parts=12, tools=24),
        # the milled part at scale: 3584 parts, 512 tool sweeps, 1024^3
        dict(name="build_milled_1024", path="build", scene="milled", nx=1024, ny=1024, nz=1024, pitch=1 / 1024, block=8, parts=3584, tools=512),
        # many recipes built together under one captured graph
        dict(name="batch_20", path="batch", count=20, smallest=64, largest=512, fewest=8, most=2048),
        # the squared distance of a 512^3 obstacle grid (2000 boxes, about 8 % filled)
        dict(name="edt_boxes_512", path="edt", mask="boxes", nx=512, ny=512, nz=512, boxes=2000, fill=0.08),
        # the paired signed distance of the reference's published plate 249 x 109 x 17
        dict(name="edt_pair_plate", path="edt_pair", mask="boxes", nx=249, ny=109, nz=17, boxes=12, fill=0.3),
        # one serving request's worth of points, few and many, on a resident field
        dict(name="query_1k", path="query", points=1000, n=64, block=8, parts=48, tools=8),
        dict(name="query_1m", path="query", points=1_000_000, n=256, block=8, parts=512, tools=64),
        # a route planner's step: clearance, valid mask, resistor network of the free space
        dict(name="clearance_320", path="clearance", nx=320, ny=288, nz=256, cell=32),
        # packing a dense field into the adaptive tree, then reading it back at random voxels
        dict(name="tree_384", path="tree", nx=384, ny=384, nz=381, samples=10_000_000),
        # the surface of a resident field as a triangle mesh
        dict(name="export_256", path="export", nx=256, ny=256, nz=250, block=8),
        # a closed triangle mesh into a signed field, host arrays in and out as the reference's call
        dict(name="mesh_field", path="mesh", fine=3, pitch=0.1),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["chain", "chain", "assembly", "batch", "edt", "edt", "edt_pair", "query", "query",
                       "clearance", "tree", "export", "mesh"])
    size = lambda lo, hi: [_log_int(rng, lo, hi) for _ in range(3)]
    if path == "chain":
        nx, ny, nz = size(48, 560)
        parts = _log_int(rng, 4, 2048)
        return dict(path="build", scene="milled", nx=nx, ny=ny, nz=nz, pitch=1 / max(nx, ny, nz),
                    block=rng.choice([4, 8, 8, 16]), parts=parts, tools=parts // 7)
    if path == "assembly":
        nx, ny, nz = size(40, 220)
        parts = rng.randint(2, 16)
        return dict(path="build", scene="assembly", nx=nx, ny=ny, nz=nz, pitch=1 / max(nx, ny, nz),
                    block=rng.choice([4, 8, 16]), parts=parts, tools=2 * parts)
    if path == "batch":
        return dict(path="batch", count=rng.randint(4, 20), smallest=64, largest=rng.choice([128, 256, 512]),
                    fewest=8, most=_log_int(rng, 64, 2048))
    if path in ("edt", "edt_pair"):
        nx, ny, nz = size(24, 512)
        return dict(path=path, mask=rng.choice(["boxes", "random", "sparse"]), nx=nx, ny=ny, nz=nz,
                    boxes=_log_int(rng, 8, 2000), fill=round(rng.uniform(0.02, 0.5), 3))
    if path == "query":
        return dict(path="query", points=_log_int(rng, 500, 1_000_000), n=_log_int(rng, 48, 300),
                    block=rng.choice([4, 8, 16]), parts=_log_int(rng, 8, 700), tools=rng.randint(0, 64))
    if path == "clearance":
        nx, ny, nz = size(40, 320)
        return dict(path="clearance", nx=nx, ny=ny, nz=nz, cell=rng.randint(10, 40))
    if path == "tree":
        nx, ny, nz = size(80, 400)
        return dict(path="tree", nx=nx, ny=ny, nz=nz, samples=_log_int(rng, 10_000, 10_000_000))
    if path == "export":
        block = rng.choice([4, 8, 16])
        nx, ny, nz = size(128 if block == 16 else 80, 270)
        return dict(path="export", nx=nx, ny=ny, nz=nz, block=block)
    return dict(path="mesh", fine=rng.randint(1, 3), pitch=round(rng.uniform(0.1, 0.3), 3))


# ------------------------------------------------------------------------------------ recipes
# A part is (kind, numbers); the recipe's nodes are made from it, and exact() evaluates it directly.

def _part(rng, kind, scale, lo, hi):
    c = rng.uniform(lo, hi, 3)
    if kind == 0:
        return ("sphere", c, rng.uniform(0.02, 0.1) * scale)
    if kind == 1:
        return ("box", c, rng.uniform(0.02, 0.08, 3) * scale)
    if kind == 2:
        d = rng.normal(size=3)
        d *= rng.uniform(0.02, 0.08) * scale / np.linalg.norm(d)
        return ("capsule", c - d, c + d, rng.uniform(0.01, 0.04) * scale)
    R = rng.uniform(0.04, 0.1) * scale
    return ("torus", c, R, R * rng.uniform(0.15, 0.4), int(rng.integers(0, 3)))


def _node(p):
    if p[0] == "sphere":
        return X.sphere(float(p[2]), p[1])
    if p[0] == "box":
        return X.box(p[2], p[1])
    if p[0] == "capsule":
        return X.capsule(p[1], p[2], float(p[3]))
    if p[0] == "torus":
        return X.torus(float(p[2]), float(p[3]), "xyz"[p[4]], p[1])
    return X.cylinder_z_infinite(float(p[2]), p[1][:2])


def _value(p, x, y, z):
    """A part's signed distance in 64 bits at float64 coordinates that broadcast."""
    if p[0] == "capsule":
        a, b = p[1], p[2]
        d = b - a
        qx, qy, qz = x - a[0], y - a[1], z - a[2]
        t = ((qx * d[0] + qy * d[1] + qz * d[2]) / float(d @ d)).clamp(0.0, 1.0)
        return torch.sqrt((qx - d[0] * t) ** 2 + (qy - d[1] * t) ** 2 + (qz - d[2] * t) ** 2) - p[3]
    c = p[1]
    qx, qy, qz = x - c[0], y - c[1], z - c[2]
    if p[0] == "sphere":
        return torch.sqrt(qx * qx + qy * qy + qz * qz) - p[2]
    if p[0] == "cylinder":
        return torch.sqrt(qx * qx + qy * qy) + 0.0 * qz - p[2]
    if p[0] == "box":
        h = p[2]
        qx, qy, qz = qx.abs() - h[0], qy.abs() - h[1], qz.abs() - h[2]
        out = torch.sqrt(qx.clamp(min=0) ** 2 + qy.clamp(min=0) ** 2 + qz.clamp(min=0) ** 2)
        return out + torch.maximum(qx, torch.maximum(qy, qz)).clamp(max=0)
    q = [qx, qy, qz]
    axial = q.pop(p[4])
    ring = torch.sqrt(q[0] * q[0] + q[1] * q[1]) - p[2]
    return torch.sqrt(ring * ring + axial * axial) - p[3]


def _scene(case, seed):
    """Groups of (parts, tools): the field is the union over the groups of (union of parts) - tools."""
    rng = np.random.default_rng(seed)
    if case["scene"] == "plate":
        hx, hy, hz = (0.475 * n * case["pitch"] for n in (case["nx"], case["ny"], case["nz"]))
        s = rng.uniform(0.95, 1.0, 4)
        return [([("box", np.zeros(3), np.array([hx, hy, hz]) * s[:3])], [("cylinder", np.zeros(3), 0.6 * hy * s[3])])]
    size = np.array([case["nx"], case["ny"], case["nz"]]) * case["pitch"]
    if case["scene"] == "assembly":  # plates, each with its own bores
        groups = []
        bores = case["tools"] // case["parts"]
        for _ in range(case["parts"]):
            c, h = rng.uniform(0.2, 0.8, 3) * size, rng.uniform(0.06, 0.2, 3) * size.min()
            tools = []
            for _ in range(bores):
                a = c + rng.uniform(-0.7, 0.7, 3) * h
                b = a.copy()
                k = int(rng.integers(0, 3))
                a[k], b[k] = c[k] - 2 * h[k], c[k] + 2 * h[k]
                tools.append(("capsule", a, b, rng.uniform(0.1, 0.3) * h.min()))
            groups.append(([("box", c, h)], tools))
        return groups
    parts, tools = case["parts"], case["tools"]
    scale = min(1.0, max(0.25, (64.0 / parts) ** (1 / 3))) if parts < 3000 else 0.25
    made = [_part(rng, k % 4, scale, 0.1 * size, 0.9 * size) for k in rng.permutation(parts)]
    cut = []
    for _ in range(tools):
        a, b = rng.uniform(0.05, 0.95, (2, 3)) * size
        cut.append(("capsule", a, b, rng.uniform(0.005, 0.02) * max(scale, 0.25)))
    return [(made, cut)]


def _recipe(groups):
    return X.union_all([X.subtract_all(X.union_all([_node(p) for p in parts]), [_node(t) for t in tools])
                        for parts, tools in groups])


def _field_value(groups, x, y, z):
    whole = None
    for parts, tools in groups:
        v = None
        for p in parts:
            w = _value(p, x, y, z)
            v = w if v is None else torch.minimum(v, w)
        for t in tools:
            v = torch.maximum(v, -_value(t, x, y, z))
        whole = v if whole is None else torch.minimum(whole, v)
    return whole


def _meta(case):
    n = (case["nx"], case["ny"], case["nz"])
    lo = [-0.5 * (k - 1) * case["pitch"] for k in n] if case.get("scene") == "plate" else [0.0, 0.0, 0.0]
    return GridMeta(*lo, case["pitch"], *n, case["block"])


def _axes(meta):
    """World coordinates of the padded grid's vertices, one past the last block's end."""
    nb = (meta.n_bx, meta.n_by, meta.n_bz)
    return [o + torch.arange(k * meta.block + 1, **F64) * meta.pitch for o, k in zip((meta.x0, meta.y0, meta.z0), nb)]


def _corner_kinds(lattice, margin):
    """(kind, min |corner|) of every block from the values at its corners (n_bx + 1, ...)."""
    a = torch.stack([lattice[i:lattice.shape[0] - 1 + i, j:lattice.shape[1] - 1 + j, k:lattice.shape[2] - 1 + k]
                     for i in (0, 1) for j in (0, 1) for k in (0, 1)])
    near = a.abs().amin(0)
    mixed = (a >= 0).any(0) & (a < 0).any(0)
    kind = torch.where((a < 0).all(0), -1, 1)
    kind[mixed | (near <= margin)] = 0
    return kind.to(torch.int32).reshape(-1), near.reshape(-1)


def _exact_build(groups, meta):
    """(None, corner minima, None, leaf tiles padded to every block) in 64 bits; None where it costs too much."""
    prims = sum(len(p) + len(t) for p, t in groups)
    if prims * meta.n_blocks * 4 > EXACT_EVALS:
        return None
    ax, ay, az = _axes(meta)
    b = meta.block
    corners = [a[::b] for a in (ax, ay, az)]
    lattice = _field_value(groups, corners[0][:, None, None], corners[1][None, :, None], corners[2][None, None, :])
    kind, near = _corner_kinds(lattice, float(np.float32(meta.margin_mm)))
    ids = torch.nonzero(kind == 0).reshape(-1)
    if prims * len(ids) * b ** 3 > EXACT_EVALS:
        return None
    tiles = torch.zeros((meta.n_blocks, b, b, b), **F64)
    step = max(1, (1 << 24) // b ** 3)
    o = torch.arange(b, device=DEV)
    for s in range(0, len(ids), step):
        i = ids[s:s + step]
        bx, by, bz = i // (meta.n_by * meta.n_bz), (i // meta.n_bz) % meta.n_by, i % meta.n_bz
        tiles[s:s + len(i)] = _field_value(groups, ax[bx[:, None] * b + o][:, :, None, None],
                                         ay[by[:, None] * b + o][:, None, :, None],
                                         az[bz[:, None] * b + o][:, None, None, :])
    return [None, near, None, tiles.reshape(meta.n_blocks, b ** 3), len(ids)]


# ------------------------------------------------------------------------------------ masks and dense fields
def _boxes(case, seed):
    """uint8 occupancy of random boxes whose expected union fills about `fill` of the grid."""
    rng = np.random.default_rng(seed)
    n = np.array([case["nx"], case["ny"], case["nz"]])
    k = case["boxes"]
    half = rng.uniform(0.5, 1.5, (k, 3))
    # Boolean model: fill = 1 - exp(-sum of volumes / V)
    scale = (-math.log(1 - case["fill"]) * float(n.prod()) / float((2 * half).prod(1).sum())) ** (1 / 3)
    c = rng.uniform(0, 1, (k, 3)) * n
    lo = np.clip(np.floor(c - half * scale), 0, n - 1).astype(int)
    hi = np.clip(np.ceil(c + half * scale), lo + 1, n).astype(int)
    g = torch.zeros(tuple(int(v) for v in n), dtype=torch.uint8, device=DEV)
    for a, b in zip(lo, hi):
        g[a[0]:b[0], a[1]:b[1], a[2]:b[2]] = 1
    return g


def _mask(case, seed):
    if case["mask"] == "boxes":
        g = _boxes(case, seed)
    else:
        gen = torch.Generator(DEV).manual_seed(seed)
        p = case["fill"] if case["mask"] == "random" else case["fill"] * 0.002
        g = (torch.rand((case["nx"], case["ny"], case["nz"]), device=DEV, generator=gen) < p).to(torch.uint8)
    g[0, 0, 0], g[-1, -1, -1] = 1, 0  # both classes present
    return g


def _min_plus(f, axis):
    """min over s of f(s) + (q - s)^2 along an axis, int32, by shifted passes."""
    n = f.shape[axis]
    out = f.clone()
    d = 1
    while d < n and d * d < int(out.max()):  # a shift whose square alone exceeds every minimum changes nothing
        a, b = out.narrow(axis, d, n - d), out.narrow(axis, 0, n - d)
        torch.minimum(a, f.narrow(axis, 0, n - d) + d * d, out=a)
        torch.minimum(b, f.narrow(axis, d, n - d) + d * d, out=b)
        d += 1
    return out


def _squared(sites):
    """Exact squared distance of every voxel to the nearest site (a bool tensor), int32."""
    never = sum((n - 1) ** 2 for n in sites.shape) + 1
    f = torch.where(sites, 0, never).to(torch.int32)
    for axis in (2, 1, 0):
        f = _min_plus(f, axis)
    return f.clamp(max=never)


def _cells(n, cell):
    """Corners of the whole cells of edge `cell` that fit a grid of n voxels per axis."""
    at = np.stack(np.meshgrid(*(np.arange(k // cell) for k in n), indexing="ij"), -1).reshape(-1, 3)
    return at * cell


def _apart(case, seed):
    """bool occupancy: a box in every cell, no two touching.  The boxes' sizes are the case's, their order
    and places the seed's, so free cells and the links among them are as many for every seed."""
    n, cell = [case["nx"], case["ny"], case["nz"]], case["cell"]
    rng = np.random.default_rng(seed)
    corners = _cells(n, cell)
    half = np.random.default_rng(cell).uniform(0.15, 0.75, (len(corners), 3)) * (cell - 2)
    size = np.maximum(1, half.astype(int))[rng.permutation(len(corners))]
    lo = corners + 1 + (rng.uniform(0, 1, size.shape) * (cell - 1 - size)).astype(int)
    g = torch.zeros(n, dtype=torch.bool, device=DEV)
    for a, b in zip(lo, lo + size):
        g[a[0]:b[0], a[1]:b[1], a[2]:b[2]] = True
    return g


def _dense(case, seed):
    """float32 signed field of balls on an nx x ny x nz grid: a ball in every cell, far
    enough from its cell's walls that the blocks near its surface are its own.  The radii are the
    case's, their order and the pitch the seed's; centres on voxels, so a ball's samples are the same wherever it is."""
    n = [case["nx"], case["ny"], case["nz"]]
    cell, most = (128, 18.0) if case.get("block") == 16 else (80, 17.0)
    corners = _cells(n, cell)
    radii = np.random.default_rng(cell).uniform(6.0, most, len(corners))
    rng = np.random.default_rng(seed)
    pitch = rng.uniform(0.5, 1.0) / max(n)
    out = None
    at = [torch.arange(k, dtype=torch.float32, device=DEV) for k in n]
    for c, r in zip(corners[rng.permutation(len(corners))] + cell // 2, radii):
        d = [(a - float(v)) ** 2 for a, v in zip(at, c)]
        v = (d[0][:, None, None] + d[1][None, :, None] + d[2][None, None, :]).sqrt_().sub_(r)
        out = v if out is None else torch.minimum(out, v, out=out)
    return out.mul_(pitch), pitch


def _sparse(dense, pitch, block):
    """The dense field's blocks as a resident sparse field: kinds by the 8-corner rule, leaf tiles."""
    n = list(dense.shape)
    meta = GridMeta(0.0, 0.0, 0.0, pitch, *n, block)
    nb = (meta.n_bx, meta.n_by, meta.n_bz)
    at = [torch.clamp(torch.arange(k * block + 1, device=DEV), max=m - 1) for k, m in zip(nb, n)]
    cor = dense[at[0][::block]][:, at[1][::block]][:, :, at[2][::block]]
    kind, near = _corner_kinds(cor, meta.margin_mm)
    ids = torch.nonzero(kind == 0).reshape(-1)
    pad = dense[at[0][:-1]][:, at[1][:-1]][:, :, at[2][:-1]]
    tiles = pad.reshape(nb[0], block, nb[1], block, nb[2], block).permute(0, 2, 4, 1, 3, 5).reshape(-1, block ** 3)
    count = torch.tensor([len(ids)], dtype=torch.int32, device=DEV)
    return B.DeviceField(meta, kind, near.float(), ids.to(torch.int32), count, tiles[ids].contiguous(), len(ids))


def _mesh(case, seed):
    """A ball, a turned box and a ring (closed, outward) between two fixed stops at the corners of the
    window, in millimetres, as vertex and face arrays."""
    rng = np.random.default_rng(seed)
    fine = case["fine"]

    def surface(f, nu, nv, closed_v):
        u = np.linspace(0, 2 * np.pi, nu, endpoint=False)
        v = np.linspace(0, 2 * np.pi, nv, endpoint=False) if closed_v else np.linspace(0, np.pi, nv + 1)
        V = np.stack(f(u[:, None], v[None, :]), -1).reshape(-1, 3)
        w = len(v)
        i, j = np.meshgrid(np.arange(nu), np.arange(nv), indexing="ij")
        a, b = i * w + j, (i + 1) % nu * w + j
        c, d = i * w + (j + 1) % w, (i + 1) % nu * w + (j + 1) % w
        return V, np.concatenate([np.stack([a, b, d], -1).reshape(-1, 3), np.stack([a, d, c], -1).reshape(-1, 3)])

    r, c = rng.uniform(2.5, 3.5), rng.uniform(4, 6, 3)
    ball = surface(lambda u, v: (c[0] + r * np.sin(v) * np.cos(u), c[1] + r * np.sin(v) * np.sin(u),
                                 c[2] - r * np.cos(v) + 0 * u), 48 * fine, 24 * fine, False)
    R, q, o = rng.uniform(3, 4), rng.uniform(0.8, 1.4), rng.uniform(5, 7, 3) + np.array([0, 8, 0])
    ring = surface(lambda u, v: (o[0] + (R + q * np.cos(v)) * np.cos(u), o[1] + (R + q * np.cos(v)) * np.sin(u),
                                 o[2] + q * np.sin(v) + 0 * u), 48 * fine, 24 * fine, True)
    h, t, m = rng.uniform(1.5, 3, 3), rng.uniform(0.2, 0.8), rng.uniform(12, 13, 3)
    cube = np.array([[x, y, z] for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)], float)
    V = cube * h
    V = V @ np.array([[math.cos(t), math.sin(t), 0], [-math.sin(t), math.cos(t), 0], [0, 0, 1]]) + m
    T = np.array([(0, 1, 3), (0, 3, 2), (4, 6, 7), (4, 7, 5), (0, 4, 5), (0, 5, 1), (2, 3, 7), (2, 7, 6), (0, 2, 6),
                  (0, 6, 4), (1, 5, 7), (1, 7, 3)])
    Vs, Ts, k = [], [], 0
    stops = [(0.3 * cube + np.array(at), T) for at in ((0.433, 0.427, 0.441), (17.61, 19.62, 16.63))]
    for W, S in (ball, ring, (V, T), *stops):
        Vs.append(W)
        Ts.append(S + k)
        k += len(W)
    return np.concatenate(Vs).astype(np.float64), np.concatenate(Ts).astype(np.int64)


# ------------------------------------------------------------------------------------ prepare and run
def _query_scene(case):
    n = case["n"]
    return dict(scene="milled", nx=n, ny=n, nz=n, pitch=1.0 / n, block=case["block"], parts=case["parts"], tools=case["tools"])


def _points(case, seed):
    """float32 points over the grid's box and a little beyond it."""
    gen = torch.Generator(DEV).manual_seed(seed)
    return torch.rand((case["points"], 3), device=DEV, generator=gen) * 1.04 - 0.02


def _batch(case, seed):
    rng = np.random.default_rng(seed)
    sizes = [n for n in (64, 128, 256, 512) if case["smallest"] <= n <= case["largest"]]
    out = []
    for k in range(case["count"]):
        prims = int(round(math.exp(rng.uniform(math.log(case["fewest"]), math.log(case["most"])))))
        n = sizes[k % len(sizes)]
        c = dict(scene="milled", nx=n, ny=n, nz=n, pitch=1.0 / n, block=(4, 8, 8, 4)[k % 4], parts=prims - prims // 8,
                 tools=prims // 8)
        out.append((_scene(c, seed * 1000 + k), _meta(c)))
    return out


def prepare(case, seed):
    path = case["path"]
    s = {"path": path}
    if path == "build":
        fb = B.FieldBuilder(_recipe(_scene(case, seed)), _meta(case), device=DEV)
        fb.active.zero_()
        s["builder"], s["capacity"] = fb, fb.meta.n_blocks
        s["tiles"] = torch.zeros((fb.meta.n_blocks, fb.meta.block ** 3), dtype=torch.float32, device=DEV)
    elif path == "batch":
        recipes = [(_recipe(g), m) for g, m in _batch(case, seed)]
        bb = BT.BatchBuilder(recipes, device=DEV, capacity=sum(m.n_blocks * m.block ** 3 for _, m in recipes))
        bb.tiles.zero_()
        for fb in bb.builders:
            fb.active.zero_()
        bb.enqueue()
        bb.ensure_capacity()
        bb.capture()
        s["batch"] = bb
    elif path in ("edt", "edt_pair"):
        s["mask"] = _mask(case, seed)
        s["pitch"] = 0.25
    elif path == "query":
        c = _query_scene(case)
        fb = B.FieldBuilder(_recipe(_scene(c, seed)), _meta(c), device=DEV)
        s["field"] = fb.build()
        s["queries"] = Q.RecipeQueries(fb.compiled, device=DEV, builder=fb)
        s["points"], s["h"] = _points(case, seed), 1.0 / case["n"]
    elif path == "clearance":
        s["occ"], s["pitch"] = _apart(case, seed), 0.5
    elif path == "tree":
        s["dense"], s["pitch"] = _dense(case, seed)
        s["at"] = _voxels(case, seed)
    elif path == "export":
        s["field"] = _sparse(*_dense(case, seed), case["block"])
    else:
        s["V"], s["T"] = _mesh(case, seed)
        s["pitch"] = case["pitch"]
    return s


def _voxels(case, seed):
    gen = torch.Generator(DEV).manual_seed(seed + 1)
    n = torch.tensor([case["nx"], case["ny"], case["nz"]], device=DEV)
    return (torch.rand((case["samples"], 3), device=DEV, generator=gen, dtype=torch.float64) * n).to(torch.int64)


def run(s):
    path = s["path"]
    if path == "build":
        fb = s["builder"]
        fb.enqueue(s["tiles"], s["capacity"])
        return [fb.kind, fb.cma, fb.active, s["tiles"], fb.count]
    if path == "batch":
        bb = s["batch"]
        bb.replay()
        return [bb.leaf_counts(), bb.tiles] + [[fb.kind, fb.cma, fb.active] for fb in bb.builders]
    if path == "edt":
        return E.squared_distance_device(s["mask"], sites_nonzero=True)
    if path == "edt_pair":
        return list(E.signed_distance_device(s["mask"], s["pitch"], with_squared=True))
    if path == "query":
        return list(s["queries"].values_and_gradients(s["points"], h=s["h"]))
    if path == "clearance":
        mm, n, nodes, u, v, kond, L = CL.fritt_natverk(s["occ"], s["pitch"])
        valid = CL.giltig_frirum(s["occ"], mm, 1.0, 2.0 * s["pitch"])
        return [mm, valid, n, nodes, u, v, kond, L.crow_indices(), L.col_indices(), L.values()]
    if path == "tree":
        t = TR.build_device(s["dense"], s["pitch"])
        tree = TR.AdaptiveBlocks.from_device(t, s["pitch"], host=False)
        return [t["packed"], t["branch"], t["value"], t["values"], tree.sample_device(s["at"])]
    if path == "export":
        m = EX.marching_cubes(s["field"], to_host=False)
        return [m.verts, m.faces, m.volume]
    gmin, shape, surface, solid, sd, diag = MS.field_stage(s["V"], s["T"], s["pitch"], np.zeros(3))
    return [gmin, solid, surface, sd, diag["n_traffar"]]


# ------------------------------------------------------------------------------------ work
def _active_share(case):
    """Expected share of the blocks that hold leaves: a Boolean model of the parts' margin shells."""
    n, p, b = (case["nx"], case["ny"], case["nz"]), case["pitch"], case["block"]
    volume = n[0] * n[1] * n[2] * p ** 3
    if case["scene"] == "plate":
        area = 2 * 0.95 ** 2 * p * p * (n[0] * n[1] + n[1] * n[2] + n[0] * n[2])
        shells = area * 2 * math.sqrt(3) * b * p
    else:
        scale = 1.0 if case["parts"] <= 64 else max(0.25, (64.0 / case["parts"]) ** (1 / 3))
        r = 0.06 * scale
        shells = case["parts"] * 4 * math.pi * r * r * min(2 * math.sqrt(3) * b * p, 2 * r)
        shells += case["tools"] * 2 * math.pi * 0.0125 * scale * 0.66 * 2 * math.sqrt(3) * b * p * 0.3
    return 1.0 - math.exp(-shells / volume)


def _build_work(case):
    blocks = 1
    for k in ("nx", "ny", "nz"):
        blocks *= -(-case[k] // case["block"])
    leaf = blocks * _active_share(case) * case["block"] ** 3
    # kinds, minima and ids once, every leaf voxel once; one primitive (25 operations) per corner and voxel
    return 8.0 * blocks + 4.0 * leaf, 25.0 * (leaf + blocks)


def work(case):
    path = case["path"]
    if path == "build":
        b, f = _build_work(case)
    elif path == "batch":
        sizes = [n for n in (64, 128, 256, 512) if case["smallest"] <= n <= case["largest"]]
        prims = math.sqrt(case["fewest"] * case["most"])
        b = f = 0.0
        for k in range(case["count"]):
            n = sizes[k % len(sizes)]
            w = _build_work(dict(scene="milled", nx=n, ny=n, nz=n, pitch=1 / n, block=(4, 8, 8, 4)[k % 4],
                                 parts=int(prims), tools=int(prims / 8)))
            b, f = b + w[0], f + w[1]
    elif path == "query":
        b, f = case["points"] * 28.0, case["points"] * 7 * 25.0
    elif path == "mesh":
        cells = 17.8 * 19.8 * 16.8 / case["pitch"] ** 3
        b, f = cells * 6.0 + 6912.0 * case["fine"] ** 2 * 36, cells * 8.0
    else:
        v = float(case["nx"] * case["ny"] * case["nz"])
        if path == "edt":
            b, f = 5.0 * v, 6.0 * v
        elif path == "edt_pair":
            b, f = 13.0 * v, 16.0 * v
        elif path == "clearance":
            free = v * 0.9
            # occupancy, clearance, mask and node map per cell; 3 edges of 16 B and 7 entries of 12 B per node
            b, f = 14.0 * v + free * (4 + 48 + 84), 30.0 * free
        elif path == "tree":
            b, f = 4.0 * v + 28.0 * case["samples"], 8.0 * v / 64
        else:
            balls = len(_cells([case["nx"], case["ny"], case["nz"]], 128 if case["block"] == 16 else 80))
            faces = balls * 4 * math.pi * 12.0 ** 2 * 2
            tiles = faces * 2 * math.sqrt(3) * case["block"]
            b, f = 4.0 * tiles + faces * (18 + 36), 40.0 * faces
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------------------------ exact
def _exact_signed(mask, pitch):
    solid = mask != 0
    out, inside = (_squared(m).double().sqrt() * pitch for m in (solid, ~solid))
    d = out - inside
    return d - torch.sign(d) * (0.5 * pitch)


def _exact_clearance(case, seed):
    pitch = 0.5
    occ = _apart(case, seed)
    mm = _squared(occ).double().sqrt() * pitch
    free = ~occ
    edges, up, down = [], [], []
    for a in range(3):
        n = occ.shape[a]
        lo, hi = (lambda t: t.narrow(a, 0, n - 1)), (lambda t: t.narrow(a, 1, n - 1))
        k = (0.5 * (lo(mm) + hi(mm)) / pitch).clamp(min=0.1) ** 1.5
        both = lo(free) & hi(free)
        edges.append(k[both])
        fwd, bwd = torch.zeros_like(mm), torch.zeros_like(mm)
        lo(fwd)[both] = k[both]
        hi(bwd)[both] = k[both]
        up.append(fwd)
        down.append(bwd)
    diag = sum(up) + sum(down)
    row = torch.stack([-down[0], -down[1], -down[2], diag, -up[2], -up[1], -up[0]], -1)[free]
    return [mm, None, None, None, None, None, torch.cat(edges), None, None, row[row != 0]]


def _exact_tree(case, seed):
    """The tree's values at the sampled voxels: the first leaf on the way down by the 8-corner rule."""
    dense, pitch = _dense(case, seed)
    at = _voxels(case, seed)
    top = torch.tensor(dense.shape, device=DEV) - 1
    out = torch.zeros(len(at), **F64)
    open_ = torch.ones(len(at), dtype=torch.bool, device=DEV)
    for side in (8, 4, 2, 1):
        o = at // side * side
        v = torch.stack([dense[tuple(torch.minimum(o + side * torch.tensor(c, device=DEV), top).unbind(1))]
                         for c in np.ndindex(2, 2, 2)])
        neg = (v < 0).any(0)
        leaf = ~((v >= 0).any(0) & neg) & ~(v.abs().amin(0) <= float(np.float32(math.sqrt(3.0) * side * pitch)))
        here = open_ & leaf
        out[here] = torch.where(neg, -1.0, 1.0).double()[here] * (math.sqrt(3.0) * side * pitch)
        open_ &= ~leaf
    out[open_] = dense[tuple(at[open_].unbind(1))].double()
    return [None, None, None, None, out]


def _exact_export(case, seed):
    """Vertices in 64 bits from the leaf tiles: blocks ascending, edges by voxel then axis, then the
    edges that enter a block across a low face from a block without leaves."""
    f = _sparse(*_dense(case, seed), case["block"])
    m, b = f.meta, case["block"]
    nb = (m.n_bx, m.n_by, m.n_bz)
    every = torch.where(f.kind < 0, -1.0e6, 1.0e6).double()[:, None].repeat(1, b ** 3)
    every[f.active.long()] = f.tiles.double()
    v = every.reshape(*nb, b, b, b).permute(0, 3, 1, 4, 2, 5).reshape(*(k * b for k in nb))[:m.nx, :m.ny, :m.nz]
    active = (f.kind == 0).reshape(nb)
    found, order = [], []
    for a in range(3):
        n = v.shape[a]
        g0, g1 = v.narrow(a, 0, n - 1), v.narrow(a, 1, n - 1)
        p = torch.nonzero((g0 < 0) != (g1 < 0))
        t = (g0 / (g0 - g1))[tuple(p.unbind(1))]
        q = p.clone()
        q[:, a] += 1
        own = active[tuple((p // b).unbind(1))]
        blk = torch.where(own[:, None], p // b, q // b)
        l, r = p % b, q % b
        inner = ((l[:, 0] * b + l[:, 1]) * b + l[:, 2]) * 3 + a
        u, w = (1 if a == 0 else 0), (1 if a == 2 else 2)
        slot = torch.where(own, inner, 3 * b ** 3 + a * b * b + r[:, u] * b + r[:, w])
        order.append(((blk[:, 0] * nb[1] + blk[:, 1]) * nb[2] + blk[:, 2]) * (3 * b ** 3 + 3 * b * b) + slot)
        x = p.double()
        x[:, a] += t
        found.append(x * m.pitch)
    return [torch.cat(found)[torch.argsort(torch.cat(order))], None, None]


def _exact_mesh(case, seed):
    """The signed field from vertical ray windings in 64 bits and the exact transform of the solid."""
    V, T = _mesh(case, seed)
    pitch = case["pitch"]
    gmin = np.floor(V.min(0) / pitch).astype(np.int64) - 2
    gmax = np.ceil(V.max(0) / pitch).astype(np.int64) + 3
    n, o = gmax - gmin, gmin * pitch
    jx, jy = pitch * 1e-4 * 0.3819660112501051, pitch * 1e-4 * 0.6180339887498949
    A, Bv, C = V[T[:, 0]], V[T[:, 1]], V[T[:, 2]]
    a2 = (Bv[:, 0] - A[:, 0]) * (C[:, 1] - A[:, 1]) - (Bv[:, 1] - A[:, 1]) * (C[:, 0] - A[:, 0])
    span = np.abs(np.concatenate([Bv - A, C - A], 1)[:, [0, 1, 3, 4]]).max(1)
    lo = np.minimum(np.minimum(A, Bv), C)[:, :2] - [jx, jy] - o[:2]
    hi = np.maximum(np.maximum(A, Bv), C)[:, :2] - [jx, jy] - o[:2]
    i0, i1 = np.maximum(np.ceil(lo / pitch), 0).astype(int), np.minimum(np.floor(hi / pitch), n[:2] - 1).astype(int)
    w = np.maximum(i1 - i0 + 1, 0) * (np.abs(a2) > 1e-12 * span * span)[:, None]
    per = w[:, 0] * w[:, 1]
    t = np.repeat(np.arange(len(T)), per)
    k = np.arange(per.sum()) - np.repeat(np.cumsum(per) - per, per)
    ii, jj = i0[t, 0] + k // w[t, 1], i0[t, 1] + k % w[t, 1]
    px, py, s = o[0] + ii * pitch + jx, o[1] + jj * pitch + jy, np.sign(a2[t])
    cross = lambda P, S: (P[t, 0] - px) * (S[t, 1] - py) - (P[t, 1] - py) * (S[t, 0] - px)
    l0, l1, l2 = cross(Bv, C), cross(C, A), cross(A, Bv)
    hit = (l0 * s >= 0) & (l1 * s >= 0) & (l2 * s >= 0)
    z = ((l0 * A[t, 2] + l1 * Bv[t, 2] + l2 * C[t, 2]) / a2[t])[hit]
    below = np.clip(np.ceil((z - o[2]) / pitch), 0, n[2]).astype(int)  # voxels under the hit
    wind = np.zeros((n[0], n[1], n[2] + 1), np.int64)
    np.add.at(wind, (ii[hit], jj[hit], below), s[hit].astype(np.int64))
    above = wind[:, :, ::-1].cumsum(2)[:, :, ::-1][:, :, 1:]
    solid = torch.from_numpy(np.ascontiguousarray(above != 0)).to(DEV)
    return [None, None, None, _exact_signed(solid, pitch), None]


def exact(case, seed):
    path = case["path"]
    if path == "build":
        f = _exact_build(_scene(case, seed), _meta(case))
        return f and f[:4] + [None]
    if path == "batch":
        made = _batch(case, seed)
        out = [_exact_build(g, m) for g, m in made]
        whole = None
        if all(out):
            whole = torch.zeros(sum(m.n_blocks * m.block ** 3 for _, m in made), **F64)
            at = 0
            for f in out:
                leaves = f[3][:f[4]].reshape(-1)
                whole[at:at + len(leaves)] = leaves
                at += len(leaves)
        return [None, whole] + [[None, f[1] if f else None, None] for f in out]
    if path == "edt":
        return None  # whole numbers
    if path == "edt_pair":
        return [_exact_signed(_mask(case, seed), 0.25), None]
    if path == "query":
        c = _query_scene(case)
        groups, p, h = _scene(c, seed), _points(case, seed).double(), 1.0 / case["n"]
        at = lambda d: _field_value(groups, *(p + torch.tensor(d, **F64)).unbind(1))
        g = [(at([h * (a == k) for k in range(3)]) - at([-h * (a == k) for k in range(3)])) / (2 * h) for a in range(3)]
        return [at([0.0, 0.0, 0.0]), torch.stack(g, 1)]
    if path == "clearance":
        return _exact_clearance(case, seed)
    if path == "tree":
        return _exact_tree(case, seed)
    if path == "export":
        return _exact_export(case, seed)
    return _exact_mesh(case, seed)
