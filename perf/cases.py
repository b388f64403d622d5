"""The work that programs built on this framework have it do, as cases that can be timed: stage 2 alone from
a few hundred faces to millions, many meshes in one batch, stage 1, stage 3, the whole ``PaMO.run`` with its
defaults, and the checks and distances that are reported beside a result. Every case goes through a public entry point
with the handle (context, system, remesher, batch) that a program keeps from one mesh to the next.

Inputs are seeded star-shaped meshes as in ``pamo_gb300.synth`` (a geodesic icosphere whose radius is perturbed by
spherical harmonics) and noisy open height fields (meshes with a boundary), made on the GPU.
"""

import math

import numpy as np
import torch

from pamo_gb300 import PaMO, api, metrics, synth
from pamo_gb300.batch import CsrBatch
from pamo_gb300.safe_project import Stage3System

DEVICE = "cuda"
#: the stage-2 and stage-3 settings of ``PaMO.run``
THRESHOLD, TOLERANCE, STAGE3_STEPS = 1e-3, 4, 5


def listed():
    return [
        # an asset of a few hundred to a thousand faces: rounds of a few microseconds of work, launches and latency
        {"name": "simplify_tiny", "op": "simplify", "mesh": "star", "n": 8, "degree": 4, "sigma": 0.04, "ratio": 0.1},
        # the benchmark's small mesh (20,480 faces) to 1 %
        {"name": "simplify_small", "op": "simplify", "mesh": "star", "n": 32, "degree": 6, "sigma": 0.03, "ratio": 0.01},
        # a scanned height field: noisy, open (boundary edges), an odd grid, reduced to 5 %
        {"name": "simplify_open", "op": "simplify", "mesh": "grid", "n": 401, "m": 357, "ratio": 0.05},
        # the benchmark's large mesh (5,242,880 faces) to 0.1 %
        {"name": "simplify_large", "op": "simplify", "mesh": "star", "n": 512, "degree": 16, "sigma": 0.02, "ratio": 0.001},
        # a data set's meshes together, as the benchmark's batch draws them (faces log-uniform 5k to 200k)
        {"name": "batch_64", "op": "batch", "count": 64, "low": 5000, "high": 200000, "ratio_low": 0.001, "ratio_high": 0.01},
        # stage 1 for a small target (the 128^3 grid) and with its default grid on a dense input
        {"name": "remesh_128", "op": "remesh", "mesh": "star", "n": 32, "degree": 6, "sigma": 0.03, "resolution": 128},
        {"name": "remesh_256", "op": "remesh", "mesh": "star", "n": 128, "degree": 8, "sigma": 0.02, "resolution": 256},
        # stage 3 of a low-poly result (1.6k faces) and of a finer one (13k) onto their inputs
        {"name": "project_small", "op": "project", "n": 64, "degree": 6, "sigma": 0.03, "ratio": 0.02},
        {"name": "project_large", "op": "project", "n": 256, "degree": 8, "sigma": 0.02, "ratio": 0.01},
        # PaMO.run with its defaults (stages 1, 2 and 3), as the command line runs it
        {"name": "run_default", "op": "run", "mesh": "star", "n": 48, "degree": 6, "sigma": 0.03, "ratio": 0.1},
        # the whole-mesh self-intersection check of a result with folds in it
        {"name": "intersect", "op": "intersect", "n": 128, "degree": 8, "sigma": 0.02, "moved": 0.01},
        # the vertices of a low-poly result against its input, as the Hausdorff distance asks for them
        {"name": "distance", "op": "distance", "n": 128, "degree": 8, "sigma": 0.02, "points": 20000},
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    def faces(lo, hi):
        return synth.frequency_for_faces(log(lo, hi))

    degree, sigma = rng.randint(4, 12), round(rng.uniform(0.01, 0.03), 4)
    op = rng.choice(["simplify", "simplify", "simplify", "batch", "remesh", "project", "project", "run", "intersect",
                     "distance"])
    star = {"op": op, "degree": degree, "sigma": sigma}
    if op == "simplify":
        ratio = round(log(0.001, 0.2), 5)
        if rng.random() < 0.3:
            n = int(log(12, 900))
            return {"op": op, "mesh": "grid", "n": n, "m": max(9, int(n * rng.uniform(0.6, 1.0))), "ratio": ratio}
        return {**star, "mesh": "star", "n": faces(320, 4.0e6), "ratio": ratio}
    if op == "batch":
        return {"op": op, "count": rng.randint(8, 64), "low": 1000, "high": int(log(20000, 200000)), "ratio_low": 0.001,
                "ratio_high": 0.1}
    if op == "remesh":
        return {**star, "mesh": "star", "n": faces(1280, 330000), "resolution": rng.choice([64, 128, 256])}
    if op == "project":
        n = faces(5000, 1.0e6)
        return {**star, "n": n, "ratio": round(min(0.3, log(300, 12000) / (20.0 * n * n)), 5)}
    if op == "run":
        return {**star, "mesh": "star", "n": faces(1280, 46000), "ratio": round(rng.uniform(0.02, 0.1), 4)}
    if op == "intersect":
        return {**star, "n": faces(8000, 1.0e6), "moved": round(rng.uniform(0.005, 0.02), 4)}
    return {**star, "n": faces(1280, 330000), "points": int(log(500, 20000))}


# ---- inputs -------------------------------------------------------------------------------------------------------

def _icosphere(n):
    """Unit geodesic icosphere of frequency n on the GPU: (float64 [10 n^2 + 2, 3], int64 [20 n^2, 3]), outward."""
    base, bfaces = synth._icosahedron()
    base = torch.cat([torch.as_tensor(base, device=DEVICE), torch.zeros(1, 3, dtype=torch.float64, device=DEVICE)])
    corners = torch.as_tensor(bfaces, device=DEVICE)
    r = torch.arange(n + 1, device=DEVICE)
    i, j = torch.meshgrid(r, r, indexing="ij")
    inside = i + j <= n
    lid = torch.full((n + 1, n + 1), -1, device=DEVICE)
    lid[inside] = torch.arange(int(inside.sum()), device=DEVICE)
    i, j = i[inside], j[inside]
    up = i + j < n
    down = i + j < n - 1
    tri = torch.cat([torch.stack([lid[i[up], j[up]], lid[i[up] + 1, j[up]], lid[i[up], j[up] + 1]], 1),
                     torch.stack([lid[i[down] + 1, j[down]], lid[i[down] + 1, j[down] + 1], lid[i[down], j[down] + 1]], 1)])
    # a lattice point is named by its corners (those of weight 0 left out, in ascending order) and their weights
    w = torch.stack([n - i - j, i, j], 1)[None].expand(20, -1, -1).reshape(-1, 3)
    c = corners[:, None, :].expand(-1, i.numel(), -1).reshape(-1, 3)
    c, order = torch.where(w > 0, c, 12).sort(dim=1, stable=True)
    w = w.gather(1, order)
    key = ((c[:, 0] * 13 + c[:, 1]) * 13 + c[:, 2]) * (n + 1) ** 2 + w[:, 0] * (n + 1) + w[:, 1]
    names, inv = torch.unique(key, return_inverse=True)
    pos = torch.empty(names.numel(), 3, dtype=torch.float64, device=DEVICE)
    at = w[:, 0:1] * base[c[:, 0]] + w[:, 1:2] * base[c[:, 1]] + w[:, 2:3] * base[c[:, 2]]
    pos[inv] = at / at.norm(dim=1, keepdim=True)  # the same bits from every face that shares the point
    faces = inv.view(20, -1)[:, tri].reshape(-1, 3)
    return pos, faces


def _radius(d, coeffs):
    """1 + sum c_lm Y_lm at unit directions d (``synth.sh_radius`` on the GPU)."""
    z = d[:, 2].clamp(-1.0, 1.0)
    st, phi = (1.0 - z * z).clamp(min=0.0).sqrt(), torch.atan2(d[:, 1], d[:, 0])
    top = max(l for l, _ in coeffs)
    r, pmm = torch.ones_like(z), torch.full_like(z, math.sqrt(1.0 / (4.0 * math.pi)))
    for m in range(top + 1):
        if m > 0:
            pmm = -math.sqrt((2.0 * m + 1.0) / (2.0 * m)) * st * pmm
        before, last = None, pmm
        a, b = torch.zeros_like(z), torch.zeros_like(z)
        for l in range(m, top + 1):
            if l == m:
                p = pmm
            elif l == m + 1:
                p = math.sqrt(2.0 * m + 3.0) * z * pmm
            else:
                s = math.sqrt((4.0 * l * l - 1.0) / (l * l - m * m))
                p = s * (z * last - math.sqrt(((l - 1.0) ** 2 - m * m) / (4.0 * (l - 1.0) ** 2 - 1.0)) * before)
            a += coeffs.get((l, m), 0.0) * p
            b += coeffs.get((l, -m), 0.0) * p
            before, last = last, p
        r += a if m == 0 else math.sqrt(2.0) * (a * torch.cos(m * phi) + b * torch.sin(m * phi))
    return r


def _star(n, degree, sigma, seed):
    """(float32 [V, 3], int32 [F, 3]) on the GPU: a star-shaped genus-0 mesh of 20 n^2 faces, free of intersections."""
    d, faces = _icosphere(n)
    rng = np.random.default_rng(seed)
    while True:
        coeffs = {(l, m): float(rng.normal(0.0, sigma * min(1.0, 3.0 / l))) for l in range(1, degree + 1)
                  for m in range(-l, l + 1)}
        coeffs[0, 0] = 0.0
        r = _radius(d, coeffs)
        if float(r.min()) >= 0.2:
            break
    return (d * r[:, None]).float().contiguous(), faces.int().contiguous()


def _grid(n, m, seed):
    """A noisy open height field of 2 n m faces (float32, int32, GPU)."""
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    a = torch.rand(6, generator=g, device=DEVICE, dtype=torch.float64)
    x, y = torch.meshgrid(torch.linspace(0, 1, n + 1, device=DEVICE, dtype=torch.float64),
                          torch.linspace(0, m / n, m + 1, device=DEVICE, dtype=torch.float64), indexing="ij")
    z = 0.08 * torch.sin((3 + 4 * a[0]) * x + 6 * a[1]) * torch.cos((2 + 5 * a[2]) * y + 6 * a[3])
    z = z + 0.02 * torch.sin(23 * x + 17 * y + 6 * a[4])
    z = z + (0.05 / n) * torch.randn(x.shape, generator=g, device=DEVICE, dtype=torch.float64)
    idx = torch.arange((n + 1) * (m + 1), device=DEVICE).view(n + 1, m + 1)
    p, q, r, s = idx[:-1, :-1].reshape(-1), idx[1:, :-1].reshape(-1), idx[1:, 1:].reshape(-1), idx[:-1, 1:].reshape(-1)
    faces = torch.cat([torch.stack([p, q, r], 1), torch.stack([p, r, s], 1)])
    return torch.stack([x, y, z], -1).view(-1, 3).float().contiguous(), faces.int().contiguous()


def _mesh(case, seed):
    if case.get("mesh") == "grid":
        return _grid(case["n"], case["m"], seed)
    return _star(case["n"], case["degree"], case["sigma"], seed)


def _batch_sizes(case):
    """The icosphere frequencies of a batch: log-uniform face counts, the same for every seed."""
    rng = np.random.default_rng(7)
    f = np.exp(rng.uniform(math.log(case["low"]), math.log(case["high"]), case["count"]))
    return [synth.frequency_for_faces(x) for x in f]


def _surface_points(v, f, count, seed):
    """Points near the surface: random barycentric points of random faces, moved by up to 1 % of the radius."""
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    pick = torch.randint(0, f.shape[0], (count,), generator=g, device=DEVICE)
    w = torch.rand(count, 3, generator=g, device=DEVICE, dtype=torch.float64)
    w = w / w.sum(1, keepdim=True)
    p = (v.double()[f[pick].long()] * w[:, :, None]).sum(1)
    return p * (1.0 + 0.01 * (2 * torch.rand(count, 1, generator=g, device=DEVICE, dtype=torch.float64) - 1))


# ---- the passes -----------------------------------------------------------------------------------------------------

def _room(nv, nf):
    """Zeroed buffers of a program's own that each pass writes its result into (a result's size follows from the
    input's values; the counts are returned beside them)."""
    return {"verts": torch.zeros(nv, 3, device=DEVICE), "faces": torch.zeros(nf, 3, dtype=torch.int32, device=DEVICE)}


def _fill(room, v, f):
    room["verts"][:v.shape[0]] = v
    room["faces"][:f.shape[0]] = f
    return {**room, "counts": [int(v.shape[0]), int(f.shape[0])]}


def prepare(case, seed):
    op = case["op"]
    if op == "batch":
        sizes = _batch_sizes(case)
        meshes = [_star(n, 6, 0.03, seed * 1009 + k) for k, n in enumerate(sizes)]
        voff = np.cumsum([0] + [v.shape[0] for v, _ in meshes])
        foff = np.cumsum([0] + [f.shape[0] for _, f in meshes])
        ratios = np.random.default_rng(seed).uniform(case["ratio_low"], case["ratio_high"], len(sizes))
        return {"op": op, "points": torch.cat([v for v, _ in meshes]), "triangles": torch.cat([f for _, f in meshes]),
                "voff": voff, "foff": foff, "ratios": ratios, "batch": CsrBatch(DEVICE + ":0"), "room": _room(voff[-1] // 4, foff[-1] // 4)}
    v, f = _mesh(case, seed)
    if op == "simplify":
        nf = min(f.shape[0], max(200000, int(4 * case["ratio"] * f.shape[0])))
        return {"op": op, "points": v, "triangles": f, "ratio": case["ratio"], "ctx": api.Context(),
                "room": _room(min(nf, v.shape[0]), nf)}
    if op == "remesh":
        return {"op": op, "points": v, "triangles": f, "resolution": case["resolution"], "mean": api.tris_mean(v, f),
                "remesher": api.Remesher(), "room": _room(10 * case["resolution"] ** 2, 20 * case["resolution"] ** 2)}
    if op == "project":
        low, low_f, _ = api.simplify(v, f, case["ratio"], TOLERANCE, THRESHOLD, min_verts=0)
        return {"op": op, "gt_v": v.double(), "gt_f": f, "v": low.double(), "f": low_f,
                "system": Stage3System(None, DEVICE + ":0"), "room": torch.zeros(v.shape[0], 3, dtype=torch.float64, device=DEVICE)}
    if op == "run":
        return {"op": op, "points": v, "triangles": f, "ratio": case["ratio"],
                "model": PaMO((v.double().cpu().numpy(), f.cpu().numpy())),
                "room": {"verts": np.zeros((f.shape[0], 3)), "faces": np.zeros((2 * f.shape[0], 3), np.int64)}}
    if op == "intersect":
        g = torch.Generator(device=DEVICE).manual_seed(seed + 1)
        pick = torch.rand(v.shape[0], 1, generator=g, device=DEVICE) < case["moved"]
        by = (torch.rand(v.shape, generator=g, device=DEVICE) - 0.5) * (4.0 / case["n"])
        return {"op": op, "points": torch.where(pick, v + by, v), "triangles": f, "ctx": api.Context()}
    if op == "distance":
        # the metrics take NumPy arrays, as the reference's do
        return {"op": op, "points": _surface_points(v, f, case["points"], seed).cpu().numpy(), "v": v.double().cpu().numpy(),
                "f": f.cpu().numpy()}
    raise ValueError(op)


def run(s):
    op = s["op"]
    if op == "simplify":
        v, f, rounds = api.simplify(s["points"], s["triangles"], s["ratio"], TOLERANCE, THRESHOLD, min_verts=0, ctx=s["ctx"])
        return {**_fill(s["room"], v, f), "rounds": rounds}
    if op == "batch":
        v, f, voff, foff = s["batch"].simplify_csr(s["points"], s["triangles"], s["voff"], s["foff"], s["ratios"], TOLERANCE,
                                                   THRESHOLD)
        return {**_fill(s["room"], v, f), "vert_offsets": voff, "face_offsets": foff}
    if op == "remesh":
        return _fill(s["room"], *s["remesher"].remesh(s["points"], s["triangles"], s["resolution"], s["mean"]))
    if op == "project":
        v = s["system"].project(s["gt_v"], s["gt_f"], s["v"], s["f"], STAGE3_STEPS)
        s["room"][:v.shape[0]] = v
        return {"verts": s["room"]}
    if op == "run":
        return _fill(s["room"], *s["model"].run(s["points"], s["triangles"], s["ratio"], min_verts=0))
    if op == "intersect":
        return {"flags": api.self_intersect(s["points"], s["triangles"], ctx=s["ctx"])}
    if op == "distance":
        d2, face = metrics.point_mesh_sqdist(s["points"], s["v"], s["f"])
        return {"sqdist": d2, "face": face}
    raise ValueError(op)


# ---- what a pass cannot do without ---------------------------------------------------------------------------------

def work(case):
    """Each input read once and each output written once (float32 vertices, int32 faces; 24-byte float64 vertices in
    stage 3 and the metrics). The arithmetic of a pass depends on its mesh (rounds, contacts, tree walks): the floor
    given is the memory's alone, and a token count of the operations that every face takes at least once."""
    op = case["op"]
    if op == "batch":
        nf = sum(20 * n * n for n in _batch_sizes(case))
        return {"bytes": 18.0 * nf, "flops": 100.0 * nf}
    nf = 2 * case["n"] * case["m"] if case.get("mesh") == "grid" else 20 * case["n"] ** 2
    nv = nf / 2 + 2
    if op == "simplify":
        return {"bytes": (12.0 * nv + 12.0 * nf) * (1 + case["ratio"]), "flops": 100.0 * nf}
    if op == "remesh":
        cells = float(case["resolution"]) ** 3
        return {"bytes": 12.0 * nv + 12.0 * nf + 36.0 * 6 * case["resolution"] ** 2, "flops": cells}
    if op == "project":
        return {"bytes": 24.0 * nv + 12.0 * nf + 36.0 * case["ratio"] * nf, "flops": 40.0 * 50 * 300 * case["ratio"] * nf}
    if op == "run":
        return {"bytes": (36.0 * nv + 24.0 * nf) * (1 + case["ratio"]), "flops": 256.0 ** 3}
    if op == "intersect":
        return {"bytes": 12.0 * nv + 13.0 * nf, "flops": 300.0 * nf}
    return {"bytes": 24.0 * nv + 12.0 * nf + 36.0 * case["points"], "flops": 100.0 * (nf + case["points"])}


# ---- values in 64 bits ------------------------------------------------------------------------------------------------

def _closest_sqdist(p, a, b, c):
    """Squared distance of points [k, 1, 3] to triangles [1, t, 3]: the plane's where the foot lies inside, else the
    least of the three edges'."""
    def edge(u, w):
        d = w - u
        t = (((p - u) * d).sum(-1) / (d * d).sum(-1).clamp(min=1e-300)).clamp(0.0, 1.0)
        return (p - u - t[..., None] * d).square().sum(-1)

    best = torch.minimum(torch.minimum(edge(a, b), edge(b, c)), edge(c, a))
    normal = torch.linalg.cross(b - a, c - a)
    height = ((p - a) * normal).sum(-1)

    def side(u, w):
        return (torch.linalg.cross((w - u).expand(p.shape[0], -1, -1), p - u) * normal).sum(-1) >= 0

    inside = side(a, b) & side(b, c) & side(c, a)
    return torch.where(inside, height * height / normal.square().sum(-1).clamp(min=1e-300), best)


def exact(case, seed):
    """The distances by trying every face for every point. The other cases' values are defined by their float32 path
    (which edges collapse, the order of the sums), so they have no other value in 64 bits."""
    if case["op"] != "distance":
        return None
    s = prepare(case, seed)
    p, v = torch.as_tensor(s["points"], device=DEVICE), torch.as_tensor(s["v"], device=DEVICE)
    t = v[torch.as_tensor(s["f"], device=DEVICE).long()]
    best = torch.full((p.shape[0],), math.inf, dtype=torch.float64, device=DEVICE)
    rows = max(1, 40_000_000 // t.shape[0])
    for i in range(0, p.shape[0], rows):
        d2 = _closest_sqdist(p[i:i + rows, None], t[None, :, 0], t[None, :, 1], t[None, :, 2])
        best[i:i + rows] = d2.amin(1)
    return {"sqdist": best.cpu().numpy(), "face": None}
