"""Stage 1 at the edges of its tiles and words, against a plain restatement: distances by trying every triangle for
every sample near it, the outside set by SciPy's connected components, and the dual extraction sample by sample.
The faces are equal. A float32 distance in the unit cube is within 5e-7 of it (a few roundings of coordinates near 1), so a
crossing v0 / (v0 - v1) is within 2 * 5e-7 / |v0 - v1| of its own, which bounds a cell's mean with its smallest
difference; 1e-6 more for the rounding of the vertex."""

import numpy as np
import pytest
import torch

from tests import meshes

pytestmark = pytest.mark.gpu


def _quad(a, b, c, d):
    return [[a, b, c], [a, c, d]]


def _box(lo, hi):
    v = np.array([[x, y, z] for z in (lo[2], hi[2]) for y in (lo[1], hi[1]) for x in (lo[0], hi[0])], float)
    f = _quad(0, 2, 3, 1) + _quad(4, 5, 7, 6) + _quad(0, 1, 5, 4) + _quad(2, 6, 7, 3) + _quad(0, 4, 6, 2) + _quad(1, 3, 7, 5)
    return v, np.array(f)


def _join(parts):
    vs, fs, n = [], [], 0
    for v, f in parts:
        vs.append(v)
        fs.append(np.asarray(f) + n)
        n += len(v)
    return np.concatenate(vs), np.concatenate(fs)


def _corridor():
    """A box without its lowest side, with plates that leave gaps at alternate ends: the outside runs to and fro along
    x, y and z to its far corner."""
    v, f = _box((0, 0, 0), (1, 0.97, 0.94))
    parts = [(v, f[2:])]
    for k, z in enumerate((0.2, 0.4, 0.6, 0.8)):
        a, b = ((0.0, 0.8), (0.2, 1.0))[k % 2]
        plate = np.array([[a, 0, z], [b, 0, z], [b, 0.97, z], [a, 0.97, z]])
        parts.append((plate, np.array(_quad(0, 1, 2, 3))))
    return _join(parts)


def _nested():
    v, f = meshes.sphere(10)
    return _join([(np.asarray(v, float), f), (0.5 * np.asarray(v, float), f[:, ::-1])])


def _mesh(name):
    if name == "sphere":
        return meshes.sphere(12)
    if name == "patch":
        return meshes.open_patch(n=9)
    if name == "box":
        return _box((0, 0, 0), (1, 0.7, 0.55))
    return {"corridor": _corridor, "nested": _nested}[name]()


def _triangle_sq(p, a, b, c):
    """Squared distances by the regions of the triangle (Ericson, Real-Time Collision Detection, 5.1.5), in float32 and in
    the kernel's order of operations: which samples are nearer than the iso value is decided by their last bits."""
    dot = lambda u, w: u[..., 0] * w[..., 0] + u[..., 1] * w[..., 1] + u[..., 2] * w[..., 2]
    ab, ac = b - a, c - a
    ap, bp, cp = p - a, p - b, p - c
    d1, d2, d3, d4, d5, d6 = dot(ab, ap), dot(ac, ap), dot(ab, bp), dot(ac, bp), dot(ab, cp), dot(ac, cp)
    va, vb, vc = d3 * d6 - d5 * d4, d5 * d2 - d1 * d6, d1 * d4 - d3 * d2
    with np.errstate(divide="ignore", invalid="ignore"):
        t, u, w = d1 / (d1 - d3), d2 / (d2 - d6), (d4 - d3) / ((d4 - d3) + (d5 - d6))
        den = np.float32(1) / (va + vb + vc)
        inner = a + ab * (vb * den)[:, None] + ac * (vc * den)[:, None]
        regions = [((d1 <= 0) & (d2 <= 0), np.broadcast_to(a, p.shape)), ((d3 >= 0) & (d4 <= d3), np.broadcast_to(b, p.shape)),
                   ((vc <= 0) & (d1 >= 0) & (d3 <= 0), a + t[:, None] * ab),
                   ((d6 >= 0) & (d5 <= d6), np.broadcast_to(c, p.shape)),
                   ((vb <= 0) & (d2 >= 0) & (d6 <= 0), a + u[:, None] * ac),
                   ((va <= 0) & (d4 - d3 >= 0) & (d5 - d6 >= 0), b + w[:, None] * (c - b))]
    r, free = inner, np.ones(len(p), bool)
    for where, point in regions:
        r = np.where((where & free)[:, None], point, r)
        free = free & ~where
    return dot(r - p, r - p)


def _restated(V, F, R, mean):
    from scipy import ndimage

    band, iso = np.float32(3.0 / R), np.float32(0.9 / R)
    margin = np.float32(3.0 / R * 2.0 + 1.0)
    p = V.astype(np.float32) - mean
    t0 = p[F.reshape(-1)].min(0)
    tmax = (p[F.reshape(-1)] - t0).max()
    q = ((p - t0) / tmax + band) / margin
    g = (np.arange(R, dtype=np.float32) + np.float32(0.5)) * (np.float32(1.0) / np.float32(R + 1))
    d2 = np.full((R, R, R), band * band)
    assert q.dtype == g.dtype == d2.dtype == np.float32
    for a, b, c in q[F]:
        lo, hi = np.minimum(np.minimum(a, b), c) - 1.01 * band, np.maximum(np.maximum(a, b), c) + 1.01 * band
        s = [slice(np.searchsorted(g, l), np.searchsorted(g, h)) for l, h in zip(lo, hi)]
        z, y, x = np.meshgrid(g[s[2]], g[s[1]], g[s[0]], indexing="ij")
        pts = np.stack([x, y, z], -1).reshape(-1, 3)
        sub = d2[s[2], s[1], s[0]]
        np.fmin(sub, _triangle_sq(pts, a, b, c).reshape(sub.shape), out=sub)
    d = np.minimum(np.sqrt(d2), band)
    far = d > iso
    label, _ = ndimage.label(far)
    edge = np.zeros((R, R, R), bool)
    for ax in range(3):
        edge.swapaxes(0, ax)[[0, -1]] = True
    out = np.isin(label, np.unique(label[edge & far])) & far
    d, iso = d.astype(np.float64), float(iso)
    field = np.where(out, d - iso, -np.abs(d - iso))
    neg = field < 0
    C = R - 1
    corner = lambda a, k: a[(k >> 2):C + (k >> 2), ((k >> 1) & 1):C + ((k >> 1) & 1), (k & 1):C + (k & 1)]
    n_neg = sum(corner(neg, k).astype(int) for k in range(8))
    active = (n_neg > 0) & (n_neg < 8)
    index = np.full(active.shape, -1)
    index[active] = np.arange(active.sum())
    cz, cy, cx = np.nonzero(active)
    vals = np.stack([corner(field, k)[active] for k in range(8)], 1)
    total, m, step = np.zeros((len(cx), 3)), np.zeros(len(cx)), np.full(len(cx), np.inf)
    for a, b in [(0, 1), (2, 3), (4, 5), (6, 7), (0, 2), (1, 3), (4, 6), (5, 7), (0, 4), (1, 5), (2, 6), (3, 7)]:
        cross = (vals[:, a] < 0) != (vals[:, b] < 0)
        with np.errstate(divide="ignore", invalid="ignore"):
            t = vals[:, a] / (vals[:, a] - vals[:, b])
        pa, pb = np.array([a & 1, (a >> 1) & 1, a >> 2]), np.array([b & 1, (b >> 1) & 1, b >> 2])
        total[cross] += pa + t[cross, None] * (pb - pa)
        m += cross
        step = np.where(cross, np.minimum(step, np.abs(vals[:, a] - vals[:, b])), step)
    c = np.stack([cx, cy, cz], 1) + total / m[:, None]
    verts = ((c + 0.5) / (R + 1) * float(margin) - float(band)) * float(tmax) + t0
    faces = []
    for z, y, x in np.argwhere(active):  # an edge that has its four cells starts in one of them
        for ax, (dz, dy, dx) in enumerate(((0, 0, 1), (0, 1, 0), (1, 0, 0))):
            u, w = ((y, z), (z, x), (x, y))[ax]
            if (x, y, z)[ax] >= R - 1 or u < 1 or w < 1 or u > C - 1 or w > C - 1:
                continue
            low = neg[z, y, x]
            if low == neg[z + dz, y + dy, x + dx]:
                continue
            if ax == 0:
                k = index[z - 1, y - 1, x], index[z - 1, y, x], index[z, y, x], index[z, y - 1, x]
            elif ax == 1:
                k = index[z - 1, y, x - 1], index[z, y, x - 1], index[z, y, x], index[z - 1, y, x]
            else:
                k = index[z, y - 1, x - 1], index[z, y - 1, x], index[z, y, x], index[z, y, x - 1]
            faces += [[k[0], k[1], k[2]], [k[0], k[2], k[3]]] if low else [[k[0], k[2], k[1]], [k[0], k[3], k[2]]]
    voxel = float(tmax) * float(margin) / (R + 1)
    return verts, np.array(faces), voxel * 2 * 5e-7 / step + 1e-6


@pytest.mark.parametrize("name, R", [("sphere", 4), ("sphere", 31), ("sphere", 32), ("nested", 33), ("patch", 47), ("box", 65),
                                     ("corridor", 64), ("sphere", 270)])
def test_remesh_equals_a_sample_by_sample_restatement(name, R):
    import pamo_gb300

    V, F = _mesh(name)
    V, F = np.asarray(V, np.float32), np.asarray(F, np.int32)
    pts, tri = torch.tensor(V, device="cuda"), torch.tensor(F, device="cuda")
    mean = np.asarray(pamo_gb300.tris_mean(pts, tri), np.float32)
    v, f = pamo_gb300.Remesher("cuda:0").remesh(pts, tri, R, mean)
    v, f = v.cpu().numpy().astype(np.float64), f.cpu().numpy()
    v0, f0, bound = _restated(V, F, R, mean)
    assert f.shape == f0.reshape(-1, 3).shape and np.array_equal(f, f0.reshape(-1, 3))
    assert v.shape == v0.shape and (np.abs(v - v0).max(1) <= bound).all()


def test_remesh_refuses_an_index_out_of_range():
    import pamo_gb300

    V, F = _mesh("box")
    F = F.copy()
    F[5, 1] = 99
    m = pamo_gb300.Remesher("cuda:0")
    with pytest.raises(Exception):
        m.remesh(torch.tensor(V, device="cuda", dtype=torch.float32), torch.tensor(F, device="cuda", dtype=torch.int32), 32,
                 np.zeros(3, np.float32))
