"""Point-to-mesh distances where float tells the triangles apart badly: points far away, a vertex far away, a flat mesh, many
equal triangles, points without a finite distance. Against NumPy brute force in float64, and against the time that the
call takes for points near the mesh."""

import time

import numpy as np
import pytest

from pamo_gb300 import metrics
from tests import meshes
from tests.test_gpu_metrics import _point_tri_sqdist

pytestmark = pytest.mark.gpu


def _flat(n=16):
    v, f = meshes.open_patch(n)
    v = v.astype(np.float64)
    v[:, 2] = 0.0
    return v, f


def _check(P, V, F):
    d2, fi = metrics.point_mesh_sqdist(P, V, F)
    all_d2 = np.stack([_point_tri_sqdist(P, V[f[0]], V[f[1]], V[f[2]]) for f in F])
    want, size = all_d2.min(0), np.abs(P).max(1) + np.abs(V[F]).max()
    # 1e-9 of the value, or what float64 loses where coordinates are larger than the distance (as in test_gpu_metrics)
    bound = 1e-9 * want + 1e-13 * size * np.sqrt(want) + (1e-13 * size) ** 2
    assert (np.abs(d2 - want) <= bound).all()
    assert (np.abs(all_d2[fi, np.arange(len(P))] - want) <= bound).all()


@pytest.mark.parametrize("far", [3.0, 30.0, 90.0, 120.0, 1e3, 1e6, 1e9])
@pytest.mark.parametrize("flat", [False, True])
def test_points_far_from_the_mesh(far, flat):
    """On both sides of the distance (100 extents) from which the walk is in float64."""
    V, F = _flat() if flat else meshes.tangled(n=6, seed=8)
    V = V.astype(np.float64)
    rng = np.random.default_rng(5)
    P = rng.normal(0, 1.0, (130, 3))
    P *= far / np.abs(P).max(1, keepdims=True)
    if flat:
        P[:65, :2] = rng.uniform(0, 1, (65, 2))  # straight above it
    _check(P, V, F)


@pytest.mark.parametrize("away", [1e2, 1e4, 1e8])
def test_a_vertex_far_from_the_rest(away):
    V, F = meshes.sphere(7)
    V = np.vstack([V.astype(np.float64), [[away, -away, away]]])
    F = np.vstack([F, [[0, 1, len(V) - 1]]]).astype(np.int32)
    rng = np.random.default_rng(6)
    P = np.vstack([V[:60] * (1 + rng.uniform(-1e-3, 1e-3, (60, 1))), rng.normal(0, 1.2, (60, 3)), 0.5 * away * rng.normal(0, 1, (20, 3))])
    _check(P, V, F)


def test_more_equal_triangles_than_the_float_walk_takes():
    """1,500 copies of each of three triangles: the float walk leaves the points to the one in float64, and the smallest
    index wins."""
    V = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [1, 1, 0.5], [2, 0, 1]], np.float64)
    T = np.array([[0, 1, 2], [1, 3, 2], [1, 4, 3]], np.int32)
    rng = np.random.default_rng(7)
    order = rng.permutation(4500)
    F = T[order % 3]
    P = np.vstack([rng.uniform(-1, 2, (70, 3)), V])
    d2, fi = metrics.point_mesh_sqdist(P, V, F)
    ref, at = metrics.point_mesh_sqdist(P, V, T)
    assert np.array_equal(d2, ref)
    first = np.array([np.flatnonzero(order % 3 == k)[0] for k in range(3)])
    # a corner or an edge may belong to several triangles at the same distance: then the smallest of all
    want = [min(first[k] for k in range(3) if _same(P[i], V, T[k], ref[i])) for i in range(len(P))]
    assert np.array_equal(fi, want)


def _same(p, V, t, d2):
    return metrics.point_mesh_sqdist(p[None], V, t[None])[0][0] == d2


@pytest.mark.parametrize("faces", [1, 2, None])
def test_points_without_a_distance(faces):
    """A point with a coordinate that is not finite is infinitely far from every triangle; the others are not affected."""
    V, F = meshes.sphere(9)
    V, F = V.astype(np.float64), F[:faces]
    P = np.random.default_rng(8).normal(0, 1, (96, 3))
    ref, at = metrics.point_mesh_sqdist(P, V, F)
    bad = np.arange(0, 96, 7)
    Q = P.copy()
    Q[bad, bad % 3] = np.where(bad % 2 == 0, np.nan, np.inf)
    d2, fi = metrics.point_mesh_sqdist(Q, V, F)
    good = np.setdiff1d(np.arange(96), bad)
    assert np.array_equal(d2[good], ref[good]) and np.array_equal(fi[good], at[good])
    assert np.isinf(d2[bad]).all() and (fi[bad] == -1).all()


def test_a_mesh_that_float_sees_as_one_point():
    """A flat mesh of 4.5M faces far below the points, which lie in the box that a far triangle spans: to float every face is
    as near as any other, more than the nodes that a walk may take; the walk in float64 tells them apart."""
    n = 1500
    x, y = np.meshgrid(np.linspace(0, 1, n + 1), np.linspace(0, 1, n + 1), indexing="ij")
    V = np.column_stack([x.ravel(), y.ravel(), np.zeros(x.size)])
    k = np.arange((n + 1) * (n + 1)).reshape(n + 1, n + 1)
    a, b, c, d = k[:-1, :-1].ravel(), k[1:, :-1].ravel(), k[1:, 1:].ravel(), k[:-1, 1:].ravel()
    F = np.concatenate([np.stack([a, b, c], 1), np.stack([a, c, d], 1), len(V) + np.arange(3)[None]]).astype(np.int32)
    V = np.vstack([V, [[4e7, 4e7, 1e7], [4e7 + 10, 4e7, 1e7], [4e7, 4e7 + 10, 1e7]]])
    P = np.column_stack([np.linspace(0.1, 0.9, 9), np.linspace(0.9, 0.1, 9), np.linspace(2e6, 5e6, 9)])
    d2, fi = metrics.point_mesh_sqdist(P, V, F)
    assert np.allclose(d2, P[:, 2] ** 2, rtol=1e-9, atol=0) and (fi >= 0).all() and (fi < len(F) - 1).all()


def _all_sqdist(p, V, F):
    """Squared distances of p to every face by the kernel's operations (Ericson, Real-Time Collision Detection, 5.1.5) in
    float64 and in its order."""
    dot = lambda u, w: u[..., 0] * w[..., 0] + u[..., 1] * w[..., 1] + u[..., 2] * w[..., 2]
    a, b, c = V[F[:, 0]], V[F[:, 1]], V[F[:, 2]]
    ab, ac, ap, bp, cp = b - a, c - a, p - a, p - b, p - c
    d1, d2, d3, d4, d5, d6 = dot(ab, ap), dot(ac, ap), dot(ab, bp), dot(ac, bp), dot(ab, cp), dot(ac, cp)
    va, vb, vc = d3 * d6 - d5 * d4, d5 * d2 - d1 * d6, d1 * d4 - d3 * d2
    with np.errstate(all="ignore"):
        t, u, w, den = d1 / (d1 - d3), d2 / (d2 - d6), (d4 - d3) / ((d4 - d3) + (d5 - d6)), 1.0 / (va + vb + vc)
        s, r = vb * den, vc * den
        q = a + (ab * s[:, None] + ac * r[:, None])
        q = np.where(((va <= 0) & (d4 - d3 >= 0) & (d5 - d6 >= 0))[:, None], b + w[:, None] * (c - b), q)
        q = np.where(((vb <= 0) & (d2 >= 0) & (d6 <= 0))[:, None], a + u[:, None] * ac, q)
        q = np.where(((d6 >= 0) & (d5 <= d6))[:, None], c, q)
        q = np.where(((vc <= 0) & (d1 >= 0) & (d3 <= 0))[:, None], a + t[:, None] * ab, q)
        q = np.where(((d3 >= 0) & (d4 <= d3))[:, None], b, q)
        q = np.where(((d1 <= 0) & (d2 <= 0))[:, None], a, q)
    return dot(q - p, q - p)


@pytest.mark.parametrize("away", [0.0, 1e3, 1e12])
@pytest.mark.parametrize("far", [1.0, 1e2, 1e6, 1e9, 1e12, 1e15, 1e18])
def test_the_smallest_index_of_equally_near_faces(far, away):
    """The face by trying all in float64, where from far away many are equally near after rounding; with a far face, whose
    box the points lie near (then the float walk takes them), and without."""
    V, F = meshes.sphere(9)
    V = V.astype(np.float64)
    if away:
        F = np.vstack([F, len(V) + np.arange(3)[None]]).astype(np.int32)
        V = np.vstack([V, away * np.array([[4, 4, 4], [4.25, 4, 4], [4, 4.25, 4]])])
    rng = np.random.default_rng(12)
    P = -far * np.abs(rng.normal(0, 1.0, (97, 3)))  # on the other side than the far face
    d2, fi = metrics.point_mesh_sqdist(P, V, F)
    for i, p in enumerate(P):
        all_d2 = _all_sqdist(p, V, F)
        assert d2[i] == all_d2.min() and fi[i] == np.flatnonzero(all_d2 == all_d2.min())[0], (far, away, i)


def _seconds(P, V, F):
    metrics.point_mesh_sqdist(P, V, F)
    best = np.inf
    for _ in range(3):
        t = time.perf_counter()
        metrics.point_mesh_sqdist(P, V, F)
        best = min(best, time.perf_counter() - t)
    return best


@pytest.mark.parametrize("kind", ["far vertex", "flat", "far points"])
def test_time_where_float_is_coarse(kind):
    """The walks stay walks: with margins of the whole scene's size every triangle was evaluated in float64 for every point,
    400 to 1,300 times the time of points near the mesh; now 2 to 25 times. 100 times is far from either."""
    rng = np.random.default_rng(9)
    if kind == "flat":
        V, F = meshes.open_patch(200)
        V = V.astype(np.float64)
        V[:, 2] = 0.0
        near = np.column_stack([rng.uniform(0, 1, (2000, 2)), rng.uniform(0, 0.01, 2000)])
        P = near * [1, 1, 1e4]
    else:
        V, F = meshes.sphere(64)
        V = V.astype(np.float64)
        n = 20000 if kind == "far vertex" else 2000
        near = V[rng.integers(0, len(V), n)] * rng.uniform(0.99, 1.01, (n, 1))
        P = near * (1e6 if kind == "far points" else 1.0)
    base = _seconds(near, V, F)
    if kind == "far vertex":
        V = np.vstack([V, [[1e6, 1e6, 1e6]]])
        F = np.vstack([F, [[0, 1, len(V) - 1]]]).astype(np.int32)
    assert _seconds(P, V, F) < 100 * base
