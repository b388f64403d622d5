"""Precision mode 2 places an edge without a cost of its own in the round (a boundary edge, or any edge of a stuck round, which
may collapse by the stale cost that the reference keeps) at its midpoint."""

import numpy as np
import pytest
import torch

from tests import meshes

pytestmark = pytest.mark.gpu


def _midpoints(v, e):
    return (v[e[:, 0]] + v[e[:, 1]]) / np.float32(2)


def test_boundary_edges_are_placed_at_their_midpoints():
    import pamo_gb300

    v, f = meshes.open_patch(14)
    e, c, p = pamo_gb300.cost_probe(torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda(), 1.0, 1e-3, 2)
    e, c, p = e.cpu().numpy(), c.cpu().numpy(), p.cpu().numpy()
    half = np.sort(np.concatenate([f[:, [0, 1]], f[:, [1, 2]], f[:, [2, 0]]]), 1)
    pairs, count = np.unique(half, axis=0, return_counts=True)
    outer = {tuple(x) for x in pairs[count == 1]}
    rim = np.array([tuple(sorted(x)) in outer for x in e])
    # the edges of the rim that have an entry (an edge is listed by the face that runs through it downwards)
    assert rim.sum() > 10 and np.isnan(c[rim]).all()
    assert np.array_equal(p[rim], _midpoints(v, e)[rim])


def test_a_stuck_round_places_at_midpoints():
    """Two rounds, the second stuck: each vertex that moved lies at the midpoint of an edge that it had."""
    import pamo_gb300

    v, f = meshes.sphere(16, seed=3)
    op = pamo_gb300.CUDSP_Free()
    dev = torch.device("cuda", 0)
    op._context(dev).set_option("precision", 2)
    none = torch.zeros(0, dtype=torch.int32, device=dev)
    V, F, occ, vmap, undo = op.forward(torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda(), none, 0, 2.0, 1e-3, False, True)
    V = V[occ.view(-1).bool()].contiguous()
    F = F[F[:, 0] >= 0]
    F = vmap.view(-1)[F.long()].to(torch.int32).contiguous()
    V2, F2, occ2, _, _ = op.forward(V, F, none, 0, 2.0, 1e-3, True, False)
    before, after, faces = V.cpu().numpy(), V2.cpu().numpy(), F.cpu().numpy()
    alive = occ2.view(-1).bool().cpu().numpy()
    moved = np.flatnonzero(alive & (before != after).any(1))
    assert len(moved) > 0
    for u in moved:
        ring = np.unique(faces[(faces == u).any(1)])
        ring = ring[ring != u]
        mid = (before[ring] + before[u]) / np.float32(2)
        assert (mid == after[u]).all(1).any()
