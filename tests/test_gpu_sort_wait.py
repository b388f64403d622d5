"""The radix sort's bounded waits: a tile whose counts have not come when the wait runs out is counted by the tile that waits,
so the sorted tree, and with it every flag and every simplified mesh, is the same whether or not a wait ran out."""

import numpy as np
import pytest
import torch

from oracle import oracle as orc
from tests import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wait", [0, 1, 3])
@pytest.mark.parametrize("n", [11, 15, 32, 40])
def test_flags_when_the_sorts_waits_run_out(n, wait):
    """2,420 to 32,000 faces: 2 to 16 tiles. With a limit of no polls at all every tile counts all those before it."""
    import pamo_gb300

    v, f = meshes.tangled(n, seed=n, frac=0.03, amp=4.0 / n)
    ref, _ = orc.Oracle().self_intersect(v, f)
    ctx = pamo_gb300.Context("cuda:0")
    ctx.set_option("test_sort_wait", wait)
    pts, tris = torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda()
    assert ref.sum() > 0
    for _ in range(2):  # the second build finds the first one's counts in the buffers
        assert np.array_equal(pamo_gb300.self_intersect(pts, tris, ctx=ctx).cpu().numpy(), ref)


def test_simplified_mesh_when_the_sorts_waits_run_out():
    import pamo_gb300

    v, f = meshes.sphere(24, seed=5)
    pts, tris = torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda()
    out = []
    for wait in (1 << 22, 0):
        ctx = pamo_gb300.Context("cuda:0")
        ctx.set_option("test_sort_wait", wait)
        V, F, rounds = pamo_gb300.simplify(pts, tris, 0.05, 4, 1e-3, min_verts=0, ctx=ctx)
        out.append((V.cpu(), F.cpu(), rounds))
    assert out[0][2] == out[1][2] and torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
