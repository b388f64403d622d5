"""The whole-mesh self-intersection check (pamo_self_intersect) against the oracle's global check."""

import numpy as np
import pytest
import torch

from oracle import oracle as orc
from tests import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed,amp", [(9, 0.25), (10, 0.4), (11, 0.1)])
def test_flags_match_oracle(seed, amp):
    import pamo_gb300

    v, f = meshes.tangled(10, seed=seed, amp=amp)
    ref, nhits = orc.Oracle().self_intersect(v, f)
    assert nhits > 0
    got = pamo_gb300.self_intersect(torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda()).cpu().numpy()
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("faces", [1, 2, 3, 31, 33, 511, 512, 513, 1025, 1537, 2880])
def test_flags_at_the_edges_of_tiles_and_warps(faces):
    """Trees of one leaf to several bottom-up tiles of 512, and walks of one to many queries a warp."""
    import pamo_gb300

    v, f = meshes.tangled(12, seed=21, amp=0.3)
    f = np.ascontiguousarray(f[np.random.default_rng(2).permutation(len(f))[:faces]])
    ref, _ = orc.Oracle().self_intersect(v, f)
    got = pamo_gb300.self_intersect(torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda()).cpu().numpy()
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("n", [40, 41])
def test_flags_at_the_edge_of_the_sort_rule(n):
    """32,000 and 33,620 faces: 16 tiles of the radix sort (a launch a pass) and 17 (a count, a scan and a scatter)."""
    import pamo_gb300

    v, f = meshes.tangled(n, seed=n, frac=0.02, amp=0.05)
    ref, _ = orc.Oracle().self_intersect(v, f)
    got = pamo_gb300.self_intersect(torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda()).cpu().numpy()
    assert ref.sum() > 0 and np.array_equal(got, ref)


def test_star_shaped_input_is_clean():
    import pamo_gb300
    from pamo_gb300 import synth

    v, f = synth.config_mesh("plain_small", seed=0)
    got = pamo_gb300.self_intersect(torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda()).cpu().numpy()
    assert got.sum() == 0
