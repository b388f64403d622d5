"""Removed faces (all three indices -1) in the centre of the stage-2 loop: NumPy's indexing takes the last vertex for them."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 600])
def test_a_removed_face_counts_as_the_last_vertex(n):
    import pamo_gb300

    rng = np.random.default_rng(n)
    v = rng.uniform(-1, 2, (40, 3)).astype(np.float32)
    f = rng.integers(0, 40, (n, 3)).astype(np.int32)
    f[::2] = -1
    s = np.zeros(3, np.float32)
    for a, b, c in f:
        s = s + ((v[a] + v[b]) + v[c]) / np.float32(3)
    got = pamo_gb300.tris_mean(torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda())
    assert s.dtype == np.float32 and np.array_equal(got, s / np.float32(n))
