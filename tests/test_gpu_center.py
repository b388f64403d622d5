"""The centre of the stage-2 loop: the chunk-parallel sequential float32 sum gives the bits of the element-by-element
sum at the chunk and window edges and for inputs whose sums tie, cross binades, cancel or are not finite."""

import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _values(kind, n):
    rng = np.random.default_rng(n)
    if kind == "positive":
        x = rng.uniform(0.5, 1.5, (n, 3))
    elif kind == "ties":  # multiples of 1/4 under sums that reach spacings of 1/2 and more
        x = rng.integers(-3, 9, (n, 3)) * 0.25 * np.array([2.0 ** 12, 2.0 ** 16, 2.0 ** 20])
        x[0] += np.array([2.0 ** 35, 2.0 ** 37, 2.0 ** 43])
    elif kind == "cancelling":
        x = rng.normal(0, 1, (n, 3))
    elif kind == "tiny":
        x = rng.normal(0, 1, (n, 3)) * np.array([1e-38, 1e-41, 1e-30])
    else:  # an infinity on one coordinate, a NaN on another
        x = rng.uniform(-1, 2, (n, 3))
        x[n // 2, 1], x[n // 3, 2] = np.inf, np.nan
    return x.astype(np.float32)


@pytest.mark.parametrize("kind", ["positive", "ties", "cancelling", "tiny", "non_finite"])
@pytest.mark.parametrize("n", [1, 3, 511, 512, 513, 1025, 32 * 512, 33 * 512 + 1, 200003])
def test_centre_is_the_sequential_sum(kind, n):
    import pamo_gb300

    v = _values(kind, n)
    f = np.repeat(np.arange(n, dtype=np.int32)[:, None], 3, axis=1)
    got = pamo_gb300.tris_mean(torch.from_numpy(v).cuda(), torch.from_numpy(f).cuda())
    with np.errstate(all="ignore"):
        want = orc.tris_mean(v, f)
    np.testing.assert_array_equal(got, want)
