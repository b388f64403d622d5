"""A limit that the build of one of stage 3's trees ran into reaches the caller."""

import numpy as np
import pytest

from tests import meshes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", [1, 0])
def test_a_tree_build_that_gave_up_is_an_error(graphs):
    """A test knob sets the trees' status words as a scan or a climb that gave up does (kErrIterLimit)."""
    from pamo_gb300 import PamoError, safe_project

    GV, GF, V, F = meshes.stage3_pair()
    s = safe_project.Stage3System(None, "cuda:0")
    s.set("use_cuda_graph", graphs)
    good = s.project(GV, GF, V, F, 1).cpu().numpy()
    s.set("test_tree_status", 8)
    with pytest.raises(PamoError) as e:
        s.project(GV, GF, V, F, 1)
    assert "BVH" in str(e.value)
    s.set("test_tree_status", 0)
    assert np.array_equal(s.project(GV, GF, V, F, 1).cpu().numpy(), good)
