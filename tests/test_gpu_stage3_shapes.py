"""The launch shapes of stage 3's solve and line search where their branches meet: contacts with a barrier term under two
threads a sum, more elements a thread than the solve's mask has bits, and searches that go past their first launch or find
no trial. cg_mode 7 (one thread a sum, two launches an iteration) and ls_mode 0 (a launch pair
a trial) give the bits to compare with."""

import numpy as np
import pytest

from tests import meshes

pytestmark = pytest.mark.gpu


def _pushed_sheets(n):
    V, F = meshes.sheet_pair(n)
    GV = V.copy()
    GV[: len(V) // 2, 2] += 0.0012  # pulls the lower sheet into the upper one
    return GV, F, V, F


def _run(case, steps, cg=0, ls=1, **cfg):
    from pamo_gb300 import safe_project

    s = safe_project.Stage3System(safe_project.Stage3Config(**cfg), "cuda:0")
    s.set("cg_mode", cg)
    s.set("ls_mode", ls)
    return s.project(*case, steps).cpu().numpy(), s.stats()


def test_contacts_with_a_barrier_term_under_two_threads_a_sum():
    """13,924 faces in two sheets 0.6 barrier distances apart: more elements than the grid has threads (152 blocks of 128)
    without the contacts, whose terms are not zero."""
    case = _pushed_sheets(60)
    out, st = _run(case, 1)
    ref, _ = _run(case, 1, cg=7)
    off, _ = _run(case, 1, coll_stiffness=0.0)
    assert st["max_contacts"] > 0 and np.isfinite(out).all()
    assert not np.array_equal(out, off)  # the barrier moved the sheets
    assert np.array_equal(out, ref)


@pytest.mark.parametrize("cg", [0, 3])
def test_more_rounds_of_elements_than_the_mask_has_bits(cg):
    """324 faces with every pair within 0.6 of the box: 8 blocks of 128 threads (4 of 256), 100 rounds of contacts."""
    case = _pushed_sheets(10)
    out, st = _run(case, 1, cg=cg, contact_detection_radius=0.3)
    assert st["max_contacts"] > 66 * 8 * 128
    assert np.array_equal(out, _run(case, 1, cg=7, contact_detection_radius=0.3)[0])


@pytest.fixture(scope="module")
def star_searches():
    case = meshes.stage3_pair()
    return {n: (_run(case, 5, ls=1, n_line_search_iters=n)[0], _run(case, 5, ls=0, n_line_search_iters=n)[0])
            for n in (1, 2, 3, 10, 11, 64, 65)}


@pytest.mark.parametrize("trials", [1, 2, 3, 10, 11, 64, 65])
def test_trials_side_by_side_and_one_after_another(star_searches, trials):
    """The first launch takes two trials, the others eight each, 65 fall back to launch pairs."""
    side_by_side, pairs = star_searches[trials]
    assert np.array_equal(side_by_side, pairs)


def test_some_searches_go_past_each_launch(star_searches):
    """The bits change with the number of trials allowed only where a search used them all: some take a third trial, and some
    lower the energy by none of ten or eleven."""
    out = {n: star_searches[n][0] for n in star_searches}
    for few, more in ((1, 2), (2, 3), (3, 10), (10, 11), (11, 64)):
        assert not np.array_equal(out[few], out[more]), (few, more)
