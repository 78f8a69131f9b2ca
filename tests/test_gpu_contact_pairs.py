"""The contact pass of an evaluation (leaf cache, pair pool, FP64 pass per
pair) against the contact query at the same state, where one thread walks the
tree and evaluates every candidate of an element in turn: bit for bit, in both
solve modes, where the pass takes its rarer ways: leaf lists in the pool and
hundreds of candidates an element (a mesh pole), more pairs than the pool
holds, and elements too far out for the leaf cache."""
import numpy as np
import pytest

import khs_native as kn
import parity
import scenes

pytestmark = pytest.mark.gpu


def _far(offset):
    sc = scenes.pole_scene(strands=24, nodes=16)
    shift = np.array([offset, 0.0, 0.0])
    roots, collider = sc.root_points_at, sc.collider_at
    sc.points, sc.vertices = sc.points + shift, sc.vertices + shift
    sc.root_points_at = lambda f: roots(f) + shift
    sc.collider_at = lambda f: collider(f) + shift
    return sc


SCENES = {
    "pole": lambda: scenes.pole_scene(strands=24, nodes=16),
    "more pairs than the pool": lambda: scenes.pole_scene(strands=900, nodes=16),
    "63 m": lambda: _far(63.0),
    "100 m": lambda: _far(100.0),
}


@pytest.mark.parametrize("mode", [kn.MODE_PLAIN_FP64, kn.MODE_MIXED])
@pytest.mark.parametrize("name", list(SCENES))
def test_contact_pass_matches_the_query(gpu_lib, name, mode):
    sc = SCENES[name]()
    s = kn.HairSolver(gpu_lib)
    scenes.load_into(s, sc)
    s.set_solve_mode(mode)
    s.set_substep_limit(1)
    s._library.khsStepAnimationFrame(s.handle, 1, sc.frame_dt)  # the records count, converged or not
    got = s.contact_records()
    q, _ = s.state()
    want = s.query_contacts(q)
    mism = parity.records_equal(got, want)
    assert all(v == 0 for v in mism.values()), mism
    assert np.array_equal(got["gap"].view(np.uint64), want["gap"].view(np.uint64))
    assert want["candidate_count"].sum() > 0
    if name == "more pairs than the pool":
        assert want["candidate_count"].sum() > 1 << 18  # the pool's size for small scenes
    s.close()
