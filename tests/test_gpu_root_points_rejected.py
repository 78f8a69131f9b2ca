"""Root target points with a non-finite coordinate are rejected on the device
with the code and message the host check gave, before a bad frame index or too
small output arrays are, whichever point it is, and change nothing."""
import numpy as np
import pytest

import khs_native as kn
import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("at", [0, 777, -1])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_non_finite_points(gpu_lib, at, value):
    sc = scenes.sphere_scene(motion=True)
    s = kn.HairSolver(gpu_lib)
    scenes.load_into(s, sc)
    good = np.ascontiguousarray(sc.root_points_at(1))
    before = s.compute_root_targets(good)
    phase = s.progress().phase
    bad = good.copy()
    bad[at, 1] = value
    lib, n = s._library, s.build_stats().internal_node_count
    out = np.zeros((n, 3))
    calls = [lambda: lib.khsUpdateRootTargets(s.handle, kn._ptr(bad), len(bad)),
             lambda: lib.khsSetRootAnimationFrame(s.handle, 10 ** 6, kn._ptr(bad), len(bad)),
             lambda: lib.khsxComputeRootTargets(s.handle, kn._ptr(bad), len(bad), kn._ptr(out), kn._ptr(out), n),
             lambda: lib.khsxComputeRootTargets(s.handle, kn._ptr(bad), len(bad), kn._ptr(out), kn._ptr(out), n - 1)]
    for call in calls:
        assert call() == kn.ERROR_INVALID_HAIR
        assert s.last_error() == "root targets have a non-finite coordinate"
        assert s.progress().phase == phase
    assert not out.any()
    after = s.compute_root_targets(good)
    assert np.array_equal(before[0], after[0]) and np.array_equal(before[1], after[1])
    s.close()
