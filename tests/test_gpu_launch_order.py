"""Frames with the contact passes on the side stream and launches that come up
early, against the same frames with one kernel after the other on one stream
(which timing the kernels one by one asks for): bit for bit, in every solve
mode."""
import ctypes

import numpy as np
import pytest

import khs_native as kn
import scenes

pytestmark = pytest.mark.gpu

SCENES = {
    "sphere": lambda: scenes.sphere_scene(motion=True, frames=3),
    "ellipsoid": lambda: scenes.ellipsoid_scene(strands=200, frames=2),
    "no collider": lambda: _bald(scenes.ellipsoid_scene(strands=60, frames=2)),
}


def _bald(sc):
    sc.vertices = sc.triangles = sc.collider_at = None
    return sc


@pytest.mark.parametrize("mode", [kn.MODE_PLAIN_FP64, kn.MODE_MIXED, kn.MODE_MIXED_FF])
@pytest.mark.parametrize("name", list(SCENES))
def test_overlapped_launches_match_one_after_the_other(gpu_lib, name, mode):
    sc = SCENES[name]()
    runs = []
    for one_by_one in (False, True):
        s = kn.HairSolver(gpu_lib)
        scenes.load_into(s, sc)
        s.set_solve_mode(mode)
        s.set_output_ring(2)
        s.set_profiling(one_by_one)
        out = []
        for f in range(1, sc.frames):
            assert s._library.khsStepAnimationFrame(s.handle, f, sc.frame_dt) == kn.OK, s.last_error()
            out += [*s.state(), s.output_frame(f)]
            out += [np.frombuffer(ctypes.string_at(ctypes.byref(x), ctypes.sizeof(x)), np.uint8) for x in s.substep_records()]
        runs.append(out)
        s.close()
    assert len(runs[0]) == len(runs[1])
    for a, b in zip(*runs):
        assert np.array_equal(a, b)
