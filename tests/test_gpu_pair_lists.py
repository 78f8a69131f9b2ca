"""The moving-collider sweep and the CCD bound with more pairs than their list
holds, where one thread per element takes over: the plain form (every
candidate a pair) against the mixed form, whose FP32 filters drop most: same result code, substep records, failure diagnostics and state."""
import ctypes

import numpy as np
import pytest

import khs_native as kn
import scenes

pytestmark = pytest.mark.gpu


def _scene(strands, drift):
    sc = scenes.pole_scene(strands=strands, nodes=16, substeps=1)
    roots, collider = sc.root_points_at, sc.collider_at
    sc.root_points_at = lambda f: roots(f) + np.array([0.0, 0.0, drift * f])
    sc.collider_at = lambda f: collider(f) + np.array([0.0, 0.0, drift * f])
    sc.desc["maximum_substeps"] = 2
    return sc


@pytest.mark.parametrize("strands, drift, full", [(12, 0.002, False), (2400, 0.03, True)])
def test_full_pair_lists_fall_back(gpu_lib, strands, drift, full):
    sc = _scene(strands, drift)
    runs = []
    for mode in (kn.MODE_PLAIN_FP64, kn.MODE_MIXED):
        s = kn.HairSolver(gpu_lib)
        scenes.load_into(s, sc)
        s.set_solve_mode(mode)
        s.set_substep_limit(1)
        s.set_profiling(True)
        r = s._library.khsStepAnimationFrame(s.handle, 1, sc.frame_dt)
        timings = s.kernel_timings()
        diag = s.failure_diagnostics()
        runs.append((r, s.state(), bytes(ctypes.string_at(ctypes.byref(diag), ctypes.sizeof(diag))),
                     [bytes(ctypes.string_at(ctypes.byref(x), ctypes.sizeof(x))) for x in s.substep_records()], timings))
        print(mode, r, sorted(timings), diag.kind)
        s.close()
    (ra, (qa, va), da, sa, ta), (rb, (qb, vb), db, sb, tb) = runs
    assert ra == rb and da == db and sa == sb
    assert np.array_equal(qa, qb) and np.array_equal(va, vb)
    if full:
        assert "k_sweep" in ta
    else:
        assert "k_sweep" not in ta
