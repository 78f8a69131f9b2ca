"""The line-search CCD bound with more pairs than its list holds: the first trial
of an iteration is discarded and one thread per element takes the bound again.
Strands of long segments laid around a turning sphere of small triangles, so that
an element's box holds a hundred of them: the plain form, whose candidates are
all pairs, against the mixed form, whose FP32 filter drops most: same result code,
substep records and state, bit for bit."""
import ctypes

import numpy as np
import pytest

import khs_native as kn
import scenes

pytestmark = pytest.mark.gpu


def _laid_around(strands, nodes=10, segment=0.015, height=2.0e-3, level=6):
    """Great-circle arcs over a sphere of 0.1 m at a height, in any direction."""
    rng = np.random.default_rng(5)
    radius = 0.1
    v, f = scenes.icosphere(level)
    v = v * radius
    n, t = rng.normal(size=(2, strands, 3))
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    t -= n * np.sum(n * t, 1, keepdims=True)
    t /= np.linalg.norm(t, axis=1, keepdims=True)
    angle = 2.0 * np.arcsin(0.5 * segment / (radius + height)) * np.arange(nodes)
    arc = np.cos(angle)[None, :, None] * n[:, None, :] + np.sin(angle)[None, :, None] * t[:, None, :]
    points, offsets = scenes._assemble(list((radius + height) * arc))

    def turned(p):
        return lambda frame: p @ scenes._rotation_z(0.5 * frame / 24.0).T

    return scenes.Scene("arcs", points, offsets, v, f, 2, 24.0, dict(substeps=1, maximum_substeps=1, fixed_root_nodes=2),
                        dict(scenes.HAIR_MATERIAL_SMALL), turned(points), turned(v))


@pytest.mark.parametrize("strands, full", [(30, False), (5000, True)])
def test_full_ccd_list_falls_back(gpu_lib, strands, full):
    sc = _laid_around(strands)
    runs = []
    for mode in (kn.MODE_PLAIN_FP64, kn.MODE_MIXED):
        s = kn.HairSolver(gpu_lib)
        scenes.load_into(s, sc)
        s.set_solve_mode(mode)
        s.set_profiling(True)
        before, _ = s.state()
        r = s._library.khsStepAnimationFrame(s.handle, 1, sc.frame_dt)
        q, v = s.state()
        records = [bytes(ctypes.string_at(ctypes.byref(x), ctypes.sizeof(x))) for x in s.substep_records()]
        timings = {k: t[0] if isinstance(t, tuple) else t for k, t in s.kernel_timings().items()}
        runs.append((r, records, q, v, timings))
        print(mode, r, len(records), timings.get("k_ccd"), float(np.abs(q - before).max()))
        assert len(records) == 1 and r == kn.OK
        assert not np.array_equal(q, before)
        s.close()
    (ra, sa, qa, va, ta), (rb, sb, qb, vb, _) = runs
    assert ("k_ccd" in ta) == full
    assert ra == rb and sa == sb
    assert np.array_equal(qa, qb) and np.array_equal(va, vb)
