"""The bytes that the serving loop reserves for a request before its solver is
built cover what the built solver holds, from the smallest grooms, where the
arena's pools have their least size, to those of the request stream."""
import pytest

import khs_native as kn
import scenes
import serving

pytestmark = pytest.mark.gpu


def _bald(sc):
    sc.vertices = sc.triangles = sc.collider_at = None
    return sc


SCENES = {
    "1 strand": lambda: _bald(scenes.ellipsoid_scene(strands=1, node_range=(3, 3), frames=1)),
    "64 strands of 32": lambda: scenes.sphere_scene(motion=True, frames=2),
    "12 at a mesh pole": lambda: scenes.pole_scene(strands=12, nodes=16),
    "3,000 of 2 or 3": lambda: _bald(scenes.ellipsoid_scene(strands=3000, node_range=(2, 3), frames=1)),
    "500 of 16-160": lambda: scenes.ellipsoid_scene(strands=500, node_range=(16, 160), frames=10, level=4),
}


@pytest.mark.parametrize("ring", [0, 10])
@pytest.mark.parametrize("name", list(SCENES))
def test_estimate_covers_the_built_solver(gpu_lib, name, ring):
    sc = SCENES[name]()
    s = kn.HairSolver(gpu_lib)
    scenes.load_into(s, sc)
    if ring:
        s.set_rollback_ring(ring)
    held, reserved = serving.resident_bytes(s), serving.estimate_bytes(sc, ring)
    s.close()
    print(name, held, reserved)
    assert held <= reserved
