"""The work a user of the solver has it do, case by case.

A case is one call a bake, a live viewport or the serving loop makes:

* ``frame``   -- one animation frame of a bake (khsStepAnimationFrame with
                 every frame's targets resident), stepped again from the
                 rollback ring's copy of the frame before it, then read back.
* ``live``    -- one frame with the roots and the collider uploaded before it
                 (khsUpdateRootTargets, khsUpdateColliderVertices, khsStep).
* ``serving`` -- one frame of several requests at once, a host thread each.
* ``roots``   -- the root targets of one set of evaluated source points
                 (khsxComputeRootTargets).

Scenes come from the package's own generators; their sizes are those of the
repository's tests, its serving stream and its benchmark.  ``plain`` is the
library's default solve mode, ``mixed`` the one bakes and the serving loop
select.
"""
import concurrent.futures
import functools
import math
import sys
from pathlib import Path

import numpy as np

PACKAGE = Path(__file__).resolve().parents[1] / "kami-hair-solver_gb300"
if str(PACKAGE) not in sys.path:
    sys.path.insert(0, str(PACKAGE))

import khs_native as kn  # noqa: E402
import scenes  # noqa: E402

MODES = {"plain": kn.MODE_PLAIN_FP64, "mixed": kn.MODE_MIXED}

# Typical Gauss-Newton iterations and substeps of one frame, for work().
ITERATIONS = {"sphere": 2, "pole": 16, "ellipsoid": 12, "body": 12}
NODES_PER_BODY_STRAND = scenes.BODY_NODES / scenes.BODY_STRANDS


def listed():
    return [
        # The smallest call: the reference's own small test scene in the
        # library's default mode, where launches and latency are the cost.
        dict(name="sphere 64 plain", kind="frame", scene="sphere", strands=64, nodes=32, substeps=4, mode="plain", frame=1),
        # An interactive viewport: new roots and collider uploaded each frame.
        dict(name="sphere 64 live", kind="live", scene="sphere", strands=64, nodes=32, substeps=4, mode="mixed", frame=1),
        # Hair across a mesh pole: few strands, hundreds of triangles around
        # each element.
        dict(name="pole 12", kind="frame", scene="pole", strands=12, nodes=16, substeps=4, mode="mixed", frame=1),
        # The smallest request of the serving stream.
        dict(name="request 100", kind="frame", scene="ellipsoid", strands=100, low=16, high=160, level=4, substeps=8,
             collider=True, mode="mixed", frame=1),
        # A test-sized groom in the default mode, with contacts.
        dict(name="ellipsoid 80 plain", kind="frame", scene="ellipsoid", strands=80, low=16, high=64, level=5, substeps=4,
             collider=True, mode="plain", frame=1),
        # The 1,000-strand contact groom of the parity reports.
        dict(name="ellipsoid 1000", kind="frame", scene="ellipsoid", strands=1000, low=20, high=120, level=5, substeps=8,
             collider=True, mode="mixed", frame=2),
        # Hair without a collider: rods, inertia and the block solve alone.
        dict(name="hair only 500", kind="frame", scene="ellipsoid", strands=500, low=16, high=160, level=4, substeps=8,
             collider=False, mode="plain", frame=2),
        # A large request of the serving stream, alone on the card.
        dict(name="request 2000", kind="frame", scene="ellipsoid", strands=2000, low=16, high=160, level=5, substeps=8,
             collider=True, mode="mixed", frame=1),
        # A thinner groom on the benchmark's collider in the default mode, at
        # its first contacts.
        dict(name="body 700 plain", kind="frame", scene="body", strands=700, mode="plain", frame=4),
        # The benchmark's full scene at a contact-heavy frame.
        dict(name="body 6757", kind="frame", scene="body", strands=6757, mode="mixed", frame=5),
        # Four requests of the stream stepping at the same time.
        dict(name="serving 4", kind="serving", requests=4, strands=200, low=16, high=160, level=4, substeps=8, mode="mixed"),
        # The root targets of a large groom, as a bake sets them frame by frame.
        dict(name="root targets 4000", kind="roots", scene="ellipsoid", strands=4000, low=16, high=160),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ellipsoid", "ellipsoid", "ellipsoid", "sphere", "body", "roots", "serving", "pole"])
    mode = rng.choice(["mixed", "mixed", "plain"])
    if kind == "sphere":
        return dict(kind=rng.choice(["frame", "live"]), scene="sphere", strands=_log_uniform(rng, 16, 1024),
                    nodes=rng.randint(9, 64), substeps=rng.choice([4, 5, 8]), mode=mode, frame=1)
    if kind == "pole":
        return dict(kind="frame", scene="pole", strands=rng.randint(7, 40), nodes=rng.randint(12, 20), substeps=4,
                    mode="mixed", frame=1)
    if kind == "ellipsoid":
        mixed = mode == "mixed"
        return dict(kind="frame", scene="ellipsoid", strands=_log_uniform(rng, 33, 1500 if mixed else 80),
                    low=rng.randint(12, 24), high=rng.randint(40, 160 if mixed else 64), level=rng.choice([4, 5]),
                    substeps=rng.choice([4, 8]) if mixed else 4, collider=rng.random() < 0.85, mode=mode,
                    frame=rng.choice([1, 2]) if mixed else 1)
    if kind == "body":
        return dict(kind="frame", scene="body", strands=_log_uniform(rng, 300, 4000 if mode == "mixed" else 700), mode=mode,
                    frame=rng.choice([1, 4, 5] if mode == "mixed" else [1, 4]))
    if kind == "roots":
        return dict(kind="roots", scene="ellipsoid", strands=_log_uniform(rng, 100, 4000), low=rng.randint(5, 24),
                    high=rng.randint(40, 160))
    return dict(kind="serving", requests=rng.randint(2, 5), strands=_log_uniform(rng, 64, 250), low=16,
                high=rng.randint(60, 160), level=4, substeps=8, mode="mixed")


def _groom(case, seed):
    frame = case.get("frame", 1)
    if case["scene"] == "sphere":
        return scenes.sphere_scene(seed=seed, strands=case["strands"], nodes=case["nodes"], substeps=case["substeps"],
                                   frames=frame, motion=True)
    if case["scene"] == "pole":
        return scenes.pole_scene(seed=seed, strands=case["strands"], nodes=case["nodes"], substeps=case["substeps"], frames=frame)
    if case["scene"] == "ellipsoid":
        sc = scenes.ellipsoid_scene(seed=seed, strands=case["strands"], node_range=(case["low"], case["high"]),
                                    level=case.get("level", 4), substeps=case.get("substeps", 8), frames=frame)
        if not case.get("collider", False):
            sc.vertices = sc.triangles = sc.collider_at = None
        return sc
    return scenes.body_scene(seed=seed, strands=case["strands"],
                             total_nodes=int(round(NODES_PER_BODY_STRAND * case["strands"])), frames=frame)


def _scene(case, seed, attempt=0):
    """The case's groom (strand counts and collider are the case's own),
    turned about the vertical by a seeded angle and moving at a seeded pace."""
    sc = _groom(case, case["strands"] + 7919 * attempt)
    rng = np.random.default_rng(seed)
    a, pace = rng.uniform(0.0, 2.0 * math.pi), rng.uniform(0.9, 1.1)
    turn = np.array([[math.cos(a), math.sin(a), 0.0], [-math.sin(a), math.cos(a), 0.0], [0.0, 0.0, 1.0]])
    roots, collider = sc.root_points_at, sc.collider_at
    sc.points = sc.points @ turn
    sc.root_points_at = lambda frame: roots(frame * pace) @ turn
    if collider is not None:
        sc.vertices = sc.vertices @ turn
        sc.collider_at = lambda frame: collider(frame * pace) @ turn
    return sc


@functools.lru_cache(maxsize=None)
def _library():
    return kn.Library()


def _built(case, seed, animation=True):
    """A built solver and its scene.  A groom with a strand that starts
    inside the collider is refused by the build; its user makes another."""
    for attempt in range(16):
        sc = _scene(case, seed, attempt)
        solver = kn.HairSolver(_library())
        try:
            scenes.load_into(solver, sc, animation=animation)
            return solver, sc
        except kn.KhsError as e:
            solver.close()
            if e.code != kn.ERROR_INITIAL_INTERSECTION:
                raise
    raise RuntimeError("no groom outside the collider")


def _baked(case, seed):
    """A solver that has baked up to the frame before the case's."""
    solver, sc = _built(case, seed)
    solver.set_solve_mode(MODES[case["mode"]])
    solver.set_rollback_ring(2)
    for f in range(1, case["frame"]):
        solver.step_animation_frame(f, sc.frame_dt)
    return dict(kind="frame", solver=solver, frame=case["frame"], dt=sc.frame_dt)


def prepare(case, seed):
    if case["kind"] == "frame":
        return _baked(case, seed)
    if case["kind"] == "live":
        solver, sc = _built(case, seed, animation=False)
        solver.set_solve_mode(MODES[case["mode"]])
        # Frame 0 is the start that every pass goes back to.
        solver.allocate_animation(1)
        solver.set_root_animation_frame(0, sc.root_points_at(0))
        solver.set_collider_animation_frame(0, sc.collider_at(0))
        solver.finalize_animation()
        solver.set_rollback_ring(1)
        return dict(kind="live", solver=solver, dt=sc.frame_dt, points=sc.root_points_at(1), vertices=sc.collider_at(1))
    if case["kind"] == "serving":
        # Requests of the stream's mixed sizes: strand counts spread around
        # the case's.
        states = []
        for k in range(case["requests"]):
            one = dict(case, scene="ellipsoid", collider=True, frame=1, strands=max(33, int(case["strands"] * 2.0 ** (k - 1.5))))
            states.append(_baked(one, seed + 104729 * (k + 1)))
        pool = concurrent.futures.ThreadPoolExecutor(max_workers=case["requests"])
        list(pool.map(lambda _: None, range(case["requests"])))
        return dict(kind="serving", states=states, pool=pool)
    solver, sc = _built(case, seed, animation=False)
    return dict(kind="roots", solver=solver, points=_roots_points(seed, sc))


def _roots_points(seed, scene):
    """Evaluated source points away from the rest pose: the head turned and
    swaying, every strand bent a little."""
    rng = np.random.default_rng(seed + 17)
    a = 0.4 + 0.2 * rng.uniform()
    turn = np.array([[math.cos(a), -math.sin(a), 0.0], [math.sin(a), math.cos(a), 0.0], [0.0, 0.0, 1.0]])
    p = scene.root_points_at(1) @ turn.T
    return p + 0.002 * np.sin(40.0 * p[:, [1, 2, 0]] + rng.uniform(0, 6.0, size=3))


def _result(solver, positions, stats):
    q, v = solver.state()
    return dict(positions=positions, q=q, v=v,
                counts=np.array([stats.substeps, stats.converged_substeps, stats.newton_iterations, stats.linear_solves,
                                 stats.line_search_evaluations, stats.contact_candidate_count, stats.active_contact_count],
                                dtype=np.int64),
                energies=np.array([stats.kinetic_energy, stats.elastic_energy, stats.contact_energy]),
                gap=np.array([min(stats.minimum_gap, 1.0), stats.ccd_step_limit]))


def _frame(state):
    solver = state["solver"]
    solver.rollback_to_frame(state["frame"] - 1)
    return _result(solver, *solver.step_animation_frame(state["frame"], state["dt"]))


def run(state):
    if state["kind"] == "frame":
        return _frame(state)
    if state["kind"] == "live":
        solver = state["solver"]
        solver.rollback_to_frame(0)
        solver.update_roots(state["points"])
        solver.update_collider(state["vertices"])
        return _result(solver, *solver.step(state["dt"]))
    if state["kind"] == "serving":
        return list(state["pool"].map(_frame, state["states"]))
    return list(state["solver"].compute_root_targets(state["points"]))


def work(case):
    if case["kind"] == "roots":
        nodes = 0.5 * (case["low"] + case["high"]) * case["strands"]
        return dict(bytes=nodes * (24 + 72 + 20 + 48), flops=nodes * 300)
    if case["kind"] == "serving":
        one = [work(dict(case, kind="frame", scene="ellipsoid", collider=True, frame=1,
                         strands=max(33, int(case["strands"] * 2.0 ** (k - 1.5))))) for k in range(case["requests"])]
        return dict(bytes=sum(w["bytes"] for w in one), flops=sum(w["flops"] for w in one))
    if case["scene"] == "body":
        nodes, substeps = NODES_PER_BODY_STRAND * case["strands"], {1: 8, 4: 16, 5: 32}[case["frame"]]
    else:
        per = case["nodes"] if case["scene"] in ("sphere", "pole") else 0.5 * (case["low"] + case["high"])
        nodes, substeps = per * case["strands"], case["substeps"]
    iterations = substeps * ITERATIONS[case["scene"]]
    # Per iteration: the state, constants and targets read and the new state
    # written once (280 B a node, 56 B an element); the rods' gradient and
    # Gauss-Newton blocks, the rotations and the block-tridiagonal solve.
    return dict(bytes=iterations * nodes * (280 + 56), flops=iterations * nodes * (1089 + 365 + 1872))


# ---------------------------------------------------------------------------
# Root targets in 64 bits: positions are the source points; each node's frame
# carries its first director along the strand by the minimal rotation between
# tangents, and the rotation vector is that of frame * rest frame^T.

def _unit(a):
    return a / np.linalg.norm(a, axis=-1, keepdims=True)


def _frames(x, first, count, start):
    """Frames [N, 3, 3] (columns d1 d2 d3) along every strand of points x."""
    n = len(x)
    last = first + count - 1
    ends, starts = np.zeros(n, bool), np.zeros(n, bool)
    ends[last], starts[first] = True, True
    idx = np.arange(n)
    t = _unit(x[np.where(ends, idx, np.minimum(idx + 1, n - 1))] - x[np.where(starts, idx, np.maximum(idx - 1, 0))])
    frames = np.empty((n, 3, 3))

    def put(node, d1):
        d3 = t[node]
        d1 = _unit(d1 - d3 * np.sum(d1 * d3, 1, keepdims=True))
        d2 = _unit(np.cross(d3, d1))
        frames[node] = np.stack([_unit(np.cross(d2, d3)), d2, d3], 2)

    put(first, start)
    for k in range(1, int(count.max())):
        live = count > k
        node = first[live] + k
        a, b = t[node - 1], t[node]
        axis = np.cross(a, b)
        s = np.linalg.norm(axis, axis=1, keepdims=True)
        c = np.clip(np.sum(a * b, 1, keepdims=True), -1.0, 1.0)
        bent = s > 1.0e-12
        axis = np.where(bent, axis / np.where(bent, s, 1.0), 0.0)
        d = frames[node - 1][:, :, 0]
        turned = d * c + np.cross(axis, d) * s + axis * np.sum(axis * d, 1, keepdims=True) * (1.0 - c)
        put(node, np.where(bent, turned, d))
    return frames


def exact(case, seed):
    if case["kind"] != "roots":
        return None
    scene = _scene(case, seed)
    offsets = scene.offsets.astype(np.int64)
    count = np.diff(offsets)
    points = _roots_points(seed, scene)
    hint = np.tile([1.0, 0.0, 0.0], (len(count), 1))
    d3 = _unit(scene.points[offsets[:-1] + 1] - scene.points[offsets[:-1]])
    hint = np.where((np.abs(d3[:, :1]) > 1.0 - 1.0e-9), [[0.0, 1.0, 0.0]], hint)
    rest = _frames(scene.points, offsets[:-1], count, hint)
    now = _frames(points, offsets[:-1], count, rest[offsets[:-1]][:, :, 0])
    r = now @ rest.transpose(0, 2, 1)
    v = 0.5 * np.stack([r[:, 2, 1] - r[:, 1, 2], r[:, 0, 2] - r[:, 2, 0], r[:, 1, 0] - r[:, 0, 1]], 1)
    s = np.linalg.norm(v, axis=1, keepdims=True)
    angle = np.arctan2(s, 0.5 * (np.trace(r, axis1=1, axis2=2)[:, None] - 1.0))
    return [points, v * np.where(s > 1.0e-12, angle / np.where(s > 1.0e-12, s, 1.0), 1.0)]
