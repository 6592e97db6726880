"""The pruned rigid CCD's single-precision search (csrc/ccd_filter.cuh): its
earliest time of impact is the double-precision search's bit for bit, at the
edges of its range: bodies that turn too fast for its series (time depths
from 7 on in double precision) or not at all, angles beyond its range, far
from the origin, resting and touching contacts, few and many candidates, every
time window and number of seeds, batched scenes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cubes(seed, n, omega, speed, gap, offset=0.0, spin=0.0):
    """Columns of n cubes `gap` apart, cube i turned by spin about y."""
    from rigc import scene as S

    rng = np.random.default_rng(seed)
    V, F = S.meshes.cube()
    bodies = []
    for c in range(2):
        for i in range(n):
            b = S.make_body(V, F)
            th = np.array([0.0, spin + 0.3 * c + rng.uniform(-0.2, 0.2), 0.0])
            b.pose = np.concatenate([[offset + 1.8 * c, 0.5 + gap + i * (1.0 + gap), offset], th])
            b.velocity = np.concatenate([rng.normal(0, speed, 3), rng.normal(0, 1, 3) * omega])
            bodies.append(b)
    V, F = S.meshes.plane(20.0)
    p = S.make_body(V, F, position=(offset, 0, offset), is_dof_fixed=True, body_type="static")
    bodies.append(p)
    S.assign_group_ids(bodies)
    return S.Scene(bodies=bodies, timestep=0.01)


def _check(ctx, x0, x1, windows=(-1,), seeds=(-1,)):
    ctx.detect_collision_candidates_rigid(x0, x1, True, 0.0)
    toi, per, _ = ctx.earliest_toi(x0, x1, prune=False, per_candidate=True)
    assert toi == (per.min() if len(per) else np.inf)
    for w in windows:
        for k in seeds:
            ctx.set_ccd_window(w)
            ctx.set_tune(ccd_seeds_log2=k)
            assert ctx.earliest_toi(x0, x1, prune=True) == toi, (w, k)
    ctx.set_ccd_window(-1)
    ctx.set_tune()
    return toi


@pytest.mark.parametrize("omega", [0.0, 0.5, 20.0, 400.0])
@pytest.mark.parametrize("speed,gap", [(0.2, 5e-4), (3.0, 5e-3), (0.0, 2e-4)])
def test_turning_cubes(omega, speed, gap):
    import rigc

    sc = _cubes(1, 2, omega, speed, gap)
    _check(rigc.Context(sc), sc.poses(), sc.predictor_poses(), (-1, 0, 1, 6, 12), (-1, 0, 5))


@pytest.mark.parametrize("offset", [0.0, 1e3, 1e5])
@pytest.mark.parametrize("spin", [0.0, 3.1, 4.39, 6.0])
def test_far_and_turned_cubes(offset, spin):
    """Positions up to 1e5 m, rotation vectors inside and beyond the series' range."""
    import rigc

    sc = _cubes(2, 1, 1.0, 0.5, 1e-3, offset, spin)
    _check(rigc.Context(sc), sc.poses(), sc.predictor_poses(), (-1, 0, 9), (0, 3))


@pytest.mark.parametrize("n", [2, 9, 40])
def test_sphere_piles(n):
    import rigc
    from rigc import scene as S

    sc = S.scene_from_json(S.spec_icospheres(seed=n, n=n))
    x0 = S.packed_pile_poses(sc, seed=n)
    ctx = rigc.Context(sc)
    _check(ctx, x0, sc.predictor_poses(x0), (-1, 0, 3, 12), (-1, 0, 5))
    # no motion at all, and the same motion a hundred times slower
    _check(ctx, x0, x0.copy())
    _check(ctx, x0, sc.predictor_poses(x0, dt=1e-4))


def test_one_candidate_and_none():
    import rigc

    sc = _cubes(3, 1, 0.5, 0.0, 5e-3)
    sc.bodies[0].velocity[1] = -2.0  # 2 cm down, onto the plane
    x0, x1 = sc.poses(), sc.predictor_poses()
    ctx = rigc.Context(sc)
    ee, fv = ctx.detect_collision_candidates_rigid(x0, x1, True, 0.0)
    assert len(fv)
    none = np.zeros((0, 2), np.int32)
    for e, f in ((none, fv[:1]), (ee[:1], none), (none, none)):
        ctx.set_candidates(e, f)
        toi = ctx.earliest_toi(x0, x1, prune=False)
        assert ctx.earliest_toi(x0, x1, prune=True) == toi


def test_batched_scenes():
    """Per-scene running minima: scenes of different motions in one context."""
    import rigc
    from rigc import scene as S

    scenes = [_cubes(k, 1 + k % 3, o, v, g) for k, (o, v, g) in enumerate(
        [(0.0, 0.2, 5e-4), (400.0, 1.0, 1e-3), (1.0, 3.0, 5e-3), (0.0, 0.0, 2e-4), (20.0, 0.5, 1e-3)])]
    big, sob = S.concat_scenes(scenes)
    cb = rigc.Context(big, scene_of_body=sob)
    X0 = np.concatenate([s.poses() for s in scenes])
    X1 = np.concatenate([s.predictor_poses() for s in scenes])
    alone = [_check(rigc.Context(s), s.poses(), s.predictor_poses()) for s in scenes]
    for w in (-1, 0, 3, 12):
        cb.set_ccd_window(w)
        cb.compute_earliest_toi(X0, X1)
        assert np.array_equal(cb.scene_tois(), np.array(alone)), w


@pytest.mark.parametrize("gap", [0.0, 1e-6, 9e-5, 1.1e-4, 2.1e-4, 3e-4])
def test_starts(gap):
    """Starts around the length tolerance (1e-4): whether f over the first
    tolerance's box contains zero sets the candidate's time tolerance."""
    import rigc

    sc = _cubes(2, 1, 0.0, 0.0, gap)
    for v in (0.0, -1e-3, -0.5):
        sc.bodies[0].velocity[1] = v
        _check(rigc.Context(sc), sc.poses(), sc.predictor_poses())
