"""The piecewise-linear CCD's work-item kernel (pieces and boxes one per
thread, boxes decided in single precision where that is certain) against the
one-candidate-per-warp double-precision kernel, per candidate and bit for
bit: few and many candidates, minimum separations, fast turns, poses far from
the origin, near-touching starts (halvings at t = 0 beyond the work-item
kernel's depth, which hands those candidates on) and no motion."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cubes(n, gap, omega, speed, offset=0.0):
    from rigc import scene as S

    rng = np.random.default_rng(5)
    V, F = S.meshes.cube()
    bodies = []
    for i in range(n):
        b = S.make_body(V, F)
        b.pose = np.concatenate([[offset, offset + 0.5 + gap + i * (1.0 + gap), offset],
                                 [0.0, rng.uniform(-0.2, 0.2), 0.0]])
        b.velocity = np.concatenate([rng.normal(0, speed, 3), rng.normal(0, 1, 3) * omega])
        b.velocity[1] = -speed
        bodies.append(b)
    V, F = S.meshes.plane(20.0)
    bodies.append(S.make_body(V, F, position=(offset, offset, offset), is_dof_fixed=True, body_type="static"))
    S.assign_group_ids(bodies)
    return S.Scene(bodies=bodies, timestep=0.01)


def _same(ctx, x0, x1, dmin=0.0):
    got = {}
    for mode in (0, 1, -1):
        ctx.set_pl_search(mode)
        got[mode] = ctx.earliest_toi_piecewise_linear(x0, x1, dmin, per_candidate=True)
        assert ctx.earliest_toi_piecewise_linear(x0, x1, dmin) == got[mode][0]
    for mode in (1, -1):
        assert np.array_equal(got[mode][1], got[0][1])
        assert got[mode][0] == got[0][0] and got[mode][2] == got[0][2]
    return got[0]


@pytest.mark.parametrize("dmin", [0.0, 1e-4])
@pytest.mark.parametrize("omega,speed,gap,offset", [
    (0.0, 0.5, 1e-3, 0.0), (0.5, 0.5, 1e-3, 0.0), (30.0, 2.0, 5e-3, 0.0), (0.2, 0.5, 1e-3, 1e4),
    (0.0, 1.0, 1e-9, 0.0), (0.0, 0.0, 5e-4, 0.0)])
def test_cubes(omega, speed, gap, offset, dmin):
    import rigc

    sc = _cubes(3, gap, omega, speed, offset)
    x0, x1 = sc.poses(), sc.predictor_poses()
    ctx = rigc.Context(sc)
    ctx.detect_collision_candidates_rigid(x0, x1, True, dmin / 2)
    _same(ctx, x0, x1, dmin)


@pytest.mark.parametrize("n", [2, 7, 30])
def test_sphere_piles(n):
    import rigc
    from rigc import scene as S

    sc = S.scene_from_json(S.spec_icospheres(seed=n, n=n))
    x0 = S.packed_pile_poses(sc, seed=n)
    x1 = sc.predictor_poses(x0)
    ctx = rigc.Context(sc)
    ee, fv = ctx.detect_collision_candidates_rigid(x0, x1, True, 0.0)
    _same(ctx, x0, x1)
    # the first candidates alone: one block's batch and its edges
    for k in (0, 1, 3, 4, 5, 255, 256, 257, 1217):
        if k <= len(ee):
            ctx.set_candidates(ee[:k], fv[:1])
            _same(ctx, x0, x1)
