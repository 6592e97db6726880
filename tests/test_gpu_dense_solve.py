"""The dense Newton solve at the edges of its panels (32 unknowns) and tiles
(16): columns of m cubes in contact (6 m unknowns, each cube coupled to its
neighbours and the floor), one time step against the oracle's.  Poses agree to
the accuracy of the Newton solves (1e-7, as the whole time step's tests ask)."""
import numpy as np
import pytest

from conftest import contact_poses

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 3, 5, 6, 8, 11, 16, 22])
def test_columns(oracle, m):
    import rigc
    from rigc import scene as S

    spec = S.spec_cubes(5, n=3, vel_sigma=0.2)
    bodies = spec["rigid_body_problem"]["rigid_bodies"]
    floor = bodies.pop()
    # whole columns first, so that neighbours are in contact
    spec["rigid_body_problem"]["rigid_bodies"] = sorted(
        bodies, key=lambda b: (round(b["position"][0], 3), round(b["position"][2], 3), b["position"][1]))[:m] + [floor]
    sc = S.scene_from_json(spec)
    x = contact_poses(sc, seed=m)
    for b, p in zip(sc.bodies, x.reshape(-1, 6)):
        b.pose = p.copy()
    assert np.array_equal(sc.poses(), x)
    sim = oracle.OracleSim(sc, h=0.01, gravity=(0.0, -9.81, 0.0), dhat=1e-3)
    ctx = rigc.Context(sc)
    ctx.sim_init(0.01, (0.0, -9.81, 0.0), 1e-3)
    assert len(ctx.construct_constraint_set(x, 1e-3)["type"]) > 0
    sim.step()
    ctx.sim_step(1)
    P = ctx.sim_state()[0]
    assert np.abs(P.reshape(-1) - sim.pose).max() <= 1e-7
