"""The dense Newton solve's pivots at the end of the double range: the objective is
divided by the scene's average mass, so a scene's pivots can be scaled by a factor.
Free bodies fall the same way whatever the factor, pivots above 2^1022 (their
reciprocal is subnormal) included.  The step is a few quadratic solves to double
precision; 1e-9 is asked."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _step(average_mass):
    import rigc
    from rigc import meshes
    from rigc import scene as S

    V, F = meshes.cube()
    bodies = []
    for i in range(2):
        b = S.raw_body(V, None, F, pose=[0.3 * i, 0.2, 0.1 - 0.5 * i, 0.1, 0.2, 0.3 * i])
        b.mass, b.moment_of_inertia = 0.5, np.array([0.5, 0.4, 0.45])
        b.velocity = np.array([0.1, -0.2, 0.3, 0.2, -0.1, 0.4])
        b.Qdot = S.rotvec_to_matrix(b.pose[3:]) @ S.hat(b.velocity[3:])
        b.group_id = 0  # no contact
        bodies.append(b)
    sc = S.Scene(bodies=bodies, timestep=0.01)
    sc.average_mass = average_mass
    ctx = rigc.Context(sc)
    ctx.sim_init(0.01, (0.0, -9.81, 0.0), 1e-3)
    ctx.sim_step(1)
    return ctx.sim_state()[0].reshape(-1)


@pytest.mark.parametrize("average_mass", [1e-308, 1e-290, 1e290])
def test_pivot_range(average_mass):
    ref = _step(1.0)
    assert np.abs(_step(average_mass) - ref).max() <= 1e-9
