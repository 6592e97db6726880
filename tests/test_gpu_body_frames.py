"""Rotation frames and inertial energies by a warp per body and by a thread per
body (more than 2048 bodies): both sides of the limit against the oracle's
derivatives, at angles on both sides of the series' ends, to the bars of the
whole path (gradient 1e-10 and Hessian 1e-9 of their norms)."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 33, 2048, 2049])
def test_energies(oracle, n):
    import rigc
    from rigc import meshes
    from rigc import scene as S

    b0 = S.make_body(*meshes.cube())
    rng = np.random.default_rng(n)
    bodies = []
    for i in range(n):
        # angles from 0 over the series' ends (1e-4, 1e-1) to several turns
        th = rng.normal(size=3)
        th *= (0.0, 1e-9, 5e-5, 2e-4, 0.05, 0.2, 2.0, 9.0)[i % 8] / np.linalg.norm(th)
        pose = np.concatenate([rng.uniform(-5, 5, 3), th])
        bodies.append(dataclasses.replace(b0, pose=pose, velocity=rng.normal(size=6), group_id=-1,
                                          Qdot=S.rotvec_to_matrix(th) @ S.hat(rng.normal(size=3))))
    S.assign_group_ids(bodies)
    sc = S.Scene(bodies=bodies, timestep=0.01, dhat=1e-3, gravity=(0.0, -9.81, 0.0))
    ctx = rigc.Context(sc)
    x = sc.poses() + rng.normal(0, 1e-2, 6 * n)
    e, g, H = ctx.body_energy(x)
    g, H = g.reshape(n, 6), H.reshape(n, 6, 6)
    total = 0.0
    for b in range(n):
        e_o, g_o, H_o = oracle.body_energy(sc.bodies[b], x[6 * b:6 * b + 6], sc.gravity, sc.timestep)
        total += e_o
        assert np.linalg.norm(g[b] - g_o) <= 1e-10 * np.linalg.norm(g_o), b
        assert np.linalg.norm(H[b] - H_o) <= 1e-9 * np.linalg.norm(H_o), b
    assert abs(e - total) <= 1e-10 * abs(total)
