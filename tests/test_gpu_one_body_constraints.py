"""Constraints a caller sets between vertices of one and the same body: the
gradient is the sum of the constraints' terms, whether the Hessian is asked for
(sums from its diagonal segments) or not.  Sums of k items in slices round within
1e-12 of the absolute sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 3 and 200 constraints: blocks ordered by counting; 2000: by the radix sort
@pytest.mark.parametrize("n", [3, 200, 2000])
def test_gradient(n):
    import rigc
    from rigc import meshes
    from rigc import scene as S

    V, F = meshes.cube()
    bodies = [S.raw_body(V, None, F, pose=[1.2 * i, 0.1 * i, 0, 0.1, 0.2, 0.3]) for i in range(3)]
    S.assign_group_ids(bodies)
    sc = S.Scene(bodies=bodies, timestep=0.01)
    x = sc.poses()
    rng = np.random.default_rng(n)
    b = rng.integers(0, 3, (n, 2))
    b[::2, 1] = b[::2, 0]  # every other one within a body
    v = 8 * b + rng.integers(0, 4, (n, 2)) + [0, 4]  # two of a cube's vertices, different ones
    verts = np.full((n, 4), -1)
    verts[:, :2] = v
    ctx = rigc.Context(sc)
    ctx.set_constraints(np.zeros(n), verts, v, b, rng.uniform(1, 3, n), np.zeros(n))
    dhat = 5.0  # all are active
    _, gl, _ = ctx.barrier_local_terms(x, n, dhat, project=True)
    ref, mag = np.zeros((3, 6)), np.zeros((3, 6))
    for i in range(2):
        np.add.at(ref, b[:, i], gl[:, 6 * i:6 * i + 6])
        np.add.at(mag, b[:, i], np.abs(gl[:, 6 * i:6 * i + 6]))
    assert (mag > 0).any()
    for hess in (False, True):
        _, G, _ = ctx.compute_barrier_term(x, dhat, hess=hess)
        assert (np.abs(G.reshape(3, 6) - ref) <= 1e-12 * mag).all(), hess
