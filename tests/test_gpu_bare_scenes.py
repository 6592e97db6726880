"""Scenes without faces or edges (the bodies of the reference's edge-edge CCD tests,
point clouds): every query answers, with the pairs there are, none among them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SQUARE = np.array([[0.0, 0, 0], [1, 0, 0], [1, 0, 1], [0, 0, 1]])
RING = [[0, 1], [1, 2], [2, 3], [0, 3]]


def _scene(n, edges, faces=None):
    from rigc import scene as S

    bodies = [S.raw_body(SQUARE, edges, faces, pose=[0.05 * i, 0.01 * i, 0.03 * i, 0, 0.2 * i, 0]) for i in range(n)]
    S.assign_group_ids(bodies)
    return S.Scene(bodies=bodies, timestep=0.01, dhat=1e-2)


# 80 bodies: 320 vertices and edges, several tiles
@pytest.mark.parametrize("n", [2, 80])
@pytest.mark.parametrize("kind", ["edges", "vertices", "one_meshed"])
def test_bare_scenes(oracle, n, kind):
    import rigc

    sc = _scene(n, RING if kind == "edges" else np.zeros((0, 2), np.int32))
    if kind == "one_meshed":  # one body has all the faces and edges
        from rigc import scene as S

        V, F = S.meshes.plane(3.0)
        sc.bodies[0] = S.raw_body(V, None, F, pose=sc.bodies[0].pose)
        S.assign_group_ids(sc.bodies)
        sc.refresh()
    x0 = sc.poses()
    x1 = x0 + np.random.default_rng(n).normal(0, 0.02, x0.shape)
    ctx, o = rigc.Context(sc), oracle.OracleScene(sc)
    for continuous in (False, True):
        ee, fv = ctx.detect_collision_candidates_rigid(x0, x1 if continuous else x0, continuous, 6e-3)
        ee_o, fv_o = o.detect_candidates(x0, x1 if continuous else x0, continuous, 6e-3)
        assert np.array_equal(ee, ee_o) and np.array_equal(fv, fv_o)
        assert (len(ee) > 0) == (kind == "edges")
        if kind != "one_meshed":
            assert len(fv) == 0
    assert ctx.detect_intersections(x0) == o.detect_intersections(x0)
    cs = ctx.construct_constraint_set(x0, 1e-2)
    assert (len(cs["type"]) > 0) == (kind != "vertices")
    assert ctx.compute_earliest_toi(x0, x1) == o.earliest_toi(x0, x1, *o.detect_candidates(x0, x1))
