"""The broad phase's three ways of pairing elements (all pairs of tiles, patches
of neighbouring elements, the grid) against the oracle's candidates and
intersections, on scenes at the edges of tiles (128), patches (32) and of the
patches' lists; the constraint sets and barrier sums on both sides of the
limits up to which pairs, records and blocks are ordered by counting (4096).

Candidates and constraints are whole numbers: they have to be the same.  The
gradient's sums of k items are in slices of k / 16, below 1e-12 of the absolute
sum for k < 10^5."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DHAT = 1e-2


def _scene(meshes_, positions, groups=None):
    from rigc import scene as S

    bodies = []
    for (V, F), p in zip(meshes_, positions):
        b = S.make_body(V, F)
        bodies.append(dataclasses.replace(b, pose=np.concatenate([p, b.pose[3:]]), group_id=-1))
    S.assign_group_ids(bodies)
    for b, g in zip(bodies, groups if groups is not None else ()):
        b.group_id = g
    return S.Scene(bodies=bodies, timestep=0.01, dhat=DHAT, gravity=(0.0, -9.81, 0.0))


def _hull(rng, n, r=0.5):
    from rigc import meshes

    P = rng.normal(size=(n, 3))
    return meshes.convex_hull(r * P / np.linalg.norm(P, axis=1, keepdims=True))


def _make(kind):
    """(scene, scene of each body or None, whether the grid is to be taken)"""
    from rigc import meshes

    rng = np.random.default_rng(7)
    if kind == "tiles":  # boxes of 126 to 129 edges and more, few tiles
        M = [meshes.tessellated_box((1, 1, 1), n) for n in ((2, 2, 2), (3, 2, 2), (4, 2, 2), (5, 2, 3), (5, 3, 3))]
        return _scene(M, [(0.9 * i, 0.03 * i, 0.4 * (i % 2)) for i in range(5)]), None, False
    if kind == "patches":  # 4 .. 67 vertices: every remainder of a patch
        M = [_hull(rng, n) for n in range(4, 68)] + [meshes.plane(20.0)]
        P = np.concatenate([rng.uniform(-1.3, 1.3, (64, 3)), [[0, -0.8, 0]]])
        return _scene(M, P, list(np.arange(65) // 2)), None, False
    if kind == "scenes":  # the same places in three scenes
        M = [_hull(rng, n) for n in range(20, 80)]
        return _scene(M, np.tile(rng.uniform(-0.7, 0.7, (20, 3)), (3, 1))), np.arange(60) // 20, False
    if kind == "one_large":  # one body's patches against many small ones'
        M = [meshes.icosphere(4, 2.0)] + [_hull(rng, 9, 0.2) for _ in range(50)]
        P = rng.normal(size=(50, 3))
        P = 2.1 * P / np.linalg.norm(P, axis=1, keepdims=True)
        return _scene(M, np.concatenate([[[0, 0, 0]], P])), None, False
    if kind == "floor":  # a face with more pairs than are placed by counting, one with fewer
        M = [meshes.plane(20.0), meshes.tessellated_box((2, 0.2, 2), (70, 1, 70)),
             meshes.tessellated_box((2, 0.2, 2), (20, 1, 20))]
        return _scene(M, [(0, 0, 0), (3, 0.1004, -3), (-3, 0.1004, 3)]), None, False
    if kind == "rim":  # bodies that turn at the scene's rim, more time nodes than the list takes
        P = np.stack([0.7 * (np.arange(1600) // 40), np.zeros(1600), 0.7 * (np.arange(1600) % 40)], 1)
        return _scene([_hull(rng, 16 + i % 9) for i in range(1600)], P), None, False
    # boxes in one another: their patches all overlap, their elements do not
    M = [meshes.cube(1.0 + 0.01 * i) for i in range(400)] + [_hull(rng, 40) for _ in range(6)]
    P = np.concatenate([np.zeros((400, 3)), rng.uniform(-0.5, 0.5, (6, 3)) + [9, 0, 0]])
    return _scene(M, P), None, True


@pytest.mark.parametrize("continuous", [False, True])
@pytest.mark.parametrize("kind", ["tiles", "patches", "scenes", "one_large", "nested", "rim", "floor"])
def test_candidates(oracle, kind, continuous):
    import rigc

    sc, sob, grid = _make(kind)
    rng = np.random.default_rng(3)
    x0 = sc.poses()
    x1 = x0 + rng.normal(0, 0.02, x0.shape) if continuous else x0
    if continuous and kind == "rim":
        x1.reshape(-1, 6)[:, 3:] = x0.reshape(-1, 6)[:, 3:] + rng.normal(0, 2.0, (sc.num_bodies, 3))
    infl = 0.0 if continuous else 1e-3
    ctx = rigc.Context(sc, scene_of_body=sob)
    ee, fv = ctx.detect_collision_candidates_rigid(x0, x1, continuous, infl)
    assert (ctx.stats()["grid_items"] > 0) == grid
    o = oracle.OracleScene(sc)
    ee_o, fv_o = o.detect_candidates(x0, x1, continuous, infl)
    if sob is not None:
        # the scenes' own pairs: box inclusion looks at the scene's bodies alone,
        # discrete boxes do not depend on it
        es, fs, vs = (np.repeat(sob, np.diff(s)) for s in (sc.body_edge_start, sc.body_face_start, sc.body_vertex_start))
        ee_o = ee_o[es[ee_o[:, 0]] == es[ee_o[:, 1]]]
        fv_o = fv_o[fs[fv_o[:, 0]] == vs[fv_o[:, 1]]]
    assert len(ee_o) > 0
    assert np.array_equal(ee, ee_o) and np.array_equal(fv, fv_o)


@pytest.mark.parametrize("kind", ["tiles", "patches", "one_large", "nested"])
def test_intersections(oracle, kind):
    import rigc

    sc, _, _ = _make(kind)
    x = sc.poses()
    n = oracle.OracleScene(sc).detect_intersections(x)
    assert n > 0
    assert rigc.Context(sc).detect_intersections(x) == n


@pytest.mark.parametrize("n", [2, 6, 10, 14, 18, 22])
def test_constraint_sets(oracle, n):
    """Two slabs of n x n quads a little apart: some 300 to 30 000 candidates."""
    import rigc
    from rigc import meshes

    box = meshes.tessellated_box((1.0, 0.2, 1.0), (n, 2, n))
    sc = _scene([box, box], [(0, 0, 0), (0.01, 0.202, 0.013)])
    x = sc.poses()
    o = oracle.OracleScene(sc)
    ee, fv = o.detect_candidates(x, continuous=False, inflation=DHAT / 2)
    cs = o.constraint_set(x, ee, fv, DHAT).key_sorted()
    ctx = rigc.Context(sc)
    g = ctx.construct_constraint_set(x, DHAT)
    m = len(g["type"])
    assert m == len(cs) > 0
    order = np.lexsort((g["prims"][:, 1], g["prims"][:, 0], g["type"]))
    for k, ref in (("type", cs.types), ("prims", cs.prims), ("weight", cs.weight), ("eps", cs.eps)):
        vv = cs.types == 0
        got = g[k][order]
        if k == "prims":  # a vertex pair's primitives are the first pair of edges or face met
            got, ref = got[~vv], ref[~vv]
        assert np.array_equal(got, ref), k
    _, gl, _ = ctx.barrier_local_terms(x, m, DHAT, project=True)
    _, G, _ = ctx.compute_barrier_term(x, DHAT)
    ref, mag = np.zeros((2, 6)), np.zeros((2, 6))
    for i in range(2):
        np.add.at(ref, g["bodies"][:, i], gl[:, 6 * i:6 * i + 6])
        np.add.at(mag, g["bodies"][:, i], np.abs(gl[:, 6 * i:6 * i + 6]))
    assert (np.abs(G.reshape(2, 6) - ref) <= 1e-12 * mag).all()


@pytest.mark.parametrize("turn", [0.0, 0.3, 3.0, 9.0])
def test_frames_by_four_lanes(turn):
    """152 bodies (frames by four lanes) and one more far away, in no pair
    (frames by a thread): the same candidates and times of impact, for small
    turns, turns beyond the sinc's decrease (4.49) and none."""
    import rigc

    rng = np.random.default_rng(11)
    M = [_hull(rng, 8 + i % 9) for i in range(153)]
    P = np.concatenate([rng.uniform(-3.0, 3.0, (152, 3)), [[1e3, 0, 0]]])
    dx = np.concatenate([rng.normal(0, 0.3, (153, 3)), rng.normal(0, turn, (153, 3))], 1)
    res = []
    for n in (152, 153):
        sc = _scene(M[:n], P[:n])
        x0 = sc.poses()
        x1 = (x0.reshape(-1, 6) + dx[:n]).reshape(-1)
        ctx = rigc.Context(sc)
        ee, fv = ctx.detect_collision_candidates_rigid(x0, x1, True, 0.0)
        assert len(ee) > 0
        ctx.set_candidates(ee[::97], fv[::97])
        res.append((ee, fv, ctx.earliest_toi(x0, x1), ctx.compute_earliest_toi(x0, x1)))
    for a, b in zip(*res):
        assert np.array_equal(a, b)
