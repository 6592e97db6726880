"""The pruned rigid CCD on aligned contact, where its single-precision search
(csrc/ccd_filter.cuh) can decide little: unrotated boxes and slabs that land on,
slide along, rest on or touch one another at gaps from 1e-3 to 1e-8.  The earliest
time is the double-precision search's bit for bit, and the boxes searched are
bounded (below 2^16 a candidate, and the double-precision search's)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MOTIONS = {"fall": (0, -0.01, 0), "slide": (0.1, 0, 0), "rest": (0, 0, 0), "drift": (0.1, -1e-3, 0.05)}
DEFAULT_BUDGET = 1 << 22


def _stack(kind, gap, quads=6):
    from rigc import meshes
    from rigc import scene as S

    V, F = meshes.cube() if kind == "cubes" else meshes.tessellated_box((1.0, 0.2, 1.0), (quads, 1, quads))
    h = np.ptp(V[:, 1])
    bodies = [S.raw_body(V, None, F, pose=[0, i * (h + gap), 0, 0, 0, 0]) for i in range(2)]
    S.assign_group_ids(bodies)
    return S.Scene(bodies=bodies, timestep=0.01)


def _searches(ctx, x0, x1):
    """(time, boxes) with the single-precision search in front and without."""
    res = []
    for budget in (DEFAULT_BUDGET, DEFAULT_BUDGET - 1):
        ctx.set_ccd_budget(budget)
        t = ctx.earliest_toi(x0, x1)
        res.append((t, ctx.stats()["ccd_boxes"]))
    ctx.set_ccd_budget(DEFAULT_BUDGET)
    return res


def _check(ctx, x0, x1):
    ee, fv = ctx.detect_collision_candidates_rigid(x0, x1, True, 1.5e-3)
    n = len(ee) + len(fv)
    assert n > 0
    (t, boxes), (t64, boxes64) = _searches(ctx, x0, x1)
    print(n, "candidates:", t, boxes, "boxes,", boxes64, "in double precision alone")
    assert t == t64 == ctx.earliest_toi(x0, x1, prune=False)
    assert boxes <= boxes64 + n * 2**16
    return t


@pytest.mark.parametrize("gap", [1e-3, 1e-5, 1e-6, 1e-7, 1e-8, 0.0])
@pytest.mark.parametrize("motion", MOTIONS)
@pytest.mark.parametrize("kind", ["cubes", "slabs"])
def test_aligned(kind, motion, gap):
    import rigc

    sc = _stack(kind, gap)
    x0 = sc.poses()
    x1 = x0.copy()
    x1[6:9] += MOTIONS[motion]
    ctx = rigc.Context(sc)
    t = _check(ctx, x0, x1)
    assert t < 1 or (gap > 0 and motion in ("slide", "rest"))
    # one edge pair alone: every thread of a block on its boxes, whose stack some
    # overflow (12 000 boxes until the first reach the tolerance, then 2048 left on
    # the stack, each with up to 15 below it before the next look at its state)
    ee, _ = ctx.detect_collision_candidates_rigid(x0, x1, True, 1.5e-3)
    for i in (41, 61, 105):
        ctx.set_candidates(ee[i:i + 1], np.zeros((0, 2), np.int32))
        (t, boxes), (t64, boxes64) = _searches(ctx, x0, x1)
        assert t == t64 and boxes <= boxes64 + 2**16


@pytest.mark.parametrize("motion", ["fall", "rest"])
def test_pieces_overflow(motion):
    """Some 10^5 touching candidates leave more undecided boxes than the pieces'
    buffer holds (2^18): the call is done again in double precision alone."""
    import rigc

    sc = _stack("slabs", 0.0, 36)
    x0 = sc.poses()
    x1 = x0.copy()
    x1[6:9] += MOTIONS[motion]
    ctx = rigc.Context(sc)
    assert _check(ctx, x0, x1) == 0.0
    # and the next call of the context is not affected
    x0[7] += 1e-3
    x1 = x0.copy()
    x1[6:9] += MOTIONS[motion]
    _check(ctx, x0, x1)


def test_batched_aligned():
    import rigc
    from rigc import scene as S

    scenes = [_stack("cubes", g) for g in (1e-3, 1e-7, 0.0, 1e-5)]
    big, sob = S.concat_scenes(scenes)
    ctx = rigc.Context(big, scene_of_body=sob)
    X0 = np.concatenate([s.poses() for s in scenes])
    X1 = X0.copy()
    alone = []
    for k, (s, m) in enumerate(zip(scenes, MOTIONS.values())):
        X1[12 * k + 6:12 * k + 9] += m
        one = rigc.Context(s)
        one.detect_collision_candidates_rigid(X0[12 * k:12 * k + 12], X1[12 * k:12 * k + 12], True, 0.0)
        alone.append(one.earliest_toi(X0[12 * k:12 * k + 12], X1[12 * k:12 * k + 12], prune=False))
    ctx.compute_earliest_toi(X0, X1)
    assert np.array_equal(ctx.scene_tois(), np.array(alone))


def test_pose_not_finite():
    """Poses on the device are not checked: the search with a NaN among them ends
    with the double-precision search's answer."""
    import rigc

    sc = _stack("cubes", 1e-3)
    x0 = sc.poses()
    x1 = x0.copy()
    x1[7] -= 0.01
    ctx = rigc.Context(sc)
    ee, fv = ctx.detect_collision_candidates_rigid(x0, x1, True, 0.0)
    for k in range(3):
        y1 = x1.copy()
        y1[6 + k] = np.nan
        ctx.set_candidates(ee, fv)
        (t, boxes), (t64, boxes64) = _searches(ctx, x0, y1)
        assert t == t64
        assert boxes <= boxes64 + 2 * (len(ee) + len(fv))  # one each, then from the root in double
