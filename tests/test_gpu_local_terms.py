"""The per-constraint terms' projection and sums: every number of lanes per
constraint gives the same bits, the projected 12x12 is the raw one's positive
part by numpy's eigensolver (generic, exactly parallel and nearly singular
contacts), and the assembled blocks and gradient are the sums of the
per-constraint ones, for segments of one item and of many.

Tolerances: a backward stable eigensolver of a 9x9 leaves some 50 eps |A|; 1e-13
|A| is asked.  A sum of k items in slices of k / 16 errs by at most
(k / 16 + 16) eps of the absolute sum, below 1e-12 for k < 10^5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DHAT = 1e-3


def _slabs(kind):
    from rigc import scene as S

    sc = S.scene_from_json(S.spec_slab_stacks(3, nx=1, nz=1, n=(6, 1, 6)))
    x = sc.poses().reshape(-1, 6).copy()
    if kind != "parallel":
        a = {"turned": 0.03, "nearly_parallel": 1e-5}[kind]
        for i in range(2):
            x[i, 4] += a * (i + 1)
    return sc, x.reshape(-1)


def _positive_part(H):
    w, V = np.linalg.eigh(0.5 * (H + H.transpose(0, 2, 1)))
    return (V * np.maximum(w, 0)[:, None, :]) @ V.transpose(0, 2, 1)


@pytest.mark.parametrize("kind", ["parallel", "nearly_parallel", "turned"])
def test_projection(kind):
    import rigc

    sc, x = _slabs(kind)
    ctx = rigc.Context(sc)
    n = len(ctx.construct_constraint_set(x, DHAT)["type"])
    assert n > 20
    _, g, H = ctx.barrier_local_terms(x, n, DHAT, project=False)
    norm = np.linalg.norm(H, axis=(1, 2))
    for w in (1, 2, 4, 8, 16, 32):
        ctx.set_tune(barrier_per_warp=w)
        _, gw, Hw = ctx.barrier_local_terms(x, n, DHAT, project=True)
        if w == 1:
            g1, H1 = gw, Hw
            assert (np.linalg.norm(H1 - _positive_part(H), axis=(1, 2)) <= 1e-13 * norm + 1e-300).all()
            assert np.array_equal(g, g1)
        assert np.array_equal(gw, g1) and np.array_equal(Hw, H1), w
    # friction at the same contacts (its own kernel, by its count)
    ctx.friction_setup(x, DHAT, 1e6, 0.5)
    y = x.copy()
    y[0] += 3e-6
    _, _, F = ctx.friction_local_terms(y, n, 1e-5, project=False)
    _, _, Fp = ctx.friction_local_terms(y, n, 1e-5, project=True)
    ok = np.isfinite(F).all((1, 2))
    assert ok.any()
    fn = np.linalg.norm(F[ok], axis=(1, 2))
    assert (np.linalg.norm(Fp[ok] - _positive_part(F[ok]), axis=(1, 2)) <= 1e-13 * fn + 1e-300).all()


@pytest.mark.parametrize("repeat", [1, 5, 16, 17, 64, 65, 700])
def test_sums(repeat):
    """One constraint repeated: a block segment of `repeat` (off-diagonal) and
    as many (diagonal) items, gradient segments of `repeat`."""
    import rigc

    sc, x = _slabs("turned")
    ctx = rigc.Context(sc)
    cs = ctx.construct_constraint_set(x, DHAT)
    n = len(cs["type"])
    pick = np.concatenate([np.arange(min(n, 40)), np.full(repeat, n - 1)])
    ctx.set_constraints(*[cs[k][pick] for k in ("type", "verts", "prims", "bodies", "weight", "eps")])
    m = len(pick)
    _, g, H = ctx.barrier_local_terms(x, m, DHAT, project=True)
    e, G, (rp, col, val) = ctx.compute_barrier_term(x, DHAT)
    nb = sc.num_bodies
    grad, gabs = np.zeros((nb, 6)), np.zeros((nb, 6))
    full, fabs = np.zeros((nb, 6, nb, 6)), np.zeros((nb, 6, nb, 6))
    for k in range(m):
        for i in range(2):
            a = cs["bodies"][pick[k], i]
            grad[a] += g[k, 6 * i:6 * i + 6]
            gabs[a] += np.abs(g[k, 6 * i:6 * i + 6])
            for j in range(2):
                b = cs["bodies"][pick[k], j]
                blk = H[k, 6 * i:6 * i + 6, 6 * j:6 * j + 6]
                full[a, :, b] += blk
                fabs[a, :, b] += np.abs(blk)
    assert (np.abs(G.reshape(nb, 6) - grad) <= 1e-12 * gabs).all()
    got = np.zeros_like(full)
    for r in range(nb):
        for s in range(rp[r], rp[r + 1]):
            got[r, :, col[s]] = val[s]
    assert (np.abs(got - full) <= 1e-12 * fabs).all()
