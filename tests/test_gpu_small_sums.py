"""The deterministic sum of up to 4096 numbers by one block and of more by two
launches: both additions' orders are the same tree, restated here."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tree(v):
    while len(v) > 1:
        h = len(v) // 2
        v = v[:h] + v[h:]
    return v[0]


def _sum(v):
    part = np.zeros(1024)
    for b in range((len(v) + 255) // 256):
        w = np.zeros(256)
        w[:len(v[256 * b:256 * b + 256])] = v[256 * b:256 * b + 256]
        part[b] = _tree(w)
    return _tree(part)


@pytest.mark.parametrize("n", [1, 5, 255, 256, 257, 1024, 1025, 4096, 4097])
def test_energy_sum(n):
    """The barrier energy of one constraint taken n times with its own weight."""
    import rigc
    from rigc import scene as S

    sc = S.scene_from_json(S.spec_slab_stacks(3, nx=1, nz=1, n=(6, 1, 6)))
    x = sc.poses()
    ctx = rigc.Context(sc)
    cs = ctx.construct_constraint_set(x, 1e-3)
    m = len(cs["type"])
    pick = np.arange(n) % m
    w = np.random.default_rng(n).uniform(0.5, 2.0, n)
    ctx.set_constraints(*[cs[k][pick] for k in ("type", "verts", "prims", "bodies")], w, cs["eps"][pick])
    e, _, _ = ctx.barrier_local_terms(x, n, 1e-3, project=False)
    assert ctx.compute_barrier_term(x, 1e-3, grad=False, hess=False)[0] == _sum(np.asarray(e))
