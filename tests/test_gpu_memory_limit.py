"""With no device memory left, the CCD searches do without the buffers of their
faster paths: the same answers, no error."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fill(torch):
    """All of the device's memory down to blocks of 2 MiB."""
    held, size = [], 1 << 38
    while size >= 2 << 20:
        try:
            held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.cuda.OutOfMemoryError:
            size //= 2
    return held


def test_searches_without_memory():
    import rigc
    import torch
    from rigc import scene as S

    sc = S.scene_from_json(S.spec_icospheres(seed=1, n=40))
    x0 = S.packed_pile_poses(sc, seed=1)
    x1 = sc.predictor_poses(x0)
    ref = rigc.Context(sc)
    toi = ref.compute_earliest_toi(x0, x1)
    toi_pl = ref.compute_earliest_toi_piecewise_linear(x0, x1)
    ref.close()
    ctx = rigc.Context(sc)
    d0, d1 = ctx.device(x0), ctx.device(x1)
    # the buffers of the searches alone
    ctx.set_ccd_budget((1 << 22) - 1)
    ctx.set_pl_search(0)
    assert ctx.compute_earliest_toi(d0, d1) == toi
    assert ctx.compute_earliest_toi_piecewise_linear(d0, d1) == toi_pl
    ctx.set_ccd_budget(1 << 22)
    ctx.set_pl_search(-1)
    held = _fill(torch)
    try:
        got = ctx.compute_earliest_toi(d0, d1), ctx.compute_earliest_toi_piecewise_linear(d0, d1)
    finally:
        del held
        torch.cuda.empty_cache()
    assert got == (toi, toi_pl)
    # and with memory again
    assert ctx.compute_earliest_toi(d0, d1) == toi
    assert ctx.compute_earliest_toi_piecewise_linear(d0, d1) == toi_pl
    assert np.isfinite(toi)
