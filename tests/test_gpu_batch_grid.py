"""The CTAs per SM of a batched launch change its time, not its results."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


# few and many systems, the sizes around a tile and a row block
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("sizes", [[2049], [300] * 3 + [129, 128, 1], [257] * 700])
def test_grid_does_not_change_the_forces(ctx, nbr, oracle, prec, sizes):
    off = np.concatenate([[0], np.cumsum(sizes)])
    sub = [nbr.plummer(n, 50 + i) for i, n in enumerate(sizes)]
    st = {k: np.concatenate([s[k] for s in sub]) for k in nbr.KEYS}
    ctx.batch_upload(off, st)
    a = ctx.batch_forces(prec, eps2=1e-4)
    for per in (1, 2, 3, 4):
        ctx.batch_set_config(prec, 2, per)
        np.testing.assert_array_equal(ctx.batch_forces(prec, eps2=1e-4), a)
    ctx.batch_set_config(prec, 2, 0)
    np.testing.assert_array_equal(ctx.batch_forces(prec, eps2=1e-4), a)
    ref = oracle.accel(*[sub[0][k] for k in ("x", "y", "z", "m")], eps2=1e-4, extended=True)
    e = rel_err(a[:, :sizes[0]], ref)
    assert e.max() <= 1e-12 if prec == 0 else np.median(e) <= 1e-6 and e.max() <= 1e-4
