"""The FP64 inverse cube of the pair loops: its accuracy over the range of
distances, and the limits it shares with a reciprocal square root."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FP64 = 0
# the kernels that evaluate it: forced (ni, warps), or the default choice
CONFIGS = [(0, 0), (4, 4), (8, 2), (1, 2), (1, 8), (3, 8)]


# One source at the origin, receivers on an axis: |a| = 1 / d^2.  The result
# carries the rounding of r^2 (times 3/2), of the series, of the seed's cube, of
# their product, and of the products with the mass, the difference and the
# scale: 7.5 x 2^-53 = 8.4e-16.
@pytest.mark.parametrize("eps2", [0.0, 1e-300])
def test_pair_force_over_the_range_of_distances(ctx, eps2):
    rng = np.random.default_rng(5)
    d = np.exp(rng.uniform(np.log(1e-90 if eps2 == 0.0 else 1e-60), np.log(1e90), 3000))
    z = np.zeros_like(d)
    one = np.ones(1)
    a = ctx.accel_ij(d, z, z, 0 * one, 0 * one, 0 * one, one, precision=FP64, eps2=eps2)
    want = -1.0 / d.astype(np.longdouble) ** 2
    assert np.abs((a[0] - want) / want).max() <= 1e-15
    assert (a[1:] == 0.0).all()


# A body so far away that its squared distance overflows pulls nothing and is
# pulled by nothing, as with an exact reciprocal square root.
@pytest.mark.parametrize("ni,warps", CONFIGS)
@pytest.mark.parametrize("n,eps2", [(300, 0.0), (1025, 1e-6)])
def test_overflowing_distance_gives_zero(ctx, nbr, ni, warps, n, eps2):
    s = {k: v[:n] for k, v in nbr.plummer(n, 3).items()}
    far = {k: np.concatenate([s[k], [1e160 if k == "x" else 1.0 / n if k == "m" else 0.0]])
           for k in ("x", "y", "z", "m")}
    near = dict(far, m=np.concatenate([s["m"], [0.0]]),
                x=np.concatenate([s["x"], [0.5]]))
    try:
        ctx.set_force_config(FP64, ni, warps)
        ctx.upload(far)
        a = ctx.forces(FP64, eps2=eps2)
        ctx.upload(near)  # the same launch, the last body massless
        b = ctx.forces(FP64, eps2=eps2)
    finally:
        ctx.set_force_config(FP64)
    assert (a[:, -1] == 0.0).all()
    assert np.abs(a[:, :-1] - b[:, :-1]).max() <= 1e-15 * np.abs(b).max()


# Coincident bodies without softening are skipped; the others feel both.
@pytest.mark.parametrize("ni,warps", CONFIGS)
def test_coincident_bodies_are_skipped(ctx, nbr, ni, warps):
    s = nbr.plummer(700, 8)
    s = {k: v.copy() for k, v in s.items()}
    for k in ("x", "y", "z"):
        s[k][699] = s[k][0]
    try:
        ctx.set_force_config(FP64, ni, warps)
        ctx.upload(s)
        a = ctx.forces(FP64)
    finally:
        ctx.set_force_config(FP64)
    assert np.isfinite(a).all()
    assert np.abs(a[:, 0] - a[:, 699]).max() <= 1e-12 * np.abs(a[:, 0]).max()
