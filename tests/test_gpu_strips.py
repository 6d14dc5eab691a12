"""Newton-3 strips against the oracle at the edges of their units: batches of 32
sources, row blocks of 32 x (receivers per lane), strips of one unit or none,
and the sizes where the default takes them."""
import os

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

FP64, FP32C = 0, 1
SIZES = [1, 2, 31, 32, 33, 127, 129, 191, 193, 255, 257, 319, 321, 511, 513, 1000, 2049, 4096]


def check(a, ref, prec):
    """The bounds of the other force tests: FP64 differs by summation order
    (1e-12); FP32C by its pair arithmetic (median 1e-6, worst 1e-4)."""
    e = rel_err(a, ref)
    if prec == FP64:
        assert e.max() <= 1e-12, e.max()
    else:
        assert np.median(e) <= 1e-6 and e.max() <= 1e-4, (np.median(e), e.max())


@pytest.mark.parametrize("prec", [FP64, FP32C])
@pytest.mark.parametrize("eps2", [0.0, 1e-4])
def test_forced_strips_at_unit_edges(ctx, nbr, oracle, prec, eps2):
    ctx.set_force_config(prec, 3, 8)
    try:
        for n in SIZES:
            s = nbr.plummer(n, 40 + n)
            ctx.upload(s)
            a = ctx.forces(prec, eps2=eps2)
            ref = oracle.accel(s["x"], s["y"], s["z"], s["m"], eps2=eps2, extended=True)
            if n == 1:
                assert not a.any()
            else:
                check(a, ref, prec)
            np.testing.assert_array_equal(a, ctx.forces(prec, eps2=eps2))
    finally:
        ctx.set_force_config(prec)


@pytest.mark.parametrize("prec", [FP64, FP32C])
@pytest.mark.parametrize("n", [4097, 4100, 5119, 5121, 7681, 9984, 20481])
def test_default_strips(ctx, nbr, oracle, prec, n):
    s = nbr.plummer(n, n)
    ctx.upload(s)
    assert ctx.get_force_config(prec, 1e-6)[0] == 3
    idx = np.unique(np.concatenate([np.arange(0, n, 37), [n - 1]]))
    ref = oracle.accel_subset(s["x"], s["y"], s["z"], s["m"], idx, eps2=1e-6)
    check(ctx.forces(prec, eps2=1e-6)[:, idx], ref, prec)
    # the partial sums of several launches, accumulated: the same to rounding
    os.environ["NBR_TEST_N3_SLICES"] = "3"
    try:
        check(ctx.forces(prec, eps2=1e-6)[:, idx], ref, prec)
    finally:
        del os.environ["NBR_TEST_N3_SLICES"]


def ragged_last_batch(nbr, n, case):
    s = {k: v.copy() for k, v in nbr.plummer(n, n).items() if k in "xyzm"}
    if case == "far":  # the coordinate origin, 3e19 away, is no place for a source
        s = {k: 1e10 * v for k, v in s.items()}
        s["x"] += 3e19
        return s, 1e14
    # a body 1e-14 from the coordinate origin, last; the mean of its tile (alone,
    # or with bodies in opposite pairs) as near
    first = n - 1 - (n - 1) % 128
    pairs = np.arange(first, n - 1).reshape(2, -1)
    for k in "xyz":
        s[k][pairs[1]] = -s[k][pairs[0]]
        s[k][n - 1] = 1e-14 if k == "x" else 0.0
    return s, 0.0


# Massless padding of the last batch pulls nothing, wherever the system lies.
@pytest.mark.parametrize("prec", [FP64, FP32C])
@pytest.mark.parametrize("n", [4097, 4129, 8193])
@pytest.mark.parametrize("case", ["far", "near"])
def test_padding_of_the_last_batch(ctx, nbr, oracle, prec, n, case):
    s, eps2 = ragged_last_batch(nbr, n, case)
    ctx.upload(s)
    assert ctx.get_force_config(prec, eps2)[0] == 3
    idx = np.unique(np.concatenate([np.arange(0, n, 61), np.arange(n - 40, n)]))
    ref = oracle.accel_subset(s["x"], s["y"], s["z"], s["m"], idx, eps2=eps2)
    check(ctx.forces(prec, eps2=eps2)[:, idx], ref, prec)


# A coordinate that all particles share is as good as zero, however large
@pytest.mark.parametrize("prec", [FP64, FP32C])
@pytest.mark.parametrize("n", [4097, 4129, 8192])
@pytest.mark.parametrize("far", [1e25, 1e60, 1e154, 1e300])
def test_a_coordinate_all_share(ctx, nbr, prec, n, far):
    s = {k: v.copy() for k, v in nbr.plummer(n, n).items() if k in "xyzm"}
    a = []
    for x in (0.0, far):
        s["x"][:] = x
        ctx.upload(s)
        a.append(ctx.forces(prec, eps2=1e-4))
    assert np.isfinite(a[0]).all()
    np.testing.assert_array_equal(a[0], a[1])


# two CTAs of the reduction per SM in all, and one batch more: 148 SMs, 296 batches
@pytest.mark.parametrize("prec", [FP64, FP32C])
@pytest.mark.parametrize("n", [9471, 9472, 9473, 9505])
def test_reduction_where_its_form_changes(ctx, nbr, oracle, prec, n):
    s = nbr.plummer(n, n)
    ctx.upload(s)
    idx = np.unique(np.concatenate([np.arange(0, n, 97), np.arange(n - 40, n)]))
    ref = oracle.accel_subset(s["x"], s["y"], s["z"], s["m"], idx, eps2=1e-6)
    check(ctx.forces(prec, eps2=1e-6)[:, idx], ref, prec)


@pytest.mark.parametrize("prec,tol", [(FP64, 1e-11), (FP32C, 1e-6)])
@pytest.mark.parametrize("scheme", ["kdk", "euler"])
def test_strip_runs_between_other_kernels(ctx, nbr, oracle, prec, tol, scheme):
    """A run in strips leaves no FP32C records: a large-kernel evaluation after
    it, and a run after that, see the moved particles."""
    n, eps2 = 4500, 1e-4
    s = nbr.plummer(n, 3)
    ctx.upload(s)
    ctx.run(prec, nbr.KDK if scheme == "kdk" else nbr.EULER, 2, 1e-3, 3, eps2=eps2)
    advance = oracle.kdk if scheme == "kdk" else oracle.euler
    want = advance(s, 1e-3, 3, eps2=eps2)
    got = ctx.download()
    for k in ("x", "y", "z", "vx", "vy", "vz"):
        assert np.abs(got[k] - want[k]).max() <= tol, k
    ctx.set_force_config(prec, 4, 4)
    try:
        a = ctx.forces(prec, eps2=eps2)
    finally:
        ctx.set_force_config(prec)
    check(a, oracle.accel(got["x"], got["y"], got["z"], s["m"], eps2=eps2, extended=True), prec)


@pytest.mark.parametrize("eps2", [0.0, 1e-4])
def test_energy_by_pairs_equals_the_potential(ctx, nbr, oracle, eps2):
    """diagnostics() evaluates each pair once, potential() every ordered pair:
    the same sum to rounding, and the oracle's, at the edges of the units."""
    for n in [1, 2, 31, 33, 127, 129, 255, 257, 1000, 4097, 8191, 8193, 12345]:
        s = nbr.plummer(n, n)
        ctx.upload(s)
        d = ctx.diagnostics(eps2=eps2)
        U, phi = ctx.potential(eps2=eps2, per_particle=True)
        assert abs(d["U"] - U) <= 1e-13 * abs(U), n
        assert abs(0.5 * (s["m"] * phi).sum() - U) <= 1e-13 * abs(U), n
        if n <= 4097:
            ref = oracle.energy(s, eps2=eps2)["U"]
            assert abs(d["U"] - ref) <= 1e-13 * abs(ref), n


# r^2 subnormal (its own rounding is the reference's too), tiny, ordinary, and
# overflowing (no contribution): 4 roundings of the inverse distance and the
# two masses' products stay within 1e-15.
@pytest.mark.parametrize("d", [1e-160, 3e-157, 1e-150, 1e-100, 1.0, 1e100, 1e160])
def test_energy_of_an_extreme_pair(ctx, d):
    z = np.zeros(2)
    with np.errstate(over="ignore", under="ignore"):
        r2 = np.float64(d) * np.float64(d)
        want = -0.25 / np.sqrt(r2) if np.isfinite(r2) else 0.0
    ctx.upload({"x": np.array([0.0, d]), "y": z, "z": z, "m": np.array([0.5, 0.5])})
    for U in (ctx.diagnostics()["U"], ctx.potential(), ctx.potential(per_particle=True)[0]):
        assert abs(U - want) <= 1e-15 * abs(want)
    # a coincident pair is skipped without softening
    ctx.upload({"x": z, "y": z, "z": z, "m": np.array([0.5, 0.5])})
    assert ctx.diagnostics()["U"] == 0.0 and ctx.potential(per_particle=True)[0] == 0.0


# Where the FP64 reactions' form changes (16384 particles), and a large FP32C system,
# ragged too
@pytest.mark.parametrize("prec,n", [(FP64, 16383), (FP64, 16384), (FP64, 16385),
                                    (FP32C, 131071), (FP32C, 131072), (FP32C, 131073)])
@pytest.mark.parametrize("eps2", [0.0, 1e-6])
def test_reactions_where_their_form_changes(ctx, nbr, oracle, prec, n, eps2):
    s = nbr.plummer(n, n)
    ctx.upload(s)
    assert ctx.get_force_config(prec, eps2)[0] == 3
    idx = np.unique(np.concatenate([np.linspace(0, n - 1, 300).astype(int), np.arange(n - 3, n)]))
    ref = oracle.accel_subset(s["x"], s["y"], s["z"], s["m"], idx, eps2=eps2)
    check(ctx.forces(prec, eps2=eps2)[:, idx], ref, prec)
