"""The rounding of a force, by kernel: a kernel that a default moved to adds no
more of it than the one it replaced.  Medians over 2000 receivers of the error
against extended precision; two such medians of equal kernels differ by 3 %."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

FP64, FP32C = 0, 1


def system(nbr, n, masses):
    s = {k: v.copy() for k, v in nbr.plummer(n, n + 1).items()}
    if masses == "spread":
        s["m"] *= np.random.default_rng(n).uniform(0.5, 1.5, n)
    return s


def over_decades(nbr, n):
    """Masses over many decades, one of a hundred 1000 times as heavy."""
    s, g = nbr.plummer(n, n + 1), np.random.default_rng(n)
    s["m"] = g.lognormal(0.0, 2.0, n) * np.where(g.uniform(size=n) < 0.01, 1000.0, 1.0)
    s["m"] /= s["m"].sum()
    return s


def median_errors(ctx, oracle, s, prec, eps2, configs):
    """One median per (ni, warps); "run": the accelerations of a run's kernel, as
    the velocities after one Euler step of size 1 from rest."""
    n = len(s["x"])
    idx = np.unique(np.linspace(0, n - 1, 2000).astype(int))
    ref = oracle.accel_subset(s["x"], s["y"], s["z"], s["m"], idx, eps2=eps2)
    out = []
    for c in configs:
        ctx.upload({k: s[k] for k in "xyzm"})
        if c == "run":
            ctx.run(prec, 2, 2, 1.0, 1, eps2=eps2)
            d = ctx.download()
            a = np.stack([d["vx"], d["vy"], d["vz"]])
        else:
            try:
                ctx.set_force_config(prec, *c)
                a = ctx.forces(prec, eps2=eps2)
            finally:
                ctx.set_force_config(prec)
        out.append(np.median(rel_err(a[:, idx], ref)))
    return out


# strips against the small-system kernel with 8 lane groups, which served these sizes
@pytest.mark.parametrize("n", [4500, 9000, 14000])
@pytest.mark.parametrize("eps2", [0.0, 1e-4])
def test_fp64_strips(ctx, nbr, oracle, n, eps2):
    strips, small = median_errors(ctx, oracle, system(nbr, n, "equal"), FP64, eps2, [(3, 8), (1, 8)])
    assert strips <= 1.03 * small, (strips, small)


# and with masses over many decades
@pytest.mark.parametrize("n", [12288, 14000])
@pytest.mark.parametrize("eps2", [0.0, 1e-4])
def test_fp64_strips_masses_over_decades(ctx, nbr, oracle, n, eps2):
    strips, small = median_errors(ctx, oracle, over_decades(nbr, n), FP64, eps2, [(3, 8), (1, 8)])
    assert strips <= 1.03 * small, (strips, small)


# the persistent run against the force call of the same size
@pytest.mark.parametrize("n", [1000, 2048, 4096])
def test_fp64_persistent_run(ctx, nbr, oracle, n):
    run, small = median_errors(ctx, oracle, system(nbr, n, "equal"), FP64, 1e-4, ["run", (1, 8)])
    assert run <= 1.03 * small, (run, small)


# FP32C strips against the small-system kernel with 2 lane groups (up to 8192
# particles) and the large kernel, which served these sizes; 10 % is a third of
# what one chain of additions per reaction, or one origin per tile, adds
@pytest.mark.parametrize("n,other", [(6000, (1, 2)), (8192, (1, 2)), (12001, (8, 2))])
@pytest.mark.parametrize("eps2", [1e-6, 1e-4])
def test_fp32c_strips(ctx, nbr, oracle, n, other, eps2):
    strips, before = median_errors(ctx, oracle, system(nbr, n, "spread"), FP32C, eps2, [(3, 8), other])
    assert strips <= 1.1 * before, (strips, before)


# Median errors of the CTA grid, which served these sizes; with one chain of additions
# per reaction the strips had 8.1e-8 and 8.3e-8
@pytest.mark.parametrize("n,before", [(131073, 7.30e-8), (200000, 7.33e-8)])
def test_fp32c_strips_masses_over_decades(ctx, nbr, oracle, n, before):
    strips, = median_errors(ctx, oracle, over_decades(nbr, n), FP32C, 1e-6, [(3, 8)])
    assert strips <= before


# Masses in whole ratios carry no rounding of their own: a system whose masses are
# multiples of 1/7000 moves as one of multiples of 2^-13 (exact in 32 bits), up to
# the roundings of the factor, the sums' product with it and this quotient
@pytest.mark.parametrize("masses", ["equal", "whole"])
def test_fp32c_strips_scale_with_the_mass(ctx, nbr, masses):
    n = 7000
    s = system(nbr, n, "equal")
    ratio = np.ones(n) if masses == "equal" else np.random.default_rng(1).choice([1.0, 3.0, 1000.0], n)
    a = []
    for unit in (1.0 / 7000, 2.0 ** -13):
        ctx.upload({"x": s["x"], "y": s["y"], "z": s["z"], "m": unit * ratio})
        a.append(ctx.forces(FP32C, eps2=1e-6) / unit)
    assert np.abs(a[0] / a[1] - 1.0).max() <= 1e-15


@pytest.mark.parametrize("m0", [0.0, 0.7, 1.99999999, 1e-30, 5e-324])
def test_fp32c_strips_any_mass_of_particle_0(ctx, nbr, oracle, m0):
    s = system(nbr, 4500, "spread")
    s["m"][0] = m0
    ctx.upload(s)
    ref = oracle.accel(s["x"], s["y"], s["z"], s["m"], eps2=1e-4, extended=True)
    e = rel_err(ctx.forces(FP32C, eps2=1e-4), ref)
    assert np.median(e) <= 1e-6 and e.max() <= 1e-4


def potentials(s, eps2, idx):
    """Extended-precision potentials of the particles idx."""
    x = np.stack([s[k] for k in "xyz"]).astype(np.longdouble)
    m = s["m"].astype(np.longdouble)
    out = np.zeros(len(idx), np.longdouble)
    for k, i in enumerate(idx):
        d = x - x[:, i:i + 1]
        r2 = (d * d).sum(0) + np.longdouble(eps2)
        r2[i] = 1
        w = m / np.sqrt(r2)
        w[i] = 0
        out[k] = -w.sum()
    return out


# rms errors of a potential in the kernel with rsqrt(double): no more than these
@pytest.mark.parametrize("n,before", [(2048, 1.78e-16), (6000, 1.62e-16)])
def test_potentials(ctx, nbr, n, before):
    e = []
    for seed in range(4):
        s = nbr.plummer(n, seed)
        ctx.upload(s)
        idx = np.arange(0, n, max(1, n // 500))
        ref = potentials(s, 1e-4, idx)
        got = ctx.potential(eps2=1e-4, per_particle=True)[1][idx]
        e.append(((got - ref) / ref).astype(float))
    assert np.sqrt(np.mean(np.square(e))) <= before


# A potential energy rounds about once: half a unit in the last place at most, a
# quarter on average over systems (of 64: within 0.02), and its parts' sums a little
def test_potential_energy(ctx, nbr):
    n, e = 300, []
    for seed in range(64):
        s = nbr.plummer(n, seed)
        ctx.upload(s)
        U = (s["m"] * potentials(s, 1e-4, np.arange(n))).sum() / 2
        e.append(float(abs(ctx.diagnostics(eps2=1e-4)["U"] - U)) / np.spacing(abs(float(U))))
    assert np.mean(e) <= 1 / 3
