"""The FP64 Newton-3 CTA grid on systems small enough for the oracle (it is the
default above 196608 particles only): ragged sizes, with and without softening,
in one launch and in several, and as a run."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import PKG, rel_err

pytestmark = pytest.mark.gpu

FP64 = 0


@pytest.fixture
def grid(ctx, monkeypatch):
    monkeypatch.setenv("NBR_TEST_N3_GRID", "1")
    ctx.set_force_config(FP64, 3, 8)
    yield ctx
    ctx.set_force_config(FP64)


# 1e-12 of a force, the bound of the other FP64 kernels: summation order
@pytest.mark.parametrize("n", [1, 2, 255, 257, 2049, 4097, 20001])
@pytest.mark.parametrize("eps2", [0.0, 1e-4])
def test_forces(grid, nbr, oracle, monkeypatch, n, eps2):
    s = nbr.plummer(n, 29)
    grid.upload(s)
    a = grid.forces(FP64, eps2=eps2)
    np.testing.assert_array_equal(a, grid.forces(FP64, eps2=eps2))
    if n == 1:
        assert not a.any()
        return
    idx = np.unique(np.concatenate([np.arange(0, n, max(1, n // 500)), [n - 1]]))
    ref = oracle.accel_subset(s["x"], s["y"], s["z"], s["m"], idx, eps2=eps2)
    assert rel_err(a[:, idx], ref).max() <= 1e-12
    net = np.abs((s["m"] * a).sum(axis=1)).max()
    assert net <= 1e-12 * (s["m"] * np.linalg.norm(a, axis=0)).sum()
    # another order of the same sums than the strips
    if n > 2048:
        monkeypatch.delenv("NBR_TEST_N3_GRID")
        assert (grid.forces(FP64, eps2=eps2) != a).any()
        monkeypatch.setenv("NBR_TEST_N3_GRID", "1")
    for launches in ("2", "5"):
        monkeypatch.setenv("NBR_TEST_N3_SLICES", launches)
        assert rel_err(grid.forces(FP64, eps2=eps2)[:, idx], ref).max() <= 1e-12


@pytest.mark.parametrize("n", [4097, 4500])
def test_run(grid, nbr, oracle, n):
    s = nbr.plummer(n, 5)
    grid.upload(s)
    grid.run(FP64, nbr.KDK, 2, 1e-3, 3, eps2=1e-4)
    got, want = grid.download(), oracle.kdk(s, 1e-3, 3, eps2=1e-4)
    for k in ("x", "y", "z", "vx", "vy", "vz"):
        assert np.abs(got[k] - want[k]).max() <= 1e-11, k


@pytest.mark.parametrize("n,eps2", [(300, 0.0), (1025, 1e-6)])
def test_overflowing_distance_gives_zero(grid, nbr, n, eps2):
    s = {k: v[:n] for k, v in nbr.plummer(n, 3).items()}
    far = {k: np.concatenate([s[k], [1e160 if k == "x" else 1.0 / n if k == "m" else 0.0]])
           for k in ("x", "y", "z", "m")}
    near = dict(far, m=np.concatenate([s["m"], [0.0]]), x=np.concatenate([s["x"], [0.5]]))
    grid.upload(far)
    a = grid.forces(FP64, eps2=eps2)
    grid.upload(near)  # the same launch, the last body massless
    b = grid.forces(FP64, eps2=eps2)
    assert (a[:, -1] == 0.0).all()
    assert np.abs(a[:, :-1] - b[:, :-1]).max() <= 1e-15 * np.abs(b).max()


def test_coincident_bodies_are_skipped(grid, nbr):
    s = {k: v.copy() for k, v in nbr.plummer(700, 8).items()}
    for k in ("x", "y", "z"):
        s[k][699] = s[k][0]
    grid.upload(s)
    a = grid.forces(FP64)
    assert np.isfinite(a).all()
    assert np.abs(a[:, 0] - a[:, 699]).max() <= 1e-12 * np.abs(a[:, 0]).max()


def test_bounds_checked_build():
    """Every index of the same calls against its array's length."""
    lib = os.path.join(PKG, "libnbr_checked.so")
    if not os.path.exists(lib):
        subprocess.run(["make", "-C", PKG, "checked"], check=True, capture_output=True)
    code = ("import os, sys; sys.path.insert(0, %r); import nbr\n"
            "c = nbr.Context(0); c.set_force_config(nbr.FP64, 3, 8)\n"
            "for n in (1, 257, 2049, 4097, 20001):\n"
            "    for launches in ('0', '3'):\n"
            "        os.environ['NBR_TEST_N3_SLICES'] = launches\n"
            "        c.upload(nbr.plummer(n, 3))\n"
            "        for eps2 in (0.0, 1e-6): c.forces(nbr.FP64, eps2=eps2)\n"
            "        if n > 4096: c.run(nbr.FP64, nbr.KDK, 2, 1e-4, 2, eps2=1e-6)\n"
            "print('all in bounds')\n") % PKG
    env = dict(os.environ, NBR_LIB_PATH=lib, NBR_TEST_N3_GRID="1")
    p = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, env=env, timeout=300)
    assert p.returncode == 0 and "all in bounds" in p.stdout, p.stdout + p.stderr
