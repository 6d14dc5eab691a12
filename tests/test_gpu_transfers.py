"""Packed transfers of small arrays, at the size where a call changes to one
copy per array, and the graphs that nbr_run keeps."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

FP64, FP32C = 0, 1


# 6 x n and 3 x n doubles against 1 MiB
@pytest.mark.parametrize("n", [1, 2, 1023, 21845, 21846, 43690, 43691])
def test_download_and_forces_at_the_limit(ctx, nbr, oracle, n):
    s = nbr.plummer(n, 5)
    ctx.upload(s)
    got = ctx.download()
    for k in ("x", "y", "z", "vx", "vy", "vz"):
        np.testing.assert_array_equal(got[k], s[k])
    if n == 1:
        return
    a = ctx.forces(FP64, eps2=1e-4)
    idx = np.unique([0, n // 2, n - 1])
    ref = oracle.accel_subset(s["x"], s["y"], s["z"], s["m"], idx, eps2=1e-4)
    assert rel_err(a[:, idx], ref).max() <= 1e-12
    ctx.forces_device(FP64, eps2=1e-4)
    np.testing.assert_array_equal(ctx.forces_download(), a)


# 4 n_i + 4 n_j doubles against 1 MiB, with and without receiver masses
@pytest.mark.parametrize("n_i,n_j", [(1, 1), (1000, 1), (1, 1000), (16384, 16384), (16385, 16384)])
@pytest.mark.parametrize("prec", [FP64, FP32C])
def test_accel_ij_at_the_limit(ctx, nbr, oracle, n_i, n_j, prec):
    s, q = nbr.plummer(n_i, 6), nbr.plummer(n_j, 7)
    x, y, z = s["x"] + 0.25, s["y"], s["z"]
    args = (x, y, z, q["x"], q["y"], q["z"], q["m"])
    a = ctx.accel_ij(*args, precision=prec, eps2=1e-4)
    f = ctx.accel_ij(*args, mi=s["m"], precision=prec, eps2=1e-4, want_force=True)
    np.testing.assert_allclose(f, s["m"] * a, rtol=1e-14)
    idx = np.unique([0, n_i // 2, n_i - 1])
    d = [q[k][None, :] - v[idx][:, None] for k, v in (("x", x), ("y", y), ("z", z))]
    w = q["m"] / (d[0] ** 2 + d[1] ** 2 + d[2] ** 2 + 1e-4) ** 1.5
    ref = np.stack([(w * e).sum(axis=1) for e in d])
    assert rel_err(a[:, idx], ref).max() <= (1e-12 if prec == FP64 else 1e-4)


@pytest.mark.parametrize("n", [100, 20000])
@pytest.mark.parametrize("which", range(8))
def test_accel_ij_rejects_what_is_not_finite(ctx, nbr, n, which):
    s = nbr.plummer(n, 6)
    arrays = [s[k].copy() for k in ("x", "y", "z", "x", "y", "z", "m", "m")]
    arrays[which][n - 1] = np.inf if which % 2 else np.nan
    with pytest.raises(nbr.NbrError) as e:
        ctx.accel_ij(*arrays[:7], mi=arrays[7], eps2=1e-4, want_force=True)
    assert e.value.status == 7
    a = ctx.accel_ij(*[s[k] for k in ("x", "y", "z", "x", "y", "z", "m")], eps2=1e-4)
    assert np.isfinite(a).all()


# Runs of an odd number of position updates alternate between two graphs, and
# more kinds of calls than graphs are kept displace each other.
@pytest.mark.parametrize("prec,tol", [(FP64, 1e-11), (FP32C, 1e-6)])
def test_alternating_runs(ctx, nbr, oracle, prec, tol):
    n, eps2 = 4200, 1e-4
    s = nbr.plummer(n, 9)
    ctx.upload(s)
    steps = [3, 3, 3, 1, 2, 3, 1, 4, 5, 3]
    for k in steps:
        ctx.run(prec, nbr.KDK, 2, 1e-4, k, eps2=eps2)
    want = oracle.kdk(s, 1e-4, sum(steps), eps2=eps2)
    got = ctx.download()
    for k in ("x", "y", "z", "vx", "vy", "vz"):
        assert np.abs(got[k] - want[k]).max() <= tol, k


def test_batch_download_is_the_upload(ctx, nbr):
    sizes = [1, 127, 128, 129, 300, 5, 256]
    off = np.concatenate([[0], np.cumsum(sizes)])
    rng = np.random.default_rng(1)
    st = {k: np.abs(rng.standard_normal(off[-1])) for k in nbr.KEYS}
    ctx.batch_upload(off, st)
    got = ctx.batch_download()
    for k in ("x", "y", "z", "vx", "vy", "vz"):
        np.testing.assert_array_equal(got[k], st[k])


def test_batch_download_keeps_one_array(nbr):
    """What a download allocates and keeps is one array without padding, whichever
    arrays are asked for."""
    torch = pytest.importorskip("torch")
    sizes = np.full(64, 32700)
    off = np.concatenate([[0], np.cumsum(sizes)])
    n = int(off[-1])
    rng = np.random.default_rng(2)
    st = {k: np.abs(rng.standard_normal(n)) for k in nbr.KEYS}
    with nbr.Context(0) as c:
        c.batch_upload(off, st)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        z, vx = np.zeros(n), np.zeros(n)
        assert c.L.nbr_batch_download(c.h, None, None, nbr._p(z), nbr._p(vx), None, None) == 0
        np.testing.assert_array_equal(z, st["z"])
        np.testing.assert_array_equal(vx, st["vx"])
        got = c.batch_download()
        for k in ("x", "y", "z", "vx", "vy", "vz"):
            np.testing.assert_array_equal(got[k], st[k])
        assert free - torch.cuda.mem_get_info()[0] <= 8 * n + (4 << 20)  # allocation granularity


# Where there is no room for what a transfer or a launch would take at its
# fastest, the call does without it: the same results.
def failing_allocation(monkeypatch, call, k="1"):
    monkeypatch.setenv("NBR_TEST_FAIL_ALLOC", k)
    try:
        return call()
    finally:
        monkeypatch.delenv("NBR_TEST_FAIL_ALLOC")


def test_transfers_without_staging(nbr, monkeypatch):
    s = nbr.plummer(1500, 5)
    with nbr.Context(0) as c:
        c.upload(s)
        got = failing_allocation(monkeypatch, c.download)
        for k in ("x", "y", "z", "vx", "vy", "vz"):
            np.testing.assert_array_equal(got[k], s[k])
    args = [s[k] for k in ("x", "y", "z", "x", "y", "z", "m")]
    with nbr.Context(0) as c:
        a = failing_allocation(monkeypatch, lambda: c.accel_ij(*args, eps2=1e-4))
        np.testing.assert_array_equal(a, c.accel_ij(*args, eps2=1e-4))
    off = np.array([0, 300, 1500])
    with nbr.Context(0) as c:
        c.batch_upload(off, s)
        got = failing_allocation(monkeypatch, c.batch_download)
        for k in ("x", "y", "z", "vx", "vy", "vz"):
            np.testing.assert_array_equal(got[k], s[k])
        np.testing.assert_array_equal(c.batch_download()["x"], s["x"])


def test_strips_in_less_scratch(nbr, monkeypatch):
    """450000 particles take 2.4 GB of reactions in one launch."""
    with nbr.Context(0) as c:
        c.upload(nbr.plummer(450000, 5))
        few = failing_allocation(monkeypatch, lambda: c.forces(FP32C, eps2=1e-4))
        again = c.forces(FP32C, eps2=1e-4)
        np.testing.assert_array_equal(few, again)
        c.upload(nbr.plummer(450000, 5))
        e = rel_err(few, c.forces(FP32C, eps2=1e-4))
        assert np.median(e) <= 1e-6 and e.max() <= 1e-4


def test_download_leaves_a_pending_error(nbr, monkeypatch):
    """A download after an evaluation that timed out returns the state; the
    status is the next evaluation's, as for arrays too large to be packed."""
    s = nbr.plummer(5000, 5)
    with nbr.Context(0) as c:
        c.upload(s)
        c.set_force_config(FP64, 4, 4)
        monkeypatch.setenv("NBR_WAIT_LIMIT_MS", "50")
        monkeypatch.setenv("NBR_TEST_SKIP_TILE", "1")
        c.forces_device(FP64, eps2=1e-4)
        monkeypatch.delenv("NBR_TEST_SKIP_TILE")
        np.testing.assert_array_equal(c.download()["x"], s["x"])
        with pytest.raises(nbr.NbrError):
            c.synchronize()
        assert np.isfinite(c.forces(FP64, eps2=1e-4)).all()


def test_graphs_give_way(nbr, oracle, monkeypatch):
    """What a context keeps for speed is given back where an allocation fails."""
    small, large = nbr.plummer(4500, 5), nbr.plummer(9000, 6)
    for keep in ("graph", "batch copy"):
        with nbr.Context(0) as c:
            if keep == "graph":
                c.upload(small)
                c.run(FP64, nbr.KDK, 2, 1e-4, 2, eps2=1e-4)
            else:
                c.batch_upload(np.array([0, 4000, 4500]), small)
                c.batch_download()
            failing_allocation(monkeypatch, lambda: c.upload(large))
            ref = oracle.accel(large["x"], large["y"], large["z"], large["m"], eps2=1e-4, extended=True)
            assert rel_err(c.forces(FP64, eps2=1e-4), ref).max() <= 1e-12
            if keep == "batch copy":
                np.testing.assert_array_equal(c.batch_download()["x"], small["x"])


def test_long_graphs_are_not_all_kept(nbr):
    """Two graphs stay, of whatever length; more only while they are short."""
    torch = pytest.importorskip("torch")
    free = []
    with nbr.Context(0) as c:
        c.upload(nbr.plummer(4500, 5))
        for steps in (6000, 6001, 6002, 6003):  # about 12000 launches, 30 MB each
            c.run(FP64, nbr.EULER, 2, 1e-9, steps, eps2=1e-2)
            torch.cuda.synchronize()
            free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[1] > 16 << 20
    assert free[1] - free[3] <= 16 << 20
