"""The work that users of this solver have it do, as measurable cases.

Four kinds of calls, each through the Python binding of the C ABI (nbr.Context):

* run      advance one uploaded system by a few steps (nbr_run) and read the
           state: the solver's main loop.  Small systems come back to the host
           (nbr_system_download), as a program that logs a trajectory does;
           larger ones stay on the GPU (nbr_state_pointers), where the next
           consumer of the state works;
* forces   one force evaluation of an uploaded system into host arrays
           (nbr_forces);
* ij       receivers and sources from host arrays, forces back to the host
           (nbr_accel_ij): the drop-in for the reference's force call;
* batch    many independent systems of uneven size advanced together
           (nbr_batch_run) and copied back (nbr_batch_download).

FP64 results are kept as the 64-bit values the call returns; FP32C pair forces
are good to about 1e-7, so a program of that precision keeps what it reads in
32 bits.

Systems are Plummer spheres in N-body units (G = M = 1, scale radius 3 pi / 16)
or cold uniform balls, sampled here from the seed.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "n-body-ring-solver_b200"))
import nbr  # noqa: E402

PRECISION = {"fp64": nbr.FP64, "fp32c": nbr.FP32C}
SCHEME = {"kdk": nbr.KDK, "dkd": nbr.DKD, "euler": nbr.EULER}
STATE = ("x", "y", "z", "vx", "vy", "vz")
#: Largest system whose state a program copies to the host after every call.
HOST_N = 4096
#: Pairs that exact() evaluates within about 10 seconds.
EXACT_PAIRS = 2e11


def listed():
    run = {"kind": "run", "ic": "plummer", "scheme": "kdk", "order": 2, "dt": 1e-3, "eps": 1e-3,
           "diag": False}
    return [
        # the smallest call: a few bodies, one step at a time (interactive use,
        # or a caller that couples other physics between steps)
        dict(run, name="fp64 n64 one step", precision="fp64", n=64, steps=1),
        # the reference's small-system workload: N = 2048, 100 steps
        dict(run, name="fp64 n2048 kdk", precision="fp64", n=2048, steps=100),
        # the same in the compensated precision, at a ragged size
        dict(run, name="fp32c n1999 kdk", precision="fp32c", n=1999, steps=50),
        # a few thousand unsoftened bodies with the fourth-order Yoshida scheme
        # (the reference's -i lf -order 4; it has no softening)
        dict(run, name="fp64 n6000 yoshida4", precision="fp64", n=6000, scheme="dkd", order=4,
             dt=1e-4, eps=0.0, steps=3),
        # a mid-size compensated run, ragged
        dict(run, name="fp32c n12001 kdk", precision="fp32c", n=12001, steps=10),
        # the reference's force call through host arrays, unsoftened, FP64
        {"name": "fp64 force call n8000", "kind": "ij", "precision": "fp64", "n": 8000,
         "n_src": 8000, "eps": 0.0},
        # the cold-collapse workload: uniform ball, N = 32768
        dict(run, name="fp32c n32768 collapse", precision="fp32c", n=32768, ic="ball", eps=1e-2,
             dt=1e-4, steps=10),
        # a production FP64 run with its energy check before and after
        dict(run, name="fp64 n65500 energies", precision="fp64", n=65500, dt=5e-4, steps=3,
             diag=True),
        # the headline workload: N = 262144, compensated
        dict(run, name="fp32c n262144 kdk", precision="fp32c", n=262144, dt=5e-4, steps=1),
        # the largest single system
        dict(run, name="fp32c n1048576 kdk", precision="fp32c", n=1048576, dt=5e-4, steps=1),
        # ensembles of independent small systems, both precisions
        {"name": "fp64 batch 1000", "kind": "batch", "precision": "fp64", "systems": 1000,
         "n_min": 64, "n_max": 4096, "steps": 40, "dt": 1e-3, "eps": 1e-3},
        {"name": "fp32c batch 1000", "kind": "batch", "precision": "fp32c", "systems": 1000,
         "n_min": 64, "n_max": 4096, "steps": 80, "dt": 1e-3, "eps": 1e-3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    precision = rng.choice(["fp64", "fp32c"])
    # pairs of one pass: up to a tenth of a second or so of the slower precision
    most = 1e11 if precision == "fp64" else 2e11
    # the softened form is what FP32C is for; FP64 also stands in for the
    # reference's unsoftened solver
    eps = rng.choice([0.0, 1e-3, 1e-2] if precision == "fp64" else [1e-3, 1e-2])
    kind = rng.choice(["run", "run", "run", "run", "forces", "ij", "batch"])
    if kind == "batch":
        lo = _log_int(rng, 16, 512)
        return {"kind": "batch", "precision": precision, "systems": _log_int(rng, 16, 1000),
                "n_min": lo, "n_max": min(4096, lo * rng.randint(2, 64)),
                "steps": rng.randint(5, 40), "dt": 1e-3, "eps": max(eps, 1e-3)}
    if kind == "ij":
        return {"kind": "ij", "precision": "fp64", "n": _log_int(rng, 64, 65536),
                "n_src": _log_int(rng, 64, 65536), "eps": eps}
    if kind == "forces":
        return {"kind": "forces", "precision": "fp64", "n": _log_int(rng, 64, 131072), "eps": eps}
    scheme = rng.choice(["kdk", "kdk", "dkd", "euler"])
    order = rng.choice([2, 4, 6, 8]) if scheme == "dkd" else 2
    n = _log_int(rng, 16, 262144)
    case = {"kind": "run", "precision": precision, "n": n, "scheme": scheme, "order": order,
            "ic": rng.choice(["plummer", "ball"]), "dt": rng.choice([1e-4, 2e-4, 5e-4]),
            "eps": eps, "diag": rng.random() < 0.25}
    evals = {2: 1, 4: 3, 6: 7, 8: 15}[order]
    case["steps"] = _log_int(rng, 1, max(1, min(60, int(most / (evals * float(n) * n)))))
    return case


# ------------------------------------------------------------------ systems --
def _directions(g, n):
    w = g.uniform(-1.0, 1.0, n)
    phi = g.uniform(0.0, 2.0 * math.pi, n)
    q = np.sqrt(1.0 - w * w)
    return q * np.cos(phi), q * np.sin(phi), w


def _plummer(g, n):
    """Positions and velocities of n bodies of a Plummer sphere (Aarseth, Henon
    and Wielen 1974): radii from the inverse cumulative mass, speeds from the
    isotropic distribution function by rejection."""
    a = 3.0 * math.pi / 16.0
    r = a / np.sqrt(g.uniform(1e-9, 0.999, n) ** (-2.0 / 3.0) - 1.0)
    q = np.empty(n)
    todo = np.arange(n)
    while len(todo):
        t = g.uniform(0.0, 1.0, len(todo))
        ok = g.uniform(0.0, 0.1, len(todo)) < t * t * (1.0 - t * t) ** 3.5
        q[todo[ok]] = t[ok]
        todo = todo[~ok]
    v = q * math.sqrt(2.0) * (r * r + a * a) ** -0.25
    return [r * d for d in _directions(g, n)] + [v * d for d in _directions(g, n)]


def _ball(g, n):
    """n bodies at rest, uniform in the unit ball."""
    r = g.uniform(0.0, 1.0, n) ** (1.0 / 3.0)
    return [r * d for d in _directions(g, n)] + [np.zeros(n)] * 3


def _sizes(case):
    """The ensemble's system sizes, uniform in their logarithm: part of the case,
    whatever the seed of the bodies."""
    k, lo, hi = case["systems"], math.log(case["n_min"]), math.log(case["n_max"])
    q = (np.random.default_rng(k).permutation(k) + 0.5) / k
    return np.exp(lo + (hi - lo) * q).round().astype(np.int64)


def _inputs(case, seed):
    g = np.random.default_rng(seed)
    if case["kind"] == "batch":
        sizes = _sizes(case)
        s = dict(zip(STATE, _plummer(g, int(sizes.sum()))))
        s["m"] = np.repeat(1.0 / sizes, sizes)
        s["offsets"] = np.concatenate([[0], np.cumsum(sizes)])
        return s
    n = case["n"]
    s = dict(zip(STATE, _ball(g, n) if case.get("ic") == "ball" else _plummer(g, n)))
    s["m"] = np.full(n, 1.0 / n)
    if case["kind"] == "ij":
        k = case["n_src"]
        p = _plummer(g, k) if k != n else [s[d] for d in STATE]
        s["src"] = {"x": p[0], "y": p[1], "z": p[2], "m": np.full(k, 1.0 / k)}
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    ctx = nbr.Context(0)
    state = {"case": case, "ctx": ctx, "system": s}
    if case["kind"] == "batch":
        ctx.batch_upload(s["offsets"], s)
    elif case["kind"] in ("run", "forces"):
        ctx.upload(s)
        if case["n"] <= HOST_N:
            state["host"] = {k: np.zeros(case["n"]) for k in STATE}
        elif case["kind"] == "run":
            # the program's own copy of the state, written in the solver's
            # stream order (the context's arrays change with the next step)
            kind = torch.float32 if case["precision"] == "fp32c" else torch.float64
            state["device"] = {k: torch.zeros(case["n"], dtype=kind, device="cuda") for k in STATE}
            state["stream"] = torch.cuda.ExternalStream(ctx.stream)
    return state


def run(state):
    case, ctx = state["case"], state["ctx"]
    precision, eps2 = PRECISION[case["precision"]], case["eps"] ** 2
    narrow = case["precision"] == "fp32c"
    if case["kind"] == "ij":
        s = state["system"]
        j = s["src"]
        return ctx.accel_ij(s["x"], s["y"], s["z"], j["x"], j["y"], j["z"], j["m"], mi=s["m"],
                            precision=precision, eps2=eps2, want_force=True)
    if case["kind"] == "forces":
        return ctx.forces(precision, eps2=eps2)
    if case["kind"] == "batch":
        ctx.batch_run(precision, dt=case["dt"], steps=case["steps"], eps2=eps2)
        out = ctx.batch_download()
        return {k: v.astype(np.float32) for k, v in out.items()} if narrow else out
    r = ctx.run(precision, SCHEME[case["scheme"]], case["order"], case["dt"], case["steps"],
                eps2=eps2, diag=case["diag"])
    if "host" in state:
        out = ctx.download(state["host"])
        out = {k: v.astype(np.float32) for k, v in out.items()} if narrow else dict(out)
    else:
        out = dict(state["device"])
        with torch.cuda.stream(state["stream"]):
            for k, v in ctx.state_tensors().items():
                out[k].copy_(v[:case["n"]])
    if case["diag"]:
        for when, d in zip(("before", "after"), r["diag"]):
            out[when] = [d["T"], d["U"], d["E"], d["M"]]
    return out


# --------------------------------------------------------------------- work --
def _evals(case):
    """Force evaluations of one pass (a KDK run's first pass does one more)."""
    return case["steps"] * {2: 1, 4: 3, 6: 7, 8: 15}[case.get("order", 2)]


def work(case):
    """Bytes: the state read and written once.  Operations: per pair of bodies
    3 differences, 6 for the softened square, 4 for the inverse cube (its
    reciprocal square root counted as one), and 7 for the force on each of
    the two bodies; an energy check needs 12 per pair."""
    if case["kind"] == "batch":
        # the expected square of a size that is uniform in its logarithm
        lo, hi = float(case["n_min"]), float(case["n_max"])
        mean, square = (hi - lo) / math.log(hi / lo), (hi * hi - lo * lo) / 2 / math.log(hi / lo)
        return {"bytes": 104.0 * mean * case["systems"],
                "flops": _evals(case) * case["systems"] * square / 2 * 27.0}
    n = float(case["n"])
    if case["kind"] == "ij":
        k = float(case["n_src"])
        return {"bytes": 56.0 * n + 32.0 * k, "flops": 20.0 * n * k}
    if case["kind"] == "forces":
        return {"bytes": 56.0 * n, "flops": 13.5 * n * n}
    return {"bytes": 104.0 * n,
            "flops": n * n / 2 * (27.0 * _evals(case) + (24.0 if case["diag"] else 0.0))}


# -------------------------------------------------------------------- exact --
def _yoshida(order):
    """c and d of the symplectic schemes of order 2, 4, 6 and 8 (Yoshida 1990;
    the solution A of order 6 and D of order 8)."""
    c2 = 2.0 ** (1.0 / 3.0)
    w = {2: [], 4: [1.0 / (2.0 - c2)],
         6: [-1.17767998417887, 0.235573213359357, 0.78451361047756],
         8: [-0.161582374150097e1, -0.244699182370524e1, -0.716989419708120e-2,
             0.244002732616735e1, 0.157739928123617, 0.182020630970714e1,
             0.104242620869991e1]}[order]
    w = w[::-1] + [1.0 - 2.0 * sum(w)] + w
    d = w
    c = [w[0] / 2] + [(a + b) / 2 for a, b in zip(w, w[1:])] + [w[-1] / 2]
    return c, d


def _accel(p, q, m, eps2):
    """Accelerations at p (..., 3, n) from bodies q (..., 3, k) of masses m
    (..., k), and their potentials, in 64 bits."""
    n, k = p.shape[-1], q.shape[-1]
    a, phi = torch.zeros_like(p), torch.zeros_like(p[..., 0, :])
    rows = max(1, int(2e8 / (k * p[..., 0, 0].numel())))
    for i in range(0, n, rows):
        d = [q[..., c, None, :] - p[..., c, i:i + rows, None] for c in range(3)]
        r2 = d[0] * d[0]
        r2.addcmul_(d[1], d[1]).addcmul_(d[2], d[2])
        own = r2 == 0.0
        y = r2.add_(eps2).rsqrt_()
        y.masked_fill_(own, 0.0)
        phi[..., i:i + rows] = -(y @ m[..., None])[..., 0]
        s = (y * y).mul_(y).mul_(m[..., None, :])
        for c in range(3):
            a[..., c, i:i + rows] = (s * d[c]).sum(-1)
    return a, phi


def _advance(case, x, v, m):
    eps2, dt = case["eps"] ** 2, case["dt"]
    scheme = case.get("scheme", "kdk")

    def accel():
        return _accel(x, x, m, eps2)[0]

    if scheme == "kdk":
        a = accel()
        for _ in range(case["steps"]):
            v += 0.5 * dt * a
            x += dt * v
            a = accel()
            v += 0.5 * dt * a
    elif scheme == "euler":
        for _ in range(case["steps"]):
            a = accel()
            x += dt * v
            v += dt * a
    else:
        c, d = _yoshida(case["order"])
        for _ in range(case["steps"]):
            for ci, di in zip(c, d):
                x += ci * dt * v
                v += di * dt * accel()
            x += c[-1] * dt * v


def _energies(case, x, v, m):
    t = float((0.5 * m * (v * v).sum(0)).sum())
    u = float((0.5 * m * _accel(x, x, m, case["eps"] ** 2)[1]).sum())
    return [t, u, t + u, float(m.sum())]


def exact(case, seed):
    s = _inputs(case, seed)
    dev = torch.device("cuda")

    def up(*arrays):
        return torch.tensor(np.stack(arrays), dtype=torch.float64, device=dev)

    m = up(s["m"])[0]
    x, v = up(s["x"], s["y"], s["z"]), up(s["vx"], s["vy"], s["vz"])
    if case["kind"] == "batch":
        o = s["offsets"]
        if float(((o[1:] - o[:-1]) ** 2.0).sum()) * (case["steps"] + 1) > EXACT_PAIRS:
            return None
        # systems of about the same size together, padded with massless bodies
        by_size = np.argsort(o[1:] - o[:-1], kind="stable")
        for g in np.array_split(by_size, max(1, len(by_size) // 16)):
            k = int(max(o[i + 1] - o[i] for i in g))
            X, V, M = (torch.zeros((len(g),) + d + (k,), dtype=torch.float64, device=dev)
                       for d in ((3,), (3,), ()))
            for r, i in enumerate(g):
                w = o[i + 1] - o[i]
                X[r, :, :w], V[r, :, :w] = x[:, o[i]:o[i + 1]], v[:, o[i]:o[i + 1]]
                M[r, :w] = m[o[i]:o[i + 1]]
            _advance(case, X, V, M)
            for r, i in enumerate(g):
                w = o[i + 1] - o[i]
                x[:, o[i]:o[i + 1]], v[:, o[i]:o[i + 1]] = X[r, :, :w], V[r, :, :w]
        return dict(zip(STATE, list(x) + list(v)))
    if case["kind"] == "ij":
        j = s["src"]
        if float(case["n"]) * case["n_src"] > EXACT_PAIRS:
            return None
        q = up(j["x"], j["y"], j["z"])
        return m * _accel(x, q, up(j["m"])[0], case["eps"] ** 2)[0]
    if float(case["n"]) ** 2 * (_evals(case) + 3 if case["kind"] == "run" else 1) > EXACT_PAIRS * 2:
        return None
    if case["kind"] == "forces":
        return _accel(x, x, m, case["eps"] ** 2)[0]
    before = _energies(case, x, v, m) if case["diag"] else None
    _advance(case, x, v, m)
    out = dict(zip(STATE, list(x) + list(v)))
    if case["diag"]:
        out["before"], out["after"] = before, _energies(case, x, v, m)
    return out
