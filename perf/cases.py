"""Performance cases of the sweeping-preconditioned Helmholtz solver.

Every case is one of the calls a program makes, at a size such a program
uses, through the package's public entry points:

  apply     the global operator on a block of wavefields (FP64), the call of
            a user's own Krylov or time-harmonic post-processing loop
  sweep     one application of the preconditioner, the call of a user's own
            Krylov method (mixed: complex-single factors; fp64)
  solve     GMRES(20) to 1e-4 for a block of sources on the device, factors
            in hand (modelling many shots in one velocity model)
  plain     the reference drivers' sequence on host data: Initialize, then
            Solve, all in FP64
  preview   Initialize with a new velocity model and solve few shots (mixed)
  gradient  one misfit and velocity gradient of a waveform inversion: factor,
            forward solve, adjoint solve, gradient (mixed)
  batch     independent problems of uneven size, several in flight (mixed)

Mixed-precision fields are handed on in complex single, which is what their
factors and sweeps carry; FP64 ones in complex double.  Sizes count the PML
points.  Inputs are drawn from the seed on the GPU: smooth random velocity
anomalies or faulted layers, and Gaussian point sources.
"""
import math

import numpy as np
import torch

import psp_b200 as P
from psp_b200 import batch as psp_batch
from psp_b200.autograd import misfit_and_gradient

RESTART, RTOL = 20, 1e-4
DAMPING, PLANES, CUTOFF = 7.0, 4, 12   # DistHelmholtz defaults
STEPS = 12                             # GMRES steps that work() counts for one solve
EXACT_FLOPS = 3.0e14                   # largest elimination that exact() does (a sweep: a third of that)


def listed():
    return [
        # a unit-test sized operator call: launch and allocation latency
        dict(name="apply_tiny", path="apply", nx=22, ny=23, nz=24, k=3, pml=5, layers=0),
        # the operator on the shots of the 100^3 model with an 8-point PML
        dict(name="apply_116", path="apply", nx=116, ny=116, nz=116, k=16, pml=8, layers=0),
        # the smallest whole solve, uneven sides: latency of every launch
        dict(name="solve_tiny", path="solve", nx=22, ny=23, nz=24, k=3, pml=5, layers=0),
        # FP64 preconditioner on an odd-sized mid-size grid
        dict(name="sweep_fp64", path="sweep", nx=57, ny=53, nz=61, k=5, pml=5, layers=0, mixed=False),
        # preconditioner on the layered inversion model, 32 shots
        dict(name="sweep_96_k32", path="sweep", nx=96, ny=96, nz=76, k=32, pml=8, layers=8, mixed=True),
        # preconditioner on the 100^3 model, 16 shots
        dict(name="sweep_116_k16", path="sweep", nx=116, ny=116, nz=116, k=16, pml=8, layers=0, mixed=True),
        # preconditioner for one shot on a ragged grid (a single-source inversion step)
        dict(name="sweep_75_k1", path="sweep", nx=75, ny=67, nz=58, k=1, pml=5, layers=0, mixed=True),
        # the 40^3 interior reference problem from host buffers, factor and solve in FP64
        dict(name="plain_50", path="plain", nx=50, ny=50, nz=50, k=4, pml=5, layers=0),
        # a new velocity model looked at with two shots
        dict(name="preview_80", path="preview", nx=80, ny=84, nz=60, k=2, pml=8, layers=8),
        # many shots in one layered model (the largest case)
        dict(name="solve_140_k32", path="solve", nx=140, ny=140, nz=80, k=32, pml=10, layers=12),
        # one inversion gradient, 32 surface shots, receivers on the whole surface
        dict(name="gradient_96", path="gradient", nx=96, ny=96, nz=76, k=32, pml=8, layers=8),
        # independent uneven problems, as a parameter study submits them
        dict(name="batch_5", path="batch", nx=56, ny=48, nz=52, k=4, pml=5, layers=0, count=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["apply", "apply", "sweep", "sweep", "sweep", "sweep64", "solve", "solve", "plain", "preview",
                       "gradient", "batch"])
    pml = rng.choice([5, 8])
    layers = rng.choice([0, 8])
    lo, hi, kmax = {"apply": (20, 120, 32), "sweep": (24, 104, 32), "sweep64": (24, 60, 8), "solve": (24, 84, 32),
                    "plain": (24, 50, 6), "preview": (28, 84, 4), "gradient": (28, 64, 16),
                    "batch": (32, 52, 8)}[path]
    lo = max(lo, 2 * pml + 12)
    c = dict(path="sweep" if path == "sweep64" else path, nx=_log(rng, lo, hi), ny=_log(rng, lo, hi),
             nz=_log(rng, lo, hi), k=_log(rng, 1, kmax), pml=pml, layers=layers)
    if c["path"] == "sweep":
        c["mixed"] = path == "sweep"
    if path == "batch":
        c["count"] = rng.randint(2, 4)
    return c


# ------------------------------------------------------------------ inputs


def _disc(c, nx, ny, nz, slowest):
    """Ten points per wavelength of the slowest velocity, spacing 1 / (largest
    interior + 1), PML amplitudes of the drivers (1.5; 7.5 for km/s models)."""
    pml = c["pml"]
    h = 1.0 / (max(nx, ny, nz) - 2 * pml + 1)
    omega = 2 * math.pi * slowest / (10.0 * h)
    return P.Discretization(omega, nx, ny, nz, (nx + 1) * h, (ny + 1) * h, (nz + 1) * h, pml=(pml,) * 3,
                            sigma=7.5 if c["layers"] else 1.5)


def _velocity(c, nx, ny, nz, rng, dev):
    """Background 1 with Gaussian anomalies in [0.6, 1.8], or layers of
    1.5 - 5.5 km/s across two dipping faults; (nz, ny, nx) float64."""
    ax = [torch.arange(n, device=dev, dtype=torch.float64) / (n - 1) for n in (nz, ny, nx)]
    z, y, x = ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]
    if not c["layers"]:
        v = torch.ones(nz, ny, nx, device=dev, dtype=torch.float64)
        for _ in range(6):
            p, a, w = rng.uniform(0.1, 0.9, 3), rng.uniform(-0.4, 0.6), rng.uniform(0.08, 0.2)
            v += a * torch.exp(-((x - p[0]) ** 2 + (y - p[1]) ** 2 + (z - p[2]) ** 2) / (2 * w * w))
        return v.clamp_(0.6, 1.8)
    n = c["layers"]
    shift = torch.zeros(nz, ny, nx, device=dev, dtype=torch.float64)
    for _ in range(2):
        d, p = rng.uniform(-1, 1, 3), rng.uniform(0.3, 0.7, 3)
        side = (x - p[0]) * d[0] + (y - p[1]) * d[1] + (z - p[2]) * (0.3 + abs(d[2])) > 0
        shift += side * (rng.uniform(0.15, 0.3) / n)
    tops = torch.tensor((np.arange(1, n) + rng.uniform(-0.15, 0.15, n - 1)) / n, device=dev)
    speeds = torch.linspace(1.5, 5.5, n, device=dev, dtype=torch.float64)
    return speeds[torch.searchsorted(tops, (z - shift).contiguous())].contiguous()


def _sources(c, nx, ny, nz, k, rng, dev, surface=False):
    """Gaussian point sources of width two spacings away from the faces (or
    just under the top PML): (nz, ny, nx, k) complex128."""
    g = []
    for a, n in enumerate((nz, ny, nx)):
        at = rng.integers(c["pml"] + 2, n - c["pml"] - 2, k)
        if surface and a == 0:
            at[:] = c["pml"]
        i = torch.arange(n, device=dev, dtype=torch.float64)
        g.append(torch.exp(-((i[:, None] - torch.tensor(at, device=dev, dtype=torch.float64)) ** 2) / 8.0))
    out = torch.zeros(nz, ny, nx, k, device=dev, dtype=torch.complex128)
    torch.view_as_real(out)[..., 0] = -(g[0][:, None, None] * g[1][None, :, None] * g[2][None, None, :])
    return out


def _inputs(c, seed):
    """What exact() shares with prepare(): discretization, velocity, right-hand sides."""
    dev = torch.device("cuda", 0)
    rng = np.random.default_rng(seed)
    nx, ny, nz, k = c["nx"], c["ny"], c["nz"], c["k"]
    vel = _velocity(c, nx, ny, nz, rng, dev)
    disc = _disc(c, nx, ny, nz, 1.5 if c["layers"] else 0.8)
    if c["path"] in ("apply", "sweep"):  # Krylov vectors: dense fields
        gen = torch.Generator(device=dev).manual_seed(int(seed) + 1)
        rhs = torch.randn(nz, ny, nx, k, device=dev, dtype=torch.complex128, generator=gen)
    else:
        rhs = _sources(c, nx, ny, nz, k, rng, dev, surface=c["path"] == "gradient")
    return disc, vel, rhs, rng


def _batch_sides(c):
    """Uneven problems: the sides step down from the case's by up to a quarter."""
    return [[max(2 * c["pml"] + 12, int(c[n] * (1 - 0.06 * ((i * j + i) % 5))))
             for j, n in enumerate(("nx", "ny", "nz"))] for i in range(c["count"])]


def _mixed(c):
    return c.get("mixed", c["path"] in ("solve", "preview", "gradient", "batch"))


def prepare(case, seed):
    c = dict(case)
    disc, vel, rhs, rng = _inputs(c, seed)
    s = dict(case=c, path=c["path"], mixed=_mixed(c))
    if c["path"] == "batch":
        s["problems"] = []
        for i, n in enumerate(_batch_sides(c)):
            v = _velocity(c, *n, rng, vel.device)
            f = _sources(c, *n, 1 + i % c["k"], rng, vel.device)
            s["problems"].append(psp_batch.Problem(_disc(c, *n, 1.5 if c["layers"] else 0.8),
                                                   v.reshape(-1).cpu().numpy(),
                                                   f.reshape(-1, f.shape[-1]).cpu().numpy(), "p%d" % i))
        return s
    H = s["solver"] = P.DistHelmholtz(disc, DAMPING, PLANES, CUTOFF, device=0)
    s["stream"] = torch.cuda.ExternalStream(H.stream_ptr(), device=0)
    torch.cuda.synchronize()
    if c["path"] == "plain":
        s["velocity"] = P.DistUniformGrid(c["nx"], c["ny"], c["nz"], 1, np.float64, vel.cpu().numpy())
        s["rhs"] = rhs.cpu().numpy()
        return s
    s["velocity"], s["rhs"] = vel.reshape(-1), rhs.reshape(-1)
    if c["path"] == "gradient":
        ny, nx, pml = c["ny"], c["nx"], c["pml"]
        yy, xx = np.meshgrid(np.arange(pml, ny - pml), np.arange(pml, nx - pml), indexing="ij")
        s["receivers"] = torch.tensor((xx + nx * (yy + ny * pml)).reshape(-1), device=vel.device)
        s["rhs"] = rhs.reshape(-1, c["k"])
        # observed data: the direct wave of each shot in the slowest medium
        h, peak = disc.wx / (nx + 1), rhs[pml].real.reshape(ny * nx, -1).argmin(0)
        dx = (s["receivers"] % (nx * ny) % nx)[:, None] - (peak % nx)[None, :]
        dy = (s["receivers"] % (nx * ny) // nx)[:, None] - (peak // nx)[None, :]
        r = h * torch.sqrt((dx * dx + dy * dy).double() + 8.0)
        s["data"] = -(8 * math.pi) ** 1.5 * h ** 3 * torch.polar(1 / (4 * math.pi * r), r * (2 * math.pi / (10 * h)))
        return s
    if c["path"] != "preview":
        H.Initialize(s["velocity"], precision=P.MIXED if s["mixed"] or c["path"] == "apply" else P.FP64)
    return s


# ------------------------------------------------------------------ the calls


def run(state):
    path, H = state["path"], state.get("solver")
    if path == "batch":
        got, _ = psp_batch.solve_batch(state["problems"], RESTART, RTOL, P.MIXED, streams=4)
        return [got[i][0].astype(np.complex64) for i in range(len(state["problems"]))]
    if path == "plain":
        B = P.DistUniformGrid(*(state["case"][n] for n in ("nx", "ny", "nz", "k")), np.complex128, state["rhs"].copy())
        H.Initialize(state["velocity"], precision=P.FP64)
        H.Solve(B, RESTART, RTOL)
        return B.data
    if path == "gradient":
        J, g = misfit_and_gradient(H, state["velocity"], state["rhs"], state["receivers"], state["data"], RESTART,
                                   RTOL, precision=P.MIXED)
        return {"misfit": J.float(), "gradient": g.float()}
    B = state["rhs"].clone()
    state["stream"].wait_stream(torch.cuda.current_stream())  # the solver works on a stream of its own
    if path == "apply":
        H.multiply_device(B)
    elif path == "sweep":
        H.precondition_device(B)
    else:
        if path == "preview":
            H.Initialize(state["velocity"], precision=P.MIXED)
        H.Solve(B, RESTART, RTOL)
    return B.to(torch.complex64) if state["mixed"] else B


# ------------------------------------------------------------------ work


def _panels(c, nx, ny, nz):
    """(lowest v, depth, padding) of every panel, v = nz - 1 - z the sweep
    coordinate: a bottom panel of pml + 4 planes, inner panels of 4 planes, a
    leftover, a top panel of pml + 4 planes; all but the first are padded by
    an artificial PML below."""
    b = c["pml"]
    ends, inner = b + PLANES, nz - 2 * (b + PLANES)
    depths = [ends] + [PLANES] * (inner // PLANES) + ([inner % PLANES] if inner % PLANES else []) + [ends]
    lows = np.concatenate([[0], np.cumsum(depths)[:-1]])
    return [(int(lo), d, 0 if p == 0 else b) for p, (lo, d) in enumerate(zip(lows, depths))]


def _front_sums(disc):
    """Per panel class: nonzeros of the factors and flops of the factorization."""
    out = {}
    for cls in range(3):
        try:
            info, _ = P.analyze_class(disc, PLANES, CUTOFF, cls)
        except (P.LogicError, RuntimeError):
            continue
        s, u = info[:, 1].astype(float), info[:, 2].astype(float)
        nnz = (s + u) * s - s * (s - 1) / 2
        out[cls] = (nnz.sum(), (8 * (s ** 3 / 6 + s ** 2 * u / 2 + s * u * (u + 1) / 2)).sum())
    return out


def _work(c, nx, ny, nz, k, mixed):
    """(sweep, factor, apply) as (bytes, flops)."""
    disc = _disc(c, nx, ny, nz, 1.0)
    sums, geo = _front_sums(disc), P.panel_geometry(disc, PLANES)
    entry = 8.0 if mixed else 16.0
    N = float(nx * ny * nz)
    sweep, factor = [0.0, 0.0], [8.0 * N, 0.0]
    for p, row in enumerate(geo):
        nnz, fl = sums[int(row[3])]
        times = 2 if p < len(geo) - 1 else 1  # every panel but the top one is solved twice
        sweep[0] += times * 2 * entry * nnz   # forward and backward read the factors
        sweep[1] += times * 2 * 8.0 * nnz * k
        factor[0] += entry * nnz
        factor[1] += fl
    sweep[0] += 32.0 * N * k
    return sweep, factor, [N * (32.0 * k + 8), 56.0 * N * k]


def work(case):
    c = dict(case)
    sizes = [(c["nx"], c["ny"], c["nz"], c["k"])]
    if c["path"] == "batch":
        sizes = [(*n, 1 + i % c["k"]) for i, n in enumerate(_batch_sides(c))]
    total = np.zeros(2)
    for nx, ny, nz, k in sizes:
        sweep, factor, apply = (np.array(v) for v in _work(c, nx, ny, nz, k, _mixed(c)))
        # a solve: its sweeps and operators, and per step the basis read twice (half full on average) and x
        vec = np.array([16.0, 8.0]) * nx * ny * nz * k
        solve = (STEPS + 1) * sweep + 2 * STEPS * apply + STEPS * (STEPS + 4) * vec
        total += {"apply": apply, "sweep": sweep, "solve": solve, "plain": factor + solve, "preview": factor + solve,
                  "gradient": factor + 2 * solve + apply, "batch": factor + solve}[c["path"]]
    return {"bytes": float(total[0]), "flops": float(total[1])}


# ------------------------------------------------------------------ 64-bit values


def _stretch(lo, hi, n, b, sigma, h, omega, edge=0):
    """1-D PML stretches at indices lo .. hi - 1 (PML on both sides)."""
    out = np.ones(hi - lo, dtype=np.complex128)
    for j, i in enumerate(range(lo, hi)):
        d = (edge + b - 1) - i if i < edge + b - 1 else i - (n - b) if i > n - b else 0
        out[j] += 1j * (sigma / (b * h)) * (d / b) ** 2 * (2 * math.pi / omega)
    return out


def _operator(disc, vel, lo, hi, edge, omega):
    """The stencil on planes v = lo .. hi - 1: (centre, [x, y, v] couplings),
    arrays (v, y, x); coupling a[i] is the (positive) term between i and i + 1."""
    dev = vel.device
    n, b, w, sg = (disc.nx, disc.ny, disc.nz), disc.bx, (disc.wx, disc.wy, disc.wz), disc.sigmax
    h = [w[a] / (n[a] + 1) for a in range(3)]
    s = [_stretch(-1, n[0] + 1, n[0], b, sg, h[0], disc.omega), _stretch(-1, n[1] + 1, n[1], b, sg, h[1], disc.omega),
         _stretch(lo - 1, hi + 1, n[2], b, sg, h[2], disc.omega, edge)]
    t = [torch.tensor(v, device=dev) for v in s]
    m = [t[0][1:-1][None, None, :], t[1][1:-1][None, :, None], t[2][1:-1][:, None, None]]
    face = [((1 / t[a][1:] + 1 / t[a][:-1]) / (2 * h[a] ** 2)) for a in range(3)]
    shape = [(1, 1, -1), (1, -1, 1), (-1, 1, 1)]
    cross = [m[1] * m[2], m[0] * m[2], m[0] * m[1]]
    left = [cross[a] * face[a][:-1].reshape(shape[a]) for a in range(3)]
    right = [cross[a] * face[a][1:].reshape(shape[a]) for a in range(3)]
    v = vel.flip(0)[lo:hi]
    centre = sum(left) + sum(right) - (omega / v) ** 2 * (m[0] * m[1] * m[2])
    full = centre.shape
    return centre, [r.expand(full) for r in right], [q.expand(full) for q in left]


def _apply(disc, vel, B):
    """A B for a natural-order (z, y, x, k) block."""
    centre, right, left = _operator(disc, vel, 0, disc.nz, 0, disc.omega)
    X = B.flip(0)
    Y = centre[..., None] * X
    Y[:, :, :-1] -= right[0][:, :, :-1, None] * X[:, :, 1:]
    Y[:, :, 1:] -= left[0][:, :, 1:, None] * X[:, :, :-1]
    Y[:, :-1] -= right[1][:, :-1, :, None] * X[:, 1:]
    Y[:, 1:] -= left[1][:, 1:, :, None] * X[:, :-1]
    Y[:-1] -= right[2][:-1, ..., None] * X[1:]
    Y[1:] -= left[2][1:, ..., None] * X[:-1]
    return Y.flip(0).contiguous()


def _eliminate(op, B, along, kept=None):
    """Solves the stencil system op X = B, B (v, y, x, k), by block
    elimination over planes of array dimension `along`; `kept`: a list that
    holds the eliminated blocks from one call with op to the next."""
    centre, right, _ = op
    axis = {2: 0, 1: 1, 0: 2}  # array dimension -> coupling number
    order = [along] + [d for d in range(3) if d != along]
    c = centre.permute(order)
    out = right[axis[along]].permute(order)
    ins = [right[axis[d]].permute(order) for d in order[1:]]
    n, p, q = c.shape
    rhs = B.permute(order + [3]).reshape(n, p * q, -1)
    idx = torch.arange(p * q, device=c.device).reshape(p, q)

    def block(i):
        D = torch.diag(c[i].reshape(-1))
        for a, (u, v) in zip(ins, ((idx[:-1], idx[1:]), (idx[:, :-1], idx[:, 1:]))):
            e = -(a[i][:-1] if u.shape[0] < p else a[i][:, :-1]).reshape(-1)
            D[u.reshape(-1), v.reshape(-1)] = e
            D[v.reshape(-1), u.reshape(-1)] = e
        return D

    inv, y = kept if kept is not None else [], []
    for i in range(n):
        e = out[i - 1].reshape(-1, 1) if i else None
        if len(inv) == i:
            inv.append(torch.linalg.inv(block(i) - e * inv[-1] * e.T if i else block(i)))
        y.append(rhs[i] + e * (inv[i - 1] @ y[-1]) if i else rhs[i])
    x = [None] * n
    for i in range(n - 1, -1, -1):
        r = y[i] if i == n - 1 else y[i] + out[i].reshape(-1, 1) * x[i + 1]
        x[i] = inv[i] @ r
    back = [0, 0, 0]
    for j, d in enumerate(order):
        back[d] = j
    return torch.stack(x).reshape(n, p, q, -1).permute(back + [3]).contiguous()


def _sweep(disc, vel, B, c):
    """The preconditioner: block LDL^T sweep over the panels, each panel's
    subproblem (artificial PML below it, damped frequency) solved directly."""
    panels = _panels(c, disc.nx, disc.ny, disc.nz)
    kept = [[] for _ in panels]
    X = B.flip(0).clone()
    _, right, left = _operator(disc, vel, 0, disc.nz, 0, disc.omega)

    def solve(p, R):
        lo, depth, pad = panels[p]
        op = _operator(disc, vel, lo - pad, lo + depth, lo - pad, disc.omega + 1j * DAMPING)
        full = torch.zeros(pad + depth, *R.shape[1:], device=R.device, dtype=R.dtype)
        full[pad:] = R
        return _eliminate(op, full, 2, kept[p])[pad:]

    for p, (lo, depth, _) in enumerate(panels):
        R = X[lo:lo + depth].clone()
        if p:
            R[0] += left[2][lo][..., None] * X[lo - 1]
        X[lo:lo + depth] = solve(p, R)
    for p in range(len(panels) - 2, -1, -1):
        lo, depth, _ = panels[p]
        R = torch.zeros_like(X[lo:lo + depth])
        R[-1] = right[2][lo + depth - 1][..., None] * X[lo + depth]
        X[lo:lo + depth] += solve(p, R)
    return X.flip(0).contiguous()


def exact(case, seed):
    c = dict(case)
    if c["path"] in ("gradient", "batch"):
        return None
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    dims = (nz, ny, nx)
    along = dims.index(max(dims))
    flops = 22.0 * max(dims) * (nx * ny * nz / max(dims)) ** 3
    if c["path"] == "sweep":
        flops = sum(22.0 * nx * (ny * (d + pad)) ** 3 for _, d, pad in _panels(c, nx, ny, nz))
    if c["path"] != "apply" and flops > EXACT_FLOPS / (3 if c["path"] == "sweep" else 1):
        return None
    disc, vel, rhs, _ = _inputs(c, seed)
    if c["path"] == "apply":
        X = _apply(disc, vel, rhs)
    elif c["path"] == "sweep":
        X = _sweep(disc, vel, rhs, c)
    else:
        X = _eliminate(_operator(disc, vel, 0, nz, 0, disc.omega), rhs.flip(0), along).flip(0).contiguous()
    return X.cpu().numpy() if c["path"] == "plain" else X.reshape(-1)
