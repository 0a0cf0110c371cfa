"""The work a program has this framework do, as cases that can be timed and compared.

Every pass is a whole call of a public entry point on prepared chunks: the
device-resident timestep (`Host.solve_device`), the timestep through the
reference's drivers over run_* (`Host.solve`), the field summary, the
iterative-refinement timestep, the batched timestep and the 3D adjoint
gradient. A pass starts from the deck's initial energy (run_store_energy
copies it back), so every pass of a state does the same work.

Decks are seeded as tealeaf_b200.problems describes them: ambient density
100 and energy 1e-4, boxes and discs of density 0.1 with energy uniform in
[0.1, 25], dt 0.004, reciprocal conductivity. A full 4096^2 timestep takes
thousands of iterations; the big cases stop at `max_iters`, which leaves the
rate of the loop and its start and end, as the benchmark's CPU arm does.
"""
import ctypes
import math
import random

import numpy as np
import torch

from tealeaf_b200.batch import Batch
from tealeaf_b200.host import Host
from tealeaf_b200.problems import Problem

AMBIENT = (100.0, 1e-4)
DOMAIN = 10.0
DT = 0.004
HALO = 2


# ------------------------------------------------------------------- cases --

def listed():
    return [
        # The smallest calls: a mesh of a test or a teaching run, to convergence, with its field summary.
        dict(name="cg2d_64", kind="device", dims=2, nx=64, ny=64, solver="cg", max_iters=20000, summary=True),
        # The mesh of the reference's own sample decks and of the CPU-runnable workload, whole timestep.
        dict(name="cg2d_512", kind="device", dims=2, nx=512, ny=512, solver="cg", max_iters=20000, summary=True),
        # A ragged mesh with odd sides and the block preconditioner, to convergence.
        dict(name="pcg2d_odd", kind="device", dims=2, nx=1013, ny=777, solver="cg", max_iters=20000, summary=False,
             precond="jac_block"),
        # The drop-in benchmark: FP64 CG at 4096^2.
        dict(name="cg2d_4096", kind="device", dims=2, nx=4096, ny=4096, solver="cg", max_iters=200, summary=False),
        # The same benchmark's other two solvers, past their CG presteps.
        dict(name="cheby2d_4096", kind="device", dims=2, nx=4096, ny=4096, solver="cheby", max_iters=300,
             summary=False),
        dict(name="ppcg2d_2048", kind="device", dims=2, nx=2048, ny=2048, solver="ppcg", max_iters=100,
             summary=False),
        # 3D drop-in: the benchmark's CG mesh, and a ragged mesh with Chebyshev.
        dict(name="cg3d_256", kind="device", dims=3, nx=256, ny=256, nz=256, solver="cg", max_iters=100,
             summary=False),
        dict(name="cheby3d_ragged", kind="device", dims=3, nx=130, ny=97, nz=110, solver="cheby", max_iters=200,
             summary=True),
        # The reference's own drivers calling run_* (one host round trip per dot product) and their summary.
        dict(name="drivers2d_1000", kind="drivers", dims=2, nx=1000, ny=1000, solver="cg", max_iters=300,
             summary=True),
        # Mixed precision: FP32 sweeps inside FP64 refinement to a relative residual of 1e-10.
        dict(name="refine2d_1536", kind="refine", dims=2, nx=1536, ny=1536, solver="cg", max_iters=20000,
             precision=32),
        # Many uneven problems in one persistent launch.
        dict(name="batch_24", kind="batch", dims=2, count=24, lo=64, hi=768, meshes=5),
        # Gradient of a scalar of the final temperature through several 3D timesteps.
        dict(name="adjoint3d_48", kind="adjoint", dims=3, nx=48, ny=48, nz=48, solver="cg", max_iters=20000,
             steps=4, every=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["device2", "device2", "device2", "device3", "device3", "drivers", "refine", "batch",
                       "adjoint"])
    if kind == "device2":
        nx, ny = _log(rng, 48, 4096), _log(rng, 48, 4096)
        solver = rng.choice(["cg", "cg", "cheby", "ppcg"])
        # cut by work: no more than the largest listed case's
        cap = min(20000, 3_000_000_000 // (nx * ny))
        if solver == "ppcg":
            cap = min(400, cap // 5)
        elif solver == "cheby":
            cap = min(2000, cap)
        c = dict(kind="device", dims=2, nx=nx, ny=ny, solver=solver, max_iters=max(40, cap),
                 summary=rng.random() < 0.5)
        if solver == "cg" and nx * ny <= 1 << 20 and rng.random() < 0.4:
            c.update(precond=rng.choice(["jac_diag", "jac_block"]), max_iters=20000)
        return c
    if kind == "device3":
        n = [_log(rng, 16, 256) for _ in range(3)]
        solver = rng.choice(["cg", "cg", "cheby", "ppcg"])
        cap = min(2000, 1_500_000_000 // (n[0] * n[1] * n[2]))
        if solver == "ppcg":
            cap = min(200, cap // 5)
        return dict(kind="device", dims=3, nx=n[0], ny=n[1], nz=n[2], solver=solver, max_iters=max(40, cap),
                    summary=rng.random() < 0.5)
    if kind == "drivers":
        nx, ny = _log(rng, 48, 2048), _log(rng, 48, 2048)
        return dict(kind="drivers", dims=2, nx=nx, ny=ny, solver=rng.choice(["cg", "cheby", "ppcg"]),
                    max_iters=rng.randint(60, 300), summary=True)
    if kind == "refine":
        return dict(kind="refine", dims=2, nx=_log(rng, 96, 1536), ny=_log(rng, 96, 1536),
                    solver=rng.choice(["cg", "ppcg"]), max_iters=20000, precision=rng.choice([32, 32, 64]))
    if kind == "batch":
        return dict(kind="batch", dims=2, count=rng.randint(4, 24), lo=64, hi=rng.randint(256, 768),
                    meshes=rng.randrange(1000))
    n = [_log(rng, 16, 56) for _ in range(3)]
    return dict(kind="adjoint", dims=3, nx=n[0], ny=n[1], nz=n[2], solver="cg", max_iters=20000,
                steps=rng.randint(2, 4), every=rng.choice([1, 2]))


# ------------------------------------------------------------------- decks --

def _shapes(rng, dims, boxes, discs):
    """Painted states after the ambient one: (lo, hi, None, energy) boxes, (centre, None, radius, energy) discs."""
    out = []
    for _ in range(boxes):
        lo = [rng.uniform(0.0, DOMAIN) for _ in range(dims)]
        hi = [min(a + rng.uniform(0.5, 5.0), DOMAIN) for a in lo]
        out.append((lo, hi, None, rng.uniform(0.1, 25.0)))
    for _ in range(discs):
        out.append(([rng.uniform(0.0, DOMAIN) for _ in range(dims)], None, rng.uniform(0.3, 2.0),
                    rng.uniform(0.1, 25.0)))
    return out


def _problems(case, seed):
    """The decks of a case: [(cells, shapes, eps)]."""
    rng = random.Random(seed)
    if case["kind"] == "batch":
        out, sides = [], random.Random(case["meshes"])
        for _ in range(case["count"]):
            cells = [_log(sides, case["lo"], case["hi"]) for _ in range(2)]
            out.append((cells, _shapes(rng, 2, 3, 0), 1e-12))
        return out
    cells = [case["nx"], case["ny"]] + ([case["nz"]] if case["dims"] == 3 else [])
    return [(cells, _shapes(rng, case["dims"], 6, 0 if case["dims"] == 3 else 3), 1e-15)]


def _deck(case, cells, shapes, eps):
    states = ["density=%r energy=%r" % AMBIENT]
    axes = "xyz"[: case["dims"]]
    for lo, hi, radius, energy in shapes:
        word = ("rectangle" if case["dims"] == 2 else "cuboid") if radius is None else "circular"
        ext = " ".join("%smin=%r" % (a, v) for a, v in zip(axes, lo))
        ext += " " + " ".join("%smax=%r" % (a, v) for a, v in zip(axes, lo if hi is None else hi))
        states.append("density=0.1 energy=%r geometry=%s %s%s"
                      % (energy, word, ext, "" if radius is None else " radius=%r" % radius))
    poly = case.get("solver") in ("cheby", "ppcg")
    return Problem(dims=case["dims"], cells=cells, states=states, solver=case.get("solver", "cg"), eps=eps,
                   max_iters=case.get("max_iters", 20000), dt=DT, presteps=30, ppcg_inner_steps=10,
                   check_result=False, halo_depth=HALO, error_switch=poly, eps_lim=1e30,
                   preconditioner=case.get("precond", "none"), name="perf").tea_in()


# ------------------------------------------------------------------ passes --

class _Field:
    """A chunk's device field as a tensor without a copy; keeps what frees it (the host, or its batch) alive."""

    def __init__(self, owner, host, name):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=tuple(host.shape), typestr="<f8", strides=None, version=3,
                                             data=(getattr(host.chunk, name), False))


def _field(owner, host, name):
    if host.dims == 3 and name == "u":
        name = "vec_u"
    return torch.as_tensor(_Field(owner, host, name), device="cuda")


def _restart(host):
    host.lib.run_store_energy(ctypes.byref(host.chunk), ctypes.byref(host.settings))


def prepare(case, seed):
    decks = [_deck(case, *p) for p in _problems(case, seed)]
    if case["kind"] == "batch":
        return case, Batch(decks)
    return case, Host(decks[0], dims=case["dims"])


BOX = (6.0, 9.0, 6.0, 9.0, 6.0, 9.0)


def run(state):
    case, h = state
    if case["kind"] == "batch":
        for one in h.hosts:
            _restart(one)
        h.step()
        return {"u": [_field(h, one, "u") for one in h.hosts]}
    _restart(h)
    out = {}
    if case["kind"] == "adjoint":
        j, grad, _ = h.adjoint_gradient(case["steps"], case["every"], BOX, 1e-12)
        return {"J": j, "grad": grad}
    if case["kind"] == "refine":
        h.refine_step(0, 1e-10, case["precision"], summary=False)
    elif case["kind"] == "drivers":
        out["summary"] = h.solve(0).summary
    else:
        r = h.solve_device(0, summary=case["summary"])
        if case["summary"]:
            out["summary"] = r.summary
    out["u"], out["energy"] = _field(h, h, "u"), _field(h, h, "energy")
    return out


# -------------------------------------------------------------------- work --

def _trips(case, cells):
    """Iterations of a timestep: the cap, or about what these decks take to eps 1e-15."""
    return min(case.get("max_iters", 20000), 2 * max(cells))


def work(case):
    """Compulsory traffic of the method: the streams of one iteration (operands in, results out, each once) times
    its iterations; meshes that fit on chip need only the fields in and out."""
    total_b = total_f = 0.0
    for cells, _, _ in _problems(case, 0):
        n = float(np.prod(cells))
        t = _trips(case, cells)
        solver = case.get("solver", "cg")
        flops = 24.0 if case["dims"] == 2 else 32.0
        per = 96.0 if case["dims"] == 2 else 104.0
        if case["kind"] == "adjoint":
            t *= 2 * case["steps"]
        if case["kind"] == "batch" or case.get("precision") == 32:
            per = 48.0
        if solver == "cheby":
            per, flops = 14.0, 20.0
        elif solver == "ppcg":
            per, flops = per + 160.0, flops + 200.0
        if n * 48 < 60e6:
            total_b += 64.0 * n
        else:
            total_b += per * n * t
        total_f += flops * n * t
    return {"bytes": total_b, "flops": total_f}


# ------------------------------------------------------- 64-bit references --
# The timestep in plain torch double precision (arrays [z,] y, x with a halo
# of HALO cells), written from the equations.

def _paint(dims, cells, shapes, dev):
    size = [n + 2 * HALO for n in reversed(cells)]
    rho = torch.full(size, AMBIENT[0], dtype=torch.float64, device=dev)
    e = torch.full(size, AMBIENT[1], dtype=torch.float64, device=dev)
    lo_v, hi_v, centre = [], [], []
    for ax, n in enumerate(cells):
        d = DOMAIN / n
        k = torch.arange(n + 2 * HALO, dtype=torch.float64, device=dev) - HALO
        shape = [1] * dims
        shape[dims - 1 - ax] = -1
        a, b = (d * k).reshape(shape), (d * (k + 1)).reshape(shape)
        lo_v.append(a)
        hi_v.append(b)
        centre.append(0.5 * (a + b))
    for lo, hi, radius, energy in shapes:
        # the deck's extents are drawn in by a hundredth of a cell, a disc's centre moved by it (2d/parse_config.c)
        nudge = [DOMAIN / n / 100.0 for n in cells]
        lo = [a + b for a, b in zip(lo, nudge)]
        hi = hi and [a - b for a, b in zip(hi, nudge)]
        hit = torch.ones(size, dtype=torch.bool, device=dev)
        if radius is None:
            for ax in range(dims):
                hit &= (hi_v[ax] >= lo[ax]) & (lo_v[ax] < hi[ax])
        else:
            hit = (sum((centre[ax] - lo[ax]) ** 2 for ax in range(dims)).sqrt() <= radius).expand(size)
        rho[hit] = 0.1
        e[hit] = energy
    return rho, e


def _reflect(f, depth):
    """The reflective halo of every face, `depth` layers, interior span only."""
    d = f.dim()
    for ax in range(d):
        n = f.shape[ax]
        v = f[tuple(slice(None) if a == ax else slice(HALO, -HALO) for a in range(d))]
        for k in range(depth):
            v.select(ax, HALO - 1 - k).copy_(v.select(ax, HALO + k))
            v.select(ax, n - HALO + k).copy_(v.select(ax, n - HALO - 1 - k))


def _in(f):
    return f[(slice(HALO, -HALO),) * f.dim()]


class _Operator:
    """A = I + sum over faces of k (difference) with reflective faces, on interior arrays."""

    def __init__(self, rho, cells):
        dims = rho.dim()
        w = 1.0 / rho
        self.k = []
        for ax in range(dims):   # tensor axis; its physical axis is dims - 1 - ax
            d = DOMAIN / cells[dims - 1 - ax]
            n = rho.shape[ax]
            inner = [slice(HALO, -HALO)] * dims
            a, b = list(inner), list(inner)
            a[ax], b[ax] = slice(HALO, n - HALO - 1), slice(HALO + 1, n - HALO)
            wa, wb = w[tuple(a)], w[tuple(b)]
            self.k.append((DT / (d * d)) * (wa + wb) / (2.0 * wa * wb))

    def __call__(self, u):
        out = u.clone()
        for ax, k in enumerate(self.k):
            n = u.shape[ax]
            f = k * (u.narrow(ax, 1, n - 1) - u.narrow(ax, 0, n - 1))
            out.narrow(ax, 0, n - 1).sub_(f)
            out.narrow(ax, 1, n - 1).add_(f)
        return out


def _cg(A, b, u, eps, max_iters, stop=None, record=None):
    r = b - A(u)
    p = r.clone()
    rro = float((r * r).sum())
    t = 0
    while t < max_iters and rro > 0.0:
        if stop is not None and stop(t, rro):
            break
        w = A(p)
        alpha = rro / float((p * w).sum())
        u = u + alpha * p
        r = r - alpha * w
        rrn = float((r * r).sum())
        beta = rrn / rro
        if record is not None:
            record.append((alpha, beta))
        rro = rrn
        p = r + beta * p
        t += 1
        if abs(rrn) < eps:
            break
    return u, r, p, rro, t


def _bounds(record):
    n = len(record)
    d = np.zeros(n)
    o = np.zeros(max(0, n - 1))
    for i, (al, be) in enumerate(record):
        d[i] = 1.0 / al + (record[i - 1][1] / record[i - 1][0] if i else 0.0)
        if i < n - 1:
            o[i] = math.sqrt(be) / al
    ev = np.linalg.eigvalsh(np.diag(d) + np.diag(o, 1) + np.diag(o, -1))
    return 0.95 * float(ev[0]), 1.05 * float(ev[-1])


def _coefs(lo, hi, count):
    theta, delta = (hi + lo) / 2.0, (hi - lo) / 2.0
    sigma = theta / delta
    rho, a, b = 1.0 / sigma, [], []
    for _ in range(count):
        new = 1.0 / (2.0 * sigma - rho)
        a.append(new * rho)
        b.append(2.0 * new / delta)
        rho = new
    return theta, a, b


def _solve(case, A, b, eps):
    """The solution of one timestep as the case's solver leaves it, and u where the u halo was last refreshed."""
    cap, solver = case.get("max_iters", 20000), case.get("solver", "cg")
    if case["kind"] in ("refine", "batch"):
        u = _cg(A, b, b.clone(), 1e-26 * float((b * b).sum()), 40000)[0]
        return u, u
    if case.get("precond"):
        u = _cg(A, b, b.clone(), 1e-20, 40000)[0]
        return u, u
    limit = eps * eps if case["dims"] == 3 else eps
    if solver == "cg":
        u = _cg(A, b, b.clone(), limit, cap)[0]
        return u, u
    rec = []
    u, r, p, rro, t = _cg(A, b, b.clone(), limit, cap, stop=lambda n, _: n > 20, record=rec)
    lo, hi = _bounds(rec)
    if solver == "cheby":
        theta, ca, cb = _coefs(lo, hi, cap - t)
        r = b - A(u)
        p = r / theta
        u = u + p
        bb, err, est, n = float((b * b).sum()), None, 0, 0
        while t < cap:
            n += 1
            r = b - A(u)
            p = ca[n] * p + cb[n] * r if n < len(ca) else 0.0 * p   # past the table: zeros
            u = u + p
            if n == 1 or (n >= est and (t + 1) % 10 == 0):
                err = float((r * r).sum())
                if n == 1:
                    cn = math.sqrt(hi / lo)
                    g = (cn - 1.0) / (cn + 1.0)
                    est = round(math.log(2.220446049250313e-16 * bb / (4.0 * err)) / (2.0 * math.log(g)))
                if (math.sqrt(err) if case["dims"] == 3 else err) < eps:
                    break
            t += 1
        return u, u
    theta, ca, cb = _coefs(lo, hi, 10)
    halo_u = u
    r = b - A(u)
    while t < cap:
        w = A(p)
        alpha = rro / float((p * w).sum())
        u = u + alpha * p
        r = r - alpha * w
        sd = r / theta
        for i in range(10):
            r = r - A(sd)
            u = u + sd
            sd = ca[i] * sd + cb[i] * r
        rrn = float((r * r).sum())
        p = r + (rrn / rro) * p
        rro = rrn
        if (math.sqrt(rrn) if case["dims"] == 3 else rrn) < eps:
            break
        t += 1
    return u, halo_u


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed, dev)
    us = []
    for cells, shapes, eps in _problems(case, seed):
        rho, e0 = _paint(case["dims"], cells, shapes, dev)
        e = e0.clone()
        _reflect(rho, HALO)
        _reflect(e, HALO)
        e0 = e.clone()
        full = e * rho
        u, last = _solve(case, _Operator(rho, cells), _in(full).clone(), eps)
        if case["kind"] not in ("batch", "refine"):   # those leave the halo of u as cg_init made it
            _in(full).copy_(last)
            _reflect(full, 1)
        _in(full).copy_(u)
        us.append(full)
    if case["kind"] == "batch":
        return {"u": us}
    _in(e).copy_(u / _in(rho))
    _reflect(e, 1)
    out = {"u": us[0], "energy": e}
    if case.get("summary") or case["kind"] == "drivers":
        vol = 1.0
        for n in cells:
            vol *= DOMAIN / n
        m = vol * _in(rho)
        out["summary"] = [vol * m.numel(), float(m.sum()), float((m * _in(e0)).sum()), float((m * u).sum())]
    return out


def _exact_adjoint(case, seed, dev):
    cells, shapes, _ = _problems(case, seed)[0]
    rho, e = _paint(3, cells, shapes, dev)
    _reflect(rho, HALO)
    d = [DOMAIN / n for n in cells]
    vol = d[0] * d[1] * d[2]
    A = _Operator(rho, cells)
    r_in, e_in = _in(rho).clone(), _in(e).clone()
    us = [e_in * r_in]
    for _ in range(case["steps"]):
        us.append(_cg(A, us[-1], us[-1].clone(), 1e-32, 20000)[0])
    inside = torch.ones_like(r_in)
    for ax, n in enumerate(cells):
        c = (torch.arange(n, dtype=torch.float64, device=dev) + 0.5) * d[ax]
        shape = [1, 1, 1]
        shape[2 - ax] = -1
        inside = inside * ((c >= BOX[2 * ax]) & (c <= BOX[2 * ax + 1])).reshape(shape)
    j = float((vol * r_in * us[-1] * inside).sum())
    lam = [None] * (case["steps"] + 1)
    g = vol * r_in * inside
    for n in range(case["steps"], 0, -1):
        lam[n] = _cg(A, g, torch.zeros_like(g), 1e-26 * float((g * g).sum()), 20000)[0]
        g = lam[n]
    var = rho.clone().requires_grad_(True)
    op = _Operator(var, cells)
    s = (vol * _in(var) * us[-1] * inside).sum() + (lam[1] * e_in * _in(var)).sum()
    for n in range(1, case["steps"] + 1):   # lam . A u as the sum over faces of k (difference)(difference)
        for ax, k in enumerate(op.k):
            m = us[n].shape[ax]
            du = us[n].narrow(ax, 1, m - 1) - us[n].narrow(ax, 0, m - 1)
            dl = lam[n].narrow(ax, 1, m - 1) - lam[n].narrow(ax, 0, m - 1)
            s = s - (k * du * dl).sum()
    s.backward()
    grad = _in(var.grad) * r_in
    return {"J": j, "grad": grad.cpu().numpy()}
