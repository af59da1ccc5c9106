"""Performance cases of the framework: what its users have it do, through the public Python entry points.

A case is one of six kinds of work:

* ``flow``    steps of a resident single-phase solve, then the report (Error
              and Comput_Perm) and the rho/u fields, as the program does at
              every output interval; with ``state`` the populations too, as
              at a checkpoint;
* ``solve``   one whole permeability solve from a host mask: creation, the
              run to the stop test, the fields, and the end of the solver;
* ``batch``   many subsamples to the stop test in one node pool, with all
              of their fields;
* ``serve``   a burst of permeability requests through a running server;
* ``cg``      steps of a resident colour-gradient two-phase solve, then the
              report and its fields;
* ``solute``  steps of a D3Q7 or D3Q19 solute on a given velocity field, then
              the concentration.

Geometries are overlapping spheres or straight cylinders with the porosities,
radii, viscosities and forces of the benchmark configurations and of the
tests; all inputs follow from the seed.  The C ABI returns every field in
64-bit arrays; the fields and numbers of 32- and 16-bit solves are kept here
as what they hold, 32-bit values.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "jianhui-lbm_b200"))

import lbm_b200  # noqa: E402

CS2 = 1.0 / 3.0


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest calls: a coarse test geometry stepped a few steps
        # between reports, where launches and synchronisations count
        dict(name="flow_f32_small", kind="flow", precision="f32", nx=33, ny=31, nz=35, porosity=0.45, r0=3.0, r1=5.0,
             steps=20, force="x", faces=False, state=False),
        # the headline workload: 256^3, porosity 0.35, FP32, one output interval
        dict(name="flow_f32_large", kind="flow", precision="f32", nx=256, ny=256, nz=256, porosity=0.35, r0=4.0,
             r1=10.0, steps=500, force="x", faces=False, state=False),
        # half-precision storage on a ragged scan
        dict(name="flow_f16_ragged", kind="flow", precision="f16", nx=187, ny=201, nz=163, porosity=0.4, r0=4.0,
             r1=10.0, steps=300, force="x", faces=False, state=False),
        # the bit-exact FP64 solve up to a checkpoint (all populations)
        dict(name="flow_f64_checkpoint", kind="flow", precision="f64", nx=104, ny=96, nz=88, porosity=0.4, r0=6.0,
             r1=6.0, steps=200, force="x", faces=False, state=True),
        # a pressure-driven sample (constant-density x faces, no body force)
        dict(name="flow_f32_faces", kind="flow", precision="f32", nx=150, ny=121, nz=135, porosity=0.4, r0=4.0, r1=8.0,
             steps=200, force="none", faces=True, state=False),
        # one permeability solve of a small sample from its mask to its fields
        dict(name="solve_f32_64", kind="solve", precision="f32", nx=64, ny=64, nz=64, porosity=0.4, r0=6.0, r1=6.0,
             tol=1e-6, check=100, cap=6000),
        # subsamples of uneven size in one pool
        dict(name="batch_f32", kind="batch", precision="f32", count=8, lo=40, hi=96, plo=0.25, phi=0.5, r0=5.0, r1=5.0,
             tol=1e-5, check=100, cap=3000),
        # a burst of requests to a resident server
        dict(name="serve_f32", kind="serve", precision="f32", count=6, lo=32, hi=80, plo=0.2, phi=0.5, r0=3.0, r1=8.0,
             tol=1e-5, check=100, cap=3000),
        # the two-phase workload: 128^3 cylinders, porosity 0.6, saturation 0.5
        dict(name="cg_f32_128", kind="cg", precision="f32", nx=128, ny=128, nz=128, porosity=0.6, r0=3.0, r1=3.0,
             steps=300),
        # the bit-exact two-phase solve of a validation sample
        dict(name="cg_f64_ragged", kind="cg", precision="f64", nx=75, ny=64, nz=61, porosity=0.6, r0=3.0, r1=3.0,
             steps=100),
        # solute on the headline geometry's size, the seven-direction program
        dict(name="solute7_f32", kind="solute", precision="f32", lattice=7, nx=192, ny=192, nz=192, porosity=0.35,
             r0=4.0, r1=10.0, steps=400),
        # the nineteen-direction solute in FP64
        dict(name="solute19_f64", kind="solute", precision="f64", lattice=19, nx=111, ny=96, nz=130, porosity=0.4,
             r0=4.0, r1=8.0, steps=200),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["flow", "flow", "flow", "solve", "batch", "serve", "cg", "cg", "solute"])
    if kind in ("flow", "solve", "cg", "solute"):
        edge = {"flow": 230, "solve": 88, "cg": 128, "solute": 200}[kind]
        base = _log(rng, 24, edge)
        nx, ny, nz = (max(16, min(edge, base + rng.randint(-base // 6, base // 6))) for _ in range(3))
        c = dict(kind=kind, nx=nx, ny=ny, nz=nz, porosity=round(rng.uniform(0.3, 0.55), 3))
        c["r0"] = round(rng.uniform(3.0, 6.0), 2)
        c["r1"] = round(c["r0"] + rng.uniform(0.0, 4.0), 2)
    if kind == "flow":
        c["precision"] = rng.choice(["f32", "f32", "f32", "f16", "f64", "f64fast"])
        # node-updates within those of the largest listed case
        nodes = nx * ny * nz * c["porosity"]
        c["steps"] = max(1, min(_log(rng, 5, 800), int((1.4e9 if "64" not in c["precision"] else 4e8) / nodes)))
        c["faces"] = rng.random() < 0.25
        c["force"] = "none" if c["faces"] else rng.choice(["x", "xyz"])
        c["state"] = nodes < 4e5 and rng.random() < 0.4
    elif kind == "solve":
        c.update(precision=rng.choice(["f32", "f32", "f64fast"]), tol=rng.choice([1e-4, 1e-5]),
                 check=rng.choice([50, 100]), cap=3000)
    elif kind in ("batch", "serve"):
        lo = _log(rng, 24, 56)
        c = dict(kind=kind, precision=rng.choice(["f32", "f32", "f16"]), count=rng.randint(2, 10), lo=lo,
                 hi=min(96, lo + rng.randint(4, 48)), plo=0.25, phi=0.5, r0=3.0, r1=6.0, tol=rng.choice([1e-4, 1e-5]),
                 check=rng.choice([50, 100]), cap=1500)
    elif kind == "cg":
        c["precision"] = rng.choice(["f32", "f32", "f64"])
        c["porosity"] = round(rng.uniform(0.45, 0.7), 3)
        nodes = nx * ny * nz * c["porosity"]
        c["steps"] = max(1, min(_log(rng, 5, 400), int((3.8e8 if c["precision"] == "f32" else 6e7) / nodes)))
    else:
        c["precision"] = rng.choice(["f32", "f64"])
        c["lattice"] = rng.choice([7, 19])
        c["steps"] = max(1, min(_log(rng, 5, 600), int(9e8 / (nx * ny * nz * c["porosity"]))))
    return c


# ------------------------------------------------------------------- inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _solid_cells(dist, porosity):
    """uint8 mask of the cells nearest to the solids: as many as leave the
    given pore fraction (to a cell, so that every seed has as many pores)."""
    pores = max(1, int(round(porosity * dist.numel())))
    mask = torch.zeros(dist.numel(), dtype=torch.uint8, device=dist.device)
    mask[torch.sort(dist.reshape(-1), stable=True).indices[:dist.numel() - pores]] = 1
    return mask.reshape(dist.shape).cpu().numpy()


def _spheres(nx, ny, nz, porosity, r0, r1, seed):
    """[nz, ny, nx] uint8 mask of overlapping periodic spheres: as many as
    leave the given pore fraction on average, their surfaces then moved by
    the fraction of a cell that is missing."""
    rng = np.random.RandomState(seed)
    dev = _device()
    mean = 4.0 / 3.0 * math.pi * ((r1**4 - r0**4) / (4.0 * (r1 - r0)) if r1 > r0 else r0**3)
    n = max(1, int(round(-math.log(porosity) * nx * ny * nz / mean)))
    c = torch.from_numpy(rng.uniform(0, 1, (n, 3)) * np.array([nx, ny, nz])).to(dev)
    r = torch.from_numpy(rng.uniform(r0, r1, n) if r1 > r0 else np.full(n, float(r0))).to(dev)
    k = int(math.ceil(max(r0, r1))) + 2
    o = torch.arange(-k, k + 1, device=dev)
    off = torch.stack(torch.meshgrid(o, o, o, indexing="ij"), -1).reshape(-1, 3)
    ext = torch.tensor([nx, ny, nz], device=dev)
    dist = torch.full((nx * ny * nz,), 1e9, dtype=torch.float64, device=dev)
    for a in range(0, n, 1024):
        ca, ra = c[a:a + 1024, None, :], r[a:a + 1024, None]
        cell = torch.floor(ca).to(torch.int64) + off[None]
        d = ((cell.double() - ca) ** 2).sum(-1).sqrt() - ra
        w = cell % ext
        dist.scatter_reduce_(0, (w[..., 0] + nx * (w[..., 1] + ny * w[..., 2])).reshape(-1), d.reshape(-1), "amin")
    return _solid_cells(dist.reshape(nz, ny, nx), porosity)


def _cylinders(nx, ny, nz, porosity, radius, seed):
    """Straight cylinders of random position and direction until the pore
    fraction falls to the given one, which the last surfaces then meet."""
    rng = np.random.RandomState(seed)
    dev = _device()
    dist = torch.full((nz, ny, nx), 1e9, dtype=torch.float64, device=dev)
    while float((dist > radius * radius).double().mean()) > porosity:
        p = rng.uniform(0, 1, 3) * np.array([nx, ny, nz])
        v = rng.normal(size=3)
        v /= np.linalg.norm(v)
        d = []
        for size, q in ((nx, p[0]), (ny, p[1]), (nz, p[2])):
            x = torch.arange(size, device=dev, dtype=torch.float64) - q
            d.append(x - size * torch.round(x / size))
        dx, dy, dz = d[0][None, None, :], d[1][None, :, None], d[2][:, None, None]
        t = dx * v[0] + dy * v[1] + dz * v[2]
        dist = torch.minimum(dist, dx * dx + dy * dy + dz * dz - t * t)
    return _solid_cells(dist, porosity)


def _blobs(mask, seed):
    """+1 / -1 phase per pore (0 on solids): a thresholded sum of Gaussian
    blobs at a saturation of one half."""
    nz, ny, nx = mask.shape
    rng = np.random.RandomState(seed)
    dev = _device()
    sigma = max(nx, ny, nz) / 16.0
    field = torch.zeros((nz, ny, nx), dtype=torch.float64, device=dev)
    for _ in range(64):
        c = rng.uniform(0, 1, 3) * np.array([nx, ny, nz])
        s = rng.choice([-1.0, 1.0])
        e = []
        for size, q in ((nx, c[0]), (ny, c[1]), (nz, c[2])):
            x = torch.arange(size, device=dev, dtype=torch.float64) - q
            x = x - size * torch.round(x / size)
            e.append(torch.exp(-x * x / (2 * sigma * sigma)))
        field += s * e[2][:, None, None] * e[1][None, :, None] * e[0][None, None, :]
    pore = torch.from_numpy(mask == 0).to(dev)
    v, _ = torch.sort(field[pore])
    psi = torch.where(field > v[(v.numel() - 1) // 2], 1.0, -1.0).double()
    psi[~pore] = 0.0
    return psi.cpu().numpy()


def _fluid_cells(mask):
    """x, y, z of the pore cells in the reference's order (x fastest)."""
    nz, ny, nx = mask.shape
    c = np.flatnonzero(mask.reshape(-1) == 0)
    return c % nx, (c // nx) % ny, c // (nx * ny)


def _solute_inputs(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    mask = _spheres(nx, ny, nz, case["porosity"], case["r0"], case["r1"], seed)
    rng = np.random.RandomState(seed + 17)
    x, y, z = _fluid_cells(mask)
    ph = rng.uniform(0, 2 * math.pi, 6)
    ax, ay, az = 2 * math.pi * x / nx, 2 * math.pi * y / ny, 2 * math.pi * z / nz
    u = np.zeros((x.size + 1, 3))
    # a smooth creeping flow: a mean along x with recirculation
    u[1:, 0] = 2e-3 * (1.0 + 0.5 * np.sin(ay + ph[0]) * np.sin(az + ph[1]))
    u[1:, 1] = 1e-3 * np.sin(ax + ph[2]) * np.sin(az + ph[3])
    u[1:, 2] = 1e-3 * np.sin(ax + ph[4]) * np.sin(ay + ph[5])
    # a slug, one value per cell
    c0 = np.zeros(mask.shape)
    c0[:, :, nx // 8:nx // 2] = 1.0
    return mask, u, c0


def _flow_inputs(case, seed):
    mask = _spheres(case["nx"], case["ny"], case["nz"], case["porosity"], case["r0"], case["r1"], seed)
    g = {"x": (1e-6, 0.0, 0.0), "xyz": (1e-6, 4e-7, -3e-7), "none": (0.0, 0.0, 0.0)}[case.get("force", "x")]
    return mask, 0.1, g


# INPUT.dat face order xp, xn, yp, yn, zp, zn
_FACE_RHO = (0.9995, 1.0005)


def _packs(case, seed):
    """Cubes of uneven size: edges spread over the logarithm of their range,
    porosities and radii over theirs, in an order of their own."""
    rng = np.random.RandomState(seed)
    n, out = case["count"], []
    for i in range(n):
        t, w = (i + 0.5) / n, ((i * 5) % n + 0.5) / n
        e = int(round(case["lo"] * (case["hi"] / case["lo"]) ** ((i * 3 % n + 0.5) / n)))
        por, r = case["plo"] + (case["phi"] - case["plo"]) * t, case["r0"] + (case["r1"] - case["r0"]) * w
        out.append((_spheres(e, e, e, por, r, r, int(rng.randint(1 << 30))), 0.1, (1e-6, 0.0, 0.0)))
    return out


_CG = dict(nu_l=0.1, nu_g=0.1, psi_solid=0.70711, cap_a=1e-3, g=(1e-5, 0.0, 0.0), body_force_phase=-1)


def _cg_inputs(case, seed):
    mask = _cylinders(case["nx"], case["ny"], case["nz"], case["porosity"], case["r0"], seed)
    return mask, _blobs(mask, seed + 1)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "flow":
        mask, nu, g = _flow_inputs(case, seed)
        bc = None
        if case["faces"]:
            bc = dict(sub_bc=0, in_bc=1, pressure=(1, 1, 0, 0, 0, 0), rho=_FACE_RHO + (1.0,) * 4)
        s["solver"] = lbm_b200.SinglePhase(mask, nu, g=g, precision=case["precision"], bc=bc)
    elif kind == "solve":
        s["input"] = _flow_inputs(case, seed)
    elif kind == "batch":
        s["batch"] = lbm_b200.Batch(_packs(case, seed), precision=case["precision"])
    elif kind == "serve":
        s["packs"] = _packs(case, seed)
        s["server"] = lbm_b200.Server(capacity_nodes=4 * 1024 * 1024, precision=case["precision"], tol=case["tol"],
                                      check_every=case["check"], max_steps=case["cap"])
    elif kind == "cg":
        mask, psi = _cg_inputs(case, seed)
        s["solver"] = lbm_b200.ColourGradient(mask, psi, precision=case["precision"], **_CG)
    else:
        mask, u, c0 = _solute_inputs(case, seed)
        s["solver"] = lbm_b200.Solute(mask, c0, 0.01, u_nodes=u, precision=case["precision"],
                                      lattice=case["lattice"])
    return s


# --------------------------------------------------------------------- runs
def _keep(case, values):
    """An array of the solve's own precision."""
    a = torch.from_numpy(np.ascontiguousarray(values, dtype=np.float64))
    return a if case["precision"].startswith("f64") else a.float()


def _flow_numbers(case, d):
    return {"perm": _keep(case, d["perm"][0]), "mass": _keep(case, d["mass"]),
            "speeds": _keep(case, [d["u_ave"], d["u_max"], d["u_mean_speed"]])}


def _pool_numbers(case, res):
    return {k: _keep(case, [r["perm"][0] if k == "perm" else r[k] for r in res]) for k in ("perm", "u_ave", "mass")}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "flow":
        s = state["solver"]
        s.step(case["steps"])
        d = s.reduce()
        rho, u = s.fields()
        out = {"report": _flow_numbers(case, d), "rho": _keep(case, rho), "u": _keep(case, u)}
        if case["state"]:
            out["f"] = _keep(case, s.populations())
        return out
    if kind == "solve":
        mask, nu, g = state["input"]
        with lbm_b200.SinglePhase(mask, nu, g=g, precision=case["precision"]) as s:
            d = s.run_to_convergence(tol=case["tol"], check_every=case["check"], max_steps=case["cap"])
            rho, u = s.fields()
        return {"steps": d["step"], "report": _flow_numbers(case, d), "rho": _keep(case, rho),
                "u": _keep(case, u)}
    if kind == "batch":
        b = state["batch"]
        b.reset()
        res = b.run(tol=case["tol"], check_every=case["check"], max_steps=case["cap"])
        fields = [b.fields(i) for i in range(len(res))]
        return {"steps": np.array([r["steps"] for r in res]),
                "report": _pool_numbers(case, res),
                "rho": [_keep(case, f[0]) for f in fields], "u": [_keep(case, f[1]) for f in fields]}
    if kind == "serve":
        srv = state["server"]
        for mask, nu, g in state["packs"]:
            srv.submit(mask, nu, g)
        res = []
        while True:
            active, queued = srv.pump()
            res += srv.poll()
            if active == 0 and queued == 0 and len(res) == len(state["packs"]):
                break
        res.sort(key=lambda r: r["request_id"])
        return {"steps": np.array([r["steps"] for r in res]),
                "report": _pool_numbers(case, res)}
    if kind == "cg":
        s = state["solver"]
        s.step(case["steps"])
        d = s.reduce()
        f = s.fields()
        out = {k: _keep(case, f[k]) for k in ("rho", "u", "psi", "rho_r", "rho_b")}
        out["report"] = {"saturation": _keep(case, d["saturation"]), "mass": _keep(case, d["mass"]),
                         "speeds": _keep(case, [d["u_max"], d["u_mean_speed"]])}
        return out
    s = state["solver"]
    s.step(case["steps"])
    return _keep(case, s.concentration())


# --------------------------------------------------------------------- work
def work(case):
    """Populations read and written once a step, the neighbour bits of the
    geometry (one per direction), and the fields that the call returns."""
    s = {"f64": 8, "f64fast": 8, "f32": 4, "f16": 2}[case["precision"]]
    kind = case["kind"]
    if kind in ("batch", "serve"):
        edge = math.sqrt(case["lo"] * case["hi"])
        n = case["count"] * edge**3 * 0.5 * (case["plo"] + case["phi"])
        steps = min(case["cap"], 1000)
        return {"bytes": n * (steps * (38 * s + 18 / 8) + (32 if kind == "batch" else 0)), "flops": n * steps * 500}
    n = case["nx"] * case["ny"] * case["nz"] * case["porosity"]
    if kind == "flow":
        return {"bytes": n * (case["steps"] * (38 * s + 18 / 8) + 32 + (152 if case["state"] else 0)),
                "flops": n * case["steps"] * 500}
    if kind == "solve":
        steps = min(case["cap"], 1000)
        return {"bytes": n * (steps * (38 * s + 18 / 8) + 32), "flops": n * steps * 500}
    if kind == "cg":
        return {"bytes": n * (case["steps"] * (38 * s + 4 * s + 18 / 8) + 56), "flops": n * case["steps"] * 1500}
    q = 6 if case["lattice"] == 7 else 19
    return {"bytes": n * (case["steps"] * (2 * q * s + 3 * s + q / 8) + 8), "flops": n * case["steps"] * 8 * q}


# ------------------------------------------------- the same in 64 bits, plainly
_E = np.array([(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, 1, 0),
               (1, -1, 0), (-1, -1, 0), (0, 1, 1), (0, -1, 1), (0, 1, -1), (0, -1, -1), (1, 0, 1), (-1, 0, 1),
               (1, 0, -1), (-1, 0, -1)])
_W = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12)
_OPP = [int(np.flatnonzero((_E == -e).all(1))[0]) for e in _E]


def _pull_table(masks, q_count=19):
    """[q, n] flat sources of the streaming step over all masks' pores, with
    halfway bounce-back, and [q, n] whether the cell at x - e_q is a pore."""
    dev = _device()
    total = sum(int((m == 0).sum()) for m in masks)
    src = torch.empty((q_count, total), dtype=torch.int64, device=dev)
    flu = torch.empty((q_count, total), dtype=torch.bool, device=dev)
    at = 0
    for m in masks:
        pore = torch.from_numpy(m == 0).to(dev)
        n = int(pore.sum())
        ids = torch.full(pore.shape, -1, dtype=torch.int64, device=dev)
        ids[pore] = torch.arange(at, at + n, device=dev)
        own = torch.arange(at, at + n, device=dev)
        for q in range(q_count):
            ex, ey, ez = (int(v) for v in _E[q])
            nb = torch.roll(ids, shifts=(ez, ey, ex), dims=(0, 1, 2))[pore]
            src[q, at:at + n] = torch.where(nb >= 0, q * total + nb, _OPP[q] * total + own)
            flu[q, at:at + n] = nb >= 0
        at += n
    return src, flu


def _sp_moments():
    M = np.zeros((19, 19))
    for q, (x, y, z) in enumerate(_E):
        c = x * x + y * y + z * z
        M[:, q] = [1, 19 * c - 30, (21 * c * c - 53 * c + 24) / 2, x, (5 * c - 9) * x, y, (5 * c - 9) * y, z,
                   (5 * c - 9) * z, 3 * x * x - c, (3 * c - 5) * (3 * x * x - c), y * y - z * z,
                   (3 * c - 5) * (y * y - z * z), x * y, y * z, x * z, (y * y - z * z) * x, (z * z - x * x) * y,
                   (x * x - y * y) * z]
    return M


class _Flow64:
    """D3Q19 MRT with Guo's force on the pores of one or more masks."""

    def __init__(self, masks, nu, g, faces=None):
        dev = _device()
        self.src, _ = _pull_table(masks)
        n = self.src.shape[1]
        sv = 1.0 / (3.0 * nu + 0.5)
        so = 8 * (2 - sv) / (8 - sv)
        S = np.array([0, sv, sv, 0, so, 0, so, 0, so, sv, sv, sv, sv, sv, sv, sv, so, so, so])
        M = _sp_moments()
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
        self.K = t(np.linalg.inv(M) @ np.diag(S) @ M)
        self.E, self.W = t(_E), t(_W)
        self.g = t(np.array(g, dtype=np.float64))
        self.eg = self.E @ self.g
        self.rho = torch.ones(n, dtype=torch.float64, device=dev)
        self.u = torch.zeros((3, n), dtype=torch.float64, device=dev)
        self.f = (self.W[:, None] * self.rho[None]).contiguous()
        self.face = faces or []  # [(index of the face's nodes, density)]

    def step(self):
        eu = self.E @ self.u
        uu = (self.u * self.u).sum(0)
        h = self.W[:, None] * (3.0 * (self.eg[:, None] - (self.g @ self.u)[None]) + 9.0 * eu * self.eg[:, None])
        d = self.f + 0.5 * h
        d -= (self.W[:, None] * self.rho[None]) * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * uu[None])
        self.f += h
        self.f -= self.K @ d
        self.f = self.f.view(-1)[self.src]
        for at, rho in self.face:
            self.f[:, at] = self.W[:, None] * rho
        self.rho = self.f.sum(0)
        self.u = (self.E.T @ self.f + 0.5 * self.g[:, None]) / self.rho[None]

    def rows(self, a=0, b=None):
        """rho [n + 1] and u [n + 1, 3] with the unused row 0."""
        rho, u = self.rho[a:b], self.u[:, a:b]
        z = torch.zeros(1, dtype=torch.float64, device=rho.device)
        return torch.cat([z, rho]), torch.cat([z.expand(3)[None], u.T])

    def report(self, cells, drive, nu, a=0, b=None):
        u, n = self.u[:, a:b], self.u[:, a:b].shape[1]
        q = u.sum(1)
        speed = (u * u).sum(0).sqrt()
        t = lambda v: torch.as_tensor(v, dtype=torch.float64)  # noqa: E731
        return {"perm": t(float(q[0]) / cells * nu / drive), "mass": t(float(self.rho[a:b].sum())),
                "speeds": t([float((q / n).norm()), float(speed[:-1].max()), float(speed[:-1].sum()) / n])}


def _to_stop(masks, nu, g, case):
    """Every mask's solve to its own stop test: [(steps, report, rho, u)]."""
    flow = _Flow64(masks, nu, g)
    n = [int((m == 0).sum()) for m in masks]
    at = np.concatenate([[0], np.cumsum(n)])
    prev, out = [None] * len(masks), [None] * len(masks)
    steps = 0
    while any(o is None for o in out) and steps < case["cap"]:
        k = min(case["check"], case["cap"] - steps)
        for _ in range(k):
            flow.step()
        steps += k
        for i, m in enumerate(masks):
            if out[i] is not None:
                continue
            rep = flow.report(m.size, g[0], nu, int(at[i]), int(at[i + 1]))
            ave = float(rep["speeds"][0])
            if (prev[i] is not None and abs((prev[i] - ave) / prev[i]) < case["tol"]) or steps >= case["cap"]:
                out[i] = (steps, rep) + tuple(x.clone() for x in flow.rows(int(at[i]), int(at[i + 1])))
            prev[i] = ave
    return out


# colour-gradient direction order and basis
_EC = np.array([(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0),
                (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, -1, -1),
                (0, 1, -1), (0, -1, 1)])


class _TwoPhase64:
    """The colour-gradient model, directions in its own order."""

    def __init__(self, mask, psi):
        dev = _device()
        src, flu = _pull_table([mask])
        n = src.shape[1]
        rows = [int(np.flatnonzero((_E == e).all(1))[0]) for e in _EC]  # flow direction of each of this model's
        back = torch.tensor([rows.index(q) for q in range(19)], device=dev)
        self.src = torch.stack([back[src[r] // n] * n + src[r] % n for r in rows])
        # neighbour x + e_t: the source of the opposite direction's pull
        self.fluid = torch.stack([flu[_OPP[r]] for r in rows])
        self.nb = torch.stack([src[_OPP[r]] % n for r in rows])
        self.wall = (~self.fluid).any(0)
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
        M = np.zeros((19, 19))
        for q, (x, y, z) in enumerate(_EC):
            c = x * x + y * y + z * z
            M[:, q] = [1, c - 1, 3 * c * c - 6 * c + 1, x, (3 * c - 5) * x, y, (3 * c - 5) * y, z, (3 * c - 5) * z,
                       3 * x * x - c, (2 * c - 3) * (3 * x * x - c), y * y - z * z, (2 * c - 3) * (y * y - z * z),
                       x * y, y * z, x * z, (y * y - z * z) * x, (z * z - x * x) * y, (x * x - y * y) * z]
        self.M, self.MI, self.E, self.W = t(M), t(np.linalg.inv(M)), t(_EC), t(_W)
        p = torch.from_numpy(psi.astype(np.float32).astype(np.float64)[mask == 0]).to(dev)
        self.psi, self.rho = p, torch.ones_like(p)
        self.rr = (p + 1.0) / 2
        self.rb = 1.0 - self.rr
        self.u = torch.zeros((3, n), dtype=torch.float64, device=dev)
        self.f = self.MI[:, :1] @ self.rho[None]
        self.g = t(np.array(_CG["g"]))
        self.eg = self.E @ self.g

    def step(self):
        W, E, u, psi = self.W[:, None], self.E, self.u, self.psi
        ps = torch.where(self.fluid, psi[self.nb], torch.full_like(psi, _CG["psi_solid"])[None])
        C = 3.0 * (E.T @ (W * ps))
        C = C * (~(((self.rr - self.rb).abs() >= 0.9) & self.wall)).double()
        cc = (C * C).sum(0).sqrt()
        nrm = torch.where(cc > 0, C / torch.where(cc > 0, cc, torch.ones_like(cc)), torch.zeros_like(C))
        eu = E @ u
        uu = (u * u).sum(0)
        guo = W * (3.0 * (self.eg[:, None] - (self.g @ u)[None]) + 9.0 * eu * self.eg[:, None])
        guo = guo * (psi <= -0.99).double()  # body force on the non-wetting phase alone
        ux, uy, uz = u
        a, b, c = nrm
        ck = 0.5 * _CG["cap_a"] * cc
        meq = torch.zeros_like(self.f)
        meq[0], meq[3], meq[5], meq[7] = self.rho, ux, uy, uz
        meq[1] = uu + 2.0 * ck
        meq[9] = 2 * ux * ux - uy * uy - uz * uz + ck * (2 * a * a - b * b - c * c)
        meq[11] = uy * uy - uz * uz + ck * (b * b - c * c)
        meq[13] = ux * uy + ck * a * b
        meq[14] = uy * uz + ck * b * c
        meq[15] = ux * uz + ck * a * c
        wl, wg, dl = 1.0 / (3 * _CG["nu_l"] + 0.5), 1.0 / (3 * _CG["nu_g"] + 0.5), 0.1
        w0 = 2 * wl * wg / (wl + wg)
        l1, g1 = 2 * (wl - w0) / dl, 2 * (w0 - wg) / dl
        sv = torch.where(psi > 0, torch.where(psi > dl, wl, w0 + l1 * psi - l1 / (2 * dl) * psi * psi),
                         torch.where(psi < -dl, wg, w0 + g1 * psi + g1 / (2 * dl) * psi * psi))
        so = 8 * (2 - sv) / (8 - sv)
        m, fh = self.M @ self.f, self.M @ guo
        z = torch.zeros_like(sv)
        S = torch.stack([z, sv, sv, z, so, z, so, z, so] + [sv] * 7 + [so] * 3)
        self.f = (self.MI @ (m - S * (m - meq) + (1 - 0.5 * S) * fh)).view(-1)[self.src]
        eq = W * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * uu[None])
        gr, gb = self.rr[None] * eq, self.rb[None] * eq
        cp = torch.minimum(torch.minimum(gr[1::2], gr[2::2]), torch.minimum(gb[1::2], gb[2::2])) * (E[1::2] @ nrm)
        gr[1::2] += cp
        gr[2::2] -= cp
        gb[1::2] -= cp
        gb[2::2] += cp
        self.rr, self.rb = gr.view(-1)[self.src].sum(0), gb.view(-1)[self.src].sum(0)
        self.rho = self.f.sum(0)
        self.u = (E.T @ self.f + 0.5 * self.g[:, None]) / self.rho[None]
        self.psi = (self.rr - self.rb) / (self.rr + self.rb)


def _solute64(case, seed):
    mask, u, c0 = _solute_inputs(case, seed)
    dev = _device()
    q0, q1 = (1, 7) if case["lattice"] == 7 else (0, 19)
    src, _ = _pull_table([mask], q1)
    n = src.shape[1]
    src = src[q0:] - q0 * n
    t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
    E, u, c = t(_E[q0:q1]), t(u[1:].T.copy()), t(c0[mask == 0])
    W = torch.full((6,), 1.0 / 6.0, dtype=torch.float64, device=dev) if q0 else t(_W)
    eu = E @ u
    k = W[:, None] * (1.0 + 3.0 * eu) if q0 else W[:, None] * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * (u * u).sum(0)[None])
    tau = 3.0 * 0.01 + 0.5
    # the program sets g before it loads the velocity: the equilibrium at rest
    f = (W[:, None] * c[None]).contiguous()
    for _ in range(case["steps"]):
        f = (f - (f - k * c[None]) / tau).view(-1)[src]
        c = f.sum(0)
    return torch.cat([torch.zeros(1, dtype=torch.float64, device=dev), c])


def exact(case, seed):
    kind = case["kind"]
    t = lambda v: torch.as_tensor(v, dtype=torch.float64)  # noqa: E731
    if kind == "flow":
        mask, nu, g = _flow_inputs(case, seed)
        faces, drive = None, g[0]
        if case["faces"]:
            x = torch.from_numpy(_fluid_cells(mask)[0]).to(_device())
            faces = [(torch.nonzero(x == case["nx"] - 1)[:, 0], _FACE_RHO[0]),
                     (torch.nonzero(x == 0)[:, 0], _FACE_RHO[1])]
            drive = abs(_FACE_RHO[0] - _FACE_RHO[1]) * CS2 / case["nx"]
        flow = _Flow64([mask], nu, g, faces)
        for _ in range(case["steps"]):
            flow.step()
        rho, u = flow.rows()
        out = {"report": flow.report(mask.size, drive, nu), "rho": rho, "u": u}
        if case["state"]:
            out["f"] = torch.cat([torch.zeros((1, 19), dtype=torch.float64, device=rho.device), flow.f.T])
        return out
    if kind == "solve":
        mask, nu, g = _flow_inputs(case, seed)
        steps, rep, rho, u = _to_stop([mask], nu, g, case)[0]
        return {"steps": None, "report": rep, "rho": rho, "u": u}
    if kind in ("batch", "serve"):
        packs = _packs(case, seed)
        res = _to_stop([p[0] for p in packs], packs[0][1], packs[0][2], case)
        out = {"steps": None, "report": {"perm": t([float(r[1]["perm"]) for r in res]), "mass": t([float(r[1]["mass"]) for r in res]),
                                         "u_ave": t([float(r[1]["speeds"][0]) for r in res])}}
        if kind == "batch":
            out.update(rho=[r[2] for r in res], u=[r[3] for r in res])
        return out
    if kind == "cg":
        mask, psi = _cg_inputs(case, seed)
        s = _TwoPhase64(mask, psi)
        for _ in range(case["steps"]):
            s.step()
        z = torch.zeros(1, dtype=torch.float64, device=s.psi.device)
        row = lambda v: torch.cat([z, v])  # noqa: E731
        speed = (s.u * s.u).sum(0).sqrt()
        rep = {"saturation": t(float((s.psi >= 0).double().mean())), "mass": t(float(s.rho.sum())),
               "speeds": t([float(speed.max()), float(speed.sum()) / mask.size])}
        return {"rho": row(s.rho), "u": torch.cat([z.expand(3)[None], s.u.T]), "psi": row(s.psi),
                "rho_r": row(s.rr), "rho_b": row(s.rb), "report": rep}
    return _solute64(case, seed)
