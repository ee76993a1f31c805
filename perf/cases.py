"""Timed workloads of the library: what its users run, over the sizes they run it at.

Five kinds of case, each through the public Python entry points:

* ``batch``: many independent Dirichlet Poisson problems in one call
  (``BatchPoisson.solve_device``), FP64 and FP32-inner / FP64-outer.
* ``plane``: a run of the 2D drivers (periodic layer, oblique layer, rotating annulus):
  the start state loaded, a few time steps, the fields read back.
* ``meridian``: the same for the axisymmetric annulus, on its uniform and its
  tanh-stretched grid.
* ``annulus3d``: the same for the 3D rotating annulus.
* ``sweep``: requests of a parameter sweep served together (``GangServer``).

A run of a driver starts from its start state in every pass, so that each pass does the
same steps.  The fields, Nusselt numbers and sweep counts all come back.
"""
import math

import numpy as np
import torch

from codesthesis_dir_gb300 import initial, lib, serve
from codesthesis_dir_gb300.axi import AXI, stretched_grid
from codesthesis_dir_gb300.batch import BatchPoisson
from codesthesis_dir_gb300.prb import PRB
from codesthesis_dir_gb300.r3d import R3D

BATCH_PRECISION = {"fp64": lib.BATCH_FP64, "mixed": lib.BATCH_MIXED_F64OUTER, "pairs": lib.BATCH_MIXED}
PRECISION = {"fp64": lib.PRB_FP64, "mixed": lib.PRB_MIXED}
ORDER = {"lex": lib.SMOOTHER_LEX, "zebra": lib.SMOOTHER_ZEBRA}
VARIANT = {"layer": lib.PRB_LAYER, "oblique": lib.PRB_OBLIQUE, "annulus": lib.PRB_ANNULUS}


def _batch(nprob, sizes, precision, inner):
    return {"kind": "batch", "nprob": nprob, "sizes": sizes, "precision": precision, "inner": inner}


def _plane(variant, nr, np_, order, precision, tolcon, steps):
    return {"kind": "plane", "variant": variant, "nr": nr, "np": np_, "order": order, "precision": precision,
            "tolcon": tolcon, "steps": steps}


def _meridian(nr, nz, stretch, order, precision, tolcon, steps):
    return {"kind": "meridian", "nr": nr, "nz": nz, "stretch": stretch, "order": order, "precision": precision,
            "tolcon": tolcon, "steps": steps}


def _annulus3d(nr, nz, np_, order, precision, steps):
    return {"kind": "annulus3d", "nr": nr, "nz": nz, "np": np_, "order": order, "precision": precision,
            "steps": steps}


def _sweep(requests, largest, precision, lo, hi):
    return {"kind": "sweep", "requests": requests, "largest": largest, "precision": precision, "lo": lo, "hi": hi}


def listed():
    return [
        # a handful of small problems in one call: a caller's single solves, bound by launches and latency
        dict(_batch(8, "17,33,65", "mixed", 1), name="batch_small_mixed"),
        # the batched benchmark: 256 uneven problems, FP32 cycles inside FP64 defect correction
        dict(_batch(256, "65,129,257,513", "mixed", 3), name="batch_256_mixed"),
        # the same solver in plain FP64 on a middling batch
        dict(_batch(48, "65,129,257", "fp64", 1), name="batch_48_fp64"),
        # the drop-in path: the reference's own line order and tolerance, FP64, a small layer
        dict(_plane("layer", 32, 64, "lex", "fp64", 2e-6, 2), name="layer_lex_fp64"),
        # the 129 x 65 benchmark layer, plain FP64, two-colour lines
        dict(_plane("layer", 64, 128, "zebra", "fp64", 1e-10, 4), name="layer_fp64"),
        # the same layer with mixed-precision velocity solves
        dict(_plane("layer", 64, 128, "zebra", "mixed", 1e-10, 4), name="layer_mixed"),
        # the rotating annulus at the size of the deck it ships with
        dict(_plane("annulus", 272, 1200, "zebra", "mixed", 1e-5, 1), name="annulus_mixed"),
        # the axisymmetric annulus at the reference's largest uniform grid, plain FP64
        dict(_meridian(128, 128, 0.0, "zebra", "fp64", 1e-6, 4), name="meridian_fp64"),
        # the 257 x 257 stretched annulus benchmark, mixed precision
        dict(_meridian(256, 256, 1.5, "zebra", "mixed", 1e-9, 3), name="meridian_stretched_mixed"),
        # the 3D annulus at half its benchmark's grid in each direction, plain FP64
        dict(_annulus3d(32, 32, 64, "zebra", "fp64", 1), name="annulus3d_fp64"),
        # the 3D annulus benchmark, mixed precision
        dict(_annulus3d(64, 64, 128, "zebra", "mixed", 2), name="annulus3d_mixed"),
        # a parameter sweep of layers and annuli of several grids, served together
        dict(_sweep(16, 128, "mixed", 16, 32), name="sweep_mixed"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _times(rng, unit, lo, hi):
    """A multiple of `unit` in [lo, hi], even over the logarithm."""
    return unit * max(1, min(hi // unit, round(_log(rng, lo, hi) / unit)))


def draw(rng):
    kind = rng.choice(["batch", "batch", "plane", "plane", "meridian", "meridian", "annulus3d", "sweep"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "batch":
        precision = rng.choice(["fp64", "mixed", "mixed", "pairs"])
        sizes = rng.choice(["17,33,65", "33,129", "65,129,257", "65,129,257,513", "129,257", "257,513", "9,65,257"])
        inner = 1 if precision == "fp64" else rng.choice([1, 2, 3, 4])
        return _batch(round(_log(rng, 3, 96 if precision == "fp64" else 240)), sizes, precision, inner)
    if kind == "plane":
        variant = rng.choice(["layer", "layer", "oblique", "annulus"])
        order = rng.choice(["zebra", "zebra", "zebra", "lex"])
        nr = _times(rng, 8, 16, 32 if order == "lex" else 128)
        np_ = 16 * max(1, round(nr * rng.uniform(1.6, 2.4) / 16))
        return _plane(variant, nr, np_, order, precision, rng.choice([2e-6, 1e-7]), rng.choice([1, 2, 3]))
    if kind == "meridian":
        stretch = rng.choice([0.0, 1.0, 1.5])
        nr = _times(rng, 16, 32, 256)
        nz = nr if rng.random() < 0.5 else min(256, 16 * max(2, round(nr * rng.uniform(0.8, 1.25) / 16)))
        return _meridian(nr, nz, stretch, "zebra", precision, 1e-6, rng.choice([1, 2, 3]))
    if kind == "annulus3d":
        nr = _times(rng, 8, 16, 64 if precision == "mixed" else 32)
        nz = nr if rng.random() < 0.5 else _times(rng, 8, 16, 64 if precision == "mixed" else 32)
        np_ = 16 * max(2, min(8, round(2 * nr * rng.uniform(0.7, 1.0) / 16)))
        return _annulus3d(nr, nz, np_, "zebra", precision, 1)
    return _sweep(rng.randint(2, 24), rng.choice([64, 128]), precision, rng.randint(4, 12), rng.randint(13, 28))


# -- inputs --------------------------------------------------------------------------------------------------------


def _sizes(case, seed):
    choice = [int(s) for s in case["sizes"].split(",")]
    # every size of the mix occurs; the rest are drawn
    rng = np.random.default_rng(7)
    n = np.concatenate([choice, rng.choice(choice, size=max(0, case["nprob"] - len(choice)))])[: case["nprob"]]
    return n.astype(np.int32)


def _right_hand_sides(sizes, seed):
    """Zero-mean, unit-variance Gaussian random fields with squared-exponential correlation of
    length 0.05 of the domain, zero on the boundary, packed row-major."""
    gen = torch.Generator(device="cuda").manual_seed(1000 + seed)
    out = [None] * len(sizes)
    for n in sorted(set(int(s) for s in sizes)):
        at = [p for p, s in enumerate(sizes) if s == n]
        w = torch.randn((len(at), n, n), dtype=torch.float64, device="cuda", generator=gen)
        k = torch.fft.fftfreq(n, d=1.0 / (n - 1), dtype=torch.float64, device="cuda")
        filt = torch.exp(-((2 * math.pi) ** 2) * (k[:, None] ** 2 + k[None, :] ** 2) * 0.05 ** 2 / 4.0)
        g = torch.fft.ifft2(torch.fft.fft2(w) * filt).real
        g = (g - g.mean(dim=(1, 2), keepdim=True)) / g.std(dim=(1, 2), keepdim=True)
        g[:, 0, :] = g[:, -1, :] = g[:, :, 0] = g[:, :, -1] = 0.0
        for j, p in enumerate(at):
            out[p] = -g[j].reshape(-1)
    return torch.cat(out)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        sizes = _sizes(case, seed)
        f = _right_hand_sides(sizes, seed)
        solver = BatchPoisson(sizes, precision=BATCH_PRECISION[case["precision"]], inner=case["inner"])
        return {"kind": kind, "solver": solver, "f": f, "psi": torch.zeros_like(f)}
    if kind == "plane":
        nr, np_, variant = case["nr"], case["np"], VARIANT[case["variant"]]
        par = dict(tolcon=case["tolcon"], smoother=ORDER[case["order"]], precision=PRECISION[case["precision"]],
                   variant=variant)
        if case["variant"] == "annulus":
            r0, rmax = 0.5, 1.0
            g = PRB(nr, np_, dt=2e-8, r0=r0, rmax=rmax, Ra=8e8, Pr=0.71, Re=1.06148e5, **par)
        else:
            r0, rmax = 0.0, 1.0
            g = PRB(nr, np_, dt=1e-5, r0=r0, rmax=rmax, xx=2.0, Ra=1e5, Pr=1.0, **par)
        fields = initial.initial_fields(nr, np_, r0, rmax, variant, 1, seed, 1e-3)
        return {"kind": kind, "run": g, "fields": fields, "steps": case["steps"], "out": ("vel", "uel", "C", "th")}
    if kind == "meridian":
        nr, nz = case["nr"], case["nz"]
        grid = stretched_grid(nr, nz, 0.5, 1.0, 0.5, case["stretch"]) if case["stretch"] else None
        big = max(nr, nz) > 128
        g = AXI(nr, nz, dt=2e-7 if big else 1e-6, r0=0.5, rmax=1.0, zmax=0.5, Ra=1e8 if big else 1e6,
                Re=math.sqrt(1e5) / 2.0, Pr=1.0, tolcon=case["tolcon"], smoother=ORDER[case["order"]],
                precision=PRECISION[case["precision"]], grid=grid)
        fields = serve.axi_initial(nr, nz, 0.5, 1.0, seed, 1e-4, r=None if grid is None else grid.r[1])
        return {"kind": kind, "run": g, "fields": fields, "steps": case["steps"],
                "out": ("phi", "omeg", "vel", "theta")}
    if kind == "annulus3d":
        nr, nz, np_ = case["nr"], case["nz"], case["np"]
        g = R3D(nr, nz, np_, dt=4e-6, r0=0.5, rmax=1.0, zmax=0.5, Ra=1e6, Re=500.0, Pr=7.0,
                smoother=ORDER[case["order"]], precision=PRECISION[case["precision"]])
        fields = initial.r3d_initial_fields(nr, nz, np_, 0.5, 1.0, 3, 1e-3, noise=1e-5, seed=seed)
        return {"kind": kind, "run": g, "fields": fields, "steps": case["steps"],
                "out": ("wel", "vel", "uel", "A", "B", "C", "th")}
    return {"kind": kind, "requests": _requests(case, seed), "precision": PRECISION[case["precision"]]}


def _requests(case, seed):
    grids = [g for g in serve.SWEEP_GRIDS if g[0] <= case["largest"]]
    out = serve.sweep_requests(n=case["requests"], rate=50.0, seed=seed, steps=(case["lo"], case["hi"]), grids=grids)
    fixed = serve.sweep_requests(n=case["requests"], rate=50.0, seed=11, steps=(case["lo"], case["hi"]), grids=grids)
    for q, p in zip(out, fixed):
        # the mix of kinds, grids and lengths belongs to the case, the physics and the start to the seed;
        # all requests are there at the start
        q.kind, q.nx, q.nz, q.steps, q.Ta, q.arrival = p.kind, p.nx, p.nz, p.steps, p.Ta, 0.0
    return out


# -- one pass ------------------------------------------------------------------------------------------------------


def run(state):
    kind = state["kind"]
    if kind == "batch":
        f, psi = state["f"], state["psi"]
        status, cycles, relres = state["solver"].solve_device(f.data_ptr(), psi.data_ptr(),
                                                              torch.cuda.current_stream().cuda_stream)
        return {"psi": psi, "cycles": cycles, "status": status}
    if kind == "sweep":
        results = serve.GangServer(keep_fields=True, precision=state["precision"]).run(state["requests"])
        return {"nu": np.concatenate([np.ravel(r.nu) for r in results]),
                "steps": np.array([r.steps_done for r in results]),
                "status": np.array([r.status for r in results]),
                "fields": [np.concatenate([np.ravel(r.fields[n]) for n in sorted(r.fields)]) for r in results]}
    g = state["run"]
    for name, a in state["fields"].items():
        g.set(name, a)
    g.kt = 0
    nu, sweeps = g.step(state["steps"])
    return {"nu": nu, "sweeps": sweeps, "fields": {n: g.get(n) for n in state["out"]}}


# -- what a pass cannot do without ---------------------------------------------------------------------------------


def work(case):
    """Bytes: the inputs read once, the outputs written once.  Operations: one multigrid cycle per
    decade of residual for a solve (about 60 operations a point and cycle in 2D, 110 in 3D), and
    about 200 (2D) or 500 (3D) a point and step for the transport."""
    kind = case["kind"]
    if kind == "batch":
        points = float(sum(int(n) ** 2 for n in _sizes(case, 0)))
        return {"bytes": 16.0 * points, "flops": 10 * 60.0 * points}
    if kind == "plane":
        points = float(case["nr"] * case["np"])
        return {"bytes": 8.0 * points * (8 + 4), "flops": case["steps"] * points * (200 + 2 * 5 * 60)}
    if kind == "meridian":
        points = float(case["nr"] * case["nz"])
        return {"bytes": 8.0 * points * (7 + 4), "flops": case["steps"] * points * (200 + 5 * 60)}
    if kind == "annulus3d":
        points = float(case["nr"] * case["nz"] * case["np"])
        return {"bytes": 8.0 * points * (14 + 7), "flops": case["steps"] * points * (500 + 3 * 5 * 110)}
    reqs = _requests(case, 0)
    return {"bytes": 8.0 * sum(q.nx * q.nz for q in reqs) * 12,
            "flops": float(sum(q.steps * q.nx * q.nz for q in reqs)) * (200 + 2 * 5 * 60)}


# -- in 64 bits, without the library -------------------------------------------------------------------------------


def exact(case, seed):
    """The batched problems' discrete solutions by sine transforms.  The drivers' runs have no
    short restatement: their steps hold iterative solves stopped at a tolerance."""
    if case["kind"] != "batch":
        return None
    sizes = _sizes(case, seed)
    f = _right_hand_sides(sizes, seed)
    off = np.concatenate([[0], np.cumsum(sizes.astype(np.int64) ** 2)])
    psi = torch.zeros_like(f)
    for n in sorted(set(int(s) for s in sizes)):
        m = n - 2
        i = torch.arange(1, m + 1, dtype=torch.float64, device="cuda")
        s = torch.sin(math.pi * ((i[:, None] * i[None, :]) % (2 * (n - 1))) / (n - 1)) * math.sqrt(2.0 / (n - 1))
        lam = -4.0 * (n - 1) ** 2 * torch.sin(math.pi * i / (2.0 * (n - 1))) ** 2
        at = [p for p, q in enumerate(sizes) if q == n]
        g = torch.stack([f[off[p]:off[p + 1]].reshape(n, n)[1:-1, 1:-1] for p in at])
        u = s @ ((s @ g @ s) / (lam[:, None] + lam[None, :])) @ s
        for j, p in enumerate(at):
            psi[off[p]:off[p + 1]].reshape(n, n)[1:-1, 1:-1] = u[j]
    return {"psi": psi, "cycles": None, "status": None}
