"""Workloads by which the transport engine's speed is followed.

Each case is one thing a user's program has the engine do, through the public calls of
``moquimc_gb300`` (capi.Context, dij, beamline) or of the C ABI: transport one spot, many spots one
call each, a phantom, a whole plan with its statistics, robust scenarios, masked LET scoring, a
beamline in front of a phantom; score and build a Dij matrix; take an optimisation step on it;
convert a CT.  ``listed()`` names twelve of them with the sizes the package's workloads, tests and
benchmark use (scaled so that a pass stays below a second), and ``draw()`` gives more from the same
ranges.

Every transport pass clears the tallies, transports, and copies each tally to a buffer of the
caller's, as a planning program does for each dose it asks for.
"""
import ctypes as C
import math

import numpy as np
import torch

from moquimc_gb300 import beamline, capi, dij
from moquimc_gb300 import phantom as ph

DEV = "cuda"
FLOPS_PER_STEP = 600      # FP32 operations of one condensed-history voxel step, random numbers included

# grids: voxels, pitch in mm, centre in mm
GRIDS = {
    "water": ((200, 200, 350), (0.5, 0.5, 1.0), (0.0, 0.0, -175.0)),     # the phantom example
    "slab": ((256, 256, 256), (1.0, 1.0, 1.0), (0.0, 0.0, -128.0)),      # water with a lung and a bone slab
    "box": ((100, 100, 200), (1.0, 1.0, 1.0), (0.0, 0.0, -100.0)),       # the beamline phantom
    "dose_ct": ((256, 256, 200), (1.96, 1.96, 2.0), (0.0, 0.0, 0.0)),    # a CT on a dose grid
    "ct": ((512, 512, 200), (0.98, 0.98, 2.0), (0.0, 0.0, 0.0)),         # a CT at its own resolution
}


def listed():
    return [
        # a lone spot of a plan checked by itself: launches and the longest track decide
        {"name": "spot_600", "kind": "vertices", "grid": "slab", "histories": 600, "energy": 110.0,
         "beam": "gaussian", "debug": False, "scorer": "dose"},
        # moqui's per-spot simulation: one transport call for each spot of a small field
        {"name": "per_spot", "kind": "plan", "grid": "dose_ct", "spots": 12, "median": 2500, "scorer": "dose",
         "per_spot": True, "scenarios": 1},
        # the phantom example: uniform 200 MeV field in water, debug physics
        {"name": "water_100k", "kind": "vertices", "grid": "water", "histories": 100000, "energy": 200.0,
         "beam": "uniform", "debug": True, "scorer": "edep"},
        # the benchmark's heterogeneous phantom at its full history count
        {"name": "slab_1m", "kind": "vertices", "grid": "slab", "histories": 1000000, "energy": 150.0,
         "beam": "gaussian", "debug": False, "scorer": "dose"},
        # one pass of a field on a CT in one call, with the statistics that decide when to stop
        {"name": "ct_plan_stat", "kind": "plan", "grid": "ct", "spots": 211, "median": 9900, "scorer": "dose_stat",
         "per_spot": False, "scenarios": 1},
        # robust evaluation: 21 setup and density scenarios of a few spots in one call
        {"name": "robust_21", "kind": "plan", "grid": "dose_ct", "spots": 17, "median": 5000, "scorer": "dose_stat",
         "per_spot": False, "scenarios": 21},
        # dose and LETd numerator and denominator inside a contoured organ
        {"name": "let_contour", "kind": "plan", "grid": "dose_ct", "spots": 30, "median": 6000,
         "scorer": "let_contour", "per_spot": False, "scenarios": 1},
        # range shifter and aperture in front of a phantom: three child grids
        {"name": "beamline_250k", "kind": "beamline", "grid": "box", "histories": 250000, "energy": 150.0},
        # a field's Dij: transport into the table, build both layouts, read the CSR
        {"name": "dij_build", "kind": "dij_build", "grid": "ct", "spots": 75, "median": 9900},
        # one forward and backward of a small plan's optimisation, in double (finite-difference checks)
        {"name": "dij_step_small_f64", "kind": "dij_step", "grid": "slab", "spots": 37, "median": 1500,
         "dtype": "float64"},
        # one forward and backward of a large plan's optimisation, in single
        {"name": "dij_step_large", "kind": "dij_step", "grid": "ct", "spots": 500, "median": 9900,
         "dtype": "float32"},
        # a CT of odd size taken from HU to density on the device, before every robust density scenario
        {"name": "hu_ct", "kind": "hu", "nx": 511, "ny": 509, "nz": 199, "scale": 1.035},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["vertices", "vertices", "plan", "plan", "robust", "let", "beamline", "dij_build", "dij_step",
                       "dij_step", "hu"])
    energy = round(rng.uniform(70.0, 230.0), 1)
    if kind == "vertices":
        grid = rng.choice(["water", "slab"])
        return {"kind": "vertices", "grid": grid, "histories": _log(rng, 300, 1000000), "energy": energy,
                "beam": rng.choice(["uniform", "gaussian"]), "debug": rng.random() < 0.4,
                "scorer": rng.choice(["dose", "edep", "dose_stat"])}
    if kind == "plan":
        if rng.random() < 0.4:
            return {"kind": "plan", "grid": rng.choice(["dose_ct", "slab"]), "spots": rng.randint(3, 20),
                    "median": _log(rng, 500, 8000), "scorer": rng.choice(["dose", "dose_stat"]), "per_spot": True,
                    "scenarios": 1}
        return {"kind": "plan", "grid": rng.choice(["ct", "dose_ct"]), "spots": rng.randint(20, 210),
                "median": _log(rng, 1000, 9900), "scorer": rng.choice(["dose", "dose_stat"]), "per_spot": False,
                "scenarios": 1}
    if kind == "robust":
        return {"kind": "plan", "grid": "dose_ct", "spots": rng.randint(3, 17), "median": _log(rng, 500, 5000),
                "scorer": rng.choice(["dose", "dose_stat"]), "per_spot": False, "scenarios": rng.choice([3, 7, 21])}
    if kind == "let":
        return {"kind": "plan", "grid": "dose_ct", "spots": rng.randint(5, 40), "median": _log(rng, 500, 6000),
                "scorer": "let_contour", "per_spot": False, "scenarios": 1}
    if kind == "beamline":
        return {"kind": "beamline", "grid": "box", "histories": _log(rng, 2000, 400000),
                "energy": round(rng.uniform(110.0, 170.0), 1)}
    if kind == "dij_build":
        return {"kind": "dij_build", "grid": rng.choice(["ct", "dose_ct", "slab"]), "spots": rng.randint(5, 75),
                "median": _log(rng, 500, 9900)}
    if kind == "dij_step":
        return {"kind": "dij_step", "grid": rng.choice(["ct", "dose_ct", "slab"]), "spots": _log(rng, 20, 400),
                "median": _log(rng, 800, 9900), "dtype": rng.choice(["float32", "float32", "float64"])}
    return {"kind": "hu", "nx": rng.randint(64, 512), "ny": rng.randint(64, 512), "nz": rng.randint(20, 200),
            "scale": rng.choice([1.0, 1.035, 0.965])}


# ---- inputs ---------------------------------------------------------------------------------

def _edges(grid, shift=(0.0, 0.0, 0.0)):
    n, d, c = GRIDS[grid]
    lxyz = tuple(float(np.float32(a * b)) for a, b in zip(n, d))
    pos = tuple(float(np.float32(a) + np.float32(b)) for a, b in zip(c, shift))
    return ph.phantom_box_edges(lxyz, pos, n)


def _ct_hu(n, d, seed):
    """int16 HU [nz][ny][nx] of an ellipsoidal body in air: a Gaussian-smoothed (5 mm) random field
    of mean 40 and s.d. 150.  Smoothed by shifted sums, whose bits do not depend on a library's
    choice of algorithm."""
    gen = torch.Generator(DEV).manual_seed(seed)
    rad = [int(math.ceil(12.5 / p)) for p in d]
    a = torch.randn([m + 2 * r for m, r in zip(n[::-1], rad[::-1])], generator=gen, device=DEV)
    norm = 1.0
    for axis in range(3):
        r, p = rad[2 - axis], d[2 - axis]
        w = [math.exp(-0.5 * (k * p / 5.0) ** 2) for k in range(-r, r + 1)]
        norm *= math.sqrt(sum(x * x for x in w))
        m = a.shape[axis] - 2 * r
        out = a.narrow(axis, 0, m) * w[0]
        for k in range(1, 2 * r + 1):
            out.add_(a.narrow(axis, k, m), alpha=w[k])
        a = out
    a.mul_(150.0 / norm).add_(40.0).round_().clamp_(-1000.0, 1500.0)
    q = [((torch.arange(m, device=DEV, dtype=torch.float64) + 0.5) / m - 0.5) / s
         for m, s in zip(n, (0.359, 0.239, 0.45))]
    body = (q[2] ** 2)[:, None, None] + (q[1] ** 2)[None, :, None] + (q[0] ** 2)[None, None, :] <= 1.0
    return torch.where(body, a, torch.full_like(a, -1000.0)).to(torch.int16).cpu().numpy()


def _hu(grid, seed):
    n, d, _ = GRIDS[grid]
    if grid in ("ct", "dose_ct"):
        return _ct_hu(n, d, seed)
    hu = np.zeros(n[::-1], np.int16)
    if grid == "slab":
        rng = np.random.default_rng(seed)
        lung, bone = int(rng.integers(25, 60)), int(rng.integers(95, 130))
        hu[n[2] - lung - 30:n[2] - lung] = -700     # the beam enters at the largest z
        hu[n[2] - bone - 15:n[2] - bone] = 1200
    return hu


def _spots(case, seed):
    """Gaussian spots on a 5 mm grid, energies over the range that ends inside the grid, lognormal
    history counts."""
    rng = np.random.default_rng(seed)
    n = case["spots"]
    nx = max(1, int(round(math.sqrt(1.25 * n))))
    i = np.arange(n)
    sp = np.zeros(n, capi.SPOT_DTYPE)
    sp["mean"][:, 0] = (i % nx - 0.5 * (nx - 1)) * 5.0
    sp["mean"][:, 1] = (i // nx - 0.5 * (-(-n // nx) - 1)) * 5.0
    ct = case["grid"] in ("ct", "dose_ct")
    sp["mean"][:, 2] = 195.0 if ct else 0.5
    sp["sigma"][:, :2] = 4.0
    sp["energy"] = rng.uniform(70.0, 230.0 if ct else 180.0, n).astype(np.float32)
    sp["rot"] = np.eye(3, dtype=np.float32).ravel()
    m = case["median"]
    sp["histories"] = np.clip(np.rint(m * np.exp(0.99 * rng.standard_normal(n))), max(1, m // 10), 10 * m)
    return sp


def _vertices(case, seed):
    rng = np.random.default_rng(seed)
    make = ph.uniform_spot_vertices if case["beam"] == "uniform" else ph.gaussian_spot_vertices
    return make(case["histories"], rng, case["energy"], (0.0, 0.0, 0.5),
                (30.0, 30.0) if case["beam"] == "uniform" else (4.0, 4.0))


def _contour(grid):
    """A spherical organ at the grid's centre as a contour ROI: start, stride, accumulated stride."""
    n, d, _ = GRIDS[grid]
    q = [(np.arange(m) + 0.5 - 0.5 * m) * p for m, p in zip(n, d)]
    m = ((q[2] ** 2)[:, None, None] + (q[1] ** 2)[None, :, None] + (q[0] ** 2)[None, None, :] <= 60.0 ** 2).ravel()
    edge = np.flatnonzero(np.diff(np.concatenate([[0], m.view(np.int8), [0]])))
    start, stop = edge[0::2], edge[1::2]
    stride = (stop - start).astype(np.uint32)
    return start.astype(np.uint32), stride, np.cumsum(stride, dtype=np.uint64).astype(np.uint32)


def _add_scorers(ctx, cid, case):
    """Scorer ids; a dose_stat run's pair comes last."""
    what = case.get("scorer", "dose")
    if what == "edep":
        return [ctx.add_scorer(cid, capi.EDEP)]
    if what == "let_contour":
        st, sr, ac = _contour(case["grid"])
        roi = {"roi_method": capi.ROI_CONTOUR, "start": st, "stride": sr, "acc": ac}
        return [ctx.add_scorer(cid, t, **roi) for t in (capi.DOSE_W, capi.LETD_NUM, capi.LETD_DEN)]
    ids = [ctx.add_scorer(cid, capi.DOSE_W)]
    if what == "dose_stat":
        ids += list(ctx.add_stat_scorers(cid))
    return ids


def _scenarios(grid, n):
    """n of the 21 robust scenarios: setup shifts of 0 and +-3 mm per axis, each with density scale
    1, 1.035 and 0.965."""
    shifts = [(0.0, 0.0, 0.0)] + [tuple(s * 3.0 if i == ax else 0.0 for i in range(3)) for ax in range(3) for s in (1, -1)]
    return [(sh, sc) for sh in shifts for sc in (1.0, 1.035, 0.965)][:n]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "seed": seed * 2654435761 + 12345}
    if kind == "hu":
        n = case["nx"] * case["ny"] * case["nz"]
        d = tuple(500.0 / case[k] for k in ("nx", "ny", "nz"))
        s["hu"] = torch.from_numpy(_ct_hu((case["nx"], case["ny"], case["nz"]), d, seed)).to(DEV)
        s["rho"] = torch.empty(n, dtype=torch.float32, device=DEV)
        s["ctx"] = capi.Context(0)
        return s
    ctx = s["ctx"] = capi.Context(0)
    grid = case["grid"]
    ctx.set_physics(bool(case.get("debug", False)))
    if kind == "beamline":
        for child in beamline.children_from_devices([
                ("rangeshifter", (-100.0, -10.0, -100.0), (100.0, 10.0, 100.0), 1.19, (math.pi / 2, 0.0, 0.0),
                 (0.0, 0.0, 50.0)),
                ("aperture", (0.0, 0.0, 25.0), (80.0, 80.0, 10.0), [beamline.circle(20.0, 12)], (0.0, 0.0, 0.0),
                 (0.0, 0.0, 0.0))]):
            child.add_to(ctx)
    cid = ctx.add_child(*_edges(grid))
    if case.get("scenarios", 1) > 1:
        sc = _scenarios(grid, case["scenarios"])
        e = [_edges(grid, sh) for sh, _ in sc]
        ctx.set_scenarios(cid, [x[0] for x in e], [x[1] for x in e], [x[2] for x in e], [x for _, x in sc])
    ctx.set_hu(cid, _hu(grid, seed))
    if kind in ("vertices", "beamline"):
        if kind == "beamline":
            v = ph.uniform_spot_vertices(case["histories"], np.random.default_rng(seed), case["energy"],
                                         (0.0, 0.0, 100.0), (30.0, 30.0))
        else:
            v = _vertices(case, seed)
        ctx.set_vertices(v)
    else:
        s["total"] = ctx.set_spot_plan(_spots(case, seed))
    if kind in ("dij_build", "dij_step"):
        # slots: twice an upper estimate of the entries (at most a beam's column of voxels per spot)
        n, d, _ = GRIDS[grid]
        need = min(s["total"] * 400, case["spots"] * int(6.0e5 * 1.92 / (d[0] * d[1] * d[2])))
        slots = 1 << max(16, (2 * need - 1).bit_length())
        s["dij"] = ctx.add_dij_scorer(cid, capacity=slots)
        if kind == "dij_build":     # the CSR's arrays, with room for any entry count the table can reach
            s["indptr"] = torch.zeros(case["spots"] + 1, dtype=torch.int64, device=DEV)
            s["indices"] = torch.zeros(slots, dtype=torch.int32, device=DEV)
            s["data"] = torch.zeros(slots, dtype=torch.float32, device=DEV)
        if kind == "dij_step":
            ctx.transport_plan(0, s["total"], s["seed"])
            s["op"] = ctx.dij_build(s["dij"])
            s.update(_step_inputs(case, seed))
        return s
    s["ids"] = _add_scorers(ctx, cid, case)
    n_vox = int(np.prod(GRIDS[grid][0])) * case.get("scenarios", 1)
    s["out"] = [torch.empty(n_vox, dtype=torch.float64, device=DEV) for _ in s["ids"]]
    return s


def _step_inputs(case, seed):
    """Spot weights and the objective's gradient with respect to the dose: signed, in the voxels of
    the target and around it."""
    dt = getattr(torch, case["dtype"])
    gen = torch.Generator(DEV).manual_seed(seed + 1)
    n_vox = int(np.prod(GRIDS[case["grid"]][0]))
    w = torch.rand(case["spots"], generator=gen, device=DEV, dtype=torch.float32) + 0.5
    g = torch.randn(n_vox, generator=gen, device=DEV, dtype=torch.float32)
    return {"w": w.to(dt), "g": g.to(dt)}


# ---- passes ---------------------------------------------------------------------------------

def run(s):
    case, kind, ctx = s["case"], s["case"]["kind"], s["ctx"]
    if kind == "hu":
        ctx._check(ctx.lib.mqi_hu_to_density(ctx.h, C.c_void_p(s["hu"].data_ptr()), C.c_void_p(s["rho"].data_ptr()),
                                             s["rho"].numel(), C.c_float(case["scale"]), 1), ctx.h)
        return s["rho"]
    if kind == "dij_step":
        w = s["w"].detach().requires_grad_(True)
        dose = dij.dose(s["op"], w)
        dose.backward(s["g"])
        return {"dose": dose.detach(), "grad": w.grad}
    ctx.reset()
    if kind == "dij_build":
        ctx.transport_plan(0, s["total"], s["seed"])
        ctx.dij_build(s["dij"])
        csr = {k: s[k] for k in ("indptr", "indices", "data")}
        ctx._check(ctx.lib.mqi_dij_get_csr(ctx.h, s["dij"], *[C.c_void_p(t.data_ptr()) for t in csr.values()], 1), ctx.h)
        return csr
    res = {}
    if kind in ("vertices", "beamline"):
        ctx.transport(0, case["histories"], s["seed"])
        n = case["histories"]
    elif case["per_spot"]:
        cum = ctx.plan_cum
        for k in range(case["spots"]):
            ctx.transport_plan(int(cum[k]), int(cum[k + 1]), s["seed"])
        n = s["total"]
    elif case["scorer"] == "dose_stat":
        # one pass of the plan and its estimate: the loop of a run that stops on its statistics
        _, res["sigma"] = ctx.run_plan_until_stat(s["ids"][1], s["ids"][2], 1e-6, 0.5, 1, s["seed"])
    else:
        ctx.transport_plan(0, s["total"], s["seed"])
    if case.get("scorer") == "dose_stat" and "sigma" not in res:
        res["sigma"] = ctx.stat_uncertainty(s["ids"][1], s["ids"][2], n, 0.5)[0]
    for i, b in zip(s["ids"], s["out"]):
        ctx.tally_to_device(i, b.data_ptr())
    res["tally"] = s["out"]
    return res


# ---- what a pass cannot do without ------------------------------------------------------------

def _steps_per_history(case):
    """Voxel steps of a history: about 1.6 for each mm of its range in water."""
    e = case.get("energy", 150.0)
    return 1.6 * 0.022 * e ** 1.77


def work(case):
    kind = case["kind"]
    if kind == "hu":
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 6.0 * n, "flops": 4.0 * n}
    n, d, _ = GRIDS[case["grid"]]
    vox = float(np.prod(n))
    hist = float(case.get("histories", 0)) or case["spots"] * case["median"] * 1.5
    steps = hist * _steps_per_history(case)
    if kind.startswith("dij"):
        # entries: a spot's column fills with its histories, up to a beam's column of voxels
        nnz = case["spots"] * min(1.5 * case["median"] * 60.0, 4.5e5 / (d[0] * d[1] * d[2]))
        if kind == "dij_step":
            es = 8.0 if case["dtype"] == "float64" else 4.0
            return {"bytes": 16.0 * nnz + 2 * es * vox, "flops": 4.0 * nnz}
        return {"bytes": 8.0 * nnz + 4.0 * vox, "flops": FLOPS_PER_STEP * steps}
    scen = case.get("scenarios", 1)
    tallies = {"dose_stat": 3, "let_contour": 3}.get(case.get("scorer"), 1)
    src = 28.0 * hist if kind != "plan" else 112.0 * case["spots"]
    return {"bytes": src + 4.0 * vox + 8.0 * vox * scen * tallies, "flops": FLOPS_PER_STEP * steps * scen}


def exact(case, seed):
    """The Dij products in 64 bits from the matrix a program holds.  Transports and builds are Monte
    Carlo sums over random streams that only the engine draws: they have no such value."""
    if case["kind"] != "dij_step":
        return None
    s = prepare(case, seed)
    indptr, voxel, value = s["op"].csr()
    spot = torch.repeat_interleave(torch.arange(case["spots"], device=DEV),
                                   torch.from_numpy(np.diff(indptr)).to(DEV))
    voxel = torch.from_numpy(voxel.astype(np.int64)).to(DEV)
    value = torch.from_numpy(value).to(DEV).double()
    dose = torch.zeros(s["g"].numel(), dtype=torch.float64, device=DEV)
    dose.index_add_(0, voxel, value * s["w"].double()[spot])
    grad = torch.zeros(case["spots"], dtype=torch.float64, device=DEV)
    grad.index_add_(0, spot, value * s["g"].double()[voxel])
    return {"dose": dose, "grad": grad}
