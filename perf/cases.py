"""Performance cases of the FIM simulator: report steps through `ReservoirSimulator.step` and
`Ensemble.step`, the linear-solver seam and the adjoint, each as a program with its own deck runs
it.  A case is a dict of plain values; `prepare` builds the deck and the device context from a
seed, `run` is one pass.

A step pass uploads the state it starts from (`rf_set_state`), takes one report step and reads the
state and the well BHPs back, so every pass does the same work.  The permeability and porosity
fields come from the seed; everything else of a deck (wells, fluids, controls) is the generator's.
"""
import ctypes as C
import math

import numpy as np
import torch

from ressim_b200 import Ensemble, ReservoirSimulator, _abi, _lib, decks, linear_solve_bsr

_dp = C.POINTER(C.c_double)


def listed():
    return [
        # the 1D waterflood configuration: the smallest deck a program steps, launches and the
        # dense coarse inverse count
        {"name": "1d-200", "kind": "step", "fluid": "1d", "nx": 200, "ny": 1, "nz": 1, "dt": 10.0,
         "precision": "fp64"},
        # a teaching-size black-oil deck whose Newton systems take the direct LU
        {"name": "bo-direct-5x5x4", "kind": "step", "fluid": "blackoil", "nx": 5, "ny": 5, "nz": 4, "dt": 5.0,
         "precision": "fp64"},
        # SPE1's grid with the black-oil fluid: the smallest iterative black-oil deck
        {"name": "bo-10x10x3", "kind": "step", "fluid": "blackoil", "nx": 10, "ny": 10, "nz": 3, "dt": 10.0,
         "precision": "fp64"},
        # ordinary single decks, odd sizes: with gravity, and the middle of the ensemble's sizes
        {"name": "wf-33x29x7-gravity", "kind": "step", "fluid": "waterflood-gravity", "nx": 33, "ny": 29, "nz": 7,
         "dt": 1.0, "precision": "fp64"},
        {"name": "wf-45x61x7", "kind": "step", "fluid": "waterflood", "nx": 45, "ny": 61, "nz": 7, "dt": 1.0,
         "precision": "fp64"},
        # the 72,000-cell black-oil configuration
        {"name": "bo-60x60x20", "kind": "step", "fluid": "blackoil", "nx": 60, "ny": 60, "nz": 20, "dt": 0.25,
         "precision": "fp64"},
        # a large mixed-precision waterflood (the 2M-cell configuration's kind, a quarter of its size)
        {"name": "wf-127x101x40-mixed", "kind": "step", "fluid": "waterflood", "nx": 127, "ny": 101, "nz": 40,
         "dt": 0.1, "precision": "mixed"},
        # the sensitivity ensemble, in FP64 and in the mixed form: variants of uneven sizes
        {"name": "ensemble-16", "kind": "ensemble", "first": 0, "count": 16, "dt": 1.0, "precision": "fp64"},
        {"name": "ensemble-12-mixed", "kind": "ensemble", "first": 40, "count": 12, "dt": 1.0,
         "precision": "mixed"},
        # comparison runs with tight tolerances: refined solves, Newton to CNV 1e-8 / MB 1e-10
        {"name": "matched-21x20x5", "kind": "matched", "fluid": "waterflood", "nx": 21, "ny": 20, "nz": 5, "dt": 1.0,
         "precision": "fp64"},
        # the linear-solver seam on a host matrix (another simulator's Newton system)
        {"name": "seam-40x31x5", "kind": "seam", "nx": 40, "ny": 31, "nz": 5},
        # gradients: two recorded report steps and the backward pass
        {"name": "adjoint-12x11x4", "kind": "adjoint", "fluid": "blackoil", "nx": 12, "ny": 11, "nz": 4, "dt": 1.0,
         "steps": 2},
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "step", "ensemble", "matched", "seam", "adjoint"])
    if kind == "ensemble":
        return {"kind": kind, "first": rng.randrange(64, 4096), "count": rng.randint(2, 12), "dt": rng.choice([0.25, 1.0]),
                "precision": rng.choice(["fp64", "mixed"])}
    fluid = rng.choice(["waterflood", "waterflood-gravity", "blackoil"])
    top = {"step": 300000.0, "matched": 4000.0, "seam": 12000.0, "adjoint": 600.0}[kind]
    cells = math.exp(rng.uniform(math.log(100.0), math.log(top)))
    nz = rng.randint(2, 40 if cells > 40000 else 16 if cells > 2500 else 5)
    aspect = math.exp(rng.uniform(-0.5, 0.5))
    nx = max(4, round(math.sqrt(cells / nz) * aspect))
    ny = max(4, round(math.sqrt(cells / nz) / aspect))
    if kind == "seam":
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz}
    if kind == "adjoint":
        return {"kind": kind, "fluid": "blackoil", "nx": nx, "ny": ny, "nz": nz, "dt": 1.0, "steps": 2}
    n = nx * ny * nz
    dt = rng.choice([1.0, 5.0]) if n < 10000 else 0.25 if n < 90000 else 0.1
    return {"kind": kind, "fluid": fluid, "nx": nx, "ny": ny, "nz": nz, "dt": dt,
            "precision": rng.choice(["fp64", "fp64", "mixed"]) if kind == "step" else "fp64"}


def _deck(case, seed):
    nx, ny, nz, fluid = case["nx"], case["ny"], case["nz"], case["fluid"]
    if fluid == "1d":
        d, _, _ = decks.waterflood_1d(nx)
        kh, _ = decks.lognormal_field((1, 1, nx), seed, math.log(100.0), 0.3, 5.0)
        d.set_permeability_field(kh, kh, kh)
        return d
    if fluid == "blackoil":
        return decks.black_oil_3d(nx, ny, nz, seed=seed, rate_per_perf=5.0)
    return decks.waterflood_3d(nx, ny, nz, seed=seed, rate_per_perf=10.0, gravity=fluid == "waterflood-gravity")


def _variant(index, seed):
    """Variant `index` of the ensemble (its sizes, fluids and controls) with the seed's rock."""
    d = decks.ensemble_variant(index)
    kh, z = decks.lognormal_field((d.nz, d.ny, d.nx), 1000 * seed + index, math.log(100.0), 1.0, 5.0)
    d.set_permeability_field(kh, kh, 0.1 * kh)
    d.set_porosity_field(np.clip(0.1 + 0.02 * z, 0.05, 0.3))
    return d


def _host_state(d):
    """The deck's state in pinned host memory, as a coupled program holds it."""
    return [torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).pin_memory()
            for a in (d.pressure, d.sat_water, d.sat_gas, d.rs)]


def _upload(handle, host):
    rc = _lib.load().rf_set_state(handle, *[C.cast(t.data_ptr(), _dp) for t in host], C.c_double(0.0))
    if rc != _abi.RF_OK:
        raise RuntimeError(f"rf_set_state failed: {_lib.last_error(handle)}")


def _seam_system(case, seed):
    """A Newton-like 3x3 block system on the grid's 7-point pattern: a transmissibility Laplacian
    with compressibility in the pressure unknown, upwinded transport in the saturations."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    rng = np.random.default_rng(seed)
    kh, z = decks.lognormal_field((nz, ny, nx), seed, 0.0, 1.0, 3.0)
    idx = np.arange(n)
    i, j, k = idx % nx, (idx // nx) % ny, idx // (nx * ny)
    pot = rng.standard_normal(n) + 0.05 * (i + j)
    acc = 0.05 + 0.02 * rng.random(n)
    rows, cols, blocks = [], [], []
    diag = np.zeros((n, 3, 3))
    diag[:, 0, 0] = 1e-3
    diag[:, 0, 1] = 0.2 * acc
    diag[:, 1, 0] = 1e-3 * acc
    diag[:, 1, 1] = acc
    diag[:, 2, 2] = 1.0
    for ok, off, geo in ((i > 0, -1, 1.0), (i < nx - 1, 1, 1.0), (j > 0, -nx, 1.0), (j < ny - 1, nx, 1.0),
                         (k > 0, -nx * ny, 3.0), (k < nz - 1, nx * ny, 3.0)):
        r = idx[ok]
        c = r + off
        t = geo * 2.0 / (1.0 / kh[r] + 1.0 / kh[c])
        up_here = pot[r] >= pot[c]
        lam = np.where(up_here, 0.3 + 0.4 * acc[r], 0.3 + 0.4 * acc[c])
        flow = 0.02 * t * np.abs(pot[r] - pot[c])
        b = np.zeros((len(r), 3, 3))
        b[:, 0, 0] = -t
        b[:, 1, 0] = -t * lam
        b[:, 1, 1] = np.where(up_here, 0.0, -flow)
        diag[r, 0, 0] += t
        diag[r, 1, 0] += t * lam
        diag[r, 1, 1] += np.where(up_here, flow, 0.0)
        rows.append(r)
        cols.append(c)
        blocks.append(b)
    rows = np.concatenate([idx] + rows)
    cols = np.concatenate([idx] + cols)
    blocks = np.concatenate([diag] + blocks)
    order = np.lexsort((cols, rows))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    rhs = (rng.standard_normal((n, 3)) * np.array([1.0, 0.3, 0.0])).ravel()
    return rp, cols[order].astype(np.int32), np.ascontiguousarray(blocks[order].reshape(-1)), rhs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "seam":
        d = decks.waterflood_3d(case["nx"], case["ny"], case["nz"], seed=seed)
        d.wells = []
        sim = ReservoirSimulator.from_deck(d)
        sim.get_pressures()  # the device context
        return {"kind": kind, "sim": sim, "system": _seam_system(case, seed)}
    if kind == "ensemble":
        ds = [_variant(case["first"] + v, seed) for v in range(case["count"])]
        ens = Ensemble(ds, precision=case["precision"])
        return {"kind": kind, "ens": ens, "hosts": [_host_state(d) for d in ds], "dt": case["dt"]}
    d = _deck(case, seed)
    sim = ReservoirSimulator.from_deck(d)
    state = {"kind": kind, "sim": sim, "host": _host_state(d), "dt": case["dt"]}
    if kind == "adjoint":
        sim.set_controller_options(True, 1e-9, 1e-11)
        state["steps"] = case["steps"]
    else:
        sim.set_linear_precision(case["precision"])
    if kind == "matched":
        sim.set_controller_options(False, 1e-8, 1e-10)
        sim.set_linear_refinement(1e-10)
    return state


def run(state):
    kind = state["kind"]
    if kind == "seam":
        x, _ = linear_solve_bsr(state["sim"], *state["system"])
        return {"x": x}
    if kind == "ensemble":
        ens = state["ens"]
        for h, host in zip(ens._ctx, state["hosts"]):
            _upload(h, host)
        ens.step(state["dt"])
        return [{k: s[k] for k in ("pressure", "sat_water")} | {"bhp": ens.well_bhp(v)}
                for v, s in ((v, ens.state(v)) for v in range(len(ens)))]
    sim = state["sim"]
    _upload(sim._context(), state["host"])
    if kind == "adjoint":
        sim.adjoint_record(True)
        for _ in range(state["steps"]):
            sim.step(state["dt"])
        value, grad, controls = sim.backward()
        s = sim.state()
        return {"value": value, "grad": grad, "controls": controls, "pressure": s["pressure"], "sat_gas": s["sat_gas"]}
    sim.step(state["dt"])
    s = sim.state()
    return {k: s[k] for k in ("pressure", "sat_water", "sat_gas", "rs")} | {"bhp": sim.get_well_bhp()}


def _cells(case):
    if case["kind"] != "ensemble":
        return case["nx"] * case["ny"] * case["nz"]
    total = 0
    for v in range(case["count"]):  # the sizes decks.ensemble_variant draws
        rng = np.random.default_rng(1000 + case["first"] + v)
        nx, ny = (int(a) for a in rng.integers(20, 65, size=2))
        total += nx * ny * int(rng.integers(5, 17))
    return total


def work(case):
    """One pass at the least a report step can take: the state read and written once, and three
    Newton iterations (the controller accepts none before) that each write the block Jacobian
    (7 blocks of 3x3 per cell) once and read it once with the residual and the update.  The seam
    reads its matrix and right-hand side and writes x."""
    n = _cells(case)
    newton = n * (2 * 7 * 72 + 2 * 24)
    if case["kind"] == "seam":
        return {"bytes": n * (7 * 72 + 7 * 4 + 48), "flops": n * 7 * 18}
    steps = case.get("steps", 1)
    per_step = n * 8 * 14 + 3 * newton
    both = 2 if case["kind"] == "adjoint" else 1
    return {"bytes": both * steps * per_step, "flops": both * steps * 3 * n * 7 * 18}


def exact(case, seed):
    """Systems of at most 512 rows are solved to rounding (direct LU); larger ones, and every step,
    stop at a tolerance, which has no exact value."""
    if case["kind"] != "seam" or 3 * _cells(case) > 512:
        return None
    rp, cols, vals, rhs = _seam_system(case, seed)
    n = len(rp) - 1
    a = np.zeros((3 * n, 3 * n))
    for r in range(n):
        for e in range(rp[r], rp[r + 1]):
            c = cols[e]
            a[3 * r:3 * r + 3, 3 * c:3 * c + 3] = vals[9 * e:9 * e + 9].reshape(3, 3)
    return {"x": np.linalg.solve(a, rhs)}
