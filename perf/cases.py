"""The calls that the framework is timed on.

Each case is one call of a public entry point as a caller makes it: a fresh
solve of device arrays (`SolveODE`), an operator-split step that continues
from a kept workspace, a solve of host arrays, a driver's ladder of t_stop
values, several networks in one launch, and the conversion between mass
fractions and number densities.  Inputs are the seeded distributions of
`odevec_b200.workloads`.

`SolveODE` updates its arrays in place, so every pass starts from copies of
the kept initial state (a hydro code that may have to redo a step holds the
same copy).  Device calls run with `raise_on_failure=False`, as the driver,
the multi-network and the serving code of this repository do: the status
array comes back with the other results and nothing waits on the host.
"""
import math

import numpy as np
import torch

from odevec_b200 import driver as D, multi as M, solver as S, workloads as W

# Mean floating-point operations per cell of a whole solve of each network's
# workload, from the integrator's own counters (steps, Newton iterations,
# Jacobians) and the generated code's operation counts: what the method
# needs, without the step-size selection.
SOLVE_FLOPS = {"PRIMORDIAL": 299e3, "OREGO": 177e3, "ROBER": 30.7e3, "SYN64": 3.87e6, "HCTOY": 40e3}
# one continued operator-split step of a PRIMORDIAL cell (about 12 steps)
STEP_FLOPS = 16e3
NEQ = {"PRIMORDIAL": 16, "OREGO": 3, "ROBER": 3, "SYN64": 64, "HCTOY": 9}


def listed():
    return [
        # the benchmark configuration: a million cells of one network, the
        # throughput form
        {"name": "primordial-1m-fp32lu", "kind": "solve", "workload": "PRIMORDIAL",
         "network": "PRIMORDIAL_CSC_FF", "ncells": 1048576, "precision": "fp32_lu", "group": 1},
        # a caller whose arrays live in pinned host memory (the Fortran or C
        # hydro code), in the reference's own precision
        {"name": "primordial-host-fp64", "kind": "host", "workload": "PRIMORDIAL",
         "network": "PRIMORDIAL_CSC_FF", "ncells": 150001, "precision": "fp64", "group": 1},
        # one hydro step of an operator-split run: every cell continues from
        # its kept integrator state for a short span; some cells are masked
        {"name": "primordial-step-fma", "kind": "step", "workload": "PRIMORDIAL",
         "network": "PRIMORDIAL_CSC_FF", "ncells": 100003, "precision": "fp64_fma", "group": 1,
         "hydro": 1e8, "mask": True},
        # a small request of a serving stream (1k cells is its smallest)
        {"name": "primordial-1k-fp32lu", "kind": "solve", "workload": "PRIMORDIAL",
         "network": "PRIMORDIAL_CSC_FF", "ncells": 1000, "precision": "fp32_lu", "group": 1},
        # the smallest call: one lockstep group of the reference's nvector = 32
        {"name": "rober-32-fp64", "kind": "solve", "workload": "ROBER", "network": "ROBER_DENSE_NONE",
         "ncells": 32, "precision": "fp64", "group": 32},
        # the ROBER configuration
        {"name": "rober-4096-fp64", "kind": "solve", "workload": "ROBER", "network": "ROBER_DENSE_NONE",
         "ncells": 4096, "precision": "fp64", "group": 32},
        # the OREGO configuration: an end time per cell, long oscillating runs
        {"name": "orego-65536-fp64", "kind": "solve", "workload": "OREGO", "network": "OREGO_CSC_CMK",
         "ncells": 65536, "precision": "fp64", "group": 1},
        # the large network, a quarter of its configuration's cells
        {"name": "syn64-65536-fp32lu", "kind": "solve", "workload": "SYN64", "network": "SYN64_CSC_CMK",
         "ncells": 65536, "precision": "fp32_lu", "group": 1},
        # the large network as a small request
        {"name": "syn64-3001-fp64", "kind": "solve", "workload": "SYN64", "network": "SYN64_CSC_CMK",
         "ncells": 3001, "precision": "fp64", "group": 1},
        # a hydro code's mass fractions to number densities and back
        {"name": "convert-1m", "kind": "convert", "workload": "PRIMORDIAL", "network": "PRIMORDIAL_CSC_FF",
         "ncells": 1048576},
        # the reference driver's ladder (conversion, solve, conversion back,
        # ten calls of 1e8 s each), replayed as a CUDA graph
        {"name": "ladder-primordial-8192", "kind": "ladder", "workload": "PRIMORDIAL",
         "network": "PRIMORDIAL_CSC_FF", "ncells": 8192, "precision": "fp64", "calls": 10},
        # the serving mix in one launch
        {"name": "mix-fused-fp32lu", "kind": "mix", "workload": "MIX", "rober": 16384, "primordial": 65536,
         "syn64": 4096, "precision": "fp32_lu"},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any of the kinds above, the other shipped variants and
    the options (masks, CheckNegatives) among them."""
    kind = rng.choice(["solve"] * 6 + ["host", "step", "convert", "ladder", "mix"])
    prec = rng.choice(["fp64", "fp64_fma", "fp32_lu"])
    if kind == "convert":
        return {"kind": kind, "workload": "PRIMORDIAL", "network": "PRIMORDIAL_CSC_FF",
                "ncells": _size(rng, 100, 1048576)}
    if kind == "mix":
        return {"kind": kind, "workload": "MIX", "rober": _size(rng, 64, 32768),
                "primordial": _size(rng, 64, 131072), "syn64": _size(rng, 16, 8192), "precision": prec}
    if kind in ("host", "step", "ladder"):
        c = {"kind": kind, "workload": "PRIMORDIAL", "network": "PRIMORDIAL_CSC_FF",
             "ncells": _size(rng, 50, 65536 if kind == "ladder" else 200000), "precision": prec}
        if kind == "ladder":
            c["calls"] = rng.randint(2, 12)
            return c
        c["group"] = 1
        c["mask"] = rng.random() < 0.3
        if kind == "step":
            c["hydro"] = 10.0 ** rng.uniform(6.0, 11.0)
        return c
    wl = rng.choice(["PRIMORDIAL", "PRIMORDIAL", "OREGO", "ROBER", "SYN64", "HCTOY"])
    group = 1
    if wl == "PRIMORDIAL":
        net = rng.choice(["PRIMORDIAL_CSC_FF"] * 3 + ["PRIMORDIAL_CSC_CMK", "PRIMORDIAL_DENSE_NONE",
                                                      "PRIMORDIAL_DENSE_NONE_LU3"])
        n = _size(rng, 1, 1000000 if net == "PRIMORDIAL_CSC_FF" and prec == "fp32_lu" else 200000)
    elif wl == "OREGO":
        net = rng.choice(["OREGO_CSC_CMK", "OREGO_CSC_CMK", "OREGO_DENSE_NONE", "OREGO_DENSE_NONE_LU2"])
        n = _size(rng, 1, 262144)
    elif wl == "ROBER":
        net = rng.choice(["ROBER_DENSE_NONE", "ROBER_DENSE_NONE", "ROBER_CSC_NONE", "ROBER_DENSE_NONE_LU2",
                          "ROBER_DENSE_NONE_LU3"])
        group = rng.choice([1, 32])
        n = _size(rng, 1, 65536)
        if group == 32:
            n = 32 * max(1, n // 32)
    elif wl == "SYN64":
        net, n = "SYN64_CSC_CMK", _size(rng, 1, 32768)
    else:
        net, n = "HCTOY_DENSE_NONE", _size(rng, 1, 131072)
    return {"kind": kind, "workload": wl, "network": net, "ncells": n, "precision": prec, "group": group,
            "mask": rng.random() < 0.2, "check_negatives": rng.random() < 0.2}


class _Solver:
    """An initialised solver object, closed with the state that holds it."""

    def __init__(self, wl, case, max_cells=0, **kw):
        self.ode = S.Odevec(wl.network, max_cells=max_cells, RelativeTolerance=kw.pop("rtol", wl.rtol),
                            AbsoluteTolerance=wl.atol, MinimalTimestep=wl.dt_min, nvector=case.get("group", 1),
                            precision=case["precision"], CheckNegatives=bool(case.get("check_negatives")),
                            raise_on_failure=False, **kw)
        S.InitOdevec(self.ode)

    def __del__(self):
        try:
            S.CloseOdevec(self.ode)
        except Exception:
            pass


def _workload(case, seed):
    build = {"PRIMORDIAL": W.primordial, "OREGO": W.orego, "ROBER": W.rober, "SYN64": W.syn64, "HCTOY": W.hctoy}
    return build[case["workload"]](ncells=case["ncells"], seed=seed, network=case["network"])


def _mask(case, seed):
    """Cells of a hydro grid that are left out of the chemistry (every tenth
    or so)."""
    if not case.get("mask"):
        return None
    m = np.random.default_rng(seed + 1).random(case["ncells"]) >= 0.1
    m[0] = True
    return m


def _convert_inputs(case, seed):
    """Mass fractions and gas density of the workload's cells (the rows
    without a mass pass through)."""
    n = _workload(case, seed).y
    mass = np.array(MASSES)[:, None]
    rho = (n * mass).sum(0)
    return np.where(mass > 0.0, n * mass / rho, n), rho


# g; electron, H-, H, He, H2, D, HD, H+, He+, H2+, D+, He++, and four rows without a mass
MASSES = [9.10938188e-28, 1.67444345638e-24, 1.67353251819e-24, 6.69206503638e-24, 3.34706503638e-24,
          3.34603251819e-24, 5.01956503638e-24, 1.67262158e-24, 6.69115409819e-24, 3.34615409819e-24,
          3.34512158e-24, 6.69024316e-24, 0.0, 0.0, 0.0, 0.0]
# 1/g, with the digits that KROME's tables give
IMASSES = [1.09776932527e+27, 5.9721335838e+23, 5.97538433901e+23, 1.49430705554e+23, 2.9876921695e+23,
           2.98861411108e+23, 1.99220448934e+23, 5.97863863505e+23, 1.4945104915e+23, 2.98850552203e+23,
           2.98942796572e+23, 1.49471398286e+23, 0.0, 0.0, 0.0, 0.0]


def _device(a):
    return torch.tensor(a, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "convert":
        x, rho = _convert_inputs(case, seed)
        x = _device(x)
        return {"kind": kind, "network": case["network"], "x": x, "rho": _device(rho),
                "n": torch.empty_like(x), "back": torch.empty_like(x)}
    if kind == "mix":
        jobs, init, keep = [], [], []
        for k, wl in enumerate((W.rober(case["rober"], seed), W.primordial(case["primordial"], seed),
                                W.syn64(case["syn64"], seed))):
            s = _Solver(wl, {"precision": case["precision"]}, escalation=False)
            arrs = [_device(a) for a in (wl.t0, wl.dt0, wl.t_stop, wl.y)]
            init.append([a.clone() for a in arrs])
            jobs.append((s.ode, *arrs))
            keep.append(s)
        return {"kind": kind, "many": M.SolveMany(jobs, fused=True), "jobs": jobs, "init": init, "keep": keep}
    wl = _workload(case, seed)
    n = wl.ncells
    if kind == "ladder":
        x, rho = _convert_inputs(case, seed)
        s = _Solver(wl, case, rtol=1e-4)
        y0, y = _device(x), _device(x)
        dt0 = float(wl.dt0[0])
        lad = D.Ladder(s.ode, y, 0.0, dt0, [1e8 * (k + 1) for k in range(case["calls"])], rho=_device(rho),
                       graph=True, chunk=case["calls"])
        st = {"kind": kind, "lad": lad, "y0": y0, "y": y, "t0": lad.t.clone(), "d0": lad.d.clone(), "keep": s}
        run(st)  # captures the graph, once per run of the program
        return st
    mask = _mask(case, seed)
    if kind == "host":
        s = _Solver(wl, case, max_cells=n)
        pin = lambda a: torch.tensor(a).pin_memory()  # noqa: E731
        st = {"kind": kind, "ode": s.ode, "keep": s, "mask": None if mask is None else pin(mask.astype(np.uint8)).numpy(),
              "ts": pin(wl.t_stop).numpy()}
        for k, a in (("y", wl.y), ("t", wl.t0), ("dt", wl.dt0)):
            st[k + "0"], st[k] = pin(a), pin(a)
        return st
    s = _Solver(wl, case)
    st = {"kind": kind, "ode": s.ode, "keep": s, "mask": None if mask is None else _device(mask.astype(np.uint8)),
          "y0": _device(wl.y), "t0": _device(wl.t0), "dt0": _device(wl.dt0), "ts": _device(wl.t_stop)}
    if kind == "step":
        # the state that the run has reached after its first hydro step
        st["ws0"] = S.Workspace(s.ode, n)
        st["ts"] = torch.full((n,), 2.0 * case["hydro"], dtype=torch.float64, device="cuda")
        S.SolveODE(s.ode, st["t0"], st["dt0"], 0.5 * st["ts"], st["y0"], Mask=st["mask"], workspace=st["ws0"])
        st["ws"] = torch.empty_like(st["ws0"])
    return st


def run(st):
    kind = st["kind"]
    if kind == "convert":
        D.x2n(st["network"], st["x"], st["rho"], out=st["n"])
        D.n2x(st["network"], st["n"], st["rho"], out=st["back"])
        return {"n": st["n"], "x": st["back"]}
    if kind == "ladder":
        lad = st["lad"]
        st["y"].copy_(st["y0"])
        lad.t.copy_(st["t0"])
        lad.d.copy_(st["d0"])
        t, d, failed = lad.run()
        return {"y": st["y"], "t": t, "dt": d, "status": failed}
    if kind == "mix":
        for job, first in zip(st["jobs"], st["init"]):
            for k in (0, 1, 3):  # time, dt, y
                job[k + 1].copy_(first[k])
        status = st["many"].run()
        return [{"y": j[4], "t": j[1], "dt": j[2], "status": s} for j, s in zip(st["jobs"], status)]
    if kind == "host":
        for k in ("y", "t", "dt"):
            st[k].copy_(st[k + "0"])
        y, t, dt = (st[k].numpy() for k in ("y", "t", "dt"))
        S.SolveODE(st["ode"], t, dt, st["ts"], y, Mask=st["mask"], in_place=True)
        return {"y": y, "t": t, "dt": dt, "status": st["ode"].status, "stats": st["ode"].stats}
    y, t, dt = st["y0"].clone(), st["t0"].clone(), st["dt0"].clone()
    if kind == "step":
        ws = st["ws"].copy_(st["ws0"])
        t, dt = S.SolveODE(st["ode"], t, dt, st["ts"], y, Mask=st["mask"], workspace=ws, resume=True)
        return {"y": y, "t": t, "dt": dt, "status": st["ode"].status, "stats": st["ode"].stats, "workspace": ws}
    t, dt = S.SolveODE(st["ode"], t, dt, st["ts"], y, Mask=st["mask"])
    return {"y": y, "t": t, "dt": dt, "status": st["ode"].status, "stats": st["ode"].stats}


def work(case):
    """Bytes: state, time, step and end time in, state, time, step and status
    out.  Operations: the method's own, at the workload's mean counts."""
    kind = case["kind"]
    if kind == "mix":
        b = f = 0.0
        for key in ("rober", "primordial", "syn64"):
            w = key.upper()
            b += case[key] * (16.0 * NEQ[w] + 44.0)
            f += case[key] * SOLVE_FLOPS[w]
        return {"bytes": b, "flops": f}
    n, neq = case["ncells"], NEQ[case["workload"]]
    if kind == "convert":
        # both directions: the rows in, the rows out, the density
        return {"bytes": 2.0 * n * (16.0 * neq + 8.0), "flops": 2.0 * n * 24.0}
    if kind == "ladder":
        # the first call starts at order 1 (about 60 steps), as every call does
        return {"bytes": n * (16.0 * neq + 44.0) * case["calls"], "flops": n * 80e3 * case["calls"]}
    if kind == "step":
        return {"bytes": n * (16.0 * neq + 44.0 + 2.0 * 864.0), "flops": n * STEP_FLOPS}
    return {"bytes": n * (16.0 * neq + 44.0), "flops": n * SOLVE_FLOPS[case["workload"]]}


def _robertson(y, t_end):
    """Robertson's problem from 0 to t_end for all columns of y at once:
    three-stage Radau IIA (order 5) on a geometric grid."""
    s6 = math.sqrt(6.0)
    A = np.array([[(88 - 7 * s6) / 360, (296 - 169 * s6) / 1800, (-2 + 3 * s6) / 225],
                  [(296 + 169 * s6) / 1800, (88 + 7 * s6) / 360, (-2 - 3 * s6) / 225],
                  [(16 - s6) / 36, (16 + s6) / 36, 1.0 / 9.0]])
    f = lambda u: np.stack([-0.04 * u[..., 0] + 1e4 * u[..., 1] * u[..., 2],  # noqa: E731
                            0.04 * u[..., 0] - 3e7 * u[..., 1] ** 2 - 1e4 * u[..., 1] * u[..., 2],
                            3e7 * u[..., 1] ** 2], axis=-1)
    u = y.T.copy()
    grid = np.concatenate([[0.0], np.geomspace(1e-6, t_end, 260)])
    eye = np.eye(9)
    for h in np.diff(grid):
        z = np.zeros((u.shape[0], 3, 3))
        for _ in range(8):
            v = u[:, None, :] + z
            J = np.zeros((u.shape[0], 3, 3, 3))
            J[..., 0, 0], J[..., 0, 1], J[..., 0, 2] = -0.04, 1e4 * v[..., 2], 1e4 * v[..., 1]
            J[..., 1, 0] = 0.04
            J[..., 1, 1], J[..., 1, 2] = -6e7 * v[..., 1] - 1e4 * v[..., 2], -1e4 * v[..., 1]
            J[..., 2, 1] = 6e7 * v[..., 1]
            res = h * np.einsum("ij,cjk->cik", A, f(v)) - z
            mat = eye - h * np.einsum("ij,cjkl->cikjl", A, J).reshape(-1, 9, 9)
            dz = np.linalg.solve(mat, res.reshape(-1, 9, 1)).reshape(-1, 3, 3)
            z += dz
            if np.abs(dz).max() < 1e-15:
                break
        u = u + z[:, 2, :]
    return u.T


def exact(case, seed):
    """The conversion in NumPy; Robertson's problem by an independent method
    of higher order.  The other networks' solutions (stiff, 12 to 64 species,
    or long oscillating runs with an end time per cell) take minutes in NumPy.
    The time at the end is t_stop for every cell; the next step size, status
    and counters have no value outside the method."""
    kind = case["kind"]
    if kind == "convert":
        x, rho = _convert_inputs(case, seed)
        m, im = np.array(MASSES)[:, None], np.array(IMASSES)[:, None]
        n = np.where(m > 0.0, rho * x * im, x)
        return {"n": n, "x": np.where(m > 0.0, n * m / rho, n)}
    if kind == "mix":
        return [{"y": None, "t": w.t_stop, "dt": None, "status": None}
                for w in (W.rober(case["rober"], seed), W.primordial(case["primordial"], seed),
                          W.syn64(case["syn64"], seed))]
    n = case["ncells"]
    if kind == "ladder":
        return {"y": None, "t": np.full(n, 1e8 * case["calls"]), "dt": None, "status": None}
    if kind == "step":
        return {"y": None, "t": np.full(n, 2.0 * case["hydro"]), "dt": None, "status": None, "stats": None,
                "workspace": None}
    wl = _workload(case, seed)
    y = None
    if case["workload"] == "ROBER" and n <= 4096:
        y = _robertson(wl.y, float(wl.t_stop[0]))
        mask = _mask(case, seed)
        if mask is not None:
            y = np.where(mask, y, wl.y)
    return {"y": y, "t": wl.t_stop, "dt": None, "status": None, "stats": None}
