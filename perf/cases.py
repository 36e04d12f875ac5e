"""Workloads of the framework over the range its users run, through its public
entry points (cardiacfoam_gb300.api).

listed() names twelve of them, draw() gives further ones of the same ranges,
prepare() makes what a program holds before the call, run() is one pass,
work() what a pass cannot do without, and exact() the same results from plain
numpy in 64 bits where the model is short enough to be written out here.

Fields of the mixed form (32-bit gates and currents) are returned in 32 bits,
which is what they carry; those of the FP64 form, and of the float-pair
solves, as they are.  A monodomain or bidomain context advances by `steps`
time steps a pass and hands its fields to the host, as a run does between two
write times.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from cardiacfoam_gb300 import api, io, lib, lv
from cardiacfoam_gb300 import verification as ver
from cardiacfoam_gb300.fields import gaussian_random_field
from cardiacfoam_gb300.mesh import box_mesh

SIGMA = (0.1334, 0.0, 0.0, 0.0176, 0.0, 0.0176)
CHI, CM = 140000.0, 0.01
TISSUE = {"TNNP": "epicardialCells", "ORd": "myocyte", "ToRORd_dynCl": "endocardialCells",
          "BuenoOrovio": "epicardialCells"}
# operations of one right-hand-side evaluation (csrc/models/opcounts.json) and states
OPS = {"TNNP": (476, 17), "ORd": (1182, 41), "ToRORd_dynCl": (1430, 45), "BuenoOrovio": (89, 4)}
EVALS = 7          # six RKF45 stages and the current at the end of the step


def listed():
    return [
        # one cell driven step by step from the host, as singleCellSolver does:
        # the smallest call there is, all launch and copy latency
        dict(name="single_cell_tnnp", kind="cell", model="TNNP", n=1, steps=20, dt=1e-5),
        # the ionic update as a plug-in of a host-side solver: Vm in, current
        # out, host arrays, mixed form, an odd cell count
        dict(name="ionic_call_ord", kind="ionic", model="ORd", n=52501, steps=4, dt=5e-6,
             mixed=True),
        # the tutorial-sized cuboid at h = 0.5 mm in the plain FP64 form
        dict(name="slab_tnnp_3k", kind="slab", model="TNNP", nx=40, ny=14, nz=6, dt=1e-5,
             steps=20, mixed=False),
        # the cuboid at h = 0.1 mm, the configuration production runs use
        dict(name="slab_ord_420k", kind="slab", model="ORd", nx=200, ny=70, nz=30, dt=5e-6,
             steps=100, mixed=True),
        # the same cuboid at h = 0.2 mm in FP64, the reference arithmetic
        dict(name="slab_ord_52k_fp64", kind="slab", model="ORd", nx=100, ny=35, nz=15, dt=5e-6,
             steps=4, mixed=False),
        # left ventricle of tetrahedra with fibres and three cell types: the
        # general mesh, corrected Laplacian, working set beyond L2
        dict(name="lv_tnnp_564k", kind="lv", nt=12, m=38, nr=42, dt=1e-5, steps=5, mixed=True),
        # the Niederer benchmark as the regression test runs it: explicit
        # diffusion, BuenoOrovio, FP64
        dict(name="niederer_explicit_52k", kind="niederer", nx=100, ny=35, nz=15, steps=20),
        # a population of independently parameterised cells, from creation to
        # results (SingleCellSolver for many cells)
        dict(name="batch_torord_16k", kind="batch", model="ToRORd_dynCl", n=16384, steps=300,
             dt=1e-5, mixed=True),
        # the bidomain tutorial's manufactured cube, float-pair solves
        dict(name="bidomain_cube_64k", kind="bidomain", n=40, steps=2, pairs=True),
        # gradient of a probe misfit on the two-dimensional sheet, forward and
        # backward
        dict(name="adjoint_sheet_16k", kind="adjoint", n=128, steps=40, mixed=True),
        # pseudo-ECG recorded while a ventricle runs
        dict(name="ecg_lv_564k", kind="ecg", nt=12, m=38, nr=42, electrodes=5, rows=32),
        # a Purkinje network alone, of the tutorial's order of size (193 nodes)
        dict(name="purkinje_network", kind="purkinje", depth=5, segment=6, steps=20),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cell", "ionic", "slab", "slab", "lv", "niederer", "batch", "bidomain",
                       "adjoint", "ecg", "purkinje"])
    if kind == "cell":
        return dict(kind=kind, model=rng.choice(["TNNP", "BuenoOrovio"]), n=_log_int(rng, 1, 64),
                    steps=rng.randint(5, 20), dt=rng.choice([1e-5, 2e-5]))
    if kind == "ionic":
        return dict(kind=kind, model=rng.choice(["TNNP", "ORd", "ToRORd_dynCl"]),
                    n=_log_int(rng, 100, 60000), steps=rng.randint(1, 4), dt=5e-6,
                    mixed=rng.random() < 0.7)
    if kind == "slab":
        h = math.exp(rng.uniform(math.log(0.1), math.log(0.5)))
        d = [max(2, int(round(v / h))) for v in (20.0, 7.0, 3.0)]
        mixed = rng.random() < 0.6 or d[0] > 110
        return dict(kind=kind, model=rng.choice(["TNNP", "ORd", "ToRORd_dynCl"]), nx=d[0],
                    ny=d[1], nz=d[2], dt=5e-6, steps=rng.randint(5, 20) if mixed else 3,
                    mixed=mixed)
    if kind == "lv":
        s = math.exp(rng.uniform(math.log(0.35), 0.0))
        return dict(kind=kind, nt=max(3, int(12 * s)), m=2 * int(19 * s), nr=int(42 * s),
                    dt=1e-5, steps=rng.randint(2, 5), mixed=s > 0.5 or rng.random() < 0.5)
    if kind == "niederer":
        h = math.exp(rng.uniform(math.log(0.2), math.log(0.5)))
        d = [max(2, int(round(v / h))) for v in (20.0, 7.0, 3.0)]
        return dict(kind=kind, nx=d[0], ny=d[1], nz=d[2], steps=rng.randint(10, 20))
    if kind == "batch":
        return dict(kind=kind, model=rng.choice(["TNNP", "ORd", "ToRORd_dynCl"]),
                    n=_log_int(rng, 64, 16384), steps=rng.randint(50, 300), dt=1e-5, mixed=True)
    if kind == "bidomain":
        pairs = rng.random() < 0.7
        return dict(kind=kind, n=rng.randint(12, 40 if pairs else 28), steps=rng.randint(1, 2),
                    pairs=pairs)
    if kind == "adjoint":
        mixed = rng.random() < 0.7
        return dict(kind=kind, n=_log_int(rng, 24, 128 if mixed else 64),
                    steps=10 * rng.randint(2, 4 if mixed else 2), mixed=mixed)
    if kind == "ecg":
        s = math.exp(rng.uniform(math.log(0.35), 0.0))
        return dict(kind=kind, nt=max(3, int(12 * s)), m=2 * int(19 * s), nr=int(42 * s),
                    electrodes=rng.randint(1, 12), rows=rng.randint(8, 32))
    return dict(kind="purkinje", depth=rng.randint(2, 7), segment=rng.randint(2, 9),
                steps=rng.randint(5, 20))


# ------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=4)
def _box(nx, ny, nz, lx, ly, lz):
    return box_mesh(nx, ny, nz, lx, ly, lz)


@functools.lru_cache(maxsize=2)
def _ventricle(nt, m, nr):
    return lv.left_ventricle(nt, m, nr)


@functools.lru_cache(maxsize=2)
def _cube(n):
    return ver.geometry_mesh_for(3, n)


def _vm_field(centres, seed, radius, rest=-0.084):
    """Tissue at rest with a smooth variation of about 2 mV and one ball of the
    given radius, somewhere inside, that has just been depolarised."""
    rng = np.random.default_rng(seed)
    lo, hi = centres.min(axis=0), centres.max(axis=0)
    x = (centres - lo) / np.where(hi > lo, hi - lo, 1.0)
    v = np.full(len(centres), rest)
    for _ in range(4):
        k, ph = rng.uniform(1.0, 6.0, 3), rng.uniform(0.0, 2.0 * np.pi)
        v += 1e-3 * rng.uniform(0.2, 1.0) * np.cos(x @ k + ph)
    mid = centres[rng.integers(0, len(centres))]
    r = np.sqrt(((centres - mid) ** 2).sum(axis=1)) / radius
    return v + 0.1 / (1.0 + np.exp(8.0 * (r - 1.0)))


def _corner_box():
    return [((0.0, 0.0, 0.0), (1.5e-3, 1.5e-3, 1.5e-3), 0.0, 2e-3, 5e4)]


def _precision(case):
    return lib.PRECISION_MIXED if case.get("mixed") else lib.PRECISION_FP64


def _carried(case, a):
    return a.astype(np.float32) if case.get("mixed") else a


def _niederer_case(case):
    mesh = _box(case["nx"], case["ny"], case["nz"], 20e-3, 7e-3, 3e-3)
    # a Courant-limited step: the largest h^2 the explicit step is stable at
    h = 20e-3 / case["nx"]
    return mesh, min(5e-5, 0.1 * h * h * CHI * CM / SIGMA[0])


def _ecg_points(L, count):
    base = L.ecg_electrodes()
    t = np.arange(count)[:, None]
    return base[np.arange(count) % len(base)] * (1.0 + 0.1 * (t // len(base)))


def _tree(case, seed):
    """Edges of a branching network whose segments and conductances vary."""
    e, _, _ = io.synthetic_purkinje_tree(case["depth"], case["segment"], 2.5e-4, seed=seed)
    rng = np.random.default_rng(seed)
    e[:, 2:] *= np.exp(0.2 * rng.standard_normal((len(e), 2)))
    return e


def _bidomain_start(mesh, seed):
    V, pe, _, u1, u2, u3 = ver.bidomain_fields(mesh.centres, 0.0, 3)
    rng = np.random.default_rng(seed)
    k = rng.integers(1, 4, 3)
    V = V + 0.02 * np.cos(mesh.centres @ (np.pi * k))
    return V, pe, u1, u2, u3


def _ionic_vm(n, seed, k):
    rng = np.random.default_rng(seed)
    base = -0.086 + 0.11 * rng.random(n) ** 4
    return np.ascontiguousarray(base + 1e-4 * k * rng.standard_normal(n))


def _cell_states(case, seed, y0):
    rng = np.random.default_rng(seed)
    return y0 * (1.0 + 1e-3 * rng.standard_normal((len(y0), case["n"])))


# ------------------------------------------------------------------ prepare

def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "cell":
        stim = api.stimulus_desc(0.0, 1000.0, 1.0, 20.0 if case["model"] == "TNNP" else 0.4, 3)
        ion = api.IonicModel(case["model"], TISSUE[case["model"]], case["n"], case["dt"],
                             solve_vm_within_ode=True, ode=api.ode_desc(max_steps=10 ** 6),
                             stimulus=stim)
        ion.set_states(_cell_states(case, seed, ion.states()[:, :1]))
        s.update(ion=ion, t=0.0)
    elif kind == "ionic":
        s.update(ion=api.IonicModel(case["model"], TISSUE[case["model"]], case["n"], case["dt"],
                                    precision=_precision(case),
                                    ode=api.ode_desc(max_steps=10 ** 6)),
                 vm=[_ionic_vm(case["n"], seed, k) for k in range(case["steps"])], t=0.0)
    elif kind == "slab":
        mesh = _box(case["nx"], case["ny"], case["nz"], 20e-3, 7e-3, 3e-3)
        md = api.Monodomain(mesh, case["model"], TISSUE[case["model"]], SIGMA, CHI, CM,
                            dt=case["dt"], precision=_precision(case), boxes=_corner_box())
        md.set_field(lib.FIELD_VM, _vm_field(mesh.centres, seed, 2e-3))
        s.update(md=md, dt=case["dt"])
    elif kind == "lv":
        L = _ventricle(case["nt"], case["m"], case["nr"])
        lo, hi = L.apex_box(2e-3)
        md = api.Monodomain(L.mesh, "TNNP", "epicardialCells", dt=case["dt"],
                            precision=_precision(case), boxes=[(lo, hi, 0.0, 2e-3, 5e4)],
                            tissue_per_cell=L.tissue, conductivity_per_cell=L.conductivity,
                            stencil=False)
        md.set_field(lib.FIELD_VM, _vm_field(L.mesh.centres, seed, 1e-2))
        s.update(md=md, dt=case["dt"])
    elif kind == "niederer":
        mesh, dt = _niederer_case(case)
        md = api.Monodomain(mesh, "BuenoOrovio", "epicardialCells", SIGMA, CHI, CM, dt=dt,
                            implicit=False, boxes=_corner_box())
        md.set_field(lib.FIELD_VM, _vm_field(mesh.centres, seed, 2e-3))
        s.update(md=md, dt=dt)
    elif kind == "batch":
        rng = np.random.default_rng(seed)
        n = case["n"]
        cl, beats = rng.uniform(300.0, 1000.0, n), rng.integers(5, 51, n)
        start = rng.uniform(0.1, 1.0, n)
        s.update(stimuli=[api.stimulus_desc(float(start[c]), float(cl[c]), 1.0, 53.0,
                                            int(beats[c])) for c in range(n)],
                 scales=np.exp(rng.uniform(np.log(0.5), np.log(2.0), (6, n))),
                 end=np.full(n, case["steps"] * case["dt"]))
    elif kind == "bidomain":
        mesh = _cube(case["n"])
        dt = 0.2 / (2.5 * case["n"] ** 2) / 40.0 * 7.0
        V, pe, u1, u2, u3 = _bidomain_start(mesh, seed)
        bd = api.Bidomain(mesh, model="bidomainFDAManufactured", tissue="3D",
                          sigma_i=ver.BIDOMAIN_SIGMA_I, sigma_e=ver.BIDOMAIN_SIGMA_E,
                          chi=ver.CHI, cm=ver.CM, dt=dt, pcg_tol=1e-12, phie_tol=1e-12,
                          phie_max_iter=4000, n_outer=2, ref_point=ver.BIDOMAIN_REF_POINT,
                          grad_scheme=lib.GRAD_GAUSS_LINEAR)
        bd.set_pcg_arithmetic(lib.PCG_FLOAT_PAIRS if case["pairs"] else lib.PCG_FP64)
        bd.set_field(lib.FIELD_VM, V)
        bd.set_field(lib.FIELD_PHIE, pe)
        bd.set_states(np.stack([V, u1, u2, u3]))
        s.update(bd=bd, dt=dt)
    elif kind == "adjoint":
        n, h = case["n"], 2.5e-4
        mesh = box_mesh(n, n, 1, n * h, n * h, h)
        rng = np.random.default_rng(seed)
        a, b = (gaussian_random_field((n, n), h, 5e-3, 0.2, seed + k).ravel() for k in (1, 2))
        p = api.AdjointProblem(mesh, case["steps"], 1e-5, rng.choice(n * n, 64, replace=False),
                               10, checkpoint_every=20,
                               boxes=[((0.0, 0.0, 0.0), (1.5e-3, 1.5e-3, h), 0.0, 2e-3, 5e4)],
                               precision=_precision(case))
        p.set_target(-0.08 + 0.01 * rng.standard_normal((case["steps"] // 10, 64)))
        s.update(problem=p, gna=a, gk1=b)
    elif kind == "ecg":
        L = _ventricle(case["nt"], case["m"], case["nr"])
        ecg = api.PseudoECG(L.mesh, _ecg_points(L, case["electrodes"]),
                            conductivity_per_cell=L.conductivity, max_rows=case["rows"])
        fields = [torch.from_numpy(_vm_field(L.mesh.centres, seed + k, 2e-2)).cuda()
                  for k in range(3)]
        s.update(ecg=ecg, vm=fields)
    elif kind == "purkinje":
        e = _tree(case, seed)
        s.update(pk=api.Purkinje(e, "BuenoOrovio", "epicardialCells", dt=1e-5,
                                 root_stimulus=(0, 0.0, 2e-3, 5e5)))
    return s


# ------------------------------------------------------------------ run

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("slab", "lv", "niederer"):
        md = s["md"]
        md.run(s["dt"], case["steps"])
        return {"vm": _carried(case, md.vm()), "iion": _carried(case, md.iion()),
                "activation": _carried(case, md.activation())}
    if kind == "cell":
        ion, out = s["ion"], []
        im = np.zeros(case["n"])
        for _ in range(case["steps"]):
            ion.solveODE(s["t"], case["dt"], None, im)
            s["t"] += case["dt"]
            out.append(im.copy())
        return {"current": np.array(out), "states": ion.states()}
    if kind == "ionic":
        ion, out = s["ion"], []
        for vm in s["vm"]:
            im = np.zeros(case["n"])
            ion.solveODE(s["t"], case["dt"], vm, im)
            s["t"] += case["dt"]
            out.append(_carried(case, im))
        return out
    if kind == "batch":
        b = api.BatchCells(case["model"], TISSUE[case["model"]], case["dt"], s["stimuli"],
                           s["end"], precision=_precision(case), scales=s["scales"],
                           ode=api.ode_desc(max_steps=10 ** 6))
        b.run()
        beats, apd, t_up, ca = b.results()
        states = b.states()
        b.close()
        return {"beats": beats, "apd": _carried(case, apd), "t_up": _carried(case, t_up),
                "ca": _carried(case, ca), "states": _carried(case, states)}
    if kind == "bidomain":
        bd = s["bd"]
        bd.run(s["dt"], case["steps"])
        return {"vm": bd.vm(), "phie": bd.phie(), "phii": bd.phii()}
    if kind == "adjoint":
        p = s["problem"]
        loss, trace = p.forward(s["gna"], s["gk1"], 0.1334, 0.1334)
        ga, gb, gs = p.backward()
        return {"loss": _carried(case, np.array([loss])), "trace": _carried(case, trace),
                "gna": _carried(case, ga), "gk1": _carried(case, gb), "sigma": _carried(case, gs)}
    if kind == "ecg":
        ecg = s["ecg"]
        ecg.reset()
        for k in range(case["rows"]):
            ecg.record(s["vm"][k % len(s["vm"])], k * 1e-3)
        t, v = ecg.series()
        return {"times": t, "phi": v}
    pk = s["pk"]
    for _ in range(case["steps"]):
        pk.step(1e-5)
    return {"vm": pk.vm(), "iion": pk.iion()}


# ------------------------------------------------------------------ work

def work(case):
    """Inputs read once and outputs written once; operations of the model's
    right-hand sides and, for a field solve, of one matrix product and the
    vector updates of an iteration."""
    kind = case["kind"]
    if kind in ("slab", "niederer", "lv"):
        if kind == "lv":
            n = case["nt"] * (case["m"] ** 2 + 4 * case["m"] * case["nr"]) * 6
            model, evals, its, row = "TNNP", 30, 11, 4 * 24
        else:
            n = case["nx"] * case["ny"] * case["nz"]
            model = case.get("model", "BuenoOrovio")
            evals, its, row = EVALS, (8 if kind == "slab" else 1), 0
        ops, ns = OPS[model]
        word = 4 if case.get("mixed") else 8
        return {"bytes": n * (2 * ns * word + 8 * 8 + row),
                "flops": n * case["steps"] * (evals * ops + its * 28)}
    if kind == "cell":
        ops, ns = OPS[case["model"]]
        return {"bytes": case["n"] * 16 * (ns + case["steps"]),
                "flops": case["n"] * case["steps"] * EVALS * ops}
    if kind == "ionic":
        ops, ns = OPS[case["model"]]
        return {"bytes": case["n"] * (2 * ns * (4 if case["mixed"] else 8) + 16 * case["steps"]),
                "flops": case["n"] * case["steps"] * EVALS * ops}
    if kind == "batch":
        ops, ns = OPS[case["model"]]
        return {"bytes": case["n"] * (8 * ns + 6 * 8 + 56),
                "flops": case["n"] * case["steps"] * EVALS * ops}
    if kind == "bidomain":
        n = case["n"] ** 3
        # about 10 iterations per direction and cell for each of the two solves
        return {"bytes": n * 8 * 8.0, "flops": n * case["steps"] * 2 * 10.0 * case["n"] * 28}
    if kind == "adjoint":
        n = case["n"] ** 2
        # five fixed substeps forward, twice (run and recompute), and the reverse
        return {"bytes": n * 8 * 8.0,
                "flops": n * case["steps"] * OPS["TNNP"][0] * (2 * 31 + 3 * 31)}
    if kind == "ecg":
        n = case["nt"] * (case["m"] ** 2 + 4 * case["m"] * case["nr"]) * 6
        return {"bytes": n * 8.0 * (case["electrodes"] + 3),
                "flops": 2.0 * n * case["electrodes"] * case["rows"]}
    n = case["segment"] * (2 ** (case["depth"] + 1) - 1) + 1
    return {"bytes": n * 8.0 * 12,
            "flops": n * case["steps"] * (2 * EVALS * OPS["BuenoOrovio"][0] + 12)}


# ------------------------------------------------------------------ exact

def _rk4(f, y, t, dt, sub):
    """y(t + dt) of dy/dt = f(t, y) by `sub` classical Runge-Kutta steps: far
    below the solver tolerance of the framework's adaptive steps."""
    h = dt / sub
    for k in range(sub):
        x = t + k * h
        k1 = f(x, y)
        k2 = f(x + 0.5 * h, y + 0.5 * h * k1)
        k3 = f(x + 0.5 * h, y + 0.5 * h * k2)
        k4 = f(x + h, y + h * k3)
        y = y + (h / 6.0) * (k1 + 2.0 * k2 + 2.0 * k3 + k4)
    return y


def _bueno(y, stim=None):
    """Bueno-Orovio, Cherry and Fenton (2008), epicardial cells: rates and
    ionic current of the states u, v, w, s (time in ms)."""
    u, v, w, s = y
    H = lambda x: (x > 0).astype(float)  # noqa: E731
    hv, hw, ho = H(u - 0.3), H(u - 0.13), H(u - 0.006)
    tau_so = 30.0181 + (0.9957 - 30.0181) * (1.0 + np.tanh(2.0458 * (u - 0.65))) / 2.0
    tau_o = (1.0 - ho) * 400.0 + ho * 6.0
    fi = -v * hv * (u - 0.3) * (1.55 - u) / 0.11
    so = u * (1.0 - hw) / tau_o + hw / tau_so
    si = -hw * w * s / 1.8875
    tau_v = (1.0 - ho) * 60.0 + ho * 1150.0
    tau_w = 60.0 + (15.0 - 60.0) * (1.0 + np.tanh(65.0 * (u - 0.03))) / 2.0
    tau_s = (1.0 - hw) * 2.7342 + hw * 16.0
    v_inf = H(0.006 - u)
    w_inf = (1.0 - ho) * (1.0 - u / 0.07) + ho * 0.94
    dv = (1.0 - hv) * (v_inf - v) / tau_v - hv * v / 1.4506
    dw = (1.0 - hw) * (w_inf - w) / tau_w - hw * w / 200.0
    ds = ((1.0 + np.tanh(2.0994 * (u - 0.9087))) / 2.0 - s) / tau_s
    J = fi + so + si
    du = -J - stim if stim is not None else np.zeros_like(u)
    return np.stack([du, dv, dw, ds]), J


TNNP_START = (-86.2, 138.3, 11.6, 0.0002, 0.0, 1.0, 0.0, 0.0, 0.75, 0.75, 0.0, 1.0, 1.0, 1.0,
              0.0, 0.2, 1.0)


def _tnnp(y, stim=None):
    """ten Tusscher, Noble, Noble and Panfilov (2004), epicardial cells, in
    the framework's order of states: rates and membrane current (time in ms)."""
    V, Ki, Nai, Cai, xr1, xr2, xs, m, h, j, d, f, fca, s, r, casr, g = y
    E = np.exp
    RTF, cm, vc, F = 8.314 * 310.0 / 96.485, 185.0, 16404.0, 96.485
    low = V < -40.0
    gate = lambda x, inf, tau: (inf - x) / tau  # noqa: E731
    dm = gate(m, 1 / (1 + E((-56.86 - V) / 9.03)) ** 2, 1 / (1 + E((-60 - V) / 5)) *
              (0.1 / (1 + E((V + 35) / 5)) + 0.1 / (1 + E((V - 50) / 200))))
    hj = 1 / (1 + E((V + 71.55) / 7.43)) ** 2
    ah = np.where(low, 0.057 * E(-(V + 80) / 6.8), 0.0)
    bh = np.where(low, 2.7 * E(0.079 * V) + 310000.0 * E(0.3485 * V),
                  0.77 / (0.13 * (1 + E((V + 10.66) / -11.1))))
    aj = np.where(low, (-25428.0 * E(0.2444 * V) - 6.948e-6 * E(-0.04391 * V)) * (V + 37.78) /
                  (1 + E(0.311 * (V + 79.23))), 0.0)
    bj = np.where(low, 0.02424 * E(-0.01052 * V) / (1 + E(-0.1378 * (V + 40.14))),
                  0.6 * E(0.057 * V) / (1 + E(-0.1 * (V + 32))))
    dh, dj = (hj - h) * (ah + bh), (hj - j) * (aj + bj)
    dd = gate(d, 1 / (1 + E((-5 - V) / 7.5)), (1.4 / (1 + E((-35 - V) / 13)) + 0.25) * 1.4 /
              (1 + E((V + 5) / 5)) + 1 / (1 + E((50 - V) / 20)))
    df = gate(f, 1 / (1 + E((V + 20) / 7)),
              1125 * E(-(V + 27) ** 2 / 240) + 80 + 165 / (1 + E((25 - V) / 10)))
    ds = gate(s, 1 / (1 + E((V + 20) / 5)),
              85 * E(-(V + 45) ** 2 / 320) + 5 / (1 + E((V - 20) / 5)) + 3)
    dr = gate(r, 1 / (1 + E((20 - V) / 6)), 9.5 * E(-(V + 40) ** 2 / 1800) + 0.8)
    dxr1 = gate(xr1, 1 / (1 + E((-26 - V) / 7)),
                450 / (1 + E((-45 - V) / 10)) * 6 / (1 + E((V + 30) / 11.5)))
    dxr2 = gate(xr2, 1 / (1 + E((V + 88) / 24)),
                3 / (1 + E((-60 - V) / 20)) * 1.12 / (1 + E((V - 60) / 20)))
    dxs = gate(xs, 1 / (1 + E((-5 - V) / 14)),
               1100 / np.sqrt(1 + E((-10 - V) / 6)) / (1 + E((V - 60) / 20)))
    fca_inf = (1 / (1 + (Cai / 0.000325) ** 8) + 0.1 / (1 + E((Cai - 0.0005) / 0.0001)) +
               0.2 / (1 + E((Cai - 0.00075) / 0.0008)) + 0.23) / 1.46
    dfca = np.where((fca_inf > fca) & (V > -60.0), 0.0, (fca_inf - fca) / 2.0)
    q = Cai / 0.00035
    g_inf = np.where(Cai < 0.00035, 1 / (1 + q ** 6), 1 / (1 + q ** 16))
    dg = np.where((g_inf > g) & (V > -60.0), 0.0, (g_inf - g) / 2.0)
    Ena, Ek = RTF * np.log(140.0 / Nai), RTF * np.log(5.4 / Ki)
    Eks, Eca = (RTF * np.log((5.4 + 0.03 * 140) / (Ki + 0.03 * Nai)),
                0.5 * RTF * np.log(2.0 / Cai))
    v = V / RTF
    nak = 1.362 * 5.4 / 6.4 * Nai / (Nai + 40) / (1 + 0.1245 * E(-0.1 * v) + 0.0353 * E(-v))
    ina, ibna = 14.838 * m ** 3 * h * j * (V - Ena), 0.00029 * (V - Ena)
    naca = (1000 * (E(0.35 * v) * Nai ** 3 * 2 - E(-0.65 * v) * 140.0 ** 3 * Cai * 2.5) /
            ((87.5 ** 3 + 140.0 ** 3) * (1.38 + 2) * (1 + 0.1 * E(-0.65 * v))))
    ak1 = 0.1 / (1 + E(0.06 * (V - Ek - 200)))
    bk1 = (3 * E(0.0002 * (V - Ek + 100)) + E(0.1 * (V - Ek - 10))) / (1 + E(-0.5 * (V - Ek)))
    ik1 = 5.405 * ak1 / (ak1 + bk1) * (V - Ek)
    ito, ikr = 0.294 * r * s * (V - Ek), 0.096 * xr1 * xr2 * (V - Ek)
    iks = 0.245 * xs ** 2 * (V - Eks)
    ical = (0.175 * d * f * fca * 4 * v * F * (Cai * E(2 * v) - 0.341 * 2) / np.expm1(2 * v))
    ibca, ipk = 0.000592 * (V - Eca), 0.0146 * (V - Ek) / (1 + E((25 - V) / 5.98))
    ipca = 0.825 * Cai / (Cai + 0.0005)
    total = (ik1 + ito + ikr + iks + ical + nak + ina + ibna + naca + ibca + ipk + ipca)
    ist = stim if stim is not None else 0.0
    dNa = -(ina + ibna + 3 * nak + 3 * naca) * cm / (vc * F)
    dK = -(ik1 + ito + ikr + iks + ipk + ist - 2 * nak) * cm / (vc * F)
    rel = (0.016464 * casr ** 2 / (0.25 ** 2 + casr ** 2) + 0.008232) * d * g
    up, leak = 0.000425 / (1 + 0.00025 ** 2 / Cai ** 2), 8e-5 * (casr - Cai)
    dCa = ((-(ical + ibca + ipca - 2 * naca) / (2 * vc * F) * cm + leak - up + rel) /
           (1 + 0.15 * 0.001 / (Cai + 0.001) ** 2))
    dSR = vc / 1094 * (up - (rel + leak)) / (1 + 10 * 0.3 / (casr + 0.3) ** 2)
    dV = -total - ist if stim is not None else np.zeros_like(V)
    return np.stack([dV, dK, dNa, dCa, dxr1, dxr2, dxs, dm, dh, dj, dd, df, dfca, ds, dr, dSR,
                     dg]), total


def _box_laplacian(case, h, vol):
    """V -> V_c div(sigma grad V) on the uniform box, zero-gradient walls."""
    shape = (case["nz"], case["ny"], case["nx"])
    coef = [SIGMA[5] * vol / h[2] ** 2, SIGMA[3] * vol / h[1] ** 2, SIGMA[0] * vol / h[0] ** 2]

    def lap(v):
        v = v.reshape(shape)
        out = np.zeros(shape)
        for ax in range(3):
            d = coef[ax] * np.diff(v, axis=ax)
            lo = [slice(None)] * 3
            hi = [slice(None)] * 3
            lo[ax], hi[ax] = slice(0, -1), slice(1, None)
            out[tuple(lo)] += d
            out[tuple(hi)] -= d
        return out.ravel()
    return lap


def _conjugate_gradient(A, b, x):
    r = b - A(x)
    p, rr, stop = r, r @ r, 1e-30 * (b @ b)
    for _ in range(500):
        if rr <= stop:
            break
        q = A(p)
        al = rr / (p @ q)
        x, r = x + al * p, r - al * q
        rn = r @ r
        p, rr = r + rn / rr * p, rn
    return x


def _tissue_exact(case, seed, mesh, dt, implicit, model, y, to_state, scale, sub):
    h = (20e-3 / case["nx"], 7e-3 / case["ny"], 3e-3 / case["nz"])
    vol = h[0] * h[1] * h[2]
    lap = _box_laplacian(case, h, vol)
    vm = _vm_field(mesh.centres, seed, 2e-3)
    box = (mesh.centres <= 1.5e-3).all(axis=1)
    old, oldold, chicm, t = vm, vm, CHI * CM, 0.0
    for k in range(case["steps"]):
        oldold, old = (old, vm) if k else (vm, vm)
        y[0] = to_state(old)
        y = _rk4(lambda _, q: model(q)[0], y, 0.0, dt * 1000.0, sub)
        iion = scale * model(y)[1]
        src = np.where(box & (t <= 2e-3), 5e4, 0.0)
        if implicit or k:
            c, c0, c00 = 1.5, 2.0, 0.5
        else:
            c, c0, c00 = 1.0, 1.0, 0.0
        rhs = chicm * vol * (c0 * old - c00 * oldold) / dt + (src - chicm * iion) * vol
        diag = chicm * vol * c / dt
        vm = (_conjugate_gradient(lambda x: diag * x - lap(x), rhs, old) if implicit
              else (rhs + lap(old)) / diag)
        t += dt
    return {"vm": vm, "iion": iion, "activation": None}


def _ecg_exact(case, seed):
    L = _ventricle(case["nt"], case["m"], case["nr"])
    m, n = L.mesh, L.mesh.n_cells
    P, N, C = m.owner, m.neighbour, m.centres
    d = C[N] - C[P]
    k = 1.0 / (d * d).sum(axis=1)
    nb = m.boundary_sf / np.linalg.norm(m.boundary_sf, axis=1)[:, None]
    db = nb * (nb * (m.boundary_centres - C[m.boundary_cell])).sum(axis=1)[:, None]
    kb = 1.0 / (db * db).sum(axis=1)
    add = lambda at, w: np.bincount(at, w, n)  # noqa: E731
    dd = np.zeros((n, 3, 3))
    for a in range(3):
        for b in range(3):
            w = k * d[:, a] * d[:, b]
            dd[:, a, b] = add(P, w) + add(N, w) + add(m.boundary_cell, kb * db[:, a] * db[:, b])
    inv = np.linalg.inv(dd)
    g = L.conductivity
    full = g[:, [0, 1, 2, 1, 3, 4, 2, 4, 5]].reshape(n, 3, 3)
    pts = _ecg_points(L, case["electrodes"])
    rows = []
    for q in range(3):
        v = _vm_field(C, seed + q, 2e-2)
        w = k * (v[N] - v[P])
        rhs = np.stack([add(P, w * d[:, a]) + add(N, w * d[:, a]) for a in range(3)], axis=1)
        dip = (full @ (inv @ rhs[:, :, None]))[:, :, 0] * m.volumes[:, None]
        r = C[None] - pts[:, None]
        rows.append(((dip[None] * r).sum(axis=2) / np.linalg.norm(r, axis=2) ** 3).sum(axis=1))
    count = case["rows"]
    return {"times": np.arange(count) * 1e-3, "phi": np.array([rows[i % 3] for i in range(count)])}


def _purkinje_exact(case, seed):
    e = _tree(case, seed)
    a, b = e[:, 0].astype(int), e[:, 1].astype(int)
    n, dt, chicm = max(a.max(), b.max()) + 1, 1e-5, CHI * CM
    if n > 2500:
        return None
    length = np.bincount(a, 0.5 * e[:, 2], n) + np.bincount(b, 0.5 * e[:, 2], n)
    A = np.eye(n)
    c = dt * e[:, 3] / e[:, 2] / chicm
    np.add.at(A, (a, a), c / length[a])
    np.add.at(A, (b, b), c / length[b])
    A[a, b] -= c / length[a]
    A[b, a] -= c / length[b]
    inv = np.linalg.inv(A)
    y = np.tile(np.array([0.0, 1.0, 1.0, 0.0])[:, None], (1, n))
    vm, iion = np.full(n, -0.084), None

    def ionic():
        nonlocal y
        y[0] = (vm * 1000.0 + 84.0) / 85.7
        y = _rk4(lambda _, q: _bueno(q)[0], y, 0.0, dt * 500.0, 4)
        return 85.7 * _bueno(y)[1]

    for _ in range(case["steps"]):
        iion = ionic()
        rhs = vm - dt * iion
        rhs[0] += dt * 5e5 / chicm
        vm = inv @ rhs
        iion = ionic()
    return {"vm": vm, "iion": iion}


def _cell_exact(case, seed):
    tn = case["model"] == "TNNP"
    model, amp = (_tnnp, 20.0) if tn else (_bueno, 0.4)
    y0 = np.array(TNNP_START if tn else (0.0, 1.0, 1.0, 0.0))[:, None]
    y, out = _cell_states(case, seed, y0), []
    sub = 100 if tn else 8
    for _ in range(case["steps"]):
        y = _rk4(lambda _, q: model(q, -amp)[0], y, 0.0, case["dt"] * 1000.0, sub)
        out.append((1.0 if tn else 85.7) * model(y)[1])
    return {"current": np.array(out), "states": y}


def exact(case, seed):
    kind = case["kind"]
    if kind == "cell":
        return _cell_exact(case, seed)
    if kind == "purkinje":
        return _purkinje_exact(case, seed)
    if kind == "ecg":
        return _ecg_exact(case, seed)
    if kind == "niederer":
        mesh, dt = _niederer_case(case)
        y = np.tile(np.array([0.0, 1.0, 1.0, 0.0])[:, None], (1, mesh.n_cells))
        return _tissue_exact(case, seed, mesh, dt, False, _bueno, y,
                             lambda v: (v * 1000.0 + 84.0) / 85.7, 85.7, 4)
    if kind == "slab" and case["model"] == "TNNP" and case["nx"] <= 50 and not case["mixed"]:
        mesh = _box(case["nx"], case["ny"], case["nz"], 20e-3, 7e-3, 3e-3)
        y = np.tile(np.array(TNNP_START)[:, None], (1, mesh.n_cells))
        return _tissue_exact(case, seed, mesh, case["dt"], True, _tnnp, y,
                             lambda v: v * 1000.0, 1.0, 60)
    return None     # models of 40 states, and solves of hundreds of iterations
