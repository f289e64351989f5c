"""The work that a user of this framework has it do, as cases that can be timed.

A case marches one turbomachine (or a batch of them) some LOOP iterations
from its deck's initial guess on, reports its performance, or differentiates
one step of it, through the Python binding of the C ABI (mgpu.lib): the
machines are the nozzle row, the single-stage turbine and the four-stage
compressor that the benchmark and the tests use, at their sizes and at others.
A seed sets the operating point (inlet stagnation pressure and temperature,
exit static pressure); the blades and the grid belong to the case.
"""
import copy
import functools
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "multall-open-18.3_gb300"))
from mgpu import case as mcase  # noqa: E402
from mgpu import common_setup, lib  # noqa: E402

STATE = ("RO", "ROVX", "ROVR", "RORVT", "ROE")
# a LOOP iteration reads and writes five conserved variables and their SCREE
# histories and reads nine geometry arrays and four body forces, FP32
STEP_BYTES, STEP_FLOPS = 132, 700
# a transposed step: fourteen adjoint arrays read and written, and the same
# geometry and the thirteen recorded arrays read
ADJ_BYTES, ADJ_FLOPS = 200, 1500


def listed():
    def c(name, kind, machine, im, jm, km, steps, ilos=10, order=0, members=1):
        return {"name": name, "kind": kind, "machine": machine, "im": im, "jm": jm, "km": km, "steps": steps,
                "ilos": ilos, "order": order, "members": members}

    return [
        # a teaching-size row driven one mgpu_step at a time with its monitors,
        # as a Fortran LOOP calls the library: launches and latency
        c("step_row_small", "step", "row", 9, 29, 7, 10),
        # the tests' small stage, marched
        c("march_stage_small", "march", "stage", 9, 25, 7, 50),
        # the nozzle row of the benchmark configurations
        c("march_row", "march", "row", 37, 97, 33, 50),
        # the headline stage, J per row
        c("march_stage", "march", "stage", 65, 121, 49, 25),
        # plain FP32 sums on a ragged grid
        c("march_stage_plain", "march", "stage", 50, 83, 38, 25, order=2),
        # the other two viscous models
        c("march_stage_newloss", "march", "stage", 43, 69, 35, 25, ilos=100),
        c("march_stage_sa", "march", "stage", 49, 81, 41, 25, ilos=200),
        # eight rows, the largest grid
        c("march_compressor", "march", "compressor", 73, 89, 57, 25),
        # 64 operating points on eight grids of uneven size in one graph
        c("batch_64", "batch", "stage", 0, 0, 0, 10, members=64),
        # the efficiency report of a running stage
        c("report_stage", "report", "stage", 65, 121, 49, 0),
        # gradients of the efficiency: record, seed, iterate, geometry pass
        c("adjoint_stage", "adjoint", "stage", 65, 121, 49, 25),
        c("adjoint_row_small", "adjoint", "row", 21, 61, 17, 25),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(("march", "march", "march", "march", "step", "batch", "report", "adjoint"))
    machine = rng.choice(("row", "stage", "stage", "stage"))
    c = {"kind": kind, "machine": machine, "im": size(9, 73), "jm": size(49, 140), "km": size(9, 57),
         "steps": 5 * size(2, 8), "ilos": rng.choice((10, 10, 10, 100, 200)), "order": rng.choice((0, 0, 0, 2)),
         "members": 1}
    if c["ilos"] >= 100:
        # the eddy-viscosity models are run on grids that resolve the passage
        c.update(im=size(31, 61), jm=size(57, 121), km=size(31, 49))
    if c["machine"] == "stage" and 18 <= c["km"] <= 26:
        # a span of 18 to 26 points puts a single cell in the rotor's tip gap,
        # and a long march of some such stages ends in a non-finite field
        c["km"] += 9
    if kind == "march" and rng.random() < 0.15:
        c.update(machine="compressor", im=size(17, 41), jm=89, km=size(13, 29), ilos=10)
    if kind == "step":
        c.update(steps=size(5, 20))
    if kind == "batch":
        c.update(machine="stage", im=0, jm=rng.randrange(1000), km=0, steps=5, ilos=10, members=size(3, 40))
    if kind == "report":
        c.update(machine="stage", steps=0, ilos=10)
    if kind == "adjoint":
        c.update(ilos=10)
    return c


def _spec(c):
    if c["machine"] == "row":
        jm = c["jm"]
        if jm < 40:
            spec = mcase.small_nozzle(im=c["im"], jm=jm, km=c["km"])
        else:
            spec = mcase.nozzle_row(im=c["im"], jm=jm, km=c["km"], jle=round(jm * 18 / 97), jte=round(jm * 74 / 97))
    elif c["machine"] == "compressor":
        spec = mcase.compressor_4stage(im=c["im"], jm_row=c["jm"], km=c["km"])
    elif c["jm"] < 40:
        spec = mcase.small_stage(im=c["im"], jm_row=c["jm"], km=c["km"])
    else:
        spec = mcase.turbine_stage(im=c["im"], jm_row=c["jm"], km=c["km"])
    spec.ilos = c["ilos"]
    return spec


@functools.lru_cache(maxsize=12)
def _machine(machine, im, jm, km, ilos):
    return common_setup.build_common(_spec({"machine": machine, "im": im, "jm": jm, "km": km, "ilos": ilos}))


@functools.lru_cache(maxsize=12)
def _member(number):
    return common_setup.build_common(mcase.batch_instance(number))


def _operating_point(base, rng, order):
    """The machine's deck at an operating point near its design point."""
    cd = copy.copy(base)
    cd.ints, cd.reals, cd.arrays = dict(base.ints), dict(base.reals), dict(base.arrays)
    po, to, pe = 1.0 + 0.004 * rng.uniform(-1, 1), 1.0 + 0.01 * rng.uniform(-1, 1), 1.0 + 0.01 * rng.uniform(-1, 1)
    cd.arrays["PO1"] = (base.arrays["PO1"] * po).astype(np.float32)
    cd.arrays["RPO1"] = (1.0 / cd.arrays["PO1"]).astype(np.float32)
    cd.arrays["TO1"] = (base.arrays["TO1"] * to).astype(np.float32)
    cd.arrays["PD"] = (base.arrays["PD"] * pe).astype(np.float32)
    for n in ("PDOWN_HUB", "PDOWN_TIP"):
        cd.reals[n] = base.reals[n] * pe
    # a long march: neither the step limit nor the convergence test ends it
    cd.ints["NSTEPS_MAX"], cd.reals["CONLIM"] = 10 ** 9, 1e-9
    cd.ints["REDUCE_ORDER"] = order
    return cd


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "batch":
        # jm numbers the first of the eight machines that the members share
        bases = [_member(8 * case["jm"] + m) for m in range(min(8, case["members"]))]
        decks = [_operating_point(bases[m % len(bases)], rng, case["order"]) for m in range(case["members"])]
    else:
        base = _machine(case["machine"], case["im"], case["jm"], case["km"], case["ilos"])
        decks = [_operating_point(base, rng, case["order"])]
    problems = [lib.Problem(cd) for cd in decks]
    nodes = [p.cd.im * p.cd.jm * p.cd.km for p in problems]
    s = {"kind": kind, "steps": case["steps"], "problems": problems}
    # the flow state comes back into pinned host buffers that the program keeps
    names = STATE + (("TRANS_DYN_VIS",) if case["ilos"] >= 200 else ())
    s["out"] = {n: torch.zeros(sum(nodes), pin_memory=True) for n in names}
    at = np.concatenate([[0], np.cumsum(nodes)])
    s["view"] = {n: [t.numpy()[at[m]:at[m + 1]] for m in range(len(nodes))] for n, t in s["out"].items()}
    if kind == "batch":
        s["batch"] = lib.Batch(problems)
    if kind == "report":
        problems[0].run(25)
    if kind == "adjoint":
        problems[0].run(200)
    return s


def run(state):
    kind, p = state["kind"], state["problems"][0]
    if kind == "report":
        i, g = p.integrals(), p.stage(1)
        return {"flow_in": i.mass_flow_in, "flow_out": i.mass_flow_out, "eta_tt": i.eta_tt, "eta_ts": i.eta_ts,
                "po_ratio": i.po_ratio, "to_ratio": i.to_ratio, "stage_po_ratio": g.po_ratio,
                "stage_eta_tt": g.eta_tt, "stage_eta_poly": g.eta_poly}
    if kind == "adjoint":
        p.adjoint_prepare()
        value = p.adjoint_objective("eta_tt")
        p.adjoint_iterate(state["steps"])
        return {"value": value, "gradient": p.adjoint_gradient(), "theta": p.adjoint_gradient_theta(),
                "adjoint": {n: p.adjoint_get(n) for n in STATE}}
    if kind == "batch":
        _, mons = state["batch"].run(state["steps"])
        flow = [v for m in mons for v in (m.flow_in, m.flow_out)]
    elif kind == "step":
        flow = []
        for _ in range(state["steps"]):
            m = p.step()
            flow += [m.flow_in, m.flow_out]
        flow = flow[-10:]
    else:
        _, m = p.run(state["steps"])
        flow = [m.flow_in, m.flow_out]
    for n, views in state["view"].items():
        for q, v in zip(state["problems"], views):
            q.get_into(n, v)
    return {"state": state["out"], "flow": np.array(flow, np.float32)}


def work(case):
    if case["kind"] == "batch":
        specs = [mcase.batch_instance(8 * case["jm"] + m % 8) for m in range(case["members"])]
        nodes = sum(s.im * sum(r.jm for r in s.rows) * s.km for s in specs)
    else:
        spec = _spec(case)
        nodes = spec.im * sum(r.jm for r in spec.rows) * spec.km
    if case["kind"] == "report":
        return {"bytes": 28 * nodes, "flops": 60 * nodes}
    if case["kind"] == "adjoint":
        n = case["steps"] + 1
        return {"bytes": nodes * (n * ADJ_BYTES + STEP_BYTES), "flops": nodes * (n * ADJ_FLOPS + STEP_FLOPS)}
    return {"bytes": case["steps"] * STEP_BYTES * nodes, "flops": case["steps"] * STEP_FLOPS * nodes}


def exact(case, seed):
    """The performance report in 64 bits; a march and an adjoint have no
    independent 64-bit value that is quick to form."""
    if case["kind"] != "report":
        return None
    p = prepare(case, seed)["problems"][0]
    cd = p.cd
    vx, vr, vt, ho, pr, flow = (p.get(n).astype(np.float64) for n in ("VX", "VR", "VT", "HO", "P", "FLOWX"))
    cp, ga = np.float64(np.float32(cd.reals["CP"])), np.float64(np.float32(cd.reals["GA"]))
    fga = (ga - 1.0) / ga
    kmid = int(0.5 * cd.km) - 1
    po1, to1 = np.float64(cd.arrays["PO1"][kmid]), np.float64(cd.arrays["TO1"][kmid])
    # per node: stagnation temperature and pressure, with the floors that the
    # report applies
    tstag = np.maximum(ho / cp, 0.1 * to1)
    tstat = np.maximum((ho - 0.5 * (vx * vx + vr * vr + vt * vt)) / cp, 0.1 * to1)
    pstag = np.maximum(pr, 0.02 * po1) * (tstag / tstat) ** (1.0 / fga)

    def station(j):                       # 1-based: mass flow and mass-averaged PO, TO and P
        w = -flow[:-1, j - 1, :-1] * np.float64(cd.arrays["NBLADE"][j - 1])

        def mean(a):
            a = a[:, j - 1, :]
            return float((w * 0.25 * (a[:-1, :-1] + a[:-1, 1:] + a[1:, 1:] + a[1:, :-1])).sum() / w.sum())

        return float(w.sum()), mean(pstag), mean(tstag), mean(pr)

    f1, p1, t1, _ = station(1 if cd.ints["NSTAGES"] == 1 else 2)
    f2, p2, t2, ps2 = station(cd.jm - 1)

    def efficiency(pratio):
        ideal, actual = t1 * (pratio ** fga - 1.0), t2 - t1
        return ideal / actual if actual > 0.0 else actual / ideal if actual < 0.0 else 1.0

    poly = np.log(t2 / t1) / np.log(p2 / p1) / fga
    poly = 1.0 / poly if t2 > t1 else poly
    # a single stage's own stations are the machine's
    eta = efficiency(max(p2 / p1, 0.01))
    return {"flow_in": f1, "flow_out": f2, "eta_tt": eta, "eta_ts": efficiency(ps2 / p1), "po_ratio": p2 / p1,
            "to_ratio": t2 / t1, "stage_po_ratio": p2 / p1, "stage_eta_tt": eta, "stage_eta_poly": poly}
