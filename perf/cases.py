"""The work that users of this package have it do, as cases that can be timed and compared.

Three public paths, each over the range of sizes it is used at:
  run   ``GreensteinWinslow.run``: one call simulates one cell from host arrays to host records, as
        the reference's Python does (FP64 by default, FP32 for production).
  ens   ``gwgb300.Ensemble.run``: the next stretch of an ensemble that the program keeps on the
        device, with the records it asked for.
  grad  one step of a parameter fit: the voltage trace of every cell and the gradient of a loss of
        it, through ``GradEngine`` (kept over the fit) or ``VoltageTrace`` (torch autograd).

Cells start in one of three phases of the paced beat.  The globals and the CRUs' channel occupancies
and Ca quantiles of "release" and "plateau" are those of a 1,250-CRU cell 20 and 120 ms after the
stimulus; "rest" is the reference's initial state with the stimulus at t = 0.

``exact`` restates the model in 64-bit torch (float64 state, the same counter-based draws), and for
the fits differentiates it with torch autograd on the frozen jump trajectory.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "gw-model_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import GreensteinWinslow as GW  # noqa: E402
from gwgb300 import engine  # noqa: E402
from gwgb300.adjoint import GradEngine, TraceSpec, VoltageTrace, scaled_params  # noqa: E402

DT = 1e-3             # global step [ms]
PULSE = (0.0, 0.0, 0.5, 100.0)  # stimulus start, period, duration, amplitude

# ------------------------------------------------------------------------------------------
# The model's parameters and the three phases.
# ------------------------------------------------------------------------------------------
PARAMS = dict(
    T=310.0, CSA=153.4, Vcyto=25.84, VNSR=1.113, VJSR=22.26e-6, VSS=0.2303e-6, NCaRU=12500, Ko=4.0, Nao=138.0,
    Cao=2.0, Clo=150.0, Clcyto=20.0, f=0.85, g=2.0, f1=0.005, g1=7.0, a=2.0, b=1.9356, gamma0=0.44, omega=0.02158,
    PCaL=9.13e-13, kfClCh=13.3156, kbClCh=2.0, Pto2=2.65e-15, k12=877.5, k21=250.0, k23=2.358e8, k32=9.6,
    k34=1.415e6, k43=13.65, k45=0.07, k54=93.385, k56=1.887e7, k65=30.0, k25=2.358e6, k52=0.001235, rRyR=3.92,
    rxfer=200.0, rtr=0.333, riss=20.0, BSRT=0.047, KBSR=0.00087, BSLT=1.124, KBSL=0.0087, CSQNT=13.5, KCSQN=0.63,
    CMDNT=0.05, KCMDN=0.00238, GNa=12.8, GKr=0.024, Kf=0.0266, Kb=0.1348, GKs=0.00271, GKv43=0.1389,
    alphaa0Kv43=0.5437, aaKv43=0.02898, betaa0Kv43=0.08019, baKv43=0.04684, alphai0Kv43=0.04984, aiKv43=3.37302e-4,
    betai0Kv43=8.1948e-4, biKv43=5.374e-8, f1Kv43=1.8936, f2Kv43=14.225, f3Kv43=158.574, f4Kv43=142.937,
    b1Kv43=6.7735, b2Kv43=15.621, b3Kv43=28.753, b4Kv43=524.576, PKv14=1.989e-7, alphaa0Kv14=1.8931,
    aaKv14=0.006950, betaa0Kv14=0.01179, baKv14=0.08527, alphai0Kv14=0.002963, aiKv14=0.0, betai0Kv14=1.0571e-4,
    biKv14=0.0, f1Kv14=0.2001, f2Kv14=0.3203, f3Kv14=13.509, f4Kv14=1151.765, b1Kv14=2.230, b2Kv14=12.0,
    b3Kv14=5.370, b4Kv14=5.240, Csc=1.0e6, GK1=3.0, KmK1=13.0, GKp=0.002659, kNaCa=0.27, KmNa=87.5, KmCa=1.38,
    ksat=0.2, eta=0.35, INaKmax=0.901, KmNai=10.0, KmKo=1.5, IpCamax=0.03, KmpCa=0.0005, GCab=0.0002536,
    GNab=0.00264, kHTRPNp=20.0, kHTRPNm=6.60e-5, kLTRPNp=40.0, kLTRPNm=0.04, HTRPNtot=0.140, LTRPNtot=0.070,
    Vmaxf=0.0002096, Vmaxr=0.0002096, Kmf=0.000260, Kmr=1.8, Hf=0.75, Hr=0.75)

# V, Nai, Ki, Cai, CaNSR, CaLTRPN, CaHTRPN, m, h, j, xKs, Kr[5], Kv43[10], Kv14[10]
GLOBALS = {
    "rest": [-91.382, 10.0, 131.84, 1.45273e-4, 0.908882, 8.9282e-3, 0.137617, 5.33837e-4, 0.996345, 0.997315,
             2.04171e-4, 0.999503, 4.13720e-4, 7.27568e-5, 8.73984e-6, 1.36159e-6, 0.953060, 0.0253906, 2.53848e-4,
             1.12796e-6, 1.87950e-9, 0.0151370, 0.00517622, 8.96600e-4, 8.17569e-5, 2.24032e-6, 0.722328, 0.101971,
             0.00539932, 1.27081e-4, 1.82742e-6, 0.152769, 0.00962328, 0.00439043, 0.00195348, 0.00143629],
    "release": [-3.7155, 10.0039, 131.835, 4.02258e-4, 0.881251, 0.0124178, 0.137661, 0.992079, 1.62797e-47, 0.0037773,
                0.0102443, 0.886991, 0.0966165, 0.0135658, 0.0019791, 8.47614e-4, 1.28724e-4, 0.00241111, 0.0165456,
                0.0483376, 0.0580828, 3.32196e-8, 6.57902e-6, 7.03505e-4, 0.0403787, 0.833405, 6.49141e-10,
                2.87313e-7, 4.74354e-5, 0.00344368, 0.0907773, 9.39219e-13, 1.89215e-10, 2.77791e-7, 3.87611e-4,
                0.905343],
    "plateau": [8.94974, 9.99824, 131.835, 7.71387e-4, 0.656815, 0.0305527, 0.138975, 0.998037, 0.0, 6.20314e-16,
                0.0597608, 0.591685, 0.269997, 0.0441698, 0.020248, 0.0738998, 2.33677e-8, 1.26598e-6, 2.57249e-5,
                2.32381e-4, 7.85381e-4, 4.03245e-10, 2.7711e-7, 9.68455e-5, 0.0178409, 0.981017, 2.49781e-13,
                3.68447e-10, 2.03809e-7, 5.01062e-5, 0.00461952, 8.91942e-15, 5.85152e-12, 2.77432e-8, 1.29731e-4,
                0.9952],
}
QUANTILES = [0.0, 0.01, 0.1, 0.25, 0.5, 0.75, 0.9, 0.99, 1.0]
CRUS = {
    "rest": dict(LCC=[0.958, 0.038, 0, 0, 0, 0, 0.004, 0, 0, 0, 0, 0], gate=0.9425, clch=0.002,
                 RyR=[0.609, 0, 0, 0, 0.1955, 0.1955]),
    "release": dict(LCC=[0.0090, 0.0722, 0.2262, 0.2796, 0.1496, 0.0602, 0.0, 0.0012, 0.0138, 0.0656, 0.1224, 0.0002],
                    gate=0.8782, clch=0.0518, RyR=[0.4171, 0.0, 0.0139, 0.1032, 0.2683, 0.1975],
                    CaSS=[3.88e-4, 3.891e-4, 3.977e-4, 5.794e-4, 2.482e-3, 0.01411, 0.02856, 0.05163, 0.0729],
                    CaJSR=[0.53, 0.5752, 0.6732, 0.7512, 0.8354, 0.9022, 0.9022, 0.9022, 0.9023]),
    "plateau": dict(LCC=[0.0004, 0.0034, 0.0274, 0.0976, 0.0914, 0.0414, 0.0, 0.0006, 0.0086, 0.1480, 0.5810, 0.0002],
                    gate=0.6862, clch=0.0146, RyR=[0.1609, 0.0, 0.0009, 0.0138, 0.6269, 0.1975],
                    CaSS=[7.717e-4, 7.718e-4, 7.718e-4, 7.719e-4, 7.756e-4, 1.040e-3, 2.411e-3, 0.01854, 0.04396],
                    CaJSR=[0.45, 0.5061, 0.5821, 0.6190, 0.6465, 0.6557, 0.6593, 0.6611, 0.6612]),
}
VARIED = ("PCaL", "GKr", "GKs", "Vmax", "rRyR")  # log-normal between the cells of an ensemble


# ------------------------------------------------------------------------------------------
# Cases.
# ------------------------------------------------------------------------------------------
def _run(name, ncru, steps, every, precision, phase):
    return dict(name=name, kind="run", ncru=ncru, steps=steps, every=every, precision=precision, phase=phase)


def _ens(name, cells, lo, hi, steps, every, precision, phase, sums=False, codec=False, cluster=0):
    return dict(name=name, kind="ens", cells=cells, lo=lo, hi=hi, steps=steps, every=every, precision=precision,
                phase=phase, sums=sums, codec=codec, cluster=cluster)


def _grad(name, cells, lo, hi, steps, sample, checkpoint, phase, autograd):
    return dict(name=name, kind="grad", cells=cells, lo=lo, hi=hi, steps=steps, sample=sample, checkpoint=checkpoint,
                phase=phase, autograd=autograd)


def listed():
    return [
        # a try-out of the reference's API: a few CRUs for a fraction of a millisecond, in its arithmetic
        _run("run_fp64_64", 64, 300, 30, "fp64", "rest"),
        # the reference's own size (1,250 CRUs standing for 12,500) in its arithmetic, amid the release
        _run("run_fp64_1250", 1250, 500, 100, "fp64", "release"),
        # a small odd cell, as for a parameter scan by single calls
        _run("run_fp32_777", 777, 2000, 250, "fp32", "plateau"),
        # the full-size cell, production precision: the upstroke, and the Ca release
        _run("run_fp32_12500_rest", 12500, 1000, 333, "fp32", "rest"),
        _run("run_fp32_12500_release", 12500, 1000, 333, "fp32", "release"),
        # the reference-arithmetic ensemble: eight cells of very different sizes
        _ens("ens_fp64_8", 8, 5, 1200, 200, 50, "fp64", "plateau"),
        # a population of mid-size cells with currents' sums and one cell's CRUs recorded often
        _ens("ens_fp32_24_records", 24, 500, 3000, 1000, 20, "fp32", "release", sums=True, codec=True),
        # 256 mixed cells amid their Ca release (launch shape as the autotuner picks it)
        _ens("ens_fp32_256", 256, 2000, 12500, 100, 50, "fp32", "release", sums=True, cluster=6),
        # 1,024 full-size cells paced from rest
        _ens("ens_fp32_1024", 1024, 12500, 12500, 50, 25, "fp32", "rest", cluster=6),
        # one iteration of a fit of three small cells through torch autograd
        _grad("grad_autograd_3", 3, 180, 420, 200, 20, 200, "rest", True),
        # one iteration of a fit of 32 cells of 5,000 CRUs
        _grad("grad_32x5000", 32, 5000, 5000, 60, 20, 30, "release", False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "ens", "ens", "grad"])
    phase = rng.choice(["rest", "release", "plateau"])
    precision = rng.choice(["fp32", "fp32", "fp64"])
    if kind == "run":
        ncru = _log_int(rng, 20, 12500 if precision == "fp32" else 1400)
        steps = _log_int(rng, 100, 2000 if precision == "fp32" else 500)
        c = _run("", ncru, steps, max(20, steps // rng.randint(1, 5)), precision, phase)
    elif kind == "ens":
        cells = _log_int(rng, 2, 256 if precision == "fp32" else 24)
        hi = _log_int(rng, 100, 12500 if precision == "fp32" else 1300)
        lo = max(5, int(hi * rng.uniform(0.1, 1.0)))
        big = precision == "fp32" and cells * hi > 400000
        steps = _log_int(rng, 50, 100 if big else 400)
        c = _ens("", cells, lo, hi, steps, max(10, steps // rng.randint(1, 6)), precision, phase, sums=rng.random() < 0.5,
                 codec=rng.random() < 0.3, cluster=6 if big and hi > 2000 else 0)
    else:
        cells = _log_int(rng, 1, 32)
        hi = _log_int(rng, 50, 5000)
        steps = _log_int(rng, 30, 60 if cells * hi > 20000 else 150)
        c = _grad("", cells, max(20, int(hi * rng.uniform(0.3, 1.0))), hi, steps, rng.randint(3, 20),
                  rng.choice([20, 50, 200]), phase, rng.random() < 0.3)
    del c["name"]
    return c


def _sizes(case):
    """CRUs per cell, spread over [lo, hi]."""
    if case["kind"] == "run":
        return [case["ncru"]]
    lo, hi = case["lo"], case["hi"]
    return [int(n) for n in np.random.default_rng([case["cells"], lo, hi]).integers(lo, hi + 1, case["cells"])]


def work(case):
    """Bytes: each cell's state read and written once (72 B per CRU with an FP32 state, 108 B with an
    FP64 one) and the records written once.  Operations: ~300 per CRU-step (fluxes, rates, Ca updates,
    draw) and ~1,500 per global step, three times that with the reverse pass."""
    n = sum(_sizes(case))
    cells, steps = case.get("cells", 1), case["steps"]
    flops = steps * (300.0 * n + 1500.0 * cells)
    if case["kind"] == "grad":
        return {"bytes": 2.0 * 108 * n + 8.0 * cells * (2 * (steps // case["sample"]) + 8), "flops": 3.0 * flops}
    state = 72 if case["precision"] == "fp32" else 108
    rec = steps // case["every"]
    out = rec * 36 * 8.0 * cells
    if case["kind"] == "run":
        out += rec * n * (184.0 if case["precision"] == "fp64" else 168.0)
    elif case["sums"]:
        out += rec * 28 * 8.0 * cells
    if case.get("codec"):
        out += rec * 36.0 * n / cells
    return {"bytes": 2.0 * state * n + out, "flops": flops}


# ------------------------------------------------------------------------------------------
# Inputs.
# ------------------------------------------------------------------------------------------
def _pick(rng, p, shape):
    """Indices drawn with (not quite normalised) weights p."""
    c = np.cumsum(p)
    return np.searchsorted(c / c[-1], rng.random(shape), side="right").clip(0, len(p) - 1)


def _crus(rng, n, phase, f32):
    """n CRUs of a phase: channel states by occupancy, Ca by quantile (values that float32 holds for
    an FP32 run, so that every precision starts from the same state)."""
    q = CRUS[phase]
    ryr = _pick(rng, q["RyR"], (n, 4, 5))
    s = dict(LCC=(1 + _pick(rng, q["LCC"], (n, 4))).astype(np.int32),
             LCC_inactivation=(rng.random((n, 4)) < q["gate"]).astype(np.int32),
             ClCh=(rng.random((n, 4)) < q["clch"]).astype(np.int32),
             RyR=np.stack([(ryr == k).sum(-1) for k in range(6)], -1).astype(np.int32))
    if phase == "rest":
        s["CaSS"], s["CaJSR"] = np.full((n, 4), 1.45370e-4), np.full(n, 0.908408)
    else:
        s["CaSS"] = np.exp(np.interp(rng.random((n, 4)), QUANTILES, np.log(q["CaSS"])))
        s["CaJSR"] = np.interp(rng.random(n), QUANTILES, q["CaJSR"])
    if f32:
        s["CaSS"], s["CaJSR"] = (s[k].astype(np.float32).astype(np.float64) for k in ("CaSS", "CaJSR"))
    return s


def _inputs(case, seed):
    """Sizes, parameters, globals, CRU states and stimulus of every cell, from the seed alone."""
    rng = np.random.default_rng([seed & 0xFFFFFFFF, 77])
    sizes = _sizes(case)
    f32 = case.get("precision") == "fp32"
    pool = _crus(rng, min(sum(sizes), 16384), case["phase"], f32)
    m = len(pool["CaJSR"])
    cells = []
    for n in sizes:
        p = dict(PARAMS)
        if case["kind"] != "run":
            z = np.exp(rng.normal(0.0, 0.1, len(VARIED)))
            for k, name in enumerate(VARIED):
                for field in (("Vmaxf", "Vmaxr") if name == "Vmax" else (name,)):
                    p[field] *= float(z[k])
        g = np.array(GLOBALS[case["phase"]])
        g[:11] *= 1.0 + 1e-3 * rng.standard_normal(11)
        at = np.arange(n) if len(sizes) == 1 and n <= m else rng.integers(0, m, n)
        cells.append(dict(n=n, params=p, globals=g, crus={k: v[at] for k, v in pool.items()}))
    return dict(cells=cells, seed=int(rng.integers(1, 1 << 62)), rng=rng)


def _state(c):
    return engine.CRUState(**{k: c["crus"][k] for k in ("CaSS", "CaJSR", "LCC", "LCC_inactivation", "RyR", "ClCh")})


def _pulse(t):
    return PULSE[3] if PULSE[0] <= t < PULSE[0] + PULSE[2] else 0.0


def _istim(case):
    """Samples of the stimulus at the accumulated time of every step (only from rest: later phases
    lie after it)."""
    out, t = np.zeros(case["steps"]), 0.0
    for i in range(case["steps"]):
        out[i] = _pulse(t) if case["phase"] == "rest" else 0.0
        t += DT
    return out


def _scales(inputs):
    """Per-cell scales of the eight fitted parameters (THETA's order)."""
    return 1.0 + inputs["rng"].uniform(-0.2, 0.2, (len(inputs["cells"]), 8))


def _target(inputs, case):
    """The trace that a fit compares V with: one value per cell and sample."""
    V0 = inputs["cells"][0]["globals"][0]
    return torch.from_numpy(V0 + inputs["rng"].normal(0.0, 5.0, (len(inputs["cells"]), case["steps"] // case["sample"])))


def prepare(case, seed):
    if case["kind"] == "ens" and case["phase"] == "rest" and case["cells"] * case["hi"] > 400000:
        return _prepare_large(case, seed)
    inp = _inputs(case, seed)
    cells = inp["cells"]
    if case["kind"] == "run":
        p, g, s = GW.GWParameters(), GW.GWGlobalState(), GW.GWCRUState(case["ncru"])
        for k, v in cells[0]["params"].items():
            setattr(p, k, v)
        G = cells[0]["globals"]
        for i, k in enumerate(_SCALARS):
            setattr(g, k, G[i])
        g.XKr, g.XKv43, g.XKv14 = G[11:16], G[16:26], G[26:36]
        for k, v in cells[0]["crus"].items():
            setattr(s, k, v)
        return dict(case=case, params=p, globals=g, crus=s, istim=_istim(case), seed=inp["seed"])
    plist = [engine.params_from(c["params"]) for c in cells]
    sizes = [c["n"] for c in cells]
    pulse = PULSE if case["phase"] == "rest" else (0.0, 0.0, 0.0, 0.0)
    if case["kind"] == "ens":
        e = engine.Ensemble(sizes, plist, precision=case["precision"], seed=inp["seed"], cluster_ctas=case["cluster"])
        for i, c in enumerate(cells):
            e.set_globals(i, c["globals"])
            e.set_crus(i, _state(c))
        e.set_pulse(*pulse)
        return dict(case=case, ens=e)
    scales = _scales(inp)
    target = _target(inp, case)
    if case["autograd"]:
        base = engine.params_from(PARAMS)
        spec = TraceSpec(ncru=sizes, base=base, states=[(c["globals"], _state(c)) for c in cells], seed=inp["seed"],
                         n_steps=case["steps"], dt=DT, checkpoint_every=case["checkpoint"],
                         sample_every=case["sample"], stim=pulse)
        return dict(case=case, spec=spec, target=target, scales=torch.from_numpy(scales))
    plist = [scaled_params(engine.params_from(PARAMS), z) for z in scales]
    eng = GradEngine(sizes, plist, n_steps=case["steps"], dt=DT, seed=inp["seed"], checkpoint_every=case["checkpoint"],
                     sample_every=case["sample"], stim=pulse)
    for i, c in enumerate(cells):
        eng.set_state(i, c["globals"], _state(c))
    return dict(case=case, eng=eng, target=target)


def _prepare_large(case, seed):
    """A large ensemble from rest: its CRUs are the device's own draw of the reference's initial
    distributions (keyed on the seed), its parameters log-normal, its pacing at 2 Hz."""
    rng = np.random.default_rng([seed & 0xFFFFFFFF, 78])
    sizes, plist = _sizes(case), []
    for z in np.exp(rng.normal(0.0, 0.15, (case["cells"], len(VARIED)))):
        plist.append(engine.params_from(None, PCaL=PARAMS["PCaL"] * z[0], GKr=PARAMS["GKr"] * z[1],
                                        GKs=PARAMS["GKs"] * z[2], Vmaxf=PARAMS["Vmaxf"] * z[3],
                                        Vmaxr=PARAMS["Vmaxr"] * z[3], rRyR=PARAMS["rRyR"] * z[4]))
    e = engine.Ensemble(sizes, plist, precision=case["precision"], seed=int(rng.integers(1, 1 << 62)),
                        cluster_ctas=case["cluster"])
    e.set_pulse(PULSE[0], 500.0, PULSE[2], PULSE[3])
    return dict(case=case, ens=e)


# ------------------------------------------------------------------------------------------
# One pass.
# ------------------------------------------------------------------------------------------
_SCALARS = ("V", "Nai", "Ki", "Cai", "CaNSR", "CaLTRPN", "CaHTRPN", "m", "h", "j", "xKs")
_CRU_FIELDS = ("CaJSR", "CaSS", "LCC", "LCC_inactivation", "RyR", "ClCh")


def run(state):
    case = state["case"]
    if case["kind"] == "run":
        r = GW.run(state["params"], case["ncru"], DT, case["steps"], state["istim"], case["every"], state["crus"],
                   state["globals"], seed=state["seed"], precision=case["precision"])
        out = {k: getattr(r, k) for k in _CRU_FIELDS}
        # the 36 global states of every record side by side, as the ensemble's trace has them
        out.update(t=r.t, globals=np.column_stack([getattr(r, k) for k in _SCALARS] + [r.XKr, r.XKv43, r.XKv14]))
        if case["precision"] == "fp32":  # the records of an FP32 state hold float32 values
            out["CaSS"], out["CaJSR"] = out["CaSS"].astype(np.float32), out["CaJSR"].astype(np.float32)
        return out
    if case["kind"] == "ens":
        tr = state["ens"].run(DT, case["steps"], case["every"], cru_cell=0 if case["codec"] else None,
                              codec=case["codec"], sums=case["sums"], currents=case["sums"])
        out = dict(t=tr.t, globals=tr.globals)
        if case["sums"]:
            out.update(sums=tr.cru_sums, currents=tr.currents)
        if case["codec"]:
            out.update({"cru_" + k: v for k, v in tr.codec.items()})
        return out
    if case["autograd"]:
        scales = state["scales"].clone().requires_grad_(True)
        V = VoltageTrace.apply(scales, state["spec"])
        loss = ((V - state["target"]) ** 2).mean()
        loss.backward()
        return dict(V=V.detach(), loss=loss.detach(), grad=scales.grad)
    V = state["eng"].forward()
    r = V - state["target"].numpy()
    return dict(V=V, sens=state["eng"].backward(2.0 * r / r.size))


# ------------------------------------------------------------------------------------------
# The same in 64 bits.
# ------------------------------------------------------------------------------------------
_M32 = 0xFFFFFFFF
_LCC_NEXT = [[0, 0, 0], [2, 7, 7], [1, 3, 8], [2, 4, 9], [3, 5, 10], [4, 6, 11], [5, 5, 5], [1, 8, 8], [2, 7, 9],
             [3, 8, 10], [4, 9, 11], [5, 10, 12], [11, 11, 11]]
_RYR_FROM = [0, 1, 1, 2, 3, 4, 1, 2, 3, 4, 4, 5]
_RYR_TO = [1, 2, 4, 3, 4, 5, 0, 1, 2, 1, 3, 4]


def _uniform(k, cru, step, cell, seed, bits):
    """Draw k of (seed, cell, CRU, step): Philox4x32-10, its 64-bit word as a 53- or 24-bit uniform."""
    c = [k >> 1, cru, torch.full_like(k, step & _M32), cell]
    k0, k1 = seed & _M32, (seed >> 32) & _M32
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & _M32) ^ c[1] ^ k0, p1 & _M32, ((p0 >> 32) & _M32) ^ c[3] ^ k1, p0 & _M32]
        k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
    odd = (k & 1) == 1
    hi, lo = torch.where(odd, c[3], c[1]), torch.where(odd, c[2], c[0])
    m = (hi >> 8) if bits == 24 else (hi << 21) + (lo >> 11)
    return m.clamp(min=1).double() * 2.0 ** -bits


class _Exact:
    """Cells of the model side by side: P maps a parameter to a [cells] tensor."""

    def __init__(self, P, cells, seed, bits, device):
        self.P, self.seed, self.bits = P, seed, bits
        t = lambda v, dt: torch.as_tensor(np.concatenate(v), device=device, dtype=dt)  # noqa: E731
        ns = [c["n"] for c in cells]
        self.C = len(cells)
        self.at = torch.as_tensor(np.repeat(np.arange(self.C), ns), device=device)
        self.cru = torch.as_tensor(np.concatenate([np.arange(n) for n in ns]), device=device)
        cr = lambda k, dt: t([c["crus"][k] for c in cells], dt)  # noqa: E731
        self.x, self.J = cr("CaSS", torch.float64), cr("CaJSR", torch.float64)
        self.lcc, self.gate = cr("LCC", torch.int64), cr("LCC_inactivation", torch.int64)
        self.cl, self.ryr = cr("ClCh", torch.int64), cr("RyR", torch.int64)
        self.L = torch.zeros_like(self.x)
        G = torch.as_tensor(np.stack([c["globals"] for c in cells]), device=device)
        self.g = [G[:, i] for i in range(36)]
        n = torch.as_tensor(ns, device=device).double()
        self.factor = P["NCaRU"] / n
        self.sum_tr = n * (P["rtr"] * (0.908882 - 0.908408)).detach()
        self.sum_xf = 4 * n * (P["rxfer"] * (1.45370e-4 - 1.45273e-4)).detach()
        self.next = torch.tensor(_LCC_NEXT, device=device)
        self.rfrom, self.rto = torch.tensor(_RYR_FROM, device=device), torch.tensor(_RYR_TO, device=device)
        self.step = 0

    def _cells_sum(self, v):
        return torch.zeros(self.C, dtype=torch.float64, device=v.device).index_add(0, self.at, v)

    # ---- the CRUs over one step (V, Cai, CaNSR of the step's start) ----
    def _lcc_table(self, V):
        """Outgoing LCC rates by state, [cells, 13, 3] (without the Ca-dependent ones)."""
        P = self.P
        al, be = 2.0 * torch.exp(0.012 * (V - 35.0)), 0.0882 * torch.exp(-0.05 * (V - 35.0))
        z, a, b, om = torch.zeros_like(V), P["a"], 1.0 / P["b"], P["omega"]
        rows = [[z, z, z], [4 * al, z, z], [be, 3 * al, z], [2 * be, 2 * al, z], [3 * be, al, z],
                [4 * be, P["f"], z], [P["g"], z, z], [om, 4 * al * a, z], [om * b, be * b, 3 * al * a],
                [om * b ** 2, 2 * be * b, 2 * al * a], [om * b ** 3, 3 * be * b, al * a],
                [om * b ** 4, 4 * be * b, P["f1"]], [P["g1"], z, z]]
        return torch.stack([torch.stack(r, -1) for r in rows], 1)

    def _rates(self, i, x, table, inact):
        """LCC [n, 4, 3], gate [n, 4], RyR [n, 4, 12] and ClCh [n, 4] rates of CRUs i at CaSS x."""
        at, R = self.at[i], self.ryr[i].double()
        P = {k: self.P[k].detach()[at][:, None] for k in (
            "gamma0", "a", "k12", "k21", "k23", "k25", "k32", "k34", "k43", "k45", "k52", "k54", "k56", "k65",
            "kfClCh", "kbClCh")}
        lcc = self.lcc[i]
        rl = table[at[:, None], lcc].clone()
        gx = P["gamma0"] * P["a"] ** (lcc - 1).clamp(0, 4) * x
        rl[..., 1] = torch.where(lcc == 1, gx, rl[..., 1])
        rl[..., 2] = torch.where((lcc >= 2) & (lcc <= 5), gx, rl[..., 2])
        rg = torch.where(self.gate[i] == 0, inact[0][at][:, None], inact[1][at][:, None])
        x2, hi34, hi56, z = x * x, x > 3.685e-2, x > 1.15e-4, torch.zeros_like(x)
        tau, eq = 1.0 / (P["k34"] * x2 + P["k43"]), P["k65"] / (P["k56"] * x2 + P["k65"])
        R34, R56 = R[..., 2] + R[..., 3], R[..., 4] + R[..., 5]
        rr = torch.stack([
            R[..., 0] * P["k12"] * x2, R[..., 1] * P["k23"] * x2, R[..., 1] * P["k25"] * x2,
            torch.where(hi34, z, R[..., 2] * P["k34"] * x2),
            torch.where(hi34, R34 * P["k45"] * P["k34"] * x2 * tau, R[..., 3] * P["k45"]),
            torch.where(hi56, z, R[..., 4] * P["k56"] * x2), R[..., 1] * P["k21"],
            torch.where(hi34, R34 * P["k32"] * P["k43"] * tau, R[..., 2] * P["k32"]),
            torch.where(hi34, z, R[..., 3] * P["k43"]),
            torch.where(hi56, R56 * P["k52"] * eq, R[..., 4] * P["k52"]),
            torch.where(hi56, R56 * P["k54"] * x2 * eq, R[..., 4] * P["k54"] * x2),
            torch.where(hi56, z, R[..., 5] * P["k65"])], -1)
        rc = torch.where(self.cl[i] == 0, P["kfClCh"] * x, P["kbClCh"])
        return rl, rg, rr, rc

    def _draw(self, i, k):
        return _uniform(k, self.cru[i], self.step, self.at[i], self.seed, self.bits)

    def _resplit(self, i, k, x, new):
        """Binomial re-splits of the CRUs i whose CaSS falls through a threshold; the draws used."""
        used = torch.zeros_like(k)
        k56, k34 = (x > 1.15e-4) & (new <= 1.15e-4), (x > 0.03685) & (new <= 0.03685)
        k34 &= ~k56
        rows = (k56 | k34).any(1).nonzero()[:, 0]
        if not rows.numel():
            return used
        ii, kr, x = i[rows], k[rows] + 1, x[rows]
        ryr, P = self.ryr[ii], {n: self.P[n].detach()[self.at[ii]] for n in ("k34", "k43", "k56", "k65")}
        for j in range(4):
            for mask, lo, down, up in ((k56[rows, j], 4, P["k65"], P["k56"]), (k34[rows, j], 2, P["k43"], P["k34"])):
                if not bool(mask.any()):
                    continue
                n = torch.where(mask, ryr[:, j, lo] + ryr[:, j, lo + 1], 0).clamp(min=0)
                p, X = down / (down + up * x[:, j] ** 2), torch.zeros_like(n)
                for q in range(int(n.max())):
                    X += ((q < n) & (self._draw(ii, kr + q) < p)).long()
                ryr[:, j, lo] = torch.where(mask, X, ryr[:, j, lo])
                ryr[:, j, lo + 1] = torch.where(mask, n - X, ryr[:, j, lo + 1])
                kr, used[rows] = kr + n, used[rows] + n
        self.ryr[ii] = ryr
        return used

    def _crus_step(self, V, Cai, CaNSR):
        P, at0 = self.P, self.at
        with torch.no_grad():
            Vd = V.detach()
            table = self._lcc_table(Vd)
            yinf = 0.4 / (1.0 + torch.exp((Vd + 12.5) / 5.0)) + 0.6
            tau = 340.0 / (1.0 + torch.exp((Vd + 30.0) / 12.0)) + 60.0
            inact = (yinf / tau, (1.0 - yinf) / tau)
        F_RT = 1.0 / (8.314 * P["T"] / 96.5)
        je = torch.exp(2.0 * V * F_RT)
        jm = 2.0e6 * P["PCaL"] / P["VSS"] * V * F_RT / (je - 1.0)
        fxf, ftr = None, None
        open_ = (self.ryr[..., 2] + self.ryr[..., 3]).double()
        rel = P["rRyR"][at0][:, None] * open_ * (self.J[:, None] - self.x)
        t = torch.zeros_like(self.J)
        k = torch.zeros_like(self.cru)
        i = torch.arange(len(self.cru), device=self.cru.device)
        while i.numel():
            at = at0[i]
            x, J, L, rl_ = self.x[i], self.J[i], self.L[i], rel[i]
            p = lambda n: P[n][at][:, None]  # noqa: E731
            jtr = P["rtr"][at] * (CaNSR[at] - J)
            jis = p("riss") * (torch.roll(x, -1, 1) + torch.roll(x, 1, 1) - 2 * x)
            jxf = p("rxfer") * (x - Cai[at][:, None])
            with torch.no_grad():
                xd = x.detach()
                rl, rg, rr, rc = self._rates(i, xd, table, inact)
                sub = rl.sum(-1) + rg + rr.sum(-1) + rc
                total = sub.sum(1)
                jump = -torch.log(self._draw(i, k[i])) / total
                last = ~(t[i] + jump < DT)
                h = torch.where(last, DT - t[i], jump)
            beta = 1.0 / (1.0 + p("KBSR") * p("BSRT") / (p("KBSR") + x) ** 2 + p("KBSL") * p("BSLT") / (p("KBSL") + x) ** 2)
            new = x + h[:, None] * (L + rl_ - jxf + jis) * beta
            with torch.no_grad():
                used = self._resplit(i, k[i], xd, new.detach())
            bj = 1.0 / (1.0 + P["KCSQN"][at] * P["CSQNT"][at] / (P["KCSQN"][at] + J) ** 2)
            Jn = J + h * bj * (jtr - P["VSS"][at] / P["VJSR"][at] * rl_.sum(1))
            whole = i.numel() == len(self.cru)
            self.x = new if whole else self.x.index_put((i,), new)
            self.J = Jn if whole else self.J.index_put((i,), Jn)
            xs = jxf.sum(1)
            fxf, ftr = (xs, jtr) if whole else (fxf.index_put((i,), xs), ftr.index_put((i,), jtr))
            e = (~last).nonzero()[:, 0]
            if not e.numel():
                break
            ie = i[e]
            with torch.no_grad():
                kk = k[ie] + 1 + used[e]
                u = self._draw(ie, kk) * total[e]
                j = (sub[e].cumsum(1)[:, :3] < u[:, None]).sum(1)
                r3, r12 = rl[e, j], rr[e, j]
                s3, sg, sc, ss = r3.sum(1), rg[e, j], rc[e, j], sub[e, j]
                s12 = ss - (s3 + sg + sc)
                u = self._draw(ie, kk + 1) * ss
                act = torch.where(u < s3, 1, torch.where(u < s3 + sg, 2, torch.where(u < s3 + sg + s12, 3, 4)))
                u = self._draw(ie, kk + 2)
                t3 = (r3.cumsum(1)[:, :2] < (u * s3)[:, None]).sum(1)
                t12 = (r12.cumsum(1)[:, :11] < (u * s12)[:, None]).sum(1)
                k[ie] = kk + 2 + ((act == 1) | (act == 3)).long()
                t[ie] = t[ie] + jump[e]
                frm = self.lcc[ie, j]
                to = self.next[frm, t3]
                self.lcc[ie, j] = torch.where(act == 1, to, frm)
                self.gate[ie, j] = torch.where(act == 2, 1 - self.gate[ie, j], self.gate[ie, j])
                self.cl[ie, j] = torch.where(act == 4, 1 - self.cl[ie, j], self.cl[ie, j])
                d = (act == 3).long()
                self.ryr[ie, j, self.rfrom[t12]] -= d
                self.ryr[ie, j, self.rto[t12]] += d
                entered = (act == 1) & (((frm == 5) & (to == 6)) | ((frm == 11) & (to == 12)))
                left = (act == 1) & ((frm == 6) | (frm == 12))
                g1, opn = self.gate[ie, j] == 1, (self.lcc[ie, j] == 6) | (self.lcc[ie, j] == 12)
                setj = (entered & g1) | ((act == 2) & g1 & opn)
                zero = (entered & ~g1) | left | ((act == 2) & ~g1)
            ae = at0[ie]
            opened = jm[ae] * (0.341 * P["Cao"][ae] - je[ae] * self.x[ie, j])
            self.L = self.L.index_put((ie, j), torch.where(setj, opened, torch.where(zero, 0.0, self.L[ie, j])))
            nopen = (self.ryr[ie, j, 2] + self.ryr[ie, j, 3]).double()
            nrel = P["rRyR"][ae] * nopen * (self.J[ie] - self.x[ie, j])
            rel = rel.index_put((ie, j), torch.where(act == 3, nrel, rel[ie, j]))
            i = ie
        self.sum_xf, self.sum_tr = self._cells_sum(fxf), self._cells_sum(ftr)

    # ---- the global step ----
    def advance(self, istim):
        P, e = self.P, torch.exp
        V, Nai, Ki, Cai, CaNSR, LT, HT, m, hh, jj, xKs = self.g[:11]
        Kr, K43, K14 = self.g[11:16], self.g[16:26], self.g[26:36]
        sum_L, sum_cl = self._cells_sum(self.L.sum(1)), self._cells_sum(self.cl.sum(1).double())
        RT_F = 8.314 * P["T"] / 96.5
        v = V / RT_F
        ev, F, CSA = e(-v), 96.5, P["CSA"]
        ENa, EK = torch.log(P["Nao"] / Nai) * RT_F, torch.log(P["Ko"] / Ki) * RT_F
        INa = P["GNa"] * m ** 3 * hh * jj * (V - ENa)
        INab = P["GNab"] * (V - ENa)
        e1 = e(P["eta"] * v)
        e2 = e1 * ev
        INaCa = (5000.0 * P["kNaCa"] / ((P["KmNa"] ** 3 + P["Nao"] ** 3) * (P["KmCa"] + P["Cao"]))
                 * (e1 * Nai ** 3 * P["Cao"] - e2 * P["Nao"] ** 3 * Cai) / (1.0 + P["ksat"] * e2))
        sigma = (e(P["Nao"] / 67.3) - 1.0) / 7.0
        INaK = (P["INaKmax"] * P["Ko"] / (P["Ko"] + P["KmKo"]) / (1.0 + 0.1245 * e(-0.1 * v) + 0.0365 * sigma * ev)
                / (1.0 + (P["KmNai"] / Nai) ** 1.5))
        IKr = P["GKr"] * torch.sqrt(P["Ko"]) / (1.0 + 1.4945 * e(0.0446 * V)) * Kr[3] * (V - EK) * 0.5
        EKs = torch.log((P["Ko"] + 0.01833 * P["Nao"]) / (Ki + 0.01833 * Nai)) * RT_F
        IKs = P["GKs"] * xKs ** 2 * (V - EKs)
        IKv14 = (P["PKv14"] / P["Csc"] * F * v * K14[4] / (1 - ev)
                 * ((Ki - P["Ko"] * ev) + 0.02 * (Nai - P["Nao"] * ev)) * 1.0e9)
        Ito1 = IKv14 + P["GKv43"] * K43[4] * (V - EK)
        Ito2 = sum_cl * (1.0e9 * P["Pto2"] * F * self.factor / CSA) * v * (P["Clcyto"] * ev - P["Clo"]) / (ev - 1.0)
        IK1 = P["GK1"] / (2.0 + e(1.5 * (V - EK) / RT_F)) * P["Ko"] / (P["Ko"] + P["KmK1"]) * (V - EK)
        IKp = P["GKp"] / (1.0 + e((7.488 - V) / 5.98)) * (V - EK)
        ICaL = sum_L * (-1000.0 * 2.0 * F * P["VSS"] * self.factor / CSA)
        ICab = P["GCab"] * (V - 0.5 * EK)
        IpCa = P["IpCamax"] * Cai / (P["KmpCa"] + Cai)
        fu, ru = (Cai / P["Kmf"]) ** P["Hf"], (CaNSR / P["Kmr"]) ** P["Hr"]
        Jup = (P["Vmaxf"] * fu - P["Vmaxr"] * ru) / (1.0 + fu + ru)
        Jtr, Jxf = self.sum_tr * self.factor, self.sum_xf * self.factor
        bc = 1.0 / (1.0 + P["KCMDN"] * P["CMDNT"] / (P["KCMDN"] + Cai) ** 2)
        dLT = P["kLTRPNp"] * Cai * (P["LTRPNtot"] - LT) - P["kLTRPNm"] * LT
        dHT = P["kHTRPNp"] * Cai * (P["HTRPNtot"] - HT) - P["kHTRPNm"] * HT
        CF = CSA / (1000 * P["Vcyto"] * F)
        d = [istim - (INa + ICaL + IKr + IKs + Ito1 + IK1 + IKp + Ito2 + INaK + INaCa + IpCa + ICab + INab),
             -CF * (INa + INab + 3 * INaCa + 3 * INaK), -CF * (IKr + IKs + Ito1 + IK1 + IKp - 2 * INaK),
             bc * (-0.5 * CF * (ICab + IpCa - 2 * INaCa) + P["VSS"] / P["Vcyto"] * Jxf - Jup - (dLT + dHT)),
             P["Vcyto"] / P["VNSR"] * Jup - P["VJSR"] / P["VNSR"] * Jtr, dLT, dHT]
        hi = V >= -40.0
        z = torch.zeros_like(V)
        am, bm = 0.32 * (V + 47.13) / (1.0 - e(-0.1 * (V + 47.13))), 0.08 * e(-V / 11.0)
        ah = torch.where(hi, z, 0.135 * e(-(V + 80.0) / 6.8))
        bh = torch.where(hi, 1.0 / (0.13 * (1.0 + e(-(V + 10.66) / 11.1))), 3.56 * e(0.079 * V) + 3.1e5 * e(0.35 * V))
        aj = torch.where(hi, z, (-127140.0 * e(0.2444 * V) - 3.474e-5 * e(-0.04391 * V)) * (V + 37.78)
                         / (1.0 + e(0.311 * (V + 79.23))))
        bj = torch.where(hi, 0.3 * e(-2.535e-7 * V) / (1.0 + e(-0.1 * (V + 32.0))),
                         0.1212 * e(-0.01052 * V) / (1.0 + e(-0.1378 * (V + 40.14))))
        xinf = 1.0 / (1.0 + e(-(V - 24.7) / 13.6))
        w = V - 10.0
        tinv = 0.0000719 * w / (1.0 - e(-0.148 * w)) + 0.000131 * w / (e(0.0687 * w) - 1.0)
        d += [am * (1 - m) - bm * m, ah * (1 - hh) - bh * hh, aj * (1 - jj) - bj * jj, (xinf - xKs) * tinv]
        q23, q24 = 0.0218 * e(0.0262 * V), 1.29e-5 * e(2.71e-6 * V)
        q32, q34, q43 = 0.0009 * e(-0.0269 * V), 0.0622 * e(0.0120 * V), 0.0059 * e(-0.0443 * V)
        edges = [(0, 1, 0.0069 * e(0.0272 * V)), (1, 0, 0.0227 * e(-0.0431 * V)), (1, 2, P["Kf"]), (2, 1, P["Kb"]),
                 (2, 3, q23), (2, 4, q24), (3, 2, q32), (3, 4, q34), (4, 3, q43), (4, 2, q32 * q43 * q24 / (q23 * q34))]
        d += self._chain(Kr, edges)
        for x, n in ((K43, "Kv43"), (K14, "Kv14")):
            p = lambda k: P[k + n]  # noqa: B023, E731
            aa, ba = p("alphaa0") * e(p("aa") * V), p("betaa0") * e(-p("ba") * V)
            ai, bi = p("alphai0") * e(-p("ai") * V), p("betai0") * e(p("bi") * V)
            fs, bs = [1.0] + [p("f%d" % q) for q in (1, 2, 3, 4)], [1.0] + [p("b%d" % q) for q in (1, 2, 3, 4)]
            edges = []
            for q in range(4):
                edges += [(q, q + 1, (4 - q) * aa), (q + 1, q, (q + 1) * ba),
                          (5 + q, 6 + q, (4 - q) * aa * bs[q + 1] / bs[q]), (6 + q, 5 + q, (q + 1) * ba * fs[q] / fs[q + 1])]
            for q in range(5):
                edges += [(q, 5 + q, fs[q] * bi), (5 + q, q, ai / bs[q])]
            d += self._chain(x, edges)
        self._crus_step(V, Cai, CaNSR)
        self.g = [x + DT * y for x, y in zip(self.g, d)]
        self.step += 1

    @staticmethod
    def _chain(x, edges):
        d = [torch.zeros_like(x[0]) for _ in x]
        for a, b, q in edges:
            w = q * x[a]
            d[a], d[b] = d[a] - w, d[b] + w
        return d


def _tensors(cells, device):
    return {k: torch.tensor([float(c["params"][k]) for c in cells], dtype=torch.float64, device=device) for k in PARAMS}


_THETA_FIELDS = (("PCaL",), ("GKr",), ("GKs",), ("GK1",), ("INaKmax",), ("Vmaxf", "Vmaxr"), ("rRyR",), ("CSQNT",))


def exact(case, seed):
    n = sum(_sizes(case))
    grad = case["kind"] == "grad"
    steps = case["steps"] if grad else (case["steps"] // case["every"] - 1) * case["every"] + 1
    # a step takes 5 to 10 ms while its launches set the time, more for the largest states
    if steps * (1.0 + n / 20000.0) > (250 if grad else 1900) or n > (4000 if grad else 60000):
        return None
    inp = _inputs(case, seed)
    cells = inp["cells"]
    device = "cuda" if n > 3000 and torch.cuda.is_available() else "cpu"
    P = _tensors(cells, device)
    istim = _istim(case)
    if grad:
        z = torch.from_numpy(_scales(inp)).requires_grad_(True)
        target = _target(inp, case)
        for k, v in PARAMS.items():
            P[k] = torch.full((len(cells),), float(v), dtype=torch.float64)
        for k, fields in enumerate(_THETA_FIELDS):
            for f in fields:
                P[f] = P[f] * z[:, k]
        sim, V = _Exact(P, cells, inp["seed"], 53, "cpu"), []
        for s in range(steps):
            sim.advance(float(istim[s]))
            if (s + 1) % case["sample"] == 0:
                V.append(sim.g[0])
        V = torch.stack(V, 1)
        loss = ((V - target) ** 2).mean()
        loss.backward()
        if case["autograd"]:
            return dict(V=V.detach(), loss=loss.detach(), grad=z.grad)
        return dict(V=V.detach(), sens=(z.grad * z).detach())
    bits = 24 if case["precision"] == "fp32" else 53
    with torch.no_grad():
        sim = _Exact(P, cells, inp["seed"], bits, device)
        t, rec = 0.0, []
        for s in range(steps):
            sim.advance(float(istim[s]))
            t += DT
            if s % case["every"] == 0:
                rec.append((t, torch.stack(sim.g, 1).cpu().numpy(), sim.x.cpu().numpy(), sim.J.cpu().numpy()))
    G = np.stack([r[1] for r in rec], 1)  # [cells, records, 36]
    ts = np.array([r[0] for r in rec])
    if case["kind"] == "ens":
        out = dict(t=ts, globals=G)
        if case["sums"]:
            out.update(sums=None, currents=None)
        if case["codec"]:
            n0 = cells[0]["n"]
            out.update({"cru_" + k: None for k in ("LCC", "LCC_inactivation", "ClCh", "RyR")})
            out["cru_CaSS"] = np.stack([r[2][:n0] for r in rec])
            out["cru_CaJSR"] = np.stack([r[3][:n0] for r in rec])
        return out
    out = dict.fromkeys(_CRU_FIELDS)
    out.update(t=ts, globals=G[0], CaSS=np.stack([r[2] for r in rec]), CaJSR=np.stack([r[3] for r in rec]))
    return out
