"""Performance cases: the sweeps that users of this package run.

Each listed case is one call of a public entry point on a workload of this
repository (its circuits, tests and benchmark); ``draw`` gives more of the
same ranges.  ``prepare`` makes what a program holds before the call (context,
uploaded circuit, settings, output buffers, matrices), ``run`` is one pass,
``exact`` the same results in plain 64-bit torch arithmetic.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import spicier_gb300 as sg
from spicier_gb300 import abi, configs
from spicier_gb300.api import Mlp, newton_dc_learned_device

DEV = "cuda"
F64 = torch.float64

# ---------------------------------------------------------------------------
# Circuits as plain data: (kind, name, nodes, values, pulse); a value is a
# number or a draw ("G", mean, sigma, index), ("U", lo, hi, index) or
# ("L", lo, hi, index).  MOSFET values: (vto, kp, lambda, w), all L = 1 um.
# ---------------------------------------------------------------------------


def _mos(name, d, g, s, pmos, vto, kp, lam, w):
    return ("P" if pmos else "N", name, (d, g, s), (vto, kp, lam, w), None)


def cs_nmos_elements():
    """The common-source NMOS amplifier (RD, RS, VTO and KP drawn)."""
    return [
        ("V", "VDD", ("vdd", "0"), (5.0,), None),
        ("R", "R1", ("vdd", "gate"), (100e3,), None),
        ("R", "R2", ("gate", "0"), (47e3,), None),
        ("R", "RD", ("vdd", "drain"), (("G", 10e3, 0.05 * 10e3, 0),), None),
        ("R", "RS", ("source", "0"), (("G", 1e3, 0.05 * 1e3, 1),), None),
        _mos("M1", "drain", "gate", "source", False, ("G", 0.7, 0.03, 2), ("G", 110e-6, 0.10 * 110e-6, 3), 0.02, 10e-6),
    ], {}


OPAMP = (
    ("M1", "n1", "out", "tail", False, 20e-6), ("M2", "n2", "vin", "tail", False, 20e-6),
    ("M3", "n1", "n1", "vdd", True, 20e-6), ("M4", "n2", "n1", "vdd", True, 20e-6),
    ("M5", "tail", "bias", "vss", False, 20e-6), ("M6", "out", "n2", "vdd", True, 80e-6),
    ("M7", "out", "bias", "vss", False, 40e-6), ("M8", "bias", "bias", "vss", False, 10e-6),
)


def opamp_elements():
    """The two-stage Miller op-amp buffer (VIN uniform; VTO and KP of each device Gaussian)."""
    els = [
        ("V", "VDD", ("vdd", "0"), (3.3,), None),
        ("V", "VSS", ("vss", "0"), (0.0,), None),
        ("V", "VIN", ("vin", "0"), (("U", 1.0, 2.3, 0),), None),
        ("I", "IBIAS", ("vdd", "bias"), (20e-6,), None),
    ]
    for k, (name, d, g, s, pmos, w) in enumerate(OPAMP):
        vto, kp = (-0.8, 50e-6) if pmos else (0.7, 110e-6)
        els.append(_mos(name, d, g, s, pmos, ("G", vto, 0.020, 1 + 2 * k), ("G", kp, 0.05 * kp, 2 + 2 * k), 0.04, w))
    els += [("R", "RZ", ("n2", "nz"), (2e3,), None), ("C", "CC", ("nz", "out"), (2e-12,), None)]
    return els, dict(vdd=3.3, vss=0.0, vin=1.65, out=1.65, n1=2.3, n2=2.3, nz=2.3, tail=0.8, bias=0.9)


def rlc_elements():
    """The Monte Carlo RLC network of the fixed-step transient tests: two V
    sources, a current source, two inductors, two capacitors, 9 unknowns."""
    return [
        ("V", "V1", ("in", "0"), (0.0,), (0.0, 1.0, 2e-6, 1e-6, 1e-6, 10e-6, 40e-6)),
        ("R", "R1", ("in", "a"), (("G", 100.0, 5.0, 0),), None),
        ("L", "L1", ("a", "b"), (("L", 1e-6, 1e-5, 1),), None),
        ("C", "C1", ("b", "0"), (("L", 1e-9, 1e-8, 2),), None),
        ("R", "R2", ("b", "c"), (("G", 200.0, 10.0, 3),), None),
        ("C", "C2", ("c", "0"), (("L", 1e-9, 1e-8, 4),), None),
        ("R", "R3", ("c", "bias"), (1e3,), None),
        ("V", "V2", ("bias", "0"), (("G", 0.5, 0.01, 5),), None),
        ("I", "I1", ("0", "c"), (1e-4,), (0.0, 1e-4, 5e-6, 1e-6, 1e-6, 5e-6, 20e-6)),
        ("L", "L2", ("c", "d"), (2e-6,), None),
        ("R", "R4", ("d", "0"), (("G", 50.0, 2.0, 6),), None),
    ], {}


def rc_elements():
    """The same network without its inductors (the reference's TR-BDF2 update
    of an inductor is unstable, so that method's users run R, C circuits)."""
    els, nodeset = rlc_elements()
    ohms = {"L1": ("G", 20.0, 1.0, 1), "L2": 10.0}
    return [("R", "R" + nm, nodes, (ohms[nm],), None) if kind == "L" else (kind, nm, nodes, vals, pulse)
            for kind, nm, nodes, vals, pulse in els], nodeset


ELEMENTS = {"cs_nmos": cs_nmos_elements, "opamp": opamp_elements, "rlc": rlc_elements, "rc": rc_elements}


def build_circuit(name):
    """The same circuit through the package's circuit builder."""
    if name == "bsim3_chain":
        return configs.bsim3_cmos_chain()
    els, nodeset = ELEMENTS[name]()

    def val(v):
        if isinstance(v, tuple):
            return {"G": sg.Gauss, "U": sg.Uniform, "L": sg.LogUniform}[v[0]](*v[1:])
        return v

    c = sg.Circuit(name)
    for kind, nm, nodes, vals, pulse in els:
        vals = [val(v) for v in vals]
        p = sg.Pulse(*pulse) if pulse else None
        if kind in "NP":
            c.M(nm, *nodes, pmos=kind == "P", vto=vals[0], kp=vals[1], lam=vals[2], w=vals[3], l=1e-6)
        elif kind in "VI":
            getattr(c, kind)(nm, *nodes, vals[0], pulse=p)
        else:
            {"R": c.R, "C": c.Cap, "L": c.L}[kind](nm, *nodes, vals[0])
    c.nodeset = dict(nodeset)
    return c


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # the smallest sweep of everyday use: 1,024 samples of a one-transistor amplifier, plain FP64
        dict(name="cs_nmos_1k_fp64", kind="newton", circuit="cs_nmos", samples=1024, precision="fp64", warm="none",
             moments=False, resid=False),
        # the Monte Carlo operating points with statistics: op-amp, mixed precision, from the nodeset
        dict(name="opamp_64k_mixed", kind="newton", circuit="opamp", samples=65536, precision="mixed", warm="none",
             moments=True, resid=False),
        # the same sweep started from the learned linear warm start (the benchmark's headline arm)
        dict(name="opamp_64k_learned", kind="newton", circuit="opamp", samples=65536, precision="mixed",
             warm="linear", moments=True, resid=False),
        # the library's default precision, with the KCL residual a sign-off run asks for
        dict(name="opamp_64k_fp64", kind="newton", circuit="opamp", samples=65536, precision="fp64", warm="none",
             moments=False, resid=True),
        # the host-buffer call on BSIM3 devices (generic kernels, results in host memory)
        dict(name="bsim3_8k_host", kind="newton_host", circuit="bsim3_chain", samples=8192, precision="mixed"),
        # BatchedLuSolver at the sizes the reference publishes: 50 x 50 x 5,000 and 100 x 100 x 2,000
        dict(name="lu_50x5000", kind="lu", n=50, batch=5000, precision="fp64"),
        dict(name="lu_100x2000", kind="lu", n=100, batch=2000, precision="fp64"),
        # AC small-signal Monte Carlo of the op-amp, 8 decades at 10 points per decade
        dict(name="ac_opamp_8k", kind="ac", samples=8192, per_decade=10, precision="fp64"),
        # fixed-step trapezoidal transients of the RLC network, waveform recorded
        dict(name="rlc_16k_trap", kind="transient", samples=16384, steps=150, method=1),
        # adaptive RC-diode ladder transients of uneven size (an eighth of the benchmark's 4,096)
        dict(name="ladders_512_mixed", kind="ladder", count=512, max_sections=512, precision="mixed"),
        # power-grid corners on the 64 x 64 mesh, all 256 of the benchmark
        dict(name="grid_256_mixed", kind="grid", count=256, rows=64, cols=64, sinks=512, precision="mixed"),
        # one gradient step of the warm-start network's trainer (17 -> 3 x 256 -> 12, its batch of 4,096)
        dict(name="mlp_grad_4k", kind="mlp", rows=4096, hidden=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["newton", "newton", "newton", "newton_host", "lu", "lu", "ac", "transient", "ladder", "grid", "mlp"])
    if kind == "newton":
        circuit = rng.choice(["cs_nmos", "opamp", "opamp"])
        precision = rng.choice(["fp64", "mixed"])
        warm = rng.choice(["none", "linear"]) if circuit == "opamp" and precision == "mixed" else "none"
        top = 131072 if precision == "fp64" else 262144
        return dict(kind=kind, circuit=circuit, samples=_log(rng, 500, top), precision=precision, warm=warm,
                    moments=rng.random() < 0.5, resid=rng.random() < 0.5)
    if kind == "newton_host":
        return dict(kind=kind, circuit=rng.choice(["bsim3_chain", "opamp", "cs_nmos"]), samples=_log(rng, 500, 20000),
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "lu":
        n = _log(rng, 5, 150)
        most = min(65535, int(9e9 / n ** 3), int(3e8 / n ** 2))
        return dict(kind=kind, n=n, batch=_log(rng, 500, max(most, 600)),
                    precision=rng.choice(["fp64", "fp64", "mixed"]))
    if kind == "ac":
        return dict(kind=kind, samples=_log(rng, 200, 8192), per_decade=rng.choice([5, 7, 10]),
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "transient":
        return dict(kind=kind, samples=_log(rng, 300, 16384), steps=_log(rng, 40, 150), method=rng.choice([0, 1, 2]))
    if kind == "ladder":
        return dict(kind=kind, count=_log(rng, 30, 512), max_sections=rng.choice([40, 123, 257, 512]),
                    precision=rng.choice(["mixed", "fp64"]))
    if kind == "grid":
        rows, cols = rng.randint(12, 64), rng.randint(12, 64)
        return dict(kind=kind, count=_log(rng, 8, 128), rows=rows, cols=cols, sinks=max(1, rows * cols // 8),
                    precision="mixed")
    return dict(kind=kind, rows=64 * _log(rng, 8, 64), hidden=rng.choice([64, 128, 256]))


PREC = {"fp64": abi.SP_PREC_FP64, "mixed": abi.SP_PREC_MIXED}
_CTX = []


def _ctx():
    """The process's one context (a program opens it once)."""
    if not _CTX:
        _CTX.append(sg.Context(0))
    return _CTX[0]


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _lu_system(case, seed):
    n, b = case["n"], case["batch"]
    g = _gen(seed)
    A = torch.randn((b, n, n), dtype=F64, device=DEV, generator=g)
    A += 4.0 * torch.eye(n, dtype=F64, device=DEV) * torch.rand((b, 1, 1), dtype=F64, device=DEV, generator=g)
    rhs = torch.randn((b, n), dtype=F64, device=DEV, generator=g)
    return A, rhs


def _ac_cfg(case):
    c = build_circuit("opamp")
    return abi.ac_config(10.0, 1e9, case["per_decade"], abi.SP_AC_DEC,
                         probes=(c.node("out"), c.node("n2")), precision=PREC[case["precision"]])


TRAN_H = 0.2e-6


def prepare(case, seed):
    s = dict(case=case, seed=seed)
    kind = case["kind"]
    ctx = s["ctx"] = _ctx()
    if kind in ("newton", "newton_host"):
        s["circuit"] = c = build_circuit(case["circuit"])
        s["cfg"] = abi.newton_config(precision=PREC[case["precision"]])
        if kind == "newton_host":
            return s
        n, k = c.n, case["samples"]
        s["topo"] = ctx.topology(c)
        s["x"] = torch.empty((k, n), dtype=F64, device=DEV)
        s["iters"] = torch.empty(k, dtype=torch.int32, device=DEV)
        s["status"] = torch.empty(k, dtype=torch.uint8, device=DEV)
        s["resid"] = torch.empty(k, dtype=F64, device=DEV) if case["resid"] else None
        s["moments"] = torch.empty((n, 5), dtype=F64, device=DEV) if case["moments"] else None
        if case["warm"] == "linear":
            mean, lin, out = linear_fit(case["circuit"])
            slots = [j for j, p in enumerate(c.params) if p[0] != abi.SP_DRAW_FIXED]
            s["mlp"] = m = Mlp(ctx, len(slots), n, 128, 3)
            m.set_linear(lin)
            m.set_io(slots, mean, np.ones(len(slots)), out, np.zeros(n))
            m.set_inference_kernel(abi.SP_MLP_KERNEL_LINEAR)
            s["cfg"].warm_max_iterations = 8
    elif kind == "lu":
        A, rhs = _lu_system(case, seed)
        s["A"] = A.transpose(1, 2).contiguous()  # the solver's column-major layout
        s["rhs"] = rhs
        s["x"] = torch.empty_like(rhs)
        s["sing"] = torch.empty(case["batch"], dtype=torch.uint8, device=DEV)
    elif kind == "ac":
        c = build_circuit("opamp")
        s["topo"], s["cfg"], s["ac"] = ctx.topology(c), abi.newton_config(), _ac_cfg(case)
        nf = len(ctx.ac_frequencies(s["ac"]))
        s["probe"] = torch.empty((case["samples"], nf, 2, 2), dtype=F64, device=DEV)
        s["status"] = torch.empty(case["samples"], dtype=torch.uint8, device=DEV)
    elif kind == "transient":
        c = build_circuit(_tran_net(case))
        s["topo"], s["cfg"] = ctx.topology(c), abi.newton_config()
        s["tc"] = abi.transient_config(TRAN_H, _tstop(case), case["method"], c.node("c"), abi.SP_PREC_FP64)
        s["x"] = torch.empty((case["samples"], c.num_nodes + 2), dtype=F64, device=DEV)
        s["status"] = torch.empty(case["samples"], dtype=torch.uint8, device=DEV)
        s["probe"] = torch.empty((case["samples"], case["steps"] + 1), dtype=F64, device=DEV)
    elif kind == "ladder":
        s["cfg"] = cfg = abi.ladder_config(precision=PREC[case["precision"]], max_sections=case["max_sections"])
        k = case["count"]
        s["out"] = dict(x=torch.empty((k, cfg.max_sections + 2), dtype=F64, device=DEV),
                        probe=torch.empty((k, cfg.num_probe), dtype=F64, device=DEV),
                        status=torch.empty(k, dtype=torch.uint8, device=DEV),
                        **{w: torch.empty(k, dtype=torch.int32, device=DEV)
                           for w in ("n", "accepted", "rejected", "iterations")})
    elif kind == "grid":
        s["cfg"] = abi.grid_config(precision=PREC[case["precision"]], rows=case["rows"], cols=case["cols"],
                                   num_sinks=case["sinks"])
        k = case["count"]
        s["out"] = dict(x=torch.empty((k, case["rows"] * case["cols"] + 1), dtype=F64, device=DEV),
                        newton=torch.empty(k, dtype=torch.int32, device=DEV),
                        krylov=torch.empty(k, dtype=torch.int32, device=DEV),
                        status=torch.empty(k, dtype=torch.uint8, device=DEV),
                        resid=torch.empty(k, dtype=F64, device=DEV))
    else:
        X, T, flat = _mlp_data(case, seed)
        s["mlp"] = m = Mlp(ctx, 17, 12, case["hidden"], 3)
        m.set_params(flat.cpu().numpy())
        s["X"], s["T"] = X, T
        s["grads"] = torch.empty(m.num_params, dtype=torch.float32, device=DEV)
        s["loss"] = torch.empty(1, dtype=torch.float32, device=DEV)
    return s


def _stream():
    return torch.cuda.current_stream().cuda_stream


def run(s):
    case, ctx, kind = s["case"], s["ctx"], s["case"]["kind"]
    if kind == "newton":
        k, kw = case["samples"], dict(iters=s["iters"], status=s["status"], resid=s["resid"], moments=s["moments"],
                                      stream=_stream())
        if case["warm"] == "linear":
            newton_dc_learned_device(ctx, s["topo"], s["mlp"], s["cfg"], s["seed"], k, s["x"], **kw)
        else:
            ctx.newton_dc_device(s["topo"], s["cfg"], s["seed"], k, s["x"], **kw)
        out = dict(x=s["x"], iters=s["iters"], status=s["status"])
        if s["resid"] is not None:
            out["resid"] = s["resid"]
        if s["moments"] is not None:  # sp_moments: a 64-bit count, then sum, sum of squares, min, max
            out["count"], out["moments"] = s["moments"].view(torch.int64)[:, 0], s["moments"][:, 1:]
        return out
    if kind == "newton_host":
        r = ctx.newton_dc(s["circuit"], s["cfg"], s["seed"], case["samples"])
        return dict(x=r.x, iters=r.iters, status=r.status, resid=r.resid)
    if kind == "lu":
        ctx.solve_batch_device(s["A"], s["rhs"], case["n"], case["batch"], s["x"], s["sing"],
                               precision=PREC[case["precision"]], stream=_stream())
        return dict(x=s["x"], sing=s["sing"])
    if kind == "ac":
        ctx.ac_sweep_device(s["topo"], s["cfg"], s["ac"], s["seed"], case["samples"], s["probe"], s["status"],
                            stream=_stream())
        return dict(probe=s["probe"], status=s["status"])
    if kind == "transient":
        ctx.transient_device(s["topo"], s["cfg"], s["tc"], s["seed"], case["samples"], s["x"], s["status"],
                             probe=s["probe"], stream=_stream())
        return dict(x=s["x"], probe=s["probe"], status=s["status"])
    if kind == "ladder":
        o = s["out"]
        ctx.ladder_transient_device(s["cfg"], s["seed"], case["count"], o["x"], o["n"], o["accepted"], o["rejected"],
                                    o["iterations"], o["status"], probe=o["probe"], stream=_stream())
        return dict(o)
    if kind == "grid":
        o = s["out"]
        ctx.grid_solve_device(s["cfg"], s["seed"], case["count"], o["x"], o["newton"], o["krylov"], o["status"],
                              o["resid"], stream=_stream())
        return dict(o)
    s["mlp"].gradients_device(s["X"], s["T"], case["rows"], s["grads"], s["loss"], stream=_stream())
    return dict(grads=s["grads"], loss=s["loss"])


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------


def work(case):
    kind = case["kind"]
    if kind in ("newton", "newton_host"):
        n, draws, its = {"cs_nmos": (5, 4, 5), "opamp": (12, 17, 3), "bsim3_chain": (6, 7, 42)}[case["circuit"]]
        k = case["samples"]
        # outputs written once; draws (~100 operations each) and its Newton steps on a sparse system (~12 n^2)
        return dict(bytes=k * (8 * n + 13), flops=k * (100 * draws + its * 12 * n * n))
    if kind == "lu":
        n, b = case["n"], case["batch"]
        return dict(bytes=8 * b * (n * n + 2 * n) + b, flops=b * (2 * n ** 3 / 3 + 2 * n * n))
    if kind == "ac":
        k, nf = case["samples"], 8 * case["per_decade"] + 1
        return dict(bytes=k * nf * 32 + k, flops=k * nf * 12.0 * 12 * 8)  # one sparse complex solve per point
    if kind == "transient":
        k, stages = case["samples"], 2 if case["method"] == 2 else 1
        return dict(bytes=k * (8 * (case["steps"] + 10) + 1), flops=k * case["steps"] * stages * 2.0 * 9 * 9)
    if kind == "ladder":
        # about 300 steps of two stages with two Newton iterations, some 60 operations per section
        k, sec = case["count"], (8 + case["max_sections"]) / 2
        return dict(bytes=k * 8 * (case["max_sections"] + 2 + 101), flops=k * 300.0 * 4 * 60 * sec)
    if kind == "grid":
        # Arnoldi steps (grows with the mesh's diameter) of a stencil and one orthogonalisation pass
        k, n = case["count"], case["rows"] * case["cols"] + 1
        steps = 20.0 * max(case["rows"], case["cols"])
        return dict(bytes=k * 8 * n, flops=k * steps * n * (10 + 4 * 15))
    h, r = case["hidden"], case["rows"]
    w = 17 * h + 2 * h * h + 12 * h
    return dict(bytes=4 * (r * 29 + 2 * w), flops=6.0 * r * w)


# ---------------------------------------------------------------------------
# 64-bit results
# ---------------------------------------------------------------------------
_K1, _K2 = 0x517CC1B727220A95, 0x5851F42D4C957F2D


def _i64(v):
    v &= (1 << 64) - 1
    return v - (1 << 64) if v >= 1 << 63 else v


def _shr(x, k):
    return (x >> k) & ((1 << (64 - k)) - 1)


def _uniform(seed, sweep, param):
    """Hash-RNG uniforms of sweep indices `sweep` (int64 tensor) and parameter indices `param`."""
    x = sweep * _i64(_K1)
    x = x ^ (_i64(param * _K2) if isinstance(param, int) else param * _i64(_K2)) ^ _i64(seed)
    x = x + _i64(0x9E3779B97F4A7C15)
    x = (x ^ _shr(x, 30)) * _i64(0xBF58476D1CE4E5B9)
    x = (x ^ _shr(x, 27)) * _i64(0x94D049BB133111EB)
    x = x ^ _shr(x, 31)
    return _shr(x, 11).to(F64) * 2.0 ** -53


def _value(spec, seed, sweep):
    if not isinstance(spec, tuple):
        return torch.full(sweep.shape, float(spec), dtype=F64, device=sweep.device)
    kind, a, b, idx = spec
    if kind == "G":
        u1 = _uniform(seed, sweep, 2 * idx).clamp(min=1e-10)
        u2 = _uniform(seed, sweep, 2 * idx + 1)
        return a + torch.sqrt(-2.0 * torch.log(u1)) * torch.cos(6.283185307179586 * u2) * b
    u = _uniform(seed, sweep, idx)
    return a + u * (b - a) if kind == "U" else a * torch.exp(u * math.log(b / a))


class _Net:
    """A circuit's MNA bookkeeping and the drawn values of `count` samples."""

    def __init__(self, name, seed, count):
        self.els, nodeset = ELEMENTS[name]()
        self.index, nb = {}, 0
        for _, _, nodes, _, _ in self.els:
            for nm in nodes:
                if nm != "0" and nm not in self.index:
                    self.index[nm] = len(self.index)
        self.nn, self.branch = len(self.index), {}
        for kind, nm, _, _, _ in self.els:
            if kind in "VL":
                self.branch[nm] = self.nn + nb
                nb += 1
        self.n = self.nn + nb
        sweep = torch.arange(count, dtype=torch.int64, device=DEV)
        self.val = {nm: [_value(v, seed, sweep) for v in vals] for _, nm, _, vals, _ in self.els}
        self.start = torch.zeros(self.n, dtype=F64, device=DEV)
        for nm, v in nodeset.items():
            self.start[self.index[nm]] = v

    def nodes(self, nodes):
        return [self.index.get(nm, -1) for nm in nodes]

    def add(self, A, r, c, v):
        if r >= 0 and c >= 0:
            A[:, r, c] += v

    def cond(self, A, i, j, g):
        self.add(A, i, i, g), self.add(A, j, j, g), self.add(A, i, j, -g), self.add(A, j, i, -g)

    def mos(self, kind, nm, nodes, x):
        """(ids, gds, gm, vgs, vds) of a Level-1 MOSFET at x."""
        d, g, s = self.nodes(nodes)
        v = lambda i: x[:, i] if i >= 0 else torch.zeros_like(x[:, 0])  # noqa: E731
        vto, kp, lam, w = self.val[nm]
        beta, vth, sign = kp * w / 1e-6, vto.abs(), -1.0 if kind == "P" else 1.0
        vgs, vds = sign * (v(g) - v(s)), sign * (v(d) - v(s))
        vov, q = vgs - vth, 1.0 + lam * vds
        off, lin = vgs < vth, vds < vgs - vth
        quad = vov * vds - 0.5 * vds * vds
        ids = torch.where(lin, beta * quad * q, 0.5 * beta * vov * vov * q)
        gds = torch.where(lin, beta * (vov - vds) * q + beta * quad * lam, 0.5 * beta * vov * vov * lam)
        gm = torch.where(lin, beta * vds * q, beta * vov * q)
        z = torch.zeros_like(ids)
        ids, gds, gm = torch.where(off, z, ids), torch.where(off, z, gds).clamp(min=1e-12), torch.where(off, z, gm)
        return sign * ids, gds, gm, sign * vgs, sign * vds

    def newton(self, x):
        """Plain Newton with the sweep's convergence test; (x, converged operating point, KCL residual)."""
        B = x.shape[0]
        done = torch.zeros(B, dtype=torch.bool, device=DEV)
        for _ in range(50):
            A = torch.zeros((B, self.n, self.n), dtype=F64, device=DEV)
            b = torch.zeros((B, self.n), dtype=F64, device=DEV)
            for kind, nm, nodes, _, _ in self.els:
                idx, val = self.nodes(nodes), self.val[nm]
                if kind == "R":
                    self.cond(A, idx[0], idx[1], 1.0 / val[0])
                elif kind in "VL":
                    br = self.branch[nm]
                    self.add(A, idx[0], br, 1.0), self.add(A, br, idx[0], 1.0)
                    self.add(A, idx[1], br, -1.0), self.add(A, br, idx[1], -1.0)
                    if kind == "V":
                        b[:, br] += val[0]
                elif kind == "I":
                    for k, sg_ in ((0, -1.0), (1, 1.0)):
                        if idx[k] >= 0:
                            b[:, idx[k]] += sg_ * val[0]
                elif kind in "NP":
                    ids, gds, gm, vgs, vds = self.mos(kind, nm, nodes, x)
                    d, g, s = idx
                    self.cond(A, d, s, gds)
                    self.add(A, d, g, gm), self.add(A, d, s, -gm), self.add(A, s, g, -gm), self.add(A, s, s, gm)
                    ieq = ids - gds * vds - gm * vgs
                    if d >= 0:
                        b[:, d] -= ieq
                    if s >= 0:
                        b[:, s] += ieq
            xn = torch.linalg.solve(A, b)
            tol = 1e-3 * torch.maximum(xn.abs(), x.abs())
            tol[:, :self.nn] += 1e-6
            tol[:, self.nn:] += 1e-12
            ok = ((xn - x).abs() <= tol).all(1)
            x = torch.where(done[:, None], x, xn)
            done |= ok
            if bool(done.all()):
                break
        return x, done

    def conductances(self, A, x):
        """Real small-signal stamps at x into A, as Newton's without the equivalent currents."""
        for kind, nm, nodes, _, _ in self.els:
            idx, val = self.nodes(nodes), self.val[nm]
            if kind == "R":
                self.cond(A, idx[0], idx[1], 1.0 / val[0])
            elif kind in "VL":
                br = self.branch[nm]
                self.add(A, idx[0], br, 1.0), self.add(A, br, idx[0], 1.0)
                self.add(A, idx[1], br, -1.0), self.add(A, br, idx[1], -1.0)
            elif kind in "NP":
                _, gds, gm, _, _ = self.mos(kind, nm, nodes, x)
                d, g, s = idx
                self.cond(A, d, s, gds)
                self.add(A, d, g, gm), self.add(A, d, s, -gm), self.add(A, s, g, -gm), self.add(A, s, s, gm)


_FIT = {}


def linear_fit(name):
    """(input means, linear term [n][inputs], output means) of the least-squares
    warm start on 4,096 operating points of seed 7."""
    if name not in _FIT:
        net = _Net(name, 7, 4096)
        x, ok = net.newton(net.start.expand(4096, -1).clone())
        P, mean = [], []
        for _, nm, _, vals, _ in net.els:
            for v, spec in zip(net.val[nm], vals):
                if isinstance(spec, tuple):
                    P.append(v)
                    mean.append(spec[1] if spec[0] == "G" else 0.5 * (spec[1] + spec[2]))
        P = torch.stack(P, 1)[ok].cpu().numpy() - np.array(mean)
        scale = P.std(0)
        A = np.column_stack([P / scale, np.ones(len(P))])
        coef = np.linalg.lstsq(A, x[ok].cpu().numpy(), rcond=None)[0]
        _FIT[name] = (np.array(mean), (coef[:-1] / scale[:, None]).T.copy(), coef[-1].copy())
    return _FIT[name]


def _exact_newton(case, seed):
    if case["circuit"] == "bsim3_chain":
        return None
    k = case["samples"]
    net = _Net(case["circuit"], seed, k)
    start = net.start.expand(k, -1).clone()
    if case.get("warm") == "linear":
        mean, lin, outm = (torch.as_tensor(a, dtype=F64, device=DEV) for a in linear_fit(case["circuit"]))
        P = torch.stack([v for _, nm, _, vals, _ in net.els for v, spec in zip(net.val[nm], vals)
                         if isinstance(spec, tuple)], 1)
        start = outm + (P - mean) @ lin.T
    x, _ = net.newton(start)
    out = dict(x=x, iters=None, status=None)
    if case["kind"] == "newton_host":
        return dict(x=x.cpu().numpy(), iters=None, status=None, resid=None)
    if case["resid"]:
        out["resid"] = None  # a rounding residue: it has no value of its own
    if case["moments"]:
        out["count"] = None
        out["moments"] = torch.stack([x.sum(0), (x * x).sum(0), x.min(0).values, x.max(0).values], 1)
    return out


def _exact_lu(case, seed):
    A, rhs = _lu_system(case, seed)
    x = torch.empty_like(rhs)
    for i in range(0, len(A), 4096):
        x[i:i + 4096] = torch.linalg.solve(A[i:i + 4096], rhs[i:i + 4096])
    return dict(x=x, sing=None)


def _exact_ac(case, seed):
    k = case["samples"]
    net = _Net("opamp", seed, k)
    x, _ = net.newton(net.start.expand(k, -1).clone())
    G = torch.zeros((k, net.n, net.n), dtype=F64, device=DEV)
    net.conductances(G, x)
    C = torch.zeros_like(G)
    b = torch.zeros((k, net.n), dtype=torch.complex128, device=DEV)
    for kind, nm, nodes, _, _ in net.els:
        if kind == "C":
            i, j = net.nodes(nodes)
            net.cond(C, i, j, net.val[nm][0])
        elif kind == "V":
            b[:, net.branch[nm]] += 1.0
    ppd = case["per_decade"]
    out = []
    for i in range(8 * ppd + 1):
        f = 10.0 * 10.0 ** (i / ppd)
        h = torch.linalg.solve(torch.complex(G, 2.0 * math.pi * f * C), b)
        out.append(torch.view_as_real(h[:, [net.index["out"], net.index["n2"]]]))
    return dict(probe=torch.stack(out, 1), status=None)


def _tran_net(case):
    return "rc" if case["method"] == 2 else "rlc"


def _tstop(case):
    return TRAN_H * (case["steps"] - 0.5)  # ceil(tstop / h) is the step count, whatever its rounding


def _pulse(p, t):
    v1, v2, td, tr, tf, pw, per = p
    if t < td:
        return v1
    r = math.fmod(t - td, per)
    if r < tr:
        return v1 + (v2 - v1) * r / tr
    if r < tr + pw:
        return v2
    if r < tr + pw + tf:
        return v2 - (v2 - v1) * (r - tr - pw) / tf
    return v1


def _exact_transient(case, seed):
    """DC operating point, then fixed steps of BE, TRAP or TR-BDF2 with the
    companion models and state updates the fixed-step solver states."""
    k, h = case["samples"], TRAN_H
    net = _Net(_tran_net(case), seed, k)
    dc, _ = net.newton(net.start.expand(k, -1).clone())
    vsrc = [e[1] for e in net.els if e[0] == "V"]
    nt = net.nn + len(vsrc)
    v_of = lambda x, i: x[:, i] if i >= 0 else torch.zeros(k, dtype=F64, device=DEV)  # noqa: E731
    gamma = 2.0 - math.sqrt(2.0)
    rho = (1.0 - gamma) / gamma
    den = 1.0 + 2.0 * rho
    a1, a2, b0 = (1.0 + rho) ** 2 / den, -rho * rho / den, (1.0 + rho) / den
    h2, hg, alpha = (1.0 - gamma) * h, gamma * h, (1.0 - gamma) / (gamma * (2.0 - gamma))
    st = {}
    x = torch.empty((k, nt), dtype=F64, device=DEV)
    x[:, :net.nn] = dc[:, :net.nn]
    for j, nm in enumerate(vsrc):
        x[:, net.nn + j] = dc[:, net.branch[nm]]
    for kind, nm, nodes, _, _ in net.els:
        if kind in "CL":
            i, j = net.nodes(nodes)
            zero = torch.zeros(k, dtype=F64, device=DEV)
            st[nm] = [v_of(dc, i) - v_of(dc, j), dc[:, net.branch[nm]].clone() if kind == "L" else zero, zero]

    def geq(kind, nm, stage):
        v = net.val[nm][0]
        if stage == 0:
            return v / h if kind == "C" else h / v
        if stage == 1:
            hh = hg if case["method"] == 2 else h
            return 2.0 * v / hh if kind == "C" else hh / (2.0 * v)
        return v / (b0 * h2) if kind == "C" else b0 * h2 / v

    def matrix(stage):
        A = torch.zeros((k, nt, nt), dtype=F64, device=DEV)
        for kind, nm, nodes, _, _ in net.els:
            idx = net.nodes(nodes)
            if kind == "R":
                net.cond(A, idx[0], idx[1], 1.0 / net.val[nm][0])
            elif kind in "CL":
                net.cond(A, idx[0], idx[1], geq(kind, nm, stage))
            elif kind == "V":
                row = net.nn + vsrc.index(nm)
                for i, sgn in zip(idx, (1.0, -1.0)):
                    net.add(A, i, row, sgn), net.add(A, row, i, sgn)
        return torch.linalg.lu_factor(A)

    def solve(stage, t):
        b = torch.zeros((k, nt), dtype=F64, device=DEV)

        def inject(i, cur):
            if i >= 0:
                b[:, i] += cur

        for kind, nm, nodes, _, pulse in net.els:
            idx = net.nodes(nodes)
            src = _pulse(pulse, t) if pulse else net.val[nm][0]
            if kind == "V":
                b[:, net.nn + vsrc.index(nm)] = src
            elif kind == "I":
                inject(idx[0], -src), inject(idx[1], src)
            elif kind in "CL":
                v, i, pp = st[nm]
                g = geq(kind, nm, stage)
                if kind == "C":
                    ieq = g * v if stage == 0 else g * v + i if stage == 1 else g * (a1 * v + a2 * pp)
                    inject(idx[0], ieq), inject(idx[1], -ieq)
                else:
                    ieq = i if stage == 0 else i + g * v if stage == 1 else a1 * i + a2 * pp
                    inject(idx[0], -ieq), inject(idx[1], ieq)
        return torch.linalg.lu_solve(*lu[stage], b[:, :, None])[:, :, 0]

    method = case["method"]
    lu = {q: matrix(q) for q in ((1, 2) if method == 2 else (method,))}
    probe = [x[:, net.index["c"]].clone()]
    for step in range(1, case["steps"] + 1):
        t = step * h
        if method == 2:
            y = solve(1, t)
            for kind, nm, nodes, _, _ in net.els:
                if kind in "CL":
                    i, j = net.nodes(nodes)
                    v, c, _ = st[nm]
                    nv, val = v_of(y, i) - v_of(y, j), net.val[nm][0]
                    st[nm] = [nv, 2.0 * val / hg * (nv - v) - c, v] if kind == "C" else \
                        [nv, c + hg / (2.0 * val) * (nv + v), c]
        x = solve(method, t)
        for kind, nm, nodes, _, _ in net.els:
            if kind in "CL":
                i, j = net.nodes(nodes)
                v, c, pp = st[nm]
                nv, val = v_of(x, i) - v_of(x, j), net.val[nm][0]
                if kind == "C":
                    nc = (val / h * (nv - v), 2.0 * val / h * (nv - v) - c,
                          val / h * ((1.0 + alpha) * nv - (1.0 + 2.0 * alpha) * v + alpha * pp))[method]
                    st[nm] = [nv, nc, v]
                else:
                    nc = c + (h / val * nv, h / (2.0 * val) * (nv + v),
                              h / val * ((1.0 + alpha) * nv - (1.0 + 2.0 * alpha) * v + alpha * v))[method]
                    st[nm] = [nv, nc, nc]
        probe.append(x[:, net.index["c"]].clone())
    return dict(x=x, probe=torch.stack(probe, 1), status=None)


def _exact_grid(case, seed):
    """Newton on the mesh with each linear system solved by block elimination
    over its rows (the driven corner's voltage is known, so the straps are
    diagonal terms)."""
    R, C, K, S = case["rows"], case["cols"], case["count"], case["sinks"]
    if R * C * C * C * K > 3e10:
        return None
    inst = torch.arange(K, dtype=torch.int64, device=DEV)
    lay, corner = inst // 4, inst % 4
    nh, nv, nn = R * (C - 1), (R - 1) * C, R * C
    e = torch.arange(nh + nv, dtype=torch.int64, device=DEV)
    scale = torch.where(corner % 2 == 1, 1.1, 0.9).to(F64)[:, None]
    g = 1.0 / (0.5 * torch.exp(_uniform(seed, lay[:, None], e[None, :]) * math.log(4.0)) * scale)
    gh, gv = g[:, :nh].reshape(K, R, C - 1), g[:, nh:].reshape(K, R - 1, C)
    si = nh + nv + 2 * torch.arange(S, dtype=torch.int64, device=DEV)
    node = torch.floor(nn * _uniform(seed, lay[:, None], si[None, :])).to(torch.int64)
    vov = 0.8 + _uniform(seed, lay[:, None], si[None, :] + 1) * (1.2 - 0.8)
    vov = vov - torch.where(corner >= 2, 0.75, 0.65).to(F64)[:, None]
    beta, lam = 110e-6 * 5e-6 / 0.5e-6, 0.04
    base = torch.zeros((K, R, C), dtype=F64, device=DEV)
    base[:, :, 1:] += gh
    base[:, :, :-1] += gh
    base[:, 1:] += gv
    base[:, :-1] += gv
    for r, c in ((0, C - 1), (R - 1, 0), (R - 1, C - 1)):
        base[:, r, c] += 1e3
    x = torch.zeros((K, nn), dtype=F64, device=DEV)
    done = torch.zeros(K, dtype=torch.bool, device=DEV)
    isrc = torch.zeros(K, dtype=F64, device=DEV)
    for _ in range(30):
        vds = torch.gather(x, 1, node)
        lin, q = vds < vov, 1.0 + lam * vds
        quad = vov * vds - 0.5 * vds * vds
        ids = torch.where(lin, beta * quad * q, 0.5 * beta * vov * vov * q)
        gds = torch.where(lin, beta * (vov - vds) * q + beta * quad * lam, 0.5 * beta * vov * vov * lam).clamp(min=1e-12)
        d = base.reshape(K, nn).clone().scatter_add_(1, node, gds).reshape(K, R, C)
        b = torch.zeros((K, nn), dtype=F64, device=DEV).scatter_add_(1, node, gds * vds - ids)
        d0, b0 = d[:, 0, 0].clone(), b[:, 0].clone()
        b = b.reshape(K, R, C)
        # node 0 is the driven corner at 1 V: its row is replaced, its neighbours get its current
        b[:, 0, 1] += gh[:, 0, 0]
        b[:, 1, 0] += gv[:, 0, 0]
        for r, c in ((0, C - 1), (R - 1, 0), (R - 1, C - 1)):
            b[:, r, c] += 1e3
        b[:, 0, 0], d[:, 0, 0] = 1.0, 1.0
        up = gv.clone()
        up[:, 0, 0] = 0.0
        side = gh.clone()
        side[:, 0, 0] = 0.0
        D, F = [], []
        for r in range(R):
            M = torch.diag_embed(d[:, r])
            M -= torch.diag_embed(side[:, r], 1) + torch.diag_embed(side[:, r], -1)
            f = b[:, r].clone()
            if r:
                W = torch.linalg.solve(D[-1], torch.cat([torch.diag_embed(up[:, r - 1]), F[-1][:, :, None]], 2))
                M -= up[:, r - 1][:, :, None] * W[:, :, :C]
                f += up[:, r - 1] * W[:, :, C]
            D.append(M)
            F.append(f)
        y = [None] * R
        for r in reversed(range(R)):
            f = F[r] if r == R - 1 else F[r] + up[:, r] * y[r + 1]
            y[r] = torch.linalg.solve(D[r], f)
        xn = torch.stack(y, 1).reshape(K, nn)
        cur = b0 - d0 * xn[:, 0] + gh[:, 0, 0] * xn[:, 1] + gv[:, 0, 0] * xn[:, C]
        for p in (C - 1, (R - 1) * C, nn - 1):
            cur += 1e3 * (xn[:, p] - xn[:, 0])
        ok = ((xn - x).abs() <= 1e-3 * torch.maximum(xn.abs(), x.abs()) + 1e-6).all(1)
        ok &= (cur - isrc).abs() <= 1e-3 * torch.maximum(cur.abs(), isrc.abs()) + 1e-12
        x, isrc = torch.where(done[:, None], x, xn), torch.where(done, isrc, cur)
        done |= ok
        if bool(done.all()):
            break
    return dict(x=torch.cat([x, isrc[:, None]], 1), newton=None, krylov=None, status=None, resid=None)


def _mlp_data(case, seed):
    g = _gen(seed)
    rows, h = case["rows"], case["hidden"]
    X = torch.randn((rows, 17), device=DEV, generator=g)
    T = torch.randn((rows, 12), device=DEV, generator=g) * 0.5
    flat = []
    for out, inp, ro, ri in ((h, 32, h, 17), (h, h, h, h), (h, h, h, h), (32, h, 12, h)):
        W = torch.zeros((out, inp), device=DEV)
        W[:ro, :ri] = (torch.rand((ro, ri), device=DEV, generator=g) * 2.0 - 1.0) * math.sqrt(6.0 / ri)
        flat += [W.reshape(-1), torch.zeros(out, device=DEV)]
    return X, T, torch.cat(flat)


def _exact_mlp(case, seed):
    X, T, flat = _mlp_data(case, seed)
    h, flat = case["hidden"], flat.to(F64).requires_grad_(True)
    a, o = torch.nn.functional.pad(X.to(F64), (0, 15)), 0
    shapes = ((h, 32), (h, h), (h, h), (32, h))
    for i, (r, c) in enumerate(shapes):
        W, b = flat[o:o + r * c].reshape(r, c), flat[o + r * c:o + r * c + r]
        o += r * c + r
        a = a @ W.T + b
        if i < 3:
            a = torch.nn.functional.gelu(a, approximate="tanh")
    loss = ((a[:, :12] - T.to(F64)) ** 2).mean()
    loss.backward()
    return dict(grads=flat.grad, loss=loss.detach().reshape(1))


def exact(case, seed):
    kind = case["kind"]
    if kind == "ladder":  # thousands of dependent adaptive steps: minutes in plain torch
        return None
    return dict(newton=_exact_newton, newton_host=_exact_newton, lu=_exact_lu, ac=_exact_ac,
                transient=_exact_transient, grid=_exact_grid, mlp=_exact_mlp)[kind](case, seed)
