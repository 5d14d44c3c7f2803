"""FP64 AC sweeps on the circuit's pattern: the oracle's bits at every probed
unknown (zero parts' signs included), for purely real and purely imaginary
entries, units of one warp that pivot differently, systems that outgrow the
slots, and values the dense kernel has to take."""
import numpy as np
import pytest

import oracle
from spicier_gb300 import abi, configs
from spicier_gb300.api import Context
from spicier_gb300.circuit import Circuit, Gauss, LogUniform, Table

pytestmark = pytest.mark.gpu


def reactive():
    """Inductor loops and capacitor-only nodes (imaginary pivots), reversed elements."""
    c = Circuit("reactive")
    c.V("V1", "0", "in", 1.0)
    c.L("L1", "in", "a", LogUniform(1e-9, 1e-3, 0))
    c.Cap("C1", "a", "b", LogUniform(1e-15, 1e-6, 1))
    c.Cap("C2", "b", "0", LogUniform(1e-15, 1e-6, 2))
    c.R("R0", "b", "0", LogUniform(1.0, 1e9, 3))
    c.L("L2", "0", "a2", LogUniform(1e-9, 1e-3, 4))
    c.R("RL", "a2", "a", 1e-3)  # (two inductors across the source alone have no DC point)
    c.R("R1", "0", "a", LogUniform(1.0, 1e9, 5))
    c.V("V2", "x", "a", 0.0)
    c.R("R2", "x", "y", 50.0)
    c.R("R3", "y", "0", 1e12)
    return c


def mesh(nodes):
    """Every node tied to five others by R and C of widely spread values: fill, and pivots that differ."""
    c = Circuit(f"mesh{nodes}")
    c.V("V1", "a0", "0", 1.0)
    for i in range(nodes):
        for k, d in enumerate((1, 3, 7, 11, 13)):
            j = (i + d) % (nodes + 1)
            a, b = f"a{i}", (f"a{j}" if j < nodes else "0")
            if a == b:
                continue
            if (i + k) % 2:
                c.Cap(f"C{i}_{k}", a, b, LogUniform(1e-15, 1e-6, 10 * i + k))
            else:
                c.R(f"R{i}_{k}", a, b, LogUniform(1.0, 1e9, 10 * i + k))
        c.R(f"G{i}", f"a{i}", "0", 1e9)
    return c


def opamp_more():
    c = configs.miller_opamp()
    c.Cap("CL", "out", "0", Gauss(1e-12, 1e-13, 90))
    c.Cap("CT", "tail", "vss", 1e-13)
    return c


CASES = {"reactive": reactive, "mesh6": lambda: mesh(6), "mesh27": lambda: mesh(27), "opamp_more": opamp_more}


@pytest.mark.parametrize("count", [1, 5, 33])
@pytest.mark.parametrize("name", list(CASES))
def test_bits_at_every_unknown(ctx, name, count):
    c = CASES[name]()
    dc = abi.newton_config(precision=abi.SP_PREC_FP64_EXACT)
    for lo in range(0, c.n, 8):
        probes = list(range(lo, min(lo + 8, c.n)))
        cfg = abi.ac_config(1e1, 1e10, 3, abi.SP_AC_DEC, probes)
        h, st = ctx.ac_sweep(c, dc, cfg, 5, count)
        with oracle.math_mode("cr"):
            ho, so = oracle.ac_sweep(c, dc, 5, count, Context.ac_frequencies(cfg), probes)
        assert np.array_equal(st, so)
        ok = (st & abi.SP_ST_MASK) == 0
        assert ok.all()
        assert np.array_equal(h[ok].view(np.uint64), ho[ok].view(np.uint64)), (probes,)


def test_extreme_values_and_singular_points(ctx):
    """Infinite, zero and huge element values and a sample without a path: status and values as the oracle."""
    c = Circuit("extreme")
    c.V("V1", "in", "0", 1.0)
    c.R("R1", "in", "a", Table(0))
    c.Cap("C1", "a", "b", Table(1))
    c.R("R2", "b", "0", Table(2))
    c.L("L1", "b", "d", Table(3))
    c.R("R3", "d", "0", 1e3)
    rng = np.random.default_rng(2)
    vals = np.array([0.0, 1e300, 1e-300, 1e160, np.inf, -1e3, 1e-310])
    T = np.where(rng.random((150, 4)) < 0.25, vals[rng.integers(0, len(vals), (150, 4))],
                 10.0 ** np.column_stack([rng.uniform(0, 6, 150), rng.uniform(-15, -6, 150), rng.uniform(0, 6, 150),
                                          rng.uniform(-9, -3, 150)]))
    dc = abi.newton_config(precision=abi.SP_PREC_FP64_EXACT, fallback=0)
    probes = list(range(c.n))
    cfg = abi.ac_config(1e1, 1e9, 3, abi.SP_AC_DEC, probes)
    h, st = ctx.ac_sweep(c, dc, cfg, 1, 150, table=T)
    ho, so = oracle.ac_sweep(c, dc, 1, 150, Context.ac_frequencies(cfg), probes, table=T)
    assert np.array_equal(st, so)
    ok = (st & abi.SP_ST_MASK) == 0
    assert ok.sum() > 60
    g, w = h[ok].view(np.float64), ho[ok].view(np.float64)
    nan = np.isnan(w)
    assert np.array_equal(np.isnan(g), nan)
    assert np.array_equal(g[~nan].view(np.uint64), w[~nan].view(np.uint64))
