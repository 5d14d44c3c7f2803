"""The warp-wide sparse solve of the generic Newton kernels against the oracle's
dense one: sweeps that do not fill a warp, samples of one warp that pivot
differently, zero pivots, and parameters that make entries zero, infinite or NaN."""
import numpy as np
import pytest

import oracle
from spicier_gb300 import abi, configs
from spicier_gb300.circuit import Circuit, Gauss, LogUniform, Table

pytestmark = pytest.mark.gpu


def mesh28():
    """28 unknowns, the largest the kernels take: a resistor grid with two sources, a
    controlled path through MOSFETs, and widely spread resistances (pivot choices
    that differ from sample to sample)."""
    c = Circuit("mesh28")
    c.V("V1", "a0", "0", 3.0)
    for i in range(24):
        c.R(f"R{i}", f"a{i}", f"a{i + 1}", LogUniform(10.0, 1e6, i))
        c.R(f"S{i}", f"a{i + 1}", f"a{(7 * i + 3) % 25}", LogUniform(10.0, 1e6, 30 + i))
    c.V("V2", "b", "a12", Gauss(0.3, 0.05, 60))
    c.M("M1", "a20", "b", "0", vto=Gauss(0.7, 0.05, 61), kp=1e-4, lam=0.02)
    c.M("M2", "a24", "a24", "0", vto=0.6, kp=1e-4, lam=0.02)
    return c


def table_net():
    """Every element value from the table, so that a row can hold anything."""
    c = Circuit("table_net")
    c.V("V1", "in", "0", Table(0))
    c.R("R1", "in", "out", Table(1))
    c.R("R2", "out", "0", Table(2))
    c.R("R3", "out", "x", Table(3))
    c.R("R4", "x", "0", 1e3)
    c.M("M1", "out", "in", "0", vto=0.7, kp=1e-4, lam=0.02)
    c.I("I1", "0", "x", Table(4))
    return c


def floating():
    c = Circuit("floating")
    c.V("V1", "a", "0", 1.0)
    c.R("R1", "a", "b", Gauss(1e3, 10.0, 0))
    c.R("R2", "c", "d", 1e3)  # no path to ground
    return c


CIRCUITS = {"cs_nmos": configs.cs_nmos_amp, "opamp": configs.miller_opamp, "bjt_diode": configs.bjt_diode_bias,
            "bsim3": configs.bsim3_cmos_chain, "mesh28": mesh28, "floating": floating}


@pytest.mark.parametrize("count", [1, 31, 32, 33, 97])
@pytest.mark.parametrize("name", list(CIRCUITS))
def test_iterations_status_and_solution(ctx, name, count):
    c = CIRCUITS[name]()
    assert c.n <= 28
    cfg = abi.newton_config(fallback=0)
    with oracle.math_mode("cr"):
        x, it, st, _ = oracle.newton_dc(c, cfg, seed=3, count=count)
    g = ctx.newton_dc(c, cfg, 3, count)
    assert np.array_equal(g.status, st)
    assert np.array_equal(g.iters, it)
    ok = (st & abi.SP_ST_MASK) == abi.SP_ST_CONVERGED
    assert ok.any() == (name != "floating")
    scale = np.maximum(np.abs(x[ok]), 1e-9)
    assert (np.abs(g.x[ok] - x[ok]) <= 1e-9 * scale + 1e-13).all()


@pytest.mark.parametrize("precision", [abi.SP_PREC_FP64, abi.SP_PREC_MIXED])
def test_extreme_table_values(ctx, precision, monkeypatch):
    """Rows with zeros, infinities, NaN and huge or tiny values: the bits, status
    and iterations of the dense solve.  The dense solve runs in the fallback
    kernel, which restarts a sample cold when its warm start misses: a far start
    capped at one iteration misses."""
    monkeypatch.setenv("SPICIER_GB300_GENERIC", "1")
    rng = np.random.default_rng(5)
    vals = np.array([0.0, 1.0, 1e3, -1e3, 1e300, 1e-300, 1e-310, np.inf, -np.inf, np.nan])
    T = np.where(rng.random((200, 5)) < 0.3, vals[rng.integers(0, len(vals), (200, 5))],
                 10.0 ** rng.uniform(0, 4, (200, 5)))
    T[:8] = 100.0
    c = table_net()
    g = ctx.newton_dc(c, abi.newton_config(precision=precision, fallback=0), 1, 200, table=T)
    x0 = rng.uniform(100.0, 200.0, (200, c.n))
    d = ctx.newton_dc(c, abi.newton_config(precision=precision, fallback=0, warm_max_iterations=1), 1, 200, table=T, x0=x0)
    cold = (d.status & abi.SP_ST_FLAG_COLD) != 0
    # a NaN step passes the convergence test, and a linear sample converges at once from anywhere it lands
    assert cold.sum() >= 150
    assert np.array_equal(g.status[cold] & abi.SP_ST_MASK, d.status[cold] & abi.SP_ST_MASK)
    assert np.array_equal(g.iters[cold], d.iters[cold] - 1)
    gx, dx = g.x[cold], d.x[cold]
    nan = np.isnan(dx)
    assert np.array_equal(np.isnan(gx), nan)
    assert np.array_equal(gx[~nan], dx[~nan])
    assert {0, abi.SP_ST_NONFINITE, abi.SP_ST_SINGULAR} <= set((d.status[cold] & abi.SP_ST_MASK).tolist())
