"""Level-1 MOSFETs whose threshold, KP, LAMBDA or width is NaN, infinite or zero:
the generic Newton kernels give such samples the status, iterations and bits of
the dense solve, and the status of the exact mode."""
import numpy as np
import pytest

from spicier_gb300 import abi
from spicier_gb300.circuit import Circuit, Table

pytestmark = pytest.mark.gpu


def stages():
    """An NMOS stage that drives a PMOS stage, every model value from the table."""
    c = Circuit("table_mos")
    c.V("VDD", "vdd", "0", 3.0)
    c.V("VIN", "in", "0", Table(8))
    c.R("R1", "vdd", "a", 1e4)
    c.M("M1", "a", "in", "0", vto=Table(0), kp=Table(1), lam=Table(2), w=Table(3))
    c.M("M2", "b", "a", "vdd", pmos=True, vto=Table(4), kp=Table(5), lam=Table(6), w=Table(7))
    c.R("R2", "b", "0", 1e4)
    return c


def table():
    """A plain row, then one extreme value at a time in every column, then rows of several."""
    plain = np.array([0.7, 1e-4, 0.02, 1e-5, -0.8, 5e-5, 0.02, 2e-5, 1.2])
    extreme = np.array([np.nan, -np.nan, np.inf, -np.inf, 0.0])
    rows = [plain]
    for col in range(8):
        for v in extreme:
            rows.append(plain.copy())
            rows[-1][col] = v
    rng = np.random.default_rng(11)
    several = np.where(rng.random((64, 8)) < 0.25, extreme[rng.integers(0, len(extreme), (64, 8))], plain[:8])
    rows += [np.append(r, rng.uniform(0.0, 3.0)) for r in several]
    return np.array(rows)


@pytest.mark.parametrize("precision", [abi.SP_PREC_FP64, abi.SP_PREC_MIXED])
def test_nonfinite_mos_parameters(ctx, precision, monkeypatch):
    monkeypatch.setenv("SPICIER_GB300_GENERIC", "1")
    c, T = stages(), table()
    count = len(T)
    g = ctx.newton_dc(c, abi.newton_config(precision=precision, fallback=0), 1, count, table=T)
    # the dense solve: the fallback kernel's cold restart of a sample whose far start, capped at one iteration, misses
    x0 = np.random.default_rng(3).uniform(100.0, 200.0, (count, c.n))
    d = ctx.newton_dc(c, abi.newton_config(precision=precision, fallback=0, warm_max_iterations=1), 1, count, table=T, x0=x0)
    e = ctx.newton_dc(c, abi.newton_config(precision=abi.SP_PREC_FP64_EXACT, fallback=0), 1, count, table=T)
    assert np.array_equal(g.status == abi.SP_ST_NONFINITE, e.status == abi.SP_ST_NONFINITE)
    if precision == abi.SP_PREC_FP64:
        assert np.array_equal(g.status, e.status)
    cold = (d.status & abi.SP_ST_FLAG_COLD) != 0
    assert cold.sum() >= count // 2
    assert np.array_equal(g.status[cold], d.status[cold] & abi.SP_ST_MASK)
    assert np.array_equal(g.iters[cold], d.iters[cold] - 1)
    nan = np.isnan(d.x[cold])
    assert np.array_equal(np.isnan(g.x[cold]), nan)
    assert np.array_equal(g.x[cold][~nan], d.x[cold][~nan])
    # a NaN threshold is no cutoff
    assert (g.status[np.isnan(T[:, 0]) | np.isnan(T[:, 4])] == abi.SP_ST_NONFINITE).all()
    assert g.status[0] == abi.SP_ST_CONVERGED
