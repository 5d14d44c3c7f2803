"""Samples of a team of lanes that turn non-finite: they walk the whole fallback chain
(a NaN iterate passes the convergence test, so every gmin level "converges" and the
source ramp follows) and end with the status, iterations and bits of single lanes."""
import numpy as np
import pytest

import oracle
from spicier_gb300 import abi
from spicier_gb300.circuit import Circuit, Table


def chain(devices):
    c = Circuit(f"b3_table_{devices}")
    c.V("VDD", "vdd", "0", 1.8)
    c.V("VIN", "n0", "0", Table(0))
    for i in range(devices):
        pmos = bool(i % 2)
        s = "vdd" if pmos else "0"
        c.B3(f"M{i}", f"n{i + 1}", f"n{i}", s, s, pmos=pmos, vth0=Table(1 + i), w=2e-6)
        c.R(f"R{i}", f"n{i + 1}", "0" if pmos else "vdd", 1e4)
    return c


def table(devices, rows):
    """Half of the rows hold a NaN or an infinite threshold somewhere."""
    rng = np.random.default_rng(devices)
    vth = np.where(np.arange(devices) % 2, -0.4, 0.4) + rng.normal(0.0, 0.02, (rows, devices))
    bad = np.array([np.nan, np.inf, -np.inf])
    vth[np.arange(0, rows, 2), rng.integers(0, devices, (rows + 1) // 2)] = bad[rng.integers(0, 3, (rows + 1) // 2)]
    return np.column_stack([rng.normal(0.8, 0.05, rows), vth])


@pytest.mark.gpu
@pytest.mark.parametrize("devices", [2, 5])
@pytest.mark.parametrize("prec", [abi.SP_PREC_MIXED, abi.SP_PREC_FP64])
def test_nonfinite_samples_of_a_team(ctx, devices, prec):
    c, few = chain(devices), 67
    # 20,000 rows: no teams, and a fallback list of some 10,000 samples, too long for them
    T = np.tile(table(devices, few), (300, 1))[:20000]
    cfg = abi.newton_config(precision=prec)
    a, b = ctx.newton_dc(c, cfg, 1, few, table=T[:few]), ctx.newton_dc(c, cfg, 1, len(T), table=T)
    for f in ("iters", "status"):
        assert np.array_equal(getattr(a, f), getattr(b, f)[:few]), f
    for f in ("x", "resid"):
        u, v = getattr(a, f), getattr(b, f)[:few]
        nan = np.isnan(v)
        assert np.array_equal(np.isnan(u), nan) and np.array_equal(u[~nan], v[~nan]), f
    nanrow = np.isnan(T[:few]).any(axis=1)
    both = abi.SP_ST_FLAG_GMIN | abi.SP_ST_FLAG_SOURCE
    assert nanrow.any() and (a.status[nanrow] == (abi.SP_ST_NONFINITE | both)).all()
    with oracle.math_mode("cr"):
        _, it, st, _ = oracle.newton_dc(c, abi.newton_config(), seed=1, count=few, table=T[:few])
    assert np.array_equal(a.status[nanrow], st[nanrow]) and np.array_equal(a.iters[nanrow], it[nanrow])
