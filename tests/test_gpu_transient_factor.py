"""Fixed-step transients on the factors kept from the first step: the same bits
as the oracle's per-step solve in the exact mode, over both edges of the sample
blocks, several element orders, singular circuits, and more pulse sources than
the waveform table holds."""
import numpy as np
import pytest

import oracle
from spicier_gb300 import abi
from spicier_gb300.circuit import Circuit, Gauss, LogUniform, Pulse

pytestmark = pytest.mark.gpu

PULSE = Pulse(0.0, 1.0, 2e-6, 1e-6, 1e-6, 5e-6, 15e-6)


def sources_last():
    """Reactive elements first, sources last and reversed, a node tied by inductors only."""
    c = Circuit("sources_last")
    c.Cap("C1", "a", "b", LogUniform(1e-9, 1e-8, 0))
    c.L("L1", "b", "0", 1e-5)
    c.L("L2", "a", "b", LogUniform(1e-6, 1e-5, 1))
    c.R("R1", "a", "in", Gauss(100.0, 5.0, 2))
    c.R("R2", "b", "0", 1e3)
    c.Cap("C2", "0", "a", 1e-9)
    c.I("I1", "a", "b", Gauss(1e-4, 1e-5, 3), pulse=PULSE)
    c.V("V1", "0", "in", Gauss(0.5, 0.01, 4), pulse=PULSE)
    c.I("I2", "0", "b", 1e-5)
    return c


def many_pulses(k):
    c = Circuit("many_pulses")
    c.V("V1", "in", "0", 0.0, pulse=PULSE)
    c.R("R1", "in", "out", Gauss(1e3, 10.0, 0))
    c.Cap("C1", "out", "0", 1e-9)
    for i in range(k):
        c.I(f"I{i}", "0", "out", 0.0, pulse=Pulse(0.0, 1e-6 * (i % 7), 1e-6 * (i % 5), 1e-6, 1e-6, 2e-6, 9e-6))
    return c


def two_sources(k):
    """Two parallel V sources: the matrix is singular, DC point included (k = 0), or
    only in the transient, where the inductor across a source is a conductance (k = 1)."""
    c = Circuit("two_sources")
    c.V("V1", "in", "0", 1.0)
    if k == 0:
        c.V("V2", "in", "0", 1.0)
    c.R("R1", "in", "out", 1e3)
    c.Cap("C1", "out", "x", 1e-9)
    if k == 1:
        c.Cap("C2", "x", "out", 1e-9)
    c.R("R2", "out", "0", 1e3)
    c.R("R3", "x", "0", 1e6)
    return c


CIRCUITS = {"sources_last": sources_last, "pulses_17": lambda: many_pulses(17), "pulses_600": lambda: many_pulses(600),
            "singular": lambda: two_sources(0), "parallel_caps": lambda: two_sources(1)}


@pytest.mark.parametrize("method", [abi.SP_TRAN_BE, abi.SP_TRAN_TRAP, abi.SP_TRAN_TRBDF2])
@pytest.mark.parametrize("name", list(CIRCUITS))
def test_bits_of_the_per_step_solve(ctx, name, method):
    c = CIRCUITS[name]()
    count, probe = 33, c.num_nodes - 1
    cfg = abi.transient_config(0.2e-6, 13.1e-6, method, probe, abi.SP_PREC_FP64_EXACT)  # 66 steps: two waveform tables and a rest
    dc = abi.newton_config(precision=abi.SP_PREC_FP64_EXACT)
    g = ctx.transient(c, dc, cfg, 2, count)
    with oracle.math_mode("cr"):
        x, pr, st = oracle.transient(c, dc, 2, count, method, 0.2e-6, 13.1e-6, probe_idx=probe)
    assert np.array_equal(g["status"], st)
    ok = (st & abi.SP_ST_MASK) == 0
    assert ok.all() == (name != "singular")
    assert np.array_equal(g["x"][ok].view(np.uint64), x[ok].view(np.uint64))
    assert np.array_equal(g["probe"][ok].view(np.uint64), pr[ok].view(np.uint64))
    # the contracted build: the same steps to rounding, growing with the number of steps
    cfg.precision = abi.SP_PREC_FP64
    f = ctx.transient(c, abi.newton_config(), cfg, 2, count)
    assert np.array_equal(f["status"], st)
    scale = max(1.0, np.abs(pr[ok]).max()) if ok.any() else 1.0
    if ok.any():
        assert np.abs(f["probe"][ok] - pr[ok]).max() <= 1e-9 * scale
