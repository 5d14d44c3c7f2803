"""Fixed-step transients beyond everyday values: quotients of the kept factor near
the smallest doubles, samples whose matrix is singular only in the transient
beside regular ones, and more reactive elements than shared memory keeps
conductances for."""
import numpy as np
import pytest

import oracle
from spicier_gb300 import abi
from spicier_gb300.circuit import Circuit, Pulse, Table

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("amps", [1.0, 1e-300, 3e-305, 1e-306, 3e-308, 1e-310])
def test_quotients_are_ieee(ctx, amps):
    """A current step into R || C from rest: the first backward-Euler voltage is the
    amplitude over 1 / R + C / h, one division of the substitution."""
    h, cap = 1e-6, 3e-9
    c = Circuit("step")
    c.I("I1", "0", "a", 0.0, pulse=Pulse(0.0, amps, 0.0, 1e-9, 1e-9, 1.0, 0.0))
    c.R("R1", "a", "0", Table(0))
    c.Cap("C1", "a", "0", cap)
    r = 10.0 ** np.random.default_rng(7).uniform(0.0, 4.0, (20000, 1))
    cfg = abi.transient_config(h, 0.9e-6, abi.SP_TRAN_BE, 0, abi.SP_PREC_FP64)
    g = ctx.transient(c, abi.newton_config(), cfg, 1, len(r), table=r)
    assert (g["status"] == 0).all()
    want = amps / (1.0 / r[:, 0] + cap / h)
    assert np.array_equal(g["probe"][:, 1].view(np.uint64), want.view(np.uint64))


def cancelling():
    """A node whose negative resistor can cancel its capacitor's companion conductance
    (all values powers of two), driven by a pulse, beside a regular RC branch."""
    c = Circuit("cancelling")
    c.V("V1", "in", "0", 1.0)
    c.R("R1", "in", "out", 1024.0)
    c.Cap("C1", "out", "0", 2.0 ** -30)
    c.I("I1", "0", "x", 2.0 ** -10, pulse=Pulse(0.0, 2.0 ** -10, 2.0 ** -20, 2.0 ** -20, 2.0 ** -20, 2.0 ** -18, 2.0 ** -17))
    c.R("R2", "x", "0", Table(0))
    c.Cap("C2", "x", "0", 2.0 ** -30)
    return c


@pytest.mark.parametrize("method, ohms", [(abi.SP_TRAN_BE, -1024.0), (abi.SP_TRAN_TRAP, -512.0)])
@pytest.mark.parametrize("precision", [abi.SP_PREC_FP64_EXACT, abi.SP_PREC_FP64])
def test_singular_in_the_transient_only(ctx, method, ohms, precision):
    """C / h = 2^-10 (2 C / h = 2^-9 for the trapezoid) cancels 1 / R exactly: the DC
    point exists, every step's solve fails.  Regular samples lie in the same warps."""
    c = cancelling()
    count, h, tstop = 70, 2.0 ** -20, 6.5 * 2.0 ** -20
    table = np.where(np.arange(count) % 3 == 0, ohms, 4096.0)[:, None]
    cfg = abi.transient_config(h, tstop, method, c.node("x"), precision)
    dc = abi.newton_config(precision=precision)
    g = ctx.transient(c, dc, cfg, 2, count, table=table)
    with oracle.math_mode("cr"):
        x, pr, st = oracle.transient(c, abi.newton_config(precision=abi.SP_PREC_FP64_EXACT), 2, count, method, h, tstop,
                                     probe_idx=c.node("x"), table=table)
    singular = np.arange(count) % 3 == 0
    assert np.array_equal(st & abi.SP_ST_MASK, np.where(singular, abi.SP_ST_SINGULAR, abi.SP_ST_CONVERGED))
    assert np.array_equal(g["status"], st)
    # the waveform of a singular sample ends with its DC point, its state stays there
    assert np.isnan(g["probe"][singular, 1:]).all()
    assert np.isfinite(g["probe"][~singular]).all()
    if precision == abi.SP_PREC_FP64_EXACT:
        pr[singular, 1:] = g["probe"][singular, 1:]
        assert np.array_equal(g["probe"].view(np.uint64), pr.view(np.uint64))
        assert np.array_equal(g["x"].view(np.uint64), x.view(np.uint64))


@pytest.mark.parametrize("method, caps", [(abi.SP_TRAN_BE, 10500), (abi.SP_TRAN_TRAP, 10500), (abi.SP_TRAN_TRBDF2, 6000)])
def test_conductances_not_kept(ctx, method, caps):
    """One sample's v, i and conductances pass 227 KB: the conductances are worked out
    at every use, with the bits of the kept ones."""
    c = Circuit("parallel")
    c.V("V1", "in", "0", 0.0, pulse=Pulse(0.0, 1.0, 1e-6, 1e-6, 1e-6, 4e-6, 9e-6))
    c.R("R1", "in", "a", Table(0))
    for k in range(caps):
        c.Cap(f"C{k}", "a", "0", 1e-13 * (1 + k % 7))
    table = np.array([[1e3], [2e3], [3.3e3]])
    cfg = abi.transient_config(0.5e-6, 2.4e-6, method, c.node("a"), abi.SP_PREC_FP64_EXACT)
    dc = abi.newton_config(precision=abi.SP_PREC_FP64_EXACT)
    g = ctx.transient(c, dc, cfg, 1, 3, table=table)
    with oracle.math_mode("cr"):
        x, pr, st = oracle.transient(c, dc, 1, 3, method, 0.5e-6, 2.4e-6, probe_idx=c.node("a"), table=table)
    assert np.array_equal(g["status"], st) and (st == 0).all()
    assert np.array_equal(g["x"].view(np.uint64), x.view(np.uint64))
    assert np.array_equal(g["probe"].view(np.uint64), pr.view(np.uint64))
