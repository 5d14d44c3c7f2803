"""Ladder transients at the section counts where the block-per-ladder kernel
changes: the elimination's block count (N / 2 below 64 sections, then 32), a
row more than a multiple of 32, the thread-count rules, and arrays in the
global workspace (too long for shared memory)."""
import numpy as np
import pytest

import oracle
from spicier_gb300 import abi

pytestmark = pytest.mark.gpu

SIZES = [2, 3, 5, 8, 31, 48, 49, 62, 63, 64, 65, 96, 97, 160, 161]


def cfg_of(n, **kw):
    return abi.ladder_config(min_sections=n, max_sections=n, tstop=12e-9, h_max=1e-9, num_probe=7, **kw)


@pytest.mark.parametrize("n", SIZES)
def test_exact_bits(ctx, n):
    cfg = cfg_of(n, precision=abi.SP_PREC_FP64_EXACT)
    g = ctx.ladder_transient(cfg, 3, 3)
    with oracle.math_mode("cr"):
        o = oracle.ladder_transient(cfg, 3, 3)
    for k in ("n", "accepted", "rejected", "iterations", "status"):
        assert np.array_equal(g[k], o[k]), k
    assert np.array_equal(g["x"].view(np.uint64), o["x"].view(np.uint64))
    assert np.array_equal(g["probe"].view(np.uint64), o["probe"].view(np.uint64))


@pytest.mark.parametrize("n,prec", [(n, p) for n in SIZES for p in (abi.SP_PREC_FP64, abi.SP_PREC_MIXED)] +
                         [(1200, abi.SP_PREC_FP64), (2800, abi.SP_PREC_MIXED)])
def test_replay_of_its_own_steps(ctx, n, prec):
    """The bars of the full-size test: FP64 1e-9 relative, MIXED the SPICE tolerance per node."""
    cfg = cfg_of(n, precision=prec)
    g = ctx.ladder_transient_steps(cfg, 3, 3)
    assert (g["status"] == 0).all()
    with oracle.math_mode("cr"):
        rep = oracle.ladder_replay(cfg_of(n), 3, g["steps"], g["accepted"])
    x, w = g["x"], rep["x"]
    if prec == abi.SP_PREC_FP64:
        scale = np.maximum(np.abs(w), 1e-9 * np.abs(w).max(axis=1, keepdims=True))
        assert (np.abs(x - w) <= 1e-9 * scale + 1e-18).all()
    else:
        tol = 1e-3 * np.abs(w) + 1e-6
        tol[:, n + 1] = 1e-3 * np.abs(w[:, n + 1]) + 1e-12
        assert (np.abs(x - w) <= tol).all()


def test_longer_ladders_are_refused_as_before(ctx):
    import spicier_gb300 as sg
    for n, prec in ((1791, abi.SP_PREC_FP64), (3583, abi.SP_PREC_MIXED), (1791, abi.SP_PREC_FP64_EXACT)):
        with pytest.raises(sg.SpicierError) as e:
            ctx.ladder_transient(cfg_of(n, precision=prec), 1, 1)
        assert e.value.kind == "InvalidDimension"
