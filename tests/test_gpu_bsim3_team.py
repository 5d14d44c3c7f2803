"""BSIM3 devices of one sample spread over a team of lanes: the same bits as one
lane that evaluates them all (which large sweeps and long fallback lists use)."""
import numpy as np
import pytest

from spicier_gb300 import abi
from spicier_gb300.circuit import Circuit, Gauss


def chain(devices):
    """VDD, a gate source and `devices` common-source stages in a row (odd ones PMOS)."""
    c = Circuit(f"b3_chain_{devices}")
    c.V("VDD", "vdd", "0", 1.8)
    c.V("VIN", "n0", "0", Gauss(0.8, 0.05, 0))
    for i in range(devices):
        pmos = bool(i % 2)
        s = "vdd" if pmos else "0"
        c.B3(f"M{i}", f"n{i + 1}", f"n{i}", s, s, pmos=pmos,
             vth0=Gauss(-0.4 if pmos else 0.4, 0.02, i + 1), w=2e-6)
        c.R(f"R{i}", f"n{i + 1}", "0" if pmos else "vdd", 1e4)
    return c


# 1: no team; 2, 3 (one lane idle), 8: one round; 9 and 11: a second, partial round
@pytest.mark.gpu
@pytest.mark.parametrize("devices", [1, 2, 3, 8, 9, 11])
@pytest.mark.parametrize("prec", [abi.SP_PREC_MIXED, abi.SP_PREC_FP64])
@pytest.mark.parametrize("limit", [50, 3])  # 3 iterations: every sample goes through the fallback
def test_team_of_lanes(ctx, devices, prec, limit):
    c, cfg = chain(devices), abi.newton_config(precision=prec, max_iterations=limit)
    few, many = (ctx.newton_dc(c, cfg, 7, n) for n in (67, 20000))
    for f in ("x", "iters", "status", "resid"):
        a, b = np.asarray(getattr(few, f)), np.asarray(getattr(many, f))[:67]
        assert a.tobytes() == b.tobytes(), f
