"""BSIM3 lane teams at the edges of their rules: fallback lists of as many samples as
the launch has blocks and of one more, and sweeps on both sides of the primary
kernel's line, give the bits of single lanes."""
import numpy as np
import pytest

from spicier_gb300 import abi
from spicier_gb300.circuit import Circuit, Gauss

pytestmark = pytest.mark.gpu


def chain(devices):
    c = Circuit(f"b3_edges_{devices}")
    c.V("VDD", "vdd", "0", 1.8)
    c.V("VIN", "n0", "0", Gauss(0.8, 0.05, 0))
    for i in range(devices):
        pmos = bool(i % 2)
        s = "vdd" if pmos else "0"
        c.B3(f"M{i}", f"n{i + 1}", f"n{i}", s, s, pmos=pmos,
             vth0=Gauss(-0.4 if pmos else 0.4, 0.02, i + 1), w=2e-6)
        c.R(f"R{i}", f"n{i + 1}", "0" if pmos else "vdd", 1e4)
    return c


def same(a, b, rows):
    for f in ("x", "iters", "status", "resid"):
        u, v = np.asarray(getattr(a, f))[:rows], np.asarray(getattr(b, f))[:rows]
        assert u.tobytes() == v.tobytes(), f


@pytest.mark.parametrize("prec", [abi.SP_PREC_MIXED, abi.SP_PREC_FP64])
@pytest.mark.parametrize("extra", [-1, 0, 1, 33])
def test_list_as_long_as_the_launch(ctx, prec, extra):
    """Three iterations: every sample is listed (two blocks per SM when there are as many samples)."""
    import torch
    n = 2 * torch.cuda.get_device_properties(0).multi_processor_count + extra
    c, cfg = chain(3), abi.newton_config(precision=prec, max_iterations=3)
    few, many = ctx.newton_dc(c, cfg, 5, n), ctx.newton_dc(c, cfg, 5, 20000)
    assert ((few.status & abi.SP_ST_FLAG_GMIN) != 0).all()
    same(few, many, n)


@pytest.mark.parametrize("prec, devices, warps", [(abi.SP_PREC_MIXED, 3, 8), (abi.SP_PREC_FP64, 3, 8),
                                                  (abi.SP_PREC_MIXED, 9, 8), (abi.SP_PREC_FP64, 9, 6)])
def test_both_sides_of_the_primary_line(ctx, prec, devices, warps):
    import torch
    team = 4 if devices == 3 else 8
    n = torch.cuda.get_device_properties(0).multi_processor_count * 32 * warps // team
    c, cfg = chain(devices), abi.newton_config(precision=prec, fallback=0)
    same(ctx.newton_dc(c, cfg, 6, n), ctx.newton_dc(c, cfg, 6, n + 1), n)
