"""FP64 AC sweeps of circuits on both sides of the line between the sparse and the
dense kernel, and of the estimated fill that sizes the sparse kernel's slots: the
oracle's bits."""
import random

import numpy as np
import pytest

import oracle
from spicier_gb300 import abi
from spicier_gb300.api import Context
from spicier_gb300.circuit import Circuit, Gauss

pytestmark = pytest.mark.gpu


def net(n, degree, seed):
    """n unknowns: a chain of drawn resistors driven at one end, with R and C between
    random pairs up to `degree` elements a node."""
    rng = random.Random(seed)
    nodes = n - 1
    c = Circuit(f"net{n}_{degree}")
    c.V("V1", "a0", "0", 1.0)
    for i in range(nodes - 1):
        c.R(f"P{i}", f"a{i}", f"a{i + 1}", Gauss(1e3, 10.0, i))
    for e in range(int(nodes * degree / 2) - (nodes - 1)):
        i, j = rng.sample(range(nodes), 2)
        if rng.random() < 0.5:
            c.Cap(f"C{e}", f"a{i}", f"a{j}", 1e-12 * (1 + rng.random()))
        else:
            c.R(f"R{e}", f"a{i}", f"a{j}", 1e3 * (1 + rng.random()))
    c.R("G", f"a{nodes - 1}", "0", 1e3)
    c.Cap("CG", "a1", "0", 1e-12)
    return c


# small and sparse, dense at every size, and the sizes where slots end (28 unknowns at 3 fit one warp per SM)
@pytest.mark.parametrize("n, degree", [(3, 2), (5, 4), (8, 6), (10, 6), (12, 11), (14, 4), (14, 6), (16, 2), (16, 10),
                                       (20, 3), (20, 4), (20, 10), (24, 2), (28, 3), (28, 4), (28, 20)])
@pytest.mark.parametrize("count", [2, 260])
def test_bits_on_both_sides(ctx, n, degree, count):
    c = net(n, degree, 100 * n + degree)
    assert c.n == n
    dc = abi.newton_config(precision=abi.SP_PREC_FP64_EXACT)
    probes = sorted({0, n // 2, n - 1})
    cfg = abi.ac_config(1e3, 1e10, 3, abi.SP_AC_DEC, probes)
    h, st = ctx.ac_sweep(c, dc, cfg, 4, count)
    with oracle.math_mode("cr"):
        ho, so = oracle.ac_sweep(c, dc, 4, count, Context.ac_frequencies(cfg), probes)
    assert np.array_equal(st, so) and ((st & abi.SP_ST_MASK) == 0).all()
    assert np.array_equal(h.view(np.uint64), ho.view(np.uint64))
