"""Uploading a circuit costs memory in proportion to its elements, whatever its size
(a matrix of flags for 60,000 unknowns would be 3.6 GB of host memory); the dense
solvers refuse what they do not take."""
import resource

import pytest

from spicier_gb300 import abi
from spicier_gb300._lib import SpicierError
from spicier_gb300.circuit import Circuit


@pytest.mark.gpu
def test_creation_without_a_matrix(ctx):
    import torch
    n = 60000
    c = Circuit("long_chain")
    c.V("V1", "n0", "0", 1.0)
    for i in range(n):
        c.R(f"R{i}", f"n{i}", f"n{i + 1}", 1e3)
    before = resource.getrusage(resource.RUSAGE_SELF).ru_maxrss
    topo = ctx.topology(c)
    grown_kb = resource.getrusage(resource.RUSAGE_SELF).ru_maxrss - before
    assert grown_kb < 512 * 1024
    x = torch.empty((1, c.n), dtype=torch.float64, device="cuda")
    with pytest.raises(SpicierError, match="exceeds the dense Newton limit"):
        ctx.newton_dc_device(topo, abi.newton_config(), 1, 1, x)
    topo.close()
