"""Weight and bias gradients of every layer, reduced together: widths and row
counts with partial blocks and chunks, and more layers than one launch of the
final bias sums takes."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo
from spicier_gb300 import abi
from spicier_gb300.api import Mlp
from test_gpu_mlp import gradients, rel

pytestmark = pytest.mark.gpu


# layers + 1 bias vectors: 2, 8 (one full launch), 9 (a second one); 64 rows: a single chunk
@pytest.mark.parametrize("H,nl,rows", [(32, 1, 64), (96, 7, 192), (64, 8, 64), (32, 8, 4160)])
@pytest.mark.parametrize("kind", [abi.SP_MLP_KERNEL_TCGEN05, abi.SP_MLP_KERNEL_MMA_SYNC])
def test_every_layer(ctx, H, nl, rows, kind):
    """BF16 activations leave 3e-2 on the 4-layer networks of test_gpu_mlp; with
    the depth that grows about in proportion (9 layers: 7e-2).  A sum that went
    to another layer, or missed a chunk, is off by its own size."""
    m = Mlp(ctx, 10, 12, H, nl, seed=H + nl)
    m.set_training_kernel(kind)
    rng = np.random.default_rng(rows)
    X = rng.standard_normal((rows, 10)).astype(np.float32)
    T = rng.standard_normal((rows, 12)).astype(np.float32)
    gpu, loss = gradients(m, X, T, rows)
    again, _ = gradients(m, X, T, rows)
    _, lo, go = mo.forward_backward(m.unflatten(m.get_params()), X, T, 12)
    assert abs(loss - lo) <= 1e-2 * lo
    for l in range(len(go)):
        for a, b, o in zip(gpu[l], again[l], go[l]):
            assert np.array_equal(a, b), l
            assert rel(a, o) < 1e-1, l
    assert m.fault() == 0
    m.close()
