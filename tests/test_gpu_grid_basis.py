"""Mixed power-grid solves with the Krylov basis on chip: every home of a basis
vector (tensor, shared and global memory), the rows past 4,096 and the edges of
the meshes each kernel instance takes."""
import numpy as np
import pytest

from spicier_gb300 import abi

MIXED, FP64 = abi.SP_PREC_MIXED, abi.SP_PREC_FP64


def solve(ctx, prec, rows, cols, **kw):
    kw.setdefault("num_sinks", max(1, rows * cols // 8))
    return ctx.grid_solve(abi.grid_config(rows=rows, cols=cols, precision=prec, **kw), 3, 4)


# n = rows * cols + 1: up to 1,024, 2,048, 4,096 (no tail), 4,097, and a tail of
# more than 256 rows; restart up to 16 / 26 / 32 vectors (the homes' edges)
@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols", [(2, 2), (2, 300), (31, 33), (32, 32), (23, 89), (32, 64), (63, 65), (64, 64),
                                       (67, 68), (2, 2303)])
@pytest.mark.parametrize("restart,steps", [(1, 3), (16, 16), (17, 35), (26, 27), (32, 32)])
def test_first_solve_against_fp64(ctx, rows, cols, restart, steps):
    """`steps` Krylov steps from x = 0: in exact arithmetic both precisions have
    the same iterate.  FP32 leaves about steps * sqrt(n) * 2^-24 of the
    largest entry (35 * 68 * 6e-8 = 1.4e-4); a vector read from the wrong place
    leaves orders of magnitude more."""
    g, r = (solve(ctx, p, rows, cols, restart=restart, max_newton=1, max_krylov=steps) for p in (MIXED, FP64))
    scale = np.abs(r["x"]).max(axis=1, keepdims=True)
    small = rows * cols <= 4  # the FP64 solve may have stopped before `steps`
    assert small or np.array_equal(g["krylov"], r["krylov"])
    assert (np.abs(g["x"] - r["x"]) <= 1e-3 * scale).all()


@pytest.mark.gpu
@pytest.mark.parametrize("rows,cols,restart", [(12, 17, 30), (32, 40, 30), (46, 50, 32), (63, 65, 30)])
def test_converged(ctx, rows, cols, restart):
    """To convergence: the residual target, and the FP64 solution within the SPICE tolerance."""
    g, r = (solve(ctx, p, rows, cols, restart=restart) for p in (MIXED, FP64))
    n = rows * cols
    assert (g["status"] == 0).all() and g["resid"].max() <= abi.grid_config().resid_target
    assert (np.abs(g["x"][:, :n] - r["x"][:, :n]) <= 1e-3 * np.abs(r["x"][:, :n]) + 1e-6).all()
    again = solve(ctx, MIXED, rows, cols, restart=restart)
    assert all(np.array_equal(g[k], again[k]) for k in g)


@pytest.mark.gpu
def test_sinks_on_one_node(ctx):
    """More sinks than nodes: each node's are added in order, by one thread."""
    g, r = (solve(ctx, p, 5, 6, num_sinks=1200) for p in (MIXED, FP64))
    assert (g["status"] == 0).all() and np.array_equal(g["status"], r["status"])
    assert (np.abs(g["x"] - r["x"])[:, :30] <= 1e-3 * np.abs(r["x"])[:, :30] + 1e-6).all()
