"""The batched LU's kernel setting is kept per precision: what was chosen for FP64
solves leaves the mixed ones alone, and where FP64 has one kernel only nothing is timed."""
import numpy as np
import pytest

from spicier_gb300 import abi
from spicier_gb300.autotune import Autotuner, TuneCache, key

pytestmark = pytest.mark.gpu


def solve(ctx, n, precision, A, b):
    import torch
    x = torch.empty_like(b)
    s = torch.empty(len(b), dtype=torch.uint8, device="cuda")
    ctx.solve_batch_device(A, b, n, len(b), x, s, precision=precision)
    torch.cuda.synchronize()
    assert not s.any()
    return x.cpu().numpy()


@pytest.mark.parametrize("n", [5, 16, 17, 28])
def test_fp64_setting_leaves_mixed_alone(ctx, n, tmp_path):
    import torch
    t = Autotuner(ctx, TuneCache(str(tmp_path / "t.json")))
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.rand((300, n, n), dtype=torch.float64, device="cuda", generator=g) + n * torch.eye(n, dtype=torch.float64, device="cuda")
    b = torch.rand((300, n), dtype=torch.float64, device="cuda", generator=g)
    plain = {p: solve(ctx, n, p, A, b) for p in (abi.SP_PREC_FP64, abi.SP_PREC_MIXED)}
    t.set(key("lu.cta", n), 1)
    try:
        for p, want in plain.items():
            assert np.array_equal(solve(ctx, n, p, A, b).view(np.uint64), want.view(np.uint64))
    finally:
        t.set(key("lu.cta", n), 0)
    # the mixed solve's own setting: the FP64 elimination of a CTA
    t.set(key("lu.cta.mixed", n), 1)
    try:
        assert np.array_equal(solve(ctx, n, abi.SP_PREC_MIXED, A, b).view(np.uint64), plain[abi.SP_PREC_FP64].view(np.uint64))
    finally:
        t.set(key("lu.cta.mixed", n), 0)


def test_one_kernel_is_not_timed(ctx, tmp_path):
    t = Autotuner(ctx, TuneCache(str(tmp_path / "t.json")))
    assert t.tune_lu(sizes=(20, 28), batch=64) == {20: 0, 28: 0}
    assert t.cache.settings(t.gpu) == {} and t.get(key("lu.cta", 20)) is None


def test_mixed_choice_has_its_own_key(ctx, tmp_path):
    t = Autotuner(ctx, TuneCache(str(tmp_path / "t.json")), reps=2)
    best = t.tune_lu(sizes=(12,), batch=512, precision=abi.SP_PREC_MIXED)[12]
    try:
        assert t.cache.settings(t.gpu) == {key("lu.cta.mixed", 12): best}
        assert t.get(key("lu.cta", 12)) is None and t.get(key("lu.cta.mixed", 12)) == (best or None)
    finally:
        t.set(key("lu.cta.mixed", 12), 0)
