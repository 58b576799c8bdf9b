"""The operator cache of a context is emptied when it would grow beyond 16 GiB.  A mixed-precision level reads its
FP64 operators while it makes the split ones from them: emptying the cache for the split ones must not take the FP64
ones away.

Each solve below has a cube of its own, so it adds one level's FP64 operators (316 * 224 * 216 doubles, 122 MB) and
their BF16 split (63 MB); the first adds FP64 operators alone (a kernel without a split), so that the 92nd solve's FP64
operators still fit under the limit and its split does not.  1/r scales as 1/s with the points: every solve is
compared with the first, to the 1e-5 of the split products."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def test_split_of_operators_survives_an_emptied_cache():
    import fmma_b200
    r = np.random.default_rng(2)
    t, s, w = r.random((64, 3)), r.random((64, 3)), r.standard_normal(64)
    ctx = fmma_b200.Context(0)
    ctx.set_kernel("sum_over_r2")
    ctx.solve(t, s, w, poly_ord=5, depth=3)
    ctx.set_kernel("inv_r_safe")
    first, _ = ctx.solve(t, s, w, poly_ord=5, depth=3, precision="bf16x3")
    for i in range(1, 96):
        k = 1.0 + i / 64.0
        got, _ = ctx.solve(k * t, k * s, w, poly_ord=5, depth=3, precision="bf16x3")
        assert rel_l2(k * got, first) <= 1e-5
    ctx.close()
