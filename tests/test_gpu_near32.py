"""The mixed near field's target-lane kernel at the leaf sizes where its chunks of targets change: two chunks sharing
the sources (49 to 64 targets), one group with idle lanes (17 to 31), lane groups (16 and fewer), a chunk after a pair.
Depth 2: every leaf is a neighbour of every other, so the result is the direct sum; the oracle's exact sum is the
reference.  Tolerance 1e-6: FP32 kernel values (2^-23) of 200 to 700 terms of both signs, compensated sums."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 2, 3])
@pytest.mark.parametrize("per_leaf", [1, 5, 16, 17, 31, 32, 33, 48, 49, 64, 65, 81, 97, 130])
@pytest.mark.parametrize("nrhs", [1, 3, 16])
def test_chunks(ctx, oracle, d, per_leaf, nrhs):
    r = np.random.default_rng(per_leaf + 100 * d + nrhs)
    # one crowded leaf of exactly per_leaf targets, a few in the others
    crowd = r.random((per_leaf, d)) * 0.49
    t = np.concatenate([crowd, 0.51 + r.random((7, d)) * 0.49])
    s = np.concatenate([r.random((211 + per_leaf, d)), np.zeros((1, d)), np.ones((1, d))])
    w = r.uniform(-1, 1, (nrhs, len(s)))
    ctx.set_kernel("multiquadric", 1e-2)
    got, _ = ctx.solve(t, s, w if nrhs > 1 else w[0].copy(), poly_ord=2, depth=2, precision="tf32x3")
    got = np.atleast_2d(got)
    for k in {0, nrhs - 1}:
        want = oracle.exact_rows(d, 5, 1e-2, np.arange(len(t)), t, s, w[k].copy())
        assert rel_l2(got[k], want) <= 1e-6


@pytest.mark.parametrize("d", [1, 2, 3])
@pytest.mark.parametrize("n", [49, 50, 63, 64, 81, 96, 113, 128, 145])
def test_pairs_of_chunks_sum_as_chunks_alone(ctx, d, n):
    """One rhs: chunks of 32 targets of a leaf go in pairs where the second holds at least 17.  A chunk's sums do not
    depend on the company: the leaf's targets at once and 32 at a time give the same bits."""
    r = np.random.default_rng(n + 1000 * d)
    t = r.random((n, d)) * 0.49  # one leaf; its order is that of the targets
    s = np.concatenate([r.random((500, d)), np.zeros((1, d)), np.ones((1, d))])
    w = r.uniform(-1, 1, len(s))
    ctx.set_kernel("multiquadric", 1e-2)

    def solve(x):
        return ctx.solve(np.ascontiguousarray(x), s, w, poly_ord=2, depth=2, precision="tf32x3")[0]
    whole = solve(t)
    np.testing.assert_array_equal(whole, np.concatenate([solve(t[i:i + 32]) for i in range(0, n, 32)]))
