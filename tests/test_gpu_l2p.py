"""L2P on the FP64 tensor cores (l2p.cu) at the sizes where it can go wrong, through the fmm, against the oracle.

Tolerance: relative L2 <= 1e-12, that of the plain FP64 parity tests: sums of at most 512 terms in another order.

Every node count of the range; leaves from one target to several tiles of 32, most with remainders; right-hand sides
around the choice between the split and the plain form and around a column group of 8; problems of different depths in
one forest, one without expansions.

The gradient against differences of the potential, which within a leaf is a polynomial of degree below 8 plus a
Gaussian's near field: (4 D(eps/2) - D(eps)) / 3 at eps = 1e-4 of a leaf width of 0.125 leaves (8e-4)^4 * 7^5 ~ 1e-8 of
truncation at worst and 2^-53 / eps ~ 1e-12 of rounding: 1e-6 of the largest component."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _solve(ctx, t, s, w, **kw):
    ctx.set_schedule_options(l2p_mode=1)  # lanes over targets for every leaf
    try:
        return ctx.solve(t, s, w, **kw)[0]
    finally:
        ctx.set_schedule_options()


@pytest.mark.parametrize("d,n,depth", [(1, 300, 5), (2, 900, 4), (3, 1500, 3)])
@pytest.mark.parametrize("poly_ord", [1, 2, 3, 4, 5, 6, 7])
def test_every_node_count(ctx, oracle, d, n, depth, poly_ord):
    r = np.random.default_rng(10 * d + poly_ord)
    t, s, w = r.random((n, d)) ** 2, r.random((n + 9, d)), r.standard_normal((9, n + 9))  # crowded towards the origin
    kid = 1
    ctx.set_kernel(kid, 0.0)
    for nrhs in (1, 3, 9):
        got = np.asarray(_solve(ctx, t, s, w[:nrhs], poly_ord=poly_ord, depth=depth)).reshape(nrhs, -1)
        for k in (0, nrhs - 1):
            want, _ = oracle.fmm(d, kid, 0.0, poly_ord, depth, 1, t, s, w[k].copy())
            assert rel_l2(got[k], want) <= TOL


@pytest.mark.parametrize("nrhs", [1, 2, 4, 5, 7, 8, 16, 17])
def test_right_hand_sides(ctx, oracle, nrhs):
    r = np.random.default_rng(nrhs)
    t, s, w = r.random((1300, 3)), r.random((1200, 3)), r.standard_normal((nrhs, 1200))
    ctx.set_kernel("inv_r_safe")
    got = np.asarray(_solve(ctx, t, s, w, poly_ord=4, depth=3)).reshape(nrhs, -1)
    for k in (0, nrhs - 1):
        want, _ = oracle.fmm(3, 1, 0.0, 4, 3, 1, t, s, w[k].copy())
        assert rel_l2(got[k], want) <= TOL


@pytest.mark.parametrize("nrhs", [1, 16])
def test_forest_with_a_problem_without_expansions(ctx, oracle, nrhs):
    r = np.random.default_rng(3)
    sizes, depths = [40, 1700, 3, 700], [2, 4, 3, 5]
    off = np.concatenate([[0], np.cumsum(sizes)])
    t, s = r.random((off[-1], 2)), r.random((off[-1], 2))
    w = r.standard_normal((nrhs, off[-1]))
    ctx.set_kernel("multiquadric", 1e-2)
    ctx.set_schedule_options(l2p_mode=1)
    try:
        got = np.asarray(ctx.forest_solve(t, off, s, off, w, depths, poly_ord=4)).reshape(nrhs, -1)
    finally:
        ctx.set_schedule_options()
    for p, depth in enumerate(depths):
        a, b = off[p], off[p + 1]
        want, _ = oracle.fmm(2, 5, 1e-2, 4, depth, 1, t[a:b], s[a:b], w[nrhs - 1, a:b].copy())
        assert rel_l2(got[nrhs - 1, a:b], want) <= TOL


@pytest.mark.parametrize("d,depth", [(2, 4), (3, 4)])
@pytest.mark.parametrize("poly_ord", [1, 2, 3, 4, 5, 6, 7])
def test_gradient(ctx, d, depth, poly_ord):
    r = np.random.default_rng(100 * d + poly_ord)
    n = 250
    leaf = 0.5 ** (depth - 1)
    cells = r.integers(0, 1 << (depth - 1), (n, d)) // 2 * 2  # in every second leaf: some with several targets
    t = (cells + r.uniform(0.2, 0.8, (n, d))) * leaf
    s = np.concatenate([r.random((600, d)), np.zeros((1, d)), np.ones((1, d))])  # the corners hold the tree in place
    w = r.standard_normal((2, len(s)))
    ctx.set_kernel("gaussian", 0.3)
    for nrhs in (1, 2):
        kw = dict(poly_ord=poly_ord, depth=depth)
        pot, grad = ctx.solve_grad(t, s, w[:nrhs], **kw)[:2]
        pot, grad = np.asarray(pot).reshape(nrhs, n), np.asarray(grad).reshape(nrhs, n, d)

        def at(shift):
            return np.asarray(ctx.solve(t + shift, s, w[:nrhs], **kw)[0]).reshape(nrhs, n)

        assert rel_l2(pot, at(0.0)) <= TOL
        for q in range(d):
            e = np.eye(d)[q]
            d1, d2 = ((at(h * e) - at(-h * e)) / (2 * h) for h in (1e-4, 5e-5))
            assert np.abs(grad[:, :, q] - (4 * d2 - d1) / 3).max() <= 1e-6 * np.abs(grad).max()


@pytest.mark.parametrize("mode", [0, 2])
@pytest.mark.parametrize("d,n", [(1, 1), (1, 8), (1, 9), (1, 16), (2, 1), (2, 5), (2, 6), (2, 8), (2, 9), (2, 10), (2, 11),
                                 (2, 12), (2, 13), (2, 14), (2, 15), (2, 16), (3, 1), (3, 2), (3, 3), (3, 4), (3, 5),
                                 (3, 6), (3, 7)])
def test_every_expansion_size(ctx, oracle, d, n, mode):
    # P2M and L2P have a kernel for every expansion size that is accepted, by default and with lanes over coefficients
    r = np.random.default_rng(16 * d + n)
    depth = {1: 6, 2: 4, 3: 3}[d]
    t, s, w = r.random((300, d)), r.random((310, d)), r.standard_normal((3, 310))
    ctx.set_kernel("inv_r_safe")
    ctx.set_schedule_options(l2p_mode=mode)
    try:
        one, _ = ctx.solve(t, s, w[2].copy(), poly_ord=n - 1, depth=depth)
        many, _ = ctx.solve(t, s, w, poly_ord=n - 1, depth=depth)
    finally:
        ctx.set_schedule_options()
    want, _ = oracle.fmm(d, 1, 0.0, n - 1, depth, 1, t, s, w[2].copy())
    assert rel_l2(one, want) <= TOL and rel_l2(many[2], want) <= TOL
