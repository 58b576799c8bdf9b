"""The FP64 near field and the exact sum (near64.cu) at the sizes where their cuts change, against the oracle, and
1/r's own inverse square root against extended precision.

Tolerances: the sums differ from the oracle's only in order and in the last place of f: 1e-13 relative L2 for the exact
sum (the parity tests' bound), 1e-12 through the fmm.  A single 1/r: r^2 rounded once (2^-54 of 1/r) and at most one ulp
(2^-52) of the inverse square root."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

P0 = {4: 0.3, 5: 1e-2}


@pytest.mark.parametrize("kid", [0, 1, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("nt,ns", [(1, 1), (3, 63), (255, 64), (256, 65), (257, 1000), (2048, 129), (5000, 4097)])
def test_exact_sizes(ctx, oracle, kid, nt, ns):
    r = np.random.default_rng(nt + ns + kid)
    d = 1 + (nt + ns) % 3
    t, s, w = r.random((nt, d)), r.random((ns, d)), r.standard_normal((3, ns))
    ctx.set_kernel(kid, P0.get(kid, 0.0))
    one, _ = ctx.solve(t, s, w[0].copy(), solver="exact")
    want = oracle.exact_rows(d, kid, P0.get(kid, 0.0), np.arange(nt), t, s, w[0].copy())
    assert rel_l2(one, want) <= 1e-13
    many, _ = ctx.solve(t, s, w, solver="exact")  # four per pass
    for k in range(3):
        want = oracle.exact_rows(d, kid, P0.get(kid, 0.0), np.arange(nt), t, s, w[k].copy())
        assert rel_l2(many[k], want) <= 1e-13


@pytest.mark.parametrize("d,n,depth", [(1, 700, 5), (2, 97, 3), (2, 4000, 4), (2, 9000, 3), (3, 5000, 3), (3, 40, 4)])
@pytest.mark.parametrize("nrhs", [1, 2, 3, 9])
def test_near_field_cuts(ctx, oracle, d, n, depth, nrhs):
    """Leaves of one to hundreds of targets (whole, three-quarter and split chunks), one to four units a row, every
    right-hand-side block."""
    r = np.random.default_rng(n + depth + nrhs)
    t, s = r.random((n, d)) ** 2, r.random((n + 13, d)) ** 2  # crowded towards the origin
    w = r.standard_normal((nrhs, n + 13))
    ctx.set_kernel("log_r")
    got, _ = ctx.solve(t, s, w, poly_ord=3, depth=depth)
    for k in {0, nrhs - 1}:
        want, _ = oracle.fmm(d, 3, 0.0, 3, depth, 1, t, s, w[k].copy())
        assert rel_l2(got[k], want) <= 1e-12


def test_one_unit_per_warp(ctx, oracle):
    # more leaf rows than eight waves of warps: no sharing of a unit
    r = np.random.default_rng(3)
    n = 60000
    t, s, w = r.random((n, 2)), r.random((n, 2)), r.standard_normal(n)
    ctx.set_kernel("inv_r_safe")
    got, _ = ctx.solve(t, s, w, poly_ord=2, depth=9)
    want, _ = oracle.fmm(2, 1, 0.0, 2, 9, 1, t, s, w)
    assert rel_l2(got, want) <= 1e-12


@pytest.mark.parametrize("kid", [0, 1, 3, 4, 5, 6])
def test_near_gradient_is_the_exact_one(ctx, kid):
    # Depth 2: every leaf is a neighbour, the fmm is the direct sum
    r = np.random.default_rng(kid)
    t, s, w = r.random((500, 3)), r.random((400, 3)), r.standard_normal((2, 400))
    ctx.set_kernel(kid, P0.get(kid, 0.0))
    c, g, _ = ctx.solve_grad(t, s, w, poly_ord=2, depth=2)
    ce, ge, _ = ctx.solve_grad(t, s, w, solver="exact")
    assert rel_l2(c, ce) <= 1e-13
    assert rel_l2(g, ge) <= 1e-12


@pytest.mark.parametrize("d,kid", [(1, k) for k in range(7)] + [(2, k) for k in (0, 1, 3, 4, 5, 6)] + [(3, 1), (3, 6)])
@pytest.mark.parametrize("coincident", [False, True])
def test_near_gradient_in_every_dimension(ctx, d, kid, coincident):
    # against the exact gradient, which another kernel sums pair by pair; coincident points take the guards
    r = np.random.default_rng(20 * d + kid)
    t, s, w = r.random((300, d)), r.random((280, d)), r.standard_normal((2, 280))
    if coincident:
        t[:40] = s[:40]
    ctx.set_kernel(kid, P0.get(kid, 0.0))
    c, g, _ = ctx.solve_grad(t, s, w, poly_ord=2, depth=2)
    ce, ge, _ = ctx.solve_grad(t, s, w, solver="exact")
    ok = np.isfinite(ce)  # at r = 0 the potential of 1/r is infinite and that of s/r^2 undefined
    np.testing.assert_array_equal(np.isfinite(c), ok)
    assert ok.all() == (not coincident or kid not in (0, 6))
    assert rel_l2(c[ok], ce[ok]) <= 1e-13
    assert np.isfinite(ge).all() and rel_l2(g, ge) <= 1e-12


def test_inverse_square_root(ctx):
    r = np.random.default_rng(1)
    x = np.concatenate([r.uniform(1, 4, 20000), 10.0 ** r.uniform(-150, 150, 20000)])
    # one source at the origin, unit weight, coordinates kept as they are by the exact solver
    ctx.set_kernel("inv_r_safe")
    got, _ = ctx.solve(x[:, None].copy(), np.zeros((1, 1)), np.ones(1), solver="exact")
    want = 1 / x.astype(np.longdouble)
    err = np.abs((got.astype(np.longdouble) - want) / want)
    assert float(err.max()) <= 2.0 ** -52 + 2.0 ** -54
    # outside the normal range of r^2: subnormal, zero, infinite
    edge = np.array([[1e-160], [0.0], [-0.0], [1e200], [1.4e-154]])
    got, _ = ctx.solve(edge, np.zeros((1, 1)), np.ones(1), solver="exact")
    assert got[1] == 0 and got[2] == 0 and got[3] == 0
    assert abs(got[0] * 1e-160 - 1) < 1e-3  # r^2 = 1e-320 has 11 bits
    assert abs(got[4] * 1.4e-154 - 1) < 1e-12
    ctx.set_kernel("inv_r")
    got, _ = ctx.solve(edge, np.zeros((1, 1)), np.ones(1), solver="exact")
    assert np.isinf(got[1]) and got[3] == 0
    # a Gaussian whose width takes the plain division, and distances outside the fast one's range
    for p0 in (0.3, 1e-200, 1e200):
        ctx.set_kernel("gaussian", p0)
        y = np.array([0.0, 0.1, 1.0, 7.0, 1e-170, 1e170]) * np.sqrt(p0)
        got, _ = ctx.solve(y[:, None].copy(), np.zeros((1, 1)), np.ones(1), solver="exact")
        with np.errstate(over="ignore", under="ignore"):
            np.testing.assert_allclose(got, np.exp(-(y * y) / p0), rtol=1e-13, atol=0)


@pytest.mark.parametrize("d,depth,per,rhs", [(1, 8, 10, 1), (1, 8, 22, 1), (1, 8, 30, 4), (1, 13, 3, 1), (1, 13, 25, 2),
                                             (2, 5, 5, 1), (2, 5, 8, 3), (2, 7, 2, 1), (2, 7, 31, 1), (2, 7, 60, 1),
                                             (3, 3, 2, 1), (3, 3, 3, 8), (3, 5, 1, 1), (3, 5, 10, 1), (3, 5, 20, 1)])
def test_units_of_one_and_of_four_warps(ctx, oracle, d, depth, per, rhs):
    # lists and numbers of units on both sides of the rule that has four warps share a unit; the other stages are as
    # in the parity tests: 1e-12
    r = np.random.default_rng(100 * d + depth + per)
    n = per * 2 ** (d * (depth - 1))
    t, s, w = r.random((n, d)), r.random((n, d)), r.standard_normal((rhs, n))
    ctx.set_kernel("inv_r_safe")
    got, _ = ctx.solve(t, s, w if rhs > 1 else w[0].copy(), poly_ord=1, depth=depth)
    want, _ = oracle.fmm(d, 1, 0.0, 1, depth, 1, t, s, w[rhs - 1].copy())
    assert rel_l2(np.atleast_2d(got)[rhs - 1], want) <= 1e-12


@pytest.mark.parametrize("d,depth,per", [(1, 11, 1), (1, 11, 4), (1, 11, 5), (1, 11, 6), (2, 7, 1), (2, 7, 2)])
@pytest.mark.parametrize("kid", [1, 4])
def test_sparse_leaves(ctx, oracle, d, depth, per, kid):
    # lists of fewer than 16 sources in 1-D and 2-D have a form of their own: both sides of the line, one to nine rhs
    # the gradient is below, where the near field is all there is
    r = np.random.default_rng(10 * d + per)
    n = per * 2 ** (d * (depth - 1))
    t, s, w = r.random((n, d)), r.random((n, d)), r.standard_normal((9, n))
    ctx.set_kernel(kid, P0.get(kid, 0.0))
    for rhs in (1, 3, 9):
        got, _ = ctx.solve(t, s, w[:rhs] if rhs > 1 else w[0].copy(), poly_ord=1, depth=depth)
        want, _ = oracle.fmm(d, kid, P0.get(kid, 0.0), 1, depth, 1, t, s, w[rhs - 1].copy())
        assert rel_l2(np.atleast_2d(got)[rhs - 1], want) <= 1e-12


@pytest.mark.parametrize("d", [1, 2])
@pytest.mark.parametrize("kid", [1, 2, 4, 6])
def test_gradient_on_sparse_leaves(ctx, d, kid):
    # Depth 2 with a point or two a leaf: the direct sum, by the sparse form
    if kid == 2 and d > 1:
        pytest.skip("1/(x-y) is one-dimensional")
    r = np.random.default_rng(kid)
    ctx.set_kernel(kid, P0.get(kid, 0.0))
    for n in (2, 3, 5):
        t, s, w = r.random((n, d)), r.random((n, d)), r.standard_normal((2, n))
        c, g, _ = ctx.solve_grad(t, s, w, poly_ord=2, depth=2)
        ce, ge, _ = ctx.solve_grad(t, s, w, solver="exact")
        assert rel_l2(c, ce) <= 1e-13 and rel_l2(g, ge) <= 1e-12
