"""The FP64 M2L on the reflection symmetry of the grid (radial kernels in 3-D, 3 to 8 nodes per
dimension) against the oracle.

Tolerance: relative L2 <= 1e-12, that of the plain FP64 parity tests: the same sums in another order,
P terms per far box and at most 189 boxes, in FP64 (2^-53 sqrt(189 * 512) ~ 3e-14).

Sizes where it can go wrong: every node count of its range (odd ones have a centre node without an odd
part), tiles of 64 (32 from 7 nodes) rows with a few rows only and with remainders, levels split over
several blocks and levels that are not, orbits with no source for some row groups (clustered points),
several right-hand sides sharing a tile, and several problems with operator tables of their own."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

KERNELS = [(0, 0.0), (1, 0.0), (3, 0.0), (4, 0.3), (5, 1e-2)]  # 1/r, 1/r (0 at r = 0), log r, Gaussian, multiquadric
TOL = 1e-12


def _points(r, n, clustered):
    if not clustered:
        return r.random((n, 3))
    c = r.uniform(0.1, 0.9, (4, 3))
    return np.clip(c[r.integers(0, 4, n)] + 0.03 * r.standard_normal((n, 3)), 0.0, 1.0)


@pytest.mark.parametrize("poly_ord", [2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("clustered", [False, True])
def test_every_node_count(ctx, oracle, poly_ord, clustered):
    r = np.random.default_rng(poly_ord)
    depth = 4 if poly_ord <= 4 else 3
    n = 700 if poly_ord == 7 else (3000 if clustered else 2500)
    t, s, w = _points(r, n, clustered), _points(r, n + 77, clustered), r.uniform(-1, 1, n + 77)
    kid, p0 = KERNELS[poly_ord % len(KERNELS)]
    ctx.set_kernel(kid, p0)
    # 8 nodes: dense leaves need more shared memory in the target-lane L2P than there is
    ctx.set_schedule_options(l2p_mode=2 if poly_ord == 7 else 0)
    try:
        got, _ = ctx.solve(t, s, w, poly_ord=poly_ord, depth=depth)
    finally:
        ctx.set_schedule_options()
    want, _ = oracle.fmm(3, kid, p0, poly_ord, depth, 1, t, s, w)
    assert rel_l2(got, want) <= TOL


@pytest.mark.parametrize("kid,p0", KERNELS)
def test_every_radial_kernel(ctx, oracle, kid, p0):
    r = np.random.default_rng(17 + kid)
    t, s, w = r.random((900, 3)), r.random((1100, 3)) * [1.0, 0.4, 0.7], r.standard_normal(1100)
    ctx.set_kernel(kid, p0)
    got, _ = ctx.solve(t, s, w, poly_ord=3, depth=4)
    want, _ = oracle.fmm(3, kid, p0, 3, 4, 1, t, s, w)
    assert rel_l2(got, want) <= TOL


def test_right_hand_sides_and_unsplit_level(ctx, oracle):
    # 4096 leaves x 7 rhs = 56 tiles per class, 448 in all: the leaf level in one or two parts, the others split
    r = np.random.default_rng(5)
    t, s, w = r.random((20000, 3)), r.random((20000, 3)), r.standard_normal((7, 20000))
    ctx.set_kernel("inv_r_safe")
    got, _ = ctx.solve(t, s, w, poly_ord=4, depth=5)
    for k in (0, 6):
        want, _ = oracle.fmm(3, 1, 0.0, 4, 5, 1, t, s, w[k])
        assert rel_l2(got[k], want) <= TOL


@pytest.mark.parametrize("poly_ord", [3, 4, 6])
@pytest.mark.parametrize("rhs", [1, 2, 3, 4, 5, 8, 9])
def test_used_row_groups(ctx, oracle, poly_ord, rhs):
    # all 64 boxes of level 2, 8 of every class: tiles of exactly rhs row groups of 8 (8 and 9: full and 1 more)
    r = np.random.default_rng(20 + rhs)
    t, s, w = r.random((900, 3)), r.random((1000, 3)), r.standard_normal((rhs, 1000))
    ctx.set_kernel("inv_r_safe")
    got, _ = ctx.solve(t, s, w, poly_ord=poly_ord, depth=3)
    got = np.asarray(got).reshape(rhs, -1)
    for k in (0, rhs - 1):
        want, _ = oracle.fmm(3, 1, 0.0, poly_ord, 3, 1, t, s, w[k])
        assert rel_l2(got[k], want) <= TOL


def test_few_points(ctx, oracle):
    r = np.random.default_rng(8)
    for n in (1, 2, 9, 40):
        t, s, w = r.random((n, 3)), r.random((n, 3)), r.standard_normal(n)
        ctx.set_kernel("inv_r_safe")
        got, _ = ctx.solve(t, s, w, poly_ord=4, depth=4)
        want, _ = oracle.fmm(3, 1, 0.0, 4, 4, 1, t, s, w)
        assert np.linalg.norm(got - want) <= TOL * max(np.linalg.norm(want), 1e-300) + 1e-300


def test_forest_of_different_boxes(ctx, oracle):
    r = np.random.default_rng(9)
    sizes = [300, 1500, 37]
    off = np.concatenate([[0], np.cumsum(sizes)])
    side = np.repeat([0.5, 3.0, 1.0], sizes)[:, None]
    t, s = (side * r.random((off[-1], 3)) for _ in range(2))
    w = r.standard_normal((2, off[-1]))
    ctx.set_kernel("multiquadric", 1e-2)
    got = ctx.forest_solve(t, off, s, off, w, [3, 4, 3], poly_ord=4)
    for p, depth in enumerate([3, 4, 3]):
        a, b = off[p], off[p + 1]
        for k in range(2):
            want, _ = oracle.fmm(3, 5, 1e-2, 4, depth, 1, t[a:b], s[a:b], w[k, a:b])
            assert rel_l2(got[k, a:b], want) <= TOL


def test_plan_replay_is_the_solve(ctx):
    r = np.random.default_rng(10)
    t, s, w = r.random((5000, 3)), r.random((5000, 3)), r.standard_normal((2, 5000))
    ctx.set_kernel("inv_r_safe")
    plan = ctx.plan(t, [0, 5000], s, [0, 5000], 2, [4], poly_ord=5)
    want, _ = ctx.solve(t, s, w, poly_ord=5, depth=4)
    np.testing.assert_array_equal(plan.execute(w), want)
    np.testing.assert_array_equal(plan.execute(w), want)
    plan.close()


@pytest.mark.parametrize("poly_ord,depth", [(3, 4), (4, 4), (4, 3), (6, 3)])
def test_wait_that_gives_up_reports_and_context_recovers(poly_ord, depth):
    """The gathering warps never report a stage and the waits are bounded at 2e6 SM clocks (~1 ms): the multiplying
    warps' first wait gives up, both sides leave, the solve raises status 5 (timeout), and the same context then
    solves bit for bit as before.  Even and odd node counts, full tiles and tiles whose upper half has no rows."""
    import fmma_b200
    r = np.random.default_rng(poly_ord)
    t, s, w = r.random((2000, 3)), r.random((2100, 3)), r.standard_normal(2100)
    c = fmma_b200.Context(0)
    try:
        c.set_kernel("inv_r_safe")
        ref, _ = c.solve(t, s, w, poly_ord=poly_ord, depth=depth)
        c.debug_m2l_wait(2_000_000, hold_issuer=True)
        with pytest.raises(fmma_b200.FmmaError) as e:
            c.solve(t, s, w, poly_ord=poly_ord, depth=depth)
        assert e.value.status == 5, e.value
        c.debug_m2l_wait(200_000_000)  # a bound that nothing runs into
        out, _ = c.solve(t, s, w, poly_ord=poly_ord, depth=depth)
        np.testing.assert_array_equal(out, ref)
    finally:
        c.debug_m2l_wait()
        c.close()


@pytest.mark.parametrize("poly_ord", [3, 4, 5, 7])
@pytest.mark.parametrize("power", [1023, -900])
def test_weights_of_any_size(ctx, poly_ord, power):
    # A power of two in the weights is one in the result, bit for bit, up to where the sums offset by offset would
    # overflow: one source near the centre of each of the 64 boxes, weights up to 2^1023 of one sign, 1/r below 2^-9.
    r = np.random.default_rng(poly_ord)
    grid = np.stack(np.meshgrid(*[np.arange(4.0)] * 3, indexing="ij"), -1).reshape(-1, 3)
    s = 1024.0 * (grid + 0.5 + r.uniform(-0.1, 0.1, (64, 3)))
    s = np.concatenate([s, [[0.0] * 3, [4096.0] * 3]])  # the cube; weightless
    w = np.concatenate([r.uniform(0.6, 1.0, 64), [0.0, 0.0]])
    t = 4096.0 * r.random((900, 3))
    ctx.set_kernel("inv_r_safe")
    base, _ = ctx.solve(t, s, w, poly_ord=poly_ord, depth=3)
    got, _ = ctx.solve(t, s, np.ldexp(w, power), poly_ord=poly_ord, depth=3)
    np.testing.assert_array_equal(got, np.ldexp(base, power))


@pytest.mark.parametrize("poly_ord", [2, 3, 4, 7])
def test_operators_of_a_narrow_gaussian(ctx, poly_ord):
    """The far field of a Gaussian whose exponent is some hundreds at the far boxes, against the same sum in extended
    precision: P2M, M2L and L2P with the double nodes, in long double.  Only far pairs count here (targets left,
    sources right), positive weights.  Plain double arithmetic in the exponent alone is off by about 300 * 2^-53 =
    3e-14 in every term; what is left otherwise is the rounding of P2M, L2P (4 (n - 1) + 4 steps a factor, three
    factors) and of the M2L's sums, 64 * 2^-53 of the terms' absolute sum, which is kappa (2 to 3) times the result.
    Node counts whose nodes nearest to the far box are exactly symmetric, as the symmetry assumes; the others carry
    the nodes' own rounding."""
    LD, n, p0 = np.longdouble, poly_ord + 1, 3e-4
    r = np.random.default_rng(poly_ord)
    t, s = r.random((60, 3)) * [0.2, 0.99, 0.99], r.random((70, 3)) * [0.2, 0.99, 0.99] + [0.55, 0.0, 0.0]
    s = np.concatenate([s, [[0.0, 0.0, 0.0], [1.0, 1.0, 1.0]]])  # the unit cube; weightless
    w = np.concatenate([r.uniform(0.5, 1.0, 70), [0.0, 0.0]])
    ctx.set_kernel("gaussian", p0)
    got, _ = ctx.solve(t, s, w, poly_ord=poly_ord, depth=3)

    import math
    node = np.array([math.cos((2.0 * k + 1.0) / (2 * n) * math.pi) for k in range(n)])

    def factors(y):  # S_n(node, y), T_j by the recurrence
        T = [np.ones_like(y), y]
        X = [np.ones(n, LD), node.astype(LD)]
        for _ in range(2, n):
            T.append(2 * y * T[-1] - T[-2])
            X.append(2 * node.astype(LD) * X[-1] - X[-2])
        return LD(1) / n + LD(2) / n * sum(np.multiply.outer(T[j], X[j]) for j in range(1, n))

    def boxes(p):
        i = np.minimum((p * 4).astype(int), 3)
        f = [factors(2 * (p[:, q].astype(LD) * 4 - i[:, q]) - 1) for q in range(3)]
        return i, np.einsum("pi,pj,pk->pijk", *f).reshape(len(p), n ** 3)
    ti, tf = boxes(t)
    si, sf = boxes(s)
    half = np.stack(np.meshgrid(*[node.astype(LD) / 2] * 3, indexing="ij"), -1).reshape(-1, 3)
    want, terms = np.zeros(len(t), LD), np.zeros(len(t), LD)
    for b in {tuple(x) for x in si[:70]}:
        wb = (w * (si == b).all(1)).astype(LD)
        for a in {tuple(x) for x in ti}:
            d = (half[:, None] - (half[None] + np.subtract(b, a))) / 4
            here = (ti == a).all(1)
            K = np.exp(-(d * d).sum(-1) / LD(p0))
            want[here] += tf[here] @ (K @ (wb @ sf))
            terms[here] += abs(tf[here]) @ (K @ (wb @ abs(sf)))
    err, scale = (np.linalg.norm(x.astype(float)) for x in (got - want, terms))
    assert err <= 64 * 2.0 ** -53 * scale, err / scale


@pytest.mark.parametrize("points", [80, 700, 3000])
@pytest.mark.parametrize("rhs", [1, 3])
def test_eight_nodes_on_sparse_and_dense_leaves(ctx, oracle, points, rhs):
    # the default leaf evaluation, which 8 nodes in 3-D have at every density
    r = np.random.default_rng(points)
    t, s, w = r.random((points, 3)), r.random((points, 3)), r.standard_normal((rhs, points))
    ctx.set_kernel("inv_r_safe")
    got, _ = ctx.solve(t, s, w, poly_ord=7, depth=3)
    want, _ = oracle.fmm(3, 1, 0.0, 7, 3, 1, t, s, w[rhs - 1])
    assert rel_l2(np.atleast_2d(got)[rhs - 1], want) <= TOL


def test_gaussian_of_points_beyond_its_range(ctx):
    # far boxes at a distance whose square overflows: their operators are zero, not undefined
    r = np.random.default_rng(2)
    s = 1e160 * r.random((600, 3))
    w = r.standard_normal(600)
    ctx.set_kernel("gaussian", 0.01)
    got, _ = ctx.solve(s, s, w, poly_ord=4, depth=4)
    np.testing.assert_array_equal(got, w)  # only the coincident pair of every point counts
