"""M2M and L2L by parent (translate.cu) at the sizes where they can go wrong, through the fmm, against the oracle.

Tolerance: relative L2 <= 1e-12, that of the plain FP64 parity tests: sums of a few hundred terms in another order.

Every node count in its range and one above it; trees of depth 5 and more, so that both run over several levels;
crowded points (parents with one child and with all), targets and sources in different corners (children with one of
them only); right-hand sides that leave a warp's last unit group partly filled and that split a parent over two groups;
problems of different depths."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-12


@pytest.mark.parametrize("d,poly_ord,depth", [(1, p, 6) for p in (0, 1, 4, 7, 8, 11, 15)]
                         + [(2, p, 5) for p in (0, 1, 2, 3, 4, 5, 6, 7, 8)]
                         + [(3, p, 4) for p in (0, 1, 2, 3, 4, 5, 6, 7)])
def test_every_node_count(ctx, oracle, d, poly_ord, depth):
    r = np.random.default_rng(16 * d + poly_ord)
    n = 60 if (d, poly_ord) == (3, 7) else 400
    t, s = r.random((n, d)) ** 2, 1.0 - r.random((n + 11, d)) ** 3  # crowded towards opposite corners
    w = r.standard_normal((3, n + 11))
    ctx.set_kernel("inv_r_safe")
    for nrhs in (1, 3):
        got = np.asarray(ctx.solve(t, s, w[:nrhs], poly_ord=poly_ord, depth=depth)[0]).reshape(nrhs, -1)
        for k in (0, nrhs - 1):
            want, _ = oracle.fmm(d, 1, 0.0, poly_ord, depth, 1, t, s, w[k].copy())
            assert rel_l2(got[k], want) <= TOL


@pytest.mark.parametrize("d,poly_ord", [(1, 5), (2, 4), (3, 2), (3, 4)])
@pytest.mark.parametrize("nrhs", [2, 5, 7, 16, 33])
def test_right_hand_sides(ctx, oracle, d, poly_ord, nrhs):
    r = np.random.default_rng(nrhs + d)
    t, s, w = r.random((500, d)), r.random((450, d)), r.standard_normal((nrhs, 450))
    ctx.set_kernel("inv_r_safe")
    got = np.asarray(ctx.solve(t, s, w, poly_ord=poly_ord, depth=6 - d)[0]).reshape(nrhs, -1)
    for k in (0, nrhs // 2, nrhs - 1):
        want, _ = oracle.fmm(d, 1, 0.0, poly_ord, 6 - d, 1, t, s, w[k].copy())
        assert rel_l2(got[k], want) <= TOL


@pytest.mark.parametrize("nrhs", [1, 6])
def test_forest_of_different_depths(ctx, oracle, nrhs):
    r = np.random.default_rng(6)
    sizes, depths = [900, 30, 5, 400, 2000], [4, 2, 3, 6, 5]
    off = np.concatenate([[0], np.cumsum(sizes)])
    t, s, w = r.random((off[-1], 2)), r.random((off[-1], 2)), r.standard_normal((nrhs, off[-1]))
    ctx.set_kernel("multiquadric", 1e-2)
    got = np.asarray(ctx.forest_solve(t, off, s, off, w, depths, poly_ord=4)).reshape(nrhs, -1)
    for p, depth in enumerate(depths):
        a, b = off[p], off[p + 1]
        want, _ = oracle.fmm(2, 5, 1e-2, 4, depth, 1, t[a:b], s[a:b], w[nrhs - 1, a:b].copy())
        assert rel_l2(got[nrhs - 1, a:b], want) <= TOL
