"""Block transforms on the FP64 matrix instruction at every basis size (tile remainders of 2k and of k), against the FP64
CPU oracle: adaptive projection and compression, products and sums whose factors lack nodes by one and by several levels, the
device-side union grid, and inner products.

Bar: integer tree structure identical; FP64 coefficients within 1e-10 of the largest one (the repository's bar), plus what
the two sides' two-scale filters differ by (each builds its own by Gram-Schmidt, whose conditioning grows with the order: 1e-11
at order 9, 3e-10 at 10, 2e-9 at 11): three directions of 2k terms each."""
import numpy as np
import pytest

from test_gpu_parity import assert_same_tree, pair, to_oracle

pytestmark = pytest.mark.gpu

PREC = {3: 1e-2, 4: 1e-3, 5: 1e-3, 6: 1e-4, 7: 1e-4, 8: 1e-5, 9: 1e-5, 10: 1e-5, 11: 1e-5}
SHARP, WIDE = (60.0, (0.31, -0.17, 0.23)), (0.8, (0.1, 0.2, -0.3))


def bar(mg, mo):
    d = np.abs(mg.filter() - mo.filter())
    return 1e-10 + 3 * len(d) * d.max()


def project_both(G, O, mg, mo, prec, spec):
    f = G.gauss_params([spec[0] ** 0.75], [spec[0]], [spec[1]], [(1, 0, 2)])  # with a polynomial factor
    tg, to = G.FunctionTree(mg), O.FunctionTree(mo)
    G.project(prec, tg, f)
    O.project(prec, to, f)
    return tg, to


@pytest.mark.parametrize("order", sorted(PREC))
def test_projection_and_dot(gpu_mod, oracle_mod, order):
    G, O = gpu_mod, oracle_mod
    mg, mo = pair(G, O, order)
    a, ao = project_both(G, O, mg, mo, PREC[order], SHARP)
    b, bo = project_both(G, O, mg, mo, PREC[order], WIDE)
    tol = bar(mg, mo)
    assert_same_tree(a.export(), ao.export(), tol)
    assert_same_tree(b.export(), bo.export(), tol)
    scale = np.sqrt(a.square_norm() * b.square_norm())
    for x, y, xo, yo in ((a, b, ao, bo), (b, a, bo, ao), (a, a, ao, ao)):
        assert abs(G.dot(x, y) - O.dot(xo, yo)) < tol * scale


@pytest.mark.parametrize("order", [q for q in sorted(PREC) if q <= 10])
def test_products_and_sums_below_coarse_factors(gpu_mod, oracle_mod, order):
    """on the sharp function's grid the wide one is generated, several levels below its leaves at the centre"""
    G, O = gpu_mod, oracle_mod
    mg, mo = pair(G, O, order)
    a, _ = project_both(G, O, mg, mo, PREC[order], SHARP)
    b, _ = project_both(G, O, mg, mo, PREC[order], WIDE)
    assert a.export(False)["depth"].max() >= b.export(False)["depth"].max() + (2 if order < 9 else 1)
    ao, bo = to_oracle(O, mo, a), to_oracle(O, mo, b)
    for x, y, xo, yo in ((a, b, ao, bo), (b, a, bo, ao), (a, a, ao, ao)):
        g, o = G.FunctionTree(mg), O.FunctionTree(mo)
        for t, to in ((x, xo), (y, yo)):
            G.build_grid(g, t)
            O.build_grid(o, to)
        n = g.nnodes()
        G.build_grid(g, x)  # nothing to add
        assert g.nnodes() == n
        G.multiply(-1.0, g, 0.7, x, y, 0)
        O.multiply(-1.0, o, 0.7, xo, yo, 0)
        assert_same_tree(g.export(), o.export(), bar(mg, mo))
        G.add(-1.0, g, [0.3, -1.1], [x, y], 0)
        O.add(-1.0, o, [0.3, -1.1], [xo, yo], 0)
        assert_same_tree(g.export(), o.export(), bar(mg, mo))


def test_union_grid_keeps_blocks(gpu_mod):
    """nodes added between a function's own leave its blocks and norms as they are, through several growths"""
    G = gpu_mod
    mg = G.MultiResolutionAnalysis(-2, (-5, -5, -5), (10, 10, 10), 5, 14)
    t = G.FunctionTree(mg)
    G.project(1e-3, t, G.gauss_params([1.0], [4.0], [(0.1, 0.2, 0.3)]))
    before = t.export()
    key = lambda e: {(int(d), *map(int, x)): i for i, (d, x) in enumerate(zip(e["depth"], e["trans"]))}
    for q in range(4):
        u = G.FunctionTree(mg)
        G.project(1e-3, u, G.gauss_params([1.0], [300.0 * 4 ** q], [(6.0 - 4 * q, -5.0 + 3 * q, 2.0 * q)]))
        G.build_grid(t, u)
        ku, kt = key(u.export(False)), key(t.export(False))
        assert set(ku) <= set(kt)
    after = t.export()
    kb, ka = key(before), key(after)
    for k, i in kb.items():
        assert np.array_equal(before["coef"][i], after["coef"][ka[k]])
    for k, i in ka.items():
        if k not in kb:
            assert not after["coef"][i].any()
        p = after["parent"][i]
        assert p < 0 if k[0] == 0 else (int(after["depth"][p]), *map(int, after["trans"][p])) == (k[0] - 1, *(x >> 1 for x in k[1:]))
    assert np.all(np.diff(after["depth"]) >= 0)
