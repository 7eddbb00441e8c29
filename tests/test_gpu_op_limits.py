"""Operator tables at the limits of their construction (mw_optab.cu): groups whose lists are built one operator at a time,
and lists beyond 32-bit positions.

Bar: tables equal those of an operator built alone bit for bit; what is refused is an error and leaves the context usable."""
import math

import pytest

from test_gpu_parity import WORLD, assert_same_tree, two_gaussians

pytestmark = pytest.mark.gpu


def row_world(G, boxes, order=3):
    """a row of boxes: the bands of the wide terms reach over all of it, in every direction"""
    return G.MultiResolutionAnalysis(-2, (-(boxes // 2), 0, 0), (boxes, 1, 1), order, 10)


def test_large_lists_of_a_group(gpu_mod):
    """about 14 million records each at the root: more than one group holds, 32-bit counts apart"""
    G = gpu_mod
    m = row_world(G, 40)
    f = G.FunctionTree(m)
    G.project(1e-2, f, G.gauss_params([1.0], [2.0], [(0.3, 1.9, 2.2)]))
    precs = [1e-3, 2e-3, 5e-3]
    ops = [G.PoissonOperator(m, p) for p in precs]
    outs = [G.FunctionTree(m) for _ in ops]
    G.apply_batched(1e-2, outs, ops, [f] * 3)
    for p, out in zip(precs, outs):
        one = G.FunctionTree(m)
        G.apply(1e-2, one, G.PoissonOperator(m, p), f)
        assert one.square_norm() > 0.0
        assert_same_tree(out.export(), one.export(), tol=0.0)


def test_lists_beyond_32_bit_positions_are_refused(gpu_mod):
    """about 4e9 records of one operator"""
    G = gpu_mod
    m = row_world(G, 256)
    f = G.FunctionTree(m)
    G.project(1e-2, f, G.gauss_params([1.0], [2.0], [(0.3, 1.9, 2.2)]))
    out = G.FunctionTree(m)
    for ops in ([G.PoissonOperator(m, 1e-3)], [G.PoissonOperator(m, 1e-3), G.PoissonOperator(m, 2e-3)]):
        with pytest.raises(G.MWError, match="offset list too large"):
            G.apply_batched(1e-2, [out, G.FunctionTree(m)][: len(ops)], ops, [f] * len(ops))
    G.apply(1e-2, out, G.HelmholtzOperator(m, 20.0, 1e-3), f)  # the context goes on
    assert out.square_norm() > 0.0


def test_operator_without_terms(gpu_mod):
    """a decay length far below the finest scale leaves no term of the expansion: the operator gives zero, alone and at
    any place of a batch"""
    G = gpu_mod
    prec, depth = 1e-3, 10
    m = G.MultiResolutionAnalysis(*WORLD, 5, depth)
    eps, r_min = 0.1 * prec, 0.01 * 4.0 * 2.0 ** -depth
    h = math.pi ** 2 / (2.0 * math.log(2.0 * math.sqrt(2.0) / eps))
    s_hi = math.log((math.sqrt(-math.log(0.1 * eps)) + 1.0) / r_min)
    mu = 2.0 * math.sqrt(-math.log(1e-3 * eps)) * math.exp(s_hi + 1.5 * h)  # one and a half steps beyond the range
    none = G.HelmholtzOperator(m, mu, prec)
    assert len(none.terms()[0]) == 0
    f = G.FunctionTree(m)
    G.project(prec, f, two_gaussians(G))
    out = G.FunctionTree(m)
    G.apply(prec, out, none, f)
    assert out.square_norm() == 0.0 and out.nnodes() == 1000
    some = G.HelmholtzOperator(m, 1.0, prec)
    one = G.FunctionTree(m)
    G.apply(prec, one, some, f)
    for where in range(3):
        ops = [G.HelmholtzOperator(m, 1.0, prec) for _ in range(2)]
        ops.insert(where, G.HelmholtzOperator(m, mu, prec))
        outs = [G.FunctionTree(m) for _ in ops]
        G.apply_batched(prec, outs, ops, [f] * 3)
        for q, t in enumerate(outs):
            if q == where:
                assert t.square_norm() == 0.0
            else:
                assert_same_tree(t.export(), one.export(), tol=0.0)


def test_bands_wider_than_the_lists(gpu_mod):
    """At order 3 and operator precision 1e-6 the scaling blocks of the widest term reach 1014 offsets at depth 10, its bounds
    far fewer: the matrices are held, the lists fit.  The self-energy of six Gaussians of unit charge about one point,
    each finding the next on the grid, against 2 / sqrt(pi) sum (a b / (a + b))^(1/2); the bar is the apply's precision
    carried through <f|V>, 1e-4 ||f|| ||V||, 18 of 2189."""
    G = gpu_mod
    m = G.MultiResolutionAnalysis(-2, (0, 0, 0), (1, 1, 1), 3, 14)
    alpha = [16.0 * 8.0 ** j for j in range(6)]
    f, out = G.FunctionTree(m), G.FunctionTree(m)
    G.project(1e-4, f, G.gauss_params([(a / math.pi) ** 1.5 for a in alpha], alpha, [(2.1, 1.9, 2.05)] * 6))
    G.apply(1e-4, out, G.PoissonOperator(m, 1e-6), f)
    assert out.export(False)["depth"].max() >= 10
    energy = sum(2.0 / math.sqrt(math.pi) * math.sqrt(a * b / (a + b)) for a in alpha for b in alpha)
    assert abs(G.dot(f, out) - energy) < 1e-4 * math.sqrt(f.square_norm() * out.square_norm())
