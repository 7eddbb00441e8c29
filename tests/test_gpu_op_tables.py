"""Operator tables built on the device (mw_optab.cu): groups of operators against operators built alone, bands
wider than the first scratch (64 offsets), and worlds of few boxes, the latter two against the FP64 CPU oracle.

Bar: a group's tables equal single ones bit for bit (each term is computed by itself); against the oracle the
repository's bar for FP64 applies, identical trees and triple counts, coefficients within 1e-10 of the largest."""
import numpy as np
import pytest

from test_gpu_parity import WORLD, assert_same_tree, pair, to_oracle, two_gaussians

pytestmark = pytest.mark.gpu


def test_operators_of_a_batch_equal_single_ones(gpu_mod):
    """ten operators (more than one group), one of them listed twice, Poisson among them"""
    G = gpu_mod
    prec = 1e-4
    m = G.MultiResolutionAnalysis(*WORLD, 7, 14)
    f = G.FunctionTree(m)
    G.project(prec, f, two_gaussians(G))
    mus = [0.0, 0.5, 0.9, 1.3, 1.7, 2.1, 2.5, 2.9, 3.3, 3.7]
    ops = [G.ConvolutionOperator(m, mu, prec) for mu in mus]
    ops.append(ops[4])
    outs = [G.FunctionTree(m) for _ in ops]
    G.apply_batched(prec, outs, ops, [f] * len(ops))
    for mu, out in zip(mus + [mus[4]], outs):
        one = G.FunctionTree(m)
        G.apply(prec, one, G.ConvolutionOperator(m, mu, prec), f)
        assert_same_tree(out.export(), one.export(), tol=0.0)


@pytest.mark.parametrize("order,prec", [(3, 1e-3)])
def test_wide_bands(gpu_mod, oracle_mod, order, prec):
    """at order 3 the widest band of depth 3 has 79 offsets per side, of depth 4 159"""
    G, O = gpu_mod, oracle_mod
    mg, mo = pair(G, O, order)
    f = G.FunctionTree(mg)
    G.project(prec, f, G.gauss_params([1.0], [30.0], [(0.1, -0.2, 0.3)]))
    out, out_o = G.FunctionTree(mg), O.FunctionTree(mo)
    sg = G.apply(prec, out, G.PoissonOperator(mg, prec), f)
    so = O.apply(prec, out_o, O.PoissonOperator(mo, prec), to_oracle(O, mo, f))
    assert sg[2] >= 4 and sg[0] == so[0]
    assert_same_tree(out.export(), out_o.export())


@pytest.mark.parametrize("corner,boxes", [((-1, 0, -1), (3, 1, 2)), ((0, 0, 0), (1, 1, 1)), ((-1, -1, -1), (2, 2, 2))])
def test_small_worlds(gpu_mod, oracle_mod, corner, boxes):
    G, O = gpu_mod, oracle_mod
    order, prec = 6, 1e-4
    mg = G.MultiResolutionAnalysis(-2, corner, boxes, order, 14)
    mo = O.MultiResolutionAnalysis(-2, corner, boxes, order, 14)
    f = G.FunctionTree(mg)
    G.project(prec, f, G.gauss_params([1.0], [6.0], [(0.9, 0.8, 1.1)]))
    out, out_o = G.FunctionTree(mg), O.FunctionTree(mo)
    sg = G.apply(prec, out, G.HelmholtzOperator(mg, 0.6, prec), f)
    so = O.apply(prec, out_o, O.HelmholtzOperator(mo, 0.6, prec), to_oracle(O, mo, f))
    assert sg[0] == so[0]
    assert_same_tree(out.export(), out_o.export())
    assert np.isfinite(out.square_norm())
