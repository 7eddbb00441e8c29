"""The FP64 engine (matrix-instruction contraction) at every basis size it is instantiated for, against the
FP64 CPU oracle: the tile remainders of 2k (0, 2, 4, 6 mod 8), planes of one and of several lines, generated
inputs, and the s->s correction.

Bar: integer tree structure and triple counts identical; FP64 coefficients within 1e-10 of the largest one
(the repository's bar for FP64 applies: sums of at most a few thousand products of rounding 1e-16)."""
import numpy as np
import pytest

from test_gpu_parity import assert_same_tree, pair, to_oracle, two_gaussians

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk", [1, 48, 4096])
@pytest.mark.parametrize("order,prec", [(3, 1e-2), (4, 1e-3), (5, 1e-3), (6, 1e-4), (7, 1e-4), (8, 1e-5), (9, 1e-5),
                                        (10, 1e-5), (11, 1e-5)])
def test_orders_against_oracle(gpu_mod, oracle_mod, order, prec, chunk):
    G, O = gpu_mod, oracle_mod
    mg, mo = pair(G, O, order)
    inp = G.FunctionTree(mg)
    G.project(prec, inp, two_gaussians(G))
    out, out_o = G.FunctionTree(mg), O.FunctionTree(mo)
    before = mg.ctx.chunk_triples(G.APPLY_FP64)
    mg.ctx.set_chunk_triples(G.APPLY_FP64, chunk)
    try:
        sg = G.apply(prec, out, G.HelmholtzOperator(mg, 0.7, prec), inp)
    finally:
        mg.ctx.set_chunk_triples(G.APPLY_FP64, before)
    so = O.apply(prec, out_o, O.HelmholtzOperator(mo, 0.7, prec), to_oracle(O, mo, inp))
    assert sg[0] == so[0]
    assert_same_tree(out.export(), out_o.export())
    assert np.isfinite(out.square_norm())
