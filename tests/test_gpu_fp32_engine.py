"""The FP32 engine at every basis size it is instantiated for, against the FP64 engine: the tile shapes of
P = 8, 12, 16, 20 and 24 columns per slice, threads past the last tile, generated inputs, the s->s correction,
and chunks of one triple and of whole nodes.

Bar: identical tree structure; relative L2 error at most 3 * 24 * 2^-24 = 4.3e-6, three mode products of at
most 24 FP32 multiply-adds each, every one rounding at 2^-24 of the largest partial sum."""
import numpy as np
import pytest

from test_gpu_parity import keyed, pair, two_gaussians

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk", [1, 4096])
@pytest.mark.parametrize("order,prec", [(3, 1e-2), (4, 1e-3), (5, 1e-3), (6, 1e-4), (7, 1e-4), (8, 1e-5), (9, 1e-5),
                                        (10, 1e-5), (11, 1e-5)])
def test_orders_against_fp64(gpu_mod, oracle_mod, order, prec, chunk):
    G = gpu_mod
    mg, _ = pair(G, oracle_mod, order)
    inp = G.FunctionTree(mg)
    G.project(prec, inp, two_gaussians(G))
    op = G.HelmholtzOperator(mg, 0.7, prec)
    outs = []
    for flags in (G.APPLY_FP64, G.APPLY_FP32):
        before = mg.ctx.chunk_triples(flags)
        mg.ctx.set_chunk_triples(flags, chunk)
        try:
            out = G.FunctionTree(mg)
            triples = G.apply(prec, out, op, inp, flags)[0]
        finally:
            mg.ctx.set_chunk_triples(flags, before)
        outs.append((triples, out.export()))
    (t64, a), (t32, b) = outs
    assert t64 == t32
    ka, kb = keyed(a), keyed(b)
    assert set(ka) == set(kb)
    ca = np.stack([a["coef"][ka[q]] for q in ka])
    cb = np.stack([b["coef"][kb[q]] for q in ka])
    assert np.linalg.norm(ca - cb) <= 3 * 24 * 2.0**-24 * np.linalg.norm(ca)
