"""Inner products of trees with more nodes than the kernel has groups of warps (below k = 8: 8 blocks of two groups per SM,
which take nodes in turn; from k = 8 up a group a node), with equal and with different grids, against the allocation-free inner product, which sums per node.

Bar: 1e-12 relative, that of the other inner products."""
import numpy as np
import pytest

from test_gpu_parity import WORLD

pytestmark = pytest.mark.gpu


def spikes(G, m, prec, n, box, seed):
    rng = np.random.default_rng(seed)
    a = np.exp(rng.uniform(np.log(0.5), np.log(3e3), n))
    t = G.FunctionTree(m)
    G.project(prec, t, G.gauss_params(list((a / np.pi) ** 0.75), list(a), [tuple(x) for x in rng.uniform(-box, box, (n, 3))]))
    return t


@pytest.mark.parametrize("order,prec,coarse,nodes", [(3, 1e-4, 1e-2, 18000), (4, 1e-5, 1e-3, 13000), (6, 3e-6, 1e-4, 5000),
                                                     (7, 1e-7, 1e-5, 19000)])
def test_dot_of_large_trees(gpu_mod, order, prec, coarse, nodes):
    G = gpu_mod
    m = G.MultiResolutionAnalysis(*WORLD, order, 15)
    a, b = spikes(G, m, prec, 60, 9.0, order), spikes(G, m, coarse, 60, 9.0, order)
    assert a.nnodes() > nodes
    for x, y in ((a, a), (a, b), (b, a)):
        ref = G.nalloc_dot(x, y)
        assert abs(G.dot(x, y) - ref) <= 1e-12 * abs(ref)
    assert G.dot(a, b) == G.dot(a, b)  # a fixed order of sums
