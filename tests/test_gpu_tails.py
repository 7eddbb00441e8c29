"""Factors generated many levels below a leaf where the function decays: a block generated level by level is accurate relative
to its own size at every level, not to that of the leaf it comes from, so that a product far below its factors is a smooth
function and not rounding noise that refinement chases.

Bars: the product's tree against the CPU oracle's, which generates level by level too: its size within a factor of two (both
sides' leaves carry rounding of their own).  Below a leaf the function is one polynomial, so the wavelet part of every node of
its sum or product with one is rounding: 1e-12 of the node's own largest coefficient (of the products 1e-11: they pass
through point values, 1 / sqrt(w) and sqrt(w) per direction)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,basis", [(4, 0), (6, 1), (7, 0), (9, 0), (10, 0)])
def test_product_of_separated_functions(gpu_mod, oracle_mod, order, basis):
    G, O = gpu_mod, oracle_mod
    size = []
    for M in (G, O):
        m = M.MultiResolutionAnalysis(0, (-2, 0, 0), (4, 1, 1), order, 7, basis)
        a, b, out = M.FunctionTree(m), M.FunctionTree(m), M.FunctionTree(m)
        M.project(1e-3, a, M.gauss_params([1.0], [345.0], [(0.73, 0.79, 0.19)], [(0, 1, 2)]))
        M.project(1e-3, b, M.gauss_params([1.0], [83.0], [(-1.84, 0.53, 0.46)], [(0, 1, 2)]))
        M.multiply(1e-3, out, -1.3, a, b)
        size.append(out.nnodes())
    assert size[0] <= 2 * size[1] and size[1] <= 2 * size[0], size


@pytest.mark.parametrize("order", range(3, 11))
def test_generated_blocks_are_smooth(gpu_mod, order):
    """sums and products on a grid five levels deep in the tail of a function whose tree ends at the root there"""
    G = gpu_mod
    k = order + 1
    m = G.MultiResolutionAnalysis(0, (-2, 0, 0), (4, 1, 1), order, 9)
    f, one, grid, out = (G.FunctionTree(m) for _ in range(4))
    G.project(1e-3, f, G.gauss_params([1.0], [83.0], [(-1.84, 0.53, 0.46)]))
    G.project(-1.0, one, G.gauss_params([1.0], [0.0], [(0.0, 0.0, 0.0)]))
    # a grid refined towards the end of the box that is farther from the function
    G.project(1e-2, grid, G.gauss_params([1.0] * 4, [500.0, 4e3, 3e4, 2.4e5], [(0.93, 0.6, 0.6)] * 4))
    e = f.export()
    tree = {(int(d), *map(int, x)): c for d, x, c in zip(e["depth"], e["trans"], e["coef"])}
    assert (0, 2, 0, 0) in tree and (1, 4, 0, 0) not in tree  # box [0, 1]: one leaf, values falling by many decades
    for kind in ("add", "multiply"):
        G.copy_grid(out, grid)
        if kind == "add":
            G.add(-1.0, out, [0.7], [f])
        else:
            G.multiply(-1.0, out, 0.7, f, one, 0)
        e = out.export()
        deep, small = 0, 1.0
        for d, x, c in zip(e["depth"], e["trans"], e["coef"].reshape(-1, 2 * k, 2 * k, 2 * k)):
            if d < 1 or int(x[0]) >> int(d) != 2:
                continue
            w = c.copy()
            w[:k, :k, :k] = 0.0
            size = np.abs(c).max()
            assert np.abs(w).max() <= (1e-12 if kind == "add" else 1e-11) * size, (d, x, kind)
            deep, small = max(deep, int(d)), min(small, size)
        assert deep >= 5 and small < 1e-6 * np.abs(tree[(0, 2, 0, 0)]).max()
