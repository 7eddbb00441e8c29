"""Device memory that a pass holds at once, from the device pool's high-water mark."""
import ctypes

import pytest

from test_gpu_parity import WORLD, two_gaussians

pytestmark = pytest.mark.gpu

USED_CURRENT, USED_HIGH = 7, 8  # CU_MEMPOOL_ATTR_USED_MEM_*


class Pool:
    """the device's default memory pool (driver API)"""

    def __init__(self):
        self.L = ctypes.CDLL("libcuda.so.1")
        dev, self.h = ctypes.c_int(), ctypes.c_void_p()
        assert self.L.cuDeviceGet(ctypes.byref(dev), 0) == 0
        assert self.L.cuDeviceGetDefaultMemPool(ctypes.byref(self.h), dev) == 0

    def get(self, attr):
        v = ctypes.c_uint64()
        assert self.L.cuMemPoolGetAttribute(self.h, attr, ctypes.byref(v)) == 0
        return v.value

    def reset_high(self):
        v = ctypes.c_uint64(0)
        assert self.L.cuMemPoolSetAttribute(self.h, USED_HIGH, ctypes.byref(v)) == 0


@pytest.mark.parametrize("order,flags", [(3, 0), (4, 1)])
def test_pass_holds_sorted_triples_only(gpu_mod, order, flags):
    """While the partial blocks exist, of the triples only the sorted keys and values (16 bytes each) do: the unsorted ones
    are given back after the sort.  One pass (roots only), one CTA per 48 triples: per triple 16 bytes of them are a
    fifth of what a partial block takes at this order."""
    G = gpu_mod
    ctx = G.Context.default()
    m = G.MultiResolutionAnalysis(*WORLD, order, 0)
    f = G.FunctionTree(m)
    # one box per Gaussian for many input nodes: their root blocks are all non-zero
    c = [(4.0 * x + 2.0, 4.0 * y + 2.0, 4.0 * z + 2.0) for x in range(-4, 4, 2) for y in range(-4, 4, 2) for z in range(-4, 4, 2)]
    G.project(1e-3, f, G.gauss_params([1.0] * len(c), [0.05] * len(c), c))
    op, out, pool = G.PoissonOperator(m, 1e-3), G.FunctionTree(m), Pool()
    assert G.apply(1e-4, out, op, f, flags)[2] == 1  # tables and tree arrays exist from here on
    ctx.profile(True)
    ctx.synchronize()
    base = pool.get(USED_CURRENT)
    pool.reset_high()
    trip = G.apply(1e-4, out, op, f, flags)[0]
    ctx.synchronize()
    high, ctas = pool.get(USED_HIGH) - base, ctx.profile_ctas()
    ctx.profile(False)
    assert trip > 4_000_000
    block, ncand = 8 * (2 * (order + 1)) ** 3, 1000 * 1000
    # partial blocks, sorted triples, chunk lists (with their sorted copy), candidates, block images and generated nodes
    held = ctas * (block + 48) + 16 * trip + 33 * ncand + 1000 * 4 * block
    sort = 32 * trip + 20 * trip + 33 * ncand  # the sort itself: both sides and its scratch
    assert high <= max(held, sort) + (32 << 20), (high, held, sort)


def test_union_grid_keeps_little_spare_room(gpu_mod):
    """A grid made in a tree that once held many more nodes: the merged arrays keep room to grow, but no more than 1 GiB of
    it beside the tree's own (the old ones are still there while they are filled)."""
    import numpy as np

    G = gpu_mod
    ctx = G.Context.default()
    m = G.MultiResolutionAnalysis(*WORLD, 9, 14)
    rng = np.random.default_rng(1)
    a = np.exp(rng.uniform(np.log(0.5), np.log(3e3), 120))
    big, small, pool = G.FunctionTree(m), G.FunctionTree(m), Pool()
    G.project(1e-8, big, G.gauss_params(list((a / np.pi) ** 0.75), list(a), [tuple(x) for x in rng.uniform(-9, 9, (120, 3))]))
    G.project(1e-5, small, two_gaussians(G))
    block, n = 8 * 20 ** 3, small.nnodes()
    assert big.nnodes() * block > 2 << 30
    G.clear(big)
    ctx.synchronize()
    base = pool.get(USED_CURRENT)
    pool.reset_high()
    G.build_grid(big, small)
    ctx.synchronize()
    assert big.nnodes() == n
    assert pool.get(USED_HIGH) - base <= n * block + (1 << 30) + (32 << 20)
    assert pool.get(USED_CURRENT) < base
    G.multiply(1e-5, big, 1.0, small, small)  # and it grows again
    assert big.square_norm() > 0.0
