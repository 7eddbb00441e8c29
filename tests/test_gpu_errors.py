"""A call that fails for want of device memory is an error of that call alone: the next call on the context answers."""
import pytest

from test_gpu_parity import WORLD, two_gaussians

pytestmark = pytest.mark.gpu


def test_calls_go_on_after_a_failed_allocation(gpu_mod):
    G = gpu_mod
    ctx = G.Context(0)
    m = G.MultiResolutionAnalysis(*WORLD, 5, 10, ctx=ctx)
    f, out = G.FunctionTree(m), G.FunctionTree(m)
    G.project(1e-3, f, two_gaussians(G))
    op = G.PoissonOperator(m, 1e-3)
    for call in (lambda: G.project(1e-3, f, two_gaussians(G)), lambda: G.apply(1e-3, out, op, f), lambda: G.dot(f, f)):
        with pytest.raises(G.MWError):
            ctx.reserve(1 << 46)  # 64 TB: refused at once
        call()
    assert out.square_norm() > 0.0
