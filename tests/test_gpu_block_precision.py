"""Block transforms and the FP64 contraction at every order against numpy with the library's own two-scale filter and operator
matrices, so that the comparison is not loosened by what two Gram-Schmidt filters differ by: projection, compression, sums and
products of factors that lack nodes, and one output node of an apply (own and generated input nodes, root and next level).

Bar: 1e-12 of the largest coefficient.  A separable transform with an orthogonal 2k x 2k matrix loses at most 3 2k 2^-53 of a
fibre's norm, which is at most (2k)^(1/2) times its largest entry per direction: 9e-13 at k = 12 if every rounding went
the same way.  Products pass through point values (1 / sqrt(w) per direction, 6 at k = 11) and back: 1e-11."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BAR = 1e-12
WORLD = (-2, (-2, -2, -2), (4, 4, 4))


def modes(A, X, B=None, C=None):
    """(C (x) B (x) A) X for blocks X[..., z, y, x]"""
    B, C = A if B is None else B, A if C is None else C
    return np.einsum("cz,...zyx->...cyx", C, np.einsum("by,...zyx->...zbx", B, np.einsum("ax,...zyx->...zya", A, X)))


class Tree:
    def __init__(self, t):
        e = t.export()
        k2 = 2 * t.mra.k
        self.child0, self.coef = e["child0"], e["coef"].reshape(-1, k2, k2, k2)
        self.at = {(int(d), *map(int, x)): i for i, (d, x) in enumerate(zip(e["depth"], e["trans"]))}
        self.scale = np.abs(self.coef).max()

    def block(self, key, F):
        """the block at a node, generated below the deepest node on the path (zero wavelets)"""
        if key in self.at:
            return self.coef[self.at[key]]
        d, x = key[0], key[1:]
        k = len(F) // 2
        up = self.block((d - 1, *(q >> 1 for q in x)), F)
        s = modes(F.T, up)
        out = np.zeros_like(up)
        out[:k, :k, :k] = s[tuple(slice((q & 1) * k, (q & 1) * k + k) for q in reversed(x))]
        return out


def check_compressed(t, F):
    k = len(F) // 2
    for key, i in t.at.items():
        c0 = t.child0[i]
        if c0 < 0:
            continue
        ch = t.coef[c0:c0 + 8, :k, :k, :k].reshape(2, 2, 2, k, k, k).transpose(0, 3, 1, 4, 2, 5).reshape(2 * k, 2 * k, 2 * k)
        assert np.abs(modes(F, ch) - t.coef[i]).max() <= BAR * t.scale


def quadrature(k):
    q, w = np.polynomial.legendre.leggauss(k)
    return 0.5 * (q + 1.0), 0.5 * w


def setup(G, order):
    m = G.MultiResolutionAnalysis(*WORLD, order, 5)
    k = order + 1
    q, w = quadrature(k)
    F = m.filter()
    assert np.abs(F @ F.T - np.eye(2 * k)).max() < 1e-12
    PF = F @ np.diag(np.tile(np.sqrt(w), 2))      # interpolating basis: phi_j(x_q) = delta_jq / sqrt(w_q)
    MV = np.diag(np.tile(1.0 / np.sqrt(w), 2)) @ F.T
    return m, k, q, F, PF, MV


SHARP, WIDE = (40.0, (0.31, 0.27, 0.23)), (0.4, (0.2, 0.1, 0.3))
PREC = {3: 1e-2, 4: 1e-3, 5: 1e-3, 6: 1e-4, 7: 1e-4, 8: 1e-5, 9: 1e-5, 10: 1e-6, 11: 1e-6}


@pytest.mark.parametrize("order", range(3, 12))
def test_projection_and_compression(gpu_mod, order):
    G = gpu_mod
    m, k, q, F, PF, _ = setup(G, order)
    t = G.FunctionTree(m)
    G.project(PREC[order], t, G.gauss_params([1.7, -0.6], [SHARP[0], 3.0], [SHARP[1], (-1.0, 0.5, 0.2)], [(1, 0, 2), (0, 1, 0)]))
    T = Tree(t)
    assert max(key[0] for key in T.at) >= 2
    check_compressed(T, F)
    leaves = 0
    for key, i in T.at.items():
        if T.child0[i] >= 0:
            continue
        d, x = key[0], np.array(key[1:])
        h = 2.0 ** -(-2 + d + 1)
        p = [-8.0 + (2 * x[a] + np.concatenate([q, q + 1.0])) * h for a in range(3)]
        v = 0.0
        for c, a, r, pw in ((1.7, SHARP[0], SHARP[1], (1, 0, 2)), (-0.6, 3.0, (-1.0, 0.5, 0.2), (0, 1, 0))):
            f = [(p[e] - r[e]) ** pw[e] * np.exp(-a * (p[e] - r[e]) ** 2) for e in range(3)]
            v = v + c * f[2][:, None, None] * f[1][None, :, None] * f[0][None, None, :]
        assert np.abs(modes(PF, v) * 2.0 ** (-1.5 * (-2 + d + 1)) - T.coef[i]).max() <= BAR * T.scale
        leaves += 1
    assert leaves > 64


@pytest.mark.parametrize("order", range(3, 11))
def test_sums_and_products_below_coarse_factors(gpu_mod, order):
    G = gpu_mod
    m, k, q, F, PF, MV = setup(G, order)
    a, b, g = G.FunctionTree(m), G.FunctionTree(m), G.FunctionTree(m)
    G.project(PREC[order], a, G.gauss_params([1.0], [SHARP[0]], [SHARP[1]]))
    G.project(PREC[order], b, G.gauss_params([1.0], [WIDE[0]], [WIDE[1]]))
    A, B = Tree(a), Tree(b)
    G.copy_grid(g, a)
    G.build_grid(g, b)
    for kind in ("add", "multiply"):
        if kind == "add":
            G.add(-1.0, g, [0.3, -1.1], [a, b], 0)
        else:
            G.multiply(-1.0, g, 0.7, a, b, 0)
        out, missing = Tree(g), 0
        check_compressed(out, F)
        for key, i in out.at.items():
            if out.child0[i] >= 0:
                continue
            x, y = A.block(key, F), B.block(key, F)
            missing += key not in A.at or key not in B.at
            if kind == "add":
                ref, bar = 0.3 * x - 1.1 * y, BAR * max(A.scale, B.scale)
            else:
                ref = 0.7 * modes(PF, modes(MV, x) * modes(MV, y)) * 2.0 ** (1.5 * (-2 + key[0] + 1))
                bar = 1e-11 * out.scale
            assert np.abs(ref - out.coef[i]).max() <= bar
        assert missing > 8


@pytest.mark.parametrize("order", range(3, 12))
def test_one_output_node_of_an_apply(gpu_mod, order):
    """a leaf of depth 1: its own contributions and the child's part of its root's, summed over every term and every input
    node of the two levels.  The operator's and the apply's screening lie four digits below the bar."""
    G = gpu_mod
    k = order + 1
    m = G.MultiResolutionAnalysis(*WORLD, order, 1)
    F = m.filter()
    f, out = G.FunctionTree(m), G.FunctionTree(m)
    G.project(1e-3, f, G.gauss_params([1.0], [1.5], [(1.4, 1.2, 1.6)]))
    op = G.HelmholtzOperator(m, 8.0, 1e-10)
    beta = op.terms()[1]
    G.apply(1e-15, out, op, f)
    A, O = Tree(f), Tree(out)
    node = (1, 5, 5, 5)  # the upper child of the box that holds the Gaussian's centre
    kinds = set()

    def contribution(key, root):
        depth, x = key[0], key[1:]
        n, ext = -2 + depth, 4 << depth
        blocks = {}
        total = np.zeros((2 * k,) * 3)
        for t in range(len(beta)):
            L = op.band(t, n)
            if L < 0:
                continue
            M = {l: op.ns_matrix(t, n, l) for l in range(-L, L + 1)}
            near = [[s for s in range(ext) if abs(x[e] - s) <= L] for e in range(3)]
            for sz in near[2]:
                plane, low = 0.0, 0.0
                for sy in near[1]:
                    line, lown = 0.0, 0.0
                    for sx in near[0]:
                        if (sx, sy, sz) not in blocks:
                            kinds.add((root, (depth, sx, sy, sz) in A.at))
                            blocks[sx, sy, sz] = A.block((depth, sx, sy, sz), F)
                        X, Mx = blocks[sx, sy, sz], M[x[0] - sx]
                        line = line + X @ Mx.T
                        lown = lown + X[:k, :k, :k] @ Mx[:k, :k].T
                    My = M[x[1] - sy]
                    plane = plane + np.matmul(My, line)
                    low = low + np.matmul(My[:k, :k], lown)
                Mz = M[x[2] - sz]
                total += beta[t] * np.einsum("cz,zyx->cyx", Mz, plane)
                if not root:
                    total[:k, :k, :k] -= beta[t] * np.einsum("cz,zyx->cyx", Mz[:k, :k], low)
        return total

    root = contribution((0, *(q >> 1 for q in node[1:])), True)
    ref = contribution(node, False)
    s = modes(F.T, root)
    ref[:k, :k, :k] += s[tuple(slice((q & 1) * k, (q & 1) * k + k) for q in reversed(node[1:]))]
    assert kinds == {(True, True), (False, True), (False, False)}
    assert np.abs(ref - O.coef[O.at[node]]).max() <= BAR * np.abs(root).max()
    check_compressed(O, F)
