"""Timed cases of the multiwavelet framework: what a quantum-chemistry program built on it calls.

A case is a dict of plain values.  ``prepare`` makes what the program already holds (function trees on
the device, operators), ``run`` is one pass through the public entry points and returns whole outputs:
node keys and coefficient blocks of every output tree as views of the library's device arrays, or the
number a call returns.  ``exact`` restates projection, products, sums and inner products with plain
torch in 64 bits.

Kinds of work:
  apply     out_i = O_i f_i with Poisson (mu = 0) or Helmholtz operators, one batch (config 1, 2, 4)
  scf       the same with the Helmholtz operators made inside the pass: the energies, so the exponents
            mu, are new in every iteration of a self-consistent-field solver
  multiply  adaptive pair products of orbitals (exchange)
  add       linear combination of orbitals on their union grid (rotation of an orbital set)
  deriv     gradient of an orbital, three directions (momentum and kinetic energy)
  project   Gaussian sums onto adaptive trees (initial guess)
  dot       one overlap <a|b>
"""
import math

import numpy as np
import torch

from mrchem_b200 import mrcpp as mw

# [-20, 20]^3 as 10^3 boxes of edge 4, the world of every configuration and test
WORLD = dict(min_scale=-2, corner=(-5, -5, -5), boxes=(10, 10, 10))
MAX_DEPTH = 15
ENGINES = {"fp64": mw.APPLY_FP64, "fp32": mw.APPLY_FP32, "bf16x3": mw.APPLY_BF16X3}
POOL = 40 << 30  # device pool reserved once by the program, as bench.py does


def listed():
    return [
        # unit-test size: an overlap of two small functions; host latency and two launches
        dict(name="dot_order5", kind="dot", source="orbitals", molecule=1, order=5, prec=1e-3, n=2),
        # smallest apply (the smoke test's): launch and read-back latency
        dict(name="poisson_order5", kind="apply", source="charges", molecule=2,
            order=5, prec=1e-3, n=1, poisson=True, engine="fp64"),
        # Poisson potential of three charges, order 7, prec 1e-5: one ordinary call, the default engine
        dict(name="poisson_order7", kind="apply", source="charges", molecule=3,
            order=7, prec=1e-5, n=1, poisson=True, engine="fp64"),
        # batch of Helmholtz applies in the default engine, half the benchmark's batch
        dict(name="helmholtz16_fp64", kind="apply", source="orbitals", molecule=4,
            order=9, prec=1e-6, n=16, poisson=False, engine="fp64"),
        # the benchmark's batch: 32 orbitals, mixed precision with the tensor-core x step
        dict(name="helmholtz32_bf16x3", kind="apply", source="orbitals", molecule=5,
            order=9, prec=1e-6, n=32, poisson=False, engine="bf16x3"),
        # potential of a 20-atom density at order 9, FP32 products
        dict(name="density_order9_fp32", kind="apply", source="density", molecule=6,
            order=9, prec=1e-6, n=1, poisson=True, engine="fp32"),
        # the same at order 11 in the default engine (largest basis of the density sweep)
        dict(name="density_order11_fp64", kind="apply", source="density", molecule=7,
            order=11, prec=1e-5, n=1, poisson=True, engine="fp64"),
        # one solver iteration of a small molecule: new operators, then the batch
        dict(name="scf4_order7", kind="scf", source="orbitals", molecule=8,
            order=7, prec=1e-5, n=4, poisson=False, engine="fp64"),
        # 28 exchange pair products of 7 orbitals
        dict(name="products28_order9", kind="multiply", source="orbitals", molecule=9, order=9, prec=1e-6, n=7),
        # one rotated orbital of a set of 8, on the union grid
        dict(name="sum8_order9", kind="add", source="orbitals", molecule=10, order=9, prec=1e-6, n=8),
        # gradient of one orbital
        dict(name="gradient_order9", kind="deriv", source="orbitals", molecule=11, order=9, prec=1e-6, n=1),
        # initial guess: 6 Gaussian-sum orbitals
        dict(name="project6_order9", kind="project", source="orbitals", molecule=12, order=9, prec=1e-6, n=6),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["apply", "apply", "apply", "scf", "multiply", "add", "deriv", "project", "dot"])
    order = rng.choice([4, 5, 6, 7, 8, 9, 9, 10])
    prec = 10.0 ** -rng.uniform(2.5, {4: 3.5, 5: 4.5, 6: 5.0, 7: 5.5}.get(order, 6.0))
    case = dict(kind=kind, source="orbitals", molecule=rng.randrange(1, 10 ** 6), order=order, prec=float("%.3g" % prec))
    if kind == "apply":
        case["source"] = rng.choice(["orbitals", "orbitals", "charges", "density"])
        case["n"] = _log_int(rng, 1, 16) if case["source"] == "orbitals" and order < 10 else 1
        case["poisson"] = case["source"] != "orbitals" or rng.random() < 0.3
        case["engine"] = rng.choice(["fp64", "fp64", "fp32", "bf16x3"])
    elif kind == "scf":
        case.update(n=_log_int(rng, 1, 4), poisson=False, engine=rng.choice(["fp64", "bf16x3"]))
    else:
        case["n"] = {"multiply": rng.randint(2, 7), "add": _log_int(rng, 2, 16), "deriv": 1,
                     "project": rng.randint(1, 6), "dot": 2}[kind]
    return case


# ---------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------
def _functions(case, seed):
    """(coefficients, exponents, centres) per input function, as the configurations draw them.  The
    case's molecule fixes positions and exponents relative to the molecular frame; the seed its orientation (one
    of the 48 of the cubic world) and the amplitudes, so that inputs of another seed are other functions
    on trees of the same size."""
    rng, pose = np.random.default_rng(case["molecule"]), np.random.default_rng(seed)
    axes, mirror = pose.permutation(3), pose.choice([-1.0, 1.0], 3)
    turn = lambda r: r[:, axes] * mirror
    size = lambda: pose.uniform(0.5, 2.0)
    if case["source"] == "charges":  # three unit charges in [-2, 2]^3
        a = rng.uniform(1.0, 50.0, 3)
        return [(size() * (a / np.pi) ** 1.5, a, turn(rng.uniform(-2.0, 2.0, (3, 3))))]
    if case["source"] == "density":  # 20 atoms in a 12 Bohr box, four unit charges each
        sites = np.repeat(rng.uniform(-6.0, 6.0, (20, 3)), 4, axis=0)
        a = np.exp(rng.uniform(np.log(0.3), np.log(1e3), 80))
        return [(size() * (a / np.pi) ** 1.5, a, turn(sites))]
    # orbitals: 2 to 6 Gaussians on 8 atoms, the first one a valence tail; pairs that are multiplied or
    # overlapped are those of neighbouring atoms (a program screens the others: their product is rounding)
    near = case["kind"] in ("multiply", "dot")
    half = 1.5 if near else 3.0
    sites = rng.uniform(-half, half, (8, 3))
    out = []
    for _ in range(case["n"]):
        ng = int(rng.integers(2, 7))
        a = np.exp(rng.uniform(np.log(0.5), np.log(200.0), ng))
        if near:
            a[0] = rng.uniform(0.5, 1.0)
        r = sites[rng.integers(0, 8, ng)]
        c = rng.uniform(0.5, 1.5, ng)
        d2 = ((r[:, None] - r[None]) ** 2).sum(-1)
        p = a[:, None] + a[None]
        s = (np.pi / p) ** 1.5 * np.exp(-a[:, None] * a[None] / p * d2)
        out.append((size() * c / np.sqrt(c @ s @ c), a, turn(r)))
    return out


def _exponents(case):
    """Helmholtz exponents of the batch"""
    return np.random.default_rng(case["molecule"] + 1000).uniform(0.5, 3.0, case["n"])


def _weights(case, seed):
    """coefficients of a linear combination (a row of a rotation)"""
    w = np.random.default_rng(seed + 2000).normal(size=case["n"])
    return w / np.linalg.norm(w)


def _pairs(n):
    return [(i, j) for i in range(n) for j in range(i, n)]


_reserved = []


def prepare(case, seed):
    ctx = mw.Context.default()
    if not _reserved:
        ctx.reserve(POOL)
        _reserved.append(True)
    mra = mw.MultiResolutionAnalysis(WORLD["min_scale"], WORLD["corner"], WORLD["boxes"], case["order"], MAX_DEPTH, ctx=ctx)
    kind = case["kind"]
    fs = [mw.gauss_params(c, a, r) for c, a, r in _functions(case, seed)]
    st = dict(case=case, mra=mra, prec=case["prec"], funcs=fs)
    n_out = {"multiply": len(_pairs(case["n"])), "add": 1, "deriv": 3, "dot": 0}.get(kind, len(fs))
    st["out"] = [mw.FunctionTree(mra) for _ in range(n_out)]
    if kind == "project":
        return st
    st["inp"] = [mw.FunctionTree(mra) for _ in fs]
    for t, f in zip(st["inp"], fs):
        mw.project(case["prec"], t, f)
    if kind in ("apply", "scf"):
        st["flags"] = ENGINES[case["engine"]]
        st["mus"] = [float(m) for m in _exponents(case)]
        if kind == "apply":
            st["ops"] = ([mw.PoissonOperator(mra, case["prec"])] * len(fs) if case["poisson"] else
                         [mw.HelmholtzOperator(mra, m, case["prec"]) for m in st["mus"]])
    elif kind == "add":
        st["weights"] = _weights(case, seed)
    elif kind == "deriv":
        st["op"] = mw.ABGVOperator(mra, 0.5, 0.5)
    return st


class _Array:
    """A device array of a tree for torch (CUDA array interface); keeps the tree alive."""

    def __init__(self, tree, ptr, shape, typestr):
        self.tree = tree
        self.__cuda_array_interface__ = dict(shape=shape, typestr=typestr, data=(ptr, False), version=3, strides=None)


def _view(tree):
    """(node keys, coefficient blocks) of a tree, no copy"""
    n, bs = tree.nnodes(), (2 * tree.mra.k) ** 3
    coef, key, _ = tree.device_arrays()
    return (torch.as_tensor(_Array(tree, key, (n,), "<i8"), device="cuda"),
            torch.as_tensor(_Array(tree, coef, (n, bs), "<f8"), device="cuda"))


def run(state):
    kind, prec, out = state["case"]["kind"], state["prec"], state["out"]
    inp = state.get("inp")
    if kind == "dot":
        return mw.dot(inp[0], inp[1])
    if kind == "apply":
        mw.apply_batched(prec, out, state["ops"], inp, state["flags"])
    elif kind == "scf":
        ops = [mw.HelmholtzOperator(state["mra"], mu, prec) for mu in state["mus"]]
        mw.apply_batched(prec, out, ops, inp, state["flags"])
        for t in out:
            t.rescale(-0.5 / math.pi)
    elif kind == "multiply":
        for t in out:
            mw.clear(t)
        pairs = _pairs(len(inp))
        mw.multiply_batched(prec, out, None, [inp[i] for i, _ in pairs], [inp[j] for _, j in pairs])
    elif kind == "add":
        mw.clear(out[0])
        for t in inp:
            mw.build_grid(out[0], t)
        mw.add(-1.0, out[0], state["weights"], inp)
    elif kind == "deriv":
        for d in range(3):
            mw.apply_derivative(out[d], state["op"], inp[0], d)
    elif kind == "project":
        for t, f in zip(out, state["funcs"]):
            mw.project(prec, t, f)
    return [_view(t) for t in out]


# ---------------------------------------------------------------------------------------------------
# work: blocks read and written once, and the operations of the method
# ---------------------------------------------------------------------------------------------------
def _nodes(case):
    """Nodes of one projected function: the root boxes, and refined ones (fitted to measured trees)."""
    digits, k = -math.log10(case["prec"]), case["order"] + 1
    share = {"charges": 0.13, "density": 1.0}.get(case["source"], 0.11)
    return 1000 + share * 4200 * (8.0 / k) ** 1.85 * 1.8 ** (digits - 5)


def _triples(case):
    """(output node, input node, Gaussian term) contributions above the screening, per apply (fitted)."""
    digits = -math.log10(case["prec"])
    if case["source"] == "density":
        return 1.2e6 * 10 ** (0.235 * (digits - 5))
    if case["source"] == "charges":
        return 6.7e4 * 10 ** (0.224 * (digits - 3))
    return 3.9e4 * 10 ** (0.095 * (digits - 5))


def work(case):
    k, n = case["order"] + 1, case["n"]
    block, mode = 8.0 * (2 * k) ** 3, 2.0 * (2 * k) ** 4  # bytes of a node block, flops of a mode product
    nodes = _nodes(case)
    kind = case["kind"]
    if kind == "dot":
        return dict(bytes=2 * block * nodes, flops=2 * (2 * k) ** 3 * nodes)
    if kind == "project":
        return dict(bytes=n * block * nodes, flops=n * 3 * mode * nodes)
    if kind == "multiply":
        m = len(_pairs(n))
        return dict(bytes=block * nodes * (n + m), flops=9 * mode * nodes * m)
    if kind == "add":
        return dict(bytes=block * nodes * (n + 1), flops=2.0 * (2 * k) ** 3 * nodes * n)
    if kind == "deriv":  # offsets -1, 0, 1 along one direction
        return dict(bytes=4 * block * nodes, flops=3 * 3 * mode * nodes)
    # applies: summed along lines and planes, a triple costs about 1.9 of its 3 mode products
    return dict(bytes=2 * n * block * nodes, flops=n * _triples(case) * 1.9 * mode)


# ---------------------------------------------------------------------------------------------------
# 64-bit restatement of projection, product, sum and inner product in plain torch
# ---------------------------------------------------------------------------------------------------
class _Basis:
    """Interpolating scaling functions of order k - 1 on [0, 1], their two-scale filter and quadrature."""

    def __init__(self, k, dev):
        x, w = np.polynomial.legendre.leggauss(k)
        self.x, w = 0.5 * (x + 1.0), 0.5 * w
        norm = np.sqrt(2.0 * np.arange(k) + 1.0)

        def values(t):  # [len(t), k]
            leg = lambda u: np.polynomial.legendre.legvander(2.0 * np.asarray(u) - 1.0, k - 1) * norm
            return leg(t) @ leg(self.x).T * np.sqrt(w)

        gx, gw = np.polynomial.legendre.leggauss(2 * k)
        gx, gw = 0.5 * (gx + 1.0), 0.5 * gw
        F = np.zeros((2 * k, 2 * k))
        for c in (0, 1):
            F[:k, c * k:(c + 1) * k] = values(0.5 * (gx + c)).T @ (gw[:, None] * values(gx)) / np.sqrt(2.0)
        for j in range(k):  # wavelets: orthonormal complement from the antisymmetric pairs
            v = np.zeros(2 * k)
            v[j], v[k + j] = 1.0 / np.sqrt(2.0), -1.0 / np.sqrt(2.0)
            for _ in range(2):
                for r in range(k + j):
                    v = v - (F[r] @ v) * F[r]
            F[k + j] = v / np.linalg.norm(v)
        two = lambda a: np.kron(np.eye(2), a)
        put = lambda a: torch.tensor(a, dtype=torch.float64, device=dev)
        self.k, self.F = k, put(F)
        self.PF = put(F @ two((w[:, None] * values(self.x)).T))  # point values on the children -> block
        self.MV = put(two(values(self.x)) @ F.T)  # block -> point values on the children


def _modes(M, A):
    """M applied along the three dimensions of blocks A[n, z, y, x]"""
    return torch.einsum("ax,nzyx->nzya", M, torch.einsum("by,nzyx->nzbx", M, torch.einsum("cz,nzyx->ncyx", M, A)))


def _morton(t):
    m = torch.zeros(len(t), dtype=torch.int64, device=t.device)
    for b in range(19):
        for d in range(3):
            m |= ((t[:, d] >> b) & 1) << (3 * b + d)
    return m


class _Tree:
    """Levels of (translations [n, 3], blocks [n, 2k, 2k, 2k]) in Morton order"""

    def __init__(self, basis):
        self.b, self.t, self.c, self.split = basis, [], [], []

    def grow(self, prec, block):
        """Adaptive construction from `block(depth, translations)`, refined while a node's wavelet norm
        exceeds prec ||f|| 2^(-depth/2), then compressed bottom-up."""
        k, dev = self.b.k, self.b.F.device
        g = [torch.arange(n, device=dev) for n in WORLD["boxes"]]
        t = torch.stack([a.reshape(-1) for a in torch.meshgrid(*g, indexing="ij")], 1)
        t = t[torch.argsort(_morton(t))]
        leaves = torch.zeros((), dtype=torch.float64, device=dev)
        while len(t):
            d = len(self.t)
            c = block(d, t)
            n2 = c.square().sum((1, 2, 3))
            wav = c.clone()
            wav[:, :k, :k, :k] = 0.0
            w2 = wav.square().sum((1, 2, 3))
            leaves = leaves + n2.sum()
            s = torch.nonzero(w2.sqrt() > prec * leaves.sqrt() * 2.0 ** (-0.5 * d)).flatten()
            leaves = leaves - n2[s].sum()
            self.t.append(t)
            self.c.append(c)
            self.split.append(s)
            off = torch.tensor([[q & 1, (q >> 1) & 1, q >> 2] for q in range(8)], device=dev)
            t = (2 * t[s][:, None] + off).reshape(-1, 3)
        return self.compress()

    def compress(self):
        k = self.b.k
        for d in range(len(self.t) - 2, -1, -1):
            s = self.split[d]
            ch = self.c[d + 1][:, :k, :k, :k].reshape(len(s), 2, 2, 2, k, k, k)
            ch = ch.permute(0, 1, 4, 2, 5, 3, 6).reshape(len(s), 2 * k, 2 * k, 2 * k)
            self.c[d][s] = _modes(self.b.F, ch)
        return self

    def on(self, depth, t, parents):
        """Blocks at nodes t of a depth: the tree's own, or scaling blocks generated from the parents' blocks"""
        k = self.b.k
        out = torch.zeros((len(t), 2 * k, 2 * k, 2 * k), dtype=torch.float64, device=t.device)
        own = torch.zeros(len(t), dtype=torch.bool, device=t.device)
        if depth < len(self.t):
            have, want = _morton(self.t[depth]), _morton(t)
            i = torch.searchsorted(have, want).clamp(max=len(have) - 1)
            own = have[i] == want
            out[own] = self.c[depth][i[own]]
        if not bool(own.all()):
            par_t, par_c = parents
            miss = torch.nonzero(~own).flatten()
            i = torch.searchsorted(_morton(par_t), _morton(t[miss] >> 1))
            r = _modes(self.b.F.T.contiguous(), par_c[i]).reshape(len(miss), 2, k, 2, k, 2, k)
            bit = t[miss] & 1
            out[miss, :k, :k, :k] = r[torch.arange(len(miss), device=t.device), bit[:, 2], :, bit[:, 1], :, bit[:, 0], :]
        return out

    def outputs(self):
        keys = torch.cat([_morton(t) | (d << 59) for d, t in enumerate(self.t)])
        return keys, torch.cat(self.c).reshape(len(keys), -1)


def _project(basis, prec, func):
    dev, k = basis.F.device, basis.k
    c, a, r = (torch.tensor(np.asarray(v), dtype=torch.float64, device=dev) for v in func)
    q = torch.tensor(np.concatenate([basis.x, basis.x + 1.0]), dtype=torch.float64, device=dev)
    lo = torch.tensor([v * 2.0 ** -WORLD["min_scale"] for v in WORLD["corner"]], dtype=torch.float64, device=dev)

    def block(d, t):
        h = 2.0 ** -(WORLD["min_scale"] + d + 1)
        p = lo[None, :, None] + (2 * t[:, :, None] + q) * h  # [n, 3, 2k]
        e = [torch.exp(-a[None, :, None] * (p[:, None, i] - r[None, :, i, None]).square()) for i in range(3)]
        v = torch.einsum("g,ngz,ngy,ngx->nzyx", c, e[2], e[1], e[0])
        return _modes(basis.PF, v) * 2.0 ** (-1.5 * (WORLD["min_scale"] + d + 1))

    return _Tree(basis).grow(prec, block)


def _combine(basis, prec, fs, weights):
    """sum_i w_i f_i on the union grid"""
    out, prev = _Tree(basis), [None] * len(fs)
    for d in range(max(len(f.t) for f in fs)):
        t = torch.unique(torch.cat([f.t[d] for f in fs if d < len(f.t)]), dim=0)
        t = t[torch.argsort(_morton(t))]
        blocks = [f.on(d, t, p) for f, p in zip(fs, prev)]
        prev = [(t, b) for b in blocks]
        out.t.append(t)
        out.c.append(sum(w * b for w, b in zip(weights, blocks)))
    for d in range(len(out.t) - 1):
        have = _morton(out.t[d])
        out.split.append(torch.searchsorted(have, _morton(out.t[d + 1][::8] >> 1)))
    return out.compress()


def _product(basis, prec, a, b):
    last = {}

    def block(d, t):
        blocks = [f.on(d, t, last.get(i)) for i, f in enumerate((a, b))]
        last.update({i: (t, c) for i, c in enumerate(blocks)})
        v = _modes(basis.MV, blocks[0]) * _modes(basis.MV, blocks[1])
        return _modes(basis.PF, v) * 2.0 ** (1.5 * (WORLD["min_scale"] + d + 1))

    return _Tree(basis).grow(prec, block)


def _dot(a, b):
    k, s = a.b.k, 0.0
    for d in range(min(len(a.t), len(b.t))):
        ha, hb = _morton(a.t[d]), _morton(b.t[d])
        i = torch.searchsorted(hb, ha).clamp(max=len(hb) - 1)
        m = hb[i] == ha
        p = a.c[d][m] * b.c[d][i[m]]
        if d > 0:
            p[:, :k, :k, :k] = 0.0
        s += float(p.sum())
    return s


def exact(case, seed):
    if case["kind"] in ("apply", "scf", "deriv"):
        return None  # operator tables and the adaptive apply: minutes in plain torch
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    basis, prec = _Basis(case["order"] + 1, dev), case["prec"]
    fs = [_project(basis, prec, f) for f in _functions(case, seed)]
    if case["kind"] == "dot":
        return _dot(fs[0], fs[1])
    if case["kind"] == "project":
        return [f.outputs() for f in fs]
    if case["kind"] == "add":
        return [_combine(basis, prec, fs, _weights(case, seed)).outputs()]
    return [_product(basis, prec, fs[i], fs[j]).outputs() for i, j in _pairs(case["n"])]
