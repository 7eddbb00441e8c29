"""The non-standard-form matrices that the contraction reads (device tables, mw_optab.cu) against quadrature in numpy that
shares no code with the library or the oracle: every order, both bases, terms from the widest to the narrowest of a depth,
offsets of every launch of the construction (0 .. 3, 4 .. 11, from 12 on), both signs, root and deeper scales.

Bar: 1e-12 times the scale's factor 2^-n, which bounds every entry of T^n (orthonormal scaling functions, kernel at most one).
The construction adds 2k products per entry three times, of magnitude at most sqrt(4k) each: 2k sqrt(4k) 2^-53, 4e-14 at
k = 12, and the exponential's argument, at most 40 where it counts, rounds to 1e-14."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LEGENDRE = 1


def values(x, k, basis):
    """scaling functions on [0, 1] at the points x, [len(x), k]"""
    norm = np.sqrt(2.0 * np.arange(k) + 1.0)
    leg = lambda t: np.polynomial.legendre.legvander(2.0 * t - 1.0, k - 1) * norm
    if basis == LEGENDRE:
        return leg(x)
    q, w = np.polynomial.legendre.leggauss(k)
    return leg(x) @ leg(0.5 * (q + 1.0)).T * np.sqrt(0.5 * w)


def edges(a, centre, lo, hi):
    """panel edges of [lo, hi], graded away from the point closest to the Gaussian's centre"""
    near = min(max(centre, lo), hi)
    dist = abs(centre - near)
    unit = 1.0 / np.sqrt(a) if dist == 0.0 else min(1.0 / np.sqrt(a), 0.5 / (a * dist))
    steps = unit * np.concatenate([[0.0], 0.5 * 2.0 ** np.arange(60)])
    e = np.concatenate([near - steps, near + steps, [lo, hi]])
    return np.unique(e[(e >= lo) & (e <= hi)])


def t_block(a, l, k, basis):
    """int int phi_i(u) phi_j(v) exp(-a (u - v + l)^2): over t = u - v outside, over u inside (exact for polynomials)"""
    gx, gw = np.polynomial.legendre.leggauss(40)
    ux, uw = np.polynomial.legendre.leggauss(k)
    T = np.zeros((k, k))
    for lo, hi in ((-1.0, 0.0), (0.0, 1.0)):
        e = edges(a, -float(l), lo, hi)
        for p, q in zip(e[:-1], e[1:]):
            t = p + 0.5 * (q - p) * (gx + 1.0)
            g = 0.5 * (q - p) * gw * np.exp(-a * (t + l) ** 2)
            if not g.any():
                continue
            u0, u1 = np.maximum(0.0, t), np.minimum(1.0, 1.0 + t)
            u = u0[:, None] + 0.5 * (u1 - u0)[:, None] * (ux + 1.0)
            w = g[:, None] * 0.5 * (u1 - u0)[:, None] * uw
            pu, pv = values(u.ravel(), k, basis), values((u - t[:, None]).ravel(), k, basis)
            T += (pu * w.ravel()[:, None]).T @ pv
    return T


def ns_reference(alpha, n, l, F, k, basis, cache):
    def T(d):
        if d not in cache:
            cache[d] = t_block(alpha * 4.0 ** -(n + 1), d, k, basis) * 2.0 ** -(n + 1)
        return cache[d]

    return F @ np.block([[T(2 * l), T(2 * l - 1)], [T(2 * l + 1), T(2 * l)]]) @ F.T


@pytest.mark.parametrize("order,basis", [(o, 0) for o in range(3, 12)] + [(5, LEGENDRE), (9, LEGENDRE)])
def test_tables_against_quadrature(gpu_mod, order, basis):
    G = gpu_mod
    k, n0 = order + 1, -2
    m = G.MultiResolutionAnalysis(n0, (-10, 0, 0), (20, 1, 1), order, 10, basis)
    op = G.PoissonOperator(m, 1e-3)
    F, alpha = m.filter(), op.terms()[0]
    seen, widest = set(), 0
    for depth in (0, 1, 3):
        n = n0 + depth
        band = np.array([op.band(t, n) for t in range(len(alpha))])
        active = np.flatnonzero(band >= 0)
        assert len(active) > 3
        by_width = active[np.argsort(band[active], kind="stable")]
        widest = max(widest, band.max())
        for t in {by_width[0], by_width[len(by_width) // 2], by_width[-1]}:
            L, cache = int(band[t]), {}
            for l in sorted({0, 1, -1, 3, 4, -5, 11, 12, -13, L, -L}):
                if abs(l) > L:
                    continue
                ref = ns_reference(alpha[t], n, l, F, k, basis, cache)
                assert np.abs(op.ns_matrix(t, n, l) - ref).max() < 1e-12 * 2.0 ** -n, (depth, t, l)
                seen.add(l)
    assert widest >= 19 and {0, 4, 12, -13, 19, -19} <= seen


def test_matrices_beyond_the_tables(gpu_mod):
    """offsets outside the band, scales outside the world and inactive terms are still answered"""
    G = gpu_mod
    order, k = 4, 5
    m = G.MultiResolutionAnalysis(-2, (-5, -5, -5), (10, 10, 10), order, 6)
    op = G.PoissonOperator(m, 1e-3)
    F, alpha = m.filter(), op.terms()[0]
    t = len(alpha) // 2
    L = op.band(t, 0)
    for n, l in ((0, L + 1), (0, -(L + 2)), (-4, 1), (9, 0)):
        ref = ns_reference(alpha[t], n, l, F, k, 0, {})
        assert np.abs(op.ns_matrix(t, n, l) - ref).max() < 1e-12 * 2.0 ** -n
    assert op.band(t, -4) == -1 and op.band(t, 9) == -1
    off = [q for q in range(len(alpha)) if op.band(q, 4) < 0]
    assert off
    for q in (off[0], off[-1]):
        assert np.abs(op.ns_matrix(q, 4, 0) - ns_reference(alpha[q], 4, 0, F, k, 0, {})).max() < 1e-12 * 2.0 ** -4
    wide = G.MultiResolutionAnalysis(-2, (-128, 0, 0), (256, 1, 1), 3, 6)  # lists too large to build
    op = G.PoissonOperator(wide, 1e-3)
    alpha = op.terms()[0]
    assert op.band(5, -2) == -1
    ref = ns_reference(alpha[5], -2, 3, wide.filter(), 4, 0, {})
    assert np.abs(op.ns_matrix(5, -2, 3) - ref).max() < 1e-12 * 4.0
