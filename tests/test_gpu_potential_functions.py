"""GPU parity: the Y functions and term sums of YPOT and XPOT (gg_ypot,
gg_xpot) against the oracle at the sizes where their splits end: grids whose
chains fill one pass of the scan or need several, odd and even, and a grid too
long for the scan's shared memory; lists of one term, around a chunk, and of
many chunks.

Bar: a function is a sum of a few hundred products and a potential one of up
to 1,500 functions, each rounded to 1.1e-16 of its size, so 1e-13 of the
largest value holds with room (the sums' terms have either sign).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEY = 215


def _lists(nw, n, kmax, seed):
    r = np.random.default_rng(seed)
    k = r.integers(0, kmax + 1, n)
    a, b, io = (r.integers(1, nw + 1, n) for _ in range(3))
    return (((b * KEY + a) * KEY + k).astype(np.int32), (((io * KEY + b) * KEY + a) * KEY + k).astype(np.int32),
            r.normal(size=n))


def _setup(n, h):
    """Smooth two-component orbitals on n points of step h, ends from a dozen
    points to the whole grid, normalised by the grid's trapezoid sum."""
    from grasp_gb300 import Context
    import oracle
    rnt, z, c = 2e-7, 10.0, 137.035999139
    r = rnt * np.expm1(h * np.arange(n))
    rp = rnt * np.exp(h * np.arange(n))
    zz = np.full(n, z)
    nak = [-1, -1, 1, -2, 2, -3, -1, 1]
    mf = [n // 8 + 12, n // 2, n // 2 + 1, n // 2 + 2, n // 2 + 3, 3 * n // 4, n - 1, n]
    pf, qf = np.zeros((len(nak), n)), np.zeros((len(nak), n))
    for j, (k, m) in enumerate(zip(nak, mf)):
        l = k if k > 0 else -k - 1
        a = 12.0 / r[m - 1]  # fallen to e^-12 at its end
        p = r ** (l + 1) * np.exp(-a * r) * (1.0 - 0.3 * a * r)
        p /= np.sqrt(h * np.sum(p[:m] ** 2 * rp[:m]))
        pf[j, :m] = p[:m]
        qf[j, :m] = -0.01 * p[:m] * np.cos(a * r[:m])
    ctx, g = Context(0), oracle.Oracle(n=n, rnt=rnt, h=h, c=c, zz=zz)
    ctx.set_grid(n, rnt, h, c, zz)
    for t in (ctx, g):
        t.set_orbitals(np.array(nak), np.array(mf), pf, qf)
    return g, ctx, len(nak)


def _close(a, b):
    assert np.abs(a - b).max() <= 1e-13 * max(np.abs(b).max(), 1e-300), np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("n,h", [(120, 0.2), (481, 0.05), (590, 0.04), (636, 0.04), (641, 0.04), (1283, 0.02), (2560, 0.01), (2561, 0.01)])
def test_functions_by_grid(gpu_ready, oracle_mod, n, h):
    g, ctx, nw = _setup(n, h)
    nya, nxa, co = _lists(nw, 300, 6, n)
    _close(ctx.ypot(nya, co), g.ypot(nya, co))
    for x, x0 in zip(ctx.xpot(nxa, co), g.xpot(nxa, co)):
        _close(x, x0)


@pytest.mark.parametrize("terms", [0, 1, 3, 255, 256, 257, 511, 1500])
@pytest.mark.parametrize("orbs", [1, None])
def test_sums_by_terms(gpu_ready, oracle_mod, terms, orbs):
    """orbs = 1: every term on one orbital, one run per chunk."""
    g, ctx, nw = _setup(590, 0.04)
    nya, nxa, co = _lists(nw, terms, 6, terms + 1)
    if orbs:
        nxa = (nxa % KEY**3 + KEY**3 * orbs).astype(np.int32)
    _close(ctx.ypot(nya, co), g.ypot(nya, co))
    for x, x0 in zip(ctx.xpot(nxa, co), g.xpot(nxa, co)):
        _close(x, x0)
