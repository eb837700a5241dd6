"""YPOT and XPOT over so many distinct Y functions that the call waits for
their number before it reserves memory for them (the bound, 8,400 functions
and the six arrays of their long build, passes 256 MB), and on a grid so long
that the call's buffers pass the 512 MB a context keeps: the buffers go back
and the next calls, a short one and the long one again, give the same bits.

Bar: 8,400 terms of either sign, each rounded to 1.1e-16 of its size, are off
by 9e-13 of the largest value at worst; 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEY = 215


def _setup(n, nw):
    from grasp_gb300 import Context
    import oracle
    h, rnt, z, c = 23.6 / n, 2e-7, 10.0, 137.035999139
    r, rp = rnt * np.expm1(h * np.arange(n)), rnt * np.exp(h * np.arange(n))
    nak = np.array([(-1, 1, -2, 2, -3)[j % 5] for j in range(nw)])
    mf = np.array([n - 1 - (n // 3) * j // nw for j in range(nw)])
    pf, qf = np.zeros((nw, n)), np.zeros((nw, n))
    for j in range(nw):
        l = nak[j] if nak[j] > 0 else -nak[j] - 1
        a = 12.0 / r[mf[j] - 1]  # fallen to e^-12 at its end
        p = r ** (l + 1) * np.exp(-a * r) * (1.0 - 0.3 * a * r)
        p /= np.sqrt(h * np.sum(p[:mf[j]] ** 2 * rp[:mf[j]]))
        pf[j, :mf[j]] = p[:mf[j]]
        qf[j, :mf[j]] = -0.01 * p[:mf[j]] * np.cos(a * r[:mf[j]])
    ctx, o = Context(0), oracle.Oracle(n=n, rnt=rnt, h=h, c=c, zz=np.full(n, z))
    ctx.set_grid(n, rnt, h, c, np.full(n, z))
    for t in (ctx, o):
        t.set_orbitals(nak, mf, pf, qf)
    return ctx, o


@pytest.mark.parametrize("n", [590, 2561])
def test_many_functions(gpu_ready, oracle_mod, n):
    nw = 20
    ctx, o = _setup(n, nw)
    rng = np.random.default_rng(n)
    k, a, b = (x.ravel() for x in np.meshgrid(np.arange(21), np.arange(1, nw + 1), np.arange(1, nw + 1)))
    p = rng.permutation(k.size)
    k, a, b = k[p], a[p], b[p]
    nya = ((b * KEY + a) * KEY + k).astype(np.int32)
    nxa = (((rng.integers(1, nw + 1, k.size) * KEY + b) * KEY + a) * KEY + k).astype(np.int32)
    co = rng.normal(size=k.size)
    y, x = ctx.ypot(nya, co), ctx.xpot(nxa, co)
    for got, ref in zip([y, *x], [o.ypot(nya, co), *o.xpot(nxa, co)]):
        assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
    few, ref = ctx.ypot(nya[:50], co[:50]), o.ypot(nya[:50], co[:50])
    assert np.abs(few - ref).max() <= 1e-12 * np.abs(ref).max()
    np.testing.assert_array_equal(ctx.ypot(nya, co), y)
    for got, first in zip(ctx.xpot(nxa, co), x):
        np.testing.assert_array_equal(got, first)
