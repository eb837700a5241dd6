"""RINTI, the I(ab) table, SETLAG and SLATER on grids around the lengths where
their working arrays leave shared memory (k_rinti above 1,174 points,
k_setlag_quad above 24,024, k_quad_items above 5,990), against the oracle.

Bars: a RINTI runs the oracle's operations in their order up to QUAD's log, so
1e-12 of the table's largest value holds with room for the cancellation of its
four integrals; the multipliers' bar is test_setlag_matches_oracle's; a SLATER
runs the oracle's operations in their order up to QUAD's log: 1e-14."""
import numpy as np
import pytest

from tests.test_gpu_potential_functions import KEY, _lists, _setup

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [590, 1174, 1175, 1198, 1199, 1283, 2561, 24024, 24025, 24537])
def test_one_electron_integrals_and_multipliers(gpu_ready, oracle_mod, n):
    o, ctx, nw = _setup(n, 23.6 / n)
    nak = [-1, -1, 1, -2, 2, -3, -1, 1]
    pairs = [(a, b) for b in range(1, nw + 1) for a in range(1, nw + 1) if nak[a - 1] == nak[b - 1]]
    iab = ctx.iabint_table()
    ref = np.array([o.rinti(a, b) for a, b in pairs])
    got = np.array([iab[a - 1, b - 1] for a, b in pairs])
    assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
    assert ctx.rinti(*pairs[1]) == got[1]
    cofs = []
    for j in range(nw):
        nya, nxa, co = _lists(nw, 60, 6, j + 1)
        cofs.append(dict(nya=nya, ya=co, nxa=nxa, xa=co, nda=np.array([1 + j % nw], np.int32), da=np.array([0.1])))
    iecc = np.array([a + KEY * b for a, b in pairs if a < b], np.int32)
    for fixed, spread in ((1, 1.0), (0, 1.0), (0, 0.01)):  # every case of SETLAG's
        ucf = 1.0 + spread * np.arange(nw)
        lfix = np.zeros(nw, np.int32)
        lfix[[1, 2]] = fixed
        ecv, ecv0 = ctx.setlag(iecc, ucf, lfix, cofs), o.setlag(iecc, ucf, lfix, cofs)
        assert np.abs(ecv - ecv0).max() <= 1e-12 * max(1.0, np.abs(ecv0).max())


@pytest.mark.parametrize("n", [590, 5990, 5991, 24537])
def test_slater(gpu_ready, oracle_mod, n):
    o, ctx, _ = _setup(n, 23.6 / n)
    for a, b, c, d, k in [(1, 2, 1, 2, 0), (3, 8, 8, 3, 0), (2, 4, 7, 5, 1), (6, 6, 6, 6, 2), (8, 7, 8, 7, 0)]:
        v, v0 = ctx.slater(a, b, c, d, k), o.slater(a, b, c, d, k)
        assert abs(v - v0) <= 1e-14 * abs(v0), (a, b, c, d, k)
