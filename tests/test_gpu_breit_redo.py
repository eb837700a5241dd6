"""Breit tables evaluated term by term (an orbital too short for the
contraction). One with more entries than one launch of k_br_redo takes (524,288):
the pieces meet without a gap. Bar: 1e-13 of the table's largest value, the
tables' own (each value is the reference's sum up to the rounding of log, sin
and cos)."""
import numpy as np
import pytest

from inputs import synth as S
from tests.common import oracle_for

pytestmark = pytest.mark.gpu


def test_term_by_term_table_in_pieces(gpu_ready, oracle_mod):
    from grasp_gb300 import Context
    orbs, n, z = S.orbital_set(6, 3), 590, 26.0
    rnt, r = S.grid(n, z)
    ob = S.hydrogenic_orbitals(orbs, z, S.screenpar([k for _, k in orbs], 1), r, n=n)
    ob.mf[1] = 9
    ob.pf[1, 9:] = 0.0
    ob.qf[1, 9:] = 0.0
    case = dict(n=n, rnt=rnt, h=0.05, c=S.CVAC, zz=np.full(n, z), orb=ob)
    e = -np.linspace(50.0, 1.0, len(ob.nak))
    o = oracle_for(case)
    ctx = Context(0)
    ctx.set_grid(n, rnt, 0.05, S.CVAC, case["zz"])
    ctx.set_orbitals(ob.nak, ob.mf, ob.pf, ob.qf)
    ind, val, kst, _ = ctx.genintbreit(1, 1.0, e)
    assert len(ind) > 1 << 19
    ind0, val0, kst0, _ = o.genintbreit(1, 1.0, e, nthreads=16)
    np.testing.assert_array_equal(ind, ind0)
    np.testing.assert_array_equal(kst, kst0)
    assert np.abs(val - val0).max() <= 1e-13 * np.abs(val0).max()


def test_two_terms_take_two_threads(gpu_ready):
    """A type 2 table without a frequency has two terms per integral where one
    with frequencies has three or four: it takes about half the kernels' time
    (0.37 measured; 0.71 with idle threads for the terms it does not have)."""
    from grasp_gb300 import Context
    orbs, n, z = S.orbital_set(5, 3), 590, 26.0
    rnt, r = S.grid(n, z)
    ob = S.hydrogenic_orbitals(orbs, z, S.screenpar([k for _, k in orbs], 1), r, n=n)
    ob.mf[1] = 9
    ob.pf[1, 9:] = 0.0
    ob.qf[1, 9:] = 0.0
    ctx = Context(0)
    ctx.set_grid(n, rnt, 0.05, S.CVAC, np.full(n, z))
    ctx.set_orbitals(ob.nak, ob.mf, ob.pf, ob.qf)
    e = -np.linspace(50.0, 1.0, len(ob.nak))

    def kernels(wfact):
        ms = []
        for _ in range(4):
            ctx.genintbreit(2, wfact, e)
            ms.append(ctx.stage_stat(33))
        return min(ms)

    assert kernels(0.0) < 0.55 * kernels(1.0)
