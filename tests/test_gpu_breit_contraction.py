"""GENINTBREIT1/2 by contraction (k_br_*) where its grouping can go wrong:
orbital sets whose ends coincide (one column bucket), lie one point apart or
far apart (the shared part of the vectors short or long, QUAD's last point on
every residue class), zero frequencies among others, a source whose chain
starts with zeros or changes sign (entries evaluated term by term), and an
orbital too short for the contraction (the whole table term by term), for
grids of both parities. Bar: 1e-13 of the table's largest value, the tables'
own (the sums differ from the oracle's in the order of some 400 FP64
additions, a few 1e-16 of the largest partial sum)."""
import numpy as np
import pytest

from inputs import synth as S
from tests.common import oracle_for

pytestmark = pytest.mark.gpu


def _ends(ob, e, ends):
    for j, m in ends.items():
        ob.mf[j] = m


SETS = {
    "as_is": lambda ob, e: None,
    "equal_ends": lambda ob, e: _ends(ob, e, {j: 300 for j in range(len(e))}),
    "adjacent_ends": lambda ob, e: _ends(ob, e, {j: 290 + j for j in range(len(e))}),
    "shortest_taken": lambda ob, e: _ends(ob, e, {0: 16, 3: 17, 4: 18, 5: 19}),
    "too_short": lambda ob, e: _ends(ob, e, {1: 9}),
    "zeros_at_the_start": lambda ob, e: (ob.pf[2].__setitem__(slice(0, 6), 0.0), ob.qf[2].__setitem__(slice(0, 6), 0.0)),
    "sign_change": lambda ob, e: ob.pf[3].__setitem__(2, -ob.pf[3][2]),
    "degenerate_energies": lambda ob, e: e.__setitem__(slice(1, 6), [e[3], e[2], e[3], e[4], e[4] + 1e-8]),
}


def _case(n, z=10.0):
    orbs = S.orbital_set(3, 2)
    rnt, r = S.grid(n, z)
    ob = S.hydrogenic_orbitals(orbs, z, S.screenpar([k for _, k in orbs], 1), r, n=n)
    return dict(n=n, rnt=rnt, h=0.05, c=S.CVAC, zz=np.full(n, z), orb=ob)


@pytest.mark.parametrize("n", [590, 513])
@pytest.mark.parametrize("wfact", [1.0, 0.0])
@pytest.mark.parametrize("itype", [1, 2])
@pytest.mark.parametrize("which", sorted(SETS))
def test_contraction_matches_oracle(gpu_ready, oracle_mod, which, itype, wfact, n):
    from grasp_gb300 import Context
    case = _case(n)
    ob = case["orb"]
    nw = len(ob.nak)
    e = -np.linspace(50.0, 1.0, nw)
    SETS[which](ob, e)
    for j in range(nw):
        ob.pf[j, ob.mf[j]:] = 0.0
        ob.qf[j, ob.mf[j]:] = 0.0
    o = oracle_for(case)
    ctx = Context(0)
    ctx.set_grid(case["n"], case["rnt"], case["h"], case["c"], case["zz"])
    ctx.set_orbitals(ob.nak, ob.mf, ob.pf, ob.qf)
    ind, val, kst, j2 = ctx.genintbreit(itype, wfact, e)
    ind0, val0, kst0, j20 = o.genintbreit(itype, wfact, e, nthreads=8)
    assert j2 == j20
    np.testing.assert_array_equal(ind, ind0)
    np.testing.assert_array_equal(kst, kst0)
    assert np.abs(val - val0).max() <= 1e-13 * np.abs(val0).max()
