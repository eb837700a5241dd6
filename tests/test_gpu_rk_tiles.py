"""GPU parity: the R^k contractions (gg_genintrk) at the sizes where their
tilings change: the FP64 form's tiles of 8, 4, 2 or 1 rows, the tensor-core
form's tiles split over the grid (fewer tiles than SMs), one per SM and several
in turn; odd and even grids, orbitals that end on the last grid point or
within the first few.

Bar: 1e-12 of the largest |R^k| (tests/test_gpu_radial.py): against the oracle
for the small sets, between the two forms for the large ones.
"""
import numpy as np
import pytest

from inputs import synth as S

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _case(nmax, lmax, n, z=18.0):
    orbs = S.orbital_set(nmax, lmax)
    rnt, r = S.grid(n, z)
    ob = S.hydrogenic_orbitals(orbs, z, S.screenpar([k for _, k in orbs], 1), r, n=n)
    return dict(n=n, rnt=rnt, h=0.05, c=S.CVAC, zz=np.full(n, z), orb=ob)


def _context(case):
    from grasp_gb300 import Context
    ctx = Context(0)
    ctx.set_grid(case["n"], case["rnt"], case["h"], case["c"], case["zz"])
    ob = case["orb"]
    ctx.set_orbitals(ob.nak, ob.mf, ob.pf, ob.qf)
    return ctx


@pytest.mark.parametrize("nmax,lmax,n", [(1, 0, 590), (2, 1, 401), (3, 1, 590), (3, 2, 513), (4, 3, 590)])
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("ends", ["as_is", "last_point", "short"])
def test_small_sets_match_oracle(gpu_ready, oracle_mod, nmax, lmax, n, precision, ends):
    from tests.common import oracle_for
    case = _case(nmax, lmax, n)
    if ends == "last_point":
        case["orb"].mf[0] = n
    elif ends == "short":
        case["orb"].mf[-1] = 24
    ctx = _context(case)
    ctx.genintrk(precision=precision)
    ind, val, kst = ctx.rk_table()
    ind0, val0, kst0, _ = oracle_for(case).genintrk()
    np.testing.assert_array_equal(ind, ind0)
    np.testing.assert_array_equal(kst, kst0)
    assert np.abs(val - val0).max() <= TOL * np.abs(val0).max()


@pytest.mark.parametrize("nmax,lmax,n,kmax", [(5, 4, 590, -1), (6, 4, 589, 5), (7, 3, 590, 8), (7, 4, 513, 8)])
def test_large_sets_agree(gpu_ready, nmax, lmax, n, kmax):
    case = _case(nmax, lmax, n)
    ctx = _context(case)
    ctx.genintrk(kmax, precision=0)
    ind, val, _ = ctx.rk_table()
    ctx.genintrk(kmax, precision=1)
    ind1, val1, _ = ctx.rk_table()
    np.testing.assert_array_equal(ind, ind1)
    assert np.abs(val - val1).max() <= TOL * np.abs(val).max()
    ctx.genintrk(kmax, precision=1)
    np.testing.assert_array_equal(ctx.rk_table()[1], val1)
