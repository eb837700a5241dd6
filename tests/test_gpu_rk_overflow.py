"""The R^k table where QUAD's integrands leave the range of a double: the head
index is the reference's (quad.f90: TA(i) != 0 and not TA(i+1)/TA(i) <= 0), so
an entry is not a number where the oracle's is, a point whose ratio to the
next underflows or is infinite is no head where it is none for the oracle, and
the other entries are the usual ones. Bar: test_gpu_radial's, 1e-12 of the
value or 1e-14 of the table's usual size."""
import numpy as np
import pytest

from tests.common import hydrogenic_case, oracle_for

pytestmark = pytest.mark.gpu


def _large(ob):
    ob.pf[2] *= 1e100
    ob.qf[2] *= 1e100
    ob.pf[5] *= 1e-100
    ob.qf[5] *= 1e-100


def _larger(ob):
    ob.pf[2] *= 1e140
    ob.qf[2] *= 1e140
    ob.pf[5] *= 1e-140
    ob.qf[5] *= 1e-140


def _first_point(p0, p1):
    def change(ob):  # zero up to a point, then p0, p1 and the orbital as it was
        ob.pf[1, :40] = 0.0
        ob.qf[1, :40] = 0.0
        ob.pf[1, 40:42] = p0, p1
        ob.qf[1, 40:42] = 0.0
    return change


def _not_a_number(ob):
    ob.pf[1, 30] = np.nan


CASES = {"large": _large, "larger": _larger, "infinite_first": _first_point(1e160, 1e-3),
         "underflow": _first_point(1e3, 3e-160), "nan": _not_a_number}


@pytest.mark.parametrize("which", sorted(CASES))
def test_entries_out_of_range(gpu_ready, oracle_mod, which):
    from grasp_gb300 import Context
    case = hydrogenic_case(nmax=4, lmax=3, z=26.0)
    ob = case["orb"]
    usual = np.abs(oracle_for(case).genintrk(nthreads=8)[1]).max()
    CASES[which](ob)
    ctx = Context(0)
    ctx.set_grid(case["n"], case["rnt"], case["h"], case["c"], case["zz"])
    ctx.set_orbitals(ob.nak, ob.mf, ob.pf, ob.qf)
    ctx.genintrk()
    ind, val, _ = ctx.rk_table()
    ind0, val0, _, _ = oracle_for(case).genintrk(nthreads=8)
    np.testing.assert_array_equal(ind, ind0)
    np.testing.assert_array_equal(np.isnan(val), np.isnan(val0))
    inf = np.isinf(val0)
    np.testing.assert_array_equal(val[inf], val0[inf])
    fin = np.isfinite(val0)
    assert (np.abs(val[fin] - val0[fin]) <= 1e-12 * np.abs(val0[fin]) + 1e-14 * usual).all()
