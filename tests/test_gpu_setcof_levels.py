"""SETCOF's sums for numbers of levels around the 32 that a warp holds at a
time (k_dsubrs_pos), EOL and EAL, against the oracle: labels entry for entry,
values to 1e-14 of each list's largest (the label sums' own bar; the sums run
over at most a few hundred contributions, the diagonal ones over 120 CSFs)."""
import numpy as np
import pytest

from tests.common import hydrogenic_case, oracle_for
from tests.test_setcof_oracle import _blocks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nev", [1, 31, 32, 33, 65, 0])
def test_levels_match_oracle(gpu_ready, oracle_mod, nev):
    from grasp_gb300 import Context, HMatrix
    case = hydrogenic_case(nmax=4, lmax=3, z=10.0)
    o = oracle_for(case)
    ob = case["orb"]
    ctx = Context(0)
    ctx.set_grid(case["n"], case["rnt"], case["h"], case["c"], case["zz"])
    ctx.set_orbitals(ob.nak, ob.mf, ob.pf, ob.qf)
    ctx.genintrk()
    ctx.iabint_table()
    _, blocks = _blocks(two_js=(0, 2))
    rng = np.random.default_rng(nev)
    eol = nev > 0
    for b in blocks:
        b["wt"] = rng.uniform(0.1, 1.0, nev if eol else b["ncf"])
        if eol:
            b["evec"] = np.linalg.qr(rng.normal(size=(b["ncf"], nev)))[0]
    hs = []
    for b in blocks:
        h = HMatrix(ctx, b["ncf"], b["iendc"], b["irow"])
        h.setham_upload(b["iq"], b["tlist"], b["vlists"])
        hs.append(h)
    ctx.setcof_prepare(hs, [b["wt"] for b in blocks], [b["evec"] for b in blocks] if eol else None, eol=eol)
    for j in range(1, len(ob.nak) + 1):
        got, ref = ctx.setcof(j, 1.25), o.setcof(blocks, eol, j, 1.25)
        for key in ("nya", "nxa", "nda"):
            np.testing.assert_array_equal(got[key], ref[key])
        for key in ("ya", "xa", "da"):
            scale = max(1e-300, np.abs(ref[key]).max(initial=0.0))
            assert np.abs(got[key] - ref[key]).max(initial=0.0) <= 1e-14 * scale, (j, key)
