"""gg_setcof_prepare's pieces: the label sums of a block whose DSUBRS do not
fit the workspace are formed some positions at a time (k_dsubrs_pos<true>,
k_label_sums<true>). Pieces of one position, of a few, that cut rows, and one
short of the whole block, around the 32 levels a warp holds, EOL and EAL,
against the oracle: labels entry for entry, values to 1e-14 of each list's
largest (the label sums' own bar: a few hundred contributions)."""
import numpy as np
import pytest

from tests.common import hydrogenic_case, oracle_for
from tests.test_setcof_oracle import _blocks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nev", [2, 33, 0])
@pytest.mark.parametrize("positions", [1, 37, 1000, -1])
def test_pieces_match_oracle(gpu_ready, oracle_mod, positions, nev):
    from grasp_gb300 import Context, HMatrix, _lib
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
    hs = []
    for b in blocks:
        b["wt"] = rng.uniform(0.1, 1.0, nev if eol else b["ncf"])
        if eol:
            b["evec"] = np.linalg.qr(rng.normal(size=(b["ncf"], nev)))[0]
        h = HMatrix(ctx, b["ncf"], b["iendc"], b["irow"])
        h.setham_upload(b["iq"], b["tlist"], b["vlists"])
        hs.append(h)
    p = positions if positions > 0 else max(len(b["irow"]) for b in blocks) - 1
    args = (hs, [b["wt"] for b in blocks], [b["evec"] for b in blocks] if eol else None)

    def launches():
        n0 = _lib.gpu().gg_launch_count()
        ctx.setcof_prepare(*args, eol=eol)
        return _lib.gpu().gg_launch_count() - n0

    assert _lib.gpu().gg_test_setcof_positions(ctx._h, p) == 0
    n = launches()
    got = [ctx.setcof(j, 1.25) for j in range(1, len(ob.nak) + 1)]
    # two launches for every piece but a block's first; the hook is for one call
    assert n - launches() == 2 * sum((len(b["irow"]) - 1) // p for b in blocks)
    for j, g in enumerate(got, 1):
        ref = o.setcof(blocks, eol, j, 1.25)
        for key in ("nya", "nxa", "nda"):
            np.testing.assert_array_equal(g[key], ref[key])
        for key in ("ya", "xa", "da"):
            scale = max(1e-300, np.abs(ref[key]).max(initial=0.0))
            assert np.abs(g[key] - ref[key]).max(initial=0.0) <= 1e-14 * scale, (j, key)
