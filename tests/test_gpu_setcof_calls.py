"""gg_setcof_prepare forms the sums, gg_setcof one orbital's lists: a caller
who asks for few orbitals does not pay for the merging of every orbital's
lists over the blocks. Over three blocks, one preparation takes less time than
the lists of all 23 orbitals (it took 25 times as long when it formed them)."""
import time

import numpy as np
import pytest

from inputs import synth as S

pytestmark = pytest.mark.gpu


def test_preparation_leaves_the_lists_to_the_calls(gpu_ready):
    from grasp_gb300 import Context, HMatrix
    orbs, n, z = S.orbital_set(5, 3), 590, 10.0
    rnt, r = S.grid(n, z)
    ob = S.hydrogenic_orbitals(orbs, z, S.screenpar([k for _, k in orbs], 1), r, n=n)
    ctx = Context(0)
    ctx.set_grid(n, rnt, 0.05, S.CVAC, np.full(n, z))
    ctx.set_orbitals(ob.nak, ob.mf, ob.pf, ob.qf)
    ctx.genintrk()
    ctx.iabint_table()
    refs = [S.occupation(orbs, {(1, -1): 2, (2, -1): 2}), S.occupation(orbs, {(1, -1): 2, (2, 1): 2})]
    rng = np.random.default_rng(1)
    hs, evec = [], []
    for tj in (0, 2, 4):
        b = S.ci_block(orbs, refs, [0] * len(orbs), two_j=tj, parity=0, seed=3)
        h = HMatrix(ctx, b.ncf, b.iendc, b.irow)
        h.setham_upload(b.iq, b.tlist, b.vlists)
        hs.append(h)
        evec.append(np.linalg.qr(rng.normal(size=(b.ncf, 4)))[0])
    wt = [np.ones(4) / 4] * len(hs)

    def timed(f):
        t0 = time.perf_counter()
        f()
        return time.perf_counter() - t0

    prepare = min(timed(lambda: ctx.setcof_prepare(hs, wt, evec)) for _ in range(4))
    calls = min(timed(lambda: [ctx.setcof(j, 1.2) for j in range(1, len(orbs) + 1)]) for _ in range(4))
    assert prepare < calls, (prepare, calls)
