"""gg_brint from several threads on one table: the first look-ups, which copy
the table to the host, give the table's values like the later ones, for a new
table each time (a smaller one after a larger one among them)."""
import threading

import numpy as np
import pytest

from tests.test_gpu_breit import _hyd

pytestmark = pytest.mark.gpu


def test_first_lookups_from_several_threads(gpu_ready, oracle_mod):
    ctx, _, nw, e = _hyd()
    key = nw + 1
    for itype, wfact in [(1, 1.0), (2, 1.0), (1, 0.0), (2, 0.0)] * 5:
        ind, val, kst, _ = ctx.genintbreit(itype, wfact, e)
        k = np.repeat(np.arange(len(kst) - 1), np.diff(kst))
        bad, gate = [], threading.Barrier(8)

        def look(seed):
            gate.wait()
            for t in np.random.default_rng(seed).integers(0, len(ind), 40):
                a, b, c, d = (int(ind[t]) // key ** p % key for p in (3, 2, 1, 0))
                if ctx.brint(itype, a, b, c, d, int(k[t])) != val[t]:
                    bad.append(t)

        threads = [threading.Thread(target=look, args=(s,)) for s in range(8)]
        for th in threads:
            th.start()
        for th in threads:
            th.join()
        assert not bad
