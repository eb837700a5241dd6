"""Stage statistics of gg_genintbreit: 32 is the host's time up to the last
launch, so the table kernels, most of whose time comes after it, are in 31
(the call) and 33 (the kernels) and not in 32."""
import numpy as np
import pytest

from inputs import synth as S

pytestmark = pytest.mark.gpu


def test_host_stage_excludes_the_kernels(gpu_ready):
    from grasp_gb300 import Context
    orbs, n, z = S.orbital_set(6, 3), 590, 26.0
    rnt, r = S.grid(n, z)
    ob = S.hydrogenic_orbitals(orbs, z, S.screenpar([k for _, k in orbs], 1), r, n=n)
    ctx = Context(0)
    ctx.set_grid(n, rnt, 0.05, S.CVAC, np.full(n, z))
    ctx.set_orbitals(ob.nak, ob.mf, ob.pf, ob.qf)
    e = -np.linspace(50.0, 1.0, len(ob.nak))
    after = []
    for _ in range(6):
        ctx.genintbreit(1, 1.0, e)
        total, host, kernels = (ctx.stage_stat(i) for i in (31, 32, 33))
        assert 0 < host < total and 0 < kernels < total
        after.append((total - host) / kernels)
    assert max(after) > 0.25, after
