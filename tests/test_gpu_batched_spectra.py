"""GPU parity: the projected eigensolver of gg_maneig_batched on blocks solved
in the full unit basis (NCF <= LIM), where it diagonalises the block itself:
sizes at the edges of the warp and of LIM, and spectra that take each of its
branches - isolated roots, clusters, exact degeneracy, decoupled rows.

Bars: the tridiagonalisation's backward error is of order m eps |H| (2.8e-14
at m = 128), so eigenvalues and residuals within 1e-12 |H|; roots closer than
1e-3 |H| are orthogonalised and for the others that error over the gap stays
below 1e-9.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 3, 5, 31, 32, 33, 34, 64, 65, 96, 127, 128)


def _matrix(kind, n, rng):
    if kind == "diagonal":
        return np.diag(np.sort(rng.normal(size=n)))
    if kind == "decoupled":
        a = rng.normal(size=(4, 4))
        return np.kron(np.eye(-(-n // 4)), a + a.T)[:n, :n]
    if kind == "ci":
        a = rng.normal(size=(n, n)) * 0.05
        return a + a.T + np.diag(-100.0 + 3.0 * np.sqrt(np.arange(n)))
    q = np.linalg.qr(rng.normal(size=(n, n)))[0]
    w = np.linspace(-1.0, 9.0, n)
    w[: min(n, 3)] = (-5.0, -5.0 + (1e-9 if kind == "close" else 0.0), -4.9999)[: min(n, 3)]
    h = q @ np.diag(w) @ q.T
    return 0.5 * (h + h.T)


@pytest.mark.parametrize("kind", ["ci", "close", "degenerate", "decoupled", "diagonal"])
def test_full_basis_blocks(gpu_ready, kind):
    from grasp_gb300 import Context, HMatrix, maneig_batched
    rng = np.random.default_rng(11)
    ctx = Context(0)
    mats = [_matrix(kind, n, rng) for n in SIZES]
    hs, nvec = [], []
    for h in mats:
        n = h.shape[0]
        ap = np.concatenate([h[i, : i + 1] for i in range(n)])
        hs.append(HMatrix.packed(ctx, n, ap))
        nvec.append(min(n, 4))
    res, info = maneig_batched(ctx, hs, nvec, lim=128)
    assert (info["ierr"] == 0).all()
    for h, (ev, vec), r in zip(mats, res, nvec):
        w = np.linalg.eigvalsh(h)
        nrm = np.abs(w).max()
        assert np.abs(ev - w[:r]).max() <= 1e-12 * nrm, (h.shape, ev - w[:r])
        assert np.abs(h @ vec - vec * ev).max() <= 1e-12 * nrm, h.shape
        assert np.abs(vec.T @ vec - np.eye(r)).max() <= 1e-9, h.shape
