"""GPU parity: block Davidson passes in FP64 (gg_maneig with MBLOCK = NVEC)
at the widths and orders where the Gram dots change form: few pairs (each
pair's two sums in two warps) up to more than half a block of them, row chunks
full, ragged and single, columns per grid row narrowed on idle SMs or not.

Bar: the solver stops on a residual below 1e-9, and an eigenvalue's error is
of second order in it: 1e-10 of the spectrum, as the dense reference's own
error is far below; the vectors' by the residual over the smallest gap, 1e-6.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [65, 128, 361, 1021])
@pytest.mark.parametrize("nvec", [1, 2, 3, 4, 5, 8, 12, 16])
def test_block_pass_widths(gpu_ready, n, nvec):
    from grasp_gb300 import Context, HMatrix
    rng = np.random.default_rng(n + nvec)
    a = rng.normal(size=(n, n)) * 0.02
    h = a + a.T + np.diag(-20.0 + 0.37 * np.arange(n) ** 0.9)
    m = HMatrix.packed(Context(0), n, np.concatenate([h[i, : i + 1] for i in range(n)]))
    ev, vec, _ = m.maneig(nvec, precision=0, mblock=nvec)
    w, u = np.linalg.eigh(h)
    assert np.abs(ev - w[:nvec]).max() <= 1e-10 * np.abs(w).max()
    u = u[:, :nvec] * np.sign(np.sum(u[:, :nvec] * vec, axis=0))
    assert np.abs(vec - u).max() <= 1e-6
    np.testing.assert_allclose(vec.T @ vec, np.eye(nvec), atol=1e-12)
