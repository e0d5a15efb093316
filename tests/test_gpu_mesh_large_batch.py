"""Batches of more than 65,535 k-points, and of more than 65,535 samples, at tiny orders: the same
results as in smaller calls (which the mesh tests compare with the oracle)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# The same arithmetic per sample up to the order of a convergence test's sums: 1e-12 for energies
# of order 1; Chern numbers as in the mesh-edge tests.
E_TOL, C_TOL = 1e-12, 1e-8


def _same(whole, parts, scale):
    e, c = (np.concatenate([p[i] for p in parts]) for i in (0, 1))
    assert np.abs(whole[0] - e).max() <= E_TOL * scale
    assert np.abs(whole[1] - c).max() <= C_TOL


@pytest.mark.parametrize("n_phi,g,samples", [(3, 8, 900), (16, 64, 16)])
def test_rlm_more_than_65535_k_points(n_phi, g, samples):
    import rlmb
    ctx = rlmb.Context(0)
    assert samples * (g + 1) ** 2 > 65535
    whole = ctx.rlm_mesh_solve(n_phi, 1.0, 16.0, g, 7, 0, samples)
    part = samples // 4
    parts = [ctx.rlm_mesh_solve(n_phi, 1.0, 16.0, g, 7, s, part) for s in range(0, samples, part)]
    _same(whole, parts, np.abs(whole[0]).max())
    ctx.close()


@pytest.mark.parametrize("lx,ly,g,samples", [(6, 3, 32, 64), (3, 2, 1, 66000)])
def test_hlm_more_than_65535_k_points(lx, ly, g, samples):
    import rlmb
    ctx = rlmb.Context(0)
    assert samples * (g + 1) * g > 65535
    pots = rlmb.hlm_potentials(7, lx * ly, samples)
    whole = ctx.hlm_mesh_solve(lx, ly, 3, 0, g, pots)
    part = samples // 4
    parts = [ctx.hlm_mesh_solve(lx, ly, 3, 0, g, pots[s:s + part]) for s in range(0, samples, part)]
    _same(whole, parts, np.abs(whole[0]).max())
    ctx.close()
