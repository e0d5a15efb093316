"""Mesh pipelines at the edges of their launch shapes, against the CPU oracle: states that do
not fill a plaquette CTA, meshes on both sides of each slot-count boundary (g = 4 | 5, 32 | 33),
several samples, orders below the impurity band's width."""
import numpy as np
import pytest

from oracle import hlm as ohlm
from oracle import rlm as orlm

pytestmark = pytest.mark.gpu

# Energies: 1e-12 of the largest (n <= 40: backward error n eps with a margin of 100).  Chern
# numbers: eigenvector errors of ~1e-15 |H| / gap, gaps above ~1e-5 |H| on these inputs, summed
# over the g^2 plaquettes: 1e-8 leaves two orders of magnitude.
E_TOL, C_TOL = 1e-12, 1e-8


def _close(e, c, ref):
    assert np.abs(e - ref["energies"]).max() <= E_TOL * np.abs(ref["energies"]).max()
    assert np.abs(c - ref["chern"]).max() <= C_TOL


@pytest.mark.parametrize("n_phi,g,samples", [(3, 1, 2), (5, 4, 3), (17, 4, 1), (16, 5, 2), (33, 5, 1), (7, 32, 1),
                                             (6, 33, 2)])
def test_rlm_mesh_edges(n_phi, g, samples):
    import rlmb
    ctx = rlmb.Context(0)
    e, c = ctx.rlm_mesh_solve(n_phi, 1.0, 16.0, g, 11, 0, samples)
    for k, ref in enumerate(orlm.run(orlm.RlmParams(n_phi, 1.0, 16.0, g, samples, 11))):
        _close(e[k], c[k], ref)
    ctx.close()


@pytest.mark.parametrize("lx,ly,g,samples", [(3, 1, 3, 2), (6, 3, 4, 3), (9, 6, 5, 2), (6, 2, 33, 2)])
def test_hlm_mesh_edges(lx, ly, g, samples):
    import rlmb
    ctx = rlmb.Context(0)
    p = ohlm.HlmParams(lx, ly, 3, 0, g, samples, 11)
    pots = rlmb.hlm_potentials(11, p.n_sites, samples)
    e, c = ctx.hlm_mesh_solve(lx, ly, 3, 0, g, pots)
    for k in range(samples):
        _close(e[k], c[k], ohlm.run_sample(p, pots[k]))
    ctx.close()
