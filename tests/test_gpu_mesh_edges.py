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


@pytest.mark.parametrize("n_phi,g", [(8, 70), (70, 130), (65, 3)])
def test_assemble_theta_groups(n_phi, g):
    """More distinct theta_2 than one launch's list holds, unsorted and repeated; every entry
    within 1e-13 of the largest one (sums of at most dim^2 = 1225 terms, n eps)."""
    import torch

    import rlmb
    ctx = rlmb.Context(0)
    p = orlm.RlmParams(n_phi, 1.0, 16.0, g, 1, 3)
    cmn, cmt, cjm = orlm.prepare_coeff(p)
    rng = np.random.default_rng(5)
    v = rng.standard_normal(p.dim ** 2) + 1j * rng.standard_normal(p.dim ** 2)
    t2 = np.concatenate([rng.permutation(g + 1), rng.integers(0, g + 1, 5)])
    t1 = rng.integers(0, g + 1, len(t2))
    got = ctx.rlm_assemble(*(torch.from_numpy(a).cuda() for a in (v, cmt, cjm)), n_phi, p.off_head, g, t1, t2)
    for i in range(0, len(t2), max(1, len(t2) // 40)):
        ref = orlm.assemble(p, v, cmt, cjm, int(t1[i]), int(t2[i])).reshape(n_phi, n_phi)
        assert np.abs(got[i].cpu().numpy() - ref).max() <= 1e-13 * np.abs(ref).max()
    ctx.close()


@pytest.mark.parametrize("lx,ly,g", [(24, 8, 2), (24, 16, 3), (48, 8, 2), (48, 16, 2)])
def test_hlm_links_block_sizes(lx, ly, g):
    """Bloch blocks of 8 and 16 in either direction (the tensor-path link kernel)."""
    import rlmb
    ctx = rlmb.Context(0)
    p = ohlm.HlmParams(lx, ly, 3, 0, g, 1, 4)
    pots = rlmb.hlm_potentials(4, p.n_sites, 1)
    e, c = ctx.hlm_mesh_solve(lx, ly, 3, 0, g, pots)
    _close(e[0], c[0], ohlm.run_sample(p, pots[0]))
    ctx.close()
