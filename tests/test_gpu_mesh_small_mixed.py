"""Mesh solves of orders up to 20 in the mixed mode: double precision as in the FP64 mode, whatever
the number of refinement steps, against the CPU oracle with the tolerances of the double-precision
mesh tests; exported eigenvectors with those of the export test, and against the batched eigensolver."""
import os

import numpy as np
import pytest

from oracle import hlm as ohlm
from oracle import rlm as orlm
from oracle import vsl
from test_gpu_mesh_edges import _close

pytestmark = pytest.mark.gpu


def _context(steps):
    import rlmb
    ctx = rlmb.Context(0)
    ctx.precision = ctx.MIXED
    ctx.set_refinement_steps(steps)
    return ctx


@pytest.mark.parametrize("steps", [1, 2])
@pytest.mark.parametrize("n_phi", [12, 13, 16, 18, 20])
def test_mixed_rlm_small(n_phi, steps):
    ctx = _context(steps)
    e, c = ctx.rlm_mesh_solve(n_phi, 1.0, 16.0, 6, 3, 0, 2)
    for k, ref in enumerate(orlm.run(orlm.RlmParams(n_phi, 1.0, 16.0, 6, 2, 3))):
        _close(e[k], c[k], ref)
    ctx.close()


@pytest.mark.parametrize("steps", [1, 2])
@pytest.mark.parametrize("lx,ly", [(6, 6), (9, 6), (6, 10), (12, 4)])
def test_mixed_hlm_small(lx, ly, steps):
    import rlmb
    ctx = _context(steps)
    p = ohlm.HlmParams(lx, ly, 3, 0, 6, 2, 5)
    pots = rlmb.hlm_potentials(5, p.n_sites, 2)
    e, c = ctx.hlm_mesh_solve(lx, ly, 3, 0, 6, pots)
    for k in range(2):
        _close(e[k], c[k], ohlm.run_sample(p, pots[k]))
    ctx.close()


@pytest.mark.parametrize("steps", [1, 2])
@pytest.mark.parametrize("n", [13, 20])
def test_mixed_export_small(n, steps, tmp_path):
    ctx = _context(steps)
    g, sample = 3, 1
    ctx.rlm_mesh_export(n, 1.0, 16.0, g, 1, sample, str(tmp_path))
    ctx.close()
    p = orlm.RlmParams(n, 1.0, 16.0, g, 1, 1)
    cmn, cmt, cjm = orlm.prepare_coeff(p)
    vmn = orlm.potential_coeff(*vsl.rlm_disorder(p.impurity_num, p.L1, p.L2, p.seed, sample), cmn, p.dim, p.off_head)
    for t1 in range(g + 1):
        for t2 in range(g + 1):
            x = np.fromfile(os.path.join(tmp_path, f"wfs_{t1}_{t2}.bin"), np.complex128).reshape(n, n).T
            h = orlm.assemble(p, vmn, cmt, cjm, t1, t2).reshape(n, n).T
            assert np.linalg.norm(h @ x - x * np.linalg.eigvalsh(h)) <= 1e-12 * np.linalg.norm(h)
            assert np.linalg.norm(x.conj().T @ x - np.eye(n)) <= 1e-12


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n", [12, 13, 16, 20, 21])
def test_export_phases(n, mixed, tmp_path):
    """Exported vectors are the batched eigensolver's, phases included: both come from the same
    arithmetic up to the order of the sums, so gaps above 1e-3 |H| leave 1e-12; 1e-9 is asserted
    (the mixed mode above order 20: 1e-6, its vectors carry the refinement's error)."""
    import torch
    ctx = _context(2)
    if not mixed:
        ctx.precision = ctx.FP64
    g, sample = 3, 0
    ctx.rlm_mesh_export(n, 1.0, 16.0, g, 1, sample, str(tmp_path))
    p = orlm.RlmParams(n, 1.0, 16.0, g, 1, 1)
    cmn, cmt, cjm = orlm.prepare_coeff(p)
    vmn = orlm.potential_coeff(*vsl.rlm_disorder(p.impurity_num, p.L1, p.L2, p.seed, sample), cmn, p.dim, p.off_head)
    points = [(t1, t2) for t1 in range(g + 1) for t2 in range(g + 1)]
    h = np.stack([orlm.assemble(p, vmn, cmt, cjm, *t).reshape(n, n) for t in points])
    a = torch.from_numpy(h).cuda()
    ctx.heevd(a)
    got = np.stack([np.fromfile(os.path.join(tmp_path, f"wfs_{t1}_{t2}.bin"), np.complex128).reshape(n, n)
                    for t1, t2 in points])
    assert np.abs(got - a.cpu().numpy()).max() <= (1e-6 if mixed and n > 20 else 1e-9)
    ctx.close()
