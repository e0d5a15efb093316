"""Divide and conquer pinned at the smallest orders, where a cluster of CTAs reaches its first shared
merge at once, and on spectra that deflate wholly (no root is left to share): against LAPACK
with the tolerances of the divide-and-conquer tests.  The Householder path is pinned as well: the
batched eigensolver would take Jacobi at these orders."""
import numpy as np
import pytest

from test_gpu_parity import _check_eig, _hermitian, _run_heevd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch,kind", [(2, 1, "random"), (2, 148, "random"), (3, 2, "random"), (5, 1, "random"),
                                          (7, 1, "identity"), (7, 30, "random"), (20, 3, "degenerate"),
                                          (33, 18, "random"), (65, 2, "tridiag_split"), (513, 4, "identity"),
                                          (600, 3, "diagonal")])
def test_dc_small(n, batch, kind):
    import rlmb
    ctx = rlmb.Context(0)
    if n <= 80:
        ctx.set_heev_solver(n, ctx.SOLVER_HOUSEHOLDER)
    ctx.set_tridiag_solver(n, ctx.TRIDIAG_DC)
    rng = np.random.default_rng(n + batch)
    mats = [_hermitian(rng, n, kind) for _ in range(min(batch, 3))]
    mats += [mats[-1]] * (batch - len(mats))
    w, x = _run_heevd(ctx, mats)
    for b in {0, 1 % batch, batch - 1}:
        _check_eig(mats[b], w[b], x[b], np.linalg.eigvalsh(mats[b]))
    ctx.close()
