"""Divide-and-conquer merges shared by clusters of CTAs: chunk sizes that give a matrix 8, 5, 3
and 1 CTAs, orders whose upper levels leave a single child, degenerate spectra (deflation and
its rotations), against LAPACK with the tolerances of the divide-and-conquer tests."""
import numpy as np
import pytest

from test_gpu_parity import _check_eig, _hermitian, _run_heevd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch,kind", [(513, 1, None), (600, 25, None), (520, 40, None), (300, 150, None),
                                          (1030, 3, None), (33, 1, None), (64, 2, None),
                                          (7, 1, "identity"), (513, 6, "degenerate"), (700, 26, "blocks"),
                                          (640, 2, "tridiag_split")])
def test_dc_cluster(n, batch, kind):
    import torch

    import rlmb
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ctx = rlmb.Context(0)
    ctx.set_tridiag_solver(n, ctx.TRIDIAG_DC)
    rng = np.random.default_rng(n + batch)
    first = _hermitian(rng, n, kind) if kind else _hermitian(rng, n)
    mats = [first] + [_hermitian(rng, n) for _ in range(min(batch, 3) - 1)]
    mats += [mats[-1]] * (batch - len(mats))
    w, x = _run_heevd(ctx, mats)
    for b in {0, 1 % batch, batch - 1}:
        _check_eig(mats[b], w[b], x[b], np.linalg.eigvalsh(mats[b]))
    ctx.close()
