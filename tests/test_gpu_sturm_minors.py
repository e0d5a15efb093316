"""Bisection on tridiagonals whose leading minors vanish or all but vanish: diagonal entries and
couplings that are zero or many powers of two below the norm, spectra with exact zeros on the
grid of the first counts.  Eigenvalues against LAPACK with the tolerance of the bisection tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIAGONAL = [0.0, 0.0, 0.5, -0.5, 0.25] + [s * 2.0 ** -k for k in (100, 200, 300) for s in (1, -1)]
COUPLING = [0.0, 0.0, 0.5, 0.25, 2.0 ** -60, 2.0 ** -150, 2.0 ** -300]


@pytest.mark.parametrize("n,batch", [(8, 8000), (12, 8000), (17, 4000), (40, 2000), (129, 300)])
def test_vanishing_minors(n, batch):
    import torch

    import rlmb
    rng = np.random.default_rng(n)
    d, e = rng.choice(DIAGONAL, (batch, n)), rng.choice(COUPLING, (batch, n - 1))
    d[:, 0], d[:, 1], e[:, :2] = -0.5, 0.5, 0.5   # a Gershgorin interval around zero
    t = np.zeros((batch, n, n))
    i = np.arange(n)
    t[:, i, i], t[:, i[:-1], i[1:]], t[:, i[1:], i[:-1]] = d, e, e
    ctx = rlmb.Context(0)
    if n <= 80:
        ctx.set_heev_solver(n, ctx.SOLVER_HOUSEHOLDER)
    ctx.set_tridiag_solver(n, ctx.TRIDIAG_BISECTION)
    w = ctx.heevd(torch.from_numpy(t.astype(complex)).cuda()).cpu().numpy()
    assert np.abs(w - np.linalg.eigvalsh(t)).max() <= 1e-12
    ctx.close()
