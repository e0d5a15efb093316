"""The unblocked reduction at the edges of its 16 x 16 tiles, thread counts and storage (per-tile
sums up to order 144, shared atomics above; the triangle resident up to order ~155), few and
many matrices, both precisions, against LAPACK eigenvalues and the eigenvectors' residual."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W_TOL, R_TOL, O_TOL = 1e-13, 1e-12, 1e-10   # n eps |H| with n <= 255: 6e-14


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n,batch", [(1, 3), (2, 3), (3, 200), (15, 5), (16, 200), (17, 200), (33, 150), (48, 149),
                                     (49, 149), (64, 3), (65, 3), (100, 149), (101, 149), (144, 2), (145, 149),
                                     (160, 3), (200, 2), (255, 2)])
def test_unblocked_reduction(n, batch, mixed):
    import torch

    import rlmb
    rng = np.random.default_rng(n)
    h = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    h = (h + h.conj().swapaxes(1, 2)) / 2
    if batch > 2:
        h[1] = np.diag(h[1].diagonal().real)   # every reflector inactive
    ctx = rlmb.Context(0)
    ctx.precision = ctx.MIXED if mixed else ctx.FP64
    ctx.set_heev_solver(n, ctx.SOLVER_HOUSEHOLDER)
    a = torch.from_numpy(np.ascontiguousarray(h.swapaxes(1, 2))).cuda()   # column-major
    w = ctx.heevd(a).cpu().numpy()
    x = a.transpose(1, 2).cpu().numpy()
    for b in sorted({0, 1, batch - 1}):
        ref = np.linalg.eigvalsh(h[b])
        scale = np.abs(ref).max()
        assert np.abs(w[b] - ref).max() <= W_TOL * scale
        assert np.abs(h[b] @ x[b] - x[b] * w[b]).max() <= R_TOL * scale
        assert np.abs(x[b].conj().T @ x[b] - np.eye(n)).max() <= O_TOL
    ctx.close()
