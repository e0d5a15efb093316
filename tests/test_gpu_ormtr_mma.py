"""The double-precision back-transformation with X resident on the SM, at the edges of its tiles
(8 rows, 16 reflectors, 32 or 16 columns), of its CTA shapes (n = 120 | 121, 272 | 273) and of
its range (408 | 409), against LAPACK eigenvalues and the eigenvectors' residual."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W_TOL, R_TOL, O_TOL = 1e-12, 1e-12, 1e-10   # n eps |H| with n <= 409: 9e-14


@pytest.mark.parametrize("n,batch", [(2, 4), (7, 3), (8, 3), (16, 150), (17, 3), (18, 3), (31, 3), (34, 3), (120, 2),
                                     (121, 2), (128, 150), (129, 2), (241, 2), (272, 3), (273, 3), (280, 2), (281, 2),
                                     (408, 2), (409, 2)])
def test_resident_back_transformation(n, batch):
    import torch

    import rlmb
    rng = np.random.default_rng(n)
    h = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    h = (h + h.conj().swapaxes(1, 2)) / 2
    ctx = rlmb.Context(0)
    if n <= 80:
        ctx.set_heev_solver(n, ctx.SOLVER_HOUSEHOLDER)
    assert ctx.heev_config(n)[1]["gemm_bt"] == (1 if n > 408 else 0)
    a = torch.from_numpy(np.ascontiguousarray(h.swapaxes(1, 2))).cuda()   # column-major
    w = ctx.heevd(a).cpu().numpy()
    x = a.transpose(1, 2).cpu().numpy()
    for b in {0, batch - 1}:
        ref = np.linalg.eigvalsh(h[b])
        scale = np.abs(ref).max()
        assert np.abs(w[b] - ref).max() <= W_TOL * scale
        assert np.abs(h[b] @ x[b] - x[b] * w[b]).max() <= R_TOL * scale
        assert np.abs(x[b].conj().T @ x[b] - np.eye(n)).max() <= O_TOL
    ctx.close()
