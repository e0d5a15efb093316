"""Inverse iteration on clusters of equal eigenvalues whose vectors live on all but decoupled blocks:
an iterate that is one of the earlier vectors up to rounding has to be cleaned of it again.
Tridiagonals with entries 0 and 1 and couplings 0, 1 and 1e-9, against LAPACK with the
tolerances of the bisection tests."""
import numpy as np
import pytest

from test_gpu_bisection import O_TOL, R_TOL, W_TOL

pytestmark = pytest.mark.gpu

# diagonal, couplings; 9 stands for 1e-9
CASES = ["01100100011001110 0191990101009001", "10110111111100110 0011009101919190",
         "11111111110001111 0919119009100101", "10011001100111011 1101919100109990",
         "10011111000010111 0001091911191009", "01110011011110111 0090101011191990",
         "10100011010111100111110010011001 9000091110119191911009190901999",
         "00110010111010111000101001001001 9011199010090001919199999109191",
         "00111011111000010111111000000101 1019190010019090900901101191010"]


@pytest.mark.parametrize("case", CASES)
def test_degenerate_clusters(case):
    import torch

    import rlmb
    d, e = ([{"0": 0.0, "1": 1.0, "9": 1e-9}[c] for c in part] for part in case.split())
    n = len(d)
    t = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
    ctx = rlmb.Context(0)
    ctx.set_heev_solver(n, ctx.SOLVER_HOUSEHOLDER)
    ctx.set_tridiag_solver(n, ctx.TRIDIAG_BISECTION)
    a = torch.from_numpy(t.astype(complex)[None].copy()).cuda()
    info = torch.full((1,), -7, dtype=torch.int32, device="cuda")
    w = ctx.heevd(a, info=info)[0].cpu().numpy()
    assert not info.any()
    x = a[0].T.cpu().numpy()
    ref = np.linalg.eigvalsh(t)
    scale = np.abs(ref).max()
    assert np.abs(w - ref).max() <= W_TOL * scale
    assert np.abs(t @ x - x * w).max() <= R_TOL * scale
    assert np.linalg.norm(x.conj().T @ x - np.eye(n)) <= O_TOL
    ctx.close()
