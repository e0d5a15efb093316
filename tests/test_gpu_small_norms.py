"""Eigensolves of matrices of small norm, where the squares of a reflector's entries are denormal in
the reduction's precision (single in the mixed mode) but not yet zero: against LAPACK on the
matrix of unit scale."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# Squares of entries x ~ scale: relative error 2^-149 / x^2 in single precision (1e-5 at 1e-20, which
# two refinement steps take back), 2^-1074 / x^2 in double (1e-14 at 1e-155, times n per column).
@pytest.mark.parametrize("mixed,n,scale,tol", [(True, 40, 1e-19, 1e-12), (True, 40, 3e-20, 1e-12), (True, 150, 1e-20, 1e-11),
                                               (True, 300, 1e-20, 1e-11), (False, 40, 1e-154, 1e-12),
                                               (False, 40, 1e-155, 1e-11), (False, 150, 1e-155, 1e-11),
                                               (False, 300, 1e-155, 1e-11)])
def test_small_norm(mixed, n, scale, tol):
    import torch

    import rlmb
    rng = np.random.default_rng(n)
    h = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    h = (h + h.conj().T) / 2
    ctx = rlmb.Context(0)
    ctx.precision = ctx.MIXED if mixed else ctx.FP64
    if n <= 80:
        ctx.set_heev_solver(n, ctx.SOLVER_HOUSEHOLDER)
    a = torch.from_numpy(np.ascontiguousarray((h * scale).T)[None]).cuda()   # column-major
    info = torch.full((1,), -7, dtype=torch.int32, device="cuda")
    w = ctx.heevd(a, info=info)[0].cpu().numpy() / scale
    assert not info.any()
    x = a[0].T.cpu().numpy()
    ref = np.linalg.eigvalsh(h)
    norm = np.abs(ref).max()
    assert np.abs(w - ref).max() <= tol * norm
    assert np.abs(h @ x - x * w).max() <= tol * norm
    assert np.abs(x.conj().T @ x - np.eye(n)).max() <= 10 * tol
    ctx.close()
