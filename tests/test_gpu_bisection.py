"""The bisection tridiagonal solver on tridiagonals that strain its integer sign and range tests,
its power-of-two scaling and its twisted factorisation, at the edges of its thread counts (one
CTA of 32 to 256 threads per matrix, two CTAs from order 257 on in small chunks): against
LAPACK's tridiagonal eigenvalues, and the eigenvectors' residual and orthogonality."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# as the Householder tests: eigenvalues and residual 1e-12 |T|, orthogonality 1e-11 (Frobenius)
W_TOL, R_TOL, O_TOL = 1e-12, 1e-12, 1e-11


def _tridiagonal(kind, n):
    rng = np.random.default_rng(n)
    d, e = rng.uniform(-1, 1, n), rng.uniform(0.1, 1, max(n - 1, 0))
    if kind == "huge":
        d, e = d * 2.0 ** 400, e * 2.0 ** 400
    elif kind == "tiny":
        d, e = d * 2.0 ** -400, e * 2.0 ** -400
    elif kind == "split":          # zero couplings: independent blocks
        e[rng.random(n - 1) < 0.2] = 0.0
    elif kind == "weak":           # couplings down to 1e-12: near-splits, tiny minors
        e *= 10.0 ** rng.uniform(-12, 0, n - 1)
    elif kind == "wilkinson":      # pairs of eigenvalues agreeing to working precision
        d, e = np.abs(np.arange(n) - (n - 1) / 2.0), np.ones(n - 1)
    elif kind == "toeplitz":       # zero minors at x = 0
        d, e = np.zeros(n), np.ones(n - 1)
    elif kind == "graded":
        s = 10.0 ** -np.linspace(0, 10, n)
        d, e = d * s, e * s[1:]
    return d, e


@pytest.mark.parametrize("batch", [1, 160])
@pytest.mark.parametrize("kind,n", [("plain", n) for n in (2, 3, 4, 5, 31, 32, 33, 63, 65, 128, 129, 256, 257, 300, 384, 385)]
                         + [(k, n) for k in ("huge", "tiny", "split", "weak", "wilkinson", "toeplitz", "graded")
                            for n in (21, 64, 150, 301)])
def test_bisection(kind, n, batch):
    import scipy.linalg
    import torch

    import rlmb
    d, e = _tridiagonal(kind, n)
    t = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
    ctx = rlmb.Context(0)
    if n <= 80:
        ctx.set_heev_solver(n, ctx.SOLVER_HOUSEHOLDER)
    ctx.set_tridiag_solver(n, ctx.TRIDIAG_BISECTION)
    a = torch.from_numpy(np.repeat(t[None].astype(complex), batch, axis=0)).cuda()
    info = torch.full((batch,), -7, dtype=torch.int32, device="cuda")
    w = ctx.heevd(a, info=info).cpu().numpy()
    assert not info.any()
    x = a.transpose(1, 2)[[0, batch - 1]].cpu().numpy()
    ref = scipy.linalg.eigvalsh_tridiagonal(d, e)
    scale = np.abs(ref).max()
    for i, b in enumerate((0, batch - 1)):
        assert np.abs(w[b] - ref).max() <= W_TOL * scale
        assert np.abs((t / scale) @ x[i] - x[i] * (w[b] / scale)).max() <= R_TOL
        assert np.linalg.norm(x[i].conj().T @ x[i] - np.eye(n)) <= O_TOL
    ctx.close()
