"""The reduction's panels by a cluster of CTAs per matrix (few matrices of order >= 256), against
LAPACK eigenvalues and the eigenvectors' residual and orthogonality: orders off the 16-column
strips and 32-row blocks, both panel widths, one matrix (16 CTAs) up to the chunk sizes where the
cluster shrinks to two CTAs, inactive reflectors; and by one CTA per matrix in chunks of more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Backward errors of the reduction are below n eps |H| (7e-13 at n = 3000); orthogonality of
# the tridiagonal solvers' vectors and of two mixed refinement steps as in the other solver tests.
W_TOL, R_TOL, O_TOL, O_TOL_MIXED = 1e-12, 1e-11, 1e-10, 1e-8


def _matrices(kind, n, batch, seed):
    rng = np.random.default_rng(seed)
    h = rng.standard_normal((batch, n, n)) + 1j * rng.standard_normal((batch, n, n))
    h = (h + h.conj().swapaxes(1, 2)) / 2
    if kind == "diagonal":        # every reflector inactive
        h = np.stack([np.diag(d) for d in h.diagonal(axis1=1, axis2=2).real]).astype(complex)
    elif kind == "blocks":        # inactive reflectors among active ones
        k = n // 3
        h[:, :k, k:] = h[:, k:, :k] = 0
        h[:, 2 * k:, :2 * k] = h[:, :2 * k, 2 * k:] = 0
    return h


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("kind,n,batch", [("random", 256, 1), ("random", 257, 18), ("random", 273, 5),
                                          ("random", 300, 36), ("random", 511, 74), ("random", 513, 26),
                                          ("random", 1031, 9), ("random", 1500, 2), ("diagonal", 260, 3),
                                          ("blocks", 301, 4), ("blocks", 1060, 2),
                                          # one CTA per matrix: 512, 256 and 128 threads
                                          ("random", 258, 100), ("random", 256, 150), ("blocks", 261, 297),
                                          ("random", 257, 600), ("random", 520, 160)])
def test_cluster_panels(kind, n, batch, mixed):
    import torch

    import rlmb
    h = _matrices(kind, n, batch, n + batch)
    ctx = rlmb.Context(0)
    ctx.precision = ctx.MIXED if mixed else ctx.FP64
    a = torch.from_numpy(np.ascontiguousarray(h.swapaxes(1, 2))).cuda()   # column-major
    w = ctx.heevd(a)
    x = a.transpose(1, 2)
    hd = torch.from_numpy(h).cuda()
    for b in sorted({0, batch // 2, batch - 1}):
        ref = np.linalg.eigvalsh(h[b])
        scale = np.abs(ref).max()
        assert np.abs(w[b].cpu().numpy() - ref).max() <= W_TOL * scale
        assert (hd[b] @ x[b] - x[b] * w[b]).abs().max().item() <= R_TOL * scale
        eye = torch.eye(n, dtype=x.dtype, device="cuda")
        assert (x[b].conj().T @ x[b] - eye).abs().max().item() <= (O_TOL_MIXED if mixed else O_TOL)
    ctx.close()
