"""Reductions whose vectors leave the cluster panels' staging no room (double precision): a single
matrix above order 5080, and about as many matrices as SMs above order 3000."""
import time

import pytest

pytestmark = pytest.mark.gpu

# Residual and orthogonality: n eps with a margin of 10 (divide and conquer up to order 3600), and
# bisection's 1e-10 above.  Time of a second call: 1.6 s; one CTA of few threads for all panels takes 10.
@pytest.mark.parametrize("n,batch,res,orth,seconds", [(5200, 1, 1e-11, 1e-10, 5.0), (3100, 100, 1e-11, 1e-11, None)])
def test_long_vectors(n, batch, res, orth, seconds):
    import torch

    import rlmb
    torch.manual_seed(n)
    h = torch.randn(n, n, dtype=torch.complex128, device="cuda")
    h = (h + h.mH) / 2
    ctx = rlmb.Context(0)
    a = torch.empty((batch, n, n), dtype=h.dtype, device="cuda")
    for rep in range(2 if seconds else 1):
        a[:] = h.T
        torch.cuda.synchronize()
        t = time.perf_counter()
        w = ctx.heevd(a)
        torch.cuda.synchronize()
        t = time.perf_counter() - t
    ctx.close()
    for b in {0, batch - 1}:
        x = a[b].T
        assert (torch.linalg.norm(h @ x - x * w[b]) / torch.linalg.norm(h)).item() <= res
        assert (x.mH @ x - torch.eye(n, device="cuda")).abs().max().item() <= orth
        assert abs((w[b].sum() - h.diagonal().real.sum()).item()) <= 1e-9 * w[b].abs().max().item()
    assert not seconds or t <= seconds
