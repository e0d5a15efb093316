"""The largest orders the eigensolver takes, and the first ones it refuses: before any work."""
import pytest

pytestmark = pytest.mark.gpu


def _hermitian(n):
    import torch
    torch.manual_seed(n)
    h = torch.randn(n, n, dtype=torch.complex128, device="cuda")
    return (h + h.mH) / 2


def _check(ctx, n):
    import torch
    h = _hermitian(n)
    a = h.T[None].contiguous()
    w = ctx.heevd(a)[0]
    x = a[0].T
    assert (torch.linalg.norm(h @ x - x * w) / torch.linalg.norm(h)).item() <= 1e-11   # n eps, a margin of 7
    assert (x.mH @ x - torch.eye(n, device="cuda")).abs().max().item() <= 1e-10        # as the bisection solver's


def test_largest_order():
    import rlmb
    ctx = rlmb.Context(0)
    _check(ctx, 6370)
    ctx.close()


@pytest.mark.parametrize("n", [6400, 6500])
def test_orders_beyond_are_refused(n):
    import torch

    import rlmb
    ctx = rlmb.Context(0)
    a = _hermitian(n)[None].contiguous()
    before = a.clone()
    with pytest.raises(rlmb.RlmbError):
        ctx.heevd(a)
    assert torch.equal(a, before)
    _ok = ctx.heevd(_hermitian(40)[None].contiguous())   # the context works on
    assert bool(torch.isfinite(_ok).all())
    ctx.close()


def test_unblocked_limit():
    """The unblocked reduction pinned: four vectors of 16-byte entries in shared memory, up to order 3628;
    above, an argument error before any work."""
    import torch

    import rlmb
    ctx = rlmb.Context(0)
    for n in (3628, 3629):
        ctx.set_heev_config(n, 0, -1, 0, 0, 0)
    _check(ctx, 3628)
    a = _hermitian(3629)[None].contiguous()
    before = a.clone()
    with pytest.raises(rlmb.RlmbError, match="status -1"):
        ctx.heevd(a)
    assert torch.equal(a, before)
    ctx.close()
