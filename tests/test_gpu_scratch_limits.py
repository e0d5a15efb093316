"""Small calls take little memory, run where little is left, and bring their results home without
pinned memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_small_call_takes_little_memory():
    """hlm 6 x 6, g = 8, one sample: 72 matrices of order 12, 0.2 MB in all."""
    import rlmb
    pots = rlmb.hlm_potentials(3, 36, 1)
    for k in range(2):   # (the first call also loads kernels)
        before = _free()
        ctx = rlmb.Context(0)
        ctx.hlm_mesh_solve(6, 6, 3, 0, 8, pots)
        taken = before - _free()
        ctx.close()
    assert taken <= 8 << 20


def test_small_call_in_scarce_memory():
    """rlm n_phi = 32, g = 8: about 7 MB in a new context, with 20 MB left on the device."""
    import torch

    import rlmb
    ctx = rlmb.Context(0)
    ref = ctx.rlm_mesh_solve(32, 1.0, 16.0, 8, 1, 0, 1)
    ctx.close()
    torch.cuda.empty_cache()
    held = torch.empty(_free() - (20 << 20), dtype=torch.uint8, device="cuda")
    try:
        assert _free() <= 24 << 20
        ctx = rlmb.Context(0)
        got = ctx.rlm_mesh_solve(32, 1.0, 16.0, 8, 1, 0, 1)
        ctx.close()
    finally:
        del held
        torch.cuda.empty_cache()
    assert all(np.array_equal(a, b) for a, b in zip(got, ref))


def _pinned_bytes(ctx):
    """The context's count of pinned host bytes, read from its start: device, stream, launches, then
    pointer and size of the workspace, of the pipeline buffer and of the pinned buffer."""
    import ctypes
    words = (ctypes.c_size_t * 9).from_address(ctypes.cast(ctx.h, ctypes.c_void_p).value)
    assert words[0] & 0xffffffff == 0 and words[4] % (1 << 20) == 0 and words[6] % (1 << 20) == 0 and words[6] > 0
    return words[8]


def test_no_pinned_memory_for_small_results():
    """Pinned memory takes 1 to 3 ms to allocate, more than the first call of a small lattice."""
    import rlmb
    ctx = rlmb.Context(0)
    ctx.hlm_mesh_solve(6, 6, 3, 0, 8, rlmb.hlm_potentials(3, 36, 2))
    ctx.rlm_mesh_solve(16, 1.0, 16.0, 4, 1, 0, 2)
    assert _pinned_bytes(ctx) == 0
    ctx.close()


@pytest.mark.parametrize("samples", [1, 700])
def test_results_of_either_size(samples):
    """Results in one copy, and above 256 KB straight to the caller's arrays: as on the device."""
    import torch

    import rlmb
    ctx = rlmb.Context(0)
    n = 32
    pots = rlmb.hlm_potentials(5, 96, samples)
    e, c = ctx.hlm_mesh_solve(12, 8, 3, 0, 1, pots)
    de, dc = (torch.empty((samples, n), dtype=torch.float64, device="cuda") for _ in range(2))
    ctx.hlm_mesh_solve_device(12, 8, 3, 0, 1, torch.from_numpy(pots).cuda(), de, dc)
    assert np.array_equal(e, de.cpu().numpy()) and np.array_equal(c, dc.cpu().numpy())
    e, c = ctx.rlm_mesh_solve(n, 1.0, 16.0, 1, 5, 0, samples)
    ctx.rlm_mesh_solve_device(n, 1.0, 16.0, 1, 5, 0, de, dc)
    assert np.array_equal(e, de.cpu().numpy()) and np.array_equal(c, dc.cpu().numpy())
    ctx.close()


def test_results_of_several_batches():
    """More than the 40 GB of a batch (580 samples of 289 matrices of order 128): as on the device.
    (Up to order 144 every sum has a fixed order, so that two calls agree bit for bit.)"""
    import torch

    import rlmb
    ctx = rlmb.Context(0)
    n, samples = 128, 580
    e, c = ctx.rlm_mesh_solve(n, 1.0, 16.0, 16, 5, 0, samples)
    assert _pinned_bytes(ctx) > 0
    de, dc = (torch.empty((samples, n), dtype=torch.float64, device="cuda") for _ in range(2))
    ctx.rlm_mesh_solve_device(n, 1.0, 16.0, 16, 5, 0, de, dc)
    assert np.array_equal(e, de.cpu().numpy()) and np.array_equal(c, dc.cpu().numpy())
    ctx.close()


def test_potential_of_many_samples():
    """V_mn of 3,000 samples of 2,064 impurities on 47 x 47 coefficients, 33 splits of 35 kB each: its
    scratch is bounded (3.5 GB at once otherwise), the sums are those of a call of one sample."""
    import torch

    import rlmb
    ctx = rlmb.Context(0)
    samples, nimp, o = 3000, 2064, 23
    dim = 2 * o + 1
    gen = torch.Generator(device="cuda").manual_seed(4)
    x, y, s = (torch.rand((samples, nimp), dtype=torch.float64, device="cuda", generator=gen) for _ in range(3))
    cmn = torch.randn((dim, dim), dtype=torch.complex128, device="cuda", generator=gen)
    ctx.rlm_potential(x[:1], y[:1], s[:1], cmn, o)   # (loads the kernels)
    torch.cuda.empty_cache()
    out = torch.empty((samples, dim * dim), dtype=torch.complex128, device="cuda")   # as large as the call's own
    before = _free()
    del out
    v = ctx.rlm_potential(x, y, s, cmn, o)
    assert before - _free() <= 300 << 20
    for k in (0, 1, 503, 504, samples - 1):
        one = ctx.rlm_potential(x[k:k + 1].contiguous(), y[k:k + 1].contiguous(), s[k:k + 1].contiguous(), cmn, o)
        assert torch.equal(v[k].reshape(-1), one.reshape(-1))
    ctx.close()
