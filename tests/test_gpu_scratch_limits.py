"""Small calls take little memory and run where little is left."""
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
