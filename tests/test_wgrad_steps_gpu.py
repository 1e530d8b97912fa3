"""The halo-tile weight gradient over many steps per CTA: the refilled stages, the
release barriers in both phases and the sums that stay in tensor memory across
steps.  Every channel instantiation with five steps or more per CTA of 148
(odd and even numbers of them, a step count that the grid does not divide, a
ragged grid).  Inputs are whole numbers, every product and partial sum stays
below 2^24, so FP32 sums are exact and one lost voxel shows."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("cin,cout,n,B,up", [
    (8, 16, (64, 64, 64), 2, 0), (8, 8, (60, 50, 62), 2, 0),
    (16, 16, (64, 64, 64), 2, 0), (16, 4, (64, 64, 63), 2, 0), (16, 32, (64, 64, 33), 1, 0),
    (32, 16, (64, 64, 64), 2, 1), (32, 32, (44, 40, 37), 2, 0), (32, 64, (32, 32, 32), 2, 0),
    (64, 64, (32, 32, 32), 2, 0), (64, 32, (36, 36, 34), 1, 1)])
def test_weight_gradient_over_many_steps(cin, cout, n, B, up):
    import torch
    from lowmachmixtures_b200 import _native
    lib = _native.load()
    nx, ny, nz = n
    # steps per CTA: planes of a step and columns of a slice by channel count
    planes, cols = {8: (3, 16), 64: (1, 16)}.get(cin) or ((1, 32) if -(-cout // 16) % 2 == 0 else ({16: 3, 32: 2}[cin], 16))
    steps = -(-nx // 8) * -(-ny // 16) * -(-nz // planes) * B
    assert steps >= 5 * (148 // -(-cout // cols))
    gen = torch.Generator(device="cuda").manual_seed(cin + cout + nx + nz)
    x = torch.randint(-2, 3, (B, nz >> up, ny >> up, nx >> up, cin), device="cuda", generator=gen).to(torch.bfloat16)
    gy = torch.randint(-2, 3, (B, nz, ny, nx, cout), device="cuda", generator=gen).to(torch.bfloat16)
    cg = -(-cout // 8) * 8
    g = torch.nn.functional.pad(gy, (0, cg - cout)).contiguous()
    dw = torch.zeros(cout, 27, cin, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.lmm_nn_conv3d_wgrad(_p(x), _p(g), _p(dw), B, nx, ny, nz, up, cin, cg, cout, _p(err), s) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    xd = x.double()
    for d in (1, 2, 3):
        xd = xd.repeat_interleave(2, d) if up else xd
    gd = gy.double().reshape(-1, cout)
    for t in range(27):
        sh = torch.roll(xd, (1 - t // 9, 1 - t // 3 % 3, 1 - t % 3), (1, 2, 3)).reshape(-1, cin)
        assert torch.equal(dw[:, t].double(), gd.T @ sh)
