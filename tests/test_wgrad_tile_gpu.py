"""The halo-tile weight gradient at the edges of its tiles: every channel
instantiation, grids that do not tile by 8 x 16, plane counts that are not a
multiple of the planes of a step, fewer steps than SMs, upsampled inputs, and
the channel counts that stay with the gathered kernel."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("cin,cout,n,B,up", [
    (8, 16, (8, 16, 3), 1, 0), (8, 5, (12, 10, 7), 2, 0),
    (16, 16, (8, 16, 1), 1, 0), (16, 4, (20, 18, 5), 1, 0), (16, 32, (4, 4, 4), 2, 0), (16, 48, (9, 17, 2), 1, 0),
    (32, 16, (24, 24, 12), 1, 1), (32, 32, (10, 34, 3), 1, 0), (32, 64, (8, 8, 8), 2, 0),
    (64, 64, (8, 8, 8), 2, 0), (64, 32, (12, 20, 6), 1, 1), (64, 8, (1, 1, 1), 1, 0),
    (24, 16, (9, 6, 5), 1, 0),
])
def test_weight_gradient_at_tile_edges(cin, cout, n, B, up):
    import torch
    from lowmachmixtures_b200 import _native
    lib = _native.load()
    nx, ny, nz = n
    gen = torch.Generator().manual_seed(cin * 100 + cout + nx)
    x = torch.randn(B, nz >> up, ny >> up, nx >> up, cin, generator=gen).to(torch.bfloat16).cuda()
    cg = (cout + 7) // 8 * 8
    gy = torch.zeros(B, nz, ny, nx, cg, dtype=torch.bfloat16, device="cuda")
    gy[..., :cout] = torch.randn(B, nz, ny, nx, cout, generator=gen).to(torch.bfloat16).cuda()
    dw0 = torch.randn(cout, 27, cin, generator=gen).cuda()
    dw = dw0.clone()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert lib.lmm_nn_conv3d_wgrad(_p(x), _p(gy), _p(dw), B, nx, ny, nz, up, cin, cg, cout, _p(err), s) == 0
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    xd = x.double()
    for d in (1, 2, 3):
        xd = xd.repeat_interleave(2, d) if up else xd
    g = gy[..., :cout].double()
    ref, mag = [], []
    for t in range(27):
        sh = torch.roll(xd, (1 - t // 9, 1 - t // 3 % 3, 1 - t % 3), (1, 2, 3))
        ref.append(torch.einsum("bzyxo,bzyxc->oc", g, sh))
        mag.append(torch.einsum("bzyxo,bzyxc->oc", g.abs(), sh.abs()))
    ref = torch.stack(ref, 1) + dw0.double()
    mag = torch.stack(mag, 1) + dw0.double().abs()
    # exact products, at most 8192 of them added in FP32 (the tensor core truncates): 2^13 x 2^-24 of the sum of magnitudes
    assert ((dw.double() - ref).abs() <= 2.0 ** -11 * mag + 1e-30).all()
