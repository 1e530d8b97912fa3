"""The operator and the residual by pairs of cells against the kernels that take
one face or cell per thread: arrays that do not start on a pair take the latter
for the operator, the fused residual + restriction (residual_fusion = 1)
replaces the former's residual.  Rows of one pair to several blocks, row counts
that do not fill a block, uniform and varying alpha."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("uniform", [True, False])
@pytest.mark.parametrize("visc", [-1, -2, -3])
@pytest.mark.parametrize("n", [(2, 4, 6), (6, 2, 4), (18, 10, 6), (34, 4, 10), (66, 6, 4), (130, 2, 2)])
def test_operator_by_pairs_equals_operator_by_cells(n, visc, uniform):
    import torch
    from lowmachmixtures_b200 import abi
    from lowmachmixtures_b200.gmres import StokesSolver
    gen = torch.Generator(device="cuda").manual_seed(sum(n) - visc)
    shape = tuple(reversed(n))

    def rand(lo, hi, off=0):
        a = torch.empty(int(np.prod(shape)) + off, dtype=torch.float64, device="cuda")[off:].view(shape)
        return a.copy_(lo + (hi - lo) * torch.rand(shape, dtype=torch.float64, device="cuda", generator=gen))

    alpha = [torch.full(shape, 1.25, dtype=torch.float64, device="cuda") if uniform else rand(0.5, 1.5) for _ in range(3)]
    x = [rand(-1, 1) for _ in range(4)]
    with StokesSolver(3, n, 1.0 / n[0], knobs=abi.make_knobs(precon_type=2, visc_type=visc, gmres_verbose=0, autotune=-1)) as s:
        s.load_coeffs(alpha, rand(0.2, 5), [rand(0.2, 5) for _ in range(3)], rand(0.1, 0.5), 3.7)
        outs = []
        for off in (0, 1):   # one entry past a pair: the kernel by cells
            xo = [rand(0, 1, off).copy_(a) for a in x]
            out = [rand(0, 1, off) for _ in range(4)]
            torch.cuda.synchronize()
            s.apply_matrix(xo[:3], xo[3], out[:3], out[3])
            torch.cuda.synchronize()
            outs.append([o.cpu().numpy() for o in out])
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [(64, 64, 64), (96, 48, 64), (16, 8, 72)])
def test_residual_by_pairs_equals_fused_residual(n, precision):
    import torch
    from lowmachmixtures_b200 import abi
    from lowmachmixtures_b200.gmres import StokesSolver
    gen = torch.Generator(device="cuda").manual_seed(5 + sum(n))
    shape = tuple(reversed(n))

    def rand(lo, hi):
        return lo + (hi - lo) * torch.rand(shape, dtype=torch.float64, device="cuda", generator=gen)

    bu = [rand(-1, 1) for _ in range(3)]
    bu = [b - b.mean() for b in bu]
    bp = torch.zeros(shape, dtype=torch.float64, device="cuda")
    coef = ([torch.ones_like(bp) for _ in range(3)], rand(0.2, 5), [rand(0.2, 5) for _ in range(3)], rand(0.1, 0.5))
    res = []
    for fusion in (0, 1):   # tail_cells = -1: every level by per-level kernels
        k = abi.make_knobs(precon_type=2, visc_type=-2, method=abi.LMM_METHOD_FGMRES, precision=precision, residual_fusion=fusion,
                           tail_cells=-1, gmres_max_iter=4, gmres_max_outer=1, gmres_verbose=0, autotune=-1)
        xu, xp = [torch.zeros_like(bp) for _ in range(3)], torch.zeros_like(bp)
        with StokesSolver(3, n, 1.0 / n[0], knobs=k) as s:
            s.solve_device(bu, bp, xu, xp, *coef, 0.1 * n[0] ** 2)
        torch.cuda.synchronize()
        res.append([a.cpu().numpy() for a in xu] + [xp.cpu().numpy()])
    for a, b in zip(*res):
        assert np.isfinite(a).all()
        np.testing.assert_array_equal(a, b)
