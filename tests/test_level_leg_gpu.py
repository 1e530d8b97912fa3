"""The cluster legs of the V-cycle are bitwise neutral: a solve with them equals
the same solve with one launch per colour (tail_cells = -1 turns the legs and
the single-block tails off).  Sizes at which slabs are one plane thick, of
unequal thickness, span 8 and 16 CTAs and one and two pairs of cells per
thread, in 2D and 3D, periodic and with walls in every direction."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P, NS, SL = -1, 100, 200
CASES = [
    (2, (64, 64), None), (2, (96, 48), None), (2, (192, 96), None), (2, (32, 208), None),
    (2, (64, 48), ((P, P), (NS, NS))), (2, (80, 96), ((SL, NS), (P, P))), (2, (48, 80), ((NS, NS), (NS, SL))),
    (3, (16, 16, 16), None), (3, (32, 32, 32), None), (3, (48, 24, 40), None), (3, (16, 48, 80), None),
    (3, (32, 16, 24), ((P, P), (P, P), (NS, NS))), (3, (32, 32, 32), ((NS, NS), (P, P), (SL, NS))),
    (3, (24, 48, 24), ((NS, SL), (NS, NS), (NS, NS))),
]


def _solve(dm, n, bc, visc, mixed, **kw):
    import torch
    from lowmachmixtures_b200 import abi
    from lowmachmixtures_b200.gmres import StokesSolver
    gen = torch.Generator(device="cuda").manual_seed(17 + sum(n) + dm)

    def ext(nodal):
        e = [n[d] + (1 if d in nodal and abi.walled(bc, d) else 0) for d in range(dm)]
        return tuple(reversed(e))

    def rand(shape, lo, hi):
        return lo + (hi - lo) * torch.rand(shape, dtype=torch.float64, device="cuda", generator=gen)

    cells = ext(())
    bu = []
    for d in range(dm):
        r = rand(cells, -1.0, 1.0)
        r -= r.mean()
        if abi.walled(bc, d):
            r.select(dm - 1 - d, 0).zero_()
        bu.append(r)
    bp = torch.zeros(cells, dtype=torch.float64, device="cuda")
    alpha = [rand(cells, 0.5, 1.5) for _ in range(dm)]
    beta = rand(cells, 0.2, 5.0)
    bed = [rand(ext(abi.edge_nodal(dm, e)), 0.2, 5.0) for e in range(1 if dm == 2 else 3)]
    gamma = rand(cells, 0.1, 0.5)
    xu, xp = [torch.zeros_like(bp) for _ in range(dm)], torch.zeros_like(bp)
    k = dict(precon_type=2, visc_type=visc, gmres_max_iter=6, gmres_max_outer=2, gmres_verbose=0, autotune=-1, **kw)
    if mixed:
        k.update(method=abi.LMM_METHOD_FGMRES, precision=abi.LMM_PRECISION_FP32, orthogonalization=1)
    with StokesSolver(dm, n, 1.0 / n[0], knobs=abi.make_knobs(**k), bc=bc) as s:
        s.solve_device(bu, bp, xu, xp, alpha, beta, bed, gamma, 0.1 * n[0] ** 2)
    torch.cuda.synchronize()
    return [a.cpu().numpy() for a in xu] + [xp.cpu().numpy()]


@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("visc", [-1, -2, -3])
@pytest.mark.parametrize("dm,n,bc", CASES)
def test_legs_are_bitwise_neutral(dm, n, bc, visc, mixed):
    for a, b in zip(_solve(dm, n, bc, visc, mixed), _solve(dm, n, bc, visc, mixed, tail_cells=-1)):
        assert np.isfinite(a).all()
        np.testing.assert_array_equal(a, b)
