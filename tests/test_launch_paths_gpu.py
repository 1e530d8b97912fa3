"""Which path a size takes, and that the paths agree: V-cycle levels that run as
cluster legs (by the launches of one V-cycle), the pair kernels of the residual
and the prolongation against those of one face per thread (arrays that start an
entry past a pair), and the reductions at the sizes where their launch changes
(1 to 8 blocks: one cluster; up to 148: split by component; more: neither)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

P, NS, SL = -1, 100, 200


def _solver(dm, n, bc=None, **kw):
    from lowmachmixtures_b200 import abi
    from lowmachmixtures_b200.gmres import StokesSolver
    k = dict(precon_type=2, visc_type=-2, gmres_verbose=0, autotune=-1)
    return StokesSolver(dm, n, 1.0 / n[0], knobs=abi.make_knobs(**{**k, **kw}), bc=bc)


def _problem(dm, n, bc=None):
    from test_caller_arrays_gpu import _problem as make
    return make(dm, n, bc)


# launches of one V-cycle: a leg 1 down and 1 up, the coarse tail 1, a level of
# colour launches 2 x 2 dm colours + residual + restriction down, prolongation +
# 2 x 2 dm colours up (27 in 3D, 19 in 2D)
@pytest.mark.parametrize("dm,n,bc,which,launches", [
    (3, (16, 16, 16), None, 4, 3), (3, (16, 16, 16), None, 5, 3), (3, (32, 32, 32), None, 5, 5), (3, (32, 32, 32), None, 4, 30),
    (3, (64, 64, 64), None, 5, 32), (3, (32, 16, 24), ((P, P), (P, P), (NS, NS)), 5, 5), (3, (16, 16, 16), ((NS, SL), (P, P), (NS, NS)), 4, 3),
    (2, (64, 64), None, 5, 3), (2, (192, 96), None, 5, 7), (2, (192, 96), None, 4, 24), (2, (64, 48), ((P, P), (NS, NS)), 5, 3)])
def test_levels_run_as_legs(dm, n, bc, which, launches):
    import torch
    from lowmachmixtures_b200 import abi
    _, _, coef, _ = _problem(dm, n, bc)
    with _solver(dm, n, bc, method=abi.LMM_METHOD_FGMRES, precision=abi.LMM_PRECISION_FP32) as s:
        torch.cuda.synchronize()
        s.load_coeffs(*coef, 2.5)
        before = s.lib.lmm_kernel_launches()
        s.time_op(which, 1)   # one V-cycle to warm up, one timed
        assert s.lib.lmm_kernel_launches() - before == 2 * launches


@pytest.mark.parametrize("visc", [-1, -2, -3])
@pytest.mark.parametrize("dm,n,bc", [(2, (8, 12), None), (2, (20, 8), ((NS, SL), (P, P))), (3, (4, 8, 12), None), (3, (36, 4, 8), None),
                                     (3, (8, 12, 4), ((P, P), (SL, NS), (NS, NS)))])
def test_pairs_equal_single_faces(dm, n, bc, visc):
    import torch
    rhs, _, coef, (phi, _) = _problem(dm, n, bc)
    phi = [torch.where(r == 0, r, p) for r, p in zip(rhs, phi)]   # zero on the walls, as rhs
    coarse = tuple(m // 2 for m in reversed(n))
    gen = torch.Generator(device="cuda").manual_seed(sum(n))
    corr = [torch.randn(coarse, dtype=torch.float64, device="cuda", generator=gen) for _ in range(dm)]

    def at(arrays, off):
        return [torch.empty(a.numel() + off, dtype=torch.float64, device="cuda")[off:].view(a.shape).copy_(a) for a in arrays]

    got = []
    with _solver(dm, n, bc, visc_type=visc) as s:
        torch.cuda.synchronize()
        s.load_coeffs(*coef, 2.5)
        for off in (0, 1):
            f, r, out = at(phi, off), at(rhs, off), at([torch.zeros_like(c) for c in corr], off)
            torch.cuda.synchronize()
            s.residual_restrict(0, r, f, out)
            s.prolong_add(0, at(corr, off), f)
            torch.cuda.synchronize()
            got.append([a.cpu().numpy() for a in (*out, *f)])
    for a, b in zip(*got):
        assert np.isfinite(a).all() and np.abs(a).max() > 0
        np.testing.assert_array_equal(a, b)


# blocks of 2048 entries: 1, 2 | 3, 8 (too many to split by component too) | 9 | 148 | 149 | 592 (the most);
# odd counts read entry by entry
SIZES = [(2, (16, 16)), (2, (64, 64)), (2, (64, 96)), (2, (128, 128)), (2, (128, 144)), (2, (99, 187)),
         (3, (8, 8, 8)), (3, (16, 16, 16)), (3, (17, 15, 19)), (3, (32, 32, 16)), (3, (32, 24, 24)), (3, (64, 64, 74)), (3, (64, 32, 149)),
         (3, (128, 96, 100))]


@pytest.mark.parametrize("dm,n", SIZES)
def test_reductions_of_whole_numbers_are_exact(dm, n):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(sum(n))
    shape = tuple(reversed(n))
    a, b = ([torch.randint(-9, 10, shape, device="cuda", generator=gen).double() for _ in range(dm + 1)] for _ in range(2))

    def total(x, c, w):   # face component c: the seam plane counts w times
        return float(x.sum() + ((w - 1) * x.select(dm - 1 - c, 0).sum() if c < dm else 0))

    with _solver(dm, n) as s:
        torch.cuda.synchronize()
        dots, means = s.inner_prod(a[:dm], a[dm], b[:dm], b[dm]), s.sum_umac_press(a[:dm], a[dm])
    assert dots == [total(x * y, c, 3) for c, (x, y) in enumerate(zip(a, b))]
    w = [3] + [3 if m < 16 else 2 for m in n[1:]]
    cells = float(np.prod(n))
    assert means == [total(a[dm], dm, 1) / cells] + [total(a[c], c, w[c]) / cells for c in range(dm)]


@pytest.mark.parametrize("dm,n", SIZES)
def test_gram_schmidt_passes(dm, n):
    """Classical Gram-Schmidt (its fused passes, 1 to 8 vectors each) against the modified one (a dot product and
    a subtraction per vector): the same iterates but for rounding.  Sums of up to 2^21 terms are off by 2^-32 of
    their magnitude, eight columns of a basis whose condition is below 1e2 keep the solutions within 1e-6."""
    import torch
    from lowmachmixtures_b200 import abi
    bu, bp, coef, (xu, xp) = _problem(dm, n)
    res = []
    for orth in (0, 1):
        with _solver(dm, n, method=abi.LMM_METHOD_FGMRES, orthogonalization=orth, gmres_max_inner=9, gmres_max_iter=9,
                     gmres_max_outer=1) as s:
            yu, yp = [a.clone() for a in xu], xp.clone()
            torch.cuda.synchronize()
            st = s.solve_device(bu, bp, yu, yp, *coef, 0.1 * n[0] ** 2)[2]
            torch.cuda.synchronize()
        assert st["total_iter"] >= 3
        res.append([a.cpu().numpy() for a in (*yu, yp - yp.mean())])
    for a, b in zip(*res):
        assert np.isfinite(a).all()
        np.testing.assert_allclose(a, b, rtol=0, atol=1e-6 * np.abs(a).max())
