"""Where the caller's arrays may lie: kernels read and write those of the
handle's device in place, every other array that a copy takes goes through the
handle's buffers (pinned host memory, an address that is not a multiple of 8),
with the same results; a missing array is an error and leaves the handle usable;
an operator whose output overlaps an input goes through the handle's vectors."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [(2, (32, 24), None), (2, (24, 32), ((-1, -1), (100, 200))), (3, (16, 8, 12), None), (3, (15, 9, 5), None)]


class _At:
    """One array in memory of the given form, with the address the ABI takes."""

    def __init__(self, src, form):
        import torch
        src = src.contiguous()
        self.src, n = src, src.numel()
        if form == "pinned":
            self.t = torch.empty(n, dtype=torch.float64).pin_memory()
        elif form == "misaligned":
            self.t = torch.empty(8 * n + 16, dtype=torch.uint8, device="cuda")[4:4 + 8 * n]
        elif form == "inside":   # an odd entry inside a larger allocation
            self.t = torch.empty(n + 7, dtype=torch.float64, device="cuda")[3:3 + n]
        else:
            self.t = torch.empty(n, dtype=torch.float64, device="cuda")
        flat = src.reshape(-1)
        self.t.copy_(flat.view(torch.uint8) if form == "misaligned" else flat)

    def data_ptr(self):
        return self.t.data_ptr()

    def value(self):
        import torch
        t = self.t.clone()
        return (t.view(torch.float64) if t.dtype == torch.uint8 else t).reshape(self.src.shape).cpu().numpy()


def _problem(dm, n, bc):
    import torch
    from lowmachmixtures_b200 import abi
    gen = torch.Generator(device="cuda").manual_seed(3 + sum(n) + dm)

    def ext(nodal):
        return tuple(reversed([n[d] + (1 if d in nodal and abi.walled(bc, d) else 0) for d in range(dm)]))

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
    coef = ([rand(cells, 0.5, 1.5) for _ in range(dm)], rand(cells, 0.2, 5.0),
            [rand(ext(abi.edge_nodal(dm, e)), 0.2, 5.0) for e in range(1 if dm == 2 else 3)], rand(cells, 0.1, 0.5))
    x0 = [rand(cells, -0.1, 0.1) for _ in range(dm)], rand(cells, -0.1, 0.1)
    return bu, bp, coef, x0


def _solver(dm, n, bc):
    from lowmachmixtures_b200 import abi
    from lowmachmixtures_b200.gmres import StokesSolver
    k = abi.make_knobs(precon_type=2, visc_type=-3, gmres_max_iter=4, gmres_max_outer=1, gmres_verbose=0, autotune=-1)
    return StokesSolver(dm, n, 1.0 / n[0], knobs=k, bc=bc)


def _run(dm, n, bc, form):
    import torch
    bu, bp, (alpha, beta, bed, gamma), (xu, xp) = _problem(dm, n, bc)

    def at(a):
        return [_At(q, form) for q in a] if isinstance(a, list) else _At(a, form)

    coef = (at(alpha), at(beta), at(bed), at(gamma))
    yu, yp = at(xu), at(xp)
    ou, op = at(xu), at(xp)
    vu, vp = at(bu), at(xp)
    with _solver(dm, n, bc) as s:
        torch.cuda.synchronize()
        s.solve_device(at(bu), at(bp), yu, yp, *coef, 0.1 * n[0] ** 2)
        s.load_coeffs(*coef, 2.5)
        s.apply_matrix(vu, vp, ou, op)
        torch.cuda.synchronize()
    return [a.value() for a in (*yu, yp, *ou, op)]


@pytest.mark.parametrize("form", ["inside", "misaligned", "pinned"])
@pytest.mark.parametrize("dm,n,bc", CASES)
def test_arrays_anywhere_give_the_same_results(dm, n, bc, form):
    for a, b in zip(_run(dm, n, bc, "device"), _run(dm, n, bc, form)):
        assert np.isfinite(a).all() and np.abs(a).max() > 0
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("missing", ["b_u", "b_p", "x_p", "alpha", "beta", "beta_ed"])
def test_a_missing_array_is_an_error(missing):
    import torch
    from lowmachmixtures_b200.gmres import LmmError
    n = (16, 8, 12)
    bu, bp, (alpha, beta, bed, gamma), (xu, xp) = _problem(3, n, None)
    full = dict(b_u=bu, b_p=bp, x_u=xu, x_p=xp, alpha_fc=alpha, beta=beta, beta_ed=bed, gamma=gamma)
    name = {"alpha": "alpha_fc"}.get(missing, missing)
    short = dict(full)
    short[name] = [full[name][0], None, full[name][2]] if isinstance(full[name], list) else None
    with _solver(3, n, None) as s:
        torch.cuda.synchronize()
        with pytest.raises(LmmError):
            s.solve_device(**short, theta_alpha=1.0)
        assert s.solve_device(**full, theta_alpha=1.0)[2]["total_iter"] > 0


@pytest.mark.parametrize("dm,n,bc", CASES)
def test_operator_with_overlapping_arrays(dm, n, bc):
    import torch
    bu, _, coef, (xu, xp) = _problem(dm, n, bc)
    size = xp.numel()
    with _solver(dm, n, bc) as s:
        torch.cuda.synchronize()
        s.load_coeffs(*coef, 2.5)
        ref = [torch.empty_like(xp) for _ in range(dm + 1)]
        s.apply_matrix(bu, xp, ref[:dm], ref[dm])
        # in place, the components exchanged; then each output half over the next input
        x = [a.clone() for a in bu] + [xp.clone()]
        torch.cuda.synchronize()
        s.apply_matrix(x[:dm], x[dm], x[dm - 1::-1], x[dm])
        for a, b in zip(x[dm - 1::-1] + [x[dm]], ref):
            assert torch.equal(a, b)
        buf = torch.zeros((dm + 1) * size + size // 2, dtype=torch.float64, device="cuda")
        x = [buf[c * size:(c + 1) * size].view(xp.shape).copy_(a) for c, a in enumerate([*bu, xp])]
        b = [buf[size // 2 + c * size:size // 2 + (c + 1) * size] for c in range(dm + 1)]
        torch.cuda.synchronize()
        s.apply_matrix(x[:dm], x[dm], b[:dm], b[dm])
        for a, r in zip(b, ref):
            assert torch.equal(a.view(xp.shape), r)
