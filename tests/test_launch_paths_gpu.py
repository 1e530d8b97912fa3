"""Which path a size takes: V-cycle levels that run as cluster legs, by the
launches of one V-cycle."""
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
