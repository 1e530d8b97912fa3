"""A handle of a periodic box holds no face coefficients of its own on the finest
pressure level (it shares 1/alpha there); one with walls does."""
import pytest

pytestmark = pytest.mark.gpu


def _held(bc):
    import torch
    from lowmachmixtures_b200 import abi
    from lowmachmixtures_b200.gmres import StokesSolver
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    with StokesSolver(3, (96, 96, 96), 1.0 / 96, knobs=abi.make_knobs(precon_type=2, visc_type=-2, gmres_verbose=0, autotune=-1), bc=bc):
        return before - torch.cuda.mem_get_info()[0]


def test_periodic_box_shares_the_finest_pressure_coefficients():
    for _ in range(2):   # the first handles of a process also load modules
        periodic, walled = _held(None), _held(((-1, -1), (100, 100), (-1, -1)))
    # three faces in FP64 and FP32; allocations come in 2 MiB
    assert walled - periodic >= 3 * (8 + 4) * 96 ** 3 - (2 << 20)
