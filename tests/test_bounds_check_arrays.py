"""The bounds-check build covers the coefficient hierarchy, the cluster legs and
the operator on the caller's arrays: their loads go through the checked helpers,
and device-array solves, coefficient loads and operators of that build report no
load out of range, with the default build's bits in FP64."""
import os
import re
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "lowmachmixtures_b200", "csrc")
P, NS, SL = -1, 100, 200
# (dm, n, bc): pairs of cells, odd counts, walls whose edge arrays have n + 1 nodes; sizes whose levels run as legs
CASES = [(2, (64, 48), None), (2, (48, 80), ((NS, NS), (NS, SL))), (3, (32, 32, 32), None), (3, (15, 9, 5), None),
         (3, (24, 48, 24), ((NS, SL), (P, P), (NS, NS)))]


def _kernel(file, name):
    """The source of one kernel, without comments."""
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, file)).read())
    start = text.index(name + "(")
    return text[start:text.index("\n}", start)]


@pytest.mark.parametrize("file,name,arrays", [
    ("coeffs.cu", "k_coeffs_fine", "alpha|beta|gamma|bed"), ("coeffs.cu", "k_coeffs_coarse", "alpha|beta|gamma|bed|pa"),
    ("coeffs.cu", "face_mean", "a"), ("coeffs.cu", "cell_mean", "a"), ("leg.cuh", "k_level_leg", "rhs")])
def test_loads_are_checked(file, name, arrays):
    body = _kernel(file, name)
    assert "__ldg" not in body
    # an element of an input read by an index instead of through ld / ldp (outputs are o_*, f_* and crhs)
    raw = re.findall(rf"(?:= *|\( *)(?:A\.)?(?:{arrays})(?:\[\w+\])?\[[^\]]*\][ ,;)]", body)
    assert not [r for r in raw if re.search(r"\]\[|A\.(beta|gamma)\[", r)], raw


def _results():
    import torch
    from lowmachmixtures_b200 import _native, abi
    from lowmachmixtures_b200.gmres import StokesSolver
    from test_caller_arrays_gpu import _problem
    res = {"library": np.array(os.path.basename(_native.load()._name))}
    for q, (dm, n, bc) in enumerate(CASES):
        bu, bp, coef, (xu, xp) = _problem(dm, n, bc)
        for tag, kw in (("fp64", {}), ("mixed", dict(method=abi.LMM_METHOD_FGMRES, precision=abi.LMM_PRECISION_FP32))):
            k = abi.make_knobs(precon_type=2, visc_type=-3, gmres_max_iter=4, gmres_max_outer=1, gmres_verbose=0, autotune=-1, **kw)
            with StokesSolver(dm, n, 1.0 / n[0], knobs=k, bc=bc) as s:
                yu, yp = [a.clone() for a in xu], xp.clone()
                torch.cuda.synchronize()
                s.solve_device(bu, bp, yu, yp, *coef, 0.1 * n[0] ** 2)
                s.load_coeffs(*coef, 2.5)
                out = [torch.empty_like(xp) for _ in range(dm + 1)]
                torch.cuda.synchronize()
                s.apply_matrix(bu, xp, out[:dm], out[dm])
                torch.cuda.synchronize()
            for c, a in enumerate([*yu, yp, *out]):
                res[f"{tag}_{q}_{c}"] = a.cpu().numpy()
    return res


@pytest.mark.gpu
def test_device_arrays_in_the_bounds_check_build(tmp_path):
    got = []
    for check in ("0", "1"):
        out = str(tmp_path / f"r{check}.npz")
        # a status other than LMM_OK (LMM_ERR_BOUNDS) raises in the child
        r = subprocess.run([sys.executable, os.path.abspath(__file__), out], env=dict(os.environ, LMM_BOUNDS_CHECK=check),
                           capture_output=True, text=True, timeout=900)
        assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
        got.append(dict(np.load(out)))
    plain, checked = got
    assert (str(plain.pop("library")), str(checked.pop("library"))) == ("liblmmstokes.so", "liblmmstokes_bc.so")
    assert set(plain) == set(checked)
    for k, a in plain.items():
        assert np.isfinite(a).all() and np.isfinite(checked[k]).all(), k
        # (mixed: contraction differs between the builds, and four iterations do not converge; the status is the check)
        if k.startswith("fp64"):
            np.testing.assert_array_equal(checked[k], a, err_msg=k)


if __name__ == "__main__":
    sys.path.insert(0, os.path.dirname(HERE))
    np.savez(sys.argv[1], **_results())
